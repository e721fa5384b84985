// The dense field solve of uniformly refined Cartesian runs (a5g_uniform.cu).
#ifndef A5_UNIFORM_H
#define A5_UNIFORM_H
#include "a5_internal.h"

struct A5Uniform;
// What a solve works on: the run's slots, the applied potential and the
// multigrid schedule (mixed: that of the FP32 correction solve).
struct A5UniformArgs {
  double *cc, *fx, *fy;
  long long capacity;
  double voltage;
  int n_cycle_base;
  bool mixed;
  int fmg, sw_down, sw_up, sw_base, n_corr;  // cycles
};
// The dense levels of a topology, or null where it is not uniform (or too
// large for their 32-bit indices, or without memory): the box phases serve.
// Its tables are uploaded on the run's stream, which does not order with the
// default stream.
A5Uniform *a5u_build(const A5Topo &topo, const double *lv_dr, void *stream);
void a5u_destroy(A5Uniform *u);
// Settings or storage behind a captured solve have changed.
void a5u_changed(A5Uniform *u);
bool a5u_ready(A5Uniform *u, const A5UniformArgs &a, void *stream);
int a5u_solve(A5Uniform *u, bool mixed, void *stream);  // a cudaError_t
#endif
