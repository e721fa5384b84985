"""The 3D form's dense multigrid (every level one colour-split grid, the
coarsest ones in one block) against the oracle, bit for bit, on base grids
and levels where its pieces change: one base box and several, odd counts,
coarse levels too large for the one-block section (no such section at all on
the largest base grid here), a finest level right above it."""
import numpy as np
import pytest

import a5ref
from a5_streamer_b200 import config, device3
from test_gpu_3d import _compare, _upload

pytestmark = pytest.mark.gpu

# n_base, level: (1,1,1) 1 has its whole coarse hierarchy in one warp;
# (5,5,5) keeps level 0 (8,000 cells) out of the one-block section, (9,8,8)
# every level (4,608 cells on the coarsest)
SHAPES = [((1, 1, 1), 1), ((1, 1, 1), 2), ((1, 1, 1), 4), ((2, 1, 3), 2), ((3, 2, 1), 3), ((1, 7, 2), 2),
          ((5, 5, 5), 1), ((9, 8, 8), 1)]


def _cfg(n_base, level):
    return config.cube_16mm_uniform(level, n_base=n_base, domain_len=tuple(16e-3 * n for n in n_base))


def _pair(n_base, level, eps=True):
    """A run in the oracle's initial state; eps False: the permittivity as
    set_init_cond leaves it (known to be 1, which the fused transport needs)
    instead of uploaded."""
    cfg = _cfg(n_base, level)
    sim = a5ref.Sim3(cfg, n_threads=8)
    sim.init()
    rc, xmin, inv, n = sim.table()
    run = device3.Run3(cfg, table=(rc, xmin, inv, n))
    if eps:
        _upload(sim, run)
    else:
        run.set_init_cond()
        for iv in range(8):
            run.set_cc(iv, sim.cc(iv))
        for d in range(3):
            for f in range(2):
                run.set_fc(d, f, sim.fc(d, f))
    return cfg, sim, run


@pytest.mark.parametrize("n_base,level", SHAPES)
def test_field_solve_from_any_state(n_base, level):
    """compute_fld from random potentials, densities and |E| (ghost, edge and
    corner entries too): all slots of all variables as the reference leaves
    them."""
    cfg, sim, run = _pair(n_base, level)
    rng = np.random.default_rng(3)
    for iv, scale in ((0, 1e15), (1, 1e15), (4, 1e3), (5, 1e6), (6, 1e8)):
        x = sim.cc(iv)
        x[:] = scale * (rng.random(x.shape) - 0.5)
        sim.set_cc(iv, x)
        run.set_cc(iv, sim.cc(iv))
    for _ in range(2):
        sim.op("compute_fld", 0)
        run.compute_fld(False)
    run.sync()
    _compare(sim, run, f"{n_base} level {level}")


@pytest.mark.parametrize("n_base,level", SHAPES)
@pytest.mark.parametrize("eps", [True, False])
def test_steps_parity(n_base, level, eps):
    """Whole steps from a state whose densities vary in every cell and whose
    ghost entries agree with no neighbour; between steps a change of n_e by
    the caller, which the next step has to see."""
    cfg, sim, run = _pair(n_base, level, eps)
    rng = np.random.default_rng(4)
    dt = sim.get_max_dt()
    for k in range(3):
        for iv in (0, 1) if k == 0 else (0,):
            x = sim.cc(iv)
            x *= 1 + 0.2 * rng.random(x.shape)
            sim.set_cc(iv, x)
            run.set_cc(iv, sim.cc(iv))
        sim.step(dt)
        run.step(dt)
    run.sync()
    _compare(sim, run, f"{n_base} level {level}")


@pytest.mark.parametrize("n_base,level", SHAPES)
def test_mixed_steps_fused_equals_plain(n_base, level):
    """The mixed form's steps through the fused transport (eps known to be 1)
    and through the box-slot kernels (eps uploaded)."""
    runs = [_pair(n_base, level, eps)[2] for eps in (True, False)]
    for r in runs:
        r.set_precision(True)
        dt = r.get_max_dt()
        for _ in range(3):
            r.step(dt)
        r.sync()
    for iv in range(9):
        assert np.array_equal(runs[0].cc(iv), runs[1].cc(iv)), iv
    for d in range(3):
        for f in range(2):
            assert np.array_equal(runs[0].fc(d, f), runs[1].fc(d, f)), (d, f)


def test_step_after_eps_is_written():
    """A captured step does not outlive a write of eps (a dielectric region:
    n_e moves into n_i there), nor the return to eps = 1."""
    cfg, sim, run = _pair((1, 1, 1), 2, eps=False)
    dt = sim.get_max_dt()
    for val in (None, 2.0):
        if val:
            x = sim.cc(8)
            x[:, ::7] = val
            sim.set_cc(8, x)
            run.set_cc(8, sim.cc(8))
            sim.op("fld_from_pot")
            run.op("fld_from_pot")
        sim.step(dt)
        run.step(dt)
        if val:
            # the oracle's multigrid keeps eps operators out of the 3D form; compare the transport
            _compare(sim, run, f"eps {val}", ivs=(0, 1, 2, 3), faces=False)
        else:
            _compare(sim, run, "eps 1")


class _Emulated:
    """The mixed form's FP32 correction solve on dense grids in numpy, every
    operation rounded to float32 in the order of the reference's expressions
    (afivo/src/m_aX_mg.f90:208-255, 430-549, 714-848): arrays [z, y, x] with
    one layer of ghost cells, wall value 0."""

    def __init__(self, n_base, level, dr_base):
        self.lo, self.hi = -1, level
        self.n, self.dx2, self.inv, self.p, self.f, self.o = {}, {}, {}, {}, {}, {}
        for l in range(self.lo, level + 1):
            m = 8 * 2 ** (l - 1) if l >= 1 else 8 >> (1 - l)
            self.n[l] = tuple(k * m for k in n_base[::-1])
            h = dr_base * 0.5 ** (l - 1)
            self.dx2[l], self.inv[l] = np.float32(h * h), np.float32(1 / (h * h))
            self.p[l], self.f[l], self.o[l] = (np.zeros([k + 2 for k in self.n[l]], np.float32) for _ in range(3))

    @staticmethod
    def sides(a):
        """The six neighbours of the cells, x- x+ y- y+ z- z+."""
        c = slice(1, -1)
        return (a[c, c, :-2], a[c, c, 2:], a[c, :-2, c], a[c, 2:, c], a[:-2, c, c], a[2:, c, c])

    @staticmethod
    def fill(a):
        a[:, :, 0], a[:, :, -1] = a[:, :, 1], a[:, :, -2]
        a[:, 0], a[:, -1] = a[:, 1], a[:, -2]
        a[0], a[-1] = -a[1], np.float32(0) - a[-2]

    def lpl(self, a, l):
        xm, xp, ym, yp, zm, zp = self.sides(a)
        return self.inv[l] * (((((xm + xp) + ym) + yp) + zm) + zp - np.float32(6) * a[1:-1, 1:-1, 1:-1])

    def smooth(self, l, cycles):
        par = np.indices(self.n[l]).sum(0) & 1
        for it in range(2 * cycles):
            self.fill(self.p[l])
            xm, xp, ym, yp, zm, zp = self.sides(self.p[l])
            s = ((((xp + xm) + yp) + ym) + zp) + zm
            new = np.float32(1 / 6.0) * (s - self.dx2[l] * self.f[l][1:-1, 1:-1, 1:-1])
            c = self.p[l][1:-1, 1:-1, 1:-1]
            c[par == (it & 1)] = new[par == (it & 1)]
        self.fill(self.p[l])

    @staticmethod
    def restrict(a):
        s = a[0::2, 0::2, 0::2]
        for k in range(1, 8):
            s = s + a[(k >> 2)::2, ((k >> 1) & 1)::2, (k & 1)::2]
        return a.dtype.type(0.125) * s

    def down(self, l):
        i = (slice(1, -1),) * 3
        r = self.restrict(self.f[l][i] - self.lpl(self.p[l], l))
        self.p[l - 1][i] = self.restrict(self.p[l][i])
        self.fill(self.p[l - 1])
        self.f[l - 1][i] = self.lpl(self.p[l - 1], l - 1) + r
        self.o[l - 1] = self.p[l - 1].copy()

    def correct(self, l):
        c = self.p[l - 1] - self.o[l - 1]
        i1 = [(np.arange(1, k + 1) + 1) >> 1 for k in self.n[l]]
        i2 = [a + 1 - 2 * (np.arange(1, k + 1) & 1) for a, k in zip(i1, self.n[l])]
        at = lambda z, y, x: c[np.ix_(z, y, x)]
        s = at(i1[0], i1[1], i1[2]) + at(i1[0], i1[1], i2[2])
        s = s + at(i1[0], i2[1], i1[2])
        s = s + at(i2[0], i1[1], i1[2])
        v = self.p[l][1:-1, 1:-1, 1:-1]
        v[...] = v + np.float32(0.25) * s
        self.fill(self.p[l])

    def cycle(self, top, sched):
        for l in range(top, self.lo, -1):
            self.smooth(l, sched[1])
            self.down(l)
        self.smooth(self.lo, sched[3])
        for l in range(self.lo + 1, top + 1):
            self.correct(l)
            self.smooth(l, sched[2])

    def solve(self, res, sched):
        i = (slice(1, -1),) * 3
        self.f[self.hi][i] = res.astype(np.float32)
        if sched[0] == 0:
            return self.cycle(self.hi, sched)
        for l in range(self.hi, self.lo, -1):
            self.f[l - 1][i] = self.restrict(self.f[l][i])
        for l in range(self.lo, self.hi + 1):
            self.o[l] = self.p[l].copy()
            if l > self.lo:
                self.correct(l)
            self.cycle(l, sched)


def _dense(run, meta, ids, x):
    """The cells of one level's boxes as one array [z, y, x]."""
    nc = int(meta[ids[0], 20])
    g = nc + 2
    at = (meta[ids, 2:5] - 1) * nc
    out = np.zeros((at.max(0) + nc)[::-1])
    for id_, (a, b, c) in zip(ids, at):
        out[c:c + nc, b:b + nc, a:a + nc] = x[id_, :g ** 3].reshape(g, g, g)[1:-1, 1:-1, 1:-1]
    return out


@pytest.mark.parametrize("n_base,level", SHAPES)
@pytest.mark.parametrize("schedule", [(1, 2, 2, 8, 1), (0, 1, 1, 4, 1), (1, 3, 1, 2, 1)])
def test_mixed_solve_equals_emulation(n_base, level, schedule):
    cfg, sim, run = _pair(n_base, level)
    run.set_precision(True, schedule)
    meta, levels = run.meta(), run.levels()
    phi, e, p = run.cc(4), run.cc(0), run.cc(1)
    run.compute_fld(False)
    new = run.cc(4)
    em = _Emulated(n_base, level, cfg.dr_base)
    hi = levels[level][0]
    a = np.pad(_dense(run, meta, hi, phi), 1)
    em.fill(a)
    a[-1] = 2 * cfg.applied_voltage - a[-2]
    xm, xp, ym, yp, zm, zp = em.sides(a)
    dr = cfg.dr_at(level)
    lap = (1 / (dr * dr)) * (((((xm + xp) + ym) + yp) + zm) + zp - 6 * a[1:-1, 1:-1, 1:-1])
    rhs = 1.6022e-19 / 8.8541878176e-12 * (_dense(run, meta, hi, e) - _dense(run, meta, hi, p))
    em.solve(rhs - lap, schedule)
    for l in range(run.min_lvl, level + 1):
        want = _dense(run, meta, levels[l][0], phi) + em.p[l][1:-1, 1:-1, 1:-1].astype(np.float64)
        assert np.array_equal(_dense(run, meta, levels[l][0], new), want), f"level {l}"
