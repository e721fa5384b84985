"""The device code's set-up work (no GPU needed). Runs and batches own
non-blocking streams, which do not order with the default stream, so nothing
that their kernels read may be copied or cleared on the default stream: a
clear, or a copy from pageable memory, may return before the device has it."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEFAULT_STREAM = re.compile(r"\bcudaMem(?:cpy|cpy2D|cpy3D|cpyToSymbol|cpyFromSymbol|set|set2D|set3D)\s*\(")
ON_STREAM_0 = re.compile(r"\bcudaMem(?:cpy|set)\w*Async\s*\([^;]*,\s*(?:0|nullptr|cudaStreamLegacy)\s*\)\s*[;)!=]")


def _code(path):
    src = open(path).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return re.sub(r"//[^\n]*", "", src)


def test_no_set_up_on_the_default_stream():
    files = [f for ext in ("cu", "cuh", "cpp", "h")
             for f in glob.glob(os.path.join(ROOT, "a5_streamer_b200", "csrc", "*." + ext))]
    assert len(files) >= 5
    bad = []
    for f in files:
        text = _code(f)
        bad += [(os.path.basename(f), m.group(0)) for p in (DEFAULT_STREAM, ON_STREAM_0) for m in p.finditer(text)]
        # every run's and batch's stream is a non-blocking one
        assert not re.search(r"\bcudaStreamCreate\s*\(", text), f
    assert not bad, bad
