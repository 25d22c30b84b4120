"""The allocation-free step beside the rest of the process: a wait that gave up elsewhere
is still reported after it (its kernel has no waits of its own), and the first
call of a process may be captured."""
import pathlib
import subprocess
import sys

import pytest
import torch

from comcot_b200 import _lib
from test_zz_no_alloc import _buffers, _case, _two_calls

pytestmark = pytest.mark.gpu

GC_ETIMEOUT = -5


def test_noalloc_step_keeps_a_raised_timeout():
    lib = _lib.load()
    bufs = _buffers([_case(97, 81, 61)], torch.device("cuda", 0))
    stream = torch.cuda.current_stream().cuda_stream
    lib.gcomcot_sync()
    assert lib.gcomcot_inject_timeout() == 0
    torch.cuda.synchronize()
    _two_calls(lib, bufs, stream)
    torch.cuda.synchronize()
    assert lib.gcomcot_sync() == GC_ETIMEOUT
    _two_calls(lib, bufs, stream)
    torch.cuda.synchronize()
    assert lib.gcomcot_sync() == 0


FIRST_CALL_CAPTURED = """
import sys
sys.path[:0] = {paths!r}
import numpy as np, torch
from comcot_b200 import _lib
from test_zz_no_alloc import _buffers, _case, _results, _two_calls
lib, dev = _lib.load(), torch.device("cuda", 0)
cases = [_case(150, 70, 62)]
a, b = _buffers(cases, dev), _buffers(cases, dev)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    _two_calls(lib, a, torch.cuda.current_stream().cuda_stream)
g.replay()
_two_calls(lib, b, torch.cuda.current_stream().cuda_stream)
torch.cuda.synchronize()
x, y = _results(a[0]), _results(b[0])
assert all(np.array_equal(x[k].view(np.uint32), y[k].view(np.uint32)) for k in x)
"""


def test_first_call_of_a_process_inside_a_capture():
    here = pathlib.Path(__file__).resolve().parent
    paths = [str(here), str(here.parent / "gpu-comcot_b200"), str(here.parent / "oracle")]
    p = subprocess.run([sys.executable, "-c", FIRST_CALL_CAPTURED.format(paths=paths)], capture_output=True, text=True,
                       timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
