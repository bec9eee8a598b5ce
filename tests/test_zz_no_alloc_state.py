"""The allocation-free entry point keeps nothing but its twiddle tables between
calls: calls of other splits, streams and captured graphs in a row, against the
FP64 oracle."""
import ctypes as C
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from rawspec_gb300 import api
from test_zz_no_alloc import _blocks, entry, oracle_path
from util import REL_TOL, normalized_error

pytestmark = pytest.mark.gpu

# long integrations of few channels, split over many CTAs, and of more channels
CALLS = [
    dict(Nc=1, Np=2, nbits=8, Ntpb=262144, nt=8, na=32768, npol=4, conj=0, fft_dir=1, seed=61),
    dict(Nc=3, Np=2, nbits=8, Ntpb=131072, nt=2048, na=64, npol=-4, conj=1, fft_dir=-1, seed=62),
    dict(Nc=2, Np=1, nbits=16, Ntpb=65536, nt=64, na=1024, npol=1, conj=0, fft_dir=1, seed=63),
    dict(Nc=40, Np=2, nbits=8, Ntpb=16384, nt=256, na=64, npol=1, conj=0, fft_dir=-1, seed=64),
]


class Call:
    def __init__(self, f, c):
        import torch
        self.f, self.c = f, c
        blocks = _blocks(c)
        self.d_in = torch.from_numpy(blocks[0].copy()).cuda()
        nd = c["Ntpb"] // (c["nt"] * c["na"])
        self.out = torch.full((nd * abs(c["npol"]) * c["Nc"] * c["nt"],), float("nan"), dtype=torch.float32, device="cuda")
        self.ref = oracle_path(blocks, c)[None, :]

    def __call__(self, stream):
        c = self.c
        return self.f(C.c_void_p(self.d_in.data_ptr()), c["Nc"], c["Np"], c["nbits"], c["Ntpb"], c["nt"], c["na"],
                      c["npol"], c["fft_dir"], c["conj"], C.cast(C.c_void_p(self.out.data_ptr()), C.POINTER(C.c_float)),
                      C.c_void_p(stream.cuda_stream))

    def check(self):
        c = self.c
        err = normalized_error(self.out.cpu().numpy()[None, :], self.ref, c["npol"], c["Nc"], c["nt"])
        assert err < REL_TOL, (c, err)
        self.out.fill_(float("nan"))


def test_calls_on_changing_streams(cuda_device):
    import torch
    calls = [Call(entry(api.load_library()), c) for c in CALLS]
    streams = [torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    for i in range(3 * len(calls)):
        call, s = calls[i % len(calls)], streams[i % len(streams)]
        torch.cuda.synchronize()
        assert call(s) == 0
        torch.cuda.synchronize()
        call.check()


def test_captured_calls_between_others(cuda_device):
    import torch
    calls = [Call(entry(api.load_library()), c) for c in CALLS]
    assert calls[3](torch.cuda.current_stream()) == 0  # tables filled
    graphs = []
    for call in calls[:2]:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            assert call(torch.cuda.current_stream()) == 0
        graphs.append(g)
    for _ in range(3):
        for g, call in zip(graphs, calls):
            g.replay()
            torch.cuda.synchronize()
            call.check()
        assert calls[2](torch.cuda.current_stream()) == 0
        torch.cuda.synchronize()
        calls[2].check()


FIRST_CAPTURED = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
import torch
from rawspec_gb300 import api
from test_zz_no_alloc import entry
from test_zz_no_alloc_state import CALLS, Call
f = entry(api.load_library())
calls = [Call(f, c) for c in CALLS]
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, capture_error_mode="relaxed"):
    assert calls[1](torch.cuda.current_stream()) == 0
for k in (0, 2, 3):  # replays before and after the calls that fill the tables
    g.replay()
    torch.cuda.synchronize()
    calls[1].check()
    assert calls[k](torch.cuda.current_stream()) == 0
    torch.cuda.synchronize()
    calls[k].check()
print("ok")
"""


def test_first_call_of_a_process_captured(cuda_device):
    """It fills a table of its own in the graph."""
    tests = Path(__file__).resolve().parent
    res = subprocess.run([sys.executable, "-c", FIRST_CAPTURED.format(root=str(tests.parent), tests=str(tests))],
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "ok" in res.stdout, res.stderr[-2000:]
