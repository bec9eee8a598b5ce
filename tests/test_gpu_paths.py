"""Each long-FFT kernel on inputs that its rule sends to it, against the FP64 oracle.

Every test asserts which kernel computed the product: the fused four-step
kernel takes three transforms or more of two 8-bit polarisations, one a unit."""
import numpy as np
import pytest

from oracle import oracle as O
from rawspec_gb300 import api
from test_gpu_edges import codes
from util import REL_TOL, normalized_error

pytestmark = pytest.mark.gpu


def check_kernel(kernel, Nc, Np, Ntpb, nbits, product, buffers=1, fft_dir=1, conj=0, seed=1):
    nt, na, npol = product
    rng = np.random.default_rng(seed)
    blocks = codes(rng, (buffers, Nc, Ntpb, Np, 2), nbits).view(np.uint8).reshape(buffers, -1)
    spec = api.Spectrometer(Nc, Np, Ntpb, nbits, [product], Nb=1, conj=conj)
    try:
        assert spec.product_kernel(0) == kernel
        spec.process(blocks, fft_dir=fft_dir)
        got = np.array(spec.dumps[0])
    finally:
        spec.close()
    cfg = O.make_cfg(Nc, Np, Ntpb, 1, nbits, [product], conj=conj, inverse=1 if fft_dir <= 0 else 0)
    ref = O.run_oracle(cfg, blocks)[0][0]
    assert got.shape == ref.shape
    err = normalized_error(got, ref, npol, Nc, nt)
    print(f"2^{nt.bit_length() - 1} {kernel}: {err:.2e}")
    assert err < REL_TOL


# Two-kernel path above 2^18: columns of 512 to 4096 points (staged, and read
# directly at 2048 and 4096), rows of up to 4096, results written directly
# (three spectra a unit) and staged (one).
@pytest.mark.parametrize("logn,Np,nbits,npol,na", [(19, 2, 16, 1, 3), (20, 1, 8, 1, 3), (20, 2, 8, -4, 3),
                                                   (20, 2, 16, 4, 1), (21, 2, 16, -4, 1), (21, 1, 16, 1, 3),
                                                   (21, 2, 8, 1, 3), (22, 2, 16, 4, 1), (22, 1, 8, 1, 1),
                                                   (22, 2, 16, 1, 2), (23, 1, 16, 1, 1), (23, 2, 8, -4, 1),
                                                   (24, 1, 8, 1, 1), (24, 2, 16, 1, 1)])
def test_two_kernel_long_lengths(cuda_device, logn, Np, nbits, npol, na):
    nt = 1 << logn
    check_kernel("large_a", 1, Np, nt * na, nbits, (nt, na, npol), fft_dir=-1 if logn % 2 else 1, conj=1, seed=logn)


# The fused kernel at every split and radix it has, written and added over two
# buffers, total power and four planes; 2^18 and 2^19 in total power are the
# lengths at which 32 values a thread begin.
@pytest.mark.parametrize("npol", [1, 4, -4])
@pytest.mark.parametrize("logn", [16, 17, 18, 19, 20, 21])
def test_fused_lengths(cuda_device, logn, npol):
    nt = 1 << logn
    check_kernel("large_fused", 3, 2, nt, 8, (nt, 2, npol), buffers=2, fft_dir=-1 if logn % 2 else 1, conj=1, seed=logn)


# Rows of one spectrum staged in shared memory, two polarisations.
@pytest.mark.parametrize("npol", [1, 4])
@pytest.mark.parametrize("logn", [16, 18])
def test_two_kernel_single_spectra(cuda_device, logn, npol):
    nt = 1 << logn
    check_kernel("large_a", 2, 2, nt, 8, (nt, 2, npol), buffers=2, fft_dir=-1, conj=1, seed=logn)


# Compensated integration from the fused kernel's staging plane (its output map
# of its own), and from the two-kernel path's.
@pytest.mark.parametrize("Nc,kernel", [(3, "large_fused"), (1, "large_a")])
@pytest.mark.parametrize("npol", [1, 4])
def test_compensation_of_long_products(cuda_device, monkeypatch, Nc, kernel, npol):
    nt = 1 << 16
    dumps = []
    for kahan in ("1", "0"):
        monkeypatch.setenv("RAWSPEC_GB300_KAHAN", kahan)
        check_kernel(kernel, Nc, 2, nt, 8, (nt, 6, npol), buffers=6, seed=npol)
        rng = np.random.default_rng(9)
        blocks = codes(rng, (6, Nc, nt, 2, 2), 8).view(np.uint8).reshape(6, -1)
        with api.Spectrometer(Nc, 2, nt, 8, [(nt, 6, npol)], Nb=1) as spec:
            spec.set_profiling(True)
            spec.process(blocks)
            dumps.append(np.array(spec.dumps[0]))
            assert spec.profile(api.KERNEL_CLASS_NAMES.index("merge"))[1] == (5 if kahan == "1" else 0)
    assert normalized_error(dumps[0], dumps[1].astype(np.float64), npol, Nc, nt) < 1e-6
