"""The kernels at the edges of their splits, against the FP64 oracle.

Every bin is within REL_TOL of the oracle, the bound of the FP32 path."""
import numpy as np
import pytest

from oracle import oracle as O
from rawspec_gb300 import api
from util import REL_TOL, normalized_error

pytestmark = pytest.mark.gpu


def codes(rng, shape, nbits):
    """Every code of the format, the lowest one included."""
    if nbits == 16:
        return rng.integers(-32768, 32768, shape, dtype=np.int16)
    if nbits == 4:
        return rng.integers(0, 256, shape[:-1], dtype=np.uint8)  # both components in a byte
    return rng.integers(-128, 128, shape, dtype=np.int8)


def check(Nc, Np, Ntpb, Nb, nbits, products, fft_dir=1, conj=0, buffers=1, combined=False, seed=1):
    rng = np.random.default_rng(seed)
    x = codes(rng, (Nb * buffers, Nc, Ntpb, Np, 2), nbits)
    blocks = x.view(np.uint8).reshape(Nb * buffers, -1)
    spec = api.Spectrometer(Nc, Np, Ntpb, nbits, products, Nb=Nb, conj=conj)
    try:
        spec.process(blocks, fft_dir=fft_dir, combined=combined)
        got = [np.array(d) for d in spec.dumps]
    finally:
        spec.close()
    if nbits == 4:  # first component in the high nibble
        v = x.view(np.int8)
        blocks = np.stack([v >> 4, (v << 4).view(np.int8) >> 4], -1).view(np.uint8).reshape(Nb * buffers, -1)
    cfg = O.make_cfg(Nc, Np, Ntpb, Nb, max(nbits, 8), products, conj=conj, inverse=1 if fft_dir <= 0 else 0)
    ref, _ = O.run_oracle(cfg, blocks)
    for i, (nt, na, npol) in enumerate(products):
        assert got[i].shape == ref[i].shape
        err = normalized_error(got[i], ref[i], npol, Nc, nt)
        assert err < REL_TOL, (nt, na, npol, err)


# One polarisation: spectra in pairs, with odd and single counts; lengths on
# both sides of a change of the values per thread.
@pytest.mark.parametrize("nbits", [8, 16])
@pytest.mark.parametrize("nt", [4, 8, 16, 32, 64, 256, 512, 1024, 2048, 4096])
def test_pairs_of_spectra(cuda_device, monkeypatch, nt, nbits):
    monkeypatch.setenv("RAWSPEC_GB300_TENSOR_DFT", "0")
    for na, nd in ((1, 3), (5, 3), (8, 2)):
        check(3, 1, nt * na * nd, 1, nbits, [(nt, na, 1)], fft_dir=-1 if na == 5 else 1, conj=1, seed=nt + na)


# Units on one CTA, on a pair, on a cluster of up to eight, on more CTAs than a
# cluster holds; the last chunk shorter than the others; two products of a
# buffer; a launch with fewer units than the GPU has SMs and one with more.
@pytest.mark.parametrize("Nc,nt,na,nd,npol", [(1, 2048, 2, 1, 4), (4, 2048, 8, 1, 4), (4, 4096, 7, 1, -4),
                                              (3, 1024, 13, 2, 1), (2, 512, 61, 1, -4), (1, 64, 997, 1, 4),
                                              (1, 8, 20011, 1, 1), (1, 16, 4099, 2, -4), (64, 2048, 6, 3, 4),
                                              (40, 4096, 11, 5, 1)])
def test_units_over_ctas(cuda_device, monkeypatch, Nc, nt, na, nd, npol):
    monkeypatch.setenv("RAWSPEC_GB300_TENSOR_DFT", "0")
    check(Nc, 2, nt * na * nd, 1, 8, [(nt, na, npol), (nt // 2, 2 * na, npol)], fft_dir=-1 if na % 2 else 1, seed=na)


# Two-kernel path: every split of the length, the staged rows (at most two
# spectra) and the direct ones, pairs of rows for one polarisation, odd counts.
@pytest.mark.parametrize("Np,npol", [(2, 1), (2, 4), (2, -4), (1, 1)])
@pytest.mark.parametrize("logn", [13, 14, 15, 16, 17, 18])
def test_two_kernel_lengths(cuda_device, logn, Np, npol):
    nt = 1 << logn
    for na, Nc in ((1, 3), (3, 2)) if logn < 17 else ((3, 1),):
        check(Nc, Np, nt * na, 1, 16 if logn == 15 else 8, [(nt, na, npol)], fft_dir=-1 if na == 1 else 1, seed=logn)


# Small copies, gathered by a kernel: rows on and off the 16-byte grid, 4-bit
# samples, the block limit of a launch and one more, separate and combined
# calls, an integration over two buffers.
@pytest.mark.parametrize("combined", [False, True])
@pytest.mark.parametrize("Np,nbits,Ntpb,Nb", [(2, 8, 64, 1), (1, 8, 33, 8), (1, 4, 33, 8), (2, 4, 40, 16),
                                              (2, 16, 5, 16), (1, 8, 8, 17), (1, 4, 8, 17)])
def test_small_copies(cuda_device, Np, nbits, Ntpb, Nb, combined):
    total = Ntpb * Nb
    check(5, Np, Ntpb, Nb, nbits, [(8, 2 * total // 8, 1)], buffers=2, combined=combined, seed=Ntpb)


# Units of one group of threads, which writes its sums itself: one spectrum a
# unit, written and added over two buffers, and a chunk of one iteration.
@pytest.mark.parametrize("npol", [1, 4])
@pytest.mark.parametrize("nt", [1, 2, 8, 16, 32, 64, 512, 1024, 4096])
def test_units_of_one_group(cuda_device, monkeypatch, nt, npol):
    monkeypatch.setenv("RAWSPEC_GB300_TENSOR_DFT", "0")
    check(5, 2, nt, 1, 8, [(nt, 2, npol)], buffers=4, fft_dir=-1, conj=1, seed=nt)
    check(3, 2, 3 * nt, 1, 16, [(nt, 1, npol)], seed=nt + 1)
    check(70, 2, 2 * nt, 1, 8, [(nt, 2, npol)], seed=nt + 2)


# Fewer units than a CTA has sets of groups: their sums are shared out over all
# of its threads, written and added, on one CTA and on more.
@pytest.mark.parametrize("npol", [1, -4])
@pytest.mark.parametrize("Nc,nt,na", [(1, 32, 4), (3, 32, 2), (5, 8, 4), (1, 64, 8), (2, 256, 3), (9, 16, 6), (1, 512, 2),
                                      (1, 128, 300), (3, 16, 700)])
def test_few_units(cuda_device, monkeypatch, Nc, nt, na, npol):
    monkeypatch.setenv("RAWSPEC_GB300_TENSOR_DFT", "0")
    check(Nc, 2, nt * na, 1, 8, [(nt, 2 * na, npol)], buffers=4, fft_dir=-1 if na % 2 else 1, conj=1, seed=nt)
    check(Nc, 2, nt * na, 1, 16, [(nt, na, npol)], seed=nt + 1)


# Units whose partial sums a kernel of its own adds, alone and in shared launches
# (one channel, four planes), written and added.
@pytest.mark.parametrize("nt,na,npol", [(4096, 64, 4), (2048, 70, -4), (4096, 129, 1)])
def test_units_summed_by_a_kernel(cuda_device, monkeypatch, nt, na, npol):
    monkeypatch.setenv("RAWSPEC_GB300_TENSOR_DFT", "0")
    check(1, 2, nt * na, 1, 8, [(nt, 2 * na, npol)], buffers=4, fft_dir=-1, conj=1, seed=na)
    rng = np.random.default_rng(na)
    blocks = [codes(rng, (1, 1, nt * na, 2, 2), 8).view(np.uint8).reshape(1, -1) for _ in range(2)]
    specs = [api.Spectrometer(1, 2, nt * na, 8, [(nt, na, npol)], Nb=1) for _ in blocks]
    try:
        alone = []
        for spec, b in zip(specs, blocks):
            spec.process(b)
            alone.append(np.array(spec.dumps[0]))
            spec.load_blocks(b)
            spec.copy_to_gpu()
        before = specs[0].kernel_launches()
        api.start_group(specs, [1, 1])
        for spec in specs:
            assert spec.wait() == 0
        assert specs[0].kernel_launches() - before == 2  # the shared launch and the sum
        for spec, a in zip(specs, alone):
            assert np.array_equal(np.array(spec.dumps[0])[-1:], a[-1:])
    finally:
        for spec in specs:
            spec.close()


# A copy goes by the kernel or by the copy engines, whichever is the faster; the
# bytes are the same.
@pytest.mark.parametrize("Nc,Np,nbits,Ntpb,Nb,kernels", [(2, 1, 8, 262143, 1, 0), (3, 2, 8, 4096, 1, 0), (3, 2, 8, 4096, 4, 1),
                                                         (3, 1, 8, 4095, 16, 1), (5, 2, 4, 4096, 1, 1), (5, 1, 4, 262143, 1, 0),
                                                         (30000, 1, 8, 8, 4, 0), (600, 1, 8, 63, 4, 1)])
def test_small_copies_by_kernel_or_engine(cuda_device, Nc, Np, nbits, Ntpb, Nb, kernels):
    spec = api.Spectrometer(Nc, Np, Ntpb, nbits, [(1, Ntpb * Nb, 1)], Nb=Nb)
    try:
        spec.copy_to_gpu()
        before = spec.kernel_launches()
        spec.copy_to_gpu()
        launched = spec.kernel_launches() - before
    finally:
        spec.close()
    # the engines' copies of 4-bit samples are followed by their expansion
    assert launched == (1 if nbits == 4 else kernels)
    check(Nc, Np, Ntpb, Nb, nbits, [(1, Ntpb * Nb, 1)], buffers=1, seed=Ntpb)
