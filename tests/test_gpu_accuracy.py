"""Rounding errors of the products against NumPy's FFT in 64 bits.

The tolerance of the parity tests is a hundred times the rounding of an FP32
transform; these tests hold the rounding itself."""
from fractions import Fraction

import numpy as np
import pytest

from rawspec_gb300 import api

pytestmark = pytest.mark.gpu


def rms_error(Nc, Np, nt, na, npol, nbits=8, buffers=1, seed=11):
    """RMS error of the first plane (both of a full-polarisation product) over the RMS total power, `na` spectra
    in each of `buffers` buffers."""
    rng = np.random.default_rng(seed)
    lim, sigma = (32767, 2500.0) if nbits == 16 else (127, 20.0)
    x = np.clip(np.rint(rng.normal(0.0, sigma, (buffers, Nc, nt * na, Np, 2))), -lim, lim)
    x = x.astype(np.int16 if nbits == 16 else np.int8)
    spec = api.Spectrometer(Nc, Np, nt * na, nbits, [(nt, na * buffers, npol)], Nb=1)
    try:
        spec.process(x.view(np.uint8).reshape(buffers, -1))
        got = np.array(spec.dumps[0], np.float64).reshape(abs(npol), Nc, nt)
    finally:
        spec.close()
    ref = np.zeros((2, Nc, nt))
    for b in x:
        for c in range(Nc):
            z = b[c].astype(np.float64) / lim
            z = (z[..., 0] + 1j * z[..., 1]).reshape(na, nt, Np)
            p = np.abs(np.fft.fftshift(np.fft.fft(z, axis=1), axes=1)) ** 2
            for q in range(Np):
                ref[q, c] += p[..., q].sum(0)
    total = ref.sum(0)
    scale = np.sqrt(np.mean(total ** 2))
    err = got[:2] - ref if npol == 4 else got[:1] - total
    return float(np.sqrt(np.mean(err ** 2)) / scale)


# The bounds are 1.1 times the errors measured with twiddles of separately
# rounded cosines and sines; with tangents rounded by themselves they were 1.2
# times these.
@pytest.mark.parametrize("nt,na,npol,before", [(256, 16, 4, 4.43e-8), (256, 4, -4, 9.11e-8), (2048, 16, 4, 5.02e-8)])
def test_twiddles_add_no_error(cuda_device, nt, na, npol, before):
    err = rms_error(64, 2, nt, na, npol)
    print(f"{nt} points, {na} spectra, Npolout {npol}: {err:.2e}")
    assert err < 1.1 * before


def f32(x):
    """The float32 nearest to an exact value (a Fraction)."""
    y = np.float32(float(x))
    near = [np.nextafter(y, np.float32(-np.inf)), y, np.nextafter(y, np.float32(np.inf))]
    return min(near, key=lambda v: (abs(Fraction(float(v)) - x), int(v.view(np.int32)) & 1))


# A buffer's sum enters the running sum of the two-kernel path with one rounding.
# Constant voltages show every one of them: bin 0 of a transform is N times the
# code, times 128/127 in the twiddles; its square, the sum of the spectra and the
# running sum round, the scale 2^-14 does not.  (With the scale 1/127^2 as a
# float the product with it rounded as well.)
@pytest.mark.parametrize("Nc,logn,na,fft_dir", [(1, 16, 1, 1), (1, 16, 1, -1), (1, 16, 3, 1), (2, 13, 3, -1), (1, 20, 2, 1)])
def test_sums_are_added_with_one_rounding(cuda_device, Nc, logn, na, fft_dir):
    nt = 1 << logn
    f = f32(Fraction(128, 127))
    for c1, c2 in ((1, 3), (7, 43), (10, 92), (37, 120), (64, 43), (118, 106)):
        x = np.zeros((2, Nc, nt * na, 1, 2), np.int8)
        x[0, ..., 0], x[1, ..., 1] = c1, c2
        spec = api.Spectrometer(Nc, 1, nt * na, 8, [(nt, 2 * na, 1)], Nb=1)
        try:
            assert spec.product_kernel(0) == "large_a"
            spec.process(x.view(np.uint8).reshape(2, -1), fft_dir=fft_dir)
            got = np.array(spec.dumps[0]).reshape(Nc, nt)
        finally:
            spec.close()
        sums = []
        for c in (c1, c2):
            v = f32(Fraction(float(f)) * c)
            p, s = f32(Fraction(float(v)) ** 2), np.float32(0)
            for _ in range(na):
                s = f32(Fraction(float(s)) + Fraction(float(p)))
            sums.append(Fraction(float(s)))
        want = float(f32(sum(sums))) * nt ** 2 / 2 ** 14
        assert np.all(got[:, nt // 2] == want), (c1, c2, got[:, nt // 2], want)
