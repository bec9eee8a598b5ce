"""Rounding errors of the products against NumPy's FFT in 64 bits.

The tolerance of the parity tests is a hundred times the rounding of an FP32
transform; these tests hold the rounding itself."""
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
