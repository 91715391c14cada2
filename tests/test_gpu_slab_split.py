"""The correlation's transform along a where a block splits it over its warps (k_slab_split: columns of
128 points, and 64-point columns of 128 to a slab), against a float64 inverse FFT, and its values against the
shared-memory transform's bits; 64-point columns of 64 to a slab against the FFT too (GPU only).

Tolerance: a value is a sum of L terms f·V·e with Σ|f V| <= s, through log2(n) stages of single-precision
butterflies: |error| <= 2 (log2 n + 2) 2^-24 s for its column's s, scaled by rden.
"""
import ctypes
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _sp():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _tw():
    t = -2j * math.pi * torch.arange(1024, dtype=torch.float64) / 1024
    return torch.view_as_real(torch.exp(t).to(torch.complex64)).contiguous().cuda()


def _dims(L, fold):
    from zebsdsolve_b200 import _native as N

    n = 16
    while n < 2 * L - 1:
        n *= 2
    return N.So3Dims(L, n, n // 2 + 1, n // fold, fold, (L - 1) // fold, L * (L + 1) // 2)


def _peaks(U, n, d, rden, div):
    from zebsdsolve_b200 import _native as N

    peaks = torch.zeros(n, 8, device="cuda")
    scratch = torch.empty(N.load().zeb_peaks_scratch_bytes(ctypes.byref(d), n), dtype=torch.uint8, device="cuda")
    N.call("zeb_correlate_peaks", _p(U), n, ctypes.byref(d), _p(_tw()), _p(rden), div, _p(peaks), _p(scratch), _sp())
    return peaks


@pytest.mark.parametrize("L,fold,n,div", [(128, 4, 5, 1 << 30), (65, 4, 3, 2), (92, 2, 2, 1), (64, 2, 9, 1 << 30),
                                          (33, 1, 4, 3), (64, 1, 3, 1 << 30)])
def test_split_transform_finds_the_volume_s_largest_value(L, fold, n, div):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d = _dims(L, fold)
    g = torch.Generator(device="cuda")
    g.manual_seed(L * 8 + fold)
    U = torch.randn(n, d.nb, L, d.nc, 2, device="cuda", generator=g)
    volumes = -(-n // min(div, n))
    rden = torch.rand(volumes, d.nb, d.nc, d.n, device="cuda", generator=g) + 0.5
    rden.view(-1)[::13] = 0
    peaks = _peaks(U, n, d, rden, div)
    V = torch.view_as_complex(U.double()).transpose(2, 3)  # [b][j][c][m']
    pad = torch.zeros(n, d.nb, d.nc, d.n // 2 + 1, dtype=torch.complex128, device="cuda")
    pad[..., :L] = V.conj()
    which = torch.arange(n, device="cuda") // min(div, n)
    vol = torch.fft.irfft(pad, n=d.n, dim=-1) * d.n * rden[which].double()
    s = 2 * V.abs().sum(-1) * 1.5  # (rden <= 1.5)
    tol = float(2 * (math.log2(d.n) + 2) * 2.0 ** -24 * s.max())
    best = vol.reshape(n, -1).max(1).values
    assert (peaks[:, 4].double() - best).abs().max() <= tol
    # the cell the angles round to holds that value
    k = torch.round(peaks[:, 5:8].double() * d.n / (2 * math.pi)).long()
    at = vol[torch.arange(n, device="cuda"), k[:, 1], k[:, 2] % d.nc, k[:, 0] % d.n]
    assert (at - best).abs().max() <= 2 * tol


@pytest.mark.parametrize("L,fold", [(128, 4), (64, 1)])
def test_split_transform_keeps_the_first_of_equal_values(L, fold):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d = _dims(L, fold)
    U = torch.zeros(2, d.nb, L, d.nc, 2, device="cuda")
    U[..., 0, :, 0] = 1.0  # the volume is 1 everywhere, -1 for the second item
    U[1] *= -1
    rden = torch.ones(d.nb, d.nc, d.n, device="cuda")
    rden[0, 0, :3] = 0.5
    peaks = _peaks(U, 2, d, rden, 1 << 30).cpu().numpy()
    step = 2 * math.pi / d.n
    # first among 1's past the damped cells; first among the -0.5's (the largest of the negatives)
    assert abs(peaks[0, 4] - 1) < 1e-6 and np.allclose(peaks[0, 5:8], [3 * step, 0, 0], atol=0.51 * step)
    assert abs(peaks[1, 4] + 0.5) < 1e-6 and np.allclose(peaks[1, 6:8], 0, atol=1e-6) and peaks[1, 5] <= 0.51 * step


@pytest.mark.parametrize("L,fold,n,div", [(128, 4, 5, 1 << 30), (65, 4, 6, 4), (80, 2, 3, 1), (92, 2, 2, 1 << 30),
                                          (33, 1, 4, 3), (64, 1, 3, 1 << 30)])
def test_split_transform_gives_the_shared_memory_transform_s_bits(L, fold, n, div):
    """Every slab's candidate is the largest of zeb_correlate_volume's values (k_slab, the transform that a
    slab of these sizes took before) times its denominators: the same stages with the same twiddles."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zebsdsolve_b200 import _native as N

    d = _dims(L, fold)
    g = torch.Generator(device="cuda")
    g.manual_seed(L * 16 + fold)
    U = torch.randn(n, d.nb, L, d.nc, 2, device="cuda", generator=g)
    volumes = -(-n // min(div, n))
    rden = torch.rand(volumes, d.nb, d.nc, d.n, device="cuda", generator=g) + 0.5
    vol = torch.empty(n, d.nb, d.nc, d.n, device="cuda")
    tw = _tw()
    N.call("zeb_correlate_volume", _p(U), n, ctypes.byref(d), _p(tw), _p(vol), _sp())
    want = (vol * rden[torch.arange(n, device="cuda") // min(div, n)]).reshape(n, d.nb, -1)
    peaks = torch.zeros(n, 8, device="cuda")
    scratch = torch.empty(N.load().zeb_peaks_scratch_bytes(ctypes.byref(d), n), dtype=torch.uint8, device="cuda")
    N.call("zeb_correlate_peaks", _p(U), n, ctypes.byref(d), _p(tw), _p(rden), div, _p(peaks), _p(scratch), _sp())
    key = scratch.view(torch.int32).view(n, d.nb, 2).cpu().numpy().view(np.uint32)
    top = key[..., 1]
    value = np.where(top >> 31 == 1, top ^ np.uint32(1 << 31), ~top).astype(np.uint32).view(np.float32)
    index = (~key[..., 0]).astype(np.int64) - np.arange(d.nb) * d.nc * d.n
    best = want.max(-1).values
    assert np.array_equal(value, best.cpu().numpy())
    at = want.gather(2, torch.as_tensor(index, device="cuda")[..., None])[..., 0]
    assert torch.equal(at, best) and torch.equal(peaks[:, 4], best.max(1).values)
