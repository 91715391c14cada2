"""The slab entry points called on tensors, and what their results are held to (for the tests of the
correlation's transform along a)."""
import ctypes
import math

import numpy as np
import torch


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def twiddles():
    t = -2j * math.pi * torch.arange(1024, dtype=torch.float64) / 1024
    return torch.view_as_real(torch.exp(t).to(torch.complex64)).contiguous().cuda()


def dims(L, fold):
    from zebsdsolve_b200 import _native as N

    n = 16
    while n < 2 * L - 1:
        n *= 2
    return N.So3Dims(L, n, n // 2 + 1, n // fold, fold, (L - 1) // fold, L * (L + 1) // 2)


def peaks(U, n, d, rden, div):
    """zeb_correlate_peaks: the peaks [n, 8] and the scratch with every slab's candidate."""
    from zebsdsolve_b200 import _native as N

    out = torch.zeros(n, 8, device="cuda")
    scratch = torch.empty(N.load().zeb_peaks_scratch_bytes(ctypes.byref(d), n), dtype=torch.uint8, device="cuda")
    N.call("zeb_correlate_peaks", ptr(U), n, ctypes.byref(d), ptr(twiddles()), ptr(rden), div, ptr(out), ptr(scratch),
           stream())
    return out, scratch


def volume(U, n, d, guard=0):
    """zeb_correlate_volume [n, nb, nc, n], and `guard` floats of 9 past its end."""
    from zebsdsolve_b200 import _native as N

    count = n * d.nb * d.nc * d.n
    vol = torch.full((count + guard,), 9.0, device="cuda")
    N.call("zeb_correlate_volume", ptr(U), n, ctypes.byref(d), ptr(twiddles()), ptr(vol), stream())
    return vol[:count].view(n, d.nb, d.nc, d.n), vol[count:]


def exact_volume(U, d):
    """The volume by a float64 inverse FFT, and each column's Σ|V|."""
    V = torch.view_as_complex(U.double()).transpose(2, 3)  # [b][j][c][m']
    pad = torch.zeros(*V.shape[:3], d.n // 2 + 1, dtype=torch.complex128, device="cuda")
    pad[..., :d.L] = V.conj()
    return torch.fft.irfft(pad, n=d.n, dim=-1) * d.n, V.abs().sum(-1)


def inputs(L, fold, n, div, seed):
    """U [n, nb, L, nc, 2] and the denominators [volumes, nb, nc, n]."""
    d = dims(L, fold)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    U = torch.randn(n, d.nb, L, d.nc, 2, device="cuda", generator=g)
    rden = torch.rand(-(-n // min(div, n)), d.nb, d.nc, d.n, device="cuda", generator=g) + 0.5
    return d, U, rden


def check_largest(L, fold, n, div):
    """An item's peak is its volume's largest value. A value is a sum of L terms f·V·e with Σ|f V| <= s, through
    log2(n) stages of single-precision butterflies: |error| <= 2 (log2 n + 2) 2^-24 s for its column's s, scaled
    by rden (<= 1.5)."""
    d, U, rden = inputs(L, fold, n, div, L * 8 + fold)
    rden.view(-1)[::13] = 0
    got, _ = peaks(U, n, d, rden, div)
    vol, size = exact_volume(U, d)
    which = torch.arange(n, device="cuda") // min(div, n)
    vol = vol * rden[which].double()
    tol = float(2 * (math.log2(d.n) + 2) * 2.0 ** -24 * (2 * size * 1.5).max())
    best = vol.reshape(n, -1).max(1).values
    assert (got[:, 4].double() - best).abs().max() <= tol
    # the cell the angles round to holds that value
    k = torch.round(got[:, 5:8].double() * d.n / (2 * math.pi)).long()
    at = vol[torch.arange(n, device="cuda"), k[:, 1], k[:, 2] % d.nc, k[:, 0] % d.n]
    assert (at - best).abs().max() <= 2 * tol


def split_candidates(scratch, n, d):
    """k_slab_split's candidates: (value, index within the slab's own nc·n cells, −1 for none) [n, nb]."""
    key = scratch.view(torch.int32).view(n, d.nb, 2).cpu().numpy().view(np.uint32)
    top, low = key[..., 1], key[..., 0]
    value = np.where(top >> 31 == 1, top ^ np.uint32(1 << 31), ~top).astype(np.uint32).view(np.float32)
    index = (~low).astype(np.int64) - np.arange(d.nb) * d.nc * d.n
    return value, np.where(low == 0, -1, index)


def check_split_bits(U, rden, n, d, div):
    """Every slab's candidate is the first largest of zeb_correlate_volume's values (k_slab, the transform that a
    slab of these sizes took before) times its denominators, NaN passed over: the same stages with the same
    twiddles."""
    vol, _ = volume(U, n, d)
    want = (vol * rden[torch.arange(n, device="cuda") // min(div, n)]).reshape(n, d.nb, -1)
    want = torch.nan_to_num(want, nan=-math.inf, posinf=math.inf, neginf=-math.inf)
    got, scratch = peaks(U, n, d, rden, div)
    value, index = split_candidates(scratch, n, d)
    best = want.max(-1).values
    none = (best <= -3.4e38).cpu().numpy()
    assert np.array_equal(value, np.where(none, np.float32(-3.4e38), best.cpu().numpy()))
    assert np.array_equal(index == -1, none)
    at = want.gather(2, torch.as_tensor(np.maximum(index, 0), device="cuda")[..., None])[..., 0]
    some = torch.as_tensor(~none, device="cuda")
    assert torch.equal(at[some], best[some])
    items = some.any(1)
    assert torch.equal(got[items, 4], best.max(1).values[items])
    return got
