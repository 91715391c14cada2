"""The FP32 form's spectrum on the tensor cores (zeb_spectrum_x2) against the float64 product, beside the
plain FP32 kernel's error on the same operands (GPU only).

Bounds: its error is no larger than k_spectrum_f32's, relative to the result's 2-norm (what the split is
taken for); a single value is off by at most the dropped 2^-22 of |g|·|Y| summed over its terms and the
accumulator's truncation, 2^-23 a step of 16 terms: (2^-22 + K/16 · 3 · 2^-23) Σ|g||Y|.
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


def _dims(L, fold):
    from zebsdsolve_b200 import _native as N

    n = 16
    while n < 2 * L - 1:
        n *= 2
    return N.So3Dims(L, n, n // 2 + 1, n // fold, fold, (L - 1) // fold, L * (L + 1) // 2)


# (K a whole number of blocks and not; one pattern tile, a ragged second, the largest bandwidth)
@pytest.mark.parametrize("L,fold,n", [(24, 4, 5), (33, 4, 129), (64, 4, 200), (64, 2, 127), (48, 1, 40), (97, 4, 10),
                                      (128, 4, 17)])
def test_split_spectrum_is_as_exact_as_fp32(L, fold, n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zebsdsolve_b200 import _native as N

    d = _dims(L, fold)
    cols = d.nb * d.nc
    g = torch.Generator(device="cuda")
    g.manual_seed(L + n)
    l = torch.cat([torch.arange(m, L) for m in range(L)]).cuda()
    alm = torch.randn(n, d.n_pairs, 2, device="cuda", generator=g) / (1 + l)[None, :, None]  # a pattern's decay
    alm = (alm / alm.flatten(1).norm(dim=1)[:, None, None]).contiguous()
    Y = torch.randn(d.n_pairs, cols, 2, device="cuda", generator=g, dtype=torch.float64) / (1 + l)[:, None, None]
    scale = 2.0 ** math.floor(math.log2(16384 / float(Y.abs().max())))
    A = torch.empty(N.load().zeb_x2_master_bytes(ctypes.byref(d)), dtype=torch.uint8, device="cuda")
    B = torch.empty(N.load().zeb_x2_patterns_bytes(ctypes.byref(d), n), dtype=torch.uint8, device="cuda")
    N.call("zeb_x2_pack_master", ctypes.byref(d), _p(Y), scale, _p(A), _sp())
    guard = 4096
    U = torch.full((n * d.nb * L * d.nc * 2 + guard,), 9.0, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    N.call("zeb_spectrum_x2", _p(alm), n, ctypes.byref(d), _p(A), scale, _p(B), _p(U), _p(status), _sp())
    plain = torch.empty(n * d.nb * L * d.nc * 2, device="cuda")
    Yf = Y.float().contiguous()
    N.call("zeb_spectrum_f32", _p(alm), n, ctypes.byref(d), _p(Yf), _p(plain), _sp())
    assert int(status) == 0 and bool((U[-guard:] == 9.0).all())
    U = U[:-guard].view(n, d.nb, L, d.nc, 2)
    plain = plain.view(n, d.nb, L, d.nc, 2)
    gc, Yc = torch.view_as_complex(alm.double()), torch.view_as_complex(Y)
    split = fp32 = 0.0
    for m in range(L):
        p0 = m * L - m * (m - 1) // 2
        a, y = gc[:, p0:p0 + L - m], Yc[p0:p0 + L - m]
        want = torch.view_as_real((a.conj() @ y).view(n, d.nb, d.nc))
        size = (alm[:, p0:p0 + L - m].double().abs().sum(-1) @ Y[p0:p0 + L - m].abs().sum(-1)).view(n, d.nb, d.nc, 1)
        off = (U[:, :, m].double() - want).abs()
        steps = math.ceil(2 * (L - m) / 64) * 4
        assert bool((off <= (2.0 ** -22 + 3 * steps * 2.0 ** -23) * size).all())
        split += float((off ** 2).sum())
        fp32 += float(((plain[:, :, m].double() - want) ** 2).sum())
    assert split <= fp32


def test_split_spectrum_refuses_what_it_cannot_take():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zebsdsolve_b200 import _native as N

    x = torch.zeros(64, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    for L in (8, 23, 129, 160):
        d = _dims(L, 4)
        assert N.load().zeb_x2_master_bytes(ctypes.byref(d)) == 0
        with pytest.raises(N.NativeError, match="unsupported dims"):
            N.call("zeb_spectrum_x2", _p(x), 1, ctypes.byref(d), _p(x), 1.0, _p(x), _p(x), _p(st), _sp())
