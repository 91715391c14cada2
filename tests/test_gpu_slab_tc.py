"""The tensor-core transform along a (k_slab_tc: one group of epilogue warps for columns of 128 points, two
for shorter ones), each slab's candidate against a float64 inverse transform (GPU only).

Tolerance: a value is Σ f·V·e with e rounded to FP16 (2^-12 of 1 at most: |e| <= 1) and FP32 accumulation of
exact products that may truncate (2^-23 of the running sum a term, 2L terms): |error| <= (2^-11.5 + 2L 2^-23) s
for s = Σ f (|Re V| + |Im V|), scaled by rden, whose own rounding (2^-23 of the value) the margin holds.
"""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("L,fold,items", [(16, 4, 1), (16, 1, 300), (32, 4, 129), (32, 2, 700), (64, 4, 127),
                                          (64, 2, 260), (64, 1, 2)])
def test_every_slab_s_candidate(L, fold, items):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zebsdsolve_b200 import _native as N

    n, nb, nc = 2 * L, L + 1, 2 * L // fold
    d = N.So3Dims(L, n, nb, nc, fold, (L - 1) // fold, L * (L + 1) // 2)
    g = torch.Generator(device="cuda")
    g.manual_seed(L * 8 + fold)
    tiles = -(-items // 128)
    U = torch.randn(tiles, nb, nc, L, 2, 128, device="cuda", generator=g).half()
    rden = torch.rand(nb, nc, n, device="cuda", generator=g) + 0.5
    rden.view(-1)[::13] = 0
    scratch = torch.empty(N.load().zeb_peaks_scratch_bytes(ctypes.byref(d), items), dtype=torch.uint8, device="cuda")
    peaks = torch.zeros(items, 8, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    N.call("zeb_correlate_peaks_h", _p(U), items, ctypes.byref(d), 4.0, _p(rden), _p(peaks), _p(scratch), _p(status),
           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert int(status.item()) == 0

    cand = scratch[: items * nb * 8].view(items, nb, 2, 4)
    value = cand[:, :, 0].contiguous().view(torch.float32)[..., 0].double()
    index = cand[:, :, 1].contiguous().view(torch.int32)[..., 0].long()
    V = U.permute(0, 5, 1, 2, 3, 4).reshape(tiles * 128, nb, nc, L, 2)[:items].double() / 4.0
    f = torch.full((L,), 2.0, dtype=torch.float64, device="cuda")
    f[0] = 1.0
    angle = 2 * torch.pi * torch.arange(L, device="cuda", dtype=torch.float64)[:, None] * torch.arange(
        n, device="cuda", dtype=torch.float64) / n
    bound = 2.0 ** -11.5 + 2 * L * 2.0 ** -23
    for i in range(0, items, 32):
        v = V[i:i + 32]
        vol = torch.einsum("pjcm,ma->pjca", v[..., 0] * f, angle.cos()) + torch.einsum(
            "pjcm,ma->pjca", v[..., 1] * f, angle.sin())
        tol = (v.abs().sum(-1) * f).sum(-1)[..., None] * rden.double() * bound
        vol, tol = (vol * rden.double()).reshape(v.shape[0], nb, -1), tol.reshape(v.shape[0], nb, -1)
        at = index[i:i + 32] - torch.arange(nb, device="cuda") * nc * n
        assert bool(((at >= 0) & (at < nc * n)).all())
        got = value[i:i + 32]
        there = vol.gather(2, at[..., None])[..., 0]
        near = tol.gather(2, at[..., None])[..., 0]
        assert bool(((got - there).abs() <= near).all()), float(((got - there).abs() / near).max())
        assert bool((got >= (vol - tol).amax(-1)).all())
