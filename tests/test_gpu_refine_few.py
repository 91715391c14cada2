"""The refinement over a pixel list, few patterns to a launch and many (more threads' registers, and for the longest
lists the pattern's values in shared memory, against more patterns an SM): the same sums in the same order, so
the same bits (GPU only)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# (h, w, the launches' patterns): lists of 256 threads (from 4 609 pixels; many from 445 and from 889) and of
# 512 (from 9 217 to the longest taken; many from 149), and one of 128, which has one form
CASES = [(60, 60, (3, 200)), (80, 80, (3, 444, 445, 600, 889)), (108, 108, (1, 444, 445)), (110, 110, (2, 148, 149)),
         (160, 160, (2, 148, 149)), (180, 180, (1, 150))]


@pytest.mark.parametrize("h,w,counts", CASES)
@pytest.mark.parametrize("form", ["zeb_refine_list", "zeb_refine_list_h"])
def test_few_and_many_patterns_give_the_same_records(h, w, counts, form):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zebsdsolve_b200 import _native as N

    def p(t):
        return ctypes.c_void_p(t.data_ptr())

    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    g = torch.Generator(device="cuda")
    g.manual_seed(h)
    side, held = 101, 16
    sheets = torch.randn(2, side, side, device="cuda", generator=g)
    grad = torch.empty(2 * side * side * 4, device="cuda")
    N.call("zeb_master_gradient", p(sheets), p(grad), side, stream)
    vpair, gpair = torch.empty(2 * side * side * 2, device="cuda"), torch.empty(2 * side * side * 8, device="cuda")
    N.call("zeb_master_pairs", p(sheets), p(grad), side, p(vpair), p(gpair), stream)
    quads = torch.empty(2 * side * side * 32, dtype=torch.uint8, device="cuda")
    N.call("zeb_master_quads", p(grad), side, p(quads), stream)
    fr = N.Frame()
    fr.h, fr.w = h, w
    fr.c0[:], fr.c1[:], fr.c2[:] = (0.0, 0.01, 0.0), (0.01, 0.0, 0.0), (0.0, 0.0, 0.01)
    fr.mask[:] = (0.5 * (h - 1), 0.5 * (w - 1), (0.5 * min(h, w)) ** 2)
    npix = N.load().zeb_mask_pixels(ctypes.byref(fr))
    lst = torch.empty(npix, dtype=torch.int32, device="cuda")
    N.call("zeb_mask_list", ctypes.byref(fr), p(lst), stream)
    pats = torch.randn(held, h * w, device="cuda", generator=g)
    pats = (pats / pats.norm(dim=1, keepdim=True)).contiguous()
    o = N.RefineOpts()
    for k, v in dict(iters=6, max_step=0.05, scale0=1.0, scale_min=0.02, scale_max=1e4, nmi_bins=16, stamp=1.0).items():
        setattr(o, k, v)
    which = torch.arange(max(counts), device="cuda") % held
    items = torch.tensor([-0.005 * w, -0.005 * h, 0.006 * h, 0.0], device="cuda").repeat(len(which), 1)
    items[:, 3] = which
    q = torch.randn(held, 4, device="cuda", generator=g)
    q = (q / q.norm(dim=1, keepdim=True))[which].contiguous()
    table = gpair if form == "zeb_refine_list" else quads
    got = []
    for n in counts:
        rec = torch.full((n, 8), float("nan"), device="cuda")
        N.call(form, p(pats), p(items), p(q), 4, n, ctypes.byref(fr), p(lst), npix, p(vpair), p(table), side, ctypes.byref(o),
               p(rec), stream)
        got.append(rec.cpu().numpy())
    assert np.isfinite(got[-1]).all() and (got[-1][:, 4] > -1).all()
    for rec in got:
        assert np.array_equal(rec, got[-1][np.arange(len(rec)) % held])
