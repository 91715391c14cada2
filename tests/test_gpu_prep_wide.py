"""The wide blur from tables made once a call (k_prep_wide) against the general kernel (k_prep), which a
scratch pointer on an 8-byte boundary only still takes: the same sums in the same order, so the same bits
(GPU only)."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# (stored h, w, patterns, pixel type, factor): two boxes a cell and more, sizes that leave short last boxes,
# not square, one pattern, reduced, an image too large for two blocks an SM
CASES = [(80, 80, 3, 0, 1.0), (83, 101, 5, 1, 1.0), (60, 160, 2, 2, 1.0), (161, 120, 3, 1, 1.0), (96, 96, 1, 2, 1.0),
         (170, 190, 3, 1, 2.0), (240, 250, 4, 1, 2.5), (210, 200, 2, 0, 1.0)]


@pytest.mark.parametrize("h,w,n,pixel,factor", CASES)
@pytest.mark.parametrize("dynamic,normalize", [(1, 1), (2, 1), (1, 0), (3, 0)])
def test_wide_blur_tables_give_the_general_kernel_s_bits(h, w, n, pixel, factor, dynamic, normalize):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zebsdsolve_b200 import _native as N

    def p(t, off=0):
        return ctypes.c_void_p(t.data_ptr() + off)

    g = torch.Generator(device="cuda")
    g.manual_seed(h * w + dynamic)
    raw = torch.rand(n, h, w, device="cuda", generator=g) * 250
    raw = raw.to(torch.uint8) if pixel == 0 else raw.to(torch.int32).to(torch.uint16) if pixel == 1 else raw
    if pixel == 2 and n > 1:
        raw[0, 3, 5] = float("inf")  # a bad pixel reaches the cells it reached, no others
        raw[1, 7, 2] = float("nan")
    oh, ow = int(h / factor + 1e-9), int(w / factor + 1e-9)
    bg = torch.rand(oh, ow, device="cuda", generator=g) * 100
    sigma = max(0.15 * ow, 12.5)
    r = 0.5 * min(oh, ow)
    mask = (ctypes.c_float * 3)(0.5 * (oh - 1), 0.5 * (ow - 1), r * r)
    scratch = torch.zeros(N.load().zeb_prep_scratch_bytes(n, oh, ow, sigma) + 16, dtype=torch.uint8, device="cuda")
    out = []
    for off in (0, 8):
        o = torch.zeros(n * oh * ow, device="cuda")
        N.call("zeb_prep_reduced", p(raw), pixel, n, h, w, factor, p(bg), dynamic, sigma, mask, normalize, p(o),
               p(scratch, off), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        out.append(o)
    a, b = out
    assert torch.equal(torch.isnan(a), torch.isnan(b))
    assert torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
