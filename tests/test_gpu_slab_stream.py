"""The correlation's transform along a with the next slab on its way (k_slab_stream: 32 or 64 columns
of 64 points to a slab, one denominator volume) against the kernel that holds its loads in
registers (k_slab_cols, which U on an 8-byte boundary takes): the same arithmetic in the same order, so the same
bits; 64 columns also against the float64 transform, as test_gpu_slab_split has it (GPU only).
"""
import ctypes

import pytest
import test_gpu_slab_split as split

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("L,n,fold", [(64, 1, 4), (64, 13, 4), (33, 200, 4), (63, 77, 4), (48, 300, 4), (64, 700, 4),
                                      (64, 40, 2), (35, 9, 2)])
def test_streamed_slabs_give_the_same_peaks(L, n, fold):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zebsdsolve_b200 import _native as N

    nc = 128 // fold
    d = N.So3Dims(L, 128, 65, nc, fold, (L - 1) // fold, L * (L + 1) // 2)
    g = torch.Generator(device="cuda")
    g.manual_seed(L * 1000 + n)
    count = n * 65 * L * nc * 2
    both = torch.empty(count + 4, device="cuda")
    U = torch.randn(count, device="cuda", generator=g)
    rden = torch.rand(65 * nc * 128, device="cuda", generator=g) + 0.5
    rden[::13] = 0
    t = -2j * torch.pi * torch.arange(1024, dtype=torch.float64) / 1024
    tw = torch.view_as_real(torch.exp(t).to(torch.complex64)).contiguous().cuda()
    got = []
    for shift in (0, 2):  # floats: a 16-byte boundary, and an 8-byte one
        u = both[shift:shift + count]
        u.copy_(U)
        assert u.data_ptr() % 16 == 4 * shift
        scratch = torch.empty(N.load().zeb_peaks_scratch_bytes(ctypes.byref(d), n), dtype=torch.uint8, device="cuda")
        peaks = torch.zeros(n, 8, device="cuda")
        N.call("zeb_correlate_peaks", _p(u), n, ctypes.byref(d), _p(tw), _p(rden), 1 << 30, _p(peaks), _p(scratch),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        got.append((peaks, scratch[: n * 65 * 8].clone()))
    assert torch.equal(got[0][1], got[1][1])
    assert torch.equal(got[0][0], got[1][0])


@pytest.mark.parametrize("L,n", [(64, 1), (33, 30), (63, 13), (48, 40)])
def test_sixty_four_columns(L, n):
    split.test_split_transform_finds_the_volume_s_largest_value(L, 2, n, 1 << 30)
