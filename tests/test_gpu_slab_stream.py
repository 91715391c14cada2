"""The correlation's transform along a with the next slab on its way (k_slab_stream: 32 or 64 columns of 64 points
to a slab, one denominator volume) against the kernel that holds its loads in registers (k_slab_cols, which U
on an 8-byte boundary takes): the same arithmetic in the same order, so the same bits; 64 columns also against
the float64 transform (GPU only; its tolerance stands in slab_calls).
"""
import math

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def device():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _both(U, n, d, rden):
    """The peaks and candidates of U on a 16-byte boundary and on an 8-byte one."""
    import slab_calls as sc

    held = torch.empty(U.numel() + 4, device="cuda")
    got = []
    for shift in (0, 2):  # floats
        u = held[shift:shift + U.numel()]
        u.copy_(U.reshape(-1))
        assert u.data_ptr() % 16 == 4 * shift
        peaks, scratch = sc.peaks(u, n, d, rden, 1 << 30)
        got.append((peaks.view(torch.int32), scratch))
    return got


@pytest.mark.parametrize("L,n,fold", [(64, 1, 4), (64, 13, 4), (33, 200, 4), (63, 77, 4), (48, 300, 4), (64, 700, 4),
                                      (64, 40, 2), (35, 9, 2)])
def test_streamed_slabs_give_the_same_peaks(L, n, fold):
    import slab_calls as sc

    d, U, rden = sc.inputs(L, fold, n, 1 << 30, L * 1000 + n)
    rden.view(-1)[::13] = 0
    a, b = _both(U, n, d, rden)
    assert torch.equal(a[1], b[1]) and torch.equal(a[0], b[0])


@pytest.mark.parametrize("fold", [4, 2])
def test_values_that_are_not_finite(fold):
    import slab_calls as sc

    n = 6
    d, U, rden = sc.inputs(64, fold, n, 1 << 30, fold)
    U[1, 4, 7, 3, 0] = math.nan  # one column
    U[2] = math.nan
    U[3, 6, 1, 9, 1] = math.inf
    U[4, 6, 0, 9, 0] = -math.inf
    rden[0, 2] = 0
    a, b = _both(U, n, d, rden)
    assert torch.equal(a[1], b[1]) and torch.equal(a[0], b[0])


@pytest.mark.parametrize("L,n", [(64, 1), (33, 30), (63, 13), (48, 40)])
def test_sixty_four_columns(L, n):
    import slab_calls as sc

    sc.check_largest(L, 2, n, 1 << 30)
