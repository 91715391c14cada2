"""The correlation's transform along a where a block splits it over its warps (k_slab_split: columns of
128 points, and 64-point columns of 128 to a slab), against a float64 inverse FFT, and its values against the
shared-memory transform's bits; 64-point columns of 64 to a slab against the FFT too (GPU only; the tolerances
stand in slab_calls).
"""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
FOR_ALL = 1 << 30


@pytest.fixture(autouse=True)
def device():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("L,fold,n,div", [(128, 4, 5, FOR_ALL), (65, 4, 3, 2), (92, 2, 2, 1), (64, 2, 9, FOR_ALL),
                                          (33, 1, 4, 3), (64, 1, 3, FOR_ALL)])
def test_split_transform_finds_the_volume_s_largest_value(L, fold, n, div):
    import slab_calls as sc

    sc.check_largest(L, fold, n, div)


@pytest.mark.parametrize("L,fold", [(128, 4), (64, 1)])
def test_split_transform_keeps_the_first_of_equal_values(L, fold):
    import slab_calls as sc

    d = sc.dims(L, fold)
    U = torch.zeros(2, d.nb, L, d.nc, 2, device="cuda")
    U[..., 0, :, 0] = 1.0  # the volume is 1 everywhere, -1 for the second item
    U[1] *= -1
    rden = torch.ones(d.nb, d.nc, d.n, device="cuda")
    rden[0, 0, :3] = 0.5
    peaks = sc.peaks(U, 2, d, rden, FOR_ALL)[0].cpu().numpy()
    step = 2 * math.pi / d.n
    # first among 1's past the damped cells; first among the -0.5's (the largest of the negatives)
    assert abs(peaks[0, 4] - 1) < 1e-6 and np.allclose(peaks[0, 5:8], [3 * step, 0, 0], atol=0.51 * step)
    assert abs(peaks[1, 4] + 0.5) < 1e-6 and np.allclose(peaks[1, 6:8], 0, atol=1e-6) and peaks[1, 5] <= 0.51 * step


@pytest.mark.parametrize("L,fold,n,div", [(128, 4, 5, FOR_ALL), (65, 4, 6, 4), (80, 2, 3, 1), (92, 2, 2, FOR_ALL),
                                          (33, 1, 4, 3), (64, 1, 3, FOR_ALL)])
def test_split_transform_gives_the_shared_memory_transform_s_bits(L, fold, n, div):
    import slab_calls as sc

    d, U, rden = sc.inputs(L, fold, n, div, L * 16 + fold)
    sc.check_split_bits(U, rden, n, d, div)


@pytest.mark.parametrize("L,fold", [(128, 4), (64, 1)])
def test_values_that_are_not_finite(L, fold):
    """NaN is passed over as before; an item of nothing else has no candidate and gives the volume's first cell.
    An infinity stays with its own slab."""
    import slab_calls as sc

    n = 5
    d, U, rden = sc.inputs(L, fold, n, FOR_ALL, L + fold)
    U[1, 4, 7, 3, 0] = math.nan  # one column
    U[2] = math.nan
    rden[0, 2] = 0
    got = sc.check_split_bits(U, rden, n, d, FOR_ALL)
    assert bool((got[2, 4] == -3.4e38) & (got[2, 5:8].abs() <= 1.001 * math.pi / d.n).all())
    clean = [sc.split_candidates(sc.peaks(U, n, d, rden, FOR_ALL)[1], n, d)][0]
    U[3, 6, 1, 9, 1] = math.inf
    peaks, scratch = sc.peaks(U, n, d, rden, FOR_ALL)
    value, index = sc.split_candidates(scratch, n, d)
    assert ((index >= -1) & (index < d.nc * d.n)).all() and bool(torch.isfinite(peaks[3, 5:8]).all())
    others = np.ones((n, d.nb), bool)
    others[3, 6] = False
    assert np.array_equal(value[others], clean[0][others]) and np.array_equal(index[others], clean[1][others])
