"""Slabs wider than one block's shared memory (bandwidths above 92 with a two-fold master, above 64 without a
fold): the volume by groups of columns against a float64 inverse FFT, and a two-fold master indexed at L = 128
(GPU only).

Tolerance of the volume: as slab_calls has it, 2 (log2 n + 2) 2^-24 of its column's 2 Σ|V|; of the orientations:
test_gpu_configs' for the same bandwidth.
"""
import ctypes
import math
import tempfile

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def device():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("L,fold,n", [(93, 2, 2), (128, 2, 3), (65, 1, 2), (128, 1, 1), (92, 2, 1), (64, 1, 2)])
def test_the_volume_of_a_wide_slab(L, fold, n):
    import slab_calls as sc

    d, U, _ = sc.inputs(L, fold, n, 1 << 30, L + fold)
    vol, past = sc.volume(U, n, d, guard=4096)
    assert bool((past == 9.0).all())
    want, size = sc.exact_volume(U, d)
    tol = 2 * (math.log2(d.n) + 2) * 2.0 ** -24 * 2 * size[..., None]
    assert bool(((vol.double() - want).abs() <= tol).all())


@pytest.mark.parametrize("L,fold,n,div", [(128, 2, 3, 1 << 30), (93, 2, 4, 2), (65, 1, 2, 1)])
def test_the_peaks_of_a_wide_slab(L, fold, n, div):
    import slab_calls as sc

    d, U, rden = sc.inputs(L, fold, n, div, L * 16 + fold)
    sc.check_split_bits(U, rden, n, d, div)


def test_slabs_without_a_split_stay_refused():
    import slab_calls as sc
    from zebsdsolve_b200 import _native as N

    x = torch.zeros(64, device="cuda")
    d = sc.dims(160, 4)  # 256-point columns, 128 of them
    with pytest.raises(N.NativeError, match="shared memory"):
        N.call("zeb_correlate_volume", sc.ptr(x), 1, ctypes.byref(d), sc.ptr(x), sc.ptr(x), sc.stream())
    with pytest.raises(N.NativeError, match="shared memory"):
        sc.peaks(x, 1, d, x, 1)


@pytest.mark.parametrize("precision", ["f32", "bf16"])
def test_a_two_fold_master_at_bandwidth_128(precision):
    import zebsdsolve_b200 as ze
    from zebsdsolve_b200 import synthetic as syn
    from zebsdsolve_b200.master import write_npz

    path = tempfile.mkdtemp() + "/m.npz"
    sheets = syn.master_sheets(3, side=401, lmax=96, group="622", device="cuda")
    write_npz(path, sheets, 401, syn.group_matrices("622"), syn.POINT_GROUP["622"])
    s = ze.Solver()
    s.configure(static_background="none", dynamic_background="none", bandwidth=128, precision=precision)
    s.add_phase(path)
    s.set_patterns(np.zeros((3, 5, 60, 60), np.float32))
    s.set_geometry(pc=(0.5, 0.3, 0.6), sample_tilt_deg=70, detector_tilt_deg=0)
    rng = np.random.default_rng(21)
    q = syn.uniform_quaternions(rng, 15)
    pats = s.simulate(q, cells=np.arange(15), phase=0).reshape(15, 60, 60)
    pats = pats + 0.5 * pats.std() * rng.normal(size=pats.shape)
    s.set_patterns(pats.astype(np.float32).reshape(3, 5, 60, 60))
    dis = np.degrees(s.disorientation(s.index()["quaternions"].reshape(-1, 4), q))
    assert np.median(dis) < 0.15 and dis.max() < 1.0, (np.median(dis), dis.max())
