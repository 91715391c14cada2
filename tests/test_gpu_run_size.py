"""The FP32 form's record of a cell is the same bits however many cells run with it: a look at a few cells,
a region, the whole map, refined and not; and a blank master is indexed (GPU only)."""
import tempfile

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROWS, COLS = 10, 14


def _master(sheets, side):
    from zebsdsolve_b200 import synthetic as syn
    from zebsdsolve_b200.master import write_npz

    path = tempfile.mkdtemp() + "/m.npz"
    write_npz(path, sheets, side, syn.group_matrices("432"), 30)
    return path


def _solver(L, master, patterns):
    import zebsdsolve_b200 as ze

    s = ze.Solver()
    s.configure(bandwidth=L)
    s.add_phase(master)
    s.set_patterns(patterns)
    s.set_geometry(pc=(0.5, 0.3, 0.6), sample_tilt_deg=70, detector_tilt_deg=0)
    return s


@pytest.fixture(scope="module")
def scan():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zebsdsolve_b200 import synthetic as syn

    n = ROWS * COLS
    master = _master(syn.master_sheets(6, side=201, lmax=48, group="432", device="cuda"), 201)
    s = _solver(32, master, np.zeros((ROWS, COLS, 60, 60), np.uint16))
    sims = s._e.simulate_device(0, np.arange(n), syn.uniform_quaternions(np.random.default_rng(12), n))
    return master, syn.counted_patterns(sims, seed=2).cpu().numpy().reshape(ROWS, COLS, 60, 60)


@pytest.mark.parametrize("L,refine", [(32, True), (32, False), (64, True)])
def test_a_cell_s_record_does_not_depend_on_the_run_s_size(scan, L, refine):
    s = _solver(L, *scan)
    s.configure(refine=refine)
    n = ROWS * COLS
    whole = s.index_cells(np.arange(n))
    for size in (5, 64, 65):
        for at in (0, 37):
            part = s.index_cells(np.arange(at, at + size))
            for k, v in part.items():
                assert np.array_equal(v, whole[k][:, at:at + size]), (size, at, k)


def test_a_blank_master_is_indexed():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    s = _solver(32, _master(np.zeros((2, 201, 201), np.float32), 201),
                np.random.default_rng(3).integers(0, 250, (ROWS, COLS, 60, 60)).astype(np.uint8))
    r = s.index_cells(np.arange(ROWS * COLS))
    assert np.isfinite(r["quaternions"]).all() and (r["ncc"] <= 0).all()
