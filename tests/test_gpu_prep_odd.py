"""The wide blur of a detector with an odd number of pixels, too large for shared memory: its partial sums
(pairs of floats) start on an 8-byte boundary of every pattern's scratch (GPU only; the filter chain
against the oracle's)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3])
def test_wide_blur_of_a_large_odd_detector(n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import oracle.geometry as og
    import oracle.prep as op
    from zebsdsolve_b200 import _native as N

    h = w = 151
    sigma = 0.15 * w
    raw = np.random.default_rng(4).integers(0, 4000, (n, h, w)).astype(np.uint16)
    mask = og.mask_of(h, w)
    lib = N.load()
    scratch = torch.zeros(lib.zeb_prep_scratch_bytes(n, h, w, sigma), dtype=torch.uint8, device="cuda")
    dev = torch.as_tensor(raw, device="cuda")
    out = torch.empty(n * h * w, device="cuda")

    def p(t):
        return ctypes.c_void_p(t.data_ptr())

    N.call("zeb_prep_ex", p(dev), 1, n, h, w, None, 1, sigma, (ctypes.c_float * 3)(*mask), 1, p(out), p(scratch),
           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    got = out.view(n, h, w).cpu().numpy()
    for k in range(n):
        want = op.run(raw[k], dynamic="subtract", dynamic_sigma=sigma, mask=mask)
        assert np.abs(got[k] - want).max() <= 2e-6  # as the other filter tests, on unit-norm images
