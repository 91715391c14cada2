"""Kernels whose dynamic shared memory alone fits the 48 KB that need no leave, but not beside their static
arrays: patterns of such sizes are filtered as the first work of a process, where no larger call has raised
the limit (GPU only)."""
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CODE = """
import ctypes, sys, torch
sys.path.insert(0, {root!r})
from zebsdsolve_b200 import _native as N
p = lambda t: ctypes.c_void_p(t.data_ptr())
h, w, dynamic, sigma = {case}
n = 3
raw = torch.rand(n, h, w, device="cuda")
out = torch.full((n, h, w), float("nan"), device="cuda")
scratch = torch.zeros(N.load().zeb_prep_scratch_bytes(n, h, w, sigma) + 16, dtype=torch.uint8, device="cuda")
mask = (ctypes.c_float * 3)(0.5 * (h - 1), 0.5 * (w - 1), 1e9)
N.call("zeb_prep_reduced", p(raw), 2, n, h, w, 1.0, None, dynamic, sigma, mask, 1, p(out), p(scratch),
       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
torch.cuda.synchronize()
norm = out.double().flatten(1).norm(dim=1)
assert bool(((norm - 1).abs() < 1e-4).all()), norm
"""


@pytest.mark.parametrize("case", [(72, 85, 0, 0.0), (80, 80, 1, 12.0)])  # k_prep; k_prep_wide
def test_first_call_of_a_process(case, request):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, "-c", CODE.format(root=str(request.config.rootpath), case=case)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
