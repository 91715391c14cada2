"""One round of the six-unknown settle (zeb_settle6) against the same steps in plain FP64 tensor operations
(GPU only).

Tolerance: both are FP64; the steps solve systems of condition below 1e6 by elimination, so that a trial
differs by some 1e6 · 2^-52 of its size at most: 1e-8; the statistics by a few roundings: 1e-12.
"""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

F64 = torch.float64


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _sums(n, width, g):
    """Sums of 200 invented pixels a pattern: the statistics of the master's values M, their derivatives D and
    the pattern's values e (the pattern part of M, so that the NCC is well off 0)."""
    D = torch.randn(n, 200, 6, generator=g, dtype=F64, device="cuda")
    M = torch.randn(n, 200, generator=g, dtype=F64, device="cuda")
    e = M + 0.7 * torch.randn(n, 200, generator=g, dtype=F64, device="cuda") + 0.05 * D.sum(-1)
    e = e - e.mean(1, keepdim=True)
    e = e / e.norm(dim=1, keepdim=True)
    iu = torch.triu_indices(6, 6)
    s = [torch.full((n, 1), 200.0, dtype=F64, device="cuda"), M.sum(1)[:, None], (M * M).sum(1)[:, None],
         (M * e).sum(1)[:, None], D.sum(1), (M[..., None] * D).sum(1), (e[..., None] * D).sum(1),
         torch.einsum("bpi,bpj->bij", D, D)[:, iu[0], iu[1]]]
    if width == 61:
        E = D + 0.01 * torch.randn(n, 200, 6, generator=g, dtype=F64, device="cuda")
        s += [E.sum(1), (M[..., None] * E).sum(1), (e[..., None] * E).sum(1)]
    return torch.cat(s, 1).float().contiguous()


def _qmul(a, b):
    aw, ax, ay, az = a.unbind(-1)
    bw, bx, by, bz = b.unbind(-1)
    return torch.stack([aw * bw - ax * bx - ay * by - az * bz, aw * bx + ax * bw + ay * bz - az * by,
                        aw * by - ax * bz + ay * bw + az * bx, aw * bz + ax * by - ay * bx + az * bw], -1)


def _unit(q):
    return q / q.norm(dim=-1, keepdim=True) * torch.where(q[..., :1] < 0, -1.0, 1.0)


def _trial(adjoint, s, q, shift, lam, trust):
    ok, ncc, g, H = adjoint.local_of(s[:, :43])
    if s.shape[1] == 61:
        g = torch.where(ok[:, None], adjoint.adjoint_gradient(s), torch.zeros_like(g))
    dg = torch.diagonal(H, dim1=1, dim2=2)
    A = H + torch.diag_embed(dg * lam[:, None] + (1e-9 * dg.sum(-1) + 1e-30)[:, None])
    d = torch.zeros_like(g)
    d[ok] = torch.linalg.solve(A[ok], g[ok])
    th = d[:, 3:].norm(dim=1, keepdim=True)
    half = torch.where(th < 1e-6, 0.5 - th * th / 48, torch.sin(th / 2) / torch.where(th < 1e-6, 1.0, th))
    turned = _unit(_qmul(torch.cat([torch.cos(th / 2), half * d[:, 3:]], 1), q))
    return (ok, ncc, torch.where(ok[:, None], turned, q),
            torch.where(ok[:, None], (shift + d[:, :3]).clamp(-trust, trust), shift))


@pytest.mark.parametrize("n,width", [(1, 43), (31, 61), (32, 43), (33, 61), (1000, 43)])
def test_two_rounds(n, width):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zebsdsolve_b200 import _native as N
    from zebsdsolve_b200 import adjoint

    g = torch.Generator(device="cuda")
    g.manual_seed(n * 64 + width)
    trust = 0.05
    s1, s2 = _sums(n, width, g), _sums(n, width, g)
    s1[3::7, 2] = 0  # no variance: nothing to step on
    s2[5::9, 2] = 0
    q0 = torch.randn(n, 4, generator=g, dtype=F64, device="cuda")
    state = torch.zeros(N.ZEB_SETTLE6_STATE, n, dtype=F64, device="cuda")
    state[29:33] = q0.t()
    x = torch.zeros(n, 6, device="cuda")
    qf = torch.zeros(n, 4, device="cuda")
    parts = torch.full(((n + 31) // 32, 3), float("nan"), dtype=F64, device="cuda")

    def step(s, first):
        N.call("zeb_settle6", _p(s), width, n, trust, first, _p(state), _p(x), _p(qf), _p(parts),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()

    step(s1, 1)
    lam = torch.full((n,), 1e-3, dtype=F64, device="cuda")
    q, shift = _unit(q0), torch.zeros(n, 3, dtype=F64, device="cuda")
    ok1, ncc1, qt, st = _trial(adjoint, s1, q, shift, lam, trust)
    near = lambda a, b, t: float((a - b).abs().max()) <= t  # noqa: E731
    assert near(state[0], ncc1, 1e-12) and near(state[29:33].t(), q, 1e-14) and near(state[37:41].t(), qt, 1e-8)
    assert near(state[41:44].t(), st, 1e-8) and torch.equal(qf, state[37:41].t().float())
    assert torch.equal(x[:, :3], state[41:44].t().float()) and bool((x[:, 3:] == 0).all())
    qt, st = state[37:41].t().clone(), state[41:44].t().clone()
    step(s2, 0)
    _, ncc2, _, _ = _trial(adjoint, s2, qt, st, lam, trust)
    better = ncc2 > ncc1
    gain, kept, damp = parts.sum(0).tolist()
    assert kept == int(better.sum()) and damp == n - kept
    assert abs(gain - float((ncc2 - ncc1)[better].sum())) <= 1e-12 * n
    keep = lambda a, b: torch.where(better.view(-1, *([1] * (a.dim() - 1))), a, b)  # noqa: E731
    lam = torch.where(better, lam / 3, lam * 5)
    assert near(state[36], lam, 1e-15)
    assert near(state[29:33].t(), keep(qt, q), 1e-14)
    assert near(state[0], keep(ncc2, ncc1), 1e-12)
    q, shift = keep(qt, q), keep(st, shift)
    _, _, qn, sn = _trial(adjoint, torch.where(better[:, None], s2, s1), q, shift, lam, trust)
    assert near(state[33:36].t(), shift, 1e-15)
    assert near(state[37:41].t(), qn, 1e-8) and near(state[41:44].t(), sn, 1e-8)


@pytest.mark.parametrize("width", [43, 61])
def test_damping_at_its_bounds_and_small_rotations(width):
    """λ set by hand before a round that keeps or loses the trial: it stays within [1e-4, 1e8], a loss at 1e8 is no
    longer counted as damped, and at 1e8 the next step's rotation is far below the 1e-6 where its sine's series
    takes over. The systems are then all but diagonal: a step is right to 1e-10 of its size, and a trial beside
    it to the rounding of a unit quaternion, 2e-15."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zebsdsolve_b200 import _native as N
    from zebsdsolve_b200 import adjoint

    n, trust = 96, 0.05
    g = torch.Generator(device="cuda")
    g.manual_seed(width)
    s1, s2 = _sums(n, width, g), _sums(n, width, g)
    state = torch.zeros(N.ZEB_SETTLE6_STATE, n, dtype=F64, device="cuda")
    state[29:33] = torch.randn(4, n, generator=g, dtype=F64, device="cuda")
    x, qf = torch.zeros(n, 6, device="cuda"), torch.zeros(n, 4, device="cuda")
    parts = torch.empty((n + 31) // 32, 3, dtype=F64, device="cuda")

    def step(s, first):
        N.call("zeb_settle6", _p(s), width, n, trust, first, _p(state), _p(x), _p(qf), _p(parts),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()

    step(s1, 1)
    given = torch.tensor([1e-4, 2e-4, 3e7, 1e8], dtype=F64, device="cuda").repeat(n // 4)
    state[36] = given
    was, q, qt, st = state[0].clone(), state[29:33].t().clone(), state[37:41].t().clone(), state[41:44].t().clone()
    step(s2, 0)
    _, ncc, _, _ = adjoint.local_of(s2[:, :43])
    better = ncc > was
    assert 4 <= int(better.sum()) <= n - 4
    lam = torch.where(better, (given / 3).clamp(min=1e-4), (given * 5).clamp(max=1e8))
    assert torch.equal(state[36], lam)
    _, kept, damp = parts.sum(0).tolist()
    assert kept == int(better.sum()) and damp == int((~better & (given < 1e8)).sum())
    q, shift = torch.where(better[:, None], qt, q), torch.where(better[:, None], st, 0 * st)
    _, _, qn, sn = _trial(adjoint, torch.where(better[:, None], s2, s1), q, shift, lam, trust)
    small = lam >= 1e7
    d = 2 * (qn - q)[small].norm(dim=1)
    assert int(small.sum()) >= 40 and float(d.max()) < 1e-6
    assert bool(((state[37:41].t() - qn)[small].abs() <= 1e-10 * d[:, None] + 2e-15).all())
    assert bool(((state[41:44].t() - sn)[small].abs() <= 1e-10 * (sn - shift)[small].abs() + 1e-17).all())


def test_solve6():
    """Random systems, some with a pivot that has to be fetched from another row, some singular, one with a NaN: the
    residual is the rounding of an elimination with partial pivoting, 6^2 · 2^-52 (|A||x| + |b|) with room for the
    growth of 6 pivots (2^5)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zebsdsolve_b200 import _native as N

    n = 300
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    A = torch.randn(n, 6, 6, generator=g, dtype=F64, device="cuda")
    A[1::5, 0, 0] = 0
    A[2::5, 2:4, 2] = 0
    A[3::5, :, 4] = 0  # singular
    A[4] = 0
    A[9, 3, 3] = float("nan")
    b = torch.randn(n, 6, generator=g, dtype=F64, device="cuda")
    x = torch.full((n, 6), 7.0, dtype=F64, device="cuda")
    ok = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    N.call("zeb_solve6", _p(A), _p(b), n, _p(x), _p(ok), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    want = torch.ones(n, dtype=torch.int32, device="cuda")
    want[3::5] = 0
    want[4] = 0
    assert torch.equal(ok, want) and bool((x[ok == 0] == 0).all()) and bool(torch.isnan(x[9]).any())
    use = ok != 0
    use[9] = False
    A, b, x = A[use], b[use], x[use]
    off = (torch.einsum("nij,nj->ni", A, x) - b).abs()
    bound = 36 * 32 * 2.0 ** -52 * (torch.einsum("nij,nj->ni", A.abs(), x.abs()) + b.abs()).amax(1, keepdim=True)
    assert bool((off <= bound).all())
