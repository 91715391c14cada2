"""Refinement of six unknowns per pattern on the detector: the source's shift (equivalently its
pattern centre) and the crystal's orientation (config 3; the per-pattern step of the reference's
plane fit, `planefit.zig:570-622` settle with k = 6, Winkelmann et al. / kikuchipy's
refine_orientation_projection_center).

`ProjectedNCC` is the detector projection + NCC as a `torch.autograd.Function`: forward and
backward are the CUDA kernels of `zeb_det6` (mode 0 and mode 1); the backward recomputes the
projection of every pixel from the parameters instead of keeping the projected patterns.
`refine6` runs the reference's Levenberg–Marquardt settle over all the given patterns at once,
each round's verdicts and damped 6 × 6 solves in one FP64 kernel (`zeb_settle6`), the
Gauss–Newton matrix from the reference's 43 sums (`zeb_det6` mode 2); the gradient is the reference's (the gradient
table's) or the exact adjoint's (the kernel behind ProjectedNCC's backward).
"""
import ctypes

import numpy as np
import torch

from . import _native as N
from .device import ptr, stream_ptr


class Plan:
    """What a batch of patterns needs besides its parameters: preprocessed patterns, items,
    frame, and the master's pair tables."""

    def __init__(self, pats, items, frame, vpair, gpair, side, pixels=None):
        self.pats, self.items, self.frame = pats, items, frame
        self.vpair, self.gpair, self.side = vpair, gpair, side
        self.pixels = pixels  # the frame's masked-pixel list (zeb_mask_list), or None
        self.n = items.shape[0]

    def run(self, mode, x, q0):
        width = (1, 7, 43, 61)[mode]
        out = torch.empty(self.n * width, dtype=torch.float32, device=x.device)
        if self.pixels is not None:
            N.call("zeb_det6_list", mode, ptr(self.pats), ptr(self.items), self.n, ctypes.byref(self.frame),
                   ptr(self.pixels), self.pixels.numel(), ptr(self.vpair), ptr(self.gpair), self.side, ptr(x), ptr(q0),
                   ptr(out), stream_ptr())
        else:
            N.call("zeb_det6", mode, ptr(self.pats), ptr(self.items), self.n, ctypes.byref(self.frame),
                   ptr(self.vpair), ptr(self.gpair), self.side, ptr(x), ptr(q0), ptr(out), stream_ptr())
        return out.view(self.n, width) if width > 1 else out


class ProjectedNCC(torch.autograd.Function):
    """NCC[b] of pattern b with the master projected at x[b] = (δt (pixels), φ (radians)) about
    its base orientation q0[b]; backward by the hand-written adjoint kernel."""

    @staticmethod
    def forward(ctx, x, q0, plan):
        x = x.detach().to(torch.float32).contiguous()
        q0 = q0.detach().to(torch.float32).contiguous()
        ctx.save_for_backward(x, q0)
        ctx.plan = plan
        return plan.run(0, x, q0).clone()

    @staticmethod
    def backward(ctx, grad_out):
        x, q0 = ctx.saved_tensors
        res = ctx.plan.run(1, x, q0)  # the projection recomputed, its derivatives summed
        return grad_out.to(torch.float32)[:, None] * res[:, :6], None, None


def projected_ncc(x, q0, plan):
    return ProjectedNCC.apply(x, q0, plan)


def pc_jacobian(geo, rows, cols):
    """∂t/∂(pcx, pcy, pcz) of the source's place t = R·(0.5 − pcy·rows, 0.5 − pcx·cols, pcz·rows)
    (geometry.zig:153-161): a 3 × 3 matrix, columns per pattern-centre coordinate."""
    R = geo.rotation()
    return np.stack([R @ np.array([0.0, -cols, 0.0]), R @ np.array([-rows, 0.0, 0.0]), R @ np.array([0.0, 0.0, rows])],
                    1)


def _qstd(q):
    n = torch.linalg.norm(q, dim=-1, keepdim=True)
    n = torch.where(n == 0, torch.ones_like(n), n)
    return q / n * torch.where(q[..., :1] < 0, -1.0, 1.0)


def local_of(s):
    """planefit.zig:176-200 (localOf) for every pattern, FP64: (ok, NCC, g [n,6], H [n,6,6])
    from the 43 sums [n, 43]."""
    s = s.to(torch.float64)
    n = torch.clamp(s[:, 0], min=1.0)
    mean = s[:, 1] / n
    var_n = s[:, 2] - n * mean * mean
    ok = var_n > 1e-12
    inv = torch.where(ok, torch.rsqrt(torch.where(ok, var_n, torch.ones_like(var_n))), torch.zeros_like(var_n))
    ncc = s[:, 3] * inv
    sd = s[:, 4:10]
    au = (s[:, 10:16] - mean[:, None] * sd) * inv[:, None]
    g = (s[:, 16:22] - ncc[:, None] * au) * inv[:, None]
    iu = torch.triu_indices(6, 6)
    P = torch.zeros(s.shape[0], 6, 6, dtype=torch.float64, device=s.device)
    P[:, iu[0], iu[1]] = s[:, 22:43]
    P = P + torch.triu(P, 1).transpose(1, 2)
    H = (P - sd[:, :, None] * sd[:, None, :] / n[:, None, None] - au[:, :, None] * au[:, None, :]) * (inv * inv)[:, None, None]
    ncc = torch.where(ok, ncc, torch.full_like(ncc, -2.0))
    return ok, ncc, g, H


def adjoint_gradient(s):
    """∂NCC/∂x from the one-pass sums of zeb_det6 mode 3 [n, 61] (FP64): the NCC's statistics
    (sums 0-3) with the exact derivatives' ΣD', ΣM·D', Σe·D' (sums 43-60), by the formula of
    planefit.zig:176-200 (au = (ΣM·D' − mean·ΣD')/σ, g = (Σe·D' − NCC·au)/σ)."""
    s = s.to(torch.float64)
    n = torch.clamp(s[:, 0], min=1.0)
    mean = s[:, 1] / n
    var_n = s[:, 2] - n * mean * mean
    ok = var_n > 1e-12
    inv = torch.where(ok, torch.rsqrt(torch.where(ok, var_n, torch.ones_like(var_n))), torch.zeros_like(var_n))
    ncc = s[:, 3] * inv
    au = (s[:, 49:55] - mean[:, None] * s[:, 43:49]) * inv[:, None]
    return (s[:, 55:61] - ncc[:, None] * au) * inv[:, None]


def refine6(plan, q0, trust, most=60, gradient="reference"):
    """planefit.zig:570-622 (settle, k = 6) over every pattern of `plan` at once: λ from 1e-3;
    each round every pattern's damped step (its shift clamped to ±trust pixels, its rotation
    exp(d)·q) is kept where its own NCC rose (λ ← max(λ/3, 1e-4)), else λ ← min(5λ, 1e8); until
    a round gains the patterns' mean NCC less than 1e-7 (a round in which every step overshot
    goes again while some λ < 1e8) or after `most` rounds. gradient: "reference" (the gradient
    table's, as the reference) or "adjoint" (the exact derivative of the forward, ProjectedNCC's
    backward: the derivatives of its adjoint kernel summed in the same pass as the GN sums, mode 3).
    Returns (q [n,4] f64, shift [n,3] f64 pixels, NCC [n], rounds)."""
    dev = q0.device
    n = plan.n
    mode, width = (3, 61) if gradient == "adjoint" else (2, 43)
    state = torch.zeros(N.ZEB_SETTLE6_STATE, n, dtype=torch.float64, device=dev)
    state[29:33] = q0.t()
    x = torch.zeros(n, 6, dtype=torch.float32, device=dev)
    qf = _qstd(q0.to(torch.float64)).to(torch.float32).contiguous()
    parts = torch.empty((n + 31) // 32, 3, dtype=torch.float64, device=dev)

    def step(first):
        # the sums at (x, qf), held until the call that reads them, then the round's verdicts and the next (x, qf)
        sums = plan.run(mode, x, qf)
        N.call("zeb_settle6", ptr(sums), width, n, float(trust), first, ptr(state), ptr(x), ptr(qf),
               ptr(parts), stream_ptr())

    step(1)
    count = max(n, 1)
    rounds = 0
    while rounds < most:
        step(0)
        gain, kept, damp = parts.sum(0).tolist()
        if kept == 0 and damp > 0:  # (every step overshot: they go again, damped more)
            rounds += 1
            continue
        if gain / count < 1e-7:  # (the round that ends the loop is not counted, as the reference's)
            break
        rounds += 1
    return state[29:33].t().contiguous(), state[33:36].t().contiguous(), state[0], rounds
