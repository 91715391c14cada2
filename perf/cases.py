"""The framework's performance cases: whole indexing runs, the six-unknown refinement and the
dictionary match, through the calls a user's program makes (`Solver.index`,
`Solver.refine_patterns`, the C ABI of include/zebsdsolve_b200.h for the match), over the range of
scans, detectors, bandwidths, arithmetic forms and options the framework is used with.

`exact` gives each case's outputs from plain torch in 64 bits: the definitions of the path (the
filters, the spherical harmonics, the SO(3) correlation and its peak, the Gauss–Newton and
Levenberg–Marquardt refinements, the scores) written out over the same inputs.

Patterns are simulated here from seeded masters (SH degree up to 96, symmetrized by their point
group): grains over the map, Poisson counts over a Gaussian background.
"""
import ctypes
import functools
import math
import os
import tempfile

import numpy as np
import torch

import zebsdsolve_b200 as ze
from zebsdsolve_b200 import _native as native
from zebsdsolve_b200 import synthetic
from zebsdsolve_b200.master import write_npz

PC = (0.5, 0.3, 0.6)
TILT_DEG = 70.0
DETECTOR_MM = 24.0
SIDE, LMAX = 401, 96
MASTERS = (("432", 2), ("622", 3))  # the first phase, and the second where a case has two
MASTER_SMOOTH, DYNAMIC_SIGMA, STATIC_PATTERNS = 0.3, 0.15, 1024
NMI_BINS, REFINE_ITERS, REFINE_STEP_DEG = 16, 8, 2.0
ACCEPT_Z, ACCEPT_STEP_DEG = 15.0, 5.0  # matches are accepted by their score alone
ROI_AT = 3  # where a region of interest starts, rows and columns
GRAIN_SPREAD_DEG = 0.5
F64, C128 = torch.float64, torch.complex128


# ── the cases ──

def _index(name, rows, cols, h, w, pixel, precision, L, **more):
    case = {"kind": "index", "rows": rows, "cols": cols, "h": h, "w": w, "pixel": pixel, "precision": precision,
            "L": L, "phases": 1, "sweeps": 1, "binning": 1, "refine": True, "nlpar": False, "new_scan": False, "roi": 0}
    case.update(more)
    return dict(case, name=name)


def listed():
    return [
        # a few cells of an open scan indexed while looking at it: the smallest call, its latency
        _index("look_4x4", 55, 75, 60, 60, "u8", "f32", 64, roi=4),
        # a laboratory map of the reference's own scan's size at the default settings
        _index("map_55x75", 55, 75, 60, 60, "u8", "f32", 64),
        # the same map in two sweeps (a coarse one for most cells, the full bandwidth for the rest),
        # each time a scan newly set: what indexing one file after another costs
        _index("two_sweeps_55x75", 55, 75, 60, 60, "u8", "f32", 64, sweeps=2, new_scan=True),
        # the same map averaged with its neighbours first (noisy scans)
        _index("nlpar_55x75", 55, 75, 60, 60, "u8", "f32", 64, nlpar=True),
        # a large map at the default settings
        _index("map_160x160", 160, 160, 60, 60, "u16", "f32", 64),
        # the largest map: the BF16 form, the throughput setting
        _index("bf16_map_256x256", 256, 256, 60, 60, "u16", "bf16", 64),
        # correlation alone at half the bandwidth: a first look, no refinement
        _index("coarse_64x64", 64, 64, 60, 60, "u16", "f32", 32, refine=False),
        # two candidate phases on a mid-size detector
        _index("two_phases_48x64", 48, 64, 96, 96, "u16", "bf16", 64, phases=2),
        # large detectors unreduced (float patterns, not square)
        _index("detector_120x160", 32, 48, 120, 160, "f32", "f32", 64),
        # large detectors binned to half, the highest bandwidth
        _index("binned_L128", 24, 32, 160, 160, "u16", "bf16", 128, binning=2),
        # every pattern's orientation and pattern centre refined, by the exact gradient
        {"name": "refine6_64x64", "kind": "refine6", "rows": 64, "cols": 64, "h": 120, "w": 120, "pixel": "u16",
         "gradient": "adjoint"},
        # patterns' coefficients matched against a dictionary's
        {"name": "match_16384x32768", "kind": "match", "n": 16384, "entries": 32768, "cols": 512},
    ]


def _loguniform(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["index"] * 8 + ["refine6", "refine6", "match"])
    pixel = rng.choice(["u8", "u16", "u16", "f32"])
    if kind == "match":
        n, entries, cols = _loguniform(rng, 64, 16384), _loguniform(rng, 2000, 32768), rng.choice([256, 300, 512])
        return {"kind": "match", "n": n, "entries": entries, "cols": cols}
    h = rng.randint(40, 140)
    w = h if rng.random() < 0.6 else rng.randint(40, 140)
    if kind == "refine6":
        n = _loguniform(rng, 16, max(17, min(4096, (40 << 20) // (h * w))))
        rows = max(1, int(math.sqrt(n) * rng.uniform(0.7, 1.2)))
        return {"kind": "refine6", "rows": rows, "cols": max(1, n // rows), "h": h, "w": w, "pixel": pixel,
                "gradient": rng.choice(["adjoint", "reference"])}
    L = rng.choice([16, 24, 32, 48, 64, 64, 64, 80, 128])
    phases = rng.choice([1, 1, 1, 2])
    most = min(16384 if L <= 64 else 768, (40 << 20) // (h * w)) // phases
    n = _loguniform(rng, 300, most)
    rows = max(1, int(math.sqrt(n) * rng.uniform(0.6, 1.3)))
    c = _index("", rows, max(1, n // rows), h, w, pixel, rng.choice(["f32", "bf16"]), L, phases=phases,
               sweeps=rng.choice([1, 1, 1, 2]) if L > 32 else 1, binning=rng.choice([1, 1, 1, 2]) if min(h, w) > 90 else 1,
               refine=rng.random() < 0.85, nlpar=rng.random() < 0.1 and n < 4096, new_scan=rng.random() < 0.25,
               roi=rng.randint(1, 8) if rng.random() < 0.15 else 0)
    del c["name"]
    return c


def _mask_pixels(h, w):
    return int(_mask(h, w).sum())


def work(case):
    """Bytes and operations of one pass that the path cannot do without: the stored patterns read
    and the records written once; the correlation's products (8 operations a complex product, every
    pattern with every column of the master's table) and the detector's lookups."""
    if case["kind"] == "match":
        n, e, k = case["n"], case["entries"], case["cols"]
        return {"bytes": 4.0 * (n * k + e * k + 8 * n), "flops": 2.0 * n * e * k}
    n = case["rows"] * case["cols"] if not case.get("roi") else case["roi"] ** 2
    size = {"u8": 1, "u16": 2, "f32": 4}[case["pixel"]]
    stored = float(n * case["h"] * case["w"] * size)
    if case["kind"] == "refine6":
        return {"bytes": stored + 64.0 * n, "flops": 5 * 300.0 * n * _mask_pixels(case["h"], case["w"])}
    b = case["binning"]
    pix = _mask_pixels(case["h"] // b, case["w"] // b)
    flops = 0.0
    for k in range(case["phases"]):
        L = 32 if case["sweeps"] == 2 else case["L"]
        size_n = _fft_size(L)
        nc = size_n // (4 if MASTERS[k][0] == "432" else 2)
        cols = (size_n // 2 + 1) * nc
        flops += n * (8.0 * cols * L * (L + 1) / 2 + 5.0 * cols * size_n * math.log2(size_n))
        flops += n * pix * 100.0 * (1 + (REFINE_ITERS if case["refine"] else 0))
    return {"bytes": stored + 48.0 * n, "flops": flops}


# ── masters and scans ──

@functools.lru_cache(maxsize=None)
def _master(k):
    """(path of the master's file, its sheets [2, side, side], its rotations as quaternions)."""
    group, seed = MASTERS[k]
    sheets = synthetic.master_sheets(seed, side=SIDE, lmax=LMAX, group=group, device="cuda")
    path = os.path.join(tempfile.mkdtemp(prefix="cases_"), f"m{group}.npz")
    write_npz(path, sheets, SIDE, synthetic.group_matrices(group), synthetic.POINT_GROUP[group])
    return path, sheets, _group(group)


def _qmul(a, b):
    aw, ax, ay, az = a.unbind(-1)
    bw, bx, by, bz = b.unbind(-1)
    return torch.stack([aw * bw - ax * bx - ay * by - az * bz, aw * bx + ax * bw + ay * bz - az * by,
                        aw * by - ax * bz + ay * bw + az * bx, aw * bz + ax * by - ay * bx + az * bw], -1)


def _qstd(q):
    q = q / q.norm(dim=-1, keepdim=True)
    return torch.where(q[..., :1] < 0, -q, q)


def _exp(v):
    th = v.norm(dim=-1, keepdim=True)
    k = torch.where(th < 1e-6, 0.5 - th * th / 48, torch.sin(0.5 * th) / torch.where(th < 1e-6, torch.ones_like(th), th))
    return torch.cat([torch.cos(0.5 * th), k * v], -1)


def _rotate(q, v):
    """q v q* (q broadcast over v's leading axes)."""
    u = q[..., 1:].expand(v.shape)
    t = 2 * torch.linalg.cross(u, v)
    return v + q[..., :1] * t + torch.linalg.cross(u, t)


def _group(name):
    """The rotations of 432 (axes along x, y, z) or 622 (six-fold along z, two-fold along x)."""
    r = math.sqrt(0.5)
    gens = [(r, 0, 0, r), (0.5, 0.5, 0.5, 0.5)] if name == "432" else [(math.sqrt(3) / 2, 0, 0, 0.5), (0, 1, 0, 0)]
    out = [torch.tensor([1.0, 0, 0, 0], dtype=F64)]
    for a in out:
        for g in gens:
            q = _qmul(torch.tensor(g, dtype=F64), a)
            if all(abs(float((q * b).sum())) < 1 - 1e-9 for b in out):
                out.append(q)
    return torch.stack(out)


def _square(v):
    """Unit vectors → coordinates in [−1, 1]² of their own hemisphere's equal-area square."""
    ax, ay = v[..., 0].abs(), v[..., 1].abs()
    s = ax * ax + ay * ay
    xn = torch.sqrt(math.pi / 2 * s / (1 + v[..., 2].abs()))
    big = ax >= ay
    ang = 4 / math.pi * torch.atan2(torch.where(big, ay, ax), torch.where(big, ax, ay).clamp(min=1e-30))
    u, w = torch.where(big, xn, xn * ang), torch.where(big, xn * ang, xn)
    sc = math.sqrt(2 / math.pi)
    return sc * torch.where(v[..., 0] < 0, -u, u), sc * torch.where(v[..., 1] < 0, -w, w)


def _lookup(table, v):
    """Bilinear values of a table [2, side, side(, k)] at directions v."""
    side = table.shape[1]
    x, y = _square(v)
    last = side - 1.0
    fj, fi = ((x + 1) * 0.5 * last).clamp(0, last), ((y + 1) * 0.5 * last).clamp(0, last)
    c0, r0 = fj.detach().floor().clamp(max=side - 2).long(), fi.detach().floor().clamp(max=side - 2).long()
    tj, ti = fj - c0, fi - r0
    o = (v[..., 2] < 0).long() * side * side + r0 * side + c0
    flat = table.reshape(2 * side * side, *table.shape[3:])
    if table.dim() == 4:
        tj, ti = tj[..., None], ti[..., None]
    return (flat[o] * (1 - tj) + flat[o + 1] * tj) * (1 - ti) + (flat[o + side] * (1 - tj) + flat[o + side + 1] * tj) * ti


class _Detector:
    """The detector of h × w pixels (a stored size over a binning) and the map's cells before it."""

    def __init__(self, case, dtype=F64, device="cuda"):
        b = case.get("binning", 1)
        self.h, self.w, self.dtype, self.device = case["h"] // b, case["w"] // b, dtype, device
        rows, cols = case["rows"], case["cols"]
        a = math.radians(-TILT_DEG)
        s, c = math.sin(a), math.cos(a)
        self.R = torch.tensor([[-s, 0, c], [0, 1, 0], [-c, 0, -s]], dtype=dtype, device=device)
        fh, fw = case["h"] / b, case["w"] / b
        t0 = self.R @ torch.tensor([0.5 - PC[1] * fh, 0.5 - PC[0] * fw, PC[2] * fh], dtype=dtype, device=device)
        px_um = 1000.0 * DETECTOR_MM / case["w"] * b
        cell = torch.arange(rows * cols, device=device)
        off = torch.stack([-(cell // cols - 0.5 * (rows - 1)) / px_um, -(cell % cols - 0.5 * (cols - 1)) / px_um,
                           torch.zeros(rows * cols, device=device)], 1).to(dtype)
        self.t0, self.t = t0, t0 - off
        self.angle = b / (PC[2] * case["h"])  # of a pixel, radians
        self.mask = torch.as_tensor(_mask(self.h, self.w), device=device)
        rr, cc = torch.meshgrid(torch.arange(self.h, device=device), torch.arange(self.w, device=device), indexing="ij")
        self.plane = rr.to(dtype)[..., None] * self.R[:, 0] + cc.to(dtype)[..., None] * self.R[:, 1]

    def rays(self, t, masked=True):
        """Every (masked) pixel's ray from sources t [n, 3]: [n, pixels, 3]."""
        p = self.plane[self.mask] if masked else self.plane.reshape(-1, 3)
        return p[None] + t[:, None, :]


def _mask(h, w):
    r = 0.5 * min(h, w)
    y, x = np.arange(h)[:, None] - 0.5 * (h - 1), np.arange(w)[None, :] - 0.5 * (w - 1)
    return y * y + x * x <= r * r


def _scan(case, seed):
    """(stored patterns on the device [n, h, w], orientations [n, 4], phases [n]): grains of uniform
    orientations over the map, a little spread in each, Poisson counts over a Gaussian hump."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    rows, cols, h, w = case["rows"], case["cols"], case["h"], case["w"]
    n, phases = rows * cols, case.get("phases", 1)
    k = max(1, min(200, n // 16))
    at = torch.rand(k, 2, device="cuda", generator=g) * torch.tensor([rows, cols], device="cuda")
    gq = _qstd(torch.randn(k, 4, device="cuda", generator=g, dtype=F64))
    cell = torch.arange(n, device="cuda")
    place = torch.stack([cell // cols + 0.5, cell % cols + 0.5], 1)
    grain = torch.cdist(place.float(), at).argmin(1)
    spread = math.radians(GRAIN_SPREAD_DEG) / math.sqrt(3)
    q = _qstd(_qmul(_exp(spread * torch.randn(n, 3, device="cuda", generator=g, dtype=F64)), gq[grain]))
    phase = grain % phases
    full = _Detector(dict(case, binning=1), torch.float32)
    yy = torch.arange(h, device="cuda")[:, None] + 0.5 - 0.5 * h
    xx = torch.arange(w, device="cuda")[None, :] + 0.5 - 0.5 * w
    hump = torch.exp(-(xx * xx + yy * yy) / (2 * (0.4 * w) ** 2))
    hump = hump * (h * w) / hump.sum()
    shift = torch.zeros(n, 3, device="cuda")
    if case["kind"] == "refine6":  # each pattern's own source, some way off the map's
        shift = (torch.rand(n, 3, device="cuda", generator=g) - 0.5) * 0.01 * h
    counts = 90.0 if case["pixel"] == "u8" else 1000.0
    out = torch.empty(n, h, w, dtype={"u8": torch.uint8, "u16": torch.int32, "f32": torch.float32}[case["pixel"]],
                      device="cuda")
    sheets = [torch.as_tensor(_master(p)[1], device="cuda") for p in range(phases)]
    chunk = max(1, (24 << 20) // (h * w))
    for i in range(0, n, chunk):
        sl = slice(i, min(n, i + chunk))
        u = full.rays(full.t[sl] + shift[sl], masked=False)
        v = _rotate(q[sl].float()[:, None], u / u.norm(dim=-1, keepdim=True))
        m = _lookup(sheets[0], v)
        if phases == 2:
            m = torch.where(phase[sl][:, None] == 1, _lookup(sheets[1], v), m)
        lam = (counts * (0.6 + 0.4 * m.reshape(-1, h, w)) * hump).clamp(min=0)
        out[sl] = torch.poisson(lam, generator=g).clamp(0, 255 if case["pixel"] == "u8" else 65535).to(out.dtype)
    return out, q, phase


def _host(x):
    x = x.cpu().numpy()
    return x.astype(np.uint16) if x.dtype == np.int32 else x


def _settings(case):
    c = {"precision": case.get("precision", "f32"), "bandwidth": case.get("L", 64), "refine": case.get("refine", True),
         "binning": float(case.get("binning", 1)), "nlpar": case.get("nlpar", False),
         "accept_step_deg": ACCEPT_STEP_DEG}
    if case.get("roi"):
        c.update(roi_x=ROI_AT, roi_y=ROI_AT, roi_w=case["roi"], roi_h=case["roi"])
    if case.get("sweeps", 1) == 2:
        c.update(sweeps=2, sweep_bandwidth=32)
    return c


def prepare(case, seed):
    if case["kind"] == "match":
        return _prepare_match(case, seed)
    pats, q, _ = _scan(case, seed)
    host = _host(pats).reshape(case["rows"], case["cols"], case["h"], case["w"])
    s = ze.Solver()
    s.configure(**_settings(case))
    for k in range(case.get("phases", 1)):
        s.add_phase(_master(k)[0])
    s.set_patterns(host)
    s.set_geometry(pc=PC, sample_tilt_deg=TILT_DEG, detector_tilt_deg=0.0)
    state = {"case": case, "solver": s, "patterns": host}
    if case["kind"] == "refine6":
        state["cells"] = np.arange(case["rows"] * case["cols"])
        state["q0"] = _start(q, seed).cpu().numpy()
    return state


def _start(q, seed):
    """Starting orientations a degree or two off the true ones."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 104729 + 5)
    ax = torch.randn(len(q), 3, device="cuda", generator=g, dtype=F64)
    ang = torch.deg2rad(1 + torch.rand(len(q), 1, device="cuda", generator=g, dtype=F64))
    return _qstd(_qmul(_exp(ax / ax.norm(dim=1, keepdim=True) * ang), q))


def run(state):
    case = state["case"]
    if case["kind"] == "match":
        return _run_match(state)
    s = state["solver"]
    if case["kind"] == "refine6":
        return s.refine_patterns(state["cells"], quaternions=state["q0"], gradient=case["gradient"], rounds=5)
    if case["new_scan"]:
        s.set_patterns(state["patterns"])
    return s.index()


# ── the dictionary match, through the C ABI ──

def _match_inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 31 + 3)
    n, e, k = case["n"], case["entries"], case["cols"]
    d = torch.randn(e, k, device="cuda", generator=g) / torch.arange(1, k + 1, device="cuda").sqrt()
    d /= d.norm(dim=1, keepdim=True)
    x = d[torch.randint(0, e, (n,), device="cuda", generator=g)] + \
        0.02 * torch.randn(n, k, device="cuda", generator=g)
    x /= x.norm(dim=1, keepdim=True)
    q = torch.randn(e, 4, device="cuda", generator=g)
    return x.contiguous(), d.contiguous(), (q / q.norm(dim=1, keepdim=True)).contiguous()


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _prepare_match(case, seed):
    x, d, q = _match_inputs(case, seed)
    n, e, k = case["n"], case["entries"], case["cols"]
    lib = native.load()
    panels = [torch.empty(lib.zeb_panel_bytes(m, k), dtype=torch.uint8, device="cuda") for m in (n, e)]
    native.call("zeb_pack_panel", _p(d), e, k, k, _p(panels[1]), _stream())
    slices = lib.zeb_match_slices(n, e, k, 1)
    return {"case": case, "x": x, "d": d, "q": q, "panels": panels, "slices": slices,
            "cand_v": torch.empty(n, slices, 8, device="cuda"),
            "cand_i": torch.full((n, slices, 8), -1, dtype=torch.int32, device="cuda"),
            "status": torch.zeros(1, dtype=torch.int32, device="cuda"), "seeds": torch.zeros(n, 8, device="cuda")}


def _run_match(s):
    n, e, k = s["case"]["n"], s["case"]["entries"], s["case"]["cols"]
    native.call("zeb_pack_panel", _p(s["x"]), n, k, k, _p(s["panels"][0]), _stream())
    native.call("zeb_match_bf16", _p(s["panels"][0]), n, _p(s["panels"][1]), e, k, s["slices"], _p(s["cand_v"]),
                _p(s["cand_i"]), _p(s["status"]), _stream())
    native.call("zeb_match_best", _p(s["x"]), n, _p(s["d"]), e, k, _p(s["cand_i"]), s["slices"] * 8, _p(s["q"]),
                _p(s["seeds"]), _stream())
    return {"seeds": s["seeds"], "status": s["status"]}


def _exact_match(case, seed):
    x, d, q = _match_inputs(case, seed)
    seeds = torch.zeros(len(x), 8, dtype=F64, device="cuda")
    for i in range(0, len(x), 2048):
        v, at = (x[i:i + 2048].double() @ d.double().T).max(1)
        seeds[i:i + 2048, :4] = q[at].double()
        seeds[i:i + 2048, 4], seeds[i:i + 2048, 5] = v, at.double()
    return {"seeds": seeds, "status": None}


# ── the path in 64 bits ──

def _lattice(rows, cols, want):
    gy, gx = rows, cols
    if rows * cols > want:
        gy = int(min(max(round(math.sqrt(want * rows / cols)), 1), rows))
        gx = int(min(max(want // gy, 1), cols))
    r, c = (2 * np.arange(gy) + 1) * rows // (2 * gy), (2 * np.arange(gx) + 1) * cols // (2 * gx)
    return torch.as_tensor((r[:, None] * cols + c[None, :]).reshape(-1), device="cuda")


def _blur_matrix(n, sigma):
    """The Gaussian background's weights along an axis of n pixels (before normalization): direct
    taps to ceil(3σ) below σ = 12 pixels; above, boxes of ⌊σ/6⌋ pixels under a coarse Gaussian,
    spread back to the pixels by a narrow one."""
    x = np.arange(n)
    s = int(math.floor(sigma / 6))
    if s < 2:
        d = np.abs(x[:, None] - x[None, :])
        return np.where(d <= max(1, math.ceil(3 * sigma)), np.exp(-d * d / (2.0 * sigma * sigma)), 0.0)
    cs = math.sqrt(sigma * sigma - s * s - (s * s - 1) / 12)
    reach, pad = math.ceil(4 * cs), 3
    ns = -(-n // s)

    def cell(j):
        lo, hi = j * s, j * s + s
        if j >= 0 and lo < n:
            hi = min(hi, n)
        return 0.5 * (lo + hi - 1), float(hi - lo)

    box = np.zeros((ns, n))
    for j in range(ns):
        box[j, j * s:min((j + 1) * s, n)] = 1
    coarse = np.zeros((ns + 2 * pad, ns))
    for t in range(ns + 2 * pad):
        c = cell(t - pad)[0]
        for j in range(max(math.floor((c - reach) / s), 0), min(math.floor((c + reach) / s), ns - 1) + 1):
            coarse[t, j] = math.exp(-(cell(j)[0] - c) ** 2 / (2 * cs * cs))
    spread = np.zeros((n, ns + 2 * pad))
    for i in range(n):
        for t in range(2 * pad + 1):
            c, width = cell(i // s + t - pad)
            spread[i, i // s + t] = width * math.exp(-(i - c) ** 2 / (2.0 * s * s))
    return spread @ coarse @ box


def _load(pats, b):
    """Stored patterns → FP64, reduced by a whole binning."""
    p = pats.to(F64)
    if b > 1:
        n, h, w = p.shape
        p = p[:, : h // b * b, : w // b * b].reshape(n, h // b, b, w // b, b).mean((2, 4))
    return p


def _average_neighbours(p, rows, cols, radius=3, lam=0.7):
    """One pass of non-local averaging over (2·radius + 1)² cells."""
    n, h, w = p.shape
    P = p.reshape(rows, cols, h * w)

    def pairs(dy, dx):
        ys, yo = slice(max(-dy, 0), rows + min(-dy, 0)), slice(max(dy, 0), rows + min(dy, 0))
        xs, xo = slice(max(-dx, 0), cols + min(-dx, 0)), slice(max(dx, 0), cols + min(dx, 0))
        return (ys, xs), (yo, xo)

    offsets = [(dy, dx) for dy in range(-radius, radius + 1) for dx in range(-radius, radius + 1)
               if (dy or dx) and abs(dy) < rows and abs(dx) < cols]
    least = torch.full((rows, cols), math.inf, dtype=F64, device="cuda")
    dist = {}
    for o in offsets:
        a, b = pairs(*o)
        dist[o] = ((P[a] - P[b]) ** 2).mean(-1)
        if max(abs(o[0]), abs(o[1])) == 1:
            least[a] = torch.minimum(least[a], dist[o])
    sig = 0.5 * torch.where(torch.isfinite(least), least, torch.zeros_like(least))
    total, acc = torch.ones(rows, cols, dtype=F64, device="cuda"), P.clone()
    for o in offsets:
        a, b = pairs(*o)
        e, d = sig[a] + sig[b], dist[o]
        far = torch.exp(-math.sqrt(h * w / 2) * (d / e.clamp(min=1e-300) - 1) / lam ** 2)
        wt = torch.where(d <= e, torch.ones_like(d), torch.where(e > 0, far, torch.zeros_like(d)))
        acc[a] += wt[..., None] * P[b]
        total[a] += wt
    return (acc / total[..., None]).reshape(n, h, w)


def _filter(p, static, det):
    """Static and dynamic background subtracted, zero mean and unit norm under the mask."""
    p = p - static
    sigma = DYNAMIC_SIGMA * det.w
    By, Bx = (torch.as_tensor(_blur_matrix(m, sigma), device="cuda") for m in (det.h, det.w))
    By, Bx = By / By.sum(1, keepdim=True), Bx / Bx.sum(1, keepdim=True)
    p = (p - By @ p @ Bx.T)[:, det.mask]
    p = p - p.mean(1, keepdim=True)
    return p / p.norm(dim=1, keepdim=True)  # [n, masked pixels]


def _sheet_directions(side):
    x = torch.linspace(-1, 1, side, dtype=F64, device="cuda")
    X, Y = x[None, :].expand(side, side), x[:, None].expand(side, side)
    sc = math.sqrt(math.pi / 2)
    xa, ya = X.abs() * sc, Y.abs() * sc
    big = xa >= ya
    xn, yn = torch.maximum(xa, ya), torch.minimum(xa, ya)
    r = 2 * xn / math.pi * torch.sqrt((math.pi - xn * xn).clamp(min=0))
    ang = math.pi * yn / (4 * xn.clamp(min=1e-300))
    u, v = r * torch.cos(ang), r * torch.sin(ang)
    hx, hy = torch.where(big, u, v) * torch.where(X < 0, -1.0, 1.0), torch.where(big, v, u) * torch.where(Y < 0, -1.0, 1.0)
    z = 1 - 2 * xn * xn / math.pi
    d = torch.stack([torch.stack([hx, hy, z], -1), torch.stack([hx, hy, -z], -1)])
    return d / d.norm(dim=-1, keepdim=True)


def _tangents(d):
    ref = torch.zeros_like(d)
    far = d[..., 0].abs() > 0.8
    ref[..., 0], ref[..., 1] = torch.where(far, 0.0, 1.0), torch.where(far, 1.0, 0.0)
    e1 = torch.linalg.cross(d, ref)
    e1 = e1 / e1.norm(dim=-1, keepdim=True)
    return e1, torch.linalg.cross(d, e1)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _normalized(s):
    s = s - s.mean()
    return s / torch.sqrt((s * s).mean())


def _bake(k, angle):
    """Phase k's sheets as the detector's pixels see them: smoothed on the sphere by
    MASTER_SMOOTH pixels (the pixel's width in steps of 5 %), normalized; and their gradient table
    [2, side, side, 4]."""
    sheets = _normalized(torch.as_tensor(_master(k)[1], device="cuda").to(F64))
    px = angle * SIDE / math.sqrt(2 * math.pi)
    sigma = MASTER_SMOOTH * 1.05 ** math.floor(math.log(px) / math.log(1.05) + 0.5)
    d = _sheet_directions(SIDE)
    e1, e2 = _tangents(d)
    if sigma > 0.05:
        left, s = sigma * sigma, min(sigma, 2.0)
        while left > 1e-6:
            if s * s > left or left - s * s < 0.02 * left:
                s = math.sqrt(left)
            left -= s * s
            sr = s * math.sqrt(2 * math.pi) / SIDE
            acc, total = torch.zeros_like(sheets), 0.0
            for i in range(-4, 5):
                for j in range(-4, 5):
                    a, b = 0.6 * sr * i, 0.6 * sr * j
                    wt = math.exp(-(a * a + b * b) / (2 * sr * sr))
                    acc += wt * _lookup(sheets, _unit(d + a * e1 + b * e2))
                    total += wt
            sheets = acc / total
            s *= 2
        sheets = _normalized(sheets)
    h = math.sqrt(2 * math.pi) / SIDE
    g = sum(((_lookup(sheets, _unit(d + h * e)) - _lookup(sheets, _unit(d - h * e))) / (2 * h))[..., None] * e
            for e in (e1, e2))
    return sheets, torch.cat([g, sheets[..., None]], -1)


def _fft_size(L):
    n = 16
    while n < 2 * L - 1:
        n *= 2
    return n


def _legendre(L, x):
    """Normalized P̄_l^m(x) with the Condon–Shortley sign: [m][l − m][x]."""
    s = torch.sqrt((1 - x * x).clamp(min=0))
    pmm = torch.full_like(x, math.sqrt(1 / (4 * math.pi)))
    out = []
    for m in range(L):
        if m:
            pmm = -math.sqrt((2 * m + 1) / (2 * m)) * s * pmm
        col = [pmm]
        if m + 1 < L:
            col.append(math.sqrt(2 * m + 3) * x * pmm)
        for l in range(m + 2, L):
            a = math.sqrt((4 * l * l - 1) / (l * l - m * m))
            b = math.sqrt(((l - 1) ** 2 - m * m) / (4 * (l - 1) ** 2 - 1))
            col.append(a * (x * col[-1] - b * col[-2]))
        out.append(torch.stack(col))
    return out


def _rings(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return torch.as_tensor(x, device="cuda"), torch.as_tensor(w, device="cuda")


def _directions(x, n_phi):
    phi = 2 * math.pi * torch.arange(n_phi, dtype=F64, device="cuda") / n_phi
    s = torch.sqrt(1 - x * x)[:, None]
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), x[:, None].expand(-1, n_phi)], -1)


def _analyze(samples, w, plm):
    """Samples [..., rings, φ] → coefficients, one tensor [..., L − m] an order m."""
    F = torch.fft.rfft(samples, dim=-1) * (2 * math.pi / samples.shape[-1])
    return [((F[..., m] * w) @ p.T.to(C128)) for m, p in enumerate(plm)]


class _Sphere:
    """The spherical correlation at bandwidth L against a baked master."""

    def __init__(self, L, det, masters, folds):
        self.L, self.n, self.det = L, _fft_size(L), det
        x, self.wq = _rings(self.n)
        self.plm = _legendre(L, x)
        self.dirs = _directions(x, 2 * self.n)
        self.nd = self.dirs @ det.R[:, 2]
        win, _ = self._sample(None, det.t0[None])
        area = float((win * self.wq[:, None]).sum()) * 2 * math.pi / (2 * self.n)
        wlm = [c[None] for c in _analyze(win[0], self.wq, self.plm)]
        self.tables = []
        self._wigner(folds)
        for sheets, fold in zip(masters, folds):
            f, f2 = self._harmonics(sheets, fold)
            Y, Y2 = self._table(f, fold), self._table(f2, fold)
            v, v2 = self._volume(wlm, Y, fold), self._volume(wlm, Y2, fold)
            var = v2 - v * v / area
            rden = torch.where(var > 1e-6 * area, 1 / torch.sqrt(var.clamp(min=1e-300)), torch.zeros_like(var))
            self.tables.append((Y, rden, fold))
        self.d = None

    def _sample(self, pats, t):
        """Patterns (full frames, None: the window) on the sphere from sources t: (values, window)."""
        det = self.det
        h, w = det.h, det.w
        ok = self.nd > 1e-4
        hit = ((t @ det.R[:, 2])[:, None, None] / torch.where(ok, self.nd, torch.ones_like(self.nd)))[..., None] * \
            self.dirs - t[:, None, None, :]
        row, col = hit @ det.R[:, 0], hit @ det.R[:, 1]
        r = 0.5 * min(h, w)
        inside = ok & (row >= 0) & (row <= h - 1) & (col >= 0) & (col <= w - 1) & \
            ((row - 0.5 * (h - 1)) ** 2 + (col - 0.5 * (w - 1)) ** 2 <= r * r)
        win = inside.to(F64)
        if pats is None:
            return win, win
        row, col = torch.where(inside, row, torch.zeros_like(row)), torch.where(inside, col, torch.zeros_like(col))
        r0, c0 = row.floor().clamp(max=h - 2).long(), col.floor().clamp(max=w - 2).long()
        fr, fc = row - r0, col - c0
        o = (r0 * w + c0).reshape(len(t), -1)

        def at(k):
            return torch.gather(pats, 1, o + k).reshape(row.shape)

        val = (at(0) * (1 - fc) + at(1) * fc) * (1 - fr) + (at(w) * (1 - fc) + at(w + 1) * fc) * fr
        return val * win, win

    def _harmonics(self, sheets, fold):
        """The master's coefficients up to L (its mean left out, the orders its symmetry forbids
        zeroed) and those of its square: [l, m ≥ 0]."""
        L = self.L
        nt = max(4 * L, 512)
        x, w = _rings(nt)
        # the sheets meet the sphere at 32 bits, as every user's stored master does
        c = _analyze(_lookup(sheets.float().to(F64), _directions(x, 2 * nt)), w, _legendre(L, x))
        f = torch.zeros(L, L, dtype=C128, device="cuda")
        for m in range(L):
            f[m:, m] = c[m]
        f[0, 0] = 0
        l, m = torch.arange(L, device="cuda")[:, None], torch.arange(L, device="cuda")[None, :]
        e = f.abs() ** 2 * torch.where(m == 0, 1.0, 2.0)
        total = e.sum()
        keep = torch.ones_like(e, dtype=torch.bool)
        if e[l[:, 0] % 2 == 1].sum() < 1e-5 * total:
            keep &= l % 2 == 0
        if torch.where((l + m) % 2 == 1, e, 0.0).sum() < 1e-5 * total:
            keep &= (l + m) % 2 == 0
        for order in (6, 4, 3, 2):
            if torch.where(m % order != 0, e, 0.0).sum() < 1e-5 * total:
                keep &= m % order == 0
                break
        f = torch.where(keep, f, torch.zeros_like(f))
        x, w = _rings(2 * L)
        plm = _legendre(L, x)
        G = torch.stack([(plm[m].to(C128) * f[m:, m, None]).sum(0) for m in range(L)], -1)
        s = torch.fft.irfft(G, n=4 * L, dim=-1) * 4 * L
        c = _analyze(s * s, w, plm)
        f2 = torch.zeros_like(f)
        for m in range(L):
            f2[m:, m] = c[m]
        return f, f2

    def _wigner(self, folds):
        """d^l_{m'm}(b_j) at b_j = 2πj/n, j ≤ n/2, from the eigenvectors of J_y: [l] of [j][m' ≥ 0][m]."""
        beta = 2 * math.pi * torch.arange(self.n // 2 + 1, dtype=F64, device="cuda") / self.n
        self.d = []
        for l in range(self.L):
            m = torch.arange(-l, l, dtype=F64, device="cuda")
            up = torch.sqrt(l * (l + 1) - m * (m + 1))
            Jy = torch.zeros(2 * l + 1, 2 * l + 1, dtype=C128, device="cuda")
            i = torch.arange(2 * l, device="cuda")
            Jy[i + 1, i], Jy[i, i + 1] = up / 2j, -up / 2j
            _, V = torch.linalg.eigh(Jy)
            lam = torch.arange(-l, l + 1, dtype=F64, device="cuda")
            e = torch.exp(-1j * beta[:, None] * lam)
            self.d.append(((V[None, l:] * e[:, None, :]) @ V.conj().T).real)

    def _table(self, f, fold):
        """Y[m'] of [l − m'][j·nc + c]: the sums over the master's orders of f_lm d^l_{m'm}(b_j) e^{−imc}."""
        L, n = self.L, self.n
        nc, nb = n // fold, n // 2 + 1
        Y = [torch.zeros(L - mp, nb * nc, dtype=C128, device="cuda") for mp in range(L)]
        c = 2 * math.pi * torch.arange(nc, dtype=F64, device="cuda") / n
        for l in range(L):
            m = torch.arange(-(l // fold) * fold, l + 1, fold, device="cuda")
            fl = f[l, m.abs()]
            fl = torch.where(m < 0, fl.conj() * torch.where(m % 2 == 0, 1.0, -1.0), fl)
            T = (self.d[l][:, :, m + l].to(C128) * fl) @ torch.exp(-1j * m[:, None].to(F64) * c)  # [j][m'][c]
            for mp in range(l + 1):
                Y[mp][l - mp] = T[:, mp].reshape(-1)
        return Y

    def _volume(self, g, Y, fold):
        """Correlations [n][j][c][a] of coefficients g with a table."""
        L, n = self.L, self.n
        nc, nb = n // fold, n // 2 + 1
        U = torch.zeros(len(g[0]), nb, nc, n // 2 + 1, dtype=C128, device="cuda")
        for mp in range(L):
            U[..., mp] = (g[mp] @ Y[mp].conj()).reshape(-1, nb, nc)  # (conj of conj(g) Y, for the inverse FFT)
        return torch.fft.irfft(U, n=n, dim=-1) * n

    def peaks(self, pats, t):
        """The best orientation and score of each pattern (masked values) with each master."""
        det = self.det
        full = torch.zeros(len(pats), det.h * det.w, dtype=F64, device="cuda")
        full[:, det.mask.reshape(-1)] = pats
        out = [[] for _ in self.tables]
        cells = self.n ** 3 // 2 // min(f for _, _, f in self.tables)
        step = max(1, min((96 << 20) // cells, (64 << 20) // (2 * self.n * self.n)))
        for i in range(0, len(pats), step):
            val, win = self._sample(full[i:i + step], t[i:i + step])
            wq = self.wq[:, None]
            mean = (val * wq).sum((1, 2)) / (win * wq).sum((1, 2))
            g = _analyze((val - mean[:, None, None]) * win, self.wq, self.plm)
            power = sum((c.abs() ** 2).sum(-1) * (1 if m == 0 else 2) for m, c in enumerate(g))
            g = [c / torch.sqrt(power)[:, None] for c in g]
            for k, (Y, rden, fold) in enumerate(self.tables):
                out[k].append(self._peak(self._volume(g, Y, fold) * rden, fold))
        return [torch.cat(o) for o in out]

    def _peak(self, vol, fold):
        n, nb = self.n, self.n // 2 + 1
        nc = n // fold
        m = len(vol)
        flat = vol.reshape(m, -1)
        v0, at = flat.max(1)
        j, c, a = at // (nc * n), at // n % nc, at % n
        who = torch.arange(m, device="cuda")

        def vertex(lo, hi):
            den = lo - 2 * v0 + hi
            return torch.where(den >= -1e-12, torch.zeros_like(den), (0.5 * (lo - hi) / den).clamp(-0.5, 0.5))

        da = vertex(vol[who, j, c, (a - 1) % n], vol[who, j, c, (a + 1) % n])
        dc = vertex(vol[who, j, (c - 1) % nc, a], vol[who, j, (c + 1) % nc, a])
        inner = (j > 0) & (j < n // 2)
        dj = vertex(vol[who, (j - 1).clamp(min=0), c, a], vol[who, (j + 1).clamp(max=nb - 1), c, a])
        dj = torch.where(inner, dj, torch.zeros_like(dj))
        A, B, C = ((k + d) * (2 * math.pi / n) for k, d in ((a, da), (j, dj), (c, dc)))
        # conj(Rz(A) Ry(B) Rz(C))
        cb, sb = torch.cos(B / 2), torch.sin(B / 2)
        q = torch.stack([cb * torch.cos((A + C) / 2), sb * torch.sin((A - C) / 2), -sb * torch.cos((A - C) / 2),
                         -cb * torch.sin((A + C) / 2)], 1)
        return _qstd(q)


def _solve(H, g):
    return torch.linalg.solve(H, g[..., None])[..., 0]


def _refine(det, t, q, pats, grad, iters):
    """Gauss–Newton on the orientation, iters steps from the best point so far: (q, NCC, the last
    improving step's length)."""
    n, N = len(q), pats.shape[1]
    u = _unit(det.rays(t))
    best = torch.full((n,), -2.0, dtype=F64, device="cuda")
    mu = torch.ones(n, dtype=F64, device="cuda")
    promised = torch.zeros_like(mu)
    accepted = torch.zeros(n, dtype=torch.bool, device="cuda")
    taken, last = torch.zeros_like(mu), torch.zeros_like(mu)
    qb, gb, Hb = q.clone(), torch.zeros(n, 3, dtype=F64, device="cuda"), torch.zeros(n, 3, 3, dtype=F64, device="cuda")
    for it in range(iters + 1):
        c = _rotate(q[:, None], u)
        G = _lookup(grad, c)
        m = G[..., 3]
        D = torch.linalg.cross(c, G[..., :3])
        mean = m.mean(1)
        inv = 1 / torch.sqrt((m * m).sum(1) - N * mean * mean)
        ncc = (m * pats).sum(1) * inv
        sd = D.sum(1)
        au = ((m[..., None] * D).sum(1) - mean[:, None] * sd) * inv[:, None]
        g = ((pats[..., None] * D).sum(1) - ncc[:, None] * au) * inv[:, None]
        H = (D.transpose(1, 2) @ D - sd[:, :, None] * sd[:, None] / N - au[:, :, None] * au[:, None]) * \
            (inv * inv)[:, None, None]
        up = ncc > best
        rho = (ncc - best) / promised.clamp(min=1e-300)
        gain = torch.minimum(torch.maximum(mu * (2 - rho), mu / 3), mu * 3)
        mu = torch.where(up, torch.where(accepted & (promised > 1e-6), gain, mu), mu * 3).clamp(0.02, 1e4)
        qb, gb = torch.where(up[:, None], q, qb), torch.where(up[:, None], g, gb)
        last = torch.where(up, taken, last)
        Hb, best, accepted = torch.where(up[:, None, None], H, Hb), torch.where(up, ncc, best), accepted | up
        if it == iters:
            break
        Hs = Hb * mu[:, None, None]
        tr = Hs.diagonal(dim1=1, dim2=2).sum(1).clamp(min=1e-20)
        Hs = Hs + 1e-6 * tr[:, None, None] * torch.eye(3, dtype=F64, device="cuda")
        step = _solve(Hs, gb)
        ln = step.norm(dim=1, keepdim=True)
        step = step * torch.where(ln > math.radians(REFINE_STEP_DEG), math.radians(REFINE_STEP_DEG) / ln, torch.ones_like(ln))
        promised = (gb * step).sum(1) - 0.5 * (step[:, None] @ Hs @ step[..., None])[:, 0, 0]
        taken = step.norm(dim=1)
        q = _qmul(_exp(step), qb)
        q = q / q.norm(dim=1, keepdim=True)
    return qb, best, last


def _nmi(det, t, q, pats, sheets):
    """2 I(A;B) / (H(A) + H(B)) of the patterns with the simulations, binned between their extremes."""
    s = _lookup(sheets, _rotate(q[:, None], _unit(det.rays(t))))
    n, N, B = len(q), pats.shape[1], NMI_BINS

    def bins(v):
        lo = v.amin(1, keepdim=True)
        return ((v - lo) * (B / (v.amax(1, keepdim=True) - lo))).long().clamp(max=B - 1)

    at = bins(pats) * B + bins(s) + torch.arange(n, device="cuda")[:, None] * B * B
    hist = torch.bincount(at.reshape(-1), minlength=n * B * B).reshape(n, B, B).to(F64) / N

    def entropy(p):
        return -torch.xlogy(p, p).sum(-1)

    marg = entropy(hist.sum(2)) + entropy(hist.sum(1))
    return 2 * (marg - entropy(hist.reshape(n, -1))) / marg


def _chance(det, cells, pats, sheets, draws=8):
    """(median, spread) of the NMI of up to 256 patterns at random orientations (Shoemake's, from a
    32-bit hash of the pattern's number and the draw's)."""
    def rand(x):
        x = x & 0xFFFFFFFF
        v = (x * 747796405 + 2891336453) & 0xFFFFFFFF
        w = (((v >> ((v >> 28) + 4)) ^ v) * 277803737) & 0xFFFFFFFF
        return ((w >> 22) ^ w) & 0xFFFFFFFF

    b = torch.arange(len(cells), device="cuda")
    got = []
    for k in range(draws):
        s = rand(b + 1) ^ ((k * 0x9E3779B9) & 0xFFFFFFFF)
        u, a, c = ((rand(s + i) >> 8).to(F64) / 16777216.0 for i in range(3))
        a, c = 2 * math.pi * a, 2 * math.pi * c
        ra, rb = torch.sqrt(1 - u), torch.sqrt(u)
        q = torch.stack([ra * torch.sin(a), ra * torch.cos(a), rb * torch.sin(c), rb * torch.cos(c)], 1)
        got.append(_nmi(det, det.t[cells], q, pats, sheets))
    v = torch.cat(got).sort().values
    med = v[len(v) // 2]
    return med, (1.4826 * (v - med).abs().sort().values[len(v) // 2]).clamp(min=1e-6)


def _reduced(q, ops):
    """Orientations in the fundamental zone: the equivalent of largest w."""
    c = _qstd(_qmul(ops.to("cuda")[None], q[:, None]))
    return c[torch.arange(len(q), device="cuda"), c[..., 0].argmax(1)]


def _bunge(q):
    w, x, y, z = q.unbind(-1)
    chi = torch.sqrt((w * w + z * z) * (x * x + y * y))
    e = torch.stack([torch.atan2(x * z - w * y, -w * x - y * z), torch.atan2(2 * chi, w * w + z * z - x * x - y * y),
                     torch.atan2(w * y + x * z, y * z - w * x)], -1)
    return torch.where(e < 0, e + 2 * math.pi, e)


def _exact_index(case, seed):
    stored, _, _ = _scan(case, seed)
    det = _Detector(case)
    rows, cols, b = case["rows"], case["cols"], case["binning"]
    n = rows * cols
    static = _load(stored[_lattice(rows, cols, STATIC_PATTERNS)], b).mean(0)
    if case["nlpar"]:
        averaged = _average_neighbours(_load(stored, b), rows, cols)

    def patterns(cells):
        return _filter(averaged[cells] if case["nlpar"] else _load(stored[cells], b), static, det)

    baked = [_bake(k, det.angle) for k in range(case["phases"])]
    folds = [4 if MASTERS[k][0] == "432" else 2 for k in range(case["phases"])]
    left = torch.arange(n, device="cuda").reshape(rows, cols)
    if case["roi"]:
        left = left[ROI_AT:ROI_AT + case["roi"], ROI_AT:ROI_AT + case["roi"]]
    left = left.reshape(-1)
    some = min(len(left), 256)
    cells = left[torch.as_tensor(((2 * np.arange(some) + 1) * len(left)) // (2 * some), device="cuda")]
    calm = [_chance(det, cells, patterns(cells), s) for s, _ in baked]
    chunk = max(1, (3 << 20) // _mask_pixels(det.h, det.w))
    r = torch.zeros(n, 8, dtype=F64, device="cuda")  # q, NCC, NMI, z, the last improving step
    r[:, 0] = 1  # (cells outside the region of interest)
    euler = torch.zeros(n, 3, dtype=F64, device="cuda")
    for sweep, L in enumerate([32, case["L"]][2 - case["sweeps"]:]):
        sphere = _Sphere(L, det, [s for s, _ in baked], folds) if len(left) else None
        for i in range(0, len(left), chunk):
            c = left[i:i + chunk]
            p, t = patterns(c), det.t[c]
            per = []
            for k, seeds in enumerate(sphere.peaks(p, t)):
                q, ncc, step = _refine(det, t, seeds, p, baked[k][1], REFINE_ITERS if case["refine"] else 0)
                nmi = _nmi(det, t, q, p, baked[k][0])
                per.append(torch.cat([_reduced(q, _master(k)[2]), torch.stack(
                    [ncc, nmi, (nmi - calm[k][0]) / calm[k][1], step], 1)], 1))
            per = torch.stack(per)
            new = per[per[..., 5].argmax(0), torch.arange(len(c), device="cuda")]
            # a later sweep's match is taken where it is accepted or better
            good = (new[:, 6] >= ACCEPT_Z) & (new[:, 7] <= math.radians(ACCEPT_STEP_DEG))
            better = good | (new[:, 6] > r[c, 6]) | (sweep == 0)
            r[c] = torch.where(better[:, None], new, r[c])
            euler[c] = _bunge(r[c, :4])
        left = left[(r[left, 6] < ACCEPT_Z) | (r[left, 7] > math.radians(ACCEPT_STEP_DEG))]
    return {"quaternions": r[:, :4].reshape(rows, cols, 4), "euler": euler.reshape(rows, cols, 3),
            "ncc": r[:, 4].reshape(rows, cols), "nmi": r[:, 5].reshape(rows, cols), "z": r[:, 6].reshape(rows, cols),
            "phase": None, "sweep": None}


def _projected(det, t, q, shift, pats, sheets):
    """NCC of the patterns with the master seen from shifted sources."""
    m = _lookup(sheets, _rotate(q[:, None], _unit(det.rays(t + shift))))
    m = m - m.mean(1, keepdim=True)
    return (m * pats).sum(1) / m.norm(dim=1)


def _local(det, t, q, shift, pats, sheets, grad, adjoint):
    """NCC, its gradient over (shift, rotation) and the Gauss–Newton matrix, a pattern."""
    u = det.rays(t + shift)
    dist = u.norm(dim=-1, keepdim=True)
    c = _rotate(q[:, None], u / dist)
    G = _lookup(grad, c)
    m, N = G[..., 3], pats.shape[1]
    conj = q[:, None] * torch.tensor([1.0, -1, -1, -1], dtype=F64, device="cuda")
    D = torch.cat([_rotate(conj, G[..., :3]) / dist, torch.linalg.cross(c, G[..., :3])], -1)
    mean = m.mean(1)
    inv = 1 / torch.sqrt((m * m).sum(1) - N * mean * mean)
    ncc = (m * pats).sum(1) * inv
    sd = D.sum(1)
    au = ((m[..., None] * D).sum(1) - mean[:, None] * sd) * inv[:, None]
    g = ((pats[..., None] * D).sum(1) - ncc[:, None] * au) * inv[:, None]
    H = (D.transpose(1, 2) @ D - sd[:, :, None] * sd[:, None] / N - au[:, :, None] * au[:, None]) * (inv * inv)[:, None, None]
    if adjoint:  # the exact derivative of the projection itself
        s = shift.clone().requires_grad_(True)
        f = torch.zeros_like(shift).requires_grad_(True)
        total = _projected(det, t, _qmul(_small(f), q), s, pats, sheets).sum()
        g = torch.cat(torch.autograd.grad(total, (s, f)), 1)
    return ncc, g, H


def _small(f):
    """exp of rotation vectors about 0, to the first order (all a derivative there sees)."""
    return torch.cat([torch.ones_like(f[:, :1]), 0.5 * f], 1)


def _exact_refine6(case, seed, rounds=5):
    stored, q_true, _ = _scan(case, seed)
    det = _Detector(case)
    rows, cols, h, w = case["rows"], case["cols"], case["h"], case["w"]
    n = rows * cols
    static = _load(stored[_lattice(rows, cols, STATIC_PATTERNS)], 1).mean(0)
    sheets, grad = _bake(0, det.angle)
    q0 = _qstd(_start(q_true, seed))
    eye = torch.eye(6, dtype=F64, device="cuda")
    trust = 0.05 * h
    parts = []
    chunk = max(1, (3 << 20) // _mask_pixels(h, w))
    for i in range(0, n, chunk):
        c = torch.arange(i, min(n, i + chunk), device="cuda")
        p, t, q = _filter(_load(stored[c], 1), static, det), det.t[c], q0[c]
        shift = torch.zeros(len(c), 3, dtype=F64, device="cuda")
        lam = torch.full((len(c),), 1e-3, dtype=F64, device="cuda")
        ncc, g, H = _local(det, t, q, shift, p, sheets, grad, case["gradient"] == "adjoint")
        for _ in range(rounds):
            diag = H.diagonal(dim1=1, dim2=2)
            A = H + eye * (diag * lam[:, None])[:, :, None] + eye * (1e-9 * diag.sum(1))[:, None, None]
            d = _solve(A, g)
            st, qt = (shift + d[:, :3]).clamp(-trust, trust), _qstd(_qmul(_exp(d[:, 3:]), q))
            now = _local(det, t, qt, st, p, sheets, grad, case["gradient"] == "adjoint")
            up = now[0] > ncc
            q, shift = torch.where(up[:, None], qt, q), torch.where(up[:, None], st, shift)
            ncc, g = torch.where(up, now[0], ncc), torch.where(up[:, None], now[1], g)
            H = torch.where(up[:, None, None], now[2], H)
            lam = torch.where(up, (lam / 3).clamp(min=1e-4), (lam * 5).clamp(max=1e8))
        parts.append(torch.cat([q, shift, ncc[:, None]], 1))
    r = torch.cat(parts)
    J = torch.stack([det.R @ torch.tensor(v, dtype=F64, device="cuda") for v in
                     ((0.0, -float(w), 0.0), (-float(h), 0.0, 0.0), (0.0, 0.0, float(h)))], 1)
    pc = torch.tensor(PC, dtype=F64, device="cuda") + r[:, 4:7] @ torch.linalg.inv(J).T
    return {"quaternions": r[:, :4], "shift": r[:, 4:7], "pc": pc, "ncc": r[:, 7], "rounds": None}


def exact(case, seed):
    if case["kind"] == "match":
        return _exact_match(case, seed)
    if case["kind"] == "refine6":
        return _exact_refine6(case, seed)
    return _exact_index(case, seed)
