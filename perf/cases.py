"""The calls whose speed is measured: the SRRF map of a series (device, host, block lists, time batches), the drift
refinement's forward and backward, and the 3B localisation step's two inner calls (spot optimisation, Gibbs draws).

A case names its call ("kind"), the series [T][D][H][W], the magnification per axis and the options that matter;
everything else is the configuration the benchmark workloads use (ring radius 0.5, 6 axes, smoothed gradient with
ranges 1, intensity weighting). Series are made on the GPU: blinking Gaussian emitters over a background with Poisson
and read noise, the model of rfba_gb300/synth.py."""
import math

import numpy as np
import torch

from rfba_gb300 import drift, srrf

DEV = "cuda"
METHODS = {"TRM": 0, "TRA": 1, "TRPPM": 2, "TRAC": 3}


def listed():
    def srrf_case(name, kind, T, D, H, W, mag, method, order=2, itc=0, dtype="u16", emitters=40, curves=0, **more):
        return {"name": name, "kind": kind, "T": T, "D": D, "H": H, "W": W, "mx": mag[0], "my": mag[1], "mz": mag[2],
                "method": method, "order": order, "itc": itc, "dtype": dtype, "emitters": emitters, "curves": curves,
                "smooth": 1, **more}

    return [
        # a crop around one structure, looked at while parameters are chosen: latency and launches count
        srrf_case("forward_tiny", "forward", 5, 10, 12, 12, (2, 2, 2), "TRA", emitters=10),
        # the small benchmark series
        srrf_case("forward_small", "forward", 30, 32, 32, 32, (2, 2, 2), "TRA"),
        # the reference's own entry point on one float block in host memory, shipped defaults: magnification 5, no
        # gradient smoothing, temporal mean
        {**srrf_case("legacy_host_block", "legacy", 20, 16, 20, 20, (5, 5, 5), "TRA", itc=1, dtype="f32"), "smooth": 0},
        # a float series cropped to an odd box, third-order cumulants
        srrf_case("forward_odd_f32", "forward", 37, 33, 61, 75, (3, 3, 3), "TRAC", order=3, dtype="f32", emitters=120),
        # integrated lag times (the shipped ITC default) at magnification 4
        srrf_case("forward_itc1", "forward", 64, 24, 48, 48, (4, 4, 4), "TRAC", order=4, itc=1, emitters=80),
        # the mid-size series at 4 x 4 x 2: the headline workload
        srrf_case("forward_mid", "forward", 100, 64, 128, 128, (4, 4, 2), "TRAC", emitters=600, curves=20),
        # a series cut into 29^3 blocks with 1 voxel of border and uneven edge blocks, as before localisation
        srrf_case("blocks_29", "blocks", 50, 64, 70, 80, (3, 3, 3), "TRA", emitters=400, curves=12),
        # a series too long for its stacks, reduced in batches of 25 volumes
        srrf_case("forward_batches", "batches", 100, 32, 64, 64, (4, 4, 2), "TRAC", order=4, emitters=150, batch=25),
        # one iteration of the drift refinement: drift-corrected map, its objective's derivative, the adjoint
        srrf_case("drift_pair", "drift", 60, 64, 64, 64, (2, 2, 2), "TRAC", dtype="f32", emitters=300),
        # the same on a small crop at 4 x 4 x 2, fourth-order cumulants
        srrf_case("drift_pair_small", "drift", 12, 18, 37, 45, (4, 4, 2), "TRAC", order=4, dtype="f32", emitters=60),
        # 3B: one spot's conjugate-gradient optimisation on 10 background draws of a 29^3 block
        {"name": "spot_optimise", "kind": "spot", "S": 10, "F": 100, "D": 29, "H": 29, "W": 29},
        # 3B: 10 Gibbs draws of 20 spots' states on a 29^3 block
        {"name": "gibbs_draws", "kind": "gibbs", "K": 20, "F": 100, "D": 29, "H": 29, "W": 29, "draws": 10},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["forward", "forward", "forward", "legacy", "blocks", "batches", "drift", "drift", "spot", "gibbs"])
    if kind == "spot":
        return {"kind": kind, "S": rng.randint(4, 20), "F": log_int(20, 150), "D": rng.randint(9, 29),
                "H": rng.randint(9, 29), "W": rng.randint(9, 29)}
    if kind == "gibbs":
        return {"kind": kind, "K": rng.randint(4, 24), "F": log_int(20, 150), "D": rng.randint(9, 29),
                "H": rng.randint(11, 29), "W": rng.randint(11, 29), "draws": rng.randint(2, 10)}
    c = {"kind": kind}
    mag = rng.choice([(2, 2, 2), (3, 3, 3), (4, 4, 2), (4, 4, 4), (5, 5, 5), (2, 2, 1)])
    # voxel-volumes of the map: up to half of the largest listed case's for a forward, a fifth of that where each
    # costs several times as much or goes through host memory
    units = math.exp(rng.uniform(math.log(1e6), math.log(1.6e9 if kind == "forward" else 2.5e8)))
    c["T"] = log_int(40, 120) if kind == "batches" else log_int(6, 120)
    if kind == "legacy":
        mag, units = (rng.choice([2, 3, 4, 5]),) * 3, min(units, 4e7)
    side = (units / c["T"] / (mag[0] * mag[1] * mag[2])) ** (1 / 3)
    lo = 32 if kind == "blocks" else 8
    c["D"] = max(lo, int(round(side * rng.uniform(0.5, 1.0))))
    c["H"] = max(lo, int(round(side * rng.uniform(0.8, 1.3))))
    c["W"] = max(lo, int(round(side * rng.uniform(0.8, 1.3))))
    if rng.random() < 0.3:
        c["W"] = (c["W"] + 7) // 8 * 8
    c["mx"], c["my"], c["mz"] = mag
    c["method"] = "TRAC" if kind in ("batches", "drift") else rng.choice(["TRA", "TRAC", "TRAC", "TRPPM", "TRM"])
    c["order"] = rng.choice([2, 2, 3, 4])
    c["itc"] = 1 if kind in ("forward", "legacy") and rng.random() < 0.25 else 0
    c["dtype"] = "f32" if kind in ("drift", "legacy") else rng.choice(["u16", "u16", "f32"])
    c["emitters"] = max(8, min(600, c["D"] * c["H"] * c["W"] // 900))
    c["curves"] = 0
    c["smooth"] = 0 if kind == "legacy" and rng.random() < 0.5 else 1
    if kind == "batches":
        c["batch"] = 25
    return c


# ---- inputs ------------------------------------------------------------------

def _series(case, g, drifted):
    """[T][D][H][W] float32 on the GPU and the drift [T][3] that was put in."""
    T, D, H, W, n = case["T"], case["D"], case["H"], case["W"], case["emitters"]
    f64 = {"dtype": torch.float64, "device": DEV}
    dims = torch.tensor([W, H, D], **f64)
    if case["curves"]:
        c = case["curves"]
        ctrl = 3 + torch.rand(c, 4, 3, generator=g, **f64) * (dims - 6)
        ctrl = ctrl[torch.arange(n, device=DEV) % c]
        s = torch.rand(n, 1, generator=g, **f64)
        pos = ((1 - s) ** 3 * ctrl[:, 0] + 3 * (1 - s) ** 2 * s * ctrl[:, 1] + 3 * (1 - s) * s * s * ctrl[:, 2]
               + s ** 3 * ctrl[:, 3])
    else:
        pos = 2 + torch.rand(n, 3, generator=g, **f64) * (dims - 4)
    on = torch.zeros(T, n, **f64)
    state = torch.rand(n, generator=g, **f64) < 0.25
    for t in range(T):
        on[t] = state.double()
        u = torch.rand(n, generator=g, **f64)
        state = torch.where(state, u >= 0.3, u < 0.1)
    walk = torch.zeros(T, 3, **f64)
    if drifted:
        step = 0.15 * torch.randn(T, 3, generator=g, **f64)
        step[0] = 0
        walk = torch.cumsum(step, 0)

    def axis(mu, sigma, length):
        edges = torch.arange(length + 1, **f64)
        c = torch.special.erf((edges - mu[..., None]) / (sigma * math.sqrt(2)))
        return 0.5 * (c[..., 1:] - c[..., :-1])

    out = torch.empty(T, D, H, W, dtype=torch.float32, device=DEV)
    for t in range(T):
        p = pos - walk[t]  # the shift that undoes it is +walk
        wx, wy, wz = axis(p[:, 0], 1.2, W), axis(p[:, 1], 1.2, H), axis(p[:, 2], 2.5, D)
        zy = (500.0 * on[t])[:, None, None] * wz[:, :, None] * wy[:, None, :]
        lam = 100.0 + (zy.reshape(n, D * H).t().float() @ wx.float()).reshape(D, H, W).clamp_min(0)
        noise = torch.randn(D, H, W, generator=g, device=DEV)
        out[t] = torch.poisson(lam, generator=g) + 2.0 * noise
    return out, walk


def _config(case):
    return srrf.Config.make(mag=(case["mx"], case["my"], case["mz"]), method=METHODS[case["method"]], itc=case["itc"],
                            trac_order=case["order"], gradient_smooth=case["smooth"], main_range=1, x_range=1,
                            y_range=1, z_range=1, intensity_w=1, axes_in_ring=6, ring_radius=0.5)


_handles = {}


def _context(batch=0):
    """The program's context, kept between calls (one for each time-batch setting)."""
    if batch not in _handles:
        c = srrf.Context(0)
        if batch:
            c.set_time_batch(batch)
        _handles[batch] = c
    return _handles[batch]


def _threeb_model():
    return srrf.ThreeBModel.make([[0.16, 0.84, 0.0], [0.495, 0.495, 0.01], [0.0, 0.0, 1.0]], [0.5, 0.5, 0.0])


def _threeb_block(case, g, n_spots):
    """Voxels [P][3] in (z, y, x) order, spot shapes, the spots and a generator of series."""
    D, H, W = case["D"], case["H"], case["W"]
    f64 = {"dtype": torch.float64, "device": DEV}
    zz, yy, xx = torch.meshgrid(torch.arange(D, device=DEV), torch.arange(H, device=DEV), torch.arange(W, device=DEV),
                                indexing="ij")
    px = torch.stack([xx.reshape(-1), yy.reshape(-1), zz.reshape(-1)], 1).to(torch.int32)
    dims = torch.tensor([W, H, D], **f64)
    centre = 2 + torch.rand(n_spots, 3, generator=g, **f64) * (dims - 5)
    bright = 30 + 50 * torch.rand(n_spots, generator=g, **f64)
    blur = 0.9 + 0.5 * torch.rand(n_spots, generator=g, **f64)
    d = px.double()[None] - centre[:, None]
    shapes = (bright / (blur * math.sqrt(2 * math.pi)))[:, None] * torch.exp(-(d * d).sum(2) / (2 * blur ** 2)[:, None])
    return px, shapes, centre, bright, blur


def prepare(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    kind = case["kind"]
    if kind == "spot":
        S, F = case["S"], case["F"]
        px, shapes, centre, bright, blur = _threeb_block(case, g, 6)
        on = (torch.rand(F, 6, generator=g, device=DEV) < 0.5).double()
        pix = on @ shapes + torch.randn(F, len(px), generator=g, dtype=torch.float64, device=DEV)
        son = (torch.rand(S, F, 6, generator=g, device=DEV) < 0.5).double()
        son[:, :, 0] = 0
        spot = np.array([float(bright[0]) * 0.9, float(blur[0]) * 1.1, *(centre[0] + 0.3).tolist()])
        lim = np.array([0.5 * math.sqrt((math.exp(1.0) - 1) * math.exp(2 * 3.5 + 1.0)), 0.5, 0.5, 0.5, 0.5])
        return {"case": case, "ctx": _context(), "model": _threeb_model(), "bg": (son @ shapes).contiguous(),
                "pix": pix.contiguous(), "px": px, "spot": spot, "limit": lim}
    if kind == "gibbs":
        K, F = case["K"], case["F"]
        px, shapes, centre, bright, blur = _threeb_block(case, g, K)
        on = (torch.rand(F, K, generator=g, device=DEV) < 0.25).double()
        pix = on @ shapes + torch.randn(F, len(px), generator=g, dtype=torch.float64, device=DEV)
        near = centre + 0.2 * torch.randn(K, 3, generator=g, dtype=torch.float64, device=DEV)
        spots = torch.cat([bright[:, None], blur[:, None], near], 1).cpu().numpy()
        pixels = px.cpu().numpy()
        return {"case": case, "ctx": _context(), "model": _threeb_model(), "pix": pix.cpu().numpy(), "px": pixels,
                "spots": spots, "masks": srrf.spot_masks_3b(pixels, spots), "seed": int(seed)}
    x, walk = _series(case, g, kind == "drift")
    s = {"case": case, "cfg": _config(case), "ctx": _context(case.get("batch", 0))}
    if kind == "drift":
        # a refinement somewhere between its start and the truth
        s["x"], s["shifts"] = x, (0.5 * walk + 0.25).float().contiguous()
        s["map"] = torch.empty(_map_shape(case), device=DEV)
        s["din"], s["dshift"] = torch.empty_like(x), torch.empty_like(s["shifts"])
        return s
    if kind == "legacy":
        conf = srrf.SRRFConf(RingRadius=0.5, Magnification=case["mx"], AxesinRing=6, MainRange=1, XRange=1, YRange=1,
                             ZRange=1, Method=METHODS[case["method"]], ITC=case["itc"], TRACOrder=case["order"],
                             RemoveCon=0, Renormalize=0, GradientSmooth=case["smooth"], IntensityW=1, blockSizeX=16,
                             blockSizeY=16, blockSizeZ=16)
        # 3B hands over series in units of their standard deviation
        return {"case": case, "conf": conf, "x": (x / x.std()).cpu().numpy()}
    s["x"] = x.round().clamp(0, 65535).to(torch.int32).to(torch.int16) if case["dtype"] == "u16" else x
    if kind == "blocks":
        blocks, n, elems = srrf.blocks_dosplit(s["cfg"], x.shape, 29, 1)
        s.update(blocks=blocks, n=n, elems=elems, map=torch.zeros(elems, device=DEV))
    else:
        s["map"] = torch.empty(_map_shape(case), device=DEV)
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "spot":
        return list(s["ctx"].optimise_spot_3b(s["model"], s["bg"], s["pix"], s["px"], s["spot"], s["limit"], 5))
    if kind == "gibbs":
        c = s["case"]
        return list(s["ctx"].gibbs_sample_3b(s["model"], s["pix"], s["px"], s["spots"], s["masks"],
                                             n_draws=c["draws"], seed=s["seed"]))
    if kind == "legacy":
        return srrf.SRRFGradientCalcGPU(s["x"], s["conf"])
    if kind == "blocks":
        return s["ctx"].forward_blocks(s["cfg"], s["x"], s["blocks"], s["n"], s["elems"], out=s["map"])
    if kind == "drift":
        m = s["ctx"].forward_shifted(s["cfg"], s["x"], s["shifts"], out=s["map"])
        gx, gs = s["ctx"].backward(s["cfg"], s["x"], s["shifts"], drift.grad_map(m), din=s["din"], dshift=s["dshift"])
        return [m, gx, gs]
    return s["ctx"].forward(s["cfg"], s["x"], out=s["map"])


# ---- what a pass cannot do without -----------------------------------------------

def _map_shape(case):
    return case["D"] * case["mz"], case["H"] * case["my"], case["W"] * case["mx"]


def work(case):
    kind = case["kind"]
    if kind in ("spot", "gibbs"):
        P = case["D"] * case["H"] * case["W"]
        if kind == "spot":
            # samples and data read once; about 100 evaluations over the spot's support (some 3,500 voxels) of
            # 8 operations a voxel, frame and sample
            n = case["S"] * case["F"]
            return {"bytes": 8.0 * P * (n + case["F"]), "flops": 100.0 * n * min(P, 3500) * 16}
        # data in, the draws' intensities and states out; the emission sums over each spot's mask (some 1,800 voxels)
        nu = case["K"] * case["draws"] * case["F"]
        return {"bytes": 8.0 * P * case["F"] * (1 + case["draws"]) + nu, "flops": nu * min(P, 1800) * 6.0}
    voxels = case["T"] * case["D"] * case["H"] * case["W"]
    if kind == "blocks":
        # overlapping borders are computed in both blocks
        blocks, n, elems = srrf.blocks_dosplit(_config(case), (case["T"], case["D"], case["H"], case["W"]), 29, 1)
        out = elems
    else:
        out = case["D"] * case["H"] * case["W"] * case["mx"] * case["my"] * case["mz"]
    size = 2 if case["dtype"] == "u16" else 4
    flops = srrf.flops_per_voxel_volume(_config(case)) * out * case["T"]
    if kind == "drift":
        # forward; then the forward's interpolation again, the derivative and the transposed passes
        return {"bytes": 4.0 * (2 * voxels + 3 * out), "flops": 3.5 * flops}
    return {"bytes": float(size * voxels + 4 * out), "flops": flops}


# ---- the same in 64 bits ---------------------------------------------------------

def _ring(radius, axes):
    """The ring's distinct points with their multiplicities, from the reference's float construction."""
    n = 2 * axes
    step = np.float32(np.float32(3.141592654) * np.float32(2)) / np.float32(n)
    a = (step * np.arange(n, dtype=np.float32)).astype(np.float32)
    sin, cos, r = np.sin(a), np.cos(a), np.float32(radius)
    x, y = (r * sin)[:, None] * cos[None], (r * sin)[:, None] * sin[None]
    z = np.repeat((r * cos)[:, None], n, 1)
    p = np.stack([x, y, z], -1).reshape(-1, 3).astype(np.float64)
    p[np.abs(p) <= 1e-6 * radius] = 0
    reps, mult = [], []
    for q in p:
        for i, u in enumerate(reps):
            if np.abs(u - q).max() <= 1e-6 * radius:
                mult[i] += 1
                break
        else:
            reps.append(q)
            mult.append(1)
    return np.array(reps), np.array(mult), n


def _cubic(v):
    a = np.abs(v)
    return np.where(a < 1, a * a * (1.5 * a - 2.5) + 1, np.where(a < 2, -0.5 * a ** 3 + 2.5 * a * a - 4 * a + 2, 0))


def _taps(length, mag, rho):
    """Four clamped tap indices and weights for every fine position at offset rho, and which pass the window."""
    q = (np.arange(length * mag) + 0.5 + rho) / mag
    u0 = np.floor(q - 0.5).astype(np.int64)
    at = u0[:, None] + np.arange(-1, 3)
    w = _cubic(q[:, None] - (at + 0.5))
    qf = (np.arange(length * mag, dtype=np.float32) + np.float32(0.5) + np.float32(rho)) / np.float32(mag)
    ok = ~((qf < 1.5) | (qf > np.float32(length) - np.float32(1.5)))
    return (torch.from_numpy(at.clip(0, length - 1)).to(DEV), torch.from_numpy(w).to(DEV), torch.from_numpy(ok).to(DEV))


def _along(v, taps, dim):
    """v resampled along `dim` by four taps."""
    at, w, _ = taps
    shape = [1] * v.dim()
    shape[dim] = -1
    return sum(v.index_select(dim, at[:, k]) * w[:, k].reshape(shape) for k in range(4))


def _gradient(v, smooth):
    """(Gx, Gy, Gz) of [T][D][H][W] with edge clamping: ranges 1, or the central difference."""
    p = torch.nn.functional.pad(v, (1, 1, 1, 1, 1, 1), mode="replicate")

    def box(a, dim):
        n = a.shape[dim] - 2
        parts = [a.narrow(dim, k, n) for k in range(3)]
        return parts[0] + parts[1] + parts[2] if smooth else parts[1]

    def diff(a, dim):
        n = a.shape[dim] - 2
        return a.narrow(dim, 2, n) - a.narrow(dim, 0, n)

    return diff(box(box(p, 1), 2), 3), diff(box(box(p, 1), 3), 2), diff(box(box(p, 2), 3), 1)


def _radiality(v, case):
    """Radiality and intensity [T][Z][Y][X] of float64 volumes."""
    mag, dims = (case["mx"], case["my"], case["mz"]), v.shape[:0:-1]
    points, mult, n = _ring(0.5, 6)
    taps = [{r: _taps(dims[a], mag[a], r) for r in set(points[:, a].tolist()) | {0.0}} for a in range(3)]
    grad = _gradient(v, case["smooth"])
    S = 0
    for x in sorted(taps[0]):
        here = [i for i in range(len(points)) if points[i, 0] == x]
        gx = [_along(c, taps[0][x], 3) for c in grad] if here else None
        for y in sorted(set(points[here, 1].tolist())):
            gy = [_along(c, taps[1][y], 2) for c in gx]
            for i in (i for i in here if points[i, 1] == y):
                z, u = points[i, 2], points[i] / 0.5
                G = [_along(c, taps[2][z], 1) for c in gy]
                dot = G[0] * u[0] + G[1] * u[1] + G[2] * u[2]
                cr = [G[1] * u[2] - G[2] * u[1], G[2] * u[0] - G[0] * u[2], G[0] * u[1] - G[1] * u[0]]
                sin = torch.sqrt((cr[0] ** 2 + cr[1] ** 2 + cr[2] ** 2) / (G[0] ** 2 + G[1] ** 2 + G[2] ** 2))
                D = (1 - sin) ** 2 * (float(mult[i]) / n)
                S = S + torch.where(dot > 0, -D, D)
    inside = [torch.stack([taps[a][r][2] for r in set(points[:, a].tolist())]).all(0) for a in range(3)]
    ok = inside[2][:, None, None] & inside[1][:, None] & inside[0]
    S = torch.where(ok, S, torch.full_like(S, math.nan))
    I = _along(_along(_along(v, taps[0][0.0], 3), taps[1][0.0], 2), taps[2][0.0], 1).clamp_min(0)
    ok = taps[2][0.0][2][:, None, None] & taps[1][0.0][2][:, None] & taps[0][0.0][2]
    return S, torch.where(ok, I, torch.zeros_like(I))


def _temporal(S, I, case):
    T, k, method = S.shape[0], case["order"], case["method"]
    if method == "TRA":
        return (S * I).mean(0)
    if method == "TRM":
        v = S * I
        return torch.where(torch.isnan(v), torch.zeros_like(v), v).amax(0).clamp_min(0)
    if method == "TRPPM":
        r = torch.where(torch.isnan(S), torch.zeros_like(S), S).clamp_min(0)
        return 0.5 * (r.sum(0) ** 2 + (r * r).sum(0)) / max(0.5 * T * (T + 1), 1) * I.mean(0)
    mean, weight = S.mean(0), (S * I).mean(0)
    rows, n, out = list(S.unbind(0)) + [torch.zeros_like(mean)] * 4, T, 0
    zero = torch.zeros_like(mean)
    ABC, ABCD, CD, AC, BD, AD, BC = (zero for _ in range(7))
    while True:
        AB = zero
        for t in range(n - k):
            a, b = rows[t] - mean, rows[t + 1] - mean
            AB = AB + a * b
            if k == 3:
                ABC = ABC + a * b * (rows[t + 2] - mean)
            if k == 4:
                c, d = rows[t + 2] - mean, rows[t + 3] - mean
                ABCD, CD, AC, BD, AD, BC = (ABCD + a * b * c * d, CD + c * d, AC + a * c, BD + b * d, AD + a * d,
                                            BC + b * c)
            if case["itc"]:
                # entry t becomes the mean of k entries; itself reads as 0, and so does what lies past the series
                rows[t] = sum((zero if j == t or j >= T else rows[j]) for j in range(t * k, t * k + k)) / k \
                    if t * k < n else zero
        if n > k or not case["itc"]:
            C = AB if k == 2 else ABC if k == 3 else ABCD - AB * CD - AC * BD - AD * BC
            out = out + C.abs() / n
        n //= k
        if not case["itc"] or n <= k:
            return weight * out


def _blocks_exact(x, case):
    """The packed blocks of the doSplit rule, each reduced by itself."""
    blocks, n, elems = srrf.blocks_dosplit(_config(case), x.shape, 29, 1)
    out = torch.zeros(elems, dtype=torch.float64, device=DEV)
    for i in range(n):
        b = blocks[i]
        o, s = list(b.origin), list(b.size)
        m = _temporal(*_radiality(x[:, o[2]:o[2] + s[2], o[1]:o[1] + s[1], o[0]:o[0] + s[0]], case), case)
        out[b.out_offset:b.out_offset + m.numel()] = m.reshape(-1)
    return out


def _shifted(x, shifts):
    """The volumes resampled at x + shift by clamped Catmull-Rom taps, one axis at a time; differentiable in both."""
    def kernel(u):
        a = u.abs()
        return torch.where(a < 1, a * a * (1.5 * a - 2.5) + 1, -0.5 * a ** 3 + 2.5 * a * a - 4 * a + 2)

    vols = []
    for v, d in zip(x.unbind(0), shifts.unbind(0)):
        for dim, s in ((2, d[0]), (1, d[1]), (0, d[2])):
            n = v.shape[dim]
            pos = torch.arange(n, device=DEV) + s
            base = torch.floor(pos.detach()).long()
            shape = [1, 1, 1]
            shape[dim] = n
            v = sum(v.index_select(dim, (base + k).clamp(0, n - 1)) * kernel(pos - (base + k)).reshape(shape)
                    for k in range(-1, 3))
        vols.append(v)
    return torch.stack(vols)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("spot", "gibbs"):
        return None  # a search's path and a random chain
    units = case["T"] * case["D"] * case["H"] * case["W"] * case["mx"] * case["my"] * case["mz"]
    if units > (2e7 if kind == "drift" else 6e8):
        return None
    s = prepare(case, seed)
    x = s["x"]
    if kind == "legacy":
        x = torch.from_numpy(x).to(DEV)
    elif case["dtype"] == "u16":
        x = x.to(torch.int32) & 0xffff
    x = x.double()
    if kind == "blocks":
        return _blocks_exact(x, case)
    if kind != "drift":
        stacks = [_radiality(v, case) for v in x.split(max(1, int(2.5e8 * case["T"] / units)))]
        m = _temporal(torch.cat([a for a, _ in stacks]), torch.cat([b for _, b in stacks]), case)
        return m.cpu().numpy() if kind == "legacy" else m
    x.requires_grad_(True)
    shifts = s["shifts"].double().requires_grad_(True)
    y = _shifted(x, shifts)
    v = y.detach()
    with torch.no_grad():
        stacks = [_radiality(v[t:t + 1], case) for t in range(len(v))]
    S = torch.cat([a for a, _ in stacks]).requires_grad_(True)
    I = torch.cat([b for _, b in stacks]).requires_grad_(True)
    bad = torch.isnan(S).any(0)
    m = torch.where(bad, math.nan, _temporal(S, I, case).detach())
    f = torch.nan_to_num(m, nan=0.0)
    gm = -f / f.norm()
    inner = _temporal(torch.where(bad, 0.0, S), torch.where(bad, 0.0, I), case)
    gS, gI = torch.autograd.grad((torch.where(bad, 0.0, inner) * gm).sum(), [S, I])
    gv = torch.zeros_like(v)
    for t in range(len(v)):
        vt = v[t:t + 1].clone().requires_grad_(True)
        a, b = _radiality(vt, case)
        total = (torch.where(bad, 0.0, a[0]) * gS[t]).sum() + (torch.where(bad, 0.0, b[0]) * gI[t]).sum()
        gv[t] = torch.autograd.grad(total, vt)[0][0]
    gx, gs = torch.autograd.grad(y, [x, shifts], gv)
    return [m, gx, gs]
