"""Performance cases of the light-field projector and reconstruction path.

Each case is one call of a public entry point on inputs that live where a user's program has
them (device arrays, a resident PSF, a reusable solver), over the sizes this repository is
used at: lenslet pitch 15 px, patches of 11 to 71 lenslets per side, 7 to 51 depth planes,
point-spread functions of 61 to 231 px, sensor movies of 100 to 2000 frames.

kinds:
  conv       mex_lfm_convolution_vec(bitmap, kernels): the MEX projector
  solve      RLSolver.run(lfimg, iterations): the Richardson-Lucy reconstruction of a patch
  batch      BatchSolver.run(images, iterations): patches of a carpet solved together
  forward    RLSolver.forward_project(volume): light-field image of a volume
  backward   RLSolver.backward_view(image, u, v): back projection of one sub-aperture view
  summary    summary_image(movie): rank-1 background, detrend and temporal deviation
  rectify    image_load_module_aug(patch, SI, frames): raw frames to the sensor movie
"""
import math

import torch

import mesolf_gb300.api as api

N = 15  # lenslet pitch (the reference's Nnum)
DEV = "cuda"


def listed():
    return [
        # interactive use of the projector on a crop, the size of the installation check
        {"name": "conv_crop", "kind": "conv", "W": 40, "H": 35, "n": 2, "kw": 21},
        # one depth of a segment's slices, even kernel width, sides off the lenslet grid
        {"name": "conv_depth", "kind": "conv", "W": 253, "H": 198, "n": 4, "kw": 136},
        # the reference's own test input: 77 slices of 376 x 376 with 241-px kernels
        {"name": "conv_stack", "kind": "conv", "W": 376, "H": 376, "n": 77, "kw": 241},
        # the CPU-runnable reconstruction (11 x 11 lenslets, 21 planes), launch-bound
        {"name": "solve_11x11x21", "kind": "solve", "La": 11, "Lb": 11, "Z": 21, "z0": -10, "K0": 61, "iters": 8,
         "precision": "fp32"},
        # the headline reconstruction: 1005 x 1005 px, 51 planes, 231-px PSF, 3 iterations
        {"name": "solve_67x67x51", "kind": "solve", "La": 67, "Lb": 67, "Z": 51, "z0": 0, "K0": 231, "iters": 3,
         "precision": "fp32"},
        # one carpet patch in the mixed precision that serving uses
        {"name": "solve_mixed_45x70x51", "kind": "solve", "La": 45, "Lb": 70, "Z": 51, "z0": 0, "K0": 231, "iters": 3,
         "precision": "bf16x2"},
        # uneven patches with plane ranges of one PSF solved together
        {"name": "batch_mixed_6", "kind": "batch", "patches": 6, "Lmin": 31, "Lmax": 60, "Zmin": 13, "Z": 26, "z0": -13,
         "K0": 171, "iters": 3, "precision": "bf16x2"},
        # light-field image of a segment volume (seed library, peeling)
        {"name": "forward_31x40x26", "kind": "forward", "La": 31, "Lb": 40, "Z": 26, "z0": -13, "K0": 141},
        # back projection of one sub-aperture image
        {"name": "backward_52x37x31", "kind": "backward", "La": 52, "Lb": 37, "Z": 31, "z0": -15, "K0": 201, "u": 3, "v": 9},
        # summary image of a small patch over a short recording
        {"name": "summary_465x450x500", "kind": "summary", "rows": 465, "cols": 450, "T": 500, "mode": "pixelwise"},
        # summary image of a full patch over a 2000-frame recording, the defaults
        {"name": "summary_1005x1005x2000", "kind": "summary", "rows": 1005, "cols": 1005, "T": 2000, "mode": "pixelwise"},
        # raw 16-bit camera frames of a patch to the sensor movie, the defaults
        {"name": "rectify_1100x1100x2000", "kind": "rectify", "rows": 1100, "cols": 1100, "T": 2000, "dtype": "u16",
         "step": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _psf_size(Z, z0, extra):
    """Odd PSF side that holds the widest plane inside the phase-space crop."""
    far = max(abs(z0), abs(z0 + Z - 1))
    return min(231, max(61, 2 * (int(math.ceil(2 + 1.65 * far)) + 22) + 1 + 2 * extra))


def draw(rng):
    kind = rng.choice(["conv", "solve", "solve", "solve", "batch", "forward", "backward", "summary", "rectify"])
    if kind == "conv":
        return {"kind": kind, "W": _log(rng, 31, 400), "H": _log(rng, 31, 400), "n": _log(rng, 1, 60),
                "kw": _log(rng, 15, 241)}
    if kind in ("solve", "forward", "backward"):
        Z = rng.randint(7, 33)
        z0 = -(Z // 2)
        c = {"kind": kind, "La": _log(rng, 11, 60), "Lb": _log(rng, 11, 60), "Z": Z, "z0": z0,
             "K0": _psf_size(Z, z0, rng.randint(0, 40))}
        if kind == "solve":
            c["iters"] = rng.randint(1, 3)
            c["precision"] = rng.choice(["fp32", "fp32", "bf16x2", "bf16x3"])
        if kind == "backward":
            c["u"], c["v"] = rng.randint(3, 11), rng.randint(3, 11)
        return c
    if kind == "batch":
        Z = rng.randint(11, 26)
        Lmin = rng.randint(18, 31)
        return {"kind": kind, "patches": rng.randint(2, 7), "Lmin": Lmin, "Lmax": rng.randint(Lmin + 2, 60),
                "Zmin": max(7, Z // 2), "Z": Z, "z0": -(Z // 2), "K0": _psf_size(Z, -(Z // 2), rng.randint(0, 20)),
                "iters": rng.randint(1, 3), "precision": "bf16x2"}
    if kind == "summary":
        return {"kind": kind, "rows": N * _log(rng, 11, 67), "cols": N * _log(rng, 11, 67), "T": _log(rng, 130, 1600),
                "mode": rng.choice(["pixelwise", "pixelwise", "global"])}
    return {"kind": kind, "rows": _log(rng, 200, 1100), "cols": _log(rng, 200, 1100), "T": _log(rng, 24, 1200),
            "dtype": rng.choice(["u16", "u16", "f32"]), "step": rng.choice([1, 1, 2, 3])}


# ----------------------------------------------------------------------------- inputs
def _gen(seed, device=DEV):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def _col(t):
    """(..., c, b, a) contiguous memory seen in MATLAB index order (a, b, c, ...)."""
    return t.permute(*reversed(range(t.dim())))


def _psf(K0, Z, z0, seed):
    """(Z, N, N, K0, K0) contiguous PSF: a defocused disc (Gaussian profile, hard edge) per
    plane and source position, shifted with depth, with a per-slice amplitude jitter."""
    jit = 0.9 + 0.2 * torch.rand((Z, N, N), generator=_gen(seed), device=DEV)
    H = torch.empty((Z, N, N, K0, K0), device=DEV)
    x = torch.arange(K0, device=DEV, dtype=torch.float64)
    off = torch.arange(N, device=DEV, dtype=torch.float64) - (N - 1) / 2
    for k in range(Z):
        z = z0 + k
        radius = 2.0 + 0.6 * abs(z)
        d2 = (x[None, :] - ((K0 - 1) / 2 + off * z * 0.15)[:, None]) ** 2       # (N, K0)
        d = d2[:, None, :, None] + d2[None, :, None, :]                         # (b, a, y, x)
        g = torch.exp(-d / (2 * (radius / 2) ** 2)) * (d <= radius * radius)
        g = g / g.sum(dim=(2, 3), keepdim=True)
        H[k] = (g * jit[k][:, :, None, None]).float()
    return H


def _image(H, La, Lb, planes, seed):
    """Photon-counting light-field image (Lb*N, La*N) of random point sources in `planes`."""
    K0, m = H.shape[-1], H.shape[-1] // 2
    Xr, Xc = La * N, Lb * N
    n_obj = max(20, min(240, Xr * Xc // 3000))
    g = _gen(seed + 1, "cpu")
    r = torch.randint(0, Xr, (n_obj,), generator=g).tolist()
    c = torch.randint(0, Xc, (n_obj,), generator=g).tolist()
    z = torch.randint(planes[0], planes[0] + planes[1], (n_obj,), generator=g).tolist()
    amp = torch.exp(0.5 * torch.randn(n_obj, generator=g)).tolist()
    img = torch.zeros((Xc + 2 * m, Xr + 2 * m), device=DEV)
    for i in range(n_obj):
        img[c[i]:c[i] + K0, r[i]:r[i] + K0].add_(H[z[i], c[i] % N, r[i] % N], alpha=amp[i])
    img = img[m:m + Xc, m:m + Xr]
    img = img / img.max() + 0.01
    return torch.poisson(2000.0 * img, generator=_gen(seed + 2)).contiguous()


def _rot(H):
    return H.flip(-1, -2).contiguous()


def _volume(La, Lb, Z, seed):
    v = torch.rand((Z, Lb * N, La * N), generator=_gen(seed + 3), device=DEV)
    return 0.02 + v ** 8  # sparse bright voxels on a constant background


def _batch_geometry(case, seed):
    g = _gen(1000 * case["Lmin"] + case["Lmax"], "cpu")  # the carpet's layout does not depend on the data
    P = case["patches"]
    L = torch.randint(case["Lmin"], case["Lmax"] + 1, (P, 2), generator=g).tolist()
    nz = torch.randint(case["Zmin"], case["Z"] + 1, (P,), generator=g).tolist()
    z0 = [int(torch.randint(0, case["Z"] - k + 1, (1,), generator=g)) for k in nz]
    return L, list(zip(z0, nz))


def _movie(P, T, seed):
    """(T, P) fluorescence movie: baseline with bleaching, decaying transients, noise."""
    g = _gen(seed)
    base = 100 + 500 * torch.rand(P, generator=g, device=DEV)
    Y = torch.randn((T, P), generator=g, device=DEV)
    c = torch.zeros(P, device=DEV)
    for j in range(T):
        k = torch.rand(P, generator=g, device=DEV)
        c.mul_(0.8825).add_(torch.clamp(k - 0.996, min=0.0), alpha=300 / 0.004)
        Y[j].mul_(8.0).add_(base, alpha=1 - 0.2 * j / T).add_(c)
    return Y


def _frames(rows, cols, T, dtype, seed):
    """(T, cols, rows) raw camera frames: a lenslet pattern with shot noise."""
    g = _gen(seed)
    base = 200 + 3000 * torch.rand((cols, rows), generator=g, device=DEV)
    out = torch.empty((T, cols, rows), device=DEV, dtype=torch.int16 if dtype == "u16" else torch.float32)
    for j in range(0, T, 50):
        k = min(50, T - j)
        f = base + base.sqrt() * torch.randn((k, cols, rows), generator=g, device=DEV)
        out[j:j + k] = f.clamp_(0, 32000)
    return out.view(torch.uint16) if dtype == "u16" else out


def _axis(center, size, dx):
    """Kept query coordinates (1-based, FP64) of one axis of the rectified patch."""
    s = dx / N
    left = [center - s * k for k in range(int(math.floor((center + s) / s + 1e-9)) + 1)][::-1]
    right = [center + s * k for k in range(1, int(math.floor((size + 0.9 - center) / s + 1e-9)) + 1)]
    q = left + right
    q = q[(len(left) - N // 2) % N:]
    return q[:N * (len(q) // N)]


RECT_DX = 15.27


def _rect_geometry(case):
    """Raw cut (1-based, inclusive), lenslet centre inside it and the query axes."""
    y0, y1, x0, x1 = 4, case["rows"] - 3, 6, case["cols"] - 2
    h, w = y1 - y0 + 1, x1 - x0 + 1
    yc, xc = h / 2 + 0.3, w / 2 - 0.4
    return (y0, y1, x0, x1), (yc, xc), (_axis(yc, h, RECT_DX), _axis(xc, w, RECT_DX))


def prepare(case, seed):
    k = case["kind"]
    if k == "conv":
        g = _gen(seed)
        W, H, n, kw = case["W"], case["H"], case["n"], case["kw"]
        bm = torch.rand((n, H, W), generator=g, device=DEV)
        bm = torch.where(bm > 0.9, bm * 10, torch.zeros((), device=DEV))        # sparse segment slices
        ker = torch.rand((N, N, kw, kw), generator=g, device=DEV) / (kw * kw)
        return {"kind": k, "bitmap": _col(bm), "kernels": _col(ker)}
    if k in ("solve", "forward", "backward"):
        H = _psf(case["K0"], case["Z"], case["z0"], seed)
        psf = api.PhaseSpacePSF(_col(H), _col(_rot(H)))
        s = {"kind": k, "psf": psf, "solver": api.RLSolver(psf, (case["La"] * N, case["Lb"] * N))}
        if k == "solve":
            s["lf"] = _col(_image(H, case["La"], case["Lb"], (0, case["Z"]), seed))
            s["iters"], s["precision"] = case["iters"], case["precision"]
        elif k == "forward":
            s["vol"] = _col(_volume(case["La"], case["Lb"], case["Z"], seed))
        else:
            s["proj"] = _col(0.5 + torch.rand((case["Lb"], case["La"]), generator=_gen(seed + 3), device=DEV))
            s["u"], s["v"] = case["u"], case["v"]
        return s
    if k == "batch":
        H = _psf(case["K0"], case["Z"], case["z0"], seed)
        psf = api.PhaseSpacePSF(_col(H), _col(_rot(H)))
        L, planes = _batch_geometry(case, seed)
        imgs = [_col(_image(H, a, b, p, seed + 10 * i)) for i, ((a, b), p) in enumerate(zip(L, planes))]
        return {"kind": k, "psf": psf, "solver": api.BatchSolver(psf, [(a * N, b * N) for a, b in L], planes),
                "lf": imgs, "iters": case["iters"], "precision": case["precision"]}
    if k == "summary":
        return {"kind": k, "movie": _movie(case["rows"] * case["cols"], case["T"], seed).T, "mode": case["mode"]}
    cut, centre, axes = _rect_geometry(case)
    info = {"size": (len(axes[0]), len(axes[1])), "raw_cut": [[cut[0], cut[1]], [cut[2], cut[3]]],
            "raw_cut_yCenter": centre[0], "raw_cut_xCenter": centre[1]}
    return {"kind": k, "info": info, "SI": {"Nnum": N, "frames_dx": RECT_DX, "frames_step": case["step"]},
            "frames": _col(_frames(case["rows"], case["cols"], case["T"], case["dtype"], seed))}


def run(state):
    k = state["kind"]
    if k == "conv":
        return api.mex_lfm_convolution_vec(state["bitmap"], state["kernels"])
    if k in ("solve", "batch"):
        return state["solver"].run(state["lf"], state["iters"], precision=state["precision"], want_stats=False)
    if k == "forward":
        return state["solver"].forward_project(state["vol"])
    if k == "backward":
        return state["solver"].backward_view(state["proj"], state["u"], state["v"])
    if k == "summary":
        return api.summary_image(state["movie"], detrend_mode=state["mode"])
    return api.image_load_module_aug(state["info"], state["SI"], state["frames"])


# ----------------------------------------------------------------------------- work
def _crop(K0):
    """Side and first pixel of the phase-space crop of a K0-px PSF."""
    S = K0 - (K0 - N) % (2 * N)
    return S, int(math.floor(K0 / 2 + 0.5)) - S // 2 - 1


def _step_flops(La, Lb, Z, K0):
    """Multiply-adds of one direction of one view: every lenslet meets S*S/N/N taps per channel."""
    return 2.0 * La * Lb * Z * _crop(K0)[0] ** 2


#: Share of the N*N views whose weight passes the reference's 0.2 cut (142 of 225 at the headline size).
VIEWS = 142


def work(case):
    k = case["kind"]
    if k == "conv":
        px, kk = case["W"] * case["H"] * case["n"], case["kw"] ** 2
        return {"bytes": 8.0 * px + 4.0 * kk * N * N, "flops": 2.0 * px * kk}
    if k in ("solve", "forward", "backward"):
        La, Lb, Z, K0 = case["La"], case["Lb"], case["Z"], case["K0"]
        px, taps = La * Lb * N * N, 4.0 * _crop(K0)[0] ** 2 * Z
        one = _step_flops(La, Lb, Z, K0)
        if k == "solve":
            return {"bytes": 4.0 * px * (1 + Z) + 2 * VIEWS * taps, "flops": 2.0 * VIEWS * case["iters"] * one}
        if k == "forward":
            return {"bytes": 4.0 * px * (1 + Z) + N * N * taps, "flops": N * N * one}
        return {"bytes": 4.0 * px * Z + 4.0 * La * Lb + taps, "flops": one}
    if k == "batch":
        L, planes = _batch_geometry(case, 0)
        b, f = 2 * VIEWS * 4.0 * _crop(case["K0"])[0] ** 2 * case["Z"], 0.0
        for (La, Lb), (_, nz) in zip(L, planes):
            b += 4.0 * La * Lb * N * N * (1 + nz)
            f += 2.0 * VIEWS * case["iters"] * _step_flops(La, Lb, nz, case["K0"])
        return {"bytes": b, "flops": f}
    if k == "summary":
        P, T = case["rows"] * case["cols"], case["T"]
        return {"bytes": 4.0 * P * T + 8.0 * P + 4.0 * T, "flops": 40.0 * P * T}
    cut, _, axes = _rect_geometry(case)
    n_out = (case["T"] - 1) // case["step"] + 1
    raw, out = (cut[1] - cut[0] + 1) * (cut[3] - cut[2] + 1) * case["T"], len(axes[0]) * len(axes[1]) * n_out
    return {"bytes": (2.0 if case["dtype"] == "u16" else 4.0) * raw + 4.0 * out, "flops": 6.0 * out + raw}


# ----------------------------------------------------------------------------- 64-bit results
#: Bytes of gathered FP64 windows above which a reconstruction is not repeated in 64 bits.
EXACT_BYTES = 5e12


def _exact_conv(case, seed):
    s = prepare(case, seed)
    bm, ker = _col(s["bitmap"]).double(), _col(s["kernels"])       # (n, H, W), (b, a, ky, kx)
    n, Hh, W = bm.shape
    kw = ker.shape[-1]
    hk = kw // 2
    if kw % 2 == 0:  # the reference never reads the last row and column for even widths
        bm[:, -1, :] = 0
        bm[:, :, -1] = 0
    E = (Hh + kw, W + kw)
    F = torch.fft.rfft2(bm, s=E)
    out = torch.zeros_like(bm)
    for b in range(min(N, Hh)):
        for a in range(min(N, W)):
            full = torch.fft.irfft2(F * torch.fft.rfft2(ker[b, a].double(), s=E).conj(), s=E)
            full = torch.roll(full, (hk, hk), (1, 2))
            out[:, b::N, a::N] = full[:, :Hh, :W][:, b::N, a::N]
    return _col(out)


def _view_psf(H, sums, u, v):
    """(Z, S, S) phase-space PSF (rows p, columns q) of view (u, v); H is (Z, b, a, y, x)."""
    S, i1 = _crop(H.shape[-1])
    p = torch.arange(S, device=H.device)
    ru, rv = p + u - (N - 1) // 2, p + v - (N - 1) // 2
    ok = ((ru >= 0) & (ru < S))[:, None] & ((rv >= 0) & (rv < S))[None, :]
    x, y = ru.clamp(0, S - 1) + i1, rv.clamp(0, S - 1) + i1
    ab = N - 1 - p % N
    h = H[:, ab[None, :], ab[:, None], y[None, :], x[:, None]].double()
    return h * ok / sums[:, None, None]


def _windows(X, S):
    """(Z, La*Lb, S*S) windows of the (Z, Xr, Xc) volume around every lenslet centre."""
    m, c0 = S // 2, (N + 1) // 2 - 1
    Xp = torch.nn.functional.pad(X, (m - c0, m, m - c0, m)) if m >= c0 else None
    w = Xp.unfold(1, S, N).unfold(2, S, N)[:, :X.shape[1] // N, :X.shape[2] // N]
    return w.reshape(X.shape[0], -1, S * S)


def _back(t, R, u, v):
    """(Z, Xr, Xc) back projection of R (La, Lb) with the (Z, S, S) kernel t."""
    Z, S, _ = t.shape
    La, Lb = R.shape
    size = ((La - 1) * N + S, (Lb - 1) * N + S)
    cols = t.reshape(Z, S * S, 1) * R.reshape(1, 1, -1)
    full = torch.nn.functional.fold(cols, size, S, stride=N)[:, 0]
    m = S // 2
    out = torch.zeros((Z, La * N, Lb * N), dtype=torch.float64, device=R.device)
    r0, c0 = m - u, m - v  # row of `full` that is row 0 of the image
    full = torch.nn.functional.pad(full, (0, N + m, 0, N + m))
    lo_r, lo_c = max(0, -r0), max(0, -c0)
    out[:, lo_r:, lo_c:] = full[:, r0 + lo_r:r0 + La * N, c0 + lo_c:c0 + Lb * N]
    return out


def _spiral():
    """Views (u, v) from the rim inwards, in the reference's order."""
    order = []
    for k in range((N + 1) // 2):
        lo, hi = k, N - 1 - k
        if lo == hi:
            order.append((lo, lo))
            continue
        order += [(i, lo) for i in range(lo, hi + 1)]
        order += [(hi, j) for j in range(lo + 1, hi + 1)]
        order += [(i, hi) for i in range(hi - 1, lo - 1, -1)]
        order += [(lo, j) for j in range(hi - 1, lo, -1)]
    return order


def _filter(X):
    """Flux-preserving low-pass of the planes around the middle, (Z, Xr, Xc) in place."""
    Z, Xr, Xc = X.shape
    R = int(math.ceil(Z / 3))
    R += R % 2
    nb, half = 3 * R, int(math.floor(Z / 2 + 0.5))
    x = torch.arange(1, Xr + 1, device=X.device, dtype=torch.float64) - Xr / 2
    y = torch.arange(1, Xc + 1, device=X.device, dtype=torch.float64) - Xc / 2
    for z1 in range(1, Z + 1):
        if not half - nb / 2 + 1 <= z1 <= half + nb / 2:
            continue
        axis = (z1 - half + nb / 2) - nb / 2
        w = max(0.2, (N - 7) * math.exp(-(axis / 100 * 2 * math.sqrt(math.log(2))) ** 2))
        gx, gy = torch.fft.fft(torch.exp(-(x / w) ** 2)).abs(), torch.fft.fft(torch.exp(-(y / w) ** 2)).abs()
        flt = (gx / gx.max())[:, None] * (gy / gy.max())[None, :]
        img = X[z1 - 1]
        buf = torch.fft.ifft2(torch.fft.fft2(img) * flt).real
        total = buf.sum()
        X[z1 - 1] = img.sum() * buf / total if float(total) != 0 else 0.0


def _solve64(H, lf, iters):
    """The reconstruction of lf (Xr, Xc) with PSF planes H (Z, b, a, y, x), (Z, Xr, Xc) FP64."""
    Z, S = H.shape[0], _crop(H.shape[-1])[0]
    i1 = _crop(H.shape[-1])[1]
    sums = H.double().sum(dim=(1, 2, 3, 4))
    Ht = _rot(H)
    hps = {(u, v): _view_psf(H, sums, u, v) for u in range(N) for v in range(N)}
    w = torch.stack([torch.stack([hps[u, v].sum() for v in range(N)]) for u in range(N)])
    w = w / w.sum()
    w = w - w.min()
    w = w / w.max()
    w = torch.where(w < 0.2, torch.zeros_like(w), w) * 0.3
    lf = lf.double()
    X = torch.ones((Z,) + tuple(lf.shape), dtype=torch.float64, device=lf.device)
    X = X / X.sum() * lf.sum()
    La, Lb = lf.shape[0] // N, lf.shape[1] // N
    ones = torch.ones((La, Lb), dtype=torch.float64, device=lf.device)
    for _ in range(iters):
        for u, v in _spiral():
            wv = float(w[u, v])
            if wv == 0:
                continue
            h = hps[u, v].flip(1, 2).reshape(Z, S * S, 1)
            HX = torch.bmm(_windows(X, S), h).sum(0).reshape(La, Lb)
            R = lf[u::N, v::N] / HX
            R = torch.where(torch.isfinite(R), R, torch.zeros_like(R))
            t = (Ht[:, v, u, i1:i1 + S, i1:i1 + S].double() / sums[:, None, None]).transpose(1, 2)
            C, D = _back(t, R, u, v), _back(t, ones, u, v)
            Xc = X * C / D
            Xc = torch.where(torch.isfinite(Xc) & (Xc > 0), Xc, torch.zeros_like(Xc))
            X = (Xc * wv + (1 - wv) * X).clamp_(min=0)
        _filter(X)
    return X


def _solve_bytes(La, Lb, Z, K0, iters):
    return 8.0 * La * Lb * Z * _crop(K0)[0] ** 2 * VIEWS * iters


def _exact_solve(case, seed):
    if case["kind"] == "solve":
        if _solve_bytes(case["La"], case["Lb"], case["Z"], case["K0"], case["iters"]) > EXACT_BYTES:
            return None
        H = _psf(case["K0"], case["Z"], case["z0"], seed)
        lf = _image(H, case["La"], case["Lb"], (0, case["Z"]), seed).T
        return _solve64(H, lf, case["iters"]).permute(1, 2, 0)
    L, planes = _batch_geometry(case, seed)
    if sum(_solve_bytes(a, b, nz, case["K0"], case["iters"]) for (a, b), (_, nz) in zip(L, planes)) > EXACT_BYTES:
        return None
    H = _psf(case["K0"], case["Z"], case["z0"], seed)
    imgs = [_image(H, a, b, p, seed + 10 * i).T for i, ((a, b), p) in enumerate(zip(L, planes))]
    return [_solve64(H[z0:z0 + nz], im, case["iters"]).permute(1, 2, 0) for im, (z0, nz) in zip(imgs, planes)]


def _exact_forward(case, seed):
    La, Lb, Z, K0 = case["La"], case["Lb"], case["Z"], case["K0"]
    S = _crop(K0)[0]
    if 8.0 * La * Lb * S * S * Z > 2e11:
        return None
    H, vol = _psf(K0, Z, case["z0"], seed), _volume(La, Lb, Z, seed).transpose(1, 2).double()
    one = torch.ones(1, dtype=torch.float64, device=DEV)
    out = torch.zeros((N * N, La * Lb), dtype=torch.float64, device=DEV)
    for z in range(Z):
        win = _windows(vol[z:z + 1], S)[0]
        taps = torch.stack([_view_psf(H[z:z + 1], one, u, v)[0].flip(0, 1).reshape(-1) for u in range(N) for v in range(N)])
        out += taps @ win.T
    return out.reshape(N, N, La, Lb).permute(2, 0, 3, 1).reshape(La * N, Lb * N)


def _exact_backward(case, seed):
    La, Lb, Z, K0 = case["La"], case["Lb"], case["Z"], case["K0"]
    S, i1 = _crop(K0)
    H = _psf(K0, Z, case["z0"], seed)
    R = (0.5 + torch.rand((Lb, La), generator=_gen(seed + 3), device=DEV)).double().T
    out = torch.empty((La * N, Lb * N, Z), dtype=torch.float64, device=DEV)
    Ht = _rot(H)
    for z in range(Z):
        t = Ht[z, case["v"], case["u"], i1:i1 + S, i1:i1 + S].double().T / Ht[z].double().sum()
        out[:, :, z] = _back(t[None], R, case["u"], case["v"])[0]
    return out


def _moving_mean(y, w):
    """MATLAB movmean along dim 0: floor(w/2) samples before, the rest after, shrinking ends."""
    T, b = y.shape[0], w // 2
    cs = torch.cat([torch.zeros_like(y[:1]), torch.cumsum(y, 0)])
    i = torch.arange(T, device=y.device)
    lo, hi = (i - b).clamp(min=0), (i + w - b).clamp(max=T)
    return (cs[hi] - cs[lo]) / (hi - lo).double()[:, None]


def _exact_summary(case, seed):
    P, T = case["rows"] * case["cols"], case["T"]
    Y = _movie(P, T, seed).double()                       # (T, P)
    M = Y.max()
    t = Y.sum(1)
    for it in range(5):
        t = t / t.norm()
        s = (t @ Y) / M
        if it < 4:
            t = Y @ s
    img = torch.empty(P, dtype=torch.float64, device=DEV)
    if case["mode"] == "global":
        B, C = Y.mean(0) / M, t.mean()
        v = ((Y / M) ** 2).sum(0)
        img = ((v - s ** 2) / T - B ** 2 + 2 * B * s * C - s ** 2 * C ** 2).clamp(min=0).sqrt()
    else:
        for p in range(0, P, 65536):
            y = Y[:, p:p + 65536] / M
            x = _moving_mean(y - _moving_mean(y, 100), 20) ** 3
            img[p:p + 65536] = ((x ** 2).mean(0) - x.mean(0) ** 2).clamp(min=0).sqrt()
    return img / img.max(), s, t


def _exact_rectify(case, seed):
    (y0, y1, x0, x1), _, (qy, qx) = _rect_geometry(case)
    fr = _frames(case["rows"], case["cols"], case["T"], case["dtype"], seed)
    fr = fr.view(torch.int16) if case["dtype"] == "u16" else fr

    def cells(q, n):
        q = torch.tensor(q, dtype=torch.float64, device=DEV)
        c = q.floor().clamp(1, n - 1)
        return c.long() - 1, q - c

    iy, wy = cells(qy, y1 - y0 + 1)
    ix, wx = cells(qx, x1 - x0 + 1)
    n_out = (case["T"] - 1) // case["step"] + 1
    out = torch.empty((n_out, len(qx), len(qy)), dtype=torch.float64, device=DEV)
    for i in range(n_out):
        f = fr[i * case["step"]:(i + 1) * case["step"], x0 - 1:x1, y0 - 1:y1].double().mean(0)
        c = f[ix] * (1 - wx)[:, None] + f[ix + 1] * wx[:, None]
        out[i] = c[:, iy] * (1 - wy) + c[:, iy + 1] * wy
    out = out.reshape(n_out, -1)
    return out.div_(out.max()).T


def exact(case, seed):
    return {"conv": _exact_conv, "solve": _exact_solve, "batch": _exact_solve, "forward": _exact_forward,
            "backward": _exact_backward, "summary": _exact_summary, "rectify": _exact_rectify}[case["kind"]](case, seed)
