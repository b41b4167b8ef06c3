"""Workloads of the B200 match_template framework, timed through its public Python entry points.

A case is one pass of something a user of the framework runs again and again:

  search    one (pixel size, defocus) plane of ``TemplateMatchingCore``: reset, every orientation of
            the range, the result maps back on the host
  windows   the fine search of the learned proposal: angular bins over an image set of small windows
            (``SearchCore.run_plane_images``)
  refine    one ``RefineCore.score`` batch of refine_template (one candidate per peak)
  whiten    ``core.whiten_micrograph`` of one micrograph, host buffers in and out
  network   one gradient evaluation of the proposal network (forward, loss and backward)

Inputs are synthetic and made on the GPU from the seed: Gaussian-atom templates, white-noise
micrographs holding CTF-modulated projections at orientations of the searched list, so that the
maps have noise and clear peaks as real ones do.  Sums and the histogram are returned as FP32, the
type of the statistics written to the output files; best angles are returned where a peak stands
out of the noise (elsewhere the argmax of noise is decided by the last bit).
"""
import math

import numpy as np
import torch

from cistem_downstream_bah_b200 import core, hostprep, prep, proposal

DEV = "cuda"
PEAK = 8.0          # correlation (in units of its standard deviation) above which a pixel is a peak
N_FULL = 4096 * 4096  # the micrograph whose windows the window search takes

# (template box, padded width, padded height) of the camera formats and window sizes with kernels of their own
COMPILED = [(32, 256, 256), (32, 512, 512), (64, 512, 512), (64, 1024, 1024), (128, 1024, 1024), (128, 2048, 2048),
            (256, 2048, 2048), (256, 2048, 1944), (256, 2048, 2592), (128, 2048, 2916), (256, 4096, 4096),
            (128, 4096, 4096), (384, 4096, 4096), (128, 4096, 3888), (256, 4096, 5184), (256, 4096, 5832)]


# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest search: a quick look with a small template, where launches and latency count
        dict(name="search_256_t32", kind="search", T=32, X=256, Y=256, step=30.0, psi=30.0, positions=40, batch=0),
        # the CPU-runnable configuration as a whole: 1024^2, 64^3, 15 / 15 degrees, every orientation
        dict(name="search_1024_t64", kind="search", T=64, X=1024, Y=1024, step=15.0, psi=15.0, positions=188, batch=0),
        # a share of the full-size configuration: 4096^2, 256^3, 2.5 / 1.5 degrees, at the batch its autotuner picks
        dict(name="search_4096_t256", kind="search", T=256, X=4096, Y=4096, step=2.5, psi=1.5, positions=25, batch=128),
        # the uneven micrographs of the batched configuration: 3838 x 3710
        dict(name="search_4096x3888_t256", kind="search", T=256, X=4096, Y=3888, step=3.0, psi=2.0, positions=20,
             batch=128),
        # the stress configuration's geometry: 5760 x 4092 with a 384^3 template
        dict(name="search_4096x5832_t384", kind="search", T=384, X=4096, Y=5832, step=2.5, psi=1.5, positions=9,
             batch=128),
        # a binned camera format: 2880 x 2046
        dict(name="search_2048x2916_t256", kind="search", T=256, X=2048, Y=2916, step=3.0, psi=2.0, positions=24,
             batch=128),
        # a size without compiled kernels: 2700^2
        dict(name="search_2700_t256", kind="search", T=256, X=2700, Y=2700, step=3.0, psi=2.0, positions=5, batch=64),
        # the learned proposal's fine search: 2T windows, a few of them sharing each angular bin
        dict(name="windows_512_t256", kind="windows", T=256, W=512, images=5, bins=6, per_bin=723, batch=256),
        # refine_template with many peaks: one candidate per peak, a quarter with a pixel-size change
        dict(name="refine_256_t256", kind="refine", T=256, TP=256, n=256, resampled=0.25),
        # refine_template with a handful of peaks left
        dict(name="refine_5_t128", kind="refine", T=128, TP=128, n=5, resampled=0.25),
        # preparation of one micrograph
        dict(name="whiten_4096", kind="whiten", X=4096, Y=4096),
        # one training evaluation of the proposal network: 128 tiles, as its training draws them
        dict(name="network_128", kind="network", n=128, tile=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "search", "search", "windows", "refine", "whiten", "network"])
    if kind == "search":
        if rng.random() < 0.6:
            T, X, Y = rng.choice(COMPILED)
        else:   # a micrograph of any size, padded as match_template pads it
            T = rng.choice([32, 64, 128, 256])
            X, Y = (prep.factorize_dimension(_log(rng, 300, 3000), T) for _ in range(2))
            while min(X, Y) < T or max(X, Y) > 8192:
                X, Y = (prep.factorize_dimension(_log(rng, 300, 3000), T) for _ in range(2))
        psi = rng.choice([1.5, 2.0, 5.0, 15.0])
        n_psi = int(360.0 / psi) + 1
        speed = 1.0 if (T, X, Y) in COMPILED else 5.0
        # enough orientations for the histogram to be well filled, at most the largest listed search's points
        most = max(1, int(0.5 * 4096 * 4096 * 6025 / (X * Y * n_psi * speed)))
        least = max(1, min(most, int(math.ceil(3.0e7 / (X * Y * n_psi)))))
        step = rng.choice([2.5, 3.0, 7.5])
        return dict(kind="search", T=T, X=X, Y=Y, step=step, psi=psi, batch=rng.choice([0, 32, 64, 128]),
                    positions=min(1000, _log(rng, least, most)))
    if kind == "windows":
        T = rng.choice([64, 128, 256])
        return dict(kind="windows", T=T, W=max(2 * T, 256), images=rng.randint(1, 12), bins=rng.randint(1, 8),
                    per_bin=_log(rng, 241, 2410), batch=256)
    if kind == "refine":
        T = rng.choice([64, 128, 256, 384])
        return dict(kind="refine", T=T, TP=rng.choice([T, T, 2 * T]) if T < 256 else T, n=_log(rng, 1, 300),
                    resampled=rng.choice([0.0, 0.25, 1.0]))
    if kind == "whiten":
        T, X, Y = rng.choice(COMPILED)
        if rng.random() < 0.4:
            X, Y = (prep.factorize_dimension(_log(rng, 400, 4000), 256) for _ in range(2))
        return dict(kind="whiten", X=X, Y=Y)
    return dict(kind="network", n=_log(rng, 8, 256), tile=rng.choice([32, 64, 64]))


# ---------------------------------------------------------------------------------------------
# synthetic inputs, on the GPU
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _logical(n):
    i = torch.arange(n, device=DEV)
    return torch.where(i >= (n + 1) // 2, i - n, i)


def _swap(ny, nx):
    """Phase of the quadrant swap on the half plane."""
    a = (nx // 2) * torch.arange(nx // 2 + 1, device=DEV, dtype=torch.float64)[None, :] / nx
    b = (ny // 2) * _logical(ny).double()[:, None] / ny
    return torch.exp(-2j * math.pi * (a + b))


def _template(T, g):
    """Template volume of Gaussian atoms in a ball and its quadrant-swapped spectrum (complex64)."""
    n = min(120000, 4 * T * T)
    d = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64)
    r = torch.rand(n, 1, generator=g, device=DEV, dtype=torch.float64) ** (1.0 / 3.0)
    xyz = (d / d.norm(dim=1, keepdim=True) * r * (0.36 * T) + T / 2).round().long()
    vol = torch.zeros(T, T, T, device=DEV, dtype=torch.float64)
    vol.index_put_((xyz[:, 2], xyz[:, 1], xyz[:, 0]), torch.ones(n, device=DEV, dtype=torch.float64), accumulate=True)
    k = _logical(T).double() / T
    kx = torch.arange(T // 2 + 1, device=DEV).double() / T
    spec = torch.fft.rfftn(vol) / T ** 3
    spec *= torch.exp(-2.0 * (math.pi * 1.5) ** 2 * (k[:, None, None] ** 2 + k[None, :, None] ** 2 + kx[None, None, :] ** 2))
    par = (_logical(T)[:, None, None] + _logical(T)[None, :, None] + torch.arange(T // 2 + 1, device=DEV)) & 1
    spec = torch.where(par == 1, -spec, spec)
    spec[0, 0, 0] = 0
    return spec.to(torch.complex64)


def _rotations(angles):
    """The two used columns of the Euler rotation, FP32 as match_template forms it: (n, 6)."""
    f = np.float32
    a = (np.asarray(angles, f) * f(3.14159265359)).astype(np.float64) / 180.0
    c, s = np.cos(a.astype(f)), np.sin(a.astype(f))
    cp, ct, cs, sp, st, ss = c[:, 0], c[:, 1], c[:, 2], s[:, 0], s[:, 1], s[:, 2]
    m = np.stack([cp * ct * cs - sp * ss, -cp * ct * ss - sp * cs, sp * ct * cs + cp * ss, -sp * ct * ss + cp * cs,
                  -st * cs, st * ss], 1)
    return torch.from_numpy(m.astype(f)).to(DEV)


def _project(tspec, angles, filt=None):
    """Real projections (n, T, T), unscaled, FP64: trilinear Fourier slice x filter, inverse transform."""
    T = tspec.shape[0]
    vol = torch.view_as_real(tspec.to(torch.complex128)).reshape(-1, 2)
    m = _rotations(angles)
    i = torch.arange(T // 2 + 1, device=DEV).float()[None, :]
    jl = torch.where(torch.arange(T, device=DEV) < T // 2, torch.arange(T, device=DEV), torch.arange(T, device=DEV) - T)
    j = jl.float()[:, None].expand(T, T // 2 + 1)
    # the i = 0 column holds conjugate pairs: negative j (but -T/2) from positive j
    mirror = (i == 0) & (j < 0) & (j != -(T // 2))
    j = torch.where(mirror, -j, j)
    out = []
    for a in m:
        c = [a[2 * q] * i + a[2 * q + 1] * j for q in range(3)]   # FP32 coordinates (x, y, z)
        neg = c[0] < 0
        lo = [torch.floor(v) for v in c]
        ok = (lo[1] >= -(T // 2)) & (lo[1] + 1 <= T // 2 - 1) & (lo[2] >= -(T // 2)) & (lo[2] + 1 <= T // 2 - 1)
        ok &= torch.where(neg, lo[0] >= -(T // 2), lo[0] + 1 <= T // 2)
        acc = torch.zeros(T, T // 2 + 1, 2, device=DEV, dtype=torch.float64)
        for dz in (0, 1):
            for dy in (0, 1):
                for dx in (0, 1):
                    p = [(lo[q] + d).long() for q, d in enumerate((dx, dy, dz))]
                    w = 1.0
                    for q in range(3):
                        w = w * (1.0 - (c[q].double() - p[q].double()).abs())
                    s = torch.where(neg, -1, 1)
                    px, py, pz = (s * v for v in p)
                    idx = ((pz % T) * T + py % T) * (T // 2 + 1) + px.clamp(0, T // 2)
                    v = vol[idx]
                    acc[..., 0] += torch.where(ok, w * v[..., 0], 0.0)
                    acc[..., 1] += torch.where(ok, w * s * v[..., 1], 0.0)
        acc[..., 1] = torch.where(mirror, -acc[..., 1], acc[..., 1])
        sl = torch.view_as_complex(acc)
        sl[0, 0] = 0
        par = (jl[:, None] + torch.arange(T // 2 + 1, device=DEV)) & 1
        sl = torch.where(par == 1, -sl, sl)
        if filt is not None:
            sl = sl * filt.double()
        col = torch.fft.ifft(sl, dim=0, norm="forward")
        out.append(torch.fft.irfft(col, n=T, dim=1, norm="forward"))
    return torch.stack(out)


def _ctf(T):
    """CTF of the planted particles and of the filters (300 kV, 2.7 mm, 1.2 um, 1 A/px)."""
    return torch.from_numpy(prep.projection_filter(T, np.ones(64), kv=300.0, cs_mm=2.7, amplitude_contrast=0.07,
                                                   defocus1=12000.0, defocus2=12000.0, pixel_size=1.0)).to(DEV)


def _micrograph(X, Y, tspec, angles, g, z=16.0):
    """Unit white noise plus one particle per row of angles whose matched-filter score is about z."""
    T = tspec.shape[0]
    img = torch.randn(Y, X, generator=g, device=DEV, dtype=torch.float64)
    proj = _project(tspec, angles, _ctf(T))
    at = torch.rand(len(proj), 2, generator=g, device=DEV)
    for p, (u, v) in zip(proj, at.tolist()):
        p = p - p.mean()
        y0, x0 = int(u * (Y - T)), int(v * (X - T))
        img[y0:y0 + T, x0:x0 + T] += p * (z / p.norm())
    return img


def _whitened(img):
    """Whitened unit-norm half spectrum (complex64) with the quadrants swapped, and the radial filter."""
    Y, X = img.shape
    spec = torch.fft.rfft2(img) / img.numel() * _swap(Y, X)
    spec[0, 0] = 0
    n = int((X / 2.0 + 1.0) * math.sqrt(2.0) + 1.0)
    f = torch.sqrt((torch.arange(X // 2 + 1, device=DEV) / X) ** 2 + (_logical(Y) / Y)[:, None] ** 2)
    b = (f * (n - 1) / (0.5 * math.sqrt(2.0))).round().long().clamp(max=n - 1).reshape(-1)
    pw = torch.zeros(n, device=DEV, dtype=torch.float64).index_add_(0, b, spec.abs().square().reshape(-1))
    cnt = torch.zeros(n, device=DEV, dtype=torch.float64).index_add_(0, b, torch.ones_like(b, dtype=torch.float64))
    c = torch.where(pw > 0, (cnt / pw.clamp(min=1e-300)).sqrt(), 0.0)
    c = c / c.max()
    spec = spec * c[b].reshape(spec.shape)
    spec = spec / (math.sqrt(2.0) * spec.norm())
    return spec.to(torch.complex64), c.cpu().numpy()


def _angles(step, psi, positions):
    grid = prep.search_grid(step)
    first = max(0, len(grid) // 2 - positions // 2)   # views around the equator
    last = min(len(grid), first + positions) - 1
    return grid, first, last


# ---------------------------------------------------------------------------------------------
def _search_inputs(case, seed):
    g = _gen(seed)
    T, X, Y = case["T"], case["X"], case["Y"]
    grid, first, last = _angles(case["step"], case["psi"], case["positions"])
    ang = core.orientation_list(grid, 0.0, case["psi"], 360.0, first, last)
    tspec = _template(T, g)
    pick = torch.randint(len(ang), (max(1, min(24, X * Y // (T * T * 4))),), generator=g, device=DEV).cpu().numpy()
    ispec, curve = _whitened(_micrograph(X, Y, tspec, ang[pick], g))
    filt = prep.projection_filter(T, curve, kv=300.0, cs_mm=2.7, amplitude_contrast=0.07, defocus1=12000.0,
                                  defocus2=12000.0, pixel_size=1.0)
    return dict(tspec=tspec, ispec=ispec, filt=filt, ang=ang, grid=grid, first=first, last=last)


def _windows_inputs(case, seed):
    g = _gen(seed)
    T, W = case["T"], case["W"]
    ang = core.orientation_list(prep.search_grid(2.5), 0.0, 1.5, 360.0, 2000, 2000 + case["bins"] * case["per_bin"] // 241 + 1)
    tspec = _template(T, g)
    bins = [ang[b * case["per_bin"]:(b + 1) * case["per_bin"]] for b in range(case["bins"])]
    # every bin is wanted by some of the windows, the first by all of them
    ids = [[w for w in range(case["images"]) if b == 0 or (w + b) % 2 == 0 or w == b % case["images"]] for b in range(len(bins))]
    spectra = []
    for w in range(case["images"]):
        s, curve = _whitened(_micrograph(W, W, tspec, bins[0][[(37 * w + 5) % len(bins[0])]], g))
        spectra.append(s * (W * W / N_FULL))
    filt = prep.projection_filter(T, curve, kv=300.0, cs_mm=2.7, amplitude_contrast=0.07, defocus1=12000.0,
                                  defocus2=12000.0, pixel_size=1.0)
    return dict(tspec=tspec, spectra=torch.stack(spectra), filt=filt, bins=bins, ids=ids)


FACTORS = (0.98, 0.99, 1.01, 1.02)


def _refine_inputs(case, seed):
    g = _gen(seed)
    T, TP, n = case["T"], case["TP"], case["n"]
    tspec = _template(TP, g)
    u = torch.rand(n, 6, generator=g, device=DEV).cpu().numpy().astype(np.float32)
    euler = np.ascontiguousarray(u[:, :3] * np.float32([360.0, 180.0, 360.0]))
    n_part = min(n, 16)
    win = torch.randn(n_part, T, T, generator=g, device=DEV, dtype=torch.float64)
    proj = _project(tspec, euler[:n_part])
    o = (TP - T) // 2
    proj = proj[:, o:o + T, o:o + T]
    proj = torch.fft.irfft2(torch.fft.rfft2(proj) * _ctf(T), s=(T, T))   # the particle's CTF
    proj = proj - proj.mean(dim=(1, 2), keepdim=True)
    win += proj * (20.0 / proj.flatten(1).norm(dim=1))[:, None, None]
    par = (torch.arange(T, device=DEV)[:, None] + torch.arange(T // 2 + 1, device=DEV)) & 1
    part = torch.fft.rfft2(win) / (T * T) * torch.where(par == 1, -1.0, 1.0)
    filters = np.stack([prep.projection_filter(T, np.ones(64), kv=300.0, cs_mm=2.7, amplitude_contrast=0.07,
                                               defocus1=11900.0 + 50.0 * k, defocus2=11900.0 + 50.0 * k, pixel_size=1.0)
                        for k in range(4)])
    ops = [hostprep.pixel_size_operator(TP, T, f) for f in FACTORS] if case["resampled"] > 0 else []
    op = np.where(u[:, 4] < case["resampled"], (u[:, 5] * 3.99).astype(np.int32), -1).astype(np.int32)
    return dict(tspec=tspec, euler=euler, part=part.to(torch.complex64), filters=filters, ops=ops,
                pid=(np.arange(n) % n_part).astype(np.int32), fid=(u[:, 3] * 3.99).astype(np.int32), op=op)


def _whiten_inputs(case, seed):
    g = _gen(seed)
    X, Y = case["X"], case["Y"]
    # detector noise over a background that falls off with frequency, and a few hot pixels
    img = torch.randn(Y, X, generator=g, device=DEV, dtype=torch.float64)
    k2 = (torch.arange(X // 2 + 1, device=DEV) / X) ** 2 + (_logical(Y) / Y)[:, None] ** 2
    img = torch.fft.irfft2(torch.fft.rfft2(img) * (0.3 + 1.0 / (1.0 + 400.0 * k2)), s=(Y, X))
    hot = torch.randint(X * Y, (50,), generator=g, device=DEV)
    img.view(-1)[hot] = 40.0
    return img.float()


def _network_inputs(case, seed):
    rng = np.random.default_rng(seed)
    g = _gen(seed)
    n, t = case["n"], case["tile"]
    x = torch.randn(n, proposal.FEATURES, t, t, generator=g, device=DEV).cpu().numpy()
    lab = np.zeros((n, 4), np.float32)
    pos = rng.random(n) < 0.5   # balanced batches
    d = rng.standard_normal((n, 3))
    lab[:, 1:] = d / np.linalg.norm(d, axis=1, keepdims=True)
    lab[:, 0] = pos
    lab[~pos, 1:] = 0.0
    return x, lab, proposal.init_params(seed=seed % 100000)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "search":
        d = _search_inputs(case, seed)
        hmin, hstep = prep.histogram_scaled(case["X"], case["Y"])
        tm = core.TemplateMatchingCore()
        tm.Init(d["tspec"].cpu().numpy(), d["ispec"].cpu().numpy(), 0.0, 0.0, 1.0, 0.0, 0.0, 12000.0, 12000.0, 360.0, 0.0,
                case["psi"], d["grid"], hmin, hstep, prep.HISTOGRAM_BINS, 1.0, d["first"], d["last"], image_x=case["X"],
                orientation_batch=case["batch"])
        return dict(kind=kind, core=tm, filt=d["filt"], limit=np.float32(PEAK / math.sqrt(case["X"] * case["Y"])))
    if kind == "windows":
        d = _windows_inputs(case, seed)
        hmin, hstep = prep.histogram_scaled(4096, 4096)
        sc = core.SearchCore(case["W"], case["W"], case["T"], histogram_min_scaled=hmin, histogram_step_scaled=hstep,
                             orientation_batch=case["batch"])
        sc.set_template(d["tspec"].cpu().numpy())
        sc.set_normalization_pixels(N_FULL)
        sc.set_image_set(d["spectra"].cpu().numpy())
        return dict(kind=kind, core=sc, filt=d["filt"], bins=d["bins"], ids=d["ids"], images=case["images"],
                    limit=np.float32(PEAK / math.sqrt(N_FULL)))
    if kind == "refine":
        d = _refine_inputs(case, seed)
        rc = core.RefineCore(d["tspec"].cpu().numpy(), case["T"], max_batch=max(64, case["n"]), max_particles=16,
                             max_filters=4, max_operators=4)
        for k, p in enumerate(d["part"].cpu().numpy()):
            rc.set_particle(k, p)
        for k, f in enumerate(d["filters"]):
            rc.set_filter(k, f)
        for k, (info, *ops) in enumerate(d["ops"]):
            rc.set_operator(k, *ops, info["has_pad_value"])
        return dict(kind=kind, core=rc, args=(d["euler"], d["pid"], d["fid"], d["op"]))
    if kind == "whiten":
        return dict(kind=kind, image=_whiten_inputs(case, seed).cpu().numpy())
    x, lab, params = _network_inputs(case, seed)
    net = proposal.ProposalNet(tile=case["tile"], max_batch=max(128, case["n"]))
    net.set_params(params)
    return dict(kind=kind, net=net, x=x, lab=lab)


def _at_peaks(mip, maps, limit, most=1024):
    """The first `most` positions above the threshold (-1 after the last) and the best angles there."""
    at = np.flatnonzero(mip > limit)[:most]
    where, angles = np.full(most, -1, np.int64), np.zeros((most, 3), np.float32)
    where[:len(at)] = at
    for k, m in enumerate(maps):
        angles[:len(at), k] = m.reshape(-1)[at]
    return where, angles


def run(state):
    kind = state["kind"]
    if kind == "search":
        tm = state["core"]
        tm.RunInnerLoop(state["filt"], 0, 0)
        n = tm.total_number_of_cccs_calculated
        mip = tm.d_max_intensity_projection
        at, angles = _at_peaks(mip, (tm.d_best_phi, tm.d_best_theta, tm.d_best_psi), state["limit"])
        mean, square = (torch.from_numpy(s).div(n).float() for s in (tm.d_sum3, tm.d_sumSq3))
        return {"mip": mip, "mean": mean, "mean_square": square, "histogram": tm.histogram.astype(np.float32),
                "peaks": at, "peak_angles": angles}
    if kind == "windows":
        sc = state["core"]
        sc.reset()
        for angles, ids in zip(state["bins"], state["ids"]):
            sc.run_plane_images(state["filt"], angles, ids)
        out = {}
        for w in range(state["images"]):
            r = sc.image_results(w)
            at, angles = _at_peaks(r["mip"], (r["phi"], r["theta"], r["psi"]), state["limit"])
            out["window%d" % w] = {"mip": r["mip"], "peaks": at, "peak_angles": angles}
        return out
    if kind == "refine":
        s = state["core"].score(*state["args"])
        return {"value": s[:, 0], "shift": s[:, 1:]}
    if kind == "whiten":
        spec, curve = core.whiten_micrograph(state["image"])
        return {"spectrum": spec, "curve": curve.astype(np.float32)}
    loss, grads = state["net"].gradients(state["x"], state["lab"], 4.0, 1.0)
    return {"loss": np.float32(loss), "gradients": grads}


# ---------------------------------------------------------------------------------------------
def _orientations(case):
    if case["kind"] == "windows":
        d = [b for b in range(case["bins"])]
        pairs = sum(len([w for w in range(case["images"]) if b == 0 or (w + b) % 2 == 0 or w == b % case["images"]]) for b in d)
        return pairs * case["per_bin"]
    _, first, last = _angles(case["step"], case["psi"], case["positions"])
    return (last - first + 1) * (int(360.0 / case["psi"]) + 1)


def work(case):
    kind = case["kind"]
    if kind in ("search", "windows"):
        T = case["T"]
        n = case["X"] * case["Y"] if kind == "search" else case["W"] ** 2
        images = case.get("images", 1)
        # inputs: template spectrum, micrograph spectrum, filter; outputs: MIP, 3 angles, sum, sum of squares
        return {"bytes": 4.0 * T ** 3 + images * n * (4.0 + 4 * 4 + (16 if kind == "search" else 0)),
                # the two micrograph-size real transforms and the per-pixel update of every orientation
                "flops": float(_orientations(case)) * n * (5.0 * math.log2(n) + 10.0)}
    if kind == "refine":
        T, TP, n = case["T"], case["TP"], case["n"]
        ops = n * case["resampled"] * 2.0 * (2.0 * TP * TP * T + 2.0 * TP * T * T)
        return {"bytes": 4.0 * TP ** 3 + min(n, 16) * 4.0 * T * T + 8.0 * T * T + n * 40.0,
                "flops": n * (T * T * 2 * 5.0 * math.log2(T) * 2 + TP * TP * (5.0 * math.log2(TP) + 30.0)) + ops}
    if kind == "whiten":
        n = case["X"] * case["Y"]
        return {"bytes": 8.0 * n, "flops": n * (2.5 * math.log2(n) + 20.0)}
    n, t = case["n"], case["tile"]
    chans = (proposal.FEATURES, 32, 64, 128, 128)
    fwd = sum(2.0 * 9 * chans[i] * chans[i + 1] * (t >> i) ** 2 for i in range(4))
    back = 2.0 * fwd - 2.0 * 9 * chans[0] * chans[1] * t * t
    return {"bytes": 4.0 * n * chans[0] * t * t + 8.0 * sum(9 * chans[i] * chans[i + 1] for i in range(4)),
            "flops": n * (fwd + back)}


# ---------------------------------------------------------------------------------------------
def _correlations(proj, ispec, X, Y, norm_pixels):
    """Correlation map of one projection (T, T) with the micrograph spectrum, FP64."""
    T = proj.shape[0]
    edge = torch.cat([proj[0], proj[-1], proj[1:-1, 0], proj[1:-1, -1]]).mean()
    p = proj - edge
    r = T * T / float(norm_pixels)
    p = p / torch.sqrt(p.square().mean() * r - (p.mean() * r) ** 2)
    big = torch.zeros(Y, X, device=DEV, dtype=torch.float64)
    big[Y // 2 - T // 2:Y // 2 - T // 2 + T, X // 2 - T // 2:X // 2 - T // 2 + T] = p
    f = torch.fft.rfft2(big) / (X * Y)
    f[0, 0] = 0
    z = torch.fft.ifft(ispec * f.conj(), dim=0, norm="forward")
    return torch.fft.irfft(z, n=X, dim=1, norm="forward")


def exact(case, seed):
    kind = case["kind"]
    if kind in ("search", "windows"):
        n_or = _orientations(case)
        n_px = case["X"] * case["Y"] if kind == "search" else case["W"] ** 2
        # FP64 transforms and, per orientation, the slice's gathers
        if n_or * (n_px * 4.0e-10 + 2.0e-3) > 12.0:
            return None
    if kind == "search":
        d = _search_inputs(case, seed)
        X, Y = case["X"], case["Y"]
        filt, ispec = torch.from_numpy(d["filt"]).to(DEV), d["ispec"].to(torch.complex128)
        mip = torch.full((Y, X), -math.inf, device=DEV, dtype=torch.float64)
        s, q = torch.zeros_like(mip), torch.zeros_like(mip)
        for a in d["ang"]:
            c = _correlations(_project(d["tspec"], a[None], filt)[0], ispec, X, Y, X * Y)
            mip = torch.maximum(mip, c)
            s += c
            q += c * c
        n = len(d["ang"])
        return {"mip": mip, "mean": s / n, "mean_square": q / n, "histogram": None, "peaks": None, "peak_angles": None}
    if kind == "windows":
        d = _windows_inputs(case, seed)
        W = case["W"]
        filt, spectra = torch.from_numpy(d["filt"]).to(DEV), d["spectra"].to(torch.complex128)
        mip = torch.full((case["images"], W, W), -math.inf, device=DEV, dtype=torch.float64)
        for angles, ids in zip(d["bins"], d["ids"]):
            for a in angles:
                p = _project(d["tspec"], a[None], filt)[0]
                for w in ids:
                    mip[w] = torch.maximum(mip[w], _correlations(p, spectra[w], W, W, N_FULL))
        return {"window%d" % w: {"mip": mip[w].reshape(-1), "peaks": None, "peak_angles": None} for w in range(case["images"])}
    if kind == "refine":
        d = _refine_inputs(case, seed)
        T, TP = case["T"], case["TP"]
        i = torch.arange(T // 2 + 1, device=DEV)
        jj = _logical(T)[:, None]
        edge_x, edge_y = (i == 0) | (i == T // 2), (jj == 0) | (jj == -(T // 2))
        wgt = torch.where(edge_x & edge_y, 0.5, torch.where(edge_x & (jj < 0), 0.0, 1.0)).double()
        r = torch.arange(TP, device=DEV) - TP // 2
        disc = (r[:, None] ** 2 + r[None, :] ** 2).float() <= np.float32(np.float32(0.45) * np.float32(TP)) ** 2
        value, shift = [], []
        for k in range(case["n"]):
            p = _project(d["tspec"], d["euler"][k:k + 1])[0]
            if d["op"][k] >= 0:
                info, ar, ai, brt, bit = d["ops"][d["op"][k]]
                ar, ai, brt, bit = (torch.from_numpy(v).to(DEV).double() for v in (ar, ai, brt, bit))
                pv = p[disc].mean() if info["has_pad_value"] else 0.0
                p = ar @ (p - pv) @ brt - ai @ (p - pv) @ bit + pv
            else:
                o = TP // 2 - T // 2
                p = p[o:o + T, o:o + T]
            f = torch.fft.rfft2(p) * torch.from_numpy(d["filters"][d["fid"][k]]).to(DEV).double()
            f[0, 0] = 0
            ss = 2.0 * (f.abs().square() * wgt).sum()
            c = torch.fft.ifft(d["part"][int(d["pid"][k])].to(torch.complex128) * f.conj(), dim=0, norm="forward")
            c = torch.fft.irfft(c, n=T, dim=1, norm="forward")
            at = int(c.argmax())
            value.append(float(c.reshape(-1)[at] / torch.sqrt(ss)))
            shift.append((float(at % T - T // 2), float(at // T - T // 2)))
        return {"value": torch.tensor(value, dtype=torch.float64), "shift": torch.tensor(shift, dtype=torch.float64)}
    if kind == "whiten":
        return _exact_whiten(_whiten_inputs(case, seed).double())
    return _exact_network(case, *_network_inputs(case, seed))


def _exact_whiten(img):
    """match_template's whitening in FP64: outliers, transform, radial curve with linear interpolation, filter, norm."""
    Y, X = img.shape
    mean = img.mean()
    sd = torch.sqrt(img.square().mean() - mean ** 2)
    img = torch.where((img - mean).abs() > 5.0 * sd, mean, img)
    spec = torch.fft.rfft2(img) * _swap(Y, X)
    spec[0, 0] = 0
    n = int((X / 2.0 + 1.0) * math.sqrt(2.0) + 1.0)
    xa = torch.arange(n, device=DEV, dtype=torch.float64) * (0.5 * math.sqrt(2.0) / (n - 1))
    f = torch.sqrt((torch.arange(X // 2 + 1, device=DEV) / X).double() ** 2 + (_logical(Y) / Y).double()[:, None] ** 2)
    i = torch.searchsorted(xa, f.reshape(-1), right=True).sub(1).clamp(0, n - 2).reshape(f.shape)
    d = (f - xa[i]) / (xa[i + 1] - xa[i])
    keep = torch.ones_like(f)
    keep[(Y + 1) // 2:, 0] = 0.0   # explicit Hermitian mates
    pw, cnt = (torch.zeros(n, device=DEV, dtype=torch.float64) for _ in range(2))
    for j, w in ((i, 1.0 - d), (i + 1, d)):
        pw.index_add_(0, j.reshape(-1), (spec.abs().square() * w * keep).reshape(-1))
        cnt.index_add_(0, j.reshape(-1), (w * keep).reshape(-1))
    c = torch.where(cnt > 0, pw / cnt.clamp(min=1e-300), 0.0).sqrt()
    c = torch.where(c != 0, 1.0 / c.clamp(min=1e-300), 0.0)
    c = c / c.max()
    spec = spec * (c[i] * (1.0 - d) + c[i + 1] * d)
    spec[0, 0] = 0
    jj = _logical(Y)[:, None]
    x = torch.arange(X // 2 + 1, device=DEV)
    edge_x = (x == 0) | ((x == X // 2) & (X % 2 == 0))
    edge_y = (jj == 0) | ((jj == -(Y // 2)) & (X % 2 == 0))
    w = torch.where(edge_x & edge_y, 0.5, torch.where(edge_x & (jj < 0), 0.0, 1.0)).double()
    return {"spectrum": spec / torch.sqrt(2.0 * (spec.abs().square() * w).sum()), "curve": c}


def _exact_network(case, x, lab, params):
    """Loss and gradients in FP64 with the BF16 values of the weights (biases FP32)."""
    F = torch.nn.functional
    chans = (proposal.FEATURES, 32, 64, 128, 128)
    p = torch.from_numpy(params).to(DEV)
    parts, at = [], 0
    for ci, co, k in [(chans[i], chans[i + 1], 9) for i in range(4)] + [(128, 4, 1)]:
        w = p[at:at + ci * co * k].bfloat16().double().reshape((co, ci, 3, 3) if k == 9 else (co, ci))
        at += ci * co * k
        b = p[at:at + co].double()
        at += co
        parts += [w.requires_grad_(), b.requires_grad_()]
    h = torch.from_numpy(x).to(DEV).double()
    lab = torch.from_numpy(lab).to(DEV).double()
    for i in range(4):
        h = F.relu(F.conv2d(h, parts[2 * i], parts[2 * i + 1], padding=1))
        h = F.max_pool2d(h, 2) if i < 3 else h.amax(dim=(2, 3))
    out = F.linear(h, parts[8], parts[9])
    y = lab[:, 0]
    bce = F.binary_cross_entropy_with_logits(out[:, 0], y, reduction="none") * torch.where(y > 0.5, 4.0, 1.0)
    cos = (out[:, 1:] * lab[:, 1:]).sum(1) / torch.sqrt(out[:, 1:].square().sum(1) + 1e-12)
    loss = (bce + torch.where(y > 0.5, 1.0 - cos, 0.0)).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "gradients": torch.cat([q.grad.reshape(-1) for q in parts])}
