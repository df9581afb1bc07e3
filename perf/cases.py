"""Performance cases: the work that users of this framework have it do.

A case names a size; ``prepare`` makes what a program has in hand before the
call (seeded, on the GPU), ``run`` makes one pass through the public entry
points, ``work`` counts what a pass cannot do without and ``exact`` computes
the same outputs in 64 bits with plain torch.

Kinds:
  search  whole-orientation search of one micrograph: the drop-in
          ``core_match_template`` (results on the host) or the stateful
          ``MatchTemplateSearch`` (results left on the device), optionally
          followed by peak picking;
  refine  ``core_refine_template``: the local grid of a particle stack;
  xcorr   ``cross_correlate_particle_stack``: one correlogram per particle;
  train   forward and backward pass of the refinement's proposal network.

The searches return their continuous maps.  The decoded pose maps are step
functions of the winning index, which changes between correlograms that tie to
rounding; they are compared where a program reads them, at the picked peaks
(cases with ``peaks``).
"""

from __future__ import annotations

import math

import torch

DEV = "cuda"

# rows / columns of the correlation grids that a micrograph is zero padded to
GRID_ROWS = (48, 64, 128, 256, 288, 512, 576, 1024, 2048, 2880, 3072, 3840, 4096, 5760)
GRID_COLS = (48, 64, 80, 128, 256, 288, 512, 576, 1024, 2048, 2880, 3072, 3840, 4096, 5760)
TEMPLATES = (32, 48, 64, 96, 128, 192, 256, 288, 384, 512)
CROPS = ((64, 48), (128, 96), (256, 192), (288, 256), (512, 384))

VOLTAGE, CS_MM, AMP, PIXEL = 300.0, 2.7, 0.07, 1.06

# the proposal network's layers (kind, in, out, stride, relu)
NET = (("conv", 12, 48, 2, True), ("conv", 48, 96, 2, True), ("conv", 96, 128, 2, True),
       ("conv", 128, 128, 2, True), ("conv", 128, 128, 1, True), ("fc", 2048, 1152, 1, True),
       ("fc", 1152, 256, 1, True), ("fc", 256, 7, 1, False))


def _search(name, h, w, d, c, df, n, b, entry, peaks=False):
    return {"name": name, "kind": "search", "h": h, "w": w, "d": d, "c": c, "df": df, "n": n, "batch": b,
            "entry": entry, "peaks": peaks}


def listed():
    return [
        # a quick look at a few orientations of a small image: launches and host work count
        _search("search-512-short", 512, 512, 64, 1, 1, 24, 8, "core"),
        # the small configuration's whole 20-degree grid, then its peaks
        _search("search-512-grid", 512, 512, 64, 1, 1, 1908, 32, "core", peaks=True),
        # a binned micrograph over defocus planes and pixel sizes
        _search("search-2048", 2048, 2048, 256, 3, 7, 8, 4, "device"),
        # a frame whose sides are no FFT length: zero padded
        _search("search-3838x3710", 3838, 3710, 256, 3, 7, 4, 4, "device"),
        # the production configuration: two of its orientation batches, then the peaks
        _search("search-4096", 4096, 4096, 384, 1, 3, 128, 64, "device", peaks=True),
        # the published benchmark shape: 512 template, 11 defocus planes
        _search("search-4096-512x11", 4096, 4096, 512, 1, 11, 8, 8, "device"),
        # a wide-format camera's frame
        _search("search-5760x4092", 5760, 4092, 256, 3, 7, 4, 4, "device"),
        # one particle refined over a default-sized local grid: latency
        {"name": "refine-one", "kind": "refine", "crop": 288, "d": 256, "p": 1, "rings": 1, "inplane": 5, "df": 9,
         "batch": 32},
        # a micrograph's particles over a finer local grid
        {"name": "refine-288", "kind": "refine", "crop": 288, "d": 256, "p": 32, "rings": 2, "inplane": 7, "df": 9,
         "batch": 32},
        # larger crops, few particles
        {"name": "refine-512", "kind": "refine", "crop": 512, "d": 384, "p": 4, "rings": 1, "inplane": 5, "df": 5,
         "batch": 16},
        # every particle of a stack against its own projection
        {"name": "xcorr-288", "kind": "xcorr", "crop": 288, "d": 256, "p": 300, "mode": "valid", "batch": 1024},
        # one step of the proposal network's training at its batch size
        {"name": "train-256", "kind": "train", "p": 256},
    ]


def _grid(lengths, n):
    """The grid length that holds n pixels."""
    return min(g for g in lengths if g >= n)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "search", "refine", "refine", "xcorr", "train"])
    if kind == "search":
        h, w = _log_int(rng, 256, 5760), 2 * _log_int(rng, 128, 2880)
        d = rng.choice([t for t in TEMPLATES if t <= min(h, w) // 2])
        c, df = rng.choice([1, 1, 3]), rng.randint(1, 11)
        # correlograms in all: at least 48 for the statistics, at most 2e9 pixels of their padded grid
        most = max(48, min(4000, int(2e9 / (_grid(GRID_ROWS, h) * _grid(GRID_COLS, w)))))
        n = max(1, _log_int(rng, 48, most) // (c * df))
        n = max(n, -(-48 // (c * df)))
        b = min(max(_log_int(rng, 1, 64), n // 100), max(1, 192 // (c * df)), n)
        return {"kind": kind, "h": h, "w": w, "d": d, "c": c, "df": df, "n": n, "batch": b,
                "entry": "core" if h * w <= 1 << 20 else "device", "peaks": False}
    if kind == "train":
        return {"kind": kind, "p": _log_int(rng, 33, 255)}
    crop, d = rng.choice(CROPS)
    if kind == "refine":
        rings, inplane, df = rng.randint(0, 2), rng.choice([3, 5, 7]), rng.randint(1, 9)
        k = inplane * (1 + 3 * rings * (rings + 1))
        most = max(1, min(32, int(3e9 / (crop * crop * k * df))))
        return {"kind": kind, "crop": crop, "d": d, "p": _log_int(rng, 1, most), "rings": rings, "inplane": inplane,
                "df": df, "batch": _log_int(rng, 4, 64)}
    most = max(8, min(1000, int(1e8 / (crop * crop))))
    return {"kind": kind, "crop": crop, "d": d, "p": _log_int(rng, 1, most), "mode": rng.choice(["valid", "same"]),
            "batch": 1024}


# ---- inputs (plain torch) -------------------------------------------------------
def _euler_to_rotmat(e):
    """ZYZ Euler angles (degrees) -> R = Rz(phi) Ry(theta) Rz(psi), float64."""
    a = torch.deg2rad(e.double())
    (cp, ct, cs), (sp, st, ss) = a.cos().unbind(-1), a.sin().unbind(-1)
    r = torch.stack([cp * ct * cs - sp * ss, -cp * ct * ss - sp * cs, cp * st, sp * ct * cs + cp * ss,
                     -sp * ct * ss + cp * cs, sp * st, -st * cs, st * ss, ct], dim=-1)
    return r.reshape(*e.shape[:-1], 3, 3)


def _rotmat_to_euler(r):
    return torch.rad2deg(torch.stack([torch.atan2(r[..., 1, 2], r[..., 0, 2]), torch.acos(r[..., 2, 2].clamp(-1, 1)),
                                      torch.atan2(r[..., 2, 1], -r[..., 2, 0])], dim=-1))


def _random_euler(n, gen):
    u = torch.rand((n, 3), generator=gen, device=DEV, dtype=torch.float64)
    # theta stays off the poles, where phi and psi are one angle
    theta = torch.rad2deg(torch.acos((1 - 2 * u[:, 1]).clamp(-0.98, 0.98)))
    return torch.stack([360 * u[:, 0], theta, 360 * u[:, 2]], dim=1).float()


def _freqs(d, dtype=torch.float64):
    ky = torch.fft.fftfreq(d, dtype=dtype, device=DEV)[:, None]
    kx = torch.fft.rfftfreq(d, dtype=dtype, device=DEV)[None, :]
    return ky, kx


def _ctf(d, defocus, astig=0.0, angle_deg=0.0, cs_mm=CS_MM):
    """CTF (float64) on the rfft grid of a d x d box; defocus, astig, angle_deg: numbers or (n, 1, 1)."""
    ky, kx = (k / PIXEL for k in _freqs(d))
    k2 = kx**2 + ky**2
    v = VOLTAGE * 1e3
    h, m0, e, c = 6.62607015e-34, 9.1093837015e-31, 1.602176634e-19, 299792458.0
    lam = h / math.sqrt(2 * m0 * e * v * (1 + e * v / (2 * m0 * c * c))) * 1e10
    df = defocus + astig * torch.cos(2 * (torch.atan2(ky, kx) - torch.deg2rad(torch.as_tensor(
        angle_deg, dtype=torch.float64, device=DEV))))
    chi = (-math.pi * lam * k2 * df + 0.5 * math.pi * cs_mm * 1e7 * lam**3 * k2**2
           - math.atan(AMP / math.sqrt(1 - AMP**2)))
    return -torch.sin(chi)


def _whitening(d):
    ky, kx = _freqs(d)
    r = torch.sqrt(ky**2 + kx**2)
    return (1.0 / (1.0 + 0.6 * torch.exp(-(r / 0.08) ** 2))).float()


def _template(d, gen):
    """A particle's density as Gaussian blobs: (fftshifted rfft, blob centres, blob width)."""
    nb, sigma = (150 if d < 128 else 1000), 1.3
    v = torch.randn((nb, 3), generator=gen, device=DEV)
    r = 0.38 * d * torch.rand((nb, 1), generator=gen, device=DEV) ** (1 / 3)
    centres = v / v.norm(dim=1, keepdim=True) * r  # x, y, z
    g = torch.arange(d, device=DEV, dtype=torch.float32) - d // 2
    gx, gy, gz = (torch.exp(-((g[None] - centres[:, i : i + 1]) ** 2) / (2 * sigma**2)) for i in range(3))
    vol = torch.zeros((d * d, d), device=DEV)
    for a in range(0, nb, 250):
        zy = gz[a : a + 250, :, None] * gy[a : a + 250, None, :]
        vol += zy.reshape(zy.shape[0], d * d).t() @ gx[a : a + 250]
    vol = torch.fft.rfftn(torch.fft.fftshift(vol.reshape(d, d, d)))
    return torch.fft.fftshift(vol, dim=(0, 1)).contiguous(), centres, sigma


def _project(centres, sigma, rot, d):
    p = centres @ rot.float()
    g = torch.arange(d, device=DEV, dtype=torch.float32) - d // 2
    gx = torch.exp(-((g[None] - p[:, 0:1]) ** 2) / (2 * sigma**2))
    gy = torch.exp(-((g[None] - p[:, 1:2]) ** 2) / (2 * sigma**2))
    return gy.t() @ gx


def _unit_spectrum(img):
    """rfft2 with no DC and a mean power of one per Fourier pixel (complex64, contiguous)."""
    f = torch.fft.rfft2(img.double() if img.numel() < 1 << 23 else img)
    f[..., 0, 0] = 0
    w = f.abs().double() ** 2
    s = w.sum(dim=(-2, -1), keepdim=True) + w[..., 1:-1].sum(dim=(-2, -1), keepdim=True)
    n = img.shape[-2] * img.shape[-1]
    return (f * torch.sqrt(n / s)).to(torch.complex64).contiguous()


def _signal(proj, ctf, snr):
    s = torch.fft.irfft2(torch.fft.rfft2(proj.double()) * ctf, s=proj.shape)
    s = s - s.mean()
    return (s * (math.sqrt(snr) / s.std())).float()


def _search_inputs(case, seed):
    h, w, d = case["h"], case["w"], case["d"]
    gen = torch.Generator(device=DEV).manual_seed(seed)
    template, centres, sigma = _template(d, gen)
    euler = _random_euler(case["n"], gen)
    defocus = (torch.arange(case["df"], device=DEV, dtype=torch.float32) - case["df"] // 2) * 200.0
    pixel = (torch.arange(case["c"], device=DEV, dtype=torch.float32) - case["c"] // 2) * 0.02
    cs = [CS_MM / ((PIXEL + 0.02 * (i - case["c"] // 2)) / PIXEL) ** 4 for i in range(case["c"])]
    ctf = torch.stack([torch.stack([_ctf(d, 10000.0 + 200.0 * (j - case["df"] // 2), cs_mm=c)
                                    for j in range(case["df"])]) for c in cs]).float()
    image = torch.randn((h, w), generator=gen, device=DEV)
    box = _ctf(d, 10000.0)
    n_p = max(1, min(24, (h * w) // (6 * d * d)))
    at = torch.rand((n_p, 3), generator=gen, device=DEV).cpu()
    rot = _euler_to_rotmat(euler)
    for y, x, o in at.tolist():
        y0, x0 = int(y * (h - d)), int(x * (w - d))
        sig = _signal(_project(centres, sigma, rot[int(o * case["n"])], d), box, 0.3 if d < 128 else 0.1)
        image[y0 : y0 + d, x0 : x0 + d] -= sig
    return {"image_dft": _unit_spectrum(image), "template_dft": template, "ctf_filters": ctf.contiguous(),
            "whitening_filter_template": _whitening(d), "defocus_values": defocus, "pixel_values": pixel,
            "euler_angles": euler}


def _offsets(case):
    """Local orientation grid of 1-degree steps: rings of tilt axes times in-plane rotations."""
    out = []
    for k in range(case["inplane"]):
        om = float(k - case["inplane"] // 2)
        for r in range(case["rings"] + 1):
            for a in range(6 * r or 1):
                az = 360.0 * a / (6 * r or 1)
                out.append((az, float(r), om - az))
    return torch.tensor(out, device=DEV, dtype=torch.float32)


def _stack_inputs(case, seed):
    crop, d, p = case["crop"], case["d"], case["p"]
    gen = torch.Generator(device=DEV).manual_seed(seed)
    template, centres, sigma = _template(d, gen)
    euler = _random_euler(p, gen)
    tilt = torch.rand((p, 3), generator=gen, device=DEV).double()
    move = torch.rand((p, 3), generator=gen, device=DEV).double()
    jitter = torch.stack([360 * tilt[:, 0], 1.5 * tilt[:, 1], -360 * tilt[:, 0] + 4 * tilt[:, 2] - 2], dim=1)
    true = _euler_to_rotmat(jitter) @ _euler_to_rotmat(euler)
    images = torch.randn((p, crop, crop), generator=gen, device=DEV)
    shift = ((move[:, :2] * 2 - 1) * 3).round().int().cpu().tolist()
    ddf = ((move[:, 2] * 2 - 1) * 200).cpu().tolist()
    o = (crop - d) // 2
    for i in range(p):
        y, x = o + shift[i][0], o + shift[i][1]
        sig = _signal(_project(centres, sigma, true[i], d), _ctf(d, 10000.0 + ddf[i]), 0.2)
        images[i, y : y + d, x : x + d] -= sig
    du = 10000.0 + 150 * torch.rand(p, generator=gen, device=DEV)
    ang = 180 * torch.rand(p, generator=gen, device=DEV)
    return {"particle_stack_dft": _unit_spectrum(images), "template_dft": template, "euler_angles": euler,
            "defocus_u": du, "defocus_v": du - 100.0, "defocus_angle": ang, "gen": gen}


def _refine_inputs(case, seed):
    s = _stack_inputs(case, seed)
    gen, p, m = s.pop("gen"), case["p"], case["crop"] - case["d"] + 1
    s["euler_angle_offsets"] = _offsets(case)
    s["defocus_offsets"] = (torch.arange(case["df"], device=DEV, dtype=torch.float32) - case["df"] // 2) * 100.0
    s["pixel_size_offsets"] = torch.zeros(1, device=DEV)
    s["corr_mean"] = 0.05 * torch.randn((p, m, m), generator=gen, device=DEV)
    s["corr_std"] = 1.0 + 0.05 * torch.rand((p, m, m), generator=gen, device=DEV)
    s["projective_filters"] = _whitening(case["d"]).expand(p, -1, -1).contiguous()
    return s


def _xcorr_inputs(case, seed):
    s = _stack_inputs(case, seed)
    ctf = _ctf(case["d"], (0.5 * (s["defocus_u"] + s["defocus_v"])).double()[:, None, None], 50.0,
               s["defocus_angle"].double()[:, None, None])
    return {"particle_stack_dft": s["particle_stack_dft"], "template_dft": s["template_dft"],
            "rotation_matrices": _euler_to_rotmat(s["euler_angles"]).float().contiguous(),
            "projective_filters": (ctf * _whitening(case["d"])).float().contiguous()}


def _train_inputs(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    w, b = [], []
    for kind, cin, cout, _, _ in NET:
        shape, fan = ((cout, cin, 3, 3), 9 * cin) if kind == "conv" else ((cout, cin), cin)
        w.append(torch.randn(shape, generator=gen, device=DEV) * math.sqrt(2.0 / fan))
        b.append(0.05 * torch.randn(cout, generator=gen, device=DEV))
    # six band-limited images and the six constant maps of a first estimate, which the target is near
    x = torch.randn((case["p"], 12, 64, 64), generator=gen, device=DEV)
    ky, kx = _freqs(64, torch.float32)
    img = torch.fft.irfft2(torch.fft.rfft2(x[:, :6]) * torch.exp(-((ky**2 + kx**2) / 0.02)), s=(64, 64))
    x[:, :6] = img / img.std(dim=(2, 3), keepdim=True)
    step = torch.randn((case["p"], 6, 1, 1), generator=gen, device=DEV)
    x[:, 6:] = step
    target = torch.cat([step[:, :, 0, 0], step[:, :1, 0, 0]], dim=1)
    return w, b, x.to(torch.bfloat16), target + 0.2 * torch.randn((case["p"], 7), generator=gen, device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "search":
        return {"case": case, "kwargs": _search_inputs(case, seed)}
    if kind == "refine":
        return {"case": case, "kwargs": _refine_inputs(case, seed), "ctf_kwargs": {
            "voltage": VOLTAGE, "spherical_aberration": CS_MM, "amplitude_contrast_ratio": AMP, "ctf_B_factor": 0.0,
            "phase_shift": 0.0, "pixel_size": PIXEL, "template_shape": (case["d"], case["d"]),
            "even_zernikes": None, "odd_zernikes": None, "mag_matrix": None}}
    if kind == "xcorr":
        return {"case": case, "kwargs": _xcorr_inputs(case, seed)}
    from leopard_em_gb300.proposal import ProposalNet

    w, b, x, target = _train_inputs(case, seed)
    net = ProposalNet(DEV)
    net.load({f"w{i}": t.cpu().numpy() for i, t in enumerate(w)} | {f"b{i}": t.cpu().numpy() for i, t in enumerate(b)})
    return {"case": case, "net": net, "x": x, "target": target}


# ---- one pass ---------------------------------------------------------------------
PEAK_ROWS = 512
MAPS = ("mip", "scaled_mip", "correlation_mean", "correlation_variance")


def _run_search(case, kwargs):
    from leopard_em_gb300.backend import MatchTemplateSearch, core_match_template

    if case["entry"] == "core":
        res = core_match_template(**kwargs, device=DEV, orientation_batch_size=case["batch"])
    else:
        search = MatchTemplateSearch(**kwargs, device=DEV, orientation_batch_size=case["batch"])
        search.run()
        res = search.result(to_cpu=False)
    out = {k: res[k] for k in MAPS}
    if case["peaks"]:
        from leopard_em_gb300.peaks import extract_peaks_and_statistics_zscore

        found = extract_peaks_and_statistics_zscore(
            res["mip"], res["scaled_mip"], res["best_psi"], res["best_theta"], res["best_phi"], res["best_defocus"],
            res["correlation_mean"], res["correlation_variance"], res["total_projections"], device=DEV)
        # a table of fixed length, as many rows as no image here has peaks
        out["peaks"] = [torch.nn.functional.pad(t, (0, PEAK_ROWS - t.numel())) for t in (
            found.pos_y, found.pos_x, found.phi, found.theta, found.psi, found.relative_defocus)]
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "search":
        return _run_search(case, state["kwargs"])
    if case["kind"] == "refine":
        from leopard_em_gb300.backend import core_refine_template

        return core_refine_template(**state["kwargs"], ctf_kwargs=state["ctf_kwargs"], device=DEV,
                                    batch_size=case["batch"])
    if case["kind"] == "xcorr":
        from leopard_em_gb300.backend import cross_correlate_particle_stack

        return cross_correlate_particle_stack(**state["kwargs"], mode=case["mode"], batch_size=case["batch"])
    net = state["net"]
    out = net.forward(state["x"])
    loss, dout = net.loss_and_grad(out, state["target"])
    net.backward(dout)
    return {"out": out, "loss": loss, "gw": list(net.gw), "gb": list(net.gb)}


# ---- what a pass cannot do without ------------------------------------------------
def work(case):
    """Bytes: inputs read once, outputs written once.  FLOPs: per correlogram a
    real forward and a real inverse 2-D FFT of the image size (2.5 n log2 n
    each), the cross power and the statistics (7 n); the projection itself."""
    if case["kind"] == "train":
        n, macs, params, act, hw = case["p"], 0, 0, 12 * 64 * 64 * 2, 64
        for kind, cin, cout, stride, _ in NET:
            hw = hw // stride if kind == "conv" else 1
            size = cin * cout * (9 if kind == "conv" else 1)
            macs += size * hw * hw
            params += size + cout
        first = 12 * 48 * 9 * 32 * 32  # the first layer has no input gradient
        return {"bytes": n * (act + 7 * 8) + params * (2 + 4), "flops": 2.0 * n * (3 * macs - first)}
    d = case["d"]
    filt = d * (d // 2 + 1)
    if case["kind"] == "search":
        h, w = case["h"], case["w"]
        n_img, c = 1, case["n"] * case["c"] * case["df"]
        out = 4 * 4 * h * w
        small = case["c"] * case["df"] * filt * 4
    else:
        h = w = case["crop"]
        n_img = case["p"]
        small = n_img * filt * 4
        if case["kind"] == "xcorr":
            c = n_img
            m = h if case["mode"] == "same" else h - d + 1
            out = 4 * n_img * m * m
        else:
            c = n_img * case["inplane"] * (1 + 3 * case["rings"] * (case["rings"] + 1)) * case["df"]
            out = n_img * (40 + 8 * (h - d + 1) ** 2)
    n = float(h * w)
    flops = c * (5 * n * math.log2(n) + 7 * n + 2.5 * d * d * math.log2(d * d) + 30 * filt)
    return {"bytes": n_img * h * (w // 2 + 1) * 8 + 8 * d * filt + small + out, "flops": flops}


# ---- the same outputs in 64 bits ---------------------------------------------------
def _slices(template, rot):
    """Central slices (n, d, d//2+1) of the fftshifted spectrum: trilinear,
    Friedel mates for x < 0, zero outside; rows in fft order, DC 0, contrast flipped."""
    d, wc = template.shape[0], template.shape[2]
    ky, kx = _freqs(d)
    g = torch.stack([kx.expand(d, wc), ky.expand(d, wc), torch.zeros(d, wc, device=DEV, dtype=torch.float64)], -1)
    q = torch.einsum("nij,abj->nabi", rot.double(), g)
    conj = q[..., 0] < 0
    q = torch.where(conj[..., None], -q, q) * d
    x, y, z = q[..., 0], q[..., 1] + d // 2, q[..., 2] + d // 2
    ok = (z >= 0) & (z <= d - 1) & (y >= 0) & (y <= d - 1) & (x >= 0) & (x <= wc - 1)
    out = torch.zeros(q.shape[:-1], dtype=torch.complex128, device=DEV)
    i0 = [c.floor().long() for c in (z, y, x)]
    t = [c - i for c, i in zip((z, y, x), i0)]
    for corner in range(8):
        idx, wgt = [], 1.0
        for a, n in enumerate((d, d, wc)):
            up = (corner >> a) & 1
            idx.append((i0[a] + up).clamp(0, n - 1))
            wgt = wgt * (t[a] if up else 1 - t[a])
        out += template[idx[0], idx[1], idx[2]] * wgt
    out = torch.where(ok, torch.where(conj, out.conj(), out), 0)
    out[:, 0, 0] = 0
    return -out


def _normalised(proj, h, w):
    """Edge mean removed, scaled to unit variance of the zero-padded h x w image."""
    d = proj.shape[-1]
    edge = proj[..., 0, :].sum(-1) + proj[..., -1, :].sum(-1) + proj[..., 1:-1, 0].sum(-1) + proj[..., 1:-1, -1].sum(-1)
    proj = proj - (edge / (4 * d - 4))[..., None, None]
    rel = d * d / (h * w)
    mean = proj.mean(dim=(-2, -1), keepdim=True) * rel * rel
    var = ((proj - mean) ** 2).sum(dim=(-2, -1), keepdim=True) + (h - d) * (w - d) * mean**2
    return proj * math.sqrt(h * w) / var.clamp_min(1e-8).sqrt()


def _correlate(spectrum, slices, size, norm, dc):
    """Correlograms (size) of ``spectrum`` with the filtered slices' projections."""
    d = slices.shape[-2]
    proj = torch.fft.ifftshift(torch.fft.irfft2(slices, s=(d, d)), dim=(-2, -1))
    f = torch.fft.rfft2(_normalised(proj, *norm), s=size)
    if not dc:
        f[..., 0, 0] = 0
    return torch.fft.irfft2(spectrum * f.conj(), s=size)


def _exact_search(case, seed):
    k = _search_inputs(case, seed)
    h, w = case["h"], case["w"]
    grid = (_grid(GRID_ROWS, h), _grid(GRID_COLS, w))
    spec = k["image_dft"].to(torch.complex128)
    if grid != (h, w):
        img = torch.fft.irfft2(spec, s=(h, w))
        spec = torch.fft.rfft2(img, s=grid)
    pf = (k["ctf_filters"] * k["whitening_filter_template"]).double().reshape(-1, *k["ctf_filters"].shape[2:])
    template, rot = k["template_dft"].to(torch.complex128), _euler_to_rotmat(k["euler_angles"])
    mip = torch.full(grid, -math.inf, dtype=torch.float64, device=DEV)
    s1, s2 = torch.zeros_like(mip), torch.zeros_like(mip)
    step = max(1, int(2**26 / (grid[0] * grid[1])))
    for o in range(case["n"]):
        sl = _slices(template, rot[o : o + 1])
        for a in range(0, pf.shape[0], step):
            cc = _correlate(spec, sl * pf[a : a + step], grid, (h, w), False)
            mip = torch.maximum(mip, cc.amax(dim=0))
            s1 += cc.sum(dim=0)
            s2 += (cc**2).sum(dim=0)
    n = case["n"] * pf.shape[0]
    mean = s1 / n
    std = (s2 / n - mean**2).clamp_min(0).sqrt()
    z = torch.where(std > 0, (mip - mean) / std, torch.zeros_like(mip))
    out = {key: v[:h, :w].contiguous() for key, v in zip(MAPS, (mip, z, mean, std))}
    if case["peaks"]:
        out["peaks"] = None
    if case["entry"] == "core":
        out = {key: v.cpu() if v is not None else None for key, v in out.items()}
    return out


def _exact_refine(case, seed):
    k = _refine_inputs(case, seed)
    crop, d, p = case["crop"], case["d"], case["p"]
    m, offs = crop - d + 1, k["euler_angle_offsets"]
    template = k["template_dft"].to(torch.complex128)
    r_off, r_p = _euler_to_rotmat(offs), _euler_to_rotmat(k["euler_angles"])
    zs, ccs, eul = [], [], []
    for i in range(p):
        du, dv = float(k["defocus_u"][i]), float(k["defocus_v"][i])
        ctf = _ctf(d, 0.5 * (du + dv) + k["defocus_offsets"].double()[:, None, None], 0.5 * abs(du - dv),
                   float(k["defocus_angle"][i]))
        pf = ctf * k["projective_filters"][i].double()
        spec = k["particle_stack_dft"][i].to(torch.complex128)
        best = None
        for a in range(0, offs.shape[0], case["batch"]):
            sl = _slices(template, r_off[a : a + case["batch"]] @ r_p[i])
            top = []
            for f in pf:
                cc = _correlate(spec, sl * f, (crop, crop), (crop, crop), False)[..., :m, :m]
                z = ((cc - k["corr_mean"][i].double()) / k["corr_std"][i].double()).flatten(1).amax(dim=1)
                top.append(torch.stack([z, cc.flatten(1).amax(dim=1)], dim=1))
            top = torch.stack(top)  # (defocus, offset, 2)
            z, at = top[..., 0].flatten().max(dim=0)
            if best is None or z > best[0]:
                best = (z, top[..., 1].max(), a + int(at) % top.shape[1])
        zs.append(best[0])
        ccs.append(best[1])
        e = _rotmat_to_euler(r_off[best[2]] @ r_p[i])
        eul.append(torch.where(e < 0, e + torch.tensor([360.0, 180.0, 360.0], device=DEV, dtype=e.dtype), e))
    return {"refined_cross_correlation": torch.stack(ccs).cpu(), "refined_z_score": torch.stack(zs).cpu(),
            "refined_euler_angles": torch.stack(eul).cpu()}


def _exact_xcorr(case, seed):
    k = _xcorr_inputs(case, seed)
    crop, d = case["crop"], case["d"]
    template, out = k["template_dft"].to(torch.complex128), []
    for a in range(0, case["p"], 32):
        sl = _slices(template, k["rotation_matrices"][a : a + 32]) * k["projective_filters"][a : a + 32].double()
        cc = _correlate(k["particle_stack_dft"][a : a + 32].to(torch.complex128), sl, (crop, crop), (crop, crop), True)
        out.append(cc if case["mode"] == "same" else cc[:, : crop - d + 1, : crop - d + 1])
    return torch.cat(out).contiguous()


def _exact_train(case, seed):
    w, b, x, target = _train_inputs(case, seed)
    w = [t.to(torch.bfloat16).double().requires_grad_() for t in w]
    b = [t.double().requires_grad_() for t in b]
    a = x.double()
    for (kind, _, _, stride, relu), wi, bi in zip(NET, w, b):
        if kind == "conv":
            a = torch.nn.functional.conv2d(a, wi, bi, stride=stride, padding=1)
        else:
            a = torch.nn.functional.linear(a.flatten(1), wi, bi)
        a = torch.relu(a) if relu else a
    loss = ((a - target.double()) ** 2).sum() / case["p"]
    loss.backward()
    return {"out": a.detach(), "loss": loss.detach().reshape(1), "gw": [t.grad for t in w], "gb": [t.grad for t in b]}


def exact(case, seed):
    return {"search": _exact_search, "refine": _exact_refine, "xcorr": _exact_xcorr,
            "train": _exact_train}[case["kind"]](case, seed)
