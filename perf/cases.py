"""The workloads whose speed this framework is held to, each through its public classes.

``listed`` gives them, ``draw`` gives more of the same ranges, ``prepare`` makes
what a program holds before the call, ``run`` is one pass, ``work`` its least
traffic and arithmetic, and ``exact`` the same results in float64 from plain
torch. The atmosphere is the 9-layer profile of the benchmark (8 m telescope,
r0 = 0.157 m, L0 = 25 m, 30 degrees from zenith); shorter profiles take its
first layers.
"""

import math

import numpy as np
import torch

HEIGHTS = [0, 500, 1000, 2000, 4000, 8000, 12000, 16000, 20000]
FRACTIONS = [0.52, 0.10, 0.07, 0.06, 0.05, 0.06, 0.06, 0.05, 0.03]
DIAMETER, R0, L0, ZENITH, DT = 8.0, 0.157, 25.0, 30.0, 1e-3
WAVELENGTH = 500e-9
ARCSEC = math.pi / (180.0 * 3600.0)
DEVICE = "cuda"


def listed():
    return [
        # one small screen for a unit test or a simulation warm-up: the smallest call, all latency
        {"name": "screen_128", "kind": "screens", "n": 128, "count": 1, "levels": 3},
        # a batch of independent screens, the benchmark's first configuration
        {"name": "screens_256x64", "kind": "screens", "n": 256, "count": 64, "levels": 3},
        # screens of a length with a large prime factor (a pupil plus its field margin), default levels
        {"name": "screens_586x16", "kind": "screens", "n": 586, "count": 16, "levels": 8},
        # Monte-Carlo pupil OPDs of the whole atmosphere, the second half of the headline metric
        {"name": "sample_512x64", "kind": "sample", "n": 512, "count": 64, "layers": 9, "levels": 3},
        # two seconds of frozen-flow frames at 1 kHz, the headline workload
        {"name": "window_512x2000", "kind": "window", "n": 512, "steps": 2000, "layers": 9, "levels": 3},
        # an asterism of guide stars at one instant (tomography); the margin makes an odd-factor grid
        {"name": "pointings_512x5", "kind": "pointings", "n": 512, "stars": 5, "field": 15.0, "layers": 9, "levels": 3},
        # a few steps of a closed loop on boiling turbulence: each frame depends on the one before
        {"name": "boiling_256x4", "kind": "boiling", "n": 256, "steps": 4, "layers": 9, "levels": 3},
        # one frame through the cone of a sodium laser guide star
        {"name": "laser_512", "kind": "laser", "n": 512, "interp": "cubic", "layers": 9, "levels": 3},
        # non-periodic frozen flow, some frames of a long run, default interpolation
        {"name": "extrude_512x8", "kind": "extrude", "n": 512, "steps": 8, "interp": "cubic", "layers": 9},
        # row steps of 16 realisations of 9 layers at 1024 pixels, the benchmark's sparse stencil
        {"name": "rows_1449x144", "kind": "rows", "width": 1449, "screens": 144, "columns": 2, "form": "fp32", "steps": 8},
        # a training step on layer screens, weights and winds: 8 stars and one laser, frames of a sequence
        {"name": "fit_screens_512", "kind": "fit_screens", "n": 512, "size": 768, "batch": 4, "times": 8, "stars": 8, "layers": 9},
        # a training step on layer noise, weights and winds through the spectral frames
        {"name": "fit_spectra_256", "kind": "fit_spectra", "n": 256, "size": 256, "times": 32, "layers": 9, "levels": 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["screens", "screens", "sample", "window", "window", "pointings", "boiling",
                       "laser", "extrude", "rows", "fit_screens", "fit_spectra"])
    layers, levels = rng.randint(3, 9), rng.choice([3, 3, 8])
    # half of the sizes are powers of two, as pupils mostly are, the others anything
    def size(lo, hi):
        if rng.random() < 0.5:
            return 1 << rng.randint(int(math.log2(lo)), int(math.log2(hi)))
        return _log(rng, lo, hi)

    if kind in ("screens", "sample"):
        n = size(64, 1024) if kind == "screens" else size(128, 512)
        case = {"n": n, "count": _log(rng, 1, max(1, 64 * 512 ** 2 // n ** 2)) if n > 64 else 256, "levels": levels}
        if kind == "sample":
            case["layers"] = layers
    elif kind == "window":
        n = size(64, 640)
        case = {"n": n, "steps": _log(rng, 16, max(17, min(2000, 400 * 512 ** 2 // n ** 2))), "layers": layers, "levels": levels}
    elif kind == "pointings":
        case = {"n": size(128, 512), "stars": rng.randint(1, 8), "field": round(rng.uniform(2.0, 15.0), 2), "layers": layers, "levels": levels}
    elif kind == "boiling":
        case = {"n": size(64, 256), "steps": rng.randint(1, 6), "layers": layers, "levels": levels}
    elif kind == "laser":
        case = {"n": size(128, 512), "interp": rng.choice(["cubic", "linear", "lanczos"]), "layers": layers, "levels": levels}
    elif kind == "extrude":
        case = {"n": size(64, 512), "steps": rng.randint(2, 12), "interp": rng.choice(["cubic", "linear", "lanczos"]), "layers": layers}
    elif kind == "rows":
        case = {"width": _log(rng, 180, 1449), "screens": _log(rng, 1, 144), "columns": rng.choice([0, 2]),
                "form": rng.choice(["fp32", "fp32", "bf16x2", "bf16x3"]), "steps": 8}
    elif kind == "fit_screens":
        n = size(64, 512)
        case = {"n": n, "size": n + rng.randint(n // 4, n // 2), "batch": rng.randint(1, 3), "times": rng.randint(2, 8),
                "stars": rng.randint(1, 6), "layers": layers}
    else:
        n = size(64, 256)
        case = {"n": n, "size": n + rng.choice([0, rng.randint(1, n // 4)]), "times": rng.randint(4, 32), "layers": layers, "levels": 3}
    return {"kind": kind, **case}


# ------------------------------------------------------------------ inputs


def _winds(count):
    rng = np.random.default_rng(2024)
    speed, angle = rng.uniform(5.0, 30.0, 9), np.deg2rad(rng.uniform(0.0, 360.0, 9))
    return np.stack([speed * np.cos(angle), speed * np.sin(angle)], axis=1)[:count], speed[:count], np.rad2deg(angle)[:count]


def _fractions(count):
    f = np.asarray(FRACTIONS[:count])
    return f / f.sum()


def _atmosphere(case, seed, **options):
    import pyturb_gb300 as G

    _, speed, angle = _winds(case["layers"])
    table = [G.Layer(h, f, v, d, L0) for h, f, v, d in zip(HEIGHTS, _fractions(case["layers"]), speed, angle)]
    if "levels" in case:
        options["subharmonics"] = case["levels"]
    return G.Atmosphere(table, r0=R0, zenith_angle=ZENITH, diameter=DIAMETER, n=case["n"], seed=seed, **options)


def _start_time(seed):
    return 0.05 + 0.1 * float(np.random.default_rng(seed).uniform())


def _stars(case, seed):
    """Directions in arcsec inside the field."""
    rng = np.random.default_rng(seed + 1)
    radius = 0.95 * case.get("field", 60.0) * np.sqrt(rng.uniform(0, 1, case["stars"]))
    angle = rng.uniform(0, 2 * np.pi, case["stars"])
    return [(float(r * math.cos(a)), float(r * math.sin(a))) for r, a in zip(radius, angle)]


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _coloured(shape, gen):
    """Real Gaussian screens with a turbulence-like spectrum, unit variance."""
    n = shape[-1]
    f = torch.fft.fftfreq(n, device=DEVICE)
    amplitude = (f[:, None] ** 2 + f[None, :] ** 2 + 1.0 / n ** 2) ** (-11.0 / 12.0)
    x = torch.fft.ifft2(torch.fft.fft2(torch.randn(shape, generator=gen, device=DEVICE)) * amplitude).real
    return (x / x.std()).contiguous()


def _target(case, screens, gen):
    """What a sensor saw: a static sum of the layers with other weights."""
    n, size = case["n"], case["size"]
    c = (size - n) // 2
    weights = torch.sqrt(torch.tensor(_fractions(case["layers"]), dtype=torch.float32, device=DEVICE))
    weights = weights * (0.8 + 0.4 * torch.rand(len(weights), generator=gen, device=DEVICE))
    return torch.einsum("l,blij->bij", weights, screens[:, :, c:c + n, c:c + n])


def prepare(case, seed):
    import pyturb_gb300 as G

    kind = case["kind"]
    state = {"case": dict(case), "seed": seed}
    if kind == "screens":
        state["screen"] = G.PhaseScreen(n=case["n"], pixel_scale=DIAMETER / 256, r0=0.15, L0=L0, subharmonics=case["levels"], seed=seed)
    elif kind == "sample":
        state["atm"] = _atmosphere(case, seed)
        state["atm"].sample(1)  # makes its generators, as a program's first draw does
    elif kind == "window":
        state["loop"] = _atmosphere(case, seed).frame_loop(DT, case["steps"])
        state["t"] = _start_time(seed)
    elif kind == "pointings":
        state["atm"] = _atmosphere(case, seed, field_of_view=case["field"])
        state["t"], state["stars"] = _start_time(seed), _stars(case, seed)
    elif kind == "boiling":
        state["atm"] = _atmosphere(case, seed, tau_boil=0.05)
    elif kind == "laser":
        state["atm"] = _atmosphere(case, seed, interp=case["interp"], lgs_altitude=90e3)
        state["t"] = _start_time(seed)
    elif kind == "extrude":
        state["atm"] = _atmosphere(case, seed, engine="extrude", interp=case["interp"])
    elif kind == "rows":
        state.update(_ring(case, seed))
    elif kind == "fit_screens":
        state.update(_fit_screens(case, seed))
    else:
        state.update(_fit_spectra(case, seed))
    return state


def _ring(case, seed):
    from pyturb_gb300.backend import NoiseStream
    from pyturb_gb300.covariance import AnchorTables, anchor_modes, build_operator, sparse_points
    from pyturb_gb300.extrude import RingExtruder
    from pyturb_gb300.fourier import PhaseScreen

    W, S, form, steps = case["width"], case["screens"], case["form"], case["steps"]
    dx = DIAMETER / 1024
    sparse = sparse_points(W, 2, case["columns"])
    depth = max([steps] + [d for d, _ in sparse])
    depth = -(-depth // steps) * steps
    operator = build_operator(W, 2, dx, L0, sparse, want_float64=True, want_lo=form == "fp32" and bool(sparse),
                              increments=form == "bf16x3")
    modes = anchor_modes(W, sparse)
    anchor = AnchorTables([operator], modes) if form == "fp32" and modes else None
    r0 = R0 * _fractions(9)[np.arange(S) % 9] ** -0.6
    ring = RingExtruder(W, 2, depth + 8 * steps, [], [0] * S, list(r0 ** (-5.0 / 6.0)),
                        [NoiseStream(seed * 1000 + s, None) for s in range(S)], device_operator=operator.M, form=form,
                        sparse=sparse, operator_lo=operator.Mlo, anchor=anchor, increments=form == "bf16x3")
    side = 1 << (max(W, depth) - 1).bit_length()
    source = PhaseScreen(n=side, pixel_scale=dx, r0=1.0, L0=L0, seed=seed)
    for s in range(S):
        ring.seed_rows(s, source.generate()[:depth, :W] * float(r0[s] ** (-5.0 / 6.0)))
    return {"ring": ring, "operator": operator.M64, "sparse": sparse, "counts": np.full(S, steps, dtype=np.int32)}


def _fit_screens(case, seed):
    from pyturb_gb300.diff import DifferentiableReadout

    gen = _generator(seed)
    L, n, size = case["layers"], case["n"], case["size"]
    stars = [(x * ARCSEC, y * ARCSEC) for x, y in _stars(case, seed)] + [(0.0, 0.0)]
    t0 = _start_time(seed)
    readout = DifferentiableReadout(n, size, DIAMETER / n, HEIGHTS[:L], stars, t0 + DT * np.arange(case["times"]),
                                    source_altitudes=[None] * case["stars"] + [90e3])
    screens = _coloured((case["batch"], L, size, size), gen)
    seen = _target(case, screens, gen)
    target = seen[:, None, None].expand(-1, case["times"], len(stars), -1, -1).contiguous()
    weights = torch.sqrt(torch.tensor(_fractions(L), dtype=torch.float32, device=DEVICE))
    winds = torch.tensor(_winds(L)[0], dtype=torch.float32, device=DEVICE)
    return {"readout": readout, "target": target, "stars": stars, "t": t0, "screens": screens.requires_grad_(True),
            "weights": weights.requires_grad_(True), "winds": winds.requires_grad_(True)}


def _fit_spectra(case, seed):
    from pyturb_gb300.diff import DifferentiableSpectralFrames

    gen = _generator(seed)
    L, n, size, P = case["layers"], case["n"], case["size"], case["levels"]
    t0 = _start_time(seed)
    frames = DifferentiableSpectralFrames(n, size, DIAMETER / n, R0, L0, HEIGHTS[:L], t0 + DT * np.arange(case["times"]),
                                          subharmonics=P)
    noise = torch.randn((L, size, size, 2), generator=gen, device=DEVICE)
    low = torch.randn((L, P, 3, 3, 2), generator=gen, device=DEVICE)
    target = 10.0 * _coloured((case["times"], n, n), gen)
    weights = torch.sqrt(torch.tensor(_fractions(L), dtype=torch.float32, device=DEVICE))
    winds = torch.tensor(_winds(L)[0], dtype=torch.float32, device=DEVICE)
    return {"frames": frames, "target": target, "t": t0, "noise": torch.view_as_complex(noise).requires_grad_(True),
            "low": torch.view_as_complex(low).requires_grad_(True),
            "weights": weights.requires_grad_(True), "winds": winds.requires_grad_(True)}


# ------------------------------------------------------------------ one pass


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "screens":
        return state["screen"].generate(case["count"])
    if kind == "sample":
        return state["atm"].sample(case["count"])
    if kind == "window":
        return state["loop"].render(state["t"])
    if kind == "pointings":
        return state["atm"].opd(state["t"], directions=state["stars"])
    if kind == "boiling":
        return [state["atm"].evolve(DT) for _ in range(case["steps"])]
    if kind == "laser":
        return state["atm"].opd(state["t"])
    if kind == "extrude":
        return [frame for _, frame in state["atm"].frames(DT, case["steps"])]
    if kind == "rows":
        ring = state["ring"]
        ring.extrude(state["counts"])
        end = (int(ring.top[0]) - 1) % ring.cap + 1  # the capacity is a multiple of the steps
        return ring.buf[:, end - case["steps"]:end]
    if kind == "fit_screens":
        leaves = {k: state[k] for k in ("screens", "weights", "winds")}
        loss = torch.nn.functional.mse_loss(state["readout"](*leaves.values()), state["target"])
    else:
        leaves = {k: state[k] for k in ("noise", "weights", "winds", "low")}
        loss = torch.nn.functional.mse_loss(state["frames"](*leaves.values()), state["target"])
    grads = torch.autograd.grad(loss, list(leaves.values()))
    return {"loss": loss.detach(), **dict(zip(leaves, grads))}


# ------------------------------------------------------------------ least work


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    L, P = case.get("layers", 1), case.get("levels", 0)

    def fft(size):  # one complex transform of size x size
        return 10.0 * size * size * math.log2(size)

    if kind in ("screens", "sample"):
        count = case["count"]
        return {"bytes": 4.0 * n * n * (1 + count), "flops": count * (fft(n) / 2 + (2 + 4 * P) * n * n)}
    if kind == "rows":
        W, S, K = case["width"], case["screens"], 3 * case["width"]
        return {"bytes": 4.0 * (W * K + S * case["steps"] * W + 2 * S * W), "flops": 2.0 * W * K * S * case["steps"]}
    if kind == "extrude":  # three sampled rows' worth of new pixels a frame, and the gather
        W, taps = int(1.42 * n) + 4, {"linear": 2, "cubic": 4, "lanczos": 6}[case["interp"]]
        rows = L * case["steps"]
        return {"bytes": 4.0 * (3 * W * W + rows * 3 * W + (L + case["steps"]) * n * n),
                "flops": 2.0 * rows * 3 * W * W + rows * n * n * (2.0 * taps * taps + 20)}
    if kind == "fit_screens":
        size, images = case["size"], case["batch"] * case["times"] * (case["stars"] + 1)
        # screens read, their gradient written, the target read; forward 8 and each adjoint as many a sample
        return {"bytes": 4.0 * (2 * case["batch"] * L * size ** 2 + images * n * n), "flops": 28.0 * images * L * n * n}
    if kind == "fit_spectra":
        size, F = case["size"], case["times"]
        return {"bytes": 8.0 * 2 * L * size ** 2 + 4.0 * F * n * n,
                "flops": F * (fft(size) + 3 * 8.0 * L * size ** 2 / 2 + 12 * P * n * n)}
    frames = case.get("steps", case.get("stars", 1))
    grid = n
    if kind == "pointings":
        grid = n + 2 * _margin(case)
    images = L if kind == "laser" else frames
    spectra = 8.0 * L * grid ** 2 * (2 * frames if kind == "boiling" else 1)
    extra = 50.0 * n * n * L if kind == "laser" else 20.0 * L * grid ** 2 * frames if kind == "boiling" else 0.0
    return {"bytes": spectra + 4.0 * frames * n * n if kind != "laser" else spectra + 4.0 * n * n,
            "flops": images * (fft(grid) / 2 + 4 * P * n * n) + 8.0 * L * grid ** 2 / 2 * frames + extra}


def _margin(case):
    top = HEIGHTS[case["layers"] - 1] / math.cos(math.radians(ZENITH))
    return math.ceil(top * math.tan(case["field"] * ARCSEC) / (DIAMETER / case["n"]))


# ------------------------------------------------------------------ the same in float64


def exact(case, seed):
    return {"screens": _exact_screens, "sample": _exact_sample, "window": _exact_window, "pointings": _exact_pointings,
            "boiling": _exact_boiling, "laser": _exact_laser, "extrude": _exact_extrude, "rows": _exact_rows,
            "fit_screens": _exact_fit_screens, "fit_spectra": _exact_fit_spectra}[case["kind"]](case, seed)


def _t(x):
    return torch.as_tensor(np.asarray(x), device=DEVICE)


def _philox(index, call, domain, key):
    """Philox4x32-10 (Salmon et al., SC'11): the four words of each counter."""
    mask = 0xFFFFFFFF
    x = [index & mask, (index >> 32) & mask, torch.full_like(index, call & mask),
         torch.full_like(index, ((call >> 32) & 0xFFFFFF) | (domain << 24))]
    k0, k1 = key & mask, (key >> 32) & mask
    for _ in range(10):
        p0, p1 = x[0] * 0xD2511F53, x[2] * 0xCD9E8D57  # the low 64 bits; their upper words by a masked shift
        x = [((p1 >> 32) & mask) ^ x[1] ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ x[3] ^ k1, p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return x


def _normals(a, b):
    """Box-Muller on the top 24 bits of two words."""
    r = torch.sqrt(-2.0 * torch.log(((a >> 8).double() + 1.0) / 2 ** 24))
    angle = 2.0 * math.pi * ((b >> 8).double() / 2 ** 24 - 0.5)
    return torch.complex(-r * torch.cos(angle), -r * torch.sin(angle))


def _noise(index, call, domain, key):
    words = _philox(index, call, domain, key)
    return _normals(words[0], words[1]), _normals(words[2], words[3])


def _key(seed):
    state = np.random.SeedSequence(int(seed)).generate_state(2, dtype=np.uint32)
    return int(state[0]) | (int(state[1]) << 32)


def _psd(f2, r0):
    return 0.023 * r0 ** (-5.0 / 3.0) * (f2 + L0 ** -2) ** (-11.0 / 6.0)


def _band(fx, fy, width, r0):
    """The amplitude of a mode that stands for a cell of frequencies."""
    o = ((np.arange(33) + 0.5) / 33 - 0.5) * width
    f2 = (fx + o[:, None]) ** 2 + (fy + o[None, :]) ** 2
    p = _psd(f2, r0)
    return math.sqrt(p.mean() * width ** 2 * (p * f2).sum() / p.sum() / (fx ** 2 + fy ** 2))


def _amplitudes(n, dx, r0, P):
    """The von Karman filter (n, n), the level frequencies (P, 3) and amplitudes (P, 3, 3)."""
    df, f = 1.0 / (n * dx), np.fft.fftfreq(n, d=dx)
    f2 = f[:, None] ** 2 + f[None, :] ** 2
    f2[0, 0] = 1.0
    amp = np.sqrt(_psd(f2, r0)) * df
    amp[0, 0] = 0.0
    near = min(8, (n - 1) // 2)
    for i in range(-near, near + 1):
        for j in range(-near, near + 1):
            if i or j:
                amp[i, j] = _band(f[i], f[j], df, r0)
    freqs, low = np.zeros((P, 3)), np.zeros((P, 3, 3))
    for p in range(P):
        width = df / 3.0 ** (p + 1)
        freqs[p] = np.array([-1.0, 0.0, 1.0]) * width
        for i in range(3):
            for j in range(3):
                if i != 1 or j != 1:
                    low[p, i, j] = _band(freqs[p, i], freqs[p, j], width, r0)
    return _t(amp), freqs, _t(low)


def _low_order(coef, freqs, n, dx):
    """Re sum coef b_i(x) b_j(y) less its mean, for coef (..., P, 3, 3)."""
    x = (np.arange(n) - n / 2.0) * dx
    basis = _t(np.exp(2j * np.pi * np.asarray(freqs)[:, :, None] * x))  # (P, 3, n)
    s = torch.einsum("...pij,pix,pjy->...xy", coef, basis, basis).real
    return s - s.mean(dim=(-2, -1), keepdim=True)


def _draw_screens(n, dx, r0, P, count, key, call):
    amp, freqs, low = _amplitudes(n, dx, r0, P)
    pairs, half = (count + 1) // 2, (n + 1) // 2
    rows = torch.arange(pairs * n, device=DEVICE).reshape(pairs, n, 1)
    first, second = _noise(rows * half + torch.arange(half, device=DEVICE), call, 0x11, key)
    z = torch.cat([first, second[..., :n - half]], dim=-1) * amp
    x = torch.fft.ifft2(z) * (n * n)
    out = torch.cat([x.real, x.imag])[:count]
    gc, p, ij = (torch.arange(k, device=DEVICE) for k in (count, P, 9))
    z, _ = _noise((gc[:, None, None] * 16 + p[:, None]) * 9 + ij, call, 0x22, key)
    return out + _low_order(z.reshape(count, P, 3, 3) * low, freqs, n, dx)


def _exact_screens(case, seed):
    return _draw_screens(case["n"], DIAMETER / 256, 0.15, case["levels"], case["count"], _key(seed), 0)


def _r0_line_of_sight():
    return R0 * math.cos(math.radians(ZENITH)) ** 0.6


def _exact_sample(case, seed):
    # the spawn order of Atmosphere: the layers, two boiling streams, one stream for the one outer scale
    master = np.random.SeedSequence(seed)
    master.spawn(case["layers"] + 2)
    key = _key(master.spawn(1)[0].generate_state(1)[0])
    n = case["n"]
    screens = _draw_screens(n, DIAMETER / n, _r0_line_of_sight(), case["levels"], case["count"], key, 1)
    return screens * (WAVELENGTH / (2.0 * math.pi))


def _realisation(atm):
    """The layer spectra (L, ns, ns) and level coefficients (P, L, 3, 3) that an atmosphere holds."""
    spec = atm._spec
    return (torch.view_as_complex(spec.spectra).to(torch.complex128),
            torch.view_as_complex(spec.sh_coef).to(torch.complex128)[:spec.P])


def _phases(n, dx, shift):
    return torch.exp(2j * math.pi * torch.fft.fftfreq(n, d=dx, device=DEVICE, dtype=torch.float64) * shift[..., None])


def _moved(spectra, low, shifts, n, dx, P, per_layer=False):
    """Frames (F, n, n) of the spectra moved by shifts (F, L, 2); (F, L, n, n) per layer."""
    freqs = np.stack([np.array([-1.0, 0.0, 1.0]) / (n * dx) / 3.0 ** (p + 1) for p in range(P)])
    out = []
    for s in _t(shifts).split(8):
        px, py = _phases(n, dx, s[..., 0]), _phases(n, dx, s[..., 1])
        x = 0.0 if not per_layer else []
        for l in range(spectra.shape[0]):
            term = spectra[l] * px[:, l, :, None] * py[:, l, None, :]
            x = x + term if not per_layer else x + [term]
        x = torch.stack(x, dim=1) if per_layer else x
        fr = _t(freqs)
        ex = torch.exp(2j * math.pi * s[:, :, 0, None, None] * fr)[..., :, None]
        ey = torch.exp(2j * math.pi * s[:, :, 1, None, None] * fr)[..., None, :]
        c = low.permute(1, 0, 2, 3) * ex * ey  # (F, L, P, 3, 3)
        out.append(torch.fft.ifft2(x).real * (n * n) + _low_order(c if per_layer else c.sum(1), freqs, n, dx))
    return torch.cat(out)


def _to_opd(phase):
    return phase * (WAVELENGTH / (2.0 * math.pi))


def _exact_window(case, seed):
    atm = prepare(case, seed)["loop"].atm
    times = _start_time(seed) + DT * np.arange(case["steps"])
    shifts = times[:, None, None] * _winds(case["layers"])[0]
    return _to_opd(_moved(*_realisation(atm), shifts, case["n"], DIAMETER / case["n"], case["levels"]))


def _exact_pointings(case, seed):
    state = prepare(case, seed)
    n, m = case["n"], _margin(case)
    height = np.asarray(HEIGHTS[:case["layers"]]) / math.cos(math.radians(ZENITH))
    tangents = np.tan(np.asarray(state["stars"]) * ARCSEC)
    shifts = state["t"] * _winds(case["layers"])[0] + height[:, None] * tangents[:, None, :]
    frames = _moved(*_realisation(state["atm"]), shifts, n + 2 * m, DIAMETER / n, case["levels"])
    return _to_opd(frames[:, m:m + n, m:m + n])


def _exact_boiling(case, seed):
    atm = prepare(case, seed)["atm"]
    n, L, P = case["n"], case["layers"], case["levels"]
    dx = DIAMETER / n
    spectra, low = _realisation(atm)
    master = np.random.SeedSequence(seed)
    master.spawn(L)
    key = _key(master.spawn(1)[0].generate_state(1)[0])
    amp, freqs, low_amp = _amplitudes(n, dx, _r0_line_of_sight(), P)
    per_layer = _t(_fractions(L) ** 0.5)  # r0^(-5/6) of a layer of that fraction

    def decay(f):
        return torch.exp(-DT / (0.05 * torch.clamp(_t(f) * L0, min=1.0) ** (-2.0 / 3.0)))

    f = np.fft.fftfreq(n, d=dx)
    a, a_low = decay(np.hypot(f[:, None], f[None, :])), decay(np.hypot(freqs[:, :, None], freqs[:, None, :]))[:, None]
    amp, low_amp = amp * per_layer[:, None, None], low_amp[:, None] * per_layer[None, :, None, None]
    out = []
    for k in range(case["steps"]):
        z, _ = _noise(torch.arange(L * n * n, device=DEVICE), k, 0x66, key)
        spectra = a * spectra + torch.sqrt(1.0 - a * a) * z.reshape(L, n, n) * amp
        z, _ = _noise((1 << 40) + torch.arange(P * L * 9, device=DEVICE), k, 0x66, key)
        low = a_low * low + torch.sqrt(1.0 - a_low * a_low) * z.reshape(P, L, 3, 3) * low_amp
        shifts = (k + 1) * DT * _winds(L)[0][None]
        out.append(_to_opd(_moved(spectra, low, shifts, n, dx, P)[0]))
    return out


def _taps(t, interp):
    """Offsets and weights of an interpolation at the fractions t."""
    if interp == "linear":
        return (0, 1), (1.0 - t, t)
    if interp == "cubic":
        return (-1, 0, 1, 2), (0.5 * (-t + 2 * t ** 2 - t ** 3), 0.5 * (2 - 5 * t ** 2 + 3 * t ** 3),
                               0.5 * (t + 4 * t ** 2 - 3 * t ** 3), 0.5 * (t ** 3 - t ** 2))
    offsets = tuple(range(-2, 4))
    raw = [torch.sinc(t - o) * torch.sinc((t - o) / 3.0) for o in offsets]
    return offsets, [r / sum(raw) for r in raw]


def _exact_laser(case, seed):
    state = prepare(case, seed)
    n, L = case["n"], case["layers"]
    shifts = (state["t"] * _winds(L)[0])[None]
    layers = _moved(*_realisation(state["atm"]), shifts, n, DIAMETER / n, case["levels"], per_layer=True)[0]
    out = 0.0
    for l in range(L):
        pos = (n - 1) / 2.0 + (torch.arange(n, device=DEVICE, dtype=torch.float64) - (n - 1) / 2.0) * (1.0 - HEIGHTS[l] / 90e3)
        offsets, weights = _taps(pos - pos.floor(), case["interp"])
        take = [(pos.floor().long() + o).clamp(0, n - 1) for o in offsets]
        rows = sum(w[:, None] * layers[l][i] for w, i in zip(weights, take))
        out = out + sum(w * rows[:, i] for w, i in zip(weights, take))
    return _to_opd(out)


def _extend(rows, operator, count, sparse, key, scale):
    """More rows of one screen: [A | B] on the two newest rows, the sparse points and the row's noise."""
    rows = [r for r in rows.double()]
    W = rows[0].numel()
    for _ in range(count):
        top = len(rows)
        index = torch.arange((W + 1) // 2, device=DEVICE)
        z, _ = _noise(index, top, 0x55, key)
        beta = torch.view_as_real(z).reshape(-1)[:W] * scale
        points = [torch.stack([rows[top - d][c] for d, c in sparse])] if sparse else []
        rows.append(operator @ torch.cat([rows[top - 2], rows[top - 1], *points, beta]))
    return torch.stack(rows)


def _plain_form(operator, W, sparse):
    """The operator on the rows themselves, from the one on their differences that gives an increment."""
    m = operator.clone()
    eye = torch.eye(W, dtype=m.dtype, device=DEVICE)
    m[:, W:2 * W] = operator[:, W:2 * W] - operator[:, :W] + eye
    for k, (_, c) in enumerate(sparse):
        m[:, W + c] -= operator[:, 2 * W + k]
    return m


def _exact_rows(case, seed):
    state = prepare(case, seed)
    ring, W, steps = state["ring"], case["width"], case["steps"]
    operator = _plain_form(state["operator"], W, state["sparse"]) if case["form"] == "bf16x3" else state["operator"]
    start = int(ring.top[0])
    rows = ring.buf[:, :start].double()
    for k in range(steps):
        top = start + k
        noise = [torch.view_as_real(_noise(torch.arange((W + 1) // 2, device=DEVICE), top, 0x55, st.key)[0]).reshape(-1)[:W] * b
                 for st, b in zip(ring.streams, ring.bscale)]
        points = [rows[:, top - d, c][:, None] for d, c in state["sparse"]]
        x = torch.cat([rows[:, top - 2], rows[:, top - 1], *points, torch.stack(noise)], dim=1)
        rows = torch.cat([rows, (x @ operator.T)[:, None]], dim=1)
    return rows[:, start:]


def _exact_extrude(case, seed):
    atm = prepare(case, seed)["atm"]
    ring, n, dx = atm._ext._ring, case["n"], DIAMETER / case["n"]
    W, half = ring.W, (n - 1) / 2.0
    winds, _, _ = _winds(case["layers"])
    g = torch.arange(n, device=DEVICE, dtype=torch.float64) - half
    out = [0.0] * case["steps"]
    for l, (vx, vy) in enumerate(winds):
        speed = math.hypot(vx, vy)
        c, s = vx / speed, vy / speed
        reach = half * (abs(c) + abs(s))
        base = math.floor(-reach) - 2
        travel = [speed * k * DT / dx for k in range(case["steps"])]
        last = math.ceil(reach + travel[-1]) + 2 - base
        held = int(ring.top[l])
        rows = _extend(ring.buf[l, :held], ring.M[ring.groups[l]].double(), max(0, last + 1 - held), [],
                       ring.streams[l].key, ring.bscale[l])
        for k in range(case["steps"]):
            r = g[:, None] * c + g[None, :] * s + travel[k] - base
            q = -g[:, None] * s + g[None, :] * c + W / 2.0
            offsets, wr = _taps(r - r.floor(), case["interp"])
            _, wq = _taps(q - q.floor(), case["interp"])
            for a, u in zip(offsets, wr):
                i = (r.floor().long() + a).clamp(0, len(rows) - 1)
                for b, v in zip(offsets, wq):
                    out[k] = out[k] + u * v * rows[i, (q.floor().long() + b).clamp(0, W - 1)]
    return [_to_opd(x) for x in out]


def _leaves(state, *names):
    return [state[k].detach().to(torch.complex128 if state[k].is_complex() else torch.float64).requires_grad_(True) for k in names]


def _exact_fit_screens(case, seed):
    state = prepare(case, seed)
    names = ("screens", "weights", "winds")
    screens, weights, winds = leaves = _leaves(state, *names)
    n, S, dx = case["n"], case["size"], DIAMETER / case["n"]
    grid = torch.arange(n, device=DEVICE, dtype=torch.float64)
    grads = [torch.zeros_like(x) for x in leaves]
    total = 0.0
    scale = 1.0 / state["target"].numel()
    for t in range(case["times"]):
        for d, star in enumerate(state["stars"]):
            image = 0.0
            for l, h in enumerate(HEIGHTS[:case["layers"]]):
                mag = 1.0 - h / 90e3 if d == case["stars"] else 1.0
                shift = winds[l] * (state["t"] + DT * t) + h * _t(star)
                layer = screens[:, l]
                for axis in (0, 1):
                    u = (S - 1) / 2.0 - mag * (n - 1) / 2.0 + shift[axis] / dx + mag * grid
                    i, f = u.detach().floor().long(), u - u.detach().floor()
                    f = f[:, None] if axis == 0 else f
                    lo, hi = layer.index_select(axis + 1, i % S), layer.index_select(axis + 1, (i + 1) % S)
                    layer = lo + f * (hi - lo)
                image = image + weights[l] * layer
            part = ((image - state["target"][:, t, d].double()) ** 2).sum() * scale
            for g, x in zip(grads, torch.autograd.grad(part, leaves)):
                g += x
            total = total + part.detach()
    return {"loss": total, **dict(zip(names, grads))}


def _exact_fit_spectra(case, seed):
    state = prepare(case, seed)
    names = ("noise", "weights", "winds", "low")
    noise, weights, winds, low = leaves = _leaves(state, *names)
    n, S, L, P, dx = case["n"], case["size"], case["layers"], case["levels"], DIAMETER / case["n"]
    c = (S - n) // 2
    amp, freqs, low_amp = _amplitudes(S, dx, R0, P)
    loss = 0.0
    grads = [torch.zeros_like(x) for x in leaves]
    for k in range(case["times"]):
        shift = winds * (state["t"] + DT * k)
        x = sum(weights[l] * noise[l] * amp * _phases(S, dx, shift[l, 0])[:, None] * _phases(S, dx, shift[l, 1]) for l in range(L))
        fr = _t(freqs)
        ex = torch.exp(2j * math.pi * shift[:, 0, None, None] * fr)[..., :, None]
        ey = torch.exp(2j * math.pi * shift[:, 1, None, None] * fr)[..., None, :]
        coef = (weights[:, None, None, None] * low * low_amp * ex * ey).sum(0)
        frame = torch.fft.ifft2(x).real * (S * S) + _low_order(coef, freqs, S, dx)
        part = ((frame[c:c + n, c:c + n] - state["target"][k].double()) ** 2).sum() / state["target"].numel()
        for g, y in zip(grads, torch.autograd.grad(part, leaves)):
            g += y
        loss = loss + part.detach()
    return {"loss": loss, **dict(zip(names, grads))}
