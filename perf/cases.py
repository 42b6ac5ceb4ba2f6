"""The work a user of the framework has it do, as timed cases.

Each case is one call (or one short sequence of calls) through the public entry points:
``Integrator`` in its three precisions, from the grids of the golden fixtures to the headline grid;
``Ensemble``; the analysis of a sampled field; the currents of a state; and the learned stepper,
its network's training pass and its macro steps. Fields are near-uniform states phi0 + noise or
states that have separated a little, as runs meet them.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "active-model-bplus_gb300"))

DT = 1e-3
AMBP = dict(a=-0.25, b=0.0, c=0.25, kappa=1.0, lamb=-1.0, zeta=-4.0)   # the noisy AMB+ configuration
MODEL_B = dict(a=-0.25, b=0.0, c=0.25, kappa=1.0, lamb=0.0, zeta=0.0)  # the passive spinodal configuration
HEADLINE = dict(a=-0.25, b=0.0, c=0.25, kappa=1.0, lamb=0.5, zeta=-1.0)
PARAMS = {"ambp": AMBP, "model_b": MODEL_B, "headline": HEADLINE}
K_MACRO = 50


def listed():
    return [
        # the reference's precision on the small active grid of the golden fixtures: latency counts
        dict(name="f64 64", kind="step", precision="f64", ny=64, nx=64, params="ambp", T=0.05, steps=100),
        # the deterministic spinodal of the parity configuration
        dict(name="f64 256 T0", kind="step", precision="f64", ny=256, nx=256, params="model_b", T=0.0, steps=100),
        # a noisy grid whose sides suit no tile and no quad
        dict(name="f64 odd", kind="step", precision="f64", ny=701, nx=907, params="ambp", T=0.05, steps=20),
        # a production run in the default precision
        dict(name="f64 2048", kind="step", precision="f64", ny=2048, nx=2048, params="ambp", T=0.05, steps=10),
        # compensated FP32 on a small ragged grid
        dict(name="f32c odd", kind="step", precision="f32c", ny=250, nx=333, params="ambp", T=0.05, steps=100),
        # the single-field run that the learned stepper is compared with
        dict(name="f32c 512", kind="step", precision="f32c", ny=512, nx=512, params="ambp", T=0.05, steps=100),
        # the headline grid
        dict(name="f32c 4096", kind="step", precision="f32c", ny=4096, nx=4096, params="headline", T=0.05, steps=50),
        # a parameter sweep: replicas of uneven sizes and parameters
        dict(name="ensemble", kind="ensemble", replicas=32, lo=128, hi=1024, steps=64),
        # S(k) and droplets of a sampled field
        dict(name="analysis 1024", kind="analysis", ny=1024, nx=1024, precision="f64"),
        # sampling the currents along a run
        dict(name="currents 512", kind="currents", ny=512, nx=512, precision="f64", steps=10),
        # one training iteration's passes of the flux network on 128^2 pairs
        dict(name="train 16x128", kind="train", batch=16, ny=128, nx=128),
        # macro steps of the learned stepper with their residual check
        dict(name="learned 512", kind="learned", ny=512, nx=512, macro=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["f64", "f64", "f32", "f32", "ensemble", "analysis", "currents", "train", "learned"])
    if kind == "f64":
        ny, nx = _log(rng, 48, 2048), _log(rng, 48, 2048)
        return dict(kind="step", precision="f64", ny=ny, nx=nx, params=rng.choice(["ambp", "model_b", "headline"]),
                    T=rng.choice([0.0, 0.05]), steps=max(10, min(100, (1 << 22) * 10 // (ny * nx))))
    if kind == "f32":
        ny, nx = _log(rng, 64, 4096), _log(rng, 64, 4096)
        if rng.random() < 0.6:
            nx = max(64, nx // 4 * 4)
        return dict(kind="step", precision=rng.choice(["f32", "f32c"]), ny=ny, nx=nx,
                    params=rng.choice(["ambp", "headline"]), T=rng.choice([0.0, 0.05]),
                    steps=max(20, min(100, (1 << 24) * 20 // (ny * nx))))
    if kind == "ensemble":
        lo = rng.choice([128, 192, 256])
        return dict(kind="ensemble", replicas=_log(rng, 3, 16), lo=lo, hi=rng.choice([lo, 512, 1024]),
                    steps=rng.choice([64, 100]))
    if kind == "analysis":
        return dict(kind="analysis", ny=_log(rng, 96, 2048), nx=_log(rng, 96, 2048), precision=rng.choice(["f64", "f32c"]))
    if kind == "currents":
        return dict(kind="currents", ny=_log(rng, 64, 1024), nx=_log(rng, 64, 1024), precision=rng.choice(["f64", "f32c"]),
                    steps=10)
    if kind == "train":
        ny, nx = rng.choice([(128, 128), (96, 128), (130, 256)])
        return dict(kind="train", batch=rng.randint(2, (16 << 14) // (ny * nx)), ny=ny, nx=nx)
    ny, nx = _log(rng, 96, 768), 128 * rng.randint(1, 6)
    return dict(kind="learned", ny=ny, nx=nx, macro=min(rng.choice([10, 40]), (40 << 18) // (ny * nx)))


# ------------------------------------------------------------------ inputs

def _normal(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)


def _field(ny, nx, seed, phi0=-0.4, amp=0.01):
    return (phi0 + amp * _normal((ny, nx), seed)).cpu().numpy()


def _separated(ny, nx, seed):
    """A field with droplets some ten sites wide in the two bulk phases."""
    ky = 2 * math.pi * torch.fft.fftfreq(ny, dtype=torch.float64, device="cuda")[:, None]
    kx = 2 * math.pi * torch.fft.rfftfreq(nx, dtype=torch.float64, device="cuda")[None, :]
    k2 = kx * kx + ky * ky
    s = torch.fft.irfft2(torch.fft.rfft2(_normal((ny, nx), seed)) * k2 * torch.exp(-8.0 * k2), s=(ny, nx))
    return torch.tanh(2.0 * (s / s.std() - 0.6)) + 0.05 * _normal((ny, nx), seed + 1)


def _model(case):
    from activemodelbplus.integrator import Model
    return Model(T=case["T"], **PARAMS[case["params"]])


def _stencil():
    from activemodelbplus.integrator import Stencil
    return Stencil(dt=DT, dx=1.0, dy=1.0)


def _replicas(case, seed):
    """The replicas' shapes (the case's alone) and their parameters (the seed's)."""
    shapes, rng = np.random.default_rng(case["replicas"]), np.random.default_rng(seed)
    sides = sorted({s for s in (128, 192, 256, 384, 512, 768, 1024) if case["lo"] <= s <= case["hi"]} | {case["lo"]})
    reps = []
    for _ in range(case["replicas"]):
        ny, nx = (int(s) for s in shapes.choice(sides, 2))
        reps.append(dict(ny=ny, nx=nx, a=-0.25, b=0.0, c=0.25, kappa=1.0, lamb=float(rng.uniform(-1, 1)),
                         zeta=float(rng.uniform(-4, 4)), T=float(rng.uniform(0.01, 0.1)), phi0=float(rng.uniform(-0.6, 0.6)),
                         seed=int(rng.integers(1 << 62))))
    return reps


def _weights():
    import activemodelbplus
    return os.path.join(os.path.dirname(activemodelbplus.__file__), "weights", "fluxnet_k50.npz")


def _train_inputs(case, seed):
    B, ny, nx = case["batch"], case["ny"], case["nx"]
    phi = torch.stack([_separated(ny, nx, 1000 * seed + 7 * b) for b in range(B)]).float()
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand((B, 3), device="cuda", generator=g)
    params = torch.stack([8 * u[:, 0] - 4, 2 * u[:, 1] - 1, 0.1 * u[:, 2]], dim=1).contiguous()
    dflux = 1e-3 * torch.randn((B, 2, ny, nx), device="cuda", generator=g)
    return phi, params, dflux


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        from activemodelbplus.integrator import Integrator
        return dict(case=case, sim=Integrator(_field(case["ny"], case["nx"], seed), _stencil(), _model(case),
                                              precision=case["precision"], seed=seed))
    if kind == "ensemble":
        from activemodelbplus.integrator import Ensemble, Model
        reps = _replicas(case, seed)
        models = [Model(**{k: r[k] for k in ("a", "b", "c", "kappa", "lamb", "zeta", "T")}) for r in reps]
        fields = [_field(r["ny"], r["nx"], seed + i, r["phi0"]) for i, r in enumerate(reps)]
        return dict(case=case, ens=Ensemble(fields, _stencil(), models, precision="f32c", seeds=[r["seed"] for r in reps]))
    if kind == "analysis":
        f = _separated(case["ny"], case["nx"], seed)
        return dict(case=case, field=f if case["precision"] == "f64" else f.float())
    if kind == "currents":
        from activemodelbplus.integrator import Integrator, Model
        return dict(case=case, sim=Integrator(_separated(case["ny"], case["nx"], seed).cpu().numpy(), _stencil(),
                                              Model(T=0.05, **AMBP), precision=case["precision"], seed=seed))
    if kind == "train":
        from activemodelbplus.learned import FluxNet
        return dict(case=case, net=FluxNet.load(_weights()), inputs=_train_inputs(case, seed))
    from activemodelbplus.integrator import Model
    from activemodelbplus.learned import FluxNet, LearnedStepper
    return dict(case=case, st=LearnedStepper(FluxNet.load(_weights()), _field(case["ny"], case["nx"], seed), _stencil(),
                                             Model(T=0.05, **AMBP), K=K_MACRO, seed=seed, residual_sigma=2.0))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        sim = state["sim"]
        sim.run(case["steps"])
        return sim.field_tensor
    if kind == "ensemble":
        state["ens"].run(case["steps"])
        return state["ens"].gather()
    if kind == "analysis":
        from activemodelbplus import analysis
        k, S, counts = analysis.structure_factor(state["field"])
        labels, n = analysis.label_droplets(state["field"], 0.0)
        return [S, counts.astype(np.int64), labels, n]
    if kind == "currents":
        sim = state["sim"]
        sim.run(case["steps"])
        return [sim.current, sim.passive_current, sim.active_current]
    if kind == "train":
        from activemodelbplus.learned import network_input
        net, (phi, params, dflux) = state["net"], state["inputs"]
        net.refresh()  # the optimiser changed the weights
        flux = net.forward(network_input(phi, params), train=True)
        gw, gb = net.backward(dflux)
        return [flux, gw, gb]
    st = state["st"]
    st.advance(case["macro"])
    return st.phi_f


# ------------------------------------------------------------------ work

# Arithmetic operations of one site update that no arrangement saves: stage A 26, J2 and its
# divergence 18, the four order-8 derivatives 32, noise and update 5 (fused ones counted as two).
STEP_FLOPS = 110
NET_FLOPS = 2 * 25 * (5 * 32 + 4 * 32 * 32 + 32 * 2)  # per site, one evaluation


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        sites = sum(r["ny"] * r["nx"] for r in _replicas(case, 0))
    elif kind == "train":
        sites = case["batch"] * case["ny"] * case["nx"]
    else:
        sites = case["ny"] * case["nx"]
    if kind in ("step", "ensemble"):
        per = {"f64": 16, "f32": 8, "f32c": 12}[case.get("precision", "f32c")]
        return dict(bytes=sites * case["steps"] * per, flops=sites * case["steps"] * STEP_FLOPS)
    if kind == "analysis":
        return dict(bytes=sites * ({"f64": 8, "f32c": 4}[case["precision"]] + 4), flops=sites * 2.5 * math.log2(sites))
    if kind == "currents":
        return dict(bytes=sites * (16 * case["steps"] + 6 * 8), flops=sites * STEP_FLOPS * (case["steps"] + 1))
    if kind == "train":
        return dict(bytes=sites * 4 * 5, flops=3 * sites * NET_FLOPS)
    return dict(bytes=sites * case["macro"] * 12, flops=(case["macro"] + 1) * sites * NET_FLOPS)


# ------------------------------------------------------------------ the same in 64 bits

def _roll(f, dy, dx):
    """f at (row + dy, column + dx), periodic."""
    return torch.roll(f, (-dy, -dx), dims=(0, 1))


def _d8(f, axis):
    c = (4.0 / 5, -1.0 / 5, 4.0 / 105, -1.0 / 280)
    return sum(cj * (torch.roll(f, -(j + 1), dims=axis) - torch.roll(f, j + 1, dims=axis)) for j, cj in enumerate(c))


def _tj(f, axis):
    d = torch.roll(f, -1, dims=axis) - torch.roll(f, 1, dims=axis)
    return 0.1 * (torch.roll(d, 1, dims=1 - axis) + torch.roll(d, -1, dims=1 - axis)) + 0.3 * d


def _laplacian(f):
    def second(g, axis):
        return torch.roll(g, 1, dims=axis) - 2 * g + torch.roll(g, -1, dims=axis)

    def across(g, axis):
        return -0.25 * (torch.roll(g, 1, dims=axis) + torch.roll(g, -1, dims=axis)) + 1.5 * g
    return across(second(f, 1), 0) + across(second(f, 0), 1)


def _philox(c0, c1, c2, c3, key):
    """Philox4x32-10 of counters given as int64 tensors (or ints) of 32-bit words."""
    mask = 0xFFFFFFFF

    def mulhilo(m, x):
        lo16, hi16 = m * (x & 0xFFFF), m * (x >> 16)
        return (hi16 + (lo16 >> 16)) >> 16, (lo16 + ((hi16 & 0xFFFF) << 16)) & mask
    k0, k1 = key & mask, key >> 32
    for _ in range(10):
        h0, l0 = mulhilo(0xD2511F53, c0)
        h1, l1 = mulhilo(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c0, c1, c2, c3


def _box_muller(xa, xb):
    ua, ub = ((xa >> 8) + 1).double() * 2.0**-24, (xb >> 8).double() * 2.0**-24
    r, th = torch.sqrt(-2 * torch.log(ua)), 2 * math.pi * (ub - 0.5)
    return r * torch.cos(th), r * torch.sin(th)


def _noise(ny, nx, seed, step, comp):
    """The normals of one component at every site: one Philox call per four columns of a row."""
    nq = (nx + 3) // 4
    rows = torch.arange(ny, device="cuda")[:, None].expand(ny, nq)
    quads = torch.arange(nq, device="cuda")[None, :].expand(ny, nq)
    x = _philox(quads, rows, torch.full_like(rows, step & 0xFFFFFFFF), torch.full_like(rows, ((step >> 32) << 1) | comp), seed)
    z = _box_muller(x[0], x[1]) + _box_muller(x[2], x[3])
    return torch.stack(z, dim=2).reshape(ny, 4 * nq)[:, :nx]


def _terms(f, m, T, seed, step):
    lap, gy, gx = _laplacian(f), _tj(f, 0), _tj(f, 1)
    mup = ((m["c"] * f + m["b"]) * f + m["a"]) * f - m["kappa"] * lap
    mua = m["lamb"] * (gx * gx + gy * gy)
    out = []
    for comp, axis, g in ((0, 0, gy), (1, 1, gx)):
        jr = torch.zeros_like(f)
        if T > 0:
            jr = math.sqrt(2 * T / DT) * _noise(*f.shape, seed, step, comp)
        out.append(dict(p=-_d8(mup, axis), l=-_tj(mua, axis), c=m["zeta"] * lap * g, r=jr))
    return out


def _exact_steps(f, m, T, seed, steps, step0=0):
    f = torch.as_tensor(f, dtype=torch.float64, device="cuda")
    for s in range(step0, step0 + steps):
        y, x = _terms(f, m, T, seed, s)
        div = _d8(y["p"] + y["r"], 0) + _d8(x["p"] + x["r"], 1) + _tj(y["l"] + y["c"], 0) + _tj(x["l"] + x["c"], 1)
        f = f - DT * div
    return f


def _exact_spectrum(f):
    ny, nx = f.shape
    p = torch.fft.fft2(f - f.mean()).abs().square().cpu().numpy().ravel()
    ky = 2 * np.pi * np.fft.fftfreq(ny)[:, None]
    kx = 2 * np.pi * np.fft.fftfreq(nx)[None, :]
    edges = np.linspace(0, 3, 300)[1:]
    l = np.digitize(np.sqrt(kx * kx + ky * ky).ravel(), edges, right=True)
    s = np.bincount(l, weights=p, minlength=len(edges) + 1)[:len(edges) - 1]
    c = np.bincount(l, minlength=len(edges) + 1)[:len(edges) - 1]
    with np.errstate(invalid="ignore", divide="ignore"):
        return np.where(c > 0, s / np.maximum(c, 1), np.nan)


def _net_layers():
    z = np.load(_weights())
    n = sum(1 for k in z.files if k[:1] == "w" and k[1:].isdigit())
    as64 = lambda v: torch.from_numpy(v).double().cuda()  # noqa: E731
    return [as64(z[f"w{l}"]) for l in range(n)], [as64(z[f"b{l}"]) for l in range(n)]


def _net_forward(phi, params, ws, bs):
    """The flux network in 64 bits: phi [B, H, W], params [B, 3]."""
    hi = phi.bfloat16().double()
    p = (params.double() * torch.tensor([0.25, 1.0, 10.0], dtype=torch.float64, device="cuda"))[:, :, None, None]
    x = torch.cat([hi[:, None], 256 * (phi.double() - hi)[:, None], p.expand(-1, -1, *phi.shape[1:])], dim=1)
    for l, (w, b) in enumerate(zip(ws, bs)):
        x = torch.nn.functional.conv2d(torch.nn.functional.pad(x, (2, 2, 2, 2), mode="circular"), w, b[: w.shape[0]])
        if l < len(ws) - 1:
            x = torch.nn.functional.gelu(x, approximate="tanh")
    return x


def _exact_train(case, seed):
    phi, params, dflux = _train_inputs(case, seed)
    ws, bs = _net_layers()
    for v in ws + bs:
        v.requires_grad_(True)
    flux = []
    for b in range(case["batch"]):  # one sample at a time: the sums over samples are the accumulated gradients
        f = _net_forward(phi[b:b + 1], params[b:b + 1], ws, bs)
        f.backward(dflux[b:b + 1].double())
        flux.append(f.detach())
    return [torch.cat(flux), [w.grad for w in ws], [b.grad for b in bs]]


def _spectral_noise(ny, nx, seed, step):
    """The rfft2 spectra of two white-noise fields, drawn mode by mode."""
    nk = nx // 2 + 1
    r = torch.arange(ny, device="cuda")[:, None].expand(ny, nk)
    k = torch.arange(nk, device="cuda")[None, :].expand(ny, nk)
    herm = (k == 0) | ((k == nx // 2) if nx % 2 == 0 else torch.zeros_like(k, dtype=torch.bool))
    conj = herm & (r > ny // 2)
    rr = torch.where(conj, ny - r, r)
    x = _philox(k, rr, torch.full_like(r, step & 0xFFFFFFFF), torch.full_like(r, (step >> 32) << 1), seed ^ 0x5BD1E995A5A5A5A5)
    real = herm & ((rr == 0) | ((rr == ny // 2) if ny % 2 == 0 else torch.zeros_like(r, dtype=torch.bool)))
    out = []
    for z in (_box_muller(x[0], x[1]), _box_muller(x[2], x[3])):
        re = z[0] * math.sqrt(ny * nx) * torch.where(real, 1.0, math.sqrt(0.5))
        im = z[1] * math.sqrt(0.5 * ny * nx) * torch.where(real, 0.0, torch.where(conj, -1.0, 1.0).double())
        out.append(torch.complex(re, im))
    return out


def _exact_learned(case, seed):
    ny, nx = case["ny"], case["nx"]
    T, dtk = 0.05, K_MACRO * DT
    phi = torch.from_numpy(_field(ny, nx, seed)).cuda()
    ty = 2 * math.pi * torch.fft.fftfreq(ny, dtype=torch.float64, device="cuda")[:, None]
    tx = 2 * math.pi * torch.fft.rfftfreq(nx, dtype=torch.float64, device="cuda")[None, :]
    c = (4.0 / 5, -1.0 / 5, 4.0 / 105, -1.0 / 280)
    s2 = sum((2 * sum(cd * torch.sin((d + 1) * t) for d, cd in enumerate(c))) ** 2 for t in (tx, ty))
    lap = (1.5 - 0.5 * torch.cos(ty)) * (2 * torch.cos(tx) - 2) + (1.5 - 0.5 * torch.cos(tx)) * (2 * torch.cos(ty) - 2)
    a = 1 - DT * s2 * (-2 * AMBP["a"] - AMBP["kappa"] * lap)
    d = [1 - torch.exp(-1j * ty), 1 - torch.exp(-1j * tx)]
    den = d[0].abs() ** 2 + d[1].abs() ** 2
    den[0, 0] = 1.0
    om = 1 - a * a
    g = torch.sqrt(torch.where(om.abs() > 1e-12, (1 - a ** (2 * K_MACRO)) / (K_MACRO * om), 1.0).clamp(min=0))
    w8 = [sum(c[q - 1] for q in range(max(e, 1 - e), 5)) for e in range(-3, 5)]
    face = [g * sum(w * torch.exp(1j * t * e) for w, e in zip(w8, range(-3, 5))) for t in (ty, tx)]
    linear = [-(a ** K_MACRO - 1) * di.conj() / den / dtk for di in d]
    ws, bs = _net_layers()
    params = torch.tensor([[AMBP["zeta"], AMBP["lamb"], T]], dtype=torch.float64, device="cuda")
    with torch.no_grad():
        for n in range(case["macro"]):
            spec, xi = torch.fft.rfft2(phi), _spectral_noise(ny, nx, seed, n)
            fy, fx = (torch.fft.irfft2(spec * l + math.sqrt(2 * T / dtk) * z * w, s=(ny, nx)) + f
                      for l, z, w, f in zip(linear, xi, face, _net_forward(phi[None], params, ws, bs)[0]))
            phi = phi - dtk * ((fx - torch.roll(fx, 1, dims=1)) + (fy - torch.roll(fy, 1, dims=0)))
    return phi


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        if case["ny"] * case["nx"] * case["steps"] > 1 << 30:
            return None
        return _exact_steps(_field(case["ny"], case["nx"], seed), PARAMS[case["params"]], case["T"], seed, case["steps"])
    if kind == "ensemble":
        return torch.cat([_exact_steps(_field(r["ny"], r["nx"], seed + i, r["phi0"]), r, r["T"], r["seed"], case["steps"]).ravel()
                          for i, r in enumerate(_replicas(case, seed))])
    if kind == "analysis":
        f = _separated(case["ny"], case["nx"], seed)
        return [_exact_spectrum(f if case["precision"] == "f64" else f.float().double()), None, None, None]
    if kind == "currents":
        f = _exact_steps(_separated(case["ny"], case["nx"], seed), AMBP, 0.05, seed, case["steps"])
        t = _terms(f, AMBP, 0.05, seed, case["steps"])
        return [[v["c"] + v["l"] + v["p"] + v["r"] for v in t], [v["p"] for v in t], [v["c"] + v["l"] for v in t]]
    if kind == "train":
        return _exact_train(case, seed)
    return _exact_learned(case, seed)
