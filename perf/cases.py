"""Performance cases of the encode and decode path.

Each case is one call (or the few calls that a program always makes together)
through the public Python classes, on inputs of the kind the path meets: a
Dirichlet-bandlimited video seen through Gabor and centre-surround receptive
fields, and the spike trains of ideal integrate-and-fire neurons driven by it.
All inputs are made with numpy and torch alone, from the seed alone.

Kinds of work:

  project      vrf_bank.filter: the video projected on every receptive field
  iaf          IAF_encode.encode_blocks and the pairing of its spikes
  prep         prep_from_banks: Dirichlet coefficients, spatial functions and
               cross-weights of a decoder's receptive fields
  gram         dirichlet.compute_q and compute_G: the n x n spike Gram
  reconstruct  dirichlet.reconstruct: the video from the spike weights
  plain        one whole window of the plain float64 decoder
  decode       CoeffDecoder.decode: one whole window in the coefficient space
  rnn          CoeffDecoder.rnn_coefficients and synthesize: the gradient-flow decoder
  rnn3         neural_network.rnn3 on the n x n Gram
  batch        BatchDecoder.run: uneven clips decoded together

Windows are at least one temporal period long and hold more spike intervals
than there are coefficients, so that no eigenvalue lies at the
pseudoinverse's truncation threshold and every output is well determined.
"""
import math

import numpy as np
import torch

DEV = "cuda"
F64 = torch.float64
C128 = torch.complex128
WT = 2 * math.pi * 20.0        # temporal bandwidth of every workload, rad/s
DT = 1e-4                      # sample spacing of every workload, s
KAPPA = 2.5                    # Gabor modulation
SIGMA_C, SIGMA_S = 0.05, 0.15  # centre and surround widths


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the small configuration's encoder: 32x32, 0.2 s, 128 receptive fields; bound by latency
        {"name": "project_small", "kind": "project", "side": 32, "frames": 2000, "neurons": 128, "precision": "f64",
         "layout": "neuron", "video": "float64"},
        # the GPU configuration's encoder in the reference's precision: 64x64, 1 s, 1024 receptive fields
        {"name": "project_gpu", "kind": "project", "side": 64, "frames": 10000, "neurons": 1024, "precision": "f64",
         "layout": "neuron", "video": "float64"},
        # a served clip's projection on the tensor cores: float32 video, odd frame and neuron counts
        {"name": "project_served", "kind": "project", "side": 48, "frames": 4999, "neurons": 777,
         "precision": "bf16x3", "layout": "neuron", "video": "float32"},
        # the GPU configuration's spike encoding: 1024 neurons, 1 s
        {"name": "iaf_gpu", "kind": "iaf", "neurons": 1024, "frames": 10000, "Mt": 8, "delta": 0.12},
        # preparing a decoder for the GPU configuration's receptive fields
        {"name": "prep_gpu", "kind": "prep", "side": 64, "M": 6, "neurons": 1024},
        # the plain decoder's Gram at the size the reference states it can hold, 25k spikes
        {"name": "gram_gpu", "kind": "gram", "side": 64, "M": 6, "Mt": 8, "neurons": 1024, "samples": 10000,
         "delta": 0.12, "intervals": 24001},
        # the plain decoder's synthesis at the GPU configuration
        {"name": "reconstruct_gpu", "kind": "reconstruct", "side": 64, "M": 6, "Mt": 8, "neurons": 1024,
         "samples": 10000, "delta": 0.12},
        # one whole window of the plain decoder at the small configuration
        {"name": "plain_small", "kind": "plain", "side": 32, "M": 3, "Mt": 4, "neurons": 128, "samples": 2000,
         "delta": 0.04},
        # one whole window of the mixed-precision decoder at the GPU configuration: the headline decode
        {"name": "mixed_gpu", "kind": "decode", "solver": "mixed", "side": 64, "M": 6, "Mt": 8, "neurons": 1024,
         "samples": 10000, "delta": 0.12, "out": "float64"},
        # the float64 decoder (the default solver) on a clip of the batch's ranges, ragged sizes
        {"name": "float64_clip", "kind": "decode", "solver": "auto", "side": 48, "M": 5, "Mt": 6, "neurons": 701,
         "samples": 4501, "delta": 0.075, "out": "float64"},
        # the gradient-flow decoder at the GPU configuration: 2000 steps at 1 / lambda_max
        {"name": "rnn_gpu", "kind": "rnn", "side": 64, "M": 6, "Mt": 8, "neurons": 1024, "samples": 10000,
         "delta": 0.12, "steps": 2000},
        # twelve clips of uneven size decoded together, three refinement sweeps
        {"name": "batch_12", "kind": "batch", "clips": 12, "sizes": 2, "sweeps": 3},
    ]


def draw(rng):
    kind = rng.choice(["project", "project", "iaf", "prep", "gram", "reconstruct", "plain", "decode", "decode",
                       "decode", "rnn", "rnn3", "batch"])
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if kind == "project":
        prec = rng.choice(["f64", "f64", "bf16x3"])
        return {"kind": kind, "side": rng.choice([16, 25, 32, 48, 64]), "frames": log(101, 10000),
                "neurons": log(32, 1024), "precision": prec, "layout": rng.choice(["neuron", "neuron", "time"]),
                "video": rng.choice(["float64", "float32"])}
    if kind == "iaf":
        return {"kind": kind, "neurons": log(32, 1024), "frames": log(500, 10000), "Mt": rng.randint(3, 8),
                "delta": rng.choice([0.04, 0.075, 0.12])}
    if kind == "batch":
        return {"kind": kind, "clips": rng.randint(4, 12), "sizes": rng.randint(3, 1 << 30), "sweeps": 3}
    M = rng.randint(2, 6)
    side = rng.choice([16, 32, 48, 64])
    if kind == "prep":
        return {"kind": kind, "side": side, "M": M, "neurons": log(32, 1024)}
    Mt = rng.randint(3, 8)
    if kind in ("plain", "rnn3"):
        M, Mt = rng.randint(2, 3), rng.randint(3, 4)
    period = Mt / 20.0 / DT                     # samples in one temporal period
    samples = int(rng.uniform(1.1 * period, max(1.3 * period, 5000 if kind not in ("plain", "rnn3") else 2000)))
    delta = 0.04 if kind in ("plain", "rnn3") else 0.075
    per_neuron = 3.0 * samples * DT / delta     # spikes of one neuron
    K = ellipse(M).size * (2 * Mt + 1)
    low = max(48, int(2.5 * K / per_neuron), 3 * ellipse(M).size)
    c = {"kind": kind, "side": side, "M": M, "Mt": Mt, "neurons": log(low, max(low + 16, 160 if kind in (
        "plain", "rnn3") else 1000)), "samples": samples, "delta": delta}
    if kind == "decode":
        c["solver"] = rng.choice(["mixed", "mixed", "auto"])
        c["out"] = rng.choice(["float64", "float64", "float32"])
    if kind in ("rnn", "rnn3"):
        c["steps"] = log(200, 2000)
    if kind in ("gram", "rnn3"):
        c["intervals"] = int(0.9 * c["neurons"] * (per_neuron - 1))
    return c


# ------------------------------------------------------------------ inputs

def ellipse(M):
    """Flat indices of the spatial ellipse mx^2 + my^2 <= M^2 in the (2M+1) x (2M+1) coefficient grid."""
    m = np.arange(-M, M + 1)
    return np.nonzero((m[::-1, None] ** 2 + m[None, :] ** 2 <= M * M).reshape(-1))[0]


def fields(neurons, rng):
    """Receptive-field parameters: three quarters Gabor, one quarter centre-surround, near unit norm."""
    ng = max(1, 3 * neurons // 4)
    nc = neurons - ng
    g = {"h_alpha": rng.choice([0.05, 0.1, 0.2], ng), "h_l": rng.choice(8, ng) * math.pi / 8,
         "h_x0": rng.uniform(-0.5, 0.5, ng), "h_y0": rng.uniform(-0.5, 0.5, ng),
         "h_ab": (np.arange(ng) % 2).astype(np.int32), "h_gain": np.full(ng, math.sqrt(2.0))}
    c = {"h_alpha": np.ones(nc), "h_x0": rng.uniform(-0.5, 0.5, nc), "h_y0": rng.uniform(-0.5, 0.5, nc),
         "h_gain": np.full(nc, 0.2)}
    return g, c


def bank_objects(g, c, side, scale):
    """The framework's RF objects on the video grid (scale 1) or on a decoder's grid over one period (scale 4)."""
    from vtem_b200 import vrf
    px = side if scale == 1 else -(-side // 16) * 16
    banks = []
    gb = vrf.vrf_gabor((px, px), dx=1.0 / px, dy=1.0 / px, scale=scale)
    gb.load_parameters(num_neurons=len(g["h_alpha"]), KAPPA=KAPPA, **g)
    banks.append(gb)
    if len(c["h_alpha"]):
        cb = vrf.vrf_cs((px, px), dx=1.0 / px, dy=1.0 / px, scale=scale)
        cb.load_parameters(num_neurons=len(c["h_alpha"]), sigma_center=SIGMA_C, sigma_surround=SIGMA_S, **c)
        banks.append(cb)
    return banks


def field_values(g, c, px):
    """The receptive fields (neurons, px, px) on a px x px grid of the unit square, by their formulas."""
    t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=DEV)[:, None, None]
    x = (torch.arange(px, dtype=F64, device=DEV) * (1.0 / px) - 0.5)[None, None, :]
    y = -(torch.arange(px, dtype=F64, device=DEV) * (1.0 / px) - 0.5)[None, :, None]
    al = 1.0 / t(g["h_alpha"])
    xs, ys = al * (x - t(g["h_x0"])), al * (y - t(g["h_y0"]))
    ct, st = torch.cos(t(g["h_l"])), torch.sin(t(g["h_l"]))
    X, Y = xs * ct + ys * st, -xs * st + ys * ct
    env = al / math.sqrt(2 * math.pi) * torch.exp(-(4 * X * X + Y * Y) / 8)
    parts = [env * torch.where(t(g["h_ab"]) == 0, torch.cos(KAPPA * X), torch.sin(KAPPA * X)) * t(g["h_gain"])]
    if len(c["h_alpha"]):
        al = 1.0 / t(c["h_alpha"])
        xs, ys = al * (x - t(c["h_x0"])), al * (y - t(c["h_y0"]))
        r2 = -(xs * xs + ys * ys)
        v = torch.exp(r2 / (2 * SIGMA_C ** 2)) / SIGMA_C ** 2 - 0.9 * torch.exp(r2 / (2 * SIGMA_S ** 2)) / SIGMA_S ** 2
        parts.append(al * v / (2 * math.pi) * t(c["h_gain"]))
    return torch.cat(parts, 0)


def signs(M):
    m = torch.arange(-M, M + 1, device=DEV)
    return (1 - 2 * ((m[:, None] + m[None, :]) % 2)).to(F64)     # (-1)^(mx + my)


def dirichlet_coefficients(g, c, side, M):
    """(neurons, 2M+1, 2M+1) complex coefficients of every receptive field: row M - my, column mx + M."""
    px = 4 * (-(-side // 16) * 16)
    rows = torch.arange(M, -M - 1, -1, device=DEV) % px
    cols = torch.arange(-M, M + 1, device=DEV) % px
    mask = torch.zeros((2 * M + 1) ** 2, dtype=F64, device=DEV)
    mask[torch.as_tensor(ellipse(M), device=DEV)] = 1.0
    out = []
    ng, nc = len(g["h_alpha"]), len(c["h_alpha"])
    for a in range(0, max(ng, nc), 256):
        for p, q in (({k: v[a:a + 256] for k, v in g.items()}, None), (None, {k: v[a:a + 256] for k, v in c.items()})):
            none = {k: v[:0] for k, v in (c if q is None else g).items()}
            p, q = (none if p is None else p), (none if q is None else q)
            if not len(p["h_alpha"]) + len(q["h_alpha"]):
                continue
            f = torch.fft.fft2(field_values(p, q, px))[:, rows][:, :, cols]
            out.append((0 if len(p["h_alpha"]) else 1, f * (signs(M) * mask.reshape(2 * M + 1, -1) / (px * px))))
    return torch.cat([f for k, f in sorted(out, key=lambda o: o[0])], 0)


def spatial_basis(M, side):
    """phi_s on the side x side grid for the whole (2M+1)^2 coefficient grid: ((2M+1)^2, side * side)."""
    m = torch.arange(-M, M + 1, dtype=F64, device=DEV)
    p = torch.arange(side, dtype=F64, device=DEV)
    e = torch.exp(2j * math.pi * torch.outer(m, p) / side)
    px1 = e[None, :, None, :] * torch.flip(e, (0,))[:, None, :, None] * signs(M)[:, :, None, None]
    return px1.reshape((2 * M + 1) ** 2, side * side)


def spikes(case, seed):
    """What one encode leaves: spike intervals grouped by neuron (the first ``intervals`` of them where the case
    states a number), neuron parameters and the RF coefficients."""
    rng = np.random.default_rng([seed, 11])
    N, M, Mt, T = case["neurons"], case["M"], case["Mt"], case["samples"] * DT
    g, c = fields(N, rng)
    Ds = dirichlet_coefficients(g, c, case["side"], M)
    sm = torch.as_tensor(ellipse(M), device=DEV)
    d = Ds.reshape(N, -1)[:, sm]
    a = rng.standard_normal((len(sm), 2 * Mt + 1)) + 1j * rng.standard_normal((len(sm), 2 * Mt + 1))
    a = torch.as_tensor(0.5 * (a + np.conj(a[::-1, ::-1])), device=DEV)
    u = d.conj() @ a                                    # each neuron's drive: harmonics -Mt..Mt
    W = WT / Mt
    m = torch.arange(-Mt, Mt + 1, dtype=F64, device=DEV)
    grid = torch.exp(1j * W * torch.outer(m, torch.arange(0.0, 2 * math.pi / W, 1e-3, dtype=F64, device=DEV)))
    u = u * (0.9 / float((u @ grid).real.abs().max()))
    b = torch.as_tensor(rng.uniform(2, 4, N), device=DEV)
    delta = torch.as_tensor(np.abs(rng.normal(case["delta"], case["delta"] / 10, N)), device=DEV)
    v0 = torch.as_tensor(rng.uniform(0, 1, N), device=DEV) * delta
    up = u[:, Mt + 1:] / (1j * W * m[Mt + 1:])

    def area(t):                                        # int_0^t (b + u_n): increasing, as b > |u|
        z = torch.exp(1j * W * t)
        s = torch.zeros_like(z)
        for k in range(Mt - 1, -1, -1):
            s = (s + up[:, k, None]) * z
        return (b[:, None] + u[:, Mt, None].real) * t + 2 * (s.real - up.sum(1)[:, None].real)

    most = int(float(((4.9 * T + delta) / delta).max())) + 2
    target = delta[:, None] * torch.arange(1, most + 1, dtype=F64, device=DEV) - v0[:, None]
    lo, hi = torch.zeros_like(target), torch.full_like(target, T)
    inside = target < area(torch.full((N, 1), T, dtype=F64, device=DEV))
    for _ in range(54):
        mid = 0.5 * (lo + hi)
        over = area(mid) > target
        lo, hi = torch.where(over, lo, mid), torch.where(over, mid, hi)
    t = 0.5 * (lo + hi)
    both = inside[:, 1:]
    ind = torch.arange(N, device=DEV, dtype=torch.int32)[:, None].expand(both.shape)
    n = case.get("intervals")
    return {"tk1": t[:, :-1][both][:n].clone(), "tk2": t[:, 1:][both][:n].clone(), "ind": ind[both][:n].clone(),
            "kappa": torch.ones(N, dtype=F64, device=DEV), "delta": delta, "bias": b, "Ds": Ds, "fields": (g, c),
            "T": T, "norm": np.ones(N)}


def harmonics_T(tk1, tk2, Mt):
    """int over each interval of e^{jmWt}, m = -Mt..Mt: (intervals, 2Mt+1)."""
    W = WT / Mt
    m = torch.arange(-Mt, Mt + 1, dtype=F64, device=DEV)
    m1 = torch.where(m == 0, torch.ones_like(m), m)
    d, mid = tk2 - tk1, 0.5 * (tk1 + tk2)
    amp = torch.where(m[None] == 0, d[:, None], 2.0 / (m1 * W)[None] * torch.sin(0.5 * W * d[:, None] * m1[None]))
    return amp * torch.exp(1j * W * mid[:, None] * m[None])


def video_of(a, M, Mt, side, T):
    """Real video (frames, side, side) of the coefficients a (ellipse entries, 2Mt+1)."""
    sm = torch.as_tensor(ellipse(M), device=DEV)
    w = (spatial_basis(M, side)[sm].T @ a).T            # (2Mt+1, pixels)
    t = torch.as_tensor(np.arange(0, T, DT), device=DEV)
    m = torch.arange(-Mt, Mt + 1, dtype=F64, device=DEV)
    e = torch.exp(1j * (WT / Mt) * torch.outer(t, m))
    return (e.real @ w.real - e.imag @ w.imag).reshape(len(t), side, side)


def video(case, seed):
    from vtem_b200 import workloads
    side, F = case["side"], case["frames"]
    a = workloads.bandlimited_coeffs(6, 6, 8, seed)
    v = workloads.bandlimited_video(a, 6, 6, 8, 12 * math.pi, 12 * math.pi, WT, side, side, F, DT, device=DEV)
    return (v / v.abs().max()).to(getattr(torch, case["video"]))


def clip_sizes(case):
    """The sizes of a batch's clips: frame side, orders, duration and neuron count, uneven."""
    rng, out = np.random.default_rng(case["sizes"]), []
    for _ in range(case["clips"]):
        M, Mt = int(rng.integers(2, 7)), int(rng.integers(3, 9))
        samples = int(rng.uniform(1.1, 1.25) * Mt / 20.0 / DT)
        K = ellipse(M).size * (2 * Mt + 1)
        low = max(96, int(2.5 * K / (3.0 * samples * DT / 0.075)), 3 * ellipse(M).size)
        out.append({"side": int(rng.choice([16, 32, 48, 64])), "M": M, "Mt": Mt, "samples": samples, "delta": 0.075,
                    "neurons": int(rng.integers(low, max(low + 64, 1025)))})
    return out


# ------------------------------------------------------------------ the calls

def prep_result(c, s, side, M):
    from vtem_b200 import vtdm
    return vtdm.PrepResult(s["Ds"], None, None, s["norm"], M, M, side, side, side, side)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "project":
        from vtem_b200 import vrf
        g, c = fields(case["neurons"], np.random.default_rng([seed, 1]))
        banks = bank_objects(g, c, case["side"], 1)
        s.update(bank=vrf.vrf_bank(banks), V=video(case, seed))
    elif kind == "iaf":
        from vtem_b200 import ensemble_encode
        x, b, delta, v0 = iaf_inputs(case, seed)
        iaf = ensemble_encode.IAF_encode(case["neurons"], DT)
        iaf.load_parameters(h_kappa=np.ones(case["neurons"]), h_bias=b, h_delta=delta, h_v0=v0)
        s.update(iaf=iaf, x=x, v0=torch.as_tensor(v0, device=DEV), T=case["frames"] * DT)
    elif kind == "prep":
        g, c = fields(case["neurons"], np.random.default_rng([seed, 1]))
        s.update(banks=bank_objects(g, c, case["side"], 4), norm=np.ones(case["neurons"]))
    elif kind in ("gram", "reconstruct", "plain", "rnn3"):
        s.update(spikes(case, seed))
        M, side = case["M"], case["side"]
        flat = s["Ds"].reshape(case["neurons"], -1)
        s["Dsw"] = (flat.conj() @ flat.T).real.contiguous()
        if kind in ("reconstruct", "plain"):
            s["dirich"] = (flat @ spatial_basis(M, side)).real.reshape(-1, side, side).contiguous()
        if kind == "reconstruct":
            r = np.random.default_rng([seed, 5]).standard_normal(len(s["tk1"]))
            s["c"] = torch.as_tensor(r, device=DEV).reshape(-1, 1)
        if kind == "rnn3":
            s["G"], s["q"] = spike_gram(s, case["Mt"])
            s["step"] = 1.0 / top_eigenvalue(lambda v: s["G"] @ v, len(s["tk1"]))
    elif kind in ("decode", "rnn"):
        from vtem_b200 import fast
        s.update(spikes(case, seed))
        s["dec"] = fast.from_prep(prep_result(case, s, case["side"], case["M"]), WT, case["Mt"],
                                  solver=case.get("solver", "auto"))
        if kind == "rnn":
            P = phi(s, case)
            s["step"] = 1.0 / top_eigenvalue(lambda v: P.mH @ (P @ v), P.shape[1])
    elif kind == "batch":
        from vtem_b200 import batch
        probs = []
        for i, c in enumerate(clip_sizes(case)):
            k = spikes(c, seed * 1000 + i)
            probs.append(batch.ClipProblem(prep_result(c, k, c["side"], c["M"]), WT, c["Mt"], k["tk1"], k["tk2"],
                                           k["ind"], k["kappa"], k["delta"], k["bias"], k["T"], DT))
        s["bd"] = batch.BatchDecoder(probs, sweeps=case["sweeps"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "project":
        return s["bank"].filter(s["V"], out_layout=case["layout"], precision=case["precision"])
    if kind == "iaf":
        from vtem_b200 import spike_store
        s["iaf"].d_v0.copy_(s["v0"])          # every clip starts from its own membrane values
        sp = s["iaf"].encode_blocks(s["x"], layout="neuron")
        return [sp.count] + list(spike_store.device_pairs(sp, s["T"]))
    if kind == "prep":
        from vtem_b200 import vtdm
        M, side = case["M"], case["side"]
        w = 2 * math.pi * M
        r = vtdm.prep_from_banks(s["banks"], s["norm"], M, M, w, w, side, side, 1.0, 1.0)
        return [r.Ds, r.dirich, r.Dsw]
    if kind in ("gram", "reconstruct", "plain"):
        from vtem_b200 import dirichlet, linalg
        cp = dirichlet.dirichlet(case["neurons"], s["tk1"], s["tk2"], s["ind"], s["kappa"], s["delta"], s["bias"],
                                 s["norm"], WT, case["Mt"])
        if kind == "reconstruct":
            cp.d_q = s["c"]
            return cp.reconstruct(s["dirich"], [0, s["T"]], DT)
        cp.compute_q()
        cp.compute_G(s["Dsw"], lower_only=kind == "plain")
        if kind == "gram":
            return [cp.d_q, cp.d_G]
        cp.d_q = linalg.solve_eq_sym(cp.d_G, cp.d_q)
        cp.freeG()
        return cp.reconstruct(s["dirich"], [0, s["T"]], DT)
    if kind == "rnn3":
        from vtem_b200 import neural_network
        return neural_network.rnn3(s["G"], s["q"], dt=s["step"], alpha=1.0, steps=case["steps"])
    if kind == "batch":
        return s["bd"].run()
    dec, spk = s["dec"], (s["tk1"], s["tk2"], s["ind"], s["kappa"], s["delta"], s["bias"])
    if kind == "rnn":
        a, _ = dec.rnn_coefficients(*spk, dt_alpha=s["step"], steps=case["steps"])
        return [a, dec.synthesize(a, s["T"], DT)]
    u = dec.decode(*spk, s["T"], DT, out_dtype=getattr(torch, case["out"]))
    return [dec.a, u]


# ------------------------------------------------------------------ the same in 64 bits, without the framework

def iaf_inputs(case, seed):
    """Projections (neurons, frames) of a bandlimited video with no mean over the clip, |x| < 1, and the
    parameters of one population, the same for every clip (so that every clip has as many spikes)."""
    rng = np.random.default_rng([seed, 3])
    N, F, Mt = case["neurons"], case["frames"], case["Mt"]
    c = torch.as_tensor(rng.standard_normal((N, Mt + 1)) + 1j * rng.standard_normal((N, Mt + 1)), device=DEV)
    t = torch.arange(F, dtype=F64, device=DEV) * DT
    m = torch.arange(0, Mt + 1, dtype=F64, device=DEV)
    x = (c @ torch.exp(1j * (WT / Mt) * torch.outer(m, t))).real
    x = x - ((x[:, :-1] + x[:, 1:]).sum(1) / (2 * (F - 1)))[:, None]
    rng = np.random.default_rng([N, F])
    delta = np.abs(rng.normal(case["delta"], case["delta"] / 10, N))
    return (x * (0.9 / x.abs().max())).contiguous(), rng.uniform(2, 4, N), delta, rng.uniform(0, 1, N) * delta


def phi(s, case):
    """The spike-interval operator (intervals, coefficients): q = phi a."""
    sm = torch.as_tensor(ellipse(case["M"]), device=DEV)
    d = s["Ds"].reshape(case["neurons"], -1)[:, sm].conj()[s["ind"].long()]
    T = harmonics_T(s["tk1"], s["tk2"], case["Mt"])
    return (d[:, :, None] * T[:, None, :]).reshape(len(s["tk1"]), -1)


def measurements(s):
    k = s["ind"].long()
    return (s["kappa"][k] * s["delta"][k] - s["bias"][k] * (s["tk2"] - s["tk1"])).reshape(-1, 1)


def spike_gram(s, Mt):
    T = harmonics_T(s["tk1"], s["tk2"], Mt)
    R = torch.cat([T.real, T.imag], 1)
    G = R @ R.T
    k = s["ind"].long()
    for a in range(0, len(k), 2048):
        G[a:a + 2048] *= s["Dsw"][k[a:a + 2048]][:, k]
    return G, measurements(s)


def top_eigenvalue(mul, n):
    v = torch.ones(n, dtype=C128, device=DEV)
    try:
        mul(v)
    except RuntimeError:
        v = v.real
    for _ in range(30):
        w = mul(v)
        lam = float(w.norm() / v.norm())
        v = w / w.norm()
    return 1.05 * lam


def iaf_exact(case, seed):
    """Spike times by stepping every neuron at once, block by block of 101 frames."""
    x, b, delta, v = iaf_inputs(case, seed)
    y = (x.cpu().numpy() + b[:, None]).T
    N, F, step = case["neurons"], case["frames"], 100
    v, tc = v.copy(), np.zeros(N)
    times = [[] for _ in range(N)]
    for i in range(F - 1):
        if i % step == 0:
            tc[:] = 0.0
        y1, y2 = y[i], y[i + 1]
        area = (y1 + y2) / 2 * DT
        for n in np.nonzero(v + area >= delta)[0]:
            p, left, ar = y1[n], DT, area[n]
            while v[n] + ar >= delta[n]:
                a = (y2[n] - p) / left
                r = (delta[n] - v[n]) / p if abs(a) <= 1e-12 else (math.sqrt(p * p + 2 * (delta[n] - v[n]) * a) - p) / a
                tc[n] += r
                times[n].append(tc[n] + (i // step) * (step * DT))
                ar, v[n], left, p = ar - (delta[n] - v[n]), 0.0, left - r, p + r * a
            v[n] += ar - area[n]                 # the common update below adds the whole step's area
            tc[n] += left - DT
        v += area
        tc += DT
    t1 = np.concatenate([np.array(t[:-1]) for t in times])
    t2 = np.concatenate([np.array(t[1:]) for t in times])
    ind = np.concatenate([np.full(max(0, len(t) - 1), n, np.int32) for n, t in enumerate(times)])
    return [np.array([len(t) for t in times], np.int32), t1, t2, ind]


def solve_window(s, case):
    """Reconstruction coefficients (ellipse entries, 2Mt+1) of one window: least squares by the normal equations."""
    P = phi(s, case)
    q = measurements(s).to(C128)
    A = P.mH @ P
    L = torch.linalg.cholesky(A)
    a = torch.cholesky_solve(P.mH @ q, L)
    for _ in range(2):
        a = a + torch.cholesky_solve(P.mH @ (q - P @ a), L)
    return a.reshape(-1, 2 * case["Mt"] + 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "project":
        g, c = fields(case["neurons"], np.random.default_rng([seed, 1]))
        side = case["side"]
        rf = field_values(g, c, side).reshape(case["neurons"], -1)
        V = video(case, seed).to(F64).reshape(case["frames"], -1)
        L = (V @ rf.T) * (1.0 / (side * side))
        return L if case["layout"] == "time" else L.T.contiguous()
    if kind == "iaf":
        return iaf_exact(case, seed)
    if kind == "prep":
        g, c = fields(case["neurons"], np.random.default_rng([seed, 1]))
        Ds = dirichlet_coefficients(g, c, case["side"], case["M"])
        flat = Ds.reshape(case["neurons"], -1)
        dirich = (flat @ spatial_basis(case["M"], case["side"])).real
        return [Ds, dirich.reshape(-1, case["side"], case["side"]), (flat.conj() @ flat.T).real]
    if kind == "batch":
        out = []
        for i, c in enumerate(clip_sizes(case)):
            k = spikes(c, seed * 1000 + i)
            out.append(video_of(solve_window(k, c), c["M"], c["Mt"], c["side"], k["T"]))
        return out
    s = prepare_plain(case, seed)
    if kind == "gram":
        G, q = spike_gram(s, case["Mt"])
        return [q, G]
    if kind == "rnn3":
        G, q = spike_gram(s, case["Mt"])
        h = 1.0 / top_eigenvalue(lambda v: G @ v, len(s["tk1"]))
        x = torch.zeros_like(q)
        for _ in range(case["steps"] + 1):
            x = x + h * (q - G @ x)
        return x
    M, Mt, side = case["M"], case["Mt"], case["side"]
    if kind == "reconstruct":
        r = np.random.default_rng([seed, 5]).standard_normal(len(s["tk1"]))
        w = torch.zeros((case["neurons"], 2 * Mt + 1), dtype=C128, device=DEV)
        w.index_put_((s["ind"].long(),), torch.as_tensor(r, device=DEV)[:, None] * harmonics_T(
            s["tk1"], s["tk2"], Mt).conj(), accumulate=True)
        sm = torch.as_tensor(ellipse(M), device=DEV)
        return video_of(s["Ds"].reshape(case["neurons"], -1)[:, sm].T @ w, M, Mt, side, s["T"])
    if kind == "rnn":
        P = phi(s, case)
        h = 1.0 / top_eigenvalue(lambda v: P.mH @ (P @ v), P.shape[1])
        A, b = P.mH @ P, P.mH @ measurements(s).to(C128)
        a = torch.zeros_like(b)
        for _ in range(case["steps"] + 1):
            a = a + h * (b - A @ a)
        a = a.reshape(-1, 2 * Mt + 1)
        return [a.reshape(-1), video_of(a, M, Mt, side, s["T"])]
    a = solve_window(s, case)
    u = video_of(a, M, Mt, side, s["T"])
    return u if kind == "plain" else [a.reshape(-1), u]


def prepare_plain(case, seed):
    """spikes() with the cross-weights: the inputs of exact()."""
    s = spikes(case, seed)
    flat = s["Ds"].reshape(case["neurons"], -1)
    s["Dsw"] = (flat.conj() @ flat.T).real
    return s


# ------------------------------------------------------------------ what a pass cannot do without

def window_work(c, out_bytes=8):
    """One window in the coefficient space: temporal Grams, the Hermitian system, one factorisation, two products
    with the operator, and the synthesis."""
    N, Mt = c["neurons"], c["Mt"]
    Ks, Kt = ellipse(c["M"]).size, 2 * Mt + 1
    K = Ks * Kt
    n = N * 3.0 * c["samples"] * DT / c["delta"]
    vox = c["samples"] * c["side"] ** 2
    flops = 8.0 * n * Kt * (Kt + 1) / 2 + 8.0 * N * (Ks * (Ks + 1) / 2) * (Kt * (Kt + 1) / 2) + K ** 3 / 3.0
    flops += 4 * 8.0 * N * Ks * Kt + 2.0 * vox * Kt / 2
    return {"bytes": 20.0 * n + 16.0 * N * Ks + out_bytes * vox, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "project":
        P, F, N = case["side"] ** 2, case["frames"], case["neurons"]
        return {"bytes": F * P * (8.0 if case["video"] == "float64" else 4.0) + 8.0 * N * P + 8.0 * F * N,
                "flops": 2.0 * F * P * N}
    if kind == "iaf":
        N, F = case["neurons"], case["frames"]
        return {"bytes": 8.0 * N * F + 20.0 * N * 3.0 * F * DT / case["delta"], "flops": 6.0 * N * F}
    if kind == "prep":
        N, M, P = case["neurons"], case["M"], case["side"] ** 2
        px = 4 * (-(-case["side"] // 16) * 16)
        k = 2 * M + 1
        return {"bytes": 16.0 * N * k * k + 8.0 * N * P + 8.0 * N * N,
                "flops": N * (20.0 * px * px + 4.0 * px * px * k + 8.0 * px * k * k + 8.0 * k * k * case["side"]
                              + 4.0 * k * P) + 4.0 * N * N * ellipse(M).size}
    if kind == "batch":
        w = [window_work(c) for c in clip_sizes(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    N, Mt = case["neurons"], case["Mt"]
    n = case.get("intervals") or N * 3.0 * case["samples"] * DT / case["delta"]
    vox = case["samples"] * case["side"] ** 2
    if kind == "gram":
        return {"bytes": 8.0 * n * n + 20.0 * n + 8.0 * N * N, "flops": n * n * (2.0 * (2 * Mt + 1) + 1)}
    if kind == "reconstruct":
        P = case["side"] ** 2
        return {"bytes": 28.0 * n + 8.0 * N * P + 8.0 * vox, "flops": (2.0 * N * P + 2.0 * vox) * (2 * Mt + 1)}
    if kind == "plain":
        return {"bytes": 4.0 * n * n + 8.0 * N * case["side"] ** 2 + 8.0 * vox,
                "flops": n * n * (2 * Mt + 1) + 4.0 / 3.0 * n ** 3 + 2.0 * vox * (2 * Mt + 1)}
    if kind == "rnn3":
        return {"bytes": 8.0 * n * n, "flops": 2.0 * n * n * (case["steps"] + 1)}
    w = window_work(case, 4 if case.get("out") == "float32" else 8)
    if kind == "rnn":
        K = ellipse(case["M"]).size * (2 * Mt + 1)
        w["flops"] += 2.0 * K * K * (case["steps"] + 1) - K ** 3 / 3.0
    return w
