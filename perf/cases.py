"""Performance cases of the photon transport, through the package's public entry points.

``listed()`` names the cases, ``draw(rng)`` makes one more of the same ranges,
``prepare(case, seed)`` builds what a program has in hand before the call, ``run(state)`` is
one pass, ``work(case)`` the bytes and operations a pass cannot do without and
``exact(case, seed)`` the outputs in 64 bits where plain numpy or torch gives them quickly.

Scenes are the package's own workloads (``luminis_mc_b200.workloads``); a case's seed is the
seed of its photon streams (and, for the set-up tables, of the particle sizes).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "luminis-mc_b200"))

import luminis_mc_b200 as lm  # noqa: E402
from luminis_mc_b200 import workloads as W  # noqa: E402
from luminis_mc_b200.adjoint import AdjointTransport, lr_transport  # noqa: E402
from luminis_mc_b200.device import DeviceRun  # noqa: E402
from luminis_mc_b200.sweep import SweepRun  # noqa: E402

DEVICE = "cuda:0"
FLOPS_PER_EVENT = 300.0          # binary operations of one scattering event (reference arithmetic)
FLOPS_PER_PAIR = 480.0           # of one estimated (vertex, bin) pair
EVENTS = {"cbs": 317.0, "bilayer": 166.0, "bilayer_hg": 170.0, "mixture": 258.0}


def listed():
    return [
        # a first look or a parity check: one call of the drop-in function with few photons
        {"name": "call_cbs_10k", "kind": "call", "scene": "cbs", "precision": "fp32", "photons": 10_007},
        # the small configuration at its own size, again as one call
        {"name": "call_cbs_1m", "kind": "call", "scene": "cbs", "precision": "fp32", "photons": 1_000_000},
        # the reference's own precision on the bilayer, time-resolved sensors on the host
        {"name": "call_bilayer_fp64", "kind": "call", "scene": "bilayer", "precision": "fp64",
         "photons": 2_000_003},
        # the headline workload: production statistics, tallies resident on the GPU
        {"name": "run_bilayer_50m", "kind": "run", "scene": "bilayer", "precision": "fp32",
         "photons": 50_000_000},
        # an inversion step: outputs and the gradient of a loss over them
        {"name": "gradient_hg_3m", "kind": "gradient", "precision": "fp32", "photons": 3_000_001},
        # a parameter study over many media, one launch
        {"name": "sweep_256", "kind": "sweep", "scenes": 256, "photons": 11_000_000, "gradients": False},
        # the same with each medium's derivatives, fewer media
        {"name": "sweep_gradients_32", "kind": "sweep", "scenes": 32, "photons": 2_500_000,
         "gradients": True},
        # last-flight estimation of the cone: smooth curves from few photons
        {"name": "estimator_100", "kind": "estimator", "precision": "fp32", "photons": 100_003, "bins": 100},
        # a three-species mixture with the absorption map
        {"name": "mixture_absorption", "kind": "mixture", "precision": "fp32", "photons": 2_000_000,
         "absorption": True},
        # fluence and statistics at depths inside the slab, crossed any number of times
        {"name": "depth_planes", "kind": "depth", "precision": "fp32", "photons": 1_000_003, "planes": 3},
        # speckle and a narrow cone at very long paths (weak absorption)
        {"name": "long_paths", "kind": "long", "precision": "fp32", "photons": 100_000,
         "max_events": 100_000},
        # set-up tables of a study's particles
        {"name": "tables_256", "kind": "tables", "species": 256, "divisions": 1000},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["call", "call", "run", "run", "gradient", "sweep", "estimator", "mixture",
                       "depth", "long", "tables"])
    c = {"kind": kind}
    if kind in ("call", "run", "gradient", "estimator", "mixture", "depth", "long"):
        c["precision"] = rng.choice(["fp32", "fp32", "fp64"])
    half = 2 if c.get("precision") == "fp64" else 1
    if kind == "call":
        c.update(scene=rng.choice(["cbs", "bilayer"]), photons=log_int(1_000, 2_000_000))
    elif kind == "run":
        c.update(scene=rng.choice(["bilayer", "bilayer_hg"]), photons=log_int(100_000, 40_000_000 // half))
    elif kind == "gradient":
        c["photons"] = log_int(20_000, 6_000_000 // half)
    elif kind == "sweep":
        c.update(scenes=log_int(2, 256), photons=log_int(300_000, 11_000_000),
                 gradients=rng.random() < 0.4)
    elif kind == "estimator":
        c.update(photons=log_int(2_000, 200_000 // (2 * half)), bins=rng.randrange(30, 160))
    elif kind == "mixture":
        c.update(photons=log_int(30_000, 6_000_000 // half), absorption=rng.random() < 0.6)
    elif kind == "depth":
        c.update(photons=log_int(20_000, 2_000_000 // half), planes=rng.randrange(1, 5))
    elif kind == "long":
        c.update(photons=log_int(2_000, 100_000 // half), max_events=log_int(5_000, 60_000 // half))
    else:
        c.update(species=log_int(2, 256), divisions=log_int(150, 3_000))
    return c


# --------------------------------------------------------------------------- scenes
def scene(case, seed):
    """The workload spec of a transport case."""
    kind, n = case["kind"], case["photons"]
    name = case.get("scene")
    if kind == "estimator":
        spec = W.mie_cbs_small(n, seed)
        spec["sensors"] = [dict(spec["sensors"][0], estimator=True, d_theta=0.1 / case["bins"])]
    elif kind == "gradient":
        spec = W.bilayer_hg(n, seed)
    elif kind == "mixture":
        spec = W.mixture_bilayer(n, seed)
        if case["absorption"]:
            spec["absorption"] = {"radius": 5.0, "depth": 2.0, "d_r": 0.05, "d_z": 0.02}
    elif kind == "depth":
        # fluence maps at depths through both layers and statistics of the way back, beside
        # the cone at the surface
        spec = W.bilayer_rgd_mie(n, seed)
        spec["sensors"] = [spec["sensors"][0]] + [
            {"kind": "planar_fluence", "z": 0.2 * (i + 1), "len_x": 6.0, "len_y": 6.0, "len_t": 0.0,
             "dx": 0.06, "dy": 0.06, "d_t": 0.0, "absorb": False} for i in range(case["planes"])]
        spec["sensors"].append({"kind": "statistics", "z": 0.25, "absorb": False, "events": 200,
                                "theta": [0.0, 3.1416, 90], "depth": [2.0, 100],
                                "direction_limit": "backward"})
    elif kind == "long":
        spec = W.mie_long_paths(n, seed)
        spec["max_events"] = case["max_events"]
    elif name == "cbs":
        spec = W.mie_cbs_small(n, seed)
    elif name == "bilayer_hg":
        spec = W.bilayer_hg(n, seed)
    else:
        spec = W.bilayer_rgd_mie(n, seed)
        if kind == "call":                   # 11 time bins and the integrated one
            spec["sensors"][1].update(len_t=11.0)
    return spec


def sweep_media(case, seed):
    """Specs and photon counts of a parameter study."""
    n = case["scenes"]
    specs = [W.mie_sweep(i, seed=seed, count=n) for i in range(n)]
    share = W.mie_sweep_parameters(n)[3].astype(np.float64)
    counts = np.maximum(1, np.floor(share / share.sum() * case["photons"])).astype(np.uint64)
    return specs, counts


def particles(case, seed):
    """(wavelength, radius, n_particle, n_medium) of a study's spheres: 0.05 to 2 um."""
    radius = np.exp(np.random.default_rng(seed).uniform(math.log(0.05e-3), math.log(2.0e-3),
                                                        case["species"]))
    return [(W.LAMBDA, float(r), W.N_SPHERE, W.N_WATER) for r in radius]


# --------------------------------------------------------------------------- passes
def prepare(case, seed):
    kind = case["kind"]
    if kind == "tables":
        return {"kind": kind, "species": particles(case, seed), "divisions": case["divisions"]}
    if kind == "sweep":
        specs, counts = sweep_media(case, seed)
        configs = W.build_mie_sweep(lm, specs)
        sweep = SweepRun(configs, device=DEVICE)
        sweep.set_photons(counts)
        return {"kind": kind, "sweep": sweep, "seed": seed, "gradients": case["gradients"]}
    config, sensors, keep = W.build(lm, scene(case, seed))
    state = {"kind": kind, "config": config, "sensors": sensors, "keep": keep, "seed": seed,
             "photons": case["photons"], "precision": case["precision"]}
    if kind == "gradient":
        state["transport"] = AdjointTransport(config, radial_sensor=1, radial_bins=100,
                                              radial_max=5.0, device=DEVICE)
        state["theta"] = torch.tensor(state["transport"].parameters(), dtype=torch.float64)
    elif kind != "call":
        state["device"] = DeviceRun(config, device=DEVICE)
    return state


def run(state):
    kind = state["kind"]
    if kind == "tables":
        pairs = lm.mie_species(state["species"], state["divisions"])
        return {"cdf": np.stack([ph._table()[1] for ph, _ in pairs]),
                "sigma": np.array([ph.scattering_cross_section() for ph, _ in pairs]),
                "s1": np.stack([med._s1 for _, med in pairs]),
                "s2": np.stack([med._s2 for _, med in pairs])}
    if kind == "sweep":
        sweep = state["sweep"]
        sweep.zero()
        if not state["gradients"]:
            stats = sweep.run(state["seed"])
            return {"tallies": sweep.tallies, "hits": sweep.hits().astype(np.int64),
                    "events": stats["events"], "detected": stats["detected"]}
        blocks, stats = sweep.run_adjoint(state["seed"])
        return {"tallies": sweep.tallies, "events": stats["events"],
                "outputs": torch.cat([o for o, _ in blocks]),
                "jacobians": torch.cat([j.reshape(-1) for _, j in blocks])}
    if kind == "call":
        lm.run_simulation_parallel(state["config"], precision=state["precision"])
        out = {}
        for i, s in enumerate(state["sensors"]):
            names = (["S%d_coh" % q for q in range(4)] + ["S%d_incoh" % q for q in range(4)]
                     if isinstance(s, lm.FarFieldCBSSensor) else ["S%d" % q for q in range(4)])
            out["sensor%d" % i] = {"hits": s.hits}
            for q in names:
                out["sensor%d" % i][q] = list(getattr(s, q))
        return out
    if kind == "gradient":
        theta = state["theta"].clone().requires_grad_(True)
        y = lr_transport(theta, state["transport"], state["photons"], state["seed"],
                         precision=state["precision"])
        y.square().sum().backward()
        return {"outputs": y.detach(), "gradient": theta.grad,
                "tallies": state["transport"].last_tallies}
    dev = state["device"]
    dev.zero()
    stats, _ = dev.run(state["photons"], state["seed"], precision=state["precision"])
    return {"tallies": dev.tallies, "hits": stats["hits"],
            **{k: stats[k] for k in ("photons", "events", "steps", "draws", "detected", "escaped",
                                     "roulette", "cap")}}


# --------------------------------------------------------------------------- work
def tally_doubles(case):
    kind = case["kind"]
    cone, fluence = 8 * 200 * 8, 4 * 200 * 200
    if kind == "call":
        return 800 if case["scene"] == "cbs" else cone + 12 * fluence + 4 * 90 * 36
    return {"run": cone + 64 * fluence + 4 * 90 * 36, "gradient": cone + 64 * fluence + 4 * 90 * 36,
            "estimator": 8 * case.get("bins", 0), "mixture": cone + 32 * 4 * 100 * 100 + 101 * 101,
            "depth": cone + case.get("planes", 0) * 4 * 100 * 100 + 390,
            "long": 8 * 400 + 4 * 256 * 256}[kind]


def work(case):
    """Bytes: the set-up tables read once and the tallies written once.  Operations: those of
    the scattering events (mean events per photon of the workload) and estimated pairs."""
    kind = case["kind"]
    tables = 2 * (1001 * 16 + 1000 * 32)
    if kind == "tables":
        nodes = case["divisions"] + 1 + 1000
        # ~25 terms of the series on average over the radii, 22 operations a term
        return {"bytes": 8.0 * case["species"] * (case["divisions"] + 1 + 4000),
                "flops": 22.0 * 25.0 * nodes * case["species"]}
    if kind == "sweep":
        rows = 800 * (1 + (5 if case["gradients"] else 0) / 4)
        return {"bytes": case["scenes"] * (8.0 * rows + tables / 2),
                "flops": FLOPS_PER_EVENT * 250.0 * case["photons"]}
    if kind == "long":
        events = 11_069.0 * math.sqrt(case["max_events"] / 1e6)
    else:
        events = EVENTS["mixture" if kind == "mixture" else "cbs" if kind == "estimator"
                        else "bilayer_hg" if kind == "gradient" else case.get("scene", "bilayer")]
    flops = FLOPS_PER_EVENT * events * case["photons"]
    if kind == "estimator":
        flops += FLOPS_PER_PAIR * events * case["bins"] * case["photons"]
    return {"bytes": tables + 8.0 * tally_doubles(case), "flops": flops}


# --------------------------------------------------------------------------- exact values
def exact(case, seed):
    """The set-up tables, and the small cone's tallies, in 64 bits.  The other transports
    (10^8 to 10^10 events, or sensors that no plain array code states briefly) have none."""
    if case["kind"] == "tables":
        rows = [mie_tables(case["divisions"], *p) for p in particles(case, seed)]
        return {k: np.stack([r[i] for r in rows]) for i, k in enumerate(("cdf", "sigma", "s1", "s2"))}
    if case["kind"] == "call" and case["scene"] == "cbs" and case["photons"] <= 1_000_000:
        grids, hits = cone_tallies(scene(case, seed), case["precision"])
        names = ["S%d_coh" % q for q in range(4)] + ["S%d_incoh" % q for q in range(4)]
        return {"sensor0": {"hits": hits, **{n: [grids[q]] for q, n in enumerate(names)}}}
    return None


def mie_amplitudes(x, m, mu):
    """S1, S2 at cosines mu and the scattering efficiency of a sphere with real relative index m
    (W. J. Wiscombe, Appl. Opt. 19, 1505 (1980): term count, log-derivative, Riccati-Bessel
    recurrence)."""
    n_max = int(x + 4.0 * x ** (1 / 3) + 1) if x <= 8 else int(x + 4.05 * x ** (1 / 3) + 2)
    d = np.zeros(n_max + 40)                  # logarithmic derivative at m x, downward
    for n in range(len(d) - 1, 0, -1):
        d[n - 1] = n / (m * x) - 1.0 / (d[n] + n / (m * x))
    psi0, psi = math.sin(x), math.sin(x) / x - math.cos(x)
    chi0, chi = math.cos(x), math.cos(x) / x + math.sin(x)
    p0, p = np.zeros_like(mu), np.ones_like(mu)
    s1, s2, q = np.zeros(mu.shape, complex), np.zeros(mu.shape, complex), 0.0
    for n in range(1, n_max + 1):
        z0, z = complex(psi0, chi0), complex(psi, chi)
        fa, fb = d[n] / m + n / x, d[n] * m + n / x
        a, b = (fa * psi - psi0) / (fa * z - z0), (fb * psi - psi0) / (fb * z - z0)
        q += (2 * n + 1) * (abs(a) ** 2 + abs(b) ** 2)
        tau = n * mu * p - (n + 1) * p0
        f = (2 * n + 1) / (n * (n + 1))
        s1 += f * (a * p + b * tau)
        s2 += f * (a * tau + b * p)
        p0, p = p, ((2 * n + 1) * mu * p - (n + 1) * p0) / n
        psi0, psi = psi, (2 * n + 1) / x * psi - psi0
        chi0, chi = chi, (2 * n + 1) / x * chi - chi0
    return s1, s2, 2.0 / x ** 2 * q


def mie_tables(n_div, wavelength, radius, n_particle, n_medium):
    """CDF over theta (rectangle rule), cross section and the 1000-node amplitude table."""
    m = n_particle / n_medium
    theta = np.arange(n_div + 1) * (math.pi / n_div)
    s1, s2, q = mie_amplitudes(2 * math.pi * n_medium / wavelength * radius, m, np.cos(theta))
    cdf = np.cumsum((np.abs(s1) ** 2 + np.abs(s2) ** 2) * np.sin(theta))
    mu = np.cos(np.arange(1000) * (math.pi / 999))
    a1, a2, _ = mie_amplitudes(2 * math.pi * radius / wavelength, m, mu)
    return cdf / cdf[-1], np.float64(q * math.pi * radius ** 2), a1, a2


def philox(block, photon, seed):
    """Philox4x32-10 words [..., 4] of the streams (seed, photon) at the given blocks
    (J. K. Salmon et al., SC'11)."""
    mask = 0xFFFFFFFF
    c = [block, torch.zeros_like(block), photon & mask, photon >> 32]
    k0, k1 = seed & mask, (seed >> 32) & mask
    for _ in range(10):
        a, b = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((b >> 32) & mask) ^ c[1] ^ k0, b & mask, ((a >> 32) & mask) ^ c[3] ^ k1, a & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return torch.stack(c, -1)


def uniforms(draw, photon, seed, precision, count):
    """[n, count] values of the streams from position draw on: 24-bit values, four to a block,
    or 53-bit ones, two to a block."""
    per = 4 if precision == "fp32" else 2
    blocks = (count + per - 1) // per + 1
    b = (draw // per)[:, None] + torch.arange(blocks, device=draw.device)
    w = philox(b, photon[:, None].expand_as(b), seed)
    if per == 4:
        u = (2 * (w >> 9) + 1).double() * 2.0 ** -24
    else:
        hi, lo = w[..., 1::2], w[..., 0::2]
        u = (2 * ((hi << 20) | (lo >> 12)) + 1).double() * 2.0 ** -53
    u = u.flatten(1)
    return u.gather(1, (draw % per)[:, None] + torch.arange(count, device=draw.device))


def cone_tallies(spec, precision):
    """The FarFieldCBS tallies [8][theta][phi] of a semi-infinite Mie medium, all photons a
    scattering event at a time in 64-bit torch."""
    medium, sensor = spec["media"][0], spec["sensors"][0]
    ph = spec["phases"][0]
    cdf, _, a1, a2 = mie_tables(ph["nDiv"], ph["wavelength"], ph["radius"], ph["n_particle"],
                                ph["n_medium"])
    dev = DEVICE
    cdf = torch.tensor(cdf, device=dev)
    amp = torch.tensor(np.stack([a2, a1], 1), device=dev)             # S2, S1 by theta
    k0 = 2 * math.pi / medium["wavelength"]
    albedo = medium["mu_s"] / (medium["mu_s"] + medium["mu_a"])

    def amplitudes(theta):
        pos = theta * (999 / math.pi)
        i = pos.long().clamp(0, 998)
        t = (pos - i).clamp(0.0, 1.0)[:, None]
        return amp[i] + t * (amp[i + 1] - amp[i])

    def unit(v, fallback):
        n2 = (v * v).sum(-1, keepdim=True)
        return torch.where(n2 < 1e-20, fallback, v / n2.clamp_min(1e-300).sqrt())

    def turn(e, r00, r01, r10, r11):                                  # 2x2 real times Jones
        return torch.stack([r00 * e[:, 0] + r01 * e[:, 1], r10 * e[:, 0] + r11 * e[:, 1]], 1)

    def dot(a, b):
        return (a * b).sum(-1)

    def scatter(e, s_in, s_out, m_in, n_in, m_out, n_out):
        """A scatter s_in -> s_out on Jones vectors in the frames (m_in, n_in), (m_out, n_out)."""
        s = amplitudes(torch.acos(dot(s_in, s_out).clamp(-1, 1)))
        n_p = unit(torch.linalg.cross(s_in, s_out), n_in)
        m_pi = unit(torch.linalg.cross(n_p, s_in), m_in)
        m_po = unit(torch.linalg.cross(n_p, s_out), m_out)
        f = s * turn(e, dot(m_pi, m_in), dot(m_pi, n_in), dot(n_p, m_in), dot(n_p, n_in))
        return turn(f, dot(m_out, m_po), dot(m_out, n_p), dot(n_out, m_po), dot(n_out, n_p))

    n = spec["n_photons"]
    photon = torch.arange(n, device=dev)
    eye = torch.eye(3, dtype=torch.float64, device=dev)
    e0 = torch.tensor([spec["laser"]["m"], spec["laser"]["n"]], dtype=torch.complex128, device=dev)
    st = {"photon": photon, "draw": torch.zeros_like(photon),
          "pos": torch.tensor([0.0, 0.0, 1e-9], dtype=torch.float64, device=dev).expand(n, 3),
          "P": eye.expand(n, 3, 3), "E": e0.expand(n, 2),
          "w": torch.ones(n, dtype=torch.float64, device=dev)}
    st.update(r1=st["pos"], rn=st["pos"], P1=st["P"], Pn1=st["P"],
              T=torch.eye(2, dtype=torch.complex128, device=dev).expand(n, 2, 2),
              J=torch.eye(2, dtype=torch.complex128, device=dev).expand(n, 2, 2))
    n_theta = int(math.ceil(sensor["theta_max"] / sensor["d_theta"]))
    grids = torch.zeros(8, n_theta, dtype=torch.float64, device=dev)
    hits = 0
    for event in range(spec["max_events"] + 2):
        if not len(st["photon"]):
            break
        u = uniforms(st["draw"], st["photon"], spec["seed"], precision, 2 + 2 * 6)
        pos = st["pos"] - medium["mfp"] * torch.log(u[:, :1]) * st["P"][:, 2]
        out = pos[:, 2] < 0
        if out.any():
            h = {k: v[out] for k, v in st.items()}
            s = h["P"][:, 2]
            lo, hi = math.cos(sensor["theta_limit"][1]), math.cos(sensor["theta_limit"][0])
            theta = torch.acos((-s[:, 2]).clamp(-1, 1))
            it = (theta / sensor["d_theta"]).long()
            ok = (-s[:, 2] >= lo) & (-s[:, 2] <= hi) & (it < n_theta)
            h, it = {k: v[ok] for k, v in h.items()}, it[ok]
            hits += len(it)
            field = h["E"] * h["w"].sqrt()[:, None]
            lab = [field[:, :1] * h["P"][:, 0, :2] + field[:, 1:] * h["P"][:, 1, :2]]
            if event >= 2:
                z = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device=dev).expand(len(it), 3)
                x, y = eye[0].expand_as(z), eye[1].expand_as(z)
                e = scatter(e0.expand(len(it), 2), z, -h["Pn1"][:, 2], x, y, h["Pn1"][:, 0],
                            -h["Pn1"][:, 1])
                q = torch.tensor([1.0, -1.0], dtype=torch.float64, device=dev)
                e = q * torch.einsum("nij,ni->nj", h["T"], q * e)
                e = scatter(e, -h["P1"][:, 2], h["P"][:, 2], h["P1"][:, 0], -h["P1"][:, 1],
                            h["P"][:, 0], h["P"][:, 1])
                e = e / e.abs().square().sum(1, keepdim=True).sqrt().clamp_min(1e-300)
                phase = k0 * dot(h["P"][:, 2] + z, h["rn"] - h["r1"])
                e = e * (torch.polar(h["w"].sqrt(), phase))[:, None]
                lab.append(e[:, :1] * h["P"][:, 0, :2] + e[:, 1:] * h["P"][:, 1, :2])

            def stokes(f):
                xx, yy = f[:, 0].abs().square(), f[:, 1].abs().square()
                xy = f[:, 0] * f[:, 1].conj()
                return torch.stack([xx + yy, xx - yy, 2 * xy.real, 2 * xy.imag])

            grids[:4].index_add_(1, it, stokes(sum(lab)))
            grids[4:].index_add_(1, it, sum(stokes(f) for f in lab))
        keep = ~out
        st = {k: v[keep] for k, v in st.items()}
        u, pos = u[keep], pos[keep]
        v = u[:, 1].contiguous()
        i = torch.searchsorted(cdf, v).clamp_max(len(cdf) - 1)
        j = (i - 1).clamp_min(0)
        theta = (j + torch.where(i > 0, (v - cdf[j]) / (cdf[i] - cdf[j]), 0.0)) * (math.pi / (len(cdf) - 1))
        s = amplitudes(theta)
        ss, ee = s.abs().square(), st["E"].abs().square()
        a = ss[:, 0] * ee[:, 0] + ss[:, 1] * ee[:, 1]
        b = ss[:, 1] * ee[:, 0] + ss[:, 0] * ee[:, 1]
        c = 2 * (ss[:, 0] - ss[:, 1]) * (st["E"][:, 0] * st["E"][:, 1].conj()).real
        f_max = 0.5 * (a + b) + 0.5 * ((a - b) ** 2 + c * c).sqrt()
        cp, sp, f_acc = torch.zeros_like(a), torch.zeros_like(a), torch.ones_like(a)
        st["draw"] = st["draw"] + 2
        todo = torch.arange(len(a), device=dev)
        trials = u[:, 2:]
        while len(todo):                                              # six azimuth trials at a time
            phi = 2 * math.pi * trials[:, 0::2]
            ct, sn = torch.cos(phi), torch.sin(phi)
            f = a[todo, None] * ct * ct + b[todo, None] * sn * sn + c[todo, None] * ct * sn
            ok = trials[:, 1::2] * f_max[todo, None] <= f.clamp_min(0.0)
            first = ok.int().argmax(1)
            got = ok.any(1)
            at = todo[got]
            cp[at], sp[at], f_acc[at] = (t[got].gather(1, first[got][:, None])[:, 0] for t in (ct, sn, f))
            st["draw"].index_add_(0, todo, torch.where(got, 2 * first + 2, 12))
            todo = todo[~got]
            trials = uniforms(st["draw"][todo], st["photon"][todo], spec["seed"], precision, 12)
        ct, sn, zero = torch.cos(theta), torch.sin(theta), torch.zeros_like(theta)
        A = torch.stack([ct * cp, ct * sp, -sn, -sp, cp, zero, sn * cp, sn * sp, ct], 1).view(-1, 3, 3)
        J = torch.stack([s[:, 0] * cp, s[:, 0] * sp, -s[:, 1] * sp, s[:, 1] * cp], 1).view(-1, 2, 2)
        if event >= 2:                                                # interior product of the path
            T = st["J"] @ st["T"]
            st["T"] = T / T.abs().square().sum((1, 2), keepdim=True).sqrt()
        st["Pn1"], st["P"] = st["P"], A @ st["P"]
        st["E"] = (J @ st["E"][:, :, None])[:, :, 0] / f_acc.sqrt()[:, None]
        st["pos"] = st["rn"] = pos
        st["J"] = J
        if event == 0:
            st["r1"], st["P1"] = pos, st["P"]
        w = st["w"] * albedo
        low = w < 1e-4
        u = uniforms(st["draw"], st["photon"], spec["seed"], precision, 1)[:, 0]
        st["draw"] = st["draw"] + low.long()
        st["w"] = torch.where(low, w / 0.1, w)
        keep = (~low | (u < 0.1)) & (event + 1 <= spec["max_events"])
        st = {k: v[keep] for k, v in st.items()}
    return grids.cpu().numpy().reshape(8, n_theta, 1), hits
