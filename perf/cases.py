"""Workloads that the framework's speed is measured on, through its public
entry points (tfm_gb300.ccpgpu, tfm_gb300.surrogate).

Kinds of case ("kind"):
  forces   set_positions + forces of one system: what an external integrator
           or a check of a configuration calls; latency and launches count
  steps    advance + synchronize + positions of resident systems: the
           simulation loop (one ccp system, or an ensemble of replicas)
  frame    set_positions, one run of steps with a contact-map observation at
           its start, then the maps and the positions: one frame of the
           contact-map protocols
  observe  contact map, contact counts and distance sums by separation of one
           configuration: what ccp-analyze does for every trajectory frame
  walk     the confined random walk that starts every simulation
  predict  the surrogate network's contact maps of new sequences
  screen   the surrogate's P(s) of many sequences, reduced on the device
  grad     the surrogate's training loss and gradients on a batch of rows

Positions are made from the seed alone: a folded chain that fills the nucleus
at the model's density with bonds of about one sigma, every replica its own
orientation, zigzag and jitter; bead types come in blocks and lamina sites
cover the wall evenly.
"""
import math

import numpy as np
import torch

from tfm_gb300 import ccpgpu, surrogate

CCP_CHROMOSOMES = (0, 2284, 4599, 6687, 9338, 12508, 15193, 17477, 19792, 21880, 24531, 27701,
                   30386)


def listed():
    return [
        # forces of one small ccp system from host positions: the smallest call
        dict(name="forces-ccp-2048", kind="forces", preset="ccp", n=2048, chains=1),
        # ccp-profile's smallest benchmark shape, stepped on the device
        dict(name="steps-ccp-1024", kind="steps", preset="ccp", systems=1, n=1024, n_max=1024,
             chains=1, steps=100),
        # ccp's production model: 30386 beads in 12 chromosomes
        dict(name="steps-ccp-30386", kind="steps", preset="ccp", systems=1, n=30386, n_max=30386,
             chains=12, steps=50),
        # one chain of 2048 beads with a 2048^2 contact map every 100 steps
        dict(name="frame-chain-2048", kind="frame", preset="baseline", systems=1, n=2048, chains=1,
             bins=2048, steps=100),
        # one large system: 131072 beads in 16 chains, 1024^2 contact map
        dict(name="frame-single-131072", kind="frame", preset="baseline", systems=1, n=131072,
             chains=16, bins=1024, steps=32),
        # the batched ensemble: 512 replicas of 1024 to 16384 beads
        dict(name="steps-ensemble-512", kind="steps", preset="baseline", systems=512, n=1024,
             n_max=16384, chains=1, steps=20),
        # training data of the surrogate: equal 1024-bead replicas, 256^2 maps
        dict(name="frame-128x1024", kind="frame", preset="baseline", systems=128, n=1024, chains=1,
             bins=256, steps=100),
        # ccp-analyze on ccp's production model
        dict(name="observe-ccp-30386", kind="observe", preset="ccp", n=30386, chains=12),
        # start of a small ensemble's simulations
        dict(name="walk-64x2048", kind="walk", preset="baseline", systems=64, n=2048),
        # one new sequence: latency of a prediction
        dict(name="predict-1", kind="predict", seq_len=1024, bins=256, batch=32, count=1),
        # screening: sequences in, P(s) out, the last batch incomplete
        dict(name="screen-300", kind="screen", seq_len=1024, bins=256, batch=128, count=300),
        # one training batch of the default network
        dict(name="grad-32", kind="grad", seq_len=1024, bins=256, batch=32, count=32),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["forces", "steps", "steps", "ensemble", "frame", "frames", "observe", "walk",
                       "predict", "screen", "grad"])
    preset = rng.choice(["ccp", "baseline"])
    if kind == "forces":
        return dict(kind="forces", preset=preset, n=log(512, 32768), chains=rng.choice([1, 1, 3, 12]))
    if kind == "steps":
        return dict(kind="steps", preset=preset, systems=1, n=log(1024, 99000), n_max=0,
                    chains=rng.choice([1, 1, 2, 12, 16]), steps=rng.randint(24, 100))
    if kind == "ensemble":
        lo = log(700, 6000)
        return dict(kind="steps", preset=preset, systems=log(2, 400 if preset == "baseline" else 40), n=lo,
                    n_max=rng.randint(lo, 12000), chains=1, steps=rng.randint(10, 25))
    if kind == "frame":
        n = log(1024, 120000)
        return dict(kind="frame", preset="baseline", systems=1, n=n, chains=rng.choice([1, 2, 16]),
                    bins=min(n, rng.choice([256, 1000, 2048])), steps=rng.randint(20, 60))
    if kind == "frames":
        return dict(kind="frame", preset="baseline", systems=log(2, 128), n=log(800, 3000), chains=1,
                    bins=rng.choice([200, 256]), steps=rng.randint(30, 100))
    if kind == "observe":
        return dict(kind="observe", preset=preset, n=log(2048, 33000), chains=rng.choice([1, 2, 12]))
    if kind == "walk":
        return dict(kind="walk", preset="baseline", systems=log(1, 200), n=log(500, 2500))
    seq_len, bins = rng.choice([(256, 128), (512, 256), (1024, 128), (1024, 256)])
    if kind == "predict":
        return dict(kind="predict", seq_len=seq_len, bins=bins, batch=rng.choice([8, 32, 128]),
                    count=log(1, 140))
    if kind == "screen":
        return dict(kind="screen", seq_len=seq_len, bins=bins, batch=rng.choice([32, 128]),
                    count=log(20, 300))
    batch = rng.randint(3, 32)
    return dict(kind="grad", seq_len=seq_len, bins=bins, batch=batch, count=batch)


# ---------------------------------------------------------------- inputs

def _rotation(rng):
    q, r = np.linalg.qr(rng.standard_normal((3, 3)))
    return q * np.sign(np.diag(r))


def _close(x, r):
    """Pairs (i, j), |i - j| > 1, closer than r."""
    c = np.floor(x / r).astype(np.int64) + 512
    key = (c[:, 2] * 1024 + c[:, 1]) * 1024 + c[:, 0]
    order = np.argsort(key, kind="stable")
    ks, xs = key[order], x[order]
    found = []
    for dz in (0, 1):
        for dy in (-1, 0, 1) if dz else (0, 1):
            # three cells in a row, or from the own cell on
            own = not dz and not dy
            at = ks + (dz * 1024 + dy) * 1024
            lo = np.arange(1, len(ks) + 1) if own else np.searchsorted(ks, at - 1)
            cnt = np.searchsorted(ks, at + 1, side="right") - lo
            i = np.repeat(np.arange(len(ks)), cnt)
            j = np.arange(len(i)) - np.repeat(np.cumsum(cnt) - cnt, cnt) + np.repeat(lo, cnt)
            near = ((xs[i] - xs[j]) ** 2).sum(1) < r * r
            found.append(np.stack([order[i[near]], order[j[near]]]))
    i, j = np.concatenate(found, 1)
    far = np.abs(i - j) > 1
    return i[far], j[far]


def _chain(n, R, rng, apart):
    """A folded chain of n beads in a sphere of radius R: rows across the
    sphere walked back and forth, beads at about 0.72 sigma along the walk
    and displaced sideways by turns, so that bonds are close to one sigma."""
    r_in = R - 1.0
    a = math.sqrt(4.0 / 3.0 * math.pi * r_in ** 3 / (0.72 * n))
    for _ in range(6):
        k = np.arange(-int(r_in / a) - 1, int(r_in / a) + 2) * a
        z, y = np.meshgrid(k, k, indexing="ij")
        y[1::2] = y[1::2, ::-1]
        z, y = z.ravel(), y.ravel()
        h2 = r_in ** 2 - y ** 2 - z ** 2
        ok = h2 > 0.5
        y, z, h = y[ok], z[ok], np.sqrt(h2[ok])
        sgn = np.where(np.arange(len(h)) % 2 == 0, 1.0, -1.0)
        end = np.append(np.minimum(h[1:], h[:-1]), h[-1])  # rows turn where the next one begins
        beg = np.append(h[:1], end[:-1])
        v = np.stack([np.stack([-beg * sgn, y, z], 1), np.stack([end * sgn, y, z], 1)], 1).reshape(-1, 3)
        s = np.concatenate([[0.0], np.cumsum(np.linalg.norm(np.diff(v, axis=0), axis=1))])
        step = s[-1] / n
        if abs(step - 0.72) < 0.01:
            break
        a *= math.sqrt(step / 0.72)
    at = (np.arange(n) + 0.5) * step
    x = np.stack([np.interp(at, s, v[:, c]) for c in range(3)], 1)
    # sideways: across the walk, less where it turns
    t = np.empty_like(x)
    t[1:-1] = x[2:] - x[:-2]
    t[0], t[-1] = 2 * (x[1] - x[0]), 2 * (x[-1] - x[-2])
    l = np.linalg.norm(t, axis=1, keepdims=True) + 1e-9
    side = np.repeat(rng.standard_normal(((n + 1) // 2, 3)), 2, 0)[:n]
    side -= (side * t).sum(1, keepdims=True) / l ** 2 * t
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    side *= np.where(np.arange(n) % 2 == 0, 1.0, -1.0)[:, None] * np.clip(2.5 * l / (2 * step) - 1.5, 0.0, 1.0)
    x += 0.5 * math.sqrt(max(0.0, 1.0 - min(step, 1.0) ** 2)) * side
    x += 0.02 * rng.standard_normal((n, 3))
    # beads brought together by turns move apart: neighbours but one along the
    # chain, and with `apart` every pair
    i, j = _close(x, 1.5) if apart else (np.arange(n - 2), np.arange(2, n))
    b = np.arange(n - 1)
    for _ in range(12 if apart else 3):
        for p, q, lo, hi in ((i, j, 1.0, 9.0), (b, b + 1, 0.85, 1.15)):
            v = x[q] - x[p]
            d = np.linalg.norm(v, axis=1)
            k = np.nonzero((d < lo) | (d > hi))[0]
            v = v[k] * (0.5 - 0.5 * np.clip(d[k], lo, hi) / (d[k] + 1e-9))[:, None]
            for c in range(3):
                x[:, c] += np.bincount(p[k], v[:, c], n) - np.bincount(q[k], v[:, c], n)
    d = np.linalg.norm(x, axis=1, keepdims=True)
    x *= np.minimum(1.0, (R - 0.95) / d)
    return (x @ _rotation(rng).T).astype(np.float32)


def _model(preset):
    """Constants of the two force fields as the engine holds them (FP32)."""
    f = np.float32
    if preset == "ccp":
        rco, dt = f(1.154701), f(1.0 / 2048)
        return dict(wf=True, bend_all=False, k_e=128.0, k_b=1.0, e_att=0.5, e_rep=0.5,
                    rc_rep=float(rco), rc_att=2.0, e_w=1.0, rc_w=float(rco), depth=rco, cap=0.0,
                    dt=float(dt), sd=float(f(math.sqrt(2.0 * float(f(0.003356)) * 298.0 / 2048))))
    wca = f(2.0) ** f(1.0 / 6.0)
    dt = f(1e-3)
    return dict(wf=False, bend_all=True, k_e=100.0, k_b=2.0, e_att=0.5, e_rep=1.0,
                rc_rep=float(wca), rc_att=2.5, e_w=1.0, rc_w=float(wca), depth=wca, cap=0.1,
                dt=float(dt), sd=float(f(math.sqrt(2.0 * float(dt)))))


def _radius(preset, n):
    """Nucleus radius: ccp's chromatin volume fraction 0.2 (0.125 for the
    shapes of its benchmark below 30000 beads), the baseline's packing
    fraction 0.2."""
    if preset == "ccp":
        cvf = 0.2 if n >= 30000 else 0.125
        return float(np.float32("%.6f" % (1.154701 / 2 * (1 + (n / cvf) ** (1 / 3)))))
    return float(np.float32(0.5 * np.cbrt(n / float(np.float32(0.2)))))


def _lamina(case, R):
    """Number of lamina sites: a quarter of the wall's area (an ensemble of
    the ccp preset has none unless its text gives a number)."""
    if case["preset"] == "ccp" and case.get("systems", 1) > 1:
        return 0
    ratio = np.float32(0.5) / (np.float32(R) - _model(case["preset"])["depth"])
    return int(math.floor(0.25 * 4.0 / float(ratio) ** 2))


def _types(preset, n, rng):
    mean = 21.0 if preset == "ccp" else 16.0
    t = (rng.integers(0, 2) + np.cumsum(rng.random(n) < 1.0 / mean)) & 1
    if preset == "baseline":
        t = t | (rng.random(n) < 0.1).astype(t.dtype) << 1
    return t.astype(np.int32)


def _sizes(case, seed):
    k, lo, hi = case.get("systems", 1), case["n"], case.get("n_max", 0)
    if k == 1 or hi <= lo:
        return [lo] * k
    rng = np.random.default_rng(2026)  # the ensemble's shape, not its values
    return [int(v) for v in np.exp(rng.uniform(math.log(lo), math.log(hi), k))]


def _heads(case, n):
    c = case.get("chains", 1)
    if c == 12 and n == 30386 and case["preset"] == "ccp":
        return list(CCP_CHROMOSOMES[:-1])
    return [k * (n // c) for k in range(c)]


def _systems(case, seed):
    """Every system's beads, types and lamina sites."""
    out = []
    # the ccp steps have no cap: no overlaps there
    apart = case["preset"] == "ccp" or case.get("systems", 1) == 1
    for k, n in enumerate(_sizes(case, seed)):
        rng = np.random.default_rng([seed & 0x7FFFFFFF, k])
        R = _radius(case["preset"], n)
        m = _lamina(case, R)
        i = np.arange(m) + 0.5
        cz, ph = 1.0 - 2.0 * i / max(m, 1), i * math.pi * (1.0 + math.sqrt(5.0))
        sz = np.sqrt(np.maximum(0.0, 1.0 - cz ** 2))
        lbs = np.stack([sz * np.cos(ph), sz * np.sin(ph), cz], 1) @ _rotation(rng).T
        out.append(dict(n=n, R=R, x=_chain(n, R, rng, apart), types=_types(case["preset"], n, rng),
                        lbs=((R - float(_model(case["preset"])["depth"])) * lbs).astype(np.float32),
                        heads=_heads(case, n), seed=seed * 1000 + k))
    return out


def _engine(case, systems):
    preset, bins = case["preset"], case.get("bins", 0)
    text = "force_field %s\n" % preset
    if bins:
        text += "contact_bins %d\n" % bins
    if preset == "ccp":
        q = systems[0]
        text += "number_of_particles %d\nnucleus_radius %.6f\n" % (q["n"], q["R"])
    chains = case.get("chains", 1)
    if len(systems) == 1:
        if preset == "baseline":
            text += "number_of_particles %d\nnucleus_radius %.9g\n" % (systems[0]["n"], systems[0]["R"])
        text += "number_of_chains %d\nnumber_of_lbs %d\n" % (chains, _lamina(case, systems[0]["R"]))
        sim = ccpgpu.ChrSim(text, seed=systems[0]["seed"])
    else:
        sim = ccpgpu.Batch(text, [q["n"] for q in systems], n_chains=[chains] * len(systems),
                           radii=[q["R"] for q in systems], seeds=[q["seed"] for q in systems])
    if case["kind"] != "walk":
        sim.set_lbs(np.concatenate([q["lbs"] for q in systems]))
        sim.set_types(np.concatenate([q["types"] for q in systems]))
        sim.set_positions(np.concatenate([q["x"] for q in systems]))
    return sim


def _net_text(case):
    return "seq_len %d\nbins %d\nbatch %d\n" % (case["seq_len"], case["bins"], case["batch"])


DILATIONS = (1, 2, 4, 8, 1, 2)


def _layout(case):
    """(name, shape, standard deviation) of the network's parameters."""
    out = []
    for l in range(8):
        sd = math.sqrt(2 / 15) if l == 0 else math.sqrt(2 / 640) / math.sqrt(8)
        out += [("e%dw" % l, (5, 128, 64 if l == 0 else 128), sd), ("e%db" % l, (128,), 0.05)]
    out += [("pw", (128, 128), 0.04), ("pb", (128,), 0.05), ("E", (case["bins"], 64), 0.1)]
    for l in range(6):
        out += [("h%dw" % l, (9, 64, 64), math.sqrt(2 / 576) / math.sqrt(6)), ("h%db" % l, (64,), 0.05)]
    return out + [("wo", (64,), 0.1), ("bo", (1,), 0.0)]


def _net_data(case, seed):
    """Weights of a trained network's size, sequences of mean block length 4
    to 64 with 10 % lamina-binding beads, and noisy maps that fall off with
    the separation."""
    rng = np.random.default_rng([seed & 0x7FFFFFFF, 77])
    parts = []
    for name, shape, sd in _layout(case):
        w = sd * rng.standard_normal(shape)
        if name == "e0w":
            w[:, :, 3:] = 0.0
        parts.append(np.full(1, -5.0) if name == "bo" else w.ravel())
    n, L, M = case["count"], case["seq_len"], case["bins"]
    p = 1.0 / rng.uniform(4.0, 64.0, (n, 1))
    types = ((rng.integers(0, 2, (n, 1)) + np.cumsum(rng.random((n, L)) < p, 1)) & 1).astype(np.uint8)
    lad = (rng.random((n, L)) < 0.1).astype(np.uint8)
    maps = None
    if case["kind"] == "grad":
        i = np.arange(M)
        mean = 0.4 / (1.0 + np.abs(i[:, None] - i[None, :])) ** 1.2
        maps = rng.poisson(100.0 * np.broadcast_to(mean, (n, M, M))) / 100.0
        maps = np.tril(maps) + np.transpose(np.tril(maps, -1), (0, 2, 1))
        maps = np.minimum(maps, 1.0).astype(np.float32)
    return np.concatenate(parts).astype(np.float32), types, lad, maps


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("predict", "screen", "grad"):
        net = surrogate.Surrogate(_net_text(case), seed=1)
        params, types, lad, maps = _net_data(case, seed)
        if kind == "grad":
            net.set_dataset(types, lad, maps)
        net.set_params(params)
        rows = np.arange(case["count"], dtype=np.int32)
        return dict(case=case, net=net, types=types, lad=lad, rows=rows)
    if kind == "walk":
        systems = [dict(n=n, R=_radius(case["preset"], n), lbs=[], seed=seed * 1000 + k)
                   for k, n in enumerate(_sizes(case, seed))]
        return dict(case=case, sim=_engine(case, systems))
    systems = _systems(case, seed)
    sim = _engine(case, systems)
    return dict(case=case, sim=sim, x=np.concatenate([q["x"] for q in systems]),
                lengths=[b - a for q in systems for a, b in zip(q["heads"], q["heads"][1:] + [q["n"]])])


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "predict":
        return {"maps": state["net"].predict(state["types"], state["lad"])}
    if kind == "screen":
        return {"ps": state["net"].predict_ps(state["types"], state["lad"])}
    if kind == "grad":
        loss = state["net"].loss_grad(state["rows"])
        return {"grads": state["net"].grads(), "loss": np.float32(loss)}
    sim = state["sim"]
    if kind == "forces":
        sim.set_positions(state["x"])
        return {"forces": sim.forces()}
    if kind == "steps":
        sim.advance(case["steps"])
        sim.synchronize()
        return {"positions": sim.positions()}
    if kind == "frame":
        sim.set_positions(state["x"])
        sim.reset_observables()
        sim.advance(case["steps"], case["steps"])
        sim.synchronize()
        return {"counts": np.concatenate([sim.contact_counts(k) for k in range(case["systems"])]),
                "positions": sim.positions()}
    if kind == "observe":
        sim.set_positions(state["x"])
        sim.reset_observables()
        sim.observe(with_sdist=True)
        sep = [sim.separation_counts(c, n) for c, n in enumerate(state["lengths"])]
        return {"map": sim.contact_counts(0), "contacts": np.concatenate([c for c, _ in sep]),
                "distances": np.concatenate([d for _, d in sep]), "sums": sim.observable_sums(0)}
    draws = sim.random_walk()
    return {"draws": draws, "positions": sim.positions()}


def work(case):
    kind = case["kind"]
    if kind in ("predict", "screen", "grad"):
        n, L, M = case["count"], case["seq_len"], case["bins"]
        # encoder (the first layer has three input channels), projection,
        # pair features, head and output layer of one map, forward
        fl = 2 * L * 5 * 128 * (3 + 7 * 128) + 2 * M * 128 * 128 + 4 * 64 * M * M
        fl += 6 * 2 * 9 * 64 * 64 * M * M + 128 * M * M
        weights = 4 * sum(int(np.prod(s)) for _, s, _ in _layout(case))
        out = {"predict": 4 * n * M * M, "screen": 4 * n * M, "grad": 4 * n * M * M + weights}[kind]
        return {"bytes": 2 * n * L + weights + out, "flops": (3 if kind == "grad" else 1) * n * fl}
    sizes = _sizes(case, 0)
    beads, f = float(sum(sizes)), 0.0
    m = _model(case["preset"])
    for n in sizes:
        # unordered pairs within the cutoffs (half of the beads attract)
        rho = n / (4 / 3 * math.pi * _radius(case["preset"], n) ** 3)
        pairs = 0.5 * rho * 4 / 3 * math.pi * (0.25 * m["rc_att"] ** 3 + 0.75 * m["rc_rep"] ** 3)
        f += n * (30 * pairs + 200)
    if kind == "forces":
        return {"bytes": 24 * beads, "flops": f}
    if kind == "walk":
        return {"bytes": 24 * beads, "flops": 200 * beads}
    if kind == "observe":
        rho = beads / (4 / 3 * math.pi * _radius(case["preset"], case["n"]) ** 3)
        L = beads / case["chains"]
        contacts = 0.5 * beads * rho * 4 / 3 * math.pi * 8
        bins = beads / (8 if len(_heads(case, case["n"])) == 12 else 4)
        return {"bytes": 12 * beads + 2 * bins ** 2 + 6 * beads,
                "flops": 10 * contacts + 10 * case["chains"] * 0.375 * L * L}
    # one Heun step reads and writes 192 bytes of a bead's state (positions,
    # predictor, forces and cell lists of both stages) where the state does
    # not stay on the chip
    b = 192.0 * beads * case["steps"] + 24 * beads
    if kind == "frame":
        b += 2.0 * case["bins"] ** 2 * case["systems"]
    return {"bytes": b, "flops": case["steps"] * (2 * f + 100 * beads)}


# ---------------------------------------------------------------- the same in 64 bits

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pair_forces(x, het, m):
    """Sum over the pairs within the cutoffs, |i - j| > 1, in slabs of z."""
    order = torch.argsort(x[:, 2])
    xs, hs, n = x[order], het[order], len(x)
    zs = xs[:, 2].contiguous()
    out = torch.zeros_like(x)
    rc = max(m["rc_att"], m["rc_rep"])
    rows = max(64, min(n, (1 << 24) // max(1, min(n, 1 << 17))))
    lo = torch.searchsorted(zs, zs - rc).cpu().numpy()
    hi = torch.searchsorted(zs, zs + rc, right=True).cpu().numpy()
    for a in range(0, n, rows):
        b = min(n, a + rows)
        j0, j1 = int(lo[a]), int(hi[b - 1])
        d = xs[a:b, None, :] - xs[None, j0:j1, :]
        d2 = (d * d).sum(2)
        hh = hs[a:b, None] & hs[None, j0:j1]
        cut = torch.where(hh, m["rc_att"], m["rc_rep"]).to(d2.dtype)
        ok = (d2 <= cut * cut) & ((order[a:b, None] - order[None, j0:j1]).abs() > 1)
        s = torch.where(ok, d2, 1.0)
        if m["wf"]:
            c = m["e_att"] * 6 * (s - 4) * (3 * s - 4) / s ** 4
        else:
            e = torch.where(hh, m["e_att"], m["e_rep"]).to(d2.dtype)
            c = 24 * e * (2 / s ** 7 - 1 / s ** 4)
        c = torch.where(ok, c, 0.0)
        out[order[a:b]] = (c[:, :, None] * d).sum(1)
    return out


def _forces64(x, q, m):
    het, lad, first, lbs = q
    f = _pair_forces(x, het, m)
    # bonds inside chains and their angles
    bond = ~first[1:]
    with torch.enable_grad():
        y = x.clone().requires_grad_(True)
        v = y[1:] - y[:-1]
        d = torch.sqrt((v * v).sum(1))
        u = 0.5 * m["k_e"] * ((d - 1.0) ** 2 * bond).sum()
        fb = -torch.autograd.grad(u, y, retain_graph=True)[0]
        t = v / d[:, None]
        c = ((t[1:] * t[:-1]).sum(1) * (bond[1:] & bond[:-1])).sum()
        g = torch.autograd.grad(c, y)[0]
    f = f + fb + m["k_b"] * (g if m["bend_all"] else g * het[:, None])
    # wall
    d = torch.sqrt((x * x).sum(1))
    gap = m["R"] - d
    s = torch.where(gap <= m["rc_w"], gap, 1.0) ** 2
    c = 6 * m["e_w"] * (s - 4) * (3 * s - 4) / s ** 4 if m["wf"] else 24 * m["e_w"] * (2 / s ** 7 - 1 / s ** 4)
    c = torch.where(gap <= m["rc_w"], c, 0.0)
    f = f + (c * (1.0 - m["R"] / d))[:, None] * x
    # lamina sites
    k = torch.nonzero(lad).ravel()
    if len(k) and len(lbs):
        near = k[d[k] > m["R"] - float(m["depth"]) - 0.51]
        for part in torch.split(near, 4096):
            v = x[part][:, None, :] - lbs[None]
            n2 = (v * v).sum(2) / 0.25
            c = torch.where(n2 <= 1.0, 8.0 * (8.0 / 0.75) * (n2 ** 3 - 1.0), 0.0)
            f[part] += (c[:, :, None] * v).sum(1)
    return f


def _philox(c, key):
    """Philox4x32-10 of counters and keys, numbers or arrays."""
    M = np.uint64(0xFFFFFFFF)
    c = [np.asarray(v, np.uint64) for v in c]
    k0, k1 = (np.asarray(k, np.uint64) for k in key)
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(b >> np.uint64(32)) ^ c[1] ^ k0, b & M, (a >> np.uint64(32)) ^ c[3] ^ k1, a & M]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & M, (k1 + np.uint64(0xBB67AE85)) & M
    return c


def _noise(n, step, seed):
    z = np.zeros((n, 3))
    left = np.arange(n)
    attempt = 0
    while len(left):
        o = np.zeros_like(left)
        b = _philox([left, o + attempt, o + step, o], (seed & 0xFFFFFFFF, seed >> 32))
        u = [(v >> np.uint64(8)).astype(np.float64) for v in b]
        r0 = np.sqrt(-2 * np.log((u[0] + 1) / 16777216))
        r1 = np.sqrt(-2 * np.log((u[2] + 1) / 16777216))
        p0, p1 = 2 * math.pi * u[1] / 16777216, 2 * math.pi * u[3] / 16777216
        z[left] = np.stack([r0 * np.cos(p0), r0 * np.sin(p0), r1 * np.cos(p1)], 1)
        left = left[(np.abs(z[left]) > 5).any(1)]
        attempt += 1
    return z


def _on_device(case, q):
    dev = _device()
    m = dict(_model(case["preset"]), R=float(np.float32(q["R"])))
    het = torch.tensor((q["types"] & 1) == 0, device=dev)
    lad = het if case["preset"] == "ccp" else torch.tensor((q["types"] & 2) != 0, device=dev)
    first = torch.zeros(q["n"], dtype=torch.bool, device=dev)
    first[q["heads"]] = True
    x = torch.tensor(q["x"], device=dev, dtype=torch.float64)
    return x, (het, lad, first, torch.tensor(q["lbs"], device=dev, dtype=torch.float64)), m


def _heun(case, q):
    x, parts, m = _on_device(case, q)

    def capped(d):
        if not m["cap"]:
            return d
        l = torch.sqrt((d * d).sum(1, keepdim=True))
        return d * torch.clamp(m["cap"] / torch.clamp(l, min=1e-30), max=1.0)

    for step in range(case["steps"]):
        z = m["sd"] * torch.tensor(_noise(q["n"], step, q["seed"]), device=x.device)
        f = _forces64(x, parts, m)
        e = _forces64(x + capped(f * m["dt"]) + z, parts, m)
        x = x + capped(0.5 * m["dt"] * (f + e)) + z
    return x


def _walk(case, seed):
    """The sequential rejection walk of every system, all systems at once."""
    n = case["n"]
    sizes = _sizes(case, seed)
    K = len(sizes)
    R = np.array([_radius(case["preset"], s) for s in sizes])
    seeds = seed * 1000 + np.arange(K, dtype=np.int64)
    keys = (seeds & 0xFFFFFFFF, seeds >> 32)
    mis, k_e, k_b = float(np.float32(0.95)), 100.0, 2.0
    c_b = 0.5 * k_b
    draw = np.zeros(K, np.int64)
    idx = np.zeros(K, np.int64)
    miss = np.zeros(K, np.int64)
    pos = np.zeros((K, n, 3))
    old, prev = np.zeros((K, 3)), np.zeros((K, 3))
    rows = np.arange(K)
    while (idx < n).any():
        o = np.zeros(K, np.int64)
        b = _philox([draw, o, o + 0x10057, o + 0x1C0DE], keys)
        u = [((v >> np.uint64(8)).astype(np.float64) + 1) / 16777216 for v in b]
        ct = 1 - 2 * u[0]
        st = np.sqrt(np.maximum(0, 1 - ct * ct))
        d = np.stack([st * np.cos(2 * math.pi * u[1]), st * np.sin(2 * math.pi * u[1]), ct], 1)
        start = idx == 0
        p0 = ((R - mis) * np.cbrt(u[2]))[:, None] * d
        with np.errstate(all="ignore"):
            per = np.cross(old, d)
            per /= np.linalg.norm(per, axis=1, keepdims=True)
            cb = np.clip(1 + np.log1p(-(1 - math.exp(-2 * c_b)) * u[2]) / c_b, -1, 1)
            nd = cb[:, None] * old + np.sqrt(1 - cb * cb)[:, None] * per
            lb = 1.0 + math.sqrt(2 / k_e) * torch.erfinv(torch.tensor(2 * u[3] - 1)).numpy()
            p = lb[:, None] * nd + prev
        p = np.where(start[:, None], p0, p)
        nd = np.where(start[:, None], d, nd)
        live = idx < n
        ok = live & (start | (np.isfinite(p).all(1) & ~(R - np.linalg.norm(p, axis=1) < mis)))
        pos[rows[live], idx[live]] = p[live]
        draw[live] += 1
        old[ok], prev[ok] = nd[ok], p[ok]
        miss = np.where(ok, 0, miss + 1)
        idx = np.where(ok, idx + 1, idx)
        back = live & ~ok & (miss > 1024)
        for k in np.nonzero(back)[0]:
            idx[k] = 2 + idx[k] * 3 // 4
            prev[k] = pos[k, idx[k] - 1]
    return {"draws": draw, "positions": pos.reshape(-1, 3)}


def _network(p, case, types, lad):
    """y [n][M][M] in FP64, channels first."""
    F = torch.nn.functional
    L, M, f = case["seq_len"], case["bins"], case["seq_len"] // case["bins"]
    t = torch.as_tensor(types, device=_device())
    x = torch.stack([t == 0, t == 1, torch.as_tensor(lad, device=t.device) != 0], 1).double()
    h = F.relu(F.conv1d(x, p["e0w"][:, :, :3].permute(1, 2, 0), p["e0b"], padding=2))
    for l in range(1, 8):
        h = h + F.relu(F.conv1d(h, p["e%dw" % l].permute(1, 2, 0), p["e%db" % l], padding=2))
    hp = h.reshape(len(t), 128, M, f).mean(3)
    uv = torch.einsum("bcm,oc->bom", hp, p["pw"]) + p["pb"][:, None]
    u, v = uv[:, :64], uv[:, 64:]
    i = torch.arange(M, device=t.device)
    dist = p["E"][(i[:, None] - i[None, :]).abs()].permute(2, 0, 1)
    z = u[:, :, :, None] * v[:, :, None, :] + u[:, :, None, :] * v[:, :, :, None] + dist
    for l, d in enumerate(DILATIONS):
        w = p["h%dw" % l].reshape(3, 3, 64, 64).permute(2, 3, 0, 1)
        z = z + F.relu(F.conv2d(z, w, p["h%db" % l], padding=d, dilation=d))
    y = torch.einsum("bcij,c->bij", z, p["wo"]) + p["bo"]
    return 0.5 * (y + y.transpose(1, 2))


def _parameters(case, flat, grad):
    leaf = torch.tensor(flat, dtype=torch.float64, device=_device(), requires_grad=grad)
    p, o = {}, 0
    for name, shape, _ in _layout(case):
        k = int(np.prod(shape))
        p[name] = leaf[o:o + k].view(*shape)
        o += k
    return leaf, p


def _surrogate64(case, seed):
    flat, types, lad, maps = _net_data(case, seed)
    leaf, p = _parameters(case, flat, case["kind"] == "grad")
    n, M = case["count"], case["bins"]
    if case["kind"] != "grad":
        out = []
        with torch.no_grad():
            for a in range(0, n, 4):
                y = _network(p, case, types[a:a + 4], lad[a:a + 4])
                m = torch.exp(torch.clamp(y, max=0.0))
                if case["kind"] == "screen":
                    m = torch.stack([torch.diagonal(m, s, 1, 2).mean(1) for s in range(M)], 1)
                out.append(m.cpu().numpy())
        return {"maps" if case["kind"] == "predict" else "ps": np.concatenate(out)}
    i = np.arange(M)
    dist = np.abs(i[:, None] - i[None, :])
    pairs = np.bincount(dist.ravel(), minlength=M).astype(np.float64)
    mean = np.bincount(dist.ravel(), weights=maps.astype(np.float64).sum(0).ravel(), minlength=M) / (n * pairs)
    w = torch.tensor((M / (np.maximum(mean, 1e-6) * pairs))[dist], device=leaf.device)
    total = 0.0
    for a in range(0, n, 2):
        t = torch.tensor(maps[a:a + 2], dtype=torch.float64, device=leaf.device)
        ys = _network(p, case, types[a:a + 2], lad[a:a + 2])
        yh = ys - (ys - torch.clamp(ys, max=0.0)).detach()
        loss = (w * (torch.exp(yh) - t - t * yh + torch.xlogy(t, t))).sum() / (n * M * M)
        loss.backward()
        total += float(loss.detach())
    return {"grads": leaf.grad.cpu().numpy(), "loss": np.float64(total)}


def _observables64(case, q):
    """Distance sums by separation and the radial profile of one frame."""
    x = torch.tensor(q["x"], dtype=torch.float64, device=_device())
    dist = []
    for a, b in zip(q["heads"], q["heads"][1:] + [q["n"]]):
        c = x[a:b]
        s = np.zeros((b - a) // 2 + 1)
        for k in range(1, len(s)):
            s[k] = float(torch.sqrt(((c[k:] - c[:-k]) ** 2).sum(1)).sum())
        dist.append(s)
    X = q["x"].astype(np.float64)
    R, a = float(np.float32(q["R"])), float(np.float32(1.154701 / 2))
    d = np.linalg.norm(X, axis=1)
    vol = np.zeros((65, q["n"]))
    for k in range(64):
        r = R * ((k + 1) / 64) ** (1 / 3)
        ca, cb = (d * d + a * a - r * r) / (2 * d * a), (r * r + d * d - a * a) / (2 * r * d)
        cap = math.pi / 3 * (a ** 3 * (2 + ca) * (1 - ca) ** 2 + r ** 3 * (2 + cb) * (1 - cb) ** 2)
        vol[k + 1] = np.where(d - a > r, 0.0, np.where(d + a < r, 4 / 3 * math.pi * a ** 3, cap))
    shell = np.diff(vol, axis=0)
    het = (q["types"] & 1) == 0
    sums = np.concatenate([X.sum(0), [(X * X).sum()], shell[:, het].sum(1), shell[:, ~het].sum(1), shell.sum(1)])
    return {"map": None, "contacts": None, "distances": np.concatenate(dist), "sums": sums}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("predict", "screen", "grad"):
        return _surrogate64(case, seed)
    if kind == "walk":
        return _walk(case, seed)
    if kind in ("steps", "frame"):
        beads = sum(_sizes(case, seed))
        if case.get("systems", 1) > 1 and case["systems"] * case["steps"] > 400 or beads * case["steps"] > 5e6:
            return None  # minutes
        x = torch.cat([_heun(case, q) for q in _systems(case, seed)]).cpu().numpy()
        return {"positions": x} if kind == "steps" else {"counts": None, "positions": x}
    q = _systems(case, seed)[0]
    if kind == "observe":
        return _observables64(case, q)
    return {"forces": _forces64(*_on_device(case, q)).cpu().numpy()}
