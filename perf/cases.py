"""The work that this engine is used for, as cases that can be timed and compared.

Each case is one pass of a user's program: advance a GPU-resident system by a few steps and read
the snapshot back into pinned host memory, evaluate forces with potentials, train or apply the
learned pair correction, or sort device-resident pairs.  Systems are seeded synthetic stand-ins
(Plummer and Hernquist spheres, Zel'dovich-displaced lattices) drawn on the GPU, at the sizes and
settings of the benchmark's workloads and at smaller and ragged ones.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from blitzar_b200._lib import Engine, load

ASSIGN = {"cic": 0, "tsc": 1, "pcs": 2}


def listed():
    return [
        # a small cluster in the reference's default integrator, a few dozen steps a snapshot:
        # launch and latency bound
        {"name": "octree_4k", "kind": "octree", "ic": "plummer", "n": 4096, "theta": 0.5, "eps": 0.01,
         "dt": 1e-3, "steps": 16, "integrator": 1},
        # the benchmark's Plummer 65k leapfrog run
        {"name": "octree_65k", "kind": "octree", "ic": "plummer", "n": 65536, "theta": 0.5,
         "eps": 0.01, "dt": 1e-3, "steps": 8, "integrator": 0},
        # the benchmark's Hernquist 4M run: the largest open-boundary system
        {"name": "octree_4m", "kind": "octree", "ic": "hernquist", "n": 4194304, "theta": 0.4,
         "eps": 0.005, "dt": 2e-4, "steps": 2, "integrator": 0},
        # a diagnostic force evaluation with potentials of an odd-sized system
        {"name": "potential_200k", "kind": "potential", "ic": "plummer", "n": 200003, "theta": 0.5,
         "eps": 0.01},
        # periodic TreePM at the settings that hold 1e-3 force error (mesh of twice the lattice,
        # PCS, analytic differentiation): a small box
        {"name": "treepm_64", "kind": "treepm", "n_side": 64, "mesh": 128, "rs": 1.0, "rcf": 5.0,
         "assign": "pcs", "gradient": 2, "node": 0.5, "order": 1, "theta": 0.5, "leaf": 16,
         "dt": 2e-5, "steps": 8},
        # the reference's literal mesh (128^3 CIC, centred differences, multipoles in the cutoff)
        {"name": "treepm_128_cic", "kind": "treepm", "n_side": 128, "mesh": 128, "rs": 1.25,
         "rcf": 4.5, "assign": "cic", "gradient": 0, "node": 0.0, "order": 2, "theta": 0.5, "leaf": 16,
         "dt": 1e-4, "steps": 4},
        # the benchmark's headline box: 256^3 particles, 512^3 mesh
        {"name": "treepm_256", "kind": "treepm", "n_side": 256, "mesh": 512, "rs": 0.95, "rcf": 5.0,
         "assign": "pcs", "gradient": 2, "node": 0.5, "order": 1, "theta": 0.5, "leaf": 48,
         "dt": 5e-4, "steps": 4},
        # the reference's own open-boundary GPU TreePM at its defaults on a 1M Plummer sphere
        {"name": "treepm_open_1m", "kind": "treepm_open", "n": 1048576, "grid": 64, "cut": 1.0,
         "assign": "cic", "gradient": 0, "theta": 0.5, "eps": 0.01, "dt": 1e-3, "steps": 2},
        # an ensemble of independent clusters with adaptive power-of-two block steps
        {"name": "ensemble_96", "kind": "ensemble", "systems": 96, "n_min": 256, "n_max": 16384,
         "a_min": 0.1, "theta": 0.5, "eps": 0.01, "dt": 1e-3, "levels": 6, "eta": 0.02, "steps": 1},
        # TreePM steps with the learned pair correction applied (r_s = 0.8 cell)
        {"name": "learned_64", "kind": "learned", "n_side": 64, "mesh": 128, "rs": 0.8, "rcf": 5.0,
         "dt": 2e-5, "steps": 4},
        # training the correction: Adam on residual samples, then the trained weights
        {"name": "train_128k", "kind": "train", "n": 131072, "steps": 200, "batch": 4096},
        # sorting device-resident (key, value) pairs without allocations, at the full 2^20 - odd
        {"name": "sort_1m", "kind": "sort", "n": 1000003, "bits": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["octree", "octree", "treepm", "treepm", "treepm", "potential", "treepm_open",
                       "ensemble", "learned", "train", "sort"])
    if kind == "octree":
        n = _log_int(rng, 2000, 2000000)
        return {"kind": kind, "ic": rng.choice(["plummer", "hernquist"]), "n": n,
                "theta": round(rng.uniform(0.4, 0.7), 3), "eps": round(rng.uniform(0.005, 0.02), 4),
                "dt": 5e-4, "steps": max(1, min(16, 2000000 // n)), "integrator": rng.randint(0, 1)}
    if kind == "potential":
        return {"kind": kind, "ic": rng.choice(["plummer", "hernquist"]), "n": _log_int(rng, 5000, 1000000),
                "theta": round(rng.uniform(0.4, 0.7), 3), "eps": round(rng.uniform(0.005, 0.02), 4)}
    if kind == "treepm":
        side = _log_int(rng, 20, 200)
        mesh = 1 << max(5, (side - 1).bit_length())
        gradient = rng.randint(0, 2)
        capped = rng.random() < 0.7
        return {"kind": kind, "n_side": side, "mesh": mesh * (2 if rng.random() < 0.5 and mesh < 256 else 1),
                "rs": round(rng.uniform(0.8, 1.3), 3), "rcf": round(rng.uniform(4.5, 5.0), 2),
                "assign": rng.choice(["cic", "tsc", "pcs"]), "gradient": gradient,
                "node": 0.5 if capped else 0.0, "order": 1 if capped else 2, "theta": 0.5,
                "leaf": rng.choice([16, 32, 48]), "dt": 2e-5,
                "steps": max(1, min(8, 4000000 // side ** 3))}
    if kind == "treepm_open":
        return {"kind": kind, "n": _log_int(rng, 20000, 1000000), "grid": rng.choice([32, 48, 64, 100, 128]),
                "cut": round(rng.uniform(1.0, 2.0), 2), "assign": rng.choice(["cic", "tsc", "pcs"]),
                "gradient": rng.randint(0, 2), "theta": round(rng.uniform(0.4, 0.7), 3), "eps": 0.01,
                "dt": 1e-3, "steps": 1}
    if kind == "ensemble":
        return {"kind": kind, "systems": rng.randint(3, 96), "n_min": 200, "n_max": _log_int(rng, 2000, 16384),
                "a_min": round(rng.uniform(0.1, 0.5), 3), "theta": round(rng.uniform(0.4, 0.7), 3),
                "eps": 0.01, "dt": 1e-3, "levels": rng.randint(3, 6), "eta": 0.02, "steps": 1}
    if kind == "learned":
        side = rng.randint(24, 96)
        return {"kind": kind, "n_side": side, "mesh": max(64, 1 << side.bit_length()), "rs": round(rng.uniform(0.7, 1.0), 3),
                "rcf": 5.0, "dt": 2e-5, "steps": 2}
    if kind == "train":
        return {"kind": kind, "n": _log_int(rng, 20000, 200000), "steps": rng.randint(20, 200),
                "batch": 128 * rng.randint(4, 64)}
    return {"kind": "sort", "n": _log_int(rng, 1000, 1048576), "bits": rng.choice([32, 48, 64, 64])}


# ------------------------------------------------------------------- seeded inputs, on the GPU

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed % 1000003) + 17)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _directions(g, n):
    v = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True)


def _plummer(g, n, a=1.0):
    """Plummer sphere of mass 1: radii by inverse CDF, speeds from the isotropic distribution
    function by its tabulated CDF."""
    u = _rand(g, n).clamp(1e-9, 0.999)
    r = a / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
    q = np.linspace(0.0, 1.0, 2001)
    cdf = np.concatenate([[0.0], np.cumsum(0.5 * np.diff(q) * ((w := q * q * (1 - q * q) ** 3.5)[1:] + w[:-1]))])
    cdf = torch.tensor(cdf / cdf[-1], device="cuda")
    t = _rand(g, n)
    k = torch.searchsorted(cdf, t).clamp(1, 2000)
    lo, hi = cdf[k - 1], cdf[k]
    speed = (k - 1 + (t - lo) / (hi - lo).clamp_min(1e-300)) / 2000.0 * torch.sqrt(2.0 / torch.sqrt(r * r + a * a))
    return r[:, None] * _directions(g, n), speed[:, None] * _directions(g, n)


def _hernquist(g, n, r_max=100.0):
    """Hernquist sphere of mass 1 truncated at r_max, isotropic speeds of half the escape speed on
    average."""
    s = torch.sqrt(_rand(g, n) * (r_max / (1.0 + r_max)) ** 2)
    r = s / (1.0 - s)
    speed = (0.25 + 0.5 * _rand(g, n)) * torch.sqrt(2.0 / (r + 1.0))
    return r[:, None] * _directions(g, n), speed[:, None] * _directions(g, n)


def _lattice(g, side, rms_cells=0.2):
    """side^3 particles of a unit periodic box displaced by a Zel'dovich field with P(k) ~ k^-2."""
    k1 = torch.fft.fftfreq(side, d=1.0 / side, device="cuda", dtype=torch.float64)
    kz = torch.fft.rfftfreq(side, d=1.0 / side, device="cuda", dtype=torch.float64)
    k2 = k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + kz[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    amp = 1.0 / k2.sqrt()
    amp[0, 0, 0] = 0.0
    white = torch.randn(side, side, side, generator=g, device="cuda", dtype=torch.float64)
    delta = torch.fft.rfftn(white) * amp / k2
    disp = torch.stack([torch.fft.irfftn(1j * k * delta, s=(side, side, side))
                        for k in (k1[:, None, None], k1[None, :, None], kz[None, None, :])], -1)
    disp *= rms_cells / side / math.sqrt(float((disp ** 2).sum(-1).mean()))
    x = (torch.arange(side, device="cuda", dtype=torch.float64) + 0.5) / side
    pos = torch.stack(torch.meshgrid(x, x, x, indexing="ij"), -1) + disp
    return torch.remainder(pos, 1.0).reshape(-1, 3), torch.zeros(side ** 3, 3, device="cuda", dtype=torch.float64)


def _sphere(case, seed):
    g = _gen(seed)
    return _hernquist(g, case["n"]) if case["ic"] == "hernquist" else _plummer(g, case["n"])


def _system(case, seed):
    """(positions, velocities, masses) on the GPU, FP64."""
    kind = case["kind"]
    if kind in ("treepm", "learned"):
        pos, vel = _lattice(_gen(seed), case["n_side"])
    elif kind == "treepm_open":
        pos, vel = _plummer(_gen(seed), case["n"])
    else:
        pos, vel = _sphere(case, seed)
    n = pos.shape[0]
    return pos, vel, torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float32)


def _ensemble(case, seed):
    g = _gen(seed)
    k = case["systems"]
    # sizes spread evenly over their logarithm (a largest one among the first), scale radii drawn
    q = (np.arange(k) * 0.6180339887 + 0.9) % 1.0
    sizes = np.rint(case["n_min"] * (case["n_max"] / case["n_min"]) ** q).astype(int)
    radii = np.exp(np.log(case["a_min"]) * _rand(g, k).cpu().numpy())
    out = []
    for n, a in zip(sizes.tolist(), radii.tolist()):
        p, v = _plummer(g, n, a)
        out.append((p.cpu().numpy(), v.cpu().numpy(), np.full(n, 1.0 / n, np.float32)))
    return out


def _config(case):
    kind = case["kind"]
    if kind in ("octree", "potential"):
        return dict(solver=0, octree_theta=case["theta"], octree_softening=case["eps"], multipole_order=2,
                    integrator=case.get("integrator", 0))
    if kind == "treepm":
        return dict(solver=1, box_length=1.0, treepm_grid_size=case["mesh"], treepm_r_split_cells=case["rs"],
                    treepm_r_cut_factor=case["rcf"], treepm_assignment=ASSIGN[case["assign"]],
                    treepm_gradient=case["gradient"], treepm_window_floor=0.0 if case["gradient"] else 0.08,
                    treepm_node_size_factor=case["node"], multipole_order=case["order"],
                    octree_theta=case["theta"], octree_softening=0.02 / case["n_side"], leaf_capacity=case["leaf"])
    if kind == "learned":
        return dict(solver=1, box_length=1.0, treepm_grid_size=case["mesh"], treepm_r_split_cells=case["rs"],
                    treepm_r_cut_factor=case["rcf"], treepm_assignment=2, treepm_gradient=2,
                    treepm_window_floor=0.0, treepm_node_size_factor=0.5, multipole_order=1,
                    octree_theta=0.5, octree_softening=0.02 / case["n_side"], leaf_capacity=16)
    if kind == "treepm_open":
        return dict(solver=1, box_length=0.0, treepm_grid_size=case["grid"], treepm_r_split_cells=case["cut"] / 4.5,
                    treepm_r_cut_factor=4.5, treepm_assignment=ASSIGN[case["assign"]],
                    treepm_gradient=case["gradient"], treepm_window_floor=0.08, octree_theta=case["theta"],
                    octree_softening=case["eps"], multipole_order=2)
    if kind == "ensemble":
        return dict(solver=0, octree_theta=case["theta"], octree_softening=case["eps"], multipole_order=2,
                    adaptive_max_level=case["levels"], adaptive_eta=case["eta"])
    return dict(solver=0)  # the MLP needs a handle, not a system


def _pinned(n, dtype=torch.float32):
    return torch.empty(n, dtype=dtype, pin_memory=True)


def _weights(g, scale):
    """MLP weights of the magnitude that training leaves (Xavier-scaled), biases small."""
    p = (2.0 * _rand(g, 1667) - 1.0).float()
    p[:512] *= math.sqrt(6.0 / 48)
    p[512:1536] *= math.sqrt(6.0 / 64)
    p[1536:1568] *= 0.1
    p[1568:1664] *= math.sqrt(6.0 / 35)
    p[1664:] *= 0.01
    return (p * scale).cpu().numpy()


def _residuals(case, seed):
    """Samples shaped like the mesh force residual: separations in a ball of four cells, source
    offsets in the cell, a target that decays with the separation and is periodic in the offsets."""
    g = _gen(seed)
    n = case["n"]
    sep = _directions(g, n) * (0.02 + 3.98 * _rand(g, n, 1) ** (1.0 / 3.0))
    off = _rand(g, n, 3)
    r2 = (sep ** 2).sum(1, keepdim=True)
    y = 0.02 * torch.exp(-0.4 * r2) * (sep + 0.5 * torch.sin(2 * math.pi * off) + 0.5 * torch.cos(2 * math.pi * (off + sep)))
    return torch.cat([sep, off], 1).float().cpu().numpy(), y.float().cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        g = _gen(seed)
        n = case["n"]
        keys = torch.randint(0, 1 << 63 if case["bits"] == 64 else 1 << case["bits"], (n,), generator=g,
                             device="cuda", dtype=torch.int64) if case["bits"] < 64 else \
            (torch.randint(0, 1 << 32, (n,), generator=g, device="cuda", dtype=torch.int64) << 31) | \
            torch.randint(0, 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int64)
        vals = torch.arange(n, device="cuda", dtype=torch.int32)
        return {"case": case, "new_keys": keys, "new_vals": vals, "keys": torch.empty_like(keys),
                "vals": torch.empty_like(vals), "lib": load()}
    if kind == "train":
        x, y = _residuals(case, seed)
        return {"case": case, "engine": Engine(1024, **_config(case)), "x": x, "y": y, "seed": seed % 1000}
    if kind == "ensemble":
        systems = _ensemble(case, seed)
        n = sum(len(m) for _, _, m in systems)
        eng = Engine(n, **_config(case))
        eng.set_ensemble(systems)
        return {"case": case, "engine": eng, "pos": _pinned(3 * n), "vel": _pinned(3 * n)}
    pos, vel, mass = _system(case, seed)
    n = pos.shape[0]
    eng = Engine(n, **_config(case))
    if kind == "learned":
        eng.set_state(pos.cpu().numpy(), vel.cpu().numpy(), mass.cpu().numpy(), f64=True)
        eng.learn_set(_weights(_gen(seed + 1), 1.0), 0.02)
        eng.learn_enable(True)
    elif kind == "potential":
        eng.set_state(pos.float().cpu().numpy(), vel.float().cpu().numpy(), mass.cpu().numpy())
        return {"case": case, "engine": eng}
    else:
        eng.set_state(pos.cpu().numpy(), vel.cpu().numpy(), mass.cpu().numpy(), f64=True)
    return {"case": case, "engine": eng, "pos": _pinned(3 * n), "vel": _pinned(3 * n), "acc": _pinned(3 * n)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sort":
        keys, vals = state["keys"], state["vals"]
        keys.copy_(state["new_keys"])
        vals.copy_(state["new_vals"])
        status = state["lib"].bz_sort_pairs_noalloc(keys.data_ptr(), vals.data_ptr(), case["n"], case["bits"],
                                                    torch.cuda.current_stream().cuda_stream)
        if status:
            raise RuntimeError(f"bz_sort_pairs_noalloc: status {status}")
        return {"keys": keys, "vals": vals}
    eng = state["engine"]
    if kind == "train":
        loss = eng.learn_train(state["x"], state["y"], steps=case["steps"], batch=case["batch"], seed=state["seed"])
        params, scale = eng.learn_get()
        return {"params": params, "loss": loss, "scale": scale}
    if kind == "potential":
        acc, pot = eng.accelerations(want_pot=True)
        return {"acc": acc, "pot": pot}
    eng.step(case["dt"], case["steps"])
    if kind == "ensemble":  # block steps keep per-particle accelerations of their own
        eng.get_state_soa(state["pos"].numpy(), state["vel"].numpy())
        return {"pos": state["pos"], "vel": state["vel"]}
    eng.get_state_acc_soa(state["pos"].numpy(), state["vel"].numpy(), state["acc"].numpy())
    return {"pos": state["pos"], "vel": state["vel"], "acc": state["acc"]}


# --------------------------------------------------------------------------- work and tolerance

def _count(case):
    kind = case["kind"]
    if kind in ("treepm", "learned"):
        return case["n_side"] ** 3
    if kind == "ensemble":  # mean of a log-uniform size
        return int(case["systems"] * (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"]))
    return case["n"]


def work(case):
    """Bytes: the FP64 state and masses read and the state and FP32 forces written once a step,
    the mesh once, the snapshot once.  Flops: with a cutoff, the pairs inside it (35 each, at the
    mean density); open systems, an opening angle's worth of quadrupole terms (about 65 flops, 28
    / theta^2 of them for each factor of two in N) and 200 near pairs of 20 flops."""
    kind = case["kind"]
    n = _count(case)
    if kind == "sort":
        return {"bytes": 24.0 * n, "flops": 0.0}
    if kind == "train":
        rows = case["steps"] * case["batch"]
        return {"bytes": 36.0 * (case["n"] + rows), "flops": 6.0 * rows * 1632}
    steps = case.get("steps", 1)
    bytes_ = steps * n * (52 + 48 + 12) + 36.0 * n
    open_flops = 65 * 28 / case.get("theta", 0.5) ** 2 * max(1.0, math.log2(n / 32)) + 20 * 200
    if kind in ("treepm", "learned"):
        mesh = case["mesh"]
        rcut = case["rs"] * case["rcf"] / mesh
        near = n * 4.0 / 3.0 * math.pi * rcut ** 3
        flops = n * near * 35 + 5.0 * mesh ** 3 * math.log2(mesh ** 3)
        bytes_ += steps * 8.0 * mesh ** 3
        if kind == "learned":
            flops += n * min(near, 25.6) * 2 * 1632
        return {"bytes": bytes_, "flops": steps * flops}
    if kind == "treepm_open":
        mesh = 2 * case["grid"]
        bytes_ += steps * 8.0 * mesh ** 3
        return {"bytes": bytes_, "flops": steps * (n * open_flops + 5.0 * mesh ** 3 * math.log2(mesh ** 3))}
    if kind == "ensemble":  # a few closed steps a particle and block
        per = case["n_max"] / math.log(case["n_max"] / case["n_min"])
        open_flops = 65 * 28 / case["theta"] ** 2 * max(1.0, math.log2(per / 32)) + 20 * 200
        return {"bytes": 8 * bytes_, "flops": 8.0 * n * open_flops}
    return {"bytes": bytes_, "flops": steps * n * open_flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "sort":
        return "exact"
    if kind == "train":
        # BF16 weights and activations and Adam's division by the gradient's own size: inputs
        # moved by one FP32 rounding move the weights by 8e-5 (largest 6e-4)
        return {"rel": 1e-3, "max": 1e-2}
    if kind == "learned":  # BF16 activations of the pair correction, on top of the forces below
        return {"rel": 1e-4, "max": 1e-2}
    # FP32 force sums and an FP32 mesh: velocities moved by one FP32 rounding move the forces by
    # 1e-6 (mesh), 2e-7 (open) and, where a particle's rounding takes it across a cell boundary,
    # a few groups by the opening criterion's own error (1e-2 at most, 2e-5 in the norm)
    if kind == "treepm" and case["order"] == 1:
        return {"rel": 5e-6, "max": 5e-4}
    return {"rel": 6e-5, "max": 6e-2} if kind == "treepm" else {"rel": 2e-5, "max": 2e-2}


# ------------------------------------------------------------------------------- 64-bit results

def _direct(pos, mass, eps, want_pot=False):
    n = pos.shape[0]
    acc = torch.empty_like(pos)
    pot = torch.empty(n, device="cuda", dtype=torch.float64)
    rows = max(1, (1 << 27) // n)
    for i in range(0, n, rows):
        d = pos[None, :, :] - pos[i:i + rows, None, :]
        s2 = (d * d).sum(-1) + eps * eps
        w = mass[None, :] * s2 ** -1.5
        acc[i:i + rows] = torch.einsum("ij,ijk->ik", w, d)
        if want_pot:
            w = mass[None, :] * s2 ** -0.5
            k = torch.arange(w.shape[0], device="cuda")
            w[k, i + k] = 0.0
            pot[i:i + rows] = -w.sum(1)
    norm = acc.norm(dim=1, keepdim=True)
    return acc * (64.0 / norm.clamp_min(64.0)), pot


def _ewald(pos, mass, eps, kmax=8):
    """Periodic accelerations in the unit box: Ewald's sum with alpha = 6.4, nearest images in the
    real part, Plummer softening on the nearest image."""
    n, alpha = pos.shape[0], 6.4
    acc = torch.empty_like(pos)
    rows = max(1, (1 << 26) // n)
    for i in range(0, n, rows):
        d = pos[None, :, :] - pos[i:i + rows, None, :]
        d -= torch.round(d)
        r2 = (d * d).sum(-1)
        k = torch.arange(r2.shape[0], device="cuda")
        r2[k, i + k] = 1.0
        r = r2.sqrt()
        w = torch.erfc(alpha * r) / (r * r2) + 2 * alpha / math.sqrt(math.pi) * torch.exp(-alpha * alpha * r2) / r2
        w += (r2 + eps * eps) ** -1.5 - 1.0 / (r * r2)
        w *= mass[None, :]
        w[k, i + k] = 0.0
        acc[i:i + rows] = torch.einsum("ij,ijk->ik", w, d)
    ks = [(a, b, c) for a in range(-kmax, kmax + 1) for b in range(-kmax, kmax + 1) for c in range(-kmax, kmax + 1)
          if 0 < a * a + b * b + c * c <= kmax * kmax]
    kv = 2 * math.pi * torch.tensor(ks, device="cuda", dtype=torch.float64)
    k2 = (kv * kv).sum(1)
    amp = 4 * math.pi / k2 * torch.exp(-k2 / (4 * alpha * alpha))
    for j in range(0, kv.shape[0], 512):
        ph = pos @ kv[j:j + 512].T
        c, s = ph.cos(), ph.sin()
        sc, ss = mass @ c, mass @ s
        acc -= ((s * sc - c * ss) * amp[j:j + 512]) @ kv[j:j + 512]
    return acc


def _features(x):
    t = 2 * math.pi
    sep, off = x[:, :3], x[:, 3:]
    f = [sep]
    for v in (off, off + sep):
        f += [torch.sin(t * v), torch.cos(t * v)]
    return torch.cat(f + [torch.ones_like(x[:, :1])], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "potential" and case["n"] <= 250000:
        pos, _, mass = _system(case, seed)
        acc, pot = _direct(pos.float().double(), mass.double(), case["eps"], True)
        return {"acc": acc, "pot": pot}
    cost = case.get("steps", 1) * float(_count(case)) ** 2 if kind in ("octree", "treepm") else 0.0
    if not ((kind == "octree" and cost <= 5e10) or
            (kind == "treepm" and case["gradient"] and case["assign"] == "pcs" and case["mesh"] >= 2 * case["n_side"] and
             case["order"] == 1 and cost <= 1e10)):
        return None
    pos, vel, mass = _system(case, seed)
    mass = mass.double()
    dt = case["dt"]
    if kind == "octree":
        def force(p):
            return _direct(p, mass, case["eps"])[0]
    else:
        def force(p):
            return _ewald(p, mass, 0.02 / case["n_side"])
    acc = force(pos)
    for _ in range(case["steps"]):
        euler = case.get("integrator", 0) == 1
        vel = vel + (dt if euler else 0.5 * dt) * acc
        pos = pos + dt * vel
        if kind == "treepm":
            pos = torch.remainder(pos, 1.0)
        acc = force(pos)
        if not euler:
            vel = vel + 0.5 * dt * acc
    return {k: v.T.contiguous().reshape(-1) for k, v in (("pos", pos), ("vel", vel), ("acc", acc))}
