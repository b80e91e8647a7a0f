"""The work that programs have this library do, as measurable cases.

Three kinds of program use the library.  The reference engine calls the force
functions through its plugin type on its own host arrays, from inside its
integrators ("force").  A resident run uploads or generates a system once,
advances it on the device and downloads a snapshot every few steps ("step",
and "ensemble" for many small systems).  Around those stand the conservation
diagnostics ("diagnostics") and the training of the learned far-field
correction ("train").

Systems are the ones that the benchmark and the tests use: Plummer spheres (the
globular_cluster preset), the two-Plummer collision, and ensembles of Plummer
systems of 32 to 4096 particles; G = 1, softening 0.01, steps of 1e-3.
"""
import ctypes as C
import math

import numpy as np
import torch

import n_body_sim_pro_b200 as nb

EPS = 0.01
DT = 1e-3
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "m")


def listed():
    return [
        # plugin, all-pairs: the engine's interactive scenes hold about a thousand
        # bodies; the call is bound by its latency
        force("force_allpairs_1k", 1000, "all_pairs"),
        # plugin, Barnes-Hut at the engine's default angle: the size of its own
        # force benchmark (an odd count, as user files have)
        force("force_bh_20k", 20011, "barnes_hut"),
        # plugin, quadrupole cells: the more accurate walk on a mid-size cluster
        force("force_bh_quadrupole_150k", 150001, "barnes_hut", order=2),
        # plugin, relative opening test on page-locked arrays: the set-up that the
        # integration guide recommends for a force-error budget
        force("force_bh_relative_1m", 1000000, "barnes_hut", ic="collision", theta=5.0, alpha=0.0045, leaf=32, pinned=True),
        # resident all-pairs: the benchmark's 16k Plummer sphere, 3 steps a snapshot
        step("step_allpairs_16k", 16384, "all_pairs", 3),
        # resident all-pairs at the precision study's size
        step("step_allpairs_262k", 262144, "all_pairs", 2, pinned=True),
        # resident Barnes-Hut on a small, odd-sized cluster: launches and latency
        step("step_bh_10k", 10007, "barnes_hut", 10),
        # resident Barnes-Hut: the benchmark's 1M collision at angle 0.7, 10 steps
        step("step_bh_1m", 1000000, "barnes_hut", 10, ic="collision", pinned=True),
        # resident Barnes-Hut: the benchmark's headline, 10M at rms error 1e-3
        step("step_bh_relative_10m", 10000000, "barnes_hut", 10, ic="collision", theta=5.0, alpha=0.0045, leaf=32, pinned=True),
        # the benchmark's ensemble of 4096 systems, 20 steps a snapshot
        {"name": "ensemble_4096", "kind": "ensemble", "systems": 4096, "lo": 32, "hi": 4096, "steps": 20},
        # energy check of a run: all global sums and the O(n^2) potential energy
        {"name": "diagnostics_100k", "kind": "diagnostics", "n": 100003},
        # one epoch of the learned correction's training, as the benchmark batches it
        {"name": "train_262k", "kind": "train", "samples": 262144, "batch": 1024, "n": 200000},
    ]


def force(name, n, algorithm, ic="plummer", theta=0.7, order=1, alpha=0.0, leaf=16, opening=0, pinned=False):
    return {"name": name, "kind": "force", "n": n, "algorithm": algorithm, "ic": ic, "theta": theta, "order": order,
            "alpha": alpha, "leaf": leaf, "opening": opening, "pinned": pinned}


def step(name, n, algorithm, steps, ic="plummer", theta=0.7, order=1, alpha=0.0, leaf=16, opening=0, pinned=False):
    return dict(force(name, n, algorithm, ic, theta, order, alpha, leaf, opening, pinned), kind="step", steps=steps)


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("force", "force", "force", "step", "step", "step", "ensemble", "diagnostics", "train"))
    if kind == "ensemble":
        lo = log_int(rng, 8, 256)
        return {"kind": kind, "systems": log_int(rng, 32, 4096), "lo": lo, "hi": log_int(rng, 2 * lo, 4096), "steps": rng.randint(1, 20)}
    if kind == "diagnostics":
        return {"kind": kind, "n": log_int(rng, 500, 200000)}
    if kind == "train":
        return {"kind": kind, "samples": log_int(rng, 16384, 524288), "batch": rng.choice((512, 1024, 2048, 4096)), "n": log_int(rng, 20000, 400000)}
    algorithm = rng.choice(("all_pairs", "barnes_hut", "barnes_hut"))
    pinned = rng.random() < 0.5
    ic = rng.choice(("plummer", "collision"))
    if algorithm == "all_pairs":
        # (through the plugin, all-pairs serves the small scenes; beyond, runs are resident)
        if kind == "force":
            case = force("", log_int(rng, 2, 2000), algorithm, ic, pinned=pinned)
        else:
            n = log_int(rng, 300, 262144)
            case = step("", n, algorithm, rng.randint(1, max(1, min(20, int(2 * (262144 / n) ** 2)))), ic, pinned=pinned)
    else:
        n = log_int(rng, 100, 1000000 if kind == "force" else 10000000)
        if rng.random() < 0.35:
            how = {"theta": rng.choice((1.0, 5.0)), "alpha": rng.choice((0.0015, 0.0045)), "leaf": rng.choice((16, 32))}
        else:
            how = {"theta": rng.choice((0.5, 0.7, 1.0)), "order": rng.choice((1, 1, 2)), "opening": rng.choice((0, 0, 1))}
        heavy = how["theta"] < 0.7 or how.get("order") == 2 or how.get("alpha") == 0.0015
        if kind == "force":
            case = force("", n, algorithm, ic, pinned=pinned, **how)
        else:
            n = min(n, 3000000) if heavy else n
            case = step("", n, algorithm, rng.randint(1, max(1, min(10, 6000000 // n))), ic, pinned=pinned, **how)
    del case["name"]
    return case


# ---- inputs ------------------------------------------------------------------


def empty(n, pinned):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy() if pinned else np.zeros(n)


def generate(context, case, seed):
    if case.get("ic") == "collision":
        context.generate_plummer_collision(case["n"], seed)
    else:
        context.generate_preset("globular_cluster", case["n"], seed)


def context_of(case):
    return nb.CudaContext(theta=case["theta"], multipole_order=case["order"], leaf_capacity=case["leaf"],
                          opening=case["opening"], relative_opening=case["alpha"])


def system_of(n, pinned):
    return nb.ParticleSystem.zeros(n, allocator=lambda k: empty(k, pinned))


def host_system(case, seed):
    """The generated system in host arrays, accelerations zero."""
    system = system_of(case["n"], case.get("pinned", False))
    with nb.CudaContext() as context:
        generate(context, case, seed)
        context.download(system)
    return system


def ensemble_sizes(case):
    """round(exp(U(ln lo, ln hi))) particles a system; the same for every seed."""
    u = np.random.default_rng(case["systems"]).uniform(math.log(case["lo"]), math.log(case["hi"]), case["systems"])
    return np.clip(np.rint(np.exp(u)).astype(np.int64), case["lo"], case["hi"])


def ensemble_system(case, seed):
    """Plummer systems (a = 1, M = 1) back to back, isotropic Gaussian velocities."""
    sizes = ensemble_sizes(case)
    owner = torch.from_numpy(np.repeat(np.arange(case["systems"]), sizes)).cuda()
    n = int(sizes.sum())
    g = torch.Generator("cuda").manual_seed(seed)
    u = 1.0 - torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 0.999
    r = 1.0 / torch.sqrt(u ** (-2.0 / 3.0) - 1.0).clamp_min(1e-3)
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    pos = r[:, None] * d / d.norm(dim=1, keepdim=True)
    vel = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    vel *= torch.sqrt(1.0 / (6.0 * torch.sqrt(1.0 + r * r)))[:, None]
    mass = (1.0 / torch.from_numpy(sizes).cuda().double())[owner]
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    return pos.cpu().numpy(), vel.cpu().numpy(), mass.cpu().numpy(), offsets


def prepare(case, seed):
    g = nb.gravity_init(1.0, EPS)
    kind = case["kind"]
    if kind == "force":
        system = host_system(case, seed)
        name = {"all_pairs": "n_body_sim_pro_gravity_compute_acceleration_cuda",
                "barnes_hut": "n_body_sim_pro_barnes_hut_compute_acceleration_cuda"}[case["algorithm"]]
        return {"kind": kind, "context": context_of(case), "system": system, "view": system.view(), "gravity": g,
                "call": getattr(nb.library(), name), "error": nb.Error()}
    if kind == "step":
        context = context_of(case)
        generate(context, case, seed)
        algorithm = nb.Algorithm.ALL_PAIRS if case["algorithm"] == "all_pairs" else nb.Algorithm.BARNES_HUT
        context.compute_acceleration(g, algorithm)
        return {"kind": kind, "context": context, "algorithm": algorithm, "gravity": g, "steps": case["steps"],
                "system": system_of(case["n"], case["pinned"])}
    if kind == "ensemble":
        pos, vel, mass, offsets = ensemble_system(case, seed)
        ensemble = nb.CudaEnsemble()
        ensemble.upload(nb.ParticleSystem.from_arrays(pos, vel, mass), offsets)
        ensemble.autotune(g, DT)
        return {"kind": kind, "ensemble": ensemble, "gravity": g, "steps": case["steps"], "system": system_of(mass.shape[0], True)}
    context = nb.CudaContext()
    generate(context, case, seed)
    if kind == "diagnostics":
        return {"kind": kind, "context": context, "gravity": g}
    with context:
        correction = nb.CudaCorrection(seed=seed)
        correction.generate(context, g, 1.0, case["samples"], seed)
    return {"kind": kind, "correction": correction, "batch": case["batch"]}


def snapshot(system):
    """What a snapshot of a stepped system holds.  Accelerations are an intermediate
    of the next step and are compared where they are the result, in the force cases."""
    return {f: getattr(system, f) for f in FIELDS[:6]}


def run(state):
    kind = state["kind"]
    if kind == "force":
        # the plugin call as the engine's integrators make it: through the C ABI
        status = state["call"](C.byref(state["view"]), C.byref(state["gravity"]), state["context"].handle, C.byref(state["error"]))
        if status != nb.Status.OK:
            raise nb.CudaError(status, state["error"].message.decode(errors="replace"))
        return {f: getattr(state["system"], f) for f in ("ax", "ay", "az")}
    if kind == "step":
        state["context"].advance(state["gravity"], DT, state["steps"], state["algorithm"])
        state["context"].download(state["system"])
        return snapshot(state["system"])
    if kind == "ensemble":
        state["ensemble"].advance(state["gravity"], DT, state["steps"])
        state["ensemble"].download(state["system"])
        return snapshot(state["system"])
    if kind == "diagnostics":
        quantities, potential = state["context"].diagnostics(state["gravity"], potential=True)
        return {"quantities": quantities, "potential": potential}
    train, validation = state["correction"].train(1, state["batch"], 1e-3)
    parameters, scaling = state["correction"].parameters()
    return {"parameters": parameters, "scaling": scaling, "train": train, "validation": validation}


# ---- what a pass cannot do without -------------------------------------------


def terms(case):
    """Interactions per target: all of them, or about what the opening test leaves
    (measured on the collision: 1830 at 1M and angle 0.7, 1120 at 10M under the
    relative test at 0.0045)."""
    n = case["n"]
    if case["algorithm"] == "all_pairs":
        return n
    if case["alpha"] > 0.0:
        return min(n, 48.0 * (0.0045 / case["alpha"]) ** 0.5 * math.log2(n + 1))
    return min(n, 45.0 / case["theta"] ** 2 * math.log2(n + 1))


def work(case):
    kind = case["kind"]
    if kind == "force":  # positions and masses in, accelerations out (the relative test reads the old ones)
        n = case["n"]
        return {"bytes": (56 + (24 if case["alpha"] > 0.0 else 0)) * n, "flops": 20.0 * n * terms(case)}
    if kind == "step":  # positions, velocities, accelerations and masses read and all but masses written per step, then the snapshot
        n = case["n"]
        return {"bytes": (152.0 * case["steps"] + 80.0) * n, "flops": 20.0 * n * terms(case) * case["steps"]}
    if kind == "ensemble":  # the state once through the device, then the snapshot; forces before the first step too
        sizes = ensemble_sizes(case).astype(np.float64)
        return {"bytes": float((152.0 + 80.0) * sizes.sum()), "flops": float(20.0 * (sizes ** 2).sum() * (case["steps"] + 1))}
    if kind == "diagnostics":
        n = case["n"]
        return {"bytes": 56.0 * n, "flops": 12.0 * n * (n - 1) / 2}
    rows = case["samples"]  # inputs (16 BF16), labels and order once each for the steps and the two losses; 3 passes of 9,856 flop forward and backward
    return {"bytes": 2.0 * rows * (32 + 12 + 4), "flops": rows * 9856.0 * 4}


# ---- the same in 64 bits -------------------------------------------------------


def direct(x, m):
    """Softened accelerations of [batch, n, 3] positions by the direct sum."""
    batch, n, _ = x.shape
    out = torch.empty_like(x)
    rows = max(1, (1 << 27) // (batch * n))
    one = torch.cat([x, torch.ones_like(x[..., :1])], dim=2)
    for i in range(0, n, rows):
        t = x[:, i:i + rows]
        r2 = torch.full((batch, t.shape[1], n), EPS * EPS, dtype=torch.float64, device=x.device)
        for k in range(3):
            d = x[:, None, :, k] - t[:, :, None, k]
            r2.addcmul_(d, d)
            del d
        r2.rsqrt_()
        w = r2 * r2
        w.mul_(r2).mul_(m[:, None, :])
        s = torch.bmm(w, one)
        out[:, i:i + rows] = s[..., :3] - s[..., 3:] * t
    return out


def leapfrog(x, v, m, steps):
    a = direct(x, m)
    for _ in range(steps):
        v = v + 0.5 * DT * a
        x = x + DT * v
        a = direct(x, m)
        v = v + 0.5 * DT * a
    return x, v


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":  # the network's products are BF16 by definition: no 64-bit value
        return None
    if kind == "ensemble":
        sizes = ensemble_sizes(case)
        if float((sizes.astype(np.float64) ** 2).sum()) * (case["steps"] + 1) > 4e11:
            return None
        pos, vel, mass, offsets = (torch.from_numpy(a.astype(np.int64) if a.dtype == np.uint64 else a).cuda() for a in ensemble_system(case, seed))
        order = np.argsort(sizes)
        for i in range(0, len(order), 64):  # 64 systems of like size at a time, padded with massless entries
            few = torch.from_numpy(order[i:i + 64]).cuda()
            count = offsets[few + 1] - offsets[few]
            slot = torch.arange(int(count.max()), device="cuda")
            there = slot[None, :] < count[:, None]
            at = torch.where(there, offsets[few][:, None] + slot[None, :], 0)
            x, v = leapfrog(pos[at], vel[at], torch.where(there, mass[at], 0.0), case["steps"])
            pos[at[there]] = x[there]
            vel[at[there]] = v[there]
        return dict(zip(FIELDS[:6], [a.cpu().numpy() for a in (*pos.T.contiguous(), *vel.T.contiguous())]))
    n = case["n"]
    evaluations = case["steps"] + 1 if kind == "step" else 1
    if float(n) * n * evaluations > 4e11:
        return None
    s = host_system(dict(case, pinned=False), seed)
    x, v, m = (torch.from_numpy(np.stack([getattr(s, f) for f in names], axis=-1)).cuda()[None] for names in (FIELDS[:3], FIELDS[3:6], FIELDS[9:]))
    m = m[..., 0]
    if kind == "force":
        return dict(zip(FIELDS[6:9], direct(x, m)[0].T.cpu().numpy()))
    if kind == "step":
        x, v = leapfrog(x, v, m, case["steps"])
        return dict(zip(FIELDS[:6], [a.cpu().numpy() for a in (*x[0].T.contiguous(), *v[0].T.contiguous())]))
    x, v, m = x[0], v[0], m[0]
    total = m.sum()
    momentum = (m[:, None] * v).sum(0)
    spin = (m[:, None] * torch.linalg.cross(x, v)).sum(0)
    centre = (m[:, None] * x).sum(0) / total
    kinetic = 0.5 * (m * (v * v).sum(1)).sum()
    potential = 0.0
    rows = max(1, (1 << 26) // n)
    for i in range(0, n, rows):
        d2 = torch.full((min(rows, n - i), n), EPS * EPS, dtype=torch.float64, device="cuda")
        for k in range(3):
            d = x[None, :, k] - x[i:i + rows, None, k]
            d2.addcmul_(d, d)
        potential -= 0.5 * float((m[i:i + rows] * (d2.rsqrt_() @ m - m[i:i + rows] / EPS)).sum())
    return {"quantities": torch.cat([kinetic[None], total[None], momentum, spin, centre]).cpu().numpy(), "potential": potential}
