"""The workloads whose speed this package is judged by.

Every case goes through the public entry points (``FastMultipoleMethod`` and
``jaccpot_b200.mutual``) with particles already on the GPU, as a simulation
holds them.  The kinds are what such a program does:

* ``step``    the whole pass on live particles over a prepared topology
              (``differentiable_accelerations`` without gradients);
* ``grad``    the same with a backward pass to positions and masses;
* ``evaluate`` leaf evaluation of a prepared state with the potential;
* ``targets`` evaluation of a prepared state at a subset of the particles;
* ``fresh``   ``compute_accelerations``: tree, lists, schedules and the pass,
              on particles that have no prepared state;
* ``leapfrog`` ``strict_run_v2``: velocity Verlet steps with a refresh of the
              prepared state at every step;
* ``blockstep`` the momentum-conserving lane with a rung per particle and a
              weight per level.

Sizes and distributions are those of the package's configurations (uniform
cube at order 4, Plummer sphere at order 6, 64-clump Plummer mixture at order
8) and of its tests.  Acceptance is the opening angle theta, or with ``eps``
above zero the error-controlled walk.
"""

import math

import torch

from jaccpot_b200 import FastMultipoleMethod, mutual

DEVICE = "cuda"
MAX_DIRECT_PAIRS = 3e11  # an FP64 direct sum above this takes too long
_BASE = {"kind": "step", "dist": "clustered", "n": 0, "order": 8, "leaf": 32, "theta": 0.6, "eps": 0.0,
         "gears": "", "kahan": False, "softening": 0.0, "graph": False, "targets": 0, "steps": 0}


def _case(name, **kw):
    return {"name": name, **_BASE, **kw}


def listed():
    return [
        # a few thousand bodies, one pass: launches and host calls are most of it
        _case("step_uniform_2k_p4", dist="uniform", n=2048, order=4, leaf=16),
        # the first configuration, called once on new particles: tree to accelerations
        _case("fresh_uniform_16k_p4", kind="fresh", dist="uniform", n=16384, order=4, leaf=16),
        # a short N-body run: each step rebuilds and compares the tree, then evaluates
        _case("leapfrog_plummer_65k_p6", kind="leapfrog", dist="plummer", n=65536, order=6, softening=1e-3, steps=2),
        # the second configuration: a Plummer sphere of a million bodies on its prepared topology
        _case("step_plummer_1m_p6", dist="plummer", n=1048576, order=6),
        # the second configuration's active subset: 65,536 of the million
        _case("targets_plummer_1m_p6", kind="targets", dist="plummer", n=1048576, order=6, targets=65536),
        # the headline: four million bodies, error-controlled walk, compensated sums, replayed as a graph
        _case("step_clustered_4m_p8", n=4194304, eps=5e-5, kahan=True, graph=True),
        # per-pair orders from the error-controlled walk, at a size that is no power of two
        _case("step_gears_500k_p8", n=500009, eps=1e-4, gears="2,4,6,8", kahan=True),
        # the adjoint configuration at full size: accelerations, then gradients of positions and masses
        _case("grad_plummer_1m_p6", kind="grad", dist="plummer", n=1048576, order=6),
        # gradients of a small softened system, as in a fit by gradient descent
        _case("grad_clustered_10k_p4", kind="grad", n=10007, order=4, leaf=16, softening=1e-3),
        # a million clustered bodies without a prepared state, error-controlled: prepass, walk and pass
        _case("fresh_clustered_1m_p8", kind="fresh", n=1000003, eps=5e-5, kahan=True),
        # the highest order with the largest leaves and the potential: an accurate energy check
        _case("evaluate_200k_p10", kind="evaluate", n=200003, order=10, leaf=64, theta=0.5, softening=1e-3,
              kahan=True),
        # block time steps: rungs and level weights on the momentum-conserving lane
        _case("blockstep_plummer_131k_p6", kind="blockstep", dist="plummer", n=131071, order=6, softening=1e-3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "grad", "evaluate", "targets", "fresh", "leapfrog", "blockstep"])
    most = {"step": 1 << 21, "grad": 1 << 19, "evaluate": 1 << 20, "targets": 1 << 20, "fresh": 1 << 19,
            "leapfrog": 1 << 17, "blockstep": 1 << 18}[kind]
    # a run in time needs bodies that are bound to each other, not a cube of unit masses
    dists = ["plummer", "clustered"] if kind in ("leapfrog", "blockstep") else ["uniform", "plummer", "clustered"]
    c = dict(_BASE, kind=kind, dist=rng.choice(dists), n=_log_int(rng, 2000, most),
             order=rng.choice([4, 4, 6, 6, 8, 8, 10] if kind not in ("grad",) else [4, 6, 8]),
             leaf=rng.choice([16, 32, 32, 64]), softening=rng.choice([0.0, 1e-3]))
    if kind in ("step", "evaluate", "fresh"):
        c["kahan"] = rng.random() < 0.5
        # the error-controlled walk is a choice of accurate runs on clustered particles
        if c["dist"] == "clustered" and c["order"] == 8 and rng.random() < 0.6:
            c["eps"] = math.exp(rng.uniform(math.log(3e-5), math.log(3e-4)))
            c["gears"] = rng.choice(["", "2,4,6,8"])
    if kind == "step":
        c["graph"] = rng.random() < 0.3
    if kind == "targets":
        c["targets"] = _log_int(rng, 100, max(200, c["n"] // 2))
    if kind == "leapfrog":
        c["steps"] = rng.randint(1, 3)
    return c


# ------------------------------------------------------------------- inputs
def _uniform(g, *shape, lo=0.0, hi=1.0):
    return torch.rand(*shape, generator=g, device=DEVICE, dtype=torch.float64) * (hi - lo) + lo


def _plummer(g, n):
    """Unit Plummer sphere cut off at 20 scale radii, isotropic."""
    u = _uniform(g, n)
    r = (u ** (1.0 / 3.0) / torch.sqrt((1.0 - u ** (2.0 / 3.0)).clamp_min(1e-12))).clamp_max(20.0)
    cos_t = _uniform(g, n, lo=-1.0)
    sin_t = torch.sqrt((1.0 - cos_t ** 2).clamp_min(0.0))
    phi = _uniform(g, n, hi=2.0 * math.pi)
    return torch.stack([r * sin_t * torch.cos(phi), r * sin_t * torch.sin(phi), r * cos_t], dim=1)


def _particles(case, seed):
    """float32 positions (N, 3) and masses (N,) on the GPU, with the
    generator left for the case's other inputs."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    n = case["n"]
    if case["dist"] == "uniform":
        pos, mass = _uniform(g, n, 3, lo=-1.0), _uniform(g, n, lo=0.5, hi=1.5)
    elif case["dist"] == "plummer":
        pos, mass = _plummer(g, n), torch.full((n,), 1.0 / n, device=DEVICE, dtype=torch.float64)
    else:
        clumps = 64
        centres = _uniform(g, clumps, 3, lo=-50.0, hi=50.0)
        scales = torch.exp(_uniform(g, clumps, lo=math.log(0.1), hi=math.log(2.0)))
        weights = -torch.log(_uniform(g, clumps).clamp_min(1e-12))  # Dirichlet(1) once normalised
        of = torch.searchsorted(torch.cumsum(weights / weights.sum(), 0), _uniform(g, n)).clamp_max(clumps - 1)
        pos = centres[of] + scales[of, None] * _plummer(g, n)
        mass = torch.exp(0.5 * torch.randn(n, generator=g, device=DEVICE, dtype=torch.float64))
        mass = mass / mass.sum()
    return pos.float(), mass.float(), g


def _rest(case, g):
    """The inputs beside the particles, drawn after them."""
    n = case["n"]
    if case["kind"] == "grad":
        return torch.randn(n, 3, generator=g, device=DEVICE, dtype=torch.float32)
    if case["kind"] == "targets":
        return torch.randperm(n, generator=g, device=DEVICE)[:case["targets"]]
    if case["kind"] == "leapfrog":
        return 0.3 * torch.randn(n, 3, generator=g, device=DEVICE, dtype=torch.float32)
    if case["kind"] == "blockstep":  # a few levels, the finer ones rarer
        return (_uniform(g, n).clamp_min(1e-9).log() / math.log(0.3)).floor().clamp(0, 3).to(torch.int32)
    return None


_DT = 1e-3  # leapfrog step
_LEVEL_WEIGHTS = (1.0, 0.5, 0.25, 0.125)


def _solver(case):
    kw = dict(theta=case["theta"], G=1.0, softening=case["softening"],
              advanced={"nearfield_compensated": case["kahan"], "cuda_graph": case["graph"]})
    if case["eps"] > 0.0:
        gears = tuple(int(o) for o in case["gears"].split(",")) if case["gears"] else (case["order"],)
        # "prepass": each prepare takes its force scale from its own particles
        kw.update(adaptive_order=True, p_gears=gears, adaptive_error_model="dehnen_paper",
                  adaptive_eps=case["eps"], mac_force_scale_mode="prepass")
    return FastMultipoleMethod(**kw)


def prepare(case, seed):
    pos, mass, g = _particles(case, seed)
    s = {"case": case, "pos": pos, "mass": mass, "extra": _rest(case, g)}
    kind = case["kind"]
    if kind == "blockstep":
        topo, _ = mutual.build_mutual_topology(pos, mass, theta=case["theta"], order=case["order"],
                                               leaf_size=case["leaf"])
        s["mutual"] = mutual.build_mutual_state(topo, softening=case["softening"])
        s["weights"] = torch.tensor(_LEVEL_WEIGHTS, device=DEVICE)
        return s
    s["fmm"] = _solver(case)
    if kind not in ("fresh", "leapfrog"):
        s["state"] = s["fmm"].prepare_state(pos, mass, leaf_size=case["leaf"], max_order=case["order"])
    if kind == "grad":
        s["pos"], s["mass"] = pos.requires_grad_(), mass.requires_grad_()
    if kind == "leapfrog":
        s["xv"] = torch.stack([pos, s["extra"]], dim=1)
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "step":
        return s["fmm"].differentiable_accelerations(s["state"], s["pos"], s["mass"])
    if kind == "grad":
        acc = s["fmm"].differentiable_accelerations(s["state"], s["pos"], s["mass"])
        gx, gm = torch.autograd.grad(acc, (s["pos"], s["mass"]), s["extra"])
        return {"acc": acc.detach(), "grad_pos": gx, "grad_mass": gm}
    if kind == "evaluate":
        acc, pot = s["fmm"].evaluate_prepared_state(s["state"], return_potential=True, as_numpy=False)
        return {"acc": acc, "pot": pot}
    if kind == "targets":
        return s["fmm"].evaluate_prepared_state(s["state"], target_indices=s["extra"])
    if kind == "fresh":
        return s["fmm"].compute_accelerations(s["pos"], s["mass"], leaf_size=case["leaf"], max_order=case["order"])
    if kind == "leapfrog":
        xv, _, _ = s["fmm"].strict_run_v2(state=s["xv"], masses=s["mass"], dt=_DT, num_steps=case["steps"],
                                          refresh_every=1, leaf_size=case["leaf"], max_order=case["order"])
        return {"pos": xv[:, 0], "vel": xv[:, 1]}
    return mutual.mutual_weighted_accelerations(s["mutual"], s["pos"], s["mass"], rung=s["extra"],
                                                level_weights=s["weights"])


# -------------------------------------------------------------------- work
def _m2l_flops(p):
    """Rotate, shift along z, rotate back: two block-diagonal rotations and
    the axial terms, a multiply and an add each."""
    rot = sum((2 * ell + 1) ** 2 for ell in range(p + 1))
    axial = sum((2 if m else 1) * sum(1 for a in range(m, p + 1) for b in range(m, p + 1) if a + b <= p)
                for m in range(p + 1))
    return 2.0 * (2 * rot + axial)


def work(case):
    """Estimated from the list lengths that the tree gives at these sizes
    (theta 0.6: leaves about 0.68 full, near field about 80 leaves wide, 60 to
    300 far pairs per leaf); flops of near pairs, far pairs and the two
    sweeps, bytes of particles, lists and results."""
    n, p, kind = case["n"], case["order"], case["kind"]
    occ = 0.68 * case["leaf"]
    leaves = max(1.0, n / occ)
    coeffs = (p + 1) ** 2
    near_leaves = min(leaves, 80.0 * (0.6 / case["theta"]) ** 3)
    far_pairs = leaves * 300.0 * min(1.0, n / 2.0 ** 20) ** 0.25 * (0.6 if case["eps"] > 0.0 else 1.0)
    near, far, leaf_ops = 20.0 * n * near_leaves * occ, far_pairs * _m2l_flops(p), 2.0 * n * coeffs * 8
    sweeps = 4.0 * leaves * _m2l_flops(p)
    lists = 4.0 * far_pairs + 4.0 * leaves * near_leaves
    whole = {"flops": near + far + leaf_ops + sweeps, "bytes": 28.0 * n + lists}
    if kind == "evaluate":
        return {"flops": near + leaf_ops, "bytes": 32.0 * n + 4.0 * leaves * (near_leaves + coeffs)}
    if kind == "targets":
        share = case["targets"] / n
        touched = min(1.0, share * occ) * leaves
        return {"flops": (near + leaf_ops) * share,
                "bytes": 16.0 * n + 20.0 * case["targets"] + 4.0 * touched * (near_leaves + coeffs)}
    if kind == "grad":
        return {"flops": 4.0 * whole["flops"], "bytes": whole["bytes"] + lists + 28.0 * n}
    if kind == "fresh":
        # the error-controlled walk starts from a pass at the plain opening angle
        return {"flops": whole["flops"] * (2.5 if case["eps"] > 0.0 else 1.0), "bytes": whole["bytes"] + 2.0 * lists}
    if kind == "leapfrog":
        k = case["steps"] + 1
        return {"flops": k * whole["flops"], "bytes": k * (whole["bytes"] + 2.0 * lists + 24.0 * n)}
    return whole


# --------------------------------------------------------------- agreement
def tolerance(case):
    """Four times the most that the kernels' other forms (one lane per target
    in the near field, per-thread row copies, undivided sweeps) show against
    the default ones over 30 drawn cases: rel 4.7e-7, max 4.9e-6.  Per-pair
    orders and error-controlled lists are decided from 32-bit multipoles and
    forces, where a rounding can move a borderline pair (max 6.3e-6 seen with
    none moved); gradients carry one more derivative."""
    if case["eps"] > 0.0:
        return {"rel": 5e-6, "max": 1e-3}
    if case["kind"] == "grad":
        return {"rel": 5e-6, "max": 5e-5}
    return {"rel": 2e-6, "max": 2e-5}


# ------------------------------------------------- direct sums in 64 bits
def _direct(case, pos, mass, targets=None, w=None):
    """Direct sums over all pairs in float64: accelerations and potential of
    `targets` (indices; None for all), and with `w` the gradients of
    sum(w * acc)."""
    x, m = pos.double(), mass.double()
    n = x.shape[0]
    t = torch.arange(n, device=DEVICE) if targets is None else targets
    e2 = case["softening"] ** 2
    out = {"acc": torch.empty(t.numel(), 3, device=DEVICE, dtype=torch.float64),
           "pot": torch.empty(t.numel(), device=DEVICE, dtype=torch.float64)}
    if w is not None:
        w = w.double()
        out.update(grad_pos=torch.empty_like(x), grad_mass=torch.empty_like(m))
    rows = max(1, int(2.5e8 // n))
    for a in range(0, t.numel(), rows):
        i = t[a:a + rows]
        d = [x[None, :, k] - x[i, k][:, None] for k in range(3)]
        r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2 + e2
        r2[torch.arange(i.numel(), device=DEVICE), i] = math.inf  # no self force
        r2[r2 == 0.0] = math.inf
        inv = torch.rsqrt(r2)
        del r2
        out["pot"][a:a + rows] = -(inv @ m)
        inv3 = inv ** 3
        for k in range(3):
            out["acc"][a:a + rows, k] = (inv3 * d[k]) @ m
        if w is not None:
            # a_i = sum_j m_j f(d), f = d / r^3, f' = J = 1 / r^3 - 3 d d^T / r^5:
            # dL/dx_i = sum_j J (m_i w_j - m_j w_i), dL/dm_i = -sum_j w_j . f(d)
            out["grad_mass"][a:a + rows] = -sum((inv3 * d[k]) @ w[:, k] for k in range(3))
            mi, wi = m[i][:, None], w[i]
            v = [mi * w[None, :, k] - m[None, :] * wi[:, k][:, None] for k in range(3)]
            dv = 3.0 * inv3 * inv ** 2 * (d[0] * v[0] + d[1] * v[1] + d[2] * v[2])
            for k in range(3):
                out["grad_pos"][a:a + rows, k] = (inv3 * v[k] - dv * d[k]).sum(1)
    return out


def exact(case, seed):
    """The same quantities by direct summation.  Block-step weights hang on the
    tree's nodes, so they have no such value."""
    kind, n = case["kind"], case["n"]
    pairs = float(n) * (case["targets"] if kind == "targets" else n)
    pairs *= {"grad": 4, "leapfrog": case["steps"] + 1}.get(kind, 1)
    if kind == "blockstep" or pairs > MAX_DIRECT_PAIRS:
        return None
    pos, mass, g = _particles(case, seed)
    extra = _rest(case, g)
    if kind == "leapfrog":
        x, v, h = pos.double(), extra.double(), _DT
        a = _direct(case, x, mass)["acc"]
        for _ in range(case["steps"]):
            v = v + 0.5 * h * a
            x = x + h * v
            a = _direct(case, x, mass)["acc"]
            v = v + 0.5 * h * a
        return {"pos": x, "vel": v}
    d = _direct(case, pos, mass, targets=extra if kind == "targets" else None, w=extra if kind == "grad" else None)
    if kind == "grad":
        return {k: d[k] for k in ("acc", "grad_pos", "grad_mass")}
    if kind == "evaluate":
        return {"acc": d["acc"], "pot": d["pot"]}
    return d["acc"]
