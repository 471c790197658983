"""The adjoint at the edges of its kernels.

* Near field: leaves from one particle to the largest (the lane groups at 8, 16
  and 32 targets, the second pass above 32), neighbour lists of one to many
  chunks, split units.  With an opening angle of 1e-6 nothing but single
  particles is far (exact to rounding at any order), and the pass is a direct
  sum, whose gradient is summed in FP64 here.  Tolerance: each component is a
  sum of n terms with fewer than 40 roundings each and partial sums below S_i,
  the sum of the terms' magnitudes: |difference| <= (104 + n / 32) 2^-23 S_i, and
  2e-5 S_i for the expansions of the far ones (some hundred roundings each).
* Far field: the sweeps straight to the leaves against the ones level by level
  (the C ABI's other sequence), massless subtrees among them, p99 within the
  1e-4 of the adjoint's parity tests."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from jaccpot_b200 import _lib, engine, tree, workloads  # noqa: E402


def _grad(topo, p, pos, mass, w, eps2, **kw):
    ps = engine.Pass(engine.DeviceTopology(topo, "cuda"), p, G=1.0, eps2=eps2, **kw)
    ps.load_particles(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda())
    gx = torch.empty(pos.shape, device="cuda")
    gm = torch.empty(pos.shape[0], device="cuda")
    ps.vjp(torch.from_numpy(w).cuda(), gx, gm)
    return gx.double().cpu().numpy(), gm.double().cpu().numpy()


@pytest.mark.parametrize("n,leaf,sources", [(1, 16, 4096), (2, 16, 4096), (8, 8, 4096), (9, 9, 4096), (16, 16, 4096),
                                            (17, 17, 4096), (32, 32, 4096), (33, 33, 4096), (64, 64, 4096),
                                            (700, 2, 4096), (700, 11, 4096), (700, 25, 4096), (700, 64, 4096),
                                            (5000, 40, 4096), (900, 30, 100)])
def test_near_field_gradient_is_the_direct_sum(n, leaf, sources):
    pos, mass = workloads.plummer(n, 3)
    mass = (mass * np.linspace(0.5, 2.0, n)).astype(np.float32)
    w = np.random.default_rng(1).normal(size=(n, 3)).astype(np.float32)
    topo = tree.build_topology(pos, mass, leaf_size=leaf, theta=1e-6, device="cuda")
    gx, gm = _grad(topo, 6, pos, mass, w, 0.0, leaf_unit_sources=sources)
    x, m, ww = pos.astype(np.float64), mass.astype(np.float64), w.astype(np.float64)
    d = x[:, None] - x[None]
    r2 = (d ** 2).sum(-1)
    np.fill_diagonal(r2, np.inf)
    q = 1.0 / np.sqrt(r2)
    u = m[None, :, None] * ww[:, None] - m[:, None, None] * ww[None]
    ud = (u * d).sum(-1)
    tx = -(q ** 3)[..., None] * u + 3 * (q ** 5 * ud)[..., None] * d
    tm = q ** 3 * (ww[None] * d).sum(-1)
    size = (q ** 3 * (m[None] * np.linalg.norm(ww, axis=1)[:, None] + m[:, None] * np.linalg.norm(ww, axis=1)[None])).sum(1)
    msize = (q ** 2 * np.linalg.norm(ww, axis=1)[None]).sum(1)
    tol = (104 + n / 32) * 2.0 ** -23
    far = 2e-5 if topo.num_far_pairs else 0.0
    assert (np.abs(gx - tx.sum(1)).max(1) <= (4 * tol + far) * size + 1e-30).all()
    assert (np.abs(gm - tm.sum(1)) <= (tol + far) * msize + 1e-30).all()


def _level_vjp(ps, w):
    """The adjoint by the level sweeps of the C ABI, on a pass that has its
    particles loaded."""
    lb, t, dt, ws = ps.lib, ps.dt.topo, ps.dt, ps.ws
    ps.run(cascade=True)  # complete locals at every node
    A = ps._adj_buffers()
    P = lambda x: x.data_ptr()
    s = torch.cuda.current_stream().cuda_stream
    ok = lambda rc: _lib.check(rc, "adjoint")
    n = t.num_particles
    xm4, cbar4 = torch.empty((n, 4), device="cuda"), torch.zeros((t.num_nodes, 4), device="cuda")
    mbar = torch.zeros_like(A["mbar"])
    ok(lb.jb_gather_sorted(n, P(w), P(A["zeros"]), P(dt.perm), P(A["w4"]), s))
    sc, msc, lo = A["sched"], A["m2l"], dt.level_offsets
    ok(lb.jb_adj_near(P(ws.pos4), P(A["w4"]), t.num_internal, int(sc.units.shape[0]), P(A["units"]), P(A["aux"]),
                      P(A["runs"]), P(dt.node_ranges), ps.G, ps.eps2, P(xm4), P(A["partials"]),
                      int(sc.split.shape[0]), P(A["split"]), s))
    ok(lb.jb_adj_leaf_far(ps.p, P(ws.pos4), P(A["w4"]), t.num_nodes, t.num_internal, P(dt.node_ranges), P(ws.centers),
                          P(ws.locals), ps.G, P(xm4), P(A["lbar"]), P(cbar4), s))
    for v in range(t.num_levels - 1, -1, -1):
        ok(lb.jb_adj_l2l_level(ps.p, lo[v], lo[v + 1], P(dt.left), P(dt.right), P(ws.centers), P(ws.locals),
                               P(A["lbar"]), P(cbar4), s))
    ok(lb.jb_adj_m2l(ps.p, int(msc.units.shape[0]), P(A["m2l_units"]), P(A["lbar"]), P(ws.centers), P(dt.far_src),
                     P(mbar), P(A["m2l_partials"]), int(msc.split.shape[0]), P(A["m2l_split"]), s))
    ok(lb.jb_adj_m2l_centers(ps.p, t.num_nodes, t.num_far_pairs, P(A["pair_tgt"]), P(dt.far_src), P(dt.far_off),
                             P(A["rev"]), P(ws.mult), P(A["lbar"]), P(ws.centers), P(A["g4"]), P(cbar4), s))
    for v in range(t.num_levels):
        ok(lb.jb_adj_m2m_level(ps.p, lo[v], lo[v + 1], P(dt.left), P(dt.right), P(ws.centers), P(ws.mult), P(mbar),
                               P(cbar4), s))
    ok(lb.jb_adj_p2m(ps.p, P(ws.pos4), t.num_nodes, t.num_internal, P(dt.node_ranges), P(ws.centers), P(mbar),
                     P(cbar4), P(xm4), s))
    out = torch.empty_like(xm4)
    out[dt.perm] = xm4
    return out.double().cpu().numpy()


@pytest.mark.parametrize("kind,n,p,leaf,massless", [("clustered", 3000, 2, 4, True), ("clustered", 3000, 5, 16, True),
                                                    ("plummer", 4000, 9, 32, True), ("clustered", 20_000, 6, 1, False),
                                                    ("uniform", 50, 4, 64, True), ("plummer", 60_000, 8, 32, False)])
def test_sweeps_straight_to_the_leaves_match_the_level_sweeps(kind, n, p, leaf, massless):
    pos, mass = workloads.GENERATORS[kind](n, 7)
    mass = (mass / mass.mean()).astype(np.float32)
    if massless:
        mass[np.argsort(pos[:, 0])[:n // 4]] = 0.0
    topo = tree.build_topology(pos, mass, leaf_size=leaf, theta=0.6, device="cuda")
    w = np.random.default_rng(2).normal(size=(n, 3)).astype(np.float32)
    gx, gm = _grad(topo, p, pos, mass, w, 1e-2)
    ps = engine.Pass(engine.DeviceTopology(topo, "cuda"), p, G=1.0, eps2=1e-2)
    ps.load_particles(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda())
    want = _level_vjp(ps, torch.from_numpy(w).cuda())
    wx, wm = want[:, :3], want[:, 3]
    assert np.isfinite(gx).all() and np.isfinite(gm).all() and np.isfinite(want).all()
    ex = np.linalg.norm(gx - wx, axis=1) / np.maximum(np.linalg.norm(wx, axis=1), 1e-3 * np.abs(wx).max())
    em = np.abs(gm - wm) / np.maximum(np.abs(wm), 1e-3 * np.abs(wm).max())
    assert np.percentile(ex, 99) <= 1e-4, np.percentile(ex, [50, 99, 100])
    assert np.percentile(em, 99) <= 1e-4, np.percentile(em, [50, 99, 100])


@pytest.mark.parametrize("cotangent", ["constant", "position", "mass", "few"])
@pytest.mark.parametrize("masses", ["equal", "spread"])
@pytest.mark.parametrize("n,leaf,sources", [(60, 8, 4096), (700, 16, 4096), (700, 25, 4096), (900, 30, 100),
                                            (1500, 64, 4096)])
def test_near_field_gradient_cancels_within_the_pair(n, leaf, sources, masses, cotangent):
    """Cotangents that vary slowly between neighbours, on particles of which half
    have a neighbour at a thousandth of the usual distance: the pair's m_l w_k -
    m_k w_l is far below its two terms.  Each component is a sum of n terms of at
    most 4 q^3 |m_l w_k - m_k w_l|, T_i in all, each with fewer than 85
    roundings, the differences among them rounded at their own size:
    |difference| <= (104 + n / 32) 2^-23 T_i.  With a constant cotangent on equal
    masses, or one proportional to the masses, T_i and the gradient are 0."""
    rng = np.random.default_rng(5)
    pos, mass = workloads.plummer(n, 3)
    pos[n // 2:] = pos[:n - n // 2] + 1e-3 * rng.normal(size=(n - n // 2, 3))
    pos = pos.astype(np.float32)
    mass = np.full(n, 1.0 / n) if masses == "equal" else np.exp(2.0 * rng.normal(size=n)) / n
    mass = mass.astype(np.float32)
    # halves and doubles are exact, so that "mass" is proportional in FP32 too
    w = {"constant": np.full((n, 3), 0.7), "position": pos, "mass": mass[:, None] * np.array([0.5, 2.0, 1.0]),
         "few": np.where(np.arange(n)[:, None] % 20 == 0, rng.normal(size=(n, 3)), 0.0)}[cotangent].astype(np.float32)
    topo = tree.build_topology(pos, mass, leaf_size=leaf, theta=1e-6, device="cuda")
    assert topo.num_far_pairs == 0
    gx, _ = _grad(topo, 4, pos, mass, w, 0.0, leaf_unit_sources=sources)
    x, m, ww = pos.astype(np.float64), mass.astype(np.float64), w.astype(np.float64)
    d = x[:, None] - x[None]
    r2 = (d ** 2).sum(-1)
    np.fill_diagonal(r2, np.inf)
    q = 1.0 / np.sqrt(r2)
    y = m[None, :, None] * ww[:, None] - m[:, None, None] * ww[None]
    want = ((q ** 3)[..., None] * (3 * (q ** 2 * (y * d).sum(-1))[..., None] * d - y)).sum(1)
    size = (4 * q ** 3 * np.linalg.norm(y, axis=-1)).sum(1)
    assert (np.abs(gx - want).max(1) <= (104 + n / 32) * 2.0 ** -23 * size).all()
