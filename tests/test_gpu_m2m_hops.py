"""The M2M by hops: its items form every internal node once, from sources that
tile its particles and were finished by the hops before, each node's items
aligned within a block's 32; and the upward sweep through them gives the
level sweep's accelerations (both in FP32; p99 within the 1e-5 of every FP32
parity test) on shallow, deep and tiny trees, with massless subtrees."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from jaccpot_b200 import engine, tree, workloads  # noqa: E402

CASES = [("uniform", 20, 16, 3), ("uniform", 40, 16, 8), ("plummer", 5000, 1, 2), ("clustered", 9001, 8, 6),
         ("uniform", 30_000, 32, 10), ("clustered", 120_000, 16, 4)]


@pytest.mark.parametrize("singles", [0, 1, 3, 16])
@pytest.mark.parametrize("kind,n,leaf,p", CASES, ids=lambda c: str(c))
def test_items_and_sweep(monkeypatch, kind, n, leaf, p, singles):
    monkeypatch.setattr(engine, "m2m_single_levels", lambda num_internal: singles)
    pos, mass = workloads.GENERATORS[kind](n, 6)
    mass = mass.copy()
    mass[np.argsort(pos[:, 0])[:n // 3]] = 0.0  # whole subtrees without mass
    topo = tree.build_topology(pos, mass, leaf_size=leaf, theta=0.6, device="cuda")
    dt = engine.DeviceTopology(topo, "cuda")
    items, off = dt.m2m_hops()
    items = items.cpu().numpy()
    ranges, ni = topo.node_ranges, topo.num_internal
    assert off[0] == 0 and off[-1] == items.shape[0] and np.all(off % 32 == 0)
    done = np.zeros(topo.num_nodes, bool)
    done[ni:] = True
    for a, b in zip(off[:-1], off[1:]):
        hop, now = items[a:b], []
        dst = hop[:, 0]
        heads = np.nonzero((dst >= 0) & np.concatenate([[True], dst[1:] != dst[:-1]]))[0]
        assert np.unique(dst[heads]).size == heads.size
        for h in heads:
            size = int((dst[h:h + 16] == dst[h]).sum())
            assert size in (2, 4, 8, 16) and h % size == 0
            src = hop[h:h + size, 1]
            src = src[src >= 0]
            assert size // 2 < src.size <= size and done[src].all()
            r = ranges[src]
            assert r[0, 0] == ranges[dst[h], 0] and r[-1, 1] == ranges[dst[h], 1]
            assert np.array_equal(r[1:, 0], r[:-1, 1] + 1)
            now.append(dst[h])
        assert not done[now].any()
        done[now] = True
    assert done.all()

    ps = engine.Pass(dt, p, G=1.0, eps2=1e-6)
    ps.load_particles(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda())
    out = {}
    for hops in (False, True):
        ps.m2m_hops = hops
        ps.ws.mult.fill_(float("nan"))
        ps.ws.centers.fill_(float("nan"))
        out[hops] = ps.run().clone().double().cpu().numpy()
        assert np.isfinite(ps.ws.mult.cpu().numpy()).all() and np.isfinite(ps.ws.centers.cpu().numpy()).all()
    e = workloads.relative_errors(out[True][:, :3], out[False][:, :3])
    assert np.percentile(e, 99) <= 1e-5, np.percentile(e, [50, 99, 100])
