"""The near field that starts from nothing: near-only and near-first write their
rows without a zeroed buffer.  NaNs in the output buffer beforehand must not
survive, near-first then far-after equals one call bit for bit, near + far the
whole and the near field the one-lane-per-target form's to FP32 rounding (p99
<= 2e-6, as between the forms at every other occupancy), with split leaves,
leaves above 32 particles, the potential and the compensated sums."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from jaccpot_b200 import _lib, engine, tree, workloads  # noqa: E402


@pytest.mark.parametrize("leaf,n,sources", [(1, 1, 4096), (16, 300, 64), (33, 33, 4096), (63, 6000, 4096),
                                            (64, 20_000, 500), (64, 128, 64), (40, 9000, 128)])
@pytest.mark.parametrize("kahan,pot", [(False, False), (True, True)])
def test_nothing_of_the_buffer_survives(leaf, n, sources, kahan, pot):
    pos, mass = workloads.plummer(n, 9)
    topo = tree.build_topology(pos, mass, leaf_size=leaf, theta=0.6, device="cuda")
    ps = engine.Pass(engine.DeviceTopology(topo, "cuda"), 4, G=1.0, eps2=1e-6, leaf_unit_sources=sources,
                     p2p_mode=_lib.JB_P2P_KAHAN if kahan else _lib.JB_P2P_FP32)
    ps.load_particles(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda())
    cols = 4 if pot else 3
    nan = lambda: torch.full((n, 4), float("nan"), device="cuda")
    near = ps.evaluate(part="near", potential=pot, out=nan())
    ps.upward()
    ps.downward()
    far = ps.evaluate(part="far", potential=pot, out=nan())
    whole = ps.evaluate(potential=pot, out=nan())
    two = ps.evaluate(part="near_first", potential=pot, out=nan())
    ps.evaluate(part="far_after", potential=pot, out=two)
    assert torch.isfinite(near[:, :cols]).all() and torch.isfinite(far[:, :cols]).all()
    assert torch.equal(whole[:, :cols], two[:, :cols])
    lb = _lib.lib()
    try:
        lb.jb_set_leaf_form(0)
        lane = ps.evaluate(part="near", potential=pot, out=nan())
    finally:
        lb.jb_set_leaf_form(1)
    for got, want in ((near, lane), (near + far, whole)):
        e = workloads.relative_errors(got[:, :3].cpu().numpy(), want[:, :3].cpu().numpy())
        assert np.percentile(e, 99) <= 2e-6, np.percentile(e, [50, 99, 100])
    if pot:
        assert torch.allclose(near[:, 3], lane[:, 3], rtol=2e-6)
