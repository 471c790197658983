"""Pass.launches_per_run against the kernels that the profiler sees in one run(),
for each form of the sweeps and the M2L."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from torch.profiler import ProfilerActivity, profile  # noqa: E402

from jaccpot_b200 import engine, tree, workloads  # noqa: E402


def _kernels(ps):
    ps.run()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        ps.run()
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    if not names:
        pytest.skip("the profiler has no kernel records on this machine")
    return sum("k_" in name for name in names)


@pytest.mark.parametrize("form", ["direct", "hops off", "cascade", "split leaves and targets", "mixed", "per_gear",
                                  "nothing far"])
def test_count_equals_the_profiler(form):
    n = 40 if form == "nothing far" else 20_000
    pos, mass = workloads.GENERATORS["clustered"](n, 3)
    topo = tree.build_topology(pos, mass, leaf_size=64 if n == 40 else 16, theta=0.6, device="cuda")
    kw = {"split leaves and targets": dict(m2l_unit_pairs=8, leaf_unit_sources=64),
          "per_gear": dict(gear_form="per_gear")}.get(form, {})
    ps = engine.Pass(engine.DeviceTopology(topo, "cuda"), 4, **kw)
    if form in ("mixed", "per_gear"):
        gears = torch.arange(topo.num_far_pairs, device="cuda", dtype=torch.int32) % 2
        ps.set_gears(gears, (2, 4))
    ps.m2m_hops = ps.m2m_hops and form != "hops off"
    ps.l2l_direct = form != "cascade"
    ps.load_particles(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda())
    assert ps.launches_per_run() == _kernels(ps)
