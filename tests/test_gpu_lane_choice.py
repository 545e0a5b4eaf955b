"""AUTO between three quarters of a cell and 1.1 cells per lane (FP64, 32 to 63
species): the cells' predicted costs choose between lanes and groups, on the host's
path as inside a graph and an asynchronous step, with the same bits."""
import numpy as np
import pytest

from test_gpu_groups import small_case

pytestmark = pytest.mark.gpu
DT = 1e-10  # a few attempts a cell


@pytest.mark.parametrize("ns", [34, 50])
@pytest.mark.parametrize("equal", [True, False])
def test_costs_choose_the_mapping(ns, equal):
    import __graft_entry__
    __graft_entry__.build()
    import torch
    from fcs import _lib
    flat, few = small_case(ns, n=16)
    n = 54000  # of 58,368 lanes
    c = few.subset(np.arange(n) % 16)
    # a predicted step count of 4 for every cell, or 1 for most and 64 for one in 64
    c.subDt[:] = DT / 4.5 if equal else np.where(np.arange(n) % 64 == 0, DT / 70, DT)

    def run(mapping, how, times=1):
        ctx = _lib.Context(0)
        ctx.load_mechanism(flat)
        ctx.set_options(mapping=mapping)
        d = {k: torch.from_numpy(np.ascontiguousarray(getattr(c, k))).cuda() for k in ("p", "rho0", "T", "Y", "subDt")}
        RR, st = torch.zeros_like(d["Y"]), torch.zeros(n, dtype=torch.int32, device="cuda")
        start = {k: d[k].clone() for k in ("T", "Y", "subDt")}
        for _ in range(times):
            for k, v in start.items():
                d[k].copy_(v)
            torch.cuda.synchronize()
            a = (n, DT, d["p"], d["rho0"], d["T"], d["Y"], d["subDt"], RR, st)
            if how == "async":
                ctx.integrate_async(*a)
                code, stats, dmin = ctx.sync()
            else:
                code, stats, dmin = ctx.integrate_raw(*a, device=True, flags=_lib.CUDA_GRAPH if how == "graph" else 0)
        assert stats["cells_integrated"] == n and stats["cells_failed"] == 0
        return stats["mapping"], dmin, [v.cpu().numpy() for v in (d["T"], d["Y"], d["subDt"], RR, st)]

    _, dmin0, ref = run(1, "plain")
    for how in ("plain", "graph", "async"):
        mapping, dmin, out = run(0, how)
        assert (mapping == 1) == equal, how
        assert dmin == dmin0
        for x, y in zip(ref, out):
            np.testing.assert_array_equal(x, y)
    # the second call goes by the attempts that the first one counted
    for how in ("plain", "graph", "async"):
        _, dmin, out = run(0, how, times=3)
        assert dmin == dmin0
        for x, y in zip(ref, out):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("flags,n,mapping", [("natural order", 54000, 1), ("", 43000, 64), ("", 65000, 1)])
def test_outside_the_choice(flags, n, mapping):
    """Below three quarters of a cell per lane groups, from 1.1 on lanes, and lanes
    where the queue keeps the natural order (no predicted costs)."""
    import __graft_entry__
    __graft_entry__.build()
    from fcs import _lib
    flat, few = small_case(34, n=16)
    c = few.subset(np.arange(n) % 16)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    T, Y, sub, RR, st = c.T.copy(), c.Y.copy(), c.subDt.copy(), np.zeros_like(c.Y), np.zeros(n, np.int32)
    code, stats, _ = ctx.integrate_raw(n, DT, c.p, c.rho0, T, Y, sub, RR, st, flags=2 if flags else 0)
    assert stats["mapping"] == mapping and stats["cells_integrated"] == n


@pytest.mark.parametrize("how", ["plain", "graph"])
def test_groups_where_the_lanes_workspace_has_no_room(how):
    """Equal costs want the lanes; when their workspace cannot be allocated the groups
    run, with the same result."""
    import __graft_entry__
    __graft_entry__.build()
    import torch
    from fcs import _lib
    flat, few = small_case(34, n=16)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)

    def step(n, equal, flags, fails):
        c = few.subset(np.arange(n) % 16)
        c.subDt[:] = DT / 4.5 if equal else np.where(np.arange(n) % 64 == 0, DT / 70, DT)
        d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (c.p, c.rho0, c.T, c.Y, c.subDt)]
        torch.cuda.synchronize()
        _lib.fail_allocations(fails)
        try:
            code, stats, _ = ctx.integrate_raw(n, DT, *d, device=True, flags=flags)
        finally:
            _lib.fail_allocations(0)
        assert code == 0 and stats["cells_integrated"] == n
        return stats["mapping"], [v.cpu().numpy() for v in d[2:]]

    step(54400, False, 0, 0)  # groups: grows the other buffers, and another batch size keeps no costs
    flags = _lib.CUDA_GRAPH if how == "graph" else 0
    mapping, a = step(54000, True, flags, 1)
    assert mapping > 1
    _, b = step(54000, True, flags, 0)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
