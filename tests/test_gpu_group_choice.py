"""AUTO's threads per cell where the cells that reside decide: other groups for few
cells than for many, with the same bits."""
import numpy as np
import pytest

from test_gpu_groups import small_case

pytestmark = pytest.mark.gpu


# sizes around those where another cell fits or stops fitting an SM
@pytest.mark.parametrize("ns,solver,precision,many", [
    (34, "OptRodas34", "fp64", (64,)), (53, "OptRodas34", "mixed", (64, 128)), (64, "OptRodas34", "fp64", (64,)),
    (70, "OptRosenbrock34", "fp64", (64, 128)), (80, "OptRodas34", "fp64", (128,)), (70, "OptSeulex", "fp64", (64, 128)),
    (80, "OptRodas34", "mixed", (64, 128)), (100, "OptRodas34", "fp64", (128,))])
def test_auto_takes_smaller_groups_for_many_cells(ns, solver, precision, many):
    import __graft_entry__
    __graft_entry__.build()
    from fcs import _lib
    flat, cells = small_case(ns, n=8)
    outs = []
    for n in (8, 10 * 152):
        ctx = _lib.Context(0)
        ctx.load_mechanism(flat)
        ctx.set_options(solver=solver, precision=precision)
        outs.append(ctx.integrate(cells.subset(np.arange(n) % 8), 1e-7))
    a, b = outs
    assert a["stats"]["mapping"] == (128 if ns < 64 else 256)
    assert b["stats"]["mapping"] in many
    for k in ("T", "Y", "subDt", "RR", "status"):
        assert np.array_equal(a[k], b[k][..., :8]) and np.array_equal(a[k], b[k][..., -8:]), k


@pytest.mark.parametrize("ns", [111, 127])
def test_one_resident_cell_keeps_the_wide_group(ns):
    import __graft_entry__
    __graft_entry__.build()
    from fcs import _lib
    flat, cells = small_case(ns, n=8)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    out = ctx.integrate(cells.subset(np.arange(10 * 152) % 8), 1e-8)
    assert out["stats"]["mapping"] == 256


@pytest.mark.parametrize("ns,solver,precision", [(12, "OptRodas34", "fp64"), (34, "OptSeulex", "mixed"),
                                                 (65, "OptRosenbrock23", "fp64"), (80, "OptRodas34", "mixed"),
                                                 (100, "OptRodas34", "fp64"), (111, "OptSeulex", "fp64")])
def test_two_blocks_of_256_threads_give_the_bits_of_one(ns, solver, precision):
    """Many cells take the kernel compiled for two blocks per SM."""
    import __graft_entry__
    __graft_entry__.build()
    from fcs import _lib
    flat, cells = small_case(ns, n=8)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    ctx.set_options(solver=solver, precision=precision, mapping=256)
    a, b = [ctx.integrate(cells.subset(np.arange(n) % 8), 1e-7) for n in (8, 5 * 152)]
    assert a["stats"]["mapping"] == 256 == b["stats"]["mapping"] and (a["status"] == 0).all()
    for k in ("T", "Y", "subDt", "RR", "status"):
        assert np.array_equal(a[k], b[k][..., :8]) and np.array_equal(a[k], b[k][..., -8:]), k


@pytest.mark.parametrize("ns", [34, 65, 100, 127, 130])
def test_evaluations_have_the_same_bits_under_the_lane_mapping(ns):
    """The lane mapping is the integrator's; the evaluations run on groups whose sums
    are those of 64 threads up to 127 species, of 128 above."""
    import __graft_entry__
    __graft_entry__.build()
    from fcs import _lib
    flat, cells = small_case(ns, n=40)
    outs = []
    for mapping in (0, 1, 64 if ns <= 127 else 128):
        ctx = _lib.Context(0)
        ctx.load_mechanism(flat)
        ctx.set_options(mapping=mapping)
        outs.append((*ctx.rates(cells.p, cells.T, cells.rho0, cells.Y), ctx.rhs(cells.p, cells.T, cells.Y),
                     *ctx.jacobian(cells.p, cells.T, cells.Y)))
    for o in outs[1:]:
        for x, y in zip(outs[0], o):
            np.testing.assert_array_equal(x, y)
