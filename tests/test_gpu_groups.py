"""The cell-group kernels at the sizes where their tilings end, against the
oracle: matrix orders with every remainder of the four-row LU panels, from
fewer species than lanes to more than a warp, on every group size.

Tolerances are those of the golden comparisons (test_gpu_large.py): 1e-7
relative in T, 1e-8 absolute in Y over one step."""
import numpy as np
import pytest

import fcs
from fcs.workloads import Cells, RU

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def built():
    import __graft_entry__
    __graft_entry__.build()
    return True


def small_case(ns, n=48, seed=3):
    mech = fcs.synthetic_mechanism(name=f"edge_{ns}", n_species=ns, n_reactions=3 * ns, n_third_body=2, n_plog=1,
                                   seed=1000 + ns)
    rng = np.random.default_rng(seed)
    T = rng.uniform(1000.0, 1500.0, n)
    p = rng.uniform(1e5, 1e6, n)
    Y = np.ascontiguousarray(rng.dirichlet(np.full(ns, 0.5), size=n).T)
    rho0 = p / (RU * T * (Y / mech.W[:, None]).sum(axis=0))
    return fcs.flatten(mech), Cells(T, p, Y, rho0, np.full(n, 1e-8))


@pytest.mark.parametrize("ns", [10, 11, 12, 13, 31, 32, 34, 65])
@pytest.mark.parametrize("mapping", [0, 32, 64, 128, 256])
def test_step_matches_oracle_at_panel_and_warp_edges(built, ns, mapping):
    import oracle
    from fcs import _lib
    flat, cells = small_case(ns)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    ctx.set_options(mapping=mapping)
    out = ctx.integrate(cells, 1e-6)
    ref = oracle.Port(flat).integrate(cells, 1e-6)
    assert (out["status"] == 0).all()
    np.testing.assert_allclose(out["T"], ref["T"], rtol=1e-7, atol=0)
    np.testing.assert_allclose(out["Y"], ref["Y"], rtol=0, atol=1e-8)


@pytest.mark.parametrize("ns,solver", [(12, "OptRodas34"), (34, "OptSeulex"), (70, "OptRodas34"), (130, "OptRosenbrock34"),
                                       (70, "OptSeulex")])
def test_auto_results_do_not_depend_on_the_number_of_cells(built, ns, solver):
    """AUTO takes other group sizes for few cells than for many; a cell's result is
    the same to the last bit."""
    from fcs import _lib
    flat, cells = small_case(ns, n=8)
    many = 12 * 152 if ns < 64 else 40
    outs = []
    for idx in (np.arange(8), np.arange(many) % 8):
        ctx = _lib.Context(0)
        ctx.load_mechanism(flat)
        ctx.set_options(solver=solver)
        outs.append(ctx.integrate(cells.subset(idx), 1e-7))
    a, b = outs
    for k in ("T", "Y", "subDt", "RR", "status"):
        assert np.array_equal(a[k], b[k][..., :8]), k


@pytest.mark.parametrize("ns", [34, 70])
def test_auto_equals_its_partial_sum_width(built, ns):
    """Up to 127 species AUTO sums as a group of 64 threads does, on any group."""
    from fcs import _lib
    flat, cells = small_case(ns, n=8)
    outs = []
    for mapping in (0, 64):
        ctx = _lib.Context(0)
        ctx.load_mechanism(flat)
        ctx.set_options(mapping=mapping)
        outs.append(ctx.integrate(cells, 1e-7))
    assert np.array_equal(outs[0]["T"], outs[1]["T"]) and np.array_equal(outs[0]["Y"], outs[1]["Y"])


@pytest.mark.parametrize("ns,solver", [(34, "OptRodas34"), (34, "OptRosenbrock23"), (50, "OptRodas34")])
def test_auto_equals_the_lanes_on_large_batches(built, ns, solver):
    """From three quarters of a cell per lane on AUTO sums as the lane mapping does:
    groups (below 1.1 cells per lane) and lanes give a cell the same bits."""
    from fcs import _lib
    flat, cells = small_case(ns, n=16)
    outs = []
    for mapping, n in ((1, 16), (0, 44000), (0, 66000)):
        ctx = _lib.Context(0)
        ctx.load_mechanism(flat)
        ctx.set_options(solver=solver, mapping=mapping)
        outs.append(ctx.integrate(cells.subset(np.arange(n) % 16), 1e-8))
    assert outs[1]["stats"]["mapping"] > 1 and outs[2]["stats"]["mapping"] == 1
    for o in outs[1:]:
        for k in ("T", "Y", "subDt", "RR", "status"):
            assert np.array_equal(outs[0][k], o[k][..., :16]), k
