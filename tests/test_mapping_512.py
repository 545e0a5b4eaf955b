"""Groups of 512 threads by request: the option, the dictionary key, and on the GPU
the kernels at panel, warp and species-per-thread edges, against the oracle.

Tolerances as in test_gpu_groups.py and test_gpu_sources.py."""
import numpy as np
import pytest

from fcs import _lib, foam_io


def test_dictionary_key(tmp_path, lib_path):
    path = str(tmp_path / "chemistryProperties")
    foam_io.write_chemistry_properties(path, mapping="block512")
    o, _ = _lib.read_chemistry_properties(path)
    assert o.mapping == 512
    foam_io.write_chemistry_properties(path, mapping="block1024")
    with pytest.raises(_lib.FcsError):
        _lib.read_chemistry_properties(path)


@pytest.mark.gpu
@pytest.mark.parametrize("ns,solver,precision", [(10, "OptRodas34", "fp64"), (13, "OptSeulex", "fp64"),
                                                 (31, "OptRosenbrock34", "fp64"), (65, "OptRodas34", "fp64"),
                                                 (130, "OptRodas34", "fp64"), (34, "OptRodas34", "mixed")])
def test_step_matches_oracle(ns, solver, precision):
    import __graft_entry__
    __graft_entry__.build()
    import oracle
    from test_gpu_groups import small_case
    flat, cells = small_case(ns, n=24)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    ctx.set_options(solver=solver, precision=precision, mapping=512)
    out = ctx.integrate(cells, 1e-6)
    if precision == "fp64":
        ref = oracle.Port(flat).integrate(cells, 1e-6, solver=solver)
    else:  # the oracle has no mixed precision: the same step on 256 threads
        ctx.set_options(solver=solver, precision=precision, mapping=256)
        ref = ctx.integrate(cells, 1e-6)
    assert out["stats"]["mapping"] == 512 and (out["status"] == 0).all()
    np.testing.assert_allclose(out["T"], ref["T"], rtol=1e-7, atol=0)
    np.testing.assert_allclose(out["Y"], ref["Y"], rtol=0, atol=1e-8)


@pytest.mark.gpu
@pytest.mark.parametrize("ns", [10, 63, 130, 255])
def test_evaluations_match_oracle(ns):
    import __graft_entry__
    __graft_entry__.build()
    import oracle
    from test_gpu_groups import small_case
    flat, c = small_case(ns, n=7)
    port = oracle.Port(flat)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    ctx.set_options(mapping=512)
    RR0, _ = port.rates(c.p, c.T, c.rho0, c.Y)
    RR, _ = ctx.rates(c.p, c.T, c.rho0, c.Y)
    assert (np.abs(RR - RR0) <= 1e-10 * np.abs(RR0).max(axis=0)).all()
    J0, _ = port.jacobian(c.p, c.T, c.Y)
    J, _ = ctx.jacobian(c.p, c.T, c.Y)
    assert (np.abs(J - J0) <= 1e-11 * np.abs(J0).max(axis=(1, 2), keepdims=True)).all()
    np.testing.assert_allclose(ctx.tc(c.p, c.T, c.rho0, c.Y), port.tc(c.p, c.T, c.rho0, c.Y), rtol=1e-10)


@pytest.mark.gpu
def test_a_reported_mapping_can_be_asked_for():
    """AUTO takes 512 threads from 128 species on; the same step by request has the
    same result to the tolerance of another summation width."""
    import __graft_entry__
    __graft_entry__.build()
    from test_gpu_groups import small_case
    flat, cells = small_case(140, n=8)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    a = ctx.integrate(cells, 1e-7)
    ctx.set_options(mapping=a["stats"]["mapping"])
    b = ctx.integrate(cells, 1e-7)
    assert a["stats"]["mapping"] == b["stats"]["mapping"] == 512
    np.testing.assert_allclose(a["T"], b["T"], rtol=1e-7, atol=0)
    for bad in (2, 16, 384, 1024):
        with pytest.raises(_lib.FcsError):
            ctx.set_options(mapping=bad)
