"""Source terms, right-hand side and chemical time scale at the edges of their
launches (cells per block, threads per cell, cells of a grid), against the
oracle.

Tolerances: a net rate is a difference of its forward and reverse parts, summed
over the reactions of a species, so its error is bounded by the rounding of the
largest species' rate: 1e-10 of that (test_gpu_parity.py bounds the rates the
same way); the time scale is a quotient of positive sums, 1e-10 relative."""
import numpy as np
import pytest

import fcs
from fcs.workloads import RU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [10, 32, 63, 64, 130])
@pytest.mark.parametrize("n", [1, 5, 257])
def test_sources_match_oracle(ns, n):
    import oracle
    from fcs import _lib
    flat = fcs.flatten(fcs.synthetic_mechanism(name=f"src_{ns}", n_species=ns, n_reactions=3 * ns, n_third_body=2,
                                               n_plog=1, seed=2000 + ns))
    rng = np.random.default_rng(n)
    T, p = rng.uniform(900.0, 2000.0, n), rng.uniform(1e5, 1e6, n)
    Y = np.ascontiguousarray(rng.dirichlet(np.full(ns, 0.5), size=n).T)
    rho = p / (RU * T * (Y / flat.W[:, None]).sum(axis=0))
    port = oracle.Port(flat)
    RR0, Q0 = port.rates(p, T, rho, Y)
    f0, t0 = port.rhs(p, T, Y), port.tc(p, T, rho, Y)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    for mapping in (0, 32, 64, 128, 256):
        ctx.set_options(mapping=mapping)
        RR, Q = ctx.rates(p, T, rho, Y)
        assert (np.abs(RR - RR0) <= 1e-10 * np.abs(RR0).max(axis=0)).all()
        hf = np.abs(RR0).max(axis=0) * 1e9 * ns  # |Hf| stays below 1e9 J/kg
        assert (np.abs(Q - Q0) <= 1e-10 * hf).all()
        f = ctx.rhs(p, T, Y)
        assert (np.abs(f - f0)[:ns] <= 1e-10 * np.abs(f0[:ns]).max(axis=0)).all()
        # dT/dt sums Ha dY / cp: |Ha| / cp below 1e5 K
        assert (np.abs(f - f0)[ns] <= 1e-10 * (np.abs(f0[ns]) + 1e5 * np.abs(f0[:ns]).max(axis=0))).all()
        np.testing.assert_allclose(ctx.tc(p, T, rho, Y), t0, rtol=1e-10)
    ctx.close()


@pytest.mark.parametrize("ns,special", [(10, 0), (14, 4), (34, 0), (63, 0), (64, 0), (112, 0), (130, 0), (200, 0)])
def test_jacobian_matches_oracle_on_every_group(ns, special):
    """AUTO takes other groups for few cells than for many: the same bits.  Against
    the oracle 1e-11 of a cell's largest element (test_gpu_parity.py: 1e-12 of the
    largest, for up to 111 species)."""
    import oracle
    from fcs import _lib
    flat = fcs.flatten(fcs.synthetic_mechanism(name=f"jac_{ns}", n_species=ns, n_reactions=3 * ns, n_third_body=2,
                                               n_plog=1, n_falloff=(special, 0, 0), seed=3000 + ns))
    n = 3
    rng = np.random.default_rng(ns)
    T, p = rng.uniform(900.0, 2000.0, n), rng.uniform(1e5, 1e6, n)
    Y = np.ascontiguousarray(rng.dirichlet(np.full(ns, 0.5), size=n).T)
    J0, f0 = oracle.Port(flat).jacobian(p, T, Y)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    for mapping in (0, 32, 64, 128, 256):
        ctx.set_options(mapping=mapping)
        J, f = ctx.jacobian(p, T, Y)
        assert (np.abs(J - J0) <= 1e-11 * np.abs(J0).max(axis=(1, 2), keepdims=True)).all()
        if mapping == 0:
            few = J, f
    ctx.set_options(mapping=0)
    many = np.arange(10 * 152 if ns < 64 else 320) % n
    J, f = ctx.jacobian(p[many], T[many], np.ascontiguousarray(Y[:, many]))
    np.testing.assert_array_equal(J[:n], few[0])
    np.testing.assert_array_equal(J[-n:], few[0][many[-n:]])
    np.testing.assert_array_equal(f[:, :n], few[1])
    ctx.close()


@pytest.mark.parametrize("falloff", [(0, 1, 0), (1, 8, 9), (2, 9, 8), (0, 0, 33)])
def test_falloff_rates_match_oracle(falloff):
    """Few Troe or SRI reactions are shared out over four lanes each, more take one
    lane each."""
    import oracle
    from fcs import _lib
    flat = fcs.flatten(fcs.synthetic_mechanism(name="fall", n_species=20, n_reactions=60, n_third_body=2, n_plog=1,
                                               n_falloff=falloff, seed=77))
    n = 33
    rng = np.random.default_rng(5)
    T, p = rng.uniform(900.0, 2000.0, n), 10.0 ** rng.uniform(3.0, 7.0, n)
    Y = np.ascontiguousarray(rng.dirichlet(np.full(20, 0.5), size=n).T)
    rho = p / (RU * T * (Y / flat.W[:, None]).sum(axis=0))
    port = oracle.Port(flat)
    RR0, _ = port.rates(p, T, rho, Y)
    J0, _ = port.jacobian(p, T, Y)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    for mapping in (0, 32, 64, 128, 256):
        ctx.set_options(mapping=mapping)
        RR, _ = ctx.rates(p, T, rho, Y)
        assert (np.abs(RR - RR0) <= 1e-10 * np.abs(RR0).max(axis=0)).all()
        J, _ = ctx.jacobian(p, T, Y)
        assert (np.abs(J - J0) <= 1e-10 * np.abs(J0).max(axis=(1, 2), keepdims=True)).all()
    ctx.close()


def test_groups_of_32_with_a_large_slot():
    """7,500 reactions: four cells' net rates exceed a block's shared memory, so
    fewer cells share a block; the rates have the bits of the larger groups."""
    from fcs import _lib
    flat = fcs.flatten(fcs.synthetic_mechanism(name="many", n_species=60, n_reactions=7500, n_third_body=2, n_plog=1,
                                               seed=9))
    n = 9
    rng = np.random.default_rng(n)
    T, p = rng.uniform(900.0, 2000.0, n), rng.uniform(1e5, 1e6, n)
    Y = np.ascontiguousarray(rng.dirichlet(np.full(60, 0.5), size=n).T)
    rho = p / (RU * T * (Y / flat.W[:, None]).sum(axis=0))
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    out = []
    for mapping in (32, 64, 256):
        ctx.set_options(mapping=mapping)
        out.append(ctx.rates(p, T, rho, Y)[0])
    np.testing.assert_array_equal(out[0], out[1])
    np.testing.assert_array_equal(out[0], out[2])
    assert np.isfinite(out[0]).all() and np.abs(out[0]).max() > 0
    ctx.close()
