"""The chemical time scale where species' Gibbs factors exp(-G/RT) overflow, vanish
or are subnormal, alone and in products with each other, against the oracle.

Tolerance: as in test_gpu_sources.py, a quotient of positive sums, 1e-10
relative."""
import numpy as np
import pytest

import fcs
from fcs.workloads import RU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponents", [(800.0, 0.0), (-800.0, 0.0), (800.0, -800.0), (-720.0, 0.0), (-720.0, -720.0),
                                       (400.0, -400.0), (800.0, 800.0)])
def test_time_scale_beyond_the_range_of_the_gibbs_factors(exponents):
    import oracle
    from fcs import _lib
    ns, n, T0 = 12, 40, 1000.0
    flat = fcs.flatten(fcs.synthetic_mechanism(name="range", n_species=ns, n_reactions=60, n_third_body=4, n_plog=2,
                                               seed=21))
    # -G/RT of every other species shifted through the enthalpy coefficient a5 (its exponent is -a5/T)
    for a in (flat.low_coeffs, flat.high_coeffs):
        c = a.reshape(ns, 7)
        c[0::4, 5] -= exponents[0] * T0
        c[2::4, 5] -= exponents[1] * T0
    rng = np.random.default_rng(3)
    T, p = rng.uniform(0.999 * T0, 1.001 * T0, n), rng.uniform(1e5, 1e6, n)
    Y = np.ascontiguousarray(rng.dirichlet(np.full(ns, 0.5), size=n).T)
    rho = p / (RU * T * (Y / flat.W[:, None]).sum(axis=0))
    ref = oracle.Port(flat).tc(p, T, rho, Y)
    assert np.isfinite(ref).all()
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    for mapping in (0, 32, 256):
        ctx.set_options(mapping=mapping)
        np.testing.assert_allclose(ctx.tc(p, T, rho, Y), ref, rtol=1e-10)
    ctx.close()
