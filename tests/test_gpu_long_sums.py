"""Species that take part in more reactions than a sum's 16-bit count holds: rates
and Jacobian against the oracle.

Tolerances as in test_gpu_sources.py and test_gpu_parity.py, times the length
of the sums: net rates and Jacobian elements are sums over up to 80,000
reactions, so 1e-16 a term of the largest."""
import numpy as np
import pytest

import fcs
from fcs.mechanism import FlatMechanism
from fcs.workloads import RU

pytestmark = pytest.mark.gpu


def repeated(flat, times):
    """The mechanism's plain reactions again and again, their rates divided by that."""
    r = np.nonzero(flat.type == 0)[0]
    side = lambda off, sp: [sp[off[k]:off[k + 1]] for k in r]
    lhs, rhs = side(flat.lhs_offset, flat.lhs_species) * times, side(flat.rhs_offset, flat.rhs_species) * times
    nr, ns = len(lhs), flat.n_species
    off = lambda s: np.concatenate([[0], np.cumsum([len(v) for v in s])]).astype(np.int32)
    arr = np.tile(flat.arrhenius.reshape(-1, 3)[r], (times, 1))
    arr[:, 0] /= times
    return FlatMechanism(
        ns, nr, flat.W, flat.T_low, flat.T_high, flat.T_common, flat.high_coeffs, flat.low_coeffs,
        np.zeros(nr, np.int32), np.tile(flat.reversible[r], times).astype(np.int32), off(lhs),
        np.concatenate(lhs).astype(np.int32), off(rhs), np.concatenate(rhs).astype(np.int32), arr.reshape(-1),
        np.zeros(nr * 3), np.zeros(nr * ns), np.zeros(nr * 5), np.zeros(nr + 1, np.int32), np.zeros(0))


@pytest.mark.parametrize("count", [33000, 65535, 80000])
def test_rates_and_jacobian_of_long_sums(count):
    import oracle
    from fcs import _lib
    small = fcs.flatten(fcs.synthetic_mechanism(name="long sums", n_species=8, n_reactions=24, n_third_body=2, n_plog=0,
                                                seed=31))
    plain = small.type == 0
    per = np.zeros(8, int)
    for k in np.nonzero(plain)[0]:
        for off, sp in ((small.lhs_offset, small.lhs_species), (small.rhs_offset, small.rhs_species)):
            np.add.at(per, sp[off[k]:off[k + 1]], 1)
    flat = repeated(small, -(-count // int(per.max())))
    n = 5
    rng = np.random.default_rng(count)
    T, p = rng.uniform(900.0, 2000.0, n), rng.uniform(1e5, 1e6, n)
    Y = np.ascontiguousarray(rng.dirichlet(np.full(8, 0.5), size=n).T)
    rho = p / (RU * T * (Y / flat.W[:, None]).sum(axis=0))
    port = oracle.Port(flat)
    RR0, _ = port.rates(p, T, rho, Y)
    J0, f0 = port.jacobian(p, T, Y)
    ctx = _lib.Context(0)
    ctx.load_mechanism(flat)
    for mapping in (0, 32, 256):
        ctx.set_options(mapping=mapping)
        RR, _ = ctx.rates(p, T, rho, Y)
        assert (np.abs(RR - RR0) <= 1e-10 * np.abs(RR0).max(axis=0)).all()
        J, f = ctx.jacobian(p, T, Y)
        assert (np.abs(J - J0) <= 1e-10 * np.abs(J0).max(axis=(1, 2), keepdims=True)).all()
        assert (np.abs(f - f0)[:8] <= 1e-10 * np.abs(f0[:8]).max(axis=0)).all()
    ctx.close()
