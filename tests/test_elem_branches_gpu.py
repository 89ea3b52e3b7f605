"""The element kernels' wet branch against the general one: states with depths at the edges of its rule (zero, the
FD step above it, just below and above twice it, dry at one level only), element by element against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau", [0.0, 0.5])
def test_depths_around_the_wet_rule_are_bit_exact(tau):
    from adh_kraken_b200.capi import SW2Model
    from adh_kraken_b200.mesh import small_delaunay_case
    from oracle.oracle import OracleModel
    case = small_delaunay_case(n=20, seed=11, nsteps=1)
    rng = np.random.default_rng(4)
    V = case.nnodes
    edge = np.array([0.0, -0.0, 1e-20, 9.9e-5, 1e-4, 1.0001e-4, 1.9999e-4, 2e-4, 2.0001e-4, 1e-3, 0.5, 1.5, -1e-20, -0.3])
    o = OracleModel(case, tau_temporal=tau)
    g = SW2Model(case)
    d, vx, vy = o.bc_values(case.t0, case.t0 + case.dt)
    g.set_step(case.dt, d, vx, vy, tau_temporal=tau)
    for share in (0.02, 0.3, 1.0):               # few, some, all nodes at an edge depth, per level
        levels = []
        for _ in range(3):
            s = case.sol0.copy()
            s[0::3] = np.abs(s[0::3]) + 0.5
            s[1::3] += 0.3 * rng.standard_normal(V)
            s[2::3] += 0.3 * rng.standard_normal(V)
            pick = rng.random(V) < share
            s[0::3][pick] = rng.choice(edge, pick.sum())
            levels.append(s)
        o.wd_flags(levels[0], levels[1])
        with np.errstate(all="ignore"):
            rt, rs = o.elem_resid(*levels)
            jt, js = o.elem_jac(*levels)
        a, b = g.elem_resid(*levels)
        assert np.array_equal(a, rt, equal_nan=True) and np.array_equal(b, rs, equal_nan=True)
        a, b = g.elem_jac(*levels)
        assert np.array_equal(a, jt, equal_nan=True) and np.array_equal(b, js, equal_nan=True)
        assert np.array_equal(g.residual(*levels), o.residual(*levels), equal_nan=True)
