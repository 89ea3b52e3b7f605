"""The element kernels' wet, dry and general branches, chosen by warp: strips of the mesh at the edges of the rules (zero, the
FD step, twice it, on both sides), so that whole warps hold one value and others mix two, at the current level alone or
at all three; on both sides of the line between the small grids' kernels and the large ones' (148 SMs: 12,544 triangles).
Element by element against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = np.array([-0.3, -2.0001e-4, -2e-4, -1.9999e-4, -1e-4, -1e-20, -0.0, 0.0, 1e-20, 1e-4, 1.9999e-4, 2e-4, 2.0001e-4, 0.5])


# 2 (n - 1)^2 triangles: 722, 12,482, 12,800
@pytest.mark.parametrize("n,tau", [(20, 0.0), (20, 0.5), (80, 0.5), (81, 0.0)])
def test_branches_are_bit_exact(n, tau):
    from adh_kraken_b200.capi import SW2Model
    from adh_kraken_b200.mesh import small_delaunay_case
    from oracle.oracle import OracleModel
    case = small_delaunay_case(n=n, seed=3, nsteps=1)
    V = case.nnodes
    rng = np.random.default_rng(n)
    o, g = OracleModel(case, tau_temporal=tau), SW2Model(case)
    d, vx, vy = o.bc_values(case.t0, case.t0 + case.dt)
    g.set_step(case.dt, d, vx, vy, tau_temporal=tau)
    column = np.arange(V) // n
    strips = EDGES[column // 4 % len(EDGES)]
    dry = np.full(V, -0.3)
    few = np.where(rng.random(V) < 0.01, rng.choice(EDGES, V), -0.3)
    wet = np.where(column % 2 == 0, 0.5, 1.5)
    # the depths of the three levels: all dry, dry with few other values, strips at all levels, at the current one over dry and
    # over wet older levels, and at the older ones under a dry current one
    for levels in ((dry, dry, dry), (few, dry, few), (strips, strips, strips), (strips, dry, dry), (strips, wet, wet), (dry, strips, wet),
                   (dry, dry, strips)):
        s = [np.stack([h, 0.3 * rng.standard_normal(V), 0.3 * rng.standard_normal(V)], axis=1).ravel() for h in levels]
        o.wd_flags(s[0], s[1])
        with np.errstate(all="ignore"):
            rt, rs = o.elem_resid(*s)
            jt, js = o.elem_jac(*s)
        a, b = g.elem_resid(*s)
        assert np.array_equal(a, rt, equal_nan=True) and np.array_equal(b, rs, equal_nan=True)
        a, b = g.elem_jac(*s)
        assert np.array_equal(a, jt, equal_nan=True) and np.array_equal(b, js, equal_nan=True)
