"""Restart lengths around the pieces a GMRES cycle is built from: its captured segments (25 steps, a cycle of up to 32 in
one), the rows of the triangular solve (16 at a time) and the groups of the Gram-Schmidt products (8)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(krylov_precision=64), dict(krylov_precision=32, krylov_basis_precision=32)])
def test_restart_lengths_reach_the_same_state(kw):
    from adh_kraken_b200.capi import SW2Model, default_opts
    from adh_kraken_b200.mesh import flume_case
    case = flume_case(nsteps=1, npx=41, npy=9)
    rng = np.random.default_rng(1)
    n = 3 * case.nnodes
    sol = case.sol0 + 1e-3 * rng.standard_normal(n)
    g = SW2Model(case)
    g.set_step(10.0, 2.0, 0.25, 0.0)
    out = {}
    for m in (8, 200, 9, 16, 17, 25, 32, 33, 49, 50, 51, 100):
        s, st = g.fe_newton(sol, sol, np.zeros(n, np.int32), opts=default_opts(krylov_restart=m, **kw))
        assert st["success"], (m, st)
        out[m] = s
    for m, s in out.items():                     # every length meets the same absolute residual test
        assert np.abs(s - out[200]).max() <= 1e-8 * np.abs(out[200]).max(), m
    # the preconditioner may change on one model: its cycle is built again
    s, st = g.fe_newton(sol, sol, np.zeros(n, np.int32), opts=default_opts(krylov_restart=100, precond=1, **kw))
    assert st["success"] and np.abs(s - out[200]).max() <= 1e-8 * np.abs(out[200]).max()
