"""Restart lengths around the pieces of a GMRES cycle's kernels on a mesh above the small meshes' solver: the Gram-Schmidt
products' groups (8 basis vectors), the captured segments (25 steps) and entries past the last 16 bytes (6210 unknowns)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(krylov_precision=64), dict(krylov_precision=32, krylov_basis_precision=32)])
def test_restart_lengths_reach_the_same_state(kw):
    from adh_kraken_b200.capi import SW2Model, default_opts
    from adh_kraken_b200.mesh import flume_case
    case = flume_case(nsteps=1, npx=46, npy=45)
    n = 3 * case.nnodes
    sol = case.sol0 + 1e-3 * np.random.default_rng(1).standard_normal(n)
    g = SW2Model(case)
    g.set_step(10.0, 2.0, 0.25, 0.0)
    out = {}
    for m in (15, 200, 16, 17, 24, 25, 32, 33, 51):
        s, st = g.fe_newton(sol, sol, np.zeros(n, np.int32), opts=default_opts(krylov_restart=m, **kw))
        assert st["success"], (m, st)
        out[m] = s
    for m, s in out.items():                     # every length meets the same absolute residual test
        assert np.abs(s - out[200]).max() <= 1e-8 * np.abs(out[200]).max(), m
