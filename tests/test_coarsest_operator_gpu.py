"""The coarsest level's operator is built for the solves that read it: an FP32 solve after FP64 solves on other matrices gives
the bits of one on a fresh model, with level 0 in the cluster (2047 nodes) and above it (2400)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = (dict(krylov_precision=64), dict(krylov_precision=32, krylov_basis_precision=32),
         dict(krylov_precision=32, krylov_basis_precision=64), dict(krylov_precision=32, krylov_method=0))


@pytest.mark.parametrize("nx,ny", [(23, 89), (60, 40)])
def test_precisions_in_turn(nx, ny):
    from adh_kraken_b200.capi import SW2Model, default_opts
    from adh_kraken_b200.mesh import flume_case
    case = flume_case(nsteps=1, npx=nx, npy=ny)
    n = 3 * case.nnodes
    rng = np.random.default_rng(nx)
    sol = [case.sol0 + 1e-3 * rng.standard_normal(n) for _ in KINDS]

    def step(g, k):
        g.set_step(10.0 + 2.0 * k, 2.0, 0.25, 0.0)
        s, st = g.fe_newton(sol[k], sol[k], np.zeros(n, np.int32), opts=default_opts(krylov_restart=50, precond=2, **KINDS[k]))
        assert st["success"], (k, st)
        return s, st["krylov_its"]

    fresh = [step(SW2Model(case), k) for k in range(len(KINDS))]
    g = SW2Model(case)
    for k in (0, 1, 0, 2, 0, 3, 1, 0):
        s, its = step(g, k)
        assert its == fresh[k][1] and np.array_equal(s, fresh[k][0]), k
