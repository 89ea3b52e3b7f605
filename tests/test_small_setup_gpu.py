"""The small meshes' solver is set up by the first preconditioner that it takes, whichever call that is: a timing of the
V-cycle before any solve, an ILU solve, or an AMG step.  The results are the same bits in every order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_order_of_first_use_does_not_matter():
    from adh_kraken_b200.capi import SW2Model, default_opts
    from adh_kraken_b200.mesh import flume_case
    case = flume_case(nsteps=1, npx=31, npy=9)
    n = 3 * case.nnodes
    sol = case.sol0 + 1e-3 * np.random.default_rng(0).standard_normal(n)

    def step(g, precond):
        s, st = g.fe_newton(sol, sol, np.zeros(n, np.int32), opts=default_opts(krylov_method=1, precond=precond))
        assert st["success"], st
        return s, st["krylov_its"]

    seen = []
    for first in (None, "time", "ilu", "amg"):
        g = SW2Model(case)
        g.set_step(10.0, 2.0, 0.25, 0.0)
        if first == "time":
            g.load_state(sol, sol, sol)
            g.jacobian(sol, sol, sol)
            g.time_kernel(6, 1)
        elif first:
            step(g, 1 if first == "ilu" else 2)
        seen.append([step(g, 1), step(g, 2)])
    for ilu, amg in seen[1:]:
        assert np.array_equal(ilu[0], seen[0][0][0]) and ilu[1] == seen[0][0][1]
        assert np.array_equal(amg[0], seen[0][1][0]) and amg[1] == seen[0][1][1]
