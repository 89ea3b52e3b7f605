"""The captured cycles of GMRES, on a mesh above the small meshes' solver (which captures nothing): a change of the
preconditioner, of the restart length or of the precisions on one model replays no cycle that was captured for another.  Runs are
reproducible, so each solve has the bits and the iteration count of the same solve on a fresh model."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case():
    from adh_kraken_b200.mesh import flume_case
    case = flume_case(nsteps=1, npx=46, npy=45)                       # 2070 nodes
    return case, case.sol0 + 1e-3 * np.random.default_rng(1).standard_normal(3 * case.nnodes)


def _step(g, sol, **kw):
    from adh_kraken_b200.capi import default_opts
    g.set_step(10.0, 2.0, 0.25, 0.0)
    s, st = g.fe_newton(sol, sol, np.zeros(sol.size, np.int32), opts=default_opts(krylov_method=1, **kw))
    assert st["success"], (kw, st)
    return s, st["krylov_its"]


PRECISION = {"fp64": dict(krylov_precision=64), "fp32": dict(krylov_precision=32, krylov_basis_precision=32),
             "mixed": dict(krylov_precision=32, krylov_basis_precision=64)}


@pytest.mark.parametrize("kind", list(PRECISION))
def test_preconditioner_changes_on_one_model(kind):
    from adh_kraken_b200.capi import SW2Model
    case, sol = _case()
    kw = dict(krylov_restart=40, **PRECISION[kind])
    amg, ilu = (_step(SW2Model(case), sol, precond=p, **kw) for p in (2, 1))
    assert amg[1] != ilu[1]                                            # a replayed cycle of the other one would show
    g = SW2Model(case)
    for p, want in ((2, amg), (1, ilu), (2, amg), (1, ilu)):
        s, its = _step(g, sol, precond=p, **kw)
        assert its == want[1] and np.array_equal(s, want[0]), (p, its, want[1])


def test_restarts_and_precisions_change_on_one_model():
    from adh_kraken_b200.capi import SW2Model
    case, sol = _case()
    # around the segments' 25 steps, the triangular solve's 16 rows and the products' 8 vectors, in an order in which the basis grows,
    # and a shorter cycle follows a longer one
    order = [("fp64", 49), ("fp32", 49), ("mixed", 50), ("fp64", 50), ("fp32", 33), ("fp32", 100), ("fp64", 100), ("mixed", 17), ("fp64", 17),
             ("fp32", 32), ("fp64", 49), ("mixed", 50)]
    fresh = {}
    g = SW2Model(case)
    for kind, m in order:
        kw = dict(precond=2, krylov_restart=m, **PRECISION[kind])
        if (kind, m) not in fresh:
            fresh[kind, m] = _step(SW2Model(case), sol, **kw)
        s, its = _step(g, sol, **kw)
        assert its == fresh[kind, m][1] and np.array_equal(s, fresh[kind, m][0]), (kind, m)
