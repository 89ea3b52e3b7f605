"""The AMG cycle's small levels in one thread-block cluster: meshes at the edges of its dispatch
(everything in the coarsest level's neighbourhood, the last size whose level 0 is in the cluster and
the first above it, a level of several thousand nodes left outside it), FP64 and FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(nx, ny):
    """A scaled Newton system of a perturbed flume at a short step, from the oracle."""
    from adh_kraken_b200.mesh import flume_case
    from oracle.oracle import OracleModel
    case = flume_case(nsteps=1, npx=nx, npy=ny)
    case.dt = 10.0
    rng = np.random.default_rng(nx * 1000 + ny)
    n = 3 * case.nnodes
    sol = case.sol0 + 1e-3 * rng.standard_normal(n)
    o = OracleModel(case)
    o.wd_flags(sol, case.sol0)
    return case, o, sol


# 3x3: one aggregate or two; 16x16: level 0 has the most nodes a coarsest level may have; 64x32 = 2048 nodes: the last
# size in the cluster from level 0; 23x89 = 2047 and 41x50 = 2050: odd sizes on both sides; 150x60: level 1 first
@pytest.mark.parametrize("nx,ny", [(3, 3), (16, 16), (23, 89), (64, 32), (41, 50), (150, 60)])
def test_preconditioned_solve_reaches_its_residual(nx, ny):
    from adh_kraken_b200.capi import SW2Model
    case, o, sol = _system(nx, ny)
    g = SW2Model(case)
    n = 3 * case.nnodes
    vals, res = o.jacobian(sol, case.sol0, case.sol0), o.residual(sol, case.sol0, case.sol0)
    v, r, x0, _, sc = g.prepare_system(vals, res, np.zeros(n), np.zeros(n, np.int32))
    x, _, it = g.bicgstab(v, r, x0, sc, max_it=2000, tol=1e-10, precond=2)
    assert 0 < it < 2000
    y = x / sc                                              # the scaled system's unknowns
    ax = np.add.reduceat(v * y[o.cols], o.indptr[:-1])
    # the recurrence's residual passed max|r| <= tol + tol max|b|; a factor 2 is left for its drift from the true one
    assert np.abs(r - ax).max() <= 2 * (1e-10 + 1e-10 * np.abs(r).max())


def _union_jack(nx, ny):
    """The flume's grid with every second node joined to all its 8 neighbours and the others to 4, the former numbered
    first: the first tiles of 64 nodes have 576 neighbour slots, more than a tile holds in shared memory."""
    import dataclasses
    from adh_kraken_b200.mesh import flume_case
    case = flume_case(nsteps=1, npx=nx, npy=ny)
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    old = np.arange(nx * ny).reshape(nx, ny)
    tri = []
    for a in range(nx - 1):
        for b in range(ny - 1):
            p, q, r, s = old[a, b], old[a + 1, b], old[a + 1, b + 1], old[a, b + 1]
            tri += [(p, q, r), (p, r, s)] if (a + b) % 2 == 0 else [(p, q, s), (q, r, s)]
    order = np.argsort(((i + j) % 2).ravel(), kind="stable")
    new = np.empty(nx * ny, np.int64)
    new[order] = np.arange(nx * ny)
    sol = case.sol0.reshape(-1, 3)[order].ravel()
    return dataclasses.replace(case, xyz=case.xyz[order], tri=new[np.array(tri)].astype(np.int32),
                               seg=new[case.seg].astype(np.int32), sol0=sol)


@pytest.mark.parametrize("nx,ny", [(3, 3), (23, 89), (64, 32), (41, 50), (150, 60), (61, 67)])
def test_fp32_cycles_step_like_fp64(nx, ny):
    """Both precisions converge Newton to the same absolute residual, so their states agree far below the step's
    tolerance on the velocities (1e-8 on the residual; the flume's smallest diagonal is of order 1)."""
    from adh_kraken_b200.capi import SW2Model, default_opts
    case, o, sol = _system(nx, ny)
    if (nx, ny) == (61, 67):                                # 4087 nodes, the last tile not full
        case = _union_jack(nx, ny)
        sol = case.sol0 + 1e-3 * np.random.default_rng(5).standard_normal(3 * case.nnodes)
        case.dt = 10.0
    g = SW2Model(case)
    g.set_step(case.dt, 2.0, 0.25, 0.0)
    out = []
    for kw in (dict(krylov_precision=64), dict(krylov_precision=32), dict(krylov_precision=32, krylov_basis_precision=32)):
        s, st = g.fe_newton(sol, sol, np.zeros(3 * case.nnodes, np.int32), opts=default_opts(krylov_restart=50, **kw))
        assert st["success"], st
        out.append(s)
    for s in out[1:]:
        assert np.abs(s - out[0]).max() <= 1e-8 * np.abs(out[0]).max()
