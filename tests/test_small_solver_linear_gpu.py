"""Single linear solves of the small meshes' cluster solver against the general kernels, which run where a Newton solve would
correct what a solver got wrong.  The general kernels get the same system on a larger mesh: the small mesh and, not joined to it
and numbered after it, a patch of still water that takes the whole above the solver's 2048 nodes.  The patch has no residual
and no part in colours, factor, aggregates or sums of the small mesh's unknowns, so the iterates on these agree up to
rounding, from the first iteration on."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Aggregation gives the small mesh of each pair the same aggregates and both meshes the same number of levels (3 for the grids, else 2).
MESHES = [("grid", 30, 65), ("grid", 32, 64), ("random", 31, 60), ("random", 32, 64), ("jack", 40, 51)]
TINY = [("grid", 2, 4), ("random", 3, 5), ("grid", 17, 17)]


def _small(kind, nx, ny):
    from adh_kraken_b200.mesh import flume_case
    case = flume_case(nsteps=1, npx=nx, npy=ny)
    if kind == "jack":                                      # every second node has 8 neighbours and itself: 9 slots
        old, tri = np.arange(nx * ny).reshape(nx, ny), []
        for a in range(nx - 1):
            for b in range(ny - 1):
                p, q, r, s = old[a, b], old[a + 1, b], old[a + 1, b + 1], old[a, b + 1]
                tri += [(p, q, r), (p, r, s)] if (a + b) % 2 == 0 else [(p, q, s), (q, r, s)]
        case = dataclasses.replace(case, tri=np.array(tri, np.int32))
    if kind != "grid":
        order = np.random.default_rng(nx).permutation(case.nnodes)
        new = np.empty(case.nnodes, np.int64)
        new[order] = np.arange(case.nnodes)
        case = dataclasses.replace(case, xyz=case.xyz[order], tri=new[case.tri].astype(np.int32), seg=new[case.seg].astype(np.int32),
                                   sol0=case.sol0.reshape(-1, 3)[order].ravel())
    return case


def _with_patch(case):
    from adh_kraken_b200.mesh import flume_case
    patch = flume_case(nsteps=1, npx=16, npy=max(4, (2112 - case.nnodes) // 16 + 1))
    xyz = patch.xyz.copy()
    xyz[:, 0] += 1e5
    xyz[:, 2] = 0.0
    still = np.tile([2.0, 0.0, 0.0], patch.nnodes)
    return dataclasses.replace(case, xyz=np.concatenate([case.xyz, xyz]),
                               tri=np.concatenate([case.tri, patch.tri + case.nnodes]).astype(np.int32),
                               sol0=np.concatenate([case.sol0, still]))


def _pair(kind, nx, ny):
    from adh_kraken_b200.capi import SW2Model
    a = _small(kind, nx, ny)
    b = _with_patch(a)
    n, rng = 3 * a.nnodes, np.random.default_rng(nx * 100 + ny)
    sol = a.sol0 + 1e-3 * rng.standard_normal(n)
    both = np.concatenate([sol, b.sol0[n:]])
    models = []
    for c in (a, b):
        g = SW2Model(c)
        g.set_step(10.0, 2.0, 0.25, 0.0)
        g.set_profiling(True)
        models.append(g)
    assert a.nnodes <= 2048 < b.nnodes
    return models, (sol, both), n


def _took(g, its, small):
    """The solver's kernels since the last look: a few for the cluster, more than one an iteration for the general path."""
    k = int(g.profile()[1][4])
    g.reset_profile()
    assert (k < its + 12) if small else (k > 4 * its), (k, its, small)


@pytest.mark.parametrize("precond,kind,nx,ny", [(p, *m) for m in MESHES for p in (1, 2)] + [(1, *m) for m in TINY])
def test_bicgstab_iterates(precond, kind, nx, ny):
    models, sols, n = _pair(kind, nx, ny)
    systems = []
    for g, s in zip(models, sols):
        vals, res = g.jacobian(s, s, s), g.residual(s, s, s)
        res[n:] = 0.0
        v, r, _, _, sc = g.prepare_system(vals, res, np.zeros(g.ndofs), np.zeros(g.ndofs, np.int32))
        systems.append((v, r, sc))
    (va, ra, _), (vb, rb, _) = systems
    assert np.array_equal(va, vb[:va.size]) and np.array_equal(ra, rb[:n])
    for g in models:
        g.reset_profile()
    # A rounding of 1e-16 grows in the quotients of a few iterations; 1e-9 leaves seven digits for that, and a wrong entry of a halo,
    # a sweep or a colour changes the iterate by far more.  Later the two recurrences part; their lengths stay close.
    for k in (1, 2, 4, 4000):
        out = []
        for (v, r, sc), g in zip(systems, models):
            x, b, it = g.bicgstab(v, r, np.zeros(g.ndofs), sc, max_it=k, tol=1e-12, precond=precond)
            _took(g, abs(it), g is models[0])
            out.append((x, it))
        (x, it), (y, jt) = out
        assert np.abs(y[n:]).max() == 0.0
        if k < 4000 and it == jt == k:
            assert np.abs(x).max() > 0 and np.abs(x - y[:n]).max() <= 1e-9 * np.abs(y).max(), k
        else:
            assert it > 0 and jt > 0 and abs(it - jt) <= max(3, 0.1 * jt), (it, jt)
            assert np.abs(x - y[:n]).max() <= 1e-6 * np.abs(y).max()


# One Newton iteration (any increment counts as converged), its linear solve to a few forcings: a handful of Krylov steps,
# a few dozen, and for the small restart several cycles.
@pytest.mark.parametrize("precond,kind,nx,ny", [(p, *m) for m in MESHES for p in (1, 2)])
@pytest.mark.parametrize("precision", [64, 32])
def test_gmres_and_fp32_iterates(precision, precond, kind, nx, ny):
    from adh_kraken_b200.capi import default_opts
    models, sols, n = _pair(kind, nx, ny)
    # FP64 as above; FP32 cycles round to 6e-8, and 1e-4 leaves three digits for its growth
    bound = 1e-9 if precision == 64 else 1e-4
    for method, tol, restart in ((1, 0.3, 30), (1, 0.03, 100), (1, 1e-3, 100), (1, 1e-2, 5)) + (((0, 0.1, 30),) if precision == 32 else ()):
        out = []
        for g, s in zip(models, sols):
            g.reset_profile()
            o = default_opts(krylov_method=method, precond=precond, krylov_precision=precision, krylov_basis_precision=precision, krylov_tol=tol,
                             krylov_restart=restart, refine_tol=0.05, tol_nonlin=1e-12, inc_nonlin=1e30, max_nonlin_it=1, max_linesearch_cuts=0)
            new, st = g.fe_newton(s, s, np.zeros(g.ndofs, np.int32), opts=o)
            assert st["success"] and st["newton_its"] == 1, st
            if method == 1:
                _took(g, st["krylov_its"] if restart > 5 else 3 * st["krylov_its"], g is models[0])
            out.append(((new - s)[:n], st["krylov_its"]))
        (x, it), (y, jt) = out
        assert it > 0 and it == jt, (method, tol, it, jt)
        assert np.abs(x - y).max() <= bound * np.abs(y).max(), (method, tol, np.abs(x - y).max() / np.abs(y).max())
