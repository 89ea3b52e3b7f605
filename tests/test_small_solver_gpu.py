"""Krylov solves of small meshes in one thread-block cluster against the general kernels (block-Jacobi BiCGStab, which it
does not take): both preconditioners, both methods and precisions, on meshes of fewer nodes than CTAs, with nodes numbered
at random (large halos, aggregates across CTAs), with more neighbours than a thread holds slots, and at the last size."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _renumbered(case, order):
    new = np.empty(case.nnodes, np.int64)
    new[order] = np.arange(case.nnodes)
    return dataclasses.replace(case, xyz=case.xyz[order], tri=new[case.tri].astype(np.int32), seg=new[case.seg].astype(np.int32),
                               sol0=case.sol0.reshape(-1, 3)[order].ravel())


def _mesh(kind, nx, ny):
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
        case = _renumbered(case, np.random.default_rng(nx).permutation(case.nnodes))
    return case


@pytest.mark.parametrize("kind,nx,ny", [("grid", 2, 4), ("random", 3, 5), ("grid", 17, 1 + 16), ("random", 31, 33),
                                        ("jack", 40, 51), ("grid", 32, 64), ("random", 2048 // 16, 16)])
def test_matches_the_general_kernels(kind, nx, ny):
    from adh_kraken_b200.capi import SW2Model, default_opts
    case = _mesh(kind, nx, ny)
    n = 3 * case.nnodes
    sol = case.sol0 + 1e-3 * np.random.default_rng(nx * 100 + ny).standard_normal(n)
    g = SW2Model(case)
    g.set_step(10.0, 2.0, 0.25, 0.0)

    def step(**kw):
        s, st = g.fe_newton(sol, sol, np.zeros(n, np.int32), opts=default_opts(**kw))
        assert st["success"], (kw, st)
        return s

    ref = step(krylov_method=0, precond=0, krylov_precision=64)
    for precond in (1, 2):
        for kw in (dict(krylov_method=0), dict(krylov_method=0, krylov_precision=32), dict(krylov_method=1, krylov_restart=30),
                   dict(krylov_method=1, krylov_restart=100),
                   dict(krylov_method=1, krylov_restart=40, krylov_precision=32, krylov_basis_precision=32)):
            # each converges Newton to the same absolute residual, 1e-8 against a diagonal of order 1 and more
            s = step(precond=precond, **kw)
            assert np.abs(s - ref).max() <= 1e-8 * np.abs(ref).max(), (precond, kw)
