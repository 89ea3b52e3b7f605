"""The end of the two-phase reductions over few, exactly 32, a little more and the most blocks: the mass (two sums) against
its terms, and the sums and maxima of a block-Jacobi BiCGStab solve by the solution they lead to."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 256 triangles a block of the mass balance: 1, 2, 31, 32, 32, 34, 65 blocks and the cap of 1184
@pytest.mark.parametrize("n", [5, 17, 63, 64, 65, 66, 92, 400])
def test_mass_is_the_sum_of_its_terms(n):
    from adh_kraken_b200.capi import SW2Model
    from adh_kraken_b200.mesh import flume_case
    case = flume_case(nsteps=1, npx=n, npy=n)
    g = SW2Model(case)
    sol = case.sol0 + 0.1 * np.random.default_rng(n).standard_normal(3 * case.nnodes)
    total, inflow, terms = g.grid_mass(sol, elem=True)
    # a sum in another order of m terms: within m u sum|terms|
    assert abs(total - math.fsum(terms)) <= len(terms) * 2.0 ** -53 * np.abs(terms).sum()
    again, same, _ = g.grid_mass(sol, elem=True)
    assert again == total and same == inflow


# 32 nodes a block of the products, 256 unknowns a block of the updates
@pytest.mark.parametrize("nx,ny", [(3, 3), (8, 4), (31, 32), (32, 32), (33, 32), (101, 11), (80, 60)])
def test_block_jacobi_solve_reaches_its_residual(nx, ny):
    from adh_kraken_b200.capi import SW2Model
    from adh_kraken_b200.mesh import flume_case
    from oracle.oracle import OracleModel
    case = flume_case(nsteps=1, npx=nx, npy=ny)
    case.dt = 1.0
    n = 3 * case.nnodes
    sol = case.sol0 + 1e-3 * np.random.default_rng(nx).standard_normal(n)
    o, g = OracleModel(case), SW2Model(case)
    o.wd_flags(sol, case.sol0)
    vals, res = o.jacobian(sol, case.sol0, case.sol0), o.residual(sol, case.sol0, case.sol0)
    v, r, x0, _, sc = g.prepare_system(vals, res, np.zeros(n), np.zeros(n, np.int32))
    x, b, it = g.bicgstab(v, r, x0, sc, max_it=2000, tol=1e-10, precond=0)
    assert 0 < it < 2000
    y = x / sc                                              # the scaled system's unknowns
    ax = np.add.reduceat(v * y[o.cols], o.indptr[:-1])
    # the recurrence's preconditioned residual passed max|M^-1 r| <= tol + tol max|M^-1 b| and b is M^-1 b now; rows of M are at
    # most 3 max|v| in sum, and a factor 2 is left for its drift from the true one
    assert np.abs(r - ax).max() <= 2 * 3 * np.abs(v).max() * (1e-10 + 1e-10 * np.abs(b).max())
