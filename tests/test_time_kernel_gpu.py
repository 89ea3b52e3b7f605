"""The bytes that sw2g_time_kernel names for the passes over level 0 are what such a pass cannot do without: the rate they
give is compared with a copy's, so none may be counted that no kernel has to read."""
import pytest

pytestmark = pytest.mark.gpu


def test_level0_passes_count_what_they_must_move():
    import numpy as np
    from adh_kraken_b200.capi import SW2Model
    from adh_kraken_b200.mesh import flume_case
    case = flume_case(nsteps=1, npx=90, npy=40)
    g = SW2Model(case)
    g.set_step(10.0, 2.0, 0.25, 0.0)
    g.jacobian(case.sol0, case.sol0, case.sol0)
    V, n, nnz = case.nnodes, 3 * case.nnodes, g.nnz
    assert nnz % 9 == 0
    index = 4 * (nnz // 9) + 4 * V                          # a column per 3x3 block, a pointer per node
    for which, b, smoother, count in ((0, 8, False, 1), (4, 8, True, 1), (5, 4, True, 1), (6, 4, True, 4), (7, 4, False, 1)):
        _, got = g.time_kernel(which, 1)
        need = b * nnz + index + 2 * b * n + (9 * b * V + b * n if smoother else 0)
        assert np.isclose(got, count * need, rtol=1e-12), (which, got, count * need)
