"""Large results come back through a pinned ring and several threads: sizes below, at the pieces' edges of and above the
ring, into fresh, used and pinned arrays, and from two models used by two host threads at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(nx, ny):
    from adh_kraken_b200.capi import SW2Model
    from adh_kraken_b200.mesh import flume_case
    case = flume_case(nsteps=1, npx=nx, npy=ny)
    g = SW2Model(case)
    g.set_step(60.0, 2.0, 0.25, 0.0)
    rng = np.random.default_rng(nx)
    return case, g, case.sol0 + 1e-3 * rng.standard_normal(3 * case.nnodes)


# values: 7.4 MB (one plain copy), 8.9 MB (above the limit, a ragged last piece), 25 MB (the ring goes round)
@pytest.mark.parametrize("nx,ny", [(191, 80), (215, 85), (400, 130)])
def test_values_match_the_oracle_whatever_the_destination(nx, ny):
    import ctypes as C
    import torch
    from adh_kraken_b200.capi import _d, lib
    from oracle.oracle import OracleModel
    case, g, sol = _model(nx, ny)
    o = OracleModel(case)
    o.wd_flags(sol, sol)
    ref = o.jacobian(sol, sol, sol)
    assert np.array_equal(g.jacobian(sol, sol, sol), ref)             # a fresh array
    used = np.full(g.nnz, 7.0)
    pinned = torch.full((g.nnz,), 7.0, dtype=torch.float64).pin_memory().numpy()
    for out in (used, pinned):
        assert lib().sw2g_assemble_jacobian(g.h, _d(sol), _d(sol), _d(sol), _d(out)) == 0
        assert np.array_equal(out, ref)


def test_two_models_in_two_threads():
    models = [_model(300, 100), _model(310, 90)]
    ref = [g.jacobian(s, s, s) for _, g, s in models]
    bad = []

    def use(k):
        _, g, s = models[k]
        for _ in range(5):
            if not np.array_equal(g.jacobian(s, s, s), ref[k]):
                bad.append(k)

    t = [threading.Thread(target=use, args=(k,)) for k in range(2)]
    [x.start() for x in t]
    [x.join() for x in t]
    assert not bad
