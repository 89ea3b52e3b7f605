"""The dense layers' kernels at the edges of their tiles and of their dispatch: node counts around 16, 128 and
128 x SMs, ragged input and output widths, and pointers that are not 16-byte aligned."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -24      # FP32 unit roundoff


def _buf(a, off):
    """A device copy of `a` whose first entry is `off` floats past a 16-byte boundary."""
    import torch
    t = torch.zeros(a.size + 8, device="cuda")
    v = t[off:off + a.size]
    v.copy_(torch.from_numpy(np.ascontiguousarray(a, np.float32).ravel()))
    return v


def _sizes():
    wide = 128 * 148
    for n, i, o, off in [(1, 4, 1, 0), (15, 8, 64, 0), (16, 12, 5, 1), (17, 64, 3, 0), (33, 60, 62, 0), (127, 256, 64, 2),
                         (129, 256, 64, 0), (700, 36, 4, 3), (wide - 1, 64, 64, 0), (wide, 256, 64, 0), (wide + 17, 44, 10, 1)]:
        yield n, i, o, off


@pytest.mark.parametrize("n,i,o,off", list(_sizes()))
def test_dense_forward_and_backward_within_their_rounding(n, i, o, off):
    import torch
    from adh_kraken_b200.learned import _L, _p
    rng = np.random.default_rng(n + 1000 * i + o)
    W = torch.from_numpy(rng.normal(0, 0.3, (o, i)).astype(np.float32)).bfloat16().cuda()
    X, R, dY = (rng.normal(0, 1, (n, k)).astype(np.float32) for k in (i, o, o))
    b = rng.normal(0, 1, o).astype(np.float32)
    dX_, dR, ddY, db = _buf(X, off), _buf(R, off), _buf(dY, off), _buf(b, 0)
    Z, Y, dZ, dX = (_buf(np.full(n * k, np.nan, np.float32), off) for k in (o, o, o, i))
    L = _L()
    assert L.sw2n_dense_fwd(n, i, o, _p(W), _p(db), _p(dX_), _p(dR), 1, _p(Z), _p(Y), None) == 0
    npb = 100
    parts = (n + npb - 1) // npb
    part, g = torch.empty(parts * (o * i + o), device="cuda"), torch.empty(o * i + o, device="cuda")
    assert L.sw2n_dense_bwd(n, i, o, _p(W), _p(dX_), _p(Z), _p(ddY), 1, _p(dZ), _p(dX), npb, _p(part), _p(g), None) == 0
    torch.cuda.synchronize()
    w, x, z, y, d = (t.double().cpu().numpy() for t in (W, dX_.view(n, i), Z.view(n, o), Y.view(n, o), dZ.view(n, o)))
    # a sum of m products in FP32: within m u sum|terms| (+ the bias and the residual added after it)
    mag = np.abs(x) @ np.abs(w).T + np.abs(b)
    assert (np.abs(z - (x @ w.T + b)) <= 1.1 * (i + 2) * U * mag).all()
    # SiLU of the stored z, with the fast exponential (2 ulp + 2 |z| u, relative) and a division, then the residual
    s = 1.0 / (1.0 + np.exp(-z))
    assert (np.abs(y - (z * s + R)) <= (8 + 4 * np.abs(z)) * U * (np.abs(z * s) + np.abs(R)) + 1e-37).all()
    ref = dY * (s * (1.0 + z * (1.0 - s)))
    assert (np.abs(d - ref) <= (16 + 8 * np.abs(z)) * U * np.abs(dY) * (1 + np.abs(z))).all()
    gx = dX.view(n, i).double().cpu().numpy()
    assert (np.abs(gx - d @ w) <= 1.1 * o * U * (np.abs(d) @ np.abs(w)) + 1e-37).all()
    gw = g.double().cpu().numpy()
    m = npb + parts                                         # in a block's nodes, then over the blocks
    assert (np.abs(gw[:o * i].reshape(o, i) - d.T @ x) <= 1.1 * m * U * (np.abs(d).T @ np.abs(x))).all()
    assert (np.abs(gw[o * i:] - d.sum(0)) <= 1.1 * m * U * np.abs(d).sum(0)).all()
