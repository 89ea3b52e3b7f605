"""Tiles of 16 and of 128 nodes give a node the same bits: every sum runs in the order of its index.  Node counts on both sides of
the lines between them (64 x 148 for more than 64 inputs, else 128 x 148) against the first nodes by themselves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("i", [64, 68, 256])
@pytest.mark.parametrize("n", [64 * 148 - 1, 64 * 148, 128 * 148 - 1, 128 * 148])
def test_rows_do_not_depend_on_the_tile(n, i):
    import torch
    from adh_kraken_b200.learned import _L, _p
    L, o, few, npb = _L(), 64, 1000, 256
    g = torch.Generator(device="cuda").manual_seed(n + i)
    W = torch.randn(o, i, device="cuda", generator=g).bfloat16()
    X, b, R, dY = (torch.randn(*s, device="cuda", generator=g) for s in ((n, i), (o,), (n, o), (n, o)))

    def layer(m):
        Z, Y, dZ, dX = (torch.empty(m, k, device="cuda") for k in (o, o, o, i))
        parts = (m + npb - 1) // npb
        part, gw = torch.empty(parts * (o * i + o), device="cuda"), torch.empty(o * i + o, device="cuda")
        assert L.sw2n_dense_fwd(m, i, o, _p(W), _p(b), _p(X), _p(R), 1, _p(Z), _p(Y), None) == 0
        assert L.sw2n_dense_bwd(m, i, o, _p(W), _p(X), _p(Z), _p(dY), 1, _p(dZ), _p(dX), npb, _p(part), _p(gw), None) == 0
        torch.cuda.synchronize()
        return [t[:few].cpu().numpy() for t in (Z, Y, dZ, dX)]

    for a, c in zip(layer(n), layer(few)):
        assert np.array_equal(a, c)
