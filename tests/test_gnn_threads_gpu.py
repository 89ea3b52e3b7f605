"""Dense layers of different widths from several host threads at once: a launch's shared memory is allowed per kernel, so
one thread's width must not have another's launch refused."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_widths_do_not_disturb_each_other():
    import ctypes as C
    import torch
    from adh_kraken_b200.learned import _L, _p
    L, refused = _L(), []
    calls, n, npb = 20000, 64, 64

    def use(i, o):
        W = torch.zeros(o, i, device="cuda").bfloat16()
        X, b, Z, Y, dZ = (torch.zeros(k, device="cuda") for k in (n * i, o, n * o, n * o, n * o))
        part, g = torch.empty(o * i + o, device="cuda"), torch.empty(o * i + o, device="cuda")
        dX, st = torch.empty(n * i, device="cuda"), torch.cuda.Stream()
        s = C.c_void_p(st.cuda_stream)
        st.wait_stream(torch.cuda.current_stream())
        for k in range(calls):
            rc = L.sw2n_dense_fwd(n, i, o, _p(W), _p(b), _p(X), None, 1, _p(Z), _p(Y), s)
            if k % 8 == 0:
                rc = rc or L.sw2n_dense_bwd(n, i, o, _p(W), _p(X), _p(Z), _p(Y), 1, _p(dZ), _p(dX), npb, _p(part), _p(g), s)
            if rc:
                refused.append((i, o, rc))
        st.synchronize()

    # widths whose shared memory is above what every kernel has without asking: wide, and narrow (few outputs)
    t = [threading.Thread(target=use, args=a) for a in ((256, 64), (192, 64), (256, 3), (128, 3))]
    [x.start() for x in t]
    [x.join() for x in t]
    assert not refused, (len(refused), refused[:3])
