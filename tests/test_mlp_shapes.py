"""The MLP kernels at ragged sizes: edges of the 128 x 64 x 64 tiles, rows that
do not start on 16 bytes (odd widths, shifted pointers), products whose K loop
is split over a cluster (dW of few tiles and many rows).

Tolerance per element: FP32 accumulation of t products in any order is within
(t + 2) 2^-23 sum |a b| of the exact sum; dZ and H additionally one BF16
rounding (2^-8) of a value computed in FP32 (1e-5 for the fast exponential)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('B,K,N,shift', [(1, 1, 1, 0), (127, 64, 64, 0), (129, 72, 136, 0), (63, 23, 69, 0),
                                         (130, 65, 63, 1), (150, 92, 512, 0), (2048, 64, 40, 1),
                                         (4096, 92, 70, 0)])
def test_layer_forward_backward(B, K, N, shift):
    torch = pytest.importorskip('torch')
    from vulcan_gb300 import _build, capi
    _build.build()
    L = capi.lib()
    g = torch.Generator().manual_seed(B + K + N)
    r = lambda *s: torch.randn(*s, generator=g)

    def dev(t):                 # a copy that starts `shift` elements into its storage
        flat = torch.zeros(t.numel() + shift, dtype=t.dtype, device='cuda')
        flat[shift:] = t.reshape(-1).cuda()
        return flat[shift:]

    X, W = r(B, K).to(torch.bfloat16), (r(K, N) / K ** 0.5).to(torch.bfloat16)
    b, dH = r(N), r(B, N)
    Xd, Wd, bd, dHd = dev(X), dev(W), dev(b), dev(dH)
    new = lambda n, t=torch.float32: dev(torch.full((n,), float('nan'), dtype=t))
    Z, H, dZ = new(B * N), new(B * N, torch.bfloat16), new(B * N, torch.bfloat16)
    dW, db, dX = new(K * N), new(N), new(B * K)
    v = lambda t: C.c_void_p(t.data_ptr())
    f = lambda t: C.cast(v(t), C.POINTER(C.c_float))
    capi.check(L.vk_mlp_forward(B, K, N, v(Xd), v(Wd), f(bd), f(Z), v(H), 1, None))
    capi.check(L.vk_mlp_backward(B, K, N, v(Xd), v(Wd), f(Z), f(dHd), 1, v(dZ), f(dW), f(db), f(dX), None))
    d = lambda t, *s: t.double().cpu().reshape(*s).numpy()
    x, w, bb, dh = (t.double().numpy() for t in (X, W, b, dH))
    z = d(Z, B, N)
    u = 2.0 ** -23

    def within(got, want, mag, terms):
        assert np.all(np.abs(got - want) <= (terms + 2) * u * mag + 1e-30)

    within(z, x @ w + bb, np.abs(x) @ np.abs(w) + np.abs(bb), K + 1)
    s = 1.0 / (1.0 + np.exp(-z))
    h = z * s
    assert np.all(np.abs(d(H, B, N) - h) <= (2.0 ** -8 + 1e-5) * np.abs(h) + 1e-30)
    want = dh * s * (1.0 + z * (1.0 - s))
    got = d(dZ, B, N)
    assert np.all(np.abs(got - want) <= 2.0 ** -8 * np.abs(want) + 1e-5 * np.abs(dh) * (1.0 + np.abs(z)))
    within(d(dW, K, N), x.T @ got, np.abs(x).T @ np.abs(got), B)
    within(d(db, N), got.sum(0), np.abs(got).sum(0), B)
    within(d(dX, B, K), got @ w.T, np.abs(got) @ np.abs(w).T, N)
