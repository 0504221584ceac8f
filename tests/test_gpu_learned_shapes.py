"""Training kernels of the sweep predictor at batch sizes around their tiles (16, 64 and 128
rows) and with pointers that are only as aligned as the entry points ask for: outputs, loss and
gradient against plain 64-bit autograd.  Tolerance: BF16 keeps 8 bits, a rounding is at most
2^-9 relative; a gradient passes through at most 11 of them (4 weight layers, 3 activations,
3 + 1 back-propagated tensors), 2.2 % in the worst case; outputs through 7, 1.4 %."""
import ctypes

import numpy as np
import pytest

import semiconductor_devices_simulator_b200 as S
from semiconductor_devices_simulator_b200 import learned as LR

pytestmark = pytest.mark.gpu


def run(lib, torch, B, X, T, P0, shift):
    """Y, G, loss through the b200m_* entry points; `shift` moves every buffer off its 16-byte
    boundary by its own smallest alignment."""
    dev, keep = "cuda", []

    def buf(n, dtype, elems):
        b = torch.zeros(n + 16, dtype=dtype, device=dev)
        keep.append(b)
        return b[elems:elems + n] if shift else b[:n]
    n, nw, nb = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
    lib.b200m_mlp_sizes(ctypes.byref(n), ctypes.byref(nw), ctypes.byref(nb))
    f32, b16 = torch.float32, torch.bfloat16
    P, G, Wb, bias = buf(n.value, f32, 1), buf(n.value, f32, 1), buf(nw.value, b16, 2), buf(nb.value, f32, 1)
    x, t = buf(B * LR.MI, b16, 2), buf(B * 3, f32, 1)
    Y, Z, H = buf(B * LR.MO, f32, 2), buf(3 * B * LR.MH, f32, 2), buf(3 * B * LR.MH, b16, 2)
    dZ, dY, loss = buf(3 * B * LR.MH, b16, 2), buf(B * LR.MO, b16, 2), buf(1, f32, 1)
    P.copy_(torch.tensor(P0)); x.copy_(X.reshape(-1)); t.copy_(T.reshape(-1))
    p, st = LR._ptr, LR._stream(torch)
    assert lib.b200m_mlp_pack(p(P), p(Wb), p(bias), st)
    assert lib.b200m_mlp_forward(p(x), B, p(Wb), p(bias), p(Y), p(Z), p(H), st)
    assert lib.b200m_mlp_backward(p(x), B, p(Wb), p(Y), p(t), p(Z), p(H), p(dZ), p(dY), p(G), p(loss), st)
    torch.cuda.synchronize()
    return Y.view(B, LR.MO)[:, :3].double().cpu(), G.double().cpu(), float(loss)


@pytest.mark.parametrize("shift", [False, True], ids=["aligned", "shifted"])
@pytest.mark.parametrize("B", [1, 15, 16, 17, 63, 64, 65, 127, 129, 3100])
def test_training_shapes(B, shift):
    import torch
    lib = S.load()
    g = torch.Generator().manual_seed(B)
    X = torch.randn(B, LR.MI, generator=g).to(torch.bfloat16)
    T = 0.3 * torch.randn(B, 3, generator=g)
    n = ctypes.c_int()
    lib.b200m_mlp_sizes(ctypes.byref(n), ctypes.byref(ctypes.c_int()), ctypes.byref(ctypes.c_int()))
    P0 = LR.init_params(n.value, seed=B)
    Y, G, loss = run(lib, torch, B, X, T, P0, shift)
    P = torch.tensor(P0, dtype=torch.float64, requires_grad=True)
    h, off = X.double(), 0
    for q, (o, i) in enumerate(((LR.MH, LR.MI), (LR.MH, LR.MH), (LR.MH, LR.MH), (LR.MO, LR.MH))):
        h = h @ P[off:off + o * i].view(o, i).T + P[off + o * i:off + o * i + o]
        off += o * i + o
        if q < 3:
            h = torch.nn.functional.silu(h)
    want = ((h[:, :3] - T.double()) ** 2).mean()
    want.backward()
    want = float(want.detach())
    rel = lambda a, b: float(np.linalg.norm(a - b) / np.linalg.norm(b))
    assert rel(Y.numpy(), h[:, :3].detach().numpy()) <= 0.014
    assert rel(G.numpy(), P.grad.numpy()) <= 0.022
    assert abs(loss - want) <= 0.028 * want + 1e-12
