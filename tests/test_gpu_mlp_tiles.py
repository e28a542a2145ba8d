"""The network's kernels at the edges of their row tiles (32, 64 and 128 rows) and of the backward
pass's row chunks, and on arrays that are not 16-byte aligned, against FP64 torch autograd.

Bars, relative to the largest entry: an output is a chain of at most 128 FP32 FMAs per layer, whose
error is at most 128 x 2^-24 = 8e-6 of its terms' magnitude: 2e-5.  A gradient sums at most
ceil(n / 152) + 192 rows in one chain and at most 304 chunks in another, with terms of both signs
(rounding errors add up as a random walk, about sqrt(length) x 2^-24 of the terms' magnitude, which
exceeds the sum's by about sqrt(n)): below 1e-4 for the sizes here."""
import numpy as np
import pytest
import torch

from fastipc_gb300 import _native as NN
from test_gpu_learned import M, _p, relmax

pytestmark = pytest.mark.gpu
SHAPES = ((128, 64), (128,), (128, 128), (128,), (128, 128), (128,), (4, 128), (4,))


def _reference(params, X, dout):
    flat = params.double().requires_grad_(True)
    parts, at = [], 0
    for shp in SHAPES:
        k = int(np.prod(shp))
        parts.append(flat[at:at + k].view(shp))
        at += k
    h = X.double()
    for k in range(3):
        h = torch.nn.functional.gelu(h @ parts[2 * k].T + parts[2 * k + 1])
    out = h @ parts[6].T + parts[7]
    (out * dout.double()).sum().backward()
    return out.detach(), flat.grad


@pytest.mark.parametrize('n', [2, 31, 32, 33, 64, 65, 383, 384, 6143, 6144, 6145, 38911, 38912, 39041])
@pytest.mark.parametrize('shift', [0, 1, 3])
def test_tiles_and_chunks(n, shift):
    if shift and n not in (33, 65, 384, 6145, 38912):
        pytest.skip('unaligned arrays: one size of every path')
    g = torch.Generator(device='cuda').manual_seed(n)
    P = torch.tensor(M.init(3), dtype=torch.float32, device='cuda')
    P[-4:] = torch.tensor([0.1, -0.2, 0.3, -0.1])

    def buf(k, fill=None):   # k floats, `shift` floats past a 16-byte boundary
        b = torch.full((k + 4,), float('nan'), device='cuda')[shift:shift + k]
        return b if fill is None else b.copy_(fill.reshape(-1))
    X = torch.randn((n, 64), generator=g, device='cuda')
    dout = torch.randn((n, 4), generator=g, device='cuda')
    Xb, Pb, db = buf(64 * n, X), buf(P.numel(), P), buf(4 * n, dout)
    Z, A, out, G, dA = buf(384 * n), buf(384 * n), buf(4 * n), buf(P.numel()), buf(256 * n)
    L = NN.lib()
    assert L.fipc_mlp_forward(n, _p(Xb), _p(Pb), _p(Z), _p(A), _p(out), NN.stream()) == 0
    assert L.fipc_mlp_backward(n, _p(Xb), _p(Pb), _p(Z), _p(A), _p(db), _p(G), _p(dA), NN.stream()) == 0
    ref, gref = _reference(P, X, dout)
    assert relmax(out.view(n, 4).cpu().numpy(), ref.cpu().numpy()) < 2e-5
    at = 0
    for shp in SHAPES:
        k = int(np.prod(shp))
        assert relmax(G[at:at + k].cpu().numpy(), gref[at:at + k].cpu().numpy()) < 1e-4, shp
        at += k
