"""Layers up to 256 units take the fused kernels, wider ones the tiled products; both add each output
in one chain of the same order, so a network with a 257th hidden unit of zero weights (tiled)
gives the bits of the one without it (fused)."""
import numpy as np
import pytest
import torch

from gammcor_gb300 import api

pytestmark = pytest.mark.gpu


def split(p, dims):
    out, off = [], 0
    for i, o in zip(dims[:-1], dims[1:]):
        out.append((p[off:off + i * o].reshape(o, i), p[off + i * o:off + i * o + o]))
        off += i * o + o
    return out


@pytest.mark.parametrize("din,dout,B", [(29, 6, 9), (16, 8, 307), (5, 1, 1)])
def test_fused_and_tiled_networks_give_the_same_bits(gpu_lib, din, dout, B):
    rng = np.random.default_rng(B)
    a, b = api.Mlp(din, 256, dout, seed=3), api.Mlp(din, 257, dout, seed=3)
    da, db = [din, 256, 256, 256, dout], [din, 257, 257, 257, dout]
    wide = []
    for (W, v), i, o in zip(split(a.params().cpu().numpy(), da), db[:-1], db[1:]):
        w = np.zeros((o, i), np.float32)
        w[:W.shape[0], :W.shape[1]] = W
        wide += [w.ravel(), np.r_[v, np.zeros(o - len(v), np.float32)]]
    b.set_params(np.concatenate(wide))
    x = rng.standard_normal((B, din)).astype(np.float32)
    t = rng.standard_normal((B, dout)).astype(np.float32)
    assert torch.equal(a.forward(x), b.forward(x))
    (la, ga), (lb, gb) = a.gradients(x, t), b.gradients(x, t)
    assert abs(la - lb) <= 1e-6 * la       # the loss is summed by blocks of rows
    for (W, v), (w, u) in zip(split(ga.cpu().numpy(), da), split(gb.cpu().numpy(), db)):
        assert np.array_equal(W, w[:W.shape[0], :W.shape[1]])
        assert np.array_equal(v, u[:len(v)])
