"""A training step at batch sizes about the tiles' edges and at odd ones (rows that are only 8-byte aligned):
every product against fp64 on the same bf16-rounded device operands, sums and Adam's images."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from no_three_in_line_b200 import _lib, learned
from test_mlp_gpu import bf16, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [64, 65, 128, 131, 514, 1023])
def test_training_step_at_batch(batch, cuda):
    ch = make(chains=64, L=16)
    lp = learned.LearnedProposal(ch, seed=5, ring_capacity=1 << 13, batch=batch, lr=1e-3)
    for _ in range(10):
        lp.step()
    p0 = lp.params.double().cpu().numpy()
    lp.train()
    H, sc, off = 256, lp.scratch.double().cpu().numpy(), 0

    def take(*shape):
        nonlocal off
        size = int(np.prod(shape))
        off += size
        return sc[off - size:off].reshape(shape)

    X, _, d = take(batch, 192), take(batch), take(batch)
    Z1, H1, Z2, H2, dZ2, dZ1 = (take(batch, H) for _ in range(6))
    g = lp.grads.double().cpu().numpy()

    def close(got, want, rtol):
        scale = max(np.abs(want).max(), 1e-30)
        assert np.allclose(got, want, rtol=rtol, atol=rtol * scale), np.abs(got - want).max() / scale

    W1, W2 = p0[:learned.O_B1].reshape(H, 192), p0[learned.O_W2:learned.O_B2].reshape(H, H)
    close(Z1, bf16(X) @ bf16(W1).T + p0[learned.O_B1:learned.O_W2], 2e-4)
    close(Z2, bf16(H1) @ bf16(W2).T + p0[learned.O_B2:learned.O_W3], 2e-4)
    close(dZ1, (bf16(dZ2) @ bf16(W2)) * (Z1 > 0), 2e-4)
    close(g[:learned.O_B1].reshape(H, 192), bf16(dZ1).T @ bf16(X), 2e-4)
    close(g[learned.O_W2:learned.O_B2].reshape(H, H), bf16(dZ2).T @ bf16(H1), 2e-4)
    close(g[learned.O_B1:learned.O_W2], dZ1.sum(0), 1e-5)
    close(g[learned.O_B2:learned.O_W3], dZ2.sum(0), 1e-5)
    close(g[learned.O_W3:learned.O_B3], H2.T @ d, 1e-5)
    close(g[learned.O_B3], d.sum(), 1e-5 * (1 + np.abs(d).sum() / max(abs(d.sum()), 1e-30)))
    # the images the next inference reads are those of the new weights
    images = lp.w2_img.clone(), lp.w1a_img.clone()
    _lib.check(_lib.lib().n3_mlp_pack(ctypes.byref(lp._desc), _lib.stream_ptr()), "n3_mlp_pack")
    assert all(bool((a == b).all()) for a, b in zip(images, (lp.w2_img, lp.w1a_img)))
    assert int(lp.counters[1]) == 1
