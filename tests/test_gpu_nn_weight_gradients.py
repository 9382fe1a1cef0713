"""The tensor-core weight gradients (csrc/nn_kernels.cuh, k_wgrad) at the edges
of their 2 x 4 x 16 voxel bricks: boxes smaller than a brick, ragged in every
axis, several bricks and batches, and more bricks than CTAs (the accumulators
carried from brick to brick).  Against the FP64 restatement that rounds to
BF16 where the device does; the tolerances are those of
tests/test_gpu_nn.py, for the same reason (BF16 roundings that differ between
FP32 and FP64 accumulation).  Needs a GB300."""
import numpy as np
import pytest

import nn_oracle as NN
from fixtures import rel_err
from test_gpu_nn import bf16, net_input, params, pg, sim_box  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 4, 4, 4), (1, 4, 12, 20), (3, 12, 4, 36), (1, 20, 36, 16)])
def test_weight_gradients_at_brick_edges(pg, shape):  # noqa: F811
    sim = sim_box(pg)
    p = params(8)
    sim.nn_set_params(p)
    x0 = net_input(shape, 9)
    t = np.random.default_rng(10).standard_normal(shape + (3,)).astype(np.float32)
    L, g = sim.nn_loss_grad(x0, t)
    Le, ge = NN.loss_and_grad(p.astype(np.float64), bf16(x0).astype(np.float64), t.astype(np.float64), bf16=True)
    assert abs(L - Le) <= 2e-3 * Le
    for name, ci, co, w0, b0 in NN.layer_offsets()[0]:
        tol = 5e-2 if name.startswith("e2") else 2e-2
        assert rel_err(g[w0:b0], ge[w0:b0]) < tol, name
        assert rel_err(g[b0:b0 + co], ge[b0:b0 + co]) < tol, name


def test_head_weight_gradient_is_the_fp32_product(pg):  # noqa: F811
    """The head's weight gradient from its own input and output gradient: with
    every other layer's weights zero but their biases, the head reads a field
    that is constant inside the box, so each tap's sum over the voxels is known
    exactly, and only FP32 accumulation is left."""
    shape = (2, 4, 8, 20)
    sim = sim_box(pg)
    p = np.zeros(NN.n_params(), dtype=np.float32)
    offs, _ = NN.layer_offsets()
    for name, ci, co, w0, b0 in offs:
        if name == "d0b":
            p[b0:b0 + co] = np.arange(1, co + 1) / 16.0   # exact in BF16
    sim.nn_set_params(p)
    t = bf16(np.random.default_rng(11).standard_normal(shape + (3,)).astype(np.float32))
    x0 = np.zeros(shape + (16,), dtype=np.float32)
    L, g = sim.nn_loss_grad(x0, t)
    name, ci, co, w0, b0 = offs[-1]
    W = g[w0:b0].reshape(27, co, ci)
    nvox = int(np.prod(shape))
    gy = bf16((np.float32(2.0) / np.float32(3 * nvox)) * -t).astype(np.float64)   # out = 0
    d0 = (np.arange(1, 17) / 16.0)
    for tap in range(27):
        kd, kh, kw = tap // 9 - 1, (tap // 3) % 3 - 1, tap % 3 - 1
        sl = []
        for k, n in zip((kd, kh, kw), shape[1:]):
            sl.append(slice(max(0, -k), n - max(0, k)))
        s = gy[:, sl[0], sl[1], sl[2], :].sum(axis=(0, 1, 2, 3))
        scale = np.abs(gy).sum(axis=(0, 1, 2, 3))
        # FP32 sums of 1,280 exact products: each addition rounds by 2^-23 of a partial sum at most
        tol = 1280 * 2.0 ** -23 * scale[:, None] * d0
        assert np.all(np.abs(W[tap, :3] - s[:, None] * d0) <= tol), tap
        assert np.all(W[tap, 3:] == 0)
