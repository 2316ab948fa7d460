"""GPU tests of the network's fused kernels (csrc/mlp_fused.cuh) at the edges of their tiles: batches around the
128-row tile, widths around the 32-column padding and the 128-column weight chunks, and the widths just beyond the
fused path.

Inputs, weights and biases are -1, 0 or 1, so every sum of a forward pass is a whole number: below 256 after the
first layer, 256 * 256 after the second and 2^24 after the third, all exact in FP32 whatever the order, and the BF16
operands round the same numbers on both sides: outputs must equal the oracle's.  Gradients (scaled by 1 / count)
are held to the general path's 2e-3 relative L2 per block (test_gpu_mlp.py), the loss to 1e-5."""
import numpy as np
import pytest
import torch

from oracle import mlp as omlp
from cufcm_fil_b200.mlp import FilamentMLP

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-30))


def check(net, p, X, T, dims, exact=True):
    n, n_out = T.shape
    xd, td = torch.tensor(X, device="cuda"), torch.tensor(T, device="cuda")
    yd = torch.full((n + 1, n_out), 7.0, device="cuda")
    torch.cuda.synchronize()
    net.forward(xd, yd)
    loss, g = net.gradients(xd, td)
    torch.cuda.synchronize()
    assert (yd[n] == 7.0).all()  # nothing beyond the batch
    if exact:
        np.testing.assert_array_equal(yd[:n].cpu().numpy(), omlp.forward(p, X, *dims)[2])
    loss_ref, g_ref = omlp.gradients(p, X, T, *dims)
    assert abs(loss - loss_ref) <= 1e-5 * loss_ref
    n_in, hid, n_out = dims
    o = 0
    for s in (n_in * hid, hid, hid * hid, hid, hid * n_out, n_out):
        assert rel(g[o:o + s], g_ref[o:o + s]) < 2e-3, o
        o += s


@pytest.mark.parametrize("dims", [(182, 256, 62), (33, 160, 5), (256, 256, 128), (7, 31, 1), (257, 64, 10), (40, 64, 129)])
@pytest.mark.parametrize("n", [1, 127, 129, 2000])
def test_tile_edges_match_oracle(dims, n):
    rng = np.random.default_rng(n)
    X = rng.integers(-1, 2, (n, dims[0])).astype(np.float32)
    T = rng.standard_normal((n, dims[2])).astype(np.float32)
    with FilamentMLP(*dims, max_batch=2048, seed=3) as net:
        p = rng.integers(-1, 2, net.params().size).astype(np.float32)
        net.set_params(p)
        check(net, p, X, T, dims)


def test_training_step_leaves_consistent_weights():
    """After optimiser steps the kernels' copies of the weights are those of params()."""
    rng = np.random.default_rng(5)
    dims, n = (50, 96, 20), 300
    X = rng.standard_normal((n, dims[0])).astype(np.float32)
    T = rng.standard_normal((n, dims[2])).astype(np.float32)
    with FilamentMLP(*dims, max_batch=512, seed=1) as net:
        xd, td = torch.tensor(X, device="cuda"), torch.tensor(T, device="cuda")
        torch.cuda.synchronize()
        before = net.params()
        for _ in range(3):
            net.train_step(xd, td, lr=1e-2)
        p = net.params()
        assert rel(p, before) > 1e-3
        check(net, p, X, T, dims, exact=False)


@pytest.mark.parametrize("n", [5, 300])
def test_output_may_overlap_the_input(n):
    rng = np.random.default_rng(n)
    dims = (182, 256, 62)
    X = rng.standard_normal((n, dims[0])).astype(np.float32)
    with FilamentMLP(*dims, max_batch=512, seed=2) as net:
        xd, yd = torch.tensor(X, device="cuda"), torch.zeros((n, dims[2]), device="cuda")
        torch.cuda.synchronize()
        net.forward(xd, yd)
        net.forward(xd, xd.view(-1)[:n * dims[2]].view(n, dims[2]))
        torch.cuda.synchronize()
        assert torch.equal(xd.view(-1)[:n * dims[2]].view(n, dims[2]), yd)
