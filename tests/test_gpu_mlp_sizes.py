"""Loss, gradient and forward pass of the network's kernels at batch sizes around their tile and
slice edges and at layer sizes outside the fused output / input kernels, against the FP64 oracle.

Tolerance: every product is an FP32 sum of at most max(width, batch) terms; with sums of length n
cut into blocks the error is below sqrt(n) rounding units of 6e-8 relative to the sum of
magnitudes, 2e-5 of the largest gradient element for the sizes here."""
import numpy as np
import pytest

from coqui_b200 import capi
from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu

SIZES = [(4, 256, 2, 1), (4, 256, 2, 15), (4, 256, 2, 257), (4, 256, 2, 5001), (4, 256, 2, 20000),
         (3, 100, 1, 700), (8, 33, 4, 513), (9, 256, 2, 300), (4, 300, 2, 300), (5, 64, 5, 1030)]


@pytest.mark.parametrize("din,width,dout,batch", SIZES)
def test_loss_gradient_and_forward(din, width, dout, batch):
    net = capi.Mlp(din, width, dout, seed=11)
    rng = np.random.default_rng(batch)
    p = (net.params() + 0.05 * rng.standard_normal(net.nparam)).astype(np.float32)
    net.set_params(p)  # nonzero biases
    X = rng.standard_normal((batch, din)).astype(np.float32)
    T = rng.standard_normal((batch, dout)).astype(np.float32)
    loss_ref, g_ref = M.loss_and_grad(p, X, T, din, width, dout)
    Y_ref, _ = M.forward(p, X, din, width, dout)
    for _ in range(2):  # the second call runs on kept workspaces
        loss, g = net.gradient(X, T)
        assert abs(loss - loss_ref) < 1e-5 * loss_ref
        assert np.abs(g - g_ref).max() < 2e-5 * np.abs(g_ref).max()
        assert np.abs(net.forward(X) - Y_ref).max() < 1e-5 * max(1.0, np.abs(Y_ref).max())
    net.close()


@pytest.mark.parametrize("din,width,dout", [(4096, 64, 2), (4, 64, 6000)])
def test_workspace_follows_the_slices_in_use(din, width, dout):
    """The widest weight gradient is cut into few slices when the batch is small: the workspace is
    a few copies of it and not one per block the GPU could run."""
    import torch
    batch = 1000
    rng = np.random.default_rng(din)
    X = rng.standard_normal((batch, din)).astype(np.float32)
    T = rng.standard_normal((batch, dout)).astype(np.float32)
    warm = capi.Mlp(din, width, dout, seed=1)
    warm.gradient(X[:10], T[:10])  # the kernels are on the device
    warm.close()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    net = capi.Mlp(din, width, dout, seed=11)
    loss, g = net.gradient(X, T)
    used = free0 - torch.cuda.mem_get_info()[0]
    loss_ref, g_ref = M.loss_and_grad(net.params(), X, T, din, width, dout)
    assert abs(loss - loss_ref) < 1e-5 * loss_ref
    assert np.abs(g - g_ref).max() < 2e-5 * np.abs(g_ref).max()
    # parameters and optimiser state (about 8 copies), inputs and activations, 4 slices per gradient
    # of 256-long K, and the 2 MB blocks of the allocator
    need = 4 * (16 * net.nparam + 2 * batch * (din + 4 * width + 3 * dout)) + (64 << 20)
    assert used < need, (used, need)
    net.close()


def test_a_batch_that_did_not_fit_leaves_the_network_usable():
    """A batch whose buffers do not fit is an error code; the next, smaller one allocates again and
    does not run on the buffers that the failed call gave up."""
    import torch
    batch, big = 300, 60000
    rng = np.random.default_rng(5)
    X = rng.standard_normal((big, 4)).astype(np.float32)
    T = rng.standard_normal((big, 2)).astype(np.float32)
    net = capi.Mlp(4, 256, 2, seed=11)
    loss_ref, g_ref = net.gradient(X[:batch], T[:batch])
    net.forward(X[:2 * batch])
    torch.cuda.empty_cache()
    ballast = torch.empty(torch.cuda.mem_get_info()[0] - (100 << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(capi.CoquiB200Error) as e:
            net.gradient(X, T)
        assert e.value.code == -4
        loss, g = net.gradient(X[:batch], T[:batch])
    finally:
        del ballast
        torch.cuda.empty_cache()
    assert loss == loss_ref and np.array_equal(g, g_ref)
    net.close()
