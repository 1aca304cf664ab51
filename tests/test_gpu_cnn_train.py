"""The batched forward / backward kernels of the warm-start CNN at the batch
sizes where their shapes change, against the FP64 oracle.

Above 16 pairs the convolutions run as chains over one image a block (up to
148 pairs) or two (above; an odd batch leaves half a block empty), FC1's
weight gradient in k steps of 8 pairs, conv4's weight gradient over 4 images a
step. Tolerance: as for the other tests of these kernels, 1% of a tensor's
norm (BF16 stored activations: one step is 0.4%).
"""
import numpy as np
import pytest

from oracle import cnn_oracle as co

pytestmark = pytest.mark.gpu


def _net_and_batch(device, batch, seed):
    import torch
    from openfusion_b200 import learned
    net = learned.WarmStartNet(device, seed=seed)
    rng = np.random.default_rng(seed)
    x = co.bf16_round(rng.normal(0.0, 0.4, (batch,) + co.IN_SHAPE))
    bits = (x.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    xin = torch.from_numpy(bits.view(np.int16).reshape(batch, -1).copy()).to(device)
    return net, x, xin, rng.normal(0.0, 1.0, (batch, 6))


@pytest.mark.parametrize("batch", [1, 17, 148, 149])
def test_gradients_at_the_batch_edges(of, cuda, batch):
    import torch
    net, x, xin, target = _net_and_batch(cuda, batch, 30 + batch)
    tgt = torch.tensor(target, dtype=torch.float32, device=cuda)
    loss = float(net.gradients(xin, tgt).item())
    p = co.unpack(co.bf16_bits_to_f64(net.params.cpu().numpy().view(np.uint16)))
    pb = co.unpack(net.master.cpu().numpy().astype(np.float64))
    p.update({name: pb[name] for name, _ in co.layout() if name.startswith("b")})
    ref_loss, _, ref = co.loss_and_grads(p, x, target, net.loss_w.cpu().numpy().astype(np.float64),
                                         bf16=True)
    assert abs(loss - ref_loss) <= 1e-2 * ref_loss
    got = co.unpack(net.grad.cpu().numpy().astype(np.float64))
    for name, _ in co.layout():
        err = np.linalg.norm(got[name] - ref[name]) / np.linalg.norm(ref[name])
        assert err < 1e-2, (name, err)


def test_unaligned_buffers_and_larger_batches_change_nothing(of, cuda):
    """Inputs at an odd 16-bit offset and a workspace off its alignment give the
    same bits; the first pairs of a larger batch get the same outputs."""
    import ctypes as C
    import torch
    from openfusion_b200 import _native as N
    net, _, xin, target = _net_and_batch(cuda, 301, 5)
    tgt = torch.tensor(target, dtype=torch.float32, device=cuda)
    st = torch.cuda.current_stream().cuda_stream
    out = net.forward(xin)
    assert torch.equal(net.forward(xin[:20].contiguous()), out[:20])
    net.gradients(xin, tgt)
    grad = net.grad.clone()
    shifted = torch.zeros(xin.numel() + 1, dtype=torch.int16, device=cuda)
    shifted[1:] = xin.reshape(-1)
    n = C.c_size_t()
    N.check("of_cnn_workspace_bytes", N.lib().of_cnn_workspace_bytes(301, C.byref(n)))
    ws = torch.empty(n.value + 4, dtype=torch.uint8, device=cuda)
    N.check("of_cnn_backward", N.lib().of_cnn_backward(
        net.params.data_ptr(), net.master.data_ptr(), shifted.data_ptr() + 2, 301, tgt.data_ptr(),
        net.loss_w.data_ptr(), ws.data_ptr() + 4, net.grad.data_ptr(), None, st))
    torch.cuda.synchronize()
    assert torch.equal(net.grad, grad)
