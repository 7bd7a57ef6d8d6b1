"""The pooling kernels by form (16 aligned channels per thread, 4 aligned ones, 4 at any address) and window
(2x2, 3x3, any) and the residual add with a ragged end, against the CPU checker, byte for byte."""
import numpy as np
import pytest

from conftest import pulpnn
from test_gpu_parity import same

pytestmark = pytest.mark.gpu
api = pulpnn.api


@pytest.fixture(scope="module")
def gpu():
    return pulpnn.GpuKernels(host_buffers=False)


@pytest.mark.parametrize("C", [1, 3, 4, 6, 16, 21, 48, 429])
@pytest.mark.parametrize("k,s,p", [(2, 2, 0), (3, 2, 1), (3, 2, 0), (3, 3, 1), (7, 7, 0), (5, 2, 1)])
def test_pool(C, k, s, p, gpu, restatement):
    rng = np.random.default_rng(C * 100 + k)
    B, H, W = 3, 15, 18
    x = rng.integers(0, 256, size=(B, H, W, C), dtype=np.uint8)
    out_hw = ((H + 2 * p - k) // s + 1, (W + 2 * p - k) // s + 1)
    kw = dict(out_hw=out_hw, kernel=(k, k), pads=(p, p, p, p), strides=(s, s))
    same(gpu.maxpool(x, **kw), restatement.maxpool(x, **kw))
    for bits, requant in ((32, 0), (32, 1), (64, 1)):
        q = dict(lam=77, out_shift=6, out_add=130, requant=requant)
        same(gpu.avgpool(bits, x, **q, **kw), restatement.avgpool(bits, x, **q, **kw))


# averages of whole 16-channel pieces: four channels a thread on either side of 256 threads of sixteen an SM, sixteen beyond
@pytest.mark.parametrize("batch", [1, 9, 10, 32])
@pytest.mark.parametrize("k,s", [(2, 2), (3, 2), (1, 2)])
def test_average_of_whole_pieces(batch, k, s, gpu, restatement):
    x = np.random.default_rng(9).integers(0, 256, size=(batch, 64, 66, 64), dtype=np.uint8)
    kw = dict(out_hw=((64 - k) // s + 1, (66 - k) // s + 1), kernel=(k, k), pads=(0, 0, 0, 0), strides=(s, s))
    for bits, requant in ((32, 0), (32, 1), (64, 1)):
        q = dict(lam=77, out_shift=6, out_add=130, requant=requant)
        got = gpu.avgpool(bits, x, **q, **kw)
        assert api.last_kernel() == "pool_kernel"
        same(got[-1:], restatement.avgpool(bits, x[-1:], **q, **kw))


def test_windows_that_pads_shift(gpu, restatement):
    """An average's window starts by padding_b and ends by padding_r."""
    rng = np.random.default_rng(5)
    x = rng.integers(0, 256, size=(2, 9, 10, 20), dtype=np.uint8)
    for pads in ((1, 0, 0, 1), (0, 1, 1, 0)):
        kw = dict(out_hw=(4, 4), kernel=(3, 3), pads=pads, strides=(2, 2))
        same(gpu.avgpool(32, x, **kw), restatement.avgpool(32, x, **kw))


@pytest.mark.parametrize("H,W,k,kernel", [(560, 560, (16, 16), "pool_kernel"), (100, 257 * 13, (1, 257), "pool_kernel"),
                                          (100, 258 * 13, (1, 258), "avgpool_kernel")])
def test_largest_sums(H, W, k, kernel, gpu, restatement):
    """Windows of up to 257 pixels are summed in 16 bits: 257 * 255 is 65535. More than 1184 of them at a channel count of
    no whole words, so that they do not go to the kernel with a block per window."""
    x = np.full((1, H, W, 21), 255, np.uint8)
    x[:, : k[0], : k[1]] = np.random.default_rng(8).integers(0, 256, size=(1, k[0], k[1], 21), dtype=np.uint8)
    kw = dict(out_hw=(H // k[0], W // k[1]), kernel=k, pads=(0, 0, 0, 0), strides=k)
    for bits, requant in ((32, 0), (32, 1), (64, 1)):
        q = dict(lam=77, out_shift=6, out_add=-50, requant=requant)
        got = gpu.avgpool(bits, x, **q, **kw)
        assert api.last_kernel() == kernel
        same(got, restatement.avgpool(bits, x, **q, **kw))


@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (1, 1, 1, 15), (2, 3, 5, 7), (3, 9, 9, 48), (5, 31, 33, 37)])
def test_add(shape, shift, gpu, restatement):
    import torch
    rng = np.random.default_rng(7)
    a, b = (rng.integers(0, 256, size=shape, dtype=np.uint8) for _ in range(2))
    want = restatement.add(a, b, m1=37, m2=91, out_shift=6)
    put = lambda x: torch.cat([torch.zeros(shift, dtype=torch.uint8), torch.from_numpy(x.reshape(-1))]).cuda()  # noqa: E731
    out = torch.full((want.size + shift + 16,), 0xA5, dtype=torch.uint8, device="cuda")
    ta, tb = put(a), put(b)
    api.set_batch(shape[0])
    api.pulp_nn_add(32, ta[shift:], tb[shift:], out[shift:], 37, 91, 6, *shape[1:])
    api.synchronize()
    got = out.cpu().numpy()
    same(got[shift:shift + want.size].reshape(shape), want)
    assert (got[:shift] == 0xA5).all() and (got[shift + want.size:] == 0xA5).all()
