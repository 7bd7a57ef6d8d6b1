"""The plane-staging depthwise kernel (3x3 and 5x5 of any channel count, row length and alignment)
against the CPU checker, byte for byte: channel groups that are full, partial and of one channel, rows
that end inside a word, bands that end inside the image, both layouts, every requantisation mode."""
import numpy as np
import pytest

from conftest import pulpnn
from test_gpu_parity import MODES, dw_kw, same

pytestmark = pytest.mark.gpu
api, wl = pulpnn.api, pulpnn.workloads
KERNEL = "depthwise_planes_kernel"


@pytest.fixture(scope="module")
def gpu():
    return pulpnn.GpuKernels(host_buffers=False)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("relu,bn", MODES)
@pytest.mark.parametrize("hwc", [False, True])
def test_modes(bits, relu, bn, hwc, gpu, restatement):
    c = wl.depthwise_case(80, 13, 11, 37, kernel=(5, 5), pads=(2, 2, 2, 2), batch=2, bits=bits, out_shift=8,
                          with_bias=True, out_mult=3, relu=relu, bn=bn, w_range=(-128, 127), k_range=(-64, 64),
                          lam_range=(-2 ** 20, 2 ** 20), hwc=hwc)
    got = gpu.depthwise(bits, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c))
    assert api.last_kernel() == KERNEL
    same(got, restatement.depthwise(bits, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c)))


@pytest.mark.parametrize("k", [3, 5])
@pytest.mark.parametrize("s", [1, 2])
@pytest.mark.parametrize("hwc", [False, True])
@pytest.mark.parametrize("H,W,C,batch", [(9, 7, 1, 3), (8, 9, 15, 2), (11, 13, 17, 2), (28, 28, 33, 40), (15, 14, 120, 3),
                                         (97, 101, 34, 1), (7, 7, 475, 5), (30, 112, 16, 2), (10, 12, 6, 700)])
def test_shapes(k, s, hwc, H, W, C, batch, gpu, restatement):
    p = k // 2
    c = wl.depthwise_case(81, H, W, C, kernel=(k, k), strides=(s, s), pads=(p, p, p, p), batch=batch, out_shift=9,
                          with_bias=True, hwc=hwc)
    got = gpu.depthwise(32, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c))
    assert api.last_kernel() == KERNEL
    same(got, restatement.depthwise(32, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c)))


# rows in one and in several strips of columns: the last strip whole, of one group of four columns and of a part of one;
# images of few rows and many, bands that would not fit shared memory in one piece. Each is followed by an ordinary call,
# which has to find nothing left over.
@pytest.mark.parametrize("k,s,hwc,H,W,C,batch", [
    (5, 1, True, 8, 773, 20, 1), (5, 1, True, 8, 784, 40, 1), (5, 1, False, 8, 776, 20, 1), (5, 2, True, 6, 900, 20, 1),
    (5, 2, False, 6, 901, 20, 1), (5, 1, True, 5, 1580, 8, 1), (3, 1, True, 4, 1050, 30, 1), (3, 1, False, 4, 1052, 20, 1),
    (3, 2, True, 6, 1270, 30, 1), (3, 1, True, 4, 2120, 7, 1), (3, 1, True, 1, 1038, 154, 1), (3, 1, True, 1, 32, 5, 3),
    (3, 1, True, 1, 33, 5, 3), (3, 1, False, 2, 36, 17, 1), (5, 2, True, 3, 65, 6, 2), (5, 2, False, 3, 72, 33, 2),
    (3, 2, False, 1, 130, 31, 2), (3, 1, True, 9, 300, 3, 200), (5, 1, False, 30, 700, 18, 40)])
def test_strips_of_columns(k, s, hwc, H, W, C, batch, gpu, restatement):
    p = k // 2
    for h, w, c, b in ((H, W, C, batch), (9, 7, 20, 1)):
        c = wl.depthwise_case(83, h, w, c, kernel=(k, k), strides=(s, s), pads=(p, p, p, p), batch=b, out_shift=9, hwc=hwc)
        got = gpu.depthwise(32, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c))
        assert api.last_kernel() == KERNEL
        c["x"] = c["x"][-1:]
        same(got[-1:], restatement.depthwise(32, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c)))


@pytest.mark.parametrize("hwc", [False, True])
@pytest.mark.parametrize("H,W,C,batch", [(1, 3, 1, 2), (1, 3, 1, 5), (1, 3, 2, 3), (1, 4, 1, 5), (2, 3, 1, 3), (1, 3, 7, 2), (3, 5, 5, 4)])
@pytest.mark.parametrize("pr", [0, 1])
def test_images_of_a_few_bytes(hwc, H, W, C, batch, pr, gpu, restatement):
    c = wl.depthwise_case(84, H, W, C, batch=batch, pads=(1, 1, 1, pr), out_shift=9, hwc=hwc)
    got = gpu.depthwise(32, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c))
    assert api.last_kernel() == KERNEL
    same(got, restatement.depthwise(32, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c)))


@pytest.mark.parametrize("hwc", [False, True])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_unaligned_input(hwc, shift, gpu, restatement):
    import torch
    c = wl.depthwise_case(82, 9, 13, 20, kernel=(5, 5), pads=(2, 2, 2, 2), batch=2, out_shift=9, hwc=hwc)
    want = restatement.depthwise(32, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c))
    x = torch.cat([torch.zeros(shift, dtype=torch.uint8), torch.from_numpy(c["x"].reshape(-1))]).cuda()
    out = torch.full((want.size + 8,), 0xA5, dtype=torch.uint8, device="cuda")
    put = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    api.set_batch(2)
    fn = api.pulpnn_depthwise_hwc if hwc else api.pulp_nn_depthwise_generic
    fn(32, x[shift:], None, None, out[shift:], put(c["w"]), None, put(c["k"]), put(c["lam"]), 1, 9, 13, 9, 20, 13, 9, 20,
       5, 5, 2, 2, 2, 2, 1, 1, 1, 1)
    api.synchronize()
    assert api.last_kernel() == KERNEL
    got = out.cpu().numpy()
    same(got[shift:shift + want.size].reshape(want.shape), want)
    assert (got[:shift] == 0xA5).all() and (got[shift + want.size:] == 0xA5).all()
