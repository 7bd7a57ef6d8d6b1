"""The gathering tensor-core kernel (channel counts and alignments no TMA box takes) against the CPU
checker, byte for byte: every requantisation mode, both trees, and the shapes at which its layout can
go wrong -- runs that end inside, at and just past a 16-byte chunk and a 128-byte slab, windows that
cross every edge of the image, tiles that end inside the last image, outputs of 1, 4 and 16 bytes'
alignment, weights that stay in shared memory and weights that do not, several tiles per CTA."""
import numpy as np
import pytest

from conftest import pulpnn
from test_gpu_parity import MODES, conv_kw, pw_kw, same

pytestmark = pytest.mark.gpu
api, wl = pulpnn.api, pulpnn.workloads
KERNEL = "conv_gather_tc_kernel"


@pytest.fixture(scope="module")
def gpu():
    return pulpnn.GpuKernels(host_buffers=False)


@pytest.fixture(autouse=True)
def _status():
    yield
    assert api.device_status() == 0


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("relu,bn", MODES)
def test_modes(bits, relu, bn, gpu, restatement):
    c = wl.conv_case(70, 13, 11, 21, 37, strides=(1, 2), batch=3, bits=bits, out_shift=9, with_bias=True, out_mult=3,
                     relu=relu, bn=bn, w_range=(-128, 127), k_range=(-64, 64), lam_range=(-2 ** 20, 2 ** 20))
    got = gpu.conv(bits, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    assert api.last_kernel() == KERNEL
    same(got, restatement.conv(bits, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))


CONVS = [  # H, W, Cin, Cout, kernel, strides, pads (top, bottom, left, right), batch
    (7, 9, 5, 16, (3, 3), (1, 1), (1, 1, 1, 1), 2),        # runs of 15 bytes
    (7, 9, 16, 33, (3, 3), (1, 1), (1, 1, 1, 1), 2),       # whole chunks, odd output
    (16, 16, 48, 256, (3, 3), (2, 2), (1, 1, 1, 1), 3),    # whole chunks, weights gathered per slab
    (9, 8, 17, 8, (1, 3), (1, 1), (0, 0, 1, 1), 1),
    (6, 70, 43, 260, (3, 3), (1, 1), (1, 1, 1, 1), 2),     # runs of 129 bytes, two channel tiles, 4-byte rows
    (6, 50, 20, 301, (3, 3), (1, 1), (0, 2, 2, 0), 2),     # two channel tiles, odd rows
    (12, 12, 3, 1, (5, 5), (3, 2), (4, 4, 4, 4), 3),       # windows wholly in the padding
    (40, 40, 20, 40, (3, 3), (1, 1), (1, 1, 1, 1), 33),    # several tiles per CTA
    (5, 5, 250, 24, (5, 5), (1, 1), (2, 2, 2, 2), 1),      # long reduction
]


@pytest.mark.parametrize("H,W,Cin,Cout,kernel,strides,pads,batch", CONVS)
def test_convolutions(H, W, Cin, Cout, kernel, strides, pads, batch, gpu, restatement):
    c = wl.conv_case(71, H, W, Cin, Cout, kernel=kernel, strides=strides, pads=pads, batch=batch, out_shift=10,
                     with_bias=True, w_range=(-128, 127))
    got = gpu.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    assert api.last_kernel() == KERNEL
    same(got, restatement.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))


@pytest.mark.parametrize("cin,cout", [(1, 1), (15, 16), (17, 20), (31, 3), (127, 130), (129, 64), (257, 256), (1000, 999), (4095, 70)])
def test_pointwise_and_linear(cin, cout, gpu, restatement):
    c = wl.pointwise_case(72, 9, 15, cin, cout, batch=2, out_shift=9, with_bias=True, w_range=(-128, 127))
    got = gpu.pointwise(32, c["x"], c["w"], c["k"], c["lam"], **pw_kw(c))
    assert api.last_kernel() == (KERNEL if cin > 12 else "conv_smallcin_kernel")
    same(got, restatement.pointwise(32, c["x"], c["w"], c["k"], c["lam"], **pw_kw(c)))
    for batch in (1, 130):
        c = wl.linear_case(73, cin, cout, batch=batch, with_bias=True)
        got = gpu.linear_out_32(c["x"], c["w"], bias32=c["bias32"])
        assert api.last_kernel() == (KERNEL if cin > 44 else "conv_generic_kernel")
        same(got, restatement.linear_out_32(c["x"], c["w"], bias32=c["bias32"]))


@pytest.mark.parametrize("shift_in,shift_w,shift_out", [(1, 0, 0), (0, 3, 0), (8, 8, 4), (5, 2, 1)])
def test_unaligned_buffers(shift_in, shift_w, shift_out, gpu, restatement):
    """Operands and output that start anywhere; bytes around the output stay as they were."""
    import torch
    c = wl.conv_case(74, 9, 10, 32, 48, batch=2, out_shift=12, with_bias=False)
    want = restatement.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    dev = lambda a, s: torch.cat([torch.zeros(s, dtype=torch.uint8), torch.from_numpy(a.reshape(-1).view(np.uint8))]).cuda()  # noqa: E731
    x, w = dev(c["x"], shift_in), dev(c["w"], shift_w)
    out = torch.full((shift_out + want.size + 16,), 0xA5, dtype=torch.uint8, device="cuda")
    k, lam = torch.from_numpy(c["k"]).cuda(), torch.from_numpy(c["lam"]).cuda()
    api.set_batch(2)
    api.pulp_nn_conv_Ho_parallel(32, x[shift_in:], None, None, out[shift_out:], w[shift_w:], k, lam, 1, 12, 10, 9, 32,
                                 10, 9, 48, 3, 3, 1, 1, 1, 1, 1, 1, 1, 1)
    api.synchronize()
    assert api.last_kernel() == KERNEL
    got = out.cpu().numpy()
    same(got[shift_out:shift_out + want.size].reshape(want.shape), want)
    assert (got[:shift_out] == 0xA5).all() and (got[shift_out + want.size:] == 0xA5).all()
