"""The convolution kernel that fetches every input pixel once per tile, against the CPU checker, byte for byte: every
requantisation mode, both slab widths, several channel chunks and tiles, patches that cross every edge of the image,
kernels that are not square, weights of one and of several channel tiles, few and many tiles per CTA."""
import numpy as np
import pytest

from conftest import pulpnn
from test_gpu_parity import MODES, conv_kw, pw_kw, same

pytestmark = pytest.mark.gpu
api, wl = pulpnn.api, pulpnn.workloads
KERNEL = "conv_halo_tc_kernel"


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
    c = wl.conv_case(110, 28, 28, 64, 64, batch=40, bits=bits, out_shift=11, with_bias=True, out_mult=3, relu=relu, bn=bn,
                     w_range=(-128, 127), k_range=(-64, 64), lam_range=(-2 ** 20, 2 ** 20))
    got = gpu.conv(bits, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    assert api.last_kernel() == KERNEL
    c["x"] = c["x"][-1:]
    same(got[-1:], restatement.conv(bits, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))


@pytest.mark.parametrize("H,W,Cin,Cout,kernel,pads,batch", [
    (28, 28, 128, 128, (3, 3), (1, 1, 1, 1), 32),
    (16, 8, 128, 128, (3, 3), (1, 1, 1, 1), 160),        # a patch is an image
    (33, 17, 64, 80, (3, 3), (1, 1, 1, 1), 60),           # ragged patches, columns that are no power of two
    (30, 31, 64, 16, (5, 5), (2, 2, 2, 2), 40),
    (20, 40, 128, 48, (3, 1), (1, 1, 0, 0), 40),
    (20, 40, 64, 64, (1, 7), (0, 0, 3, 3), 40),
    (40, 24, 64, 64, (3, 3), (0, 2, 2, 0), 50),
    (24, 24, 128, 256, (3, 3), (1, 1, 1, 1), 40),         # two channel tiles
    (16, 24, 256, 64, (3, 3), (1, 1, 1, 1), 80),          # two chunks
    (16, 24, 192, 96, (3, 3), (1, 1, 1, 1), 80),          # three chunks of 64
    (28, 28, 32, 64, (3, 3), (1, 1, 1, 1), 40),           # slabs of 32 bytes
    (17, 30, 96, 112, (3, 3), (1, 1, 1, 1), 40),
])
@pytest.mark.parametrize("strides", [(1, 1), (2, 2), (2, 1), (1, 2)])
def test_shapes(H, W, Cin, Cout, kernel, pads, batch, strides, gpu, restatement):
    c = wl.conv_case(111, H, W, Cin, Cout, kernel=kernel, pads=pads, strides=strides, batch=batch, out_shift=12)
    got = gpu.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    # where the boxes of a stride or the cuts of the channels leave another kernel ahead, or do not fit
    others = {(28, 28, 128): ((2, 1), (1, 2)), (16, 8, 128): ((2, 2),), (24, 24, 128): ((2, 2), (2, 1), (1, 2)),
              (16, 24, 256): ((2, 2), (2, 1)), (16, 24, 192): ((2, 2),)}
    assert (api.last_kernel() == KERNEL) == (strides not in others.get((H, W, Cin), ()))
    x = c["x"]
    for b in (0, batch // 2, batch - 1):
        same(got[b:b + 1], restatement.conv(32, x[b:b + 1], c["w"], c["k"], c["lam"], **conv_kw(c)))


# the most channels whose tiles find an SM each on 148 SMs, and more tiles than SMs, which are for other kernels
@pytest.mark.parametrize("Cin,Cout,kernel", [(32, 37888, (3, 3)), (32, 37904, (3, 3)), (64, 40000, (1, 3)), (32, 65520, (3, 1))])
def test_more_channel_tiles_than_sms(Cin, Cout, kernel, gpu, restatement):
    c = wl.conv_case(112, 4, 4, Cin, Cout, kernel=kernel, pads=(kernel[0] // 2,) * 2 + (kernel[1] // 2,) * 2, out_shift=12)
    got = gpu.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    assert (api.last_kernel() == KERNEL) == (Cout <= 256 * 148)
    same(got, restatement.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))


@pytest.mark.parametrize("H,C,N,batch,kernel", [(28, 64, 96, 3, KERNEL), (28, 128, 128, 40, KERNEL), (7, 512, 512, 1, "igemm_split_kernel"),
                                                (14, 256, 32, 2, "igemm_split_kernel")])
def test_between_network_layers(H, C, N, batch, kernel, restatement):
    """A convolution of a network, whose weights are fetched before the layer in front of it has ended."""
    x = np.random.default_rng(113).integers(0, 256, size=(batch, H, H, 48), dtype=np.uint8)
    first = wl.pointwise_case(114, H, H, 48, C, out_shift=10)
    conv = wl.conv_case(115, H, H, C, N, out_shift=13)
    last = wl.pointwise_case(116, H, H, N, 64, out_shift=12)
    net = api.Net(32, batch)
    for c, kind, cin, cout, extra in ((first, api.LAYER_POINTWISE, 48, C, {}), (conv, api.LAYER_CONV, C, N, dict(kernel=(3, 3), pads=(1, 1, 1, 1))),
                                      (last, api.LAYER_POINTWISE, N, 64, {})):
        net.add_layer(kind, dim_in=(H, H), ch_in=cin, dim_out=(H, H), ch_out=cout, out_shift=c["out_shift"], weights=c["w"],
                      k=c["k"], lam=c["lam"], **extra)
    net.finalize()
    for b in (0, batch - 1):
        t = restatement.pointwise(32, x[b:b + 1], first["w"], first["k"], first["lam"], **pw_kw(first))
        t = restatement.conv(32, t, conv["w"], conv["k"], conv["lam"], **conv_kw(conv))
        want = restatement.pointwise(32, t, last["w"], last["k"], last["lam"], **pw_kw(last))
        for _ in range(2):
            got = np.zeros((batch, H, H, 64), np.uint8)
            net.run(x, got, batch)
            same(got[b:b + 1], want)
    assert net.layer_kernel(1) == kernel
    net.close()
