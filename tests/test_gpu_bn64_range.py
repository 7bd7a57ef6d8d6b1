"""64-bit batch-norm parameters on both sides of the range in which the kernels compute in 32 bits: values that
just fit, values that just do not, one wide channel among narrow ones, shifts above 31, and values whose product wraps.
Every kernel family, and the network runner with pairs of which one, both or neither layer fits."""
import numpy as np
import pytest

from conftest import pulpnn
from test_gpu_parity import conv_kw, dw_kw, pw_kw, same

pytestmark = pytest.mark.gpu
api, wl = pulpnn.api, pulpnn.workloads
KINDS = ["narrow", "edge", "one_wide", "wide", "wrap"]


@pytest.fixture(scope="module")
def gpu():
    return pulpnn.GpuKernels(host_buffers=False)


def params(kind, n, terms, seed=0):
    """k, lambda, shift for sums of `terms` products of at most 255 * 128."""
    rng = np.random.default_rng(seed + n)
    top = terms * 255 * 128
    k = rng.integers(1, 65, size=n).astype(np.int64)
    lam = rng.integers(-2 ** 15, 2 ** 15, size=n).astype(np.int64)
    if kind == "edge":          # the largest k that fits, and lambda at the end of what is left
        k[:] = (2 ** 31 - 1) // top
        lam[:] = 2 ** 31 - 1 - k * top
        lam[::2] *= -1
        lam[-1] += 1            # one past the end
        return k, lam, 20
    if kind == "one_wide":
        k[n // 2] = 2 ** 33 + 5
        lam[n // 2] = -2 ** 40
        return k, lam, 18
    if kind == "wide":
        return rng.integers(-2 ** 24, 2 ** 24, size=n).astype(np.int64), rng.integers(-2 ** 44, 2 ** 44, size=n).astype(np.int64), 36
    if kind == "wrap":
        return rng.integers(-2 ** 62, 2 ** 62, size=n).astype(np.int64), rng.integers(-2 ** 62, 2 ** 62, size=n).astype(np.int64), 40
    return k, lam, 12


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("H,Cin,Cout,batch", [(28, 128, 256, 12), (14, 512, 512, 40), (7, 1024, 1024, 200), (56, 32, 64, 24),
                                              (9, 48, 100, 2), (14, 512, 512, 1)])
def test_pointwise(kind, H, Cin, Cout, batch, gpu, restatement):
    c = wl.pointwise_case(100, H, H, Cin, Cout, batch=batch, bits=64, w_range=(-128, 127), with_bias=kind == "narrow")
    c["k"], c["lam"], c["out_shift"] = params(kind, Cout, Cin)
    got = gpu.pointwise(64, c["x"], c["w"], c["k"], c["lam"], **pw_kw(c))
    for b in (0, batch - 1):
        same(got[b:b + 1], restatement.pointwise(64, c["x"][b:b + 1], c["w"], c["k"], c["lam"], **pw_kw(c)))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("H,W,Cin,Cout,s", [(20, 32, 3, 32, 2), (9, 16, 3, 64, 1), (13, 11, 21, 37, 1), (14, 14, 128, 128, 1)])
def test_convolution(kind, H, W, Cin, Cout, s, gpu, restatement):
    c = wl.conv_case(101, H, W, Cin, Cout, strides=(s, s), batch=3, bits=64, w_range=(-128, 127))
    c["k"], c["lam"], c["out_shift"] = params(kind, Cout, 9 * Cin)
    same(gpu.conv(64, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)),
         restatement.conv(64, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("H,C,hwc,s,batch", [(28, 64, True, 1, 40), (32, 64, False, 2, 40), (13, 37, True, 1, 2), (56, 36, True, 1, 60)])
def test_depthwise(kind, H, C, hwc, s, batch, gpu, restatement):
    c = wl.depthwise_case(102, H, H, C, strides=(s, s), batch=batch, bits=64, w_range=(-128, 127), hwc=hwc)
    c["k"], c["lam"], c["out_shift"] = params(kind, C, 9)
    got = gpu.depthwise(64, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c))
    c["x"] = c["x"][-2:]
    same(got[-2:], restatement.depthwise(64, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c)))


@pytest.mark.parametrize("dw_kind", ["narrow", "edge", "wide"])
@pytest.mark.parametrize("pw_kind", ["narrow", "one_wide", "wide"])
def test_network_pair(dw_kind, pw_kind, restatement):
    H, C, N, B = 28, 128, 128, 3
    x = np.random.default_rng(9).integers(0, 256, size=(B, H, H, C), dtype=np.uint8)
    dw = wl.depthwise_case(103, H, H, C, batch=1, bits=64, w_range=(-128, 127), hwc=True)
    pw = wl.pointwise_case(104, H, H, C, N, batch=1, bits=64, w_range=(-128, 127))
    dw["k"], dw["lam"], ds = params(dw_kind, C, 9)
    pw["k"], pw["lam"], ps = params(pw_kind, N, C)
    net = api.Net(64, B)
    net.add_layer(api.LAYER_DEPTHWISE, dim_in=(H, H), ch_in=C, dim_out=(H, H), ch_out=C, kernel=(3, 3), pads=(1, 1, 1, 1),
                  out_shift=ds, weights=dw["w"], k=dw["k"], lam=dw["lam"])
    net.add_layer(api.LAYER_POINTWISE, dim_in=(H, H), ch_in=C, dim_out=(H, H), ch_out=N, out_shift=ps, weights=pw["w"],
                  k=pw["k"], lam=pw["lam"])
    net.finalize()
    got = np.zeros((B, H, H, N), np.uint8)
    net.run(x, got, B)
    roles = [net.layer_role(0), net.layer_role(1)]
    net.close()
    assert roles == [1, 2]
    t = restatement.depthwise(64, x, dw["w"], dw["k"], dw["lam"], out_shift=ds, out_hw=(H, H), kernel=(3, 3), pads=(1, 1, 1, 1),
                              strides=(1, 1), in_is_hwc=True)
    same(got, restatement.pointwise(64, t, pw["w"], pw["k"], pw["lam"], out_shift=ps))
