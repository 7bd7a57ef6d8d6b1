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


# The edge itself, on sums that reach it: pixels of 255 and weights of -128 make the largest sum there is, `top` below
# zero (with a bias of -128 still 128 more), and a negative k turns it into the largest k*sum + lambda. At 2^31 - 1 it is
# 127 after the shift; one more is 128, and 0 if it were computed in 32 bits.
SHIFT = 24


def at_the_edge(n, sum_max, past):
    """k, lambda of n channels whose largest value is 2^31 - 1, and 2^31 for one of them with `past`."""
    k = np.full(n, -((2 ** 31 - 1) // sum_max), np.int64)
    lam = 2 ** 31 - 1 + k * sum_max
    lam[n // 2] += past
    return k, lam


def edge_case(c, n, terms, past, bias, w=-128):
    c["x"][:], c["w"][:] = 255, w
    c["bias"] = np.full(n, -128, np.int8) if bias else None
    c["k"], c["lam"] = at_the_edge(n, terms * 255 * -w + 128 * bias, past)
    c["out_shift"] = SHIFT
    return c


def edge_result(got, n, past):
    assert got[..., n // 2].max() == 127 + past and np.delete(got, n // 2, axis=-1).max() == 127


@pytest.mark.parametrize("bias", [0, 1])
@pytest.mark.parametrize("past", [0, 1])
@pytest.mark.parametrize("H,Cin,Cout,batch,kernel", [
    (28, 128, 256, 12, "igemm_tc_kernel"), (56, 32, 64, 24, "igemm_tc_kernel"), (14, 1024, 1024, 97, "igemm_tc2_kernel"),
    (14, 512, 512, 1, "igemm_split_kernel"), (14, 1024, 256, 1, "igemm_split_kernel"), (9, 48, 100, 2, "conv_gather_tc_kernel")])
def test_edge_pointwise(H, Cin, Cout, batch, kernel, past, bias, gpu, restatement):
    c = edge_case(wl.pointwise_case(105, H, H, Cin, Cout, batch=batch, bits=64), Cout, Cin, past, bias)
    got = gpu.pointwise(64, c["x"], c["w"], c["k"], c["lam"], **pw_kw(c))
    assert api.last_kernel() == kernel
    edge_result(got, Cout, past)
    same(got[-1:], restatement.pointwise(64, c["x"][-1:], c["w"], c["k"], c["lam"], **pw_kw(c)))


@pytest.mark.parametrize("bias", [0, 1])
@pytest.mark.parametrize("past", [0, 1])
@pytest.mark.parametrize("H,W,Cin,Cout,s,batch,kernel", [
    (20, 32, 3, 32, 2, 3, "conv_smallcin_tc_kernel"), (9, 16, 3, 64, 1, 3, "conv_smallcin_tc_kernel"),
    (13, 11, 21, 37, 1, 3, "conv_gather_tc_kernel"), (14, 14, 128, 128, 1, 3, "conv_halo_tc_kernel"),
    (7, 7, 512, 512, 1, 1, "igemm_split_kernel"), (28, 28, 224, 224, 1, 16, "igemm_tc_kernel")])
def test_edge_convolution(H, W, Cin, Cout, s, batch, kernel, past, bias, gpu, restatement):
    c = edge_case(wl.conv_case(106, H, W, Cin, Cout, strides=(s, s), batch=batch, bits=64), Cout, 9 * Cin, past, bias)
    got = gpu.conv(64, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    assert api.last_kernel() == kernel
    edge_result(got, Cout, past)
    c["x"] = c["x"][-1:]
    same(got[-1:], restatement.conv(64, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))


@pytest.mark.parametrize("bias", [0, 1])
@pytest.mark.parametrize("past", [0, 1])
@pytest.mark.parametrize("H,C,k,hwc,s,batch,kernel", [
    (28, 64, 3, True, 1, 60, "depthwise_hwc3x3_tma_kernel"), (64, 64, 3, False, 1, 20, "depthwise_chw3x3_tma_kernel"),
    (13, 37, 3, True, 1, 2, "depthwise_planes_kernel"), (13, 37, 5, False, 2, 2, "depthwise_planes_kernel"),
    (56, 36, 3, True, 1, 60, "depthwise_hwc3x3_kernel")])
def test_edge_depthwise(H, C, k, hwc, s, batch, kernel, past, bias, gpu, restatement):
    c = wl.depthwise_case(107, H, H, C, kernel=(k, k), strides=(s, s), pads=(k // 2,) * 4, batch=batch, bits=64, hwc=hwc)
    c = edge_case(c, C, k * k, past, bias)
    got = gpu.depthwise(64, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c))
    assert api.last_kernel() == kernel
    edge_result(got, C, past)
    c["x"] = c["x"][-1:]
    same(got[-1:], restatement.depthwise(64, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c)))


@pytest.mark.parametrize("bias", [0, 1])
@pytest.mark.parametrize("past", [0, 1])
@pytest.mark.parametrize("w", [-128, -100])
def test_edge_network_layers(w, past, bias, restatement):
    """The runner's own proof, by the largest weights there can be (-128) and by the layer's own sum (-100): a depthwise,
    a convolution and a pointwise layer, each the first of a network, so that its input is all 255."""
    H, C, N, B = 28, 64, 96, 2
    dw = edge_case(wl.depthwise_case(108, H, H, C, batch=B, bits=64, hwc=True), C, 9, past, bias, w)
    cv = edge_case(wl.conv_case(108, H, H, C, N, batch=B, bits=64), N, 9 * C, past, bias, w)
    pw = edge_case(wl.pointwise_case(108, H, H, C, N, batch=B, bits=64), N, C, past, bias, w)
    for kind, c, n, extra, want in (
            (api.LAYER_DEPTHWISE, dw, C, dict(kernel=(3, 3), pads=(1, 1, 1, 1)),
             restatement.depthwise(64, dw["x"], dw["w"], dw["k"], dw["lam"], **dw_kw(dw))),
            (api.LAYER_CONV, cv, N, dict(kernel=(3, 3), pads=(1, 1, 1, 1)),
             restatement.conv(64, cv["x"], cv["w"], cv["k"], cv["lam"], **conv_kw(cv))),
            (api.LAYER_POINTWISE, pw, N, {}, restatement.pointwise(64, pw["x"], pw["w"], pw["k"], pw["lam"], **pw_kw(pw)))):
        net = api.Net(64, B)
        net.add_layer(kind, dim_in=(H, H), ch_in=C, dim_out=(H, H), ch_out=n, out_shift=SHIFT, weights=c["w"], bias=c["bias"],
                      k=c["k"], lam=c["lam"], **extra)
        net.finalize()
        got = np.zeros((B, H, H, n), np.uint8)
        net.run(c["x"], got, B)
        net.close()
        edge_result(got, n, past)
        same(got, want)
