"""GEMMs of few tiles, whose reduction the CTAs of a cluster share, against the CPU checker, byte for byte: every
requantisation mode, reductions that do not divide among the CTAs, ragged rows and columns, K that ends inside a
slab, patches of a convolution that cross the image's edge, and the shapes on either side of the dispatch's lines."""
import numpy as np
import pytest

from conftest import pulpnn
from test_gpu_parity import MODES, conv_kw, pw_kw, same

pytestmark = pytest.mark.gpu
api, wl = pulpnn.api, pulpnn.workloads
KERNEL = "igemm_split_kernel"


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
    c = wl.linear_case(90, 1040, 77, batch=131, bits=bits, out_shift=9, with_bias=True, out_mult=3, relu=relu, bn=bn,
                       w_range=(-128, 127), k_range=(-64, 64), lam_range=(-2 ** 20, 2 ** 20))
    kw = dict(bias=c["bias"], out_mult=3, out_shift=c["out_shift"], relu=relu, bn=bn)
    got = gpu.linear(bits, c["x"], c["w"], c["k"], c["lam"], **kw)
    assert api.last_kernel() == KERNEL
    same(got, restatement.linear(bits, c["x"], c["w"], c["k"], c["lam"], **kw))
    c = wl.conv_case(91, 9, 13, 256, 40, batch=1, bits=bits, out_shift=12, with_bias=True, out_mult=3, relu=relu, bn=bn,
                     k_range=(-64, 64), lam_range=(-2 ** 20, 2 ** 20))
    got = gpu.conv(bits, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    assert api.last_kernel() == KERNEL
    same(got, restatement.conv(bits, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))


@pytest.mark.parametrize("batch,K,N", [(8, 1024, 16), (49, 1024, 1024), (128, 1024, 1000), (129, 4096, 33), (196, 512, 512),
                                       (200, 1168, 100), (256, 2048, 257), (300, 4096, 64), (5, 65520, 20), (300, 528, 48)])
def test_linear(batch, K, N, gpu, restatement):
    kernel = {8: "gemm_fewrows_kernel", 5: "igemm_tc_kernel", 300: KERNEL if K > 1024 else "igemm_tc_kernel"}.get(batch, KERNEL)
    c = wl.linear_case(92, K, N, batch=batch, with_bias=True)
    got = gpu.linear_out_32(c["x"], c["w"], bias32=c["bias32"])
    assert api.last_kernel() == kernel
    same(got, restatement.linear_out_32(c["x"], c["w"], bias32=c["bias32"]))
    c = wl.pointwise_case(93, batch, 1, K, N, out_shift=13, with_bias=True)
    got = gpu.pointwise(32, c["x"], c["w"], c["k"], c["lam"], **pw_kw(c))
    assert api.last_kernel() == kernel
    same(got, restatement.pointwise(32, c["x"], c["w"], c["k"], c["lam"], **pw_kw(c)))


@pytest.mark.parametrize("H,W,Cin,Cout,k,s,p,batch", [(7, 7, 512, 512, 3, 1, 1, 1), (16, 16, 256, 256, 5, 1, 2, 1),
                                                      (14, 14, 256, 100, 3, 2, 1, 3), (5, 33, 384, 24, 3, 1, 1, 1),
                                                      (14, 14, 64, 64, 3, 1, 1, 1), (32, 32, 32, 64, 3, 1, 1, 1)])
def test_convolution(H, W, Cin, Cout, k, s, p, batch, gpu, restatement):
    c = wl.conv_case(94, H, W, Cin, Cout, kernel=(k, k), strides=(s, s), pads=(p, p, p, p), batch=batch, out_shift=13)
    got = gpu.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    assert api.last_kernel() == (KERNEL if Cin >= 256 else "conv_halo_tc_kernel")
    same(got, restatement.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))


# one CTA per tile, whole 16-byte pieces: the rows leave from registers. The last tile's columns end at half a piece of 32.
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("relu,bn", MODES)
@pytest.mark.parametrize("M,K,N", [(196, 512, 512), (131, 528, 304), (49, 512, 1040)])
def test_rows_from_registers(M, K, N, bits, relu, bn, gpu, restatement):
    c = wl.pointwise_case(95, 1, M, K, N, bits=bits, out_shift=11, with_bias=True, out_mult=3, relu=relu, bn=bn,
                          k_range=(-64, 64), lam_range=(-2 ** 20, 2 ** 20))
    got = gpu.pointwise(bits, c["x"], c["w"], c["k"], c["lam"], **pw_kw(c))
    assert api.last_kernel() == (KERNEL if K == 512 else "igemm_tc_kernel")
    same(got, restatement.pointwise(bits, c["x"], c["w"], c["k"], c["lam"], **pw_kw(c)))
