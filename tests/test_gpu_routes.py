"""Calls on the far side of a line that the dispatch draws between two kernels: which one takes them, and its bytes."""
import pytest

from conftest import pulpnn
from test_gpu_parity import conv_kw, same

pytestmark = pytest.mark.gpu
api, wl = pulpnn.api, pulpnn.workloads


@pytest.fixture(scope="module")
def gpu():
    return pulpnn.GpuKernels(host_buffers=False)


@pytest.fixture(autouse=True)
def _status():
    yield
    assert api.device_status() == 0


# images of one or a few rows, of which the halo kernel's 8x16 patches would be mostly outside; long reductions of few patches
@pytest.mark.parametrize("B,H,W,Cin,Cout,kernel,strides,took", [
    (3, 1, 3340, 288, 224, (1, 3), (1, 1), "igemm_tc_kernel"), (5, 1, 1201, 160, 32, (1, 3), (1, 1), "conv_gather_tc_kernel"),
    (30, 1, 2776, 32, 448, (1, 3), (1, 2), "igemm_tc_kernel"), (105, 4, 302, 416, 16, (3, 1), (1, 1), "conv_gather_tc_kernel"),
    (1, 11, 4, 416, 32, (3, 3), (1, 1), "conv_gather_tc_kernel"), (1, 4, 4, 96, 16, (9, 9), (2, 2), "conv_gather_tc_kernel"),
    (1, 7, 7, 512, 512, (3, 3), (1, 1), "igemm_split_kernel"), (32, 28, 28, 128, 128, (3, 3), (1, 1), "conv_halo_tc_kernel")])
def test_spatial_kernels(B, H, W, Cin, Cout, kernel, strides, took, gpu, restatement):
    c = wl.conv_case(130, H, W, Cin, Cout, kernel=kernel, strides=strides, pads=(kernel[0] // 2,) * 2 + (kernel[1] // 2,) * 2,
                     batch=B, out_shift=12)
    got = gpu.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    assert api.last_kernel() == took
    c["x"] = c["x"][-1:]
    same(got[-1:], restatement.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))
