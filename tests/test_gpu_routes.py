"""Calls on the far side of a line that the dispatch draws between two kernels: which one takes them, and its bytes."""
import pytest

from conftest import pulpnn
from test_gpu_parity import conv_kw, dw_kw, same

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
    (1, 7, 7, 512, 512, (3, 3), (1, 1), "igemm_split_kernel"), (1, 102, 102, 128, 128, (3, 3), (1, 1), "conv_halo_tc_kernel"), (32, 28, 28, 128, 128, (3, 3), (1, 1), "conv_halo_tc_kernel")])
def test_spatial_kernels(B, H, W, Cin, Cout, kernel, strides, took, gpu, restatement):
    c = wl.conv_case(130, H, W, Cin, Cout, kernel=kernel, strides=strides, pads=(kernel[0] // 2,) * 2 + (kernel[1] // 2,) * 2,
                     batch=B, out_shift=12)
    got = gpu.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    assert api.last_kernel() == took
    c["x"] = c["x"][-1:]
    same(got[-1:], restatement.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))


# rows of no whole 16-byte pieces, few and many values a tile (the line: 1700 values, five slabs)
@pytest.mark.parametrize("B,K,N,took", [(24, 48, 3, "igemm_tc_kernel"), (1, 32, 38, "igemm_tc_kernel"), (300, 320, 13, "igemm_tc_kernel"),
                                        (2815, 32, 2, "igemm_tc_kernel"), (300, 320, 14, "conv_gather_tc_kernel"),
                                        (24, 16, 77, "conv_gather_tc_kernel")])
def test_ragged_rows(B, K, N, took, gpu, restatement):
    c = wl.linear_case(131, K, N, batch=B, with_bias=True)
    kw = dict(bias=c["bias"], out_mult=c["out_mult"], out_shift=9, relu=c["relu"], bn=c["bn"])
    got = gpu.linear(32, c["x"], c["w"], c["k"], c["lam"], **kw)
    assert api.last_kernel() == took
    same(got, restatement.linear(32, c["x"], c["w"], c["k"], c["lam"], **kw))
    if N % 4:
        got = gpu.linear_out_32(c["x"], c["w"], bias32=c["bias32"])
        assert api.last_kernel() == took
        same(got, restatement.linear_out_32(c["x"], c["w"], bias32=c["bias32"]))


# 32-bit outputs of short reductions of no whole 16 bytes (the line: 44 terms, one round of 64x64 tiles)
@pytest.mark.parametrize("B,K,N,took", [(2, 4, 4, "conv_generic_kernel"), (58, 8, 1896, "conv_generic_kernel"), (70, 44, 33, "conv_generic_kernel"),
                                        (70, 45, 33, "conv_gather_tc_kernel"), (2500, 12, 300, "conv_gather_tc_kernel")])
def test_short_reductions(B, K, N, took, gpu, restatement):
    c = wl.linear_case(132, K, N, batch=B, with_bias=True)
    got = gpu.linear_out_32(c["x"], c["w"], bias32=c["bias32"])
    assert api.last_kernel() == took
    same(got, restatement.linear_out_32(c["x"], c["w"], bias32=c["bias32"]))


# first layers: the kernel that walks strips of an image, and the gathering one where its strips leave the GPU idle
@pytest.mark.parametrize("B,H,W,Cin,Cout,k,took", [
    (1, 6, 6, 4, 32, 1, "conv_smallcin_kernel"), (21, 575, 291, 1, 16, 3, "conv_smallcin_kernel"), (64, 28, 28, 1, 16, 3, "conv_smallcin_kernel"),
    (1, 5, 5, 3, 32, 2, "conv_smallcin_kernel"), (16, 96, 96, 3, 24, 3, "conv_gather_tc_kernel"), (16, 28, 28, 1, 16, 5, "conv_gather_tc_kernel"),
    (1, 1, 4500, 3, 16, 4, "conv_gather_tc_kernel")])
def test_first_layers(B, H, W, Cin, Cout, k, took, gpu, restatement):
    p = k // 2
    kernel = (1, k) if H == 1 else (k, k)
    c = wl.conv_case(133, H, W, Cin, Cout, kernel=kernel, pads=(p if H > 1 else 0,) * 2 + (p, p), batch=B, out_shift=9, with_bias=True)
    got = gpu.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    assert api.last_kernel() == took
    c["x"] = c["x"][-1:]
    same(got[-1:], restatement.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))


# reductions on both sides of 18000 terms: a cluster, or slices whose sums go through memory, which a stream capture may not
# hold on to and two streams of a thread share
@pytest.mark.parametrize("B,K,N,took", [(1, 17984, 20, "igemm_split_kernel"), (5, 18000, 20, "igemm_tc_kernel"), (130, 65520, 33, "igemm_tc_kernel")])
def test_long_reductions(B, K, N, took, gpu, restatement):
    c = wl.linear_case(134, K, N, batch=B, with_bias=True)
    got = gpu.linear_out_32(c["x"], c["w"], bias32=c["bias32"])
    assert api.last_kernel() == took
    same(got, restatement.linear_out_32(c["x"], c["w"], bias32=c["bias32"]))
    kw = dict(bias=c["bias"], out_mult=c["out_mult"], out_shift=14, relu=c["relu"], bn=c["bn"])
    same(gpu.linear(32, c["x"], c["w"], c["k"], c["lam"], **kw), restatement.linear(32, c["x"], c["w"], c["k"], c["lam"], **kw))


def test_long_convolution(gpu, restatement):
    c = wl.conv_case(135, 9, 8, 448, 30, kernel=(7, 7), pads=(3, 3, 3, 3), out_shift=15)
    got = gpu.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c))
    assert api.last_kernel() == "igemm_tc_kernel"
    same(got, restatement.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))


@pytest.mark.parametrize("first", ["eager", "captured"])
def test_long_reduction_under_capture(first, restatement):
    import threading

    import torch
    c = wl.linear_case(136, 20000, 24, batch=3, with_bias=True)
    put = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    x, w, bias = put(c["x"]), put(c["w"]), put(c["bias32"])
    out = torch.zeros((3, 24), dtype=torch.int32, device="cuda")
    took = []

    def work():                                  # a thread of its own has a context of its own, without memory for sums
        torch.cuda.set_device(0)
        api.set_device(0)
        api.set_batch(3)
        s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        if first == "eager":
            api.pulp_nn_linear_out_32(32, x, bias, out, w, 20000, 24)
            took.append(api.last_kernel())
            torch.cuda.synchronize()
            out.zero_()
        with torch.cuda.graph(g, stream=s):
            api.set_stream(s.cuda_stream)
            api.pulp_nn_linear_out_32(32, x, bias, out, w, 20000, 24)
        took.append(api.last_kernel())
        g.replay()
        torch.cuda.synchronize()

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert took == ["igemm_tc_kernel"] * (first == "eager") + ["igemm_split_kernel"]
    same(out.cpu().numpy(), restatement.linear_out_32(c["x"], c["w"], bias32=c["bias32"]))


def test_long_reductions_on_two_streams(gpu, restatement):
    import torch
    cases = [wl.linear_case(138 + i, 40000, 500, batch=64, with_bias=True) for i in range(2)]
    put = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    args = [[put(c[n]) for n in ("x", "bias32", "w")] for c in cases]
    outs = [[torch.zeros((64, 500), dtype=torch.int32, device="cuda") for _ in range(2)] for _ in range(20)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    api.set_batch(64)
    try:
        for pair in outs:
            for (x, bias, w), out, s in zip(args, pair, streams):
                api.set_stream(s.cuda_stream)
                api.pulp_nn_linear_out_32(32, x, bias, out, w, 40000, 500)
                assert api.last_kernel() == "igemm_tc_kernel"
    finally:
        api.set_stream(0)
        api.set_batch(1)
    torch.cuda.synchronize()
    for i, c in enumerate(cases):
        want = restatement.linear_out_32(c["x"], c["w"], bias32=c["bias32"])
        for pair in outs:
            same(pair[i].cpu().numpy(), want)


def test_long_reduction_beside_a_capture_of_another_thread(gpu, restatement):
    """A thread that gets memory for its sums, and gives it back at its end, while another one captures a graph."""
    import threading

    import torch
    c = wl.linear_case(140, 40000, 500, batch=64, with_bias=True)
    put = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    x, w, bias = put(c["x"]), put(c["w"]), put(c["bias32"])
    out, short = (torch.zeros((64, 500), dtype=torch.int32, device="cuda") for _ in range(2))
    free, started, captured, took = [], threading.Event(), threading.Event(), []

    def work():
        torch.cuda.set_device(0)
        api.set_device(0)
        api.set_batch(64)
        api.set_stream(stream)
        api.pulp_nn_linear_out_32(32, x, bias, short, w, 4000, 500)      # what every thread allocates
        api.synchronize()
        started.set()
        captured.wait(60)
        api.pulp_nn_linear_out_32(32, x, bias, out, w, 40000, 500)
        took.append(api.last_kernel())

    for _ in range(8):
        stream, side, g = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
        out.zero_()
        torch.cuda.synchronize()
        started.clear()
        captured.clear()
        t = threading.Thread(target=work)
        t.start()
        assert started.wait(60)
        with torch.cuda.graph(g, stream=side):
            short.zero_()
            captured.set()
            t.join()
        g.replay()
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert took == ["igemm_tc_kernel"] * 8 and not short.any()
    assert free[1] - free[-1] < 8 << 20                  # the sums of one call alone are 2 MB in 16 slices each
    same(out.cpu().numpy(), restatement.linear_out_32(c["x"], c["w"], bias32=c["bias32"]))


# depthwise layers with one row of output, of which the plane kernel computes two or four
@pytest.mark.parametrize("B,W,C,k,s,hwc,took", [
    (1, 1958, 128, 3, 2, True, "depthwise_hwc3x3_tma_kernel"), (15, 80, 32, 3, 1, False, "depthwise_chw3x3_tma_kernel"),
    (1, 749, 148, 3, 1, True, "depthwise_planes_kernel"), (45, 1830, 16, 3, 2, True, "depthwise_hwc3x3_kernel"),
    (25, 101, 128, 5, 2, True, "depthwise_planes_kernel"), (5, 2109, 224, 5, 1, True, "depthwise_generic_kernel"),
    (24, 1643, 174, 3, 1, True, "depthwise_planes_kernel")])
def test_one_row_depthwise(B, W, C, k, s, hwc, took, gpu, restatement):
    p = k // 2
    c = wl.depthwise_case(137, 1, W, C, kernel=(k, k), strides=(s, s), pads=(p, p, p, p), batch=B, out_shift=9, hwc=hwc)
    got = gpu.depthwise(32, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c))
    assert api.last_kernel() == took
    c["x"] = c["x"][-1:]
    same(got[-1:], restatement.depthwise(32, c["x"], c["w"], c["k"], c["lam"], **dw_kw(c)))
