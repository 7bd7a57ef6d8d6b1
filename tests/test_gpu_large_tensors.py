"""Tensors beyond 32-bit offsets: the kernel that takes them, and its results for the first and the last images."""
import numpy as np
import pytest

from conftest import pulpnn
from test_gpu_parity import conv_kw, same

pytestmark = pytest.mark.gpu
api, wl = pulpnn.api, pulpnn.workloads


def test_first_layer(restatement):
    import torch
    pulpnn.GpuKernels()
    B, H, W, C, N = 65535, 64, 171, 3, 2                 # 2.15 GB of images
    c = wl.conv_case(120, H, W, C, N, kernel=(3, 3), strides=(2, 2), batch=1, out_shift=9, with_bias=True)
    c["x"] = np.random.default_rng(121).integers(0, 256, size=(4, H, W, C), dtype=np.uint8)
    x = torch.empty((B, H, W, C), dtype=torch.uint8, device="cuda")
    x[:2], x[-2:] = (torch.from_numpy(c["x"][i:i + 2]).cuda() for i in (0, 2))
    Ho, Wo = c["out_hw"]
    out = torch.empty((B, Ho, Wo, N), dtype=torch.uint8, device="cuda")
    w, k, lam, bias = (torch.from_numpy(c[n]).cuda() for n in ("w", "k", "lam", "bias"))
    api.set_batch(B)
    api.pulp_nn_conv_Ho_parallel(32, x, None, bias, out, w, k, lam, 1, c["out_shift"], W, H, C, Wo, Ho, N, 3, 3, 1, 1, 1, 1,
                                 2, 2, 1, 1)
    api.synchronize()
    api.set_batch(1)
    assert api.last_kernel() == "conv_smallcin_kernel"
    got = torch.cat([out[:2], out[-2:]]).cpu().numpy()
    same(got, restatement.conv(32, c["x"], c["w"], c["k"], c["lam"], **conv_kw(c)))
