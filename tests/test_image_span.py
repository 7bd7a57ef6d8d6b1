"""The words that the plane-staging depthwise kernel may read lie inside the tensor, for images of a few bytes too (host
arithmetic of csrc/unaligned16.cuh; a read past a tensor changes no output, so no comparison of results sees it)."""
import os
import subprocess

from conftest import ROOT, pulpnn


def test_words_lie_inside_the_tensor(tmp_path):
    exe = str(tmp_path / "image_span")
    subprocess.run([pulpnn._lib._nvcc(), "-std=c++17", "-I" + pulpnn._lib.CSRC, "-I" + pulpnn._lib.INCLUDE, "-o", exe,
                    os.path.join(ROOT, "tests", "data", "image_span.cu")], check=True)
    words, outside = map(int, subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert words > 10000 and outside == 0
