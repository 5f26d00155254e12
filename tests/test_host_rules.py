"""Host-side rules of the CUDA sources, compiled into a small program and run without a GPU."""

import subprocess

import pytest

import test_gpu_gemm
import test_gpu_token_channel
from gaudi_kernels_b200 import _lib, build

CLUSTER_CAPS = r"""
#include <stdio.h>
#include "common.cuh"

static bfp8::ClusterCaps caps[2];
static int asked = 0;
static int ask(bfp8::ClusterCaps& c, int dev, int cluster, bool ok, int number) {
  return bfp8::cached_clusters(c, dev, cluster, [&](int* out) { ++asked; *out = number; return ok; });
}
#define EXPECT(x) do { if (!(x)) { printf("line %d: %s (asked %d)\n", __LINE__, #x, asked); return 1; } } while (0)

int main() {
  EXPECT(ask(caps[0], 0, 4, false, 99) == 0 && asked == 1);        // a failed query: not this time
  EXPECT(ask(caps[0], 0, 4, true, 18) == 18 && asked == 2);        // but asked again
  EXPECT(ask(caps[0], 0, 4, true, 7) == 18 && asked == 2);         // an answer is kept
  EXPECT(ask(caps[0], 0, 8, true, 0) == 0 && asked == 3);          // "none" too
  EXPECT(ask(caps[0], 0, 8, true, 9) == 0 && asked == 3);
  EXPECT(ask(caps[0], 1, 4, true, 5) == 5 && asked == 4);          // by device
  EXPECT(ask(caps[1], 0, 4, true, 6) == 6 && asked == 5);          // and by kernel
  EXPECT(ask(caps[0], 64, 2, true, 3) == 3 && ask(caps[0], 64, 2, true, 4) == 4 && asked == 7);   // no slot: always asked
  EXPECT(ask(caps[0], 0, 0, true, 3) == 0 && ask(caps[0], 0, 9, true, 3) == 0 && asked == 7);
  return 0;
}
"""


def _run(source, tmp_path):
    path, exe = str(tmp_path / "host_rule.cu"), str(tmp_path / "host_rule")
    with open(path, "w") as f:
        f.write(source)
    subprocess.run([build._nvcc()] + build.ARCH_FLAGS + ["-std=c++17", "-I" + build.INCLUDE, "-I" + build.CSRC, path, "-o", exe],
                   check=True, capture_output=True, text=True, timeout=300)
    return subprocess.run([exe], capture_output=True, text=True, timeout=60)


def test_cluster_residency_is_kept_by_kernel_and_never_a_failure(tmp_path):
    res = _run(CLUSTER_CAPS, tmp_path)
    assert res.returncode == 0, res.stdout


@pytest.mark.parametrize("token_channel,shapes", [(0, test_gpu_gemm.SPLIT_SHAPES), (1, test_gpu_token_channel.FORMS)])
def test_the_gpu_tests_reach_every_cluster_size(token_channel, shapes):
    build.build()
    split = _lib.load().bfp8_gemm_k_split
    for (m, k, n), want in shapes.items():
        assert split(m, n, k, token_channel, 148) == want, (m, k, n)
    large = {want for (m, k, n), want in shapes.items() if m > 128}
    assert large >= {2, 3, 4, 5, 6, 7, 8}
    if token_channel:
        assert {want for (m, k, n), want in shapes.items() if m <= 64} >= {1, 2, 4, 8} and 1 in large
    assert split(0, 1, 1, token_channel, 148) < 0
