"""Which route small builds take where a cluster of 16 blocks does not fit: the general one, and the
context is created all the same.  The host side of csrc/small.cu compiled against a runtime that answers
as such a device does (no GPU)."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "webgpu-lvbh-demo_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

PROGRAM = r"""
#include <cstdio>
#include <cuda_runtime.h>
static cudaError_t g_attr = cudaSuccess, g_query = cudaSuccess;
static int g_clusters = 1;
template <class K> cudaError_t fake_attr(K, cudaFuncAttribute, int) { return g_attr; }
template <class K> cudaError_t fake_query(int *c, K, const cudaLaunchConfig_t *) { *c = g_clusters; return g_query; }
#define cudaFuncSetAttribute fake_attr
#define cudaOccupancyMaxActiveClusters fake_query
#include "small.cu"
static int route(cudaError_t attr, cudaError_t query, int clusters) {
    g_attr = g_query = cudaSuccess; g_clusters = 4;  // whatever an earlier device said
    lvbh::small_init();
    g_attr = attr; g_query = query; g_clusters = clusters;
    lvbh::small_init();
    return (int)lvbh::small_build(100);
}
int main() {
    std::printf("fits %d\n", route(cudaSuccess, cudaSuccess, 4));
    std::printf("too_large %d\n", (int)lvbh::small_build(lvbh::kSmallMax + 1));
    std::printf("none %d\n", route(cudaSuccess, cudaSuccess, 0));
    std::printf("query_error %d\n", route(cudaSuccess, cudaErrorInvalidClusterSize, 0));
    std::printf("query_error_stale %d\n", route(cudaSuccess, cudaErrorInvalidClusterSize, 3));
    std::printf("attr_error %d\n", route(cudaErrorInvalidValue, cudaSuccess, 4));
    std::printf("fits_again %d\n", route(cudaSuccess, cudaSuccess, 1));
}
"""


def test_small_builds_where_no_cluster_fits(tmp_path):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "route.cu", tmp_path / "route"
    src.write_text(PROGRAM)
    subprocess.run([NVCC, "-O1", "-std=c++17", "-gencode", "arch=compute_100a,code=compute_100a", "-I", CSRC, "-I",
                    os.path.join(REPO, "include"), str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert dict(x.split() for x in out.splitlines()) == {
        "fits": "1", "too_large": "0", "none": "0", "query_error": "0", "query_error_stale": "0", "attr_error": "0",
        "fits_again": "1"}


def test_no_answer_of_the_query_fails_the_context():
    """lvbh_create goes on whatever small_init finds: it has no status to fail on."""
    with open(os.path.join(CSRC, "api.cu")) as f:
        src = f.read()
    create = src[src.index("int lvbh_create("):src.index("void lvbh_destroy(")]
    assert "\n    small_init();\n" in create
