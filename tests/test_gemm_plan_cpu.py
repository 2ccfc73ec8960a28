"""How a product is shared out among the SMs (csrc/tma_gemm_kernel.cuh, tma_plan): host code, run here with a stand-in for the one question it
asks of the device."""
import os
import subprocess

import pytest

from ml_framework_b200 import build as B

PROGRAM = r"""
#include "tma_gemm_kernel.cuh"
#include <chrono>
#include <cstdio>
#include <cstring>
using namespace seera;
static int failures = 0;
extern "C" cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
extern "C" cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *c) {
    static const int fit[9] = {0, 0, 74, 48, 36, 28, 22, 20, 16};
    *n = fit[c->attrs[0].val.clusterDim.x];
    return failures-- > 0 ? cudaErrorUnknown : cudaSuccess;
}
template <class F> double least_us(F f) {
    double least = 1e9;
    for (int k = 0; k < 40; k++) {
        const auto t = std::chrono::steady_clock::now();
        for (int j = 0; j < 50; j++) f();
        const double us = std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t).count() / 50;
        if (us < least) least = us;
    }
    return least;
}
int main(int, char **argv) {
    if (!strcmp(argv[1], "counts")) {
        for (int ksteps = 4; ksteps < 3000; ksteps++) {
            int next = 2;
            for (int parts = 2; parts <= ksteps; parts++) {
                const int per = (ksteps + parts - 1) / parts, used = (ksteps + per - 1) / per;
                if (used < parts) continue;                       // the same parts as with `used` of them
                if (next != parts) { printf("%d k-steps: %d after which %d\n", ksteps, parts, next); return 1; }
                next = tma_next_parts(ksteps, parts);
            }
            if (next) { printf("%d k-steps: %d at the end\n", ksteps, next); return 1; }
        }
    } else if (!strcmp(argv[1], "clusters")) {
        failures = 2;
        for (int k = 0; k < 4; k++) printf("%d ", clusters_at_once(4));
        printf("%d %d", clusters_at_once(8), clusters_at_once(4));
    } else if (!strcmp(argv[1], "cost")) {
        volatile unsigned long long by = 3;
        volatile unsigned long long out;
        const double division = least_us([&] { unsigned long long v = ~0ull; for (int k = 0; k < 32; k++) v = v / by + (~0ull >> 1); out = v; }) / 32;
        const int product[3][4] = {{576, 128, 131072, 1}, {576, 128, 25600, 3}, {1152, 256, 6400, 3}};
        for (auto &q : product) {
            TmaGemmParams p{};
            p.M = q[0]; p.N = q[1]; p.K = q[2]; p.a_mode = TMA_A_TAPS; p.b_mn = 1;
            printf("%f\n", least_us([&] { TmaGemmParams t = p; out = tma_plan(t, q[3], true).splits; }) / division);
        }
    }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cu").write_text(PROGRAM)
    subprocess.run([B.NVCC] + B.NVCC_FLAGS + [str(d / "plan.cu"), "-o", str(d / "plan"), "-L" + B.PKG, "-lseera_b200", "-lcudart", "-Xlinker",
                                              "-rpath=" + B.PKG], check=True, capture_output=True)
    return lambda *a: subprocess.run([str(d / "plan"), *a], capture_output=True, text=True, timeout=120)


def test_every_count_of_parts_that_differs_is_tried(program):
    r = program("counts")
    assert r.returncode == 0, r.stdout


def test_a_plan_costs_few_divisions(program):
    """In 64-bit divisions, one after the other: about 265, 185 and 55 of them, and 1790, 1320 and 390 when each width was estimated several
    times over every count."""
    cost = [float(v) for v in program("cost").stdout.split()]
    assert len(cost) == 3 and all(c < limit for c, limit in zip(cost, (600, 430, 130))), cost


def test_a_failed_query_for_clusters_is_asked_again(program):
    assert program("clusters").stdout.split() == ["0", "0", "36", "36", "16", "36"]
