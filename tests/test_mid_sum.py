"""The step loops of the batched solver take v1 + v2, the sum a node's gradient
needs (cuda_get_Nodes_grad_R, graph_cuda_grad.hpp:65-84), from selection
networks (`mid_sum`, f2m_b200/csrc/f2m_device.cuh) instead of the reference's
compare chain.  This test compiles `mid_sum` for the host and compares it with
the chain, bit for bit, on lists without NaN (the solver keeps the chain for
those): ties, infinities (the padding of short lists), values at and above the
chain's 1e6 sentinels, first entry included."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
HEADER = os.path.join(os.path.dirname(HERE), "f2m_b200", "csrc", "f2m_device.cuh")

HARNESS = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__
#define __forceinline__ inline
%(code)s
static double chain(int n, const double* a) {
    double v0 = a[0], v1 = 1e6, v2 = 1e6;
    for (int i = 1; i < n; ++i) {
        const double v = a[i];
        if (v < v0) { v2 = v1; v1 = v0; v0 = v; continue; }
        if (v < v1) { v2 = v1; v1 = v; continue; }
        if (v < v2) { v2 = v; continue; }
    }
    return v1 + v2;
}
template <int K>
static long long check() {
    std::mt19937_64 rng(5 + K);
    std::uniform_real_distribution<double> U(0, 1);
    const double sp[] = {0.0, 1e6, -1e6, 1e6 + 1, 999999.5, INFINITY, 0.5, 0.5, -3.25, 2e6};
    long long bad = 0;
    double a[K];
    for (int it = 0; it < 200000; ++it) {
        const int n = 1 + (int)(U(rng) * K), mode = it %% 4;
        for (int k = 0; k < K; ++k) {
            if (mode == 0) a[k] = (U(rng) - 0.5) * 20;
            else if (mode == 1) a[k] = (double)(int)(U(rng) * 6) - 2;
            else if (mode == 2) a[k] = sp[(int)(U(rng) * 10)];
            else a[k] = (U(rng) < 0.2) ? sp[(int)(U(rng) * 10)] : (U(rng) - 0.3) * 4e6;
            if (it %% 3 == 0 && k >= n) a[k] = INFINITY;
        }
        const double r = chain(K, a), g = mid_sum<K>(a);
        if (std::memcmp(&r, &g, 8) != 0 && !(r == 0 && g == 0)) ++bad;
    }
    return bad;
}
int main() {
    const long long bad = check<3>() + check<4>() + check<5>() + check<6>() + check<8>();
    std::printf("mismatches %%lld\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_mid_sum_matches_the_reference_chain(tmp_path):
    text = open(HEADER).read()
    m = re.search(r"__device__ __forceinline__ void mid_of3\(.*?(?=// Magnitudes at which)", text, re.S)
    assert m, "mid_of3 .. mid_sum not found"
    src, exe = tmp_path / "mid.cpp", tmp_path / "mid"
    src.write_text(HARNESS % {"code": m.group(0).replace("#pragma unroll\n", "")})
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "mismatches 0" in r.stdout
