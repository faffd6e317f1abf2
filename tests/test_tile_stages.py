"""The exchanges of csrc/hex27_tile.cuh on the CPU: the header's own code, compiled for the host with a
thread for each of the block's nine warps and its named barriers between them. The thread sanitizer
looks for words that one warp reads while another may write them, the address sanitizer for
accesses past the two buffers, and the results are compared with direct sums over the element's nodes
and points. (A word is [field][line][lane]: the 32 lanes of an access are neighbours, so no two meet
in a bank and one lane stands for all.)"""
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <barrier>
#include <cstdint>
#include <cstdio>
#include <thread>
#include <vector>
#define FEMB_D static inline
#define FEMB_HD static inline
#define __ldg(p) (*(p))
#define __shfl_sync(m, x, l) (x)
struct double2 { double x, y; };
struct float2 { float x, y; };
struct { unsigned x = 0; } threadIdx;
namespace femb { template <class T> T ld(const T* p) { return *p; } }
static std::barrier<> named[7] = {std::barrier<>(9), std::barrier<>(3), std::barrier<>(3), std::barrier<>(3),
                                  std::barrier<>(3), std::barrier<>(3), std::barrier<>(3)};
static void host_bar(int id) { named[id].arrive_and_wait(); }
HEADER
using namespace femb;
// one element: nodal values in, gradients at the points out; fluxes and a value density at the points
// in, nodal sums out
template <class T, int NC, bool WIDE>
void run(const std::vector<double>& in, std::vector<double>& out) {
    std::vector<T> S1(NC * 6 * 9 * HT_E), S2(NC * 9 * 9 * HT_E);
    const double *v = in.data(), *F = v + NC * 27, *W = F + NC * 81;
    std::vector<std::thread> warps;
    for (int w = 0; w < 9; ++w)
        warps.emplace_back([&, w] {
            const int a = w % 3, b = w / 3;
            for (int lane : {0, 13, 31}) {
                T x[NC][3], g[NC][3][3], f[NC][3][3], R[NC][3];
                for (int c = 0; c < NC; ++c)
                    for (int i = 0; i < 3; ++i) x[c][i] = (T)v[c * 27 + i + 3 * w];
                ht_gradient<T, NC>(x, S1.data(), S2.data(), a, b, lane, g);
                host_bar(0);   // the caller's barrier between the two contractions
                for (int c = 0; c < NC; ++c)
                    for (int d = 0; d < 3; ++d)
                        for (int q = 0; q < 3; ++q) f[c][d][q] = (T)F[(c * 3 + d) * 27 + w + 9 * q];
                ht_scatter_z<T, NC>(f, [&](int c, int q) { return (T)W[c * 27 + w + 9 * q]; }, S2.data(), a, b, lane);
                if (WIDE) host_bar(0);
                else ht_bar_a(a);
                ht_scatter_yx<T, NC>(S1.data(), S2.data(), a, b, lane, R);
                if (lane == 13)
                    for (int c = 0; c < NC; ++c)
                        for (int i = 0; i < 3; ++i) {
                            out[NC * 81 + c * 27 + i + 3 * w] = R[c][i];
                            for (int d = 0; d < 3; ++d) out[(c * 3 + d) * 27 + w + 9 * i] = g[c][d][i];
                        }
                host_bar(0);
            }
        });
    for (auto& t : warps) t.join();
}
template <int NC>
void both(const std::vector<double>& in) {
    std::vector<double> out(NC * 108);
    for (int k = 0; k < 4; ++k) {
        if (k == 0) run<double, NC, false>(in, out);
        if (k == 1) run<double, NC, true>(in, out);
        if (k == 2) run<float, NC, false>(in, out);
        if (k == 3) run<float, NC, true>(in, out);
        for (double x : out) printf("%.17g ", x);
        printf("\n");
    }
}
int main() {
    static_assert(HT_S1 == 3 * 6 * 9 * HT_E && HT_S2 == 3 * 9 * 9 * HT_E, "the kernels' buffers");
    int nc;
    if (scanf("%d", &nc) != 1) return 1;
    std::vector<double> in(nc * 135);
    for (double& x : in) if (scanf("%lf", &x) != 1) return 1;
    if (nc == 3) both<3>(in);
    else both<1>(in);
}
"""


@pytest.fixture(scope="module", params=["thread", "address,undefined"])
def program(request, tmp_path_factory):
    with open(os.path.join(ROOT, "femtools.jl_b200", "csrc", "hex27_tile.cuh")) as f:
        s = f.read()
    s = re.sub(r'#(pragma|include)[^\n]*', "", s)
    s, n = re.subn(r'asm volatile\("bar\.sync %0, 96;" ::"r"\((\d) \+ (\w)\) : "memory"\);', r"host_bar(\1 + \2);", s)
    assert n == 2 and "asm" not in s
    d = tmp_path_factory.mktemp("tile")
    src, exe = d / "tile.cpp", d / "tile"
    src.write_text("#include <type_traits>\n" + HARNESS.replace("HEADER", s))
    subprocess.check_call(["g++", "-std=c++20", "-O1", "-g", "-pthread", "-Wno-unused", "-fsanitize=" + request.param,
                           "-fno-sanitize-recover=all", str(src), "-o", str(exe)])
    return str(exe)


@pytest.mark.parametrize("nc", [1, 3])
def test_stages(program, nc):
    rng = np.random.default_rng(nc)
    v, F, W = rng.standard_normal((nc, 27)), rng.standard_normal((nc, 3, 27)), rng.standard_normal((nc, 27))
    r = subprocess.run([program], input=" ".join(repr(float(x)) for a in ([nc], v.ravel(), F.ravel(), W.ravel()) for x in a).replace(
        repr(float(nc)), str(nc), 1), capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    x = np.array([-np.sqrt(0.6), 0.0, np.sqrt(0.6)])
    L = np.stack([x * (x - 1) / 2, 1 - x * x, x * (x + 1) / 2], axis=1)      # [q][i]
    D = np.stack([x - 0.5, -2 * x, x + 0.5], axis=1)
    grid = lambda y: y.reshape(y.shape[:-1] + (3, 3, 3))                     # index i + 3j + 9k: [k][j][i]
    B = [(L, L, D), (L, D, L), (D, L, L)]                                    # (ζ, η, ξ) factors of ∂/∂ξ, ∂/∂η, ∂/∂ζ
    g = np.stack([np.einsum("zk,yj,xi,ckji->czyx", *B[d], grid(v)) for d in range(3)], axis=1)
    R = sum(np.einsum("zk,yj,xi,czyx->ckji", *B[d], grid(F[:, d])) for d in range(3))
    R = R + np.einsum("zk,yj,xi,czyx->ckji", L, L, L, grid(W))
    want = np.concatenate([g.ravel(), R.ravel()])
    rows = r.stdout.strip().split("\n")
    assert len(rows) == 4
    for k, row in enumerate(rows):
        got = np.array([float(y) for y in row.split()])
        # sums of at most 4·27 products of order one: 200 units in the last place of order ten
        assert np.abs(got - want).max() <= (200 * 2.0 ** -53 if k < 2 else 200 * 2.0 ** -24) * 10
