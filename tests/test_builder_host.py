"""The general tree builder's kernels run on the host, one thread after
another: leaf boxes, radix tree, boxes bottom-up, treelets, cost-optimal choice
and the collapse.  Whatever the boxes hold (NaN on one axis or all, numbers
whose centres overflow), every triangle comes out once and no index leaves its
array (AddressSanitizer)."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "kiraray_gb300" / "csrc"

SHIM = r"""
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#define __host__
#define __device__
#define __global__
#define __forceinline__ inline
#define __restrict__
#define __shared__ static
#define __launch_bounds__(...)
#define KRR_HD inline
struct float4 { float x, y, z, w; };
struct uint2 { uint32_t x, y; };
struct Index { int x = 0; } blockIdx, threadIdx, gridDim, blockDim;
inline float4 make_float4(float a, float b, float c, float d) { return {a, b, c, d}; }
inline uint2 make_uint2(uint32_t a, uint32_t b) { return {a, b}; }
inline uint32_t __float_as_uint(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
inline float __uint_as_float(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
inline int __clzll(uint64_t x) { return x ? __builtin_clzll(x) : 64; }
inline int __ffs(uint32_t x) { return __builtin_ffs((int)x); }
template <class T> T atomicAdd(T *p, T v) { T o = *p; *p += v; return o; }
template <class T> T atomicMax(T *p, T v) { T o = *p; *p = std::max(*p, v); return o; }
template <class T> T __ldcg(const T *p) { return *p; }
template <class T> void __stcg(T *p, T v) { *p = v; }
inline void __threadfence() {}
inline void __syncthreads() {}
using std::max;
using std::min;
"""

MAIN = r"""
#define RUN(m, call) for (blockIdx.x = 0; blockIdx.x < (m); ++blockIdx.x) call
static float unit() { return rand() / (float)RAND_MAX * 2 - 1; }
int main(int, char **argv) {
    const int kind = atoi(argv[1]);   // 0 numbers, 1 NaN, 2 NaN on one axis, 3 huge, 4 NaN alone
    blockDim.x = 1;
    for (int round = 0; round < 60; ++round) {
        const int n = 2 + rand() % (round % 2 ? 12 : 300);
        gridDim.x = n;
        std::vector<float> v(9 * n);
        for (int i = 0; i < n; ++i) {
            const float c[3] = {unit(), unit(), unit()};
            const bool odd = kind == 4 || rand() % 5 == 0;
            for (int k = 0; k < 9; ++k) {
                float x = c[k % 3] + 0.1f * unit();
                if (odd && (kind == 1 || kind == 4 || (kind == 2 && k % 3 == 1))) x = NAN;
                if (odd && kind == 3) x *= 3e38f;
                v[9 * i + k] = x;
            }
        }
        float b[12], mag = 0, ext = 0;
        for (int k = 0; k < 12; ++k) b[k] = k % 6 < 3 ? INFINITY : -INFINITY;
        for (int i = 0; i < n; ++i) {
            const V3 p = ld3(&v[9 * i]), q = ld3(&v[9 * i + 3]), r = ld3(&v[9 * i + 6]);
            const V3 lo = vmin(p, vmin(q, r)), hi = vmax(p, vmax(q, r)), ce = (lo + hi) * 0.5f;
            for (int k = 0; k < 3; ++k) {
                b[k] = fminf(b[k], get(ce, k)); b[3 + k] = fmaxf(b[3 + k], get(ce, k));
                b[6 + k] = fminf(b[6 + k], get(lo, k)); b[9 + k] = fmaxf(b[9 + k], get(hi, k));
            }
        }
        for (int k = 0; k < 3; ++k) {
            mag = std::max(mag, std::max(std::fabs(b[6 + k]), std::fabs(b[9 + k])));
            ext = std::max(ext, b[9 + k] - b[6 + k]);
        }
        std::vector<uint64_t> keys(n), sorted(n);
        std::vector<uint32_t> vals(n), idx(n);
        std::vector<float4> tlo(n), thi(n), llo(n), lhi(n);
        RUN(n, k_leaf_setup(v.data(), n, b, std::ldexp(mag + ext, -19) + 1e-30f, 1, keys.data(), vals.data(), tlo.data(),
                            thi.data()));
        std::vector<int> by(n);
        for (int i = 0; i < n; ++i) by[i] = i;
        std::stable_sort(by.begin(), by.end(), [&](int x, int y) { return keys[x] < keys[y]; });
        for (int i = 0; i < n; ++i) { sorted[i] = keys[by[i]]; idx[i] = vals[by[i]]; }
        RUN(n, k_gather_leaf_boxes(idx.data(), n, tlo.data(), thi.data(), llo.data(), lhi.data()));
        for (int variant = 0; variant < 4; ++variant) {   // one-triangle leaves, three, cost-optimal, treelets
            std::vector<uint32_t> left(n), right(n);
            std::vector<int> count(n), pint(n), pleaf(n), flags(n, 0);
            std::vector<float4> ilo(n), ihi(n), cost(2 * n);
            std::vector<uint2> choice(n);
            RUN(n - 1, k_karras(sorted.data(), n, left.data(), right.data(), count.data(), pint.data(), pleaf.data()));
            RUN(n, k_bottom_up(n, left.data(), right.data(), pint.data(), pleaf.data(), llo.data(), lhi.data(), ilo.data(),
                               ihi.data(), flags.data()));
            std::fill(flags.begin(), flags.end(), 0);
            if (variant == 3)
                RUN(n, k_treelet(n, left.data(), right.data(), count.data(), pint.data(), pleaf.data(), ilo.data(),
                                 ihi.data(), llo.data(), lhi.data(), flags.data(), 8));
            BinTree t{left.data(), right.data(), count.data(), ilo.data(), ihi.data(), llo.data(), lhi.data(), idx.data()};
            if (variant == 2) RUN(n, k_collapse_cost(n, t, pint.data(), pleaf.data(), cost.data(), choice.data(), flags.data()));
            for (int format = 0; format < 2; ++format) {
                const int leaf = variant == 1 ? 3 : 1;
                std::vector<float4> nodes((format ? 14 : 5) * (size_t)n);
                std::vector<uint32_t> order(n, 0xffffffffu);
                std::vector<CollapseItem> in(n), out(n);
                int n_nodes = 1, n_tris = 0, depth = 0, n_in = 1;
                in[0] = {0u, 0u, 1};
                while (n_in > 0) {
                    int n_out = 0;
                    RUN(n_in, k_collapse(t, in.data(), &n_in, out.data(), &n_out, nodes.data(), &n_nodes, order.data(),
                                         &n_tris, &depth, format, leaf, leaf, variant == 2 ? choice.data() : nullptr));
                    n_in = n_out;
                    in.swap(out);
                }
                std::sort(order.begin(), order.end());
                bool all = n_tris == n && n_nodes <= n;
                for (int i = 0; i < n; ++i) all = all && order[i] == (uint32_t)i;
                if (!all) { printf("round %d variant %d: %d of %d triangles\n", round, variant, n_tris, n); return 1; }
            }
        }
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def builder(tmp_path_factory):
    accel, kmath = (CSRC / "accel.cu").read_text(), (CSRC / "kmath.cuh").read_text()
    vectors = kmath[kmath.index("struct V3"):kmath.index("// Row-major 3x4")]
    kernels = accel[accel.index("__device__ __forceinline__ uint64_t spread21"):
                    accel.index("// ------------------------------------------------------------ small trees")]
    d = tmp_path_factory.mktemp("builder")
    (d / "main.cpp").write_text(SHIM + vectors + "constexpr uint32_t kLeafBit = 0x80000000u;\n"
                                "inline V3 ld3(const float *p) { return V3{p[0], p[1], p[2]}; }\n" + kernels + MAIN)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=address", "-w", str(d / "main.cpp"), "-o", str(d / "main")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return d / "main"


@pytest.mark.parametrize("kind", range(5))
def test_every_triangle_once(builder, kind):
    r = subprocess.run([str(builder), str(kind)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
