// Fused neural-radiance-cache forward pass on the 5th-generation tensor
// cores (tcgen05), one CTA per SM.
//
// Encoder warps encode the queries (hash grid, trilinear) into 128x64 BF16
// activation tiles in shared memory while two groups of four MLP warps run
// the tiles before them: for each layer one elected thread issues four
// tcgen05.mma.kind::f16 (M=128, N=64 or 16, K=16, BF16 x BF16 -> FP32 in
// tensor memory), commits them to an mbarrier, and the group's 128 threads
// read the accumulator rows back with tcgen05.ld, apply ReLU, round to BF16
// and write the next activation tile (or the RGB output).  All weights
// (43 KB, BF16) stay resident in shared memory for the CTA's lifetime.
// Waits on mbarriers are bounded: a wait that gives up sets an error flag,
// and the CTA finishes without further tensor-core work and frees its tensor
// memory.
//
// Shared-memory operands use the canonical K-major layout without swizzle:
// 8x8-element core matrices of 128 contiguous bytes, core (i, j) of a tile
// with 64 columns at byte ((i * 8) + j) * 128, so the leading-dimension
// byte offset (next core along K) is 128 and the stride-dimension byte
// offset (next 8-row group) is 1024.
#include <algorithm>

#include "nrc.h"

namespace krr {

constexpr int kTcRows = 128;
constexpr int kLayerBytes = kNrcWidth * kNrcIn * 2;     // 8 KB
constexpr int kOutBytes = kNrcOutPad * kNrcIn * 2;      // 2 KB
constexpr uint32_t kWaitLimit = 1u << 26;

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor (tcgen05): start address, leading and
// stride byte offsets (all >> 4), descriptor version 1 at bit 46, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo & 0x3FFFFu) >> 4) << 16) |
           ((uint64_t)((sbo & 0x3FFFFu) >> 4) << 32) | (1ull << 46);
}

// Instruction descriptor, kind::f16: FP32 accumulator (bits 4-5 = 1), A and
// B BF16 (bits 7-9 and 10-12 = 1), K-major, N >> 3 at bit 17, M >> 4
// at bit 24; with `a_mn` or `b_mn` (bits 15, 16) that operand lies in shared
// memory with its M or N index contiguous instead of its K index.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n, uint32_t a_mn = 0u, uint32_t b_mn = 0u) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn << 15) | (b_mn << 16) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void tc_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}

__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t mbar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    return ok;
}

__device__ __forceinline__ void fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
        "%11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Byte offset of element (r, k) in a canonical K-major tile of 64 columns.
__host__ __device__ __forceinline__ uint32_t canon(uint32_t r, uint32_t k) {
    return (((r >> 3) * 8u + (k >> 3)) * 128u) + (r & 7u) * 16u + (k & 7u) * 2u;
}

// Packs the BF16 weights [layer][out][64] into canonical tiles.
__global__ void k_pack_weights(const __nv_bfloat16 *__restrict__ w, NrcMlp mlp, uint8_t *packed) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < mlp.n_params; e += gridDim.x * blockDim.x)
        *reinterpret_cast<__nv_bfloat16 *>(packed + nrc_packed_offset(e, mlp.layers)) = w[e];
}

// Hash-grid encoding of 16 query rows by one warp, two lanes per row: lane p
// of a pair gathers the four corners at x offset p of four levels, then the
// lanes swap halves, so that each interpolates two levels from all eight
// corners and stores their four features.  The two x neighbours of a corner
// pair lie next to each other in the table (a hashed index is x ^ (a function
// of y and z), a dense one x + (the same)), in one 32-byte sector seven times
// in eight, so a pair's two loads, issued by one instruction, share an L1
// request.  Per level the corner weights and the accumulation order are those
// of the CUDA-core encoder (nrc.cu).
constexpr int kEncGroup = 4;

struct EncInput {
    float pos[3], dir[3], mat[3];   // dir: normal (lane 0) or outgoing direction (lane 1); mat: roughness or albedo
};

__device__ __forceinline__ EncInput load_input(const float *q, int p) {
    EncInput x;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        x.pos[a] = q[a];
        x.dir[a] = q[(p ? 10 : 3) + a];
    }
    x.mat[0] = q[p ? 7 : 6];
    x.mat[1] = p ? q[8] : 0.f;
    x.mat[2] = p ? q[9] : 0.f;
    return x;
}

__device__ __forceinline__ uint32_t bf16x2(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&v);
}

// The lane's four corners (y, z) = 00, 10, 01, 11 of levels l0..l0+3; a level
// at or beyond g.levels reads entry 0 and is discarded.
__device__ __forceinline__ void gather_levels(const NrcGrid &g, const float *pos, const __nv_bfloat16 *__restrict__ table,
                                              int l0, uint32_t p, uint32_t (&v)[kEncGroup][4]) {
#pragma unroll
    for (int j = 0; j < kEncGroup; ++j) {
        const int l = (l0 + j) & (kNrcMaxLevels - 1);
        const bool valid = l0 + j < g.levels;
        const char *level = reinterpret_cast<const char *>(table) + 4 * (size_t)(valid ? g.offset[l] : 0u);
        const float res = (float)g.res[l], top = (float)(g.res[l] - 1);
        uint32_t c[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) c[a] = (uint32_t)fminf(fmaxf(floorf(pos[a] * res), 0.f), top);
        // byte offsets: the factor 4 goes into the multipliers and the mask
        const uint32_t x = 4u * (c[0] + p);
        uint32_t off[4];
        if (g.dense_mask & (1u << l)) {
            const uint32_t n1 = 4u * ((uint32_t)g.res[l] + 1u), n2 = n1 * ((uint32_t)g.res[l] + 1u);
            off[0] = x + c[1] * n1 + c[2] * n2;
            off[1] = off[0] + n1;
            off[2] = off[0] + n2;
            off[3] = off[1] + n2;
        } else {
            const uint32_t mask = valid ? 4u * (g.table_size - 1u) : 0u;
            const uint32_t y0 = c[1] * (4u * 2654435761u), z0 = c[2] * (4u * 805459861u);
            const uint32_t y1 = y0 + 4u * 2654435761u, z1 = z0 + 4u * 805459861u;
            off[0] = (x ^ y0 ^ z0) & mask;
            off[1] = (x ^ y1 ^ z0) & mask;
            off[2] = (x ^ y0 ^ z1) & mask;
            off[3] = (x ^ y1 ^ z1) & mask;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) v[j][k] = __ldg(reinterpret_cast<const uint32_t *>(level + off[k]));
    }
}

// Row r of the tile; p: the lane's place in the row's pair.  Warp-collective.
__device__ __forceinline__ void encode_row(const NrcGrid &g, const EncInput &in,
                                           const __nv_bfloat16 *__restrict__ table, uint8_t *tile, uint32_t r,
                                           uint32_t p) {
    float pos[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) pos[a] = fminf(fmaxf((in.pos[a] - g.lo[a]) * g.inv_extent[a], 0.f), 1.f);
#pragma unroll 1
    for (int l0 = 0; l0 < g.levels; l0 += kEncGroup) {
        uint32_t v[kEncGroup][4];
        gather_levels(g, pos, table, l0, p, v);
        // lane 0 keeps levels l0, l0+1 and takes their x + 1 corners, lane 1
        // keeps l0+2, l0+3 and takes their x corners
        const int first = l0 + 2 * (int)p;
        uint32_t f[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            uint32_t c[8];   // corner k at bits x | y << 1 | z << 2
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t mine = p ? v[j + 2][k] : v[j][k], other = p ? v[j][k] : v[j + 2][k];
                const uint32_t got = __shfl_xor_sync(0xffffffffu, other, 1);
                c[2 * k] = p ? got : mine;
                c[2 * k + 1] = p ? mine : got;
            }
            const int l = (l0 + j) & (kNrcMaxLevels - 1), l2 = (l0 + j + 2) & (kNrcMaxLevels - 1);
            const float res = (float)(p ? g.res[l2] : g.res[l]), top = (float)((p ? g.res[l2] : g.res[l]) - 1);
            float fr[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float s = pos[a] * res;
                fr[a] = __saturatef(s - fminf(fmaxf(floorf(s), 0.f), top));
            }
            float f0 = 0.f, f1 = 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float w = ((k & 1) ? fr[0] : 1.f - fr[0]) * (((k >> 1) & 1) ? fr[1] : 1.f - fr[1]) *
                                (((k >> 2) & 1) ? fr[2] : 1.f - fr[2]);
                f0 += w * __uint_as_float(c[k] << 16);
                f1 += w * __uint_as_float(c[k] & 0xffff0000u);
            }
            f[j] = bf16x2(f0, f1);
        }
        uint8_t *dst = tile + canon(r, 2u * (uint32_t)first);
        if (first + 2 <= g.levels) *reinterpret_cast<uint2 *>(dst) = make_uint2(f[0], f[1]);
        else if (first < g.levels) *reinterpret_cast<uint32_t *>(dst) = f[0];
    }
    // the other inputs, as nrc_encode_extras: lane 0 the normal and the
    // roughness, lane 1 the outgoing direction and the albedo; zeros behind
    const uint32_t o = 2u * (uint32_t)g.levels;
    auto put = [&](uint32_t k, float a, float b) {
        *reinterpret_cast<uint32_t *>(tile + canon(r, k)) = bf16x2(a, b);
    };
    float t, u, e[kNrcBlobBins];
    nrc_spherical(in.dir[0], in.dir[1], in.dir[2], t, u);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        nrc_one_blob(k ? u : t, e);
        put(o + 8u * p + 4u * k, e[0], e[1]);
        put(o + 8u * p + 4u * k + 2u, e[2], e[3]);
    }
    if (p == 0) {
        nrc_one_blob(1.f - expf(-in.mat[0]), e);
        put(o + 16u, e[0], e[1]);
        put(o + 18u, e[2], e[3]);
    } else {
        put(o + 20u, in.mat[0], in.mat[1]);
        put(o + 22u, in.mat[2], 0.f);
    }
    for (uint32_t k = o + 24u + 2u * p; k < (uint32_t)kNrcIn; k += 4u) put(k, 0.f, 0.f);
}

// Named barrier of n threads; true for all of them if `flag` is for one.
__device__ __forceinline__ bool bar_or(int id, int n, bool flag) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %3, 0;\n\tbar.red.or.pred p, %1, %2, q;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(r)
        : "r"(id), "r"(n), "r"((uint32_t)flag)
        : "memory");
    return r != 0u;
}

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

// Bounded wait of a whole warp, one outcome for its lanes.
__device__ __forceinline__ bool warp_wait(uint32_t mbar, uint32_t parity) {
    uint32_t spins = 0, ok = 0;
    while (!(ok = mbar_try_wait(mbar, parity)) && ++spins < kWaitLimit) {
    }
    return __all_sync(0xffffffffu, ok);
}

// One CTA of 32 warps per SM: 8 MLP warps in two groups (tensor-memory lanes
// 0-127 each, 64 columns apart) and 24 encoder warps, with kTileBuffers
// activation tiles between them.  64 registers a thread; the weights and the
// tiles take 122 KB of shared memory (five hidden layers), which leaves half
// of the SM's L1 to the table.
constexpr int kMlpGroups = 2, kEncWarps = 24, kTileBuffers = 5;
constexpr int kTileBytes = kTcRows * kNrcIn * 2;
constexpr int kUnitsPerTile = kTcRows / 16;   // an encoder warp's unit of work: 16 rows
constexpr int kFwThreads = kMlpGroups * kTcRows + 32 * kEncWarps;
constexpr uint32_t kFwCols = 64u * kMlpGroups;

// out[i * out_stride + 0..3) for i < *count (or cap); optional per-layer
// activation dump (bf16 [layers][cap][64], row-major) for the training
// backward pass.
//
// Warp-specialised: the encoder warps fill tiles of 128 rows (the hash-grid
// gathers), 16 rows at a time, while each MLP group runs the layers of every
// second tile (one thread issues the MMAs, all 128 read the accumulator rows
// back, apply ReLU and write the next layer's input in place).  Tiles are
// handed over by mbarriers: full (eight 16-row units encoded) and empty (the
// group's four warps are done).
//
// An SM takes one L1 miss per clock (296 G/s over the chip with the table in
// L2, whatever the loads' kind and the warps in flight), and a query misses
// about 50 times: 0.26 ms for 1.5M queries.  Those take 397 us; 824 us with
// one lane per row, four encoder warps and a CTA-wide handover (two CTAs of
// 8 warps), 618 us with two lanes per row and two CTAs of 8 encoder warps:
// then the loads' latency was the limit, and 24 encoder warps on 64 registers
// hide it better than deeper batches of loads in 16.
// Waits are bounded: a group (or an encoder warp) whose wait gives up raises
// an error flag and leaves, as do in turn those that wait for it.
__global__ void __launch_bounds__(kFwThreads, 1)
k_nrc_forward_tc(NrcGrid g, int layers, const float *__restrict__ in, const int32_t *d_count,
                 int64_t cap, const __nv_bfloat16 *__restrict__ table,
                 const uint8_t *__restrict__ packed_w, float *__restrict__ out, int out_stride,
                 __nv_bfloat16 *__restrict__ acts, uint32_t *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *sw = smem;                                              // weights
    uint8_t *tiles_s = smem + (layers - 1) * kLayerBytes + kOutBytes;   // activation tiles
    tiles_s = reinterpret_cast<uint8_t *>(((uintptr_t)tiles_s + 1023) & ~(uintptr_t)1023);
    uint64_t *mbars = reinterpret_cast<uint64_t *>(tiles_s + kTileBuffers * kTileBytes);
    const uint32_t full0 = smem_u32(mbars), empty0 = full0 + 8 * kTileBuffers,
                   acc0 = empty0 + 8 * kTileBuffers;   // acc: a group's accumulator is complete
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mbars + 2 * kTileBuffers + kMlpGroups);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // weights -> shared memory (16-byte copies)
    int wbytes = (layers - 1) * kLayerBytes + kOutBytes;
    for (int e = tid; e < wbytes / 16; e += blockDim.x)
        reinterpret_cast<uint4 *>(sw)[e] = reinterpret_cast<const uint4 *>(packed_w)[e];
    fence_proxy_async();   // the tensor cores read the weights through the async proxy
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(kFwCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int b = 0; b < kTileBuffers; ++b) {
            mbar_init(full0 + 8 * b, kUnitsPerTile);
            mbar_init(empty0 + 8 * b, kTcRows / 32);
        }
        for (int m = 0; m < kMlpGroups; ++m) mbar_init(acc0 + 8 * m, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    const int64_t n = d_count ? min((int64_t)*d_count, cap) : cap;
    const int64_t tiles = (n + kTcRows - 1) / kTcRows;
    // the CTA's k-th tile is tile blockIdx.x + k gridDim.x, in buffer
    // k % kTileBuffers; a buffer's k / kTileBuffers-th use flips the parity
    if (warp >= 4 * kMlpGroups) {
        // encoders: a warp's rows are 16 of each third tile (rows past the
        // last are encoded as the last: their results are never stored)
        const int e = warp - 4 * kMlpGroups;
        const uint32_t r = (uint32_t)((e % kUnitsPerTile) * 16 + (lane >> 1)), p = (uint32_t)lane & 1u;
        for (int k = e / kUnitsPerTile;; k += kEncWarps / kUnitsPerTile) {
            const int64_t t = blockIdx.x + (int64_t)k * gridDim.x;
            if (t >= tiles) break;
            const int64_t row = min(t * kTcRows + r, n - 1);
            const EncInput x = load_input(in + kNrcInputs * row, (int)p);
            const int b = k % kTileBuffers;
            if (!warp_wait(empty0 + 8 * b, (uint32_t)(k / kTileBuffers + 1) & 1u)) {
                if (lane == 0) atomicOr(err, (uint32_t)kErrLoopLimit);
                break;
            }
            encode_row(g, x, table, tiles_s + b * kTileBytes, r, p);
            fence_proxy_async();   // the tensor cores read the tile through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(full0 + 8 * b);
        }
    } else {
        const int m = warp >> 2, row_t = tid & (kTcRows - 1);
        const uint32_t acc = acc0 + 8 * m, d_cols = tmem + 64u * m;
        const uint32_t my_lane_addr = d_cols + ((uint32_t)((warp & 3) * 32) << 16);
        uint32_t phase = 0;
        bool failed = false;
        for (int k = m; !failed; k += kMlpGroups) {
            const int64_t t = blockIdx.x + (int64_t)k * gridDim.x;
            if (t >= tiles) break;
            const int b = k % kTileBuffers;
            uint8_t *sa = tiles_s + b * kTileBytes;
            failed = !warp_wait(full0 + 8 * b, (uint32_t)(k / kTileBuffers) & 1u);
            const int64_t row = t * kTcRows + row_t;
            for (int l = 0; l < layers; ++l) {
                const bool last = l + 1 == layers;
                if (row_t == 0 && !failed) {
                    fence_after_sync();
                    const uint32_t a0 = smem_u32(sa), b0 = smem_u32(sw + l * kLayerBytes);
                    const uint32_t idesc = idesc_bf16(kTcRows, last ? kNrcOutPad : kNrcWidth);
#pragma unroll
                    for (int kk = 0; kk < kNrcIn / 16; ++kk)
                        tc_mma(d_cols, smem_desc(a0 + 256u * kk, 128u, 1024u),
                               smem_desc(b0 + 256u * kk, 128u, 1024u), idesc, kk > 0 ? 1u : 0u);
                    tc_commit(acc);
                }
                __syncwarp();
                // the tile holds this layer's input X_l: the warp dumps its
                // own 32 rows for the backward pass while the MMAs read them
                // (it alone overwrites these rows, below)
                if (acts) {
                    __nv_bfloat16 *dst = acts + (size_t)l * cap * kNrcIn;
                    for (int c = lane; c < 32 * 8; c += 32) {
                        const int rr = (warp & 3) * 32 + (c >> 3), j = c & 7;
                        if (t * kTcRows + rr < n)
                            reinterpret_cast<uint4 *>(dst + (t * kTcRows + rr) * kNrcIn)[j] =
                                *reinterpret_cast<const uint4 *>(sa + canon((uint32_t)rr, (uint32_t)(8 * j)));
                    }
                    __syncwarp();
                }
                if (!failed) failed = !warp_wait(acc, phase);
                phase ^= 1u;
                if (!failed) {
                    fence_after_sync();
                    if (!last) {
#pragma unroll
                        for (int h = 0; h < 4; ++h) {   // 16 columns at a time
                            float v[16];
                            tmem_ld16(my_lane_addr + 16 * h, v);
                            tmem_wait_ld();
#pragma unroll
                            for (int q = 0; q < 16; ++q) v[q] = fmaxf(v[q], 0.f);
#pragma unroll
                            for (int j = 0; j < 2; ++j)
                                *reinterpret_cast<uint4 *>(sa + canon((uint32_t)row_t, 16u * h + 8u * j)) =
                                    make_uint4(bf16x2(v[8 * j], v[8 * j + 1]), bf16x2(v[8 * j + 2], v[8 * j + 3]),
                                               bf16x2(v[8 * j + 4], v[8 * j + 5]), bf16x2(v[8 * j + 6], v[8 * j + 7]));
                        }
                        fence_proxy_async();
                    } else {
                        float v[16];
                        tmem_ld16(my_lane_addr, v);
                        tmem_wait_ld();
                        if (row < n) {
                            out[row * out_stride + 0] = v[0];
                            out[row * out_stride + 1] = v[1];
                            out[row * out_stride + 2] = v[2];
                        }
                    }
                }
                fence_before_sync();
                failed = bar_or(1 + m, kTcRows, failed);   // one outcome for the group
            }
            if (lane == 0) mbar_arrive(empty0 + 8 * b);
        }
        if (failed && lane == 0) atomicOr(err, (uint32_t)kErrLoopLimit);
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kFwCols));
}

// ------------------------------------------------------------------ backward
//
// Per 128-row tile, from the output layer down: dX_l = dY_l . W_l (M=128,
// N=64, K=64 or 16) and dW_l += dY_l^T . X_l (M=128 of which 64 rows are
// read, N=64, K=128 rows of the tile).  The dX accumulator (64 columns) is
// read back each layer, masked by ReLU'(X_l), rounded to BF16 and becomes the
// next layer's dY tile; the dW_l accumulators (64 columns each) stay in
// tensor memory for all of the CTA's tiles and are added to the FP32 gradient
// once at the end.  Operand rounding points match the CUDA-core kernels: dY,
// W and X in BF16, FP32 accumulation.
//
// A tile [row][col] in canonical cores serves both products: K-major for dX
// (K = col; next core along K 128 bytes on, next 8 rows 1024), and M- or
// N-major for dW, where K is the row: then the stride offset (next 8 columns)
// is 128 and the leading offset (next 8 rows) 1024, and likewise W_l [out]
// [in] is the N-major B operand of dX, so nothing is transposed.  The M=128
// product over a 64-column tile reads its rows 64-127 from the cores that
// follow; those accumulator rows are never read.
//
// The chain of a layer (MMA, accumulator read, next dY tile, barrier) bounds
// the kernel, one CTA per SM by the tensor memory.  Tiles X_l arrive by
// cp.async two layers ahead, dX_l is issued before dW_l and waited for
// alone (dW_l runs under the epilogue), and the loss gradient is computed
// here.  65,536 rows, five hidden layers on GB300: 46 us; 101 us with
// element-wise transposed copies of dY and X and one wait per layer, and 9 us
// for the loss.

constexpr uint32_t kBwCols = 512;
constexpr int kBwThreads = 256;             // warps 0-3: columns 0-31 of the accumulator, 4-7: 32-63
constexpr int kBwXBuffers = 3;
constexpr int kA16Bytes = kTcRows * kNrcOutPad * 2;   // dY of the output layer, 4 KB

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

__global__ void __launch_bounds__(kBwThreads, 1)
k_nrc_backward_tc(int layers, int dx_cols, const float *__restrict__ y_out, const float *__restrict__ targets,
                  float loss_scale, const __nv_bfloat16 *__restrict__ acts, const int32_t *d_count, int64_t cap,
                  const uint8_t *__restrict__ packed_w, float *__restrict__ dx0, float *__restrict__ dw,
                  float *loss, NrcMlp mlp, uint32_t *err) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int w_bytes = (layers - 1) * kLayerBytes + kOutBytes;
    uint8_t *sw = smem;
    uint8_t *dy_s = smem + ((w_bytes + 1023) & ~1023);   // dY_l, two tiles
    uint8_t *x_s = dy_s + 2 * kTileBytes;                // X_l, kBwXBuffers tiles
    uint8_t *a16 = x_s + kBwXBuffers * kTileBytes;       // dY of the output layer, [128][16]; 2 KB behind it
    uint64_t *mbar = reinterpret_cast<uint64_t *>(a16 + kA16Bytes + 2048);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mbar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t acc = smem_u32(mbar);

    const int64_t n = d_count ? min((int64_t)*d_count, cap) : cap;
    const int64_t tiles = (n + kTcRows - 1) / kTcRows;
    // The CTA's steps: the layers of tile blockIdx.x, then of the next tile
    // gridDim.x on, and so on.  fetch() brings the X of the step after the
    // last it brought into the next buffer (pairs of lanes take a 32-byte
    // sector), nothing past the last step.
    int64_t f_tile = blockIdx.x;
    int f_layer = layers - 1, f_buf = 0;
    auto fetch = [&]() {
        if (f_tile < tiles) {
            const uint32_t dst = smem_u32(x_s + f_buf * kTileBytes);
            const __nv_bfloat16 *src = acts + (size_t)f_layer * cap * kNrcIn;
            for (int c = warp; c < 32; c += kBwThreads / 32) {
                const uint32_t r = (uint32_t)((c & 7) * 16 + (lane >> 1)), j = (uint32_t)(2 * (c >> 3) + (lane & 1));
                const int64_t row = f_tile * kTcRows + r;
                cp_async16(dst + canon(r, 8u * j), src + min(row, n - 1) * kNrcIn + 8 * j, row < n ? 16u : 0u);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        f_buf = f_buf + 1 == kBwXBuffers ? 0 : f_buf + 1;
        if (f_layer-- == 0) {
            f_layer = layers - 1;
            f_tile += gridDim.x;
        }
    };
    fetch();
    fetch();
    for (int e = tid; e < w_bytes / 16; e += blockDim.x)
        reinterpret_cast<uint4 *>(sw)[e] = reinterpret_cast<const uint4 *>(packed_w)[e];
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(kBwCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        mbar_init(acc, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    const uint32_t my_lanes = (uint32_t)((warp & 3) * 32) << 16, col0 = (uint32_t)(warp >> 2) * 32u;
    const uint32_t r = (uint32_t)(tid & (kTcRows - 1));

    const float inv = 1.f / (float)(max(n, (int64_t)1) * 3);
    float lsum = 0.f;
    uint32_t phase = 0;
    bool failed = false;
    int l = layers - 1, x_buf = 0, dy_buf = 0;   // of this step
    bool first_tile = true;
    for (int64_t t = blockIdx.x; t < tiles;) {
        const bool out_layer = l == layers - 1;
        const int64_t row = t * kTcRows + r;
        if (out_layer && tid < kTcRows) {
            // relative L2 loss and its gradient, as k_loss
            float d[3] = {0.f, 0.f, 0.f};
            if (row < n)
                for (int c = 0; c < 3; ++c) {
                    const float y = y_out[row * kNrcOutPad + c], tg = targets[3 * row + c];
                    const float den = y * y + 0.01f;
                    lsum += (y - tg) * (y - tg) / den;
                    d[c] = 2.f * (y - tg) / den * inv * loss_scale;
                }
            uint8_t *dst = a16 + (r >> 3) * 256u + (r & 7u) * 16u;
            *reinterpret_cast<uint4 *>(dst) = make_uint4(bf16x2(d[0], d[1]), bf16x2(d[2], 0.f), 0u, 0u);
            *reinterpret_cast<uint4 *>(dst + 128) = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");   // this step's X is here, the next one's may be on its way
        fence_proxy_async();
        fence_before_sync();
        failed = __syncthreads_or(failed);
        if (failed) break;
        const uint8_t *x = x_s + x_buf * kTileBytes;
        if (tid == 0) {
            fence_after_sync();
            const uint32_t dy = smem_u32(out_layer ? a16 : dy_s + dy_buf * kTileBytes), xs = smem_u32(x);
            const uint32_t w = smem_u32(sw + l * kLayerBytes);
            const uint32_t dy_rows = out_layer ? 256u : 1024u;   // next 8 rows of the dY tile
            // dX = dY_l . W_l (K = 16 for the output layer, 64 otherwise)
            for (int kk = 0; kk < (out_layer ? 1 : 4); ++kk)
                tc_mma(tmem, smem_desc(dy + 256u * kk, 128u, dy_rows), smem_desc(w + 2048u * kk, 1024u, 128u),
                       idesc_bf16(kTcRows, 64, 0u, 1u), kk > 0 ? 1u : 0u);
            tc_commit(acc);   // completes after the step before's dW too
            // dW_l += dY_l^T . X_l (K = the tile's 128 rows)
            const uint32_t dcol = tmem + 64u + 64u * (uint32_t)l;
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
                tc_mma(dcol, smem_desc(dy + 2u * dy_rows * kk, dy_rows, 128u),
                       smem_desc(xs + 2048u * kk, 1024u, 128u), idesc_bf16(kTcRows, 64, 1u, 1u),
                       (!first_tile || kk > 0) ? 1u : 0u);
        }
        __syncwarp();
        failed = !warp_wait(acc, phase);
        phase ^= 1u;
        if (!failed) fence_after_sync();
        fetch();   // into the buffer of the step before, whose dW has completed
        if (!failed && (l > 0 || (int)col0 < dx_cols)) {
            float v[32];
            tmem_ld16(tmem + my_lanes + col0, v);
            tmem_ld16(tmem + my_lanes + col0 + 16, v + 16);
            tmem_wait_ld();
            if (l > 0) {
                uint8_t *dst = dy_s + (dy_buf ^ 1) * kTileBytes;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint4 h = *reinterpret_cast<const uint4 *>(x + canon(r, col0 + 8u * j));
                    const uint32_t hw[4] = {h.x, h.y, h.z, h.w};
                    uint32_t o[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {   // X > 0, of either half
                        const float a = __uint_as_float(hw[i] << 16) > 0.f ? v[8 * j + 2 * i] : 0.f;
                        const float b = __uint_as_float(hw[i] & 0xffff0000u) > 0.f ? v[8 * j + 2 * i + 1] : 0.f;
                        o[i] = bf16x2(a, b);
                    }
                    *reinterpret_cast<uint4 *>(dst + canon(r, col0 + 8u * j)) = make_uint4(o[0], o[1], o[2], o[3]);
                }
            } else if (row < n) {
                float4 *dst = reinterpret_cast<float4 *>(dx0 + row * kNrcIn + col0);
                for (int k = 0; k < 8; ++k)
                    if ((int)col0 + 4 * k < dx_cols)
                        dst[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
            }
        }
        fence_before_sync();
        x_buf = x_buf + 1 == kBwXBuffers ? 0 : x_buf + 1;
        dy_buf ^= 1;
        if (l-- == 0) {
            l = layers - 1;
            t += gridDim.x;
            first_tile = false;
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!failed && blockIdx.x < tiles) {
        // the last dW, then the accumulators' rows 0..63 (out features) in
        // the lanes of warps 0-1 and 4-5
        if (tid == 0) tc_commit(acc);
        __syncwarp();
        failed = !warp_wait(acc, phase);
        if (!failed && (warp & 3) < 2) {
            fence_after_sync();
            for (int k = 0; k < layers; ++k) {
                const int rows = k + 1 == layers ? kNrcOutPad : kNrcWidth;
                float v[32];
                const uint32_t base = tmem + my_lanes + 64u + 64u * (uint32_t)k + col0;
                tmem_ld16(base, v);
                tmem_ld16(base + 16, v + 16);
                tmem_wait_ld();
                if ((int)r < rows) {   // 16-byte vector atomics (the row offsets are multiples of 64 floats)
                    float4 *dst = reinterpret_cast<float4 *>(dw + mlp.w_offset[k] + (size_t)r * kNrcIn + col0);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        atomicAdd(dst + i, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
                }
            }
        }
        for (int off = 16; off > 0; off >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
        if (lane == 0 && tid < kTcRows) atomicAdd(loss, lsum * inv);
    }
    if (failed && lane == 0) atomicOr(err, (uint32_t)kErrLoopLimit);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kBwCols));
}

}  // namespace

size_t nrc_tc_smem_bytes(int layers) {
    size_t w = (size_t)(layers - 1) * kLayerBytes + kOutBytes;
    size_t a = ((w + 1023) & ~(size_t)1023) + kTileBuffers * kTileBytes;
    return a + 128 + 1024;   // mbarriers, tensor-memory slot, alignment slack
}

int nrc_pack_weights(const __nv_bfloat16 *w, const NrcMlp &mlp, uint8_t *packed, cudaStream_t s) {
    cudaMemsetAsync(packed, 0, (size_t)(mlp.layers - 1) * kLayerBytes + kOutBytes, s);
    k_pack_weights<<<64, 256, 0, s>>>(w, mlp, packed);
    KRR_CUDA(cudaGetLastError());
    return KRR_OK;
}

size_t nrc_tc_bwd_smem_bytes(int layers) {
    size_t w = (size_t)(layers - 1) * kLayerBytes + kOutBytes;
    return ((w + 1023) & ~(size_t)1023) + (2 + kBwXBuffers) * kTileBytes + kA16Bytes + 2048 + 64 + 1024;
}

int nrc_backward_tc(const NrcMlp &mlp, int dx_cols, const float *d_out, const float *d_targets, float loss_scale,
                    const __nv_bfloat16 *acts, const int32_t *d_count, int64_t cap, const uint8_t *packed,
                    float *d_dx0, float *d_dw, float *d_loss, uint32_t *err, cudaStream_t s) {
    const size_t smem = nrc_tc_bwd_smem_bytes(mlp.layers);
    static OncePerDevice allowed;   // for the deepest network, whatever this one's depth
    KRR_CUDA(allow_shared(allowed, k_nrc_backward_tc, nrc_tc_bwd_smem_bytes(kNrcTcBwdLayers)));
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int64_t tiles = (cap + kTcRows - 1) / kTcRows;
    int grid = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)sms));
    k_nrc_backward_tc<<<grid, kBwThreads, smem, s>>>(mlp.layers, dx_cols, d_out, d_targets, loss_scale, acts,
                                                     d_count, cap, packed, d_dx0, d_dw, d_loss, mlp, err);
    KRR_CUDA(cudaGetLastError());
    return KRR_OK;
}

int nrc_forward_tc(const NrcGrid &g, const NrcMlp &mlp, const float *d_in, const int32_t *d_count,
                   int64_t cap, const __nv_bfloat16 *table, const uint8_t *packed, float *d_out, int out_stride,
                   __nv_bfloat16 *acts, uint32_t *err, cudaStream_t s) {
    const size_t smem = nrc_tc_smem_bytes(mlp.layers);
    static OncePerDevice allowed;   // for the deepest network, whatever this one's depth
    KRR_CUDA(allow_shared(allowed, k_nrc_forward_tc, nrc_tc_smem_bytes(kNrcMaxLayers)));
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int64_t tiles = (cap + kTcRows - 1) / kTcRows;
    int grid = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)sms));
    k_nrc_forward_tc<<<grid, kFwThreads, smem, s>>>(g, mlp.layers, d_in, d_count, cap, table, packed,
                                                    d_out, out_stride, acts, err);
    KRR_CUDA(cudaGetLastError());
    return KRR_OK;
}

}  // namespace krr
