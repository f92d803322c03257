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
constexpr int kTcThreads = 128;
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
// B BF16 (bits 7-9 and 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4
// at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
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

// Writes one row (64 values) of a canonical tile as eight 16-byte chunks.
__device__ __forceinline__ void store_row(uint8_t *tile, uint32_t r, const float *v) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        __nv_bfloat162 p0 = __floats2bfloat162_rn(v[8 * j + 0], v[8 * j + 1]);
        __nv_bfloat162 p1 = __floats2bfloat162_rn(v[8 * j + 2], v[8 * j + 3]);
        __nv_bfloat162 p2 = __floats2bfloat162_rn(v[8 * j + 4], v[8 * j + 5]);
        __nv_bfloat162 p3 = __floats2bfloat162_rn(v[8 * j + 6], v[8 * j + 7]);
        uint4 q;
        q.x = *reinterpret_cast<uint32_t *>(&p0);
        q.y = *reinterpret_cast<uint32_t *>(&p1);
        q.z = *reinterpret_cast<uint32_t *>(&p2);
        q.w = *reinterpret_cast<uint32_t *>(&p3);
        *reinterpret_cast<uint4 *>(tile + canon(r, 8 * j)) = q;
    }
}

// Packs the BF16 weights [layer][out][64] into canonical tiles.
__global__ void k_pack_weights(const __nv_bfloat16 *__restrict__ w, NrcMlp mlp, uint8_t *packed) {
    int total = mlp.n_params;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        int l = 0;
        while (l + 1 < mlp.layers && e >= mlp.w_offset[l + 1]) ++l;
        int local = e - mlp.w_offset[l];
        int r = local / kNrcIn, k = local % kNrcIn;
        *reinterpret_cast<__nv_bfloat16 *>(packed + (size_t)l * kLayerBytes + canon(r, k)) = w[e];
    }
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
// N=64, K=64 or 16) and dW_l += dY_l^T . X_l (M=128 with rows 64..127 of the
// A operand zero, N=64, K=128 rows of the tile).  The dX accumulator (64
// columns) is read back each layer, masked by ReLU'(X_l), rounded to BF16
// and becomes the next layer's dY tile (row-major and transposed copies);
// the dW_l accumulators (64 columns each) stay in tensor memory for all of
// the CTA's tiles and are added to the FP32 gradient once at the end.
// Operand rounding points match the CUDA-core kernels: dY, W and X in BF16,
// FP32 accumulation.

constexpr uint32_t kBwCols = 512;
constexpr int kT128Bytes = 128 * 128 * 2;   // [128][128] canonical tile, 32 KB
constexpr int kXtBytes = 64 * 128 * 2;      // [64][128], 16 KB
constexpr int kA64Bytes = 128 * 64 * 2;     // [128][64], 16 KB
constexpr int kA16Bytes = 128 * 16 * 2;     // [128][16], 4 KB
constexpr int kWtOutBytes = 64 * 16 * 2;    // W_out^T [64][16], 2 KB

// Byte offset of element (r, k) in a canonical K-major tile of `cols` columns.
__host__ __device__ __forceinline__ uint32_t canon_c(uint32_t r, uint32_t k, uint32_t cols) {
    return (((r >> 3) * (cols >> 3) + (k >> 3)) * 128u) + (r & 7u) * 16u + (k & 7u) * 2u;
}

// Transposed weights: hidden layer l as W_l^T [64 in][64 out] at l * 8 KB,
// the output layer as W^T [64 in][16 out] after them.
__global__ void k_pack_weights_t(const __nv_bfloat16 *__restrict__ w, NrcMlp mlp, uint8_t *packed) {
    int total = mlp.n_params;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        int l = 0;
        while (l + 1 < mlp.layers && e >= mlp.w_offset[l + 1]) ++l;
        int local = e - mlp.w_offset[l];
        int r = local / kNrcIn, k = local % kNrcIn;   // W_l[r][k]
        size_t off = l + 1 < mlp.layers ? (size_t)l * kLayerBytes + canon_c(k, r, 64)
                                        : (size_t)l * kLayerBytes + canon_c(k, r, 16);
        *reinterpret_cast<__nv_bfloat16 *>(packed + off) = w[e];
    }
}

__device__ __forceinline__ void store_bf16(uint8_t *tile, uint32_t off, float v) {
    *reinterpret_cast<__nv_bfloat16 *>(tile + off) = __float2bfloat16_rn(v);
}

// Bounded wait on the CTA's mbarrier by thread 0, decision shared through
// shared memory; returns false (all threads) when the wait gave up.
__device__ __forceinline__ bool cta_wait(uint32_t mbar, uint32_t phase, uint32_t *fail_flag,
                                         uint32_t *err) {
    if (threadIdx.x == 0) {
        uint32_t spins = 0, ok = 0;
        while (!(ok = mbar_try_wait(mbar, phase)) && ++spins < kWaitLimit) {
        }
        *fail_flag = ok ? 0u : 1u;
        if (!ok) atomicOr(err, (uint32_t)kErrLoopLimit);
    }
    __syncthreads();
    if (*fail_flag) return false;
    uint32_t spins = 0;   // already complete: returns at once
    while (!mbar_try_wait(mbar, phase) && ++spins < kWaitLimit) {
    }
    return true;
}

__global__ void __launch_bounds__(kTcThreads, 1)
k_nrc_backward_tc(int layers, const float *__restrict__ dy_out, const __nv_bfloat16 *__restrict__ acts,
                  const int32_t *d_count, int64_t cap, const uint8_t *__restrict__ packed_wt,
                  float *__restrict__ dx0, float *__restrict__ dw, NrcMlp mlp, uint32_t *err) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int wt_bytes = (layers - 1) * kLayerBytes + kWtOutBytes;
    uint8_t *swt = smem;
    uint8_t *at = smem + ((wt_bytes + 1023) & ~1023);   // dY_l^T, rows 64..127 zero
    uint8_t *at16 = at + kT128Bytes;                     // dY_out^T, rows 16..127 zero
    uint8_t *xt = at16 + kT128Bytes;                     // X_l^T
    uint8_t *a64 = xt + kXtBytes;                        // dY_l
    uint8_t *a16 = a64 + kA64Bytes;                      // dY_out
    uint64_t *mbar = reinterpret_cast<uint64_t *>(a16 + kA16Bytes);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mbar + 1);
    uint32_t *fail_flag = tmem_slot + 1;
    const int tid = threadIdx.x, warp = tid >> 5;

    for (int e = tid; e < wt_bytes / 16; e += blockDim.x)
        reinterpret_cast<uint4 *>(swt)[e] = reinterpret_cast<const uint4 *>(packed_wt)[e];
    for (int e = tid; e < 2 * kT128Bytes / 16; e += blockDim.x)
        reinterpret_cast<uint4 *>(at)[e] = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(kBwCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        mbar_init(smem_u32(mbar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    const uint32_t my_lanes = (uint32_t)(warp * 32) << 16;

    const int64_t n = d_count ? min((int64_t)*d_count, cap) : cap;
    const int64_t tiles = (n + kTcRows - 1) / kTcRows;
    uint32_t phase = 0;
    bool failed = false, any_tile = false;
    for (int64_t t = blockIdx.x; t < tiles && !failed; t += gridDim.x) {
        const int64_t row = t * kTcRows + tid;
        const bool live = row < n;
        // dY of the output layer: row-major [128][16] and transposed [16 of 128][128]
        {
            float d[kNrcOutPad];
            for (int c = 0; c < kNrcOutPad; ++c) d[c] = live ? dy_out[row * kNrcOutPad + c] : 0.f;
            for (int c = 0; c < kNrcOutPad; ++c) {
                store_bf16(a16, canon_c((uint32_t)tid, (uint32_t)c, 16), d[c]);
                store_bf16(at16, canon_c((uint32_t)c, (uint32_t)tid, 128), d[c]);
            }
        }
        for (int l = layers - 1; l >= 0 && !failed; --l) {
            const bool out_layer = l == layers - 1;
            // X_l^T and the ReLU mask of X_l
            uint64_t mask = 0;
            {
                const uint4 *src = reinterpret_cast<const uint4 *>(acts + ((size_t)l * cap + row) * kNrcIn);
                for (int j = 0; j < 8; ++j) {
                    uint4 q = live ? src[j] : make_uint4(0u, 0u, 0u, 0u);
                    const __nv_bfloat16 *h = reinterpret_cast<const __nv_bfloat16 *>(&q);
                    for (int i = 0; i < 8; ++i) {
                        const int k = 8 * j + i;
                        *reinterpret_cast<__nv_bfloat16 *>(xt + canon_c((uint32_t)k, (uint32_t)tid, 128)) = h[i];
                        if (__bfloat162float(h[i]) > 0.f) mask |= 1ull << k;
                    }
                }
            }
            fence_proxy_async();
            fence_before_sync();
            __syncthreads();
            if (tid == 0) {
                fence_after_sync();
                // dW_l += dY_l^T . X_l   (K = the tile's 128 rows)
                const uint32_t a0 = smem_u32(out_layer ? at16 : at), b0 = smem_u32(xt);
                const uint32_t dcol = tmem + 64u + 64u * (uint32_t)l;
                const uint32_t idw = idesc_bf16(kTcRows, 64);
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                    tc_mma(dcol, smem_desc(a0 + 256u * kk, 128u, 2048u), smem_desc(b0 + 256u * kk, 128u, 2048u),
                           idw, (any_tile || kk > 0) ? 1u : 0u);
                // dX = dY_l . W_l  (K = 16 for the output layer, 64 otherwise)
                const uint32_t wt = smem_u32(swt + l * kLayerBytes);
                if (out_layer) {
                    tc_mma(tmem, smem_desc(smem_u32(a16), 128u, 256u), smem_desc(wt, 128u, 256u),
                           idesc_bf16(kTcRows, 64), 0u);
                } else {
                    const uint32_t a1 = smem_u32(a64);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        tc_mma(tmem, smem_desc(a1 + 256u * kk, 128u, 1024u), smem_desc(wt + 256u * kk, 128u, 1024u),
                               idesc_bf16(kTcRows, 64), kk > 0 ? 1u : 0u);
                }
                tc_commit(smem_u32(mbar));
            }
            if (!cta_wait(smem_u32(mbar), phase, fail_flag, err)) {
                failed = true;
                break;
            }
            phase ^= 1u;
            fence_after_sync();
            float v[kNrcIn];
            tmem_ld16(tmem + my_lanes + 0, v);
            tmem_ld16(tmem + my_lanes + 16, v + 16);
            tmem_ld16(tmem + my_lanes + 32, v + 32);
            tmem_ld16(tmem + my_lanes + 48, v + 48);
            tmem_wait_ld();
            if (l > 0) {
                for (int k = 0; k < kNrcIn; ++k) {
                    const float d = ((mask >> k) & 1ull) ? v[k] : 0.f;
                    v[k] = d;
                    store_bf16(at, canon_c((uint32_t)k, (uint32_t)tid, 128), d);
                }
                store_row(a64, (uint32_t)tid, v);
                fence_proxy_async();
            } else if (live) {
                float4 *dst = reinterpret_cast<float4 *>(dx0 + row * kNrcIn);
                for (int k = 0; k < kNrcIn / 4; ++k)
                    dst[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
            }
            fence_before_sync();
            __syncthreads();
        }
        any_tile = true;
    }
    // dW accumulators: rows 0..63 (out features) live in the lanes of warps 0-1
    if (!failed && any_tile && warp < 2) {
        fence_after_sync();
        const int m = tid;   // out-feature row of dW_l
        for (int l = 0; l < layers; ++l) {
            const int rows = l + 1 == layers ? kNrcOutPad : kNrcWidth;
            float v[kNrcIn];
            const uint32_t base = tmem + my_lanes + 64u + 64u * (uint32_t)l;
            tmem_ld16(base + 0, v);
            tmem_ld16(base + 16, v + 16);
            tmem_ld16(base + 32, v + 32);
            tmem_ld16(base + 48, v + 48);
            tmem_wait_ld();
            if (m < rows) {   // 16-byte vector atomics (the row offsets are multiples of 64 floats)
                float4 *dst = reinterpret_cast<float4 *>(dw + mlp.w_offset[l] + (size_t)m * kNrcIn);
                for (int k = 0; k < kNrcIn / 4; ++k)
                    atomicAdd(dst + k, make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]));
            }
        }
    }
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
    size_t w = (size_t)(layers - 1) * kLayerBytes + kWtOutBytes;
    return ((w + 1023) & ~(size_t)1023) + 2 * kT128Bytes + kXtBytes + kA64Bytes + kA16Bytes + 64 + 1024;
}

int nrc_pack_weights_t(const __nv_bfloat16 *w, const NrcMlp &mlp, uint8_t *packed, cudaStream_t s) {
    cudaMemsetAsync(packed, 0, (size_t)(mlp.layers - 1) * kLayerBytes + kWtOutBytes, s);
    k_pack_weights_t<<<64, 256, 0, s>>>(w, mlp, packed);
    KRR_CUDA(cudaGetLastError());
    return KRR_OK;
}

int nrc_backward_tc(const NrcMlp &mlp, const float *d_dy_out, const __nv_bfloat16 *acts,
                    const int32_t *d_count, int64_t cap, const uint8_t *packed_wt, float *d_dx0,
                    float *d_dw, uint32_t *err, cudaStream_t s) {
    static bool configured = false;
    size_t smem = nrc_tc_bwd_smem_bytes(mlp.layers);
    if (!configured) {
        KRR_CUDA(cudaFuncSetAttribute(k_nrc_backward_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)nrc_tc_bwd_smem_bytes(kNrcMaxLayers)));
        configured = true;
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int64_t tiles = (cap + kTcRows - 1) / kTcRows;
    int grid = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)sms));
    k_nrc_backward_tc<<<grid, kTcThreads, smem, s>>>(mlp.layers, d_dy_out, acts, d_count, cap, packed_wt,
                                                     d_dx0, d_dw, mlp, err);
    KRR_CUDA(cudaGetLastError());
    return KRR_OK;
}

int nrc_forward_tc(const NrcGrid &g, const NrcMlp &mlp, const float *d_in, const int32_t *d_count,
                   int64_t cap, const __nv_bfloat16 *table, const uint8_t *packed, float *d_out, int out_stride,
                   __nv_bfloat16 *acts, uint32_t *err, cudaStream_t s) {
    static bool configured = false;
    size_t smem = nrc_tc_smem_bytes(mlp.layers);
    if (!configured) {   // for the deepest network, whatever this one's depth
        KRR_CUDA(cudaFuncSetAttribute(k_nrc_forward_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)nrc_tc_smem_bytes(kNrcMaxLayers)));
        configured = true;
    }
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
