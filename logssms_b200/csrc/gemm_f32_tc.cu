// 32-bit matrix product of many rows on the 5th-generation tensor cores:  C[M, N] = (A[M, K] W[N, K]^T + bias) * scale, all
// float32, with the accuracy of 32-bit arithmetic.
//
// A float32 value is the sum of three bfloat16 values: h its rounding, m the rounding of x - h, l the rounding of
// x - h - m (8 + 8 + 8 bits; what is left is below 2^-26 |x|): the published splitting of a number into parts of a shorter
// format whose products are exact (Dekker 1971; Ozaki, Ogita, Oishi and Rump 2012 for matrix products).  bfloat16 has float32's
// exponents, so the parts of a small value would fall below its smallest normal number (from |x| < 2^-108 on they would keep
// fewer bits than the value); every value is therefore split as 2^24 x: a float32 number is a multiple of 2^-149, its parts are
// multiples of 2^-125.  The sums are divided by 2^48 at the end; what leaves float32's range on the way is computed again, below.
// Of the nine products of two such sums six are taken,
// h h, h m, m h, m m, h l, l h; those left out are below 2^-25 of |a w| together.  bfloat16 products are exact in the
// tensor core; what is lost is in its sums, which drop bits below the accumulator's last place.  Therefore
//   * h h gets an accumulator of its own that is emptied into registers after every 64 values of k and added up there
//     with ordinary rounded additions (two of them in turn, so that the next block's products run meanwhile);
//   * the five small products (2^-8 of h h at most) share two others for the whole of k.
// Error against 64 bits over the float32 model's products (K 512 .. 2,048, 33 .. 2,048 rows): 0.9e-7 to 1.3e-7 relative
// (2-norm), the FFMA tiles of gemm_f32.cu 1.5e-7 to 5e-7.
//
// Bound by shared memory: per block of 64 values of k a 128 x 128 tile's 24 products read 192 KB of operands, and 96 KB
// are written; a block takes about 3,800 cycles, the tensor pipe needs 1,540 of them, the FFMA form 8,192.  601 rows of
// 4,096 x 1,024: 140 -> 66 us as 160 tiles in two waves, 49 with the second one's 12 tiles cut into 8 parts of K; of 3,352 x
// 1,024: 113 -> 35 us; of 1,024 x 1,536 and 1,024 x 2,048 (40 tiles) 29 -> 23 and 35 -> 28 us with 3 parts instead of 2; 2,048 rows 322 -> 102 us.
//
//   warps 0-7   fetch the next block of A and W (16-byte loads into registers, both 128 rows x 64 values of k), split it
//               and store the six planes (128-byte swizzle) into one of two stages
//   warps 8-15  empty the h h accumulator after every block: a thread is a row and half of the columns; at the end the
//               tile goes through shared memory, where a cluster of 2 to 8 CTAs that share a tile's K adds its parts
//               up in rank order (distributed shared memory), as in gemm_f32.cu
//   warp 8      also allocates tensor memory (all 512 columns); one of its threads issues the products
// An element whose sum is not finite is computed again in plain 32-bit arithmetic: infinity times the zero of a smaller
// plane is NaN where infinity times w is infinity, and a value past 2^104 or a sum past 2^80 overflows by the factors above.
//
// Every mbarrier wait is bounded; one that gives up records itself in `error`, the others run out of theirs, all threads
// meet the barriers, tensor memory is freed and the kernel returns.
#include <cooperative_groups.h>
#include "lb200/common.cuh"
#include "lb200/tcgen05.cuh"
using namespace lb200;
using namespace lb200::tc;
namespace cg = cooperative_groups;

namespace {
constexpr int kTile = 128, kBK = 64;
constexpr int kSplitThreads = 256, kSumThreads = 256, kThreads = kSplitThreads + kSumThreads;
constexpr uint32_t kPlane = kTile * 128;                  // 128 rows of 64 bfloat16
constexpr uint32_t kStage = 6 * kPlane;                   // A's planes h, m, l, then W's
constexpr int kOutRow = kTile + 4;
constexpr size_t kSmem = 2 * (size_t)kStage;
constexpr float kUp = 0x1p24f, kDown = 0x1p-48f;          // on a value; on a sum of products
static_assert((size_t)kTile * kOutRow * 4 <= kSmem, "the finished tile lies over the stages");

__device__ __forceinline__ void report(int* error, int role, int step) {
    if (error != nullptr) atomicCAS(error, 0, 0x08000000 | (role << 24) | ((blockIdx.x & 0xFFF) << 12) | (step & 0xFFF));
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float low(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float high(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
// two values as one register pair (packed arithmetic takes half the instructions)
__device__ __forceinline__ unsigned long long pair(float a, float b) {
    return (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
}
__device__ __forceinline__ uint32_t rounded(unsigned long long v) {
    return pack2(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)));
}
__device__ __forceinline__ unsigned long long scaled_up(float a, float b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pair(a, b)), "l"(pair(kUp, kUp)));
    return d;
}
__device__ __forceinline__ unsigned long long rest(unsigned long long v, uint32_t part) {      // v minus a part of it (exact)
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(pair(low(part), high(part))), "l"(pair(-1.f, -1.f)), "l"(v));
    return d;
}
// four values of k of one row -> their places in the three planes
__device__ __forceinline__ void split_store(uint8_t* at, const float4& v) {
    const unsigned long long a = scaled_up(v.x, v.y), b = scaled_up(v.z, v.w);
    const uint32_t h0 = rounded(a), h1 = rounded(b);
    const unsigned long long ra = rest(a, h0), rb = rest(b, h1);
    const uint32_t m0 = rounded(ra), m1 = rounded(rb);
    const uint32_t l0 = rounded(rest(ra, m0)), l1 = rounded(rest(rb, m1));
    *reinterpret_cast<uint2*>(at) = make_uint2(h0, h1);
    *reinterpret_cast<uint2*>(at + kPlane) = make_uint2(m0, m1);
    *reinterpret_cast<uint2*>(at + 2 * kPlane) = make_uint2(l0, l1);
}

// LISTED: the launch is `gridDim.x` tiles from tile0 on, along N first; else its x and y are the tile's (the division by a number of
// tiles that the first form starts with costs 1 to 4 % of the kernel: its results stay in registers that the loads' addresses need).
template <bool LISTED>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_tc_kernel(const float* __restrict__ A, long lda, const float* __restrict__ W, const float* __restrict__ bias,
                   float* __restrict__ C, long ldc, int M, int N, int K, float out_scale, int tile0, int* error) {
    extern __shared__ __align__(1024) uint8_t smem[];      // the swizzle's pattern repeats every 1024 bytes
    __shared__ __align__(8) uint64_t full[2], empty[2], sum_full[2], sum_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto place = [&](int x, int& n0, int& m0) {
        const int tiles_n = (N + kTile - 1) / kTile, tile = tile0 + x;
        n0 = LISTED ? tile % tiles_n * kTile : blockIdx.x * kTile;
        m0 = LISTED ? tile / tiles_n * kTile : blockIdx.y * kTile;
    };
    int n0, m0;
    place(blockIdx.x, n0, m0);
    const int part = blockIdx.z, parts = gridDim.z;
    const int blocks = (K + kBK - 1) / kBK;
    const int kb0 = (int)((long)blocks * part / parts), kbn = (int)((long)blocks * (part + 1) / parts) - kb0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(full + s, kSplitThreads); mbar_init(empty + s, 1);
            mbar_init(sum_full + s, 1); mbar_init(sum_empty + s, kSumThreads);
        }
        failed = 0;
        mbar_fence_init();
    }
    if (warp == 8) tmem_alloc<512>(&tmem_slot);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_slot;                       // columns 0 and 128: h h of even and odd blocks; 256 and 384: the small products
    float* out_s = reinterpret_cast<float*>(smem);

    if (warp < 8) {
        // two rows of 64 values per load instruction of a warp; a thread's rows are 16 * warp + lane / 16 + 2 i
        const int r0 = warp * 16 + (lane >> 4), kc = (lane & 15) * 4;
        float4 va[8], vw[8];
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        auto load_a = [&](int i, int k) {
            const int m = m0 + r0 + 2 * i;
            return m < M && k < K ? *reinterpret_cast<const float4*>(A + (size_t)m * lda + k) : zero;
        };
        auto load_w = [&](int i, int k) {
            const int n = n0 + r0 + 2 * i;
            return n < N && k < K ? __ldg(reinterpret_cast<const float4*>(W + (size_t)n * K + k)) : zero;
        };
#pragma unroll
        for (int i = 0; i < 8; ++i) { va[i] = load_a(i, kb0 * kBK + kc); vw[i] = load_w(i, kb0 * kBK + kc); }
        for (int kb = 0; kb < kbn; ++kb) {
            const int s = kb & 1;
            bool ok = kb < 2 || mbar_wait(empty + s, ((kb >> 1) - 1) & 1);
            if (!ok) { report(error, 1, kb); failed = 1; }
            if (!__all_sync(0xffffffffu, ok) || failed) break;
            uint8_t* stage = smem + s * kStage;
            const int k_next = kb + 1 < kbn ? (kb0 + kb + 1) * kBK + kc : K;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = r0 + 2 * i;
                uint8_t* at = stage + r * 128 + (((kc >> 3) ^ (r & 7)) << 4) + (kc & 4) * 2;
                // the registers are free as soon as a piece is stored: the next block's is asked for, under the rest's arithmetic
                split_store(at, va[i]);
                va[i] = load_a(i, k_next);
                split_store(at + 3 * kPlane, vw[i]);
                vw[i] = load_w(i, k_next);
            }
            fence_async_smem();
            mbar_arrive(full + s);
        }
    } else {
        const uint32_t idesc = umma_idesc(kTile, kTile), idesc_wide = umma_idesc(kTile, 2 * kTile);
        auto issue = [&](int kb) {                         // one thread: the products of a block
            const int s = kb & 1;
            if (!mbar_wait(full + s, (kb >> 1) & 1)) { report(error, 2, kb); failed = 1; return; }
            if (kb >= 2 && !mbar_wait(sum_empty + s, ((kb >> 1) - 1) & 1)) { report(error, 3, kb); failed = 1; return; }
            fence_after_sync();
            const uint64_t a_h = umma_desc(smem + s * kStage), w_h = umma_desc(smem + s * kStage + 3 * kPlane);
            constexpr uint64_t kM = kPlane >> 4, kL = 2 * (kPlane >> 4);
            const uint32_t d_hh = tmem + s * kTile, d_small = tmem + 2 * kTile;
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k) {
                const uint64_t a = a_h + 2 * k, w = w_h + 2 * k;
                // two planes of W side by side are one operand of 256 rows: a plane of A is read once for both
                umma_bf16(d_small, a, w + kM, idesc_wide, (kb | k) != 0);        // h (m | l)
                umma_bf16(d_small, a + kM, w, idesc_wide, 1);                    // m (h | m)
                umma_bf16(d_small, a + kL, w, idesc, 1);                         // l h
                umma_bf16(d_hh, a, w, idesc, k != 0);
            }
            umma_commit(empty + s);
            umma_commit(sum_full + s);
        };
        const int quarter = warp & 3, half = (warp - 8) >> 2, r = quarter * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16) + half * (kTile / 2);
        float sum[kTile / 2];
#pragma unroll
        for (int c = 0; c < kTile / 2; ++c) sum[c] = 0.f;
        bool ok = true;
        for (int next = 0; next <= kbn && ok; ++next) {    // the block before is emptied while the products of the next run
            if (warp == 8) {
                if (lane == 0 && next < kbn && !failed) issue(next);
                __syncwarp();
            }
            if (next == 0) continue;
            const int kb = next - 1, s = kb & 1;
            ok = mbar_wait(sum_full + s, (kb >> 1) & 1);
            if (!ok && lane == 0) { report(error, 4, kb); failed = 1; }
            ok = __all_sync(0xffffffffu, ok && !failed);
            if (!ok) break;
            fence_after_sync();
#pragma unroll
            for (int c0 = 0; c0 < kTile / 2; c0 += 32) {
                uint32_t v[32];
                tmem_ld32(lane_addr + s * kTile + c0, v);
#pragma unroll
                for (int c = 0; c < 32; ++c) sum[c0 + c] += __uint_as_float(v[c]);
            }
            fence_before_sync();
            mbar_arrive(sum_empty + s);
        }
        if (ok) {                                          // the last block's products cover the small ones, too
#pragma unroll
            for (int c0 = 0; c0 < kTile / 2; c0 += 32)
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                uint32_t v[32];
                tmem_ld32(lane_addr + (2 + side) * kTile + c0, v);
#pragma unroll
                for (int c = 0; c < 32; ++c) sum[c0 + c] += __uint_as_float(v[c]);
            }
            // every product has read its stage: the tile goes there
#pragma unroll
            for (int c = 0; c < kTile / 2; c += 4)
                *reinterpret_cast<float4*>(out_s + r * kOutRow + half * (kTile / 2) + c) = make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
        }
    }
    fence_before_sync();
    if (parts > 1) cg::this_cluster().sync(); else __syncthreads();
    if (warp == 8) tmem_free<512>(tmem);
    if (!failed) {
        int x;                                             // worked out anew: kept through the loops they spill
        asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(x));
        place(x, n0, m0);
        const int row0 = kTile * part / parts, rows = kTile * (part + 1) / parts - row0;
        const bool wide = ((uintptr_t)C & 15) == 0 && ldc % 4 == 0 && n0 + kTile <= N;
        for (int i = threadIdx.x; i < rows * (kTile / 4); i += kThreads) {
            const int r = row0 + i / (kTile / 4), c = i % (kTile / 4) * 4;
            const int m = m0 + r, n = n0 + c;
            if (m >= M || n >= N) continue;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int p = 0; p < parts; ++p) {
                const float* tile = parts > 1 ? cg::this_cluster().map_shared_rank(out_s, p) : out_s;
                const float4 t = *reinterpret_cast<const float4*>(tile + r * kOutRow + c);
                v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
            }
            float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (n + e >= N) continue;
                if (!(fabsf(o[e]) <= 3.0e38f)) {           // infinite or NaN, or close to overflow: as plain arithmetic gives it
                    float s = 0.f;
                    for (int k = 0; k < K; ++k) s = fmaf(A[(size_t)m * lda + k], W[(size_t)(n + e) * K + k], s);
                    o[e] = s;
                } else o[e] *= kDown;
                o[e] = (o[e] + (bias != nullptr ? bias[n + e] : 0.f)) * out_scale;
            }
            float* out = C + (size_t)m * ldc + n;
            if (wide) *reinterpret_cast<float4*>(out) = make_float4(o[0], o[1], o[2], o[3]);
            else
                for (int e = 0; e < 4 && n + e < N; ++e) out[e] = o[e];
        }
    }
    if (parts > 1) cg::this_cluster().sync();              // nobody leaves while another one reads its tile
}

// A launch with a tile's K in `parts` CTAs of a cluster; grid and stream are the caller's.
cudaLaunchConfig_t launch_config(cudaLaunchAttribute (&attr)[1], int parts) {
    static size_t have[2] = {};
    ensure_dynamic_smem(gemm_f32_tc_kernel<false>, kSmem, have[0]);
    ensure_dynamic_smem(gemm_f32_tc_kernel<true>, kSmem, have[1]);
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = parts;
    cfg.attrs = attr;
    cfg.numAttrs = parts > 1 ? 1 : 0;
    return cfg;
}
// Clusters of so many CTAs that the GPU holds at once; 0: none.
int clusters_held(int parts) {
    static int held[9] = {};                               // plus one; 0: not asked yet
    if (held[parts] == 0) {
        int n = 148;
        if (parts > 1) {
            cudaLaunchAttribute attr[1];
            cudaLaunchConfig_t cfg = launch_config(attr, parts);
            cfg.gridDim = dim3(148, 1, parts);
            if (cudaOccupancyMaxActiveClusters(&n, gemm_f32_tc_kernel<false>, &cfg) != cudaSuccess) {
                cudaGetLastError();                        // (the question's error is not the launch's)
                n = 0;
            }
        }
        held[parts] = n + 1;
    }
    return held[parts] - 1;
}
}  // namespace

// A: [M, K] float32 rows `lda` elements apart, W: [N, K] contiguous, C: [M, N] rows `ldc` apart; K and lda multiples of 4,
// A and W on 16-byte boundaries.  `error`: a device int that is 0 before the call; non-zero afterwards: a wait gave up.
extern "C" int lb_gemm_f32_tc(const float* A, long lda, const float* W, const float* bias, float* C, long ldc, int M, int N,
                              int K, float out_scale, int* error, void* stream) {
    if (M <= 0 || N <= 0) return kOk;
    if (K <= 0 || K % 4 || lda % 4 || (((uintptr_t)A | (uintptr_t)W) & 15)) return kBadSize;
    const long tiles_m = (M + kTile - 1) / kTile, tiles_n = (N + kTile - 1) / kTile, tiles = tiles_m * tiles_n;
    if (tiles_m > 65535 || tiles > 0x7fffffffL) return kTooLarge;
    // Parts of K: a launch takes as many rounds of clusters as the GPU does not hold at once, a round the blocks of a part and about three
    // blocks' time more (a pipeline's start, the exchange).  How many clusters it holds is asked: 45 of 3 CTAs, 33 of 4, 26 of 5, 22 of 6,
    // 15 of 7 or 8 on 148 SMs.  `fewest`: the parts that a cut in powers of two over 148 SMs takes; with fewer the sums of a part are
    // longer than they were, and their error up to 1.8 times.
    const int blocks = (K + kBK - 1) / kBK;
    auto cost = [&](long n, int p) {
        const int held = clusters_held(p);
        return held > 0 ? (double)((n + held - 1) / held) * ((blocks + p - 1) / p + 3) : 1e30;
    };
    int fewest = 1;
    double low = 1e30;
    for (int p = 1; p <= 8 && (p == 1 || blocks / p >= 2); p *= 2) {
        const double c = (double)((tiles * p + 147) / 148) * ((double)((blocks + p - 1) / p) + (p > 1 ? 3.0 : 0.0) + 2.0);
        if (c < low * 0.98) { low = c; fewest = p; }
    }
    auto best_parts = [&](long n, double& best) {
        int parts = fewest;
        best = cost(n, fewest);
        for (int p = fewest + 1; p <= 8 && blocks / p >= 2; ++p)
            if (cost(n, p) < best * 0.94) { best = cost(n, p); parts = p; }
        return parts;
    };
    // Where the last round would be a few tiles, they go in a launch of their own with K cut finer (a launch costs about a block's
    // time): 601 rows of 4,096 x 1,024 are 160 tiles, 148 and then 12 in 8 parts.
    double all, tail = 0.0;
    int parts[2] = {best_parts(tiles, all), 1};
    long count[2] = {tiles, 0};
    const long rest = tiles % 148;
    if (tiles > 148 && rest != 0) {
        const int p1 = best_parts(rest, tail);
        if (p1 > fewest && cost(tiles - rest, fewest) + tail + 1.0 < all * 0.95) {
            parts[0] = fewest; parts[1] = p1;
            count[0] = tiles - rest; count[1] = rest;
        }
    }
    int rc = 0;
    for (int i = 0; i < 2 && rc == 0 && count[i] > 0; ++i) {
        const bool listed = count[1] > 0;
        cudaLaunchAttribute attr[1];
        cudaLaunchConfig_t cfg = launch_config(attr, parts[i]);
        cfg.gridDim = listed ? dim3((unsigned)count[i], 1, parts[i]) : dim3((unsigned)tiles_n, (unsigned)tiles_m, parts[i]);
        cfg.stream = (cudaStream_t)stream;
        rc = (int)cudaLaunchKernelEx(&cfg, listed ? gemm_f32_tc_kernel<true> : gemm_f32_tc_kernel<false>, A, lda, W, bias, C, ldc, M, N, K,
                                     out_scale, i == 0 ? 0 : (int)count[0], error);
    }
    return rc != 0 ? rc : launch_status();
}
