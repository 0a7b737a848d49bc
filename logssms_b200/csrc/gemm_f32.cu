// True 32-bit matrix product for the float32 path: C[M, N] = A[M, K] * W[N, K]^T (+ bias[N]) (* out_scale).
//
// Plain FFMA accumulation in float32; no tensor cores, so no reduced-precision matrix mode can sneak in whatever the
// library defaults are.  (Many rows of many weights go to gemm_f32_tc.cu; see there for how it keeps 32 bits.)  A may be a
// row-strided view.  Two kernels:
//
//   * `stream_f32_kernel`, few rows (`kStreamRows`): bound by the bytes of W, which it reads once up to 16 rows (17 to 32
//     rows are two row blocks: the second reads W from L2).  A CTA takes F features
//     with K split over its 8 warps, so that even 768 features of K = 1,024 put 192 CTAs of 16 KB each on the chip with
//     every load of W in flight at once; with up to kPdlMaxRows rows the CTAs start under the kernel in front and have L2
//     fetch their part of W (no more than that: W may be what the kernel in front writes, and L2 is where it arrives).
//     The lanes' partial sums are exchanged so that each lane ends with its own sums (V values over 32 lanes cost about V
//     shuffles instead of 5 V).  3352 x 1024: 4.7 us at 4 rows
//     (2.9 TB/s), 3.8 us at one; 193 us with the 64 x 64 tiles of one CTA each that were here before.
//   * `tile_f32_kernel`, many rows: bound by the FFMA pipes.  128 x 64 tiles (64 x 64 up to 64 rows), 128 threads with
//     8 x 8 outputs each, packed two values of k at a time (`fma.rn.f32x2`: the register pairs that a 16-byte load of either
//     operand leaves are the instruction's operands, nothing is packed or transposed), K in steps of 32 through two
//     cp.async stages (steps of 16 through four: a tenth slower, the barrier between steps costs more than depth gains).
//     Rows of 144 bytes in shared memory: 8 rows of A (or 4 of W) fall on different banks.  Where the
//     tiles do not divide the SMs evenly, a cluster of 2, 4 or 8 CTAs shares a tile's K and adds its parts up through
//     distributed shared memory, always in the same order.  601 rows, 4096 x 1024:
//     139 us (36 TFLOP/s; 47 at 2,048 rows), 315 us with the 64 x 64 tiles of 4 x 4 outputs per thread.
#include <cooperative_groups.h>
#include "lb200/common.cuh"
using namespace lb200;
namespace cg = cooperative_groups;

namespace {
// ---------------------------------------------------------------------------------------------------- few rows
constexpr int kStreamRows = 32, kStreamWarps = 8;

__device__ __forceinline__ float4 load_once(const float* p) {
    float4 v;
    asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// V sums over the 32 lanes of a warp: while more than one value is left, a step exchanges half of them with the lane
// `o` away, each lane keeping the half its bit says.  Afterwards lane l holds the sums number `first(l)` + i, i < V / 32
// (V < 32: the sum number first(l), on several lanes).
template <int V, int O>
struct LaneSums {
    static __device__ __forceinline__ void run(float* v, int lane, int& first) {
        if constexpr (V > 1) {
            const bool upper = lane & O;
#pragma unroll
            for (int i = 0; i < V / 2; ++i) {
                const float give = upper ? v[i] : v[i + V / 2], keep = upper ? v[i + V / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, O);
            }
            if (upper) first += V / 2;
            if constexpr (O > 1) LaneSums<V / 2, O / 2>::run(v, lane, first);
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
            if constexpr (O > 1) LaneSums<1, O / 2>::run(v, lane, first);
        }
    }
};

// MT: rows of a CTA (a power of two up to 16), F: features of a CTA.  Chunks of 128 values of k go to the warps in turn.
template <int MT, int F>
__global__ void __launch_bounds__(kStreamWarps * 32, MT * F > 32 ? 1 : 2)
stream_f32_kernel(const float* __restrict__ A, long lda, const float* __restrict__ W, const float* __restrict__ bias,
                  float* __restrict__ C, long ldc, int M, int N, int K, float out_scale) {
    constexpr int V = MT * F, kHeld = V >= 32 ? V / 32 : 1;
    __shared__ float sums[kStreamWarps][V];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * F, m0 = blockIdx.y * MT;
    float acc[V];                                            // number m * F + f
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = 0.f;
    const float* wrow[F];
#pragma unroll
    for (int f = 0; f < F; ++f) wrow[f] = W + (size_t)min(n0 + f, N - 1) * K;
    auto fetch = [&](int k, float4 (&w)[F]) {
#pragma unroll
        for (int f = 0; f < F; ++f) w[f] = k < K ? load_once(wrow[f] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    constexpr int kStep = kStreamWarps * 128;
    float4 w[F], wn[F];
    int k = warp * 128 + lane * 4;
    if (lane % 8 == 0)
        for (int kk = k; kk < K; kk += kStep)
#pragma unroll
            for (int f = 0; f < F; ++f) asm volatile("prefetch.global.L2 [%0];" ::"l"(wrow[f] + kk));
    pdl_trigger();
    pdl_wait();
    fetch(k, w);
    for (int k0 = 0; k0 < K; k0 += kStep, k += kStep) {
        if (k0 + kStep < K) fetch(k + kStep, wn);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < K && m0 + m < M) x = *reinterpret_cast<const float4*>(A + (size_t)(m0 + m) * lda + k);
#pragma unroll
            for (int f = 0; f < F; ++f) {
                float s = acc[m * F + f];
                s = fmaf(x.x, w[f].x, s);
                s = fmaf(x.y, w[f].y, s);
                s = fmaf(x.z, w[f].z, s);
                acc[m * F + f] = fmaf(x.w, w[f].w, s);
            }
        }
#pragma unroll
        for (int f = 0; f < F; ++f) w[f] = wn[f];
    }
    int first = 0;
    LaneSums<V, 16>::run(acc, lane, first);
#pragma unroll
    for (int i = 0; i < kHeld; ++i) sums[warp][first + i] = acc[i];      // (V < 32: lanes with the same sum write the same)
    __syncthreads();
    for (int i = threadIdx.x; i < V; i += kStreamWarps * 32) {
        const int m = m0 + i / F, n = n0 + i % F;
        if (m >= M || n >= N) continue;
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < kStreamWarps; ++j) s += sums[j][i];
        if (bias) s += bias[n];
        C[(size_t)m * ldc + n] = s * out_scale;
    }
}

template <int MT, int F>
int launch_stream(const float* A, long lda, const float* W, const float* bias, float* C, long ldc, int M, int N, int K,
                  float out_scale, cudaStream_t s) {
    dim3 grid((N + F - 1) / F, (M + MT - 1) / MT);
    return launch_pdl_if(M <= kPdlMaxRows, stream_f32_kernel<MT, F>, grid, dim3(kStreamWarps * 32), 0, s, A, lda, W, bias, C,
                         ldc, M, N, K, out_scale);
}

// ---------------------------------------------------------------------------------------------------- many rows
constexpr int kTileN = 64, kTileK = 32, kStages = 2, kRow = kTileK + 4, kPieces = kTileK / 4, kTileThreads = 128;

__device__ __forceinline__ void copy16(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void copy4(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// MI: rows per thread (a tile has 16 * MI).  ALIGNED: rows of A and W start on 16-byte boundaries and K is a multiple of 4.
template <int MI, bool ALIGNED>
__global__ void __launch_bounds__(kTileThreads)
tile_f32_kernel(const float* __restrict__ A, long lda, const float* __restrict__ W, const float* __restrict__ bias,
                float* __restrict__ C, long ldc, int M, int N, int K, float out_scale) {
    constexpr int BM = 16 * MI, kStage = (BM + kTileN) * kRow, kOutRow = kTileN + 4;
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ty = ((lane >> 1) & 3) | ((lane >> 4) << 2), tx = (lane & 1) | (((lane >> 3) & 1) << 1);   // 8 x 4 lanes
    const int row0 = (warp >> 1) * (8 * MI) + ty, col0 = (warp & 1) * 32 + tx;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * kTileN;
    const int parts = gridDim.z, part = blockIdx.z;          // one cluster holds all parts of a tile
    const int steps = (K + kTileK - 1) / kTileK;
    const int lo = (int)((long)steps * part / parts), hi = (int)((long)steps * (part + 1) / parts);

    auto fetch = [&](int step) {
        float* stage = smem + (step - lo) % kStages * kStage;
        const int k0 = step * kTileK;
#pragma unroll
        for (int i = tid; i < (BM + kTileN) * kPieces; i += kTileThreads) {
            const int r = i / kPieces, k = k0 + i % kPieces * 4;
            const bool isA = r < BM;
            const int row = isA ? m0 + r : n0 + r - BM;
            const bool in = row < (isA ? M : N);
            const float* src = isA ? A + (size_t)(in ? row : 0) * lda : W + (size_t)(in ? row : 0) * K;
            float* dst = stage + r * kRow + i % kPieces * 4;
            if (ALIGNED) {
                const bool ok = in && k < K;
                copy16(dst, ok ? src + k : src, ok ? 16 : 0);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const bool ok = in && k + e < K;
                    copy4(dst + e, ok ? src + k + e : src, ok ? 4 : 0);
                }
            }
        }
    };
    unsigned long long acc[MI][8];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) {
        if (lo + s < hi) fetch(lo + s);
        asm volatile("cp.async.commit_group;");
    }
    for (int step = lo; step < hi; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2));
        __syncthreads();                                      // the stage is there, and nobody reads the one filled next
        if (step + kStages - 1 < hi) fetch(step + kStages - 1);
        asm volatile("cp.async.commit_group;");
        const float* a = smem + (step - lo) % kStages * kStage + row0 * kRow;
        const float* w = smem + (step - lo) % kStages * kStage + (BM + col0) * kRow;
#pragma unroll
        for (int k = 0; k < kTileK; k += 4) {
            ulonglong2 av[MI];
#pragma unroll
            for (int i = 0; i < MI; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(a + i * 8 * kRow + k);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(w + j * 4 * kRow + k);
#pragma unroll
                for (int i = 0; i < MI; ++i) fma2(acc[i][j], av[i].x, wv.x);
#pragma unroll
                for (int i = 0; i < MI; ++i) fma2(acc[i][j], av[i].y, wv.y);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;");
    __syncthreads();
    // the tile through shared memory: rows of 64 features go out together, and a cluster's parts meet there
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float even = __uint_as_float((uint32_t)acc[i][j]), odd = __uint_as_float((uint32_t)(acc[i][j] >> 32));
            smem[(row0 + i * 8) * kOutRow + col0 + j * 4] = even + odd;
        }
    const int rows = BM / parts;
    if (parts > 1) cg::this_cluster().sync(); else __syncthreads();
    const bool wide = ((uintptr_t)C & 15) == 0 && ldc % 4 == 0 && n0 + kTileN <= N;
    for (int i = tid; i < rows * (kTileN / 4); i += kTileThreads) {
        const int r = part * rows + i / (kTileN / 4), c = i % (kTileN / 4) * 4;
        const int m = m0 + r, n = n0 + c;
        if (m >= M || n >= N) continue;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int p = 0; p < parts; ++p) {
            const float* tile = parts > 1 ? cg::this_cluster().map_shared_rank(smem, p) : smem;
            const float4 t = *reinterpret_cast<const float4*>(tile + r * kOutRow + c);
            v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
        }
        float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = (o[e] + (bias && n + e < N ? bias[n + e] : 0.f)) * out_scale;
        float* out = C + (size_t)m * ldc + n;
        if (wide) *reinterpret_cast<float4*>(out) = make_float4(o[0], o[1], o[2], o[3]);
        else
            for (int e = 0; e < 4 && n + e < N; ++e) out[e] = o[e];
    }
    if (parts > 1) cg::this_cluster().sync();                 // nobody leaves while another one reads its tile
}

template <int MI, bool ALIGNED>
int launch_tile(const float* A, long lda, const float* W, const float* bias, float* C, long ldc, int M, int N, int K,
                float out_scale, cudaStream_t s) {
    constexpr int BM = 16 * MI, kSms = 148;
    constexpr size_t kRing = (size_t)kStages * (BM + kTileN) * kRow * sizeof(float), kOut = (size_t)BM * (kTileN + 4) * sizeof(float);
    constexpr size_t smem = kRing > kOut ? kRing : kOut;
    static size_t have = 0;
    ensure_dynamic_smem(tile_f32_kernel<MI, ALIGNED>, smem, have);
    const long tiles = (long)((M + BM - 1) / BM) * ((N + kTileN - 1) / kTileN);
    // Parts of K: the time is that of the SM with the most work, ceil(tiles * parts / SMs) / parts tiles, and a part more
    // costs its ring's start and the exchange, about a twentieth of a tile of K = 1,024 (4 % of it measured); no part is
    // shorter than 128 values of k.
    int parts = 1;
    double best = 1e30;
    for (int p = 1; p <= 8 && p * 128 <= (K > 128 ? K : 128); p *= 2) {
        const double cost = (double)((tiles * p + kSms - 1) / kSms) * ((double)K / p + (p > 1 ? 48.0 : 0.0));
        if (cost < best * 0.98) { best = cost; parts = p; }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((N + kTileN - 1) / kTileN, (M + BM - 1) / BM, parts);
    cfg.blockDim = dim3(kTileThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = parts;
    cfg.attrs = attr;
    cfg.numAttrs = parts > 1 ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, tile_f32_kernel<MI, ALIGNED>, A, lda, W, bias, C, ldc, M, N, K, out_scale);
}
}  // namespace

extern "C" int lb_gemm_f32(const float* A, long lda, const float* W, const float* bias, float* C, long ldc, int M,
                           int N, int K, float out_scale, void* stream) {
    if (M <= 0 || N <= 0) return kOk;
    if (K <= 0) return kBadSize;
    cudaStream_t s = (cudaStream_t)stream;
    const bool aligned = K % 4 == 0 && (lda % 4 == 0 || M == 1) && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
    if (aligned && M <= kStreamRows) {
        // 8 features a CTA share the loads of A where that still leaves each SM a CTA and more (2,048 features: 256 CTAs)
        const bool eight = N >= 2048;
        if (M == 1) return eight ? launch_stream<1, 8>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s)
                                 : launch_stream<1, 4>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s);
        if (M == 2) return eight ? launch_stream<2, 8>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s)
                                 : launch_stream<2, 4>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s);
        if (M <= 4) return eight ? launch_stream<4, 8>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s)
                                 : launch_stream<4, 4>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s);
        if (M <= 8) return eight ? launch_stream<8, 8>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s)
                                 : launch_stream<8, 4>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s);
        return launch_stream<16, 4>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s);
    }
    if (M <= 64) return aligned ? launch_tile<4, true>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s)
                                : launch_tile<4, false>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s);
    return aligned ? launch_tile<8, true>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s)
                   : launch_tile<8, false>(A, lda, W, bias, C, ldc, M, N, K, out_scale, s);
}
