// Projections of a decode step with 9 to 64 rows: y[M, N] = x[M, K] W[N, K]^T, bfloat16, on the 5th-generation tensor
// cores with the operands swapped: 128 output features (rows of W) are the M side of the instruction, the batch rows
// (padded to 16, 32, 48 or 64) its N side.
//
// The product is bound by reading W once from HBM.  The few-row kernel in linear_skinny.cu streams W through registers,
// 16 features per CTA, and every CTA reads all of x through L1/L2: at 24 rows that is 1.5 bytes of x per byte of W,
// and it ran at 2.8 TB/s (gate|up of 24,576 x 3,072: 53 us; output head of 130,048 x 3,072: 221 us).  With 128
// features per CTA the x bytes are 0.13 (16 rows) to 0.5 (64 rows) of the W bytes, TMA keeps whole stages of 16 KB of W
// in flight without registers, and the tensor core needs one thread: 33 and 133 us (4.6 and 6.0 TB/s).
//
//   warp 0    one thread issues the TMA loads (128-byte swizzle): W in a box of 128 rows x 64 values of k (for SwiGLU
//             two boxes: the gate rows and the up rows of the same 64 features), x in one box, into a ring of `stages`;
//             the first round of W is asked for before the wait for the kernel before this one (W does not depend on it)
//   warp 1    allocates tensor memory; one thread issues tcgen05.mma (M 128, N rows, K 16) and commits the stages
//   warps 2-9 read the accumulator (a thread is a feature and half of the rows) and push it, four rows per 16-byte store,
//             to the CTA of the cluster that owns those rows
// K split: few tiles of 128 features would leave most SMs idle, so up to 8 CTAs of a cluster each take a range of k and
// the sums meet in distributed shared memory: every CTA owns an equal share of the rows, gets S partial sums for each
// of its values by remote 16-byte stores (one cluster barrier, no loads across the cluster) and adds them in rank
// order, so that the result does not depend on timing.
//
// Epilogues on the float32 sums, the same rounding points as linear_skinny.cu: plain (bias, scale, bfloat16), float32
// out, SwiGLU, and the depthwise conv step of a decode batch on a range of output features.
//
// Every mbarrier wait is bounded; one that gives up records itself in `error`, all roles run out of their own bounded
// waits, every thread still meets the cluster barriers, tensor memory is freed and the kernel returns.
#include "lb200/common.cuh"
#include "lb200/tcgen05.cuh"
using namespace lb200;
using namespace lb200::tc;

namespace {
typedef __nv_bfloat16 bf16;
constexpr int kFeat = 128, kBK = 64;
constexpr int kEpiThreads = 256;                          // warps 2-9
constexpr int kThreads = 64 + kEpiThreads;
constexpr uint32_t kWBytes = kFeat * kBK * 2;
constexpr int kMaxStages = 8;
constexpr int kMaxSplit = 8;

struct RowsArgs {
    const bf16* bias; void* out; long ldo;
    int M, N, K;                                          // N: output features (for SwiGLU: half of W's rows)
    int split, stages, share;                             // CTAs per cluster; ring stages; rows a CTA of the cluster owns
    float out_scale, act_scale;
    // the conv step of a decode batch on features [conv_c0, conv_c1) (see SkinnyArgs in linear_skinny.cu)
    const float* conv_w; const float* conv_b; bf16* conv_state;
    const int* conv_slots; const int* conv_start;
    int conv_c0, conv_c1, conv_k, conv_e0, conv_e1; float conv_s0, conv_s1, conv_s2;
    int* error;
};
enum : int { kPlain = 0, kOutF32 = 1, kSwiglu = 2, kConv = 3 };

__device__ __forceinline__ void report(int* error, int role, int step) {
    if (error != nullptr) atomicCAS(error, 0, 0x10000000 | (role << 24) | ((blockIdx.x & 0xFFF) << 12) | (step & 0xFFF));
}
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t peer_addr(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void store_peer16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// has the phase with this parity completed?  (No waiting: the answer is asked for ahead of the work that precedes its use.)
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return done != 0;
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// NR: batch rows padded to a multiple of 16.
template <int NR, int EPI>
__global__ void __launch_bounds__(kThreads, 2)
linear_rows_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, RowsArgs a) {
    constexpr uint32_t kXBytes = NR * kBK * 2, kStage = kWBytes + kXBytes;
    constexpr uint32_t kTmemCols = NR <= 32 ? 32 : 64;
    constexpr int kOut = EPI == kSwiglu ? 64 : 128;        // output features per tile
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    // the partial sums that land here: [source CTA][group of 4 rows][128 features][4 rows] float32, behind the ring (a
    // peer may be done while this CTA still loads) or, in a cluster of one, over it (the ring is idle by then)
    float* recv = reinterpret_cast<float*>(a.split > 1 ? base + (size_t)a.stages * kStage : base);
    __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], acc_ready;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split = a.split, rank = split > 1 ? (int)cluster_rank() : 0;
    const int tile = blockIdx.x / split, n0 = tile * kOut;
    const int blocks = (a.K + kBK - 1) / kBK;
    const int kb0 = (int)((long)blocks * rank / split), kbn = (int)((long)blocks * (rank + 1) / split) - kb0;
    const int stages = a.stages, first = min(stages, kbn);
    auto load_w = [&](int s, int i) {
        uint8_t* w_tile = base + (size_t)s * kStage;
        mbar_expect_tx(full + s, kStage);
        tma_load_2d(w_tile, &map_w, full + s, (kb0 + i) * kBK, n0);
        if (EPI == kSwiglu) tma_load_2d(w_tile + kWBytes / 2, &map_w, full + s, (kb0 + i) * kBK, a.N + n0);
    };
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        mbar_init(&acc_ready, 1);
        failed = 0;
        mbar_fence_init();
        // this thread loads: its own barriers are ready, so the first round of W need not wait for the others
        for (int i = 0; i < first; ++i) load_w(i, i);
    }
    if (threadIdx.x == 64) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
    if (warp == 1) tmem_alloc<kTmemCols>(&tmem_slot);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_slot;
    pdl_trigger();                                         // the next kernel may start, too: it asks for its weights, and waits for this one
    if (split > 1) cluster_arrive();                       // "this CTA runs": its shared memory may be written to
    pdl_wait();

    // One thread per role runs the loop, so what it waits for on every block of k is the loop's time: a wait on an
    // mbarrier takes some 200 cycles even when the phase is long over.  Both roles therefore ask for the next block's
    // barrier before they work on the current one.
    int issued = 0;
    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < first; ++i)
                tma_load_2d(base + (size_t)i * kStage + kWBytes, &map_x, full + i, (kb0 + i) * kBK, 0);
            issued = first;
            int s = 0;
            uint32_t parity = 0;
            bool ready = false;
            for (; issued < kbn; ++issued) {
                if (!ready && !mbar_wait(empty + s, parity)) { report(a.error, 1, issued); failed = 1; break; }
                const int s1 = s + 1 == stages ? 0 : s + 1;
                const uint32_t parity1 = s1 == 0 ? parity ^ 1 : parity;
                ready = mbar_test(empty + s1, parity1);
                load_w(s, issued);
                tma_load_2d(base + (size_t)s * kStage + kWBytes, &map_x, full + s, (kb0 + issued) * kBK, 0);
                s = s1; parity = parity1;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = umma_idesc(kFeat, NR);
            int s = 0;
            uint32_t parity = 0;
            bool ready = false;
            for (int i = 0; i < kbn; ++i) {
                if (!ready && !mbar_wait(full + s, parity)) { report(a.error, 2, i); failed = 1; break; }
                const int s1 = s + 1 == stages ? 0 : s + 1;
                const uint32_t parity1 = s1 == 0 ? parity ^ 1 : parity;
                ready = i + 1 < kbn && mbar_test(full + s1, parity1);
                fence_after_sync();
                const uint64_t wdesc = umma_desc(base + (size_t)s * kStage), xdesc = umma_desc(base + (size_t)s * kStage + kWBytes);
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k) umma_bf16(tmem, wdesc + 2 * k, xdesc + 2 * k, idesc, (i | k) != 0);
                umma_commit(empty + s);
                s = s1; parity = parity1;
            }
            umma_commit(&acc_ready);
        }
        __syncwarp();
    }
    // What the epilogue reads from global memory is asked for now, under the weight stream: the bias, the conv taps and the
    // windows that this thread's first group of four rows meets (up to four taps).  The epilogue is kept short, nothing in it
    // is unrolled over groups: it runs once per CTA, and its instructions come from memory like the weights (unrolled four
    // times it took 9 us longer with the conv step).
    const int groups = a.share / 4;                        // groups of 4 rows a CTA of the cluster owns
    const int t = (int)threadIdx.x - 64, f = t & (kOut - 1), n = n0 + f;     // an epilogue thread's feature
    constexpr int kTaps = 3;
    unsigned short win[4][kTaps];
    float tap_w[kTaps + 1] = {}, conv_bias = 0.f, bias = 0.f;
    const int c = n - a.conv_c0, C = a.conv_c1 - a.conv_c0, taps = a.conv_k;
    const bool conv = EPI == kConv && t >= 0 && n < a.N && c >= 0 && c < C;
    const int lead = kTaps + 1 - taps;                     // fewer taps lie at the end of the arrays, zeros before them
    auto load_windows = [&](int grp) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int m = rank * a.share + 4 * grp + j;
            const bool live = grp < groups && m < a.M && a.conv_start[m] > 0;
            const unsigned short* st = reinterpret_cast<const unsigned short*>(a.conv_state) + ((size_t)(live ? a.conv_slots[m] : 0) * C + c) * (taps - 1);
#pragma unroll
            for (int i = 0; i < kTaps; ++i) win[j][i] = live && i >= lead ? st[i - lead] : (unsigned short)0;
        }
    };
    if (EPI != kSwiglu && t >= 0 && a.bias != nullptr && n < a.N) bias = __bfloat162float(a.bias[n]);
    if (conv && taps - 1 <= kTaps) {
#pragma unroll
        for (int i = 0; i <= kTaps; ++i) if (i >= lead) tap_w[i] = a.conv_w[(size_t)c * taps + i - lead];
        load_windows(t / kOut);
    }
    if (conv && a.conv_b != nullptr) conv_bias = a.conv_b[c];
    if (warp >= 2) {
        bool ok = mbar_wait(&acc_ready, 0);
        if (!ok && lane == 0) { report(a.error, 3, 0); failed = 1; }
        ok = __all_sync(0xffffffffu, ok);
        fence_after_sync();
    }
    if (split > 1) cluster_wait();
    if (warp >= 2) {
        // a warp may read its own quarter of tensor memory's lanes; warps w and w + 4 share one and take half of the rows each
        constexpr int kHalf = NR / 2;
        const int quarter = warp & 3, feat = quarter * 32 + lane, half = (warp - 2) >> 2;
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16) + half * kHalf;
        const uint32_t mine = smem_u32(recv) + (uint32_t)(rank * groups * kFeat + feat) * 16;
        uint32_t v[kHalf];
#pragma unroll
        for (int c = 0; c < kHalf; c += 8) tmem_ld8(lane_addr + c, v + c);
        tmem_ld_wait();
        const int grp0 = half * (kHalf / 4);
        int owner = grp0 / groups, at_grp = grp0 - owner * groups;
#pragma unroll
        for (int g = 0; g < kHalf / 4; ++g) {
            if (4 * (grp0 + g) < a.M) {
                const uint32_t at = mine + (uint32_t)at_grp * (kFeat * 16);
                if (split > 1) store_peer16(peer_addr(at, owner), v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
                else reinterpret_cast<uint4*>(recv)[(grp0 + g) * kFeat + feat] = make_uint4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
            }
            if (++at_grp == groups) { at_grp = 0; ++owner; }
        }
    }
    fence_before_sync();
    if (split > 1) { cluster_arrive(); cluster_wait(); }
    else __syncthreads();
    if (warp >= 2) {
        const int row0 = rank * a.share;
        constexpr int kStep = kEpiThreads / kOut;          // threads that share a feature's groups of rows
        if (n < a.N) {
#pragma unroll 1
            for (int grp = t / kOut; grp < groups; grp += kStep) {
                const int m0 = row0 + 4 * grp;
                if (m0 >= a.M) break;
                float s[4] = {0.f, 0.f, 0.f, 0.f}, up[4] = {0.f, 0.f, 0.f, 0.f};
                // the partial sums of up to 8 CTAs: all loads first, then the sum in rank order
                float4 v[kMaxSplit], u[EPI == kSwiglu ? kMaxSplit : 1];
#pragma unroll
                for (int src = 0; src < kMaxSplit; ++src)
                    if (src < split) {
                        const float4* p = reinterpret_cast<const float4*>(recv) + (size_t)(src * groups + grp) * kFeat + f;
                        v[src] = p[0];
                        if constexpr (EPI == kSwiglu) u[src] = p[64];
                    }
#pragma unroll
                for (int src = 0; src < kMaxSplit; ++src)
                    if (src < split) {
                        s[0] += v[src].x; s[1] += v[src].y; s[2] += v[src].z; s[3] += v[src].w;
                        if constexpr (EPI == kSwiglu) { up[0] += u[src].x; up[1] += u[src].y; up[2] += u[src].z; up[3] += u[src].w; }
                    }
                if constexpr (EPI == kSwiglu) {
                    // four rows at once, the stores last: rows beyond M are zeros (x is filled up with zeros)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        s[j] = round_to<bf16>(silu_f(round_to<bf16>(round_to<bf16>(s[j]) * a.act_scale))) * round_to<bf16>(up[j]);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (m0 + j < a.M) ((bf16*)a.out)[(size_t)(m0 + j) * a.ldo + n] = __float2bfloat16_rn(s[j]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[j] = round_to<bf16>(s[j] + bias);
                    if (conv) {
                        const float scale = c < a.conv_e0 ? a.conv_s0 : (c < a.conv_e1 ? a.conv_s1 : a.conv_s2);
                        float acc[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) s[j] = round_to<bf16>(s[j] * scale);
                        if (taps - 1 <= kTaps) {
                            if (grp >= kStep) load_windows(grp);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                float old[kTaps];
#pragma unroll
                                for (int i = 0; i < kTaps; ++i) old[i] = __uint_as_float((unsigned)win[j][i] << 16);
                                acc[j] = tap_w[kTaps] * s[j];
#pragma unroll
                                for (int i = 0; i < kTaps; ++i) acc[j] += tap_w[i] * old[i];
                                if (m0 + j < a.M) {
                                    bf16* st = a.conv_state + ((size_t)a.conv_slots[m0 + j] * C + c) * (taps - 1) - lead;
#pragma unroll
                                    for (int i = 0; i < kTaps; ++i)
                                        if (i >= lead) st[i] = __float2bfloat16_rn(i + 1 < kTaps ? old[i + 1] : s[j]);
                                }
                            }
                        } else {
#pragma unroll 1
                            for (int j = 0; j < 4; ++j) {
                                const int m = min(m0 + j, a.M - 1);
                                bf16* st = a.conv_state + ((size_t)a.conv_slots[m] * C + c) * (taps - 1);
                                float mine = j == 0 ? s[0] : j == 1 ? s[1] : j == 2 ? s[2] : s[3];
                                float sum = a.conv_w[(size_t)c * taps + taps - 1] * mine;
#pragma unroll 1
                                for (int i = 0; i < taps - 1; ++i) {
                                    const float old = a.conv_start[m] > 0 ? __bfloat162float(st[i]) : 0.f;
                                    sum += a.conv_w[(size_t)c * taps + i] * old;
                                    if (i > 0 && m0 + j < a.M) st[i - 1] = __float2bfloat16_rn(old);
                                }
                                if (m0 + j < a.M) st[taps - 2] = __float2bfloat16_rn(mine);
#pragma unroll
                                for (int e = 0; e < 4; ++e) if (e == j) acc[e] = sum;
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) s[j] = round_to<bf16>(silu_f(round_to<bf16>(acc[j] + conv_bias)));
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const size_t at = (size_t)(m0 + j) * a.ldo + n;
                        if (m0 + j < a.M) {
                            if (EPI == kOutF32) ((float*)a.out)[at] = s[j] * a.out_scale;
                            else ((bf16*)a.out)[at] = __float2bfloat16_rn(a.out_scale == 1.f ? s[j] : s[j] * a.out_scale);
                        }
                    }
                }
            }
        }
    }
    __syncthreads();
    if (failed && threadIdx.x == 0)                        // copies still under way land before the CTA leaves
        for (int i = max(0, issued - stages); i < issued; ++i) mbar_wait(full + i % stages, (i / stages) & 1);
    if (warp == 1) tmem_free<kTmemCols>(tmem);
}

template <int NR, int EPI>
int launch(const CUtensorMap& map_w, const CUtensorMap& map_x, RowsArgs a, int tiles, cudaStream_t s) {
    constexpr size_t kStage = kWBytes + (size_t)NR * kBK * 2;
    const int blocks = (a.K + kBK - 1) / kBK, per = (blocks + a.split - 1) / a.split;
    a.share = ((NR + a.split - 1) / a.split + 3) / 4 * 4;
    const size_t recv = (size_t)a.split * a.share * kFeat * 4;
    // two CTAs per SM: 113 KB each, the sums that land from the cluster's other CTAs included
    constexpr size_t kBudget = 112 * 1024;
    int stages = (int)((kBudget - 1024 - (a.split > 1 ? recv : 0)) / kStage);
    stages = stages < per ? stages : per;
    stages = stages < kMaxStages ? stages : kMaxStages;
    if (stages < 1) return kTooLarge;
    a.stages = stages;
    size_t smem = 1024 + stages * kStage + (a.split > 1 ? recv : 0);
    if (a.split == 1 && smem < 1024 + recv) smem = 1024 + recv;
    static size_t have = 0;
    ensure_dynamic_smem(linear_rows_tc_kernel<NR, EPI>, smem, have);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * a.split)); cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = smem; cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)a.split; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = a.split > 1 ? 2 : 1;
    const int rc = (int)cudaLaunchKernelEx(&cfg, linear_rows_tc_kernel<NR, EPI>, map_w, map_x, a);
    return rc != 0 ? rc : launch_status();
}

template <int EPI>
int launch_rows(const CUtensorMap& map_w, const CUtensorMap& map_x, const RowsArgs& a, int tiles, cudaStream_t s) {
    if (a.M <= 16) return launch<16, EPI>(map_w, map_x, a, tiles, s);
    if (a.M <= 32) return launch<32, EPI>(map_w, map_x, a, tiles, s);
    if (a.M <= 48) return launch<48, EPI>(map_w, map_x, a, tiles, s);
    return launch<64, EPI>(map_w, map_x, a, tiles, s);
}

// CTAs that share a tile's k.  Every doubling halves a CTA's stream and costs a larger exchange: it pays up to about one
// CTA per SM as long as two blocks of k are left to each, and up to two per SM only with five blocks or more.  Measured
// back to back (13 and 64 rows, weights from HBM, us for a split of 2 / 4 / 8): 768 x 1,024 4.6 / 3.4 / 3.1 and 7.3 / 5.1 /
// 4.2; 3,352 x 1,024 (27 tiles, 16 blocks) 4.8 / 4.6 / 4.9 and 7.7 / 5.5 / 6.5; gate|up 6,144 x 1,280 (48 tiles, 20 blocks)
// 6.9 / 6.2 / 6.4 and 10.0 / 8.2 / 11.9; 3,072 x 12,288 32.1 / 19.7 / 15.2 and 40.6 / 23.7 / 17.3.
int default_split(int tiles, int blocks) {
    int split = 1;
    while (split < kMaxSplit) {
        const long ctas = 2L * tiles * split;
        const int left = blocks / (2 * split);
        if (!((ctas <= 160 && left >= 2) || (ctas <= 296 && left >= 5))) break;
        split *= 2;
    }
    return split;
}
}  // namespace

// x: [M, K] bfloat16 rows (row stride ldx, a multiple of 8 elements, 16-byte aligned base), M <= 64; w: [N, K] bfloat16
// contiguous, 16-byte aligned ([2N, K] for the SwiGLU epilogue: gate rows, then up rows); K a multiple of 8.  epilogue: 0
// plain (bfloat16 out), 1 float32 out, 2 SwiGLU, 3 plain with the conv step on features [c0, c1).  conv_w: float32
// [c1 - c0, taps]; conv_b: float32 [c1 - c0] or null; conv_state: bfloat16 [slots, c1 - c0, taps - 1], updated in place;
// slots / start: int32 per row.  `error`: a device int that is 0 before the call; non-zero afterwards: a wait gave up.
extern "C" int lb_linear_rows_tc(const void* x, long ldx, const void* w, const void* bias, void* out, long ldo, int M, int N,
                                 int K, float out_scale, float act_scale, int epilogue, const float* conv_w,
                                 const float* conv_b, void* conv_state, const int* slots, const int* start, int c0, int c1,
                                 int taps, int e0, int e1, float s0, float s1, float s2, int* error, void* stream) {
    if (M <= 0 || N <= 0) return kOk;
    if (K <= 0 || K % 8 || ldx % 8 || epilogue < 0 || epilogue > 3) return kBadSize;
    if (M > 64) return kTooLarge;
    if (((uintptr_t)x | (uintptr_t)w) & 15) return kBadSize;
    if (epilogue == kConv && (taps < 2 || taps > 8 || c0 < 0 || c1 > N || c0 > c1)) return kBadSize;
    CUtensorMap map_w, map_x;
    const int nr = M <= 16 ? 16 : M <= 32 ? 32 : M <= 48 ? 48 : 64;
    int rc = make_tile_map(&map_w, w, epilogue == kSwiglu ? 2L * N : N, K, K, epilogue == kSwiglu ? 64 : kFeat);
    if (rc == 0) rc = make_tile_map(&map_x, x, M, K, ldx, nr);
    if (rc != 0) return rc;
    RowsArgs a{};
    a.bias = (const bf16*)bias; a.out = out; a.ldo = ldo; a.M = M; a.N = N; a.K = K;
    a.out_scale = out_scale; a.act_scale = act_scale; a.error = error;
    a.conv_w = conv_w; a.conv_b = conv_b; a.conv_state = (bf16*)conv_state; a.conv_slots = slots; a.conv_start = start;
    a.conv_c0 = c0; a.conv_c1 = c1; a.conv_k = taps; a.conv_e0 = e0; a.conv_e1 = e1;
    a.conv_s0 = s0; a.conv_s1 = s1; a.conv_s2 = s2;
    const int out_feat = epilogue == kSwiglu ? 64 : 128, tiles = (N + out_feat - 1) / out_feat;
    a.split = default_split(tiles, (K + kBK - 1) / kBK);
    if ((long)tiles * a.split > 0x7fffffffL) return kTooLarge;
    cudaStream_t s = (cudaStream_t)stream;
    switch (epilogue) {
        case kPlain: return launch_rows<kPlain>(map_w, map_x, a, tiles, s);
        case kOutF32: return launch_rows<kOutF32>(map_w, map_x, a, tiles, s);
        case kSwiglu: return launch_rows<kSwiglu>(map_w, map_x, a, tiles, s);
        default: return launch_rows<kConv>(map_w, map_x, a, tiles, s);
    }
}
