// A decode step's layers as ONE persistent kernel (bfloat16, up to 16 rows): every layer is a pre-norm block with attention and
// a Mamba2 mixer side by side on the same normed rows and a gated feed-forward behind them.
//
// What bounds such a step is not bytes but the chain of dependent kernels (0.5B-class sizes at 8 rows: 7 us of bytes a layer,
// 35 us of chain: a launch, an L2 round trip for the rows, another for the weights' first bytes, a reduction, a store, five
// times a layer).  Here the grid is one CTA per SM for the whole step, a layer is five phases with a grid-wide barrier between
// them, and what does not depend on the phase before is on its way long before it:
//   1  q|k|v and the mixer's in-projection as one product over the normed rows; epilogues: rotation and cache store, conv step
//   2  attention over the pages (half of the warps) beside the state update (the other half)
//   3  both out-projections as one product; epilogue: their scaled sum joins the residual, sums of squares for the norm
//   4  gate|up over the normed rows; epilogue: SwiGLU
//   5  down-projection; epilogue: joins the residual, sums of squares for the next layer's norm
// * Weights: a warp of its own streams the CTA's rows of all phases and layers, in the order of their use, through one ring of
//   shared memory (bulk copies; a full and an empty mbarrier per batch of tiles).  It never meets a grid barrier, so the memory
//   system works through the barriers; the ring holds 150 KB per SM, most of a layer of 0.5B-class size.
// * Products: a tile is 8 output features (the 8 columns of mma.sync m16n8k16) against all rows; the 8 consumer warps split k.
//   Rows come from L2 straight into registers, 16 bytes a lane; the order of k inside an instruction is free as long as both
//   operands agree.  Tiles go round the CTAs from where the phase before stopped, so that all CTAs stream about the same bytes.
// * A norm is a factor per row and a weight per column: the phase that makes the rows writes them times the next norm's weight,
//   rounded to bfloat16, with sums of squares per 8 columns; the consumer multiplies its float32 sums by the row's factor.
//   (One rounding, as in the chain of kernels, which rounds once more where a mixer has an input multiplier.)
// * Phase 2 splits keys (16 of them a tile) and rows of the state evenly over all CTAs, whatever the contexts' lengths; the
//   first keys, values and states are requested before the barrier in front of it.  A request's share that several CTAs hold is
//   merged by the last of them to finish.
// Rounding points otherwise as in the chain of kernels: where the reference's bfloat16 engine stores an activation.
//
// Measured (whole steps with a small head, 36 layers of 0.5B-class sizes, 2,048 keys; the chain of kernels / this): 1 row 1,007 / 881 us, 4
// rows 1,155 / 934, 8 rows 1,188 / 1,017, 12 rows 1,363 / 1,189; 16 layers of 1.5B-Deep size 637 / 538 and 780 / 674 us at 1 and 8
// rows.  A layer is 44,000 cycles at 1 row: five barriers of 2,500 (the release of a CTA's stores, an atomic, a poll) and as much again of waiting for the slowest CTA,
// four products of 1,000 cycles of L2 latency and 1,200 of instructions, 8,000 of attention and merge.  What counts is instructions
// on the way from barrier to barrier: a warp issues one in 9 cycles here (two warps a scheduler, each thing done once a layer).
// Tried and slower: 16 consumer warps (96 registers, spills), sums kept across pieces of k with predicated loads (two more copies of
// everything: 3,400 instead of 2,200 cycles a product), polling by a consumer warp, fences beside the release, 16 partial results at
// a time in the merge, asking for keys and states at the start of phase 1 instead of three phases ahead.
//
// The grid is launched cooperatively (its CTAs wait on one another); every wait is bounded, and one that gives up records
// itself in the error word and ends the kernel, its own copies landed.
#include "lb200/common.cuh"
#include "lb200/tcgen05.cuh"
using namespace lb200;

namespace {
typedef __nv_bfloat16 bf16;
constexpr int kWarps = 8;                                // consumer warps
constexpr int kThreads = kWarps * 32, kBlock = kThreads + 128;      // and a group of four: one streams the weights, one keeps the barrier
constexpr int kAttnWarps = 4;                            // consumer warps that do the attention in phase 2; the others update states
// 168 registers a thread at launch; the last group keeps 40, the other two take 232: 2 x 232 + 40 = 3 x 168
constexpr int kRegsStream = 40, kRegsWork = 232;
constexpr int kTiles = 6;                                // feature tiles of a CTA that are accumulated together
constexpr int kMaxRows = 16, kMaxLayers = 64;
constexpr int kBatches = 16;                             // batches of tiles that may be in the ring
constexpr int kKeys = 16;                                // keys of an attention tile
constexpr int kMerge = 8;                                // partial results whose loads are in flight together
constexpr int kKvBytes = 64 * 1024;                      // the attention warps' ring
constexpr uint32_t kBarrierSpins = 1u << 21;             // polls of a grid barrier before a wait gives up (about a second)

struct LayerPointers {
    const bf16 *qkv_w, *in_w, *o_w, *out_w, *gate_up_w, *down_w;
    const float *conv_w, *conv_b, *a_log, *dt_bias, *d_skip;
    const float *ff_norm, *next_norm;                    // next_norm: null behind the last layer of the model
    bf16 *conv_state, *k_cache, *v_cache;
    void* ssm_state;
    const int *block_table, *slot_mapping;
    int bt_stride, pad;
};
struct alignas(64) LayerArgs { CUtensorMap map_k, map_v; LayerPointers p; };

struct StepArgs {
    int M, H, Hq, Hkv, page_size, inner, nh, P, N, groups, C, taps, conv_e0, conv_e1, inter, table_rows, state_bf16;
    float conv_s0, conv_s1, conv_s2, dt_scale, gate_scale, attn_in, ssm_in, attn_out, ssm_out, key_scale, sm_scale, act_scale, ff_scale;
    float eps_mixer, eps_ff;
    const float* cos_sin;
    const int *positions, *slots, *start_pos;
    const bf16* x; const float* first_norm;
    bf16 *xn, *res_a, *res_b, *x_out;                    // rows x norm weight; residual after the mixers / after the feed-forward
    float* ssq;                                          // [M][H / 8] sums of squares
    bf16 *qkv, *proj, *o, *y, *h;                        // [M][...]
    float* part;                                         // [CTAs][8 heads][HD + 2]
    int *counters; unsigned* barrier; int* error;
    int layers, ring, page_shift;                        // ring: its bytes; page_shift: log2 of a page's key tiles
    uint32_t barrier_polls, key_polls, weight_polls;     // polls of a grid barrier, a key tile's copy, a batch of weights before the wait gives up
};
struct Launch { StepArgs s; LayerArgs layer[kMaxLayers]; };

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float low_f(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float high_f(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ float rnd(float v) { return round_to<bf16>(v); }
// what another SM has written comes past L1
__device__ __forceinline__ uint4 ld_cg16(const void* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ uint2 ld_cg8(const void* p) { return __ldcg(reinterpret_cast<const uint2*>(p)); }
__device__ __forceinline__ uint32_t ld_cg4(const void* p) { return __ldcg(reinterpret_cast<const uint32_t*>(p)); }
__device__ __forceinline__ float ld_cg_bf16(const bf16* p) {
    return __uint_as_float((uint32_t)__ldcg(reinterpret_cast<const unsigned short*>(p)) << 16);
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void prefetch_l2_bulk(const void* p, int bytes) {       // 16-byte boundaries
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void prefetch_l2_tile(const CUtensorMap* map, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// false: the phase did not complete within so many polls
__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity, uint32_t polls) {
    for (; polls != 0; --polls) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
// The thread's index, read anew: what a phase derives from it stays the phase's own.  Derived once, the compiler keeps rows, columns
// and addresses of every phase in registers through the whole layer loop, and spills.
__device__ __forceinline__ int thread_now() {
    int tid;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    return tid;
}
template <int THREADS, int ID> __device__ __forceinline__ void named_sync() { asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(THREADS) : "memory"); }

// the distance of a tile's 8 rows of 256 n values in the ring: 64 bytes off a multiple of 128, so that the 16-byte reads of 8 lanes
// (2 rows x 4 pieces) meet all banks once
__host__ __device__ constexpr int row_pitch(int n) { return n * 512 + 64; }

// k in pieces of `n` units of 256 (32 values of k for each warp), at most `most`, the last one what is left
struct Runs { int pieces, n, units; };
__host__ __device__ __forceinline__ Runs runs_of(int K, int most) {
    Runs r;
    r.units = K / 256;
    r.pieces = (r.units + most - 1) / most;
    r.n = (r.units + r.pieces - 1) / r.pieces;
    r.pieces = (r.units + r.n - 1) / r.n;
    return r;
}

// the feature tiles of the first product: where q, k, v, then gate z, conv x|B|C, dt end
struct InTiles { int q, k, v, z, c, all; };
__host__ __device__ __forceinline__ InTiles in_tiles(const StepArgs& s, int hd) {
    InTiles t;
    t.q = s.Hq * hd / 8;
    t.k = t.q + s.Hkv * hd / 8;
    t.v = t.k + s.Hkv * hd / 8;
    t.z = t.v + s.inner / 8;
    t.c = t.z + s.C / 8;
    t.all = t.c + (s.nh + 7) / 8;
    return t;
}

// ROWS: 8 or 16.  HD: head size of the attention.
template <int ROWS, int HD>
struct Shape {
    static constexpr int GROUPS = ROWS == 8 ? 6 : 4;     // units of k in a piece: what two pieces' rows have registers for
    static constexpr int SUMS = kTiles * kWarps * ROWS * 8 * 4, MERGE = kAttnWarps * 8 * (HD + 2) * 4;
    static constexpr int RED = ((SUMS > MERGE ? SUMS : MERGE) + 1023) / 1024 * 1024;
};

// What the warps of a CTA share, at the start of its dynamic shared memory.
struct Shared {
    StepArgs s;
    LayerPointers a;                                     // the layer's arguments, for phase 2
    int pos[kMaxRows], slot[kMaxRows], start[kMaxRows];
    float factor[kMaxRows];                              // the norm's factor of a row
    int last, dead, go, epoch;                           // epoch: grid barriers passed, for the prefetching warp
    Runs run_h, run_o, run_y, run_f;                     // how k is cut in the four kinds of product
    InTiles in;
    struct { int n, first, per; } share[4];              // the CTA's tiles in them: first + i * CTAs, in passes of `per`
    int row, head, tile0, tile1, first_cta, shares;      // phase 2: key tiles [tile0, tile1) of this row and key/value head are the CTA's, one
                                                         // of `shares` neighbouring CTAs that share them (row below zero: none are)
    int quads, quad_per;                                 // ... and quad_per quads of state rows each warp's
    int kv_count[kAttnWarps];                            // tiles that passed through an attention warp's ring
    int batch_bytes[kBatches];                           // the streaming warp's book of the ring
    alignas(8) uint64_t full[kBatches], empty[kBatches], kv_full[kAttnWarps][4];
};
extern __shared__ __align__(16) unsigned char smem_dyn[];
__device__ __forceinline__ Shared& shared() { return *reinterpret_cast<Shared*>(smem_dyn); }
constexpr int kSharedBytes = (sizeof(Shared) + 1023) / 1024 * 1024;
// behind it, on a 1024-byte boundary: the attention warps' ring, the sums, the weights' ring
__device__ __forceinline__ unsigned char* smem_rings() { return smem_dyn + kSharedBytes + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u); }
__device__ __forceinline__ float* smem_sums() { return reinterpret_cast<float*>(smem_rings() + kKvBytes); }

__device__ __forceinline__ void give_up(int role, int epoch) {
    Shared& sh = shared();
    sh.dead = 1;
    if (sh.s.error != nullptr) atomicCAS(sh.s.error, 0, (role << 24) | ((blockIdx.x & 0xFFF) << 12) | (epoch & 0xFFF));
}
// The streaming warp's wait for room in the ring, as one.  False, and the warp asks for nothing more: the limit, or its CTA gave up
// (whose consumers then release batches whose copies may not have landed).
__device__ __forceinline__ bool wait_for_room(uint64_t* bar, uint32_t parity, int epoch) {
    Shared& sh = shared();
    bool ok = false;
    for (uint32_t left = sh.s.weight_polls; left != 0 && !ok && *(volatile int*)&sh.dead == 0; --left) ok = wait_for(bar, parity, 1);
    ok = __all_sync(0xffffffffu, ok && *(volatile int*)&sh.dead == 0);
    if (!ok && (threadIdx.x & 31) == 0) give_up(0x35, epoch);
    return ok;
}
// The grid barrier.  `arrive`: every thread's writes so far become visible to the grid; nobody waits.  `meet` waits for all CTAs and
// says whether the step goes on (one thread decides for all of its CTA: a wait elsewhere may give up while others read the
// decision).  Between them stands a warp of its own, which waits for the CTA's threads, counts the CTA in and polls: 1.3 us for 148
// CTAs, under which the others look up their next phase's operands.
__device__ __forceinline__ void arrive(int& epoch) {
    asm volatile("bar.arrive 1, %0;" ::"n"(kThreads + 32) : "memory");
    ++epoch;
}
__device__ __forceinline__ bool meet() {
    named_sync<kThreads + 32, 3>();
    return *(volatile int*)&shared().go != 0;
}
__device__ __forceinline__ void keep_barrier(const StepArgs& s, int epochs) {
    Shared& sh = shared();
    for (int epoch = 1; epoch <= epochs; ++epoch) {
        named_sync<kThreads + 32, 1>();
        if ((threadIdx.x & 31) == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(s.barrier) : "memory");
            const unsigned want = epoch * gridDim.x;
            for (uint32_t spin = 0; *(volatile int*)&sh.dead == 0; ++spin) {
                unsigned have;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(have) : "l"(s.barrier) : "memory");
                if (have >= want) break;
                if (spin >= s.barrier_polls) give_up(0x32, epoch);
            }
            *(volatile int*)&sh.go = *(volatile int*)&sh.dead == 0;
            *(volatile int*)&sh.epoch = epoch;
        }
        __syncwarp();
        named_sync<kThreads + 32, 3>();
        if (*(volatile int*)&sh.go == 0) return;
    }
}

// A warp of its own asks for the states, keys and values that the CTA's phase 2 will read, into L2, three phases ahead: the memory
// system has little to do under phases 3 to 5, and phase 2 reads most of a layer's bytes at 8 rows.  `pass`: grid barriers that the
// layer's turn comes after.
template <int HD, int QUAD>
__device__ __forceinline__ void ask_ahead(const LayerArgs& layer, int pass) {
    const LayerPointers& a = layer.p;
    Shared& sh = shared();
    const StepArgs& s = sh.s;
    const int lane = threadIdx.x & 31;
    for (uint32_t spin = 0; *(volatile int*)&sh.epoch < pass && spin < kBarrierSpins; ++spin) {
        if (*(volatile int*)&sh.go == 0) return;
        __nanosleep(100);
    }
    const int q0 = blockIdx.x * (kWarps - kAttnWarps) * sh.quad_per, q1 = min(sh.quads, q0 + (kWarps - kAttnWarps) * sh.quad_per), per = s.nh * s.P / 4;
    for (int q = q0 + lane; q < q1; q += 32) {
        const int m = q / per;
        if (sh.start[m] > 0) prefetch_l2_bulk((const unsigned char*)a.ssm_state + ((size_t)sh.slot[m] * per + q - m * per) * QUAD, QUAD);
    }
    if (sh.row >= 0) {
        const int* table = a.block_table + (size_t)sh.row * a.bt_stride;
        for (int x = sh.tile0 + lane; x < sh.tile1; x += 32) {        // a lane per tile
            const int row = __ldg(table + (x >> s.page_shift)) * s.page_size + (x & ((1 << s.page_shift) - 1)) * kKeys;
#pragma unroll
            for (int blk = 0; blk < HD / 64; ++blk) {
                prefetch_l2_tile(&layer.map_k, sh.head * HD + blk * 64, row);
                prefetch_l2_tile(&layer.map_v, sh.head * HD + blk * 64, row);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------ phase 2: attention
// The first warps of a CTA take every fourth one of its key tiles each; the first ones are asked for before the grid barrier in front
// of the phase.
template <int HD>
__device__ __forceinline__ bool attend(const CUtensorMap* map_k, const CUtensorMap* map_v, int epoch) {
    constexpr int AW = kAttnWarps, TILE = kKeys * HD * 2, NS = kKvBytes / (AW * 2 * TILE), LD = HD + 2;       // TILE: bytes of a tile's keys
    static_assert(NS <= 4, "as many barriers as stages");
    Shared& sh = shared();
    const StepArgs& s = sh.s;
    const int tid = thread_now(), warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, sw = lane & 7, mi = lane >> 3;
    const int b = sh.row, kvh = sh.head, tile1 = sh.tile1;
    const int Hkv = s.Hkv, G = s.Hq / Hkv, qkv_ld = (s.Hq + 2 * Hkv) * HD;
    float* red = smem_sums();
    bf16* mine = reinterpret_cast<bf16*>(smem_rings()) + (size_t)warp * NS * TILE;       // a stage: TILE bytes of keys, as many of values
    uint32_t used = sh.kv_count[warp], issued = used;
    int ahead = b < 0 ? tile1 : sh.tile0 + warp;
    const int* table = sh.a.block_table + (size_t)max(b, 0) * sh.a.bt_stride;
    const int in_page = (1 << s.page_shift) - 1;
    // the pages of the warp's next 32 tiles, one per lane: a look-up in front of each request would wait for the table every time
    int page_l = 0, asked = 0;
    auto look_up = [&]() {
        const int x = ahead + lane * AW;
        page_l = x < tile1 ? __ldg(table + (x >> s.page_shift)) : 0;
    };
    look_up();
    auto request = [&]() {                               // tile `ahead` into the next stage
        if (asked == 32) { look_up(); asked = 0; }
        const int page = __shfl_sync(0xffffffffu, page_l, asked++);
        if (lane == 0) {
            const int row = page * s.page_size + (ahead & in_page) * kKeys;
            const int st = issued % NS;
            bf16* kd = mine + (size_t)st * TILE;
            tc::mbar_expect_tx(&sh.kv_full[warp][st], 2 * TILE);
#pragma unroll
            for (int blk = 0; blk < HD / 64; ++blk) {
                tc::tma_load_2d(kd + blk * (kKeys * 64), map_k, &sh.kv_full[warp][st], kvh * HD + blk * 64, row);
                tc::tma_load_2d(kd + TILE / 2 + blk * (kKeys * 64), map_v, &sh.kv_full[warp][st], kvh * HD + blk * 64, row);
            }
        }
        ++issued;
        ahead += AW;
    };
#pragma unroll 1
    for (int p = 0; p < NS; ++p)
        if (ahead < tile1) request();
    const float scale_log2 = s.sm_scale * 1.4426950408889634f;
    const int pos = sh.pos[max(b, 0)], r = pos % kKeys, last_tile = pos / kKeys;
    const bf16* qp = s.qkv + (size_t)max(b, 0) * qkv_ld;
    const int piece = lane % (HD / 8);
    const bool value = lane >= HD / 8;
    const bf16* own_row = qp + (s.Hq + (value ? Hkv : 0) + kvh) * HD + piece * 8;
    const int shares = sh.shares, first_cta = sh.first_cta;
    qp += (kvh * G + min(g, G - 1)) * HD + 2 * t;        // (rows of the tile beyond the group: its last head again)
    int x = sh.tile0 + warp;
    const bool alive = meet();
    if (alive && b >= 0) {
        float o[HD / 8][2], mx = -INFINITY, sum = 0.f;
#pragma unroll
        for (int i = 0; i < HD / 8; ++i) o[i][0] = o[i][1] = 0.f;
        if (x < tile1) {
            uint32_t qa[HD / 16][2];
#pragma unroll
            for (int kk = 0; kk < HD / 16; ++kk) {
                qa[kk][0] = ld_cg4(qp + kk * 16);
                qa[kk][1] = ld_cg4(qp + kk * 16 + 8);
            }
#pragma unroll 1
            for (; x < tile1; x += AW) {
                const bool own = x == last_tile;         // the tile of the token's own key, which phase 1 has just made
                uint4 fresh = make_uint4(0u, 0u, 0u, 0u);
                if (own && lane < HD / 4) fresh = ld_cg16(own_row);
                const int st = used % NS;
                // the warp gives up as one, and the tile stays among those that the wait at the end is for
                if (!__all_sync(0xffffffffu, wait_for(&sh.kv_full[warp][st], (used / NS) & 1, s.key_polls))) {
                    if (lane == 0) give_up(0x34, epoch);
                    break;
                }
                bf16* kb = mine + (size_t)st * TILE;
                bf16* vb = kb + TILE / 2;
                if (own) {
                    if (lane < HD / 4)
                        *reinterpret_cast<uint4*>((value ? vb : kb) + (piece >> 3) * (kKeys * 64) + r * 64 + (((piece & 7) ^ (r & 7)) << 3)) = fresh;
                    // rows of the page beyond hold anything: their values must not meet the zero weights as NaN or infinity
                    for (int i = lane; i < (kKeys - 1 - r) * (HD / 8); i += 32) {
                        const int rr = r + 1 + i / (HD / 8), c = i % (HD / 8);
                        *reinterpret_cast<uint4*>(vb + (c >> 3) * (kKeys * 64) + rr * 64 + (c & 7) * 8) = make_uint4(0u, 0u, 0u, 0u);
                    }
                    __syncwarp();
                }
                float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int kk = 0; kk < HD / 16; ++kk) {
                    uint32_t kf[4];
                    ldsm_x4(kf, kb + (kk >> 2) * (kKeys * 64) + ((mi >> 1) * 8 + sw) * 64 + ((((kk & 3) * 2 + (mi & 1)) ^ sw) << 3));
                    mma_bf16(s0, qa[kk][0], 0u, qa[kk][1], 0u, kf[0], kf[1]);
                    mma_bf16(s1, qa[kk][0], 0u, qa[kk][1], 0u, kf[2], kf[3]);
                }
                if (own) {
                    if (2 * t > r) s0[0] = -INFINITY;
                    if (2 * t + 1 > r) s0[1] = -INFINITY;
                    if (8 + 2 * t > r) s1[0] = -INFINITY;
                    if (9 + 2 * t > r) s1[1] = -INFINITY;
                }
                float top = fmaxf(fmaxf(s0[0], s0[1]), fmaxf(s1[0], s1[1]));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
                top = fmaxf(mx, top * scale_log2);
                if (__any_sync(0xffffffffu, top > mx)) {
                    const float alpha = tc::ex2_approx(mx - top);
                    mx = top;
                    sum *= alpha;
#pragma unroll
                    for (int i = 0; i < HD / 8; ++i) { o[i][0] *= alpha; o[i][1] *= alpha; }
                }
                const float e0 = tc::ex2_approx(fmaf(s0[0], scale_log2, -mx)), e1 = tc::ex2_approx(fmaf(s0[1], scale_log2, -mx));
                const float e2 = tc::ex2_approx(fmaf(s1[0], scale_log2, -mx)), e3 = tc::ex2_approx(fmaf(s1[1], scale_log2, -mx));
                sum += (e0 + e1) + (e2 + e3);
                const uint32_t p0 = pack_bf16(e0, e1), p1 = pack_bf16(e2, e3);
#pragma unroll
                for (int d2 = 0; d2 < HD / 16; ++d2) {
                    uint32_t vf[4];
                    ldsm_x4_t(vf, vb + (d2 >> 2) * (kKeys * 64) + ((mi & 1) * 8 + sw) * 64 + ((((d2 & 3) * 2 + (mi >> 1)) ^ sw) << 3));
                    float c0[4] = {o[2 * d2][0], o[2 * d2][1], 0.f, 0.f}, c1[4] = {o[2 * d2 + 1][0], o[2 * d2 + 1][1], 0.f, 0.f};
                    mma_bf16(c0, p0, 0u, p1, 0u, vf[0], vf[1]);
                    mma_bf16(c1, p0, 0u, p1, 0u, vf[2], vf[3]);
                    o[2 * d2][0] = c0[0]; o[2 * d2][1] = c0[1];
                    o[2 * d2 + 1][0] = c1[0]; o[2 * d2 + 1][1] = c1[1];
                }
                ++used;
                if (own) tc::fence_async_smem();         // this thread's writes to the stage, before the next copy into it
                __syncwarp();
                if (ahead < tile1) request();
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        }
        // the warps' partial results of this (row, key/value head) meet in shared memory
        float* part = red + (size_t)(warp * 8 + g) * LD;
#pragma unroll
        for (int i = 0; i < HD / 8; ++i) *reinterpret_cast<float2*>(part + i * 8 + 2 * t) = make_float2(o[i][0], o[i][1]);
        if (t == 0) *reinterpret_cast<float2*>(part + HD) = make_float2(mx, sum);
        named_sync<AW * 32, 2>();
        const int task = b * Hkv + kvh;
        bf16* out = s.o + (size_t)b * s.Hq * HD + kvh * G * HD;
#pragma unroll 1
        for (int e = tid; e < G * HD / 2; e += AW * 32) {
            const int hg = e / (HD / 2), d = e % (HD / 2) * 2;
            float2 ml[AW], os = make_float2(0.f, 0.f);
            float top = -INFINITY, ls = 0.f;
#pragma unroll
            for (int w = 0; w < AW; ++w) { ml[w] = *reinterpret_cast<const float2*>(red + (w * 8 + hg) * LD + HD); top = fmaxf(top, ml[w].x); }
#pragma unroll
            for (int w = 0; w < AW; ++w) {
                const float f = tc::ex2_approx(ml[w].x - top);
                const float2 v = *reinterpret_cast<const float2*>(red + (w * 8 + hg) * LD + d);
                ls += ml[w].y * f;
                os.x += v.x * f; os.y += v.y * f;
            }
            if (shares == 1) *reinterpret_cast<uint32_t*>(out + 2 * e) = pack_bf16(os.x / ls, os.y / ls);
            else {
                float* p = s.part + ((size_t)blockIdx.x * 8 + hg) * LD;
                *reinterpret_cast<float2*>(p + d) = os;
                if (d == 0) *reinterpret_cast<float2*>(p + HD) = make_float2(top, ls);
            }
        }
        if (shares > 1) {
            named_sync<AW * 32, 2>();
            if (tid == 0) {
                int before;
                asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(before) : "l"(s.counters + task) : "memory");
                *(volatile int*)&sh.last = before == shares - 1;
                if (before == shares - 1) s.counters[task] = 0;            // for the next layer
            }
            named_sync<AW * 32, 2>();
            if (*(volatile int*)&sh.last) {
#pragma unroll 1
                for (int e = tid; e < G * HD / 2; e += AW * 32) {
                    const int hg = e / (HD / 2), d = e % (HD / 2) * 2;
                    const float* p = s.part + ((size_t)first_cta * 8 + hg) * LD;
                    float top = -INFINITY, ls = 0.f;
                    float2 os = make_float2(0.f, 0.f);
#pragma unroll 1
                    for (int c0 = 0; c0 < shares; c0 += kMerge, p += kMerge * 8 * LD) {
                        float2 ml[kMerge], v[kMerge];
#pragma unroll
                        for (int q = 0; q < kMerge; ++q) {
                            const bool in = c0 + q < shares;
                            ml[q] = in ? __ldcg(reinterpret_cast<const float2*>(p + q * 8 * LD + HD)) : make_float2(-INFINITY, 0.f);
                            v[q] = in ? __ldcg(reinterpret_cast<const float2*>(p + q * 8 * LD + d)) : make_float2(0.f, 0.f);
                        }
                        float high = top;
#pragma unroll
                        for (int q = 0; q < kMerge; ++q) high = fmaxf(high, ml[q].x);
                        const float keep = tc::ex2_approx(top - high);
                        ls *= keep; os.x *= keep; os.y *= keep;
#pragma unroll
                        for (int q = 0; q < kMerge; ++q) {
                            const float f = tc::ex2_approx(ml[q].x - high);
                            ls += ml[q].y * f;
                            os.x += v[q].x * f; os.y += v[q].y * f;
                        }
                        top = high;
                    }
                    *reinterpret_cast<uint32_t*>(out + 2 * e) = pack_bf16(os.x / ls, os.y / ls);
                }
            }
        }
    }
    // a step that goes on has used what it asked for; one that gave up still waits for its copies, the one it gave up on among them
    for (; used < issued; ++used) tc::mbar_wait(&sh.kv_full[warp][used % NS], (used / NS) & 1);
    __syncwarp();
    if (lane == 0) sh.kv_count[warp] = used;
    return alive;
}

// ------------------------------------------------------------------------------------------------ phase 2: state update
// The other warps: quads of neighbouring rows of the state (all of one head), a lane 4 NP of a row's N = 128 NP columns.  The
// states of a warp's first NQ quads are asked for before the grid barrier, each next quad's when one has been used up.
template <typename ST, int NP>
__device__ __forceinline__ bool update_states() {
    constexpr int NQ = 4 / NP, N = 128 * NP;
    Shared& sh = shared();
    const StepArgs& s = sh.s;
    const int tid = thread_now(), lane = tid & 31, w = blockIdx.x * (kWarps - kAttnWarps) + (tid >> 5) - kAttnWarps;
    const int r0 = min(w * sh.quad_per, sh.quads), r1 = min(r0 + sh.quad_per, sh.quads);
    const int nh = s.nh, P = s.P, inner = s.inner, proj_ld = (inner + s.C + nh + 7) / 8 * 8;
    ST* states = (ST*)sh.a.ssm_state;
    // column of the lane's i-th run of four values
    auto col = [&](int i) { return sizeof(ST) == 4 ? i * 128 + lane * 4 : lane * (4 * NP) + i * 4; };
    constexpr int W = NP * (int)sizeof(ST);              // words of a row that a lane holds
    uint32_t raw[NQ][4][W];
    // the quad's row b, head h and first row p of the head's state; a lane per quad works them out for 32 of them at a time
    auto place = [&](int q, int& b, int& h, int& p) {
        const int row = q * 4, per = nh * P;
        b = row / per;
        const int rest = row - b * per;
        h = rest / P;
        p = rest - h * P;
    };
    int b_l = 0, h_l = 0, p_l = 0;
    long long at_l = -1;                                 // where the quad's states lie; below zero: a request's first token, which starts from zeros
    auto places = [&](int q32) {
        place(min(q32 + lane, r1 - 1), b_l, h_l, p_l);    // (lanes beyond the last quad: that one again)
        at_l = (((long long)sh.slot[b_l] * nh + h_l) * P + p_l) * N;
        if (sh.start[b_l] <= 0) at_l = -1 - at_l;
    };
    // (loaded whether the request has a state or not, and zeroed at its use)
    auto fetch = [&](long long off, uint32_t (&into)[4][W]) {
        const ST* at = states + (off >= 0 ? off : -1 - off);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                if constexpr (sizeof(ST) == 4) {
                    const uint4 v = ld_cg16(at + i * N + col(k));
                    into[i][4 * k] = v.x; into[i][4 * k + 1] = v.y; into[i][4 * k + 2] = v.z; into[i][4 * k + 3] = v.w;
                } else {
                    const uint2 v = ld_cg8(at + i * N + col(k));
                    into[i][2 * k] = v.x; into[i][2 * k + 1] = v.y;
                }
            }
    };
    if (r0 >= r1) return meet();
    places(r0);
#pragma unroll
    for (int q = 0; q < NQ; ++q)
        if (NP == 2 || r0 + q < r1) fetch(__shfl_sync(0xffffffffu, at_l, q), raw[q]);
    float a_log_l = 0.f, bias_l = 0.f, skip_l = 0.f;
    auto constants = [&]() {
        a_log_l = __ldg(sh.a.a_log + h_l); bias_l = __ldg(sh.a.dt_bias + h_l); skip_l = __ldg(sh.a.d_skip + h_l);
    };
    constants();
    if (!meet()) return false;
    float Bv[4 * NP], Cv[4 * NP];
    int have_bg = -1;
    float kept = 0.f;                                    // the sums of the last 8 quads: lane % 8 is the quad, the upper bits the row
#pragma unroll 1
    for (int q32 = r0; q32 < r1; q32 += 32) {
        // a lane per quad of the next 32: its x, gate, dt and decay
        uint2 x_l = make_uint2(0u, 0u), z_l = x_l;
        float dt_l = 0.f, decay_l = 0.f;
        int bg_l = -1;
        if (q32 > r0) { places(q32); constants(); }
        {
            const bf16* row = s.proj + (size_t)b_l * proj_ld;
            z_l = ld_cg8(row + h_l * P + p_l);
            x_l = ld_cg8(row + inner + h_l * P + p_l);
            const float raw_dt = ld_cg_bf16(row + inner + s.C + h_l);
            bg_l = b_l * s.groups + (s.groups == 1 ? 0 : h_l / (nh / s.groups));
            dt_l = rnd(raw_dt * s.dt_scale) + bias_l;
            dt_l = dt_l > 20.f ? dt_l : log1pf(expf(dt_l));
            decay_l = expf(-expf(a_log_l) * dt_l);
        }
#pragma unroll 1
        for (int q0 = q32; q0 < min(r1, q32 + 32); q0 += NQ) {
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
                const int q = q0 + j, from = q - q32;
                if (q >= r1) continue;
                const int bg = __shfl_sync(0xffffffffu, bg_l, from);
                const float dt = __shfl_sync(0xffffffffu, dt_l, from), decay = __shfl_sync(0xffffffffu, decay_l, from);
                const uint2 xv = make_uint2(__shfl_sync(0xffffffffu, x_l.x, from), __shfl_sync(0xffffffffu, x_l.y, from));
                if (bg != have_bg) {
                    have_bg = bg;
                    const int b = bg / s.groups, grp = bg - b * s.groups;
                    const bf16* row = s.proj + (size_t)b * proj_ld + 2 * inner;
#pragma unroll
                    for (int k = 0; k < NP; ++k) {
                        const uint2 bb = ld_cg8(row + grp * N + col(k)), cc = ld_cg8(row + (s.groups + grp) * N + col(k));
                        Bv[4 * k] = low_f(bb.x); Bv[4 * k + 1] = high_f(bb.x); Bv[4 * k + 2] = low_f(bb.y); Bv[4 * k + 3] = high_f(bb.y);
                        Cv[4 * k] = low_f(cc.x); Cv[4 * k + 1] = high_f(cc.x); Cv[4 * k + 2] = low_f(cc.y); Cv[4 * k + 3] = high_f(cc.y);
                    }
                }
                const float xs[4] = {low_f(xv.x), high_f(xv.x), low_f(xv.y), high_f(xv.y)};
                float dot[4];
                const long long off = __shfl_sync(0xffffffffu, at_l, from);
                ST* at = states + (off >= 0 ? off : -1 - off);
                if (off < 0) {                            // a request's first token
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int k = 0; k < W; ++k) raw[j][i][k] = 0u;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float u = xs[i] * dt;
                    dot[i] = 0.f;
#pragma unroll
                    for (int k = 0; k < NP; ++k) {
                        float f[4];
                        if constexpr (sizeof(ST) == 4) {
#pragma unroll
                            for (int e = 0; e < 4; ++e) f[e] = __uint_as_float(raw[j][i][4 * k + e]);
                        } else {
                            f[0] = low_f(raw[j][i][2 * k]); f[1] = high_f(raw[j][i][2 * k]);
                            f[2] = low_f(raw[j][i][2 * k + 1]); f[3] = high_f(raw[j][i][2 * k + 1]);
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            f[e] = f[e] * decay + Bv[4 * k + e] * u;
                            dot[i] += f[e] * Cv[4 * k + e];
                        }
                        if constexpr (sizeof(ST) == 4) *reinterpret_cast<float4*>(at + i * N + col(k)) = make_float4(f[0], f[1], f[2], f[3]);
                        else *reinterpret_cast<uint2*>(at + i * N + col(k)) = make_uint2(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]));
                    }
                }
                if (q + NQ < r1) {                        // the quad after next of the 32, or of the next 32
                    long long next = __shfl_sync(0xffffffffu, at_l, min(from + NQ, 31));
                    if (from + NQ >= 32) {
                        int nb, nhead, np;
                        place(q + NQ, nb, nhead, np);
                        next = (((long long)sh.slot[nb] * nh + nhead) * P + np) * N;
                    }
                    fetch(next, raw[j]);
                }
                // four sums over 32 lanes at once: lanes with bits 4, 3 of their index hold row 2 * bit 4 + bit 3
                const bool up = lane & 16, odd = lane & 8;
                float k0 = up ? dot[2] : dot[0], k1 = up ? dot[3] : dot[1];
                k0 += __shfl_xor_sync(0xffffffffu, up ? dot[0] : dot[2], 16);
                k1 += __shfl_xor_sync(0xffffffffu, up ? dot[1] : dot[3], 16);
                float r = odd ? k1 : k0;
                r += __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, 8);
                r += __shfl_xor_sync(0xffffffffu, r, 4);
                r += __shfl_xor_sync(0xffffffffu, r, 2);
                r += __shfl_xor_sync(0xffffffffu, r, 1);
                if ((lane & 7) == (from & 7)) kept = r;
                // 8 quads done, or the last one: all their rows' outputs at once
                if ((from & 7) == 7 || q == r1 - 1) {
                    const int mine = (from & ~7) + (lane & 7), row = lane >> 3;
                    const uint32_t x0 = __shfl_sync(0xffffffffu, x_l.x, mine), x1 = __shfl_sync(0xffffffffu, x_l.y, mine);
                    const uint32_t z0 = __shfl_sync(0xffffffffu, z_l.x, mine), z1 = __shfl_sync(0xffffffffu, z_l.y, mine);
                    const float skip = __shfl_sync(0xffffffffu, skip_l, mine);
                    const int to = __shfl_sync(0xffffffffu, b_l * inner + h_l * P + p_l, mine);
                    if (mine <= from) {
                        const float x = row & 1 ? high_f(row & 2 ? x1 : x0) : low_f(row & 2 ? x1 : x0);
                        const float z = row & 1 ? high_f(row & 2 ? z1 : z0) : low_f(row & 2 ? z1 : z0);
                        s.y[to + row] = __float2bfloat16_rn(rnd(kept + skip * x) * rnd(silu_f(rnd(z * s.gate_scale))));
                    }
                }
            }
        }
    }
    return true;
}

// ------------------------------------------------------------------------------------------------ the kernel
// ST, NP: the states' type and their N / 128
template <int ROWS, int HD, typename ST, int NP>
__global__ void __launch_bounds__(kBlock, 1) decode_layers_kernel(const __grid_constant__ Launch L) {
    typedef Shape<ROWS, HD> S;
    constexpr int GROUPS = S::GROUPS, HALVES = ROWS / 8, WK = kWarps, AW = kAttnWarps;      // HALVES: of the instruction's 16 rows
    Shared& sh = shared();
    const StepArgs& s = L.s;
    float* red = smem_sums();                                                // [tile][WK][ROWS][8]; phase 2: [AW][8][HD + 2]
    unsigned char* ring = smem_rings() + kKvBytes + S::RED;
    int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cta = blockIdx.x, ctas = gridDim.x, M = s.M;

    // ------------------------------------------------------------------ set up: once per step
    if (tid < M) { sh.pos[tid] = max(s.positions[tid], 0); sh.slot[tid] = s.slots[tid]; sh.start[tid] = s.start_pos[tid]; }
    if (tid == 64) {
        sh.s = s;
        sh.dead = 0;
        sh.go = 1;
        sh.epoch = 0;
        // phase 2: quad_per quads of state rows are each warp's
        sh.quads = M * s.nh * s.P / 4;
        sh.quad_per = (sh.quads + ctas * (kWarps - AW) - 1) / (ctas * (kWarps - AW));
    }
    if (tid == 96) {
        sh.run_h = runs_of(s.H, GROUPS); sh.run_o = runs_of(s.Hq * HD, GROUPS); sh.run_y = runs_of(s.inner, GROUPS); sh.run_f = runs_of(s.inter, GROUPS);
        sh.in = in_tiles(s, HD);
        int base = 0;                                     // tiles go round from where the phase before stopped
        for (int ph = 0; ph < 4; ++ph) {
            const int all = ph == 0 ? sh.in.all : (ph == 2 ? s.inter / 4 : s.H / 8);
            const int first = (cta - base + ctas) % ctas, n = first < all ? (all - first + ctas - 1) / ctas : 0;
            // tiles of a pass: their sums have room, and a batch of them leaves a quarter of the ring to the next one
            const int widest = ph == 1 ? max(sh.run_o.n, sh.run_y.n) : (ph == 3 ? sh.run_f.n : sh.run_h.n), tile = 8 * row_pitch(widest);
            const int most = min(ph == 1 ? kTiles / 2 : kTiles, max(1, s.ring / 4 * 3 / tile)), passes = (n + most - 1) / most;
            sh.share[ph].n = n; sh.share[ph].first = first; sh.share[ph].per = n > 0 ? (n + passes - 1) / passes : 1;
            base = (base + all) % ctas;
        }
    }
    if (tid == 128) sh.a = L.layer[0].p;
    if (tid == 32) {
        for (int i = 0; i < kBatches; ++i) { tc::mbar_init(&sh.full[i], 1); tc::mbar_init(&sh.empty[i], kWarps); }
        for (int i = 0; i < AW * 4; ++i) tc::mbar_init(&sh.kv_full[0][0] + i, 1);
        for (int i = 0; i < AW; ++i) sh.kv_count[i] = 0;
        tc::mbar_fence_init();
    }
    __syncthreads();
    if (tid == 0) {
        // phase 2: every row and key/value head gets CTAs by its number of key tiles, each at least one and none fewer than 8 tiles
        int total = 0, at = 0;
        for (int b = 0; b < M; ++b) total += s.Hkv * (sh.pos[b] / kKeys + 1);
        const int spare = ctas - M * s.Hkv;
        sh.row = -1;
        sh.tile0 = sh.tile1 = 0;
        for (int b = 0; b < M && sh.row < 0; ++b) {
            const int tiles = sh.pos[b] / kKeys + 1;
            int shares = min(1 + (int)((long long)tiles * spare / total), (tiles + 2 * AW - 1) / (2 * AW));
            if (shares > kMerge) shares -= shares % kMerge;       // the merge loads so many at a time
            if (cta < at + shares * s.Hkv) {
                const int i = (cta - at) % shares, per = (tiles + shares - 1) / shares;
                sh.row = b; sh.head = (cta - at) / shares; sh.shares = (tiles + per - 1) / per; sh.first_cta = cta - i;
                sh.tile0 = min(i * per, tiles); sh.tile1 = min(sh.tile0 + per, tiles);
                if (i >= sh.shares) sh.row = kMaxRows;   // rounded away: nothing to do
            }
            at += shares * s.Hkv;
        }
        if (sh.row == kMaxRows) sh.row = -1;
    }
    __syncthreads();

    if (warp >= kWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsStream));
        if (warp == kWarps + 1) keep_barrier(s, (s.x != nullptr ? 1 : 0) + 5 * s.layers - 1);
        if (warp == kWarps + 2)
            for (int l = 0; l < s.layers; ++l) ask_ahead<HD, 512 * NP * (int)sizeof(ST)>(L.layer[l], l == 0 ? 0 : 5 * l - (s.x != nullptr ? 2 : 3));
        if (warp > kWarps) return;
        // ============================================================== the warp that streams the weights
        // A batch: the tiles of one pass over one piece of k, next to one another in the ring; one full and one empty barrier.
        uint32_t batch = 0, oldest = 0;
        int at = 0, room = s.ring;
        bool ok = true;
        for (int l = 0; l < s.layers && ok; ++l) {
            const LayerPointers& a = L.layer[l].p;
#pragma unroll 1
            for (int ph = 0; ph < 4 && ok; ++ph) {        // the products of phases 1, 3, 4, 5
                const int n = sh.share[ph].n, first = sh.share[ph].first, per = sh.share[ph].per;
                for (int i0 = 0; i0 < n; i0 += per)
                    for (int part = 0; part < (ph == 1 ? 2 : 1); ++part) {
                        const Runs run = ph == 1 ? (part == 0 ? sh.run_o : sh.run_y) : (ph == 3 ? sh.run_f : sh.run_h);
                        for (int u0 = 0; u0 < run.units && ok; u0 += run.n) {
                            const int un = min(run.n, run.units - u0), pitch = row_pitch(un), f = lane & 7, nt = min(per, n - i0);
                            int bytes = nt * 8 * pitch;
                            if (at + bytes > s.ring) {     // the rest of the round stays empty
                                bytes = min(bytes + s.ring - at, s.ring);
                                at = 0;
                            }
                            while (ok && (room < bytes || batch - oldest == kBatches)) {
                                ok = wait_for_room(&sh.empty[oldest % kBatches], (oldest / kBatches) & 1, 5 * l + ph);
                                room += sh.batch_bytes[oldest % kBatches];
                                ++oldest;
                            }
                            if (!ok) break;
                            const int bi = batch % kBatches;
                            __syncwarp();
                            if (lane == 0) {
                                sh.batch_bytes[bi] = bytes;
                                tc::mbar_expect_tx(&sh.full[bi], nt * un * 4096);
                            }
                            __syncwarp();
                            for (int i = lane >> 3; i < nt; i += 4) {          // eight lanes a tile, a row each
                                const int j = first + (i0 + i) * ctas;
                                const bf16* row;
                                if (ph == 0) {
                                    if (j < sh.in.k) {     // q, k: the tile holds 4 pairs of a rotation
                                        const int head = j / (HD / 8), p = j % (HD / 8);
                                        row = a.qkv_w + (size_t)(head * HD + p * 4 + (f & 3) + (f >> 2) * (HD / 2)) * s.H;
                                    } else if (j < sh.in.v) row = a.qkv_w + (size_t)(j * 8 + f) * s.H;
                                    else row = a.in_w + (size_t)min((j - sh.in.v) * 8 + f, s.inner + s.C + s.nh - 1) * s.H;
                                } else if (ph == 1) row = (part == 0 ? a.o_w : a.out_w) + (size_t)(j * 8 + f) * (run.units * 256);
                                else if (ph == 2) row = a.gate_up_w + (size_t)(j * 4 + (f & 3) + (f >> 2) * s.inter) * s.H;
                                else row = a.down_w + (size_t)(j * 8 + f) * s.inter;
                                bulk_load(smem_u32(ring + at + (i * 8 + f) * pitch), row + u0 * 256, un * 512, &sh.full[bi]);
                            }
                            ++batch;
                            room -= bytes;
                            at += nt * 8 * pitch;
                        }
                    }
            }
        }
        // no copy may land after the CTA has gone (nothing is left to wait for unless a wait gave up)
        for (uint32_t i = batch > kBatches ? batch - kBatches : 0; i < batch; ++i) tc::mbar_wait(&sh.full[i % kBatches], (i / kBatches) & 1);
        return;
    }

    // ================================================================== the other warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsWork));
    bool ok = true;                                      // false: a wait of this thread gave up
    uint32_t batch = 0;                                  // batches of tiles taken from the ring, and where the next one may lie
    int ring_at = 0, epoch = 0;                          // grid barriers arrived at
    const int qkv_ld = (s.Hq + 2 * s.Hkv) * HD, proj_cols = s.inner + s.C + s.nh, proj_ld = (proj_cols + 7) / 8 * 8;

    auto summed = [&](int i, int m, int f) -> float {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < WK; ++w) v += red[((size_t)(i * WK + w) * ROWS + m) * 8 + f];
        return v;
    };

    // ---- the rows as the embedding left them
    if (s.x != nullptr) {
        const int tiles = s.H / 8;
        for (int e = cta * kThreads + tid; e < M * tiles; e += ctas * kThreads) {
            const int m = e / tiles, p = e - m * tiles;
            const uint4 v = *reinterpret_cast<const uint4*>(s.x + (size_t)m * s.H + p * 8);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            uint32_t out[4];
            float sq = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float a = low_f(w[i]), b = high_f(w[i]);
                sq += a * a + b * b;
                out[i] = pack_bf16(a * __ldg(s.first_norm + p * 8 + 2 * i), b * __ldg(s.first_norm + p * 8 + 2 * i + 1));
            }
            *reinterpret_cast<uint4*>(s.xn + (size_t)m * s.H + p * 8) = make_uint4(out[0], out[1], out[2], out[3]);
            *reinterpret_cast<uint4*>(s.res_b + (size_t)m * s.H + p * 8) = v;
            s.ssq[(size_t)m * tiles + p] = sq;
        }
        arrive(epoch);
    }

#pragma unroll 1
    for (int l = 0; l < s.layers; ++l) {
        const LayerArgs& layer = L.layer[l];
        const LayerPointers& a = layer.p;
#pragma unroll 1
        for (int ph = 0; ph < 4; ++ph) {                  // the products: phases 1, 3, 4, 5
            tid = thread_now(); warp = tid >> 5; lane = tid & 31;
            const int g = lane >> 2, t = lane & 3;
            const int n = sh.share[ph].n, first = sh.share[ph].first, per = sh.share[ph].per;
            // ---- k in pieces: those of the phase's product, or of phase 3's two, whose sums stay apart
            const Runs run0 = ph == 1 ? sh.run_o : (ph == 3 ? sh.run_f : sh.run_h);
            // (lanes of rows beyond the last read that one again; nobody reads their sums)
            const int row = min(g, M - 1), up = min(g + 8, M - 1) - row;
            const int n0 = run0.pieces, pieces = ph == 1 ? n0 + sh.run_y.pieces : n0;
            const bf16* src0 = (ph == 1 ? s.o : (ph == 3 ? s.h : s.xn)) + (size_t)row * (run0.units * 256) + warp * 32 + t * 8;
            const bf16* src1 = s.y + (size_t)row * s.inner + warp * 32 + t * 8;
            auto units_of = [&](int c) {
                const Runs run = c < n0 ? run0 : sh.run_y;
                return min(run.n, run.units - (c < n0 ? c : c - n0) * run.n);
            };
            // ---- what the thread's first output reads besides the sums is asked for before the barrier
            float early0 = 0.f, early1 = 0.f, early2 = 0.f, early_b = 0.f;       // conv window and bias; cos and sin; residual and norm weight
            int early_at = -1;                            // the token's place in the cache
            float4 taps = make_float4(0.f, 0.f, 0.f, 0.f);
            {
                const int j = first + tid / (ROWS * 8) * ctas, m = (tid >> 3) % ROWS, f = tid & 7;
                const bool mine = tid < min(n, per) * ROWS * 8 && m < M;
                if (ph == 0) {
                    const int c = (j - sh.in.z) * 8 + f;
                    if (mine && s.taps == 4 && j >= sh.in.z && j < sh.in.c) {
                        taps = __ldg(reinterpret_cast<const float4*>(a.conv_w) + c);
                        early_b = a.conv_b != nullptr ? __ldg(a.conv_b + c) : 0.f;
                        if (sh.start[m] > 0) {
                            const bf16* win = a.conv_state + ((size_t)sh.slot[m] * s.C + c) * 3;
                            early0 = __bfloat162float(win[0]); early1 = __bfloat162float(win[1]); early2 = __bfloat162float(win[2]);
                        }
                    }
                    if (mine && j < sh.in.v) {
                        if (j < sh.in.k) {
                            const float* cs = s.cos_sin + (size_t)min(sh.pos[m], s.table_rows - 1) * HD + j % (HD / 8) * 4 + (f & 3);
                            early0 = __ldg(cs);
                            early1 = __ldg(cs + HD / 2);
                        }
                        if (j >= sh.in.q) early_at = a.slot_mapping[m];
                    }
                    // the other columns' conv operands, and what phase 2 will read: on their way to L2
                    for (int e = tid; (n > per || per * ROWS * 8 > kThreads || s.taps != 4) && e < n * ROWS; e += kThreads) {
                        const int jj = first + (e / ROWS) * ctas, mm = e % ROWS;
                        if (mm < M && jj >= sh.in.z && jj < sh.in.c) {
                            const int cc = (jj - sh.in.z) * 8;
                            const bf16* win = a.conv_state + ((size_t)sh.slot[mm] * s.C + cc) * (s.taps - 1);
                            prefetch_l2(win);
                            prefetch_l2(win + 8 * (s.taps - 1) - 1);
                            if (mm == 0) {
                                prefetch_l2(a.conv_w + (size_t)cc * s.taps);
                                prefetch_l2(a.conv_w + (size_t)(cc + 4) * s.taps);
                                if (a.conv_b != nullptr) prefetch_l2(a.conv_b + cc);
                            }
                        }
                    }
                    if (tid == 0) {
                        asm volatile("prefetch.tensormap [%0];" ::"l"(&layer.map_k) : "memory");
                        asm volatile("prefetch.tensormap [%0];" ::"l"(&layer.map_v) : "memory");
                    }
                    if (l > 0 && tid == 32) sh.a = a;      // (the first layer's: in the set-up; no grid barrier orders it for a CTA without tiles)
                    if (tid * 32 < s.nh) { prefetch_l2(a.a_log + tid * 32); prefetch_l2(a.dt_bias + tid * 32); prefetch_l2(a.d_skip + tid * 32); }
                } else if (ph != 2 && mine && (ph == 1 || a.next_norm != nullptr)) {
                    early_b = __ldg((ph == 1 ? a.ff_norm : a.next_norm) + j * 8 + f);
                    early0 = ld_cg_bf16((ph == 1 ? s.res_b : s.res_a) + (size_t)m * s.H + j * 8 + f);
                }
            }
            const unsigned char* w_at = ring;            // the next batch in the ring, this lane's share of its first tile
            int w_pitch = 0;
            auto take = [&](int nt, int un) {
                w_pitch = row_pitch(un);
                if (ring_at + nt * 8 * w_pitch > s.ring) ring_at = 0;
                if (ok && !wait_for(&sh.full[batch % kBatches], (batch / kBatches) & 1, s.weight_polls)) { ok = false; give_up(0x33, epoch); }
                w_at = ring + ring_at + g * w_pitch + warp * 64 + t * 16;
                ring_at += nt * 8 * w_pitch;
            };
            const int un0 = units_of(0);
            if (n > 0) take(min(per, n), un0);           // the first piece's weights: as a rule they landed long ago
            if (epoch > 0 && !meet()) return;
#pragma unroll 1
            for (int i0 = 0; i0 < n; i0 += per) {
                const int nt = min(per, n - i0);
                if (i0 > 0) {
                    named_sync<kThreads, 4>();           // the sums of the pass before have been read
                    take(nt, un0);
                }
                uint4 rows[2][GROUPS][HALVES];           // two pieces' rows are on their way
                auto load_rows = [&](uint4 (&v)[GROUPS][HALVES], int c) {
                    const Runs run = c < n0 ? run0 : sh.run_y;
                    const int u0 = (c < n0 ? c : c - n0) * run.n, un = min(run.n, run.units - u0);
                    const bf16* src = (c < n0 ? src0 : src1) + u0 * 256;
#pragma unroll
                    for (int u = 0; u < GROUPS; ++u) {
                        if (u >= un) break;
                        v[u][0] = ld_cg16(src + u * 256);
                        if (HALVES == 2) v[u][HALVES - 1] = ld_cg16(src + (size_t)up * (run.units * 256) + u * 256);
                    }
                };
                load_rows(rows[0], 0);
                if (pieces > 1) load_rows(rows[1], 1);
                // the rows' sums of squares, a warp per row: the norm's factors
                float squares[HALVES] = {};
#pragma unroll
                for (int h = 0; h < HALVES; ++h)
                    if ((ph == 0 || ph == 2) && warp + 8 * h < M)
                        for (int p = lane; p < s.H / 32; p += 32) {
                            const float4 four = __ldcg(reinterpret_cast<const float4*>(s.ssq + (size_t)(warp + 8 * h) * (s.H / 8)) + p);
                            squares[h] += (four.x + four.y) + (four.z + four.w);
                        }
                // one piece against the pass's tiles, two at a time
                auto multiply = [&](const uint4 (&v)[GROUPS][HALVES], int c) {
                    const int un = units_of(c);
                    const unsigned char* w = w_at;
                    float* to = red + ((size_t)((ph == 1 && c >= n0 ? kTiles / 2 : 0) * WK + warp) * ROWS + g) * 8 + 2 * t;
                    const bool more = c > 0 && c != n0;   // a sum's later pieces
                    auto two = [&](auto groups) {
                        constexpr int U = decltype(groups)::value;
#pragma unroll 1
                        for (int i = 0; i < nt; i += 2) {
                            float c0[4] = {}, c1[4] = {}, d0[4] = {}, d1[4] = {};
                            if (i + 1 < nt) {
                                uint4 x[U], y[U];
#pragma unroll
                                for (int u = 0; u < U; ++u) x[u] = *reinterpret_cast<const uint4*>(w + u * 512);
#pragma unroll
                                for (int u = 0; u < U; ++u) y[u] = *reinterpret_cast<const uint4*>(w + 8 * w_pitch + u * 512);
#pragma unroll
                                for (int u = 0; u < U; ++u) {
                                    const uint4 lo = v[u][0], hi = HALVES == 2 ? v[u][HALVES - 1] : make_uint4(0u, 0u, 0u, 0u);
                                    mma_bf16(c0, lo.x, hi.x, lo.y, hi.y, x[u].x, x[u].y);
                                    mma_bf16(d0, lo.x, hi.x, lo.y, hi.y, y[u].x, y[u].y);
                                    mma_bf16(c1, lo.z, hi.z, lo.w, hi.w, x[u].z, x[u].w);
                                    mma_bf16(d1, lo.z, hi.z, lo.w, hi.w, y[u].z, y[u].w);
                                }
                            } else {
                                uint4 x[U];
#pragma unroll
                                for (int u = 0; u < U; ++u) x[u] = *reinterpret_cast<const uint4*>(w + u * 512);
#pragma unroll
                                for (int u = 0; u < U; ++u) {
                                    const uint4 lo = v[u][0], hi = HALVES == 2 ? v[u][HALVES - 1] : make_uint4(0u, 0u, 0u, 0u);
                                    mma_bf16(c0, lo.x, hi.x, lo.y, hi.y, x[u].x, x[u].y);
                                    mma_bf16(c1, lo.z, hi.z, lo.w, hi.w, x[u].z, x[u].w);
                                }
                            }
                            float2* at = reinterpret_cast<float2*>(to + (size_t)i * WK * ROWS * 8);
#pragma unroll
                            for (int h = 0; h < HALVES; ++h, at += 32) {
                                float2 a0 = make_float2(c0[2 * h] + c1[2 * h], c0[2 * h + 1] + c1[2 * h + 1]);
                                float2 a1 = make_float2(d0[2 * h] + d1[2 * h], d0[2 * h + 1] + d1[2 * h + 1]);
                                if (more) {
                                    const float2 b0 = at[0], b1 = i + 1 < nt ? at[WK * ROWS * 4] : b0;
                                    a0.x += b0.x; a0.y += b0.y; a1.x += b1.x; a1.y += b1.y;
                                }
                                at[0] = a0;
                                if (i + 1 < nt) at[WK * ROWS * 4] = a1;
                            }
                            w += 16 * w_pitch;
                        }
                    };
                    switch (un) {
                        case 1: two(std::integral_constant<int, 1>()); break;
                        case 2: two(std::integral_constant<int, 2>()); break;
                        case 3: two(std::integral_constant<int, 3>()); break;
                        case 4: two(std::integral_constant<int, 4>()); break;
                        case 5: two(std::integral_constant<int, GROUPS < 5 ? GROUPS : 5>()); break;
                        default: two(std::integral_constant<int, GROUPS>());
                    }
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&sh.empty[batch % kBatches]);
                    ++batch;
                    if (c + 1 < pieces) take(nt, units_of(c + 1));
                };
#pragma unroll 1
                for (int c = 0; c < pieces; c += 2) {
                    multiply(rows[0], c);
                    if (c + 2 < pieces) load_rows(rows[0], c + 2);
                    if (c + 1 < pieces) {
                        multiply(rows[1], c + 1);
                        if (c + 3 < pieces) load_rows(rows[1], c + 3);
                    }
                }
                if (ph == 0 || ph == 2) {
                    const float eps = ph == 0 ? s.eps_mixer : s.eps_ff;
#pragma unroll
                    for (int h = 0; h < HALVES; ++h) {
                        const float sum = warp_sum(squares[h]);
                        if (warp + 8 * h < M && lane == 0) sh.factor[warp + 8 * h] = rsqrtf(sum / (float)s.H + eps);
                    }
                }
                named_sync<kThreads, 4>();
                // ---- epilogue: a thread per (tile i, row m, feature f); the 8 features of a tile are 8 neighbouring lanes
                tid = thread_now();
#pragma unroll 1
                for (int e = tid; e < nt * ROWS * 8; e += kThreads) {
                    const int i = e / (ROWS * 8), m = (e >> 3) % ROWS, f = e & 7, j = first + (i0 + i) * ctas;
                    const bool early = i0 == 0 && e == tid;
                    float v = summed(i, m, f);
                    if (ph == 0) {
                        v *= sh.factor[m];
                        if (j < sh.in.v) {
                            v = rnd(v * s.attn_in);
                            if (j < sh.in.k) {
                                const int head = j / (HD / 8), p = j % (HD / 8), half = HD / 2, pair = p * 4 + (f & 3);
                                const bool key = j >= sh.in.q, low = f < 4;
                                if (key) v = rnd(v * s.key_scale);
                                const float partner = __shfl_xor_sync(0xffffffffu, v, 4);
                                if (m < M) {
                                    const float* cs = s.cos_sin + (size_t)min(sh.pos[m], s.table_rows - 1) * HD + pair;
                                    const float c = early ? early0 : __ldg(cs), sn = early ? early1 : __ldg(cs + half);
                                    const bf16 out = __float2bfloat16_rn(v * c + (low ? -partner : partner) * sn);
                                    const int d = pair + (low ? 0 : half);
                                    s.qkv[(size_t)m * qkv_ld + head * HD + d] = out;
                                    const int at = !key ? -1 : (early ? early_at : a.slot_mapping[m]);
                                    if (at >= 0) a.k_cache[((size_t)at * s.Hkv + head - s.Hq) * HD + d] = out;
                                }
                            } else if (m < M) {
                                const int d = (j - sh.in.k) * 8 + f;
                                s.qkv[(size_t)m * qkv_ld + (s.Hq + s.Hkv) * HD + d] = __float2bfloat16_rn(v);
                                const int at = early ? early_at : a.slot_mapping[m];
                                if (at >= 0) a.v_cache[(size_t)at * s.Hkv * HD + d] = __float2bfloat16_rn(v);
                            }
                        } else if (m < M) {
                            v = rnd(v * s.ssm_in);
                            const int c = (j - sh.in.v) * 8 + f;
                            if (j >= sh.in.z && j < sh.in.c) {
                                const int ch = c - s.inner;
                                const float u = rnd(v * (ch < s.conv_e0 ? s.conv_s0 : (ch < s.conv_e1 ? s.conv_s1 : s.conv_s2)));
                                bf16* win = a.conv_state + ((size_t)sh.slot[m] * s.C + ch) * (s.taps - 1);
                                float sum;
                                if (early && s.taps == 4) {
                                    sum = taps.w * u;
                                    sum += taps.x * early0; sum += taps.y * early1; sum += taps.z * early2;
                                    sum += early_b;
                                    win[0] = __float2bfloat16_rn(early1); win[1] = __float2bfloat16_rn(early2); win[2] = __float2bfloat16_rn(u);
                                } else {
                                    const bool history = sh.start[m] > 0;
                                    const float* w = a.conv_w + (size_t)ch * s.taps;
                                    sum = w[s.taps - 1] * u;
#pragma unroll 1
                                    for (int q = 0; q < s.taps - 1; ++q) {
                                        const float old = history ? __bfloat162float(win[q]) : 0.f;
                                        sum += w[q] * old;
                                        if (q > 0) win[q - 1] = __float2bfloat16_rn(old);
                                    }
                                    win[s.taps - 2] = __float2bfloat16_rn(u);
                                    if (a.conv_b != nullptr) sum += a.conv_b[ch];
                                }
                                v = silu_f(rnd(sum));
                            }
                            if (c < proj_cols) s.proj[(size_t)m * proj_ld + c] = __float2bfloat16_rn(v);
                        }
                    } else if (ph == 2) {
                        v = rnd(v * sh.factor[m]);
                        if (f < 4) v = rnd(silu_f(rnd(v * s.act_scale)));
                        const float up = __shfl_xor_sync(0xffffffffu, v, 4);
                        if (f < 4 && m < M) s.h[(size_t)m * s.inter + j * 4 + f] = __float2bfloat16_rn(v * up);
                    } else {
                        const int c = j * 8 + f;
                        const float* norm = ph == 1 ? a.ff_norm : a.next_norm;
                        v = rnd(v);
                        if (ph == 1) v = rnd(rnd(v * s.attn_out) + rnd(rnd(summed(kTiles / 2 + i, m, f)) * s.ssm_out));
                        else if (s.ff_scale != 1.f) v = rnd(v * s.ff_scale);
                        if (norm == nullptr) {            // the model's last product: the norm behind it joins the two
                            if (m < M) s.x_out[(size_t)m * s.H + c] = __float2bfloat16_rn(v);
                        } else {
                            // what the join leaves for the norm behind it: v times the norm's weight, and the sum of the tile's squares
                            const float weight = early ? early_b : __ldg(norm + c);
                            if (m < M) {
                                v += early ? early0 : ld_cg_bf16((ph == 1 ? s.res_b : s.res_a) + (size_t)m * s.H + c);
                                (ph == 1 ? s.res_a : s.res_b)[(size_t)m * s.H + c] = __float2bfloat16_rn(v);
                                s.xn[(size_t)m * s.H + c] = __float2bfloat16_rn(v * weight);
                            }
                            float sq = v * v;
                            sq += __shfl_xor_sync(0xffffffffu, sq, 1);
                            sq += __shfl_xor_sync(0xffffffffu, sq, 2);
                            sq += __shfl_xor_sync(0xffffffffu, sq, 4);
                            if (m < M && f == 0) s.ssq[(size_t)m * (s.H / 8) + j] = sq;
                        }
                    }
                }
            }
            if (ph < 3 || l + 1 < s.layers) arrive(epoch);
            if (ph == 0) {
                // ================================================ phase 2
                bool alive;
                if (thread_now() < AW * 32) alive = attend<HD>(&layer.map_k, &layer.map_v, epoch);
                else alive = update_states<ST, NP>();
                if (!alive) return;
                arrive(epoch);
            }
        }
    }
}

template <int ROWS, int HD, typename ST, int NP>
int launch_states(Launch& p, cudaStream_t stream) {
    static int sms = 0;
    static size_t have = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    if (p.s.M * p.s.Hkv > sms) return kTooLarge;         // every (row, key/value head) needs a CTA of its own
    constexpr int kMost = 232448;                        // 227 KB per CTA
    constexpr int kFixed = kSharedBytes + 1024 + kKvBytes + Shape<ROWS, HD>::RED;
    p.s.ring = (kMost - kFixed) / 1024 * 1024;
    const size_t smem = kFixed + (size_t)p.s.ring;
    ensure_dynamic_smem(decode_layers_kernel<ROWS, HD, ST, NP>, smem, have);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sms); cfg.blockDim = dim3(kBlock); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int rc = (int)cudaMemsetAsync(p.s.barrier, 0, sizeof(unsigned) * (32 + (size_t)p.s.M * p.s.Hkv), stream);
    if (rc == 0) rc = (int)cudaLaunchKernelEx(&cfg, decode_layers_kernel<ROWS, HD, ST, NP>, p);
    return rc != 0 ? rc : launch_status();
}
template <int HD, typename ST, int NP>
int launch_rows(Launch& p, cudaStream_t stream) {
    return p.s.M <= 8 ? launch_states<8, HD, ST, NP>(p, stream) : launch_states<16, HD, ST, NP>(p, stream);
}
template <int HD>
int launch(Launch& p, cudaStream_t stream) {
    if (p.s.state_bf16) return p.s.N == 128 ? launch_rows<HD, bf16, 1>(p, stream) : launch_rows<HD, bf16, 2>(p, stream);
    return p.s.N == 128 ? launch_rows<HD, float, 1>(p, stream) : launch_rows<HD, float, 2>(p, stream);
}
}  // namespace

// The layers of a decode step (see the head of the file).  ints, floats, buffers: the fields of StepArgs in their order, behind the
// ints the polls after which waits give up (below zero: as many as take about a second); layers:
// 19 pointers per layer in the order of LayerPointers and, as the 20th, the block table's row stride.  M <= 16 rows, one token each.
// buffers[17]: 32 + M * Hkv words for the grid barrier and the merge counters.
extern "C" int lb_decode_layers(const int* ints, const float* floats, const uint64_t* buffers, const uint64_t* layers, int n_layers,
                                int head_dim, long pages, void* stream) {
    if (n_layers <= 0) return kOk;
    if (n_layers > kMaxLayers) return kTooLarge;
    Launch p;
    StepArgs& s = p.s;
    int* si[] = {&s.M, &s.H, &s.Hq, &s.Hkv, &s.page_size, &s.inner, &s.nh, &s.P, &s.N, &s.groups, &s.C, &s.taps, &s.conv_e0,
                 &s.conv_e1, &s.inter, &s.table_rows, &s.state_bf16};
    for (int* f : si) *f = *ints++;
    float* sf[] = {&s.conv_s0, &s.conv_s1, &s.conv_s2, &s.dt_scale, &s.gate_scale, &s.attn_in, &s.ssm_in, &s.attn_out, &s.ssm_out,
                   &s.key_scale, &s.sm_scale, &s.act_scale, &s.ff_scale, &s.eps_mixer, &s.eps_ff};
    for (float* f : sf) *f = *floats++;
    s.cos_sin = (const float*)buffers[0];
    s.positions = (const int*)buffers[1]; s.slots = (const int*)buffers[2]; s.start_pos = (const int*)buffers[3];
    s.x = (const bf16*)buffers[4]; s.first_norm = (const float*)buffers[5];
    s.xn = (bf16*)buffers[6]; s.res_a = (bf16*)buffers[7]; s.res_b = (bf16*)buffers[8]; s.x_out = (bf16*)buffers[9];
    s.ssq = (float*)buffers[10];
    s.qkv = (bf16*)buffers[11]; s.proj = (bf16*)buffers[12]; s.o = (bf16*)buffers[13]; s.y = (bf16*)buffers[14]; s.h = (bf16*)buffers[15];
    s.part = (float*)buffers[16];
    s.barrier = (unsigned*)buffers[17]; s.counters = (int*)buffers[17] + 32;
    s.error = (int*)buffers[18];
    s.layers = n_layers;
    s.ring = s.page_shift = 0;
    s.barrier_polls = ints[0] >= 0 ? (uint32_t)ints[0] : kBarrierSpins;
    s.key_polls = ints[1] >= 0 ? (uint32_t)ints[1] : tc::kSpinLimit;
    s.weight_polls = ints[2] >= 0 ? (uint32_t)ints[2] : tc::kSpinLimit;
    while (kKeys << s.page_shift < s.page_size) ++s.page_shift;
    if (s.M < 1 || s.M > kMaxRows) return kTooLarge;
    if (s.H % 256 || s.inner % 256 || s.inter % 256 || s.Hq * head_dim % 256 || s.C % 8 || (head_dim != 64 && head_dim != 128) || s.Hkv < 1 || s.Hq % s.Hkv
        || s.Hq / s.Hkv > 8 || s.page_size != kKeys << s.page_shift || s.M * s.Hkv > 64 || (s.N != 128 && s.N != 256) || s.P % 4 || s.nh < 1 || s.groups < 1
        || s.nh % s.groups || s.inner != s.nh * s.P || s.C != s.inner + 2 * s.groups * s.N || s.taps < 2 || s.taps > 8)
        return kBadSize;
    for (int i = 0; i < n_layers; ++i) {
        const uint64_t* f = layers + 20 * i;
        for (int k = 0; k < 7; ++k)                      // 16-byte copies and loads: the matrices, the conv taps
            if (f[k] & 15) return kBadSize;
        LayerPointers& a = p.layer[i].p;
        a.qkv_w = (const bf16*)f[0]; a.in_w = (const bf16*)f[1]; a.o_w = (const bf16*)f[2]; a.out_w = (const bf16*)f[3];
        a.gate_up_w = (const bf16*)f[4]; a.down_w = (const bf16*)f[5];
        a.conv_w = (const float*)f[6]; a.conv_b = (const float*)f[7]; a.a_log = (const float*)f[8]; a.dt_bias = (const float*)f[9];
        a.d_skip = (const float*)f[10]; a.ff_norm = (const float*)f[11]; a.next_norm = (const float*)f[12];
        a.conv_state = (bf16*)f[13]; a.k_cache = (bf16*)f[14]; a.v_cache = (bf16*)f[15]; a.ssm_state = (void*)f[16];
        a.block_table = (const int*)f[17]; a.slot_mapping = (const int*)f[18]; a.bt_stride = (int)f[19]; a.pad = 0;
        if ((f[14] | f[15] | f[16]) & 15) return kBadSize;
        const long width = (long)s.Hkv * head_dim;
        int rc = tc::make_tile_map(&p.layer[i].map_k, a.k_cache, pages * s.page_size, width, width, kKeys);
        if (rc == 0) rc = tc::make_tile_map(&p.layer[i].map_v, a.v_cache, pages * s.page_size, width, width, kKeys);
        if (rc != 0) return rc;
    }
    cudaStream_t st = (cudaStream_t)stream;
    return head_dim == 64 ? launch<64>(p, st) : launch<128>(p, st);
}
