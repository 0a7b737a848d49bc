// Depthwise causal conv1d over packed portions, with per-request history kept in state slots.
//
//   u_t[ch]  = round(xBC_t[ch] * region_scale(ch))                (three regions: x | B | C)
//   c_t[ch]  = sum_{j<K} w[ch, j] * u_{t-(K-1)+j}[ch] (+ bias[ch])  ; inputs before the portion come
//              from the request's conv state (zeros when the request starts at position 0)
//   out_t    = round(silu(round(c_t)))                            (`act` 1: out_t = round(c_t), no activation)
//   state'   = the last K-1 scaled inputs u, oldest first
// (python/logssms/kernel/linear_attention/packed_conv.py:96-140; decode form
// python/logssms/kernel/linear_attention/conv_decode.py:112-278.)
//
// One launch.  A step's portions are cut into runs of tokens, one CTA each (and range of channels); only a portion's first run
// reads the request's state, and its threads rewrite it afterwards from the portion's last inputs.  Where one portion is much longer
// than the others the grid has as many CTAs as there can be runs (tokens / run + requests) and not requests x runs of the longest: of
// a bucket's 32 requests 31 had one run out of 9, and most CTAs were 256 threads that looked their portion up and left.  With that,
// runs of 32 tokens instead of 64 and the tables and taps read before the wait for the kernel in front: 18 to 13 us in a step of 576
// rows and 32 requests, 14 to 12 with 8 requests, 18.5 to 16 at 2,048 rows, and the rewrite of the state in a launch of its own (2
// to 5 us more) is gone.
#include "lb200/common.cuh"
using namespace lb200;

namespace {
struct ConvArgs {
    const void* x; long x_stride;          // [tokens, C] view, row stride in elements
    const float* weight;                   // [C, K]
    const float* bias;                     // [C] or null
    void* state;                           // [slots, C, K-1]
    void* out;                             // [tokens, C] contiguous
    const int* cu_seqlens; const int* start_pos; const int* slots;
    int C; int end0; int end1; float s0; float s1; float s2;
    int act;                               // what follows the convolution: 0 silu, 1 nothing
    int B;                                 // requests
    int shift;                             // log2 of a run's tokens
    int step;                              // first stride of the search for a run; 0: the grid has every request's runs side by side
};

// The CTA's run: request and first token (at or behind the portion's end: there is none).  By every warp for itself.  Where the longest portion is about the
// usual one the grid is requests x its runs.  Else the runs are numbered, request r's from (its first token >> shift) + r on:
// at least as many numbers as it has runs, and all together no more than (tokens >> shift) + requests.  The request of a number is
// found by a search over first tokens, 32 a look (a walk that adds up lengths takes 32 dependent loads for 1,024 requests).
__device__ __forceinline__ void find_run(const ConvArgs& a, int& b, int& t0) {
    if (a.step == 0) {
        b = blockIdx.z;
        t0 = blockIdx.y << a.shift;
        return;
    }
    const int want = blockIdx.z * gridDim.y + blockIdx.y, lane = threadIdx.x & 31;
    int lo = 0, origin = 0;                               // origin: the first token of all
    for (int step = a.step;; step >>= 5) {
        const int r = lo + lane * step, start = r < a.B ? a.cu_seqlens[r] : 0;
        if (step == a.step) origin = __shfl_sync(0xffffffffu, start, 0);
        const int number = ((start - origin) >> a.shift) + r;
        const int at = __popc(__ballot_sync(0xffffffffu, r < a.B && number <= want)) - 1;
        lo += at * step;
        if (step == 1) {
            b = lo;
            t0 = (want - __shfl_sync(0xffffffffu, number, at)) << a.shift;
            return;
        }
    }
}

template <typename T>
__device__ __forceinline__ float scaled_input(const ConvArgs& a, long token, int c, float scale) {
    return round_to<T>(to_f32(((const T*)a.x)[token * a.x_stride + c]) * scale);
}

// A channel's saved inputs after a portion of `len` tokens: the last K - 1 of the inputs before it and its own.  By the only thread
// that still reads or writes them.
template <typename T, int K>
__device__ __forceinline__ void rewrite_state(const ConvArgs& a, T* st, int begin, int len, int c, float scale, bool has_history) {
    float next[K];
#pragma unroll
    for (int j = 0; j < K - 1; ++j) {
        const int idx = len - (K - 1) + j;
        next[j] = idx >= 0 ? scaled_input<T>(a, begin + idx, c, scale) : (has_history ? to_f32(st[K - 1 + idx]) : 0.f);
    }
#pragma unroll
    for (int j = 0; j < K - 1; ++j) st[j] = from_f32<T>(next[j]);
}

// Any type and alignment, a thread per channel, in two forms.  Few tokens: runs of 8 whose inputs are all on their way before the first
// is used; one thread walking 64 tokens, each load waited for, takes 15 us however few there are.  Many tokens, or portions of a
// few: runs of up to 64 walked one by one, which read no input twice and need few registers.  (float32, 1,792 channels, us, runs of 8 /
// walked: one portion of 512 tokens 5.5 / 18.5, of 2,048 13.9 / 19.7, of 8,192 64 / 47; 8 of 60 5.8 / 16, 100 of 30 20.7 / 12.9; 64 of 7
// 5.7 / 4.2; 64 decoded tokens 3.2 / 2.4.)
constexpr int kRun = 8, kWalk = 64;

template <typename T, int K>
__global__ void conv_forward_kernel(ConvArgs a) {
    static_assert(K - 1 <= kRun, "only a portion's first run may reach back into the saved inputs");
    int b, t0;
    find_run(a, b, t0);                                   // (the step's tables are not the kernel's before this one)
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= a.C) return;
    const int begin = a.cu_seqlens[b], len = a.cu_seqlens[b + 1] - begin;
    if (t0 >= len) return;
    const int n = min(len - t0, kRun);
    const float scale = c < a.end0 ? a.s0 : (c < a.end1 ? a.s1 : a.s2);
    const bool has_history = a.start_pos[b] > 0;
    T* st = (T*)a.state + ((size_t)a.slots[b] * a.C + c) * (K - 1);
    float w[K], in[K - 1 + kRun];                         // the K - 1 inputs in front of the run, then its own
#pragma unroll
    for (int j = 0; j < K; ++j) w[j] = a.weight[(size_t)c * K + j];
#pragma unroll
    for (int j = 0; j < K - 1 + kRun; ++j) {
        const int idx = t0 - (K - 1) + j;                 // relative to the portion's first token
        if (idx >= 0) in[j] = idx < len ? scaled_input<T>(a, begin + idx, c, scale) : 0.f;
        else in[j] = has_history ? to_f32(st[K - 1 + idx]) : 0.f;
    }
    const float bias = a.bias ? a.bias[c] : 0.f;
#pragma unroll
    for (int i = 0; i < kRun; ++i) {
        if (i >= n) break;
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < K; ++j) acc += in[i + j] * w[j];
        acc = round_to<T>(acc + bias);
        ((T*)a.out)[(size_t)(begin + t0 + i) * a.C + c] = from_f32<T>(a.act == 0 ? silu_f(acc) : acc);
    }
    if (K > 1 && t0 == 0) rewrite_state<T, K>(a, st, begin, len, c, scale, has_history);
}

// ONE: no portion is longer than a walk.  (With the registers of a rewrite from memory fewer than 16 CTAs fit an SM.)
template <typename T, int K, bool ONE>
__global__ void __launch_bounds__(128, 16) conv_walk_kernel(ConvArgs a) {
    int b = blockIdx.z, t0 = 0;
    if (!ONE) find_run(a, b, t0);
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= a.C) return;
    const int begin = a.cu_seqlens[b], len = a.cu_seqlens[b + 1] - begin;
    if (t0 >= len) return;
    const int t1 = ONE ? len : min(len, t0 + kWalk);
    const float scale = c < a.end0 ? a.s0 : (c < a.end1 ? a.s1 : a.s2);
    const bool has_history = a.start_pos[b] > 0;
    T* st = (T*)a.state + ((size_t)a.slots[b] * a.C + c) * (K - 1);
    float w[K], win[K];
#pragma unroll
    for (int j = 0; j < K; ++j) w[j] = a.weight[(size_t)c * K + j];
#pragma unroll
    for (int j = 0; j < K - 1; ++j) {
        const int idx = t0 - (K - 1) + j;
        win[j] = idx >= 0 ? scaled_input<T>(a, begin + idx, c, scale) : (has_history ? to_f32(st[K - 1 + idx]) : 0.f);
    }
    const float bias = a.bias ? a.bias[c] : 0.f;
    for (int t = t0; t < t1; ++t) {
        win[K - 1] = scaled_input<T>(a, begin + t, c, scale);
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < K; ++j) acc += win[j] * w[j];
        acc = round_to<T>(acc + bias);
        ((T*)a.out)[(size_t)(begin + t) * a.C + c] = from_f32<T>(a.act == 0 ? silu_f(acc) : acc);
#pragma unroll
        for (int j = 0; j < K - 1; ++j) win[j] = win[j + 1];
    }
    if (K == 1 || t0 > 0) return;
    if (!ONE && t1 < len) rewrite_state<T, K>(a, st, begin, len, c, scale, has_history);
    else {                                                // one run: win holds the last inputs
#pragma unroll
        for (int j = 0; j < K - 1; ++j) st[j] = from_f32<T>(win[j]);
    }
}

// The same for bfloat16 with eight channels per thread and 16-byte loads and stores: channels, the region
// edges and the row stride must be multiples of 8 and the input 16-byte aligned.  Portions of up to kVecChunk
// tokens: a thread takes a whole one, its rows fetched together so that several loads are in flight.
constexpr int kVecChunk = 8;

__device__ __forceinline__ void unpack8(const uint4& v, float* f) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 p = __bfloat1622float2(h[i]); f[2 * i] = p.x; f[2 * i + 1] = p.y; }
}

template <int K>
__global__ void __launch_bounds__(128) conv_forward_vec_kernel(ConvArgs a) {
    typedef __nv_bfloat16 T;
    pdl_wait();
    const int cg = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = cg * 8;
    if (c >= a.C) return;
    const int b = blockIdx.z;
    const int begin = a.cu_seqlens[b], n = a.cu_seqlens[b + 1] - begin;
    if (n <= 0) return;
    const float scale = c < a.end0 ? a.s0 : (c < a.end1 ? a.s1 : a.s2);
    const bool has_history = a.start_pos[b] > 0;
    const T* x = (const T*)a.x;
    T* st = (T*)a.state + ((size_t)a.slots[b] * a.C + c) * (K - 1);
    // The portion's rows, the thread's taps (8 * K consecutive floats) and its biases are fetched as 16-byte
    // pieces up front, so that all of them are in flight together: one after the other, each waited for,
    // they were most of the kernel's time.
    uint4 rows[kVecChunk];
#pragma unroll
    for (int i = 0; i < kVecChunk; ++i)
        if (i < n) rows[i] = *reinterpret_cast<const uint4*>(x + (size_t)(begin + i) * a.x_stride + c);
    float w[8][K], win[8][K], bias[8];
    {
        float4 raw[2 * K];
        const float4* wp = reinterpret_cast<const float4*>(a.weight + (size_t)c * K);
#pragma unroll
        for (int i = 0; i < 2 * K; ++i) raw[i] = __ldg(wp + i);
        float4 b0 = make_float4(0.f, 0.f, 0.f, 0.f), b1 = b0;
        if (a.bias) { b0 = __ldg(reinterpret_cast<const float4*>(a.bias + c)); b1 = __ldg(reinterpret_cast<const float4*>(a.bias + c) + 1); }
        bias[0] = b0.x; bias[1] = b0.y; bias[2] = b0.z; bias[3] = b0.w; bias[4] = b1.x; bias[5] = b1.y; bias[6] = b1.z; bias[7] = b1.w;
        const float* flat = reinterpret_cast<const float*>(raw);
#pragma unroll
        for (int e = 0; e < 8; ++e)
#pragma unroll
            for (int j = 0; j < K; ++j) w[e][j] = flat[e * K + j];
    }
    // the thread's 8 channels' saved inputs are 8 * (K - 1) consecutive values: K - 1 pieces of 16 bytes, asked for
    // together (one 2-byte load per value made a decode step's conv a chain of dependent loads)
    __align__(16) T hist[8 * (K - 1)];
    if (has_history) {
#pragma unroll
        for (int j = 0; j < K - 1; ++j) reinterpret_cast<uint4*>(hist)[j] = reinterpret_cast<const uint4*>(st)[j];
    }
#pragma unroll
    for (int j = 0; j < K - 1; ++j)
#pragma unroll
        for (int e = 0; e < 8; ++e) win[e][j] = has_history ? __bfloat162float(hist[e * (K - 1) + j]) : 0.f;
#pragma unroll
    for (int i = 0; i < kVecChunk; ++i) {
        if (i < n) {
            float f[8];
            unpack8(rows[i], f);
            __nv_bfloat162 o[4];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                win[e][K - 1] = round_to<T>(f[e] * scale);
                float acc = 0.f;
#pragma unroll
                for (int j = 0; j < K; ++j) acc += win[e][j] * w[e][j];
                acc = round_to<T>(acc + bias[e]);
                if (a.act == 0) acc = silu_fast(acc);                            // the result is rounded to bfloat16 next
                if (e & 1) o[e >> 1].y = __float2bfloat16_rn(acc); else o[e >> 1].x = __float2bfloat16_rn(acc);
#pragma unroll
                for (int j = 0; j < K - 1; ++j) win[e][j] = win[e][j + 1];
            }
            *reinterpret_cast<uint4*>((T*)a.out + (size_t)(begin + i) * a.C + c) = *reinterpret_cast<uint4*>(o);
        }
    }
    __align__(16) T next[8 * (K - 1)];
#pragma unroll
    for (int e = 0; e < 8; ++e)
#pragma unroll
        for (int j = 0; j < K - 1; ++j) next[e * (K - 1) + j] = __float2bfloat16_rn(win[e][j]);
#pragma unroll
    for (int j = 0; j < K - 1; ++j) reinterpret_cast<uint4*>(st)[j] = reinterpret_cast<const uint4*>(next)[j];
}

// Long portions (bfloat16, the same alignment rules): a CTA of 256 threads stages kTileTokens + K - 1 rows of 256
// channels in shared memory, already scaled and rounded, each row fetched once with 16-byte loads that are all in
// flight together; a thread then walks 4 consecutive tokens of 8 channels.  One thread per 32 outputs instead of
// per 64 with the rows shared through shared memory: four times the warps of the register form above, which at
// 2,048 tokens left the SMs a dozen warps each.
constexpr int kTileGroups = 32, kTileThreads = 256;

template <int K, int kTileTokens>
__global__ void __launch_bounds__(kTileThreads, 3) conv_forward_tile_kernel(ConvArgs a) {
    typedef __nv_bfloat16 T;
    constexpr int kRows = kTileTokens + K - 1;
    __shared__ __align__(16) T tile[kRows][kTileGroups * 8];
    int b, t0;
    find_run(a, b, t0);
    const int begin = a.cu_seqlens[b], len = a.cu_seqlens[b + 1] - begin;
    if (t0 >= len) {
        pdl_wait();
        return;
    }
    const int c0 = blockIdx.x * kTileGroups * 8;
    const bool has_history = a.start_pos[b] > 0;
    const T* x = (const T*)a.x;
    T* st = (T*)a.state + (size_t)a.slots[b] * a.C * (K - 1);
    const int g = threadIdx.x % kTileGroups, ts = threadIdx.x / kTileGroups;
    const int c = c0 + g * 8;
    const bool live = c < a.C;
    // The CTA's taps and biases go through shared memory: its 256 channels are one contiguous run of K * 256 floats,
    // fetched coalesced.  (A thread fetching its own 8 * K floats makes every load instruction of a warp touch 32
    // different lines; that was most of this kernel's time.)  A thread's 8 channels lie 8 * K + 4 floats from the
    // next thread's, so that the 16-byte reads below spread over all banks.
    constexpr int kWPitch = 8 * K + 4;
    __shared__ __align__(16) float w_s[kTileGroups * kWPitch];
    __shared__ __align__(16) float bias_s[kTileGroups * 8];
    for (int f = threadIdx.x; f < kTileGroups * 8 * K; f += kTileThreads) {
        const int ch = f / K, j = f - ch * K;
        w_s[(ch >> 3) * kWPitch + (ch & 7) * K + j] = c0 + ch < a.C ? __ldg(a.weight + (size_t)c0 * K + f) : 0.f;
    }
    bias_s[threadIdx.x] = (a.bias != nullptr && c0 + (int)threadIdx.x < a.C) ? __ldg(a.bias + c0 + threadIdx.x) : 0.f;
    pdl_wait();                                           // tables, taps and biases are not the kernel's before this one; x is
    // rows t0 - (K - 1) .. t0 + kTileTokens - 1 of the portion; row rr of the tile, channel group g
    constexpr int kPer = (kRows + kTileThreads / kTileGroups - 1) / (kTileThreads / kTileGroups);
    const float scale = c < a.end0 ? a.s0 : (c < a.end1 ? a.s1 : a.s2);
    uint4 fetched[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int rr = ts + i * (kTileThreads / kTileGroups), idx = t0 - (K - 1) + rr;
        if (live && rr < kRows && idx >= 0 && idx < len)
            fetched[i] = *reinterpret_cast<const uint4*>(x + (size_t)(begin + idx) * a.x_stride + c);
    }
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int rr = ts + i * (kTileThreads / kTileGroups), idx = t0 - (K - 1) + rr;
        if (!live || rr >= kRows) continue;
        __nv_bfloat162 o[4];
        if (idx >= 0 && idx < len) {
            float f[8];
            unpack8(fetched[i], f);
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = __floats2bfloat162_rn(f[2 * e] * scale, f[2 * e + 1] * scale);
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) {                 // before the portion: the saved inputs, or zeros
                const T v = (idx < 0 && has_history) ? st[(size_t)(c + e) * (K - 1) + K - 1 + idx] : __float2bfloat16_rn(0.f);
                if (e & 1) o[e >> 1].y = v; else o[e >> 1].x = v;
            }
        }
        *reinterpret_cast<uint4*>(&tile[rr][g * 8]) = *reinterpret_cast<uint4*>(o);
    }
    __syncthreads();
    // the portion's first run rewrites the saved inputs once all have read them, a channel per thread: from the tile if the portion lies in it
    const int mine = c0 + threadIdx.x;
    if (t0 == 0 && mine < a.C) {
        T* to = st + (size_t)mine * (K - 1);
        if (len <= kTileTokens) {
#pragma unroll
            for (int j = 0; j < K - 1; ++j) to[j] = tile[len + j][threadIdx.x];
        } else rewrite_state<T, K>(a, to, begin, len, mine, mine < a.end0 ? a.s0 : (mine < a.end1 ? a.s1 : a.s2), has_history);
    }
    if (!live) return;
    float w[8][K], bias[8];
    {
        const float* flat = w_s + g * kWPitch;            // K * 8 floats: 16-byte reads when K is even, else single ones
#pragma unroll
        for (int e = 0; e < 8; ++e)
#pragma unroll
            for (int j = 0; j < K; ++j) w[e][j] = flat[e * K + j];
#pragma unroll
        for (int e = 0; e < 8; ++e) bias[e] = bias_s[g * 8 + e];
    }
    constexpr int kWalk = kTileTokens / (kTileThreads / kTileGroups);      // 4 consecutive tokens per thread
    const int first = ts * kWalk;
    float win[8][K];
#pragma unroll
    for (int j = 0; j < K - 1; ++j) {
        float f[8];
        unpack8(*reinterpret_cast<const uint4*>(&tile[first + j][g * 8]), f);
#pragma unroll
        for (int e = 0; e < 8; ++e) win[e][j] = f[e];
    }
#pragma unroll
    for (int i = 0; i < kWalk; ++i) {
        const int t = t0 + first + i;
        if (t >= len) break;
        float f[8];
        unpack8(*reinterpret_cast<const uint4*>(&tile[first + i + K - 1][g * 8]), f);
        __nv_bfloat162 o[4];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            win[e][K - 1] = f[e];
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < K; ++j) acc += win[e][j] * w[e][j];
            acc = round_to<T>(acc + bias[e]);
            if (a.act == 0) acc = silu_fast(acc);                            // the result is rounded to bfloat16 next
            if (e & 1) o[e >> 1].y = __float2bfloat16_rn(acc); else o[e >> 1].x = __float2bfloat16_rn(acc);
#pragma unroll
            for (int j = 0; j < K - 1; ++j) win[e][j] = win[e][j + 1];
        }
        *reinterpret_cast<uint4*>((T*)a.out + (size_t)(begin + t) * a.C + c) = *reinterpret_cast<uint4*>(o);
    }
}

// The grid for portions cut into runs of 1 << shift tokens: channels first (a row's CTAs side by side), then runs.
inline dim3 cut(ConvArgs& a, long tokens, int max_len, int shift, int across) {
    const long each = (max_len + (1L << shift) - 1) >> shift, runs = (tokens >> shift) + a.B;
    constexpr long kMost = 32768;                         // of the grid's y and z
    a.shift = shift;
    a.step = 0;
    if (each * a.B <= runs && each <= kMost && a.B <= kMost) return dim3(across, (unsigned)each, (unsigned)a.B);
    for (a.step = 1; (long)a.step * 32 < a.B;) a.step *= 32;
    return runs <= kMost ? dim3(across, (unsigned)runs) : dim3(across, (unsigned)kMost, (unsigned)((runs + kMost - 1) / kMost));
}

template <int K>
void launch_vec(ConvArgs& a, long tokens, int max_len, cudaStream_t s) {
    const int threads = 128, groups = a.C / 8;
    if (max_len <= kVecChunk) {
        launch_pdl(conv_forward_vec_kernel<K>, dim3((groups + threads - 1) / threads, 1, a.B), dim3(threads), 0, s, a);
    } else {
        // Runs of 32 tokens while they fill the GPU a few times over, then of 64: fewer inputs are read twice, fewer CTAs start (us, 32 /
        // 64: 1,792 channels and 8,192 tokens 25.9 / 26.0, 16,384 55 / 47.5; 3,584 and 8,192 56 / 48; 200 portions of 65 56 / 55).  Many portions
        // that end just behind a tile are the one range where two launches, the saved inputs in one of their own, were shorter: 3,584
        // channels, 200 portions of 65 101 us instead of 93, 100 of 130 87 instead of 83, 100 of 128 71 both ways.
        const bool large = tokens * a.C >= 18L << 20 && tokens >= 48L * a.B;
        const dim3 grid = cut(a, tokens, max_len, large ? 6 : 5, (groups + kTileGroups - 1) / kTileGroups);
        launch_pdl(large ? conv_forward_tile_kernel<K, 64> : conv_forward_tile_kernel<K, 32>, grid, dim3(kTileThreads), 0, s, a);
    }
}

inline bool vec_ok(const ConvArgs& a, int dtype) {
    return dtype == kBF16 && a.C % 8 == 0 && a.end0 % 8 == 0 && a.end1 % 8 == 0 && a.x_stride % 8 == 0 &&
           ((uintptr_t)a.x & 15) == 0 && ((uintptr_t)a.out & 15) == 0 && ((uintptr_t)a.weight & 15) == 0 &&
           ((uintptr_t)a.state & 15) == 0 &&
           (a.bias == nullptr || ((uintptr_t)a.bias & 15) == 0);
}

template <typename T>
int launch(ConvArgs& a, long tokens, int K, int max_len, cudaStream_t s) {
    // A walk's time is 0.24 us a token of the longest run plus 2; runs of 8 start at 4 and lose against it by the work there is.
    const int threads = 128, longest = max_len < kWalk ? max_len : kWalk;
    const bool walk = tokens * a.C >= 100000L * (longest - 12);
    const dim3 grid = cut(a, tokens, max_len, walk ? 6 : 3, (a.C + threads - 1) / threads);
#define LB_CONV_K(KK)                                                             \
    case KK:                                                                      \
        launch_pdl(!walk ? conv_forward_kernel<T, KK> : max_len <= kWalk && a.step == 0 ? conv_walk_kernel<T, KK, true> : conv_walk_kernel<T, KK, false>,  \
                   grid, dim3(threads), 0, s, a);                                 \
        break;
    switch (K) {
        LB_CONV_K(1) LB_CONV_K(2) LB_CONV_K(3) LB_CONV_K(4) LB_CONV_K(5) LB_CONV_K(6) LB_CONV_K(7) LB_CONV_K(8)
        default: return kBadSize;
    }
#undef LB_CONV_K
    return launch_status();
}
}  // namespace

// tokens: rows of x, all portions'; max_len: upper bound of a portion's.
extern "C" int lb_causal_conv1d(const void* x, long x_stride, const float* weight, const float* bias, void* state,
                                void* out, const int* cu_seqlens, const int* start_pos, const int* slots, int B,
                                long tokens, int max_len, int C, int K, int end0, int end1, float s0, float s1, float s2,
                                int act, int dtype, void* stream) {
    if (B <= 0 || max_len <= 0) return kOk;
    if (C <= 0 || K < 1 || K > 8 || act < 0 || act > 1) return kBadSize;
    ConvArgs a{x, x_stride, weight, bias, state, out, cu_seqlens, start_pos, slots, C, end0, end1, s0, s1, s2, act, B, 0, 0};
    if (vec_ok(a, dtype) && K >= 2 && K <= 5) {
        switch (K) {
            case 2: launch_vec<2>(a, tokens, max_len, (cudaStream_t)stream); break;
            case 3: launch_vec<3>(a, tokens, max_len, (cudaStream_t)stream); break;
            case 4: launch_vec<4>(a, tokens, max_len, (cudaStream_t)stream); break;
            default: launch_vec<5>(a, tokens, max_len, (cudaStream_t)stream); break;
        }
        return launch_status();
    }
    LB_DISPATCH_DTYPE(dtype, return launch<T>(a, tokens, K, max_len, (cudaStream_t)stream));
    return kOk;
}
