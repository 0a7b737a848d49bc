// Selective state-space scan (Mamba2), token by token.  The state is held in 32-bit while a portion runs and is kept
// between steps in 32-bit (the default) or, for bfloat16 models, in bfloat16 as the reference keeps it
// (python/logssms/cache/naive/manager.py:445-451: the state pool has the engine's dtype): half the bytes of a decode step's
// state update, one rounding of the state per step.
//
//   dt_h   = softplus(round(dt_raw_h * dt_scale) + dt_bias_h)        softplus(v) = v if v > 20 else log1p(e^v)
//   dA_h   = -exp(A_log_h) * dt_h
//   S_h   <- e^{dA_h} S_h + B_{g(h)} (x) (x_h * dt_h)                 S_h in R^{P x N}
//   y_h    = S_h C_{g(h)} + D_h x_h                                   (uses the updated state)
//   y_h   <- round(y_h) * round(silu(round(z_h * gate_scale)))          (optional: the gate of a mixer without norm)
// (python/logssms/kernel/linear_attention/mamba2.py:27-36 and :261-292; recurrence oracle
// tests/kernel/test_mamba2.py:22-38 of the reference.)
//
// This kernel runs a portion of any length from the request's saved state and writes the state back
// in place; a request whose portion starts at position 0 starts from zeros whatever the slot holds.
// A single decoded token is a portion of length one.  `req_list` restricts the launch to some requests of
// the batch (B then counts the list).  Grid (head, request, P tile of 16); 128 threads
// = 16 values of p x 8 lanes over N; each lane owns N/8 state values in registers (float4 strided),
// the sum over N ends with three shuffles.
// A second form (`beside`) walks the same items with a grid that is resident at once; see ssm_scan_persistent_kernel.
// A third one runs long portions of float32 models; see ssm_scan_blocks_kernel.  A fourth one runs the decode steps of
// bfloat16 models; see ssm_step_kernel.
#include "lb200/common.cuh"
using namespace lb200;

namespace {
constexpr int kPTile = 16;
constexpr int kLanesN = 8;

struct SsmArgs {
    const void* conv; int C; long conv_stride;   // [tokens, C] (row stride in elements): x | B | C after the conv
    const void* dt; long dt_stride;              // [tokens, nh] view
    const float* A_log; const float* dt_bias; const float* D;
    void* state;                                 // [slots, nh, P, N], float or (state_bf16) bfloat16
    void* y;                                     // [tokens, nh * P]
    const int* cu_seqlens; const int* start_pos; const int* slots;
    int nh, P, N, G; float dt_scale;
    const void* gate; long gate_stride; float gate_scale;   // optional [tokens, nh * P] view: y *= silu(gate * scale)
    const int* req_list;                         // optional: the requests (indices in the batch) to run
    int beside;                                  // the launch shares the GPU with other kernels of the step: leave them SM slots
    int state_bf16;
    int longest;                                 // upper bound of the portions' tokens (0: not known)
    long tokens;                                 // rows of the step
};

template <typename T> __device__ __forceinline__ void load4(const T* p, float* f);
template <> __device__ __forceinline__ void load4<float>(const float* p, float* f) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
}
template <> __device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float* f) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
    float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}

// four consecutive state values, from or to the dtype the state is kept in
__device__ __forceinline__ void state_load4(const float* p, float* f) { load4<float>(p, f); }
__device__ __forceinline__ void state_load4(const __nv_bfloat16* p, float* f) { load4<__nv_bfloat16>(p, f); }
__device__ __forceinline__ void state_store4(float* p, const float* f) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
}
__device__ __forceinline__ void state_store4(__nv_bfloat16* p, const float* f) {
    __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
    uint2 v;
    v.x = *reinterpret_cast<uint32_t*>(&a);
    v.y = *reinterpret_cast<uint32_t*>(&b);
    *reinterpret_cast<uint2*>(p) = v;
}

// The tokens of one portion through the state values S that the thread holds (thread (pi, nl): row p of head h, the
// state columns i * 32 + nl * 4 .. + 3): y for its row, S updated.
template <typename T, int NPT, bool ALIGNED>
__device__ __forceinline__ void scan_tokens(const SsmArgs& a, int h, int p, bool p_ok, int nl, int begin, int len, float (&S)[NPT]) {
    const int g = h / (a.nh / a.G);
    const int inner = a.nh * a.P;
    const int N = a.N;
    const float negA = -expf(a.A_log[h]);
    const float dt_bias = a.dt_bias[h], Dh = a.D[h];
    const T* conv = (const T*)a.conv;
    const T* dtp = (const T*)a.dt;
#pragma unroll 2
    for (int t = 0; t < len; ++t) {
        const size_t tok = (size_t)(begin + t);
        const T* row = conv + tok * a.conv_stride;
        float dt = round_to<T>(to_f32(dtp[tok * a.dt_stride + h]) * a.dt_scale) + dt_bias;
        dt = dt > 20.f ? dt : log1pf(expf(dt));
        const float decay = expf(negA * dt);
        const float xv = p_ok ? to_f32(row[h * a.P + p]) : 0.f;
        const float u = xv * dt;
        const T* Bp = row + inner + g * N;
        const T* Cp = Bp + a.G * N;
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < NPT / 4; ++i) {
            const int n0 = i * 32 + nl * 4;
            if (n0 < N) {
                float Bv[4], Cv[4];
                if (ALIGNED) {
                    load4<T>(Bp + n0, Bv);
                    load4<T>(Cp + n0, Cv);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) { Bv[e] = to_f32(Bp[n0 + e]); Cv[e] = to_f32(Cp[n0 + e]); }
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    S[4 * i + e] = S[4 * i + e] * decay + Bv[e] * u;
                    acc += S[4 * i + e] * Cv[e];
                }
            }
        }
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        acc += __shfl_xor_sync(0xffffffffu, acc, 4);
        if (nl == 0 && p_ok) {
            float yv = acc + Dh * xv;
            if (a.gate != nullptr) {                      // the mixer's gate when it has no norm (fused.py:9-19)
                const float zg = round_to<T>(to_f32(((const T*)a.gate)[tok * a.gate_stride + h * a.P + p]) * a.gate_scale);
                yv = round_to<T>(yv) * round_to<T>(silu_f(zg));
            }
            ((T*)a.y)[tok * inner + h * a.P + p] = from_f32<T>(yv);
        }
    }
}

// NPT: state values per thread (N <= 8 * NPT).  ALIGNED: 4-element vector loads of B and C are legal.
template <typename T, typename ST, int NPT, bool ALIGNED>
__global__ void __launch_bounds__(kPTile * kLanesN) ssm_scan_kernel(SsmArgs a) {
    pdl_trigger();
    const int h = blockIdx.x, b = a.req_list ? a.req_list[blockIdx.y] : blockIdx.y;
    const int pi = threadIdx.x / kLanesN, nl = threadIdx.x % kLanesN;
    const int p = blockIdx.z * kPTile + pi;
    const bool p_ok = p < a.P;
    const int begin = a.cu_seqlens[b], len = a.cu_seqlens[b + 1] - begin;
    if (len <= 0) {
        pdl_wait();                                       // a grid that ended without waiting would let the kernel behind it start too early
        return;
    }
    const int N = a.N;
    ST* sp = (ST*)a.state + (((size_t)a.slots[b] * a.nh + h) * a.P + (p_ok ? p : 0)) * N;

    float S[NPT];
    const bool fresh = a.start_pos[b] <= 0;
#pragma unroll
    for (int i = 0; i < NPT / 4; ++i) {
        const int n0 = i * 32 + nl * 4;
        if (!fresh && p_ok && n0 < N) {
            state_load4(sp + n0, &S[4 * i]);
        } else {
            S[4 * i] = S[4 * i + 1] = S[4 * i + 2] = S[4 * i + 3] = 0.f;
        }
    }
    // Up to here only step tables, constants and the saved state were read: with a programmatic launch that runs
    // under the kernel before (the projection and conv that make x, B, C and dt), whose results are read from here on.
    pdl_wait();
    scan_tokens<T, NPT, ALIGNED>(a, h, p, p_ok, nl, begin, len, S);
    if (p_ok) {
#pragma unroll
        for (int i = 0; i < NPT / 4; ++i) {
            const int n0 = i * 32 + nl * 4;
            if (n0 < N) state_store4(sp + n0, &S[4 * i]);
        }
    }
}

// A portion of several tokens through one row, out of line: the registers of the kernel that calls it are not its own.
template <typename T, typename ST, int NPT>
__device__ __noinline__ void walk_row(const SsmArgs& a, int h, int p, bool p_ok, int nl, int begin, int len, bool fresh, ST* state) {
    float S[NPT];
    ST* sp = state + (size_t)(p_ok ? p : 0) * a.N;
#pragma unroll
    for (int i = 0; i < NPT / 4; ++i) {
        const int n0 = i * 32 + nl * 4;
        S[4 * i] = S[4 * i + 1] = S[4 * i + 2] = S[4 * i + 3] = 0.f;
        if (!fresh && p_ok && n0 < a.N) state_load4(sp + n0, &S[4 * i]);
    }
#pragma unroll 1
    for (int t = 0; t < len; ++t) scan_tokens<T, NPT, true>(a, h, p, p_ok, nl, begin + t, 1, S);
#pragma unroll
    for (int i = 0; i < NPT / 4; ++i) {
        const int n0 = i * 32 + nl * 4;
        if (p_ok && n0 < a.N) state_store4(sp + n0, &S[4 * i]);
    }
}

// A decode step of a bfloat16 model: every request has one token (another number is walked as above).  The kernel above spends most of a CTA's life waiting, for
// the step's tables, then for the state of its 16 rows, then for dt, x, B and C, then it is gone: 2.1 TB/s at 24 requests,
// 3.1 at 64.  Here a CTA takes `tiles` tiles of 16 rows of one head, one after the other: tables, dt, decay, B and C (kept as
// bfloat16 pairs) once, the next tile's state, x and gate on their way while a tile is worked on.  V: consecutive state
// values of a lane, 16 bytes of them.  The sums have the order of the form above where V is 4 (float32 states).
// Alone, states from HBM, the general form / this one: 24 requests of 24 heads of 128 x 256, bfloat16 states (75.5 MB) 27.6 /
// 17.4 us; 24 of 64 x 256, float32 (75.5 MB) 19.5 / 15.9; 13 of them 12.9 / 10.5; 64 of 64 x 128 (101 MB) 23.9 / 21.8; 64 of
// 128 x 256 (403 MB) 79.2 / 67.6 (6.0 TB/s); 8 of 64 x 128 5.5 / 4.2.
// WHOLE: every lane's columns lie below N.
template <typename ST, int NPT, bool WHOLE>
__global__ void __launch_bounds__(kPTile * kLanesN, 4) ssm_step_kernel(const __grid_constant__ SsmArgs a, int tiles) {
    typedef __nv_bfloat16 T;
    constexpr int V = 16 / sizeof(ST), kPieces = NPT / V;
    pdl_trigger();
    const int h = blockIdx.x, b = blockIdx.y;
    const int pi = threadIdx.x / kLanesN, nl = threadIdx.x % kLanesN;
    const int begin = a.cu_seqlens[b], len = a.cu_seqlens[b + 1] - begin;
    const int slot = a.slots[b];
    const bool fresh = a.start_pos[b] <= 0;
    const int N = a.N, inner = a.nh * a.P;
    const int p0 = blockIdx.z * tiles * kPTile + pi, p_end = min(a.P, (int)(blockIdx.z + 1) * tiles * kPTile);
    ST* state = (ST*)a.state + ((size_t)slot * a.nh + h) * a.P * N;
    if (len != 1) {                                       // no token; or more than the caller promised: as the form above
        pdl_wait();
        if (len > 1)
            for (int p = p0; p - pi < p_end; p += kPTile) walk_row<T, ST, NPT>(a, h, p, p < p_end, nl, begin, len, fresh, state);
        return;
    }
    uint4 raw[kPieces];
    auto fetch = [&](int p) {
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int n0 = (i * kLanesN + nl) * V;
            raw[i] = (!fresh && p < p_end && n0 < N) ? *reinterpret_cast<const uint4*>(state + (size_t)p * N + n0) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    fetch(p0);
    const float negA = -expf(a.A_log[h]), dt_bias = a.dt_bias[h], Dh = a.D[h];
    pdl_wait();                                           // the projection and conv before this kernel: x, B, C, dt, gate
    const size_t tok = (size_t)begin;
    const T* row = (const T*)a.conv + tok * a.conv_stride;
    const T* zrow = a.gate == nullptr ? nullptr : (const T*)a.gate + tok * a.gate_stride + h * a.P;
    const T* Bp = row + inner + (h / (a.nh / a.G)) * N;
    const T* Cp = Bp + a.G * N;
    uint32_t Bv[NPT / 2], Cv[NPT / 2];                    // pairs of bfloat16
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
        const int n0 = (i * kLanesN + nl) * V;
#pragma unroll
        for (int q = 0; q < V / 4; ++q) {
            uint2 bv = make_uint2(0u, 0u), cv = bv;
            if (n0 < N) { bv = *reinterpret_cast<const uint2*>(Bp + n0 + 4 * q); cv = *reinterpret_cast<const uint2*>(Cp + n0 + 4 * q); }
            Bv[(i * V + 4 * q) / 2] = bv.x; Bv[(i * V + 4 * q) / 2 + 1] = bv.y;
            Cv[(i * V + 4 * q) / 2] = cv.x; Cv[(i * V + 4 * q) / 2 + 1] = cv.y;
        }
    }
    float xv = p0 < p_end ? to_f32(row[h * a.P + p0]) : 0.f;
    float zv = zrow != nullptr && p0 < p_end ? to_f32(zrow[p0]) : 0.f;
    float dt = round_to<T>(to_f32(((const T*)a.dt)[tok * a.dt_stride + h]) * a.dt_scale) + dt_bias;
    dt = dt > 20.f ? dt : log1pf(expf(dt));
    const float decay = expf(negA * dt);
#pragma unroll 1
    for (int p = p0; p - pi < p_end; p += kPTile) {
        float S[NPT];
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if constexpr (sizeof(ST) == 4) S[V * i + e] = __uint_as_float(w[e]);
                else { S[V * i + 2 * e] = __uint_as_float(w[e] << 16); S[V * i + 2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u); }
            }
        }
        const float x = xv, z = zv, u = x * dt;
        const int pn = p + kPTile;                        // the next tile's values are on their way from here
        fetch(pn);
        xv = pn < p_end ? to_f32(row[h * a.P + pn]) : 0.f;
        zv = zrow != nullptr && pn < p_end ? to_f32(zrow[pn]) : 0.f;
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < NPT / 2; ++j) {
            // B and C stay packed: widened ahead of the loop they would take the registers of a CTA per SM
            asm volatile("" : "+r"(Bv[j]), "+r"(Cv[j]));
            const float uj = WHOLE || (2 * j / V * kLanesN + nl) * V < N ? u : 0.f;      // columns from N on stay zeros, also under an infinite u
            S[2 * j] = S[2 * j] * decay + __uint_as_float(Bv[j] << 16) * uj;
            acc += S[2 * j] * __uint_as_float(Cv[j] << 16);
            S[2 * j + 1] = S[2 * j + 1] * decay + __uint_as_float(Bv[j] & 0xffff0000u) * uj;
            acc += S[2 * j + 1] * __uint_as_float(Cv[j] & 0xffff0000u);
        }
        if (p < p_end) {
#pragma unroll
            for (int i = 0; i < kPieces; ++i) {
                const int n0 = (i * kLanesN + nl) * V;
                if (n0 < N) {
#pragma unroll
                    for (int q = 0; q < V / 4; ++q) state_store4(state + (size_t)p * N + n0 + 4 * q, &S[V * i + 4 * q]);
                }
            }
        }
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        acc += __shfl_xor_sync(0xffffffffu, acc, 4);
        if (nl == 0 && p < p_end) {
            float yv = acc + Dh * x;
            if (zrow != nullptr) yv = round_to<T>(yv) * round_to<T>(silu_f(round_to<T>(z * a.gate_scale)));
            ((T*)a.y)[tok * inner + h * a.P + p] = from_f32<T>(yv);
        }
    }
}

// The same work as a grid that is resident all at once: every CTA walks (request, head, tile of p) items, the state of
// its next item on its way while it works on this one.  For the listed requests of a step that also holds prompt
// portions: the one-CTA-per-item grid above is thousands of CTAs that take every SM slot that frees up before any
// kernel launched after it gets one, so nothing could run beside it; this form leaves the other kernels of the step
// (the chunked kernels of the prompt portion, on another stream) their share of the SMs, while it streams the states.
constexpr int kPersistCtasPerSm = 3, kSmCount = 148;

template <typename T, typename ST, int NPT, bool ALIGNED>
__global__ void __launch_bounds__(kPTile * kLanesN) ssm_scan_persistent_kernel(SsmArgs a, int B, int ptiles) {
    extern __shared__ int facts[];                       // per listed request: state slot, starts from zeros?, first token, tokens
    pdl_trigger();
    for (int i = threadIdx.x; i < B; i += blockDim.x) {
        const int b = a.req_list ? a.req_list[i] : i;
        const int begin = b >= 0 ? a.cu_seqlens[b] : 0;
        facts[4 * i] = b >= 0 ? a.slots[b] : 0;
        facts[4 * i + 1] = b >= 0 ? (a.start_pos[b] <= 0) : 1;
        facts[4 * i + 2] = begin;
        facts[4 * i + 3] = b >= 0 ? a.cu_seqlens[b + 1] - begin : 0;      // an entry that names no request: no tokens
    }
    __syncthreads();
    const int pi = threadIdx.x / kLanesN, nl = threadIdx.x % kLanesN;
    const int N = a.N, per_request = a.nh * ptiles, total = B * per_request;
    // item -> (request index in the list, head, tile of p): tiles of a head, heads of a request follow one another, as
    // the state lies in memory
    auto state_of = [&](int item, int& bi, int& h, int& p, bool& p_ok) -> ST* {
        bi = item / per_request;
        const int r = item - bi * per_request;
        h = r / ptiles;
        p = (r - h * ptiles) * kPTile + pi;
        p_ok = p < a.P;
        return (ST*)a.state + (((size_t)facts[4 * bi] * a.nh + h) * a.P + (p_ok ? p : 0)) * N;
    };
    auto fetch = [&](int item, float (&S)[NPT]) {
        int bi, h, p; bool p_ok;
        const ST* sp = state_of(item, bi, h, p, p_ok);
        const bool read = p_ok && !facts[4 * bi + 1] && facts[4 * bi + 3] > 0;
#pragma unroll
        for (int i = 0; i < NPT / 4; ++i) {
            const int n0 = i * 32 + nl * 4;
            S[4 * i] = S[4 * i + 1] = S[4 * i + 2] = S[4 * i + 3] = 0.f;
            if (read && n0 < N) state_load4(sp + n0, &S[4 * i]);
        }
    };
    float S[NPT], Sn[NPT];
    int item = blockIdx.x;
    if (item < total) fetch(item, S);
    pdl_wait();
    while (item < total) {
        const int next = item + gridDim.x;
        if (next < total) fetch(next, Sn);               // on its way while this item is worked on
        int bi, h, p; bool p_ok;
        ST* sp = state_of(item, bi, h, p, p_ok);
        const int len = facts[4 * bi + 3];
        if (len > 0) {
            scan_tokens<T, NPT, ALIGNED>(a, h, p, p_ok, nl, facts[4 * bi + 2], len, S);
            if (p_ok) {
#pragma unroll
                for (int i = 0; i < NPT / 4; ++i) {
                    const int n0 = i * 32 + nl * 4;
                    if (n0 < N) state_store4(sp + n0, &S[4 * i]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NPT; ++i) S[i] = Sn[i];
        item = next;
    }
}

// Long portions of float32 models (no chunked form runs there): the tokens one after another as above, but in blocks of
// kBlock = 16.  B, C, x and gate of a block come to shared memory while the block before is worked on; the steps and
// the decays of 256 tokens are computed at a time, a token per thread (16 threads making them block by block, with two more
// barriers, kept the other seven warps waiting for an exponential, a logarithm and another exponential); a row's state lies over 16 lanes, so that the sums of a block's 16
// tokens over them cost 15 shuffles together; and the 16 tokens are one run of instructions without a branch (tokens past
// the end have B = C = x = 0 and a decay of 1), because with one or two warps on a scheduler the time is the chain of
// dependent instructions, not their number.  350 and 251 tokens, 24 heads of 64 x 128, beside the step's
// attention: 87 us, 115 with steps and decays block by block; alone the latter took 86, the form above 425,
// whose global loads and softplus are part of that chain.
constexpr int kBlock = 16, kLanesB = 16, kBlockThreads = kPTile * kLanesB;
static_assert(kBlock == kLanesB && kBlockThreads == kBlock * kPTile, "a thread per (token, row) of a block, a lane per token's sum");

__device__ __forceinline__ unsigned long long pair(float a, float b) {
    return (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
}
__device__ __forceinline__ float pair_sum(unsigned long long v) {
    return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// floats of one buffered block: B and C rows of Np values each, x and gate pieces
__host__ __device__ constexpr int block_floats(int Np) { return kBlock * (2 * Np + 2 * kPTile); }
static_assert(block_floats(64) % 4 == 0, "the second buffer starts on a 16-byte boundary");

// A portion of a few tokens (a decoded token beside the portions) through the row's lanes, straight from memory, in the order of
// sums of the blocks below: a block is computed whole, its 16 tokens' time for one.  Out of line: the registers of the blocks'
// form are not its own.  64 decoded tokens beside a portion of 9, 24 heads of 64 x 128: 37.9 us, 86.5 with a block each.
constexpr int kFewTokens = 4;
template <int Q, bool ALIGNED>
__device__ __noinline__ void scan_few(const SsmArgs& a, int h, int p, bool p_ok, int nl, int begin, int len, bool fresh, float* sp) {
    const int N = a.N, inner = a.nh * a.P, g = h / (a.nh / a.G);
    unsigned long long S[2 * Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        const int n0 = i * 64 + nl * 4;
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if (!fresh && p_ok && n0 < N) state_load4(sp + n0, f);
        S[2 * i] = pair(f[0], f[1]);
        S[2 * i + 1] = pair(f[2], f[3]);
    }
    const float negA = -expf(a.A_log[h]), dt_bias = a.dt_bias[h], Dh = a.D[h];
#pragma unroll 1
    for (int t = 0; t < len; ++t) {
        const size_t tok = (size_t)(begin + t);
        const float* row = (const float*)a.conv + tok * a.conv_stride;
        const float* Bp = row + inner + (size_t)g * N;
        const float* Cp = Bp + (size_t)a.G * N;
        float dt = ((const float*)a.dt)[tok * a.dt_stride + h] * a.dt_scale + dt_bias;
        dt = dt > 20.f ? dt : log1pf(expf(dt));
        const float d = expf(negA * dt), x = p_ok ? row[h * a.P + p] : 0.f;
        const unsigned long long decay = pair(d, d), u = pair(x * dt, x * dt);
        unsigned long long s0 = 0ull, s1 = 0ull;
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const int n0 = i * 64 + nl * 4;
            if (n0 < N) {
                float Bv[4], Cv[4];
                if (ALIGNED) {
                    load4<float>(Bp + n0, Bv);
                    load4<float>(Cp + n0, Cv);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) { Bv[e] = Bp[n0 + e]; Cv[e] = Cp[n0 + e]; }
                }
                S[2 * i] = fma2(S[2 * i], decay, mul2(pair(Bv[0], Bv[1]), u));
                S[2 * i + 1] = fma2(S[2 * i + 1], decay, mul2(pair(Bv[2], Bv[3]), u));
                s0 = fma2(S[2 * i], pair(Cv[0], Cv[1]), s0);
                s1 = fma2(S[2 * i + 1], pair(Cv[2], Cv[3]), s1);
            }
        }
        float acc = pair_sum(s0) + pair_sum(s1);
#pragma unroll
        for (int o = kLanesB / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (nl == 0 && p_ok) {
            float yv = acc + Dh * x;
            if (a.gate != nullptr) yv *= silu_f(((const float*)a.gate)[tok * a.gate_stride + h * a.P + p] * a.gate_scale);
            ((float*)a.y)[tok * inner + h * a.P + p] = yv;
        }
    }
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        const int n0 = i * 64 + nl * 4;
        const float f[4] = {__uint_as_float((uint32_t)S[2 * i]), __uint_as_float((uint32_t)(S[2 * i] >> 32)),
                            __uint_as_float((uint32_t)S[2 * i + 1]), __uint_as_float((uint32_t)(S[2 * i + 1] >> 32))};
        if (p_ok && n0 < N) state_store4(sp + n0, f);
    }
}

// Q: state columns per thread / 4; a row has Np = 64 * Q columns in shared memory, those from N on are zeros.  WHOLE: N is Np.
// (States of up to 64 columns: 64 registers, so that four CTAs fit an SM; with the 77 that the compiler takes otherwise it is three, and
// 16 portions of 64 tokens, 8 heads of 64 x 64, take a second wave: 22.9 us, 19.5 with four.)
template <int Q, bool ALIGNED, bool WHOLE>
__global__ void __launch_bounds__(kBlockThreads, Q == 1 ? 4 : 0) ssm_scan_blocks_kernel(const __grid_constant__ SsmArgs a) {
    constexpr int Np = 64 * Q, kBuffer = block_floats(Np);
    extern __shared__ __align__(16) float blocks[];            // two blocks, then (decay, decay) and the step of 256 tokens
    const int h = blockIdx.x, b = a.req_list ? a.req_list[blockIdx.y] : blockIdx.y;
    const int tid = threadIdx.x, pi = tid / kLanesB, nl = tid % kLanesB;
    const int p0 = blockIdx.z * kPTile, p = p0 + pi;
    const bool p_ok = p < a.P;
    const int N = a.N, inner = a.nh * a.P, g = h / (a.nh / a.G);
    unsigned long long* decays = reinterpret_cast<unsigned long long*>(blocks + 2 * kBuffer);      // [kBlockThreads]
    float* steps = reinterpret_cast<float*>(decays + kBlockThreads);                               // [kBlockThreads]
    const int begin = b >= 0 ? a.cu_seqlens[b] : 0, len = b >= 0 ? a.cu_seqlens[b + 1] - begin : 0;
    if (len <= 0) return;
    float* sp = (float*)a.state + (((size_t)a.slots[b] * a.nh + h) * a.P + (p_ok ? p : 0)) * N;
    const bool fresh = a.start_pos[b] <= 0;
    if (len <= kFewTokens) {
        scan_few<Q, ALIGNED>(a, h, p, p_ok, nl, begin, len, fresh, sp);
        return;
    }
    unsigned long long S[2 * Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        const int n0 = i * 64 + nl * 4;
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if (!fresh && p_ok && n0 < N) state_load4(sp + n0, f);
        S[2 * i] = pair(f[0], f[1]);
        S[2 * i + 1] = pair(f[2], f[3]);
    }
    const float negA = -expf(a.A_log[h]), dt_bias = a.dt_bias[h], Dh = a.D[h];
    const float* conv = (const float*)a.conv;
    auto copy4 = [](float* dst, const float* src, int bytes) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes));
    };
    // everything outside the portion, its rows or N comes as zeros
    constexpr int kPiece = ALIGNED ? 4 : 1, kPerRow = 2 * Np / kPiece;
    constexpr bool kSameColumn = kBlockThreads % kPerRow == 0;  // all of a thread's pieces of B and C are of one column: its place is worked out once
    auto column = [&](int i) { return i % kPerRow * kPiece; };
    auto place = [&](int c) { return conv + (size_t)begin * a.conv_stride + inner + (size_t)(c < Np ? g : a.G + g) * N + c % Np; };
    const int my_c = column(tid);
    const float* my_bc = place(my_c);
    const int xt = tid / kPTile, xq = tid % kPTile;
    const bool x_ok = p0 + xq < a.P;
    const float* my_x = conv + (size_t)begin * a.conv_stride + h * a.P + p0 + (x_ok ? xq : 0);
    const float* my_z = a.gate == nullptr ? nullptr : (const float*)a.gate + (size_t)begin * a.gate_stride + h * a.P + p0 + (x_ok ? xq : 0);
    auto fetch = [&](int t0) {
        float* dst = blocks + (t0 / kBlock & 1) * kBuffer;
#pragma unroll
        for (int i = tid; i < kBlock * kPerRow; i += kBlockThreads) {
            const int t = i / kPerRow, c = kSameColumn ? my_c : column(i);
            const bool ok = t0 + t < len && c % Np < N;
            const float* src = ok ? (kSameColumn ? my_bc : place(c)) + (size_t)(t0 + t) * a.conv_stride : conv;
            if (ALIGNED)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + t * 2 * Np + c)), "l"(src), "r"(ok ? 16 : 0));
            else copy4(dst + t * 2 * Np + c, src, ok ? 4 : 0);
        }
        float* xs = dst + kBlock * 2 * Np;
        const bool ok = t0 + xt < len && x_ok;
        copy4(xs + tid, ok ? my_x + (size_t)(t0 + xt) * a.conv_stride : conv, ok ? 4 : 0);
        if (a.gate != nullptr) copy4(xs + kBlockThreads + tid, ok ? my_z + (size_t)(t0 + xt) * a.gate_stride : my_z, ok ? 4 : 0);
    };
    fetch(0);
    asm volatile("cp.async.commit_group;");
    for (int t0 = 0; t0 < len; t0 += kBlock) {
        if (t0 + kBlock < len) fetch(t0 + kBlock);             // into the buffer that was read before the last barrier
        asm volatile("cp.async.commit_group;");
        if (t0 % kBlockThreads == 0) {                         // the steps and decays of the next 256 tokens
            float dt = 0.f, decay = 1.f;
            if (t0 + tid < len) {
                dt = ((const float*)a.dt)[(size_t)(begin + t0 + tid) * a.dt_stride + h] * a.dt_scale + dt_bias;
                dt = dt > 20.f ? dt : log1pf(expf(dt));
                decay = expf(negA * dt);
            }
            steps[tid] = dt;
            decays[tid] = pair(decay, decay);
        }
        asm volatile("cp.async.wait_group 1;");
        __syncthreads();
        const float* bc = blocks + (t0 / kBlock & 1) * kBuffer;
        const float* xs = bc + kBlock * 2 * Np;
        const unsigned long long* turn = decays + t0 % kBlockThreads;
        const float* step = steps + t0 % kBlockThreads;
        float acc[kBlock];
#pragma unroll
        for (int t = 0; t < kBlock; ++t) {
            const float ut = xs[t * kPTile + pi] * step[t];
            const unsigned long long decay = turn[t], u = pair(ut, ut);
            unsigned long long s0 = 0ull, s1 = 0ull;
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                const float* row = bc + t * 2 * Np + i * 64 + nl * 4;
                const ulonglong2 Bv = *reinterpret_cast<const ulonglong2*>(row);
                const ulonglong2 Cv = *reinterpret_cast<const ulonglong2*>(row + Np);
                const unsigned long long ui = WHOLE || i * 64 + nl * 4 < N ? u : 0ull;      // zeros stay zeros, also under an infinite u
                S[2 * i] = fma2(S[2 * i], decay, mul2(Bv.x, ui));
                S[2 * i + 1] = fma2(S[2 * i + 1], decay, mul2(Bv.y, ui));
                s0 = fma2(S[2 * i], Cv.x, s0);
                s1 = fma2(S[2 * i + 1], Cv.y, s1);
            }
            acc[t] = pair_sum(s0) + pair_sum(s1);
        }
        // the tokens' sums over the row's lanes: lane nl ends with token nl's
#pragma unroll
        for (int o = kLanesB / 2; o > 0; o >>= 1) {
            const bool upper = nl & o;
#pragma unroll
            for (int j = 0; j < o; ++j) {
                const float give = upper ? acc[j] : acc[j + o], keep = upper ? acc[j + o] : acc[j];
                acc[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        if (t0 + nl < len && p_ok) {
            float yv = acc[0] + Dh * xs[nl * kPTile + pi];
            if (a.gate != nullptr) yv *= silu_f(xs[kBlockThreads + nl * kPTile + pi] * a.gate_scale);
            ((float*)a.y)[(size_t)(begin + t0 + nl) * inner + h * a.P + p] = yv;
        }
        __syncthreads();
    }
    if (p_ok) {
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const int n0 = i * 64 + nl * 4;
            const float f[4] = {__uint_as_float((uint32_t)S[2 * i]), __uint_as_float((uint32_t)(S[2 * i] >> 32)),
                                __uint_as_float((uint32_t)S[2 * i + 1]), __uint_as_float((uint32_t)(S[2 * i + 1] >> 32))};
            if (n0 < N) state_store4(sp + n0, f);
        }
    }
}

template <int Q, bool ALIGNED, bool WHOLE>
void launch_blocks_form(const SsmArgs& a, int B, cudaStream_t s) {
    constexpr size_t smem = 2 * block_floats(64 * Q) * sizeof(float) + kBlockThreads * (8 + sizeof(float));
    static size_t have = 0;
    ensure_dynamic_smem(ssm_scan_blocks_kernel<Q, ALIGNED, WHOLE>, smem, have);
    ssm_scan_blocks_kernel<Q, ALIGNED, WHOLE><<<dim3(a.nh, B, (a.P + kPTile - 1) / kPTile), kBlockThreads, smem, s>>>(a);
}
template <int Q, bool ALIGNED>
void launch_blocks(const SsmArgs& a, int B, cudaStream_t s) {
    if (a.N == 64 * Q) launch_blocks_form<Q, ALIGNED, true>(a, B, s);
    else launch_blocks_form<Q, ALIGNED, false>(a, B, s);
}

template <typename T, typename ST, int NPT>
void launch_npt(const SsmArgs& a, int B, bool aligned, cudaStream_t s) {
    const int ptiles = (a.P + kPTile - 1) / kPTile;
    if constexpr (sizeof(T) == 4) {
        // From portions of a few tokens on the blocks' set-up is paid for (one decoded token: the form below starts early); but
        // where most portions are shorter than that (below 8 tokens on average) and the longest one's chain, about 1.5 us a token,
        // is over before the form below has gone through all of them (0.35 us and more a request of 24 heads of 64 x 128), that one
        // is ahead: 128 tokens beside a portion of 9 57.9 against 73.7 us, 64 portions of 4 beside it 57.3 against 74.8, 128 tokens
        // with 256 state columns 93 against 129; 24 tokens beside a portion of 20, the other way, 38.4 against 22.0, 64 portions of
        // 12 119 against 88.
        const bool chain_hidden = 3L * a.longest + 10 < (long)B * a.nh * ptiles * a.N / (96 * 128);
        if (a.longest > 8 && !(chain_hidden && a.tokens < 8L * B)) {
            constexpr int Q = NPT <= 8 ? 1 : NPT / 8;
            if (aligned) launch_blocks<Q, true>(a, B, s);
            else launch_blocks<Q, false>(a, B, s);
            return;
        }
    }
    if (a.beside && (long)B * a.nh * ptiles > kPersistCtasPerSm * kSmCount && B <= 4096) {
        const int ctas = kPersistCtasPerSm * kSmCount;
        const size_t smem = (size_t)B * 4 * sizeof(int);
        if (aligned) ssm_scan_persistent_kernel<T, ST, NPT, true><<<ctas, kPTile * kLanesN, smem, s>>>(a, B, ptiles);
        else ssm_scan_persistent_kernel<T, ST, NPT, false><<<ctas, kPTile * kLanesN, smem, s>>>(a, B, ptiles);
        return;
    }
    if constexpr (sizeof(T) == 2 && NPT >= 16 / (int)sizeof(ST)) {
        // 16-byte pieces of the state, 8-byte ones of B and C
        if (a.longest == 1 && a.req_list == nullptr && aligned && a.N % (16 / (int)sizeof(ST)) == 0 && ((uintptr_t)a.state & 15) == 0) {
            // Tiles per CTA: a CTA's start (tables, dt, B, C, the first state) takes about as long as three tiles, and
            // the CTAs come in rounds of what the SMs hold.
            const long slots = kSmCount * (NPT >= 32 ? 4 : NPT >= 16 ? 5 : 8);
            int tiles = 1;
            long best = 0;
            for (int t = 1; t < 2 * ptiles; t *= 2) {
                const long ctas = (long)B * a.nh * ((ptiles + t - 1) / t), cost = (ctas + slots - 1) / slots * (3 + (t < ptiles ? t : ptiles));
                if (t == 1 || cost < best) { best = cost; tiles = t; }
            }
            launch_pdl_if(B <= kPdlMaxRows, a.N == NPT * kLanesN ? ssm_step_kernel<ST, NPT, true> : ssm_step_kernel<ST, NPT, false>,
                          dim3(a.nh, B, (ptiles + tiles - 1) / tiles), dim3(kPTile * kLanesN), 0, s, a, tiles);
            return;
        }
    }
    dim3 grid(a.nh, B, ptiles);
    // few requests: the kernel starts under the one before it and has its state in registers when that one ends
    const bool early = B <= kPdlMaxRows;
    if (aligned) launch_pdl_if(early, ssm_scan_kernel<T, ST, NPT, true>, grid, dim3(kPTile * kLanesN), 0, s, a);
    else launch_pdl_if(early, ssm_scan_kernel<T, ST, NPT, false>, grid, dim3(kPTile * kLanesN), 0, s, a);
}

template <typename T, typename ST>
int launch_state(const SsmArgs& a, int B, cudaStream_t s) {
    const int inner = a.nh * a.P;
    const bool aligned = (inner % 4 == 0) && (a.C % 4 == 0) && (a.conv_stride % 4 == 0) && (((uintptr_t)a.conv & 15) == 0) && (a.N % 4 == 0) &&
                         (sizeof(T) == 4 || (inner % 4 == 0));
    if (a.N <= 32) launch_npt<T, ST, 4>(a, B, aligned, s);
    else if (a.N <= 64) launch_npt<T, ST, 8>(a, B, aligned, s);
    else if (a.N <= 128) launch_npt<T, ST, 16>(a, B, aligned, s);
    else if (a.N <= 256) launch_npt<T, ST, 32>(a, B, aligned, s);
    else return kTooLarge;
    return launch_status();
}

template <typename T>
int launch(const SsmArgs& a, int B, cudaStream_t s) { return launch_state<T, float>(a, B, s); }
template <>
int launch<__nv_bfloat16>(const SsmArgs& a, int B, cudaStream_t s) {
    return a.state_bf16 ? launch_state<__nv_bfloat16, __nv_bfloat16>(a, B, s) : launch_state<__nv_bfloat16, float>(a, B, s);
}
}  // namespace

// `state_bf16`: the state tensor is bfloat16 (bfloat16 models only), else float32.  `longest`: no portion has more tokens
// (0: not known); it chooses the form that is fastest if that holds, and every form runs whatever the portions bring.
// `tokens`: the rows of the step.
extern "C" int lb_ssm_scan(const void* conv, int C, long conv_stride, const void* dt, long dt_stride, const float* A_log,
                           const float* dt_bias, const float* D, void* state, void* y, const int* cu_seqlens,
                           const int* start_pos, const int* slots, int B, int nh, int P, int N, int G,
                           float dt_scale, const void* gate, long gate_stride, float gate_scale,
                           const int* req_list, int beside, int state_bf16, int longest, long tokens, int dtype, void* stream) {
    if (B <= 0) return kOk;
    if (nh <= 0 || P <= 0 || N <= 0 || G <= 0 || nh % G || N % 4) return kBadSize;
    if (C != nh * P + 2 * G * N) return kBadSize;
    if (state_bf16 && dtype != kBF16) return kBadSize;
    SsmArgs a{conv, C, conv_stride, dt, dt_stride, A_log, dt_bias, D, state, y, cu_seqlens, start_pos, slots, nh, P, N, G, dt_scale,
              gate, gate_stride, gate_scale, req_list, beside, state_bf16, longest, tokens};
    LB_DISPATCH_DTYPE(dtype, return launch<T>(a, B, (cudaStream_t)stream));
    return kOk;
}
