// Router (f32 GEMV + softmax + stable top-k), dispatch (group pairs by expert) and the weighted
// combine of the quantized MoE block.  All three are small, latency- or HBM-bound kernels.
#include "common.cuh"

#include <atomic>
#include <climits>
#include <cstdlib>

namespace cmoe {

bool pdl_enabled() {
    static const bool on = [] {
        const char* v = std::getenv("CANDLE_MOE_PDL");
        return !(v && v[0] == '0');
    }();
    return on;
}

namespace {
struct TuningTable {
    std::atomic<int64_t> v[TUNE_N_KEYS];
    TuningTable() {
        const auto env = [](const char* name, int64_t dflt) {
            const char* s = std::getenv(name);
            return s && s[0] ? (int64_t)std::atoll(s) : dflt;
        };
        v[TUNE_GEMM_ENABLED] = env("CANDLE_MOE_GEMM", 1);
        v[TUNE_GEMM_MIN_ROWS] = env("CANDLE_MOE_GEMM_MIN_ROWS", CANDLE_MOE_GEMM_ROWS_AUTO);
        v[TUNE_STREAM_MAX_ROWS] = env("CANDLE_MOE_STREAM_MAX_ROWS", (int64_t)1 << 40);
        v[TUNE_FORCE_ROWS] = env("CANDLE_MOE_FORCE_ROWS", 0);
        v[TUNE_MID_ENABLED] = env("CANDLE_MOE_MID", 1);
    }
};
TuningTable& tuning_table() {
    static TuningTable t;
    return t;
}
}  // namespace
int64_t tuning_get(int key) { return key >= 0 && key < TUNE_N_KEYS ? tuning_table().v[key].load() : 0; }
bool tuning_set(int key, int64_t value) {
    if (key < 0 || key >= TUNE_N_KEYS) return false;
    tuning_table().v[key].store(value);
    return true;
}

// ------------------------------------------------------------------------------------------------
// Router (+ activation quantization).  One CTA per token; partial sums meet through warp shuffles and shared memory in a
// fixed order.  Warp 0 then does the softmax over all E experts and k rounds of arg-max
// with "lower expert id wins a tie", which is what a stable descending sort followed by take(k)
// yields (candle-transformers/src/models/quantized_llama.rs:162-179).  Meanwhile the other warps
// quantize the same row of x the Q8K way for the expert products (one pass over x instead of two
// kernels).  Arithmetic is plain f32 FMA (no TF32): the reference's router product is full f32.
// ------------------------------------------------------------------------------------------------
// Softmax over the E logits of one token and the top-k selection, by one warp (lane r ends up holding the r-th selected
// expert, from k on -1); writes the token's ids and weights.  A round is two warp-wide integer reductions and the loop is
// rolled: eight rounds of five exchanges of three values each, written out, were 16 KB of code at the end of every router kernel,
// fetched by every launch of it (Mixtral-shaped layer at one row: 10.0 -> 8.3 us, layer 75.3 -> 73.0; 60 experts, 16 rows: 12.7 -> 11.5,
// 4096 rows: layer 1364 -> 1326 in short runs).
__device__ __forceinline__ int softmax_topk_warp(const float* s_logits, int lane, int E, int k, int renorm,
                                                 uint32_t* __restrict__ ids_row, float* __restrict__ w_row) {
    // softmax over E (candle-nn/src/ops.rs:326-339): exp(v - max) / sum, true division
    constexpr int PER = CANDLE_MOE_MAX_EXPERTS / 32;
    float p[PER];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int e = lane + 32 * j;
        p[j] = e < E ? s_logits[e] : -INFINITY;
        mx = fmaxf(mx, p[j]);
    }
    mx = warp_max(mx);
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        if (32 * j >= E) break;  // (for the whole warp)
        const int e = lane + 32 * j;
        p[j] = e < E ? expf(p[j] - mx) : 0.f;
        s += p[j];
    }
    s = warp_sum(s);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        if (32 * j >= E) break;
        p[j] = (lane + 32 * j) < E ? p[j] / s : 0.f;
    }

    // Selection in the order of Rust's f32::total_cmp (the reference sorts with it, quantized_llama.rs:166), so
    // that it is total: a row holding a NaN or an infinity turns every probability into the same NaN, all keys
    // tie, and the lowest expert ids win -- the reference's stable sort gives exactly that.  Every selected id
    // is below E whatever the input holds.
    int key[PER];
    uint32_t open_mask = 0;  // bit j: expert lane + 32 j exists and has not been selected yet
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int b = (p[j] != p[j]) ? 0x7fffffff : __float_as_int(p[j]);  // all NaNs alike (they only occur together)
        key[j] = b ^ (int)(((uint32_t)(b >> 31)) >> 1);
        if (lane + 32 * j < E) open_mask |= 1u << j;
    }
    float sum = 0.f, mine_p = 0.f;
    int mine_e = -1;
#pragma unroll 1
    for (int r = 0; r < k; ++r) {
        // a key is never INT_MIN (that would be a NaN with its sign, and NaNs are made alike): it stands for "no candidate"
        int bk = INT_MIN, be = INT_MAX;
        float bv = 0.f;
#pragma unroll
        for (int j = 0; j < PER; ++j) {  // ascending expert id inside a lane: strict > keeps the lower id
            if (((open_mask >> j) & 1u) && key[j] > bk) {
                bk = key[j];
                bv = p[j];
                be = lane + 32 * j;
            }
        }
        const int top = __reduce_max_sync(0xffffffffu, bk);
        // k <= E, so a candidate always exists; the clamp only keeps a corrupted launch inside the tables
        const int sel = min(max(__reduce_min_sync(0xffffffffu, bk == top ? be : INT_MAX), 0), E - 1);
        bv = __shfl_sync(0xffffffffu, bv, sel & 31);
        sum += bv;  // rank order, like `sum_routing_weights += routing_weight`
        if (lane == r) {
            mine_e = sel;
            mine_p = bv;
        }
        if (lane == (sel & 31)) open_mask &= ~(1u << (sel >> 5));
    }
    if (lane < k) {
        ids_row[lane] = (uint32_t)mine_e;
        w_row[lane] = renorm ? mine_p / sum : mine_p;
    }
    return mine_e;
}

// Single token (the step of one-sequence decoding): its k experts are distinct, so the dispatch is their ascending order
// and needs no pass of its own.  Run by one warp whose lane r holds the r-th selected expert.
__device__ __forceinline__ void dispatch_one_token(int sel, int lane, int E, int k, uint32_t* __restrict__ counts,
                                                   uint32_t* __restrict__ offsets, uint32_t* __restrict__ perm_token,
                                                   uint32_t* __restrict__ pair_pos) {
    for (int e0 = 0; e0 < E; e0 += 32) {
        const int e = e0 + lane;
        uint32_t hit = 0, below = 0;
        for (int r = 0; r < k; ++r) {
            const int o = __shfl_sync(0xffffffffu, sel, r);
            hit += o == e;
            below += o < e;
        }
        if (e < E) {
            counts[e] = hit;
            offsets[e] = below;
        }
    }
    uint32_t pos = 0;
    for (int r = 0; r < k; ++r) pos += __shfl_sync(0xffffffffu, sel, r) < sel;
    if (lane == 0) offsets[E] = (uint32_t)k;
    if (lane < k) {
        perm_token[pos] = 0u;
        pair_pos[lane] = pos;
    }
}

__device__ __forceinline__ void add4(float4& a, const float4& b) {
    a.x += b.x;
    a.y += b.y;
    a.z += b.z;
    a.w += b.w;
}
__device__ __forceinline__ void fma4(float4& s, const float4& a, const float4& b) {
    s.x = fmaf(a.x, b.x, s.x);
    s.y = fmaf(a.y, b.y, s.y);
    s.z = fmaf(a.z, b.z, s.z);
    s.w = fmaf(a.w, b.w, s.w);
}

// Few tokens: 1024 threads per token, latency-bound.  The row passes through shared memory once, with the
// layer's RmsNorm applied on the way where the caller asks for it (norm_w; one launch fewer), and every warp owns whole
// dot products: expert e, or for few experts one of `parts` pieces of it, so that all loads of a round are in flight at
// once and one reduction per expert and warp is left.  (Eight experts at a time across all warps, eight reductions per
// warp and two barriers per round, was 7.9 us for 8 experts of 4096 and 29.2 us for 60 experts of 2048, 16
// rows; this form 8.9 us with the norm, which was another 4.5 us, and 11.5 us.)
// Before the wait for the previous kernel the first CTA asks for the router's rows in L2: a prefetch returns no data, so
// it does not matter what that kernel still writes.
template <bool NORM>
__global__ void __launch_bounds__(1024)
router_topk_small_kernel(const float* __restrict__ x, const float* __restrict__ norm_w, float eps, const float* __restrict__ wg,
                         const float* __restrict__ bias, int d, int E, int parts, int k, int renorm, uint32_t* __restrict__ ids,
                         float* __restrict__ wout, int8_t* __restrict__ qs, float* __restrict__ scales, int16_t* __restrict__ bsums,
                         uint32_t* __restrict__ counts, uint32_t* __restrict__ offsets, uint32_t* __restrict__ perm_token,
                         uint32_t* __restrict__ pair_pos) {
    extern __shared__ __align__(16) float s_x[];  // [d]
    __shared__ float s_part[8][CANDLE_MOE_MAX_EXPERTS];
    __shared__ float s_logits[CANDLE_MOE_MAX_EXPERTS];
    __shared__ float s_red[32];
    const int64_t t = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, d4 = d >> 2;
    pdl_trigger();
    if (t == 0)
        for (int64_t i = tid; i < (int64_t)E * d / 32; i += 1024) asm volatile("prefetch.global.L2 [%0];" ::"l"(wg + 32 * i));
    pdl_wait();
    const float4* xr = reinterpret_cast<const float4*>(x + t * (int64_t)d);
    float4* sx4 = reinterpret_cast<float4*>(s_x);
    if (NORM) {
        float ss = 0.f;
        for (int i = tid; i < d4; i += 1024) {
            const float4 v = xr[i];
            sx4[i] = v;
            ss = fmaf(v.x, v.x, ss);
            ss = fmaf(v.y, v.y, ss);
            ss = fmaf(v.z, v.z, ss);
            ss = fmaf(v.w, v.w, ss);
        }
        ss = warp_sum(ss);
        if (lane == 0) s_red[warp] = ss;
        __syncthreads();
        const float m = sqrtf(warp_sum(s_red[lane]) / (float)d + eps);  // every warp adds the 32 sums in the same order
        for (int i = tid; i < d4; i += 1024) {  // the elements this thread wrote
            const float4 v = sx4[i], a = reinterpret_cast<const float4*>(norm_w)[i];
            sx4[i] = make_float4(__fmul_rn(__fdiv_rn(v.x, m), a.x), __fmul_rn(__fdiv_rn(v.y, m), a.y),
                                 __fmul_rn(__fdiv_rn(v.z, m), a.z), __fmul_rn(__fdiv_rn(v.w, m), a.w));
        }
    } else {
        for (int i = tid; i < d4; i += 1024) sx4[i] = xr[i];
    }
    __syncthreads();
    // unit u = (expert, part); part p covers float4s [p d4 / parts, (p + 1) d4 / parts)
    for (int u = warp; u < E * parts; u += 32) {
        const int e = u / parts, p = u - e * parts;
        const int i1 = d4 * (p + 1) / parts;
        const float4* wr = reinterpret_cast<const float4*>(wg + (int64_t)e * d);
        // a lane's elements are added in runs of eight per component of the float4s, runs and components on their own: ten terms
        // in a row at most, where one sum over all of them had 256 for d = 8192 (root mean square error of a logit, 60 experts,
        // 64 rows of 8192: 5.4e-7 -> 2.3e-7, eight experts of 4096 1.8e-7 -> 1.5e-7; the time is the same)
        float4 tot = make_float4(0.f, 0.f, 0.f, 0.f);
        int i = d4 * p / parts + lane;
        for (; i + 7 * 32 < i1; i += 8 * 32) {
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 8; ++j) fma4(s, sx4[i + 32 * j], wr[i + 32 * j]);
            add4(tot, s);
        }
        float4 rest = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (; i < i1; i += 32) fma4(rest, sx4[i], wr[i]);
        add4(tot, rest);
        float acc = (tot.x + tot.y) + (tot.z + tot.w);
        acc = warp_sum(acc);
        if (lane == 0) s_part[p][e] = acc;
    }
    __syncthreads();
    if (warp != 0) {
        // warps 1.. quantize the row (each 256-element block by one warp)
        if (qs) {
            const int nb = d >> 8;
            for (int b = warp - 1; b < nb; b += 31)
                quantize_q8k_block(s_x + b * 256, lane, qs + t * (int64_t)d + b * 256, scales + t * nb + b, bsums + (t * nb + b) * 16);
        }
        return;
    }
    for (int e = lane; e < E; e += 32) {
        float v = 0.f;
        for (int p = 0; p < parts; ++p) v += s_part[p][e];
        if (bias) v += bias[e];
        s_logits[e] = v;
    }
    __syncwarp();
    const int sel = softmax_topk_warp(s_logits, lane, E, k, renorm, ids + t * k, wout + t * k);
    if (counts) dispatch_one_token(sel, lane, E, k, counts, offsets, perm_token, pair_pos);
}
constexpr int ROUTER_SMALL_MAX_D = 10240;  // the row in 40 KB of shared memory
// Up to 64 tokens; rows long enough to keep 1024 threads busy up to 256 (Mixtral-shaped layer, d = 4096: 100 rows 354.8 -> 345.5 us,
// 140 rows 389 -> 375, 290 rows equal; d = 1024, 257 rows 77 against 86 us the other way round).  That holds inside the block, where
// this form asks for the router's rows in L2 while the kernel before it still runs; a router called on its own keeps the other
// forms where they are faster: beyond one CTA per SM except with many experts (other form / this, 200 rows of 4096: 8 experts
// 6.8 / 10.5 us, 16 10.3 / 12.7, 32 16.7 / 16.6, 64 31.6 / 26.2; 100 rows: 8 experts 5.8 / 5.8, 16 8.4 / 6.9), and for the one round of five
// to eight experts that the other form makes of a few rows (16 rows, 8 experts: d = 4096 5.4 / 5.7, 8192 6.4 / 7.0, but the block
// of 4096 x 14336 at one row 76.2 / 75.3; two experts 5.0 / 4.8, 16 experts 7.6 / 6.9).
constexpr int ROUTER_SMALL_WAVE = 148, ROUTER_SMALL_MANY_EXPERTS = 32;
static bool router_small(int64_t T, int d, int E, bool in_block) {
    if (d > ROUTER_SMALL_MAX_D || T > (d >= 4096 ? 256 : 64)) return false;
    if (in_block) return true;
    return T <= 64 ? E <= 4 || E > 8 : T <= ROUTER_SMALL_WAVE || E >= ROUTER_SMALL_MANY_EXPERTS;
}

// Many tokens: 256 threads per token, so that eight CTAs share an SM and their load rounds overlap.  Few tokens that the form
// above does not take: 1024 threads (d = 16384, 60 experts, 16 rows 61 -> 44 us, two experts 10.0 -> 6.8).  The forms add
// the partial sums in different orders (last-bit differences of the logits, as between any two f32 dot-product orders).
template <int ROUTER_THREADS>
__global__ void __launch_bounds__(ROUTER_THREADS)
router_topk_kernel(const float* __restrict__ x, const float* __restrict__ wg, const float* __restrict__ bias,
                   int d, int E, int k, int renorm, uint32_t* __restrict__ ids, float* __restrict__ wout,
                   int8_t* __restrict__ qs, float* __restrict__ scales, int16_t* __restrict__ bsums,
                   uint32_t* __restrict__ counts, uint32_t* __restrict__ offsets, uint32_t* __restrict__ perm_token,
                   uint32_t* __restrict__ pair_pos) {
    pdl_trigger();
    pdl_wait();
    constexpr int ROUTER_WARPS = ROUTER_THREADS / 32;
    __shared__ float s_logits[CANDLE_MOE_MAX_EXPERTS];
    __shared__ float s_part[ROUTER_WARPS][8];
    const int64_t t = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float4* xr = reinterpret_cast<const float4*>(x + t * (int64_t)d);
    const int d4 = d >> 2;

    for (int e0 = 0; e0 < E; e0 += 8) {
        float acc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
        for (int i = tid; i < d4; i += ROUTER_THREADS) {
            const float4 xv = xr[i];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (e0 + j < E) {
                    const float4 wv = reinterpret_cast<const float4*>(wg + (int64_t)(e0 + j) * d)[i];
                    acc[j] = fmaf(xv.x, wv.x, acc[j]);
                    acc[j] = fmaf(xv.y, wv.y, acc[j]);
                    acc[j] = fmaf(xv.z, wv.z, acc[j]);
                    acc[j] = fmaf(xv.w, wv.w, acc[j]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float v = warp_sum(acc[j]);
            if (lane == 0) s_part[warp][j] = v;
        }
        __syncthreads();
        if (tid < 8 && e0 + tid < E) {
            float v = 0.f;
#pragma unroll
            for (int w8 = 0; w8 < ROUTER_WARPS; ++w8) v += s_part[w8][tid];
            if (bias) v += bias[e0 + tid];
            s_logits[e0 + tid] = v;
        }
        __syncthreads();
    }
    if (warp != 0) {
        // warps 1.. quantize the row (each 256-element block by one warp)
        if (qs) {
            const int nb = d >> 8;
            for (int b = warp - 1; b < nb; b += ROUTER_WARPS - 1)
                quantize_q8k_block(x + t * (int64_t)d + b * 256, lane, qs + t * (int64_t)d + b * 256, scales + t * nb + b,
                                   bsums + (t * nb + b) * 16);
        }
        return;
    }

    const int sel = softmax_topk_warp(s_logits, lane, E, k, renorm, ids + t * k, wout + t * k);
    if (counts) dispatch_one_token(sel, lane, E, k, counts, offsets, perm_token, pair_pos);
}

// Many tokens and many experts (prefill of a fine-grained layer): the router product as a tiled f32 GEMM.  The
// one-token kernels spend their time in warp reductions -- one per (token, expert) -- which for 60 experts and 4096
// tokens is most of 0.15 ms.  Here a CTA of 128 threads takes 16 tokens x all experts (64, 96 or 128): x and the router rows
// pass through shared memory in K chunks of 64 (the next chunk is fetched into registers while this one is multiplied), a
// thread accumulates 2 tokens x 4 (6, 8) experts in registers, six 128-bit shared loads per 32 multiply-adds, and the four warps
// then do the softmax and the selection of four tokens each.  Every logit is one sequential f32 sum over K (another order than
// the one-token kernels': last-bit differences, as between any two f32 dot products).  No fused quantization: used where the
// activations are quantized by a pass of their own (Q8_0 experts).  Bound by the multiply-adds (15 us for 60 experts,
// d = 2048, 4096 tokens), the shared loads and the latency of the chunks.  Measured there: one token x eight experts per
// thread, 32 tokens per CTA of 256 threads (nine shared loads, a CTA per SM) 93 us; this 70 us.  (Four K slices per CTA took
// 47 us, but add a logit in four parts: kept as one sum, so that the logits stay what they were bit for bit.)
// NJ experts per thread: 16 NJ experts, as few as hold them all (65 experts, 4096 tokens of 2048: two passes of 64 205 us, one
// of 96 140).  MIN_CTAS: four CTAs per SM where their registers allow it; with eight experts per thread three of them do more
// (128 experts, 4096 tokens 135 against 196 us), unless the CTAs then make a second wave (8192 tokens 231 against 198).
constexpr int RT_TOK = 16, RT_KC = 64, RT_PAD = RT_KC + 4, RT_THREADS = 128;
template <int NJ, int MIN_CTAS>
__global__ void __launch_bounds__(RT_THREADS, MIN_CTAS)
router_topk_tiled_kernel(const float* __restrict__ x, const float* __restrict__ wg, const float* __restrict__ bias,
                         int64_t T, int d, int E, int k, int renorm, uint32_t* __restrict__ ids, float* __restrict__ wout) {
    constexpr int RT_EXP = 16 * NJ;
    pdl_trigger();
    pdl_wait();
    __shared__ __align__(16) float s_x[RT_TOK][RT_PAD];
    __shared__ __align__(16) float s_w[RT_EXP][RT_PAD];
    __shared__ float s_logits[RT_TOK][CANDLE_MOE_MAX_EXPERTS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t t0 = (int64_t)blockIdx.x * RT_TOK;
    const int tg = lane & 7, eg = warp * 4 + (lane >> 3);  // tokens tg, tg + 8; experts eg + 16 j
    const int col = tid & 15, row = tid >> 4;              // loads: float4 column, row + 8 i
    float acc[2][NJ];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[i][j] = 0.f;
    // rows past the end repeat the last one (their results are not used); columns past d are not read
    const float4* px[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) px[i] = reinterpret_cast<const float4*>(x + min(t0 + row + 8 * i, T - 1) * (int64_t)d) + col;
    float4 vx[2], vw[2 * NJ];
    auto fetch = [&](int c) {
        if (c + 4 * col < d) {
#pragma unroll
            for (int i = 0; i < 2; ++i) vx[i] = px[i][c >> 2];
#pragma unroll
            for (int i = 0; i < 2 * NJ; ++i)
                vw[i] = reinterpret_cast<const float4*>(wg + (int64_t)min(row + 8 * i, E - 1) * d + c)[col];
        }
    };
    fetch(0);
    for (int c = 0; c < d; c += RT_KC) {
        __syncthreads();  // the previous chunk has been consumed
#pragma unroll
        for (int i = 0; i < 2; ++i) *reinterpret_cast<float4*>(&s_x[row + 8 * i][4 * col]) = vx[i];
#pragma unroll
        for (int i = 0; i < 2 * NJ; ++i) *reinterpret_cast<float4*>(&s_w[row + 8 * i][4 * col]) = vw[i];
        __syncthreads();
        if (c + RT_KC < d) fetch(c + RT_KC);  // the next chunk travels while this one is multiplied
        const int n4 = min(RT_KC, d - c) >> 2;
#pragma unroll 8
        for (int k4 = 0; k4 < n4; ++k4) {
            float4 xv[2], wv[NJ];
#pragma unroll
            for (int i = 0; i < 2; ++i) xv[i] = *reinterpret_cast<const float4*>(&s_x[tg + 8 * i][4 * k4]);
#pragma unroll
            for (int j = 0; j < NJ; ++j) wv[j] = *reinterpret_cast<const float4*>(&s_w[eg + 16 * j][4 * k4]);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    acc[i][j] = fmaf(xv[i].x, wv[j].x, acc[i][j]);
                    acc[i][j] = fmaf(xv[i].y, wv[j].y, acc[i][j]);
                    acc[i][j] = fmaf(xv[i].z, wv[j].z, acc[i][j]);
                    acc[i][j] = fmaf(xv[i].w, wv[j].w, acc[i][j]);
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int e = eg + 16 * j;
            if (e < E) s_logits[tg + 8 * i][e] = acc[i][j] + (bias ? bias[e] : 0.f);
        }
    __syncthreads();
    for (int i = warp; i < RT_TOK; i += RT_THREADS / 32) {
        const int64_t t = t0 + i;
        if (t < T) {
            softmax_topk_warp(s_logits[i], lane, E, k, renorm, ids + t * k, wout + t * k);
        }
    }
}

// the fused norm is there only where the small form runs
bool router_fuses_norm(int64_t T, int d) { return router_small(T, d, 1, true); }

cudaError_t launch_router_topk(cudaStream_t st, const float* x, const float* router, const float* bias, int64_t T,
                               int d, int E, int k, int renorm, uint32_t* ids, float* w, int8_t* qs, float* scales,
                               int16_t* bsums, uint32_t* counts, uint32_t* offsets, uint32_t* perm_token, uint32_t* pair_pos,
                               const float* norm_w, float eps) {
    if (T == 0) return cudaSuccess;
    if (counts && (T != 1 || !offsets || !perm_token || !pair_pos)) return cudaErrorInvalidValue;  // single-token dispatch only
    if (router_small(T, d, E, norm_w || offsets)) {  // (only the block hands over where the dispatch goes)
        const int parts = E <= 4 ? 8 : (E <= 8 ? 4 : (E <= 16 ? 2 : 1));
        auto kfn = norm_w ? router_topk_small_kernel<true> : router_topk_small_kernel<false>;
        return launch_k(kfn, dim3((unsigned)T), dim3(1024), (size_t)d * sizeof(float), st, x, norm_w, eps, router, bias, d, E, parts, k,
                        renorm, ids, w, qs, scales, bsums, counts, offsets, perm_token, pair_pos);
    }
    if (norm_w) return cudaErrorInvalidValue;
    if (T >= 512 && E >= 16 && !qs && !counts && d % 32 == 0) {
        const int64_t ctas = (T + RT_TOK - 1) / RT_TOK;
        auto kfn = E <= 64                           ? router_topk_tiled_kernel<4, 4>
                   : E <= 96                         ? router_topk_tiled_kernel<6, 4>
                   : ctas > 3 * 148 && ctas <= 4 * 148 ? router_topk_tiled_kernel<8, 4>
                                                     : router_topk_tiled_kernel<8, 3>;
        return launch_k(kfn, dim3((unsigned)ctas), dim3(RT_THREADS), 0, st, x, router, bias, T, d, E, k, renorm, ids, w);
    }
    return launch_k(T > 64 ? router_topk_kernel<256> : router_topk_kernel<1024>, dim3((unsigned)T), dim3(T > 64 ? 256 : 1024), 0, st, x, router,
                    bias, d, E, k, renorm, ids, w, qs, scales, bsums, counts, offsets, perm_token, pair_pos);
}

// ------------------------------------------------------------------------------------------------
// Dispatch.  A counting sort of the T*k (token, rank) pairs by expert that keeps pair order inside
// an expert, so every expert's token list is ascending like the reference's `top_x[e]`.  One CTA:
// each warp owns experts warp, warp+32, ... and walks the pair list 32 at a time with a ballot, first
// to count, then (after an exclusive scan over experts) to place.
// ------------------------------------------------------------------------------------------------
constexpr int PERMUTE_THREADS = 1024;

// s_off[e]: counts -> exclusive prefix sums, and both to memory (offsets[E] = the total); by one warp
__device__ __forceinline__ void scan_counts(uint32_t* s_off, int lane, int E, uint32_t* __restrict__ counts, uint32_t* __restrict__ offsets) {
    constexpr int PER = CANDLE_MOE_MAX_EXPERTS / 32;
    uint32_t v[PER], sum = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int e = lane * PER + j;
        v[j] = e < E ? s_off[e] : 0u;
        sum += v[j];
    }
    uint32_t run = sum;  // inclusive over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
    }
    run -= sum;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int e = lane * PER + j;
        if (e < E) {
            counts[e] = v[j];
            offsets[e] = run;
            s_off[e] = run;
            run += v[j];
            if (e == E - 1) offsets[E] = run;
        }
    }
}

__global__ void __launch_bounds__(PERMUTE_THREADS)
permute_kernel(const uint32_t* __restrict__ ids, int64_t n_pairs, int k, int E, uint32_t* __restrict__ counts,
               uint32_t* __restrict__ offsets, uint32_t* __restrict__ perm_token, uint32_t* __restrict__ pair_pos) {
    pdl_trigger();
    pdl_wait();
    // 32-bit indices, four loads in flight, a scan by one warp: with 64-bit divisions and a serial sum over the experts 64 pairs of 60
    // experts took 6.5 us, 4.2 this way, 200 pairs of eight 7.0 and 4.5
    __shared__ uint32_t s_off[CANDLE_MOE_MAX_EXPERTS + 1];  // counts, then offsets
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = PERMUTE_THREADS / 32;
    const uint32_t n = (uint32_t)n_pairs, none = 0xffffffffu;  // (no expert has that id)
    // rounds are counted: an index that ran to n would wrap behind the last round of nearly 2^32 pairs and never end (within that round
    // the largest index is a multiple of 128 less one, 2^32 - 1 at most)
    const uint32_t rounds = (uint32_t)((n_pairs + 127) / 128);
    for (int e = warp; e < E; e += n_warps) {
        uint32_t c = 0, i0 = lane;
#pragma unroll 1
        for (uint32_t round = 0; round < rounds; ++round, i0 += 128) {
            uint32_t id[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) id[j] = i0 + 32 * j < n ? ids[i0 + 32 * j] : none;
#pragma unroll
            for (int j = 0; j < 4; ++j) c += __popc(__ballot_sync(0xffffffffu, id[j] == (uint32_t)e));
        }
        if (lane == 0) s_off[e] = c;
    }
    __syncthreads();
    if (warp == 0) scan_counts(s_off, lane, E, counts, offsets);
    __syncthreads();
    for (int e = warp; e < E; e += n_warps) {
        uint32_t base = s_off[e], i0 = lane;
#pragma unroll 1
        for (uint32_t round = 0; round < rounds; ++round, i0 += 128) {
            uint32_t id[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) id[j] = i0 + 32 * j < n ? ids[i0 + 32 * j] : none;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool hit = id[j] == (uint32_t)e;
                const uint32_t m = __ballot_sync(0xffffffffu, hit);
                if (hit) {
                    const uint32_t i = i0 + 32 * j, pos = base + __popc(m & ((1u << lane) - 1u));
                    perm_token[pos] = i / (uint32_t)k;
                    pair_pos[i] = pos;
                }
                base += __popc(m);
            }
        }
    }
}

// The same counting sort over many CTAs, for large batches: the pair list is cut into chunks of PERMUTE_CHUNK pairs.
//   count  every CTA counts its chunk's pairs per expert                       -> table[chunk][expert]
//   scan   one CTA: expert offsets, and table[chunk][expert] becomes the first position of that chunk's pairs of
//          that expert (earlier chunks first: the order inside an expert stays the pair order)
//   place  every CTA walks its chunk again, 32 pairs at a time per expert with a ballot, as the one-CTA kernel does
constexpr int PERMUTE_CHUNK = 512;

__global__ void __launch_bounds__(256)
permute_count_kernel(const uint32_t* __restrict__ ids, int64_t n_pairs, int E, uint32_t* __restrict__ table) {
    pdl_trigger();
    pdl_wait();
    __shared__ uint32_t s_hist[CANDLE_MOE_MAX_EXPERTS];
    for (int e = threadIdx.x; e < E; e += blockDim.x) s_hist[e] = 0;
    __syncthreads();
    const int64_t i0 = (int64_t)blockIdx.x * PERMUTE_CHUNK;
    for (int j = threadIdx.x; j < PERMUTE_CHUNK; j += blockDim.x) {
        const int64_t i = i0 + j;
        if (i < n_pairs) {
            const uint32_t e = ids[i];
            if (e < (uint32_t)E) atomicAdd(&s_hist[e], 1u);  // a count: the order of the additions does not matter
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) table[(size_t)blockIdx.x * E + e] = s_hist[e];
}

__global__ void __launch_bounds__(128)
permute_scan_kernel(uint32_t* __restrict__ table, int n_chunks, int E, uint32_t* __restrict__ counts,
                    uint32_t* __restrict__ offsets) {
    pdl_trigger();
    pdl_wait();
    __shared__ uint32_t s_off[CANDLE_MOE_MAX_EXPERTS + 1];
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        uint32_t c = 0;
#pragma unroll 8
        for (int b = 0; b < n_chunks; ++b) c += table[(size_t)b * E + e];
        s_off[e] = c;
    }
    __syncthreads();
    if (threadIdx.x < 32) scan_counts(s_off, threadIdx.x, E, counts, offsets);
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        uint32_t run = s_off[e];
        int b = 0;
        for (; b + 8 <= n_chunks; b += 8) {  // eight loads in flight
            uint32_t c[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) c[j] = table[(size_t)(b + j) * E + e];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                table[(size_t)(b + j) * E + e] = run;
                run += c[j];
            }
        }
        for (; b < n_chunks; ++b) {
            const uint32_t c = table[(size_t)b * E + e];
            table[(size_t)b * E + e] = run;
            run += c;
        }
    }
}

__global__ void __launch_bounds__(PERMUTE_THREADS)
permute_place_kernel(const uint32_t* __restrict__ ids, int64_t n_pairs, int k, int E, const uint32_t* __restrict__ table,
                     uint32_t* __restrict__ perm_token, uint32_t* __restrict__ pair_pos) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = PERMUTE_THREADS / 32;
    // every warp holds the chunk's ids, sixteen to a lane, and goes through its experts without another load: 16384
    // selections of 60 experts 15.8 -> 8.5 us, 4096 of eight 13.8 -> 5.3
    constexpr int PER = PERMUTE_CHUNK / 32;
    const int64_t c0 = (int64_t)blockIdx.x * PERMUTE_CHUNK;
    const uint32_t n = (uint32_t)(n_pairs - c0 < PERMUTE_CHUNK ? n_pairs - c0 : PERMUTE_CHUNK);
    uint32_t id[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) id[j] = (uint32_t)(32 * j + lane) < n ? ids[c0 + 32 * j + lane] : 0xffffffffu;  // (no expert's)
#pragma unroll 1
    for (int e = warp; e < E; e += n_warps) {
        uint32_t base = table[(size_t)blockIdx.x * E + e];
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const bool hit = id[j] == (uint32_t)e;
            const uint32_t m = __ballot_sync(0xffffffffu, hit);
            if (hit) {
                const uint32_t i = (uint32_t)c0 + 32 * j + lane, pos = base + __popc(m & ((1u << lane) - 1u));
                perm_token[pos] = i / (uint32_t)k;
                pair_pos[i] = pos;
            }
            base += __popc(m);
        }
    }
}

size_t permute_scratch_words(int64_t n_pairs, int E) {
    return (size_t)((n_pairs + PERMUTE_CHUNK - 1) / PERMUTE_CHUNK) * (size_t)E;
}

cudaError_t launch_permute(cudaStream_t st, const uint32_t* ids, int64_t T, int k, int E, uint32_t* counts,
                           uint32_t* offsets, uint32_t* perm_token, uint32_t* pair_pos, uint32_t* scratch) {
    const int64_t n_pairs = T * k;
    if (!scratch || n_pairs <= 4 * PERMUTE_CHUNK)
        return launch_k(permute_kernel, dim3(1), dim3(PERMUTE_THREADS), 0, st, ids, n_pairs, k, E, counts, offsets, perm_token,
                        pair_pos);
    const int n_chunks = (int)((n_pairs + PERMUTE_CHUNK - 1) / PERMUTE_CHUNK);
    cudaError_t e = launch_k(permute_count_kernel, dim3(n_chunks), dim3(256), 0, st, ids, n_pairs, E, scratch);
    if (e != cudaSuccess) return e;
    e = launch_k(permute_scan_kernel, dim3(1), dim3(128), 0, st, scratch, n_chunks, E, counts, offsets);
    if (e != cudaSuccess) return e;
    return launch_k(permute_place_kernel, dim3(n_chunks), dim3(PERMUTE_THREADS), 0, st, ids, n_pairs, k, E,
                    (const uint32_t*)scratch, perm_token, pair_pos);
}

__global__ void single_group_kernel(uint32_t* offsets, uint32_t rows) {
    pdl_trigger();
    pdl_wait();
    offsets[0] = 0u;
    offsets[1] = rows;
}
cudaError_t launch_single_group(cudaStream_t st, uint32_t* offsets, uint32_t rows) {
    return launch_k(single_group_kernel, dim3(1), dim3(1), 0, st, offsets, rows);
}

// ------------------------------------------------------------------------------------------------
// Combine.  CTAs of 256 threads over (token, 1024-column slab) with 128-bit accesses.  The k contributions are added
// in ascending expert id, each product rounded first (no FMA), starting from +0.0: the order of the
// reference's expert loop with broadcast_mul followed by index_add (quantized_llama.rs:185-203).
// Optional shared expert: y += shared_out * sigmoid(x . g) (qwen2_moe.rs:315-319).
// KM bounds the selections per token (2, 4 or 8): the sort by expert id and the loads are unrolled for it.  (With one form
// for eight, a token's two selections cost the sorting network of eight in every thread: Mixtral-shaped layer, 2048 rows,
// 44.8 us against 27.1; 4096 rows of four and a shared expert 78 against 57.)  The loads of up to eight K-split partials of a selection are issued before the first
// is added: one row with eight partials of two selections is a chain of two memory latencies instead of sixteen
// (5.2 -> 3.3 us).
// ------------------------------------------------------------------------------------------------
constexpr int COMBINE_THREADS = 256;

// sum of the partials p, p + stride, ... (n of them) of one float4, in split order, BATCH loads in flight
template <int BATCH>
__device__ __forceinline__ float4 sum_partials(const float4* __restrict__ p, int64_t stride4, int n) {
    float4 v = p[0];
    for (int s0 = 1; s0 < n; s0 += BATCH) {
        float4 u[BATCH];
#pragma unroll
        for (int s = 0; s < BATCH; ++s)
            if (s0 + s < n) u[s] = p[(s0 + s) * stride4];
#pragma unroll
        for (int s = 0; s < BATCH; ++s)
            if (s0 + s < n) add4(v, u[s]);
    }
    return v;
}

template <int KM, bool SPLIT>
__global__ void __launch_bounds__(COMBINE_THREADS, SPLIT || KM > 4 ? 2 : 4)
combine_kernel(const float* __restrict__ eo, int n_splits, int64_t split_stride, const uint32_t* __restrict__ ids,
               const float* __restrict__ w, const uint32_t* __restrict__ pair_pos, int k, int d,
               const float* __restrict__ shared_out, int shared_splits, int64_t shared_split_stride,
               const float* __restrict__ x, const float* __restrict__ gate, const float* __restrict__ residual,
               float* __restrict__ y) {
    pdl_trigger();
    pdl_wait();
    __shared__ float s_red[COMBINE_THREADS / 32];
    __shared__ float s_gate;
    const int64_t t = blockIdx.x;
    // every thread sorts the token's k selections by expert id (k <= KM)
    uint32_t se[KM], sp[KM];
    float sw[KM];
#pragma unroll
    for (int r = 0; r < KM; ++r) {
        if (r < k) {
            se[r] = ids[t * k + r];
            sp[r] = pair_pos[t * k + r];
            sw[r] = w[t * k + r];
        } else {
            se[r] = 0xffffffffu;
            sp[r] = 0;
            sw[r] = 0.f;
        }
    }
#pragma unroll
    for (int a = 0; a < KM - 1; ++a)
#pragma unroll
        for (int b = 0; b < KM - 1 - a; ++b)
            if (se[b] > se[b + 1]) {
                uint32_t te = se[b]; se[b] = se[b + 1]; se[b + 1] = te;
                uint32_t tp = sp[b]; sp[b] = sp[b + 1]; sp[b + 1] = tp;
                float tw = sw[b]; sw[b] = sw[b + 1]; sw[b + 1] = tw;
            }

    float g = 0.f;
    if (shared_out) {
        float part = 0.f;
        const float4* xr = reinterpret_cast<const float4*>(x + t * (int64_t)d);
        const float4* gr = reinterpret_cast<const float4*>(gate);
        for (int i = threadIdx.x; i < (d >> 2); i += COMBINE_THREADS) {
            const float4 a = xr[i], b = gr[i];
            part = fmaf(a.x, b.x, part);
            part = fmaf(a.y, b.y, part);
            part = fmaf(a.z, b.z, part);
            part = fmaf(a.w, b.w, part);
        }
        part = warp_sum(part);
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = part;
        __syncthreads();
        if (threadIdx.x == 0) {
            float v = 0.f;
            for (int i = 0; i < COMBINE_THREADS / 32; ++i) v += s_red[i];
            s_gate = sigmoid_f(v);
        }
        __syncthreads();
        g = s_gate;
    }

    float4* yr = reinterpret_cast<float4*>(y + t * (int64_t)d);
    for (int i = blockIdx.y * COMBINE_THREADS + threadIdx.x; i < (d >> 2); i += COMBINE_THREADS * gridDim.y) {
        // an expert output may arrive as K-split partials: add them in split order first
        float4 v[KM];
#pragma unroll
        for (int r = 0; r < KM; ++r)
            if (r < k) {
                const float4* p = reinterpret_cast<const float4*>(eo + (int64_t)sp[r] * d) + i;
                v[r] = SPLIT ? sum_partials<7>(p, split_stride >> 2, n_splits) : p[0];
            }
        float4 sh = make_float4(0.f, 0.f, 0.f, 0.f), rr = sh;
        if (shared_out)
            sh = sum_partials<SPLIT ? 7 : 1>(reinterpret_cast<const float4*>(shared_out + t * (int64_t)d) + i, shared_split_stride >> 2, shared_splits);
        if (residual) rr = reinterpret_cast<const float4*>(residual + t * (int64_t)d)[i];
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < KM; ++r) {
            if (r < k) {
                acc.x = __fadd_rn(acc.x, __fmul_rn(v[r].x, sw[r]));
                acc.y = __fadd_rn(acc.y, __fmul_rn(v[r].y, sw[r]));
                acc.z = __fadd_rn(acc.z, __fmul_rn(v[r].z, sw[r]));
                acc.w = __fadd_rn(acc.w, __fmul_rn(v[r].w, sw[r]));
            }
        }
        if (shared_out) {
            acc.x = __fadd_rn(acc.x, __fmul_rn(sh.x, g));
            acc.y = __fadd_rn(acc.y, __fmul_rn(sh.y, g));
            acc.z = __fadd_rn(acc.z, __fmul_rn(sh.z, g));
            acc.w = __fadd_rn(acc.w, __fmul_rn(sh.w, g));
        }
        if (residual) {  // the layer's `x + residual` after the block (quantized_llama.rs:889-891)
            acc.x = __fadd_rn(acc.x, rr.x);
            acc.y = __fadd_rn(acc.y, rr.y);
            acc.z = __fadd_rn(acc.z, rr.z);
            acc.w = __fadd_rn(acc.w, rr.w);
        }
        yr[i] = acc;
    }
}

cudaError_t launch_combine(cudaStream_t st, const float* expert_out, int n_splits, int64_t split_stride,
                           const uint32_t* ids, const float* w, const uint32_t* pair_pos, int64_t T, int k, int d,
                           const float* shared_out, int shared_splits, int64_t shared_split_stride, const float* x,
                           const float* shared_gate, float* y, const float* residual) {
    if (T == 0) return cudaSuccess;
    const unsigned slabs = (unsigned)((d / 4 + COMBINE_THREADS - 1) / COMBINE_THREADS);
    auto kfn = k <= 2   ? (n_splits > 1 ? combine_kernel<2, true> : combine_kernel<2, false>)
               : k <= 4 ? (n_splits > 1 ? combine_kernel<4, true> : combine_kernel<4, false>)
                        : (n_splits > 1 ? combine_kernel<8, true> : combine_kernel<8, false>);
    return launch_k(kfn, dim3((unsigned)T, slabs), dim3(COMBINE_THREADS), 0, st, expert_out, n_splits, split_stride, ids, w, pair_pos, k, d,
                    shared_out, shared_splits, shared_split_stride, x, shared_gate, residual, y);
}

// RmsNorm of the rows feeding the block (candle-nn/src/ops.rs:504-514): y = x / sqrt(mean(x^2) + eps) * alpha, f32.
// One CTA per row; the sum of squares is a fixed-order tree (the reference adds sequentially: last-bit
// differences only).
__global__ void __launch_bounds__(256)
rmsnorm_kernel(const float* __restrict__ x, const float* __restrict__ alpha, float eps, int d, float* __restrict__ y) {
    pdl_trigger();
    pdl_wait();
    __shared__ float s_part[8];
    __shared__ float s_m;
    const float4* xr = reinterpret_cast<const float4*>(x + (int64_t)blockIdx.x * d);
    float part = 0.f;
    for (int i = threadIdx.x; i < (d >> 2); i += 256) {
        const float4 v = xr[i];
        part = fmaf(v.x, v.x, part);
        part = fmaf(v.y, v.y, part);
        part = fmaf(v.z, v.z, part);
        part = fmaf(v.w, v.w, part);
    }
    part = warp_sum(part);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int i = 0; i < 8; ++i) t += s_part[i];
        s_m = sqrtf(t / (float)d + eps);
    }
    __syncthreads();
    const float m = s_m;
    const float4* ar = reinterpret_cast<const float4*>(alpha);
    float4* yr = reinterpret_cast<float4*>(y + (int64_t)blockIdx.x * d);
    for (int i = threadIdx.x; i < (d >> 2); i += 256) {
        const float4 v = xr[i], a = ar[i];
        yr[i] = make_float4(__fmul_rn(__fdiv_rn(v.x, m), a.x), __fmul_rn(__fdiv_rn(v.y, m), a.y),
                            __fmul_rn(__fdiv_rn(v.z, m), a.z), __fmul_rn(__fdiv_rn(v.w, m), a.w));
    }
}

cudaError_t launch_rmsnorm(cudaStream_t st, const float* x, const float* alpha, float eps, int64_t T, int d, float* y) {
    if (T == 0) return cudaSuccess;
    return launch_k(rmsnorm_kernel, dim3((unsigned)T), dim3(256), 0, st, x, alpha, eps, d, y);
}

}  // namespace cmoe
