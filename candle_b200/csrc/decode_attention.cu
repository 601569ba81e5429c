// Attention for one new token per sequence over an f32 KV cache: the `standard_attention` of
// candle-transformers' quantized_llama (quantized_llama.rs:303-317) at seq_len = 1 --
//     att = softmax(q . K^T / sqrt(head_dim)),  y = att . V
// with `repeat_kv` (utils.rs repeat_kv: query head h reads kv head h / (n_head / n_kv_head)) folded into the
// indexing instead of materialised.  A decode step at batch 32 and a 4096-token context reads 1 GB of cache per
// layer, so the kernel is a streaming one: every (sequence, kv head) pair is cut into chunks of the context, a CTA
// reads its chunk of K once for all the query heads of the group, keeps the scores in shared memory, then reads its
// chunk of V once; a second small kernel merges the chunks' partial softmax sums (the usual split-softmax algebra:
// only the order of f32 additions differs from a one-pass softmax).  f32 throughout, like the reference.
#include <algorithm>

#include "common.cuh"
#include "stream_common.cuh"
#include "tc5_common.cuh"

namespace cmoe {

namespace {

constexpr int ATT_THREADS = 256;
constexpr int ATT_MAX_GROUP = 8;    // query heads per kv head
constexpr int ATT_CHUNK = 512;      // context positions per CTA

// Sum of G per-lane values over the 32 lanes of a warp.  For G = 4 the four sums are folded as they travel (two
// exchange steps halve the values a lane carries, then three ordinary steps): 6 shuffles instead of 20; lane 8 h
// ends up with the sum of head h.  Other group sizes use the plain butterfly (every lane gets every sum).
template <int G>
__device__ __forceinline__ void warp_sum_heads(float (&acc)[G], int lane, float (&out)[G], bool& owner, int& head) {
    if constexpr (G == 4) {
        const bool hi16 = lane & 16, hi8 = lane & 8;
        const float r0 = __shfl_xor_sync(0xffffffffu, hi16 ? acc[0] : acc[2], 16);
        const float r1 = __shfl_xor_sync(0xffffffffu, hi16 ? acc[1] : acc[3], 16);
        const float k0 = (hi16 ? acc[2] : acc[0]) + r0, k1 = (hi16 ? acc[3] : acc[1]) + r1;
        const float r = __shfl_xor_sync(0xffffffffu, hi8 ? k0 : k1, 8);
        float v = (hi8 ? k1 : k0) + r;
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        out[0] = v;
        owner = (lane & 7) == 0;
        head = (hi16 ? 2 : 0) + (hi8 ? 1 : 0);
    } else {
#pragma unroll
        for (int g = 0; g < G; ++g) out[g] = warp_sum(acc[g]);
        owner = lane == 0;
        head = -1;  // lane 0 holds all of them
    }
}

// partial[(((b * n_kv + kv) * n_chunks + c) * G + g) * (D + 2)]: chunk maximum, sum of exponentials, D weighted sums
template <int D, int G>
__global__ void __launch_bounds__(ATT_THREADS)
decode_attention_chunk_kernel(const float* __restrict__ q, const float* __restrict__ kc, const float* __restrict__ vc, int n_kv,
                              int64_t max_seq, int n_ctx, float scale, int n_chunks, float* __restrict__ partial) {
    pdl_trigger();
    pdl_wait();
    constexpr int WARPS = ATT_THREADS / 32;
    __shared__ float s_q[G][D];
    __shared__ __align__(16) float s_score[ATT_CHUNK][G];  // a position's G scores side by side: one vector load in the V pass
    __shared__ __align__(16) float s_o[WARPS / 2][G][D];
    __shared__ float s_red[G][WARPS];
    __shared__ float s_max[G], s_sum[G];
    const int c = blockIdx.x, kv = blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int p0 = c * ATT_CHUNK, p1 = min(n_ctx, p0 + ATT_CHUNK), np = p1 - p0;
    const int n_head = n_kv * G;
    for (int i = tid; i < G * D; i += ATT_THREADS) s_q[i / D][i % D] = q[((int64_t)b * n_head + kv * G + i / D) * D + i % D];
    __syncthreads();
    const float* kbase = kc + (((int64_t)b * n_kv + kv) * max_seq + p0) * D;
    const float* vbase = vc + (((int64_t)b * n_kv + kv) * max_seq + p0) * D;

    // ---- scores: one warp per position, a lane holds D / 32 consecutive elements of the row ----
    constexpr int PER = D / 32;
    float qr[G][PER];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
        for (int i = 0; i < PER; ++i) qr[g][i] = s_q[g][lane * PER + i];
#pragma unroll 4
    for (int p = warp; p < np; p += WARPS) {
        float kr[PER];
        if (PER == 4) {
            const float4 v4 = reinterpret_cast<const float4*>(kbase + (int64_t)p * D)[lane];
            kr[0] = v4.x; kr[1] = v4.y; kr[2] = v4.z; kr[3] = v4.w;
        } else {
            const float2 v2 = reinterpret_cast<const float2*>(kbase + (int64_t)p * D)[lane];
            kr[0] = v2.x; kr[PER - 1] = v2.y;
        }
        float acc[G], sum[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            acc[g] = 0.f;
#pragma unroll
            for (int i = 0; i < PER; ++i) acc[g] = fmaf(qr[g][i], kr[i], acc[g]);
        }
        bool owner;
        int head;
        warp_sum_heads<G>(acc, lane, sum, owner, head);
        if (owner) {
            if (head >= 0) {
                s_score[p][head] = sum[0] * scale;
            } else {
#pragma unroll
                for (int g = 0; g < G; ++g) s_score[p][g] = sum[g] * scale;
            }
        }
    }
    __syncthreads();
    // ---- chunk maximum and sum of exponentials per query head ----
#pragma unroll
    for (int g = 0; g < G; ++g) {
        float m = -INFINITY;
        for (int p = tid; p < np; p += ATT_THREADS) m = fmaxf(m, s_score[p][g]);
        m = warp_max(m);
        if (lane == 0) s_red[g][warp] = m;
    }
    __syncthreads();
    if (tid < G) {
        float m = -INFINITY;
        for (int w = 0; w < WARPS; ++w) m = fmaxf(m, s_red[tid][w]);
        s_max[tid] = m;
    }
    __syncthreads();
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const float m = s_max[g];
        float s = 0.f;
        for (int p = tid; p < np; p += ATT_THREADS) {
            const float e = expf(s_score[p][g] - m);
            s_score[p][g] = e;
            s += e;
        }
        s = warp_sum(s);
        if (lane == 0) s_red[g][warp] = s;
    }
    __syncthreads();
    if (tid < G) {
        float s = 0.f;
        for (int w = 0; w < WARPS; ++w) s += s_red[tid][w];
        s_sum[tid] = s;
    }
    // ---- weighted sum of V: D / 4 lanes cover a row with 128-bit loads, a warp takes 32 / (D / 4) positions at a time ----
    constexpr int LPP = D / 4, PPW = 32 / LPP;  // lanes per position, positions per warp and step
    const int sub = lane / LPP, l4 = lane % LPP;
    float o[G][4];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[g][i] = 0.f;
#pragma unroll 4
    for (int p = warp * PPW + sub; p < np; p += WARPS * PPW) {
        const float4 v = reinterpret_cast<const float4*>(vbase + (int64_t)p * D)[l4];
        float w[G];
        if constexpr (G == 4) {
            const float4 w4 = *reinterpret_cast<const float4*>(&s_score[p][0]);
            w[0] = w4.x; w[1] = w4.y; w[2] = w4.z; w[3] = w4.w;
        } else {
#pragma unroll
            for (int g = 0; g < G; ++g) w[g] = s_score[p][g];
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            o[g][0] = fmaf(w[g], v.x, o[g][0]);
            o[g][1] = fmaf(w[g], v.y, o[g][1]);
            o[g][2] = fmaf(w[g], v.z, o[g][2]);
            o[g][3] = fmaf(w[g], v.w, o[g][3]);
        }
    }
    if (PPW == 2) {  // the two positions a warp handles at a time meet first
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int i = 0; i < 4; ++i) o[g][i] += __shfl_xor_sync(0xffffffffu, o[g][i], 16);
    }
    // the warps meet in shared memory, halving the number of partial sums per round (a fixed order)
    for (int half = WARPS / 2; half >= 1; half >>= 1) {
        if (warp >= half && warp < 2 * half && sub == 0) {
#pragma unroll
            for (int g = 0; g < G; ++g) *reinterpret_cast<float4*>(&s_o[warp - half][g][4 * l4]) = make_float4(o[g][0], o[g][1], o[g][2], o[g][3]);
        }
        __syncthreads();
        if (warp < half && sub == 0) {
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float4 t = *reinterpret_cast<const float4*>(&s_o[warp][g][4 * l4]);
                o[g][0] += t.x; o[g][1] += t.y; o[g][2] += t.z; o[g][3] += t.w;
            }
        }
        __syncthreads();
    }
    if (warp == 0 && sub == 0) {
        float* out = partial + ((((int64_t)b * n_kv + kv) * n_chunks + c) * G) * (D + 2);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            out[g * (D + 2) + 2 + 4 * l4 + 0] = o[g][0];
            out[g * (D + 2) + 2 + 4 * l4 + 1] = o[g][1];
            out[g * (D + 2) + 2 + 4 * l4 + 2] = o[g][2];
            out[g * (D + 2) + 2 + 4 * l4 + 3] = o[g][3];
            if (l4 == 0) {
                out[g * (D + 2)] = s_max[g];
                out[g * (D + 2) + 1] = s_sum[g];
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------
// The same chunk of work for rows of 128 floats and four query heads per kv head, as a pipeline.  HBM-bound: K and V are
// read once, and what the general kernel above loses is the time in which a CTA has no loads in flight (its barriers
// between the K pass, the softmax and the V pass).  Here every warp runs a ring of its own of bulk copies -- a tile is 8
// positions of K and the same 8 of V, 4 KB each, three tiles deep, which continues into the CTA's next chunk -- and an
// online softmax, so that a warp meets the others only once per chunk.
//   scores   a lane holds dims 4 l .. 4 l + 3 of the row and of the four queries: 32 partial dot products per tile, which
//            31 shuffles (halving the number of values a lane carries) turn into ONE score per lane, lane = 4 p + g
//   softmax  running maximum per head (3 shuffles), one exponential per lane; the weights go back to all lanes through
//            32 floats of shared memory
//   V        o[g][dims of the lane] += w[p][g] * v[p][dims], packed pairs
// Measured, 32 sequences, 8 kv heads, 4096 positions (1.07 GB of cache; 164 us at 6.5 TB/s), as part of a one-layer decode
// step: step 619 -> 566 us, of which 5 us belong to the projections.
// ------------------------------------------------------------------------------------------------
constexpr int RING_WARPS = 4, RING_THREADS = 32 * RING_WARPS, RING_TILE = 8, RING_DEPTH = 3, RING_D = 128, RING_G = 4;
constexpr int RING_HALF_BYTES = RING_TILE * RING_D * 4, RING_SMEM = RING_WARPS * RING_DEPTH * 2 * RING_HALF_BYTES;
static_assert(RING_TILE * RING_G == 32, "one score per lane");

__global__ void __launch_bounds__(RING_THREADS, 2)
decode_attention_ring_kernel(const float* __restrict__ q, const float* __restrict__ kc, const float* __restrict__ vc,
                             int64_t max_seq, int n_ctx, float scale, int chunk, int n_chunks, int n_units, float* __restrict__ partial,
                             int* status, uint32_t zero) {
    extern __shared__ __align__(128) uint8_t ring[];
    __shared__ uint64_t full[RING_WARPS][RING_DEPTH];
    __shared__ __align__(16) float s_w[RING_WARPS][32];
    __shared__ __align__(16) float s_alpha[RING_WARPS][RING_G];
    __shared__ float s_m[RING_WARPS][RING_G], s_l[RING_WARPS][RING_G];
    __shared__ __align__(16) float s_o[RING_WARPS][RING_G][RING_D];
    __shared__ int s_abort;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_trigger();
    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int w = 0; w < RING_WARPS; ++w)
            for (int i = 0; i < RING_DEPTH; ++i) mbar_init(&full[w][i], 1);
        fence_barrier_init();
    }
    __syncthreads();
    pdl_wait();
    volatile int* abort_flag = &s_abort;
    const uint32_t my_ring = smem_u32(ring) + (uint32_t)warp * (RING_DEPTH * 2 * RING_HALF_BYTES);
    uint8_t* my_ring_p = ring + warp * (RING_DEPTH * 2 * RING_HALF_BYTES);

    // a unit is one chunk of one (sequence, kv head); this warp takes its tiles warp, warp + RING_WARPS, ...
    struct Cursor {
        int unit, tile, n_tiles, np;
        int64_t row0;  // first cache row of the unit
    };
    auto open = [&](Cursor& c) {  // the warp's first tile of unit c.unit, or of a later one if it has none there
        while (c.unit < n_units) {
            const int ch = c.unit % n_chunks, bk = c.unit / n_chunks;
            c.np = min(chunk, n_ctx - ch * chunk);
            c.n_tiles = (c.np + RING_TILE - 1) / RING_TILE;
            c.row0 = (int64_t)bk * max_seq + (int64_t)ch * chunk;
            c.tile = warp;
            if (c.tile < c.n_tiles) return;
            c.unit += gridDim.x;
        }
    };
    Cursor pf;  // what to request next
    pf.unit = blockIdx.x;
    open(pf);
    uint32_t n_req = 0, n_use = 0, n_issued = 0;  // n_issued: lane 0's; equal to n_req until the abort flag is seen
    auto request = [&](uint32_t dep) {  // dep: 0, known only once the slot's old contents have arrived in registers
        if (pf.unit >= n_units) return;
        const uint32_t s = n_req % RING_DEPTH + dep;
        if (lane == 0 && !*abort_flag) {
            const uint32_t bytes = (uint32_t)min(RING_TILE, pf.np - pf.tile * RING_TILE) * (RING_D * 4);
            const int64_t row = pf.row0 + pf.tile * RING_TILE;
            mbar_expect_tx(&full[warp][s], 2 * bytes);
            bulk_g2s(my_ring_p + s * 2 * RING_HALF_BYTES, kc + row * RING_D, bytes, &full[warp][s]);
            bulk_g2s(my_ring_p + s * 2 * RING_HALF_BYTES + RING_HALF_BYTES, vc + row * RING_D, bytes, &full[warp][s]);
            n_issued = n_req + 1;
        }
        ++n_req;
        pf.tile += RING_WARPS;
        if (pf.tile >= pf.n_tiles) {
            pf.unit += gridDim.x;
            open(pf);
        }
    };
    for (int i = 0; i < RING_DEPTH; ++i) request(0);

    for (int unit = blockIdx.x; unit < n_units; unit += gridDim.x) {
        const int ch = unit % n_chunks, bk = unit / n_chunks, np = min(chunk, n_ctx - ch * chunk);
        const int n_tiles = (np + RING_TILE - 1) / RING_TILE;
        uint64_t q2[RING_G][2];  // the queries at this lane's dims, as pairs
#pragma unroll
        for (int g = 0; g < RING_G; ++g) {
            const float4 v = reinterpret_cast<const float4*>(q + ((int64_t)bk * RING_G + g) * RING_D)[lane];
            q2[g][0] = f32x2_pack(v.x, v.y);
            q2[g][1] = f32x2_pack(v.z, v.w);
        }
        uint64_t o2[RING_G][2];
#pragma unroll
        for (int g = 0; g < RING_G; ++g) o2[g][0] = o2[g][1] = 0ull;
        float m = -INFINITY, l = 0.f;  // of head lane & 3: the maximum (same in all its lanes), this lane's share of the sum
        for (int tile = warp; tile < n_tiles; tile += RING_WARPS, ++n_use) {
            const uint32_t s = n_use % RING_DEPTH;
            mbar_wait(&full[warp][s], (n_use / RING_DEPTH) & 1, abort_flag);
            const int n = min(RING_TILE, np - tile * RING_TILE);
            const uint32_t kaddr = my_ring + s * 2 * RING_HALF_BYTES + 16 * lane, vaddr = kaddr + RING_HALF_BYTES;
            float part[32];  // [4 p + g]
#pragma unroll
            for (int p = 0; p < RING_TILE; ++p) {
                const uint4 kv = lds128(kaddr + p * (RING_D * 4));
                const uint64_t k0 = f32x2_pack_bits(kv.x, kv.y), k1 = f32x2_pack_bits(kv.z, kv.w);
#pragma unroll
                for (int g = 0; g < RING_G; ++g) {
                    float a, b;
                    f32x2_unpack(f32x2_fma(q2[g][1], k1, f32x2_mul(q2[g][0], k0)), a, b);
                    part[4 * p + g] = a + b;
                }
            }
            // after step i a lane carries the values whose index agrees with its lane number in the bits done so far
            static_for<5>([&](auto Ic) {
                constexpr int half = 16 >> decltype(Ic)::value;
                const bool up = lane & half;
#pragma unroll
                for (int j = 0; j < half; ++j) {
                    const float give = up ? part[j] : part[j + half], keep = up ? part[j + half] : part[j];
                    part[j] = keep + __shfl_xor_sync(0xffffffffu, give, half);
                }
            });
            const float score = (lane >> 2) < n ? part[0] * scale : -INFINITY;
            float mt = score;
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, o));
            const float m_new = fmaxf(m, mt);
            // a maximum of -inf (every score so far is -inf) must not turn the weights into NaN: exp(-inf - 0) is 0
            const float m_ref = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = expf(m - m_ref), w = expf(score - m_ref);
            m = m_new;
            l = fmaf(l, alpha, w);
            s_w[warp][lane] = w;
            if (lane < RING_G) s_alpha[warp][lane] = alpha;
            __syncwarp();
            uint32_t arrived = 0;
            // The tile's eight positions are added on their own before they join the running sum: 8 and 16 terms in a row per
            // 512-position chunk instead of 128, for the same number of instructions (relative error against 64-bit arithmetic,
            // 32 sequences of 4096 positions: 2.4e-7 -> 1.5e-7; the general kernel, 64 terms in a row, 1.9e-7)
            uint64_t t2[RING_G][2];
#pragma unroll
            for (int p = 0; p < RING_TILE; ++p) {
                if (p < n) {  // rows past the end of the context were not copied; a tile has at least one
                    const uint4 vv = lds128(vaddr + p * (RING_D * 4));
                    arrived |= vv.x;
                    const uint64_t v0 = f32x2_pack_bits(vv.x, vv.y), v1 = f32x2_pack_bits(vv.z, vv.w);
                    const float4 wv = *reinterpret_cast<const float4*>(&s_w[warp][4 * p]);
                    const float w4[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
                    for (int g = 0; g < RING_G; ++g) {
                        const uint64_t w2 = f32x2_pack(w4[g], w4[g]);
                        t2[g][0] = p ? f32x2_fma(w2, v0, t2[g][0]) : f32x2_mul(w2, v0);
                        t2[g][1] = p ? f32x2_fma(w2, v1, t2[g][1]) : f32x2_mul(w2, v1);
                    }
                }
            }
            const float4 al = *reinterpret_cast<const float4*>(s_alpha[warp]);
            const float a4[4] = {al.x, al.y, al.z, al.w};
#pragma unroll
            for (int g = 0; g < RING_G; ++g) {
                const uint64_t a2 = f32x2_pack(a4[g], a4[g]);
                o2[g][0] = f32x2_fma(o2[g][0], a2, t2[g][0]);
                o2[g][1] = f32x2_fma(o2[g][1], a2, t2[g][1]);
            }
            // The slot may be refilled when every lane HAS its rows of V (K went into the scores): the address of the
            // refill depends on a word of each load (`zero` is 0 at run time), so it cannot be issued before.
            request(__reduce_or_sync(0xffffffffu, arrived) & zero);
        }
        // ---- the warps of the chunk meet ----
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (lane < RING_G) {
            s_m[warp][lane] = m;
            s_l[warp][lane] = l;
        }
#pragma unroll
        for (int g = 0; g < RING_G; ++g) {
            float4 v;
            f32x2_unpack(o2[g][0], v.x, v.y);
            f32x2_unpack(o2[g][1], v.z, v.w);
            *reinterpret_cast<float4*>(&s_o[warp][g][4 * lane]) = v;
        }
        __syncthreads();
        float* out = partial + (int64_t)unit * RING_G * (RING_D + 2);
        {
            const int g = warp;  // RING_WARPS == RING_G: a warp finishes one head
            float M = -INFINITY;
#pragma unroll
            for (int w = 0; w < RING_WARPS; ++w) M = fmaxf(M, s_m[w][g]);
            const float M_ref = M == -INFINITY ? 0.f : M;
            float L = 0.f, r[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int w = 0; w < RING_WARPS; ++w) {
                const float f = expf(s_m[w][g] - M_ref);
                const float4 v = *reinterpret_cast<const float4*>(&s_o[w][g][4 * lane]);
                L = fmaf(f, s_l[w][g], L);
                r[0] = fmaf(f, v.x, r[0]);
                r[1] = fmaf(f, v.y, r[1]);
                r[2] = fmaf(f, v.z, r[2]);
                r[3] = fmaf(f, v.w, r[3]);
            }
            float* og = out + g * (RING_D + 2);
            if (lane == 0) {
                og[0] = M;
                og[1] = L;
            }
            reinterpret_cast<float2*>(og + 2)[2 * lane] = make_float2(r[0], r[1]);
            reinterpret_cast<float2*>(og + 2)[2 * lane + 1] = make_float2(r[2], r[3]);
        }
        __syncthreads();
    }
    // Nothing of this CTA's copies may be in flight when it leaves.  Without the abort flag every one has been waited for; with it
    // the last ones issued (at most one per slot) may not have been.
    if (lane == 0 && *abort_flag)
        for (uint32_t i = n_issued > RING_DEPTH ? n_issued - RING_DEPTH : 0; i < n_issued; ++i)
            mbar_drain(&full[warp][i % RING_DEPTH], (i / RING_DEPTH) & 1);
    __syncthreads();
    if (threadIdx.x == 0 && s_abort) atomicOr(status, 1);
}

// y[b, head, :] = sum_c exp(m_c - M) o_c / sum_c exp(m_c - M) l_c, chunks in order, in runs of eight that are added up on their
// own first: short chunks of a long context are up to 64 and more terms, which in one row would cost accuracy (one sequence of
// 4096 positions, relative error against 64-bit arithmetic MERGE_ERR)
constexpr int MERGE_RUN = 8;
template <int D, int G>
__global__ void __launch_bounds__(D)
decode_attention_merge_kernel(const float* __restrict__ partial, int n_kv, int n_chunks, float* __restrict__ y) {
    pdl_trigger();
    pdl_wait();
    const int head = blockIdx.x, b = blockIdx.y, dim = threadIdx.x;
    const int kv = head / G, g = head % G;
    const float* base = partial + ((((int64_t)b * n_kv + kv) * n_chunks) * G + g) * (D + 2);
    const int64_t stride = (int64_t)G * (D + 2);
    float M = -INFINITY;
    for (int c = 0; c < n_chunks; ++c) M = fmaxf(M, base[c * stride]);
    float num = 0.f, den = 0.f;
    for (int c0 = 0; c0 < n_chunks; c0 += MERGE_RUN) {
        float m[MERGE_RUN], l[MERGE_RUN], o[MERGE_RUN];  // loads first: a run costs one latency, not eight
#pragma unroll
        for (int i = 0; i < MERGE_RUN; ++i) {
            if (c0 + i < n_chunks) {
                const float* p = base + (c0 + i) * stride;
                m[i] = p[0];
                l[i] = p[1];
                o[i] = p[2 + dim];
            }
        }
        float n = 0.f, d = 0.f;
#pragma unroll
        for (int i = 0; i < MERGE_RUN; ++i) {
            if (c0 + i < n_chunks) {
                const float w = expf(m[i] - M);
                d = fmaf(w, l[i], d);
                n = fmaf(w, o[i], n);
            }
        }
        den += d;
        num += n;
    }
    y[((int64_t)b * n_kv * G + head) * D + dim] = num / den;
}

// Positions per unit of the ring kernel: ATT_CHUNK, halved (down to 64, two tiles per warp) while the units do not give every
// CTA two: a single sequence of 4096 positions has 64 units of 512 for 296 CTAs, two per SM of a B200.  (The workspace bound
// rests on the constant; the device is not asked on the way: a step over a context of 16 is 6.5 us, all host time.)
constexpr int RING_MIN_CHUNK = 64, RING_CTAS = 2 * 148, RING_MIN_UNITS = 2 * RING_CTAS;
int ring_chunk(int64_t pairs, int n_ctx) {
    int chunk = ATT_CHUNK;
    while (chunk > RING_MIN_CHUNK && pairs * ((n_ctx + chunk - 1) / chunk) < RING_MIN_UNITS) chunk /= 2;
    return chunk;
}

cudaError_t launch_ring(cudaStream_t st, const float* q, const float* kc, const float* vc, int B, int n_kv, int64_t max_seq, int n_ctx,
                        float scale, float* y, float* partial) {
    int* status = nullptr;
    cudaError_t e = stream_status_ptr(&status);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(decode_attention_ring_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_SMEM);
    if (e != cudaSuccess) return e;
    const int chunk = ring_chunk((int64_t)B * n_kv, n_ctx), n_chunks = (n_ctx + chunk - 1) / chunk, n_units = B * n_kv * n_chunks;
    e = launch_k(decode_attention_ring_kernel, dim3(std::min(n_units, RING_CTAS)), dim3(RING_THREADS), (size_t)RING_SMEM, st, q, kc, vc,
                 max_seq, n_ctx, scale, chunk, n_chunks, n_units, partial, status, 0u);
    if (e != cudaSuccess) return e;
    return launch_k(decode_attention_merge_kernel<RING_D, RING_G>, dim3(n_kv * RING_G, B), dim3(RING_D), 0, st, (const float*)partial, n_kv,
                    n_chunks, y);
}

template <int D, int G>
cudaError_t launch_att(cudaStream_t st, const float* q, const float* kc, const float* vc, int B, int n_kv, int64_t max_seq, int n_ctx,
                       float scale, float* y, float* partial) {
    if constexpr (D == RING_D && G == RING_G) {
        return launch_ring(st, q, kc, vc, B, n_kv, max_seq, n_ctx, scale, y, partial);
    } else {
        const int n_chunks = (n_ctx + ATT_CHUNK - 1) / ATT_CHUNK;
        cudaError_t e = launch_k(decode_attention_chunk_kernel<D, G>, dim3(n_chunks, n_kv, B), dim3(ATT_THREADS), 0, st, q, kc, vc, n_kv,
                                 max_seq, n_ctx, scale, n_chunks, partial);
        if (e != cudaSuccess) return e;
        return launch_k(decode_attention_merge_kernel<D, G>, dim3(n_kv * G, B), dim3(D), 0, st, (const float*)partial, n_kv, n_chunks, y);
    }
}

}  // namespace

namespace {
// Interleaved rotary embedding of the new token's q and k (`rope_i`, candle-nn/src/rotary_emb.rs:53-66: pairs
// (x[2i], x[2i+1]) rotated by the angle of (position, i), product then difference / sum like the CPU loop) and the
// append of k and v to the f32 cache at that position (candle-nn/src/kv_cache.rs:143-164), in one pass.
// qkv [B, row_stride] holds q (n_head * D), k (n_kv * D), v (n_kv * D) side by side; cos / sin [D / 2] of the position.
__global__ void __launch_bounds__(256)
rope_kv_append_kernel(const float* __restrict__ qkv, int64_t row_stride, const float* __restrict__ cos, const float* __restrict__ sin,
                      int n_head, int n_kv, int D, int64_t max_seq, int pos, float* __restrict__ q_out, float* __restrict__ kc,
                      float* __restrict__ vc) {
    pdl_trigger();
    pdl_wait();
    const int b = blockIdx.x;
    const int half = D / 2, n_q = n_head * half, n_k = n_kv * half;
    const float* row = qkv + (int64_t)b * row_stride;
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < n_q + 2 * n_k; i += gridDim.y * blockDim.x) {
        if (i < n_q + n_k) {
            const bool is_q = i < n_q;
            const int j = is_q ? i : i - n_q;
            const int h = j / half, ip = j - h * half;
            const float* src = row + (is_q ? 0 : n_head * D) + h * D + 2 * ip;
            const float x0 = src[0], x1 = src[1], c = cos[ip], s = sin[ip];
            const float o0 = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s)), o1 = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
            float* dst = is_q ? q_out + ((int64_t)b * n_head + h) * D + 2 * ip
                              : kc + (((int64_t)b * n_kv + h) * max_seq + pos) * D + 2 * ip;
            dst[0] = o0;
            dst[1] = o1;
        } else {
            const int j = i - n_q - n_k;
            const int h = j / half, ip = j - h * half;
            const float* src = row + (n_head + n_kv) * D + h * D + 2 * ip;
            float* dst = vc + (((int64_t)b * n_kv + h) * max_seq + pos) * D + 2 * ip;
            dst[0] = src[0];
            dst[1] = src[1];
        }
    }
}
}  // namespace

cudaError_t launch_rope_kv_append(cudaStream_t st, const float* qkv, int64_t row_stride, const float* cos, const float* sin, int B,
                                  int n_head, int n_kv, int D, int64_t max_seq, int pos, float* q_out, float* kc, float* vc) {
    if (B == 0) return cudaSuccess;
    // a pair of values per thread: one CTA per sequence was a chain of 12 trips to memory (32 sequences, 6144 values: 6.8 us)
    const unsigned slabs = (unsigned)(((n_head + 2 * n_kv) * (D / 2) + 255) / 256);
    return launch_k(rope_kv_append_kernel, dim3(B, slabs), dim3(256), 0, st, qkv, row_stride, cos, sin, n_head, n_kv, D, max_seq, pos, q_out,
                    kc, vc);
}

size_t decode_attention_workspace_bytes(int B, int n_head, int head_dim, int n_ctx) {
    size_t rows = (size_t)B * ((n_ctx + ATT_CHUNK - 1) / ATT_CHUNK);  // chunks of all sequences
    if (head_dim == RING_D && n_head % RING_G == 0) {
        // A bound for every batch up to B and context up to n_ctx: a chunk below ATT_CHUNK means that twice its length gave
        // fewer than RING_MIN_UNITS units, so that there are fewer than 2 RING_MIN_UNITS + B n_kv of them.
        const size_t small = (size_t)2 * RING_MIN_UNITS / (n_head / RING_G) + B;
        rows = std::max(rows, std::min((size_t)B * ((n_ctx + RING_MIN_CHUNK - 1) / RING_MIN_CHUNK), small));
    }
    return rows * n_head * (head_dim + 2) * sizeof(float);
}

cudaError_t launch_decode_attention(cudaStream_t st, const float* q, const float* kc, const float* vc, int B, int n_head, int n_kv,
                                    int head_dim, int64_t max_seq, int n_ctx, float scale, float* y, float* workspace) {
    if (B == 0 || n_ctx == 0) return cudaSuccess;
    const int G = n_head / n_kv;
    if (head_dim == 128) {
        if (G == 4) return launch_att<128, 4>(st, q, kc, vc, B, n_kv, max_seq, n_ctx, scale, y, workspace);
        if (G == 1) return launch_att<128, 1>(st, q, kc, vc, B, n_kv, max_seq, n_ctx, scale, y, workspace);
        if (G == 8) return launch_att<128, 8>(st, q, kc, vc, B, n_kv, max_seq, n_ctx, scale, y, workspace);
    }
    if (head_dim == 64) {
        if (G == 4) return launch_att<64, 4>(st, q, kc, vc, B, n_kv, max_seq, n_ctx, scale, y, workspace);
        if (G == 1) return launch_att<64, 1>(st, q, kc, vc, B, n_kv, max_seq, n_ctx, scale, y, workspace);
    }
    return cudaErrorNotSupported;
}

}  // namespace cmoe
