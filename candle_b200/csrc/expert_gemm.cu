// Grouped expert products for large batches (prefill): tcgen05 tensor cores, operands and accumulators
// in tensor memory.
//
// out[p, n] = W_e[n, :] . act[row(p), :] for all grouped positions p of every expert, as a grouped GEMM
// over tiles of 128 weight rows x 128 (64, 32) grouped positions.  The integers are the reference's
// (candle-core/src/quantized/k_quants.rs:1205-1285 Q4_K, :1520-1600 Q6_K): activations are the int8
// Q8K rows, and the weight operand holds (sub-block scale) x (quant).  After every 256-element block
// the accumulator is drained and scaled by d_w(row, block) * d8(position, block) on the CUDA cores.
//   Q4_K: fp16 operand sc_j * q (at most 63 * 15, exact), `tcgen05.mma kind::f16`, fp32 accumulation in tensor memory
//         -- exact while a block's sum stays below 2^24, which it does by a wide margin for real data.  The min term: beside
//         up to 64 positions exact integers in an accumulator of its own, beside 128 three tf32 steps per block against
//         dmin / d into the main one (see prep_gemm_b_kernel).
//   Q6_K: sc_j * (q - 32) reaches 4096 and is not always an fp16 integer: two int8 planes, `kind::i8`, int32
//         accumulation (exact).  Reads the repacked layout of the decode kernels (16-byte aligned pieces; the
//         210-byte GGUF blocks are only 2-byte aligned).
//   Q8_0: see GemmQ80 and GemmQ80X.
//
// One CTA per SM, persistent over tiles, warp-specialised:
//   4 or 8 warps  epilogue: drain TMEM once per block, scale, keep CH columns per thread in registers (taken from
//                 the last warpgroup with setmaxnreg); at the end of a tile apply the SiLU gate and store
//   8 warps       unpack: two groups take the blocks in turn, a thread a weight row; the operand goes straight into
//                 TENSOR MEMORY (tcgen05.st) and never touches shared memory, whose bandwidth the B operand needs
//   4 warps       raw weight blocks -> shared memory; activation scales of the drain; TMA of the activation operand
//                 (128-byte swizzle, half a 256-wide block per stage); MMA issue (A from TMEM, B from shared memory)
// Everything goes through short rings of mbarriers: weight stages, pairs of weight slabs with their activation stage, two
// accumulators (the MMAs of block b+1 overlap the drain of block b).  gate_up interleaves rows of W1 and W3 so that the two
// factors of silu(w1 x) * (w3 x) sit in neighbouring lanes and meet with one shuffle.
//
// What bounds it: not one unit but the kernel's instruction streams.  Narrow tiles (a Mixtral-shaped layer at 100 rows, gate_up)
// took the same 0.9 us per 128 x 256 block with the unpack's arithmetic, the drain's arithmetic, most of the MMAs and half of
// the operand copies taken out: the MMA warp walked its few dozen instructions per pair of slabs at several clocks each beside
// busy warps, behind an instruction cache that 60-90 KB of code -- every wait written out with its give-up path at every place
// -- did not fit.  Hence constant ring addresses, waits of a few instructions (mbar_wait_tight), no tile search in the unpack
// warps, one barrier per pair for both operands, masks fused with the fp16 magic number (field).  Counters of the result, gate_up / down:
// issue slots busy 64 / 66 % of the active cycles at 100 rows, 66 / 72 % at 2048; tensor pipe 23 / 13 and 67 / 40 %.  Layers, before -> after: Mixtral-shaped,
// 100 rows 388 -> 315 us, 2048 rows 2471 -> 2079; 8 small experts from GGUF blocks, 257 rows 79.4 -> 72.3; 60 Q8_0 experts,
// 4096 rows 1776 -> 1710; [32000, 4096] Q6_K at 32 rows 49.4 -> 44.4, [4096, 4096] Q4_K at 777 rows 53.8 -> 48.7.
// Every mbarrier wait is bounded (see stream_common.cuh); nothing here uses cluster multicast.
#include <algorithm>
#include <cmath>
#include <cuda_fp16.h>
#include <cudaTypedefs.h>

#include "common.cuh"
#include "tc5_common.cuh"

namespace cmoe {

namespace {

constexpr int G_TILE_M = 128, G_SLAB_K = 64;  // the position tile (N) is a template parameter: 128, or 32 for small batches
constexpr int G_PAD_ROWS = 128;                // zero rows after the last position, so that no box leaves the buffers
// Barriers of the weight stages go by the stage's number modulo this, not by the slot it stands for: each then belongs to one
// group of unpack warps, which sees every phase of it (a parity wait cannot tell phase k from phase k - 2).
constexpr int G_W_BARS = 8;
constexpr int G_MIN_K = 16;     // min term of Q4_K: floats per row and block, two K steps of tf32 (64-byte rows, 64-byte swizzle)
constexpr int G_TMEM_COLS = 512;
constexpr int G_RUN = 4;  // blocks that narrow tiles add in a row

// Tensor maps of the weight matrices reach device memory as kernel PARAMETERS -- of the operand preparation that runs before the
// GEMM anyway, and of a small copy kernel for what does not fit there -- never
// from host memory on the stream: a copy node recorded while a stream is being captured into a CUDA graph reads
// its host source again at every replay, long after the array it pointed to has gone.
constexpr int MAPS_PER_CHUNK = 16;
struct MapChunk {
    CUtensorMap m[MAPS_PER_CHUNK];
    CUtensorMap* dst;
    int n;  // 0: none
};
__device__ __forceinline__ void write_maps(const MapChunk& c) {  // by one CTA, after the previous user of the scratch has finished
    const uint4* src = reinterpret_cast<const uint4*>(c.m);
    uint4* d = reinterpret_cast<uint4*>(c.dst);
    for (int i = threadIdx.x; i < c.n * (int)(sizeof(CUtensorMap) / 16); i += blockDim.x) d[i] = src[i];
}
__global__ void __launch_bounds__(128) write_maps_kernel(const __grid_constant__ MapChunk c) {
    pdl_trigger();
    pdl_wait();
    write_maps(c);
}

// ---------------------------------------------------------------------------------------------
// Operand preparation: the int8 activation rows in grouped order as fp16 (B operand), the block scales
// transposed to [block][position], and the activation side of the Q4_K min term (below).
// Inside every group of 4 k the order is (0, 2, 1, 3): the weight unpack produces that order for
// free (nibbles of bytes 0,2 and 1,3 convert pairwise), and a dot product does not care.
// Rows p >= P are zero padding so that a 128-row box never leaves the buffer.
//
// Min term of Q4_K (k_quants.rs:1262-1268): block b contributes d8[p,b] * (d[r,b] * M - dmin[r,b] * sum_j m_j bsum32_j)
// = d8 * d * (M - sum_j rho_j bsum32_j) with rho_j = dmin * m_j / d, so the min term joins the SAME accumulator
// as the integer main sum M: three more K=8 steps per block, kind::tf32 (fp32 exponent range, 10-bit
// mantissa).  rho_j (fp32) is split into tf32 terms r1 + r2 (to 2^-23), the integer bsum32 (at most 32 * 127,
// 12 bits) exactly into b1 + b2; the steps are r1 b1 + r2 b1 + r1 b2.  Per (position, block) the buffer holds
// 16 floats [b1 (8) | b2 (8)], matched by [r1 | r2] on the weight side.  The main
// sum stays an exact integer until these last three steps; what they add in error is of the order of the
// reference's own f32 rounding (2^-23 of the min term).
//
// Position tiles of up to 64 have the tensor memory for an accumulator of its own: sum_j m_j bsum32_j is ONE fp16 step of exact
// integers per block, [m (8) | m (8)] against [c1 (8) | c2 (8)] with bsum32 = c1 + c2, c1 a multiple of 4, and the drain adds
// d8 * (d M - dmin Mm) like the reference.  Relative error against 64-bit arithmetic (K = 4096, 12800 rows): 1.55e-7 with the
// joined min term, 0.87e-7 (the streaming form 1.16e-7); a layer at 100 rows is as fast.
// ---------------------------------------------------------------------------------------------
// nearest value with a 10-bit mantissa (the 13 low bits of the fp32 container zero)
__device__ __forceinline__ float tf32_head(float v) { return __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u); }

// first part of a sum of 32 activations: its ten leading bits, or (fp16 steps) its multiple of 4
__device__ __forceinline__ float min_head(float bv, int fp16) { return fp16 ? 4.0f * rintf(0.25f * bv) : tf32_head(bv); }
__device__ __forceinline__ void store_min(float* bmin, int64_t i, float v, int fp16) {
    if (fp16)
        reinterpret_cast<__half*>(bmin)[i] = __float2half_rn(v);
    else
        bmin[i] = v;
}
// four integers of at most 128 as bytes: 2^23 + 2^22 + v has v in its low bits
__device__ __forceinline__ uint32_t pack_s8(float a, float b, float c, float d) {
    const uint32_t ab = __byte_perm(__float_as_uint(a + 12582912.f), __float_as_uint(b + 12582912.f), 0x0040);
    const uint32_t cd = __byte_perm(__float_as_uint(c + 12582912.f), __float_as_uint(d + 12582912.f), 0x0040);
    return __byte_perm(ab, cd, 0x5410);
}
// Q6_K: the int8 rows themselves, in grouped order
__global__ void __launch_bounds__(256)
prep_gemm_i8_kernel(const int8_t* __restrict__ aq, const float* __restrict__ ascale, const uint32_t* __restrict__ row_of, int P, int P_pad,
                    int K, int8_t* __restrict__ b8, float* __restrict__ d8t) {
    pdl_trigger();
    pdl_wait();
    const int kb = K >> 8;
    const int lane = threadIdx.x & 31;
    const int64_t unit = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);  // (p, block)
    if (unit >= (int64_t)P_pad * kb) return;
    const int p = (int)(unit / kb), blk = (int)(unit - (int64_t)p * kb);
    uint2 v = make_uint2(0, 0);
    float d8 = 0.f;
    if (p < P) {
        const int64_t row = row_of ? (int64_t)row_of[p] : (int64_t)p;
        v = *reinterpret_cast<const uint2*>(aq + row * K + blk * 256 + lane * 8);
        d8 = ascale[row * kb + blk];
    }
    *reinterpret_cast<uint2*>(b8 + (int64_t)p * K + blk * 256 + lane * 8) = v;
    if (lane == 0) d8t[(int64_t)blk * P_pad + p] = d8;
}

__global__ void __launch_bounds__(256)
prep_gemm_b_kernel(const int8_t* __restrict__ aq, const float* __restrict__ ascale, const int16_t* __restrict__ absum,
                   const uint32_t* __restrict__ row_of, int P, int P_pad, int K, __half* __restrict__ bf16,
                   float* __restrict__ bmin, int min_fp16, float* __restrict__ d8t, const __grid_constant__ MapChunk maps) {
    pdl_trigger();
    pdl_wait();
    if (blockIdx.x == 0) write_maps(maps);
    const int kb = K >> 8;
    const int lane = threadIdx.x & 31;
    const int64_t unit = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);  // (p, block)
    if (unit >= (int64_t)P_pad * kb) return;
    const int p = (int)(unit / kb), blk = (int)(unit - (int64_t)p * kb);
    uint4 o = make_uint4(0, 0, 0, 0);
    float bm = 0.f, d8 = 0.f;
    if (p < P) {
        const int64_t row = row_of ? (int64_t)row_of[p] : (int64_t)p;
        const uint2 v = *reinterpret_cast<const uint2*>(aq + row * K + blk * 256 + lane * 8);
        const int8_t* b = reinterpret_cast<const int8_t*>(&v);
        __half2 h[4];
        h[0] = __halves2half2(__int2half_rn(b[0]), __int2half_rn(b[2]));
        h[1] = __halves2half2(__int2half_rn(b[1]), __int2half_rn(b[3]));
        h[2] = __halves2half2(__int2half_rn(b[4]), __int2half_rn(b[6]));
        h[3] = __halves2half2(__int2half_rn(b[5]), __int2half_rn(b[7]));
        o = *reinterpret_cast<uint4*>(h);
        d8 = ascale[row * kb + blk];
        const int j = lane & 7;  // word j: b1_j, word 8 + j: b2_j
        const int16_t* bs = absum + row * (K / 16) + blk * 16 + 2 * j;
        const float bv = (float)((int)bs[0] + (int)bs[1]);
        const float b1 = min_head(bv, min_fp16), b2 = bv - b1;  // exact: |bv| <= 4096
        bm = lane < 8 ? b1 : b2;
    }
    *reinterpret_cast<uint4*>(bf16 + (int64_t)p * K + blk * 256 + lane * 8) = o;
    if (lane < G_MIN_K) store_min(bmin, ((int64_t)p * kb + blk) * G_MIN_K + lane, bm, min_fp16);
    if (lane == 0) d8t[(int64_t)blk * P_pad + p] = d8;
}

// Q8_0 activations (int8 values, one f32 scale per 32, candle_moe_quantize_act) as the fp16 operand d * q, rows in
// grouped order, columns padded with zeros to K_pad (a multiple of 256); the per-block scale table is all ones.
// exact = 1: 64 d q as the fp16 pair (rounded product, exact residual), a row laid out [256 of part 0 | 256 of part 1]
// per block, and 1 / 64 in the scale table.
__global__ void __launch_bounds__(256)
prep_gemm_b_q80_kernel(const int8_t* __restrict__ aq, const float* __restrict__ ascale, const uint32_t* __restrict__ row_of, int P,
                       int P_pad, int K, int K_pad, int exact, __half* __restrict__ bf16, float* __restrict__ d8t) {
    pdl_trigger();
    pdl_wait();
    const int kb = K_pad >> 8;
    const int lane = threadIdx.x & 31;
    const int64_t unit = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);  // (p, block of 256)
    if (unit >= (int64_t)P_pad * kb) return;
    const int p = (int)(unit / kb), blk = (int)(unit - (int64_t)p * kb);
    uint4 o = make_uint4(0, 0, 0, 0), o1 = make_uint4(0, 0, 0, 0);
    const int k0 = blk * 256 + lane * 8;
    if (p < P && k0 < K) {  // K is a multiple of 32: a lane's eight values lie inside one 32-block
        const int64_t row = row_of ? (int64_t)row_of[p] : (int64_t)p;
        const uint2 v = *reinterpret_cast<const uint2*>(aq + row * K + k0);
        const int8_t* b = reinterpret_cast<const int8_t*>(&v);
        const float df = ascale[row * (K / 32) + (k0 >> 5)];  // an f16 value widened to f32
        __half r0[8], r1[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float t = __fmul_rn(__fmul_rn((float)b[i], df), exact ? 64.0f : 1.0f);  // exact in f32: 8 x 11 bits
            r0[i] = __float2half_rn(t);
            r1[i] = __float2half_rn(__fsub_rn(t, __half2float(r0[i])));
        }
        __half2 h[4] = {__halves2half2(r0[0], r0[2]), __halves2half2(r0[1], r0[3]), __halves2half2(r0[4], r0[6]), __halves2half2(r0[5], r0[7])};
        __half2 g[4] = {__halves2half2(r1[0], r1[2]), __halves2half2(r1[1], r1[3]), __halves2half2(r1[4], r1[6]), __halves2half2(r1[5], r1[7])};
        o = *reinterpret_cast<uint4*>(h);
        o1 = *reinterpret_cast<uint4*>(g);
    }
    if (exact) {
        __half* dst = bf16 + (int64_t)p * (2 * K_pad) + blk * 512 + lane * 8;
        *reinterpret_cast<uint4*>(dst) = o;
        *reinterpret_cast<uint4*>(dst + 256) = o1;
    } else {
        *reinterpret_cast<uint4*>(bf16 + (int64_t)p * K_pad + blk * 256 + lane * 8) = o;
    }
    if (lane == 0) d8t[(int64_t)blk * P_pad + p] = exact ? 1.0f / 64.0f : 1.0f;
}

// The two preparations straight from f32 rows that lie in grouped order already (hidden rows before the down product, the
// rows of a dense product): the activation quantization of quantize_act.cu -- the same values bit for bit -- and the
// operand in one pass, so that the int8 rows neither travel to memory and back nor cost a launch.  A warp takes PREP_UNITS
// (row, 256-block) units, loads first; rows at or past P are zeros.  The rounded values stay floats (they are integers of at
// most 128): no conversion to int and back.  HBM-bound: 4 bytes read and 2 (Q8_0 exact: 4) written per element.
// Measured: 4096 hidden rows of 14336 (Q6_K down) 60.9 + 41.7 us in two passes, 64.5 us in one; 16384 rows of 1408 (Q8_0 down)
// 20.5 + 22.3 us against 28.1; one unit per warp and integer conversions took 82 us for the first.
constexpr int PREP_UNITS = 2;
__global__ void __launch_bounds__(256)
prep_gemm_f32_q8k_kernel(const float* __restrict__ x, int P, int P_pad, int K, int8_t* __restrict__ b8, __half* __restrict__ bf16, float* __restrict__ bmin,
                         int min_fp16, float* __restrict__ d8t, uint32_t* __restrict__ single_group, const __grid_constant__ MapChunk maps) {
    pdl_trigger();
    pdl_wait();
    if (blockIdx.x == 0) write_maps(maps);
    if (single_group && blockIdx.x == 0 && threadIdx.x < 2) single_group[threadIdx.x] = threadIdx.x ? (uint32_t)P : 0u;
    const int kb = K >> 8;
    const int lane = threadIdx.x & 31;
    const int64_t n_units = (int64_t)P_pad * kb;
    const int64_t unit0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * PREP_UNITS;  // (p, block)
    int p[PREP_UNITS], blk[PREP_UNITS];
    float4 a[PREP_UNITS], b[PREP_UNITS];
#pragma unroll
    for (int u = 0; u < PREP_UNITS; ++u) {
        p[u] = (int)((unit0 + u) / kb);
        blk[u] = (int)(unit0 + u - (int64_t)p[u] * kb);
        a[u] = b[u] = make_float4(0.f, 0.f, 0.f, 0.f);  // zeros quantize to zeros with scale 0
        if (p[u] < P) {
            const float4* src = reinterpret_cast<const float4*>(x + (int64_t)p[u] * K + blk[u] * 256) + lane * 2;
            a[u] = src[0];
            b[u] = src[1];
        }
    }
#pragma unroll
    for (int u = 0; u < PREP_UNITS; ++u) {
        if (unit0 + u >= n_units) return;
        float q[8], d8;
        quantize_q8k_values(a[u], b[u], q, d8);
        if (d8 == 0.f) {  // zeros, or a block of denormals: what the int8 row would hold
#pragma unroll
            for (int i = 0; i < 8; ++i) q[i] = (float)(int8_t)(int)q[i];
        }
        if (b8) {  // Q6_K: as int8
            uint2 o;
            o.x = pack_s8(q[0], q[1], q[2], q[3]);
            o.y = pack_s8(q[4], q[5], q[6], q[7]);
            *reinterpret_cast<uint2*>(b8 + (int64_t)p[u] * K + blk[u] * 256 + lane * 8) = o;
        } else {
            __half2 h[4] = {__floats2half2_rn(q[0], q[2]), __floats2half2_rn(q[1], q[3]), __floats2half2_rn(q[4], q[6]), __floats2half2_rn(q[5], q[7])};
            *reinterpret_cast<uint4*>(bf16 + (int64_t)p[u] * K + blk[u] * 256 + lane * 8) = *reinterpret_cast<uint4*>(h);
            float s = 0.f;  // sums of integers of at most 128: exact
#pragma unroll
            for (int i = 0; i < 8; ++i) s += q[i];
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);  // 32 elements = four lanes
            const int j = lane & 7;  // the words of prep_gemm_b_kernel
            const float bv = __shfl_sync(0xffffffffu, s, 4 * j), b1 = min_head(bv, min_fp16), b2 = bv - b1;
            if (lane < G_MIN_K) store_min(bmin, ((int64_t)p[u] * kb + blk[u]) * G_MIN_K + lane, lane < 8 ? b1 : b2, min_fp16);
        }
        if (lane == 0) d8t[(int64_t)blk[u] * P_pad + p[u]] = d8;
    }
}

__global__ void __launch_bounds__(256)
prep_gemm_f32_q80_kernel(const float* __restrict__ x, int P, int P_pad, int K, int K_pad, int exact, __half* __restrict__ bf16,
                         float* __restrict__ d8t, uint32_t* __restrict__ single_group) {
    pdl_trigger();
    pdl_wait();
    if (single_group && blockIdx.x == 0 && threadIdx.x < 2) single_group[threadIdx.x] = threadIdx.x ? (uint32_t)P : 0u;
    const int kb = K_pad >> 8;
    const int lane = threadIdx.x & 31;
    const int64_t n_units = (int64_t)P_pad * kb;
    const int64_t unit0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * PREP_UNITS;  // (p, block of 256)
    int p[PREP_UNITS], blk[PREP_UNITS];
    float4 a[PREP_UNITS], b[PREP_UNITS];
#pragma unroll
    for (int u = 0; u < PREP_UNITS; ++u) {
        p[u] = (int)((unit0 + u) / kb);
        blk[u] = (int)(unit0 + u - (int64_t)p[u] * kb);
        a[u] = b[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int k0 = blk[u] * 256 + lane * 8;
        if (p[u] < P && k0 < K) {  // K is a multiple of 32: whole groups of four lanes
            const float4* src = reinterpret_cast<const float4*>(x + (int64_t)p[u] * K + k0);
            a[u] = src[0];
            b[u] = src[1];
        }
    }
#pragma unroll
    for (int u = 0; u < PREP_UNITS; ++u) {
        if (unit0 + u >= n_units) return;
        const float v[8] = {a[u].x, a[u].y, a[u].z, a[u].w, b[u].x, b[u].y, b[u].z, b[u].w};
        float amax = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        const float d = __fdiv_rn(amax, 127.0f);
        const float id = d != 0.f ? __fdiv_rn(1.0f, d) : 0.f;
        const float df = __fmul_rn(__half2float(__float2half_rn(d)), exact ? 64.0f : 1.0f);  // a power of two: exact
        float t[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)  // exact in f32: 8 x 11 bits
            t[i] = __fmul_rn(fmaxf(fminf(roundf(__fmul_rn(v[i], id)), 127.f), -128.f), df);
        __half2 h[4] = {__floats2half2_rn(t[0], t[2]), __floats2half2_rn(t[1], t[3]), __floats2half2_rn(t[4], t[6]), __floats2half2_rn(t[5], t[7])};
        if (exact) {
            __half2 g[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int i0 = (i >> 1) * 4 + (i & 1);
                const float2 f = __half22float2(h[i]);
                g[i] = __floats2half2_rn(__fsub_rn(t[i0], f.x), __fsub_rn(t[i0 + 2], f.y));
            }
            __half* dst = bf16 + (int64_t)p[u] * (2 * K_pad) + blk[u] * 512 + lane * 8;
            *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<uint4*>(h);
            *reinterpret_cast<uint4*>(dst + 256) = *reinterpret_cast<uint4*>(g);
        } else {
            *reinterpret_cast<uint4*>(bf16 + (int64_t)p[u] * K_pad + blk[u] * 256 + lane * 8) = *reinterpret_cast<uint4*>(h);
        }
        if (lane == 0) d8t[(int64_t)blk[u] * P_pad + p[u]] = exact ? 1.0f / 64.0f : 1.0f;
    }
}

// Q8_0 GGUF rows [n][K / 32 blocks of 34 bytes] -> [ceil(n / 8)][2 * ceil(K / 256)][1088]: 8 rows x 128 elements, two
// 512-byte regions of 64 elements (chunk_pos order, a chunk of row g holds the words at 4 t, 16 + 4 t, 32 + 4 t, 48 + 4 t)
// and [8 rows][4] f16 scales; zeros past K and past n.  The pieces the decode kernels' fragments and the GEMM's
// row-per-lane reads both take with conflict-free 128-bit shared loads.  One CTA per half-tile block, one output word per
// thread.
__global__ void __launch_bounds__(288)
prepack_q80_kernel(const uint8_t* __restrict__ raw, int64_t n_rows, int K, int kb, uint8_t* __restrict__ dst) {
    const int64_t ht = blockIdx.x / kb;
    const int blk = (int)(blockIdx.x - ht * kb);
    uint32_t* out = reinterpret_cast<uint32_t*>(dst + (size_t)blockIdx.x * Q80_HTB_BYTES);
    const int w = threadIdx.x;
    if (w < 256) {
        const int region = w >> 7, pos = (w >> 2) & 31, cw = w & 3;
        const int t = pos >> 3, g = ((pos & 7) - 2 * t) & 7;  // inverse of chunk_pos
        const int64_t row = ht * 8 + g;
        const int k0 = blk * 128 + 64 * region + 16 * cw + 4 * t;
        uint32_t v = 0;
        if (row < n_rows && k0 < K) {
            const uint16_t* q = reinterpret_cast<const uint16_t*>(raw + (row * (K / 32) + (k0 >> 5)) * Q8_0_BYTES + 2 + (k0 & 31));
            v = (uint32_t)q[0] | ((uint32_t)q[1] << 16);
        }
        out[w] = v;
    } else if (w < 272) {
        uint32_t v = 0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int idx = 2 * (w - 256) + i;  // [g][j]
            const int64_t row = ht * 8 + (idx >> 2);
            const int b32 = blk * 4 + (idx & 3);
            if (row < n_rows && b32 * 32 < K)
                v |= (uint32_t)*reinterpret_cast<const uint16_t*>(raw + (row * (K / 32) + b32) * Q8_0_BYTES) << (16 * i);
        }
        out[w] = v;
    }
}

struct GemmParams {
    ExpertPtrs wa, wb;            // gate_up: W1 / W3, down: W2 (wb unused); GGUF blocks (Q4_K) or repacked (Q6_K)
    const uint32_t* offsets;      // [E + 1]
    const float* d8t;             // [kb][P_pad]
    float* out;                   // gate_up: hidden [P, N]; down: [P, N]
    const CUtensorMap* wmaps;     // device array [E][2]: raw blocks of W1 / W3 (or W2, second unused) as byte matrices
    int* status;
    int E, K, N, kb, P, P_pad;
    int m_tiles;                  // tiles along the weight rows (N / 64 for gate_up, N / 128 for down)
    int ksplit;                   // K splits (down only): partial outputs out + ks * split_stride, summed by the caller
    long long split_stride;
    uint32_t magic;               // 0x64006400 (see field)
};

__device__ __forceinline__ __half2 h2_bits(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t bits_h2(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
// (1024 + byte b of w) in both halves: 0x64xx is 1024 + xx in fp16
__device__ __forceinline__ __half2 byte_magic2(uint32_t w, int b) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(0x64646464u), "r"(0x4040u | (uint32_t)b | ((uint32_t)b << 8)));
    return h2_bits(r);
}
// (w & MASK) | magic in one operation: fields of the bytes of w dropped into the mantissa of 1024 (magic = 0x64006400, from a
// register that the compiler knows nothing about: as constants, mask and magic take an operation each)
template <uint32_t MASK>
__device__ __forceinline__ __half2 field(uint32_t w, uint32_t magic) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "n"(MASK), "r"(magic));
    return h2_bits(r);
}
template <uint32_t MASK>
__device__ __forceinline__ uint32_t or_field(uint32_t v, uint32_t w) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "n"(MASK), "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t w4(const uint4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

// ------------------------------------------------------------------------------------------------
// The unpack formats.  An unpack thread owns a tile row of a 256-block and goes through it in two halves: elements 128 h ..
// 128 h + 127, i.e. slabs 2h and 2h + 1 of 64 elements, handed over as one pair.  A slab is 32 TMEM columns of two
// elements each (A_PARTS times); element k of the slab belongs to column k / 2, inside a group of four in the order (0, 2),
// (1, 3).  All formats read raw blocks that were staged in shared memory (`row`: the thread's place in a stage).
//
// Q4_K, GGUF layout (144-byte blocks: d, dmin, 12 scale bytes, 128 nibble bytes): bytes 32 s .. 32 s + 31 of the nibbles
// are slab s, low nibbles k = 0..31, high nibbles k = 32..63.
// ------------------------------------------------------------------------------------------------
struct GemmQ4K {
    static constexpr bool EXACT_GATE = false, I8 = false, HAS_MIN = true;
    static constexpr int A_PARTS = 1, B_PARTS = 1;
    static constexpr bool HALF_TILES = false;  // staged as rows of GGUF blocks (tensor-map boxes)
    static constexpr int W_UNITS = 1;          // stages per 256-block
    static constexpr int W_UNIT_BYTES = G_TILE_M * Q4K_BYTES;
    struct Ctx {
        uint32_t dd;            // d (low half) and dmin (high half), fp16 bits
        uint32_t sc[2], mn[2];  // 6-bit scales / mins of the sub-blocks as bytes (utils.rs:50-60)
    };
    // (rows are 36 words apart: the eight lanes of a 16-byte load phase cover all 32 banks once)
    __device__ static __forceinline__ void begin(Ctx& c, uint32_t row, int) {
        const uint4 hdr = lds128_o<0>(row);
        const uint32_t s0 = hdr.y, s1 = hdr.z, s2 = hdr.w;
        c.dd = hdr.x;
        c.sc[0] = s0 & 0x3f3f3f3fu;
        c.mn[0] = s1 & 0x3f3f3f3fu;
        c.sc[1] = (s2 & 0x0f0f0f0fu) | (((s0 >> 6) & 0x03030303u) << 4);
        c.mn[1] = ((s2 >> 4) & 0x0f0f0f0fu) | (((s1 >> 6) & 0x03030303u) << 4);
        if ((hdr.x & 0x7fffu) == 0) c.sc[0] = c.sc[1] = 0;  // d = 0: the block is its min term alone (see scale_of)
    }
    // The epilogue multiplies the block's accumulator by d; a block with d = 0 (and no main sum, above) is
    // scaled by dmin instead so that its min term survives, or by 1 if both are zero.
    __device__ static __forceinline__ float scale_of(const Ctx& c) {
        const uint32_t hb = (c.dd & 0x7fffu) ? (c.dd & 0xffffu) : (((c.dd >> 16) & 0x7fffu) ? (c.dd >> 16) : 0x3c00u);
        return half_bits_to_float((uint16_t)hb);
    }
    // slab s of half h = sub-blocks 2s (low nibbles) and 2s + 1 (high nibbles) of the half.  0x6400 | n is 1024 + n
    // and fma(1024 + n, sc, -1024 sc) rounds the exact n * sc once; 0x6400 | (n << 4) is 1024 + 16 n and
    // fma(1024 + 16 n, sc / 16, -64 sc) does the same for a nibble left in the high half of its byte.
    __device__ static __forceinline__ void emit(const Ctx& c, uint32_t row, int, int h, uint32_t magic, uint32_t ta) {
        const __half2 k1024 = __float2half2_rn(1024.f);
        const uint32_t scs = h ? c.sc[1] : c.sc[0], a = row + 64 * h;
        const uint4 q[4] = {lds128_o<16>(a), lds128_o<32>(a), lds128_o<48>(a), lds128_o<64>(a)};
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const __half2 scl = __hsub2(byte_magic2(scs, 2 * s), k1024);
            const __half2 sch = __hsub2(byte_magic2(scs, 2 * s + 1), k1024);
            const __half2 offl = __hmul2(scl, __float2half2_rn(-1024.f));
            const __half2 sch16 = __hmul2(sch, __float2half2_rn(0.0625f)), offh = __hmul2(sch, __float2half2_rn(-64.f));
            uint32_t o[32];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t x = w4(q[2 * s + (i >> 2)], i & 3), y = x >> 8;  // bytes (0, 2) and (1, 3) of the four
                o[2 * i] = bits_h2(__hfma2(field<0x000F000Fu>(x, magic), scl, offl));
                o[2 * i + 1] = bits_h2(__hfma2(field<0x000F000Fu>(y, magic), scl, offl));
                o[16 + 2 * i] = bits_h2(__hfma2(field<0x00F000F0u>(x, magic), sch16, offh));
                o[16 + 2 * i + 1] = bits_h2(__hfma2(field<0x00F000F0u>(y, magic), sch16, offh));
            }
            tmem_st32(ta + 32 * s, o);
        }
    }
    // weight side of the min term (see prep_gemm_b_kernel): the eight mins, one fp16 step, for the tiles that accumulate them on their own
    __device__ static __forceinline__ void min_operand16(const Ctx& c, uint32_t (&r)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t v;  // 1024 + m in both halves
            asm("prmt.b32 %0, %1, %2, %3;" : "=r"(v) : "r"(c.mn[i >> 1]), "r"(0x64646464u), "r"(0x4140u + 0x0202u * (i & 1)));
            r[i] = bits_h2(__hsub2(h2_bits(v), __float2half2_rn(1024.f)));
        }
    }
    __device__ static __forceinline__ float d_of(const Ctx& c) { return half_bits_to_float((uint16_t)c.dd); }
    __device__ static __forceinline__ float neg_dmin_of(const Ctx& c) { return -half_bits_to_float((uint16_t)(c.dd >> 16)); }
    // ... and for the others -rho_j = -dmin m_j / d split into tf32 terms [r1 (8) | r2 (8)].  2^23 + m as float bits is 0x4B000000 | m.
    __device__ static __forceinline__ void min_operand(const Ctx& c, uint32_t (&r)[16]) {
        const float ratio = -__fdividef(half_bits_to_float((uint16_t)(c.dd >> 16)), scale_of(c));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float mf = __uint_as_float(__byte_perm(c.mn[j >> 2], 0x4B000000u, 0x7650 | (j & 3))) - 8388608.f;
            const float a = __fmul_rn(ratio, mf), a1 = tf32_head(a);
            r[j] = __float_as_uint(a1);
            r[8 + j] = __float_as_uint(tf32_head(__fsub_rn(a, a1)));
        }
    }
};

// ------------------------------------------------------------------------------------------------
// Q6_K, repacked layout (expert_direct.cu: per 8 rows x 256 elements, 1680 bytes: low nibbles 2 x 512,
// high bit pairs 512, 128 scales, 8 d; a row's four 16-byte chunks t of a 512-byte region lie in chunk_pos order).  Word
// cw of chunk t of half h holds elements k0 = 16 cw + 4 t .. + 3 of the half's two slabs (low nibbles: first slab, high
// nibbles: second), words 2h, 2h + 1 of chunk t of the third region their high bit pairs.
// sc * (q - 32) reaches 4096, two bits more than an fp16 operand holds: it is multiplied as int8, in two planes
// p = 256 hi + lo (lo unsigned) with an int32 accumulator each, put together again when a block is drained.  The sums are
// exact, int8 steps run at twice the rate of fp16 ones, and the activation operand is the int8 row itself.  (As two fp16
// operands -- the scale in halves, or the low and the high bits of the quant -- the products took the tensor pipe twice the time
// and the unpack 600-690 clocks per 128 x 128 weights, 560 this way.)
// ------------------------------------------------------------------------------------------------
struct GemmQ6K {
    static constexpr bool EXACT_GATE = false, I8 = true, HAS_MIN = false;
    static constexpr int A_PARTS = 1, B_PARTS = 1;
    static constexpr bool HALF_TILES = true;  // staged as half-tile blocks, one bulk copy per 8 rows
    static constexpr int W_UNITS = 1;
    static constexpr int W_UNIT_BYTES = G_TILE_M / 8 * Q6K_HTB_BYTES;
    struct Ctx {
        float d;
    };
    __device__ static __forceinline__ void begin(Ctx& c, uint32_t row, int g) { c.d = half_bits_to_float((uint16_t)lds16(row + 1664 + 2 * g)); }
    __device__ static __forceinline__ float scale_of(const Ctx& c) { return c.d; }
    // columns of a pair: [lo: slab 0 (16) | slab 1 (16) | hi: slab 0 | slab 1], element k of a slab in column k / 4
    __device__ static __forceinline__ void emit(const Ctx&, uint32_t row, int g, int h, uint32_t, uint32_t ta) {
        const uint2 scw = lds64_o<1536>(row + 16 * g + 8 * h);
        uint4 ql[4];
        uint2 qh[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint32_t c = row + 16 * chunk_pos(g, t);
            ql[t] = lds128_o<0>(c + 512 * h);
            qh[t] = lds64_o<1024>(c + 8 * h);
        }
#pragma unroll
        for (int s = 0; s < 2; ++s) {
#pragma unroll
            for (int c2 = 0; c2 < 2; ++c2) {
                uint32_t lo[8], hi[8];
#pragma unroll
                for (int cx = 0; cx < 2; ++cx) {
                    const int cw = 2 * c2 + cx, sc = (int)(int8_t)((s ? scw.y : scw.x) >> (8 * cw));
                    // 32768 - 32 sc in both halves: the biased products are positive, nothing is borrowed
                    const uint32_t bias = 0x80008000u - (uint32_t)(sc * 0x00200020);
                    const int bq = 2 * ((cw >> 1) + 2 * s);  // bit position of this quarter's pair in the high-bit byte
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const uint32_t qlw = w4(ql[t], cw), qhw = (cw & 1) ? qh[t].y : qh[t].x;
                        const uint32_t l = s ? qlw >> 4 : qlw, hb = bq < 4 ? qhw << (4 - bq) : qhw >> (bq - 4);
                        const uint32_t q = (l & 0x0f0f0f0fu) | (hb & ~0x0f0f0f0fu);  // (two bits above the quant are foreign)
                        const uint32_t e = (q & 0x003f003fu) * (uint32_t)sc + bias;         // bytes 0, 2: 32768 + sc (q - 32)
                        const uint32_t o = ((q >> 8) & 0x003f003fu) * (uint32_t)sc + bias;  // bytes 1, 3
                        lo[4 * cx + t] = __byte_perm(e, o, 0x6240);
                        hi[4 * cx + t] = __byte_perm(e, o, 0x7351) ^ 0x80808080u;
                    }
                }
                tmem_st8(ta + 16 * s + 8 * c2, lo);
                tmem_st8(ta + 32 + 16 * s + 8 * c2, hi);
            }
        }
    }
};

// Matrices without copies, repacked on their way (candle_moe_api.cu), and batches that the decode kernels or the streaming form
// would take as well.  The forms that take such a layer otherwise gate with expf and
// an exact division (silu_f); the hidden rows are quantized to int8 again, where a difference in the last bit can become a
// step, so this one does the same: largest relative error of a gate 2.4e-7 (8.1e-7 with __expf and an approximate division), of
// the hidden rows against 64-bit arithmetic 0.98-1.01e-7 (streaming form 0.98-1.01e-7, row-per-warp form 1.2-1.5e-7, without
// the exact gate 1.01-1.05e-7).  It costs 3-6 % of a layer of small matrices (8 experts of 1536 x 2560, 400 rows: 457 -> 470 us).
struct GemmQ6KExact : GemmQ6K {
    static constexpr bool EXACT_GATE = true;
};
struct GemmQ4KExact : GemmQ4K {
    static constexpr bool EXACT_GATE = true;
};

// ------------------------------------------------------------------------------------------------
// Q8_0, repacked layout (prepack_q80_kernel): half-tile blocks of 8 rows x 128 elements, two of them per 256-block, rows
// padded with zeros to a multiple of 256 elements.  The reference multiplies per 32-element
// block (sum of int8 products) * d_w * d_a in f32 (k_quants.rs:636-668); here both scales are folded into the fp16
// operands -- weight d_w * q, activation d_a * q, each rounded once to fp16 (2^-12 relative) -- and the products
// are accumulated in f32 by the tensor core over the whole row, so no per-block scaling is left for the epilogue.
// The rounding of the operands is the one deviation from the reference's arithmetic on this path: it shows as a
// relative L2 error of a few 1e-4 on a product, inside the block's bound (1e-3), and is measured by the tests.
// Used for the down product only (see launch_expert_gemm for why gate_up cannot afford that rounding).
// Half h of a 256-block is its half-tile block h; word cw of chunk t of region s holds elements 16 cw + 4 t .. + 3.
// ------------------------------------------------------------------------------------------------
struct GemmQ80 {
    static constexpr bool EXACT_GATE = false, I8 = false, HAS_MIN = false;
    static constexpr int A_PARTS = 1, B_PARTS = 1;
    static constexpr bool HALF_TILES = true;
    static constexpr int W_UNITS = 2;  // a stage is the half-tile blocks of one half
    static constexpr int W_UNIT_BYTES = G_TILE_M / 8 * Q80_HTB_BYTES;
    struct Ctx {};
    __device__ static __forceinline__ void begin(Ctx&, uint32_t, int) {}
    __device__ static __forceinline__ float scale_of(const Ctx&) { return 1.0f; }  // the scales are inside the operands
    // 4 int8 -> 2 columns of fp16 pairs (k0, k2), (k1, k3): the byte plus 128 is dropped into the mantissa of 1024
    // (0x6400 | b + 128 = 1152 + b), 1152 comes off exactly, one multiply rounds
    __device__ static __forceinline__ void split4(uint32_t v, __half2& e, __half2& f) {
        const __half2 k1152 = __float2half2_rn(1152.f);
        uint32_t a, b;
        const uint32_t w = v ^ 0x80808080u;
        asm("prmt.b32 %0, %1, %2, 0x4240;" : "=r"(a) : "r"(w), "r"(0x64646464u));  // bytes 0 and 2
        asm("prmt.b32 %0, %1, %2, 0x4341;" : "=r"(b) : "r"(w), "r"(0x64646464u));  // bytes 1 and 3
        e = __hsub2(h2_bits(a), k1152);
        f = __hsub2(h2_bits(b), k1152);
    }
    __device__ static __forceinline__ void emit(const Ctx&, uint32_t row, int g, int, uint32_t, uint32_t ta) {
        const uint2 sc = lds64_o<1024>(row + 8 * g);  // 4 f16 scales, two per slab
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const __half2 d2 = h2_bits(s ? sc.y : sc.x);
            uint32_t o[32];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const uint4 q = lds128_o<0>(row + 512 * s + 16 * chunk_pos(g, t));
#pragma unroll
                for (int cw = 0; cw < 4; ++cw) {
                    __half2 e, f;
                    split4(w4(q, cw), e, f);
                    const __half2 d = cw < 2 ? __low2half2(d2) : __high2half2(d2);
                    o[8 * cw + 2 * t] = bits_h2(__hmul2(e, d));
                    o[8 * cw + 2 * t + 1] = bits_h2(__hmul2(f, d));
                }
            }
            tmem_st32(ta + 32 * s, o);
        }
    }
};

// ------------------------------------------------------------------------------------------------
// Q8_0 with EXACT operands, for the gate_up product (whose f32 result is re-quantized to int8 and therefore has to
// match the reference to f32 rounding, not to fp16 rounding).  d * q has up to 19 significant bits: it is carried as
// two fp16 numbers, the rounded product and its exact residual (one more fused multiply-add), on both sides:
//   weights      4096 d_w q  = A0 + A1      (the power of two keeps the residuals out of the fp16 subnormals;
//   activations    64 d_a q  = B0 + B1       both come off again in the epilogue's scale)
// and the tensor core accumulates A0 B0 + A1 B0 + A0 B1 in f32 (A1 B1 is below 2^-22 of a term).  Three MMAs per
// K step; the activation operand is twice as large.
// ------------------------------------------------------------------------------------------------
struct GemmQ80X : GemmQ80 {
    static constexpr int A_PARTS = 2, B_PARTS = 2;
    __device__ static __forceinline__ float scale_of(const Ctx&) { return 1.0f / 4096.0f; }
    __device__ static __forceinline__ void emit(const Ctx&, uint32_t row, int g, int, uint32_t, uint32_t ta) {
        const uint2 sc = lds64_o<1024>(row + 8 * g);
#pragma unroll 1
        for (int s = 0; s < 2; ++s) {
            const __half2 d2 = __hmul2(h2_bits(s ? sc.y : sc.x), __float2half2_rn(4096.f));  // exact (a power of two)
            uint4 q[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) q[t] = lds128_o<0>(row + 512 * s + 16 * chunk_pos(g, t));
#pragma unroll
            for (int c2 = 0; c2 < 2; ++c2) {  // one 32-element block of the slab
                const __half2 d = c2 ? __high2half2(d2) : __low2half2(d2);
                uint32_t p0[16], p1[16];
#pragma unroll
                for (int cw = 0; cw < 2; ++cw)
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        __half2 e, f;
                        split4(w4(q[t], 2 * c2 + cw), e, f);
                        const __half2 re = __hmul2(e, d), rf = __hmul2(f, d);
                        p0[8 * cw + 2 * t] = bits_h2(re);
                        p0[8 * cw + 2 * t + 1] = bits_h2(rf);
                        p1[8 * cw + 2 * t] = bits_h2(__hfma2(e, d, __hneg2(re)));  // exact: the residual of a 19-bit product has at most 8 bits
                        p1[8 * cw + 2 * t + 1] = bits_h2(__hfma2(f, d, __hneg2(rf)));
                    }
                tmem_st16(ta + 64 * s + 16 * c2, p0);
                tmem_st16(ta + 64 * s + 32 + 16 * c2, p1);
            }
        }
    }
};

// How a kernel is laid out for a format and a position tile.  The rings of the kernel are short and their lengths divide the two
// blocks that the issuing loops are unrolled over, so that every address in them is a constant: with ring positions kept in
// registers a pair cost the MMA thread 680 clocks beside busy unpack warps, with constants 240.
template <class F, int TN>
struct GemmCfg {
    static constexpr int EPI_WARPS = TN == 32 ? 4 : 8;  // a warp drains 32 rows x CH columns
    static constexpr int CH = TN / (EPI_WARPS / 4);
    static constexpr int GROUPS = 2;                    // of four unpack warps: every other block (Q8_0: every other pair)
    static constexpr int WARPS = EPI_WARPS + 4 * GROUPS + 4, THREADS = 32 * WARPS;
    // registers per thread after the trade (setmaxnreg): their sum over the warpgroups is at most the launch allocation
    static constexpr int REGS_LAUNCH = WARPS == 20 ? 96 : 128;
    static constexpr bool WIDE_I8 = F::I8 && TN == 128;
    static constexpr int REGS_EPI = TN == 32 ? 160 : (WIDE_I8 ? 152 : 136);
    // (64-wide tiles of Q4_K: with 72 for the unpack warps they spilled 32 bytes; Mixtral-shaped layer, 200 rows 366 -> 359 us.  128-wide
    // ones spill 8, and gain nothing that way)
    static constexpr bool WIDE_UNPACK = F::HAS_MIN && TN == 64;
    static constexpr int REGS_DQ = TN == 32 ? 128 : (WIDE_UNPACK ? 80 : 72), REGS_MISC = TN == 32 ? 96 : (WIDE_I8 ? 32 : (WIDE_UNPACK ? 48 : 64));
    static_assert(EPI_WARPS / 4 * REGS_EPI + GROUPS * REGS_DQ + REGS_MISC <= WARPS / 4 * REGS_LAUNCH, "more registers than the launch has");
    static_assert(THREADS * REGS_LAUNCH <= 65536, "");
    // pairs of weight slabs (half blocks) in flight, each with its activation stage: two blocks, one with two-part operands
    static constexpr int RING = F::A_PARTS == 2 ? 2 : 4;
    // int8 products have two accumulators per position; 128-wide tiles then go through a block's positions in two passes,
    // one of which is drained during the other
    static constexpr int PASSES = F::I8 && TN == 128 ? 2 : 1;
    // Q4_K beside narrow tiles: the min term has an accumulator of its own (see prep_gemm_b_kernel)
    static constexpr bool MIN_ACC = F::HAS_MIN && TN <= 64;
    static constexpr int ACC_COLS = F::I8 || MIN_ACC ? 2 * TN / PASSES : TN;  // of one of the two accumulators
    // tensor memory: [two accumulators | pairs of weight slabs | min operands of two blocks (32-wide tiles; else in shared memory)]
    static constexpr bool MIN_TM = F::HAS_MIN && TN == 32, MIN_SM = F::HAS_MIN && !MIN_TM;
    static constexpr int SLAB_COLS = 32 * F::A_PARTS, PAIR_COLS = 2 * SLAB_COLS;
    static constexpr int TM_A = 2 * ACC_COLS, TM_MIN = TM_A + RING * PAIR_COLS;
    static_assert(TM_MIN + (MIN_TM ? 2 * G_MIN_K / 2 : 0) <= G_TMEM_COLS, "");
    // shared memory: activation stages (half blocks: two slabs, B_PARTS times), min operands per block, weight stages
    static constexpr int B_TILE = TN * G_SLAB_K * 2;                        // [TN x 64] fp16 or [TN x 128] int8
    static constexpr int B_BYTES = F::I8 ? B_TILE : 2 * F::B_PARTS * B_TILE;
    static constexpr int M_ROW = G_MIN_K * (MIN_ACC ? 2 : 4);  // bytes: fp16 or tf32
    static constexpr int M_BYTES = F::HAS_MIN ? TN * M_ROW : 0, MA_BYTES = MIN_SM ? G_TILE_M * M_ROW : 0;
    static constexpr int W_BYTES = F::W_UNIT_BYTES;
    static constexpr int FIXED = RING * B_BYTES + 2 * (M_BYTES + MA_BYTES);
    static constexpr int W_ROOM = 232448 - 1024 - 3072 /* barriers, offsets, weight scales */ - (MIN_ACC ? 2048 : 0) - 4 * TN * 4 - FIXED;
    static constexpr int W_STAGES = W_ROOM / W_BYTES < G_W_BARS ? W_ROOM / W_BYTES : G_W_BARS;
    static_assert(W_STAGES >= 2, "");
    static constexpr int SMEM = FIXED + W_STAGES * W_BYTES + 1024 /* alignment slack */;
};

// weight row of tile row r: gate_up tiles hold 8 rows of W1, then the same 8 rows of W3, and so on (64 rows of each)
template <bool GATE_UP>
__device__ __forceinline__ int weight_row(int mt, int r) {
    return GATE_UP ? mt * 64 + (r >> 4) * 8 + (r & 7) : mt * 128 + r;
}

struct TileCoord {
    int e, nt, mt;
    int ks, kb0, kb1;  // K split: this work item covers the 256-blocks [kb0, kb1) and writes partial output ks
    uint32_t p0, p_end;
};

// Walks the tiles of one CTA in order: tile id -> (expert, row tile, K split, position tile); position tiles are fastest, so the
// CTAs that run at the same time share a weight tile (fetched from HBM once) and each expert's activations stay in L2.  The
// expert is kept from tile to tile: looking it up from the first one again cost every role of the kernel up to E dependent
// shared-memory reads and a 64-bit division per tile, the issuing warps in line with their tiles (60 experts, 4096 rows: layer 1752
// -> 1678 us; [32000, 4096] Q6_K at 32 rows 49.4 -> 47.9).  32 bits hold a tile id: a
// tile id stands for at least 8 KB of results.
template <int TN>
struct TileWalk {
    const uint32_t* offs;
    uint32_t E, m_tiles, ksplit, blocks;  // blocks: 256-blocks of one K split
    uint32_t tile, first, e, n_tiles;     // next tile; first tile and position tiles of expert e
    __device__ __forceinline__ TileWalk(const uint32_t* offs_, int E_, int m_tiles_, int ksplit_, int kb)
        : offs(offs_), E(E_), m_tiles(m_tiles_), ksplit(ksplit_), blocks(kb / ksplit_), tile(blockIdx.x), first(0), e(0) {
        n_tiles = (offs[1] - offs[0] + TN - 1) / TN;
    }
    // how many tiles this CTA has (before the first next())
    __device__ __forceinline__ uint32_t tiles() const {
        uint32_t all = 0;
#pragma unroll 1
        for (uint32_t i = 0; i < E; ++i) all += (offs[i + 1] - offs[i] + TN - 1) / TN;
        all *= ksplit * m_tiles;
        return all > blockIdx.x ? (all - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    }
    __device__ __forceinline__ bool next(TileCoord& tc) {
        uint32_t per_mt = n_tiles * ksplit;
#pragma unroll 1
        while (tile - first >= per_mt * m_tiles) {
            first += per_mt * m_tiles;
            if (++e >= E) {
                --e;
                n_tiles = 0;  // and stays at the end
                return false;
            }
            n_tiles = (offs[e + 1] - offs[e] + TN - 1) / TN;
            per_mt = n_tiles * ksplit;
        }
        const uint32_t local = tile - first, mt = local / per_mt, rem = local - mt * per_mt;
        const uint32_t ks = ksplit == 1 ? 0u : rem / n_tiles;
        tc.e = (int)e;
        tc.mt = (int)mt;
        tc.ks = (int)ks;
        tc.nt = (int)(rem - ks * n_tiles);
        tc.kb0 = (int)(ks * blocks);
        tc.kb1 = (int)((ks + 1) * blocks);
        tc.p0 = offs[e] + (uint32_t)tc.nt * TN;
        tc.p_end = offs[e + 1];
        tile += gridDim.x;
        return true;
    }
};

template <class F, bool GATE_UP, int TN>
__global__ void __launch_bounds__(GemmCfg<F, TN>::THREADS, 1)
expert_gemm_kernel(const __grid_constant__ GemmParams P, const __grid_constant__ CUtensorMap map_b,
                   const __grid_constant__ CUtensorMap map_bs) {
    using C = GemmCfg<F, TN>;
    extern __shared__ uint8_t smem_raw[];
    // per pair: both operands there (four unpack warps and the copy), and its MMAs done
    __shared__ uint64_t full_p[C::RING], done_p[C::RING];
    __shared__ uint64_t acc_full[2], acc_free[2], full_w[G_W_BARS], empty_w[G_W_BARS];
    __shared__ uint32_t s_offs[CANDLE_MOE_MAX_EXPERTS + 1];
    constexpr int CH = C::CH;
    __shared__ __align__(16) float s_d8[4][TN];  // activation scales of the positions, per block (ring of 4)
    __shared__ float s_dw[4][G_TILE_M];  // per block (ring of 4) and tile row: the weight scale the drain multiplies by
    __shared__ float s_dm[C::MIN_ACC ? 4 : 1][C::MIN_ACC ? G_TILE_M : 1];  // ... and -dmin
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    constexpr int WARP_DQ0 = C::EPI_WARPS, WARP_MISC0 = WARP_DQ0 + 4 * C::GROUPS;
    constexpr int WARP_LOAD = WARP_MISC0, WARP_D8 = WARP_MISC0 + 1, WARP_TMA = WARP_MISC0 + 2, WARP_MMA = WARP_MISC0 + 3;
    // the warp index through a shuffle: the compiler then knows that it is warp-uniform and keeps role
    // dispatch, loop counters and MMA / TMA operands in uniform registers
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    pdl_trigger();
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* smem_min_b = smem + C::RING * C::B_BYTES;
    uint8_t* smem_min_a = smem_min_b + 2 * C::M_BYTES;
    uint8_t* smem_w = smem_min_a + 2 * C::MA_BYTES;
    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < C::RING; ++s) {
            mbar_init(&full_p[s], 4 + 1);
            mbar_init(&done_p[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 2);  // the accumulator and the scales of its positions
            mbar_init(&acc_free[b], C::EPI_WARPS / C::PASSES);
        }
        for (int s = 0; s < G_W_BARS; ++s) {
            mbar_init(&full_w[s], 1);
            mbar_init(&empty_w[s], 4);
        }
        fence_barrier_init();
    }
    if (warp == WARP_TMA) tmem_alloc(&s_tmem_base, G_TMEM_COLS);
    pdl_wait();  // nothing above touches what the kernels before leave
    for (int i = threadIdx.x; i <= P.E; i += C::THREADS) s_offs[i] = P.offsets[i];
    tc5_fence_before_sync();
    __syncthreads();
    tc5_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, s_tmem_base, 0);
    volatile int* abort_flag = &s_abort;
    TileWalk<TN> walk(s_offs, P.E, P.m_tiles, P.ksplit, P.kb);

    // Register budget: the warpgroup with the issuing warps (and the unpack warps, where they need fewer) hands registers back to
    // the CTA's pool and the epilogue takes them, so the total stays what the launch allocated (a request beyond the pool
    // would wait forever).
    if (warp >= WARP_MISC0) reg_dealloc<C::REGS_MISC>();
    else if (warp >= WARP_DQ0 && C::REGS_DQ < C::REGS_LAUNCH) reg_dealloc<C::REGS_DQ>();
    if (warp < WARP_DQ0) {
        if (C::REGS_EPI > C::REGS_LAUNCH) reg_alloc<C::REGS_EPI>();
        // ===================== epilogue =====================
        const int quarter = warp & 3, colhalf = warp >> 2;
        const int r = 32 * quarter + lane;  // tile row = TMEM lane
        const uint32_t ta_lane = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(C::PASSES == 2 ? colhalf * C::ACC_COLS : colhalf * CH);
        uint32_t ab = 0;
        TileCoord tc;
        while (walk.next(tc)) {
            // the accumulators are kept as pairs of columns: one packed fused multiply-add per pair and block
            uint64_t acc2[CH / 2];
#pragma unroll
            for (int i = 0; i < CH / 2; ++i) acc2[i] = 0ull;
            // Narrow tiles have registers to add the blocks in runs of G_RUN, the runs on their own ([32000, 4096] Q6_K at 32
            // rows, relative error against 64-bit arithmetic: 7.8e-8 in one run of 16, 6.5e-8 in two, 6.2e-8 in four)
            constexpr bool RUNS = TN <= 64;
            uint64_t run2[RUNS ? CH / 2 : 1];
            if (RUNS) {
#pragma unroll
                for (int i = 0; i < CH / 2; ++i) run2[RUNS ? i : 0] = 0ull;
            }
            for (int blk = tc.kb0; blk < tc.kb1;) {
              const int stop = RUNS ? min(blk + G_RUN, tc.kb1) : tc.kb1;
#pragma unroll 1
              for (; blk < stop; ++blk, ++ab) {
                const int buf = C::PASSES == 2 ? colhalf : (int)(ab & 1);
                mbar_wait_tight(&acc_full[buf], C::PASSES == 2 ? ab & 1 : (ab >> 1) & 1, abort_flag);
                tc5_fence_after_sync();
                const float dw = s_dw[ab & 3][r];  // left by the unpack warps when they produced this block
                const uint64_t dw2 = f32x2_pack(dw, dw);
                uint64_t dm2 = 0;
                if constexpr (C::MIN_ACC) {
                    const float dm = s_dm[ab & 3][r];
                    dm2 = f32x2_pack(dm, dm);
                }
                const uint32_t t_main = ta_lane + (uint32_t)(C::PASSES == 2 ? 0 : buf * C::ACC_COLS);
                const uint32_t d8_addr = smem_u32(&s_d8[ab & 3][colhalf * CH]);
                // Steps of 16 columns; the load of step i+1 is in flight while step i is scaled into
                // the register accumulators: acc += (d8[col] * dw[row]) * v.
                constexpr int NS = CH / 16, PL = C::ACC_COLS / 2;
                constexpr bool TWO = F::I8 || C::MIN_ACC;
                uint32_t stg[2][16], sth[2][TWO ? 16 : 1];  // int8: low and high plane; Q4_K: main sum and min term
                tmem_ld16(t_main, stg[0]);
                if constexpr (TWO) tmem_ld16(t_main + PL, sth[0]);
                tmem_ld_wait();
                tmem_ld_pin(stg[0]);
                if constexpr (TWO) tmem_ld_pin(sth[0]);
                static_for<NS>([&](auto Cc) {
                    constexpr int c = decltype(Cc)::value, s = c & 1;
                    if constexpr (c + 1 < NS) {
                        tmem_ld16(t_main + 16 * (c + 1), stg[s ^ 1]);
                        if constexpr (TWO) tmem_ld16(t_main + PL + 16 * (c + 1), sth[s ^ 1]);
                    }
                    if constexpr (F::I8) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) stg[s][i] = __float_as_uint((float)((int)stg[s][i] + 256 * (int)sth[s][i]));
                    }
                    static_for<4>([&](auto Qc) {
                        constexpr int q = decltype(Qc)::value;
                        const uint4 dv = lds128_o<64 * c + 16 * q>(d8_addr);  // base + constant: no address arithmetic
                        // per column pair packed operations (each half is the IEEE operation of the scalar form)
                        static_for<2>([&](auto Ic) {
                            constexpr int i = decltype(Ic)::value, j = 4 * q + 2 * i;
                            const uint64_t d8 = i ? f32x2_pack_bits(dv.z, dv.w) : f32x2_pack_bits(dv.x, dv.y);
                            const uint64_t main = f32x2_pack_bits(stg[s][j], stg[s][j + 1]);
                            uint64_t& a = acc2[8 * c + 2 * q + i];
                            if constexpr (C::MIN_ACC)  // d8 * (d M - dmin Mm): the two cancel before anything is rounded to the sum
                                a = f32x2_fma(f32x2_fma(dm2, f32x2_pack_bits(sth[s][j], sth[s][j + 1]), f32x2_mul(dw2, main)), d8, a);
                            else
                                a = f32x2_fma(f32x2_mul(dw2, d8), main, a);
                        });
                    });
                    if constexpr (c + 1 < NS) {
                        tmem_ld_wait();
                        tmem_ld_pin(stg[s ^ 1]);
                        if constexpr (TWO) tmem_ld_pin(sth[s ^ 1]);
                    }
                    if (c == NS - 2) {  // every column of this thread has been read: the accumulator may be overwritten
                        tc5_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&acc_free[buf]);
                    }
                });
              }
              if (RUNS && blk < tc.kb1) {
#pragma unroll
                  for (int i = 0; i < CH / 2; ++i) {
                      run2[RUNS ? i : 0] = f32x2_add(run2[RUNS ? i : 0], acc2[i]);
                      acc2[i] = 0ull;
                  }
              }
            }
            float acc[CH];
#pragma unroll
            for (int i = 0; i < CH / 2; ++i) f32x2_unpack(RUNS ? f32x2_add(run2[RUNS ? i : 0], acc2[i]) : acc2[i], acc[2 * i], acc[2 * i + 1]);
            // ---- store the tile ----
            const int n = weight_row<GATE_UP>(tc.mt, r);
            const uint32_t pc0 = tc.p0 + colhalf * CH;
            float* out_k = P.out + (size_t)tc.ks * P.split_stride;
            if (GATE_UP) {
                // the lane with bit 3 clear holds w1 x, its partner w3 x of the same output row: the first finishes the
                // first half of this warp's columns, the other the second half, one exchange per pair of columns
                const bool up = lane & 8;
                const uint32_t p0 = pc0 + (up ? CH / 2 : 0);
                int rows = (int)(tc.p_end - p0);
                float* out_p = out_k + (size_t)p0 * P.N + n;
                // In chunks, the registers moved up in between: written out, the stores of a tile are up to 14 KB of code that every
                // tile fetches anew while the MMAs wait for the accumulators (Mixtral-shaped layer, gate_up at 2048 rows 1007 -> 960 us, at 100 rows 155 -> 144;
                // 8 small experts at 257 rows 33.4 -> 27.7)
                constexpr int CHUNK = 8;
#pragma unroll 1
                for (int q = 0; q < CH / 2; q += CHUNK) {
#pragma unroll
                    for (int c = 0; c < CHUNK; ++c, out_p += P.N) {
                        const float recv = __shfl_xor_sync(0xffffffffu, up ? acc[c] : acc[c + CH / 2], 8);
                        const float gv = up ? recv : acc[c], uv = up ? acc[c + CH / 2] : recv;
                        const float v = (F::EXACT_GATE ? silu_f(gv) : __fdividef(gv, 1.0f + __expf(-gv))) * uv;
                        if (c < rows) *out_p = v;
                    }
#pragma unroll
                    for (int i = 0; i + CHUNK < CH / 2; ++i) {
                        acc[i] = acc[i + CHUNK];
                        acc[CH / 2 + i] = acc[CH / 2 + i + CHUNK];
                    }
                    rows -= CHUNK;
                }
            } else {
                int rows = (int)(tc.p_end - pc0);
                float* out_p = out_k + (size_t)pc0 * P.N + n;
                constexpr int CHUNK = 16;
#pragma unroll 1
                for (int q = 0; q < CH; q += CHUNK) {
#pragma unroll
                    for (int c = 0; c < CHUNK; ++c, out_p += P.N)
                        if (c < rows) *out_p = acc[c];
#pragma unroll
                    for (int i = 0; i + CHUNK < CH; ++i) acc[i] = acc[i + CHUNK];
                    rows -= CHUNK;
                }
            }
        }
    } else if (warp < WARP_MISC0) {
        // ===================== weight unpack -> operand in tensor memory =====================
        // A group takes every other block, a thread a whole row of it (Q8_0, whose halves stand on their own: every other
        // half), so that a header is decoded once, and the waits, the shared-memory reads and the hand-over of one block lie
        // behind the arithmetic of the other.  The loops stay rolled: the warps of a scheduler share its instruction cache
        // with the issuing warps, whose few instructions everything waits for.
        const int quarter = warp & 3, group = (warp - WARP_DQ0) >> 2;
        const int r = 32 * quarter + lane;
        const uint32_t ta_lane = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)C::TM_A;
        // where tile row r lies in a stage: rows (gate_up: the W1 rows first, then the W3 rows) or half-tiles in tile order
        const uint32_t w_row = smem_u32(smem_w) +
                               (F::HALF_TILES ? (uint32_t)((r >> 3) * (F::W_UNIT_BYTES * 8 / G_TILE_M))
                                : GATE_UP ? (uint32_t)((((r >> 3) & 1) * (G_TILE_M / 2) + (r >> 4) * 8 + (r & 7)) * (F::W_UNIT_BYTES / G_TILE_M))
                                          : (uint32_t)(r * (F::W_UNIT_BYTES / G_TILE_M)));
        const int g = r & 7;
        const uint32_t n_units = walk.tiles() * walk.blocks * F::W_UNITS;  // weight stages of this CTA: blocks or halves
        uint32_t ws = group;
#pragma unroll 1
        for (uint32_t u = group, n = 0; u < n_units; u += 2, ++n) {
            uint64_t* const bar_w = &empty_w[u % G_W_BARS];
            const uint32_t row = w_row + ws * C::W_BYTES;
            // the raw bytes were copied to shared memory by the loader warp
            mbar_wait_tight(&full_w[u % G_W_BARS], (u / G_W_BARS) & 1, abort_flag);
            typename F::Ctx ctx;
            F::begin(ctx, row, g);
            constexpr int H = 3 - F::W_UNITS;  // pairs of a unit
            // a ring slot is taken again by the same group: pass counts its uses so far
            const uint32_t first = H == 2 ? 2 * group : (C::RING == 4 ? u & 3 : u & 1);
            const uint32_t pass = H == 1 && C::RING == 4 ? n >> 1 : n;
#pragma unroll 1
            for (int h = 0; h < H; ++h) {
                const uint32_t slot = first + h;
                if (pass > 0) mbar_wait_tight(&done_p[slot], (pass - 1) & 1, abort_flag);  // the MMAs that read it last
                tc5_fence_after_sync();
                if (H == 2 ? h == 0 : group == 0) {  // for the drain of this block
                    if constexpr (C::MIN_ACC) {
                        s_dw[u & 3][r] = F::d_of(ctx);
                        s_dm[u & 3][r] = F::neg_dmin_of(ctx);
                    } else {
                        s_dw[(H == 2 ? u : u >> 1) & 3][r] = F::scale_of(ctx);
                    }
                }
                F::emit(ctx, row, g, h, P.magic, ta_lane + slot * C::PAIR_COLS);
                if constexpr (F::HAS_MIN) {
                    if (h == 1) {
                        // (the last min MMAs on these operands came before the commit just waited for)
                        if constexpr (C::MIN_ACC) {
                            uint32_t m[4];
                            F::min_operand16(ctx, m);
                            if constexpr (C::MIN_TM) {
                                const uint32_t t = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(C::TM_MIN + group * (G_MIN_K / 2));
                                tmem_st4(t, m);
                                tmem_st4(t + 4, m);
                            } else {
                                uint8_t* const a = smem_min_a + group * C::MA_BYTES + r * C::M_ROW;  // both halves alike: no swizzle to mind
                                *reinterpret_cast<uint4*>(a) = make_uint4(m[0], m[1], m[2], m[3]);
                                *reinterpret_cast<uint4*>(a + 16) = make_uint4(m[0], m[1], m[2], m[3]);
                                fence_proxy_async_smem();
                            }
                        } else {
                            uint32_t rho[16];
                            F::min_operand(ctx, rho);
                            uint8_t* const a = smem_min_a + group * C::MA_BYTES + r * C::M_ROW;
                            const int sw = (r >> 1) & 3;  // 64-byte swizzle
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                *reinterpret_cast<uint4*>(a + ((j ^ sw) << 4)) = make_uint4(rho[4 * j], rho[4 * j + 1], rho[4 * j + 2], rho[4 * j + 3]);
                            fence_proxy_async_smem();
                        }
                    }
                }
                tmem_st_wait();
                tc5_fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&full_p[slot]);
                    if (h == H - 1) mbar_arrive(bar_w);  // every byte of the stage has been used
                }
            }
            ws += 2;
            if (ws >= C::W_STAGES) ws -= C::W_STAGES;
        }
    } else if (warp == WARP_LOAD) {
        // ===================== weight loader: raw blocks of the tile rows -> shared memory =====================
        uint32_t unit = 0, ws = 0;
        bool ok = true;
        TileCoord tc;
        if constexpr (F::HALF_TILES) {
            // half-tile blocks of the repacked layout: one bulk copy per 8 tile rows (gate_up: W1 and W3 half-tiles alternate), all
            // issued by one lane from uniform registers: issued by sixteen lanes, they went out one after the other all the same,
            // about 80 clocks each, and the loader held up the all-Q8_0 products (60 experts, 4096 rows: down
            // 202 -> 164 us, shared down 144 -> 106, gate_up 467 -> 452).
            // No requests into L2 ahead: the CTAs of a weight tile's position tiles run together and share the lines.
            constexpr int HT_BYTES = F::W_UNIT_BYTES * 8 / G_TILE_M, N_HT = G_TILE_M / 8;
            const size_t pitch = (size_t)P.kb * F::W_UNITS * HT_BYTES;  // from a half-tile of rows to the next
            while (ok && walk.next(tc)) {
                const size_t off = (size_t)tc.mt * (GATE_UP ? N_HT / 2 : N_HT) * pitch + (size_t)tc.kb0 * F::W_UNITS * HT_BYTES;
                const uint8_t *src = P.wa.p[tc.e] + off, *src3 = GATE_UP ? P.wb.p[tc.e] + off : nullptr;
#pragma unroll 1
                for (uint32_t left = walk.blocks * F::W_UNITS; left > 0; --left, ++unit) {
                    const uint32_t last = unit - C::W_STAGES;
                    uint64_t* const bar = &full_w[unit % G_W_BARS];
                    if (unit >= (uint32_t)C::W_STAGES) ok = mbar_wait_tight(&empty_w[last % G_W_BARS], (last / G_W_BARS) & 1, abort_flag);
                    if (!(ok = __all_sync(0xffffffffu, ok))) break;  // nothing is issued after a wait that gave up
                    if (elect_one()) {
                        uint8_t* const dst = smem_w + ws * C::W_BYTES;
                        mbar_expect_tx(bar, F::W_UNIT_BYTES);
#pragma unroll
                        for (int i = 0; i < N_HT; ++i)
                            bulk_g2s(dst + i * HT_BYTES, GATE_UP ? (i & 1 ? src3 : src) + (i >> 1) * pitch : src + i * pitch, HT_BYTES, bar);
                    }
                    __syncwarp();
                    src += HT_BYTES;
                    if (GATE_UP) src3 += HT_BYTES;
                    if (++ws == C::W_STAGES) ws = 0;
                }
            }
        } else {
            // One TMA box per matrix and block: [64 rows x 144 bytes] of the byte matrix [n_rows, row_bytes]
            // (gate_up: the W1 rows, then the W3 rows; a TMA destination must be 128-byte aligned, so the halves cannot
            // be skewed against each other and neighbouring lanes, which alternate between them, share banks two by
            // two).
            int fenced = -1;
            constexpr int ROW_BYTES = F::W_UNIT_BYTES / G_TILE_M, HALF = F::W_UNIT_BYTES / 2;
            while (ok && walk.next(tc)) {
                const CUtensorMap* m0 = P.wmaps + 2 * tc.e;
                // the maps were written by a kernel earlier on the stream: fence an expert's once, before their first use by this
                // warp (every lane fences: any may be elected)
                if (fenced != tc.e) {
                    fenced = tc.e;
                    tensormap_fence_acquire(m0);
                    if (GATE_UP) tensormap_fence_acquire(m0 + 1);
                }
                const int y0 = GATE_UP ? tc.mt * 64 : tc.mt * 128;
#pragma unroll 1
                for (int blk = tc.kb0; blk < tc.kb1; ++blk, ++unit) {
                    const uint32_t last = unit - C::W_STAGES;
                    uint64_t* const bar = &full_w[unit % G_W_BARS];
                    if (unit >= (uint32_t)C::W_STAGES) ok = mbar_wait_tight(&empty_w[last % G_W_BARS], (last / G_W_BARS) & 1, abort_flag);
                    if (!(ok = __all_sync(0xffffffffu, ok))) break;
                    if (elect_one()) {
                        uint8_t* dst = smem_w + ws * C::W_BYTES;
                        mbar_expect_tx(bar, F::W_UNIT_BYTES);
                        tma_load_2d(dst, m0, blk * ROW_BYTES, y0, bar);
                        if (GATE_UP)
                            tma_load_2d(dst + HALF, m0 + 1, blk * ROW_BYTES, y0, bar);
                        else
                            tma_load_2d(dst + HALF, m0, blk * ROW_BYTES, y0 + 64, bar);
                    }
                    __syncwarp();
                    if (++ws == C::W_STAGES) ws = 0;
                }
            }
        }
    } else if (warp == WARP_D8) {
        // ===================== activation scales of the drain =====================
        // From global memory two blocks ahead, to shared memory when the accumulator they go with has been drained of what it
        // held before: the epilogue then waits for one barrier per block.  (Loaded by the epilogue itself, a block's scales held
        // it for the latency of L2; requested there by asynchronous copies, for the instructions that this took, 300 clocks of
        // 1700 beside busy unpack warps.)
        constexpr int NR = TN / C::PASSES / 32;  // values per lane and pass
        TileCoord tc;
        float v[NR * C::PASSES], old[NR * C::PASSES];
        const float* dp = nullptr;
        uint32_t left = 0;
#pragma unroll 1
        for (uint32_t ab = 0;; ++ab) {  // asks for the scales of block ab, hands over those of block ab - 1
            bool more = true;
            if (left == 0) {
                more = walk.next(tc);
                left = more ? walk.blocks : 0;
                dp = P.d8t + (size_t)tc.kb0 * P.P_pad + tc.p0 + lane;
            }
            if (more) {
#pragma unroll
                for (int i = 0; i < NR * C::PASSES; ++i) v[i] = dp[32 * i];
                dp += P.P_pad;
                --left;
            }
            if (ab > 0) {
                const uint32_t bl = ab - 1;
#pragma unroll
                for (int ps = 0; ps < C::PASSES; ++ps) {
                    const uint32_t buf = C::PASSES == 2 ? ps : bl & 1, turn = C::PASSES == 2 ? bl : bl >> 1;  // uses of this accumulator so far
                    if (turn > 0) mbar_wait_tight(&acc_free[buf], (turn - 1) & 1, abort_flag);
#pragma unroll
                    for (int i = 0; i < NR; ++i) s_d8[bl & 3][32 * (NR * ps + i) + lane] = old[NR * ps + i];
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_full[buf]);
                }
            }
            if (!more) break;
#pragma unroll
            for (int i = 0; i < NR * C::PASSES; ++i) old[i] = v[i];
        }
    } else if (warp == WARP_TMA) {
        // ===================== TMA: activation operand =====================
        // One stage = the slabs of one pair: [part 0: two slabs | part 1: two slabs], int8: the 128 bytes of the half in one box;
        // a row of two-part operands holds [256 of part 0 | 256 of part 1] per block.  The min operand of a block comes with its
        // second pair.  Unrolled over two blocks, like the MMA loop.
        TileCoord tc;
        uint32_t it = 0;
        bool second = false, ok = true;
        const auto load_block = [&](auto Bc, int blk) {
            constexpr int B = decltype(Bc)::value, R = C::RING;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int st = (2 * B + h) % R;
                // use it (ring of two blocks) or 2 it + B (of one) of this stage
                if (R == 4 ? it > 0 : it > 0 || B > 0) ok = ok && mbar_wait_tight(&done_p[st], R == 4 ? (it & 1) ^ 1 : (B & 1) ^ 1, abort_flag);
                if (elect_one() && ok) {  // nothing is issued after a wait that gave up
                    uint8_t* dst = smem + st * C::B_BYTES;
                    mbar_expect_tx(&full_p[st], C::B_BYTES + (h == 1 ? C::M_BYTES : 0));
                    if constexpr (F::I8) {
                        tma_load_2d(dst, &map_b, blk * 256 + h * 128, (int)tc.p0, &full_p[st]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 2 * F::B_PARTS; ++j)
                            tma_load_2d(dst + j * C::B_TILE, &map_b, blk * 256 * F::B_PARTS + (j >> 1) * 256 + (2 * h + (j & 1)) * 64,
                                        (int)tc.p0, &full_p[st]);
                    }
                    if (F::HAS_MIN && h == 1) tma_load_2d(smem_min_b + B * C::M_BYTES, &map_bs, blk * G_MIN_K, (int)tc.p0, &full_p[st]);
                }
                __syncwarp();
            }
        };
        while (walk.next(tc)) {
            int blk = tc.kb0;
            if (second) goto tma_second;
#pragma unroll 1
            for (;;) {
                second = true;
                load_block(std::integral_constant<int, 0>{}, blk);
                if (++blk == tc.kb1) break;
            tma_second:
                second = false;
                load_block(std::integral_constant<int, 1>{}, blk);
                ++it;
                if (++blk == tc.kb1) break;
            }
        }
    } else if (warp == WARP_MMA) {
        // ===================== MMA issue =====================
        // Everything else of the kernel waits for this loop, and beside busy warps each instruction in it counts at its full
        // latency and its place in the instruction cache: one barrier to wait for per pair, constant addresses (see GemmCfg); the
        // whole warp walks it, so that operands stay in uniform registers, and one elected lane issues.
        TileCoord tc;
        uint32_t it = 0, n_eff = 0, idesc[2] = {0, 0}, idesc_min = 0;
        bool second = false, full_n = false, free_n = false;
        const uint64_t b_desc = umma_desc_sw128(smem_u32(smem));
        const uint64_t mb_desc = C::MIN_ACC ? umma_desc_sw32(smem_u32(smem_min_b)) : umma_desc_sw64(smem_u32(smem_min_b));
        const uint64_t ma_desc = C::MIN_ACC ? umma_desc_sw32(smem_u32(smem_min_a)) : umma_desc_sw64(smem_u32(smem_min_a));
        // The whole warp's answer: after a wait that gave up, on whichever lane, it leaves its loop, and no MMA or commit is issued.
        // (known: the answer to a barrier asked ahead, looked at here, after it has had its time)
        const auto wait = [&](bool known, uint64_t* bar, uint32_t parity) {
            return (bool)__all_sync(0xffffffffu, known || mbar_wait_tight(bar, parity, abort_flag));
        };
        const auto block = [&](auto Bc) {  // block 2 it + B of this CTA; false: a wait gave up
            constexpr int B = decltype(Bc)::value, R = C::RING;
#pragma unroll
            for (int ps = 0; ps < C::PASSES; ++ps) {
                const int buf = C::PASSES == 2 ? ps : B;
                // the drain of what this accumulator held last: block ab - 2, with two passes ab - 1
                if (C::PASSES == 2 ? it > 0 || B > 0 : it > 0) {
                    if (!wait(free_n, &acc_free[buf], C::PASSES == 2 ? (B & 1) ^ 1 : (it & 1) ^ 1)) return false;
                }
                const uint32_t d_main = tmem_base + buf * C::ACC_COLS;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int st = (2 * B + h) % R;
                    if (ps == 0 && !wait(full_n, &full_p[st], R == 4 ? it & 1 : B & 1)) return false;
                    tc5_fence_after_sync();
                    if constexpr (C::PASSES == 1 && TN == 128) {
                        // ask the next barriers now: the answers, 200 to 300 clocks away, arrive while the MMAs are issued (gate_up of
                        // the Mixtral-shaped layer, 2048 rows 960 -> 930 us, [4096, 4096] at 777 rows 41.5 -> 39.5; narrow tiles, whose MMAs are
                        // over by then, gain nothing)
                        const uint32_t next_it = B == 1 && h == 1 ? it + 1 : it;
                        const int nb = h == 0 ? B : B ^ 1, nst = (2 * nb + (h ^ 1)) % R;
                        full_n = mbar_test(&full_p[nst], R == 4 ? next_it & 1 : nb & 1);
                        if (h == 1) free_n = mbar_test(&acc_free[nb], (next_it & 1) ^ 1);
                    }
                    if (elect_one()) {
                        const uint32_t a_t = tmem_base + C::TM_A + st * C::PAIR_COLS;
                        const uint64_t db = umma_desc_add(b_desc, st * (C::B_BYTES >> 4));
                        if constexpr (F::I8) {
                            uint32_t id0 = idesc[0], id1 = idesc[1];
                            if (ps == 1) {  // positions 64 .. 127
                                const uint32_t n = n_eff > 64 ? n_eff - 64 : 0;
                                id0 = umma_idesc_i8(G_TILE_M, 0, false) | ((n >> 3) << 17);
                                id1 = umma_idesc_i8(G_TILE_M, 0, true) | ((n >> 3) << 17);
                            }
                            if (ps == 0 || n_eff > 64) {
                                const uint64_t dp = umma_desc_add(db, ps * (64 * 128 >> 4));
#pragma unroll
                                for (int k = 0; k < 4; ++k) {  // K steps of 32: 8 columns of A, 32 bytes of B
                                    umma_i8_ts(d_main, a_t + 8 * k, umma_desc_add(dp, 2 * k), id0, (h | k) != 0);
                                    umma_i8_ts(d_main + C::ACC_COLS / 2, a_t + 32 + 8 * k, umma_desc_add(dp, 2 * k), id1, (h | k) != 0);
                                }
                            }
                        } else {
#pragma unroll
                            for (int k = 0; k < 8; ++k) {  // two slabs of four K steps
                                const uint32_t a_k = a_t + (k >> 2) * C::SLAB_COLS + 8 * (k & 3);
                                const uint64_t b_k = umma_desc_add(db, (k >> 2) * (C::B_TILE >> 4) + 2 * (k & 3));
                                umma_f16_ts(d_main, a_k, b_k, idesc[0], (h | k) != 0);
                                if (F::A_PARTS == 2) umma_f16_ts(d_main, a_k + 32, b_k, idesc[0], true);
                                if (F::B_PARTS == 2) umma_f16_ts(d_main, a_k, umma_desc_add(b_k, 2 * (C::B_TILE >> 4)), idesc[0], true);
                            }
                        }
                        if (F::HAS_MIN && h == 1) {
                            const uint64_t dm = umma_desc_add(mb_desc, B * (C::M_BYTES >> 4));
                            const uint64_t da = umma_desc_add(ma_desc, B * (C::MA_BYTES >> 4));
                            if constexpr (C::MIN_TM) {
                                umma_f16_ts(d_main + TN, tmem_base + C::TM_MIN + B * (G_MIN_K / 2), dm, idesc[0], false);
                            } else if constexpr (C::MIN_ACC) {
                                umma_f16(d_main + TN, da, dm, idesc[0], false);
                            } else {
                                // the min term joins the same accumulator: three tf32 steps r1 b1 + r2 b1 + r1 b2, last in the block
                                umma_tf32(d_main, da, dm, idesc_min, true);
                                umma_tf32(d_main, umma_desc_add(da, 2), dm, idesc_min, true);
                                umma_tf32(d_main, da, umma_desc_add(dm, 2), idesc_min, true);
                            }
                        }
                        // the pair's operands may be overwritten once these MMAs have read them
                        if (ps == C::PASSES - 1) umma_commit(&done_p[st]);
                        if (h == 1) umma_commit(&acc_full[buf]);
                    }
                    __syncwarp();
                }
            }
            return true;
        };
        while (!__any_sync(0xffffffffu, *abort_flag) && walk.next(tc)) {
            uint32_t left = walk.blocks;
            // The last position tile of an expert is rarely full: its MMAs run N = the rows it holds, rounded up to 16
            // (an MMA's time goes with N; the columns beyond are neither computed nor stored).
            n_eff = min((uint32_t)TN, (tc.p_end - tc.p0 + 15u) & ~15u);
            if constexpr (F::I8) {
                const uint32_t n = min(n_eff, (uint32_t)(TN / C::PASSES));
                idesc[0] = umma_idesc_i8(G_TILE_M, 0, false) | ((n >> 3) << 17);  // low plane: unsigned bytes
                idesc[1] = umma_idesc_i8(G_TILE_M, 0, true) | ((n >> 3) << 17);
            } else {
                idesc[0] = umma_idesc_f16(G_TILE_M, 0) | ((n_eff >> 3) << 17);
                idesc_min = umma_idesc_tf32(G_TILE_M, 0) | ((n_eff >> 3) << 17);
            }
            if (second) goto mma_second;
#pragma unroll 1
            for (;;) {
                second = true;
                if (!block(std::integral_constant<int, 0>{})) goto mma_end;
                if (--left == 0) break;
            mma_second:
                second = false;
                if (!block(std::integral_constant<int, 1>{})) goto mma_end;
                ++it;
                if (--left == 0) break;
            }
        }
    mma_end:;
    }
    tc5_fence_before_sync();
    __syncthreads();
    // After a wait that gave up, copies and MMAs of this CTA may still be under way (the issuing warps have stopped): give them
    // time, some microseconds each at most, before the shared and tensor memory go
    if (s_abort)
        for (int i = 0; i < 5000; ++i) __nanosleep(1000);
    if (warp == WARP_TMA) {
        tc5_fence_after_sync();
        tmem_dealloc(tmem_base, G_TMEM_COLS);
    }
    if (threadIdx.x == 0 && s_abort) atomicOr(P.status, 2);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point lookup (no link-time libcuda dependency)
EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// row-major matrix [rows, cols] -> boxes of [box_rows x box_cols], as wide as the swizzle (128 or 64 bytes)
bool make_map_2d(CUtensorMap* map, const void* base, CUtensorMapDataType dt, int elem_bytes, uint64_t rows, uint64_t cols,
                 uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * (uint64_t)elem_bytes};
    const cuuint32_t box[2] = {box_cols, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// byte matrix [rows, row_bytes] -> boxes of [box_rows x box_bytes], no swizzle
bool make_map_bytes(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_bytes, uint32_t box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {row_bytes, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_bytes, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int g_gemm_sms = -1;

template <class F, bool GATE_UP, int TN>
cudaError_t launch_gemm_kernel(cudaStream_t st, const GemmParams& G, const CUtensorMap& map_b, const CUtensorMap& map_bs) {
    using C = GemmCfg<F, TN>;
    auto kfn = expert_gemm_kernel<F, GATE_UP, TN>;
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return e;
    return launch_k(kfn, dim3(g_gemm_sms), dim3(C::THREADS), (size_t)C::SMEM, st, G, map_b, map_bs);
}

}  // namespace

size_t prepacked_q80_bytes(int64_t n_rows, int k) { return (size_t)((n_rows + 7) / 8) * (size_t)((k + 255) / 256) * 2 * Q80_HTB_BYTES; }
cudaError_t launch_prepack_q80(cudaStream_t st, const void* raw, int64_t n_rows, int k, void* dst) {
    const int kb = 2 * ((k + 255) / 256);
    const int64_t grid = (n_rows + 7) / 8 * kb;
    if (grid == 0) return cudaSuccess;
    prepack_q80_kernel<<<(unsigned)grid, 288, 0, st>>>(static_cast<const uint8_t*>(raw), n_rows, k, kb, static_cast<uint8_t*>(dst));
    return cudaGetLastError();
}

// Scratch the GEMM needs for P grouped rows of length K (fp16 operand, block-sum operand, scales).
size_t expert_gemm_scratch_bytes(int64_t P, int K, int parts) {
    K = (K + 255) / 256 * 256;  // Q8_0 rows are padded to whole 256-element blocks
    const size_t p_pad = (size_t)P + G_PAD_ROWS, kb = (size_t)K / 256;
    return align_up(p_pad * K * 2 * parts, 256) + align_up(p_pad * kb * G_MIN_K * 4, 256) + align_up(kb * p_pad * 4, 256) +
           sizeof(CUtensorMap) * 2 * CANDLE_MOE_MAX_EXPERTS;
}

bool expert_gemm_takes(bool gate_up, int dtype, bool repacked, int K, int N, int64_t P) {
    const bool q80 = dtype == CANDLE_GGML_Q8_0 && repacked;
    if (!((dtype == CANDLE_GGML_Q4K && !repacked) || (dtype == CANDLE_GGML_Q6K && repacked) || q80)) return false;
    return K % (q80 ? 32 : 256) == 0 && N % (gate_up ? 64 : 128) == 0 && P > 0 && P <= (1 << 30) && encode_tiled_fn() != nullptr;
}

// Takes Q4_K weights in GGUF layout (repacked = false), Q6_K weights in the repacked layout of the decode kernels
// and Q8_0 weights in the layout of prepack_q80_kernel (repacked = true); cudaErrorNotSupported for every other
// shape / dtype / layout.
cudaError_t launch_expert_gemm(cudaStream_t st, bool gate_up, const ExpertPtrs& wa, const ExpertPtrs& wb, int dtype,
                               bool repacked, int E, int K, int N, const uint32_t* offsets, const uint32_t* row_of, int64_t P,
                               int64_t max_rows, const int8_t* aq, const float* ascale, const int16_t* absum, float* out,
                               void* scratch, int max_splits, int* n_splits_out, int64_t split_stride, float* out_whole,
                               const float* x_f32, uint32_t* single_group, bool operand_ready, bool exact_gate, int max_run) {
    if (n_splits_out) *n_splits_out = 1;
    if (!scratch || !expert_gemm_takes(gate_up, dtype, repacked, K, N, P) || (x_f32 && row_of)) return cudaErrorNotSupported;
    int tn = max_rows <= 32 ? 32 : (max_rows <= 64 ? 64 : 128);  // position tile, from the bound / hint on an expert's rows
    const bool q80 = dtype == CANDLE_GGML_Q8_0 && repacked;
    // Q8_0: the DOWN product runs with operands that carry the block scales rounded to fp16 (a few 1e-4 relative on a
    // product), which a final product tolerates.  The gate_up product does not: its f32 hidden rows are re-quantized to
    // int8 before W2, and a relative difference of 1e-4 from the reference's hidden values already moves a few per cent
    // of those int8 values by one step (1 / 127 of the block's largest value) -- measured, that amplification puts the
    // block at 3e-3 .. 5e-3 relative L2, outside its bound.  gate_up therefore takes the exact two-part operands.
    const bool q80x = q80 && gate_up;
    const int parts = q80x ? 2 : 1;
    const int K_in = K;
    if (q80) K = (K + 255) / 256 * 256;  // the repacked rows and the fp16 operand are padded with zeros
    if (g_gemm_sms < 0) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        e = cudaDeviceGetAttribute(&g_gemm_sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
    }
    const int kb = K / 256;
    const int64_t p_pad = P + G_PAD_ROWS;
    uint8_t* base = static_cast<uint8_t*>(scratch);
    __half* bf16 = reinterpret_cast<__half*>(base);
    int8_t* b8 = reinterpret_cast<int8_t*>(base);  // Q6_K: int8 operand in the same place
    const bool i8 = dtype == CANDLE_GGML_Q6K;
    float* bmin = reinterpret_cast<float*>(base + align_up((size_t)p_pad * K * 2 * parts, 256));
    float* d8t = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bmin) + align_up((size_t)p_pad * kb * G_MIN_K * 4, 256));
    const bool has_min = dtype == CANDLE_GGML_Q4K;

    // byte-matrix tensor maps of the raw weight blocks (Q4_K): [n_rows, kb * 144] with boxes of 64 rows x one block, written to
    // the scratch on the stream before the kernel: the first chunk by the operand preparation, more (beyond eight experts) by
    // copy kernels
    CUtensorMap* wmaps_dev = reinterpret_cast<CUtensorMap*>(reinterpret_cast<uint8_t*>(d8t) + align_up((size_t)kb * p_pad * 4, 256));
    MapChunk first{};
    cudaError_t e;
    if (dtype == CANDLE_GGML_Q4K) {
        const uint64_t n_rows = (uint64_t)N, rb = (uint64_t)kb * Q4K_BYTES;
        for (int m0 = 0; m0 < 2 * E; m0 += MAPS_PER_CHUNK) {
            MapChunk chunk{};
            chunk.dst = wmaps_dev + m0;
            chunk.n = std::min(MAPS_PER_CHUNK, 2 * E - m0);
            for (int i = 0; i < chunk.n; ++i) {
                const int e2 = (m0 + i) >> 1;
                const uint8_t* wp = ((m0 + i) & 1) && gate_up ? wb.p[e2] : wa.p[e2];
                if (!make_map_bytes(&chunk.m[i], wp, n_rows, rb, Q4K_BYTES, 64)) return cudaErrorNotSupported;
            }
            if (m0 == 0) {
                first = chunk;
            } else {
                e = launch_k(write_maps_kernel, dim3(1), dim3(128), 0, st, chunk);
                if (e != cudaSuccess) return e;
            }
        }
    }

    const int64_t units = p_pad * kb;
    const int64_t per_cta = 8 * (x_f32 ? PREP_UNITS : 1);
    const dim3 prep_grid((unsigned)((units + per_cta - 1) / per_cta));
    if (operand_ready)  // an earlier call prepared the same rows in the same scratch (and wrote the maps, which Q4_K alone has)
        e = dtype == CANDLE_GGML_Q4K ? cudaErrorInvalidValue : cudaSuccess;
    else if (x_f32)
        e = q80 ? launch_k(prep_gemm_f32_q80_kernel, prep_grid, dim3(256), 0, st, x_f32, (int)P, (int)p_pad, K_in, K, q80x ? 1 : 0, bf16,
                           d8t, single_group)
                : launch_k(prep_gemm_f32_q8k_kernel, prep_grid, dim3(256), 0, st, x_f32, (int)P, (int)p_pad, K, i8 ? b8 : (int8_t*)nullptr,
                           bf16, has_min ? bmin : (float*)nullptr, tn <= 64 ? 1 : 0, d8t, single_group, first);
    else
        e = q80 ? launch_k(prep_gemm_b_q80_kernel, prep_grid, dim3(256), 0, st, aq, ascale, row_of, (int)P, (int)p_pad, K_in, K,
                           q80x ? 1 : 0, bf16, d8t)
            : i8 ? launch_k(prep_gemm_i8_kernel, prep_grid, dim3(256), 0, st, aq, ascale, row_of, (int)P, (int)p_pad, K, b8, d8t)
                 : launch_k(prep_gemm_b_kernel, prep_grid, dim3(256), 0, st, aq, ascale, absum, row_of, (int)P, (int)p_pad, K, bf16, bmin, tn <= 64 ? 1 : 0, d8t,
                            first);
    if (e != cudaSuccess) return e;

    CUtensorMap map_b, map_bs;
    if (i8 ? !make_map_2d(&map_b, b8, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)p_pad, (uint64_t)K, 2 * G_SLAB_K, tn)
           : !make_map_2d(&map_b, bf16, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (uint64_t)p_pad, (uint64_t)K * parts, G_SLAB_K, tn))
        return cudaErrorNotSupported;
    if (tn <= 64 ? !make_map_2d(&map_bs, bmin, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (uint64_t)p_pad, (uint64_t)kb * G_MIN_K, G_MIN_K, tn, CU_TENSOR_MAP_SWIZZLE_32B)
                 : !make_map_2d(&map_bs, bmin, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)p_pad, (uint64_t)kb * G_MIN_K, G_MIN_K, tn, CU_TENSOR_MAP_SWIZZLE_64B))
        return cudaErrorNotSupported;

    GemmParams G{};
    G.wmaps = wmaps_dev;
    G.wa = wa;
    G.wb = wb;
    G.offsets = offsets;
    G.d8t = d8t;
    G.E = E;
    G.K = K;
    G.N = N;
    G.kb = kb;
    G.P = (int)P;
    G.P_pad = (int)p_pad;
    G.m_tiles = gate_up ? N / 64 : N / 128;
    // down with few tiles (few experts with rows, narrow outputs): split K so that every SM has work; the partial
    // outputs are summed by whoever consumes them (combine, or the expert-parallel scatter)
    int ksplit = 1;
    if (!gate_up && n_splits_out && max_splits > 1) {
        // Position tiles of all experts: of its rows where there is one expert, else expected (in whole tiles) of rows scattered
        // around their average like independent draws
        double tiles = (double)((std::min<int64_t>(max_rows, P) + tn - 1) / tn);
        if (E > 1) {
            const double experts = (double)std::min<int64_t>(E, P), avg = std::min((double)P / E, (double)max_rows);
            // tiles of an expert beyond its first: those that nearly every expert fills, and the likely ones beyond
            const double spread = 4.0 * std::sqrt(avg) + 1.0, sure = std::max(1.0, std::floor((avg - spread) / tn));
            double extra = sure - 1.0;
            for (double m = sure * tn; m < avg + spread; m += tn) extra += 0.5 * std::erfc((m + 0.5 - avg) / std::sqrt(2.0 * avg));
            tiles = std::floor(experts * (1.0 + extra) + 0.1);
        }
        const int64_t items = G.m_tiles * (int64_t)tiles;
        // Time in blocks: whole waves of items over the SMs, an item being its blocks and a turn-over (the accumulators are
        // stored and a new tile begins) of about one block for 32-wide tiles, one and a half for 64, three and a half for 128.
        // A split has to shorten that by enough: partial sums cost a little in a consumer that reads the result anyway
        // (0.95), a kernel and their traffic where an unsplit result is final (0.75: [32000, 4096] at 32 rows is 250 items, two
        // waves whether split in two or not).  By waves alone, without the turn-over, sums of few blocks were split: 16 experts,
        // top-8, d = 2048, ff = 1024 (four blocks), 1000 rows 288 -> 399 us, now 267; 32 experts, top-4, d = 1536, ff = 2048, 800 rows 257
        // -> 206; 8 experts, d = 4096, ff = 4096, 257 rows 205 -> 187; ff = 14336, 100 rows 359 -> 365 (in runs, see the epilogue).
        const double turn = tn == 32 ? 1.0 : (tn == 64 ? 1.5 : 3.5);
        const auto time = [&](int ks) { return (double)((items * ks + g_gemm_sms - 1) / g_gemm_sms) * ((double)kb / ks + turn); };
        for (int ks = 2; ks <= max_splits && kb % ks == 0; ks *= 2)
            if (time(ks) < (out_whole ? 0.75 : 0.95) * time(ksplit)) ksplit = ks;
        while (max_run && kb / ksplit > max_run && ksplit * 2 <= max_splits && kb % (ksplit * 2) == 0) ksplit *= 2;
        *n_splits_out = ksplit;
    }
    G.ksplit = ksplit;
    G.out = ksplit == 1 && out_whole ? out_whole : out;
    G.split_stride = split_stride;
    G.magic = 0x64006400u;
    e = stream_status_ptr(&G.status);
    if (e != cudaSuccess) return e;
    if (dtype == CANDLE_GGML_Q4K) {
        if (gate_up && exact_gate && tn <= 64) {
            if (tn == 32) return launch_gemm_kernel<GemmQ4KExact, true, 32>(st, G, map_b, map_bs);
            return launch_gemm_kernel<GemmQ4KExact, true, 64>(st, G, map_b, map_bs);
        }
        if (tn == 32)
            return gate_up ? launch_gemm_kernel<GemmQ4K, true, 32>(st, G, map_b, map_bs) : launch_gemm_kernel<GemmQ4K, false, 32>(st, G, map_b, map_bs);
        if (tn == 64)
            return gate_up ? launch_gemm_kernel<GemmQ4K, true, 64>(st, G, map_b, map_bs) : launch_gemm_kernel<GemmQ4K, false, 64>(st, G, map_b, map_bs);
        return gate_up ? launch_gemm_kernel<GemmQ4K, true, 128>(st, G, map_b, map_bs) : launch_gemm_kernel<GemmQ4K, false, 128>(st, G, map_b, map_bs);
    }
    if (q80x) {
        if (tn == 32) return launch_gemm_kernel<GemmQ80X, true, 32>(st, G, map_b, map_bs);
        if (tn == 64) return launch_gemm_kernel<GemmQ80X, true, 64>(st, G, map_b, map_bs);
        return launch_gemm_kernel<GemmQ80X, true, 128>(st, G, map_b, map_bs);
    }
    if (q80) {
        if (tn == 32) return launch_gemm_kernel<GemmQ80, false, 32>(st, G, map_b, map_bs);
        if (tn == 64) return launch_gemm_kernel<GemmQ80, false, 64>(st, G, map_b, map_bs);
        return launch_gemm_kernel<GemmQ80, false, 128>(st, G, map_b, map_bs);
    }
    if (gate_up && exact_gate) {
        if (tn == 32) return launch_gemm_kernel<GemmQ6KExact, true, 32>(st, G, map_b, map_bs);
        if (tn == 64) return launch_gemm_kernel<GemmQ6KExact, true, 64>(st, G, map_b, map_bs);
        return launch_gemm_kernel<GemmQ6KExact, true, 128>(st, G, map_b, map_bs);
    }
    if (tn == 32)
        return gate_up ? launch_gemm_kernel<GemmQ6K, true, 32>(st, G, map_b, map_bs) : launch_gemm_kernel<GemmQ6K, false, 32>(st, G, map_b, map_bs);
    if (tn == 64)
        return gate_up ? launch_gemm_kernel<GemmQ6K, true, 64>(st, G, map_b, map_bs) : launch_gemm_kernel<GemmQ6K, false, 64>(st, G, map_b, map_bs);
    return gate_up ? launch_gemm_kernel<GemmQ6K, true, 128>(st, G, map_b, map_bs) : launch_gemm_kernel<GemmQ6K, false, 128>(st, G, map_b, map_bs);
}

}  // namespace cmoe
