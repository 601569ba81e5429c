// Grouped expert products for large batches (prefill): tcgen05 tensor cores, operands and accumulators
// in tensor memory.
//
// out[p, n] = W_e[n, :] . act[row(p), :] for all grouped positions p of every expert, as a grouped GEMM
// over tiles of 128 weight rows x 128 grouped positions.  The integers are the reference's
// (candle-core/src/quantized/k_quants.rs:1205-1285 Q4_K, :1520-1600 Q6_K): activations are the int8
// Q8K rows, and the weight operand holds (sub-block scale) x (quant), both exact in fp16, multiplied by
// `tcgen05.mma kind::f16` with fp32 accumulation in tensor memory -- exact while a 256-element block's
// sum stays below 2^24, which it does by a wide margin for real data.  After every 256-element block
// the accumulator is drained and scaled by d_w(row, block) * d8(position, block) on the CUDA cores.
//   Q4_K: operand sc_j * q (at most 63 * 15); the min term joins the same accumulator as three tf32
//         steps per block against dmin / d (see prep_gemm_b_kernel).
//   Q6_K: sc_j * (q - 32) reaches 4096 and is not always an fp16 integer, so the int8 scale is split
//         into ceil(sc/2) + floor(sc/2) and the slab is multiplied twice (each half at most 32 * 64 =
//         2048: exact).  Reads the repacked layout of the decode kernels (16-byte aligned pieces; the
//         210-byte GGUF blocks are only 2-byte aligned).
//
// One CTA per SM, persistent over tiles, warp-specialised (20 warps, five warpgroups):
//   warps 0-7   epilogue: drain TMEM (tcgen05.ld, next load in flight) once per block, scale, keep 64
//               columns per thread in registers (128 registers per thread, taken from the last
//               warpgroup with setmaxnreg); at the end of a tile apply the SiLU gate and store
//   warps 8-15  unpack the weight nibbles of [128 rows x 64 k] to fp16 x scale with one HFMA2 per two
//               elements and store them straight into TENSOR MEMORY (tcgen05.st): the A operand never
//               touches shared memory, whose bandwidth the B operand needs
//   warp  18    TMA: the activation operand, [128 positions x 64 k] fp16 boxes, 128-byte swizzle; one
//               stage is a whole 256-wide block (four boxes + the min-term box), two stages
//   warp  19    issues the MMAs (A from TMEM, B from shared memory) and commits to mbarriers; the whole
//               warp walks the loop with warp-uniform operands, one elected lane issues
// Tensor memory: two main accumulators (2 x 128 columns: the MMAs of block b+1 overlap the drain of
// block b) and a 256-column ring of weight-operand slabs, handed over in pairs.  gate_up interleaves
// rows of W1 and W3 (tile row 2i = W1 row, 2i+1 = W3 row) so the two factors of silu(w1 x) * (w3 x)
// sit in neighbouring lanes and meet with one shuffle.
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
constexpr int G_W_STAGES_MAX = 6;  // raw weight blocks in flight per CTA (narrow position tiles leave room for a deep ring)
constexpr int G_B_STAGES = 2;   // in shared memory, one 256-wide block each (four slabs + the min-term box for Q4_K)
constexpr int G_MIN_K = 16;     // min term of Q4_K: floats per row and block, two K steps of tf32 (64-byte rows, 64-byte swizzle)
constexpr int G_MIN_A_BYTES = G_TILE_M * G_MIN_K * 4;
constexpr int G_EPI_WARPS = 8, G_DQ_WARPS = 8;
// Warp roles.  The MMA and TMA warps take the highest indices: measured, their short instruction streams
// are served far better there than at the lowest ones (1.75x on the whole kernel).
constexpr int G_WARP_EPI0 = 0, G_WARP_DQ0 = G_WARP_EPI0 + G_EPI_WARPS, G_WARP_LOAD = 16, G_WARP_TMA = 18, G_WARP_MMA = 19;
constexpr int G_THREADS = 32 * 20;  // five warpgroups: 2 epilogue, 2 unpack, 1 with the TMA and MMA warps (+ 2 idle)
constexpr int G_REGS_EPI = 128, G_REGS_MISC = 32;  // budgets after the trade: 2 * 128 + 2 * 96 + 32 = 5 * 96, the launch allocation
constexpr int G_TMEM_COLS = 512;
constexpr int G_RUN = 8;  // blocks that narrow tiles add in a row
constexpr int G_TM_MAIN = 0;    // + 128 * buffer
constexpr int G_TM_A = 256;     // weight operand ring: columns 256..511

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
// ---------------------------------------------------------------------------------------------
// nearest value with a 10-bit mantissa (the 13 low bits of the fp32 container zero)
__device__ __forceinline__ float tf32_head(float v) { return __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u); }

__global__ void __launch_bounds__(256)
prep_gemm_b_kernel(const int8_t* __restrict__ aq, const float* __restrict__ ascale, const int16_t* __restrict__ absum,
                   const uint32_t* __restrict__ row_of, int P, int P_pad, int K, __half* __restrict__ bf16,
                   float* __restrict__ bmin, float* __restrict__ d8t, const __grid_constant__ MapChunk maps) {
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
        if (bmin) {
            const int j = lane & 7;  // word j: b1_j, word 8 + j: b2_j
            const int16_t* bs = absum + row * (K / 16) + blk * 16 + 2 * j;
            const float bv = (float)((int)bs[0] + (int)bs[1]);
            const float b1 = tf32_head(bv), b2 = bv - b1;  // exact: |bv| < 4096, so b2 is -1, 0 or 1
            bm = lane < 8 ? b1 : b2;
        }
    }
    *reinterpret_cast<uint4*>(bf16 + (int64_t)p * K + blk * 256 + lane * 8) = o;
    if (bmin && lane < G_MIN_K) bmin[((int64_t)p * kb + blk) * G_MIN_K + lane] = bm;
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
prep_gemm_f32_q8k_kernel(const float* __restrict__ x, int P, int P_pad, int K, __half* __restrict__ bf16, float* __restrict__ bmin,
                         float* __restrict__ d8t, uint32_t* __restrict__ single_group, const __grid_constant__ MapChunk maps) {
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
        __half2 h[4] = {__floats2half2_rn(q[0], q[2]), __floats2half2_rn(q[1], q[3]), __floats2half2_rn(q[4], q[6]), __floats2half2_rn(q[5], q[7])};
        *reinterpret_cast<uint4*>(bf16 + (int64_t)p[u] * K + blk[u] * 256 + lane * 8) = *reinterpret_cast<uint4*>(h);
        if (bmin) {
            float s = 0.f;  // sums of integers of at most 128: exact
#pragma unroll
            for (int i = 0; i < 8; ++i) s += q[i];
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);  // 32 elements = four lanes
            const int j = lane & 7;  // the words of prep_gemm_b_kernel
            const float bv = __shfl_sync(0xffffffffu, s, 4 * j), b1 = tf32_head(bv), b2 = bv - b1;
            if (lane < G_MIN_K) bmin[((int64_t)p[u] * kb + blk[u]) * G_MIN_K + lane] = lane < 8 ? b1 : b2;
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
    uint32_t zero;                // 0 at run time, unknown to the compiler (see the release of a weight stage in the kernel)
};

__device__ __forceinline__ __half2 h2_bits(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t bits_h2(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
// (1024 + byte b of w) in both halves: 0x64xx is 1024 + xx in fp16
__device__ __forceinline__ __half2 byte_magic2(uint32_t w, int b) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(0x64646464u), "r"(0x4040u | (uint32_t)b | ((uint32_t)b << 8)));
    return h2_bits(r);
}
__device__ __forceinline__ uint4 ldg128(const uint8_t* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ uint32_t w4(const uint4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

// ------------------------------------------------------------------------------------------------
// The unpack formats.  An unpack thread owns (tile row, K half h): elements 128 h .. 128 h + 127 of every 256-block,
// i.e. slabs 2h and 2h + 1 of 64 elements, handed over as one pair.  (Splitting a row's bytes between two threads inside
// every slab instead made both decode the same scales.)  A slab is 32 TMEM columns of two elements each; element k of
// the slab belongs to column k / 2, inside a group of four in the order (0, 2), (1, 3).
//
// Q4_K, GGUF layout (144-byte blocks: d, dmin, 12 scale bytes, 128 nibble bytes): bytes 32 s .. 32 s + 31 of the nibbles
// are slab s, low nibbles k = 0..31, high nibbles k = 32..63.
// ------------------------------------------------------------------------------------------------
struct GemmQ4K {
    static constexpr bool EXACT_GATE = false;
    static constexpr bool HAS_MIN = true;
    static constexpr int A_COLS = 32, A_PARTS = 1, A_PAIRS = 4;  // 8 slabs of 32 columns: two blocks in flight
    static constexpr int B_PARTS = 1;
    static constexpr bool STAGE_W = true;      // raw blocks of the tile pass through shared memory
    static constexpr bool HALF_TILES = false;  // ... as rows of GGUF blocks (tensor-map boxes)
    static constexpr int W_ROW_BYTES = Q4K_BYTES;
    static constexpr int W_STAGES_WIDE = 3;    // staged blocks that fit beside 128-wide activation stages
    struct Row {};
    struct Pre {
        uint4 hdr, q[4];
    };
    __device__ static __forceinline__ void load(Pre&, const Row&, int, int) {}
    __device__ static __forceinline__ Row row(const uint8_t*, int, int) { return Row{}; }
    // this thread's pieces of the staged row (rows are 36 words apart: the eight lanes of a 16-byte load phase cover all
    // 32 banks once)
    __device__ static __forceinline__ void load_staged(Pre& pr, uint32_t row_addr, int h) {
        pr.hdr = lds128_o<0>(row_addr);
        const uint32_t rb = row_addr + 64 * h;
        pr.q[0] = lds128_o<16>(rb);
        pr.q[1] = lds128_o<32>(rb);
        pr.q[2] = lds128_o<48>(rb);
        pr.q[3] = lds128_o<64>(rb);
    }
    // one word of every vector load_staged fetched: a value that exists only when all of them have arrived
    __device__ static __forceinline__ uint32_t staged_words(const Pre& pr) {
        return pr.hdr.x | pr.q[0].x | pr.q[1].x | pr.q[2].x | pr.q[3].x;
    }
    // d (low half) and dmin (high half) of the block, fp16 bits
    __device__ static __forceinline__ uint32_t hdr_of(const Pre& pr) { return pr.hdr.x; }
    struct Ctx {
        uint32_t sc, mn;  // 6-bit scales / mins of this half's sub-blocks 4h .. 4h + 3 as bytes (utils.rs:50-60)
    };
    __device__ static __forceinline__ void begin(const Pre& pr, Ctx& c, int h) {
        const uint32_t s0 = pr.hdr.y, s1 = pr.hdr.z, s2 = pr.hdr.w;
        if (h == 0) {
            c.sc = s0 & 0x3f3f3f3fu;
            c.mn = s1 & 0x3f3f3f3fu;
        } else {
            c.sc = (s2 & 0x0f0f0f0fu) | (((s0 >> 6) & 0x03030303u) << 4);
            c.mn = ((s2 >> 4) & 0x0f0f0f0fu) | (((s1 >> 6) & 0x03030303u) << 4);
        }
        if ((pr.hdr.x & 0x7fffu) == 0) c.sc = 0;  // d = 0: the block is its min term alone (see scale_of)
    }
    // The epilogue multiplies the block's accumulator by d; a block with d = 0 (and no main sum, above) is
    // scaled by dmin instead so that its min term survives, or by 1 if both are zero.
    __device__ static __forceinline__ float scale_of(uint32_t hdr) {
        const uint32_t hb = (hdr & 0x7fffu) ? (hdr & 0xffffu) : (((hdr >> 16) & 0x7fffu) ? (hdr >> 16) : 0x3c00u);
        return half_bits_to_float((uint16_t)hb);
    }
    // slab s of this half = sub-blocks 2s (low nibbles) and 2s + 1 (high nibbles) of the half.  0x6400 | n is 1024 + n
    // and fma(1024 + n, sc, -1024 sc) rounds the exact n * sc once; 0x6400 | (n << 4) is 1024 + 16 n and
    // fma(1024 + 16 n, sc / 16, -64 sc) does the same for a nibble left in the high half of its byte.
    __device__ static __forceinline__ void emit(int s, const Pre& pr, const Ctx& c, uint32_t ta) {
        const __half2 k1024 = __float2half2_rn(1024.f);
        const __half2 scl = __hsub2(byte_magic2(c.sc, 2 * s), k1024);
        const __half2 sch = __hsub2(byte_magic2(c.sc, 2 * s + 1), k1024);
        const __half2 offl = __hmul2(scl, __float2half2_rn(-1024.f));
        const __half2 sch16 = __hmul2(sch, __float2half2_rn(0.0625f)), offh = __hmul2(sch, __float2half2_rn(-64.f));
        uint32_t o[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t x = w4(pr.q[2 * s + (i >> 2)], i & 3), y = x >> 8;  // bytes (0, 2) and (1, 3) of the four
            o[2 * i] = bits_h2(__hfma2(h2_bits((x & 0x000F000Fu) | 0x64006400u), scl, offl));
            o[2 * i + 1] = bits_h2(__hfma2(h2_bits((y & 0x000F000Fu) | 0x64006400u), scl, offl));
            o[16 + 2 * i] = bits_h2(__hfma2(h2_bits((x & 0x00F000F0u) | 0x64006400u), sch16, offh));
            o[16 + 2 * i + 1] = bits_h2(__hfma2(h2_bits((y & 0x00F000F0u) | 0x64006400u), sch16, offh));
        }
        tmem_st32(ta, o);
    }
    // weight side of the min term (see prep_gemm_b_kernel): -rho_j = -dmin m_j / d split into tf32 terms.  One
    // row is 16 floats [r1 (8) | r2 (8)]; half h writes its four values of each.  2^23 + m as float
    // bits is 0x4B000000 | m.
    __device__ static __forceinline__ void emit_min(const Pre& pr, const Ctx& c, uint8_t* arow, int h, int sw) {
        const float ratio = -__fdividef(half_bits_to_float((uint16_t)(pr.hdr.x >> 16)), scale_of(pr.hdr.x));
        uint32_t r1[4], r2[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float mf = __uint_as_float(__byte_perm(c.mn, 0x4B000000u, 0x7650 | j)) - 8388608.f;
            const float a = __fmul_rn(ratio, mf), a1 = tf32_head(a);
            r1[j] = __float_as_uint(a1);
            r2[j] = __float_as_uint(tf32_head(__fsub_rn(a, a1)));
        }
        *reinterpret_cast<uint4*>(arow + ((h ^ sw) << 4)) = make_uint4(r1[0], r1[1], r1[2], r1[3]);
        *reinterpret_cast<uint4*>(arow + (((2 + h) ^ sw) << 4)) = make_uint4(r2[0], r2[1], r2[2], r2[3]);
    }
};

// ------------------------------------------------------------------------------------------------
// Q6_K, repacked layout (expert_direct.cu: per 8 rows x 256 elements, 1680 bytes: low nibbles 2 x 512,
// high bit pairs 512, 128 scales, 8 d; a row's four 16-byte chunks t of a 512-byte region lie in chunk_pos order).  Word
// cw of chunk t of half h holds elements k0 = 16 cw + 4 t .. + 3 of the half's two slabs (low nibbles: first slab, high
// nibbles: second), words 2h, 2h + 1 of chunk t of the third region their high bit pairs.
// The quant is placed at mantissa bits 4..9 (0x6400 | q << 4 = 1024 + 16 q); minus 1536 leaves
// 16 (q - 32), times ceil(sc/2)/16 and floor(sc/2)/16 gives the two exact operand parts.
// ------------------------------------------------------------------------------------------------
struct GemmQ6K {
    static constexpr bool EXACT_GATE = false;
    static constexpr bool HAS_MIN = false;
    static constexpr int A_COLS = 64, A_PARTS = 2, A_PAIRS = 2;  // 4 slabs of 64 columns (two operand parts each)
    static constexpr int B_PARTS = 1;
    static constexpr bool STAGE_W = false;
    static constexpr bool HALF_TILES = false;
    static constexpr int W_ROW_BYTES = 0;
    static constexpr int W_STAGES_WIDE = 1;
    struct Row {
        const uint8_t* p;  // half-tile block 0 of the row's group of 8
        int g;
    };
    __device__ static __forceinline__ Row row(const uint8_t* w, int n, int kb) {
        return Row{w + (size_t)(n >> 3) * kb * Q6K_HTB_BYTES, n & 7};
    }
    struct Pre {
        uint4 ql[4];
        uint2 qh[4], sc;
        uint32_t d;  // fp16 bits
    };
    __device__ static __forceinline__ uint32_t hdr_of(const Pre& pr) { return pr.d; }
    __device__ static __forceinline__ void load_staged(Pre&, uint32_t, int) {}
    __device__ static __forceinline__ uint32_t staged_words(const Pre&) { return 0u; }
    __device__ static __forceinline__ void load(Pre& pr, const Row& r, int blk, int h) {
        const uint8_t* b = r.p + (size_t)blk * Q6K_HTB_BYTES;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int c = 16 * chunk_pos(r.g, t);
            pr.ql[t] = ldg128(b + 512 * h + c);
            pr.qh[t] = __ldg(reinterpret_cast<const uint2*>(b + 1024 + c + 8 * h));
        }
        pr.sc = __ldg(reinterpret_cast<const uint2*>(b + 1536 + 16 * r.g + 8 * h));
        pr.d = (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(b + 1664 + 2 * r.g));
    }
    struct Ctx {
        uint32_t xc[2], xh[2];  // per scale byte: ceil(sc/2) + 64 and floor(sc/2) + 64
    };
    __device__ static __forceinline__ void begin(const Pre& pr, Ctx& c, int) {
        const uint32_t w[2] = {pr.sc.x, pr.sc.y};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t x = w[i] ^ 0x80808080u;  // sc + 128 per byte
            c.xh[i] = (x >> 1) & 0x7f7f7f7fu;
            c.xc[i] = c.xh[i] + (x & 0x01010101u);
        }
    }
    __device__ static __forceinline__ void emit(int s, const Pre& pr, const Ctx& c, uint32_t ta) {
        const __half2 k16th = __float2half2_rn(0.0625f), km68 = __float2half2_rn(-68.f), km1536 = __float2half2_rn(-1536.f);
#pragma unroll
        for (int cw = 0; cw < 4; ++cw) {
            // (1024 + x) / 16 - 68 = (x - 64) / 16: the half scale over 16; c = -1536 m, so that
            // fma(1024 + 16 q, m, c) = (q - 32) * (half scale), an integer of at most 2048: exact
            const __half2 m1 = __hfma2(byte_magic2(c.xc[s], cw), k16th, km68);
            const __half2 m2 = __hfma2(byte_magic2(c.xh[s], cw), k16th, km68);
            const __half2 c1 = __hmul2(m1, km1536), c2 = __hmul2(m2, km1536);
            const int bq = 2 * ((cw >> 1) + 2 * s);  // bit position of this quarter's pair in the qh byte
            uint32_t o1[8], o2[8];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const uint32_t qlw = w4(pr.ql[t], cw), qhw = (cw & 1) ? pr.qh[t].y : pr.qh[t].x;
                const uint32_t a02 = s ? qlw : (qlw << 4), a13 = s ? (qlw >> 8) : (qlw >> 4);
                const uint32_t b02 = qhw << (8 - bq), b13 = qhw >> bq;
                const __half2 v02 = h2_bits(((a02 & 0x00F000F0u) | 0x64006400u) | (b02 & 0x03000300u));
                const __half2 v13 = h2_bits(((a13 & 0x00F000F0u) | 0x64006400u) | (b13 & 0x03000300u));
                o1[2 * t] = bits_h2(__hfma2(v02, m1, c1));
                o1[2 * t + 1] = bits_h2(__hfma2(v13, m1, c1));
                o2[2 * t] = bits_h2(__hfma2(v02, m2, c2));
                o2[2 * t + 1] = bits_h2(__hfma2(v13, m2, c2));
            }
            tmem_st8(ta + 8 * cw, o1);
            tmem_st8(ta + 32 + 8 * cw, o2);
        }
    }
    __device__ static __forceinline__ void emit_min(const Pre&, const Ctx&, uint8_t*, int, int) {}
    __device__ static __forceinline__ float scale_of(uint32_t hdr) { return half_bits_to_float((uint16_t)hdr); }
};

// Matrices without copies, repacked on their way (candle_moe_api.cu).  The forms that take such a layer otherwise gate with expf and
// an exact division (silu_f); the hidden rows are quantized to int8 again, where a difference in the last bit can become a
// step, so this one does the same: largest relative error of a gate 2.4e-7 (8.1e-7 with __expf and an approximate division), of
// the hidden rows against 64-bit arithmetic 0.98-1.01e-7 (streaming form 0.98-1.01e-7, row-per-warp form 1.2-1.5e-7, without
// the exact gate 1.01-1.05e-7).  It costs 3-6 % of a layer of small matrices (8 experts of 1536 x 2560, 400 rows: 457 -> 470 us).
struct GemmQ6KOnTheWay : GemmQ6K {
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
    static constexpr bool EXACT_GATE = false;
    static constexpr bool HAS_MIN = false;
    static constexpr int A_COLS = 32, A_PARTS = 1, A_PAIRS = 4;
    static constexpr int B_PARTS = 1;
    static constexpr bool STAGE_W = true;
    static constexpr bool HALF_TILES = true;  // staged as half-tile blocks, one bulk copy per 8 rows
    static constexpr int W_ROW_BYTES = 2 * Q80_HTB_BYTES / 8;
    static constexpr int W_STAGES_WIDE = 2;  // staged blocks beside 128-wide activation stages
    struct Row {};
    __device__ static __forceinline__ Row row(const uint8_t*, int, int) { return Row{}; }
    struct Pre {
        uint2 sc;       // 4 f16 scales
        uint4 q[2][4];  // per slab: chunks t = 0..3
    };
    __device__ static __forceinline__ void load(Pre&, const Row&, int, int) {}
    // ht_addr: the row's half-tile (both blocks) in the stage, g: its row inside
    __device__ static __forceinline__ void load_half_tile(Pre& pr, uint32_t ht_addr, int g, int h) {
        const uint32_t b = ht_addr + h * Q80_HTB_BYTES;
        pr.sc = lds64_o<1024>(b + 8 * g);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint32_t c = b + 16 * chunk_pos(g, t);
            pr.q[0][t] = lds128_o<0>(c);
            pr.q[1][t] = lds128_o<512>(c);
        }
    }
    __device__ static __forceinline__ void load_staged(Pre&, uint32_t, int) {}
    __device__ static __forceinline__ uint32_t staged_words(const Pre& pr) {
        uint32_t v = pr.sc.x;
#pragma unroll
        for (int t = 0; t < 4; ++t) v |= pr.q[0][t].x | pr.q[1][t].x;
        return v;
    }
    __device__ static __forceinline__ uint32_t hdr_of(const Pre&) { return 0u; }
    struct Ctx {};
    __device__ static __forceinline__ void begin(const Pre&, Ctx&, int) {}
    __device__ static __forceinline__ float scale_of(uint32_t) { return 1.0f; }  // the scales are inside the operands
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
    // scales of the two 32-element blocks of slab s
    __device__ static __forceinline__ __half2 scales(const Pre& pr, int s) { return h2_bits(s ? pr.sc.y : pr.sc.x); }
    __device__ static __forceinline__ void emit(int s, const Pre& pr, const Ctx&, uint32_t ta) {
        const __half2 d2 = scales(pr, s);
        uint32_t o[32];
#pragma unroll
        for (int cw = 0; cw < 4; ++cw) {
            const __half2 d = cw < 2 ? __low2half2(d2) : __high2half2(d2);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                __half2 e, f;
                split4(w4(pr.q[s][t], cw), e, f);
                o[8 * cw + 2 * t] = bits_h2(__hmul2(e, d));
                o[8 * cw + 2 * t + 1] = bits_h2(__hmul2(f, d));
            }
        }
        tmem_st32(ta, o);
    }
    __device__ static __forceinline__ void emit_min(const Pre&, const Ctx&, uint8_t*, int, int) {}
};

// ------------------------------------------------------------------------------------------------
// Q8_0 with EXACT operands, for the gate_up product (whose f32 result is re-quantized to int8 and therefore has to
// match the reference to f32 rounding, not to fp16 rounding).  d * q has up to 19 significant bits: it is carried as
// two fp16 numbers, the rounded product and its exact residual (one more fused multiply-add), on both sides:
//   weights      4096 d_w q  = A0 + A1      (the power of two keeps the residuals out of the fp16 subnormals;
//   activations    64 d_a q  = B0 + B1       both come off again in the epilogue's scale)
// and the tensor core accumulates A0 B0 + A1 B0 + A0 B1 in f32 (A1 B1 is below 2^-22 of a term).  Three MMAs per
// K step; the activation operand is twice as large, so its two shared-memory stages hold half a block each (see the
// kernel).
// ------------------------------------------------------------------------------------------------
struct GemmQ80X : GemmQ80 {
    static constexpr int A_COLS = 64, A_PARTS = 2, A_PAIRS = 2;
    static constexpr int B_PARTS = 2;
    static constexpr int W_STAGES_WIDE = 2;
    __device__ static __forceinline__ float scale_of(uint32_t) { return 1.0f / 4096.0f; }
    __device__ static __forceinline__ void emit(int s, const Pre& pr, const Ctx&, uint32_t ta) {
        const __half2 d2 = __hmul2(scales(pr, s), __float2half2_rn(4096.f));  // exact (a power of two)
#pragma unroll
        for (int c2 = 0; c2 < 2; ++c2) {  // one 32-element block of the slab
            const __half2 d = c2 ? __high2half2(d2) : __low2half2(d2);
            uint32_t p0[16], p1[16];
#pragma unroll
            for (int cw = 0; cw < 2; ++cw)
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    __half2 e, f;
                    split4(w4(pr.q[s][t], 2 * c2 + cw), e, f);
                    const __half2 re = __hmul2(e, d), rf = __hmul2(f, d);
                    p0[8 * cw + 2 * t] = bits_h2(re);
                    p0[8 * cw + 2 * t + 1] = bits_h2(rf);
                    p1[8 * cw + 2 * t] = bits_h2(__hfma2(e, d, __hneg2(re)));  // exact: the residual of a 19-bit product has at most 8 bits
                    p1[8 * cw + 2 * t + 1] = bits_h2(__hfma2(f, d, __hneg2(rf)));
                }
            tmem_st16(ta + 16 * c2, p0);
            tmem_st16(ta + 32 + 16 * c2, p1);
        }
    }
};

// one activation stage: a 256-wide block (four slabs) or the half of one with two operand parts, + the min-term box
template <class F, int TN>
__host__ __device__ constexpr int b_stage_bytes() {
    return 4 * (TN * G_SLAB_K * 2) + (F::HAS_MIN ? TN * G_MIN_K * 4 : 0);
}
// raw weight blocks staged per CTA (see the kernel): what fits beside the activation stages
template <class F, int TN>
__host__ __device__ constexpr int w_stages() {
    return !F::STAGE_W ? 1 : (TN <= 64 ? (F::HALF_TILES ? 4 : 6) : F::W_STAGES_WIDE);
}

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
    __device__ __forceinline__ bool next(TileCoord& tc) {
        uint32_t per_mt = n_tiles * ksplit;
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
__global__ void __launch_bounds__(G_THREADS, 1)
expert_gemm_kernel(const __grid_constant__ GemmParams P, const __grid_constant__ CUtensorMap map_b,
                   const __grid_constant__ CUtensorMap map_bs) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_a[4], empty_a[4], full_b[G_B_STAGES], empty_b[G_B_STAGES];  // A: per pair of slabs
    __shared__ uint64_t tmem_full[2], epi_done[2], full_w[G_W_STAGES_MAX], empty_w[G_W_STAGES_MAX];
    __shared__ uint32_t s_offs[CANDLE_MOE_MAX_EXPERTS + 1];
    constexpr int CH = TN / 2;            // columns (positions) per epilogue warp: two warps share a TMEM lane quarter
    constexpr int B_TILE = TN * G_SLAB_K * 2;  // one [TN x 64] fp16 activation slab
    __shared__ __align__(16) float s_d8[G_EPI_WARPS][2][CH];  // per epilogue warp: activation scales of its columns
    __shared__ float s_dw[8][G_TILE_M];  // per block (ring of 8) and tile row: the weight scale the drain multiplies by
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    // the warp index through a shuffle: the compiler then knows that it is warp-uniform and keeps role
    // dispatch, loop counters and MMA / TMA operands in uniform registers
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    pdl_trigger();
    pdl_wait();
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    // One activation stage holds a whole 256-wide block (four slabs, + the min-term box for Q4_K).  With two operand
    // parts (exact Q8_0) a whole block would be twice that, so there the two stages are the two HALVES of a block
    // -- stage pr = the slabs of pair pr: [part 0: slab 2 pr, 2 pr + 1 | part 1: slab 2 pr, 2 pr + 1] -- each
    // refilled for the next block as soon as its own pair's MMAs are done; the same shared memory then takes
    // 128-wide position tiles.
    constexpr bool B_HALF = F::B_PARTS == 2;
    constexpr int G_STAGE_BYTES = b_stage_bytes<F, TN>();
    uint8_t* smem_min_a = smem + G_B_STAGES * G_STAGE_BYTES;  // Q4_K: 2 slots of the min operand (weights side)
    // staged raw blocks of the tile rows: a ring of WS blocks, so that the copy of block b + WS - 1 is in flight while
    // block b is unpacked.  (Q4_K, 128-wide position tiles: one block and requests into L2 ahead of it, with a min-term box
    // of 32 floats per row, against three blocks beside 16 floats: 2048 rows 2470 -> 2422 us, 8 small experts at 257
    // rows 78.0 -> 75.0, [4096, 4096] at 777 rows 53.9 -> 52.9.)
    constexpr int WS = w_stages<F, TN>();
    constexpr int W_STAGE_BYTES = G_TILE_M * F::W_ROW_BYTES;
    uint8_t* smem_w = smem_min_a + (F::HAS_MIN ? 2 : 0) * G_MIN_A_BYTES;
    for (int i = threadIdx.x; i <= P.E; i += G_THREADS) s_offs[i] = P.offsets[i];
    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < 4; ++s) {
            mbar_init(&full_a[s], G_DQ_WARPS / 2);
            mbar_init(&empty_a[s], 1);
        }
        for (int s = 0; s < G_B_STAGES; ++s) {
            mbar_init(&full_b[s], 1);
            mbar_init(&empty_b[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tmem_full[b], 1);
            mbar_init(&epi_done[b], G_EPI_WARPS);
        }
        for (int s = 0; s < G_W_STAGES_MAX; ++s) {
            mbar_init(&full_w[s], 1);
            mbar_init(&empty_w[s], G_DQ_WARPS);
        }
        fence_barrier_init();
    }
    if (warp == G_WARP_TMA) tmem_alloc(&s_tmem_base, G_TMEM_COLS);
    tc5_fence_before_sync();
    __syncthreads();
    tc5_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, s_tmem_base, 0);
    volatile int* abort_flag = &s_abort;
    TileWalk<TN> walk(s_offs, P.E, P.m_tiles, P.ksplit, P.kb);
    constexpr uint32_t IDESC = umma_idesc_f16(G_TILE_M, TN), IDESC_TF32 = umma_idesc_tf32(G_TILE_M, TN);

    // Register budget: launched with 96 per thread; the TMA/MMA warpgroup hands 64 per thread back to the CTA's
    // pool and the two epilogue warpgroups take 32 more each, so the total stays what the launch allocated (a
    // request beyond the pool would wait forever).
    if (warp >= G_WARP_DQ0 + G_DQ_WARPS) reg_dealloc<G_REGS_MISC>();  // the whole last warpgroup (two idle warps, TMA, MMA)
    if (warp < G_WARP_DQ0) {
        reg_alloc<G_REGS_EPI>();
        // ===================== epilogue =====================
        const int quarter = warp & 3, colhalf = (warp - G_WARP_EPI0) >> 2, ew = warp - G_WARP_EPI0;
        const int r = 32 * quarter + lane;  // tile row = TMEM lane
        const uint32_t ta_lane = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(colhalf * CH);
        uint32_t ab = 0;
        TileCoord tc, tcn;
        bool have = walk.next(tc);
        if (have) {
            const float* dp = P.d8t + (size_t)tc.kb0 * P.P_pad + tc.p0 + colhalf * CH;
            for (int i = lane; i < CH; i += 32) s_d8[ew][0][i] = dp[i];
            __syncwarp();
        }
        while (have) {
            const bool have_n = walk.next(tcn);
            // the accumulators are kept as pairs of columns: one packed fused multiply-add per pair and block
            uint64_t acc2[CH / 2];
#pragma unroll
            for (int i = 0; i < CH / 2; ++i) acc2[i] = 0ull;
            // Narrow tiles have registers to add the blocks in runs of RUN, the runs on their own ([32000, 4096] Q6_K at 32
            // rows, relative error against 64-bit arithmetic: 7.8e-8 in one run of 16, 6.5e-8 in two; 48.8 -> 49.6 us)
            constexpr bool RUNS = TN <= 64;
            uint64_t run2[RUNS ? CH / 2 : 1];
            if (RUNS) {
#pragma unroll
                for (int i = 0; i < CH / 2; ++i) run2[RUNS ? i : 0] = 0ull;
            }
            for (int blk = tc.kb0; blk < tc.kb1;) {
              const int stop = RUNS ? min(blk + G_RUN, tc.kb1) : tc.kb1;
              for (; blk < stop; ++blk, ++ab) {
                const int buf = ab & 1;
                // scales of the next block (maybe of the next tile): in flight while this block is drained
                float d8_n0 = 0.f, d8_n1 = 0.f;
                const float* dp = nullptr;
                if (blk + 1 < tc.kb1)
                    dp = P.d8t + (size_t)(blk + 1) * P.P_pad + tc.p0 + colhalf * CH + lane;
                else if (have_n)
                    dp = P.d8t + (size_t)tcn.kb0 * P.P_pad + tcn.p0 + colhalf * CH + lane;
                const bool pre = dp != nullptr;
                if (pre) {
                    if (lane < CH) d8_n0 = dp[0];
                    if (CH > 32) d8_n1 = dp[32];
                }
                mbar_wait(&tmem_full[buf], (ab >> 1) & 1, abort_flag);
                tc5_fence_after_sync();
                const float dw = s_dw[ab & 7][r];  // left by the unpack warps when they produced this block
                const uint64_t dw2 = f32x2_pack(dw, dw);
                const uint32_t t_main = ta_lane + (uint32_t)(G_TM_MAIN + buf * TN);
                const uint32_t d8_addr = smem_u32(&s_d8[ew][buf][0]);
                // Four steps of 16 columns; the load of step i+1 is in flight while step i is scaled into
                // the register accumulators: acc += (d8[col] * dw[row]) * v.
                constexpr int NS = CH / 16;  // steps of 16 columns
                uint32_t stg[2][16];
                tmem_ld16(t_main, stg[0]);
                tmem_ld_wait();
                static_for<NS>([&](auto Cc) {
                    constexpr int c = decltype(Cc)::value;
                    if (c + 1 < NS) tmem_ld16(t_main + 16 * (c + 1), stg[(c + 1) & 1]);
                    static_for<4>([&](auto Qc) {
                        constexpr int q = decltype(Qc)::value;
                        const uint4 dv = lds128_o<64 * c + 16 * q>(d8_addr);  // base + constant: no address arithmetic
                        // per column pair: the two scale products in one packed multiply, the two accumulations in one
                        // packed fused multiply-add (each half is the IEEE fma of the scalar form)
                        acc2[8 * c + 2 * q] = f32x2_fma(f32x2_mul(dw2, f32x2_pack_bits(dv.x, dv.y)),
                                                        f32x2_pack_bits(stg[c & 1][4 * q], stg[c & 1][4 * q + 1]), acc2[8 * c + 2 * q]);
                        acc2[8 * c + 2 * q + 1] = f32x2_fma(f32x2_mul(dw2, f32x2_pack_bits(dv.z, dv.w)),
                                                            f32x2_pack_bits(stg[c & 1][4 * q + 2], stg[c & 1][4 * q + 3]),
                                                            acc2[8 * c + 2 * q + 1]);
                    });
                    if (c + 1 < NS) tmem_ld_wait();
                    if (c == (NS >= 2 ? NS - 2 : 0)) {  // every column of this thread has been read: the buffer may be overwritten
                        tc5_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&epi_done[buf]);
                    }
                });
                if (pre) {
                    if (lane < CH) s_d8[ew][buf ^ 1][lane] = d8_n0;
                    if (CH > 32) s_d8[ew][buf ^ 1][lane + 32] = d8_n1;
                }
                __syncwarp();
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
#pragma unroll
                for (int c = 0; c < CH / 2; ++c) {
                    const float recv = __shfl_xor_sync(0xffffffffu, up ? acc[c] : acc[c + CH / 2], 8);
                    const float gv = up ? recv : acc[c], uv = up ? acc[c + CH / 2] : recv;
                    const uint32_t p = pc0 + c + (up ? CH / 2 : 0);
                    if (p < tc.p_end) out_k[(size_t)p * P.N + n] = (F::EXACT_GATE ? silu_f(gv) : __fdividef(gv, 1.0f + __expf(-gv))) * uv;
                }
            } else {
#pragma unroll
                for (int c = 0; c < CH; ++c)
                    if (pc0 + c < tc.p_end) out_k[(size_t)(pc0 + c) * P.N + n] = acc[c];
            }
            tc = tcn;
            have = have_n;
        }
    } else if (warp < G_WARP_DQ0 + G_DQ_WARPS) {
        // ===================== weight unpack -> fp16 operand in tensor memory =====================
        const int quarter = warp & 3, h = (warp - G_WARP_DQ0) >> 2;
        const int r = 32 * quarter + lane;
        const uint32_t ta_lane = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)G_TM_A;
        const uint32_t min_row_off = (uint32_t)(r * G_MIN_K * 4);
        uint32_t ab = 0;
        TileCoord tc, tcn;
        bool have = walk.next(tc);
        typename F::Row rowc{}, rown{};
        typename F::Pre cur, nxt;
        // where tile row r lies in a stage: rows (gate_up: the W1 rows first, then the W3 rows) or half-tiles in tile order
        const uint32_t w_row = smem_u32(smem_w) +
                               (F::HALF_TILES ? (uint32_t)((r >> 3) * 8 * F::W_ROW_BYTES)
                                : GATE_UP ? (uint32_t)((((r >> 3) & 1) * (G_TILE_M / 2) + (r >> 4) * 8 + (r & 7)) * F::W_ROW_BYTES)
                                          : (uint32_t)(r * F::W_ROW_BYTES));
        const bool is_w3 = GATE_UP && ((r >> 3) & 1);
        if (have && !F::STAGE_W) {
            rowc = F::row(is_w3 ? P.wb.p[tc.e] : P.wa.p[tc.e], weight_row<GATE_UP>(tc.mt, r), P.kb);
            F::load(cur, rowc, tc.kb0, h);
            nxt = cur;
        }
        while (have) {
            const bool have_n = walk.next(tcn);
            if (have_n && !F::STAGE_W)
                rown = F::row(is_w3 ? P.wb.p[tcn.e] : P.wa.p[tcn.e], weight_row<GATE_UP>(tcn.mt, r), P.kb);
            for (int blk = tc.kb0; blk < tc.kb1; ++blk, ++ab) {
                if (F::STAGE_W) {
                    // this block's raw bytes were copied to shared memory by the loader warp
                    mbar_wait(&full_w[ab % WS], (ab / WS) & 1, abort_flag);
                    if constexpr (F::HALF_TILES)
                        F::load_half_tile(cur, w_row + (ab % WS) * W_STAGE_BYTES, r & 7, h);
                    else
                        F::load_staged(cur, w_row + (ab % WS) * W_STAGE_BYTES, h);
                } else if (blk + 1 < tc.kb1) {
                    F::load(nxt, rowc, blk + 1, h);
                } else if (have_n) {
                    F::load(nxt, rown, tcn.kb0, h);
                }
                typename F::Ctx ctx;
                F::begin(cur, ctx, h);
                if (h == 0) s_dw[ab & 7][r] = F::scale_of(F::hdr_of(cur));  // read by the epilogue when it drains this block
                // Handing the stage back to the loader as soon as the staged words have ARRIVED in registers.  The loads are
                // plain shared-memory loads, their results are not needed until the emits below, and an arrive that
                // merely follows them in program order was observed to overtake them -- the refill then landed under
                // loads still waiting behind the (long) wait for a free operand slot, and the first rows of a tile came
                // out with the next block's weights, rarely and only when the MMAs are the bottleneck.  So the barrier's
                // ADDRESS is made to depend on one word of every load of every lane (OR-reduced over the warp, masked
                // with a kernel parameter that is zero at run time): the arrive cannot be issued before those words
                // exist.  (Released after the emits instead, a ring of two stages gave a copy less than the time of one
                // block's emits: all-Q8_0 layer of 60 experts, 4096 rows, gate_up 562 -> 531 us, shared down 136 -> 125 us.)
                // A ring of three or four stages (narrow position tiles) has that time, and there the reduction costs more than it
                // gives: released after the emits (nothing reads the stage later than that, whatever the order of the
                // instructions), gate_up of the Mixtral-shaped layer at 100 rows takes 201 us, released here 212.
                if (F::STAGE_W && WS <= 2) {
                    const uint32_t dep = __reduce_or_sync(0xffffffffu, F::staged_words(cur)) & P.zero;
                    if (lane == 0) mbar_arrive(&empty_w[ab % WS + dep]);
                }
                // The pair goes to tensor memory; the ring holds A_PAIRS pairs (Q4_K: two blocks).  The barriers
                // go by (block parity, pair) -- each has ONE waiting MMA warp that sees every phase, so a parity
                // wait is never ambiguous -- while the TMEM slot is the pair index modulo the ring size: before
                // writing it, wait for the MMAs of the block that used it last.
                const uint32_t bidx = 2 * (ab & 1) + h, slot = bidx % F::A_PAIRS;
                if (ab >= F::A_PAIRS / 2) {
                    const uint32_t abp = ab - F::A_PAIRS / 2;
                    mbar_wait_relaxed(&empty_a[2 * (abp & 1) + h], (abp >> 1) & 1, abort_flag);
                }
                tc5_fence_after_sync();
                F::emit(0, cur, ctx, ta_lane + (uint32_t)(2 * slot * F::A_COLS));
                F::emit(1, cur, ctx, ta_lane + (uint32_t)((2 * slot + 1) * F::A_COLS));
                if (F::HAS_MIN) {
                    // weight side of the min term.  Its slot was last read by the min MMAs of block ab - 2, issued
                    // before the commit of that block's second pair.
                    if (h == 0 && ab >= 2) mbar_wait_relaxed(&empty_a[2 * (ab & 1) + 1], ((ab - 2) >> 1) & 1, abort_flag);
                    F::emit_min(cur, ctx, smem_min_a + (size_t)(ab & 1) * G_MIN_A_BYTES + min_row_off, h, (r >> 1) & 3);
                    fence_proxy_async_smem();
                }
                tmem_st_wait();
                tc5_fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&full_a[bidx]);
                    if (F::STAGE_W && WS > 2) mbar_arrive(&empty_w[ab % WS]);
                }
                if (!F::STAGE_W) cur = nxt;
            }
            tc = tcn;
            rowc = rown;
            have = have_n;
        }
    } else if (warp == G_WARP_LOAD) {
        // ===================== weight loader: raw blocks of the tile rows -> shared memory =====================
        // One TMA box per matrix and block: [64 or 128 rows x 144 bytes] of the byte matrix [n_rows, row_bytes]
        // (gate_up: the W1 rows, then the W3 rows; a TMA destination must be 128-byte aligned, so the halves cannot
        // be skewed against each other and neighbouring lanes, which alternate between them, share banks two by
        // two).
        if constexpr (F::HALF_TILES) {
            // half-tile blocks of the repacked layout: one bulk copy per 8 tile rows, lane i < 16 copies half-tile i
            // (gate_up: W1 and W3 half-tiles alternate).  No requests into L2 ahead: the CTAs of a weight tile's position tiles
            // run together and share the lines, and sixteen more instructions per block held the copies up (all-Q8_0 layer of
            // 60 experts, 4096 rows, down 236 -> 218 us, shared down 127 -> 106 us without them).
            uint32_t ab = 0;
            TileCoord tc;
            constexpr int HT_BYTES = 8 * F::W_ROW_BYTES;  // a half-tile over one 256-block
            const bool active = lane < G_TILE_M / 8, is_w3 = GATE_UP && (lane & 1);
            while (walk.next(tc)) {
                const int ht = GATE_UP ? tc.mt * 8 + (lane >> 1) : tc.mt * 16 + lane;
                const uint8_t* src = active ? (is_w3 ? P.wb.p[tc.e] : P.wa.p[tc.e]) + (size_t)ht * P.kb * HT_BYTES : nullptr;
                for (int blk = tc.kb0; blk < tc.kb1; ++blk, ++ab) {
                    const uint32_t ws = ab % WS;
                    if (ab >= (uint32_t)WS) mbar_wait(&empty_w[ws], ((ab / WS) - 1) & 1, abort_flag);
                    if (lane == 0) mbar_expect_tx(&full_w[ws], G_TILE_M * F::W_ROW_BYTES);
                    __syncwarp();
                    if (active && !*abort_flag)
                        bulk_g2s(smem_w + ws * W_STAGE_BYTES + lane * HT_BYTES, src + (size_t)blk * HT_BYTES, HT_BYTES, &full_w[ws]);
                    __syncwarp();
                }
            }
        } else if constexpr (F::STAGE_W) {
            uint32_t ab = 0;
            int fenced = -1;
            TileCoord tc;
            constexpr int HALF = G_TILE_M / 2 * F::W_ROW_BYTES;  // 9216
            while (walk.next(tc)) {
                const CUtensorMap* m0 = P.wmaps + 2 * tc.e;
                // the maps were written by a kernel earlier on the stream: fence an expert's once, before their first use by this
                // warp (every lane fences: any may be elected)
                if (fenced != tc.e) {
                    fenced = tc.e;
                    tensormap_fence_acquire(m0);
                    if (GATE_UP) tensormap_fence_acquire(m0 + 1);
                }
                const int y0 = GATE_UP ? tc.mt * 64 : tc.mt * 128;
                for (int blk = tc.kb0; blk < tc.kb1; ++blk, ++ab) {
                    const uint32_t ws = ab % WS;
                    if (ab >= (uint32_t)WS) mbar_wait(&empty_w[ws], ((ab / WS) - 1) & 1, abort_flag);
                    if (elect_one()) {
                        uint8_t* dst = smem_w + ws * W_STAGE_BYTES;
                        mbar_expect_tx(&full_w[ws], G_TILE_M * F::W_ROW_BYTES);
                        if (GATE_UP) {
                            tma_load_2d(dst, m0, blk * F::W_ROW_BYTES, y0, &full_w[ws]);
                            tma_load_2d(dst + HALF, m0 + 1, blk * F::W_ROW_BYTES, y0, &full_w[ws]);
                        } else {
                            tma_load_2d(dst, m0, blk * F::W_ROW_BYTES, y0, &full_w[ws]);
                            tma_load_2d(dst + HALF, m0, blk * F::W_ROW_BYTES, y0 + 64, &full_w[ws]);
                        }
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp == G_WARP_TMA) {
        // ===================== TMA: activation operand =====================
        // the whole warp walks the loop (uniform control flow and addresses), one elected lane issues
        uint32_t ab = 0;
        TileCoord tc;
        while (walk.next(tc)) {
            for (int blk = tc.kb0; blk < tc.kb1; ++blk, ++ab) {
                if constexpr (B_HALF) {
                    // stage pr of every block: free once the MMAs of pair pr of the block before are done
#pragma unroll
                    for (int pr = 0; pr < 2; ++pr) {
                        if (ab >= 1) mbar_wait_relaxed(&empty_b[pr], (ab - 1) & 1, abort_flag);
                        uint8_t* dst = smem + (size_t)pr * G_STAGE_BYTES;
                        if (elect_one()) {
                            mbar_expect_tx(&full_b[pr], G_STAGE_BYTES);
#pragma unroll
                            for (int j = 0; j < 4; ++j)  // a row holds [256 of part 0 | 256 of part 1] per block
                                tma_load_2d(dst + j * B_TILE, &map_b, blk * 512 + (j >> 1) * 256 + (2 * pr + (j & 1)) * 64, (int)tc.p0,
                                            &full_b[pr]);
                        }
                        __syncwarp();
                    }
                    continue;
                }
                // one stage = the whole 256-wide block: four slabs (+ the activation side of the min term), one barrier
                const int st = ab & 1;
                if (ab >= 2) mbar_wait_relaxed(&empty_b[st], ((ab >> 1) & 1) ^ 1, abort_flag);
                uint8_t* dst = smem + (size_t)st * G_STAGE_BYTES;
                if (elect_one()) {
                    mbar_expect_tx(&full_b[st], G_STAGE_BYTES);
#pragma unroll
                    for (int s4 = 0; s4 < 4; ++s4)
                        tma_load_2d(dst + s4 * B_TILE, &map_b, blk * 256 + s4 * 64, (int)tc.p0, &full_b[st]);
                    if (F::HAS_MIN) tma_load_2d(dst + 4 * B_TILE, &map_bs, blk * G_MIN_K, (int)tc.p0, &full_b[st]);
                }
                __syncwarp();
            }
        }
    } else if (warp == G_WARP_MMA) {
        // ===================== MMA issue =====================
        // (Splitting the blocks by parity over two issuing warps was measured: no gain.)
        uint32_t ita = 0, ab = 0;
        TileCoord tc;
        const uint32_t a_base = tmem_base + (uint32_t)G_TM_A;
        const uint64_t b_desc0 = umma_desc_sw128(smem_u32(smem));
        const uint64_t ma_desc0 = umma_desc_sw64(smem_u32(smem_min_a)), mb_desc0 = umma_desc_sw64(smem_u32(smem) + 4 * B_TILE);
        bool rdy_a = false, rdy_b = false;
        while (walk.next(tc)) {
            // The last position tile of an expert is rarely full: its MMAs run N = the rows it holds, rounded up to 16
            // (an MMA's time goes with N; the columns beyond are neither computed nor stored).
            const uint32_t n_eff = min((uint32_t)TN, (tc.p_end - tc.p0 + 15u) & ~15u);
            const uint32_t idesc = (IDESC & ~(0x3Fu << 17)) | ((n_eff >> 3) << 17);
            const uint32_t idesc_tf32 = (IDESC_TF32 & ~(0x3Fu << 17)) | ((n_eff >> 3) << 17);
            for (int blk = tc.kb0; blk < tc.kb1; ++blk, ++ab) {
                const int buf = ab & 1;  // main accumulator and B stage of this block
                // the drain of block ab - 2 has released this main accumulator
                if (ab >= 2) mbar_wait(&epi_done[buf], ((ab >> 1) & 1) ^ 1, abort_flag);
                const uint32_t d_main = tmem_base + (uint32_t)(G_TM_MAIN + buf * TN);
                const uint64_t db = b_desc0 + (uint64_t)((B_HALF ? 0 : buf) * (G_STAGE_BYTES >> 4));
#pragma unroll
                for (int pr = 0; pr < 2; ++pr, ita += 2) {
                    const uint32_t bidx = 2 * (ab & 1) + pr, slot = bidx % F::A_PAIRS;  // barrier, TMEM slot (see the unpack warps)
                    if (!rdy_a) mbar_wait(&full_a[bidx], (ab >> 1) & 1, abort_flag);
                    if constexpr (B_HALF) {
                        mbar_wait(&full_b[pr], ab & 1, abort_flag);
                    } else {
                        if (pr == 0 && !rdy_b) mbar_wait(&full_b[buf], (ab >> 1) & 1, abort_flag);
                    }
                    tc5_fence_after_sync();
                    // look at this warp's next barriers now: the answers arrive while the MMAs are issued
                    rdy_a = pr == 0 ? mbar_test(&full_a[bidx + 1], (ab >> 1) & 1)                    // second pair of this block
                                    : mbar_test(&full_a[2 * ((ab + 1) & 1)], ((ab + 1) >> 1) & 1);  // first pair of the next
                    if (!B_HALF && pr == 1) rdy_b = mbar_test(&full_b[buf ^ 1], ((ab + 1) >> 1) & 1);
                    const uint32_t a_t = a_base + (uint32_t)(2 * slot * F::A_COLS);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) {  // two slabs of four K steps
                            const uint32_t a_k = a_t + (uint32_t)((k >> 2) * F::A_COLS + 8 * (k & 3));
                            // slab of this K step inside its stage: whole-block stages hold slabs 0..3, half-block
                            // stages [part 0: two slabs | part 1: two slabs] of pair pr
                            const uint64_t b_k = db + (uint64_t)((B_HALF ? pr * 4 + (k >> 2) : 2 * pr + (k >> 2)) * (B_TILE >> 4) + 2 * (k & 3));
                            umma_f16_ts(d_main, a_k, b_k, idesc, (pr | k) != 0);
                            if (F::A_PARTS == 2) umma_f16_ts(d_main, a_k + 32, b_k, idesc, true);
                            if (F::B_PARTS == 2) umma_f16_ts(d_main, a_k, b_k + (uint64_t)(2 * (B_TILE >> 4)), idesc, true);
                        }
                        if (pr == 1 && F::HAS_MIN) {
                            // the min term joins the same accumulator: three tf32 steps, last in the block
                            const uint64_t da = ma_desc0 + (uint64_t)(buf * (G_MIN_A_BYTES >> 4)), dm = mb_desc0 + (uint64_t)(buf * (G_STAGE_BYTES >> 4));
                            umma_tf32(d_main, da, dm, idesc_tf32, true);      // r1 b1
                            umma_tf32(d_main, da + 2, dm, idesc_tf32, true);  // r2 b1
                            umma_tf32(d_main, da, dm + 2, idesc_tf32, true);  // r1 b2
                        }
                        umma_commit(&empty_a[bidx]);  // the stages may be refilled once these MMAs have read them
                        if (B_HALF) umma_commit(&empty_b[pr]);
                        if (pr == 1) {
                            if (!B_HALF) umma_commit(&empty_b[buf]);
                            umma_commit(&tmem_full[buf]);
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }
    tc5_fence_before_sync();
    __syncthreads();
    // After a wait that gave up, copies and MMAs of this CTA may still be under way (the issuing warps have run through their
    // remaining blocks): give them time, some microseconds each at most, before the shared and tensor memory go
    if (s_abort)
        for (int i = 0; i < 5000; ++i) __nanosleep(1000);
    if (warp == G_WARP_TMA) {
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
    const int smem_bytes = G_B_STAGES * b_stage_bytes<F, TN>() + (F::HAS_MIN ? 2 : 0) * G_MIN_A_BYTES +
                           (F::STAGE_W ? w_stages<F, TN>() * G_TILE_M * F::W_ROW_BYTES : 0) + 1024 /* alignment slack */;
    auto kfn = expert_gemm_kernel<F, GATE_UP, TN>;
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (e != cudaSuccess) return e;
    return launch_k(kfn, dim3(g_gemm_sms), dim3(G_THREADS), (size_t)smem_bytes, st, G, map_b, map_bs);
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
                : launch_k(prep_gemm_f32_q8k_kernel, prep_grid, dim3(256), 0, st, x_f32, (int)P, (int)p_pad, K, bf16,
                           has_min ? bmin : (float*)nullptr, d8t, single_group, first);
    else
        e = q80 ? launch_k(prep_gemm_b_q80_kernel, prep_grid, dim3(256), 0, st, aq, ascale, row_of, (int)P, (int)p_pad, K_in, K,
                           q80x ? 1 : 0, bf16, d8t)
                : launch_k(prep_gemm_b_kernel, prep_grid, dim3(256), 0, st, aq, ascale, absum, row_of, (int)P, (int)p_pad, K, bf16,
                           has_min ? bmin : (float*)nullptr, d8t, first);
    if (e != cudaSuccess) return e;

    CUtensorMap map_b, map_bs;
    if (!make_map_2d(&map_b, bf16, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (uint64_t)p_pad, (uint64_t)K * parts, G_SLAB_K, tn))
        return cudaErrorNotSupported;
    if (!make_map_2d(&map_bs, bmin, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)p_pad, (uint64_t)kb * G_MIN_K, G_MIN_K, tn, CU_TENSOR_MAP_SWIZZLE_64B))
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
    G.zero = 0;
    G.split_stride = split_stride;
    e = stream_status_ptr(&G.status);
    if (e != cudaSuccess) return e;
    if (dtype == CANDLE_GGML_Q4K) {
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
        if (tn == 32) return launch_gemm_kernel<GemmQ6KOnTheWay, true, 32>(st, G, map_b, map_bs);
        if (tn == 64) return launch_gemm_kernel<GemmQ6KOnTheWay, true, 64>(st, G, map_b, map_bs);
        return launch_gemm_kernel<GemmQ6KOnTheWay, true, 128>(st, G, map_b, map_bs);
    }
    if (tn == 32)
        return gate_up ? launch_gemm_kernel<GemmQ6K, true, 32>(st, G, map_b, map_bs) : launch_gemm_kernel<GemmQ6K, false, 32>(st, G, map_b, map_bs);
    if (tn == 64)
        return gate_up ? launch_gemm_kernel<GemmQ6K, true, 64>(st, G, map_b, map_bs) : launch_gemm_kernel<GemmQ6K, false, 64>(st, G, map_b, map_bs);
    return gate_up ? launch_gemm_kernel<GemmQ6K, true, 128>(st, G, map_b, map_bs) : launch_gemm_kernel<GemmQ6K, false, 128>(st, G, map_b, map_bs);
}

}  // namespace cmoe
