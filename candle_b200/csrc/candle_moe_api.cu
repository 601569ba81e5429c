// extern "C" entry points of libcandle_moe_sm100.so (declared in include/candle_moe.h): argument
// validation on the host, workspace carving, and the launch sequence of the whole block.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "api_internal.cuh"

using namespace cmoe;

namespace {

// Rows per step above which the tensor-core GEMM takes the products (below, the decode kernels).  The tuning key GEMM_MIN_ROWS
// sets them; left to itself it stands for 96, and a single-device forward goes by the rows that an expert holds on average,
// k T / E, because the decode kernels pay for every eight of them and the GEMM hardly at all (gemm_rows below).
inline bool gemm_rows_auto() { return tuning_get(TUNE_GEMM_MIN_ROWS) == CANDLE_MOE_GEMM_ROWS_AUTO; }
inline int64_t gemm_min_rows() { return gemm_rows_auto() ? 96 : tuning_get(TUNE_GEMM_MIN_ROWS); }
// When the caller knows the ACTUAL largest row count of an expert (or, in the slot form of expert parallelism, a
// bound five quarters of the expected one, so that the tile width leaves a margin), the GEMM takes over above 32 rows.
// Measured on one GPU with the experts of one rank of the Mixtral-shaped layer and a former GEMM, with which the line was not measured
// again (decode kernels / GEMM, microseconds per step): one expert, 32 rows 92 / 98, 48 rows 122 / 98, 64 rows 134 / 103, 96 rows 190 / 129, 128 rows 229 / 129;
// two experts, 32 rows each 163 / 159, 40 rows 193 / 165, 64 rows 246 / 200; four experts, 32 rows 272 / 262, 40 rows
// 323 / 263.  (An earlier measurement of 248 us for two experts of ~33 rows had position tiles of 32, so that every
// expert with a row more than expected took a second, almost empty tile.)  A single-device forward only knows the
// bound T.
constexpr int64_t GEMM_MIN_ROWS_EXACT = 32;
// The dense Q8_0 product over its repacked copy: decode kernels up to the rows that split K ([32000, 4096], int8 tiles or rows / decode
// kernels: 8 rows 309 / 37 us, 32 235 / 55, 48 172 / 85, 64 130 / 92; [2048, 4096] 64 rows 42.6 / 19.8, [1024, 512] 22.2 / 15.2;
// faster in all of 300 sizes from 1024 to 32000 by 512 to 4096).  Every sixteen rows are one more pass over the copy.
constexpr int64_t QMM_DIRECT_MAX_ROWS = 64;
constexpr int64_t QMM_GEMM_MIN_ROWS = 48;  // the dense product: one matrix, rows known exactly
// The line for Q8_0 over repacked copies, from estimated times of both forms in microseconds: the GEMM costs .33 more per expert and .065
// less per million routed weights saved (W), the decode kernels .009 W more for every row of an expert beyond eight; a shared expert, whose
// group holds every row, joins the decode kernels' launches (14 us of launches and .6 per million of its weights, S, saved) and costs them
// .006 S more per row.  Fitted to 330 sizes (8 to 128 experts, top-1 to top-8, d = 1024 to 4096, ff = 512 to 4096, with and without a
// shared expert of 2816 to 5632, 97 to 512 rows): 0.3 % slower than the better form on average, at worst 11 %.  Decode kernels / GEMM --
// 60 experts of 2048 x 1408, top-2: 160 rows 172 / 189, 352 192 / 196, 512 260 / 229; with a shared expert of 5632: 160 rows 220 / 254, 272
// 263 / 259, 512 406 / 302; 32 experts, top-2, and that shared expert: 97 rows 147 / 161, 192 183 / 180, 352 273 / 193; 128 experts of
// 2048 x 768, top-8: 97 rows 258 / 267, 160 279 / 275, 352 376 / 279; 16 experts of 1024 x 1024, top-2: 97 rows 54 / 46.  (By 22 rows of an expert
// alone, with a shared expert or not: 7 % slower than the better form on average, at worst 46 %.)
inline int64_t gemm_rows_q80(const candle_moe_weights_t* w, int64_t rows) {
    const double E = w->n_experts, k = w->top_k, W = 3e-6 * E * w->d_model * w->d_ff;
    const double S = w->d_ff_shared > 0 && w->dtype_shared13 == CANDLE_GGML_Q8_0 && w->dtype_shared2 == CANDLE_GGML_Q8_0 && w->shared_w1_prepacked &&
                             w->shared_w3_prepacked && w->shared_w2_prepacked
                         ? 3e-6 * w->d_model * w->d_ff_shared
                         : 0.0;
    const double gain = 0.065 * W - 0.33 * E + (S > 0 ? 14.0 + 0.6 * S : 0.0);
    const double eight = 8.0 * E / k, per_row = 0.009 * W * k / E, per_shared_row = 0.006 * S;
    const double line = gain <= per_shared_row * eight ? (S > 0 ? gain / per_shared_row : 0.0) : (gain + per_row * eight) / (per_row + per_shared_row);
    return std::max(rows, (int64_t)std::min(line, 512.0));  // (not measured beyond)
}
// Rows of an expert above which k-quant products over repacked copies take the GEMM: where both forms cross, which is later for layers
// of many weights (the GEMM's time per block is the same, the decode kernels gain on longer items) and for Q6_K down products (1.2 us a
// block of the GEMM instead of 0.7).  Decode kernels / GEMM, us per layer, w13 / w2.  8 experts, top-2 -- 4096 x 14336, Q4_K / Q6_K: 48 rows
// 242 / 287, 58 266 / 296, 64 310 / 302, 72 330 / 302; Q4_K / Q4_K: 52 230 / 252, 60 260 / 253; 2560 x 6144, Q4_K / Q6_K: 50 103 / 117, 60 109 /
// 113, 64 114 / 111; Q6_K / Q6_K: 50 120 / 129, 60 134 / 129; 1024 x 3584, Q4_K / Q6_K: 52 52 / 56, 60 57 / 56; Q4_K / Q4_K: 48 51 / 50, 60 54 / 52.
// 4 experts of 4096 x 14336, top-2, Q4_K / Q6_K: 25 rows 138 / 176, 32 182 / 170.  60 of 2048 x 1536, top-8: 96 rows 191 / 210.  16 of 2048 x
// 1024, top-4: 48 rows 62 / 59; 32 of them, top-8: 48 90 / 92, 57 97 / 93.  Twelve for all of them, as before, cost 3 to 25 % between the lines.
// Q6_K rows of 4096 and more are too long for the decode kernels' gate_up with two position tiles: 4096 x 14336: 48 rows 477 / 352.
inline int64_t gemm_expert_rows(const candle_moe_weights_t* w) {
    const bool q6_13 = w->dtype_w13 == CANDLE_GGML_Q6K, q6_2 = w->dtype_w2 == CANDLE_GGML_Q6K;
    if (!expert_direct_takes_gate_up(w->dtype_w13, w->d_model)) return 12;
    const double millions = 3e-6 * w->n_experts * w->d_model * w->d_ff;
    if (millions >= 350.0) return q6_13 && q6_2 ? 14 : 15;
    return w->n_experts > 8 ? 12 : (q6_2 ? 14 : 13);
}
// Rows of a step above which a layer without copies takes the GEMM, for Q4_K products beside a Q4_K gate_up (Q6_K ones stay where they are).
// Up to eight rows the streaming form has one position tile and is the faster for most layers; beyond, it pays for two, and the GEMM wins from 2.5 rows of an expert on, its
// launches for the tensor maps of many experts included -- where its tiles fill the SMs and the weights outweigh its launches.
// Streaming form / GEMM, us per layer.  8 experts, top-2 -- 1024 x 3584: 10 rows 64 / 53, 60 98 / 51; 4096 x 4096: 8 77 / 94, 10 104 / 101,
// 60 163 / 103; 4096 x 14336: 10 293 / 239, 60 500 / 240, Q6_K down 320 / 302, 579 / 415; 512 x 1024: 16 33 / 34, 32 36 / 34; top-4, 4096 x
// 4096: 6 83 / 100, 8 89 / 101, 10 110 / 100.  64 of 2048 x 1024, top-8: 21 rows 184 / 133; 128 of 2048 x 768, top-8: 42 rows 303 / 222; 32 of 512
// x 512, top-4: 24 rows 54 / 57, 64 60 / 56.  Few experts -- 4 of 4096 x 4096, top-2: 8 rows 56 / 67, 12 72 / 66; 4 of 4096 x 14336: 8 136 /
// 155, 10 174 / 153; 3 of 4096 x 4096, top-1: 9 59 / 63, 22 65 / 63; 2 of 2048 x 4096, top-1: 8 33 / 39, 12 39 / 39; 3 of 1024 x 1024: 42 rows 31 / 33.
inline int64_t gemm_rows_gguf(const candle_moe_weights_t* w, int64_t rows) {
    const int64_t E = w->n_experts;
    const double millions = 3e-6 * E * w->d_model * w->d_ff;
    int64_t halves = 5;  // of a row of an expert
    if (millions < (E < 6 ? 18.0 : 8.0)) return rows;
    if (E < 6 && millions < 500.0) halves = 12;
    else if (millions < std::max(20.0, 0.8 * E)) halves = 16;
    return std::min(rows, std::max<int64_t>(8, halves * E / (2 * w->top_k)));
}
// Only where an expert's rows are expected in a narrow tile, whose gate is as exact as that of the forms before.
inline int64_t gemm_rows(const candle_moe_weights_t* w) {
    const int64_t rows = gemm_min_rows(), E = w->n_experts, k = w->top_k;
    if (!gemm_rows_auto()) return rows;
    const bool q80_13 = w->dtype_w13 == CANDLE_GGML_Q8_0, q80_2 = w->dtype_w2 == CANDLE_GGML_Q8_0;
    const bool copies = w->w1_prepacked && w->w3_prepacked && w->w2_prepacked;
    if (copies && q80_13 && q80_2) return gemm_rows_q80(w, rows);
    if (q80_13 || q80_2 || 5 * k * rows > 4 * 64 * E) return rows;
    if (copies) return std::min(rows, gemm_expert_rows(w) * E / k);
    return w->dtype_w13 == CANDLE_GGML_Q4K ? gemm_rows_gguf(w, rows) : rows;
}
// Decode-sized batches may split K finely (more parallel items, smaller resident activations);
// larger batches get four slots, enough for the streaming form's activation rows to fit.
inline int k_split_slots(int64_t T) { return T <= gemm_min_rows() ? MAX_K_SPLITS : 4; }

struct Workspace {
    // routing
    uint32_t* topk_ids;
    float* topk_w;
    uint32_t* counts;
    uint32_t* offsets;
    uint32_t* perm_token;
    uint32_t* pair_pos;
    uint32_t* perm_scratch;  // per-chunk tables of the many-CTA dispatch
    // quantized input rows (one per token; experts gather through perm_token)
    int8_t* xq;
    float* xs;
    int16_t* xb;
    // routed experts
    float* hidden;  // [T*k, ff]
    int8_t* hq;
    float* hs;
    int16_t* hb;
    float* eo;  // [T*k, d]
    // shared expert
    uint32_t* sh_offsets;  // [2] = {0, T}
    int8_t* sxq;
    float* sxs;
    int16_t* sxb;
    float* shidden;  // [T, ff_s]
    int8_t* shq;
    float* shs;
    int16_t* shb;
    float* so;  // [T, d]
    void* gemm;  // operand scratch of the large-batch tensor-core GEMM (null for decode-sized T)
    void* repack_gemm;  // large batches over Q6_K without copies: operand scratch of that form (null: not enough workspace for it)
    uint8_t* repack;    // ... and one expert's repacked matrices
    size_t total;      // without that form
    size_t total_ext;  // with it
};

constexpr int REPACK_MAX_RUN = 12;  // see gemm_repacking
// partial outputs of that form: the room behind them is its own
constexpr int64_t REPACK_MANY_SLOT_ROWS = 2048;
inline int repack_slots(int64_t P) { return P <= REPACK_MANY_SLOT_ROWS ? 4 : 2; }
// Q6_K as the GEMM reads it is the repacked layout.  Without copies a large batch (P rows over E experts) can repack one expert
// at a time on its way through the GEMM, for shapes the repack takes (as candle_moe_prepack and the GEMM check them).  Two or
// three launches per expert, one after the other and each over one matrix: worth it only where the other forms pass over an
// expert's weights long enough.  Microseconds per expert, W = its weights in millions, r = its rows on average, fitted to the
// shapes below: repacking 5 per launch + W / 0.8 + r W / 190; streaming r W / 34 (it takes rows of whole 16 bytes, k a
// multiple of 2048); row-per-warp r W / 3 + 1.1 r / E (the latency of a row, which few small experts do not hide).  Taken with a
// margin of 1.15 for what the fit misses.
// Whole layers (both products Q6_K unless said otherwise), other form / repacking, us -- d = 1536, ff = 1536, 60 experts: 6 rows per expert 954 /
// 2145, 13 rows 1762 / 2153, 27 rows 3385 / 2412; d = 512, ff = 1024, 128 experts, 1.5 rows 234 / 3017; d = 1536, ff = 768, 128
// experts, 25 rows 3483 / 3741, 50 rows 6811 / 5288; d = 1536, ff = 2560, 8 experts, 24 rows 730 / 350; streaming: d = 2048,
// ff = 4096, 8 experts, 100 rows 592 / 604, 200 rows 1070 / 662; d = 2048, ff = 2048, 60 experts, 107 rows 2380 / 3480; d = 4096,
// ff = 14336, 8 experts, Q4_K gate_up, 75 rows 1177 / 979, 100 rows 1454 / 1177, 500 rows 6128 / 2669.
inline bool repacks_on_the_way(int dtype, bool has_copy, int n, int k, bool gate_up, int64_t P, int E) {
    if (dtype != CANDLE_GGML_Q6K || has_copy || n % (gate_up ? 64 : 128) || k % 512 || tuning_get(TUNE_FORCE_ROWS)) return false;
    const double weights = 1e-6 * n * k * (gate_up ? 2 : 1), work = weights * (double)P / E;
    const double repacking = 5.0 * (gate_up ? 3 : 2) + weights / 0.8 + work / 190.0;
    const double other = k % 2048 == 0 ? work / 34.0 : work / 3.0 + 1.1 * (double)P / E / E;
    return other > 1.15 * repacking;
}

// avail: bytes behind base_ (the optional part is handed out only if it fits)
Workspace layout(const candle_moe_weights_t* w, int64_t T, void* base_, size_t avail = 0) {
    uint8_t* base = static_cast<uint8_t*>(base_);
    Workspace ws{};
    size_t off = 0;
    const size_t Tk = (size_t)T * w->top_k, d = w->d_model, ff = w->d_ff, E = w->n_experts;
    ws.topk_ids = carve<uint32_t>(base, off, Tk);
    ws.topk_w = carve<float>(base, off, Tk);
    ws.counts = carve<uint32_t>(base, off, E);
    ws.offsets = carve<uint32_t>(base, off, E + 1);
    ws.perm_token = carve<uint32_t>(base, off, Tk);
    ws.pair_pos = carve<uint32_t>(base, off, Tk);
    ws.perm_scratch = carve<uint32_t>(base, off, permute_scratch_words((int64_t)Tk, (int)E));
    ws.xq = carve<int8_t>(base, off, (size_t)T * d);
    ws.xs = carve<float>(base, off, (size_t)T * d / act_block(w->dtype_w13));
    ws.xb = carve<int16_t>(base, off, (size_t)T * d / 16);
    ws.hidden = carve<float>(base, off, Tk * ff);
    ws.hq = carve<int8_t>(base, off, Tk * ff);
    ws.hs = carve<float>(base, off, Tk * ff / act_block(w->dtype_w2));
    ws.hb = carve<int16_t>(base, off, Tk * ff / 16);
    size_t free_at = align_up(off, 256) + repack_slots((int64_t)Tk) * Tk * d * sizeof(float);
    ws.eo = carve<float>(base, off, Tk * d * k_split_slots(T));
    if (w->d_ff_shared > 0) {
        const size_t fs = w->d_ff_shared;
        ws.sh_offsets = carve<uint32_t>(base, off, 2);
        if (act_block(w->dtype_shared13) != act_block(w->dtype_w13)) {
            ws.sxq = carve<int8_t>(base, off, (size_t)T * d);
            ws.sxs = carve<float>(base, off, (size_t)T * d / act_block(w->dtype_shared13));
            ws.sxb = carve<int16_t>(base, off, (size_t)T * d / 16);
        } else {
            ws.sxq = ws.xq;
            ws.sxs = ws.xs;
            ws.sxb = ws.xb;
        }
        ws.shidden = carve<float>(base, off, (size_t)T * fs);
        ws.shq = carve<int8_t>(base, off, (size_t)T * fs);
        ws.shs = carve<float>(base, off, (size_t)T * fs / act_block(w->dtype_shared2));
        ws.shb = carve<int16_t>(base, off, (size_t)T * fs / 16);
        ws.so = carve<float>(base, off, (size_t)T * d * k_split_slots(T));
        free_at = off;
    }
    size_t gemm_ext = 0;  // end of the GEMM's operand scratch where a workspace need not have it
    if (T > std::min(gemm_min_rows(), gemm_rows(w))) {
        // large batches: activation operand of the tcgen05 GEMM, reused by gate_up and down
        size_t g = 0;
        const auto takes = [](int dt, const void* packed) {
            return dt == CANDLE_GGML_Q4K || ((dt == CANDLE_GGML_Q6K || dt == CANDLE_GGML_Q8_0) && packed != nullptr);
        };
        if (takes(w->dtype_w13, w->w1_prepacked))
            g = std::max(g, expert_gemm_scratch_bytes((int64_t)Tk, (int)d, w->dtype_w13 == CANDLE_GGML_Q8_0 ? 2 : 1));
        if (takes(w->dtype_w2, w->w2_prepacked)) g = std::max(g, expert_gemm_scratch_bytes((int64_t)Tk, (int)ff));
        if (w->d_ff_shared > 0 && w->dtype_shared13 == CANDLE_GGML_Q8_0 && w->shared_w1_prepacked && w->shared_w3_prepacked &&
            w->shared_w2_prepacked)
            g = std::max(g, std::max(expert_gemm_scratch_bytes(T, (int)d, 2), expert_gemm_scratch_bytes(T, w->d_ff_shared)));
        if (g) {
            const size_t at = align_up(off, 1024);
            const bool optional = T <= gemm_min_rows();  // the decode kernels take the batch without it
            if (!optional) off = at + g;
            else gemm_ext = align_up(at + g, 256);
            if (!optional || avail >= gemm_ext) ws.gemm = base ? base + at : nullptr;
            if (!base) ws.gemm = reinterpret_cast<void*>(1);  // size query: only the extent matters
        }
    }
    ws.total = align_up(off, 256);
    ws.total_ext = std::max(ws.total, gemm_ext);
    if (T > gemm_min_rows()) {
        const bool r13 = repacks_on_the_way(w->dtype_w13, w->w1_prepacked && w->w3_prepacked, w->d_ff, w->d_model, true, (int64_t)Tk, w->n_experts);
        const bool r2 = repacks_on_the_way(w->dtype_w2, w->w2_prepacked != nullptr, w->d_model, w->d_ff, false, (int64_t)Tk, w->n_experts);
        if (r13 || r2) {
            // The partial outputs it does not use and the GEMM's own scratch (the other product's, done or not begun) lie free
            const size_t at = align_up(free_at, 1024);
            const size_t operand = align_up(std::max(r13 ? expert_gemm_scratch_bytes((int64_t)Tk, (int)d) : 0,
                                                     r2 ? expert_gemm_scratch_bytes((int64_t)Tk, (int)ff) : 0), 1024);
            const size_t matrices = std::max(r13 ? 2 * prepacked_bytes(CANDLE_GGML_Q6K, (int64_t)ff, (int)d) : 0,
                                             r2 ? prepacked_bytes(CANDLE_GGML_Q6K, (int64_t)d, (int)ff) : 0);
            ws.total_ext = std::max(ws.total, align_up(at + operand + matrices, 256));
            if (base && avail >= ws.total_ext) {
                ws.repack_gemm = base + at;
                ws.repack = base + at + operand;
                if (!ws.gemm) ws.gemm = ws.repack_gemm;
            }
        }
    }
    return ws;
}

// A workspace for up to T rows serves smaller batches too: its size grows with the rows except where the partial outputs become
// fewer (behind gemm_min_rows() rows; REPACK_MANY_SLOT_ROWS selections), so the largest of these holds every batch up to T.
template <class Bytes>
size_t for_every_batch(const candle_moe_weights_t* w, int64_t T, Bytes bytes) {
    const int64_t few = std::max<int64_t>(0, gemm_min_rows());
    return std::max({bytes(T), bytes(std::min(T, few)), bytes(std::min(T, REPACK_MANY_SLOT_ROWS / w->top_k))});
}

}  // namespace
int cmoe::check_weights(const candle_moe_weights_t* w) {
    if (!w) return CANDLE_MOE_E_NULL;
    if (w->d_model <= 0 || w->d_ff <= 0 || w->n_experts <= 0 || w->top_k <= 0) return CANDLE_MOE_E_SHAPE;
    if (w->n_experts > CANDLE_MOE_MAX_EXPERTS || w->top_k > CANDLE_MOE_MAX_TOPK || w->top_k > w->n_experts)
        return CANDLE_MOE_E_SHAPE;
    if (!dtype_supported(w->dtype_w13) || !dtype_supported(w->dtype_w2)) return CANDLE_MOE_E_DTYPE;
    if (w->d_model % block_elems(w->dtype_w13) || w->d_ff % block_elems(w->dtype_w2)) return CANDLE_MOE_E_SHAPE;
    if (w->d_model % 32 || w->d_ff % 32) return CANDLE_MOE_E_SHAPE;
    if (w->d_ff_shared < 0) return CANDLE_MOE_E_SHAPE;
    if (w->d_ff_shared > 0) {
        if (!dtype_supported(w->dtype_shared13) || !dtype_supported(w->dtype_shared2)) return CANDLE_MOE_E_DTYPE;
        if (w->d_model % block_elems(w->dtype_shared13) || w->d_ff_shared % block_elems(w->dtype_shared2) ||
            w->d_ff_shared % 32)
            return CANDLE_MOE_E_SHAPE;
    }
    return CANDLE_MOE_OK;
}

int cmoe::fill_ptrs(const void* const* host, int E, ExpertPtrs& out) {
    if (!host) return CANDLE_MOE_E_NULL;
    std::memset(&out, 0, sizeof(out));
    for (int e = 0; e < E; ++e) {
        if (!host[e]) return CANDLE_MOE_E_NULL;
        if (reinterpret_cast<uintptr_t>(host[e]) & 15) return CANDLE_MOE_E_ALIGN;
        out.p[e] = static_cast<const uint8_t*>(host[e]);
    }
    return CANDLE_MOE_OK;
}

namespace {
// tuning key GEMM_ENABLED = 0 keeps large batches on the streaming form (A/B checks)
inline bool gemm_enabled() { return tuning_get(TUNE_GEMM_ENABLED) != 0; }

// Optional per-stage event marks for candle_moe_forward_timed (null in normal calls).
constexpr int N_STAGES = 8;  // router, permute, quantize_x, gate_up, quantize_h, down, shared expert, combine
struct StageProbe {
    cudaEvent_t ev[N_STAGES + 1];
    bool hit[N_STAGES + 1];
};
thread_local StageProbe* g_probe = nullptr;
inline void mark(cudaStream_t st, int stage_done) {
    if (g_probe) {
        cudaEventRecord(g_probe->ev[stage_done + 1], st);
        g_probe->hit[stage_done + 1] = true;
    }
}

}  // namespace

extern "C" {

const char* candle_moe_version(void) { return "candle_moe_sm100 0.2"; }

int candle_moe_set_tuning(int32_t key, int64_t value) { return tuning_set(key, value) ? CANDLE_MOE_OK : CANDLE_MOE_E_SHAPE; }
int candle_moe_get_tuning(int32_t key, int64_t* value) {
    if (!value) return CANDLE_MOE_E_NULL;
    if (key < 0 || key >= TUNE_N_KEYS) return CANDLE_MOE_E_SHAPE;
    *value = tuning_get(key);
    return CANDLE_MOE_OK;
}

int candle_moe_workspace_bytes(const candle_moe_weights_t* w, int64_t max_tokens, size_t* out_bytes) {
    if (!out_bytes) return CANDLE_MOE_E_NULL;
    CM_TRY(check_weights(w));
    if (max_tokens < 0 || max_tokens > (int64_t)1 << 24) return CANDLE_MOE_E_SHAPE;
    *out_bytes = for_every_batch(w, max_tokens, [&](int64_t rows) { return layout(w, rows, nullptr).total_ext; });
    return CANDLE_MOE_OK;
}

int candle_moe_forward_gemm_rows(const candle_moe_weights_t* w, int64_t* out_rows) {
    if (!out_rows) return CANDLE_MOE_E_NULL;
    CM_TRY(check_weights(w));
    *out_rows = gemm_enabled() ? gemm_rows(w) : INT64_MAX;
    return CANDLE_MOE_OK;
}

int candle_moe_router_topk(void* stream, const float* x, const float* router, const float* bias, int64_t T,
                           int32_t d, int32_t E, int32_t k, int32_t renorm, uint32_t* topk_ids, float* topk_w) {
    if (!x || !router || !topk_ids || !topk_w) return CANDLE_MOE_E_NULL;
    if (T < 0 || d <= 0 || d % 4 || E <= 0 || E > CANDLE_MOE_MAX_EXPERTS || k <= 0 || k > CANDLE_MOE_MAX_TOPK || k > E)
        return CANDLE_MOE_E_SHAPE;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(router)) & 15) return CANDLE_MOE_E_ALIGN;
    return rc(launch_router_topk((cudaStream_t)stream, x, router, bias, T, d, E, k, renorm, topk_ids, topk_w));
}

int candle_moe_permute(void* stream, const uint32_t* topk_ids, int64_t T, int32_t k, int32_t E,
                       uint32_t* expert_counts, uint32_t* expert_offsets, uint32_t* perm_token, uint32_t* pair_pos) {
    if (!topk_ids || !expert_counts || !expert_offsets || !perm_token || !pair_pos) return CANDLE_MOE_E_NULL;
    if (T < 0 || k <= 0 || k > CANDLE_MOE_MAX_TOPK || E <= 0 || E > CANDLE_MOE_MAX_EXPERTS) return CANDLE_MOE_E_SHAPE;
    if (T > (int64_t)UINT32_MAX / k) return CANDLE_MOE_E_SHAPE;  // the lists hold 32-bit positions, the kernel 32-bit indices
    return rc(launch_permute((cudaStream_t)stream, topk_ids, T, k, E, expert_counts, expert_offsets, perm_token,
                             pair_pos));
}

int candle_moe_quantize_act(void* stream, const float* x, int64_t rows, int32_t kdim, int32_t for_weight_dtype,
                            int8_t* qs, float* scales, int16_t* bsums) {
    if (!x || !qs || !scales) return CANDLE_MOE_E_NULL;
    if (!dtype_supported(for_weight_dtype)) return CANDLE_MOE_E_DTYPE;
    if (for_weight_dtype != CANDLE_GGML_Q8_0 && !bsums) return CANDLE_MOE_E_NULL;
    if (rows < 0 || kdim <= 0 || kdim % act_block(for_weight_dtype)) return CANDLE_MOE_E_SHAPE;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(qs) & 7)) return CANDLE_MOE_E_ALIGN;
    return rc(launch_quantize_act((cudaStream_t)stream, x, rows, kdim, for_weight_dtype, qs, scales, bsums));
}

int candle_moe_combine(void* stream, const float* expert_out, const uint32_t* topk_ids, const float* topk_w,
                       const uint32_t* pair_pos, int64_t T, int32_t k, int32_t d, const float* shared_out,
                       const float* x, const float* shared_gate, float* y) {
    if (!expert_out || !topk_ids || !topk_w || !pair_pos || !y) return CANDLE_MOE_E_NULL;
    if (shared_out && (!x || !shared_gate)) return CANDLE_MOE_E_NULL;
    if (T < 0 || k <= 0 || k > CANDLE_MOE_MAX_TOPK || d <= 0 || d % 4) return CANDLE_MOE_E_SHAPE;
    return rc(launch_combine((cudaStream_t)stream, expert_out, 1, 0, topk_ids, topk_w, pair_pos, T, k, d, shared_out, 1,
                             0, x, shared_gate, y));
}

int candle_moe_grouped_gate_up(void* stream, const void* const* w1, const void* const* w3, int32_t dtype,
                               int32_t E, int32_t d, int32_t ff, const uint32_t* expert_offsets,
                               const uint32_t* row_of, int64_t max_rows, const int8_t* xq, const float* xscales,
                               const int16_t* xbsums, float* hidden) {
    if (!expert_offsets || !xq || !xscales || !hidden) return CANDLE_MOE_E_NULL;
    if (!dtype_supported(dtype)) return CANDLE_MOE_E_DTYPE;
    if (dtype != CANDLE_GGML_Q8_0 && !xbsums) return CANDLE_MOE_E_NULL;
    if (E <= 0 || E > CANDLE_MOE_MAX_EXPERTS || d <= 0 || ff <= 0 || d % block_elems(dtype) || max_rows < 0)
        return CANDLE_MOE_E_SHAPE;
    ExpertPtrs p1, p3;
    CM_TRY(fill_ptrs(w1, E, p1));
    CM_TRY(fill_ptrs(w3, E, p3));
    return rc(launch_grouped_gate_up((cudaStream_t)stream, p1, p3, dtype, E, d, ff, expert_offsets, row_of, max_rows,
                                     xq, xscales, xbsums, hidden));
}

int candle_moe_grouped_down(void* stream, const void* const* w2, int32_t dtype, int32_t E, int32_t d, int32_t ff,
                            const uint32_t* expert_offsets, int64_t max_rows, const int8_t* hq, const float* hscales,
                            const int16_t* hbsums, float* out) {
    if (!expert_offsets || !hq || !hscales || !out) return CANDLE_MOE_E_NULL;
    if (!dtype_supported(dtype)) return CANDLE_MOE_E_DTYPE;
    if (dtype != CANDLE_GGML_Q8_0 && !hbsums) return CANDLE_MOE_E_NULL;
    if (E <= 0 || E > CANDLE_MOE_MAX_EXPERTS || d <= 0 || ff <= 0 || ff % block_elems(dtype) || max_rows < 0)
        return CANDLE_MOE_E_SHAPE;
    ExpertPtrs p2;
    CM_TRY(fill_ptrs(w2, E, p2));
    return rc(launch_grouped_down((cudaStream_t)stream, p2, dtype, E, d, ff, expert_offsets, max_rows, hq, hscales,
                                  hbsums, out, 0, 1, nullptr));
}

}  // extern "C"

namespace cmoe {
// A large batch over Q6_K experts that have no repacked copies: expert by expert, its matrices are repacked into the workspace and
// taken through the GEMM (see repacks_on_the_way for when and what it measured).  K of the down product is split until no f32 sum
// runs over more than twelve blocks, as far as the slots go (two for more than 2048 rows, whose partial outputs weigh most):
// the forms that take the layer otherwise add in many short runs.  (Relative error against 64-bit arithmetic on the same int8
// rows, K = 14336: unsplit 1.38e-7, four splits 0.84e-7, streaming 0.72e-7; K = 4096 0.78 / 0.65 / 0.62e-7; row-per-warp K = 2560
// 0.89, here 0.58e-7.  Up to 4 % of a layer's time.)
static cudaError_t gemm_repacking(cudaStream_t st, bool gate_up, const ExpertPtrs& wa, const ExpertPtrs& wb, int E, int K, int N,
                                  const uint32_t* offsets, const uint32_t* row_of, int64_t P, int64_t tile_rows, const int8_t* aq,
                                  const float* ascale, const int16_t* absum, float* out, const ExpertBufs& b, int* n_splits,
                                  int64_t split_stride, const float* x_f32) {
    const size_t bytes = prepacked_bytes(CANDLE_GGML_Q6K, N, K);
    ExpertPtrs ra{}, rb{};
    ra.p[0] = b.repack;
    rb.p[0] = gate_up ? b.repack + bytes : b.repack;
    for (int e = 0; e < E; ++e) {
        cudaError_t ce = launch_prepack(st, CANDLE_GGML_Q6K, wa.p[e], N, K, b.repack);
        if (ce == cudaSuccess && gate_up) ce = launch_prepack(st, CANDLE_GGML_Q6K, wb.p[e], N, K, b.repack + bytes);
        if (ce == cudaSuccess)
            ce = launch_expert_gemm(st, gate_up, ra, rb, CANDLE_GGML_Q6K, true, 1, K, N, offsets + e, row_of, P, tile_rows, aq, ascale, absum,
                                    out, b.repack_gemm, n_splits ? repack_slots(P) : 1, n_splits, split_stride, nullptr, x_f32, nullptr, e > 0, true,
                                    REPACK_MAX_RUN);
        if (ce != cudaSuccess) return ce == cudaErrorNotSupported && e > 0 ? cudaErrorUnknown : ce;
    }
    return cudaSuccess;
}

// The routed experts over P rows grouped by expert (device offsets [E + 1]); no expert has more than max_rows
// rows.  Picks, per product, the decode kernels over the repacked copies, the tensor-core GEMM
// (from b.gemm_above rows on, scratch present), or the streaming / row forms.  Leaves *eo_splits partial outputs in b.eo.
int run_experts(cudaStream_t st, const candle_moe_weights_t* w, const ExpertPtrs& p1, const ExpertPtrs& p3,
                const ExpertPtrs& p2, int64_t max_rows, int64_t P, const uint32_t* offsets, const uint32_t* row_of,
                const int8_t* xq, const float* xs, const int16_t* xb, const ExpertBufs& b, int slots, int* eo_splits,
                bool marks, bool rows_exact, const uint32_t* row_limit, int64_t total_rows_hint, SharedRun* shared) {
    if (total_rows_hint <= 0) total_rows_hint = P;
    const int E = w->n_experts, d = w->d_model, ff = w->d_ff;
    const int64_t gemm_above = b.gemm_above >= 0 ? b.gemm_above : gemm_min_rows();
    const bool gemm_here = b.gemm && gemm_enabled();
    bool large = gemm_here && max_rows > (rows_exact ? GEMM_MIN_ROWS_EXACT : gemm_above);
    bool use_prepacked = w->w1_prepacked && w->w3_prepacked && w->w2_prepacked &&
                         max_rows <= std::max<int64_t>({gemm_min_rows(), gemm_above, 64}) && !large;
    bool gate_done = false, down_done = false;
    *eo_splits = 1;
    ExpertPtrs q1, q3, q2;
    // Tables with a missing or misaligned entry: an error with k-quants at every batch that the decode kernels may take, whether this
    // one takes them or not (Q4_K products on the GEMM read none)
    const bool check_copies = large && !rows_exact && max_rows <= gemm_min_rows() && w->w1_prepacked && w->w3_prepacked && w->w2_prepacked;
    if (check_copies && w->dtype_w13 != CANDLE_GGML_Q8_0 && w->dtype_w2 != CANDLE_GGML_Q8_0) {
        CM_TRY(fill_ptrs(w->w1_prepacked, E, q1));
        CM_TRY(fill_ptrs(w->w3_prepacked, E, q3));
        CM_TRY(fill_ptrs(w->w2_prepacked, E, q2));
    }
    if (use_prepacked) {
        int st_copies = fill_ptrs(w->w1_prepacked, E, q1);
        if (st_copies == CANDLE_MOE_OK) st_copies = fill_ptrs(w->w3_prepacked, E, q3);
        if (st_copies == CANDLE_MOE_OK) st_copies = fill_ptrs(w->w2_prepacked, E, q2);
        // (left alone with Q8_0 matrices, which need no copies here)
        if (st_copies != CANDLE_MOE_OK && w->dtype_w13 != CANDLE_GGML_Q8_0 && w->dtype_w2 != CANDLE_GGML_Q8_0) return st_copies;
        use_prepacked = st_copies == CANDLE_MOE_OK;
    }
    // More than gemm_min_rows() rows that the line leaves to the decode kernels: the GEMM takes what they refuse -- rows too long for
    // their shared memory (Q8_0 gate_up from d = 5120 on, down from K = 20480), tables that are no use to them.  (16 experts of 5120 x
    // 1536, top-1, 128 rows: 126 us that way, 320 on the tile kernel over the GGUF blocks.)
    const bool gemm_second = gemm_here && !large && use_prepacked && max_rows > gemm_min_rows();
    if (gemm_here && !use_prepacked && max_rows > gemm_min_rows()) large = true;
    if (use_prepacked) {
        cudaError_t ce = cudaErrorNotSupported;
        const SharedGroup* const tries[2] = {shared ? &shared->gate : nullptr, nullptr};  // with the shared expert, or without
        for (const SharedGroup* sg : tries) {
            if (ce != cudaErrorNotSupported) break;
            ce = launch_expert_direct(st, true, q1, q3, w->dtype_w13, E, d, ff, offsets, row_of, max_rows, xq, xs, xb, b.hidden, nullptr,
                                      0, 1, 0, total_rows_hint, nullptr, sg);
            if (ce == cudaSuccess && sg) shared->gate_done = true;
        }
        if (ce == cudaSuccess)
            gate_done = true;
        else if (ce != cudaErrorNotSupported)
            return (int)ce;
    }
    // Position-tile width of the GEMM: from the actual largest row count when it is known, else from five quarters
    // of the average (an expert beyond the tile width simply takes a second tile)
    const int64_t tile_rows = rows_exact ? max_rows : std::min<int64_t>(max_rows, (5 * total_rows_hint + 4 * E - 1) / (4 * E));
    if (!gate_done && (large || gemm_second)) {
        // Q6_K and Q8_0 are read from the repacked copies (their GGUF blocks are only 2-byte aligned)
        const bool rp = (w->dtype_w13 == CANDLE_GGML_Q6K || w->dtype_w13 == CANDLE_GGML_Q8_0) && w->w1_prepacked && w->w3_prepacked;
        ExpertPtrs g1 = p1, g3 = p3;
        if (rp) {
            CM_TRY(fill_ptrs(w->w1_prepacked, E, g1));
            CM_TRY(fill_ptrs(w->w3_prepacked, E, g3));
        }
        const cudaError_t ce = !rp && b.repack && repacks_on_the_way(w->dtype_w13, false, ff, d, true, P, E)
                                   ? gemm_repacking(st, true, p1, p3, E, d, ff, offsets, row_of, P, tile_rows, xq, xs, xb, b.hidden, b,
                                                    nullptr, 0, nullptr)
                                   : launch_expert_gemm(st, true, g1, g3, w->dtype_w13, rp, E, d, ff, offsets, row_of, P, tile_rows, xq, xs, xb,
                                                        b.hidden, b.gemm, 1, nullptr, 0, nullptr, nullptr, nullptr, false,
                                                        !rows_exact && max_rows <= gemm_min_rows());
        if (ce == cudaSuccess)
            gate_done = true;
        else if (ce != cudaErrorNotSupported)
            return (int)ce;
    }
    if (!gate_done)
        CM_TRY(rc(launch_grouped_gate_up(st, p1, p3, w->dtype_w13, E, d, ff, offsets, row_of, max_rows, xq, xs, xb,
                                         b.hidden)));
    if (marks) mark(st, 3);
    // The down product on the GEMM quantizes the hidden rows while it prepares its operand (not with a device-side row
    // limit: the operand is prepared for all P rows)
    const bool rp2 = (w->dtype_w2 == CANDLE_GGML_Q6K || w->dtype_w2 == CANDLE_GGML_Q8_0) && w->w2_prepacked;
    const bool repack2 = b.repack && repacks_on_the_way(w->dtype_w2, w->w2_prepacked != nullptr, d, ff, false, P, E);
    const bool fuse_h = large && !row_limit && expert_gemm_takes(false, w->dtype_w2, rp2 || repack2, ff, d, P);
    if (!fuse_h) CM_TRY(rc(launch_quantize_act(st, b.hidden, P, ff, w->dtype_w2, b.hq, b.hs, b.hb, row_limit)));
    if (shared && shared->gate_done) {
        CM_TRY(rc(launch_quantize_act(st, shared->hidden, shared->gate.rows, shared->gate.N, CANDLE_GGML_Q8_0, shared->hq, shared->hs, nullptr)));
        shared->quantized = true;
    }
    if (marks) mark(st, 4);
    if (use_prepacked) {
        cudaError_t ce = cudaErrorNotSupported;
        const SharedGroup* const tries[2] = {shared && shared->quantized ? &shared->down : nullptr, nullptr};
        for (const SharedGroup* sg : tries) {
            if (ce != cudaErrorNotSupported) break;
            ce = launch_expert_direct(st, false, q2, q2, w->dtype_w2, E, ff, d, offsets, nullptr, max_rows, b.hq, b.hs, b.hb, b.eo, eo_splits,
                                      P * d, slots, (int)(total_rows_hint < E ? total_rows_hint : E), total_rows_hint, nullptr, sg);
            if (ce == cudaSuccess && sg) shared->down_done = true;
        }
        if (ce == cudaSuccess)
            down_done = true;
        else if (ce != cudaErrorNotSupported)
            return (int)ce;
        else
            *eo_splits = 1;
    }
    if (!down_done && (large || gemm_second)) {
        ExpertPtrs g2 = p2;
        if (rp2) CM_TRY(fill_ptrs(w->w2_prepacked, E, g2));
        const cudaError_t ce = repack2 ? gemm_repacking(st, false, p2, p2, E, ff, d, offsets, nullptr, P, tile_rows, b.hq, b.hs, b.hb, b.eo, b,
                                                        eo_splits, P * d, fuse_h ? b.hidden : nullptr)
                               : launch_expert_gemm(st, false, g2, g2, w->dtype_w2, rp2, E, ff, d, offsets, nullptr, P, tile_rows,
                                                  b.hq, b.hs, b.hb, b.eo, b.gemm, slots, eo_splits, P * d, nullptr,
                                                  fuse_h ? b.hidden : nullptr);
        if (ce == cudaSuccess)
            down_done = true;
        else if (ce != cudaErrorNotSupported || fuse_h)
            return (int)ce;
    }
    if (!down_done)
        CM_TRY(rc(launch_grouped_down(st, p2, w->dtype_w2, E, d, ff, offsets, max_rows, b.hq, b.hs, b.hb, b.eo, P * d, slots,
                                      eo_splits)));
    return CANDLE_MOE_OK;
}

EpWorkspace ep_layout(const candle_moe_weights_t* w, int64_t P, void* base_) {
    uint8_t* base = static_cast<uint8_t*>(base_);
    EpWorkspace ws{};
    size_t off = 0;
    const size_t d = w->d_model, ff = w->d_ff, E = w->n_experts;
    ws.plan = carve<uint32_t>(base, off, 2048);
    ws.offsets = carve<uint32_t>(base, off, E + 1);
    ws.back = carve<uint32_t>(base, off, (size_t)P);
    ws.xq = carve<int8_t>(base, off, (size_t)P * d);
    ws.xs = carve<float>(base, off, (size_t)P * d / 256);
    ws.xb = carve<int16_t>(base, off, (size_t)P * d / 16);
    ws.eb.hidden = carve<float>(base, off, (size_t)P * ff);
    ws.eb.hq = carve<int8_t>(base, off, (size_t)P * ff);
    ws.eb.hs = carve<float>(base, off, (size_t)P * ff / 256);
    ws.eb.hb = carve<int16_t>(base, off, (size_t)P * ff / 16);
    ws.eo_rows = P * ep_eo_slots(P, (int)E);
    ws.eb.eo = carve<float>(base, off, (size_t)ws.eo_rows * d);
    if (P > GEMM_MIN_ROWS_EXACT) {
        const size_t g = std::max(expert_gemm_scratch_bytes(P, (int)d), expert_gemm_scratch_bytes(P, (int)ff));
        off = align_up(off, 1024);
        ws.eb.gemm = base ? base + off : reinterpret_cast<void*>(1);
        off += g;
    }
    ws.total = align_up(off, 256);
    return ws;
}
}  // namespace cmoe

extern "C" {

static int forward_impl(void* stream, const candle_moe_weights_t* w, const float* x, int64_t T, float* y, void* workspace,
                        size_t workspace_bytes, const float* residual, const float* norm_w = nullptr, float eps = 0.f) {
    CM_TRY(check_weights(w));
    if (!x || !y || !w->router) return CANDLE_MOE_E_NULL;
    if (T < 0 || T > (int64_t)1 << 24) return CANDLE_MOE_E_SHAPE;
    if (T == 0) return CANDLE_MOE_OK;
    if (!workspace) return CANDLE_MOE_E_NULL;
    if ((reinterpret_cast<uintptr_t>(workspace) & 255) || (reinterpret_cast<uintptr_t>(x) & 15) ||
        (reinterpret_cast<uintptr_t>(y) & 15) || (reinterpret_cast<uintptr_t>(w->router) & 15))
        return CANDLE_MOE_E_ALIGN;
    const Workspace ws = layout(w, T, workspace, workspace_bytes);
    if (workspace_bytes < ws.total) return CANDLE_MOE_E_WORKSPACE;
    const int E = w->n_experts, k = w->top_k, d = w->d_model;
    ExpertPtrs p1, p3, p2;
    CM_TRY(fill_ptrs(w->w1, E, p1));
    CM_TRY(fill_ptrs(w->w3, E, p3));
    CM_TRY(fill_ptrs(w->w2, E, p2));
    if (w->d_ff_shared > 0) {
        if (!w->shared_w1 || !w->shared_w3 || !w->shared_w2 || !w->shared_gate) return CANDLE_MOE_E_NULL;
        if (reinterpret_cast<uintptr_t>(w->shared_gate) & 15) return CANDLE_MOE_E_ALIGN;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t Tk = T * k;

    // k-quant experts: the router kernel also quantizes x (Q8K); Q8_0 experts keep the separate pass
    const bool fuse_q = w->dtype_w13 != CANDLE_GGML_Q8_0;
    if (g_probe) {
        cudaEventRecord(g_probe->ev[0], st);
        g_probe->hit[0] = true;
    }
    CM_TRY(rc(launch_router_topk(st, x, w->router, w->router_bias, T, d, E, k, w->renorm, ws.topk_ids, ws.topk_w,
                                 fuse_q ? ws.xq : nullptr, fuse_q ? ws.xs : nullptr, fuse_q ? ws.xb : nullptr,
                                 T == 1 ? ws.counts : nullptr, ws.offsets, ws.perm_token, ws.pair_pos, norm_w, eps)));
    mark(st, 0);
    // one token: the router kernel has written the dispatch itself
    if (T > 1) CM_TRY(rc(launch_permute(st, ws.topk_ids, T, k, E, ws.counts, ws.offsets, ws.perm_token, ws.pair_pos, ws.perm_scratch)));
    mark(st, 1);
    // (that pass also writes the offsets of the shared expert's one group)
    if (!fuse_q) CM_TRY(rc(launch_quantize_act(st, x, T, d, w->dtype_w13, ws.xq, ws.xs, ws.xb, nullptr, ws.sh_offsets)));
    mark(st, 2);
    // a token selects an expert at most once: no expert sees more than T rows
    int eo_splits = 1, so_splits = 1;
    const int64_t gemm_above = gemm_rows(w);
    const ExpertBufs eb{ws.hidden, ws.hq, ws.hs, ws.hb, ws.eo, ws.gemm, ws.repack, ws.repack_gemm, gemm_above};
    // over repacked Q8_0 copies the shared expert takes the decode kernels -- in the launches of the routed experts where those
    // are Q8_0 too -- and for large batches the tensor-core GEMM
    const bool sh_packed = w->d_ff_shared > 0 && w->dtype_shared13 == CANDLE_GGML_Q8_0 && w->dtype_shared2 == CANDLE_GGML_Q8_0 &&
                           w->shared_w1_prepacked && w->shared_w3_prepacked && w->shared_w2_prepacked &&
                           !((reinterpret_cast<uintptr_t>(w->shared_w1_prepacked) | reinterpret_cast<uintptr_t>(w->shared_w3_prepacked) |
                              reinterpret_cast<uintptr_t>(w->shared_w2_prepacked)) & 15);
    const int64_t sh_above = std::max(gemm_min_rows(), gemm_above);
    const bool sh_gemm = sh_packed && ws.gemm && T > sh_above && gemm_enabled();
    const bool sh_direct = sh_packed && !sh_gemm && T <= std::max<int64_t>(sh_above, 64);
    SharedRun sr;
    const bool sh_joins = sh_direct && w->dtype_w13 == CANDLE_GGML_Q8_0 && w->dtype_w2 == CANDLE_GGML_Q8_0 && ws.sxq == ws.xq;
    if (sh_joins) {
        const int fs = w->d_ff_shared;
        sr.gate = {w->shared_w1_prepacked, w->shared_w3_prepacked, T, d, fs, ws.xq, ws.xs, ws.shidden, 0, 1, nullptr};
        sr.down = {w->shared_w2_prepacked, nullptr, T, fs, d, ws.shq, ws.shs, ws.so, T * (int64_t)d, k_split_slots(T), &so_splits};
        sr.hidden = ws.shidden;
        sr.hq = ws.shq;
        sr.hs = ws.shs;
    }
    CM_TRY(run_experts(st, w, p1, p3, p2, T, Tk, ws.offsets, ws.perm_token, ws.xq, ws.xs, ws.xb, eb, k_split_slots(T),
                       &eo_splits, true, false, nullptr, 0, sh_joins ? &sr : nullptr));
    mark(st, 5);

    const float* shared_out = nullptr;
    if (w->d_ff_shared > 0) {
        const int fs = w->d_ff_shared;
        if (fuse_q) CM_TRY(rc(launch_single_group(st, ws.sh_offsets, (uint32_t)T)));
        ExpertPtrs s1{}, s3{}, s2{};
        s1.p[0] = static_cast<const uint8_t*>(w->shared_w1);
        s3.p[0] = static_cast<const uint8_t*>(w->shared_w3);
        s2.p[0] = static_cast<const uint8_t*>(w->shared_w2);
        if (ws.sxq != ws.xq)
            CM_TRY(rc(launch_quantize_act(st, x, T, d, w->dtype_shared13, ws.sxq, ws.sxs, ws.sxb)));
        bool sh_done = sr.gate_done;
        const bool sh_second = sh_direct && ws.gemm && T > gemm_min_rows() && gemm_enabled();  // as gemm_second in run_experts
        if (!sh_done && (sh_gemm || sh_direct)) {
            ExpertPtrs r1{}, r3{};
            r1.p[0] = static_cast<const uint8_t*>(w->shared_w1_prepacked);
            r3.p[0] = static_cast<const uint8_t*>(w->shared_w3_prepacked);
            cudaError_t ce = cudaErrorNotSupported;
            if (sh_direct)
                ce = launch_expert_direct(st, true, r1, r3, CANDLE_GGML_Q8_0, 1, d, fs, ws.sh_offsets, nullptr, T, ws.sxq, ws.sxs, ws.sxb,
                                          ws.shidden, nullptr, 0, 1, 0, T);
            if (ce == cudaErrorNotSupported && (sh_gemm || sh_second))
                ce = launch_expert_gemm(st, true, r1, r3, CANDLE_GGML_Q8_0, true, 1, d, fs, ws.sh_offsets, nullptr, T, T, ws.sxq, ws.sxs,
                                        ws.sxb, ws.shidden, ws.gemm);
            if (ce == cudaSuccess)
                sh_done = true;
            else if (ce != cudaErrorNotSupported)
                return (int)ce;
        }
        if (!sh_done)
            CM_TRY(rc(launch_grouped_gate_up(st, s1, s3, w->dtype_shared13, 1, d, fs, ws.sh_offsets, nullptr, T, ws.sxq,
                                             ws.sxs, ws.sxb, ws.shidden)));
        const bool fuse_sh = sh_gemm && expert_gemm_takes(false, CANDLE_GGML_Q8_0, true, fs, d, T);
        if (!fuse_sh && !sr.quantized) CM_TRY(rc(launch_quantize_act(st, ws.shidden, T, fs, w->dtype_shared2, ws.shq, ws.shs, ws.shb)));
        sh_done = sr.down_done;
        if (!sh_done && (sh_gemm || sh_direct)) {
            ExpertPtrs r2{};
            r2.p[0] = static_cast<const uint8_t*>(w->shared_w2_prepacked);
            cudaError_t ce = cudaErrorNotSupported;
            if (sh_direct)
                ce = launch_expert_direct(st, false, r2, r2, CANDLE_GGML_Q8_0, 1, fs, d, ws.sh_offsets, nullptr, T, ws.shq, ws.shs,
                                          ws.shb, ws.so, &so_splits, T * (int64_t)d, k_split_slots(T), 1, T);
            if (ce == cudaErrorNotSupported && (sh_gemm || sh_second))
                ce = launch_expert_gemm(st, false, r2, r2, CANDLE_GGML_Q8_0, true, 1, fs, d, ws.sh_offsets, nullptr, T, T, ws.shq, ws.shs,
                                        ws.shb, ws.so, ws.gemm, k_split_slots(T), &so_splits, T * (int64_t)d, nullptr,
                                        fuse_sh ? ws.shidden : nullptr);
            if (ce == cudaSuccess)
                sh_done = true;
            else if (ce != cudaErrorNotSupported || fuse_sh)
                return (int)ce;
            else
                so_splits = 1;
        }
        if (!sh_done)
            CM_TRY(rc(launch_grouped_down(st, s2, w->dtype_shared2, 1, d, fs, ws.sh_offsets, T, ws.shq, ws.shs, ws.shb,
                                          ws.so, T * (int64_t)d, k_split_slots(T), &so_splits)));
        shared_out = ws.so;
    }
    mark(st, 6);
    CM_TRY(rc(launch_combine(st, ws.eo, eo_splits, Tk * d, ws.topk_ids, ws.topk_w, ws.pair_pos, T, k, d, shared_out,
                             so_splits, T * (int64_t)d, x, w->shared_gate, y, residual)));
    mark(st, 7);
    return CANDLE_MOE_OK;
}

int candle_moe_forward(void* stream, const candle_moe_weights_t* w, const float* x, int64_t T, float* y,
                       void* workspace, size_t workspace_bytes) {
    return forward_impl(stream, w, x, T, y, workspace, workspace_bytes, nullptr);
}

int candle_moe_ffn_layer_workspace_bytes(const candle_moe_weights_t* w, int64_t T, size_t* out_bytes) {
    CM_TRY(check_weights(w));
    if (!out_bytes) return CANDLE_MOE_E_NULL;
    if (T < 0 || T > (int64_t)1 << 24) return CANDLE_MOE_E_SHAPE;
    const auto need = [&](int64_t rows) { return layout(w, rows, nullptr).total_ext + align_up((size_t)rows * w->d_model * sizeof(float), 256); };
    *out_bytes = for_every_batch(w, T, need);
    return CANDLE_MOE_OK;
}

int candle_moe_ffn_layer(void* stream, const candle_moe_weights_t* w, const float* norm_weight, float eps, const float* x,
                         int64_t T, float* y, void* workspace, size_t workspace_bytes) {
    CM_TRY(check_weights(w));
    if (!x || !y || !norm_weight) return CANDLE_MOE_E_NULL;
    if (T < 0 || T > (int64_t)1 << 24) return CANDLE_MOE_E_SHAPE;
    if (T == 0) return CANDLE_MOE_OK;
    if (!workspace) return CANDLE_MOE_E_NULL;
    if ((reinterpret_cast<uintptr_t>(workspace) & 255) || (reinterpret_cast<uintptr_t>(x) & 15) ||
        (reinterpret_cast<uintptr_t>(norm_weight) & 15))
        return CANDLE_MOE_E_ALIGN;
    const Workspace plan = layout(w, T, nullptr);
    const size_t norm_bytes = align_up((size_t)T * w->d_model * sizeof(float), 256);
    if (workspace_bytes < plan.total + norm_bytes) return CANDLE_MOE_E_WORKSPACE;
    const size_t inner = workspace_bytes >= plan.total_ext + norm_bytes ? plan.total_ext : plan.total;
    // k-quant experts and no shared expert: nothing but the router kernel reads the normalised rows
    if (router_fuses_norm(T, w->d_model) && w->dtype_w13 != CANDLE_GGML_Q8_0 && w->d_ff_shared == 0)
        return forward_impl(stream, w, x, T, y, workspace, inner, x, norm_weight, eps);
    float* xn = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + inner);
    CM_TRY(rc(launch_rmsnorm((cudaStream_t)stream, x, norm_weight, eps, T, w->d_model, xn)));
    return forward_impl(stream, w, xn, T, y, workspace, inner, x);
}

int candle_moe_forward_timed(void* stream, const candle_moe_weights_t* w, const float* x, int64_t T, float* y,
                             void* workspace, size_t workspace_bytes, float* stage_ms) {
    if (!stage_ms) return CANDLE_MOE_E_NULL;
    StageProbe probe{};
    for (int i = 0; i <= N_STAGES; ++i) {
        const cudaError_t e = cudaEventCreate(&probe.ev[i]);
        if (e != cudaSuccess) {
            for (int j = 0; j < i; ++j) cudaEventDestroy(probe.ev[j]);
            return (int)e;
        }
    }
    g_probe = &probe;
    const int st = candle_moe_forward(stream, w, x, T, y, workspace, workspace_bytes);
    g_probe = nullptr;
    cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
    for (int i = 0; i < N_STAGES; ++i) {
        stage_ms[i] = 0.f;
        if (st == CANDLE_MOE_OK && e == cudaSuccess && probe.hit[i] && probe.hit[i + 1])
            cudaEventElapsedTime(&stage_ms[i], probe.ev[i], probe.ev[i + 1]);
    }
    for (int i = 0; i <= N_STAGES; ++i) cudaEventDestroy(probe.ev[i]);
    return st != CANDLE_MOE_OK ? st : rc(e);
}

// ---- allocation-free variant -------------------------------------------------------------------
// Scratch for candle_moe_forward_static.  In host code `g_static_scratch` is only a handle for the
// symbol, not an address a kernel could use: the device address is looked up once per device with
// cudaGetSymbolAddress while that device is current, and that pointer is what the launches get.
static __device__ __align__(256) unsigned char g_static_scratch[CANDLE_MOE_STATIC_SCRATCH_BYTES];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
void* g_static_ptr[kMaxDevices] = {};

// Device address of the built-in scratch on the current device; 0 on success.
int static_scratch_ptr(void** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= kMaxDevices) return CANDLE_MOE_E_NO_DEVICE;
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess) return (int)e;
        if (!p || (reinterpret_cast<uintptr_t>(p) & 255)) return CANDLE_MOE_E_ALIGN;
        g_static_ptr[dev] = p;
    }
    *out = g_static_ptr[dev];
    return CANDLE_MOE_OK;
}
}  // namespace

int candle_moe_forward_static(void* stream, const candle_moe_weights_t* w, const float* x, int64_t T, float* y) {
    CM_TRY(check_weights(w));
    if (T < 0 || T > (int64_t)1 << 24) return CANDLE_MOE_E_SHAPE;
    const size_t need = layout(w, T, nullptr).total;
    if (need > (size_t)CANDLE_MOE_STATIC_SCRATCH_BYTES) return CANDLE_MOE_E_STATIC_SCRATCH;
    void* scratch = nullptr;
    CM_TRY(static_scratch_ptr(&scratch));
    return candle_moe_forward(stream, w, x, T, y, scratch, (size_t)CANDLE_MOE_STATIC_SCRATCH_BYTES);
}

int candle_moe_workspace_views(const candle_moe_weights_t* w, int64_t T, void* workspace, uint32_t** topk_ids,
                               float** topk_w, uint32_t** expert_counts, uint32_t** perm_token) {
    CM_TRY(check_weights(w));
    if (!workspace) return CANDLE_MOE_E_NULL;
    const Workspace ws = layout(w, T, workspace);
    if (topk_ids) *topk_ids = ws.topk_ids;
    if (topk_w) *topk_w = ws.topk_w;
    if (expert_counts) *expert_counts = ws.counts;
    if (perm_token) *perm_token = ws.perm_token;
    return CANDLE_MOE_OK;
}

int candle_moe_prepacked_bytes(int32_t dtype, int64_t n_rows, int32_t k, size_t* out_bytes) {
    if (!out_bytes) return CANDLE_MOE_E_NULL;
    if (dtype == CANDLE_GGML_Q8_0) {
        if (n_rows < 0 || k <= 0 || k % 32) return CANDLE_MOE_E_SHAPE;
        *out_bytes = prepacked_q80_bytes(n_rows, k);
        return CANDLE_MOE_OK;
    }
    if (dtype != CANDLE_GGML_Q4K && dtype != CANDLE_GGML_Q6K) return CANDLE_MOE_E_DTYPE;
    if (n_rows < 0 || k <= 0) return CANDLE_MOE_E_SHAPE;
    *out_bytes = prepacked_bytes(dtype, n_rows, k);
    return *out_bytes || n_rows == 0 ? CANDLE_MOE_OK : CANDLE_MOE_E_SHAPE;
}

int candle_moe_prepack(void* stream, int32_t dtype, const void* src_blocks, int64_t n_rows, int32_t k, void* dst) {
    if (!src_blocks || !dst) return CANDLE_MOE_E_NULL;
    if (dtype == CANDLE_GGML_Q8_0) {
        if (n_rows < 0 || k <= 0 || k % 32) return CANDLE_MOE_E_SHAPE;
        if ((reinterpret_cast<uintptr_t>(src_blocks) & 1) || (reinterpret_cast<uintptr_t>(dst) & 15)) return CANDLE_MOE_E_ALIGN;
        return rc(launch_prepack_q80((cudaStream_t)stream, src_blocks, n_rows, k, dst));
    }
    if (dtype != CANDLE_GGML_Q4K && dtype != CANDLE_GGML_Q6K) return CANDLE_MOE_E_DTYPE;
    if (n_rows < 0 || k <= 0 || k % 256 || n_rows % 8) return CANDLE_MOE_E_SHAPE;
    if ((reinterpret_cast<uintptr_t>(src_blocks) | reinterpret_cast<uintptr_t>(dst)) & 15) return CANDLE_MOE_E_ALIGN;
    if (dtype == CANDLE_GGML_Q6K && (k / 256) % 2) return CANDLE_MOE_E_SHAPE;  // rows must stay 4-byte aligned
    return rc(launch_prepack((cudaStream_t)stream, dtype, src_blocks, n_rows, k, dst));
}

int candle_moe_grouped_gate_up_prepacked(void* stream, const void* const* w1p, const void* const* w3p, int32_t dtype,
                                         int32_t E, int32_t d, int32_t ff, const uint32_t* expert_offsets,
                                         const uint32_t* row_of, int64_t max_rows, const int8_t* xq,
                                         const float* xscales, const int16_t* xbsums, float* hidden) {
    if (!expert_offsets || !xq || !xscales || !xbsums || !hidden) return CANDLE_MOE_E_NULL;
    if (dtype != CANDLE_GGML_Q4K && dtype != CANDLE_GGML_Q6K) return CANDLE_MOE_E_DTYPE;
    if (E <= 0 || E > CANDLE_MOE_MAX_EXPERTS || d <= 0 || ff <= 0 || d % 256 || max_rows < 0 || max_rows > 128)
        return CANDLE_MOE_E_SHAPE;
    ExpertPtrs p1, p3;
    CM_TRY(fill_ptrs(w1p, E, p1));
    CM_TRY(fill_ptrs(w3p, E, p3));
    const cudaError_t e = launch_expert_direct((cudaStream_t)stream, true, p1, p3, dtype, E, d, ff, expert_offsets, row_of,
                                               max_rows, xq, xscales, xbsums, hidden, nullptr, 0, 1);
    return e == cudaErrorNotSupported ? CANDLE_MOE_E_SHAPE : rc(e);
}

int candle_moe_grouped_down_prepacked(void* stream, const void* const* w2p, int32_t dtype, int32_t E, int32_t d,
                                      int32_t ff, const uint32_t* expert_offsets, int64_t max_rows, const int8_t* hq,
                                      const float* hscales, const int16_t* hbsums, float* out) {
    if (!expert_offsets || !hq || !hscales || !hbsums || !out) return CANDLE_MOE_E_NULL;
    if (dtype != CANDLE_GGML_Q4K && dtype != CANDLE_GGML_Q6K) return CANDLE_MOE_E_DTYPE;
    if (E <= 0 || E > CANDLE_MOE_MAX_EXPERTS || d <= 0 || ff <= 0 || ff % 256 || max_rows < 0 || max_rows > 128)
        return CANDLE_MOE_E_SHAPE;
    ExpertPtrs p2;
    CM_TRY(fill_ptrs(w2p, E, p2));
    const cudaError_t e = launch_expert_direct((cudaStream_t)stream, false, p2, p2, dtype, E, ff, d, expert_offsets,
                                               nullptr, max_rows, hq, hscales, hbsums, out, nullptr, 0, 1);
    return e == cudaErrorNotSupported ? CANDLE_MOE_E_SHAPE : rc(e);
}

int candle_moe_device_status(int32_t* flags) {
    if (!flags) return CANDLE_MOE_E_NULL;
    int v = 0;
    const cudaError_t e = read_stream_status(&v);
    *flags = v;
    return rc(e);
}

int candle_moe_device_status_reset(void) {
    const cudaError_t e = cudaDeviceSynchronize();
    return e != cudaSuccess ? (int)e : rc(reset_stream_status());
}

int candle_moe_selftest_bounded_wait(void* stream, int32_t poll_limit) {
    if (poll_limit < 1 || poll_limit > (1 << 20)) return CANDLE_MOE_E_SHAPE;
    return rc(launch_selftest_wait((cudaStream_t)stream, poll_limit));
}

int candle_moe_rmsnorm(void* stream, const float* x, const float* weight, float eps, int64_t rows, int32_t d, float* y) {
    if (rows < 0 || d <= 0 || d % 4) return CANDLE_MOE_E_SHAPE;
    if (rows == 0) return CANDLE_MOE_OK;
    if (!x || !weight || !y) return CANDLE_MOE_E_NULL;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(weight) | reinterpret_cast<uintptr_t>(y)) & 15) return CANDLE_MOE_E_ALIGN;
    return rc(launch_rmsnorm((cudaStream_t)stream, x, weight, eps, rows, d, y));
}

int candle_moe_rope_kv_append(void* stream, const float* qkv, int64_t row_stride, const float* cos, const float* sin, int32_t batch,
                              int32_t n_head, int32_t n_kv_head, int32_t head_dim, int64_t max_seq, int32_t index_pos, float* q_out,
                              float* k_cache, float* v_cache) {
    if (batch < 0 || n_head <= 0 || n_kv_head <= 0 || head_dim <= 0 || head_dim % 2 || index_pos < 0 || index_pos >= max_seq ||
        row_stride < (int64_t)(n_head + 2 * n_kv_head) * head_dim)
        return CANDLE_MOE_E_SHAPE;
    if (batch == 0) return CANDLE_MOE_OK;
    if (!qkv || !cos || !sin || !q_out || !k_cache || !v_cache) return CANDLE_MOE_E_NULL;
    return rc(launch_rope_kv_append((cudaStream_t)stream, qkv, row_stride, cos, sin, batch, n_head, n_kv_head, head_dim, max_seq,
                                    index_pos, q_out, k_cache, v_cache));
}

int candle_moe_decode_attention_workspace_bytes(int32_t batch, int32_t n_head, int32_t head_dim, int32_t n_ctx, size_t* out_bytes) {
    if (!out_bytes) return CANDLE_MOE_E_NULL;
    if (batch < 0 || n_head <= 0 || head_dim <= 0 || n_ctx < 0) return CANDLE_MOE_E_SHAPE;
    *out_bytes = decode_attention_workspace_bytes(batch, n_head, head_dim, n_ctx);
    return CANDLE_MOE_OK;
}

int candle_moe_decode_attention(void* stream, const float* q, const float* k_cache, const float* v_cache, int32_t batch,
                                int32_t n_head, int32_t n_kv_head, int32_t head_dim, int64_t max_seq, int32_t n_ctx, float* out,
                                void* workspace, size_t workspace_bytes) {
    if (batch < 0 || n_head <= 0 || n_kv_head <= 0 || n_head % n_kv_head || head_dim <= 0 || n_ctx < 0 || n_ctx > max_seq)
        return CANDLE_MOE_E_SHAPE;
    if (batch == 0 || n_ctx == 0) return CANDLE_MOE_OK;
    if (!q || !k_cache || !v_cache || !out || !workspace) return CANDLE_MOE_E_NULL;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) |
         reinterpret_cast<uintptr_t>(workspace)) & 15)
        return CANDLE_MOE_E_ALIGN;
    if (workspace_bytes < decode_attention_workspace_bytes(batch, n_head, head_dim, n_ctx)) return CANDLE_MOE_E_WORKSPACE;
    const float scale = 1.0f / sqrtf((float)head_dim);
    const cudaError_t e = launch_decode_attention((cudaStream_t)stream, q, k_cache, v_cache, batch, n_head, n_kv_head, head_dim,
                                                  max_seq, n_ctx, scale, out, static_cast<float*>(workspace));
    return e == cudaErrorNotSupported ? CANDLE_MOE_E_SHAPE : rc(e);
}

int candle_moe_quantize_weights(void* stream, int32_t dtype, const float* src, int64_t n_elems, void* dst) {
    if (!src || !dst) return CANDLE_MOE_E_NULL;
    if (!dtype_supported(dtype)) return CANDLE_MOE_E_DTYPE;
    if (n_elems < 0 || n_elems % block_elems(dtype)) return CANDLE_MOE_E_SHAPE;
    if (reinterpret_cast<uintptr_t>(src) & 15) return CANDLE_MOE_E_ALIGN;
    return rc(launch_quantize_weights((cudaStream_t)stream, dtype, src, n_elems, dst));
}

int candle_moe_dequantize(void* stream, int32_t dtype, const void* blocks, int64_t n_elems, float* dst) {
    if (!blocks || !dst) return CANDLE_MOE_E_NULL;
    if (!dtype_supported(dtype)) return CANDLE_MOE_E_DTYPE;
    if (n_elems < 0 || n_elems % block_elems(dtype)) return CANDLE_MOE_E_SHAPE;
    return rc(launch_dequantize((cudaStream_t)stream, dtype, blocks, n_elems, dst));
}

// ---------------------------------------------------------------------------------------------------------
// Expert parallelism (experts sharded over ranks; the host issues the all-to-alls between these calls)
// ---------------------------------------------------------------------------------------------------------
int candle_moe_ep_row_bytes(int32_t d_model, size_t* out_bytes) {
    if (!out_bytes) return CANDLE_MOE_E_NULL;
    if (d_model <= 0 || d_model % 256) return CANDLE_MOE_E_SHAPE;
    *out_bytes = ep_row_bytes(d_model);
    return CANDLE_MOE_OK;
}

int candle_moe_ep_pack(void* stream, const uint32_t* perm_token, int64_t n_rows, int32_t d_model, const int8_t* xq,
                       const float* xscales, const int16_t* xbsums, void* send_rows) {
    if (n_rows < 0 || d_model <= 0 || d_model % 256) return CANDLE_MOE_E_SHAPE;
    if (n_rows == 0) return CANDLE_MOE_OK;
    if (!xq || !xscales || !xbsums || !send_rows) return CANDLE_MOE_E_NULL;
    if ((reinterpret_cast<uintptr_t>(xq) & 15) || (reinterpret_cast<uintptr_t>(send_rows) & 15)) return CANDLE_MOE_E_ALIGN;
    return rc(launch_ep_pack((cudaStream_t)stream, perm_token, n_rows, d_model, xq, xscales, xbsums, send_rows));
}

int candle_moe_ep_workspace_bytes(const candle_moe_weights_t* w, int64_t max_rows_total, size_t* out_bytes) {
    CM_TRY(check_weights(w));
    if (!out_bytes) return CANDLE_MOE_E_NULL;
    if (max_rows_total < 0 || max_rows_total > (int64_t)1 << 26) return CANDLE_MOE_E_SHAPE;
    if (w->dtype_w13 == CANDLE_GGML_Q8_0 || w->dtype_w2 == CANDLE_GGML_Q8_0) return CANDLE_MOE_E_DTYPE;
    // as for_every_batch: the slots of the partial outputs fall from 8 to 4 behind this many rows
    const int64_t few = std::min(max_rows_total, ep_many_slot_rows(w->n_experts));
    *out_bytes = std::max(ep_layout(w, max_rows_total, nullptr).total, ep_layout(w, few, nullptr).total);
    return CANDLE_MOE_OK;
}

int candle_moe_ep_experts(void* stream, const candle_moe_weights_t* w, const void* recv_rows, const uint32_t* recv_counts,
                          int32_t n_src, int64_t n_rows, int64_t max_rows_per_expert, float* out_rows, void* workspace,
                          size_t workspace_bytes) {
    CM_TRY(check_weights(w));
    if (w->dtype_w13 == CANDLE_GGML_Q8_0 || w->dtype_w2 == CANDLE_GGML_Q8_0) return CANDLE_MOE_E_DTYPE;
    if (n_rows < 0 || n_src <= 0 || (int64_t)n_src * w->n_experts > 1024 || max_rows_per_expert < 0 ||
        max_rows_per_expert > n_rows)
        return CANDLE_MOE_E_SHAPE;
    if (n_rows == 0) return CANDLE_MOE_OK;
    if (!recv_rows || !recv_counts || !out_rows || !workspace) return CANDLE_MOE_E_NULL;
    if ((reinterpret_cast<uintptr_t>(workspace) & 255) || (reinterpret_cast<uintptr_t>(recv_rows) & 15) ||
        (reinterpret_cast<uintptr_t>(out_rows) & 15))
        return CANDLE_MOE_E_ALIGN;
    const EpWorkspace ws = ep_layout(w, n_rows, workspace);
    if (workspace_bytes < ws.total) return CANDLE_MOE_E_WORKSPACE;
    const int E = w->n_experts, d = w->d_model;
    ExpertPtrs p1, p3, p2;
    CM_TRY(fill_ptrs(w->w1, E, p1));
    CM_TRY(fill_ptrs(w->w3, E, p3));
    CM_TRY(fill_ptrs(w->w2, E, p2));
    cudaStream_t st = (cudaStream_t)stream;
    CM_TRY(rc(launch_ep_regroup(st, recv_rows, recv_counts, n_src, E, n_rows, d, ws.plan, ws.xq, ws.xs, ws.xb, ws.offsets,
                                ws.back)));
    int eo_splits = 1;
    const int slots = ep_eo_slots(n_rows, E);
    CM_TRY(run_experts(st, w, p1, p3, p2, max_rows_per_expert, n_rows, ws.offsets, nullptr, ws.xq, ws.xs, ws.xb, ws.eb, slots,
                       &eo_splits, false, true, nullptr, 0));
    return rc(launch_ep_scatter(st, ws.eb.eo, eo_splits, n_rows * d, ws.back, n_rows, d, out_rows));
}

// ---------------------------------------------------------------------------------------------------------
// One quantized matrix over a batch of rows: QMatMul::forward for the dense projections of the model
// ---------------------------------------------------------------------------------------------------------
namespace {
struct QmmWorkspace {
    int8_t* xq;
    float* xs;
    int16_t* xb;
    uint32_t* offsets;
    float* eo;    // K-split partial outputs (null: the product writes `out` itself)
    int slots;
    void* gemm;
    size_t total;
};
// One group holds every row, so the row count is exact.  The tensor-core GEMM takes the product above 48 rows, and
// from 17 rows on when the matrix has enough 128-row tiles to fill the SMs by itself.  Both lines are those of a former GEMM ([4096, 4096]
// Q4_K at 32 rows 25 us against 23 through the streaming form); the present one is ahead below them too.  Streaming form / GEMM on the
// device, us, 17 and 48 rows: [1024, 4096] Q4_K 13 / 11, 15 / 13; [4096, 4096] 20 / 15, 26 / 15; [6144, 4096] 24 / 16, 33 / 17; [12800, 4096] 36 /
// 20, 51 / 23; [32000, 4096] Q6_K 103 / 45, 160 / 50.
inline bool qmm_takes_gemm(int dtype, int64_t rows, int n) {
    return dtype != CANDLE_GGML_Q8_0 && (rows > QMM_GEMM_MIN_ROWS || (rows > 16 && n >= 12800));
}
QmmWorkspace qmm_layout(int dtype, int64_t rows, int n, int k, void* base_) {
    uint8_t* base = static_cast<uint8_t*>(base_);
    QmmWorkspace ws{};
    size_t off = 0;
    ws.xq = carve<int8_t>(base, off, (size_t)rows * k);
    ws.xs = carve<float>(base, off, (size_t)rows * k / act_block(dtype));
    ws.xb = carve<int16_t>(base, off, (size_t)rows * k / 16);
    ws.offsets = carve<uint32_t>(base, off, 2);
    // decode-sized batches split K to fill the device (a [4096, 4096] matrix has 256 row tiles for 148 SMs x 16 warps)
    ws.slots = rows <= 64 && n % 4 == 0 ? MAX_K_SPLITS : 1;
    if (ws.slots > 1) ws.eo = carve<float>(base, off, (size_t)rows * n * ws.slots);
    if (qmm_takes_gemm(dtype, rows, n)) {
        off = align_up(off, 1024);
        ws.gemm = base ? base + off : reinterpret_cast<void*>(1);
        off += expert_gemm_scratch_bytes(rows, k);
    }
    ws.total = align_up(off, 256);
    return ws;
}
}  // namespace

int candle_moe_qmatmul_workspace_bytes(int32_t dtype, int64_t rows, int32_t n, int32_t k, size_t* out_bytes) {
    if (!out_bytes) return CANDLE_MOE_E_NULL;
    if (!dtype_supported(dtype)) return CANDLE_MOE_E_DTYPE;
    if (rows < 0 || rows > (int64_t)1 << 24 || n <= 0 || k <= 0 || k % block_elems(dtype)) return CANDLE_MOE_E_SHAPE;
    *out_bytes = qmm_layout(dtype, rows, n, k, nullptr).total;
    return CANDLE_MOE_OK;
}

int candle_moe_qmatmul(void* stream, const void* w, const void* w_prepacked, int32_t dtype, int32_t n, int32_t k,
                       const float* x, int64_t rows, float* out, void* workspace, size_t workspace_bytes) {
    if (!dtype_supported(dtype)) return CANDLE_MOE_E_DTYPE;
    if (rows < 0 || rows > (int64_t)1 << 24 || n <= 0 || k <= 0 || k % block_elems(dtype)) return CANDLE_MOE_E_SHAPE;
    if (rows == 0) return CANDLE_MOE_OK;
    if (!w || !x || !out || !workspace) return CANDLE_MOE_E_NULL;
    if ((reinterpret_cast<uintptr_t>(workspace) & 255) || (reinterpret_cast<uintptr_t>(x) & 15) ||
        (reinterpret_cast<uintptr_t>(out) & 15))
        return CANDLE_MOE_E_ALIGN;
    const QmmWorkspace ws = qmm_layout(dtype, rows, n, k, workspace);
    if (workspace_bytes < ws.total) return CANDLE_MOE_E_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    ExpertPtrs pw{}, pp{};
    pw.p[0] = static_cast<const uint8_t*>(w);
    pp.p[0] = static_cast<const uint8_t*>(w_prepacked);
    const bool rp = dtype == CANDLE_GGML_Q6K && w_prepacked;
    const bool large = ws.gemm && gemm_enabled() && expert_gemm_takes(false, dtype, rp, k, n, rows);
    // the quantizer -- with the GEMM the preparation of its operand -- also writes the offsets of the one group that holds
    // every row
    if (!large) CM_TRY(rc(launch_quantize_act(st, x, rows, k, dtype, ws.xq, ws.xs, ws.xb, nullptr, ws.offsets)));
    float* dst = ws.eo ? ws.eo : out;
    const int64_t stride = rows * (int64_t)n;
    int splits = 1;
    bool done = false;
    // The decode kernels over the repacked copy of a k-quant are not used here: with a single group their tiles are too few and
    // too short, and the streaming form over the GGUF blocks is faster (measured, [4096, 4096] Q4_K / [32000, 4096]
    // Q6_K: 1 row 10.8 / 44.5 us against 17.2 / 46.2; 8 rows 13.5 / 48.6 against 17.7 / 60.1).
    // (a copy made by candle_moe_prepack is 16-byte aligned; anything else is left alone)
    if (dtype == CANDLE_GGML_Q8_0 && w_prepacked && !(reinterpret_cast<uintptr_t>(w_prepacked) & 15) && rows <= QMM_DIRECT_MAX_ROWS) {
        const cudaError_t ce = launch_expert_direct(st, false, pp, pp, dtype, 1, k, n, ws.offsets, nullptr, rows, ws.xq, ws.xs, ws.xb,
                                                    dst, &splits, stride, ws.slots, 1, rows, out);
        if (ce == cudaSuccess)
            done = true;
        else if (ce != cudaErrorNotSupported)
            return (int)ce;
        else
            splits = 1;
    }
    if (large) {
        CM_TRY(rc(launch_expert_gemm(st, false, rp ? pp : pw, rp ? pp : pw, dtype, rp, 1, k, n, ws.offsets, nullptr, rows, rows, ws.xq,
                                     ws.xs, ws.xb, dst, ws.gemm, ws.slots, &splits, stride, out, x, ws.offsets)));
        done = true;
    }
    if (!done)
        CM_TRY(rc(launch_grouped_down(st, pw, dtype, 1, n, k, ws.offsets, rows, ws.xq, ws.xs, ws.xb, dst, stride, ws.slots,
                                      &splits, out)));
    // partial sums only when K was split: an unsplit product has written `out` itself (one launch fewer: [6144, 4096] Q4_K,
    // 1 row 21.1 -> 18.7 us, [32000, 4096] Q6_K, 32 rows 76.5 -> 73.0 us)
    if (splits > 1) return rc(launch_ep_scatter(st, ws.eo, splits, stride, nullptr, rows, n, out));
    return CANDLE_MOE_OK;
}

}  // extern "C"
