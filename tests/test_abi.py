"""CPU-side checks of the drop-in boundary: the shared library loads, exports every symbol the
header declares, and rejects bad arguments on the host before anything touches a GPU."""
import ctypes as C
import os
import re

import pytest

from tests import helpers as H

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    from candle_b200.csrc import build as b
    b.build()
    from candle_b200 import _lib
    return _lib


def _declared_symbols():
    src = open(os.path.join(ROOT, "include", "candle_moe.h")).read()
    return sorted(set(re.findall(r"CANDLE_MOE_API\s+[\w\s\*]+?\b(candle_moe_\w+)\s*\(", src)))


def test_header_symbols_are_exported(lib):
    names = _declared_symbols()
    assert len(names) >= 12
    handle = C.CDLL(lib.LIB_PATH)
    for n in names:
        assert hasattr(handle, n), f"{n} declared in include/candle_moe.h but not exported"
    assert set(names) == set(lib.SYMBOLS), "ctypes prototypes and header disagree"
    assert lib.load().candle_moe_version().startswith(b"candle_moe_sm100")


def _weights(lib, **kw):
    w = lib.MoeWeightsC()
    w.d_model, w.d_ff, w.n_experts, w.top_k, w.renorm = 4096, 14336, 8, 2, 1
    w.dtype_w13, w.dtype_w2 = 12, 14
    for k, v in kw.items():
        setattr(w, k, v)
    return w


def test_workspace_query_is_host_only_and_monotonic(lib):
    L = lib.load()
    out = C.c_size_t(0)
    sizes = []
    for T in (0, 1, 8, 32, 2048):
        assert L.candle_moe_workspace_bytes(C.byref(_weights(lib)), T, C.byref(out)) == 0
        sizes.append(out.value)
    assert sizes == sorted(sizes) and sizes[-1] > 2048 * 2 * 14336 * 4
    # hidden f32 + its int8 copy dominate: [T*k, ff] * 5 bytes; two K-split slots of [T*k, d] f32
    assert sizes[-1] < 2048 * 2 * (14336 * 6 + 4096 * 20) + (1 << 20)


@pytest.mark.parametrize("kw", [{}, {"copies": True}, {"dtype_w13": 14}, {"dtype_w13": 8, "dtype_w2": 8, "n_experts": 60, "top_k": 4, "d_ff": 1408,
                                                                         "d_model": 2048, "d_ff_shared": 5632, "dtype_shared13": 8, "dtype_shared2": 8}])
def test_a_workspace_for_many_rows_holds_every_smaller_batch(lib, kw):
    """Around the row counts where the number of partial outputs falls (96 rows; 2048 selections where Q6_K is repacked on
    its way; expert parallelism 2048, 64 per expert)."""
    L, kw = lib.load(), dict(kw)
    table = (C.c_void_p * 128)(*[4096] * 128)
    if kw.pop("copies", False):
        kw.update(w1_prepacked=table, w3_prepacked=table, w2_prepacked=table)
    w, out = _weights(lib, **kw), C.c_size_t(0)
    for query, rows in ((L.candle_moe_workspace_bytes, (1, 31, 95, 96, 97, 100, 191, 193, 400, 511, 513, 1023, 1024, 1025, 1100, 2000, 4096)),
                        (L.candle_moe_ffn_layer_workspace_bytes, (1, 95, 96, 97, 130, 500, 1024, 1025)),
                        (L.candle_moe_ep_workspace_bytes, (1, 32, 33, 511, 513, 2047, 2048, 2049, 3000, 3841, 5000))):
        if query is L.candle_moe_ep_workspace_bytes and w.dtype_w13 == 8:
            continue
        sizes = []
        for T in rows:
            assert query(C.byref(w), T, C.byref(out)) == 0
            sizes.append(out.value)
        assert sizes == sorted(sizes), query.__name__


@pytest.mark.parametrize("E,k,d,ff,T,taken", [
    (8, 2, 1536, 2560, 200, True),     # 50 rows per expert, 3.9 million weights a matrix
    (16, 2, 2560, 5120, 200, True),
    (4, 2, 4096, 6144, 400, True),     # instead of the streaming form
    (60, 2, 1536, 1536, 200, False),   # 7 rows each: five launches per expert cost more than the rows do
    (60, 1, 1536, 1536, 200, False),
    (60, 4, 1536, 1536, 400, True),    # 27 rows each
    (128, 2, 512, 1024, 400, False),   # 640 launches
    (60, 4, 2048, 2048, 1600, False),  # the streaming form passes over small matrices faster than they are repacked
    (8, 2, 4096, 6144, 240, False),    # 60 rows each: the streaming form passes over a matrix four times in less
])
def test_q6k_without_copies_is_repacked_only_where_the_rows_pay_for_it(lib, E, k, d, ff, T, taken):
    """Whether a batch asks for room for one expert's repacked matrices (row counts whose own size is not below that of a
    smaller batch)."""
    w = _weights(lib, dtype_w13=14, dtype_w2=14, n_experts=E, top_k=k, d_model=d, d_ff=ff, router=4096)
    out = C.c_size_t(0)
    assert lib.load().candle_moe_workspace_bytes(C.byref(w), T, C.byref(out)) == 0
    assert (out.value > H.smallest_workspace(lib, w, T)) == taken


@pytest.mark.parametrize("field,value,code", [
    ("d_model", 4000, -2),        # not a multiple of 256 for Q4K
    ("d_ff", 100, -2),
    ("n_experts", 129, -2),
    ("top_k", 9, -2),
    ("top_k", 0, -2),
    ("dtype_w13", 2, -3),         # Q4_0 is not on this path
    ("dtype_w2", 15, -3),
])
def test_bad_shapes_and_dtypes_are_rejected(lib, field, value, code):
    out = C.c_size_t(0)
    assert lib.load().candle_moe_workspace_bytes(C.byref(_weights(lib, **{field: value})), 8, C.byref(out)) == code


def test_null_pointers_are_rejected_before_any_launch(lib):
    L = lib.load()
    w = _weights(lib)
    assert L.candle_moe_forward(None, C.byref(w), None, 4, None, None, 0) == -1
    assert L.candle_moe_router_topk(None, None, None, None, 4, 4096, 8, 2, 1, None, None) == -1
    assert L.candle_moe_permute(None, None, 4, 2, 8, None, None, None, None) == -1
    assert L.candle_moe_quantize_act(None, None, 4, 4096, 12, None, None, None) == -1
    assert L.candle_moe_combine(None, None, None, None, None, 4, 2, 4096, None, None, None, None) == -1
    assert L.candle_moe_quantize_weights(None, 12, None, 256, None) == -1
    assert L.candle_moe_workspace_bytes(None, 4, C.byref(C.c_size_t())) == -1
    # zero rows is a no-op, like an empty tensor through Module::forward
    one = C.c_float(0)
    w.router = C.cast(C.byref(one), C.c_void_p)
    assert L.candle_moe_forward(None, C.byref(w), C.byref(one), 0, C.byref(one), None, 0) == 0


def test_error_type_carries_status(lib):
    with pytest.raises(lib.CandleMoeError) as ei:
        lib.check("candle_moe_forward", -4)
    assert ei.value.status == -4 and "WORKSPACE" in str(ei.value)


def test_host_mirror_rejects_cpu_tensors(lib):
    import torch
    from candle_b200 import GgmlDType, QTensor
    with pytest.raises(ValueError):
        QTensor(torch.zeros(144, dtype=torch.uint8), GgmlDType.Q4K, (1, 256))
    assert GgmlDType.Q4K.type_size() == 144 and GgmlDType.Q6K.type_size() == 210 and GgmlDType.Q8_0.type_size() == 34


def test_tuning_switches_round_trip(lib):
    L = lib.load()
    v = C.c_int64(-1)
    assert L.candle_moe_get_tuning(lib.TUNE_GEMM_MIN_ROWS, C.byref(v)) == 0
    old = v.value
    assert L.candle_moe_set_tuning(lib.TUNE_GEMM_MIN_ROWS, 77) == 0
    assert L.candle_moe_get_tuning(lib.TUNE_GEMM_MIN_ROWS, C.byref(v)) == 0 and v.value == 77
    assert L.candle_moe_set_tuning(lib.TUNE_GEMM_MIN_ROWS, old) == 0
    assert L.candle_moe_set_tuning(99, 1) == -2 and L.candle_moe_get_tuning(99, C.byref(v)) == -2


def test_the_benchmark_counts_the_kernels_of_the_form_that_runs(lib):
    """Launches of a layer on either side of the rows from which the GEMM takes it, which the library names."""
    import bench
    L, some = lib.load(), (C.c_void_p * 8)(*[4096] * 8)
    rows = C.c_int64(0)
    cfg = {"dt13": 12, "dt2": 14, "E": 8, "k": 2, "ff_shared": 0}
    w = _weights(lib, w1_prepacked=some, w3_prepacked=some, w2_prepacked=some)
    assert L.candle_moe_forward_gemm_rows(C.byref(w), C.byref(rows)) == 0 and 32 < rows.value < 96
    # router, dispatch, gate_up, quantizer, down, combine; with the GEMM two preparations in place of the quantizer
    assert bench.block_launches(cfg, rows.value, True, w) == 6
    assert bench.block_launches(cfg, rows.value + 1, True, w) == 7
    assert bench.block_launches(cfg, 1, True, w) == 5
    old = C.c_int64(0)
    assert L.candle_moe_get_tuning(lib.TUNE_GEMM_ENABLED, C.byref(old)) == 0
    try:
        assert L.candle_moe_set_tuning(lib.TUNE_GEMM_ENABLED, 0) == 0
        assert bench.block_launches(cfg, rows.value + 1, True, w) == 6
    finally:
        assert L.candle_moe_set_tuning(lib.TUNE_GEMM_ENABLED, old.value) == 0
    assert L.candle_moe_forward_gemm_rows(C.byref(_weights(lib, top_k=9)), C.byref(rows)) == -2
    assert L.candle_moe_forward_gemm_rows(C.byref(w), None) == -1


def _line(lib, E, k, d, ff, dt13, dt2, copies=True, fs=0):
    """rows above which the GEMM takes a layer"""
    some = (C.c_void_p * E)(*[4096] * E)
    w = _weights(lib, n_experts=E, top_k=k, d_model=d, d_ff=ff, dtype_w13=dt13, dtype_w2=dt2)
    if copies:
        w.w1_prepacked = w.w3_prepacked = w.w2_prepacked = some
    if fs:
        w.d_ff_shared, w.dtype_shared13, w.dtype_shared2 = fs, 8, 8
        w.shared_w1_prepacked = w.shared_w3_prepacked = w.shared_w2_prepacked = 4096
    rows = C.c_int64(0)
    assert lib.load().candle_moe_forward_gemm_rows(C.byref(w), C.byref(rows)) == 0
    return rows.value


# rows that were measured faster on the decode kernels, and on the GEMM
@pytest.mark.parametrize("E,k,d,ff,fs,decode,gemm", [
    (60, 4, 2048, 1408, 5632, 160, 224), (60, 2, 2048, 1408, 5632, 224, 352), (60, 2, 2048, 1408, 0, 272, 448), (32, 2, 2048, 1408, 5632, 144, 224),
    (32, 2, 2048, 1408, 0, 160, 224), (16, 1, 2048, 1408, 5632, 144, 192), (16, 2, 4096, 4096, 0, 96, 128), (16, 1, 4096, 4096, 0, 192, 272),
    (64, 8, 3584, 2560, 0, 97, 128), (128, 8, 2048, 768, 2816, 128, 192), (128, 1, 1024, 1024, 4096, 96, 272), (32, 4, 1024, 1024, 0, 96, 112),
])
def test_line_of_q80_layers(lib, E, k, d, ff, fs, decode, gemm):
    assert decode <= _line(lib, E, k, d, ff, 8, 8, fs=fs) < gemm


@pytest.mark.parametrize("E,k,d,ff,dt13,dt2,decode,gemm", [
    (8, 2, 4096, 14336, 12, 14, 60, 64), (8, 2, 4096, 14336, 12, 12, 56, 64), (8, 2, 4096, 14336, 14, 14, 0, 49), (8, 2, 2048, 8192, 12, 14, 58, 64),
    (8, 2, 2560, 6144, 12, 14, 60, 64), (8, 2, 2560, 6144, 14, 14, 56, 62), (8, 2, 1024, 3584, 12, 14, 54, 64), (8, 2, 1024, 3584, 12, 12, 0, 54),
    (4, 2, 4096, 14336, 12, 14, 28, 34), (60, 8, 2048, 1536, 12, 14, 96, 97), (16, 4, 2048, 1024, 12, 14, 0, 50), (16, 8, 2048, 2048, 12, 14, 0, 28),
])
def test_line_of_k_quant_layers_over_copies(lib, E, k, d, ff, dt13, dt2, decode, gemm):
    assert decode <= _line(lib, E, k, d, ff, dt13, dt2) < gemm


@pytest.mark.parametrize("E,k,d,ff,decode,gemm", [
    (8, 2, 1024, 3584, 8, 12), (8, 2, 4096, 4096, 8, 12), (8, 4, 4096, 4096, 8, 10), (16, 8, 4096, 4096, 8, 10), (128, 8, 2048, 768, 8, 60), (64, 8, 2048, 1024, 8, 40),
    (4, 2, 4096, 4096, 8, 16), (4, 2, 4096, 14336, 8, 10), (3, 1, 4096, 4096, 14, 28), (2, 1, 2048, 4096, 8, 20), (3, 1, 1024, 1024, 42, 97), (8, 2, 512, 512, 48, 97),
    (8, 2, 512, 1024, 20, 48), (32, 4, 512, 512, 32, 96),
])
def test_line_of_q4k_layers_without_copies(lib, E, k, d, ff, decode, gemm):
    assert decode <= _line(lib, E, k, d, ff, 12, 12, copies=False) < gemm


@pytest.mark.parametrize("T,k", [(2 ** 32, 1), (2 ** 29, 8), (2 ** 61, 8)])
def test_dispatch_of_more_selections_than_its_lists_can_number_is_refused(lib, T, k):
    assert lib.load().candle_moe_permute(None, 4096, T, k, 8, 4096, 4096, 4096, 4096) == -2


@pytest.mark.parametrize("n", [1, 127, 128, 129, 2 ** 31, 2 ** 32 - 129, 2 ** 32 - 128, 2 ** 32 - 127, 2 ** 32 - 1])
def test_rounds_of_the_small_dispatch_end_at_every_length(n):
    """permute_kernel's loop in its own 32-bit arithmetic: the condition as the source has it, at the first and the last rounds."""
    src = open(os.path.join(ROOT, "candle_b200", "csrc", "routing.cu")).read()
    kernel = src[src.index("permute_kernel(const"):src.index("permute_count_kernel(")]
    loops = re.findall(r"for \(([^;]*; [^;]*; [^)]*i0 \+= 128)\)", kernel)
    assert len(loops) == 2 and len(set(loops)) == 1
    m = 2 ** 32
    rounds = (n + 127) // 128
    last = (rounds - 1) * 128 + 31  # i0 of the last lane there
    if "round < rounds" in loops[0]:
        assert "rounds = (uint32_t)((n_pairs + 127) / 128)" in kernel
    else:  # an index against n: behind the last round it must not have wrapped
        assert "i0 - lane < n" in loops[0] and (last + 128 - 31) % m >= n
    assert last + 96 < m  # no index of the last round wraps


def test_every_line_of_the_gemm_can_be_chosen(lib):
    """96 rows, the line of everything that does not go by the rows of an expert, is a fixed line like any other when it is
    set: a layer over copies then has no GEMM scratch at 90 rows, and has it again when the value found before is put back."""
    L, out, v = lib.load(), C.c_size_t(0), C.c_int64(-1)
    some = (C.c_void_p * 8)(*[4096] * 8)
    w = _weights(lib, w1_prepacked=some, w3_prepacked=some, w2_prepacked=some)

    def size(T):
        assert L.candle_moe_workspace_bytes(C.byref(w), T, C.byref(out)) == 0
        return out.value

    auto = size(90)
    assert L.candle_moe_get_tuning(lib.TUNE_GEMM_MIN_ROWS, C.byref(v)) == 0
    old = v.value
    try:
        sizes = {}
        for line in (95, 96, 97):
            assert L.candle_moe_set_tuning(lib.TUNE_GEMM_MIN_ROWS, line) == 0
            sizes[line] = size(90)
        assert sizes[95] == sizes[96] == sizes[97] < auto
    finally:
        assert L.candle_moe_set_tuning(lib.TUNE_GEMM_MIN_ROWS, old) == 0
    assert size(90) == auto


def _ep_cfg(lib, **kw):
    cfg = lib.EpConfigC()
    cfg.rank, cfg.world, cfg.n_experts_global, cfg.top_k, cfg.renorm, cfg.max_tokens = 0, 2, 8, 2, 1, 32
    one = C.c_float(0)
    cfg.router = C.cast(C.pointer(one), C.c_void_p)
    for k, v in kw.items():
        setattr(cfg, k, v)
    return cfg, one


def test_expert_parallel_geometry_is_host_only(lib):
    """Form and workspace of candle_moe_ep_forward follow from the configuration alone (no device, no NCCL)."""
    L = lib.load()
    local = _weights(lib, n_experts=4)
    form, cap, need = C.c_int32(0), C.c_int64(0), C.c_size_t(0)
    cfg, keep = _ep_cfg(lib)
    assert L.candle_moe_ep_forward_form(C.byref(cfg), C.byref(local), C.byref(form), C.byref(cap)) == 0
    assert (form.value, cap.value) == (1, 64)  # decode-sized step: slots of max_tokens * min(k, local experts) rows
    assert L.candle_moe_ep_forward_workspace_bytes(C.byref(cfg), C.byref(local), C.byref(need)) == 0 and need.value > 0
    from candle_b200.expert_parallel import choose_form
    for world, tokens, d in ((2, 32, 4096), (8, 32, 4096), (2, 4096, 6144), (4, 2048, 6144), (8, 1024, 4096)):
        cfg, keep = _ep_cfg(lib, world=world, max_tokens=tokens)
        local = _weights(lib, n_experts=8 // world, top_k=min(2, 8 // world), d_model=d, d_ff=16384)
        assert L.candle_moe_ep_forward_form(C.byref(cfg), C.byref(local), C.byref(form), C.byref(cap)) == 0
        assert form.value == choose_form(world, tokens, 2, 8 // world, d)[0]
    # ranks must divide the experts; Q8_0 experts have no expert-parallel form; a missing communicator is refused
    cfg, keep = _ep_cfg(lib, world=3)
    assert L.candle_moe_ep_forward_form(C.byref(cfg), C.byref(_weights(lib, n_experts=4)), C.byref(form), None) == -2
    cfg, keep = _ep_cfg(lib)
    assert L.candle_moe_ep_forward_form(C.byref(cfg), C.byref(_weights(lib, n_experts=4, dtype_w13=8, d_model=4096)),
                                        C.byref(form), None) == -3
