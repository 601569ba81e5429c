"""Which kernels take a batch of a single-device forward: the rows on either side of the rule's lines (candle_moe_api.cu, gemm_rows),
with repacked copies and without, against the oracle; the narrow GEMM tiles whose Q4_K min term has its own
accumulator; the dispatch lists."""
import ctypes as C

import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu


def _check(orc, torch, cfg, T, prepack):
    from candle_b200 import _lib
    blk, mw = H.random_device_block(orc, torch, cfg, 5)
    if prepack:
        blk.prepack()
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn((T, cfg["d"]), generator=g, device="cuda", dtype=torch.float32)
    y = blk.forward(x).clone()
    assert torch.equal(y, blk.forward(x))
    v = C.c_int32(-1)
    assert _lib.load().candle_moe_device_status(C.byref(v)) == 0 and v.value == 0
    xs = x.cpu().numpy()
    ref = orc.moe_forward(mw, xs)
    ids = blk.last_routing(T)[0].numpy().astype(np.uint32)
    probs = orc.router_topk(xs, mw.router, cfg["k"], cfg["renorm"], mw.router_bias)[0]
    H.check_routing(probs, ref.topk_ids, ids)
    same = (ref.topk_ids == ids).all(axis=1)
    assert H.max_rel(y.cpu().numpy()[same], ref.y[same]) <= H.MAX_REL_TOL
    assert H.rel_l2(y.cpu().numpy()[same], ref.y[same]) <= H.REL_L2_TOL
    return blk, x, y


def _cfg(dt13, dt2, E, k, d=512, ff=1024, fs=0):
    return dict(d=d, ff=ff, E=E, k=k, dt13=dt13, dt2=dt2, renorm=True, ff_shared=fs, zipf=False)


@pytest.mark.parametrize("dt13,dt2,prepack,E,k,rows", [
    (12, 14, True, 8, 2, (48, 56, 57, 96, 97)),  # 14 rows of an expert
    (12, 12, True, 8, 2, (52, 53)),           # 13
    (14, 14, True, 8, 2, (48, 56, 57)),
    (12, 14, True, 16, 4, (48, 49)),          # 12
    (12, 12, True, 3, 2, (18, 19, 96)),       # few experts: wide tiles, the old line
    (12, 12, False, 8, 2, (10, 11, 32, 33, 64)),  # GGUF blocks, a small layer: 8 rows of an expert
    (12, 12, False, 32, 8, (8, 10, 11, 40)),  # 2.5; four chunks of tensor maps
    (12, 12, False, 4, 1, (9, 64)),           # few experts of a small layer: the old line
    (12, 14, False, 8, 2, (11, 33, 96)),      # the down product stays where it was
    (14, 12, False, 8, 2, (11, 96)),
    (8, 8, True, 32, 4, (97, 176, 177)),      # 22 rows of an expert
    (8, 8, False, 32, 4, (97,)),
])
def test_rows_on_either_side_of_the_lines(orc, torch_cuda, dt13, dt2, prepack, E, k, rows):
    for T in rows:
        _check(orc, torch_cuda, _cfg(dt13, dt2, E, k, fs=512 if dt13 == 8 and prepack else 0), T, prepack)


@pytest.mark.parametrize("dt13,dt2,prepack", [(12, 14, True), (12, 12, False)])
def test_smallest_workspace_of_a_batch_stays_enough(orc, torch_cuda, dt13, dt2, prepack):
    """Up to 96 rows the GEMM's operand scratch is optional: a workspace without it is taken, by the other kernels."""
    torch = torch_cuda
    from candle_b200 import _lib
    lib, T = _lib.load(), 64
    blk, x, y = _check(orc, torch, _cfg(dt13, dt2, 8, 2), T, prepack)
    w = blk._cw
    small, full = H.smallest_workspace(_lib, w, T), C.c_size_t(0)
    assert lib.candle_moe_workspace_bytes(C.byref(w), T, C.byref(full)) == 0
    assert small < full.value
    ws = torch.empty(small, dtype=torch.uint8, device="cuda")
    out = torch.empty_like(y)
    assert lib.candle_moe_forward(torch.cuda.current_stream().cuda_stream, C.byref(w), x.data_ptr(), T, out.data_ptr(), ws.data_ptr(), small) == 0
    # the hidden rows are quantized to int8 in between: the bound of two orders of the f32 sums
    assert H.rel_l2(out.cpu().numpy(), y.cpu().numpy()) <= H.REL_L2_TOL


@pytest.mark.parametrize("rows,n,k", [(17, 12800, 256), (32, 12800, 2304), (33, 12800, 768), (49, 256, 4096), (64, 1024, 1024), (65, 1024, 1024)])
def test_min_term_of_narrow_tiles(torch_cuda, rows, n, k):
    """Q4_K products with the min term in its own accumulator (tiles of up to 64 positions) and joined (65 rows), rows of zeros and
    of one value included (d = 0, a min term alone), against 64-bit arithmetic on the same int8 rows.  A sum of K / 256 block
    terms, each rounded a few times, of values that cancel to about a third: 4 sqrt(K / 256) 2^-24."""
    torch = torch_cuda
    from candle_b200 import GgmlDType, QMatMul, QTensor, _lib
    g = torch.Generator(device="cuda").manual_seed(n + k)
    w = torch.randn((n, k), generator=g, device="cuda") * 0.02
    w[3] = 0.0
    w[5] = -0.01
    w[6, :256] = -0.01
    q = QTensor.quantize(w, GgmlDType.Q4K)
    x = torch.randn((rows, k), generator=g, device="cuda")
    qs, sc = torch.empty((rows, k), dtype=torch.int8, device="cuda"), torch.empty((rows, k // 256), device="cuda")
    bs = torch.empty((rows, k // 16), dtype=torch.int16, device="cuda")
    assert _lib.load().candle_moe_quantize_act(torch.cuda.current_stream().cuda_stream, x.data_ptr(), rows, k, 12, qs.data_ptr(), sc.data_ptr(),
                                               bs.data_ptr()) == 0
    a = (qs.double().view(rows, -1, 256) * sc.double()[:, :, None]).view(rows, k)
    ref = a @ q.dequantize().double().to("cuda").T
    got = QMatMul(q).forward(x).double()
    assert torch.isfinite(got).all()
    assert float((got - ref).norm() / ref.norm()) < 4 * (k / 256) ** 0.5 * 2 ** -24
    for r in (3, 5, 6):
        assert float((got[:, r] - ref[:, r]).abs().max()) <= 1e-5 * max(1.0, float(ref[:, r].abs().max()))


@pytest.mark.parametrize("T,k,E", [(1, 1, 1), (127, 1, 2), (16, 8, 32), (43, 3, 33), (129, 1, 128), (256, 8, 60), (257, 8, 60), (600, 4, 128),
                                   (4096, 1, 5), (1537, 3, 8)])
def test_dispatch_lists(torch_cuda, T, k, E):
    """The dispatch by one CTA against a stable sort: part of a load round, whole ones, one expert to a lane group and beyond."""
    torch = torch_cuda
    from candle_b200 import _lib
    rng = np.random.default_rng(T + E)
    ids = np.stack([rng.choice(E, size=k, replace=False) for _ in range(T)]).astype(np.uint32)
    d = torch.from_numpy(ids.astype(np.int32)).cuda()
    counts, offsets = torch.full((E,), -1, dtype=torch.int32, device="cuda"), torch.full((E + 1,), -1, dtype=torch.int32, device="cuda")
    perm, pos = torch.full((T * k,), -1, dtype=torch.int32, device="cuda"), torch.full((T * k,), -1, dtype=torch.int32, device="cuda")
    assert _lib.load().candle_moe_permute(torch.cuda.current_stream().cuda_stream, d.data_ptr(), T, k, E, counts.data_ptr(), offsets.data_ptr(),
                                          perm.data_ptr(), pos.data_ptr()) == 0
    order = np.argsort(ids.reshape(-1), kind="stable")
    assert (counts.cpu().numpy() == np.bincount(ids.reshape(-1), minlength=E)).all()
    assert (offsets.cpu().numpy() == np.concatenate([[0], np.cumsum(np.bincount(ids.reshape(-1), minlength=E))])).all()
    assert (perm.cpu().numpy() == order // k).all()
    assert (pos.cpu().numpy()[order] == np.arange(T * k)).all()


@pytest.mark.parametrize("T,k,E", [(257, 8, 60), (1537, 3, 8), (2561, 1, 3), (640, 8, 128)])
def test_dispatch_lists_of_a_large_batch(orc, torch_cuda, T, k, E):
    """The same inside a block with more than 2048 selections: chunks of 512, the last one whole or not, more chunks than a round of
    the scan loads."""
    torch = torch_cuda
    blk, _ = H.random_device_block(orc, torch, _cfg(12, 12, E, k, d=256, ff=256), 1)
    x = torch.randn((T, 256), generator=torch.Generator(device="cuda").manual_seed(T), device="cuda")
    blk.forward(x)
    ids, _, counts, perm = (v.cpu().numpy() for v in blk.last_routing(T))
    flat = ids.reshape(-1).astype(np.int64)
    assert (counts[:E] == np.bincount(flat, minlength=E)).all()
    assert (perm.reshape(-1)[:T * k] == np.argsort(flat, kind="stable") // k).all()


def _tuned(key, value, fn):
    """fn() with a kernel-selection switch set"""
    from candle_b200 import _lib
    L, old = _lib.load(), C.c_int64(0)
    assert L.candle_moe_get_tuning(key, C.byref(old)) == 0 and L.candle_moe_set_tuning(key, value) == 0
    try:
        return fn()
    finally:
        assert L.candle_moe_set_tuning(key, old.value) == 0


@pytest.mark.parametrize("cfg,T", [
    (_cfg(8, 8, 8, 1, d=5120, ff=1024), 100),         # gate_up: sixteen rows of 5120 and the rings are more than shared memory
    (_cfg(8, 8, 8, 1, d=512, ff=1024, fs=20480), 100),  # the shared expert's down product, four splits of 5120
])
def test_products_that_the_decode_kernels_refuse_go_to_the_gemm(orc, torch_cuda, cfg, T):
    """Q8_0 batches above 96 rows which the line leaves to the decode kernels: without the GEMM the refused product is the tile kernel's
    over the GGUF blocks, whose sums run in another order."""
    from candle_b200 import _lib
    blk, x, y = _check(orc, torch_cuda, cfg, T, True)
    rows = C.c_int64(0)
    assert _lib.load().candle_moe_forward_gemm_rows(C.byref(blk._cw), C.byref(rows)) == 0 and rows.value >= T
    tiles = _tuned(_lib.TUNE_GEMM_ENABLED, 0, lambda: blk.forward(x).clone())
    assert not torch_cuda.equal(y, tiles)
    assert H.rel_l2(y.cpu().numpy(), tiles.cpu().numpy()) <= H.REL_L2_TOL


@pytest.mark.parametrize("bad,status", [(None, -1), (8, -5)])
def test_bad_tables_of_copies_are_refused_on_either_side_of_the_line(orc, torch_cuda, bad, status):
    """A missing or misaligned entry among the copies of a Q4_K layer: an error up to 96 rows, also where the GEMM, which reads the
    GGUF blocks, takes the batch; beyond, the tables are not looked at."""
    torch = torch_cuda
    from candle_b200 import _lib
    blk, _ = H.random_device_block(orc, torch, _cfg(12, 12, 8, 2), 5)
    blk.prepack()
    lib, table = _lib.load(), blk._cw.w3_prepacked
    keep = table[7]
    for T, expected in ((16, status), (64, status), (96, status), (97, 0)):
        x = torch.randn((T, 512), device="cuda")
        y, ws = torch.empty_like(x), torch.empty(blk.workspace_bytes(T) + 256, dtype=torch.uint8, device="cuda")
        at = (ws.data_ptr() + 255) // 256 * 256
        run = lambda: lib.candle_moe_forward(torch.cuda.current_stream().cuda_stream, C.byref(blk._cw), x.data_ptr(), T, y.data_ptr(), at,
                                             ws.numel() - 256)
        table[7] = None if bad is None else keep + bad
        assert run() == expected, T
        table[7] = keep
        assert run() == 0, T
    torch.cuda.synchronize()
