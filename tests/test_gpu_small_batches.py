"""The small-batch router (whole dot products per warp, optional norm, single-token dispatch) at the edges of its rule, and
the operand preparation that quantizes f32 rows itself against the two-pass form."""
import ctypes as C

import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,k", [(1, 1), (4, 2), (5, 3), (8, 2), (9, 4), (16, 8), (17, 2), (33, 4), (128, 8)])
def test_router_at_the_edges_of_its_forms(orc, torch_cuda, E, k):
    torch = torch_cuda
    from candle_b200 import _lib
    # rows of few float4s, of an odd number, the longest of the small form and one beyond; the last count takes the other form
    for d in (4, 36, 1028, 4096, 10240, 10244):
        for T in (1, 64, 65) if d <= 1028 else (148, 149, 256, 257) if d == 4096 and E in (8, 17, 33) else (3,):
            rng = np.random.default_rng(E + d + T)
            x = rng.standard_normal((T, d), dtype=np.float32)
            wg = rng.standard_normal((E, d), dtype=np.float32) * np.float32(0.05)
            probs, ids_ref, w_ref = orc.router_topk(x, wg, k, True, None)
            xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(wg).cuda()
            ids = torch.empty((T, k), dtype=torch.int32, device="cuda")
            w = torch.empty((T, k), dtype=torch.float32, device="cuda")
            assert _lib.load().candle_moe_router_topk(torch.cuda.current_stream().cuda_stream, xd.data_ptr(), wd.data_ptr(), None, T, d, E, k,
                                                      1, ids.data_ptr(), w.data_ptr()) == 0
            got = ids.cpu().numpy().astype(np.uint32)
            H.check_routing(probs, ids_ref, got)
            same = (ids_ref == got).all(axis=1)
            # logits are sums of d products in another order: d 2^-24 relative to the largest term bounds them loosely
            assert np.allclose(w.cpu().numpy()[same], w_ref[same], rtol=5e-5, atol=1e-7), (d, T)


@pytest.mark.parametrize("E,d", [(8, 4096), (60, 1024), (60, 4096), (60, 8192), (128, 10240), (60, 32768)])
def test_router_logits_are_as_exact_as_short_sums(torch_cuda, E, d):
    """The logits of the forms for few rows against 64-bit arithmetic.  Sums of n terms of random sign in a row are off by about
    2^-24 sqrt(n / 6) of the root of their sum of squares (which here is the size of the sum): 2.3 units of 2^-24 for 32 terms, 6.5
    for 256, while runs of ten, four components and a tree over 32 lanes stay near 2^-24 sqrt((10 + 2 * 7) / 6) = 2.  The
    softmax's own rounding of a probability adds about one.  (Longer rows than the small form takes have 32
    terms in a row and a sum over 32 warps.)"""
    torch = torch_cuda
    from candle_b200 import _lib
    T, k = 64, 8
    g = torch.Generator(device="cuda").manual_seed(E + d)
    x, wg = torch.randn((T, d), generator=g, device="cuda"), torch.randn((E, d), generator=g, device="cuda")
    wg *= d ** -0.5  # logits of size one
    ids = torch.empty((T, k), dtype=torch.int32, device="cuda")
    w = torch.empty((T, k), dtype=torch.float32, device="cuda")
    assert _lib.load().candle_moe_router_topk(torch.cuda.current_stream().cuda_stream, x.data_ptr(), wg.data_ptr(), None, T, d, E, k, 0,
                                              ids.data_ptr(), w.data_ptr()) == 0
    ref = torch.softmax(x.double() @ wg.double().T, -1).gather(1, ids.long())
    err = torch.log(w.double()) - torch.log(ref)  # of a logit, with that of the row's normaliser
    assert float(err.pow(2).mean().sqrt()) < (3.0 if d <= 10240 else 4.0) * 2 ** -24


@pytest.mark.parametrize("E,k", [(16, 2), (60, 4), (64, 8), (65, 3), (96, 6), (97, 2), (128, 8)])
def test_tiled_router(orc, torch_cuda, E, k):
    """Many tokens and experts: rows of half a K chunk, of one and a half and of a ragged last one, a ragged last token tile,
    four, six and eight experts per thread."""
    torch = torch_cuda
    from candle_b200 import _lib
    for d, T in ((32, 512), (96, 513), (1056, 543), (64, 7105)):
        rng = np.random.default_rng(E + d)
        x = rng.standard_normal((T, d), dtype=np.float32)
        wg = rng.standard_normal((E, d), dtype=np.float32) * np.float32(0.05)
        bias = rng.standard_normal(E, dtype=np.float32)
        probs, ids_ref, w_ref = orc.router_topk(x, wg, k, True, bias)
        xd, wd, bd = (torch.from_numpy(a).cuda() for a in (x, wg, bias))
        ids = torch.empty((T, k), dtype=torch.int32, device="cuda")
        w = torch.empty((T, k), dtype=torch.float32, device="cuda")
        assert _lib.load().candle_moe_router_topk(torch.cuda.current_stream().cuda_stream, xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), T, d, E,
                                                  k, 1, ids.data_ptr(), w.data_ptr()) == 0
        got = ids.cpu().numpy().astype(np.uint32)
        H.check_routing(probs, ids_ref, got)
        same = (ids_ref == got).all(axis=1)
        assert np.allclose(w.cpu().numpy()[same], w_ref[same], rtol=5e-5, atol=1e-7), (d, T)


@pytest.mark.parametrize("T", [1, 2, 64, 65])
def test_layer_equals_norm_block_residual_in_three_steps(orc, torch_cuda, T):
    torch = torch_cuda
    from candle_b200 import _lib
    cfg = dict(d=1024, ff=1024, E=8, k=2, dt13=orc.Q4K, dt2=orc.Q6K, renorm=True)
    blk, _ = H.random_device_block(orc, torch, cfg, seed=T)
    blk.prepack()
    x = torch.from_numpy(orc.make_activations(T, T, 1024)).cuda() * 3
    nw = 1.0 + 0.1 * torch.randn(1024, generator=torch.Generator(device="cuda").manual_seed(T), device="cuda")
    xn = torch.empty_like(x)
    assert _lib.load().candle_moe_rmsnorm(torch.cuda.current_stream().cuda_stream, x.data_ptr(), nw.data_ptr(), 1e-5, T, 1024, xn.data_ptr()) == 0
    want = blk.forward(xn) + x
    ids = blk.last_routing(T)[0]
    y = blk.forward_layer(x, nw, 1e-5)
    same = (ids == blk.last_routing(T)[0]).all(dim=1).cuda()
    assert int((~same).sum()) <= 1  # a near tie may fall either way
    # the norm's sum of squares is added in another order: last bits of the rows, now and then a step of an int8 value
    assert H.rel_l2((y - x)[same].cpu().numpy(), (want - x)[same].cpu().numpy()) <= H.REL_L2_TOL


@pytest.mark.parametrize("name,k,n,rows", [("Q4K", 256, 128, 49), ("Q4K", 1024, 256, 130), ("Q6K", 512, 128, 65), ("Q6K", 1024, 384, 257)])
def test_gemm_operand_from_f32_rows(orc, torch_cuda, name, k, n, rows):
    """The dense product quantizes its rows while it prepares the operand: rows of every size, rows and blocks of zeros."""
    torch = torch_cuda
    from candle_b200 import GgmlDType, QMatMul, QTensor
    dt = getattr(orc, name)
    rng = np.random.default_rng(k + n + rows)
    x = rng.standard_normal((rows, k), dtype=np.float32) * np.exp2(rng.integers(-20, 20, (rows, 1))).astype(np.float32)
    x[3] = 0.0
    x[5, 256 * (k // 256 - 1):] = 0.0
    wq = orc.quantize(dt, rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02))
    mm = QMatMul.from_qtensor(QTensor.from_blocks(wq, GgmlDType(dt), (n, k))).prepack()
    got = mm.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    ref = orc.matmul(dt, x, wq, n)
    assert np.array_equal(got[3], np.zeros(n, np.float32))
    # the same integers; f32 sums in another order: row by row, as the rows differ in size
    for r in range(rows):
        if r != 3 and not (k == 256 and r == 5):
            assert H.rel_l2(got[r], ref[r]) < 1e-5, r


@pytest.mark.parametrize("T,d,ff,fs", [(97, 256, 384, 128), (130, 512, 1408, 640), (513, 1024, 160, 384)])
def test_q80_large_batch_with_the_fused_operand(orc, torch_cuda, T, d, ff, fs):
    """Hidden rows whose length ends inside a 256-block (routed) and not (shared); against the form without repacked copies."""
    torch = torch_cuda
    from candle_b200 import _lib
    cfg = dict(d=d, ff=ff, E=4, k=2, dt13=orc.Q8_0, dt2=orc.Q8_0, renorm=True, ff_shared=fs)
    blk, _ = H.random_device_block(orc, torch, cfg, seed=T)
    x = torch.from_numpy(orc.make_activations(T, T, d)).cuda()
    want = blk.forward(x).clone()
    blk.prepack()
    y = blk.forward(x).clone()
    assert torch.equal(y, blk.forward(x))
    v = C.c_int32(-1)
    assert _lib.load().candle_moe_device_status(C.byref(v)) == 0 and v.value == 0
    loose = 1.0 if ff >= 1024 else 2.0
    assert H.rel_l2(y.cpu().numpy(), want.cpu().numpy()) <= loose * H.REL_L2_TOL


@pytest.mark.parametrize("w13,w2,T,d,ff,E", [("Q4K", "Q6K", 200, 512, 1536, 4), ("Q6K", "Q6K", 300, 1024, 1536, 4), ("Q6K", "Q4K", 230, 512, 512, 3),
                                             ("Q6K", "Q6K", 400, 2048, 2048, 4)])
def test_large_batch_over_q6k_without_copies(orc, torch_cuda, w13, w2, T, d, ff, E):
    """One expert at a time repacked in the workspace, with an expert that no row selects; and the smallest workspace, in which
    the same batch takes the other forms (the last case the streaming one): both against the oracle."""
    torch = torch_cuda
    from candle_b200 import _lib
    cfg = dict(d=d, ff=ff, E=E, k=2, dt13=getattr(orc, w13), dt2=getattr(orc, w2), renorm=True)
    blk, mw = H.random_device_block(orc, torch, cfg, seed=T)
    bias = np.zeros(E, np.float32)
    bias[1] = -1e9
    mw.router_bias, blk.router_bias = bias, torch.from_numpy(bias).cuda()
    blk._cw.router_bias = blk.router_bias.data_ptr()
    x = torch.from_numpy(orc.make_activations(T, T, d)).cuda()
    xs = x.cpu().numpy()
    ref = orc.moe_forward(mw, xs)
    y = blk.forward(x).clone()
    assert torch.equal(y, blk.forward(x))
    _, _, counts, _ = blk.last_routing(T)
    assert int(counts[1]) == 0 and int(counts.sum()) == 2 * T
    ids = blk.last_routing(T)[0].numpy().astype(np.uint32)
    H.check_routing(orc.router_topk(xs, mw.router, 2, True, bias)[0], ref.topk_ids, ids)
    same = (ref.topk_ids == ids).all(axis=1)
    L = _lib.load()
    small = H.smallest_workspace(_lib, blk._cw, T)
    assert small < blk.workspace_bytes(T)
    ws = torch.empty(small + 256, dtype=torch.uint8, device="cuda")
    ptr = (ws.data_ptr() + 255) // 256 * 256
    y2 = torch.empty_like(y)
    assert L.candle_moe_forward(torch.cuda.current_stream().cuda_stream, C.byref(blk._cw), x.data_ptr(), T, y2.data_ptr(), ptr, small) == 0
    assert not torch.equal(y2, y)  # another kernel form: the f32 sums go in another order
    loose = 1.0 if ff >= 1024 else 2.0
    for got in (y, y2):
        assert H.rel_l2(got.cpu().numpy()[same], ref.y[same]) <= loose * H.REL_L2_TOL
        assert H.max_rel(got.cpu().numpy()[same], ref.y[same]) <= loose * H.MAX_REL_TOL
    v = C.c_int32(-1)
    assert L.candle_moe_device_status(C.byref(v)) == 0 and v.value == 0


@pytest.mark.parametrize("w13,w2,T,d,ff,E", [("Q4K", "Q6K", 97, 512, 1024, 8), ("Q6K", "Q6K", 300, 1024, 1536, 4), ("Q6K", "Q4K", 130, 512, 512, 3),
                                             ("Q6K", "Q6K", 97, 1536, 512, 8), ("Q6K", "Q6K", 640, 2048, 512, 4)])
def test_q6k_without_copies_on_either_side_of_the_rule(orc, torch_cuda, w13, w2, T, d, ff, E):
    """Layers of which the rule takes both products, one or none for the GEMM."""
    torch = torch_cuda
    cfg = dict(d=d, ff=ff, E=E, k=2, dt13=getattr(orc, w13), dt2=getattr(orc, w2), renorm=True)
    blk, mw = H.random_device_block(orc, torch, cfg, seed=T)
    x = torch.from_numpy(orc.make_activations(T, T, d)).cuda()
    xs = x.cpu().numpy()
    ref = orc.moe_forward(mw, xs)
    y = blk.forward(x).clone()
    assert torch.equal(y, blk.forward(x))
    ids = blk.last_routing(T)[0].numpy().astype(np.uint32)
    H.check_routing(orc.router_topk(xs, mw.router, 2, True, None)[0], ref.topk_ids, ids)
    same = (ref.topk_ids == ids).all(axis=1)
    loose = 1.0 if ff >= 1024 else 2.0
    assert H.rel_l2(y.cpu().numpy()[same], ref.y[same]) <= loose * H.REL_L2_TOL


@pytest.mark.parametrize("w13,w2,fs", [("Q4K", "Q6K", 0), ("Q8_0", "Q8_0", 640)])
def test_one_block_takes_batches_in_any_order(orc, torch_cuda, w13, w2, fs):
    """A block keeps its scratch: a batch just above the decode kernels' range, one just inside it (whose partial outputs
    need more), and both again after the repacked copies have been made."""
    torch = torch_cuda
    cfg = dict(d=1024, ff=512, E=8, k=2, dt13=getattr(orc, w13), dt2=getattr(orc, w2), renorm=True, ff_shared=fs)
    blk, _ = H.random_device_block(orc, torch, cfg, seed=1)
    x = torch.from_numpy(orc.make_activations(1, 400, 1024)).cuda()
    nw = torch.ones(1024, device="cuda")
    first = {}
    for step in range(2):
        for T in (97, 96, 400, 95):
            y = blk.forward(x[:T]).clone()
            blk.forward_layer(x[:T], nw, 1e-5)
            assert torch.equal(blk.forward(x[:T]), y), (step, T)
            # other kernels after the copies: the same integers, other f32 orders
            assert step == 0 or H.rel_l2(y.cpu().numpy(), first[T].cpu().numpy()) <= 2 * H.REL_L2_TOL, T
            first.setdefault(T, y)
        blk.prepack()


def _hidden_rows(torch, blk, first, T):
    """The hidden rows a call left in the block's scratch, found by the first of them."""
    words, ff = blk._ws[blk._ws_ptr() - blk._ws.data_ptr():].view(torch.float32), first.numel()
    tol = 1e-4 * float(first.abs().max())
    starts = ((words[:words.numel() - T * ff:64].double() - first[0].double()).abs() <= tol).nonzero()[:, 0].tolist()
    for o in (64 * i for i in starts):
        if torch.allclose(words[o:o + ff].double(), first.double(), rtol=0, atol=tol):
            return words[o:o + T * ff].reshape(T, ff)
    raise AssertionError("the hidden rows were not found in the scratch")


def test_gate_of_repacked_q6k_is_the_exact_one(orc, torch_cuda):
    """Q6_K gate_up repacked on its way: silu as the forms for other batch sizes compute it (expf, an exact division), since the
    hidden rows are quantized again.  Operands whose sums are exact in f32 (scales are powers of two, integers small), so that
    only the gate rounds: expf one unit in the last place, the sum and the division half a unit each, two units of 2^-23 in all."""
    torch = torch_cuda
    from candle_b200 import GgmlDType, Mlp, MlpOrMoe, QMatMul, QTensor
    d, ff, T = 512, 512, 400

    def q6k(n, k, sc, m):
        b = np.zeros((n, k // 256, 210), np.uint8)  # ql[128], qh[64], scales[16], d
        q = (m + 32).astype(np.uint8)[:, None, None]
        b[..., :128] = (q & 15) * 17
        b[..., 128:192] = (q >> 4) * 85
        b[..., 192:208] = sc.astype(np.uint8)[:, None, None]
        b[..., 208:210] = np.frombuffer(np.float16(2.0 ** -14).tobytes(), np.uint8)
        return QTensor.from_blocks(b.reshape(-1), GgmlDType.Q6K, (n, k))

    i = np.arange(ff)
    sc, m = 1 + i % 127, np.array([-32, -29, -23, 31])[i // 128]
    w1, w3 = q6k(ff, d, sc, m), q6k(ff, d, np.full(ff, 16), np.full(ff, 16))
    w2 = q6k(d, ff, np.full(d, 1), np.full(d, 1))
    blk = MlpOrMoe.moe(1, torch.zeros((1, d), device="cuda"), [Mlp(QMatMul(w1), QMatMul(w2), QMatMul(w3))])
    blk.forward(torch.full((T, d), 0.125, device="cuda"))
    gate = sc * m * (512 * 2.0 ** -14 * 0.125)  # -15.9 .. 15.4; the other product is 1
    want = torch.from_numpy(gate / (1 + np.exp(-gate))).cuda()
    got = _hidden_rows(torch, blk, want, T).double()
    assert float(((got - want) / want).abs().max()) <= 2.01 * 2 ** -23


def test_down_product_of_repacked_q6k_adds_short_runs(orc, torch_cuda):
    """The down product of 14336 columns repacked on its way, against 64-bit arithmetic on the same int8 rows.  56 block sums in
    a row are off by about 2^-24 sqrt(56 / 6) of the sum's size (1.8e-7 with nothing else, 1.4e-7 measured), four runs of 14 and
    their sum by 2^-24 sqrt((14 + 2 * 4) / 6) = 1.1e-7, less where the terms differ in size."""
    torch = torch_cuda
    from candle_b200 import GgmlDType, Mlp, MlpOrMoe, QMatMul, QTensor, _lib
    d, ff, T = 4096, 14336, 500
    g = torch.Generator(device="cuda").manual_seed(1)
    mk = lambda n, k, t: QTensor.quantize(torch.randn((n, k), generator=g, device="cuda") * 0.02, t)
    w1, w3, w2 = mk(ff, d, GgmlDType.Q4K), mk(ff, d, GgmlDType.Q4K), mk(d, ff, GgmlDType.Q6K)
    blk = MlpOrMoe.moe(1, torch.zeros((1, d), device="cuda"), [Mlp(QMatMul(w1), QMatMul(w2), QMatMul(w3))])
    x = torch.randn((T, d), generator=g, device="cuda")
    y = blk.forward(x)

    def int8_rows(v):
        rows, k = v.shape
        q = torch.empty((rows, k), dtype=torch.int8, device="cuda")
        s, bs = torch.empty((rows, k // 256), device="cuda"), torch.empty((rows, k // 16), dtype=torch.int16, device="cuda")
        assert _lib.load().candle_moe_quantize_act(torch.cuda.current_stream().cuda_stream, v.data_ptr(), rows, k, int(GgmlDType.Q6K), q.data_ptr(),
                                                   s.data_ptr(), bs.data_ptr()) == 0
        return (q.double().reshape(rows, -1, 256) * s.double()[..., None]).reshape(rows, k)

    x0 = int8_rows(x[:1].contiguous())
    gate, up = x0 @ w1.dequantize().double().T, x0 @ w3.dequantize().double().T
    hidden = _hidden_rows(torch, blk, (gate / (1 + torch.exp(-gate)) * up)[0], T)
    ref = int8_rows(hidden.contiguous()) @ w2.dequantize().double().T
    assert float((y.double() - ref).norm() / ref.norm()) < 1.1e-7


@pytest.mark.parametrize("T,E,k,d,ff,slots", [(200, 16, 8, 1024, 1024, 1), (300, 8, 8, 512, 512, 1), (130, 8, 2, 1024, 3584, 2)])
def test_sums_of_few_blocks_are_not_split(orc, torch_cuda, T, E, k, d, ff, slots):
    """How many partial outputs the down product on the GEMM leaves: none beyond the first where K has a few blocks and the tiles
    fill the device, two where they do not.  Read from the scratch, which is filled with a pattern before the call."""
    torch = torch_cuda
    cfg = dict(d=d, ff=ff, E=E, k=k, dt13=orc.Q4K, dt2=orc.Q4K, renorm=True)
    blk, _ = H.random_device_block(orc, torch, cfg, seed=2)
    x = torch.from_numpy(orc.make_activations(2, T, d)).cuda()
    blk.reserve(T)
    blk._ws.fill_(255)
    blk.forward(x)
    untouched = int((blk._ws[blk._ws_ptr() - blk._ws.data_ptr():].view(torch.int32) == -1).sum())
    int8_rows = T * k * ff * (1 + 4 / 256 + 2 / 16) / 4  # of the hidden rows: not written where the operand's preparation quantizes
    assert 4 - slots <= (untouched - int8_rows) / (T * k * d) < 4.9 - slots


@pytest.mark.parametrize("rows", [32, 64])
def test_narrow_gemm_tiles_add_in_runs(orc, torch_cuda, rows):
    """A dense Q6_K product of 4096 columns on the GEMM with K unsplit, against 64-bit arithmetic on the same int8 rows: 16 block
    sums in a row were off by 7.8e-8, two runs of eight are by 6.5e-8 (2^-24 sqrt(n / 6) and what the rounding of the scales
    adds: 0.6 of 2^-24 for n = 1)."""
    torch = torch_cuda
    from candle_b200 import GgmlDType, QMatMul, QTensor, _lib
    n, k = 12800, 4096
    g = torch.Generator(device="cuda").manual_seed(4)
    w = QTensor.quantize(torch.randn((n, k), generator=g, device="cuda") * 0.02, GgmlDType.Q6K)
    x = torch.randn((rows, k), generator=g, device="cuda")
    q = torch.empty((rows, k), dtype=torch.int8, device="cuda")
    s, bs = torch.empty((rows, k // 256), device="cuda"), torch.empty((rows, k // 16), dtype=torch.int16, device="cuda")
    assert _lib.load().candle_moe_quantize_act(torch.cuda.current_stream().cuda_stream, x.data_ptr(), rows, k, int(GgmlDType.Q6K), q.data_ptr(),
                                               s.data_ptr(), bs.data_ptr()) == 0
    ref = (q.double().reshape(rows, -1, 256) * s.double()[..., None]).reshape(rows, k) @ w.dequantize().double().T
    y = QMatMul(w).prepack().forward(x)
    assert float((y.double() - ref).norm() / ref.norm()) < 7.1e-8
