"""Q8_0 over its repacked copies at decode sizes (expert_direct.cu, DirQ80): K that ends inside a 128-element block, one
and two position tiles, groups walked more than once, outputs narrower than a round of tiles, and the shapes it refuses."""
import ctypes as C

import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n", [(32, 16), (96, 48), (160, 272), (1408, 2048), (5632, 96), (288, 21)])
def test_q80_projection_over_the_repacked_copy(orc, torch_cuda, k, n):
    torch = torch_cuda
    from candle_b200 import GgmlDType, QMatMul, QTensor
    rng = np.random.default_rng(k + n)
    wq = orc.quantize(orc.Q8_0, rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02))
    x = rng.standard_normal((65, k), dtype=np.float32)
    ref = orc.matmul(orc.Q8_0, x, wq, n)
    mm = QMatMul.from_qtensor(QTensor.from_blocks(wq, GgmlDType.Q8_0, (n, k))).prepack()
    for m in (1, 7, 8, 9, 16, 17, 33, 64, 65):
        got = mm.forward(torch.from_numpy(x[:m]).cuda()).cpu().numpy()
        # identical integers, only the order of the f32 sums differs
        assert H.max_rel(got, ref[:m]) < 2e-6 and H.rel_l2(got, ref[:m]) < 1e-6, m


@pytest.mark.parametrize("T,d,ff,E,k,fs", [(1, 288, 96, 5, 2, 0), (8, 512, 1408, 60, 4, 320), (9, 288, 1056, 4, 3, 1056),
                                           (40, 512, 1024, 3, 3, 0), (96, 1024, 1408, 16, 4, 2816), (64, 160, 96, 8, 2, 1024)])
def test_q80_block_over_the_repacked_copies(orc, torch_cuda, T, d, ff, E, k, fs):
    torch = torch_cuda
    from candle_b200 import _lib
    cfg = dict(d=d, ff=ff, E=E, k=k, dt13=orc.Q8_0, dt2=orc.Q8_0, renorm=False, ff_shared=fs)
    blk, mw = H.random_device_block(orc, torch, cfg, seed=T + d)
    x = torch.from_numpy(orc.make_activations(T, T, d)).cuda()
    plain = blk.forward(x).clone()
    blk.prepack()
    y = blk.forward(x).clone()
    assert torch.equal(y, blk.forward(x))
    v = C.c_int32(-1)
    assert _lib.load().candle_moe_device_status(C.byref(v)) == 0 and v.value == 0
    # against the kernels over the GGUF bytes: the same integers, but hidden values that differ in the last bit may move an
    # int8 value by a step when they are quantized again
    loose = 1.0 if ff >= 1024 and T > 1 else 2.0
    assert H.rel_l2(y.cpu().numpy(), plain.cpu().numpy()) <= loose * H.REL_L2_TOL
    xs = x.cpu().numpy()
    ref = orc.moe_forward(mw, xs)
    same = (ref.topk_ids == blk.last_routing(T)[0].numpy().astype(np.uint32)).all(axis=1)
    H.check_routing(orc.router_topk(xs, mw.router, k, False, None)[0], ref.topk_ids, blk.last_routing(T)[0].numpy().astype(np.uint32))
    got = y.cpu().numpy()
    assert H.max_rel(got[same], ref.y[same]) <= loose * H.MAX_REL_TOL and H.rel_l2(got[same], ref.y[same]) <= loose * H.REL_L2_TOL


def test_q80_projection_ignores_a_copy_it_cannot_read(orc, torch_cuda):
    """The decode kernels copy 16-byte vectors: a pointer that candle_moe_prepack cannot have filled is left alone."""
    torch = torch_cuda
    from candle_b200 import GgmlDType, QMatMul, QTensor
    n, k, m = 64, 256, 5
    rng = np.random.default_rng(1)
    wq = orc.quantize(orc.Q8_0, rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02))
    x = rng.standard_normal((m, k), dtype=np.float32)
    mm = QMatMul.from_qtensor(QTensor.from_blocks(wq, GgmlDType.Q8_0, (n, k))).prepack()
    mm._prepacked = torch.cat([torch.zeros(8, dtype=torch.uint8, device="cuda"), mm._prepacked])[8:]
    assert mm._prepacked.data_ptr() % 16 == 8
    assert H.rel_l2(mm.forward(torch.from_numpy(x).cuda()).cpu().numpy(), orc.matmul(orc.Q8_0, x, wq, n)) < 1e-6


@pytest.mark.parametrize("w13,w2", [("Q8_0", "Q8_0"), ("Q4K", "Q8_0"), ("Q4K", "Q6K")])
def test_tables_with_a_hole(orc, torch_cuda, w13, w2):
    """Copies for some experts only: a decode-sized batch with Q8_0 matrices runs on the GGUF blocks, bit for bit as without
    tables; k-quants refuse such tables."""
    torch = torch_cuda
    from candle_b200 import _lib
    cfg = dict(d=512, ff=512, E=4, k=2, dt13=getattr(orc, w13), dt2=getattr(orc, w2), renorm=True)
    blk, _ = H.random_device_block(orc, torch, cfg, seed=3)
    x = torch.from_numpy(orc.make_activations(3, 9, 512)).cuda()
    plain = blk.forward(x).clone()
    blk.prepack()
    for value in (None, blk._p2[2] + 8):
        blk._p2[2] = value
        if w2 == "Q8_0":
            assert torch.equal(blk.forward(x), plain)
        else:
            with pytest.raises(_lib.CandleMoeError) as e:
                blk.forward(x)
            assert e.value.status == (-1 if value is None else -5)
