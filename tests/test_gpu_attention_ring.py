"""The pipelined decode attention (rows of 128, four query heads per kv head): contexts around its tile, warp and chunk
edges, chunks of every length its rule picks, one workspace for all of them, and infinities."""
import ctypes as C
import math

import pytest

pytestmark = pytest.mark.gpu

CTX = (1, 7, 8, 9, 25, 32, 33, 63, 64, 65, 129, 511, 512, 513, 1025, 1500)


def _run(torch, q, kc, vc, n_ctx, ws):
    from candle_b200 import _lib
    B, n_head, hd = q.shape
    y = torch.full((B, n_head * hd), float("nan"), device="cuda")
    st = _lib.load().candle_moe_decode_attention(torch.cuda.current_stream().cuda_stream, q.data_ptr(), kc.data_ptr(), vc.data_ptr(), B,
                                                 n_head, kc.shape[1], hd, kc.shape[2], n_ctx, y.data_ptr(), ws.data_ptr(), ws.numel())
    assert st == 0
    return y


def _plain(torch, q, kc, vc, n_ctx):
    B, n_head, hd = q.shape
    n_kv = kc.shape[1]
    att = torch.softmax(q.double().reshape(B, n_kv, n_head // n_kv, hd) @ kc[:, :, :n_ctx].double().transpose(-1, -2) / math.sqrt(hd), dim=-1)
    return (att @ vc[:, :, :n_ctx].double()).reshape(B, n_head * hd)


@pytest.mark.parametrize("B,n_kv", [(1, 1), (2, 8), (40, 8)])
def test_contexts_around_the_edges(torch_cuda, B, n_kv):
    torch = torch_cuda
    from candle_b200 import _lib
    max_seq, hd = CTX[-1], 128
    g = torch.Generator(device="cuda").manual_seed(B)
    q = torch.randn((B, 4 * n_kv, hd), generator=g, device="cuda") * 2
    kc = torch.randn((B, n_kv, max_seq, hd), generator=g, device="cuda")
    vc = torch.randn((B, n_kv, max_seq, hd), generator=g, device="cuda")
    need = C.c_size_t(0)
    assert _lib.load().candle_moe_decode_attention_workspace_bytes(B, 4 * n_kv, hd, max_seq, C.byref(need)) == 0
    ws = torch.empty(need.value + 16, dtype=torch.uint8, device="cuda")  # one workspace for every context up to max_seq
    for n_ctx in CTX:
        got, ref = _run(torch, q, kc, vc, n_ctx, ws).double(), _plain(torch, q, kc, vc, n_ctx)
        # f32 sums: 1500 terms of rounding 2^-24 in the worst order are 9e-5; the tree order keeps it near 1e-7
        assert float((got - ref).abs().max() / ref.abs().max()) < 2e-6, n_ctx
        assert torch.equal(got, _run(torch, q, kc, vc, n_ctx, ws).double()), n_ctx
    v = C.c_int32(-1)
    assert _lib.load().candle_moe_device_status(C.byref(v)) == 0 and v.value == 0


def test_infinite_and_nan_scores(torch_cuda):
    torch = torch_cuda
    B, n_kv, max_seq, hd, n_ctx = 1, 1, 300, 128, 300
    q = torch.zeros((B, 4, hd), device="cuda")
    q[..., 0] = 1.0
    kc = torch.zeros((B, n_kv, max_seq, hd), device="cuda")
    vc = torch.randn((B, n_kv, max_seq, hd), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    ws = torch.empty(1 << 22, dtype=torch.uint8, device="cuda")
    kc[0, 0, :256, 0] = float("-inf")  # whole tiles and chunks without weight: the rest decides
    got, ref = _run(torch, q, kc, vc, n_ctx, ws).double(), _plain(torch, q, kc, vc, n_ctx)
    assert float((got - ref).abs().max() / ref.abs().max()) < 2e-6
    for value in (float("nan"), float("inf")):  # as a softmax over the whole row: everything is NaN
        kc[0, 0, 280, 0] = value
        assert torch.isnan(_plain(torch, q, kc, vc, n_ctx)).all() and torch.isnan(_run(torch, q, kc, vc, n_ctx, ws)).all()


@pytest.mark.parametrize("B,n_kv", [(80, 1), (1, 8)])
def test_long_sums_are_no_less_exact_than_short_ones(torch_cuda, B, n_kv):
    """Full chunks of 512 positions, of which a warp adds 128, and 64 short chunks to merge: the relative error must not grow with
    such a run.  A sum of n terms of random sign in a row is off by about 2^-24 sqrt(n / 6) relative to the root of its
    sum of squares (a uniform rounding error of the running sum per step, whose square averages half the final one): 2.8e-7
    for 128 terms, 1.9e-7 for 64, 0.7e-7 for 8 and 1e-7 for 16.  With the rounding of the scores and weights themselves, about
    1e-7, sums of 8 and 16 stay below 1.7e-7 and those of 64 or 128 do not."""
    torch = torch_cuda
    hd, n_ctx = 128, 4096
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn((B, 4 * n_kv, hd), generator=g, device="cuda")
    kc = torch.randn((B, n_kv, n_ctx, hd), generator=g, device="cuda") * 0.5
    vc = torch.randn((B, n_kv, n_ctx, hd), generator=g, device="cuda") * 0.5
    ws = torch.empty(1 << 24, dtype=torch.uint8, device="cuda")
    got, ref = _run(torch, q, kc, vc, n_ctx, ws).double(), _plain(torch, q, kc, vc, n_ctx)
    assert float((got - ref).norm() / ref.norm()) < 1.7e-7
