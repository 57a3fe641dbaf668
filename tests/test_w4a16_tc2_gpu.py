"""GPU: the 4-bit GEMM over pairs of SMs (prompt-sized M) against the oracle: edges of its 256-row and 32-token tiles, odd numbers of 128-row
tiles, every epilogue.  Tolerance as in test_w4a16_tc_gpu.py: relative L2 <= 1e-3 for fp16 outputs."""
import numpy as np
import pytest
import torch

from oracle import gptq, ops as oops
from tests.helpers import rel_l2
from tests.test_w4a16_tc_gpu import TOL, _setup

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def no_wait_gave_up(lib, cuda):
    yield
    torch.cuda.synchronize()
    assert lib.zl_w4_tc2_watchdog() == 0


def _x(m, k, seed):
    return torch.randn(m, k, generator=torch.Generator().manual_seed(seed)).half()


@pytest.mark.parametrize("m", [129, 160, 161, 255, 256, 257, 300, 513, 1000])
@pytest.mark.parametrize("k,n", [(128, 128), (1024, 384), (640, 512)])
def test_token_counts_and_row_tiles(lib, cuda, m, k, n):
    from zhilight_b200 import ops
    w, packed = _setup(cuda, k, n, False, 5)
    x = _x(m, k, m)
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1).float().cpu().numpy()
    ref = gptq.gemm_f32(x.numpy(), w)
    assert rel_l2(y, ref) <= TOL
    for i in (0, 31, 32, 127, 128, m - 1):
        assert rel_l2(y[i], ref[i]) <= 2 * TOL, i


@pytest.mark.parametrize("k,n,m,sym", [(4096, 6144, 200, False), (4096, 4096, 520, True), (14336, 4096, 257, False), (4096, 28672, 300, False),
                                       (14336, 512, 200, False), (14336, 512, 100, True), (4096, 6144, 70, False)])
def test_model_shapes(lib, cuda, k, n, m, sym):
    """Also shapes below 257 tokens that stay with w4a16_tc.cu, or leave it for less than 129."""
    from zhilight_b200 import ops
    w, packed = _setup(cuda, k, n, sym, 3)
    x = _x(m, k, 1)
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1)
    assert torch.equal(y, ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1))
    assert rel_l2(y.float().cpu().numpy(), gptq.gemm_f32(x.numpy(), w)) <= TOL


@pytest.mark.parametrize("m", [150, 400])
def test_bias_residual_swiglu(lib, cuda, m):
    from zhilight_b200 import ops
    k, f, n = 1024, 1344, 384
    w, packed = _setup(cuda, k, 2 * f, False, 7, ops.swiglu_row_map(f, cuda))
    x = _x(m, k, 9)
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, 2 * f, k, epilogue=ops.EPI_SWIGLU, variant=1).float().cpu().numpy()
    gu = oops._t(gptq.gemm_f32(x.numpy(), w), "f16")
    assert rel_l2(y, gu[:, :f] / (1.0 + np.exp(-gu[:, :f])) * gu[:, f:]) <= 2e-3
    w2, packed2 = _setup(cuda, k, n, True, 4)
    g = torch.Generator().manual_seed(2)
    bias, res = (torch.randn(n, generator=g) * 0.5).half(), torch.randn(m, n, generator=g).half()
    y2 = ops.w4a16_gemm_fused(x.to(cuda), packed2, n, k, bias=bias.to(cuda), residual=res.to(cuda), epilogue=ops.EPI_RESIDUAL, variant=1)
    lin = oops._t(gptq.gemm_f32(x.numpy(), w2) + bias.float().numpy(), "f16")
    assert rel_l2(y2.float().cpu().numpy(), oops._t(lin + res.float().numpy(), "f16")) <= TOL
    h = res.to(cuda)                                    # the residual stream is updated in place
    ops.w4a16_gemm_fused(x.to(cuda), packed2, n, k, bias=bias.to(cuda), residual=h, epilogue=ops.EPI_RESIDUAL, variant=1, out=h)
    assert torch.equal(h, y2)


@pytest.mark.parametrize("d,hq,hkv,k,t", [(128, 4, 2, 512, 140), (64, 4, 2, 256, 300), (128, 8, 1, 1024, 257)])
def test_qkv_rope_epilogue(lib, cuda, d, hq, hkv, k, t):
    from zhilight_b200 import ops
    n = (hq + 2 * hkv) * d
    _, packed = _setup(cuda, k, n, False, 14, ops.qkv_rope_row_map(hq + 2 * hkv, d, cuda))
    _, plain = _setup(cuda, k, n, False, 14)
    x = _x(t, k, 8).to(cuda)
    pos = torch.tensor([(5 * i) % 61 for i in range(t)], dtype=torch.int32, device=cuda)
    cos, sin = ops.rope_cos_sin(pos, d, 10000.0)
    tb = torch.tensor([i % 3 for i in range(t)], dtype=torch.int32, device=cuda)
    pl = torch.tensor([-1 if i == 7 else i // 3 for i in range(t)], dtype=torch.int32, device=cuda)   # a token that is not cached
    bufs = [[torch.zeros(t // 3 + 2, hkv, d, dtype=torch.float16, device=cuda) for _ in range(3)] for _ in range(4)]
    q = ops.w4a16_gemm_fused(x, packed, n, k, epilogue=ops.EPI_QKV_ROPE, variant=1,
                             rope=dict(cos=cos, sin=sin, token_batch=tb, placement=pl, k_bufs=bufs[0], v_bufs=bufs[1], num_heads=hq,
                                       num_kv_heads=hkv, dim_head=d))
    q2 = ops.qkv_rope_append(cos, sin, ops.w4a16_gemm_fused(x, plain, n, k, variant=1), tb, pl, bufs[2], bufs[3], hq, hkv, d)
    torch.testing.assert_close(q, q2, rtol=2 ** -9, atol=3e-3)
    for a, b in zip(bufs[0] + bufs[1], bufs[2] + bufs[3]):
        torch.testing.assert_close(a, b, rtol=2 ** -9, atol=3e-3)
    assert float(bufs[0][0].abs().max()) > 0


def test_strided_activations(lib, cuda):
    from zhilight_b200 import ops
    w, packed = _setup(cuda, 512, 256, False, 21)
    x = torch.randn(200, 576, generator=torch.Generator().manual_seed(3)).half().to(cuda)[:, :512]
    y = ops.w4a16_gemm_fused(x, packed, 256, 512, variant=1).float().cpu().numpy()
    assert rel_l2(y, gptq.gemm_f32(x.cpu().numpy(), w)) <= TOL


def behind_slow_predecessors(cuda, ms, call):
    """Runs `call` behind kernels that let their dependents start at once and take `ms` together: one block reads a long row, as often as
    that takes; each of the launches is resident and waits for the one before."""
    from zhilight_b200 import _lib, ops
    long_row = 1 << 30
    row = torch.full((1, long_row), 0.5, dtype=torch.float16, device=cuda)
    q, scale = torch.empty(long_row, dtype=torch.int8, device=cuda), torch.empty(1, device=cuda)
    stream = torch.cuda.current_stream().cuda_stream
    slow = lambda: _lib.call("zl_int8_quant_per_token", row.data_ptr(), long_row, q.data_ptr(), scale.data_ptr(), 1, long_row, ops.F16,  # noqa: E731
                             1, stream)
    begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    slow()
    begin.record()
    slow()
    end.record()
    torch.cuda.synchronize()
    times = int(ms / begin.elapsed_time(end)) + 1
    assert times <= 100                                 # resident at one time: the hardware's limit is 128
    begin.record()
    for _ in range(times):
        slow()
    call()
    end.record()
    torch.cuda.synchronize()
    return begin.elapsed_time(end)


def test_predecessor_that_takes_longer_than_a_wait_may(lib, cuda):
    """Longer than the 2e9 cycles after which a wait inside the GEMM gives up: its waits begin when the predecessor has ended."""
    from zhilight_b200 import ops
    k, n, m = 4096, 512, 300
    w, packed = _setup(cuda, k, n, False, 5)
    x = _x(m, k, 1).to(cuda)
    want = ops.w4a16_gemm_fused(x, packed, n, k, variant=1)
    got = torch.full_like(want, float("nan"))
    took = behind_slow_predecessors(cuda, 1600, lambda: ops.w4a16_gemm_fused(x, packed, n, k, variant=1, out=got, pdl=True))
    assert took > 1400
    assert torch.equal(got, want)


@pytest.mark.parametrize("m,k,n,splits", [(65, 2304, 1152, 3), (40, 3968, 1280, 4), (97, 2304, 2304, 3), (128, 4096, 4096, 2), (45, 2944, 1280, 4), (256, 3200, 1152, 3),
                                          (33, 3840, 2304, 3)])
def test_pairs_that_share_a_tile(lib, cuda, m, k, n, splits):
    """Two, three and four pairs per tile; K of an odd number of 128-k groups, parts of different lengths, an odd number of 128-row tiles, chunks of
    16 tokens that do not divide by the pairs.  Every row; with the residual updated in place; twice the same."""
    from zhilight_b200 import ops
    assert lib.zl_w4_pairs_splits(m, n, k) == splits
    w, packed = _setup(cuda, k, n, False, 6)
    x = _x(m, k, m)
    ref = gptq.gemm_f32(x.numpy(), w)
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1).float().cpu().numpy()
    assert max(rel_l2(y[i], ref[i]) for i in range(m)) <= TOL
    g = torch.Generator().manual_seed(3)
    bias, res = (torch.randn(n, generator=g) * 0.5).half().to(cuda), torch.randn(m, n, generator=g).half()
    outs = []
    for _ in range(2):
        h = res.to(cuda)
        ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, bias=bias, residual=h, epilogue=ops.EPI_RESIDUAL, variant=1, out=h)
        outs.append(h)
    assert torch.equal(*outs)
    want = oops._t(oops._t(ref + bias.float().cpu().numpy(), "f16") + res.float().numpy(), "f16")
    assert rel_l2(outs[0].float().cpu().numpy(), want) <= TOL


def test_shared_tiles_with_swiglu(lib, cuda):
    from zhilight_b200 import ops
    m, k, f = 72, 3968, 640
    assert lib.zl_w4_pairs_splits(m, 2 * f, k) > 1
    w, packed = _setup(cuda, k, 2 * f, False, 7, ops.swiglu_row_map(f, cuda))
    x = _x(m, k, 9)
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, 2 * f, k, epilogue=ops.EPI_SWIGLU, variant=1).float().cpu().numpy()
    gu = oops._t(gptq.gemm_f32(x.numpy(), w), "f16")
    assert rel_l2(y, gu[:, :f] / (1.0 + np.exp(-gu[:, :f])) * gu[:, f:]) <= 2e-3


@pytest.mark.parametrize("m,k,n,pieces", [(322, 1024, 12800, 2), (387, 1024, 13568, 2), (360, 1024, 12672, 2), (385, 1024, 13568, 2), (512, 1024, 18944, 1)])
def test_last_wave_in_halves(lib, cuda, m, k, n, pieces):
    """Tiles of the last wave in halves: one row behind the first half, an odd number of 128-row tiles, a last wave that is full (whole tiles); every row.  All
    warps take part in the epilogues: none, the residual's and SwiGLU's here, qkv's below."""
    from zhilight_b200 import ops
    assert lib.zl_w4_pairs_pieces(m, n, k) == pieces
    w, packed = _setup(cuda, k, n, False, 6)
    x = _x(m, k, m)
    ref = gptq.gemm_f32(x.numpy(), w)
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1).float().cpu().numpy()
    assert max(rel_l2(y[i], ref[i]) for i in range(m)) <= TOL
    res = torch.randn(m, n, generator=torch.Generator().manual_seed(3)).half()
    h = res.to(cuda)
    ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, residual=h, epilogue=ops.EPI_RESIDUAL, variant=1, out=h)
    want = oops._t(oops._t(ref, "f16") + res.float().numpy(), "f16")
    got = h.float().cpu().numpy()
    assert max(rel_l2(got[i], want[i]) for i in range(m)) <= TOL
    if n % 256 == 0:
        _, packed2 = _setup(cuda, k, n, False, 6, ops.swiglu_row_map(n // 2, cuda))
        act = ops.w4a16_gemm_fused(x.to(cuda), packed2, n, k, epilogue=ops.EPI_SWIGLU, variant=1).float().cpu().numpy()
        gu = oops._t(ref, "f16")
        want = gu[:, :n // 2] / (1.0 + np.exp(-gu[:, :n // 2])) * gu[:, n // 2:]
        assert max(rel_l2(act[i], want[i]) for i in range(m)) <= 2e-3


@pytest.mark.parametrize("d,hq,hkv,k,t,pieces", [(128, 92, 4, 1024, 322, 2), (64, 160, 20, 1024, 450, 2), (128, 102, 2, 1024, 387, 2), (128, 32, 8, 1024, 1000, 1),
                                                 (64, 288, 8, 512, 40, 1), (128, 144, 4, 1024, 100, 1)])
def test_qkv_rope_epilogue_over_several_tiles(lib, cuda, d, hq, hkv, k, t, pieces):
    """More tiles than pairs: a chunk's placement comes with the chunk before, and the warps that convert the next tile help; whole and halved last waves, one
    accumulator and two (40 rows).  Against the oracle's matrix turned in 64 bits: every row of q and of the caches, and nothing else written."""
    from zhilight_b200 import ops
    heads, n = hq + 2 * hkv, (hq + 2 * hkv) * d
    assert lib.zl_w4_pairs_pieces(t, n, k) == pieces and lib.zl_w4_pairs_splits(t, n, k) == 1
    rows = ops.qkv_rope_row_map(heads, d, cuda)
    w, packed = _setup(cuda, k, n, False, 14, rows)
    x, bias = _x(t, k, 8), (torch.randn(n, generator=torch.Generator().manual_seed(2)) * 0.5).half()
    pos = torch.tensor([(5 * i) % 61 for i in range(t)], dtype=torch.int32, device=cuda)
    cos, sin = ops.rope_cos_sin(pos, d, 10000.0)
    tb = [i % 3 for i in range(t)]
    pl = [-1 if i in (7, t - 1) else i // 3 for i in range(t)]      # two tokens that are not cached
    bufs = [[torch.zeros(t // 3 + 2, hkv, d, dtype=torch.float16, device=cuda) for _ in range(3)] for _ in range(2)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)  # noqa: E731
    q = ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, bias=bias.to(cuda)[rows.long()], epilogue=ops.EPI_QKV_ROPE, variant=1,
                             rope=dict(cos=cos, sin=sin, token_batch=i32(tb), placement=i32(pl), k_bufs=bufs[0], v_bufs=bufs[1], num_heads=hq,
                                       num_kv_heads=hkv, dim_head=d))
    lin = torch.from_numpy(oops._t(gptq.gemm_f32(x.numpy(), w) + bias.float().numpy(), "f16")).double().view(t, heads, d)
    turned = torch.cat([-lin[..., d // 2:], lin[..., :d // 2]], -1)
    want = lin * cos.cpu().double()[:, None] + turned * sin.cpu().double()[:, None]
    want[:, hq + hkv:] = lin[:, hq + hkv:]
    got = q.cpu().double().view(t, hq, d)
    for i in range(t):
        assert rel_l2(got[i].numpy(), want[i, :hq].numpy()) <= TOL, i
    for kind in range(2):
        ref = [torch.zeros(t // 3 + 2, hkv, d, dtype=torch.float64) for _ in range(3)]
        for i in range(t):
            if pl[i] >= 0:
                ref[tb[i]][pl[i]] = want[i, hq + kind * hkv:hq + (kind + 1) * hkv]
        for b in range(3):
            have = bufs[kind][b].cpu().double()
            for i in range(t // 3 + 2):
                assert rel_l2(have[i].numpy(), ref[b][i].numpy()) <= 2 * TOL if ref[b][i].any() else not have[i].any(), (kind, b, i)


@pytest.mark.parametrize("m,k,n", [(150, 512, 384), (322, 1024, 12800), (100, 1024, 19456), (97, 2304, 2304)])
def test_outputs_on_an_odd_address(lib, cuda, m, k, n):
    """One value per store, with one tile a pair, several, halves, and tiles that pairs share: the bits of the stores of two, and nothing beside them."""
    from zhilight_b200 import ops
    assert lib.zl_w4_pairs_route(m, n, k) == 1
    _, packed = _setup(cuda, k, n, False, 4)
    g = torch.Generator().manual_seed(2)
    x, bias, res = _x(m, k, 9).to(cuda), (torch.randn(n, generator=g) * 0.5).half().to(cuda), torch.randn(m, n, generator=g).half().to(cuda)
    call = lambda r, out, **kw: ops.w4a16_gemm_fused(x, packed, n, k, bias=bias, residual=r, variant=1, out=out, **kw)  # noqa: E731
    for kw in (dict(epilogue=ops.EPI_RESIDUAL), {}):
        want = call(res if kw else None, torch.empty_like(res), **kw)
        room = torch.full((m * n + 2,), 7.0, dtype=torch.float16, device=cuda)
        odd = room[1:-1].view(m, n)
        odd.copy_(res)
        call(odd if kw else None, odd, **kw)
        assert torch.equal(odd, want) and float(room[0]) == float(room[-1]) == 7.0
