"""GPU parity: the tcgen05 W4A16 kernels of the ZLW4I layout vs the CPU oracle: stream-k (k_w4a16_ts) and pairs of SMs (k_w4a16_tc2).  Which one serves
a shape is the answer of the route queries; the tests named stream_k, and those that force its splits, assert that it is the first.

Each rounds w = (q - z) * s to fp16 once (what the reference's M > 40 dequant + cuBLASLt route does,
q_gemm_k_major.cu:843-905, 1083-1100), multiplies fp16 x fp16 exactly and accumulates all of K in fp32 in TMEM.
Tolerance: relative L2 <= 1e-3 against the fp32 oracle for fp16 outputs."""
import numpy as np
import pytest
import torch

from oracle import gptq, ops as oops
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-3


def _dev(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def _setup(cuda, k, n, sym, seed, row_map=None):
    from zhilight_b200 import ops
    qw, qz, sc, gi = gptq.make_gptq_checkpoint(k, n, 128, sym, seed=seed)
    o_qw, o_qz, o_sc, _ = gptq.to_k_major(qw, qz, sc, gi, 128)
    w = gptq.dequant_k_major_f32(o_qw, o_qz, o_sc, sym)
    packed = ops.w4_pack(_dev(o_qw.view(np.int32), cuda), _dev(o_qz, cuda), _dev(o_sc, cuda), 128, sym, row_map,
                         variant=1)
    return w, packed


@pytest.fixture
def splits(lib):
    yield lambda s: lib.zl_w4_tc_set_splits(s)
    lib.zl_w4_tc_set_splits(0)


def _stream_k(lib, m, n, k):
    return (lib.zl_w4_int_layout_route(m, n, k), lib.zl_w4_few_rows_route(m, n, k), lib.zl_w4_pairs_route(m, n, k)) == (4, 0, 0)


def _check_watchdog(lib):
    assert lib.zl_w4_tc_watchdog() == 0 and lib.zl_w4_tc2_watchdog() == 0


def test_route_selects_tcgen05(lib):
    assert lib.zl_w4_int_layout_route(1, 4096, 4096) == 3       # exact-integer mma.sync kernel
    assert lib.zl_w4_int_layout_route(4, 4096, 4096) == 3
    assert lib.zl_w4_int_layout_route(16, 512, 1024) == 3
    assert lib.zl_w4_int_layout_route(16, 4096, 4096) == 4      # 16 staged token rows of K = 4096 do not fit beside the rings
    assert lib.zl_w4_int_layout_route(17, 4096, 4096) == 4      # tcgen05
    assert lib.zl_w4_int_layout_route(32, 4096, 14336) == 4
    assert lib.zl_w4_int_layout_route(8, 4096, 14336) == 4      # staged activations of the integer kernel do not fit
    assert lib.zl_w4_int_layout_route(2048, 6144, 4096) == 4
    assert lib.zl_w4_int_layout_route(32, 96, 4096) == 0        # N % 128 != 0: the fp16 mma.sync kernel (variant 0)


def test_every_shape_has_one_kernel(lib, cuda):
    """The queries name at most one kernel for a shape, and the fp16 mma.sync kernel where a call runs on it."""
    for m in (1, 4, 8, 9, 16, 17, 32, 33, 64, 128, 256, 300):
        for k, n in ((1024, 512), (2048, 9472), (2048, 9600), (4096, 4096), (4096, 6144), (8192, 4736), (8320, 384), (14336, 512), (14336, 4096), (4096, 28672)):
            route, few, pairs = lib.zl_w4_int_layout_route(m, n, k), lib.zl_w4_few_rows_route(m, n, k), lib.zl_w4_pairs_route(m, n, k)
            assert route in (3, 4) and few + pairs <= 1 and (lib.zl_w4_pairs_splits(m, n, k) > 0) == (pairs == 1)
            if route == 3:
                assert pairs == 0 and few == (m > 8)
            elif m <= 16:
                assert few == 1
            elif m <= 32:
                assert few == (k <= 8192 if n <= 4736 else k <= 2048 if n <= 9472 else False)
            else:
                assert few == 0 and (m <= 256 or pairs == 1)


@pytest.mark.parametrize("m", [17, 32, 33, 64, 65, 128, 200, 256, 300])
def test_token_counts(lib, cuda, m):
    """ragged last 16-token chunks on both sides of 256 rows (a small matrix: pairs of SMs)"""
    from zhilight_b200 import ops
    k, n = 1024, 512
    w, packed = _setup(cuda, k, n, False, 5)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).half()
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1).float().cpu().numpy()
    _check_watchdog(lib)
    ref = gptq.gemm_f32(x.numpy(), w)
    assert rel_l2(y, ref) <= TOL
    for i in range(m):
        assert rel_l2(y[i], ref[i]) <= 2 * TOL, i


@pytest.mark.parametrize("k,n,m,sym", [(128, 128, 17, False), (256, 128, 32, True), (4096, 6144, 32, False),
                                        (4096, 4096, 24, True), (14336, 4096, 32, False), (14336, 4096, 5, False),
                                        (4096, 28672, 48, False), (8192, 1024, 128, False)])
def test_model_shapes(lib, cuda, k, n, m, sym):
    """Llama-3.1-8B / 70B-class projection shapes, asym and sym zeros, automatic k-split"""
    from zhilight_b200 import ops
    w, packed = _setup(cuda, k, n, sym, 3)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(1)).half()
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1).float().cpu().numpy()
    _check_watchdog(lib)
    ref = gptq.gemm_f32(x.numpy(), w)
    assert rel_l2(y, ref) <= TOL


@pytest.mark.parametrize("s", [1, 2, 3, 4])
def test_split_k_is_deterministic_and_exact_enough(lib, cuda, splits, s):
    from zhilight_b200 import ops
    k, n, m = 8320, 256, 40
    assert _stream_k(lib, m, n, k)
    w, packed = _setup(cuda, k, n, False, 8)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(2)).half().to(cuda)
    splits(s)
    y1 = ops.w4a16_gemm_fused(x, packed, n, k, variant=1)
    y2 = ops.w4a16_gemm_fused(x, packed, n, k, variant=1)
    _check_watchdog(lib)
    assert torch.equal(y1, y2)                                    # partials are reduced in split order
    assert rel_l2(y1.float().cpu().numpy(), gptq.gemm_f32(x.cpu().numpy(), w)) <= TOL


@pytest.mark.parametrize("m,s", [(20, 1), (40, 2)])
def test_bias_residual_swiglu(lib, cuda, splits, m, s):
    from zhilight_b200 import ops
    k, f = 8320, 1280
    assert _stream_k(lib, m, 2 * f, k) and _stream_k(lib, m, 512, k)
    rm = ops.swiglu_row_map(f, cuda)
    w, packed = _setup(cuda, k, 2 * f, False, 7, rm)
    g = torch.Generator().manual_seed(9)
    x = (torch.randn(m, k, generator=g)).half()
    splits(s)
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, 2 * f, k, epilogue=ops.EPI_SWIGLU, variant=1).float().cpu().numpy()
    _check_watchdog(lib)
    gu = oops._t(gptq.gemm_f32(x.numpy(), w), "f16")              # T(gate), T(up) like the reference's two GEMVs
    gate, up = gu[:, :f], gu[:, f:]
    ref = gate / (1.0 + np.exp(-gate)) * up
    assert rel_l2(y, ref) <= 2e-3
    # bias + residual on a plain projection
    n = 512
    w2, packed2 = _setup(cuda, k, n, True, 4)
    bias = (torch.randn(n, generator=g) * 0.5).half()
    res = torch.randn(m, n, generator=g).half()
    y2 = ops.w4a16_gemm_fused(x.to(cuda), packed2, n, k, bias=bias.to(cuda), residual=res.to(cuda),
                              epilogue=ops.EPI_RESIDUAL, variant=1).float().cpu().numpy()
    _check_watchdog(lib)
    lin = oops._t(gptq.gemm_f32(x.numpy(), w2) + bias.float().numpy(), "f16")
    ref2 = oops._t(lin + res.float().numpy(), "f16")
    assert rel_l2(y2, ref2) <= TOL


@pytest.mark.parametrize("d,hq,hkv,k,t,s", [(128, 4, 2, 512, 24, 0), (64, 4, 2, 256, 40, 0), (128, 8, 1, 1024, 130, 0),
                                           (128, 32, 8, 4096, 32, 0), (128, 32, 8, 4096, 20, 3), (128, 32, 8, 4096, 32, 2)])
def test_qkv_rope_epilogue(lib, cuda, splits, d, hq, hkv, k, t, s):
    """fused qkv split + RoPE + KV append vs the stand-alone rope/append operator on the plain GEMM output"""
    from zhilight_b200 import ops
    n = (hq + 2 * hkv) * d
    assert s == 0 or _stream_k(lib, t, n, k)
    rm = ops.qkv_rope_row_map(hq + 2 * hkv, d, cuda)
    _, packed = _setup(cuda, k, n, False, 14, rm)
    _, packed_plain = _setup(cuda, k, n, False, 14)
    g = torch.Generator().manual_seed(8)
    x = torch.randn(t, k, generator=g).half().to(cuda)
    pos = torch.tensor([(5 * i) % 61 for i in range(t)], dtype=torch.int32, device=cuda)
    cos, sin = ops.rope_cos_sin(pos, d, 10000.0)
    tb = torch.tensor([i % 3 for i in range(t)], dtype=torch.int32, device=cuda)
    pl = torch.tensor([i // 3 for i in range(t)], dtype=torch.int32, device=cuda)     # (task, slot) pairs are unique
    slots = t // 3 + 2
    kb = [torch.zeros(slots, hkv, d, dtype=torch.float16, device=cuda) for _ in range(3)]
    vb = [torch.zeros(slots, hkv, d, dtype=torch.float16, device=cuda) for _ in range(3)]
    splits(s)
    q = ops.w4a16_gemm_fused(x, packed, n, k, epilogue=ops.EPI_QKV_ROPE, variant=1,
                             rope=dict(cos=cos, sin=sin, token_batch=tb, placement=pl, k_bufs=kb, v_bufs=vb,
                                       num_heads=hq, num_kv_heads=hkv, dim_head=d))
    _check_watchdog(lib)
    splits(0)
    qkv = ops.w4a16_gemm_fused(x, packed_plain, n, k, variant=1)
    assert torch.isfinite(q).all() and torch.isfinite(qkv).all()
    kb2 = [torch.zeros_like(b) for b in kb]
    vb2 = [torch.zeros_like(b) for b in vb]
    q2 = ops.qkv_rope_append(cos, sin, qkv, tb, pl, kb2, vb2, hq, hkv, d)
    torch.testing.assert_close(q, q2, rtol=2 ** -9, atol=3e-3)
    for a, b in zip(kb + vb, kb2 + vb2):
        torch.testing.assert_close(a, b, rtol=2 ** -9, atol=3e-3)
    assert float(kb[0].abs().max()) > 0 and float(q.abs().max()) > 0


def test_strided_activations_and_fused_norm_is_rejected(lib, cuda):
    from zhilight_b200 import ops, _lib
    k, n, m = 512, 256, 20
    w, packed = _setup(cuda, k, n, False, 21)
    big = torch.randn(m, k + 64, generator=torch.Generator().manual_seed(3)).half().to(cuda)
    x = big[:, :k]                                                # ldx = k + 64
    y = ops.w4a16_gemm_fused(x, packed, n, k, variant=1).float().cpu().numpy()
    assert rel_l2(y, gptq.gemm_f32(x.cpu().numpy(), w)) <= TOL
    with pytest.raises(_lib.ZLError):
        ops.w4a16_gemm_fused(x, packed, n, k, variant=1, ln_weight=torch.ones(k, dtype=torch.float16, device=cuda))


@pytest.mark.parametrize("m", [17, 32, 33, 64, 65, 128, 129, 200, 256])
@pytest.mark.parametrize("k,n", [(8320, 384), (14336, 512)])
def test_stream_k_token_counts(lib, cuda, m, k, n):
    """every NTOK instantiation (32 / 64 / 128 / 256), ragged last 16-token chunk; every tile is cut"""
    from zhilight_b200 import ops
    assert _stream_k(lib, m, n, k)
    w, packed = _setup(cuda, k, n, False, 5)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).half()
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1)
    assert torch.equal(y, ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1))   # the exchanged words are empty again
    _check_watchdog(lib)
    y, ref = y.float().cpu().numpy(), gptq.gemm_f32(x.numpy(), w)
    assert rel_l2(y, ref) <= TOL
    for i in range(m):
        assert rel_l2(y[i], ref[i]) <= 2 * TOL, i


@pytest.mark.parametrize("m,k,f,n", [(20, 8320, 1280, 640), (40, 4096, 1344, 640), (100, 4096, 1280, 512), (33, 4096, 14336, 28672)])
def test_stream_k_bias_residual_swiglu(lib, cuda, m, k, f, n):
    """Epilogues behind the exchange of partial tiles, and (the last shape, more tiles than blocks) of whole tiles with the residual
    fetched ahead; the residual's stores of two columns and, from an odd address, of one."""
    from zhilight_b200 import ops
    assert _stream_k(lib, m, 2 * f, k) and _stream_k(lib, m, n, k)
    g = torch.Generator().manual_seed(9)
    x = torch.randn(m, k, generator=g).half()
    w, packed = _setup(cuda, k, 2 * f, False, 7, ops.swiglu_row_map(f, cuda))
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, 2 * f, k, epilogue=ops.EPI_SWIGLU, variant=1).float().cpu().numpy()
    gu = oops._t(gptq.gemm_f32(x.numpy(), w), "f16")
    assert rel_l2(y, gu[:, :f] / (1.0 + np.exp(-gu[:, :f])) * gu[:, f:]) <= 2e-3
    del w, packed
    w2, packed2 = _setup(cuda, k, n, True, 4)
    bias, res = (torch.randn(n, generator=g) * 0.5).half(), torch.randn(m, n, generator=g).half()
    call = lambda r, out=None: ops.w4a16_gemm_fused(x.to(cuda), packed2, n, k, bias=bias.to(cuda), residual=r,  # noqa: E731
                                                    epilogue=ops.EPI_RESIDUAL, variant=1, out=out)
    y2 = call(res.to(cuda))
    lin = oops._t(gptq.gemm_f32(x.numpy(), w2) + bias.float().numpy(), "f16")
    assert rel_l2(y2.float().cpu().numpy(), oops._t(lin + res.float().numpy(), "f16")) <= TOL
    h = res.to(cuda)                                    # in place
    call(h, out=h)
    assert torch.equal(h, y2)
    odd = torch.empty(m * n + 1, dtype=torch.float16, device=cuda)[1:].view(m, n)
    odd.copy_(res)
    call(odd, out=odd)
    assert torch.equal(odd, y2)
    _check_watchdog(lib)


@pytest.mark.parametrize("t", [32, 64])
def test_stream_k_qkv_rope_epilogue(lib, cuda, t):
    from zhilight_b200 import ops
    hq, hkv, d, k = 32, 8, 128, 4096
    assert _stream_k(lib, t, (hq + 2 * hkv) * d, k)
    test_qkv_rope_epilogue(lib, cuda, lib.zl_w4_tc_set_splits, d, hq, hkv, k, t, 0)


@pytest.mark.parametrize("m,k,n", [(20, 14336, 512), (32, 4096, 6144), (100, 8192, 384), (200, 8192, 384)])
def test_stream_k_starts_ahead_of_its_predecessor(lib, cuda, m, k, n):
    """Weights are fetched and converted while the predecessor still runs; the result is that of a launch behind it."""
    from tests.test_w4a16_tc2_gpu import behind_slow_predecessors
    from zhilight_b200 import ops
    assert _stream_k(lib, m, n, k)
    _, packed = _setup(cuda, k, n, False, 5)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).half().to(cuda)
    want = ops.w4a16_gemm_fused(x, packed, n, k, variant=1)
    got = torch.full_like(want, float("nan"))
    behind_slow_predecessors(cuda, 100, lambda: ops.w4a16_gemm_fused(x, packed, n, k, variant=1, out=got, pdl=True))
    assert torch.equal(got, want)
    _check_watchdog(lib)
