"""W8A8 Linear (Int8Linear, Fp8Linear) through the C-ABI against the oracle.

INT8 is integer work with a two-multiply fp32 epilogue: bit-exact.  FP8 quantisation codes are bit-exact; the fp8
GEMM accumulates in fp32 in a different order than cuBLASLt: <= 1e-3 rel (fp16) like the reference's own Linear
tests (tests/test_linear.py:48-86)."""
import numpy as np
import pytest
import torch

from oracle import ops as oracle
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu
DT = {"f16": torch.float16, "bf16": torch.bfloat16}


def _x(m, k, tag, seed=0, amp=1.5):
    r = np.random.default_rng(seed)
    return oracle._t(r.standard_normal((m, k)) * amp, tag)


def _dev(a, tag, cuda):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(DT[tag]).to(cuda)


@pytest.mark.parametrize("tag", ["f16", "bf16"])
@pytest.mark.parametrize("m,k", [(1, 512), (7, 4096), (32, 14336), (40, 1024)])
def test_int8_quant_per_token_bit_exact(lib, cuda, tag, m, k):
    from zhilight_b200 import ops
    x = _x(m, k, tag, seed=m)
    if m > 1:
        x[m // 2] = 0                                           # all-zero token
    q, s = ops.int8_quant_per_token(_dev(x, tag, cuda))
    oq, os_ = oracle.int8_quant_per_token(x)
    np.testing.assert_array_equal(q.cpu().numpy(), oq)
    np.testing.assert_array_equal(s.cpu().numpy(), os_)


@pytest.mark.parametrize("m,k", [(1, 2048), (148, 2048), (149, 2056), (296, 4096), (297, 4104), (888, 8200), (889, 512), (444, 16392)])
def test_int8_quant_of_one_to_six_rows_per_sm(lib, cuda, m, k):
    """Its CTAs ask for shared memory by how many an SM shall take; every kernel instance, calls in a row on changing rows."""
    from zhilight_b200 import ops
    xs = [_x(m, k, "f16", seed=m + i) for i in range(3)]
    on = [_dev(x, "f16", cuda) for x in xs]
    torch.cuda.synchronize()
    got = [ops.int8_quant_per_token(x) for x in on]
    for x, (q, s) in zip(xs, got):
        oq, os_ = oracle.int8_quant_per_token(x)
        np.testing.assert_array_equal(q.cpu().numpy(), oq)
        np.testing.assert_array_equal(s.cpu().numpy(), os_)


@pytest.mark.parametrize("tag", ["f16", "bf16"])
@pytest.mark.parametrize("m,n,k,f32_scale,with_bias", [
    (1, 4096, 4096, False, False), (3, 1000, 512, True, False), (8, 6144, 4096, False, True),
    (9, 4096, 14336, False, False), (16, 64, 64, False, True), (17, 2048, 2048, True, True),
    (32, 28672, 4096, False, False), (33, 1024, 1024, False, False), (70, 512, 256, False, True),
    # M > 32: the tcgen05 kind::i8 kernel (both operands through tensor-TMA, s32 accumulators in TMEM, split-k)
    (64, 6144, 4096, False, True), (128, 4096, 14336, True, False), (300, 1000, 1024, False, True)])
def test_int8_linear_bit_exact(lib, cuda, tag, m, n, k, f32_scale, with_bias):
    from zhilight_b200 import ops
    r = np.random.default_rng(n + m)
    x = _x(m, k, tag, seed=k + m)
    w_q = r.integers(-127, 128, size=(n, k)).astype(np.int8)
    w_s = oracle._t(0.0005 + 0.003 * r.random(n), tag)
    bias = oracle._t(0.2 * r.standard_normal(n), tag) if with_bias else None
    ws_dev = torch.from_numpy(w_s).to(cuda) if f32_scale else _dev(w_s, tag, cuda)
    y = ops.int8_linear(_dev(x, tag, cuda), torch.from_numpy(w_q).to(cuda), ws_dev,
                        None if bias is None else _dev(bias, tag, cuda))
    ref = oracle.int8_linear(x, w_q, w_s, tag, bias)
    np.testing.assert_array_equal(y.float().cpu().numpy(), ref)


@pytest.mark.parametrize("tag", ["f16", "bf16"])
def test_rmsnorm_quant(lib, cuda, tag):
    from zhilight_b200 import ops
    t, d = 6, 4096
    r = np.random.default_rng(5)
    x = _x(t, d, tag, seed=3)
    x[2] = 0
    w = oracle._t(1.0 + 0.2 * r.standard_normal(d), tag)
    for scale in (1.0, 2.5):
        y, q, qs = ops.rmsnorm_quant(_dev(x, tag, cuda), _dev(w, tag, cuda), 1e-5, scale)
        oy, oq, oqs = oracle.rmsnorm_quant(x, w, 1e-5, scale, tag)
        np.testing.assert_array_equal(q.cpu().numpy(), oq)
        np.testing.assert_allclose(qs.cpu().numpy(), oqs, rtol=2e-6)
        assert rel_l2(y.float().cpu().numpy(), oy) < (1e-3 if tag == "f16" else 4e-3)


@pytest.mark.parametrize("tag", ["f16", "bf16"])
@pytest.mark.parametrize("m,k", [(1, 4096), (5, 512), (32, 14336)])
def test_fp8_quant_codes_bit_exact(lib, cuda, tag, m, k):
    from zhilight_b200 import ops
    x = _x(m, k, tag, seed=11 + m, amp=3.0)
    q, s = ops.fp8_quant_per_tensor(_dev(x, tag, cuda))
    ov, os_ = oracle.fp8_quant_per_tensor(x, dtype=tag)
    assert s.item() == os_
    np.testing.assert_array_equal(oracle.e4m3_decode(q.cpu().numpy()), ov)


@pytest.mark.parametrize("tag", ["f16", "bf16"])
@pytest.mark.parametrize("m,n,k,with_bias", [(1, 4096, 4096, False), (4, 1000, 512, True), (16, 6144, 4096, False),
                                             (32, 4096, 14336, True), (35, 256, 128, False),
                                             # M > 32: the tcgen05 kind::f8f6f4 kernel
                                             (64, 6144, 4096, True), (130, 4096, 4096, False)])
def test_fp8_linear(lib, cuda, tag, m, n, k, with_bias):
    from zhilight_b200 import ops
    r = np.random.default_rng(n)
    x = _x(m, k, tag, seed=k)
    w8 = r.integers(0, 256, size=(n, k)).astype(np.uint8)
    w8[(w8 & 0x7F) == 0x7F] = 0x30
    w8[(w8 & 0x78) > 0x50] &= 0xAF                               # keep |w| <= ~30 so fp16 outputs stay finite
    w_scale = np.float32(0.004)
    bias = oracle._t(0.2 * r.standard_normal(n), tag) if with_bias else None
    y = ops.fp8_linear(_dev(x, tag, cuda), torch.from_numpy(w8).to(cuda),
                       torch.tensor([w_scale], dtype=torch.float32, device=cuda),
                       None if bias is None else _dev(bias, tag, cuda))
    ref = oracle.fp8_linear(x, oracle.e4m3_decode(w8), w_scale, tag, bias)
    assert np.isfinite(ref).all()
    assert rel_l2(y.float().cpu().numpy(), ref) < (1e-3 if tag == "f16" else 4e-3)


def test_w8_argument_errors(lib, cuda):
    from zhilight_b200 import _lib, ops
    xq = torch.zeros((2, 96), dtype=torch.int8, device=cuda)          # K % 64 != 0
    sx = torch.ones(2, device=cuda)
    w = torch.zeros((16, 96), dtype=torch.int8, device=cuda)
    with pytest.raises(_lib.ZLError):
        ops.w8a8_gemm(xq, sx, w, torch.ones(16, device=cuda), torch.float16)
    with pytest.raises(_lib.ZLError):                                  # fp8 needs f32 scalar scales
        ops.w8a8_gemm(torch.zeros((2, 64), dtype=torch.uint8, device=cuda), sx,
                      torch.zeros((16, 64), dtype=torch.uint8, device=cuda),
                      torch.ones(1, dtype=torch.float16, device=cuda), torch.float16, kind=ops.W8_FP8)


@pytest.mark.parametrize("tag", ["f16", "bf16"])
@pytest.mark.parametrize("n", [8, 65528, 65536, 65544, 1 << 20, (1 << 22) - 8, 1 << 22])
def test_fp8_quant_one_and_two_launches_bit_exact(lib, cuda, tag, n):
    """Both sides of the size where the scale is found by a launch of its own; the largest value sits in the last place."""
    from zhilight_b200 import ops
    x = _x(1, n, tag, seed=n % 97, amp=3.0)
    x[0, -1] = -17.0
    for _ in range(2):                                  # the second call finds the first one's scale word
        q, s = ops.fp8_quant_per_tensor(_dev(x, tag, cuda))
        ov, os_ = oracle.fp8_quant_per_tensor(x, dtype=tag)
        assert s.item() == os_
        np.testing.assert_array_equal(oracle.e4m3_decode(q.cpu().numpy()), ov)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,n,k", [(1, 33000, 4160), (9, 16384, 3136), (25, 4100, 12352), (33, 130, 64), (65, 1000, 192), (300, 257, 1088)])
def test_products_on_pairs_of_sms(lib, cuda, dtype, m, n, k):
    """The dispatch lines and the edges of the 256-row, 32-row and 128-byte tiles; odd row counts, K a multiple of 64 only."""
    from zhilight_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(m)
    r = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731
    xq, w = (torch.randint(-127, 128, s, generator=g, device="cuda", dtype=torch.int8) for s in ((m, k), (n, k)))
    sx, sw, b = r(m) * 0.01, r(n) * 0.01, (r(n) - 0.5).to(dtype)
    acc = (xq.double() @ w.double().T).float()          # below 2^24 in magnitude or rounded as the kernel rounds its s32 sums
    want = ((acc * sx[:, None]) * sw).to(dtype)
    assert torch.equal(ops.w8a8_gemm(xq, sx, w, sw, dtype), want)
    assert torch.equal(ops.w8a8_gemm(xq, sx, w, sw, dtype, bias=b), (want.float() + b.float()).to(dtype))
    assert torch.equal(ops.w8a8_gemm(xq, sx, w, sw.to(dtype), dtype), ((acc * sx[:, None]) * sw.to(dtype).float()).to(dtype))
    x8, w8 = (torch.randn(*s, generator=g, device="cuda").to(torch.float8_e4m3fn) for s in ((m, k), (n, k)))
    one = r(1)
    y = ops.w8a8_gemm(x8.view(torch.uint8), one, w8.view(torch.uint8), sw, dtype, ops.W8_FP8 if n == 1 else 2, bias=b)
    ref = (x8.double() @ w8.double().T) * one.double() * sw.double() + b.double()
    mag = (x8.double().abs() @ w8.double().abs().T) * one.double() * sw.double()
    # an fp32 accumulator that may drop a unit in its last place per 32 products, and the output's rounding
    lim = (k / 32 + 4) * 2.0 ** -23 * mag + 2.0 ** (-11 if dtype == torch.float16 else -8) * ref.abs() + 2.0 ** -24
    assert not ((y.double() - ref).abs() > lim).any()
    assert lib.zl_gemm_tc_watchdog() == 0


@pytest.mark.parametrize("tag", ["f16", "bf16"])
@pytest.mark.parametrize("m,k", [(2, 8), (3, 2048), (3, 2056), (3, 4096), (2, 4104), (2, 8192), (2, 8200), (2, 16384), (3, 16392), (1, 40000)])
def test_int8_quant_row_lengths_bit_exact(lib, cuda, tag, m, k):
    """each number of chunks that a thread holds in registers, its first and last row length, and the form that reads rows twice"""
    from zhilight_b200 import ops
    x = _x(m, k, tag, seed=k)
    q, s = ops.int8_quant_per_token(_dev(x, tag, cuda))
    oq, os_ = oracle.int8_quant_per_token(x)
    np.testing.assert_array_equal(q.cpu().numpy(), oq)
    np.testing.assert_array_equal(s.cpu().numpy(), os_)


@pytest.mark.parametrize("m,n,k", [(24, 8192, 8192), (40, 256, 128), (40, 300, 4096), (300, 4096, 1024)])
def test_gemm_that_starts_during_the_quantisation(lib, cuda, m, n, k):
    """the GEMM's weights are fetched while the rows are still being quantised: the same bytes as one launch after the other"""
    from zhilight_b200 import ops
    w = torch.randint(-127, 128, (n, k), dtype=torch.int8, device=cuda)
    sw = torch.rand(n, device=cuda) * 0.01
    for seed in range(6):
        x = torch.randn(m, k, device=cuda, generator=torch.Generator(device=cuda).manual_seed(seed)).half()
        got = ops.int8_linear(x, w, sw)
        q, s = ops.int8_quant_per_token(x)
        torch.cuda.synchronize()
        assert torch.equal(got, ops.w8a8_gemm(q, s, w, sw, torch.float16, ops.W8_INT8))
        w8 = w.view(torch.uint8) & 0x77                  # finite fp8 codes
        one = torch.ones(1, device=cuda)
        got = ops.fp8_linear(x, w8, one)
        q, s = ops.fp8_quant_per_tensor(x)
        torch.cuda.synchronize()
        assert torch.equal(got, ops.w8a8_gemm(q, s, w8, one, torch.float16, ops.W8_FP8))


@pytest.mark.parametrize("m,n,k,splits", [(40, 8192, 8192, 2), (129, 1000, 16384, 4), (36, 2056, 8256, 4), (64, 5000, 12352, 2)])
def test_long_sums_of_few_tiles(lib, cuda, m, n, k, splits):
    """The pairs of a cluster share a tile's K: s32 sums stay exact through the exchange, e4m3 ones as near as those of one pair."""
    from zhilight_b200 import ops
    assert lib.zl_gemm_pairs_splits(m, n, k, 1, 1) == splits
    g = torch.Generator().manual_seed(m)
    x = torch.randint(-128, 128, (m, k), generator=g, dtype=torch.int8).cuda()
    w = torch.randint(-128, 128, (n, k), generator=g, dtype=torch.int8).cuda()
    sx, sw = torch.rand(m, generator=g).cuda(), torch.rand(n, generator=g).cuda()
    acc = (x.double() @ w.double().T).float()              # below 2^53, then one rounding as from s32
    y = ops.w8a8_gemm(x, sx, w, sw, torch.float16, ops.W8_INT8)
    assert torch.equal(y, (acc * sx[:, None] * sw[None]).half())
    xf, wf = (torch.randn(*s, generator=g).mul(2).to(torch.float8_e4m3fn).cuda() for s in ((m, k), (n, k)))
    one = torch.tensor([0.25], device=cuda)
    y = ops.w8a8_gemm(xf.view(torch.uint8), one, wf.view(torch.uint8), one, torch.bfloat16, ops.W8_FP8)
    ref = xf.double() @ wf.double().T / 16
    assert float((y.double() - ref).norm() / ref.norm()) <= 2.0 ** -8


@pytest.mark.parametrize("m,n,k,kind,pairs", [(8, 9472, 4480, 0, 1), (8, 9464, 4480, 0, 0), (1, 9472, 4416, 0, 0), (3, 3584, 19328, 0, 1), (3, 3576, 19328, 0, 0), (9, 5120, 4928, 0, 1),
                                              (16, 5112, 4992, 0, 0), (9, 4096, 11008, 0, 1), (16, 5120, 4864, 0, 0), (17, 512, 8192, 0, 1), (17, 2560, 8128, 0, 0),
                                              (32, 2576, 8192, 0, 1), (32, 5124, 4096, 0, 1), (32, 5116, 4096, 0, 0), (8, 5120, 8192, 1, 0), (8, 9472, 4480, 1, 1), (9, 3072, 4096, 1, 1),
                                              (16, 3064, 4224, 1, 0), (16, 3072, 4032, 1, 0), (17, 1544, 8192, 1, 1), (32, 1528, 8192, 1, 0)])
def test_line_between_the_kernels(lib, cuda, m, n, k, kind, pairs):
    """Both sides of each line of up to 32 rows: int8 exact, e4m3 within what an fp32 accumulator may drop and the output's rounding."""
    from zhilight_b200 import ops
    assert lib.zl_w8_pairs_route(m, n, k, kind) == pairs
    g = torch.Generator(device="cuda").manual_seed(n)
    sw, b = torch.rand(n, generator=g, device="cuda") * 0.01, torch.randn(n, generator=g, device="cuda").half()
    if kind == ops.W8_INT8:
        x, w = (torch.randint(-128, 128, s, generator=g, device="cuda", dtype=torch.int8) for s in ((m, k), (n, k)))
        sx = torch.rand(m, generator=g, device="cuda") * 0.01
        want = (((x.double() @ w.double().T).float() * sx[:, None]) * sw).half()
        assert torch.equal(ops.w8a8_gemm(x, sx, w, sw, torch.float16, bias=b), (want.float() + b.float()).half())
        return
    x, w = (torch.randn(*s, generator=g, device="cuda").to(torch.float8_e4m3fn) for s in ((m, k), (n, k)))
    one = torch.rand(1, generator=g, device="cuda") * 0.01
    y = ops.w8a8_gemm(x.view(torch.uint8), one, w.view(torch.uint8), sw[:1], torch.float16, ops.W8_FP8, bias=b)
    scale = one.double() * sw[:1].double()
    ref, mag = (x.double() @ w.double().T) * scale + b.double(), (x.double().abs() @ w.double().abs().T) * scale
    # the sum rounds once to fp16 ahead of the bias's addition and once behind it
    lim = (k / 32 + 4) * 2.0 ** -23 * mag + 2.0 ** -11 * (ref.abs() + (ref - b.double()).abs()) + 2.0 ** -24
    assert not ((y.double() - ref).abs() > lim).any()
