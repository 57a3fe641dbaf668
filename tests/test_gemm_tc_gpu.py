"""GPU: the general GEMM on the tensor cores (prompt-sized M) against the same products in 64 bits: edges of its 256-row and 32-row tiles
and of the 64-k stages, every epilogue, batches, and grouped rows with empty, one-row and more-than-one-tile groups."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

BF, HF = torch.bfloat16, torch.float16


def test_which_kernel(lib):
    """What the sizes below rely on: short sums of few tiles stay with the tile kernel, both sides of the line are tested."""
    route = lib.zl_gemm_nt_pairs_route
    assert [route(*s, 1) for s in ((32, 4096, 4096), (33, 128, 64), (257, 512, 200), (64, 100, 4096))] == [0, 0, 0, 0]
    assert [route(*s, 1) for s in ((33, 128, 576), (64, 136, 584), (257, 513, 576), (777, 2048, 328), (40, 4096, 512))] == [1, 1, 1, 1, 1]
    assert [route(33, 512, 128, 16), route(300, 512, 128, 16), route(33, 520, 640, 3), route(64, 640, 128, 64)] == [0, 1, 1, 1]


def _rand(g, *shape, dtype):
    return torch.randn(*shape, generator=g).to(dtype).cuda()


def _close(y, ref, mag, k, out_dtype):
    """mag: the sums of the products' magnitudes.  Every 16 products are added to an fp32 accumulator that may drop up to a unit in its last
    place, so the sum is off by at most (k / 16 + 2) 2^-23 of it; 16-bit outputs round by half a unit of theirs."""
    y, ref = y.double(), ref.double()
    lim = (k / 16 + 2) * 2.0 ** -23 * mag + (0 if out_dtype == torch.float32 else 2.0 ** (-8 if out_dtype == BF else -11)) * ref.abs()
    bad = (y - ref).abs() > lim
    assert not bad.any(), (int(bad.sum()), float((y - ref).abs().max()))


@pytest.fixture(autouse=True)
def no_wait_gave_up(lib, cuda):
    yield
    torch.cuda.synchronize()
    assert lib.zl_gemm_tc_watchdog() == 0


@pytest.mark.parametrize("dtype,out", [(BF, BF), (BF, torch.float32), (HF, HF), (HF, torch.float32)])
@pytest.mark.parametrize("m,n,k", [(33, 128, 64), (64, 136, 72), (65, 250, 136), (256, 256, 128), (257, 513, 448), (300, 520, 1000), (40, 4096, 512),
                                   (777, 2048, 328), (33, 128, 576), (64, 136, 584), (65, 250, 648), (256, 256, 640), (257, 513, 576)])
def test_plain(lib, cuda, dtype, out, m, n, k):
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(m + n)
    x, w, b = _rand(g, m, k, dtype=dtype), _rand(g, n, k, dtype=dtype), torch.randn(n, generator=g).cuda()
    ref, mag = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    _close(ops.gemm_nt(x, w, out_dtype=out), ref, mag, k, out)
    _close(ops.gemm_nt_bias(x, w, b, out_dtype=out), ref + b.double(), mag + b.double().abs(), k, out)


@pytest.mark.parametrize("dtype", [BF, HF])
@pytest.mark.parametrize("m,n,k", [(65, 128, 64), (95, 1000, 96), (512, 264, 2048)])
def test_skinny_entry_with_bias_and_activations(lib, cuda, dtype, m, n, k):
    """zl_dense_gemm_skinny's bias is of the input type; its activations; more rows than one of its 32-row passes."""
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(k)
    x, w, b = _rand(g, m, k, dtype=dtype) / 8, _rand(g, n, k, dtype=dtype), _rand(g, n, dtype=dtype)
    mul = torch.randn(m, n, generator=g).cuda()
    ref, mag = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    _close(ops.dense_gemm_skinny(x, w, b), ref + b.double(), mag + b.double().abs(), k, dtype)
    for act, want in ((1, F.relu(ref) ** 2), (2, torch.tanh(ref)), (3, F.gelu(ref, approximate="tanh") * mul.double())):
        y = ops.dense_gemm_skinny_mul(x, w, act, mul if act == 3 else None, out_dtype=torch.float32)
        assert float((y.double() - want).norm() / want.norm()) < 1e-5, act


@pytest.mark.parametrize("m,n,k", [(40, 130, 64), (257, 512, 200), (40, 130, 576), (257, 512, 648)])
def test_epilogues(lib, cuda, m, n, k):
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(n)
    x, w, mul = _rand(g, m, k, dtype=BF) / 8, _rand(g, n, k, dtype=BF), torch.randn(m, n, generator=g).cuda()
    ref = x.double() @ w.double().T
    a, u = ref[:, 0::2], ref[:, 1::2]
    ga, cu = a.clamp(max=1.5), u.clamp(-1.5, 1.5)
    rel = lambda y, want: float((y.double() - want).norm() / want.norm())  # noqa: E731
    f32 = torch.float32
    assert rel(ops.gemm_nt(x, w, f32, ops.GEMM_EPI_RELU2), F.relu(ref) ** 2) < 1e-5
    assert rel(ops.gemm_nt(x, w, f32, ops.GEMM_EPI_SIGMOID_GATE, mul), ref * torch.sigmoid(mul.double())) < 1e-5
    assert rel(ops.gemm_nt_bias(x, w, None, f32, ops.GEMM_EPI_TANH), torch.tanh(ref)) < 1e-5
    assert rel(ops.gemm_nt_fused(x, w, None, f32, ops.GEMM_EPI_GELU_TANH_MUL, mul), F.gelu(ref, approximate="tanh") * mul.double()) < 1e-5
    assert rel(ops.gemm_nt_fused(x, w, None, f32, ops.GEMM_EPI_SOFTCAP, limit=2.0), 2 * torch.tanh(ref / 2)) < 1e-5
    assert rel(ops.gemm_nt_fused(x, w, None, f32, ops.GEMM_EPI_GEGLU_TANH), F.gelu(a, approximate="tanh") * u) < 1e-5
    assert rel(ops.gemm_nt_glu_clamp(x, w, None, f32, 1.5, 1.7, 0.5), ga * torch.sigmoid(1.7 * ga) * (cu + 0.5)) < 1e-5


@pytest.mark.parametrize("b,m,n,k", [(3, 70, 128, 64), (5, 33, 300, 128), (90, 40, 512, 64), (3, 70, 128, 576), (5, 33, 300, 640)])
def test_batches(lib, cuda, b, m, n, k):
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(b)
    x, w = _rand(g, b, m, k, dtype=BF), _rand(g, b, n, k, dtype=BF)
    prod = lambda a, c: torch.einsum("bmk,bnk->bmn", a, c)  # noqa: E731
    _close(ops.gemm_nt(x, w, out_dtype=torch.float32), prod(x.double(), w.double()), prod(x.double().abs(), w.double().abs()), k, torch.float32)


@pytest.mark.parametrize("dtype,out", [(BF, torch.float32), (HF, HF)])
@pytest.mark.parametrize("m,n,k,splits", [(33, 512, 8192, 4), (65, 250, 8200, 4), (47, 4096, 6152, 2), (200, 1000, 8192, 4), (256, 3000, 10240, 4), (100, 130, 2056, 4)])
def test_long_sums_of_few_tiles(lib, cuda, dtype, out, m, n, k, splits):
    """The pairs of a cluster share a tile's K: chunks of 16 rows that go round between two and four owners, the last one of 1 to 16, parts of unequal
    length, epilogues behind the exchange, the same result each time."""
    from zhilight_b200 import ops
    assert lib.zl_gemm_pairs_splits(m, n, k, 1, 2) == splits
    g = torch.Generator().manual_seed(m + n)
    x, w, b = _rand(g, m, k, dtype=dtype), _rand(g, n, k, dtype=dtype), torch.randn(n, generator=g).cuda()
    ref, mag = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    y = ops.gemm_nt_bias(x, w, b, out_dtype=out)
    _close(y, ref + b.double(), mag + b.double().abs(), k, out)
    assert torch.equal(y, ops.gemm_nt_bias(x, w, b, out_dtype=out))
    y = ops.gemm_nt(x, w, torch.float32, ops.GEMM_EPI_RELU2)
    assert float((y.double() - F.relu(ref) ** 2).norm() / (F.relu(ref) ** 2).norm()) < 1e-5
    xb, wb = _rand(g, 2, 40, k, dtype=dtype), _rand(g, 2, 300, k, dtype=dtype)
    assert lib.zl_gemm_pairs_splits(40, 300, k, 2, 2) > 1
    prod = lambda a, c: torch.einsum("bmk,bnk->bmn", a, c)  # noqa: E731
    _close(ops.gemm_nt(xb, wb, out_dtype=out), prod(xb.double(), wb.double()), prod(xb.double().abs(), wb.double().abs()), k, out)


@pytest.mark.parametrize("b,m,n,k,pairs", [(1, 33, 128, 200, 0), (1, 33, 128, 216, 1), (1, 200, 256, 256, 1), (1, 384, 2050, 256, 1), (16, 33, 512, 136, 0), (16, 256, 128, 64, 0),
                                            (48, 200, 250, 128, 1), (48, 33, 1024, 256, 1), (4, 384, 512, 72, 0)])
def test_line_to_the_tile_kernel(lib, cuda, b, m, n, k, pairs):
    """Both sides of the line of short sums, at one to forty-eight matrices."""
    from zhilight_b200 import ops
    assert lib.zl_gemm_nt_pairs_route(m, n, k, b) == pairs
    g = torch.Generator().manual_seed(k)
    x, w = _rand(g, b, m, k, dtype=BF), _rand(g, b, n, k, dtype=BF)
    prod = lambda a, c: torch.einsum("bmk,bnk->bmn", a, c)  # noqa: E731
    _close(ops.gemm_nt(x, w, out_dtype=torch.float32), prod(x.double(), w.double()), prod(x.double().abs(), w.double().abs()), k, torch.float32)


@pytest.mark.parametrize("dtype", [BF, HF])
@pytest.mark.parametrize("sizes", [[0, 9, 1, 0, 31], [32, 33, 0, 64, 1], [1] * 150, [256, 0, 257, 3], [700, 12]])
@pytest.mark.parametrize("n,k", [(128, 64), (300, 200), (512, 520)])
def test_grouped(lib, cuda, dtype, sizes, n, k):
    from zhilight_b200 import ops
    rng = np.random.default_rng(sum(sizes) + n)
    g = torch.Generator().manual_seed(n)
    total, groups = sum(sizes), len(sizes)
    t = total // 2 + 1                                  # rows of x: several list entries share one
    x, w = _rand(g, t, k, dtype=dtype) / 8, _rand(g, groups, n, k, dtype=dtype)
    off = torch.tensor(np.concatenate([[0], np.cumsum(sizes)]), dtype=torch.int32, device="cuda")
    rows = torch.tensor(rng.integers(0, t, total), dtype=torch.int32, device="cuda")
    back = torch.tensor(rng.permutation(total), dtype=torch.int32, device="cuda")
    owner = torch.repeat_interleave(torch.arange(groups), torch.tensor(sizes)).cuda()
    prod = lambda a, c: torch.einsum("rk,rnk->rn", a[rows.long()], c[owner])  # noqa: E731
    ref, mag = prod(x.double(), w.double()), prod(x.double().abs(), w.double().abs())
    a, u = ref[:, 0::2].clamp(max=1.0), ref[:, 1::2].clamp(-1.0, 1.0)
    y = ops.gemm_nt_grouped(x, w, off, total, x_rows=rows, out_dtype=torch.float32, epilogue=ops.GEMM_EPI_GLU_CLAMP, limit=1.0, alpha=1.7, beta=1.0)
    want = a * torch.sigmoid(1.7 * a) * (u + 1)
    assert float((y.double() - want).norm() / want.norm()) < 1e-5
    xs = x[rows.long()].contiguous()
    y = ops.gemm_nt_grouped(xs, w, off, total, y_rows=back, out_dtype=torch.float32)
    _close(y[back.long()], ref, mag, k, torch.float32)
    _close(ops.gemm_nt_grouped(x, w, off, total, x_rows=rows), ref, mag, k, dtype)


@pytest.mark.parametrize("dtype", [BF, HF])
@pytest.mark.parametrize("sizes,n", [([40], 132), ([47], 130), ([257, 0, 300, 1], 516), ([16, 33, 500], 1026)])
def test_gated_units_of_16_bits(lib, cuda, dtype, sizes, n):
    """Two columns of a gated unit per store (n % 4 == 0) and one (n % 4 == 2); chunks of 16 rows with 1 to 16 in them, groups of several tiles.  Half a unit of the
    output's last place, 2^-9 (2^-12) of a value on average, and what fp32 sums of values of about 1 lose."""
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(n)
    total, k = sum(sizes), 576
    x, w = _rand(g, total, k, dtype=dtype) / 8, _rand(g, len(sizes), n, k, dtype=dtype)
    off = torch.tensor(np.concatenate([[0], np.cumsum(sizes)]), dtype=torch.int32, device="cuda")
    back = torch.randperm(total, generator=g).to(torch.int32).cuda()
    owner = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)).cuda()
    ref = torch.cat([x[owner == i].double() @ w[i].double().T for i in range(len(sizes))])
    a, u = ref[:, 0::2].clamp(max=1.5), ref[:, 1::2].clamp(-1.5, 1.5)
    want = a * torch.sigmoid(1.7 * a) * (u + 0.5)
    tol = 2.0 ** (-8 if dtype == BF else -11)
    rel = lambda y, want: float(((y.double() - want).norm(dim=1) / want.norm(dim=1)).max())  # noqa: E731
    y = ops.gemm_nt_grouped(x, w, off, total, y_rows=back, epilogue=ops.GEMM_EPI_GLU_CLAMP, limit=1.5, alpha=1.7, beta=0.5)
    assert rel(y[back.long()], want) < tol
    if len(sizes) == 1:
        assert rel(ops.gemm_nt_glu_clamp(x, w[0], None, dtype, 1.5, 1.7, 0.5), want) < tol
        assert rel(ops.gemm_nt_fused(x, w[0], None, dtype, ops.GEMM_EPI_GEGLU_TANH), F.gelu(ref[:, 0::2], approximate="tanh") * ref[:, 1::2]) < tol


@pytest.mark.parametrize("rows_out,listed,n,out", [(33, 20, 512, BF), (4000, 3990, 512, torch.float32), (4111, 0, 256, torch.float32), (4100, 4100, 520, HF), (2600, 30, 1030, BF)])
def test_rows_that_no_entry_lands_on(lib, cuda, rows_out, listed, n, out):
    """They are zeros, whatever the memory held: few, most, none and all rows listed, slices of the last partial one, rows of no multiple of 16 bytes, an output
    so small that it is written whole first; with and without a list of y's rows."""
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(rows_out)
    k = 128
    dtype = BF if out == torch.float32 else out
    x, w = _rand(g, max(listed, 1), k, dtype=dtype), _rand(g, 3, n, k, dtype=dtype)
    off = torch.tensor([0, listed // 3, listed // 2, listed], dtype=torch.int32, device="cuda")
    rows = torch.arange(max(listed, 1), dtype=torch.int32, device="cuda")
    for back in (None, torch.randperm(rows_out, generator=g)[:max(listed, 1)].to(torch.int32).cuda()):
        junk = torch.full((rows_out, n), float("nan"), dtype=out, device=cuda)
        del junk                                        # the allocator's next block of this size
        y = ops.gemm_nt_grouped(x, w, off, rows_out, x_rows=rows, y_rows=back, out_dtype=out)
        free = torch.ones(rows_out, dtype=torch.bool, device=cuda)
        free[(rows if back is None else back.long())[:listed]] = False
        assert int(free.sum()) == rows_out - listed and not y[free].any() and (listed == 0 or bool((y[~free].abs().sum(1) > 0).all()))


@pytest.mark.parametrize("k", [128, 640])
def test_infinities_stay_in_their_rows_and_columns(lib, cuda, k):
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(1)
    x, w = _rand(g, 70, k, dtype=BF), _rand(g, 256, k, dtype=BF)
    good = ops.gemm_nt(x, w, out_dtype=torch.float32)
    x[69, 3], w[17, 5] = float("inf"), float("nan")
    bad = ops.gemm_nt(x, w, out_dtype=torch.float32)
    assert not torch.isfinite(bad[69]).any() and torch.isnan(bad[:, 17]).all()
    keep = torch.ones_like(bad, dtype=torch.bool)
    keep[69], keep[:, 17] = False, False
    assert torch.equal(bad[keep], good[keep])


def _nt(lib, x, xb, ldx, w, wb, ldw, y, yb, ldy, m, n, k, batch, epilogue=0, gate=None, gb=0, ldg=0):
    """zl_gemm_nt on tensors of any pitches (elements)."""
    from zhilight_b200 import _lib, ops
    _lib.call("zl_gemm_nt", x.data_ptr(), ldx, xb, w.data_ptr(), ldw, wb, y.data_ptr(), ldy, yb, m, n, k, batch, ops._dt(x), ops._dt(y),
              epilogue, gate.data_ptr() if gate is not None else None, ldg, gb, 0, torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("dtype", [BF, HF])
@pytest.mark.parametrize("t", [33, 64, 300])
@pytest.mark.parametrize("h,d,r,rs", [(16, 128, 512, 512), (5, 128, 512, 576), (3, 192, 136, 140), (3, 640, 520, 576), (64, 128, 640, 640)])
def test_heads_as_the_batch(lib, cuda, dtype, t, h, d, r, rs):
    """The latent layers' products: pitch between heads smaller than the row pitch, for x and y; y's rows longer than its columns; the
    way back with a gate that is part of a wider row."""
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(t + r)
    q, uk = _rand(g, t, h, d, dtype=dtype), _rand(g, h, r, d, dtype=dtype)
    y = torch.full((t, h, rs), -7.0, device=cuda)
    _nt(lib, q, d, h * d, uk, r * d, d, y, rs, h * rs, t, r, d, h)
    prod = lambda a, c: torch.einsum("thd,hrd->thr", a.double(), c.double())  # noqa: E731
    _close(y[:, :, :r], prod(q, uk), prod(q.abs(), uk.abs()), d, torch.float32)
    assert bool((y[:, :, r:] == -7.0).all())
    lat, uv = _rand(g, t, h, r, dtype=dtype) / 8, _rand(g, h, d, r, dtype=dtype)
    wide = torch.randn(t, 24 + h * d, generator=g).cuda()
    gate = wide[:, 24:]
    for epilogue in (ops.GEMM_EPI_NONE, ops.GEMM_EPI_SIGMOID_GATE):
        out = torch.zeros(t, h, d, dtype=dtype, device=cuda)
        _nt(lib, lat, r, h * r, uv, d * r, r, out, d, h * d, t, d, r, h, epilogue, gate, d, wide.shape[1])
        s = torch.sigmoid(gate.double()).reshape(t, h, d) if epilogue else torch.ones(t, h, d, dtype=torch.float64, device=cuda)
        _close(out, prod(lat, uv) * s, prod(lat.abs(), uv.abs()) * s * 1.01, r + 64, dtype)   # + 64: a few units of fp32 for the sigmoid


@pytest.mark.parametrize("k", [128, 576])
@pytest.mark.parametrize("ldx,ldw,ldy,pad", [(8, 0, 200, 0), (896, 392, 130, 1), (0, 0, 129, 3)])
def test_row_pitches_and_odd_distances(lib, cuda, k, ldx, ldw, ldy, pad):
    """Rows apart from each other; an output whose rows, matrices and base are no multiples of two values (narrow stores)."""
    g = torch.Generator().manual_seed(ldx)
    b, m, n, ldx, ldw = 3, 45, 128, k + ldx, k + ldw
    x, w = _rand(g, b, m, ldx, dtype=BF), _rand(g, b, n, ldw, dtype=BF)
    flat = torch.full((pad + b * (m * ldy + pad),), -7.0, dtype=BF, device=cuda)
    y = flat[pad:]
    yb = m * ldy + pad
    _nt(lib, x, m * ldx, ldx, w, n * ldw, ldw, y, yb, ldy, m, n, k, b)
    xs, ws = x[:, :, :k].double(), w[:, :, :k].double()
    ref, mag = torch.einsum("bmk,bnk->bmn", xs, ws), torch.einsum("bmk,bnk->bmn", xs.abs(), ws.abs())
    for i in range(b):
        _close(y[i * yb:i * yb + m * ldy].reshape(m, ldy)[:, :n], ref[i], mag[i], k, BF)
    touched = torch.zeros_like(flat, dtype=torch.bool)
    for i in range(b):
        touched[pad + i * yb:pad + i * yb + m * ldy].reshape(m, ldy)[:, :n] = True
    assert bool((flat[~touched] == -7.0).all())


_FEW_ROWS = """
import sys, torch
sys.path.insert(0, sys.argv[1])
from zhilight_b200 import ops
g = torch.Generator(device="cuda").manual_seed(1)
groups, n, k, m = 8, 2048, 4096, 20                      # large enough for the tensor-core kernel from 9 rows on
x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
w = torch.randn(groups, n, k, generator=g, device="cuda").bfloat16()
owner = torch.arange(m, device="cuda") * groups // m
def call(lo, hi):
    off = torch.zeros(groups + 1, dtype=torch.int32, device="cuda")
    off[1:] = torch.bincount(owner[lo:hi], minlength=groups).cumsum(0)
    return ops.gemm_nt_grouped(x[lo:hi].contiguous(), w, off, hi - lo, out_dtype=torch.float32)
whole, parts = call(0, m), torch.cat([call(i, min(i + 8, m)) for i in range(0, m, 8)])
print("SAME" if torch.equal(whole, parts) else "OTHER")
"""


@pytest.mark.parametrize("limit,want", [("32", "SAME"), (None, "OTHER")])
def test_row_limit_of_the_few_rows_kernel(cuda, limit, want):
    """ZL_GEMM_GROUPED_SMALL_MAX keeps the rows of a step up to that count with the few-rows kernel, whose sums do not depend on how many rows there
    are; without it 20 rows of large matrices take the tensor-core kernel, which adds in another order."""
    import os
    import subprocess
    import sys
    env = {k: v for k, v in os.environ.items() if k != "ZL_GEMM_GROUPED_SMALL_MAX"}
    if limit:
        env["ZL_GEMM_GROUPED_SMALL_MAX"] = limit
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _FEW_ROWS, root], env=env, capture_output=True, text=True, timeout=300)
    assert r.stdout.split() == [want], r.stdout + r.stderr


@pytest.mark.parametrize("captured", [False, True])
def test_starts_under_its_predecessors_end(lib, cuda, captured):
    """Inputs that the launch before is still writing, on this stream and behind another one's event; and a dependent that reads its weights ahead of its
    own wait: they were written before this kernel, whose early start must not let the dependent overtake the writer."""
    from zhilight_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(0)
    m, n, k = 100, 512, 1024
    src = [torch.randn(*s, generator=g, device=cuda).bfloat16() for s in ((m, k), (n, k), (256, n))]
    x, w, w2 = (torch.zeros_like(t) for t in src)
    ref = src[0].float() @ src[1].float().T
    side = torch.cuda.Stream()

    def step():
        torch.cuda._sleep(200_000)
        for d, s in zip((w2, x), (src[2], src[0])):
            d.copy_(s)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            torch.cuda._sleep(200_000)
            w.copy_(src[1])
        torch.cuda.current_stream().wait_stream(side)
        y = ops.dense_gemm_skinny(x, w)
        return y, ops.dense_gemm_skinny(y[:16], w2, pdl=True)
    ops.dense_gemm_skinny(src[0], src[1])                             # prepared outside of the capture
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y, z = step()
    for _ in range(3):
        for t in (x, w, w2):
            t.zero_()
        if captured:
            graph.replay()
        else:
            y, z = step()
        torch.cuda.synchronize()
        assert ((y.float() - ref).norm() / ref.norm()).item() <= 4e-3    # bf16's rounding is at most 2^-9 of a value, fp32 sums are far below
        want = y[:16].float() @ src[2].float().T
        assert ((z.float() - want).norm() / want.norm()).item() <= 4e-3
