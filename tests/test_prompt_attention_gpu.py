"""GPU: attention of several query rows per task (portions of a prompt, tree rows) against the oracle, at the edges of the kernel's
128-row blocks and 64-key tiles, with masks of any shape, key splits and both cache layouts."""
import numpy as np
import pytest
import torch

from oracle import ops as oops
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

# fp16 / bf16 output rounding (2^-12 / 2^-9 of a value on average) plus as much again for the rounding of the probabilities
TOL = {torch.float16: ("f16", 1e-3), torch.bfloat16: ("bf16", 6e-3)}


@pytest.fixture(autouse=True)
def no_wait_gave_up(lib):
    yield
    assert lib.zl_prompt_attention_watchdog() == 0


def _run(cuda, dtype, lens, len_q, hq, hkv, d, masks, bshd=True, seed=0):
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(seed)
    q = torch.randn(len(lens), len_q, hq, d, generator=g).to(dtype)
    shapes = [(n, hkv, d) if bshd else (hkv, n, d) for n in lens]
    ks = [torch.randn(*s, generator=g).to(dtype) for s in shapes]
    vs = [torch.randn(*s, generator=g).to(dtype) for s in shapes]
    flat = None if masks is None else torch.cat([m.reshape(-1) for m in masks]).to(cuda)
    out = ops.decode_attention(q.to(cuda), torch.tensor(lens, dtype=torch.int32, device=cuda), [k.to(cuda) for k in ks], [v.to(cuda) for v in vs],
                               flat, d ** -0.5, max(lens), hkv, bshd=bshd).float().cpu().numpy()
    nat = [[t.float().numpy() if bshd else t.float().permute(1, 0, 2).contiguous().numpy() for t in x] for x in (ks, vs)]
    ones = [np.ones((len_q, n), np.int8) for n in lens]
    ref = oops.decode_attention(q.float().numpy(), nat[0], nat[1], lens, ones if masks is None else [m.numpy() for m in masks], d ** -0.5, hq // hkv,
                                TOL[dtype][0])
    return out, np.asarray(ref)


def _causal(len_q, n):
    return (torch.arange(n)[None, :] <= torch.arange(n - len_q, n)[:, None]).to(torch.int8)


@pytest.mark.parametrize("dtype", list(TOL))
@pytest.mark.parametrize("hq,hkv,d", [(8, 2, 128), (4, 4, 64), (9, 3, 64), (16, 1, 128)])
@pytest.mark.parametrize("len_q,ctx", [(16, 16), (17, 63), (64, 65), (160, 160), (321, 321), (330, 515), (1030, 1030)])
def test_causal_portions(lib, cuda, dtype, hq, hkv, d, len_q, ctx):
    """Both sides of the dispatch line."""
    out, ref = _run(cuda, dtype, [ctx], len_q, hq, hkv, d, [_causal(len_q, ctx)])
    tol = TOL[dtype][1]
    assert rel_l2(out, ref) <= tol
    for i in (0, len_q // 2, len_q - 1):                # single rows: a wrong row or head cannot hide in the whole
        for h in (0, hq - 1):
            assert rel_l2(out[0, i, h], ref[0, i, h]) <= 4 * tol, (i, h)


@pytest.mark.parametrize("bshd", [True, False])
@pytest.mark.parametrize("masked", [True, False])
def test_ragged_tasks_and_any_mask(lib, cuda, bshd, masked):
    lens, len_q = [200, 33, 1, 128], 41
    g = torch.Generator().manual_seed(4)
    masks = [(torch.rand(len_q, n, generator=g) < 0.4).to(torch.int8) * 3 for n in lens] if masked else None   # any non-zero byte is visible
    if masked:
        masks[0][5] = 0                                 # rows that see nothing give zeros
        masks[2][:] = 0
        masks[3][:, :100] = 0                           # whole tiles without a visible key before the visible ones
    out, ref = _run(cuda, torch.float16, lens, len_q, 8, 2, 128, masks, bshd, seed=1)
    assert rel_l2(out, ref) <= 1e-3
    if masked:
        assert not out[0, 5].any() and not out[2].any()


@pytest.mark.parametrize("len_q,ctx", [(33, 1500), (40, 2049)])
def test_key_splits(lib, cuda, len_q, ctx):
    """Few row blocks over many keys: the keys are split and merged."""
    out, ref = _run(cuda, torch.bfloat16, [ctx], len_q, 4, 1, 128, [_causal(len_q, ctx)], seed=2)
    assert rel_l2(out, ref) <= 6e-3


def test_infinities_and_nans_stay_in_their_rows(lib, cuda):
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(3)
    q, k, v = (torch.randn(*s, generator=g).half() for s in ((1, 320, 4, 128), (384, 1, 128), (384, 1, 128)))
    q[0, 3, 1, 7] = float("inf")
    q[0, 9, 2, 0] = float("nan")
    mask = _causal(320, 384).to(cuda)
    call = lambda q_: ops.decode_attention(q_.to(cuda), torch.tensor([384], dtype=torch.int32, device=cuda), [k.to(cuda)], [v.to(cuda)],  # noqa: E731
                                           mask, 0.125, 384, 1)
    bad = call(q)
    q[0, 3, 1] = q[0, 9, 2] = 0
    good = call(q)
    assert torch.isnan(bad[0, 3, 1]).all() and torch.isnan(bad[0, 9, 2]).all()
    keep = torch.ones(320, 4, dtype=torch.bool, device=cuda)
    keep[3, 1] = keep[9, 2] = False
    assert torch.equal(bad[0][keep], good[0][keep])


def _exact(q, k, v, visible, scale):
    """q (m, h, d), k and v (n, hk, d), visible (m, n) in 64 bits on the CPU"""
    m, h, d = q.shape
    g = h // k.shape[1]
    s = torch.einsum("mhd,nhd->hmn", q.double(), k.double().repeat_interleave(g, 1)) * scale
    s = s.masked_fill(visible[None] == 0, -torch.inf)
    return torch.einsum("hmn,nhd->mhd", torch.softmax(s, -1), v.double().repeat_interleave(g, 1))


@pytest.mark.parametrize("dtype", list(TOL))
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("rise", [0.02, 0.5])
def test_maxima_that_grow_along_the_keys(lib, cuda, dtype, d, rise):
    """Scores that rise by rise / ln 2 bits a key (the output is a mean over the last keys a row sees): a row's reference maximum has to follow,
    now by less than the kernel lets it stay behind, now in every tile."""
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(5)
    m, n, h = 192, 640, 8
    q, k, v = (torch.randn(*s, generator=g) for s in ((m, h, d), (n, 2, d), (n, 2, d)))
    q[:, :, 0], k[:, :, 0] = 4.0, (torch.arange(n) * (rise * d ** 0.5 / 4)).round(decimals=2)[:, None]
    q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
    mask = _causal(m, n)
    out = ops.decode_attention(q[None].to(cuda), torch.tensor([n], dtype=torch.int32, device=cuda), [k.to(cuda)], [v.to(cuda)], mask.to(cuda), d ** -0.5,
                               n, 2)[0]
    assert rel_l2(out.double().cpu().numpy(), _exact(q, k, v, mask, d ** -0.5).numpy()) <= TOL[dtype][1]


@pytest.mark.parametrize("hq,hkv,d,len_q,ctx", [(1, 1, 128, 127, 513), (1, 1, 128, 128, 512), (1, 1, 128, 129, 511), (3, 1, 64, 341, 1025),
                                                (8, 8, 128, 130, 130), (16, 2, 128, 50, 2100), (64, 8, 128, 33, 700), (32, 8, 64, 257, 1400)])
def test_blocks_of_rows_and_clusters_of_splits(lib, cuda, hq, hkv, d, len_q, ctx):
    """A row more or less than a block, keys in one to eight parts, q on 4 bytes, a negative scale and one of zero."""
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(6)
    q, k, v = (torch.randn(*s, generator=g).bfloat16() for s in ((len_q, hq, d), (ctx, hkv, d), (ctx, hkv, d)))
    room = torch.empty(q.numel() + 2, dtype=q.dtype, device=cuda)
    shifted = room[2:].view(1, len_q, hq, d)
    shifted.copy_(q)
    mask, lens = _causal(len_q, ctx), torch.tensor([ctx], dtype=torch.int32, device=cuda)
    for qd in (q[None].to(cuda), shifted):
        for scale in (d ** -0.5, -d ** -0.5, 0.0):
            out = ops.decode_attention(qd, lens, [k.to(cuda)], [v.to(cuda)], mask.to(cuda), scale, ctx, hkv)[0]
            assert rel_l2(out.double().cpu().numpy(), _exact(q, k, v, mask, scale).numpy()) <= TOL[torch.bfloat16][1], (qd is shifted, scale)


@pytest.mark.parametrize("d,len_q,ctx,hq,hkv,ranges", [(128, 107, 2600, 16, 2, 8), (64, 110, 4090, 16, 2, 8), (128, 100, 800, 16, 4, 4), (64, 217, 1500, 8, 8, 4), (128, 268, 4070, 8, 1, 8),
                                                       (128, 107, 2600, 8, 1, 8), (64, 91, 2600, 64, 8, 2), (128, 512, 512, 4, 4, 4)])
def test_ranges_and_places(lib, cuda, d, len_q, ctx, hq, hkv, ranges):
    """Both sides of the line to eight ranges: 14 groups, of which each CTA has an SM for itself, and 16 or 17 of many and of few keys; clusters that fill half of the SMs,
    behind the mask's kernel."""
    from zhilight_b200 import ops
    assert lib.zl_prompt_attention_ranges(1, len_q, hq, hkv, ctx) == ranges
    g = torch.Generator().manual_seed(len_q)
    q, k, v = (torch.randn(*s, generator=g).half() for s in ((len_q, hq, d), (ctx, hkv, d), (ctx, hkv, d)))
    mask, lens = _causal(len_q, ctx), torch.tensor([ctx], dtype=torch.int32, device=cuda)
    outs = [ops.decode_attention(q[None].to(cuda), lens, [k.to(cuda)], [v.to(cuda)], mask.to(cuda), d ** -0.5, ctx, hkv)[0] for _ in range(3)]
    assert rel_l2(outs[0].double().cpu().numpy(), _exact(q, k, v, mask, d ** -0.5).numpy()) <= TOL[torch.float16][1]
    assert all(torch.equal(o, outs[0]) for o in outs)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("hkv", [1, 4, 16])
@pytest.mark.parametrize("masked", [True, False])
def test_ranges_without_a_key(lib, cuda, d, hkv, masked):
    """Clusters of eight, four and two key ranges of which some have no tile: their CTAs come to the merge as soon as they run, whatever the others do.  Calls in a
    row on changing inputs, each against the same call alone, the last one against 64 bits."""
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(8)
    lens, len_q = [1500, 1, 64, 130], 33
    n = torch.tensor(lens, dtype=torch.int32, device=cuda)
    masks = [(torch.arange(m)[None, :] <= torch.arange(len_q)[:, None]).to(torch.int8) if i % 2 == 0 else torch.ones(len_q, m, dtype=torch.int8) for i, m in enumerate(lens)]
    flat = torch.cat([m.reshape(-1) for m in masks]).to(cuda) if masked else None
    sets = [(torch.randn(4, len_q, 4 * hkv, d, generator=g).half(), *([torch.randn(m, hkv, d, generator=g).half() for m in lens] for _ in range(2))) for _ in range(3)]
    on = [(q.to(cuda), [t.to(cuda) for t in k], [t.to(cuda) for t in v]) for q, k, v in sets]
    call = lambda q, k, v: ops.decode_attention(q, n, k, v, flat, d ** -0.5, max(lens), hkv)  # noqa: E731
    torch.cuda.synchronize()
    row = [call(*a) for a in on for _ in range(4)]
    torch.cuda.synchronize()
    for i, a in enumerate(on):
        alone = call(*a)
        torch.cuda.synchronize()
        assert all(torch.equal(o, alone) for o in row[4 * i:4 * i + 4])
    q, k, v = sets[-1]
    for i in range(4):
        ref = _exact(q[i], k[i], v[i], masks[i] if masked else torch.ones(len_q, lens[i]), d ** -0.5)
        assert rel_l2(row[-1][i].double().cpu().numpy(), ref.numpy()) <= 1e-3, i


@pytest.mark.parametrize("d,len_q,ctx", [(128, 200, 333), (64, 100, 1100), (128, 3, 40)])
def test_layers_that_share_a_mask(lib, cuda, d, len_q, ctx):
    """The second call uses the bits that the first one left (also where the decode kernels serve it, which have none), the third derives them again."""
    from zhilight_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(5)
    hq, hkv = 8, 2
    q = torch.randn(1, len_q, hq, d, generator=g, device=cuda).half()
    k, v = (torch.randn(ctx, hkv, d, generator=g, device=cuda).half() for _ in range(2))
    lens = torch.tensor([ctx], dtype=torch.int32, device=cuda)
    mask, other = _causal(len_q, ctx).to(cuda), (torch.rand(len_q, ctx, generator=g, device=cuda) < 0.5).to(torch.int8)
    table = torch.tensor([k.data_ptr(), v.data_ptr()], dtype=torch.int64, device=cuda)
    size = lib.zl_decode_attention_workspace_bytes(1, len_q, hq, d, ctx)
    ws = torch.empty(size, dtype=torch.uint8, device=cuda)

    def call(m):
        out = torch.empty_like(q)
        _lib.call("zl_decode_attention", q.data_ptr(), lens.data_ptr(), table.data_ptr(), table.data_ptr() + 8, m.data_ptr(), d ** -0.5, ctx, out.data_ptr(), 1,
                  len_q, hq, hkv, d, 1, ws.data_ptr(), size, ops.F16, 0, torch.cuda.current_stream().cuda_stream)
        return out
    first = call(mask)
    lib.zl_decode_attention_same_mask()
    assert torch.equal(call(mask), first)
    third = call(other)
    assert not torch.equal(third, first)
    assert torch.equal(third, ops.decode_attention(q, lens, [k], [v], other, d ** -0.5, ctx, hkv))
