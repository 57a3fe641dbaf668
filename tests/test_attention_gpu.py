"""GPU parity: batch decode attention over per-task ragged KV buffers vs the oracle
(reference semantics attention_kernel.cu:434-489, 674-725, 730-923)."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import ops as oops
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


def _case(cuda, dtype, name, hq, hkv, d, lens, len_q=1, masked=True, seed=0, bshd=True):
    from zhilight_b200 import ops
    g = torch.Generator().manual_seed(seed)
    b = len(lens)
    q = torch.randn(b, len_q, hq, d, generator=g).to(dtype)
    ks, vs, masks = [], [], []
    for lb in lens:
        shape = (lb, hkv, d) if bshd else (hkv, lb, d)
        ks.append(torch.randn(*shape, generator=g).to(dtype))
        vs.append(torch.randn(*shape, generator=g).to(dtype))
        m = torch.ones(len_q, lb, dtype=torch.int8)
        if masked:
            for qi in range(len_q):
                valid = max(1, lb - 2 - 3 * qi)           # the reference's len_buf is padded past the tokens
                m[qi, valid:] = 0
                m[qi, torch.randperm(valid, generator=g)[: valid // 7]] = 0   # beam-tree style holes
        masks.append(m)
    scale = 1.0 / np.sqrt(d)
    mask_flat = torch.cat([m.reshape(-1) for m in masks]).to(cuda)
    out = ops.decode_attention(q.to(cuda), torch.tensor(lens, dtype=torch.int32, device=cuda),
                               [k.to(cuda) for k in ks], [v.to(cuda) for v in vs], mask_flat if masked else None,
                               scale, max(lens), hkv, bshd=bshd)
    kn = [k.float().numpy() if bshd else k.float().permute(1, 0, 2).contiguous().numpy() for k in ks]
    vn = [v.float().numpy() if bshd else v.float().permute(1, 0, 2).contiguous().numpy() for v in vs]
    ref = oops.decode_attention(q.float().numpy(), kn, vn, lens, [m.numpy() for m in masks], scale, hq // hkv, name)
    return out.float().cpu().numpy(), ref


@pytest.mark.parametrize("dtype,name,tol", [(torch.float16, "f16", 1e-3), (torch.bfloat16, "bf16", 6e-3)])
@pytest.mark.parametrize("hq,hkv,d", [(32, 8, 128), (32, 8, 64), (8, 1, 128), (16, 16, 64), (64, 8, 128), (32, 2, 128)])
def test_gqa_shapes(lib, cuda, dtype, name, tol, hq, hkv, d):
    out, ref = _case(cuda, dtype, name, hq, hkv, d, [130, 64, 17, 1])
    assert rel_l2(out, ref) <= tol
    # per (task, head) as well: a wrong head/task mapping cannot hide in the global norm
    for b in range(out.shape[0]):
        for h in range(hq):
            assert rel_l2(out[b, 0, h], ref[b, 0, h]) <= 4 * tol, (b, h)


@pytest.mark.parametrize("lens", [[4096, 123], [2048] * 3, [1500, 700, 3000, 64, 65], [1], [16], [15, 33]])
def test_split_kv_and_ragged_lengths(lib, cuda, lens):
    """src/nn/tests/test_attention_rag_buffer.cpp uses lens {4096, 123}, 4 kv-heads x m_query 4."""
    out, ref = _case(cuda, torch.float16, "f16", 16, 4, 128, lens, seed=1)
    assert rel_l2(out, ref) <= 1e-3


def test_no_mask_and_beam_queries(lib, cuda):
    out, ref = _case(cuda, torch.float16, "f16", 8, 2, 128, [300, 90], len_q=3, masked=True, seed=2)
    assert rel_l2(out, ref) <= 1e-3
    out, ref = _case(cuda, torch.float16, "f16", 8, 2, 128, [300, 90], len_q=1, masked=False, seed=3)
    assert rel_l2(out, ref) <= 1e-3


def test_hsd_layout(lib, cuda):
    out, ref = _case(cuda, torch.float16, "f16", 8, 2, 64, [200, 40], seed=4, bshd=False)
    assert rel_l2(out, ref) <= 1e-3


def test_fully_masked_row_is_zero_not_nan(lib, cuda):
    from zhilight_b200 import ops
    q = torch.randn(1, 1, 4, 64, device=cuda).half()
    k = [torch.randn(32, 1, 64, device=cuda).half()]
    v = [torch.randn(32, 1, 64, device=cuda).half()]
    mask = torch.zeros(32, dtype=torch.int8, device=cuda)
    out = ops.decode_attention(q, torch.tensor([32], dtype=torch.int32, device=cuda), k, v, mask, 0.125, 32, 1)
    assert torch.isfinite(out).all() and out.abs().max() < 1e-6     # sum seeded with 1e-20 (attention_kernel.cu:466)


@pytest.mark.parametrize("dtype,name,tol", [(torch.float16, "f16", 1e-3), (torch.bfloat16, "bf16", 6e-3)])
@pytest.mark.parametrize("hq,hkv,d,longest,tasks", [(8, 2, 128, 700, 3), (4, 4, 64, 257, 2), (8, 1, 128, 2048, 2), (16, 8, 128, 2000, 2), (16, 2, 128, 1000, 4),   # 256-key CTAs: 3, 2, 8, 8, 4 splits
                                                    (8, 4, 128, 4096, 32), (8, 4, 128, 4096, 40), (16, 8, 128, 1100, 40), (8, 8, 64, 1030, 40),
                                                    (16, 16, 64, 2900, 24)])                                             # 1024-key CTAs: 4, 4, 2, 2, 3
def test_splits_that_merge_in_a_cluster(lib, cuda, dtype, name, tol, hq, hkv, d, longest, tasks):
    """Both sides of the lines to the merge in a launch of its own and to three CTAs per SM; splits without a key, heads of a partial group."""
    lens = ([longest, 1, 17, longest // 4 + 1] + [40 + i for i in range(tasks)])[:tasks]
    for masked in (True, False):
        out, ref = _case(cuda, dtype, name, hq, hkv, d, lens, masked=masked, seed=6)
        for b in range(min(tasks, 6)):
            assert rel_l2(out[b], ref[b]) <= 2 * tol, b
        assert rel_l2(out, ref) <= tol


@pytest.mark.parametrize("tasks,len_q,hq,hkv,longest", [(1, 1, 8, 2, 300), (2, 20, 8, 2, 200), (1, 150, 8, 2, 150), (1, 40, 32, 4, 700), (32, 1, 4, 1, 40), (33, 1, 4, 1, 40),
                                                        (20, 1, 8, 8, 900)])
@pytest.mark.parametrize("masked", [True, False])
def test_addresses_from_the_host(lib, cuda, tasks, len_q, hq, hkv, longest, masked):
    """With the call's first kernel (up to 32 tasks and a CTA per SM) and through a table the call writes: the same bits as through a table of the caller's, in a
    row of calls on changing buffers."""
    from zhilight_b200 import _lib, ops
    d = 128
    g = torch.Generator().manual_seed(tasks)
    lens = [max(len_q, longest - 7 * i) for i in range(tasks)]
    n = torch.tensor(lens, dtype=torch.int32, device=cuda)
    mask = torch.cat([(torch.rand(len_q, m, generator=g) < 0.7).to(torch.int8).reshape(-1) for m in lens]).to(cuda) if masked else None
    ws_bytes = lib.zl_decode_attention_workspace_bytes(tasks, len_q, hq, d, longest)
    ws = torch.empty(ws_bytes + 16, dtype=torch.uint8, device=cuda)
    stream = torch.cuda.current_stream().cuda_stream
    got, want = [], []
    for turn in range(3):
        q = torch.randn(tasks, len_q, hq, d, generator=g).half().to(cuda)
        kv = [torch.randn(m, hkv, d, generator=g).half().to(cuda) for m in lens + lens]
        addrs = torch.tensor([t.data_ptr() for t in kv], dtype=torch.int64)
        for own in (False, True):
            out, table = torch.full_like(q, float("nan")), torch.empty(2 * tasks, dtype=torch.int64, device=cuda)
            args = (mask.data_ptr() if masked else None, d ** -0.5, longest, out.data_ptr(), tasks, len_q, hq, hkv, d, 1, ws.data_ptr(), ws_bytes, ops.F16)
            if own:
                table.copy_(addrs)
                _lib.call("zl_decode_attention", q.data_ptr(), n.data_ptr(), table.data_ptr(), table.data_ptr() + 8 * tasks, *args, 0, stream)
            else:
                _lib.call("zl_decode_attention_host", q.data_ptr(), n.data_ptr(), addrs.data_ptr(), table.data_ptr(), *args, stream)
            (want if own else got).append(out)
        torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and not any(torch.isnan(a).any() for a in got)


@pytest.mark.parametrize("dtype,name,tol", [(torch.float16, "f16", 1e-3), (torch.bfloat16, "bf16", 6e-3)])
@pytest.mark.parametrize("tasks,hq,hkv,d,longest,splits,per_sm,merged", [
    (21, 8, 2, 128, 760, 3, 0, True), (24, 8, 2, 128, 760, 3, 0, False), (16, 8, 2, 128, 1000, 4, 0, True), (18, 8, 2, 128, 1000, 4, 0, False),      # 126 and 144 CTAs, 128 and 144
    (12, 4, 1, 128, 2000, 8, 0, True), (16, 4, 1, 64, 2000, 8, 0, False), (12, 8, 2, 64, 1200, 5, 0, True),                                         # 96, 128, 120
    (56, 8, 8, 128, 300, 1, 4, False), (64, 8, 4, 128, 900, 2, 4, True), (40, 8, 8, 128, 300, 1, 3, False), (96, 8, 8, 64, 300, 1, 5, False)])      # 448, 512, 320, 768
def test_places_of_the_splits(lib, cuda, dtype, name, tol, tasks, hq, hkv, d, longest, splits, per_sm, merged):
    """Both sides of the lines where clusters of 256-key CTAs find no room at once, and where an SM takes three, four or five CTAs; sequences of one length, and one
    in four whole beside short ones."""
    if name == "bf16" and per_sm == 4:
        per_sm, merged = 3, False                                                                                      # beyond its wave of three nothing is a cluster
    got = [ctypes.c_int(), ctypes.c_int()]
    assert lib.zl_decode_attention_plan(tasks, hq, hkv, d, longest, 0 if name == "f16" else 1, *map(ctypes.byref, got)) == int(merged)
    assert [v.value for v in got] == [splits, per_sm]
    for lens in ([longest] * tasks, [longest if i % 4 == 0 else longest // 8 + 1 for i in range(tasks)]):
        out, ref = _case(cuda, dtype, name, hq, hkv, d, lens, masked=False, seed=7)
        assert rel_l2(out, ref) <= tol
