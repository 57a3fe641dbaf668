"""Tables of buffer addresses, written by a kernel in stream order: every word, and buffers given up right after the call."""
import pytest
import torch

from zhilight_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 2, 255, 256, 257, 700])
def test_every_address_arrives(cuda, n):
    base = torch.empty(max(n, 1) * 8, dtype=torch.uint8, device=cuda)
    views = [base[8 * i:] for i in range(n)]
    table = ops._ptr_table(views, base.device)
    assert table.dtype == torch.int64 and table.tolist() == [base.data_ptr() + 8 * i for i in range(n)]
    half = n // 2
    (a, b), both = ops._ptr_tables(base.device, views[:half], views[half:])
    assert (a, b) == (both.data_ptr(), both.data_ptr() + 8 * half) and both.tolist() == table.tolist()


@pytest.mark.parametrize("owner", ["torch", "dlpack"])
def test_buffers_of_another_stream_live_until_the_call_ends(cuda, owner):
    """Memory that came through DLPack is another owner's to give away: the allocator's notes about streams do not reach it."""
    torch.manual_seed(3)
    hkv, d, n = 2, 128, 2048
    own = (lambda t: t) if owner == "torch" else (lambda t: torch.from_dlpack(t))
    new = lambda: (own(torch.randn(1, 1, 8, d, device=cuda).half()),  # noqa: E731
                   [own(torch.randn(n, hkv, d, device=cuda).half()) for _ in range(2)])
    lens = torch.tensor([n], dtype=torch.int32, device=cuda)
    mask = torch.ones(n, dtype=torch.int8, device=cuda)
    side = torch.cuda.Stream()
    outs, refs = [], []
    for _ in range(8):
        q, (k, v) = new()
        refs.append(ops.decode_attention(q, lens, [k], [v], mask, d ** -0.5, n, hkv))
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            torch.cuda._sleep(2_000_000)                  # the call starts when the buffers have long been given up
            outs.append(ops.decode_attention(q, lens, [k], [v], mask, d ** -0.5, n, hkv))
        del q, k, v
        for _ in range(4):
            torch.full((n, hkv, d), float("nan"), dtype=torch.float16, device=cuda)   # takes what is free
    side.synchronize()
    for out, ref in zip(outs, refs):
        assert torch.equal(out, ref)


def test_memory_of_another_owner_can_be_captured(cuda):
    """Nothing runs during a capture, so nothing is waited for; the caller keeps the buffers as for any captured call."""
    torch.manual_seed(4)
    hkv, d, n = 2, 128, 300
    q, k, v = (torch.from_dlpack(torch.randn(*s, device=cuda).half()) for s in ((1, 1, 8, d), (n, hkv, d), (n, hkv, d)))
    lens = torch.tensor([n], dtype=torch.int32, device=cuda)
    call = lambda: ops.decode_attention(q, lens, [k], [v], None, d ** -0.5, n, hkv)  # noqa: E731
    want = call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = call()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
