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


def test_buffers_of_another_stream_live_until_the_call_ends(cuda):
    torch.manual_seed(3)
    hkv, d, n = 2, 128, 2048
    new = lambda: (torch.randn(1, 1, 8, d, device=cuda).half(), [torch.randn(n, hkv, d, device=cuda).half() for _ in range(2)])  # noqa: E731
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
