"""GPU: a bounded wait that gave up inside a kernel is an error of the next call or synchronisation, once.  The tests write the word that the
kernel would write; no wait is made to run out."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def words(lib, cuda):
    torch.cuda.synchronize()
    w = ctypes.cast(lib.zl_wait_words(), ctypes.POINTER(ctypes.c_uint))
    assert w and (w[0], w[1], w[2]) == (0, 0, 0)
    yield w
    w[0] = w[1] = w[2] = 0


@pytest.mark.parametrize("which,name", [(0, "general tensor-core GEMM"), (1, "4-bit GEMM"), (2, "attention of prompt portions")])
@pytest.mark.parametrize("call", ["w4", "nt", "dense", "w8", "attention", "check"])
def test_next_call_raises_once(lib, cuda, words, which, name, call):
    from zhilight_b200 import _lib, ops
    x, w = torch.ones(40, 128, dtype=torch.float16, device=cuda), torch.ones(128, 128, dtype=torch.float16, device=cuda)
    packed = torch.zeros(int(lib.zl_w4_packed_bytes(128, 128, 128)), dtype=torch.uint8, device=cuda)
    x8, one = torch.ones(40, 128, dtype=torch.int8, device=cuda), torch.ones(128, device=cuda)
    q, kv = torch.ones(1, 64, 32, 128, dtype=torch.float16, device=cuda), torch.ones(512, 8, 128, dtype=torch.float16, device=cuda)
    lens = torch.tensor([512], dtype=torch.int32, device=cuda)
    run = {"w4": lambda: ops.w4a16_gemm_fused(x, packed, 128, 128, variant=1), "nt": lambda: ops.gemm_nt(x, w),
           "dense": lambda: ops.dense_gemm_skinny(x, w), "w8": lambda: ops.w8a8_gemm(x8, one[:40], x8.new_ones(128, 128), one, torch.float16),
           "attention": lambda: ops.decode_attention(q, lens, [kv], [kv], None, 0.09, 512, 8), "check": ops.check_waits}[call]
    run()
    words[which] = 0x3401
    codes = [lib.zl_gemm_tc_watchdog(), lib.zl_w4_tc2_watchdog(), lib.zl_prompt_attention_watchdog()]
    assert codes == [0x3401 if i == which else 0 for i in range(3)]
    with pytest.raises(_lib.ZLError, match=name + ".*0x3401"):
        run()
    run()
    torch.cuda.synchronize()
    assert (words[0], words[1], words[2]) == (0, 0, 0)


def test_decoder_raises_at_the_end_of_its_step(lib, cuda, words):
    """The step is a captured graph by then: nothing but its synchronisation can notice."""
    from zhilight_b200 import _lib
    from zhilight_b200.llama import LlamaDecoder
    c = dict(num_layers=1, dim_model=256, num_heads=2, num_kv_heads=1, dim_head=128, dim_ff=512, vocab_size=320, eps=1e-5, rope_theta=1e4)
    dec = LlamaDecoder(quant_type=0, dtype="f16", max_batch=1, max_seq=64, prefill_chunk=16, **c)
    g = np.random.default_rng(0)
    half = lambda *s: (g.standard_normal(s) * 0.05).astype(np.float16)  # noqa: E731
    t = {"token_embedding.weight": half(320, 256), "lm_head.weight": half(320, 256), "output_layernorm.weight": half(256)}
    for name, shape in {"ln_attn": (256,), "ln_ff": (256,), "attn.project_q": (256, 256), "attn.project_k": (128, 256), "attn.project_v": (128, 256),
                        "attn.attn_out": (256, 256), "ff.w_in": (512, 256), "ff.w_gated": (512, 256), "ff.w_out": (256, 512)}.items():
        t["layers.0." + name + ".weight"] = half(*shape)
    dec.load_state_dict(t)
    dec.prefill(0, np.arange(5, dtype=np.int32), 0)
    step = lambda: dec.decode(np.array([7], np.int32), np.array([5], np.int32), want_logits=True)[1]  # noqa: E731
    want = step()
    words[0] = 0x2403
    with pytest.raises(_lib.ZLError, match="0x2403"):
        step()
    np.testing.assert_array_equal(step(), want)
    for i, code in ((1, 0x3403), (2, 0x4403)):
        words[i] = code
        with pytest.raises(_lib.ZLError, match=hex(code)):
            dec.prefill(0, np.arange(5, dtype=np.int32), 0)


_CAPTURE_FIRST = """
import sys, torch
sys.path.insert(0, sys.argv[1])
from zhilight_b200 import ops
g = torch.Generator(device="cuda").manual_seed(1)
x, w = (torch.randn(64, 512, generator=g, device="cuda").half(), torch.randn(1024, 512, generator=g, device="cuda").half())
x8, w8 = x.clamp(-1, 1).mul(127).to(torch.int8), w.clamp(-1, 1).mul(127).to(torch.int8)
sx, sw = torch.rand(64, generator=g, device="cuda"), torch.rand(1024, generator=g, device="cuda")
call = lambda: (ops.gemm_nt(x, w), ops.w8a8_gemm(x8, sx, w8, sw, torch.float16))
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    got = call()
graph.replay()
torch.cuda.synchronize()
print(all(torch.equal(a, b) for a, b in zip(got, call())))
"""


def test_first_call_of_a_process_may_be_captured(cuda):
    """The words are had at the first call; inside a capture that allocation is no part of it."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CAPTURE_FIRST, root], capture_output=True, text=True, timeout=300)
    assert r.stdout.split() == ["True"], r.stdout + r.stderr
