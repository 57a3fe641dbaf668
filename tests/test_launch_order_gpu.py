"""GPU: launches that start under the end of the one before them.  Whatever the callers' `pdl` says, a row of calls gives the bits of the same calls one by one,
and the switch for ordinary launches gives these."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

K = 2048


def _chain(cuda, m):
    """4-bit, int8, fp8 and dense Linears of one row length in a row, then attention over the last one's rows; no launch of torch's stands between them."""
    from oracle import gptq
    from zhilight_b200 import layers, ops
    g = torch.Generator().manual_seed(m)
    parts = []
    for quant in (layers.QUANT_GPTQ, layers.QUANT_INT8, layers.QUANT_FP8, layers.QUANT_NONE):
        if quant == layers.QUANT_GPTQ:
            qw, qz, sc, _ = gptq.make_gptq_checkpoint(K, K, 128, False, seed=m)
            t = {"qweight": torch.from_numpy(qw), "qzeros": torch.from_numpy(qz), "scales": torch.from_numpy(sc)}
        elif quant == layers.QUANT_INT8:
            t = {"weight": torch.randint(-127, 128, (K, K), generator=g, dtype=torch.int8), "weight_scale": (0.5 + torch.rand(K, generator=g)) * 0.014 / K ** 0.5}
        elif quant == layers.QUANT_FP8:
            t = {"weight": (torch.randn(K, K, generator=g) * 60).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8),
                 "weight_scale": torch.tensor([1 / (60 * K ** 0.5)])}
        else:
            t = {"weight": torch.randn(K, K, generator=g) / K ** 0.5}
        lin = layers.Linear(K, K, "", quant, "half")
        lin.load_state_dict({name: v.to(cuda) for name, v in t.items()})
        parts.append(lin)
    kv = [torch.randn(700, 4, 128, generator=g).half().to(cuda) for _ in range(2)]
    lens = torch.tensor([700], dtype=torch.int32, device=cuda)
    parts.append(lambda h: ops.decode_attention(h.view(1, m, 16, 128), lens, kv[:1], kv[1:], None, 128 ** -0.5, 700, 4).view(m, K))
    return parts


@pytest.mark.parametrize("m", [1, 4, 24, 48, 90, 300])
def test_a_row_of_calls_gives_the_bits_of_single_calls(lib, cuda, m):
    parts = _chain(cuda, m)
    xs = [torch.randn(m, K, generator=torch.Generator().manual_seed(i)).half().to(cuda) for i in range(4)]

    def run(x, wait):
        seen = []
        for _ in range(3):
            for part in parts:
                x = part(x)
                seen.append(x)
                if wait:
                    torch.cuda.synchronize()
        return seen

    alone = [run(x, True) for x in xs]
    for turn in range(3):
        row = [run(x, False) for x in xs]
        torch.cuda.synchronize()
        for a, b in zip(alone, row):
            assert all(torch.isfinite(y).all() for y in a) and all(torch.equal(y, z) for y, z in zip(a, b)), turn


def _programmatic_edges(call):
    """Programmatic edges between the launches of two calls in a captured graph, and all of them"""
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
        call()
    n = ctypes.c_size_t(32)
    nodes = [(ctypes.c_void_p * 32)() for _ in range(2)]
    edges = (ctypes.c_uint8 * 256)()       # eight bytes an edge: two ports, the type, reserved ones
    assert ctypes.CDLL("libcudart.so.12").cudaGraphGetEdges_v2(ctypes.c_void_p(graph.raw_cuda_graph()), *nodes, edges, ctypes.byref(n)) == 0
    return sum(edges[8 * i + 2] for i in range(n.value)), n.value


@pytest.mark.parametrize("what", ["dense", "w4-1", "w4-12", "w4-48", "w4-300", "int8", "fp8", "fp8-large"])
def test_three_kinds_of_launches(lib, cuda, what):
    """pdl 0: ordinary launches, 1 and 2: programmatic dependents, of one or several kernels; the same bits, and what the Python calls ask for."""
    from oracle import gptq
    from zhilight_b200 import _lib, ops
    m = int(what.split("-")[1]) if what.startswith("w4") else 80 if what == "fp8-large" else 4
    x = torch.randn(m, K, generator=torch.Generator().manual_seed(1)).half().to(cuda)
    stream = lambda: torch.cuda.current_stream().cuda_stream  # noqa: E731
    if what == "dense":
        w, y = torch.randn(K, K, device=cuda).half(), torch.empty(m, K, dtype=torch.float16, device=cuda)
        run = lambda pdl: _lib.call("zl_dense_gemm_skinny", x.data_ptr(), K, w.data_ptr(), None, y.data_ptr(), m, K, K, ops.F16, ops.F16, pdl, stream())  # noqa: E731
        python = lambda: ops.dense_gemm_skinny(x, w)  # noqa: E731
    elif what.startswith("w4"):
        qw, qz, sc, gi = gptq.make_gptq_checkpoint(K, K, 128, False, seed=3)
        km = [torch.from_numpy(a.view(d) if d else a).to(cuda) for a, d in zip(gptq.to_k_major(qw, qz, sc, gi, 128)[:3], ("int32", None, None))]
        packed, y = ops.w4_pack(*km, 128, variant=1), torch.empty(m, K, dtype=torch.float16, device=cuda)

        def run(pdl):
            a = _lib.W4FusedArgs(x.data_ptr(), K, packed.data_ptr(), None, None, y.data_ptr(), m, K, K, 128, 0, pdl, None, 1e-5)
            a.variant = 1
            _lib.call("zl_w4a16_gemm_fused", ctypes.byref(a), stream())
        python = lambda: ops.w4a16_gemm_fused(x, packed, K, K, variant=1)  # noqa: E731
    else:
        y, s = torch.empty(m, K, dtype=torch.uint8, device=cuda), torch.empty(m, device=cuda)
        if what == "int8":
            run = lambda pdl: _lib.call("zl_int8_quant_per_token", x.data_ptr(), K, y.data_ptr(), s.data_ptr(), m, K, ops.F16, pdl, stream())  # noqa: E731
            python = lambda: ops.int8_quant_per_token(x)[0].view(torch.uint8)  # noqa: E731
        else:
            run = lambda pdl: _lib.call("zl_fp8_quant_per_tensor", x.data_ptr(), y.data_ptr(), s.data_ptr(), x.numel(), ops.F16, pdl, stream())  # noqa: E731
            python = lambda: ops.fp8_quant_per_tensor(x)[0]  # noqa: E731
    want = python().clone()
    torch.cuda.synchronize()
    kernels = 3 if what == "fp8-large" else 1
    for pdl in (0, 1, 2):
        y.zero_()
        run(pdl)
        torch.cuda.synchronize()
        assert torch.equal(y, want), pdl
        assert _programmatic_edges(lambda: run(pdl)) == ((2 * kernels - 1) * (pdl != 0), 2 * kernels - 1), pdl
    assert _programmatic_edges(python)[0] == 2 * kernels - 1


_SWITCH = """
import torch
from tests.test_launch_order_gpu import _programmatic_edges
from zhilight_b200 import ops
x, w = torch.randn(4, 1024, device="cuda").half(), torch.randn(1024, 1024, device="cuda").half()
ops.dense_gemm_skinny(x, w)
torch.cuda.synchronize()
print("edges", *_programmatic_edges(lambda: ops.dense_gemm_skinny(x, w)))
"""


@pytest.mark.parametrize("switch,programmatic", [(False, 1), (True, 0)])
def test_switch_for_ordinary_launches(lib, cuda, switch, programmatic):
    """ZL_DENSE_NO_PDL: the edge between two dense GEMMs of a captured graph is an ordinary one."""
    env = dict(os.environ, PYTHONPATH=os.path.join(os.path.dirname(__file__), ".."))
    env.pop("ZL_DENSE_NO_PDL", None)
    if switch:
        env["ZL_DENSE_NO_PDL"] = "1"
    r = subprocess.run([sys.executable, "-c", _SWITCH], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split()[-3:] == ["edges", str(programmatic), "1"]


_CAPTURED_FIRST = """
import torch
from zhilight_b200 import ops
what = %r
g = torch.Generator().manual_seed(1)
x = torch.randn(149, 2056, generator=g).half().cuda()
kv = [torch.randn(2600, 8, 128, generator=g).half().cuda() for _ in range(8)]
q = torch.randn(4, 1, 32, 128, generator=g).half().cuda()
lens = torch.tensor([1000, 900, 800, 700], dtype=torch.int32, device="cuda")
rows = torch.randn(1, 107, 16, 128, generator=g).half().cuda()
long = torch.tensor([2600], dtype=torch.int32, device="cuda")
run = {"int8": lambda: ops.int8_quant_per_token(x)[0], "one row": lambda: ops.decode_attention(q, lens, [t[:n] for t, n in zip(kv, lens_)], [t[:n] for t, n in zip(kv[4:], lens_)], None,
                                                                                              0.1, 1000, 8),
       "rows": lambda: ops.decode_attention(rows, long, kv[:1], kv[1:2], None, 0.1, 2600, 8)}[what]
lens_ = [1000, 900, 800, 700]
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    y = run()
graph.replay()
torch.cuda.synchronize()
got = y.clone()
print("same", torch.equal(got, run()), float(got.float().abs().sum()) > 0)
"""


@pytest.mark.parametrize("what", ["int8", "one row", "rows"])
def test_first_call_of_a_process_may_be_captured(cuda, what):
    """The device is asked how many clusters it holds, and a kernel is given its shared memory, inside the capture."""
    env = dict(os.environ, PYTHONPATH=os.path.join(os.path.dirname(__file__), ".."))
    r = subprocess.run([sys.executable, "-c", _CAPTURED_FIRST % what], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split() == ["same", "True", "True"]
