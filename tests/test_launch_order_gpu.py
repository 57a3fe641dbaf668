"""GPU: launches that start under the end of the one before them.  Whatever the callers' `pdl` says, a row of calls gives the bits of the same calls one by one,
and the switch for ordinary launches gives these."""
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


_EDGES = """
import ctypes
import torch
from zhilight_b200 import ops
x, w = torch.randn(4, 1024, device="cuda").half(), torch.randn(1024, 1024, device="cuda").half()
run = lambda: ops.dense_gemm_skinny(ops.dense_gemm_skinny(x, w), w)
run()
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph(keep_graph=True)
with torch.cuda.graph(graph):
    run()
n = ctypes.c_size_t(8)
nodes = [(ctypes.c_void_p * 8)() for _ in range(2)]
edges = (ctypes.c_uint8 * 64)()       # eight bytes an edge: two ports, the type, reserved ones
rc = ctypes.CDLL("libcudart.so.12").cudaGraphGetEdges_v2(ctypes.c_void_p(graph.raw_cuda_graph()), *nodes, edges, ctypes.byref(n))
print("edges", rc, n.value, edges[2])
"""


@pytest.mark.parametrize("switch,programmatic", [(False, 1), (True, 0)])
def test_switch_for_ordinary_launches(lib, cuda, switch, programmatic):
    """ZL_DENSE_NO_PDL: the edge between two dense GEMMs of a captured graph is an ordinary one."""
    env = dict(os.environ, PYTHONPATH=os.path.join(os.path.dirname(__file__), ".."))
    env.pop("ZL_DENSE_NO_PDL", None)
    if switch:
        env["ZL_DENSE_NO_PDL"] = "1"
    r = subprocess.run([sys.executable, "-c", _EDGES], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split()[-4:] == ["edges", "0", "1", str(programmatic)]
