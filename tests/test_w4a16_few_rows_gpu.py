"""GPU: up to 16 rows of x through the fp16 mma.sync kernel on the ZLW4I layout, where the integer kernel has no room for the rows."""
import numpy as np
import pytest
import torch

from oracle import gptq
from tests.helpers import rel_l2
from tests.test_w4a16_int_gpu import _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n", [(14336, 4096), (4096, 12288), (8192 + 128, 128), (12800, 9728)])
@pytest.mark.parametrize("m", [3, 8, 9, 16])
@pytest.mark.parametrize("pitch", [0, 8])
def test_few_rows(lib, cuda, k, n, m, pitch):
    """Both shapes of CTA (n up to 4736 and above), rows of x staged or not, rows on 32 and on 16 bytes, every row of the launch.  q - z is exact in
    fp16 and scales multiply fp32 sums: what is left is the rounding of the output, 2^-11 / sqrt(3) of a value at most (2.8e-4)."""
    from zhilight_b200 import ops
    w, packed, _, _ = _setup(cuda, k, n, False, 4)
    if lib.zl_w4_int_layout_route(m, n, k) != 4:
        pytest.skip("the integer kernel's")
    g = torch.Generator().manual_seed(m)
    x = torch.randn(m, k + pitch, generator=g).half()
    res, bias = torch.randn(m, n, generator=g).half(), torch.randn(n, generator=g).half()
    ref = gptq.gemm_f32(x[:, :k].numpy(), w)
    xd = x.to(cuda)[:, :k]
    y = ops.w4a16_gemm_fused(xd, packed, n, k, variant=1).float().cpu().numpy()
    assert max(rel_l2(y[i], ref[i]) for i in range(m)) <= 2.8e-4
    y = ops.w4a16_gemm_fused(xd, packed, n, k, variant=1, bias=bias.to(cuda), residual=res.to(cuda), epilogue=ops.EPI_RESIDUAL).float().cpu().numpy()
    assert max(rel_l2(y[i], ref[i] + bias.float().numpy() + res[i].float().numpy()) for i in range(m)) <= 5.6e-4   # rounded twice


@pytest.mark.parametrize("m", [9, 16])
def test_nine_to_sixteen_rows_keep_small_values_beside_large_ones(lib, cuda, m):
    """Also where the integer kernel has room: one exponent per 128 values would lose them."""
    from zhilight_b200 import ops
    k, n = 1024, 512
    w, packed, _, _ = _setup(cuda, k, n, False, 4)
    g = torch.Generator().manual_seed(m)
    x = torch.randn(m, k, generator=g).half()
    x[:, 5] = 30000.0
    ref = gptq.gemm_f32(x.numpy(), w)
    blind = np.flatnonzero(w[:, 5] == 0)
    assert len(blind) > 8
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1).float().cpu().numpy()
    assert rel_l2(y[:, blind], ref[:, blind]) <= 2.8e-4


@pytest.mark.parametrize("k,n", [(128, 128), (1152, 2304), (8192, 512), (4096, 4096 + 640), (2048, 9472), (1024, 4736 + 128)])
@pytest.mark.parametrize("m", [17, 24, 25, 32])
def test_up_to_32_rows_of_small_matrices(lib, cuda, k, n, m):
    """The edges of its range: K = 8192 of one wave of super-tiles, K = 2048 of two.  Tolerances as above, which the tcgen05 kernels' weights, rounded to
    fp16, would not keep."""
    from zhilight_b200 import ops
    w, packed, _, _ = _setup(cuda, k, n, False, 4)
    g = torch.Generator().manual_seed(m)
    x = torch.randn(m, k, generator=g).half()
    res, bias = torch.randn(m, n, generator=g).half(), torch.randn(n, generator=g).half()
    ref = gptq.gemm_f32(x.numpy(), w)
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1).float().cpu().numpy()
    assert max(rel_l2(y[i], ref[i]) for i in range(m)) <= 2.8e-4
    y = ops.w4a16_gemm_fused(x.to(cuda), packed, n, k, variant=1, bias=bias.to(cuda), residual=res.to(cuda), epilogue=ops.EPI_RESIDUAL).float().cpu().numpy()
    assert max(rel_l2(y[i], ref[i] + bias.float().numpy() + res[i].float().numpy()) for i in range(m)) <= 5.6e-4
