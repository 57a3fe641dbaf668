"""CPU: an SM never holds more CTAs of the prompt attention than its tensor memory serves (256 of 512 columns each, had by a wait without a bound), by
shared memory alone: registers are the compiler's to choose."""
import pytest

SM, PER_CTA, STATIC = 228 * 1024, 1024, 1024


@pytest.mark.parametrize("dim_head", [64, 128])
def test_two_ctas_and_no_third(lib, dim_head):
    smem = lib.zl_prompt_attention_smem_bytes(dim_head)
    assert 2 * (smem + STATIC + PER_CTA) <= SM
    assert 3 * smem > SM


def test_other_widths_have_no_such_kernel(lib):
    assert lib.zl_prompt_attention_smem_bytes(96) == 0
