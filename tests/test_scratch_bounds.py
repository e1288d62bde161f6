"""What a call may hold beside its inputs and outputs does not grow with the prompt without bound."""
import pytest


@pytest.mark.parametrize("B,kv_heads,heads,dim", [(1, 4, 16, 128), (4, 8, 32, 128), (16, 2, 2, 64), (1, 1, 1, 65), (512, 64, 64, 128)])
def test_the_delta_rule_in_chunks(B, kv_heads, heads, dim):
    from ipex_llm_b200.ggml.model import mixers_cpp
    size = mixers_cpp.lib().mixers_gated_delta_chunks_workspace
    one = size(B, 32, kv_heads, heads, dim)
    sizes = [size(B, S, kv_heads, heads, dim) for S in (64, 65, 2048, 33333, 1 << 20, (1 << 31) - 1)]
    assert all(one <= s <= max(512 << 20, one) and s % one == 0 for s in sizes)
    assert sizes[0] == min(2, max(1, (512 << 20) // one)) * one
