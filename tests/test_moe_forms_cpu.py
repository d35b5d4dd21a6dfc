"""The library's estimates of the two forms of routed experts (host only: no GPU)."""
import pytest

from llmss_b200.ops import cuda_impl as cu


@pytest.mark.parametrize("E,top,W,F", [(8, 2, 128, 512), (16, 4, 64, 256), (8, 2, 128, 16), (4, 2, 96, 40)])
def test_dense_form_of_narrow_models_has_a_cost(E, top, W, F):
    """Results of at most 128 columns, past the sizes at which the pair kernel takes them (some 3500 tokens, or K of fewer than four blocks of 64): the two
    products cost at least their launches (3.5 us each, the least that an estimate has) and their bytes, beside the pass over the hidden rows."""
    for T in (64, 512, 3000, 3552, 3553, 4096, 8192, 16384):
        dense, grouped, tile = cu.moe_forms(T, top, (E, F, W), F)
        assert dense >= 4 + T * E * F * 1e-6 + 2 * 3.5 + 2 * (E * F * W + T * E * F) / 6.5e6, (T, dense)
        assert grouped > 0 and tile % 32 == 0
