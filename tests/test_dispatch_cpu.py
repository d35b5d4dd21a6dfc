"""Host-side rules of the CUDA path, on the CPU: which kernel a call takes by its sizes, and which arena by its device."""
import pytest
import torch

from llmss_b200.ops import cuda_impl as cu


@pytest.mark.parametrize("lens,want", [
    ([1024] * 8, 0), ([576, 640, 777, 900, 1024, 1100, 1300, 1472], 0), ([1500], 0),      # long portions: all over chunks
    ([512] + [1] * 63, 64), ([1024] + [16] * 31, 64), ([512] + [33] * 63, 64),            # one long portion beside short ones
    ([96] * 64, None), ([95], None), ([1] * 64, None), ([64] * 8, None)])                 # enough in flight, or too short
def test_recurrence_goes_over_chunks_where_that_is_less_work(lens, want):
    assert cu._scan_floor(sum(lens), len(lens), max(lens), 32, 64, 64, 2) == want


@pytest.mark.parametrize("heads,dk,dv", [(32, 66, 64), (2, 132, 64), (1 << 15, 128, 256), (65536, 4, 4)])
def test_recurrence_sizes_that_chunks_do_not_take(heads, dk, dv):
    """Key sizes off the vectors, and states or grids past what the chunk kernels index, stay on the general kernels."""
    assert cu._scan_floor(4096, 2, 2048, heads, dk, dv, 2) is None


@pytest.mark.parametrize("lens", [[100, 1], [300, 7, 7], [512] + [63] * 5, [512, 64], [2000, 1, 1, 1], [590, 30] * 20, [400] * 20 + [20]])
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_a_batch_without_a_floor_has_no_short_sequences_or_many_long_ones(lens, kind):
    """Without a floor the chunk kernels take every sequence: only where no sequence is shorter than a chunk, or few sequences are
    far longer on average."""
    T, B = sum(lens), len(lens)
    if cu._scan_floor(T, B, max(lens), 32, 64, 64, kind) == 0:
        assert min(lens) >= 64 or ((T - max(lens)) / (B - 1) >= 128 and B < 16)


PROMPTS = [576, 640, 777, 900, 1024, 1100, 1300, 1472]


@pytest.mark.parametrize("heads,qk_heads,d,lens,chunks,tokens", [
    (16, 8, 128, PROMPTS, 343, 910), (16, 8, 128, [1024] * 8, 284, 640), (16, 8, 128, [1500], 278, 610), (16, 8, 128, [4096], 794, 1660), (16, 8, 128, [64] * 8, 41, 50),
    (16, 8, 128, [112] + [73] * 9 + [78], 78, 99), (16, 8, 128, [1000] + [8] * 31, 243, 667), (16, 8, 128, [200, 16] * 8, 102, 181), (32, 16, 128, [72] + [45] * 3, 49, 56),
    (32, 32, 64, [1500], 306, 554), (16, 8, 32, [1024] * 8, 277, 399), (64, 32, 128, [512] * 8, 552, 1082), (4, 4, 128, [1024] * 2, 196, 422),
    (32, 32, 64, PROMPTS, 702, 550), (32, 32, 64, [1024] * 8, 622, 386), (16, 8, 128, [64], 40, 34), (16, 8, 128, [32] * 8, 36, 31), (16, 8, 128, [71] + [47] * 11, 86, 67),
    (32, 16, 128, [46] + [30] * 21 + [37], 149, 128), (16, 8, 128, [33] + [21] * 6 + [25], 62, 31)])
def test_delta_rule_goes_over_chunks_where_that_is_faster(heads, qk_heads, d, lens, chunks, tokens):
    """Either side of the rule, with the times (us) that both forms took on a B200."""
    assert cu._delta_over_chunks(sum(lens), len(lens), max(lens), heads, qk_heads, d, d) == (chunks < tokens)


@pytest.mark.parametrize("T,B,max_q,heads,dk", [(31, 1, 31, 16, 128), (8192, 8, 1024, 16, 132), (8192, 8, 1024, 16, 256), (8192, 8, 1024, 16, 66), (70000 * 40, 70000, 40, 1, 64),
                                                (2048, 1, 2048, 65536, 64), (64, 64, 1, 16, 128)])
def test_delta_rule_sizes_that_chunks_do_not_take(T, B, max_q, heads, dk):
    """No portion of a chunk's length, key sizes off the copies or above the tiles, more sequences or heads than a grid has."""
    assert not cu._delta_over_chunks(T, B, max_q, heads, heads, dk, 128)


@pytest.mark.parametrize("device", [torch.device("cuda", 1), "cuda:1", 1])
def test_arena_by_device_name_or_index(device, monkeypatch):
    """One arena per GPU, however the device is given."""
    monkeypatch.setattr(cu, "_ARENAS", {})
    monkeypatch.setattr(cu, "_Arena", lambda d: object())
    assert cu.arena(device) is cu.arena(torch.device("cuda", 1))
    assert cu.arena(torch.device("cuda", 0)) is not cu.arena(device)
    assert cu.arena("cuda") is cu.arena(torch.device("cuda:0"))
