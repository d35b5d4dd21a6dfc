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


@pytest.mark.parametrize("device", [torch.device("cuda", 1), "cuda:1", 1])
def test_arena_by_device_name_or_index(device, monkeypatch):
    """One arena per GPU, however the device is given."""
    monkeypatch.setattr(cu, "_ARENAS", {})
    monkeypatch.setattr(cu, "_Arena", lambda d: object())
    assert cu.arena(device) is cu.arena(torch.device("cuda", 1))
    assert cu.arena(torch.device("cuda", 0)) is not cu.arena(device)
    assert cu.arena("cuda") is cu.arena(torch.device("cuda:0"))
