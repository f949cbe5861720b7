"""Host-side logic of the device-driven loops, on CPU: the replay lengths
of forward()'s graphs and the adjoint gather's block count."""
import math

from diffswe2d_b200.adjoint import level_blocks
from diffswe2d_b200.solver import replay_length, replay_lengths


def test_replay_lengths_halve_while_even():
    assert replay_lengths(32) == [32, 16, 8, 4, 2]
    assert replay_lengths(64) == [64, 32, 16, 8, 4, 2]
    assert replay_lengths(8) == [8, 4, 2]
    assert replay_lengths(2) == [2]
    assert replay_lengths(6) == [6]  # 6 / 2 = 3 would leave the state in the other buffer
    for chunk in (2, 4, 6, 8, 12, 16, 24, 32, 48, 64):
        assert all(n % 2 == 0 for n in replay_lengths(chunk))


def test_replay_length_is_the_longest_that_fits():
    sizes = replay_lengths(32)
    assert replay_length(sizes, math.inf) == 32
    assert replay_length(sizes, 40.0) == 32
    assert replay_length(sizes, 31.9) == 16
    assert replay_length(sizes, 9.5) == 8
    assert replay_length(sizes, 4.0) == 4
    assert replay_length(sizes, 1.2) == 2  # at least the shortest graph
    assert replay_length(sizes, 0.0) == 2


def test_replay_lengths_cover_a_call_with_few_idle_steps():
    """Greedy replays for a call of n steps (the dt known exactly) run at
    most one step past its end."""
    sizes = replay_lengths(32)
    for n in range(1, 200):
        done, left = 0, float(n)
        while done < n:
            m = replay_length(sizes, left)
            done += m
            left = n - done
        assert done - n <= 1


def test_level_blocks_one_cell_per_thread_up_to_1024():
    assert level_blocks(1, 1) == 1
    assert level_blocks(16, 16) == 1
    assert level_blocks(244, 393) == math.ceil(244 * 393 / 256)
    assert level_blocks(4096, 4096) == 1024


def test_ensemble_rows_follow_the_members():
    from diffswe2d_b200.autotune import ensemble_rows
    assert ensemble_rows([(2, 2)]) == 1                       # one tile: the shortest chain
    assert ensemble_rows([(122, 196)] * 8) <= 4               # few tiles: short ones
    assert ensemble_rows([(122, 196)] * 64) in (8, 12, 16)
    assert ensemble_rows([(1024, 1024)] * 1024) >= 32         # many: few halo rows


def test_rainfall_at_a_host_time_equals_the_tensor_expression():
    import pytest
    import torch
    from diffswe2d_b200 import RainfallForcing
    g = torch.Generator().manual_seed(1)
    for dtype in (torch.float32, torch.float64):
        times = torch.tensor([0.0, 1.5, 3.7, 10.0], dtype=dtype)
        f = RainfallForcing(times, torch.rand((4, 1, 5, 6), generator=g) * 1e-5)
        for t in (-1.0, 0.0, 0.3, 1.5, 2.2, 3.7, 9.999, 10.0, 11.0):
            assert torch.equal(f.at(t), f.at(torch.tensor(t, dtype=dtype)))
    f.at(0.0).zero_()  # a result of its own, not a view of the series
    assert float(f.rates[0].sum()) > 0
    with pytest.raises(ValueError):
        RainfallForcing(times.flip(0), f.rates)


def test_chunks_of_an_odd_length_are_rounded_up():
    import pytest
    from diffswe2d_b200.solver import even_chunk
    assert [even_chunk(c) for c in (1, 2, 3, 31, 32, 32.0)] == [2, 2, 4, 32, 32, 32]
    assert all(n % 2 == 0 for c in range(1, 40) for n in replay_lengths(even_chunk(c)))
    for bad in (0, -2):
        with pytest.raises(ValueError):
            even_chunk(bad)


def test_boundary_levels_from_the_host_as_new_tensor_gives_them():
    import torch
    from diffswe2d_b200 import SWE2D
    for dtype in (torch.float32, torch.float64, torch.float16):
        U = torch.zeros((1, 3, 2, 2), dtype=dtype)
        for v in (0.1, 1e-46, -0.0, 3.4028235e38, -3.4028235677973366e38, 1e300, math.inf, -math.inf, math.nan, 7):
            a, b = SWE2D._prepare_boundary_level(v, U), U.new_tensor(v)
            assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a.nan_to_num(3.0), b.nan_to_num(3.0))
