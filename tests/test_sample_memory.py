"""Where State.sample's counts live and how they are made: page-locked memory
is bounded by what the program holds, and each of the three ways to the counts
gives the same draws."""
import gc

import numpy as np
import pytest
import torch


@pytest.fixture
def plain_memory(monkeypatch):
    """torch.empty without page-locking (no GPU needed)."""
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, pin_memory=False, **k: empty(*a, **k))


def test_page_locked_results_are_counted_while_they_live(plain_memory, monkeypatch):
    from quantumflow_gb300 import states
    gc.collect()
    start = states._PinnedArray._held
    monkeypatch.setattr(states, "_PINNED_RESULTS", start + 3 * 800)
    kept = []
    for k in range(3):
        host = states._PinnedArray.make(100)
        host.tensor.fill_(k)
        kept.append(host.array().reshape(10, 10)[2:])  # a view keeps the whole
        del host
    assert states._PinnedArray.make(100) is None
    assert [int(v[0, 0]) for v in kept] == [0, 1, 2] and kept[0].flags.writeable and kept[0].dtype == np.int64
    first = torch.from_numpy(kept[0])
    del kept[0]
    gc.collect()
    assert states._PinnedArray.make(100) is None  # (the tensor on it counts too)
    assert int(first[0, 0]) == 0
    del first
    gc.collect()
    assert states._PinnedArray._held == start + 2 * 800
    again = states._PinnedArray.make(100)
    assert again is not None and states._PinnedArray.make(100) is None
    del again, kept
    gc.collect()
    assert states._PinnedArray._held == start


@pytest.mark.gpu
def test_results_a_program_keeps_do_not_lock_memory_without_end(monkeypatch):
    import quantumflow_gb300 as qf
    from quantumflow_gb300 import states
    n = 15  # 256 KiB of counts
    gc.collect()
    monkeypatch.setattr(states, "_PINNED_RESULTS", states._PinnedArray._held + (2 << 18))
    ket = qf.random_state(n)
    kept = [ket.sample(1000, seed=k) for k in range(5)]
    assert [torch.from_numpy(c).is_pinned() for c in kept] == [True, True, False, False, False]
    for k, counts in enumerate(kept):
        assert np.array_equal(counts.reshape(-1), np.bincount(ket._draws(1000, seed=k), minlength=2 ** n))
    del kept[0], counts
    gc.collect()
    assert torch.from_numpy(ket.sample(10, seed=9)).is_pinned()


@pytest.mark.gpu
def test_each_way_to_the_counts(monkeypatch):
    """Ordinary, page-locked and listed read-backs of one seed, with the sizes
    brought down; draws are listed for at most one trial in 64 outcomes."""
    import quantumflow_gb300 as qf
    from quantumflow_gb300 import states
    n = 12
    ket = qf.random_state(n)
    listed = []
    draws = states.State._draws
    monkeypatch.setattr(states.State, "_draws", lambda self, trials, seed: listed.append(trials) or
                        draws(self, trials, seed))
    for pageable, pinned in ((1 << 30, 1 << 31), (1 << 10, 1 << 31), (1 << 10, 1 << 11)):
        monkeypatch.setattr(states, "_PAGEABLE_COUNTS", pageable)
        monkeypatch.setattr(states, "_PINNED_COUNTS", pinned)
        for trials in (0, 1, 2 ** n // 64, 2 ** n // 64 + 1, 2 ** n // 8, 2 ** n):
            listed.clear()
            counts = ket.sample(trials, seed=77)
            assert bool(listed) == (pinned == 1 << 11 and 64 * trials <= 2 ** n)
            assert counts.shape == (2,) * n and counts.dtype == np.int64
            want = np.bincount(draws(ket, trials, 77), minlength=2 ** n)
            assert np.array_equal(counts.reshape(-1), want)


@pytest.mark.gpu
@pytest.mark.parametrize("trials", [1, 1000, 2 ** 24 // 64, 2 ** 24 // 64 + 1])
def test_counts_of_a_large_state(trials):
    """n = 24, on both sides of the rule, unpatched."""
    import quantumflow_gb300 as qf
    ket = qf.random_state(24)
    counts = ket.sample(trials, seed=5)
    assert np.array_equal(counts.reshape(-1), np.bincount(ket._draws(trials, seed=5), minlength=2 ** 24))
