"""The order of a chunk's runs (run_chunks in mpm_kernels_runs.cuh), restated on the host: a record that finds k records
in its run counts the run as longer than k (k < 16); a run of length l then goes behind the level[l] longer ones, at its
turn among those of its length, lengths of 16 and more together.  That must be a permutation, the longest runs first."""
import numpy as np
import pytest

BINS = 16


@pytest.mark.parametrize("longest", [1, 2, 15, 16, 17, 40, 288])
def test_places_are_a_permutation_by_length(longest):
    rng = np.random.default_rng(longest)
    for _ in range(50):
        lengths = rng.integers(1, longest + 1, rng.integers(1, 120))
        lengths[0] = longest
        outside = rng.random(len(lengths)) < 0.1  # particles outside the window: runs of one record
        lengths[outside] = 1
        level, cnt = np.zeros(BINS, int), np.zeros(len(lengths), int)
        records = np.repeat(np.arange(len(lengths)), lengths)
        rng.shuffle(records)
        for r in records:
            if outside[r]:
                level[0] += 1
                continue
            longer, cnt[r] = cnt[r], cnt[r] + 1
            if longer < BINS:
                level[longer] += 1
        taken, place = np.zeros(BINS, int), np.full(len(lengths), -1)
        for r in rng.permutation(len(lengths)):
            k = min(1 if outside[r] else cnt[r], BINS) - 1
            place[r] = (level[k + 1] if k + 1 < BINS else 0) + taken[k]
            taken[k] += 1
        assert sorted(place) == list(range(len(lengths)))
        by_place = np.minimum(lengths[np.argsort(place)], BINS)
        assert np.all(np.diff(by_place) <= 0)
