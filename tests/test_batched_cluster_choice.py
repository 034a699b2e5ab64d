"""Default cluster size of a batch: which of the launch shapes timed on the
hardware the estimate takes, and that any subset of the shapes is accepted."""
import numpy as np
import pytest

from tensormesh_gb300.batched import choose_cluster

SLOTS = {1: 304, 2: 152, 4: 74, 8: 36, 16: 14}   # resident clusters of the triangle kernel


def _rows(sizes):
    return [int(s + 1) ** 2 for s in sizes]


@pytest.mark.parametrize("sizes,fastest", [
    (np.random.default_rng(2027).integers(32, 257, size=256), 4),
    (np.random.default_rng(1).integers(20, 140, size=20), 16),
    (np.random.default_rng(1).integers(16, 64, size=56), 8),
    ([20] * 200, 1),
    ([16] * 8, 4),
])
def test_fastest_measured_shape(sizes, fastest):
    assert choose_cluster(_rows(sizes), 2, SLOTS) == fastest


@pytest.mark.parametrize("slots", [{4: 1}, {1: 1, 2: 1}, SLOTS])
@pytest.mark.parametrize("dim", [2, 3])
def test_any_batch_gets_an_offered_shape(slots, dim):
    for rows in ([1], [4] * 1000, [10 ** 7], list(range(1, 400))):
        assert choose_cluster(rows, dim, slots) in slots
