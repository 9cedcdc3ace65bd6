"""The semantic forwards with the full minimisation above 32 labels (label slots
side by side) against the oracle: label counts around the slots and around
groups of four senders, exact ties, both launch shapes."""
import pytest

from test_sem_full_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pixel", [False, True])
@pytest.mark.parametrize("L", [33, 34, 35, 36, 63, 64, 65, 66, 96, 97, 128, 129])
def test_label_counts(pixel, L):
    _check(pixel, 1, 3, 7, L, seed=L)


@pytest.mark.parametrize("pixel", [False, True])
@pytest.mark.parametrize("L", [50, 64, 90])
def test_ties(pixel, L):
    _check(pixel, 1, 4, 6, L, seed=2, q=4)


@pytest.mark.parametrize("L", [40, 130])
def test_global_many_scanlines(L):
    _check(False, 3, 220, 222, L, seed=7, iters=1)
