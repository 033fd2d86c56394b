"""Searches of many keys in lists that are not evenly spread: constant,
clustered, dense at one end, of repeated ids, at the lengths where the search
tree gains a level, against numpy."""
from __future__ import annotations

import numpy as np
import pytest

import gary_b200 as gb
from gary_b200 import setops as so

pytestmark = pytest.mark.gpu

NKEYS = 148 * 1024 * 4 + 5  # enough for the search tree
LAST = (1 << 32) - 2


def _list(shape, n, rng):
    if shape == "constant":
        return np.full(n, 12345, np.uint32)
    if shape == "clusters":  # a few dense runs far apart
        start = np.sort(rng.integers(0, LAST - n, 7))
        return np.sort((start[rng.integers(0, 7, n)] + rng.integers(0, max(n // 4, 1), n)).astype(np.uint32))
    if shape == "dense low end":
        return np.sort((LAST * rng.random(n) ** 12).astype(np.uint32))
    if shape == "dense high end":
        return np.sort((LAST - LAST * rng.random(n) ** 12).astype(np.uint32))
    if shape == "repeats":
        return np.sort(rng.integers(0, 50, n)).astype(np.uint32) * np.uint32(80_000_000)
    return np.concatenate([np.zeros(n - 1, np.uint32), np.array([LAST], np.uint32)])  # "one step"


@pytest.mark.parametrize("shape", ["constant", "clusters", "dense low end", "dense high end", "repeats", "one step"])
@pytest.mark.parametrize("n", [8191, 8192, 16385, 300007, 2_000_003])
def test_search_in_lists_of_every_shape(cuda, shape, n):
    import torch

    rng = np.random.default_rng(n)
    lst = _list(shape, n, rng)
    near = lst[rng.integers(0, n, NKEYS // 2)].astype(np.int64) + rng.integers(-2, 3, NKEYS // 2)
    keys = np.concatenate([np.clip(near, 0, LAST), rng.integers(0, LAST + 1, NKEYS - NKEYS // 2)]).astype(np.uint32)
    keys[:2] = 0, LAST
    at = np.searchsorted(lst, keys)
    want = (at < n) & (lst[np.minimum(at, n - 1)] == keys)
    dl, dk = (torch.from_numpy(x.view(np.int32)).cuda() for x in (lst, keys))
    found, count = so.search(dl, dk, 1024)
    assert np.array_equal(found.cpu().numpy().astype(bool), want)
    assert int(count.item()) == int(want.sum())
