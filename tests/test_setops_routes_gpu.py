"""The routes a pair can take through the batched intersection (a few keys
flattened over a warp, one warp, the whole CTA in parts), at the list lengths
where they meet, for the two widths of the kernel (by batch size), counts,
lists, bounds and exclusions, against numpy."""
from __future__ import annotations

import numpy as np
import pytest

from gary_b200 import setops as so

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 15, 16, 17, 31, 33, 383, 385, 1023, 1024, 1025, 1536, 1537, 3071, 3073, 9000]


@pytest.fixture(scope="module")
def pairs(cuda):
    """Every pair of lengths; the lists share ids, and some pairs are disjoint
    ranges or end on the largest id there is."""
    import torch

    rng = np.random.default_rng(5)
    a, b = [], []
    for i, la in enumerate(LENGTHS):
        for j, lb in enumerate(LENGTHS):
            pool = rng.choice(40 * max(la, lb, 1), la + lb, replace=False).astype(np.uint32)
            x, y = np.sort(pool[:la]), np.sort(rng.permutation(pool)[:lb])
            if (i + j) % 7 == 0:
                y = y + np.uint32(50 * max(la, lb, 1))
            if (i + j) % 5 == 0 and la and lb:
                x[-1] = y[-1] = 0xFFFFFFFE
            a.append(x), b.append(y)

    def pack(lists):
        ln = np.array([len(x) for x in lists], np.int32)
        off = np.concatenate([[0], np.cumsum((ln + 3) // 4 * 4)]).astype(np.int64)
        v = np.full(max(off[-1], 4), 0xFFFFFFFF, np.uint32)
        for x, o in zip(lists, off[:-1]):
            v[o:o + len(x)] = x
        return [torch.from_numpy(t).cuda() for t in (ln, off, v.view(np.int32))]

    la, ao, av = pack(a)
    lb, bo, bv = pack(b)
    return a, b, so.PairBatch(len(a), la, lb, ao, bo, av, bv)


@pytest.mark.parametrize("variant", ["auto", "merge", "search", "bitmap"])
def test_lists_at_the_route_limits(pairs, variant):
    a, b, batch = pairs
    counts, total, out, off = so.intersect(batch, so.VARIANTS[variant], materialise=True)
    out, off = out.cpu().numpy().view(np.uint32), off.cpu().numpy()
    want = [np.intersect1d(x, y) for x, y in zip(a, b)]
    assert counts.cpu().tolist() == [len(w) for w in want] and int(total.item()) == sum(map(len, want))
    for w, o in zip(want, off):
        assert np.array_equal(out[o:o + len(w)], w)


@pytest.mark.parametrize("variant", ["auto", "merge", "search"])
@pytest.mark.parametrize("npairs", [1, 8, 289, (1 << 18) - 1, 1 << 18])
def test_counts_for_every_batch_size(pairs, variant, npairs):
    import torch

    a, b, batch = pairs
    want = torch.tensor([len(np.intersect1d(x, y)) for x, y in zip(a, b)], device="cuda")
    # the same lists again and again, starting with the longest
    at = (torch.arange(npairs, device="cuda") * 288 + 288) % 289
    many = so.PairBatch(npairs, batch.la[at].contiguous(), batch.lb[at].contiguous(), batch.a_off[:-1][at].contiguous(),
                        batch.b_off[:-1][at].contiguous(), batch.a, batch.b)
    counts, total = so.intersect(many, so.VARIANTS[variant])
    assert torch.equal(counts, want[at]) and int(total.item()) == int(want[at].sum().item())


@pytest.mark.parametrize("variant", ["auto", "merge", "search"])
def test_bounds_and_exclusions(pairs, variant):
    import torch

    a, b, batch = pairs
    rng = np.random.default_rng(7)
    bound = np.array([rng.integers(0, 40 * max(len(x), len(y), 1) + 1) for x, y in zip(a, b)], np.uint32)
    bound[::9] = 0xFFFFFFFF
    ex, off, want = [], [0], []
    for x, y, m in zip(a, b, bound):
        w = np.intersect1d(x, y)
        w = w[w < m]
        drop = list(w[:3]) + list(w[:1]) + list(x[-2:])  # members, one twice, and ids past the bound or of one list
        ex += drop
        off.append(len(ex))
        want.append(len(np.setdiff1d(w, np.array(drop, np.uint32))))
    t = lambda v, dt: torch.from_numpy(np.ascontiguousarray(v).view(dt)).cuda()  # noqa: E731
    counts, total = so.intersect_num(batch, t(bound, np.int32), t(np.array(off, np.int64), np.int64),
                                     t(np.array(ex, np.uint32), np.int32), so.VARIANTS[variant])
    assert counts.cpu().tolist() == want and int(total.item()) == sum(want)


@pytest.mark.parametrize("n_list", [8191, 8192, 8193, 16385, 65543, (1 << 20) + 13])
@pytest.mark.parametrize("n_keys", [606207, 606208, 1300007, 5000003])
def test_search_of_many_keys(cuda, n_list, n_keys):
    """Every depth of the separator tree, lists with repeated ids and the ids at
    both ends of the range."""
    import torch

    rng = np.random.default_rng(n_list + n_keys)
    lst = np.sort(rng.integers(0, 4 * n_list, n_list).astype(np.uint32))
    lst[0], lst[-1], lst[-2] = 0, 0xFFFFFFFE, 0xFFFFFFFE
    keys = rng.integers(0, 4 * n_list + 8, n_keys).astype(np.uint32)
    keys[:4] = [0, 0xFFFFFFFE, 0xFFFFFFFF, 0xFFFFFFFD]
    found, count = so.search(torch.from_numpy(lst.view(np.int32)).cuda(), torch.from_numpy(keys.view(np.int32)).cuda(), 256)
    want = np.isin(keys, lst)
    assert np.array_equal(found.cpu().numpy().astype(bool), want) and int(count.item()) == int(want.sum())
