"""Clique kernels at the edges of their size classes, on graphs whose counts
have a closed form: the complete graph K_n (C(n, k) k-cliques) and the cocktail
party graph, K_n without a perfect matching (2^k C(n/2, k)).  Their lower lists
have every length up to n - 1: 64/65 (warp or CTA root), 96/97 members of a row
(compacted by a warp or by the CTA), 128/129 and 256/257 (root lists), rows in
shared memory or in global scratch, and compacted matrices without room."""
from math import comb

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLIQUES = {k: "".join("0" if i == j else "1" for i in range(k) for j in range(k))
           for k in range(4, 8)}


def _dense(gat, n, matching):
    keep = ~np.eye(n, dtype=bool)
    if matching:
        i = np.arange(n)
        keep[i, i ^ 1] = False
    rows, cols = np.nonzero(keep)
    off = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return gat.Graph.from_csr(off, cols.astype(np.int32))


@pytest.fixture(scope="module")
def schedules(gat):
    return {k: gat.Schedule(p, "exact") for k, p in CLIQUES.items()}


@pytest.mark.parametrize("n,ks", [(3, (4, 7)), (8, (4, 5, 6, 7)), (64, (4, 5, 6, 7)), (66, (4, 5, 6, 7)),
                                  (98, (4, 5, 6)), (100, (5, 7)), (130, (4, 5, 6)), (258, (4, 5)),
                                  (460, (4, 5)), (700, (4, 5))])
@pytest.mark.parametrize("rows", [True, False])
def test_closed_forms(gat, schedules, n, ks, rows):
    ex = gat.Executor()
    for matching in (False, True):
        if matching and n % 2:
            continue
        g = _dense(gat, n, matching)
        g.upload(hub_max_bytes=1 << 30 if rows else 0)
        for k in ks:
            want = (2 ** k * comb(n // 2, k)) if matching else comb(n, k)
            s = schedules[k]
            assert s.dedicated_kernel == 2
            assert ex.count(g, s).count == want, (n, k, matching)
            if n <= 130:
                assert sum(ex.count_shard(g, s, i, 5)[0] for i in range(5)) == want
                assert ex.count(g, s, balg=True).count == want
