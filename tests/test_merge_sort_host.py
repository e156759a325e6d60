"""The index algebra of the merge sort (stardust_b200/csrc/sd_resort.cu), on the CPU.

Positions sorted by their old row keys, some keys changed, one bit per position
marking at least the changed ones: the merge places every position by counts
alone, and the result must be the stable sort of the new keys, with the new row
table derived from the old one. This states the formulas the kernels evaluate
and checks them against numpy's stable argsort, including marked positions whose
key did not change (bits left over from a step whose merge never ran). The GPU
tests check the kernels themselves against the full radix sort.
"""
import numpy as np
import pytest


def merge_by_counts(old, new, marked, rows):
    """Permutation and new row table by the merge formulas (vectorised)."""
    n = len(old)
    rs_old = np.searchsorted(old, np.arange(rows + 1), side="left")
    below = np.concatenate([[0], np.cumsum(marked)])  # changed_below(x) = below[x]
    ci = np.nonzero(marked)[0]                         # C in position order
    o = np.argsort(new[ci], kind="stable")
    ck, ci = new[ci][o], ci[o]                         # C sorted by key, stable
    c_rows = np.searchsorted(ck, np.arange(rows + 1), side="left")
    perm = np.full(n, -1, np.int64)
    # changed (k, i) at rank r: r + unchanged below the old row start of k, plus the
    # unchanged ones of the old row k below i
    r = np.arange(len(ci))
    lb, ub = rs_old[ck], rs_old[ck + 1]
    m = np.minimum(ub, ci)
    u = (lb - below[lb]) + np.where(ci > lb, (m - lb) - (below[m] - below[lb]), 0)
    perm[r + u] = ci
    # unchanged (k, j): j - changed below j + C with key < k + C with key k below j
    j = np.nonzero(~marked)[0]
    k = new[j]
    before = np.searchsorted(ck * (n + 1) + ci, k * (n + 1) + j)  # C before (k, j)
    perm[j - below[j] + before] = j
    rs_new = rs_old - below[rs_old] + c_rows
    return perm, rs_new


def scene(n, rows, frac, seed, stale=0.0, clustered=False):
    rng = np.random.default_rng(seed)
    old = np.sort(rng.integers(0, rows, n)).astype(np.int64)
    new = old.copy()
    moved = rng.random(n) < frac
    if clustered:
        new[moved] = rows // 2
    else:
        new[moved] = np.clip(old[moved] + rng.choice([-16, -4, -1, 1, 4, 16], moved.sum()), 0, rows - 1)
    marked = (new != old) | (rng.random(n) < stale)
    return old, new, marked


@pytest.mark.parametrize("n,rows,frac,stale,clustered", [
    (1, 16, 1.0, 0.0, False),
    (1000, 16, 0.1, 0.0, False),
    (65536, 256, 0.01, 0.0, False),
    (200_000, 4096, 0.005, 0.0, False),
    (70_000, 1024, 0.3, 0.0, False),
    (5000, 16, 0.0, 0.0, False),          # nothing moved: the identity
    (3000, 64, 1.0, 0.0, False),          # everything moved
    (66_000, 128, 0.05, 0.0, True),       # the changed keys all in one row
    (20_000, 64, 0.02, 0.1, False),       # stale marks on unchanged positions
    (20_000, 64, 0.0, 0.3, False),
])
def test_merge_formulas_give_the_stable_sort(n, rows, frac, stale, clustered):
    old, new, marked = scene(n, rows, frac, n + rows, stale, clustered)
    perm, rs_new = merge_by_counts(old, new, marked, rows)
    ref = np.argsort(new, kind="stable")
    assert np.array_equal(perm, ref)
    assert np.array_equal(rs_new, np.searchsorted(new[ref], np.arange(rows + 1), side="left"))


def test_an_unmarked_change_breaks_the_merge():
    """The marks must cover every changed position: with one left out, the
    unchanged run it sits in is no longer sorted and the formulas place it wrong."""
    old, new, marked = scene(20_000, 64, 0.02, 7)
    i = np.nonzero(marked)[0][len(np.nonzero(marked)[0]) // 2]
    marked[i] = False
    perm, _ = merge_by_counts(old, new, marked, 64)
    assert not np.array_equal(perm, np.argsort(new, kind="stable"))


def merge_wide(old, new, marked, rows, shift):
    """The permutation where a row holds 2^shift keys (key 0, the empty slots, is a row
    of its own): a binary search of the row's unchanged positions places a changed key."""
    n = len(old)
    low = np.concatenate([[0], (np.arange(rows + 1) << shift) + 1])
    row = np.where(new > 0, ((np.maximum(new, 1) - 1) >> shift) + 1, 0)
    rs_old = np.searchsorted(old, low, side="left")
    below = np.concatenate([[0], np.cumsum(marked)])
    ci = np.nonzero(marked)[0]
    o = np.argsort(new[ci], kind="stable")
    ck, ci = new[ci][o], ci[o]
    c_rows = np.searchsorted(ck, low, side="left")
    perm = np.full(n, -1, np.int64)
    for r, (k, i) in enumerate(zip(ck, ci)):
        lo, hi = rs_old[row[i]], rs_old[row[i] + 1]
        while lo < hi:
            mid = (lo + hi) >> 1
            q = mid
            while q < hi and marked[q]:
                q += 1
            if q < hi and (new[q], q) < (k, i):
                lo = q + 1
            else:
                hi = mid
        perm[r + lo - below[lo]] = i
    for j in np.nonzero(~marked)[0]:
        a, b = c_rows[row[j]], c_rows[row[j] + 1]
        a += sum((ck[q], ci[q]) < (new[j], j) for q in range(a, b))
        perm[j - below[j] + a] = j
    return perm, rs_old - below[rs_old] + c_rows, low


@pytest.mark.parametrize("n,rows,shift,frac,stale", [(1, 16, 4, 1.0, 0.0), (700, 16, 4, 0.05, 0.0), (2000, 64, 3, 0.3, 0.1),
                                                     (900, 16, 5, 1.0, 0.0), (800, 256, 4, 0.02, 0.5)])
def test_wide_rows(n, rows, shift, frac, stale):
    rng = np.random.default_rng(n)
    old = np.sort(rng.integers(0, (rows << shift) + 1, n))
    old[: n // 20] = 0
    new = old.copy()
    moved = rng.random(n) < frac
    new[moved] = np.clip(old[moved] + rng.choice([-(1 << shift), -1, 1, 1 << shift], moved.sum()), 0, rows << shift)
    new[moved & (rng.random(n) < 0.05)] = 0  # lost
    marked = (new != old) | (rng.random(n) < stale)
    perm, rs, low = merge_wide(old, new, marked, rows, shift)
    assert np.array_equal(perm, np.argsort(new, kind="stable"))
    assert np.array_equal(rs, np.searchsorted(np.sort(new), low, side="left"))
