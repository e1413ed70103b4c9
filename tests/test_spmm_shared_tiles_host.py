"""How the CTAs that share a tile of the one-kernel SpMM find their entries (csrc/spmm_direct.cuh), restated lane by lane: the search for the ends of a part, the windows that a
group of lanes walks, and the checks.  For rows in any order every entry is scattered once, or the row is found out and computed entry by entry; ascending rows are never
found out."""
import numpy as np
import pytest

CHUNK, NONE = 128, 2**31 - 1


def search(cols, group, bound):
    """The first entry with a column of at least `bound`, as a group of lanes finds it in an ascending row."""
    lo, hi = 0, len(cols)
    while lo < hi:
        n = sum(int(cols[lo + (hi - lo) * lane // group]) < bound for lane in range(group))   # the ballot's population
        new_lo = lo + (hi - lo) * (n - 1) // group + 1 if n else lo
        new_hi = lo + (hi - lo) * n // group if n < group else hi
        lo, hi = new_lo, max(new_hi, new_lo)
    return lo


def part_of_row(cols, V, K, chunk0, chunk1, first, last):
    """(scattered entries, found out) of one CTA for one vector-row."""
    rows = 16 // V
    group, window = 32 // rows, min(rows, 8)
    begin = 0 if first else search(cols, group, chunk0 * CHUNK)
    end = len(cols) if last else search(cols, group, chunk1 * CHUNK)
    bad, end = begin > end, max(begin, end)
    scattered = []
    part_end = min(chunk1 * CHUNK, K)
    for lane in range(group):
        at = np.arange(begin + lane, end, group)                       # the lane's entries
        at = np.concatenate([at, np.full(-len(at) % window + 2 * window, -1)]).reshape(-1, window)
        col = np.where(at >= 0, cols[at], NONE)
        left = np.where(at > 0, cols[at - 1], -NONE)
        w = 0
        bad |= bool((left[0] >= col[0]).any())
        for c in range(chunk0, chunk1):
            k0, k1 = c * CHUNK, min((c + 1) * CHUNK, K)
            scattered.append(at[w][(col[w] >= k0) & (col[w] < k1)])
            while col[w, -1] < k1:
                w += 1
                bad |= bool((left[w] >= col[w]).any())
                scattered.append(at[w][(col[w] >= k0) & (col[w] < k1)])
        bad |= bool(((col[w] != NONE) & (col[w] >= part_end)).any())
    return np.concatenate(scattered), bad


def rows_of_blocks(rng, K, count):
    for i in range(count):
        c = np.sort(rng.choice(K, int(rng.integers(2, K // 2)), replace=False))
        if i % 4 == 0:
            yield c, True
        elif i % 4 == 3:   # a band first, strided columns after
            at, step = int(rng.integers(0, K - K // 8)), int(rng.integers(3, 20))
            band = np.arange(at, at + K // 8)
            yield np.concatenate([band, np.setdiff1d(np.arange(0, K, step), band)]), False
        else:
            blocks = np.split(c, np.sort(rng.choice(np.arange(1, len(c)), min(int(rng.integers(1, 5)), len(c) - 1), replace=False)))
            c = np.concatenate([blocks[j] for j in rng.permutation(len(blocks))])
            yield c, bool((np.diff(c) > 0).all())


@pytest.mark.parametrize("V", [1, 2, 4, 8])
@pytest.mark.parametrize("parts,K", [(2, 900), (4, 3072), (8, 3100)])
def test_every_entry_once_or_the_row_is_found_out(V, parts, K):
    rng = np.random.default_rng(V * K)
    chunks = (K + CHUNK - 1) // CHUNK
    disordered = 0
    for cols, ascending in rows_of_blocks(rng, K, 200):
        seen, bad = [], False
        for p in range(parts):
            s, b = part_of_row(cols, V, K, p * chunks // parts, (p + 1) * chunks // parts, p == 0, p + 1 == parts)
            seen.append(s)
            bad |= b
        assert not (ascending and bad)
        disordered += bad
        assert bad or np.array_equal(np.sort(np.concatenate(seen)), np.arange(len(cols)))
    assert disordered > 100


def test_a_run_past_the_end_of_a_part():
    """0 .. 99, 2000 .. 2200, 100 .. 1499, 2300 .. 2999 of 3072 columns in two parts: the first one's lanes stop in the run of 2000 .. 2200, ahead of the descent behind it."""
    cols = np.concatenate([np.arange(100), np.arange(2000, 2201), np.arange(100, 1500), np.arange(2300, 3000)])
    for V in (1, 2, 4, 8):
        seen, bad = part_of_row(cols, V, 3072, 0, 12, True, False)
        assert bad and len(seen) < 1500
