"""CPU restatement of the incremental sort's placement with buckets bounded by the tiles' first old keys: bucket b(k) = the
largest tile j whose first old key is <= k (0 when there is none), tile j's output = its stayers and bucket j's movers in the
order (key, stayers first, storage index). Against numpy's stable sort of (key, mover, index), over key ranges with long runs
across tiles, tiles that empty, movers outside the old range and tiles of both sizes; and the groups' ranges, put together
per tile from inner groups and open ends, against the sorted keys."""
import numpy as np
import pytest


def merge(old, new, tile):
    n = len(old)
    first = old[::tile]
    stay = old == new
    movers = np.flatnonzero(~stay)
    bucket = np.maximum(np.searchsorted(first, new[movers], side="right") - 1, 0)
    out_k, out_i = [], []
    for j in range(len(first)):
        idx = np.arange(j * tile, min(n, (j + 1) * tile))
        s, m = idx[stay[idx]], movers[bucket == j]
        both = np.concatenate([s, m])
        o = np.lexsort((both, np.concatenate([np.zeros(len(s)), np.ones(len(m))]), new[both]))
        out_k.append(new[both[o]])
        out_i.append(both[o])
    return out_k, out_i


def ranges(out_k, shift):
    """(start, stop) per group as the tiles emit them: whole ranges inside a tile, starts and ends that meet through the group's entry"""
    n, pred, base, found, open_ = sum(map(len, out_k)), None, 0, [], {}
    for j, k in enumerate(out_k):
        g = k >> shift
        heads = [p for p in range(len(k)) if (g[p - 1] if p else pred) != g[p]]
        last_tile = j + 1 == len(out_k)
        for i, p in enumerate(heads):
            stop = heads[i + 1] if i + 1 < len(heads) else (len(k) if last_tile else None)
            if stop is None:
                assert open_.setdefault(int(g[p]), [None, None])[0] is None
                open_[int(g[p])][0] = base + p
            else:
                found.append((base + p, base + stop))
        if heads and pred is not None:
            open_.setdefault(int(pred), [None, None])[1] = base + heads[0]
        if not heads and last_tile:
            open_.setdefault(int(g[-1]) if len(k) else int(pred), [None, None])[1] = n
        if len(k):
            pred = g[-1]
        base += len(k)
    assert all(s is not None and e is not None for s, e in open_.values())
    return sorted(found + [tuple(v) for v in open_.values()])


@pytest.mark.parametrize("tile", [512, 2048])
@pytest.mark.parametrize("n", [1, 511, 512, 513, 2048, 5000, 9000])
@pytest.mark.parametrize("keys, moving", [(3, 0.3), (40, 0.02), (40, 1.0), (4000, 0.1), (4000, 1.0), (100000, 0.5)])
def test_merge_equals_a_stable_sort(tile, n, keys, moving):
    rng = np.random.default_rng(n * 7 + keys + tile)
    old = np.sort(rng.integers(5, 5 + keys, n))
    new = np.where(rng.random(n) < moving, rng.integers(0, 10 + keys, n), old)  # some below and above the old range
    if n > 2 * tile:
        new[tile:2 * tile] = rng.integers(0, 10 + keys, tile)  # a tile whose particles nearly all move
    out_k, out_i = merge(old, new, tile)
    want = np.lexsort((np.arange(n), old != new, new))
    assert np.array_equal(np.concatenate(out_i), want)
    assert np.array_equal(np.concatenate(out_k), new[want])
    shift = 3
    g = new[want] >> shift
    heads = np.flatnonzero(np.r_[True, g[1:] != g[:-1]])
    assert ranges(out_k, shift) == list(zip(heads.tolist(), np.r_[heads[1:], n].tolist()))
