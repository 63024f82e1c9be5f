"""Index arithmetic the kernels rely on, checked on the CPU.

* ``k_energy_sum`` (csrc/reduce_md.cu) puts chunk c of system b into slot
  b + floor(start_b / 1024) + c, with max(1, ceil(n_b / 1024)) chunks per
  system, and sizes its partial array as natoms // 1024 + nsys + 1 slots:
  the slots must be distinct and inside that bound for any batch.
* ``div_small`` (csrc/aev.cu) forms q = floor(v / n) from a float32
  reciprocal, (v + 1/2) * float32(1/n), for the triplet indices of the
  adjoint (v < 256 * 256 + 256 * 2, n <= 256, the largest angular staging);
  it must be exact there without its correction step (which stays in the
  kernel as a guard).
* ``Share`` / ``Items`` (csrc/mlp_fused.cu) cut the (tile, model) items of the
  tiles left over into contiguous ranges, one per CTA, each item's dX going to
  a slot of its CTA; ``k_mlp_join`` must add, for every tile, each of its
  models once and nothing else, within the slots of the workspace.
"""

import numpy as np
import pytest

CHUNK = 1024


def slots_of(sys_start):
    out = []
    for b in range(len(sys_start) - 1):
        n = sys_start[b + 1] - sys_start[b]
        base = b + sys_start[b] // CHUNK
        for c in range(max(1, -(-n // CHUNK))):
            out.append(base + c)
    return out


@pytest.mark.parametrize("seed", range(20))
def test_energy_slots_distinct_and_bounded(seed):
    rng = np.random.default_rng(seed)
    nsys = int(rng.integers(1, 60))
    # sizes from empty to several chunks, with chunk-boundary cases mixed in
    sizes = rng.choice([0, 1, 7, 1023, 1024, 1025, 2048, 3000, 5000], size=nsys)
    sizes = np.where(rng.random(nsys) < 0.5, rng.integers(0, 4000, nsys), sizes)
    start = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    slots = slots_of(start)
    natoms = int(start[-1])
    assert len(set(slots)) == len(slots)
    assert max(slots) < natoms // CHUNK + nsys + 1


def test_energy_slots_single_large_system():
    start = np.array([0, 98_304])
    assert slots_of(start) == list(range(96))


def test_div_small_exact_without_correction():
    n = np.arange(1, 257, dtype=np.int64)
    rn = (np.float32(1.0) / n.astype(np.float32)).astype(np.float32)
    v = np.arange(0, 256 * 256 + 2 * 256, dtype=np.int64)
    for k in range(n.size):
        q = ((v.astype(np.float32) + np.float32(0.5)) * rn[k]).astype(np.int64)  # float32 product, truncation
        np.testing.assert_array_equal(q, v // n[k])


def _written_and_joined(ntiles, M, ndx, sms=148):
    """For every shared tile: the slots its models' sums end in, with the models of
    each, and the slots that the join adds; and the slots a CTA has."""
    blocks = min(ntiles * M, sms)
    whole = ntiles // blocks
    left = ntiles - whole * blocks
    first = [left * M * c // blocks for c in range(blocks + 1)]
    most = -(-left * M // blocks)
    apart = ndx <= 16 or most <= 1
    slots = max(1, most if apart else min(most, 2))
    # what a slot holds when the CTA is done: (tile, models), None for a whole tile's sum
    held = {(c, 0): None for c in range(blocks)} if whole else {}
    for c in range(blocks):
        for item in range(first[c], first[c + 1]):
            tile, m = divmod(item, M)
            slot = item - first[c] if apart else (0 if tile == first[c] // M else 1)
            assert slot < slots
            old = held.get((c, slot))
            joined = not apart and old is not None and old[0] == tile and m > max(0, first[c] - tile * M)
            held[c, slot] = (tile, old[1] + [m] if joined else [m])
    owner = [c for c in range(blocks) for _ in range(first[c + 1] - first[c])]
    added = []
    for tile in range(left):
        if apart:
            added.append([(owner[i], i - first[owner[i]]) for i in range(tile * M, tile * M + M)])
        else:
            added.append([(c, 0 if first[c] // M == tile else 1)
                          for c in range(owner[tile * M], owner[tile * M + M - 1] + 1)])
    return held, added, slots


@pytest.mark.parametrize("ndx", [8, 64])
@pytest.mark.parametrize("M", [2, 3, 5, 8, 11])
def test_join_adds_every_model_of_a_shared_tile_once(M, ndx):
    for ntiles in list(range(1, 460)) + [900, 1037, 2961]:
        held, added, slots = _written_and_joined(ntiles, M, ndx)
        for tile, parts in enumerate(added):
            models = []
            for at in parts:
                assert held.get(at) is not None and held[at][0] == tile, (ntiles, tile, at)
                models += held[at][1]
            assert models == list(range(M)), (ntiles, tile, models)
        # the workspace: two slots of 64 groups, or a slot of 16 per item of a CTA
        blocks = min(ntiles * M, 148)
        most = -(-ntiles * M // blocks) if ntiles < 148 else M
        assert slots * ndx <= max(min(most, 2) * 64, most * 16)
