"""The levels of a marching tile's block (tile_levels): the choice whose blocks,
handed in order to the slots as they come free, end first.  The library's
arithmetic against a simulation of that schedule, on the CPU."""
import ctypes as C
import heapq
import random

import pytest

from cm1_b200 import binding


def _levels():
    f = binding.lib()._ZN4cm1g11tile_levelsEliiiii
    f.argtypes, f.restype = [C.c_long] + [C.c_int] * 5, C.c_int
    return f


def _end(tiles, nk, slots, over, kc):
    """End of the last block: the full chunks of all tiles, then every tile's last."""
    nch = -(-nk // kc)
    free = [0] * slots
    for n in range(tiles * nch):
        length = over + (kc if n < tiles * (nch - 1) else nk - (nch - 1) * kc)
        heapq.heapreplace(free, free[0] + length)
    return max(free)


def _simulated(tiles, nk, slots, over, kcmin, kcmax):
    best = None
    kc = kcmin
    while kc <= kcmax:
        end = _end(tiles, nk, slots, over, kc)
        if best is None or end < best[0]:
            best = (end, kc)
        if kc >= nk:
            break
        kc += 1 if kc < 16 else 2 if kc < 32 else 4
    return best[1]


@pytest.mark.parametrize("seed", range(6))
def test_choice_is_the_simulated_one(seed):
    rng, f = random.Random(seed), _levels()
    for _ in range(60):
        slots = rng.choice((1, 2, 3, 7, 12, 37))          # any number of slots; the kernels have 296 and 444
        tiles = rng.choice((1, 2, slots, slots + 1, rng.randint(1, 4 * slots)))
        a = (tiles, rng.randint(5, 70), slots, rng.choice((2, 3)), rng.choice((1, 4)), rng.choice((16, 32, 64, 128)))
        assert f(*a) == _simulated(*a), a


@pytest.mark.parametrize("a", [(1, 6, 444, 2, 1, 16), (297, 80, 296, 3, 4, 64), (234, 128, 296, 3, 1, 128),
                               (216, 79, 444, 2, 4, 16), (296, 40, 444, 2, 4, 32), (444, 64, 444, 2, 4, 32),
                               (445, 65, 444, 2, 1, 32)])
def test_choice_at_the_kernels_slots(a):
    assert _levels()(*a) == _simulated(*a)
