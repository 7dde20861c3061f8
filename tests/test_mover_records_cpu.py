"""The room that the host lays out for the pair loop's mover records, against where the step
kernel puts and reads them (restated here from mover_slot and MoverLane): every plan of
every molecule fits, whatever its size, charged part, system and launch shape."""
import ctypes
import random

import cgppd_gb300


def lanes(n, N, C, W):
    """Lanes per other residue: the cheapest g, ties to the smaller."""
    def cost(g):
        per = W * (32 // g)
        passes = (-(-(N - n) // C) + per - 1) // per
        return passes * (-(-n // g) + 2 + (g - 1).bit_length())
    return min(range(1, min(32, n) + 1), key=lambda g: (cost(g), g))


def test_every_plan_fits():
    cgppd_gb300.build()
    L = cgppd_gb300.lib()
    records, size = L._ZN5cgppd13mover_recordsEiiiii, L._ZN5cgppd10mover_sizeEi
    rng, seen = random.Random(1), set()
    for _ in range(6000):
        n = rng.choice([rng.randint(1, 70), rng.randint(1, 500)])
        n1 = rng.choice([0, n, rng.randint(0, n)])
        N = n + rng.choice([0, rng.randint(0, 200), rng.randint(0, 20000)])
        C, W = rng.choice([1, 2, 3, 4, 5, 6, 8, 16]), rng.choice([4, 8, 16])
        g = lanes(n, N, C, W)
        seen.add(g)
        (k1, r1), (k2, r2) = divmod(n1, g), divmod(n - n1, g)
        second = (k1 + (r1 > 0) + 1) // 2 * g
        room = records(n, n1, N, C, W)
        for o in range(n):                       # written
            k, slot = divmod(o if o < n1 else o - n1, g)
            assert (0 if o < n1 else second) + k // 2 * g + slot < room
        for sub in range(g):                     # read
            K1, slot2 = k1 + (sub < r1), (sub - r1) % g
            K2 = k2 + (slot2 < r2)
            assert K1 == 0 or sub + (K1 - 1) // 2 * g < room
            assert K2 == 0 or second + slot2 + (K2 - 1) // 2 * g < room
        assert 2 * room >= n                     # a flex move's displacements fit as well
        bound = size(room)
        assert (bound + 1) // 2 + 2 * min(bound, 32) >= room
    assert {1, 2, 3, 4, 31, 32} <= seen
