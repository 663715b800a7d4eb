"""The cost by which the layout chooses the JFA passes' sub-tile depths, against its
definition: every chain position worked out by itself."""
import ctypes
import random


def _cost(D, zrun, step, depth, most):
    z = [a for r in range(min(step, D)) for a in range(r, D, step)]
    cost = 0
    for t0 in range(0, D, zrun):
        for p0 in range(t0, min(t0 + zrun, D), depth):
            p1 = min(p0 + depth, t0 + zrun, D)
            slots = p1 - p0 + 2
            if any(z[p] + step >= D for p in range(p0, p1 - 1)):          # a chain ends inside
                slots += (z[p0] > step) + (z[p1 - 1] + step < D - 1)
            if slots > most:
                return -1
            cost += 4 * (slots + 3) + (p1 - p0) % 2
    return cost


def test_cost_of_any_cut(asv):
    f = getattr(asv.load(), "_ZN3asv13sub_tile_costEiiiii")               # asv::sub_tile_cost
    f.argtypes, f.restype = [ctypes.c_int] * 5, ctypes.c_int
    rng = random.Random(3)
    cases = [(D, zrun, step, d, 20) for D in (2, 5, 12, 30, 31) for zrun in (1, 4, D) for step in (1, 2, 5, 6, 40) for d in (4, 7, 16)]
    cases += [(rng.randint(2, 400), rng.randint(1, 40), rng.randint(1, 6), rng.randint(4, 16), rng.choice((12, 18, 20)))
              for _ in range(2000)]
    for c in cases:
        assert f(*c) == _cost(*c), c
