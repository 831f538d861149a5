"""The MRG32k3a jump-ahead of the path-start cursor (mrg_jump): matrix
powers of the two component recurrences (L'Ecuyer 1999) against stepping the
recurrences one by one in Python integers."""
import numpy as np

from oracle import oracle

M1, M2 = 4294967087, 4294944443


def step(s1, s2):
    """One step of both components, states oldest value first."""
    p1 = (1403580 * s1[1] - 810728 * s1[0]) % M1
    p2 = (527612 * s2[2] - 1370589 * s2[0]) % M2
    return [s1[1], s1[2], p1], [s2[1], s2[2], p2]


def test_jump_matches_stepping():
    rng = np.random.default_rng(3)
    for steps in (0, 1, 2, 3, 5, 24, 27, 192, 3 * 1024):
        s1 = [int(x) for x in rng.integers(1, M1, 3)]
        s2 = [int(x) for x in rng.integers(1, M2, 3)]
        a, b = list(s1), list(s2)
        for _ in range(steps):
            a, b = step(a, b)
        j1, j2 = oracle.mrg_jump(steps, s1, s2)
        assert [int(x) for x in j1] == a, steps
        assert [int(x) for x in j2] == b, steps


def test_jump_extreme_states():
    """States at the top of each modulus exercise every reduction branch."""
    for s1, s2 in (([M1 - 1] * 3, [M2 - 1] * 3), ([0, 0, 1], [1, 0, 0]), ([M1 - 1, 0, M1 - 1], [0, M2 - 1, 0])):
        a, b = list(s1), list(s2)
        for _ in range(24):
            a, b = step(a, b)
        j1, j2 = oracle.mrg_jump(24, s1, s2)
        assert [int(x) for x in j1] == a
        assert [int(x) for x in j2] == b


def test_powers_match_stepping():
    rng = np.random.default_rng(4)
    s1 = [int(x) for x in rng.integers(1, M1, 3)]
    s2 = [int(x) for x in rng.integers(1, M2, 3)]
    for steps in (3, 15, 24):
        for power in range(7):
            a, b = list(s1), list(s2)
            for _ in range(steps << power):
                a, b = step(a, b)
            j1, j2 = oracle.mrg_jump(steps, s1, s2, power)
            assert ([int(x) for x in j1], [int(x) for x in j2]) == (a, b), (steps, power)


def test_draws_match_stepping():
    """The recurrences in 64-bit integers with folded high words, against Python
    integers: random states and those at the ends of each modulus; uniforms are
    z / m1 to a float's rounding."""
    rng = np.random.default_rng(5)
    states = [([M1 - 1] * 3, [M2 - 1] * 3), ([0, 0, 1], [1, 0, 0]), ([M1 - 1, 0, M1 - 1], [0, M2 - 1, 0]),
              ([M1 - 1, 1, 0], [M2 - 1, 0, 1]), ([0, M1 - 1, 0], [0, 0, M2 - 1])]
    states += [([int(x) for x in rng.integers(0, M1, 3)], [int(x) for x in rng.integers(0, M2, 3)]) for _ in range(200)]
    for s1, s2 in states:
        z, u, e1, e2 = oracle.mrg_draws(50, s1, s2)
        a, b = s1, s2
        for k in range(50):
            a, b = step(a, b)
            d = (a[2] - b[2]) % M1
            want = d if d else M1
            assert int(z[k]) == want
            assert abs(float(u[k]) - want / M1) <= 2.0 ** -24 * want / M1 and 0 < u[k] <= 1
        assert ([int(x) for x in e1], [int(x) for x in e2]) == (a, b)
