"""The float cell indices of the plain kernels against the reference's double ones, emulated on the
CPU: a float product rounded toward zero (mover) or down (deposit) has the integer part the double
product has, and compares alike with the node array's bounds."""
import numpy as np
import pytest


def rounded(prod, down):
    """The exact product as a float rounded down, or toward zero."""
    r = prod.astype(np.float32)
    over = r.astype(np.float64) > prod if down else np.abs(r.astype(np.float64)) > np.abs(prod)
    return np.where(over, np.nextafter(r, np.float32(-np.inf) if down else np.float32(0)), r)


@pytest.mark.parametrize("cells,L", [(61, 20.0), (128, 20.0), (7, 3.1), (3, 1e-3), (1000, 0.77),
                                     (1 << 21, 5.0)])
def test_float_cells_equal_double_cells(cells, L):
    rng = np.random.default_rng(cells)
    inv = np.float32(1.0 / (L / cells))
    n = cells + 3
    x = (rng.integers(-3, cells + 4, 200000) * (L / cells)).astype(np.float32)
    for _ in range(3):
        k = rng.integers(-1, 2, x.size)
        x = np.where(k < 0, np.nextafter(x, np.float32(-1e9)),
                     np.where(k > 0, np.nextafter(x, np.float32(1e9)), x))
    x = np.concatenate([x, (rng.uniform(-3, 1.01, 100000) * L).astype(np.float32),
                        np.float32([0.0, -0.0, 1e-45, -1e-45, 1e30, -1e30])])
    prod = x.astype(np.float64) * np.float64(inv)   # exact: 24 + 24 bits
    rz, rd = rounded(prod, False), rounded(prod, True)
    i_mover = 2 + np.trunc(np.clip(prod, -8.0, n + 8.0)).astype(np.int64)
    i_dep = 2 + np.floor(np.clip(prod, -8.0, n + 8.0)).astype(np.int64)
    in_mover = (rz > np.float32(-2)) & (rz < np.float32(n - 2))
    in_dep = (rd >= np.float32(-1)) & (rd < np.float32(n - 2))
    assert np.array_equal(in_mover, (i_mover >= 1) & (i_mover <= n - 1))
    assert np.array_equal(in_dep, (i_dep >= 1) & (i_dep <= n - 1))
    assert np.array_equal(2 + np.trunc(rz[in_mover]).astype(np.int64), i_mover[in_mover])
    assert np.array_equal(2 + np.floor(rd[in_dep]).astype(np.int64), i_dep[in_dep])


def test_final_velocity_and_reciprocal():
    rng = np.random.default_rng(1)
    n = 400000
    # 2 u' - u in double and then float = one rounding of the exact difference (long double holds
    # it for exponents up to 40 apart; further apart the larger term is the result of both)
    up = (rng.standard_normal(n) * 10.0 ** rng.uniform(-6, 6, n)).astype(np.float32)
    u = (rng.standard_normal(n) * 10.0 ** rng.uniform(-6, 6, n)).astype(np.float32)
    u[: n // 4] = np.nextafter(2 * up[: n // 4], np.float32(0))
    ref = (2.0 * up.astype(np.float64) - u.astype(np.float64)).astype(np.float32)
    if np.finfo(np.longdouble).nmant >= 63:
        one = (2 * up.astype(np.longdouble) - u.astype(np.longdouble)).astype(np.float32)
        gap = np.abs(np.log2(np.abs(2.0 * up)) - np.log2(np.abs(u) + 1e-300)) < 38
        assert np.array_equal(ref[gap], one[gap])
        far = ~gap
        big = np.where(np.abs(2.0 * up) > np.abs(u), 2 * up, -u).astype(np.float32)
        assert np.array_equal(ref[far], big[far])
    # the reciprocal: an approximation within 2^-22 and one third-order step lies within one unit
    # in the last place of the quotient, so away from midpoints of floats it rounds alike
    o = (10.0 ** rng.uniform(-12, 17, n)).astype(np.float32)
    d = 1.0 + o.astype(np.float64)
    r = ((1.0 / d) * (1 + rng.uniform(-1, 1, n) * 2.0 ** -22)).astype(np.float32).astype(np.float64)
    LD = np.longdouble
    e = (1 - LD(1) * d * r).astype(np.float64)
    q = (LD(1) * r + LD(1) * r * (e + e * e)).astype(np.float64)
    low = q.view(np.int64) & 0x1FFFFFFF
    slow = (low >= 0x0FFFFFFE) & (low <= 0x10000002)
    assert np.abs(q.view(np.int64) - (1.0 / d).view(np.int64)).max() <= 1
    assert np.array_equal(q[~slow].astype(np.float32), (1.0 / d)[~slow].astype(np.float32))


@pytest.mark.parametrize("nb,L", [(33, 20.0), (1, 7.7), (64, 1e-3), (1000, 3.3), (65536, 1e3)])
def test_sort_bins_from_products(nb, L):
    """floor(x / dist) in float arithmetic against floor(x * (1 / dist)) where the latter is used:
    farther than 4.8e-7 of its value from an integer."""
    rng = np.random.default_rng(nb)
    dist = np.float32(L / np.float32(nb))
    inv = np.float32(1.0 / np.float64(dist))
    x = (rng.integers(-2, nb + 3, 200000) * np.float64(dist)).astype(np.float32)
    for _ in range(6):
        k = rng.integers(-1, 2, x.size)
        x = np.where(k < 0, np.nextafter(x, np.float32(-1e9)),
                     np.where(k > 0, np.nextafter(x, np.float32(1e9)), x))
    x = np.concatenate([x, (rng.uniform(-1, 1.1, 200000) * L).astype(np.float32),
                        np.float32([0.0, -0.0, 1e-45, -1e-45, 1e30, -1e30])])
    ref = np.floor(x / dist)
    q = x * inv
    used = np.abs(q - np.rint(q)) > np.abs(q) * np.float32(4.8e-7)
    assert used.mean() > 0.3
    assert np.array_equal(np.floor(q[used]), ref[used])
