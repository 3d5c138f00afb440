"""The level-scheduled sweep, in one thread-block cluster or over the grid,
against the sequential sweep in numpy: one row, rows with more off-diagonal
blocks than a warp fetches ahead, one and two sweeps, both precisions, sizes
around the largest whose z fits in a 16-CTA cluster (5 x 5 blocks: 16 x 204,800 /
40 = 81,920 rows; one more row takes the grid-wide sweep), and levels of up to
256 rows (the cluster's), a little more and half of the matrix (the grid's).

1e-12: FP64 substitutions of well-conditioned blocks (unit roundoff times the
rows a value passes through); the FP32 matrix is compared with the numpy sweep
on the rounded values and FP32-rounded factors, 2e-6."""
import time

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _matrix(n, bs, degree, seed):
    rng = np.random.default_rng(seed)
    cols_of = [{i} for i in range(n)]
    for i in range(n):
        for j in rng.integers(max(0, i - 40), min(n, i + 41), size=degree):
            cols_of[i].add(int(j))
            cols_of[int(j)].add(i)
    row_ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols_of])]).astype(np.int32)
    cols = np.concatenate([sorted(c) for c in cols_of]).astype(np.int32)
    rows = np.repeat(np.arange(n), np.diff(row_ptr))
    vals = 0.3 * rng.standard_normal((len(cols), bs, bs))
    d = rows == cols
    vals[d] += (2.0 * np.diff(row_ptr))[:, None, None] * np.eye(bs)
    return row_ptr, cols, vals


def _sequential(row_ptr, cols, vals, r, sweeps):
    n, bs = len(row_ptr) - 1, vals.shape[1]
    z, r = np.zeros((n, bs)), r.reshape(n, bs)
    for _ in range(sweeps):
        for order in (range(n), range(n - 1, -1, -1)):
            for i in order:
                s = r[i].copy()
                for k in range(row_ptr[i], row_ptr[i + 1]):
                    if cols[k] == i:
                        d = vals[k]
                    else:
                        s -= vals[k] @ z[cols[k]]
                z[i] = np.linalg.solve(d, s)
    return z.ravel()


@pytest.mark.parametrize("n,bs,degree", [(1, 5, 0), (15, 6, 2), (300, 5, 3), (257, 6, 4), (90, 5, 14)])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("sweeps", [1, 2])
def test_matches_sequential_sweep(cb, n, bs, degree, mixed, sweeps):
    row_ptr, cols, vals = _matrix(n, bs, degree, 3)
    r = np.random.default_rng(4).standard_normal(n * bs)
    A = cb.Bsr(row_ptr, cols, bs, cb.PREC_MIXED if mixed else cb.PREC_FP64)
    A.set_values(vals)
    A.sgs_setup(cb.SGS_LEVEL, sweeps)
    ref = _sequential(row_ptr, cols, vals.astype(np.float32).astype(np.float64) if mixed else vals, r, sweeps)
    assert rel_err(A.sgs_apply(r), ref) < (2e-6 if mixed else 1e-12)


@pytest.mark.parametrize("n", [81918, 81920, 81922])
def test_largest_cluster_sizes(cb, n):
    """Coupled pairs of rows: two wide levels, any size, a closed form."""
    bs, rng = 5, np.random.default_rng(5)
    row_ptr = np.arange(0, 2 * n + 1, 2, dtype=np.int32)
    first = np.arange(0, n, 2)
    cols = np.stack([first, first + 1, first, first + 1], axis=1).astype(np.int32).ravel()
    vals = 0.3 * rng.standard_normal((2 * n, bs, bs))
    d0, u, lo, d1 = (vals[k::4] for k in range(4))
    d0 += 4.0 * np.eye(bs)
    d1 += 4.0 * np.eye(bs)
    r = rng.standard_normal((n, bs))
    A = cb.Bsr(row_ptr, cols, bs)
    A.set_values(vals)
    A.sgs_setup(cb.SGS_LEVEL, 1)
    z = A.sgs_apply(r.ravel()).reshape(n, bs)

    def solve(d, s):
        return np.linalg.solve(d, s[:, :, None])[:, :, 0]

    y0 = solve(d0, r[0::2])
    z1 = solve(d1, r[1::2] - np.einsum("kij,kj->ki", lo, y0))
    z0 = solve(d0, r[0::2] - np.einsum("kij,kj->ki", u, z1))
    assert rel_err(z[1::2], z1) < 1e-12
    assert rel_err(z[0::2], z0) < 1e-12


@pytest.mark.parametrize("n,width", [(81918, 256), (81920, 256), (81922, 256), (10241, 255), (10300, 480), (10300, 520)])
def test_chains(cb, n, width):
    """`width` chains of rows side by side: level k is rows k * width on, solved
    for all chains at once in numpy."""
    bs, rng = 5, np.random.default_rng(6)
    i = np.arange(n)
    cols = np.stack([i - width, i, i + width], axis=1)
    have = (cols >= 0) & (cols < n)
    row_ptr = np.concatenate([[0], np.cumsum(have.sum(axis=1))]).astype(np.int32)
    vals = 0.3 * rng.standard_normal((n, 3, bs, bs))
    vals[:, 1] += 4.0 * np.eye(bs)
    r = rng.standard_normal((n, bs))
    A = cb.Bsr(row_ptr, cols[have].astype(np.int32), bs)
    A.set_values(vals[have])
    A.sgs_setup(cb.SGS_LEVEL, 1)
    z = np.zeros((n, bs))
    for side in (0, 2):
        for k in (range(0, n, width) if side == 0 else reversed(range(0, n, width))):
            q = slice(k, min(k + width, n))
            s = r[q].copy()
            for c in (0, 2):
                m = have[q, c]
                s[m] -= np.einsum("kij,kj->ki", vals[q, c][m], z[cols[q, c][m]])
            z[q] = np.linalg.solve(vals[q, 1], s[:, :, None])[:, :, 0]
    assert rel_err(A.sgs_apply(r.ravel()).reshape(n, bs), z) < 1e-12


def test_wide_levels_take_the_whole_gpu(cb):
    """Two levels of 20,000 rows, 61 us a sweep over the grid: 5.9 times the
    multicolour sweep of the same rows.  One cluster takes 566 us, 54 times; the
    bound of 18 lies between."""
    n, bs, sweeps = 40000, 5, 40
    row_ptr = np.arange(0, 2 * n + 1, 2, dtype=np.int32)
    half = np.arange(n // 2)
    cols = np.concatenate([np.stack([half, half + n // 2], axis=1)] * 2).astype(np.int32).ravel()
    vals = np.tile(0.1 * np.ones((bs, bs)), (2 * n, 1, 1))
    vals[np.repeat(np.arange(n), 2) == cols] += 4.0 * np.eye(bs)
    r = np.random.default_rng(7).standard_normal(n * bs)
    times = {}
    for ordering in (cb.SGS_COLOR, cb.SGS_LEVEL):
        A = cb.Bsr(row_ptr, cols, bs)
        A.set_values(vals)
        took = {}
        for count in (1, sweeps):  # the difference leaves the copies out
            A.sgs_setup(ordering, count)
            for _ in range(6):
                t = time.perf_counter()
                A.sgs_apply(r)
                took.setdefault(count, []).append(time.perf_counter() - t)
        times[ordering] = min(took[sweeps]) - min(took[1])
    assert times[cb.SGS_LEVEL] < 18.0 * times[cb.SGS_COLOR]
