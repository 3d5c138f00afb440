"""Small block systems for the reduced multicolour BiCGSTAB: a box (two
colours), a random graph (several colours), in natural or colour order, and a
pattern without symmetry."""
import numpy as np

import colour_sgs as CS


def _graph(kind, n, rng):
    edges = set()
    if kind == "box":
        nx, ny = 5, 3
        for i in range(n):
            for j in (i + 1 if (i + 1) % nx else -1, i + nx if (i // nx) % ny + 1 < ny else -1, i + nx * ny):
                if 0 <= j < n:
                    edges |= {(i, j), (j, i)}
    else:
        for i in range(n):
            for j in rng.integers(0, n, size=2):
                if i != j:
                    edges |= {(i, int(j)), (int(j), i)}
        if kind == "one_sided":  # half of the lower entries are missing
            edges = {(i, j) for i, j in sorted(edges) if i < j or rng.random() < 0.5}
    return edges


def system(kind, n, bs, order, seed=0):
    """(row_ptr, cols, values, colour of each row) of a diagonally dominant matrix."""
    rng = np.random.default_rng(seed)
    edges = _graph(kind, n, rng)
    row_ptr, cols = np.zeros(n + 1, dtype=np.int32), []
    for i in range(n):
        cols += sorted([i] + [j for a, j in edges if a == i])
        row_ptr[i + 1] = len(cols)
    cols = np.array(cols, dtype=np.int32)
    rows = np.repeat(np.arange(n), np.diff(row_ptr))
    vals = 0.3 / bs * rng.standard_normal((len(cols), bs, bs)) - 0.7 * np.eye(bs)
    deg = np.diff(row_ptr)
    d = rows == cols
    vals[d] = (0.8 * deg[:, None, None] + 1.0) * np.eye(bs) + 0.4 / bs * rng.standard_normal((n, bs, bs))
    vals = vals.ravel()
    if order == "colour":
        row_ptr, cols, vals, _, _ = CS.colour_order(row_ptr, cols, vals, bs)
    return row_ptr, cols, vals, colours(row_ptr, cols)


def mix_equations(row_ptr, vals, bs, cond, seed=1):
    """The system with each row's equations combined by a matrix of condition
    `cond`: the same solution, diagonal blocks of that condition."""
    rng = np.random.default_rng(seed)
    n = len(row_ptr) - 1
    q, p = (np.linalg.qr(rng.standard_normal((n, bs, bs)))[0] for _ in range(2))
    t = np.einsum("kij,j,klj->kil", q, np.logspace(0.0, np.log10(cond), bs), p)
    rows = np.repeat(np.arange(n), np.diff(row_ptr))
    return np.einsum("kij,kjl->kil", t[rows], vals.reshape(-1, bs, bs)).ravel()


def diagonal(row_ptr, cols, vals, bs):
    rows = np.repeat(np.arange(len(row_ptr) - 1), np.diff(row_ptr))
    return vals.reshape(-1, bs, bs)[rows == cols]


def colours(row_ptr, cols):
    """The colours of the sweep: greedy over the row's columns and, where that
    leaves rows of a colour coupled, over the rows that list it too."""
    colour = CS.greedy_colours(row_ptr, cols)
    n = len(row_ptr) - 1
    rows = np.repeat(np.arange(n), np.diff(row_ptr))
    if not np.any((colour[rows] == colour[cols]) & (rows != cols)):
        return colour
    pairs = sorted(set(zip(rows, cols)) | set(zip(cols, rows)))
    both = np.array([j for _, j in pairs], dtype=np.int32)
    ptr = np.searchsorted([i for i, _ in pairs], np.arange(n + 1))
    return CS.greedy_colours(ptr, both)


def dense(row_ptr, cols, vals, bs):
    n = len(row_ptr) - 1
    M = np.zeros((n * bs, n * bs))
    blocks = vals.reshape(-1, bs, bs)
    for i in range(n):
        for k in range(row_ptr[i], row_ptr[i + 1]):
            M[i * bs:(i + 1) * bs, cols[k] * bs:(cols[k] + 1) * bs] = blocks[k]
    return M


def colour_sgs(M, colour, bs, fp32=False):
    """z = M^-1 r of one symmetric sweep in colour order, dense; fp32: with the
    diagonal inverses of a mixed-precision system, rounded to FP32."""
    c = np.repeat(colour, bs)
    unit = np.repeat(np.arange(len(colour)), bs)
    same = unit[:, None] == unit[None, :]
    low = np.where((c[None, :] < c[:, None]) & ~same, M, 0.0)
    up = np.where((c[None, :] > c[:, None]) & ~same, M, 0.0)
    D = np.where(same, M, 0.0)
    if not fp32:
        return lambda r: np.linalg.solve(D + up, D @ np.linalg.solve(D + low, r))
    inv = np.linalg.inv(D).astype(np.float32).astype(np.float64)

    def apply(r):
        z = np.zeros_like(r)
        for g in range(colour.max() + 1):
            z = np.where(c == g, inv @ (r - low @ z), z)
        for g in range(colour.max(), -1, -1):
            z = np.where(c == g, z - inv @ (up @ z), z)
        return z

    return apply
