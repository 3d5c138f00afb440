"""GMRES over bases that fill, half fill and exceed the vectors one inner-product
launch takes (1, 8, 16, 24; on vectors of more than 303,104 entries 1 and 8): after k steps of one cycle the residual is the
smallest one over x = V y, V an orthonormal basis of the Krylov space (built
here with two Gram-Schmidt passes).  That minimum is flat in V and y, so an
error of 1e-15 times the Hessenberg matrix's condition (below 1e4 here) in
either leaves it equal to 1e-10."""
import numpy as np
import pytest

import reduced_systems as RS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bs", [(1, 5), (60, 5), (47, 6)])
@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 16, 17, 24, 25, 33])
def test_smallest_residual(cb, n, bs, k):
    rp, cl, _, _ = RS.system("box", n, bs, "natural")
    rng = np.random.default_rng(k)
    vals = rng.standard_normal((len(cl), bs, bs))
    vals[np.repeat(np.arange(n), np.diff(rp)) == cl] += 4.0 * np.eye(bs)  # far from converged after 33 steps
    vals = vals.ravel()
    k = min(k, n * bs - 1)
    b = rng.standard_normal(n * bs)
    A = cb.Bsr(rp, cl, bs)
    A.set_values(vals)
    x, info = A.gmres(b, precond=cb.PC_NONE, rel_tol=1e-15, max_it=k, restart=k)
    M = RS.dense(rp, cl, vals, bs)
    _is_smallest(lambda u: M @ u, b, x, info, k)


def _is_smallest(product, b, x, info, k):
    V = [b / np.linalg.norm(b)]
    for _ in range(k - 1):
        w = product(V[-1])
        for _ in range(2):
            w -= np.array(V).T @ (np.array(V) @ w)
        V.append(w / np.linalg.norm(w))
    MV = np.stack([product(v) for v in V], axis=1)
    best = np.linalg.norm(b - MV @ np.linalg.lstsq(MV, b, rcond=None)[0])
    assert info.iterations == k
    assert abs(np.linalg.norm(b - product(x)) - best) <= 1e-10 * np.linalg.norm(b)
    assert abs(info.final_residual - best) <= 1e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("n", [303104, 303105])
@pytest.mark.parametrize("k", [9, 17])
def test_long_vectors(cb, n, k):
    """A tridiagonal matrix of 1 x 1 blocks on both sides of 303,104 rows."""
    rng = np.random.default_rng(k)
    rows = np.arange(n)
    cols = np.stack([rows - 1, rows, rows + 1], axis=1)
    have = (cols >= 0) & (cols < n)
    vals = rng.standard_normal((n, 3))
    vals[:, 1] += 4.0
    row_ptr = np.concatenate([[0], np.cumsum(have.sum(axis=1))]).astype(np.int32)
    A = cb.Bsr(row_ptr, cols[have].astype(np.int32), 1)
    A.set_values(vals[have])
    b = rng.standard_normal(n)
    x, info = A.gmres(b, precond=cb.PC_NONE, rel_tol=1e-15, max_it=k, restart=k)
    pad = lambda u: np.concatenate([[0.0], u, [0.0]])  # noqa: E731
    _is_smallest(lambda u: (vals * np.stack([pad(u)[:-2], u, pad(u)[2:]], axis=1)).sum(axis=1), b, x, info, k)
