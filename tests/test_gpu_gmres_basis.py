"""GMRES over bases that fill, half fill and exceed the vectors one inner-product
launch takes (1, 8, 16, 24): after k steps of one cycle the residual is the
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
    V = [b / np.linalg.norm(b)]
    for _ in range(k - 1):
        w = M @ V[-1]
        for _ in range(2):
            w -= np.array(V).T @ (np.array(V) @ w)
        V.append(w / np.linalg.norm(w))
    MV = M @ np.array(V).T
    best = np.linalg.norm(b - MV @ np.linalg.lstsq(MV, b, rcond=None)[0])
    assert info.iterations == k
    assert abs(np.linalg.norm(b - M @ x) - best) <= 1e-10 * np.linalg.norm(b)
    assert abs(info.final_residual - best) <= 1e-10 * np.linalg.norm(b)
