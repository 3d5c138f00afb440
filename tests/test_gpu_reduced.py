"""BiCGSTAB with the multicolour sweep on the GPU against the same iterations
in numpy on the full system: two colours in natural and colour order, more
colours, block sizes, one to many warps of rows, a starting vector, and a
pattern without symmetry (coloured against its transpose too).

FP64 runs reduced, an FP32 matrix in the full form: the numpy run then uses the
matrix and the diagonal inverses rounded to FP32.  1e-10 as for the numpy
restatement."""
import numpy as np
import pytest

import colour_sgs as CS
import reduced_systems as RS
from conftest import rel_err

pytestmark = pytest.mark.gpu

CASES = [("box", 2, 5, "natural"), ("box", 13, 6, "natural"), ("box", 300, 6, "natural"), ("box", 301, 5, "colour"),
         ("box", 64, 1, "natural"), ("box", 95, 4, "colour"), ("graph", 40, 5, "colour"), ("graph", 211, 6, "colour"),
         ("graph", 97, 3, "colour"), ("graph", 33, 5, "natural"), ("one_sided", 90, 5, "natural"), ("one_sided", 91, 5, "colour")]


@pytest.mark.parametrize("kind,n,bs,order", CASES)
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("guess", [False, True])
def test_iterations_match_numpy(cb, kind, n, bs, order, mixed, guess):
    rp, cl, vals, colour = RS.system(kind, n, bs, order)
    rng = np.random.default_rng(3)
    b = rng.standard_normal(n * bs)
    x0 = rng.standard_normal(n * bs) if guess else None
    A = cb.Bsr(rp, cl, bs, cb.PREC_MIXED if mixed else cb.PREC_FP64)
    A.set_values(vals)
    A.sgs_setup(cb.SGS_COLOR, 1)
    its = 1 if n == 2 else 6
    x, info = A.bicgstab(b, x0=x0, rel_tol=1e-15, abs_tol=1e-300, max_it=its)
    M = RS.dense(rp, cl, vals.astype(np.float32).astype(np.float64) if mixed else vals, bs)
    full = CS.bicgstab(lambda u: M @ u, RS.colour_sgs(M, colour, bs, mixed), b, its, x0)
    assert info.iterations == its
    assert rel_err(x, full) < 1e-10
    r = np.linalg.norm(b - M @ full)
    if r > 1e-6 * np.linalg.norm(b):
        assert abs(info.final_residual - r) < 1e-6 * r


@pytest.mark.parametrize("kind,n,bs,order", [("box", 300, 6, "natural"), ("graph", 211, 5, "colour")])
@pytest.mark.parametrize("mixed", [False, True])
def test_preconditioner_is_that_of_the_handle(cb, kind, n, bs, order, mixed):
    """The solve runs on the operators that the handle's product and sweep
    apply.  1e-10 as above; an inverse of another precision moves the
    first iterate by 3e-9."""
    rp, cl, vals, _ = RS.system(kind, n, bs, order)
    b = np.random.default_rng(3).standard_normal(n * bs)
    A = cb.Bsr(rp, cl, bs, cb.PREC_MIXED if mixed else cb.PREC_FP64)
    A.set_values(vals)
    A.sgs_setup(cb.SGS_COLOR, 1)
    x, _ = A.bicgstab(b, rel_tol=1e-15, abs_tol=1e-300, max_it=1)
    assert rel_err(x, CS.bicgstab(A.spmv, A.sgs_apply, b, 1)) < 1e-10


@pytest.mark.parametrize("kind,n,bs,order", [("box", 120, 5, "natural"), ("box", 121, 6, "colour"),
                                             ("graph", 97, 3, "colour"), ("graph", 64, 4, "colour")])
@pytest.mark.parametrize("cond", [1.0, 3.0, 10.0, 1e4, 1e7, 1e10])
def test_converged_is_the_true_residual(cb, kind, n, bs, order, cond):
    """Diagonal blocks on both sides of the limit on their growth: a solve that
    reports convergence has reached its tolerance, and one run to the end reaches
    what the full iteration in numpy does.  1.5e-15 |b|: four times the 2.2e-16 to
    3.7e-16 that it ends at."""
    rp, cl, vals, colour = RS.system(kind, n, bs, order)
    vals = RS.mix_equations(rp, vals, bs, cond)
    M = RS.dense(rp, cl, vals, bs)
    b = M @ np.random.default_rng(3).standard_normal(n * bs)
    A = cb.Bsr(rp, cl, bs)
    A.set_values(vals)
    A.sgs_setup(cb.SGS_COLOR, 1)
    for tol in (1e-8, 1e-12):
        x, info = A.bicgstab(b, rel_tol=tol, max_it=100)
        assert info.status == cb.KRYLOV_CONVERGED
        assert np.linalg.norm(b - M @ x) <= 1.01 * tol * np.linalg.norm(b)
    x, _ = A.bicgstab(b, rel_tol=1e-30, abs_tol=1e-300, max_it=14)
    assert np.linalg.norm(b - M @ x) < 1.5e-15 * np.linalg.norm(b)


@pytest.mark.parametrize("order", ["natural", "colour"])
@pytest.mark.parametrize("cond", [1.0, 1e8])
def test_long_solves(cb, order, cond):
    """More than 32 iterations (the residual is formed from the vector every 32),
    and the same handle on new values: the form follows the matrix."""
    n, bs = 360, 5
    rp, cl, vals, _ = RS.system("box", n, bs, order)
    rows = np.repeat(np.arange(n), np.diff(rp))
    v = vals.reshape(-1, bs, bs)
    deg = np.diff(rp) - 1
    v[rows == cl] += (0.7 * deg - 0.8 * (deg + 1) - 0.95)[:, None, None] * np.eye(bs)  # 48 iterations and more
    A = cb.Bsr(rp, cl, bs)
    for c in (1.0, cond):
        w = RS.mix_equations(rp, vals, bs, c)
        M = RS.dense(rp, cl, w, bs)
        b = M @ np.random.default_rng(3).standard_normal(n * bs)
        A.set_values(w)
        A.sgs_setup(cb.SGS_COLOR, 1)
        x, info = A.bicgstab(b, rel_tol=1e-10, max_it=500)
        assert info.status == cb.KRYLOV_CONVERGED and info.iterations > 32
        assert np.linalg.norm(b - M @ x) <= 1.01e-10 * np.linalg.norm(b)


def test_set_up_at_the_memory_limit(cb):
    """Memory for the factors (115 MB, pivots, row lists) and 8 MB more, but not for
    the reduced solve's 21 MB of vectors: the solve takes the full form."""
    torch = pytest.importorskip("torch")
    n, bs = 400000, 6
    half = np.arange(n // 2)
    row_ptr = np.arange(0, 2 * n + 1, 2, dtype=np.int32)
    cols = np.concatenate([np.stack([half, half + n // 2], axis=1)] * 2).astype(np.int32).ravel()
    vals = np.tile(0.1 * np.ones((bs, bs)), (2 * n, 1, 1))
    vals[np.repeat(np.arange(n), 2) == cols] += 4.0 * np.eye(bs)
    b = np.random.default_rng(3).standard_normal(n * bs)

    def solve(A):
        A.sgs_setup(cb.SGS_COLOR, 1)
        return A.bicgstab(b, rel_tol=1e-10, max_it=20)

    first = cb.Bsr(row_ptr, cols, bs)  # loads the kernels
    first.set_values(vals)
    x, _ = solve(first)
    first.close()
    A = cb.Bsr(row_ptr, cols, bs)
    A.set_values(vals)
    room = n * (bs * bs * 8 + bs + 4 * 4) + (8 << 20)
    torch.cuda.synchronize()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
    A.sgs_setup(cb.SGS_COLOR, 1)
    del hold
    torch.cuda.empty_cache()
    y, info = A.bicgstab(b, rel_tol=1e-10, max_it=20)
    assert info.status == cb.KRYLOV_CONVERGED
    assert rel_err(y, x) < 1e-9
