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
