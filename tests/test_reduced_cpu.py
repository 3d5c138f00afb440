"""The reduced multicolour BiCGSTAB (oracle/colour_sgs.py) against BiCGSTAB
on the full system with the same preconditioner, on the CPU.  The two agree
in exact arithmetic; 1e-10 covers the rounding of ten iterations on these
well-conditioned systems (unit roundoff times the growth of the recurrences,
measured below 1e-13)."""
import numpy as np
import pytest

import colour_sgs as CS
import reduced_systems as RS
from conftest import rel_err


@pytest.mark.parametrize("kind,n,bs,order", [("box", 2, 5, "natural"), ("box", 60, 6, "natural"),
                                             ("box", 61, 1, "colour"), ("graph", 40, 5, "colour"),
                                             ("graph", 57, 3, "colour")])
@pytest.mark.parametrize("guess", [False, True])
def test_reduced_iterations_are_the_full_iterations(kind, n, bs, order, guess):
    rp, cl, vals, colour = RS.system(kind, n, bs, order)
    assert colour.max() >= (2 if kind == "graph" else 1)
    rng = np.random.default_rng(3)
    b = rng.standard_normal(n * bs)
    x0 = rng.standard_normal(n * bs) if guess else None
    M = RS.dense(rp, cl, vals, bs)
    its = 1 if n == 2 else 6
    full = CS.bicgstab(lambda x: M @ x, RS.colour_sgs(M, colour, bs), b, its, x0)
    assert rel_err(CS.bicgstab_reduced(rp, cl, vals, bs, colour, b, its, x0), full) < 1e-10
