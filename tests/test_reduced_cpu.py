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


@pytest.mark.parametrize("order", ["natural", "colour"])
@pytest.mark.parametrize("cond", [1.0, 5.0, 1e4, 1e8])
def test_growth_tells_the_reduced_residual(order, cond):
    """Blocks within the limit of 8 leave the true residual where the full
    iteration has it (4e-16 |b|; measured 2.2e-16 to 3.4e-16), blocks of condition
    1e4 and more do not."""
    n, bs = 120, 5
    rp, cl, vals, colour = RS.system("box", n, bs, order)
    vals = RS.mix_equations(rp, vals, bs, cond)
    M = RS.dense(rp, cl, vals, bs)
    b = M @ np.random.default_rng(3).standard_normal(n * bs)
    x = CS.bicgstab_reduced(rp, cl, vals, bs, colour, b, 14)
    within = CS.growth(RS.diagonal(rp, cl, vals, bs)).max() <= 8.0
    assert within == (cond < 1e3)
    assert (np.linalg.norm(b - M @ x) < 4e-16 * np.linalg.norm(b)) == within


def test_growth_ignores_units():
    """Rows and columns in other units: 1e-4 to 1e4 move it by less than the
    quarter that four steps leave; cond(D) passes 1e8."""
    rng = np.random.default_rng(0)
    d = 6.2 * np.eye(6) + 0.1 * rng.standard_normal((500, 6, 6))
    s, t = (10.0 ** rng.uniform(-4.0, 4.0, (500, 6)) for _ in range(2))
    scaled = s[:, :, None] * d * t[:, None, :]
    assert np.linalg.cond(scaled).max() > 1e8
    assert CS.growth(d).max() < 1.5 and CS.growth(scaled).max() < 1.25 * CS.growth(d).max() + 0.5
    stiff = d + 1e6 * rng.standard_normal((500, 6, 1)) * rng.standard_normal((500, 1, 6))
    assert CS.growth(s[:, :, None] * stiff * t[:, None, :]).min() > 1e4
