"""The sweeps and products on the sliced copy of a matrix larger than L2 (kept
with the device loop) against the row-by-row kernels (host loop): every sum is
formed in the same order, so the iterates are equal to the bit.  Two colours
and more, rows of unequal length, both block sizes and matrix precisions, one
and two sweeps, and last slices and windows that are not full."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {  # odd sizes whose matrix is a little over twice L2
    "plate_fp64": ("plate", (93, 67, 43), False),
    "sa_mixed": ("sa_plate", (107, 73, 47), True),
    "bump_mixed": ("bump", (117, 39, 29), True),
}


def _slices(s):
    """Whether a step keeps a sliced copy: its set-up profiles the factorisation and
    the copies, else the factorisation alone."""
    s.profile(True)
    s.newton_step(5.0)
    launches = s.profile_read()["lu"]["launches"]
    s.profile(False)
    assert launches in (1, 2)
    return launches == 2


def _steps(cb, case, mesh, loop, state):
    case.cfg.krylov_loop = loop
    out = []
    with cb.Solver(mesh, case.cfg, case.bcs) as s:
        s.set_state(state)
        assert _slices(s) == (loop == cb.KRYLOV_DEVICE_LOOP)
        s.set_state(state)
        for _ in range(2):
            r = s.newton_step(5.0)
            out.append((r.krylov_iterations, r.krylov_status, r.krylov_initial, r.krylov_final))
        return out, s.get(cb.FIELD_U), s.get(cb.FIELD_DU)


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("sweeps", [1, 2])
def test_slices_are_the_rows(cb, name, sweeps):
    make, size, mixed = CASES[name]
    case = getattr(cb.cases, make)(mixed=mixed)
    case.spec.nx, case.spec.ny, case.spec.nz = size
    case.cfg.sgs_sweeps = sweeps
    case.cfg.pre_freeze = cb.PREFREEZE_CONFIGURED  # FP32 from the first step on
    case.cfg.lin_rel_tol, case.cfg.lin_abs_tol, case.cfg.lin_max_iterations = 1e-30, 1e-300, 6
    mesh = cb.HostMesh(case.spec)
    state = cb.cases.perturbed_state(case, mesh.n_cells)
    a, b = (_steps(cb, case, mesh, loop, state) for loop in (cb.KRYLOV_DEVICE_LOOP, cb.KRYLOV_HOST_LOOP))
    assert a[0] == b[0]
    assert np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])


def test_slices_come_when_memory_does(cb):
    """Less memory than eight times the copy at the first steps: the rows are used,
    and the slices once it is free again."""
    torch = pytest.importorskip("torch")
    make, size, mixed = CASES["plate_fp64"]
    case = getattr(cb.cases, make)(mixed=mixed)
    case.spec.nx, case.spec.ny, case.spec.nz = size
    case.cfg.lin_max_iterations = 2
    mesh = cb.HostMesh(case.spec)
    with cb.Solver(mesh, case.cfg, case.bcs) as s:
        s.set_state(cb.cases.perturbed_state(case, mesh.n_cells))
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (1500 << 20), dtype=torch.uint8, device="cuda")
        assert not _slices(s)
        del hold
        torch.cuda.empty_cache()
        for _ in range(32):
            s.newton_step(5.0)
        assert _slices(s)
