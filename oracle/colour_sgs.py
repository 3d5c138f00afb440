"""Numpy restatement of the multicolour SGS apply that the GPU runs on a
colour-ordered matrix (test infrastructure only; the checker of the
algorithms in distributed-cfd-solver_b200/csrc/kernels_linalg.cu and
csrc/kernels_reduced.cu).

On a matrix whose rows are ordered colour by colour (a greedy colouring in
row order, colours ascending), the sweep is:
  forward, colours ascending:  y_i = D_i^-1 (r_i - sum_{j<i} A_ij y_j)
  backward, colours descending (the last colour already final):
      t_i = sum_{j>i} A_ij z_j,  z_i = y_i - D_i^-1 t_i
with D_i^-1 the explicit inverse of the diagonal block; the product of a
colour-0 row (swept last) is (A z)_i = t_i + A_ii z_i.
The reference's sequential SGS (bsr_sgs_sweep, natural row order, one
symmetric sweep from z = 0) is the same preconditioner on such a matrix:
rows of one colour do not couple.
"""
from __future__ import annotations

import numpy as np


def greedy_colours(row_ptr, cols):
    """Smallest colour not used by an already coloured neighbour, rows in
    order (BsrSystem::build_ordering, colour branch)."""
    n = len(row_ptr) - 1
    colour = np.full(n, -1, dtype=np.int64)
    for i in range(n):
        used = {int(colour[j]) for j in cols[row_ptr[i]:row_ptr[i + 1]] if j != i and colour[j] >= 0}
        c = 0
        while c in used:
            c += 1
        colour[i] = c
    return colour


def colour_order(row_ptr, cols, vals, bs):
    """The matrix with rows and columns permuted colour by colour (stable
    within a colour), columns sorted per row; returns (row_ptr, cols, vals,
    colour offsets, permutation new -> old)."""
    n = len(row_ptr) - 1
    colour = greedy_colours(row_ptr, cols)
    order = np.argsort(colour, kind="stable")
    new_of = np.empty(n, dtype=np.int64)
    new_of[order] = np.arange(n)
    blocks = np.asarray(vals).reshape(-1, bs, bs)
    rp = np.zeros(n + 1, dtype=np.int32)
    cl, vb = [], []
    for r, i in enumerate(order):
        ks = np.arange(row_ptr[i], row_ptr[i + 1])
        cn = new_of[cols[ks]]
        srt = np.argsort(cn)
        cl.extend(cn[srt])
        vb.append(blocks[ks[srt]])
        rp[r + 1] = len(cl)
    ncol = int(colour.max()) + 1
    off = np.zeros(ncol + 1, dtype=np.int64)
    for c in range(ncol):
        off[c + 1] = off[c] + int((colour == c).sum())
    return rp, np.asarray(cl, dtype=np.int32), np.concatenate(vb).ravel(), off, order


def split_sweep_with_product(row_ptr, cols, vals, bs, off, r):
    """z = M^-1 r by the split first sweep with explicit diagonal inverses,
    and A z with the colour-0 rows' product taken from the backward pass."""
    n = len(row_ptr) - 1
    A = np.asarray(vals, dtype=np.float64).reshape(-1, bs, bs)
    rr = np.asarray(r, dtype=np.float64).reshape(n, bs)
    diag = np.array([row_ptr[i] + int(np.searchsorted(cols[row_ptr[i]:row_ptr[i + 1]], i)) for i in range(n)])
    dinv = np.linalg.inv(A[diag])
    z = np.zeros((n, bs))
    ncol = len(off) - 1
    for c in range(ncol):                       # forward: lower blocks only
        for i in range(off[c], off[c + 1]):
            s = rr[i].copy()
            for k in range(row_ptr[i], diag[i]):
                s -= A[k] @ z[cols[k]]
            z[i] = dinv[i] @ s
    t = np.zeros((n, bs))
    for c in range(ncol - 2, -1, -1):           # backward: upper blocks only
        for i in range(off[c], off[c + 1]):
            for k in range(diag[i] + 1, row_ptr[i + 1]):
                t[i] += A[k] @ z[cols[k]]
            z[i] = z[i] - dinv[i] @ t[i]
    az = np.zeros((n, bs))
    for i in range(n):
        if i < off[1]:                          # colour 0: every off-diagonal block is in t
            az[i] = t[i] + A[diag[i]] @ z[i]
        else:
            for k in range(row_ptr[i], row_ptr[i + 1]):
                az[i] += A[k] @ z[cols[k]]
    return z.ravel(), az.ravel()


def bicgstab(product, precond, b, its, x0=None):
    """`its` iterations of BiCGSTAB (src/linalg/bicgstab.cpp:42-201) with
    right preconditioning, in numpy."""
    x = np.zeros_like(b) if x0 is None else x0.copy()
    r = b - product(x)
    r0, p, rho = r.copy(), r.copy(), r @ r
    for _ in range(its):
        ph = precond(p)
        v = product(ph)
        alpha = rho / (r0 @ v)
        s = r - alpha * v
        sh = precond(s)
        t = product(sh)
        omega = (t @ s) / (t @ t)
        x = x + alpha * ph + omega * sh
        r = s - omega * t
        rho_new = r0 @ r
        beta = rho_new / rho * alpha / omega
        p = r + beta * (p - omega * v)
        rho = rho_new
    return x


def bicgstab_reduced(row_ptr, cols, vals, bs, colour, b, its, x0=None):
    """The same iterations on the rows outside colour 0: the product is
    A z = p - L e with e = D^-1 U z, the colour-0 parts of the vectors are
    multiples of the initial residual's, and x on colour 0 follows at the
    end.  `colour` gives each row's colour; rows of a colour do not couple."""
    n = len(row_ptr) - 1
    A = np.asarray(vals, dtype=np.float64).reshape(-1, bs, bs)
    rows = np.repeat(np.arange(n), np.diff(row_ptr))
    cols = np.asarray(cols)
    dinv = np.linalg.inv(A[rows == cols])
    kr, kc = colour[rows], colour[cols]
    zero, rest = colour == 0, colour > 0

    def part(keep, x):
        y = np.zeros((n, bs))
        np.add.at(y, rows[keep], np.einsum("kij,kj->ki", A[keep], x[cols[keep]]))
        return y

    upper, lower, mid = kc > kr, kc < kr, (kc < kr) & (kc > 0)
    D = lambda x: np.einsum("kij,kj->ki", dinv, x)  # noqa: E731
    bb = b.reshape(n, bs)
    x = np.zeros((n, bs)) if x0 is None else x0.reshape(n, bs).copy()
    r0 = bb - part(np.ones(len(cols), dtype=bool), x)
    eta = np.where(zero[:, None], D(r0), 0.0)
    w = part(kc == 0, eta)
    q0 = (r0[zero] ** 2).sum()
    r, p = np.where(rest[:, None], r0, 0.0), np.where(rest[:, None], r0, 0.0)
    rr = r.copy()
    cr = cp = 1.0

    def apply(src, c):
        z, e = np.zeros((n, bs)), np.zeros((n, bs))
        for g in range(1, colour.max() + 1):
            z = np.where((colour == g)[:, None], D(src - c * w - part(mid, z)), z)
        for g in range(colour.max() - 1, -1, -1):
            t = D(part(upper, z))
            e = np.where((colour == g)[:, None], t, e)
            if g:
                z = np.where((colour == g)[:, None], z - t, z)
        return z, np.where(rest[:, None], src - part(lower, e), 0.0)

    rho = (r0 ** 2).sum()
    for _ in range(its):
        zp, v = apply(p, cp)
        alpha = rho / ((rr * v).sum() + cp * q0)
        s = r - alpha * v
        cs = cr - alpha * cp
        zs, t = apply(s, cs)
        omega = ((t * s).sum() + cs * cs * q0) / ((t * t).sum() + cs * cs * q0)
        x = np.where(rest[:, None], x + alpha * zp + omega * zs, x)
        rho_new = (rr * s).sum() + cs * q0 - omega * ((rr * t).sum() + cs * q0)
        r = s - omega * t
        cr = cs - omega * cs
        beta = rho_new / rho * alpha / omega
        p = r + beta * (p - omega * v)
        cp = cr + beta * (cp - omega * cp)
        rho = rho_new
    x0_rows = D(bb - cr * r0 - part(upper, np.where(rest[:, None], x, 0.0)))
    return np.where(zero[:, None], x0_rows, x).ravel()


def growth(blocks):
    """How much more rounding D (D^-1 s) takes than the product with D itself:
    max_i (G x)_i / x_i of G = |D| |D^-1|, x after three steps x <- G x from ones
    (an upper bound of the spectral radius of G, near it whatever the scales of
    the block's rows and columns); per block."""
    g = np.abs(blocks) @ np.abs(np.linalg.inv(blocks))
    x = np.ones(blocks.shape[:2])
    for _ in range(4):
        x, old = np.einsum("kij,kj->ki", g, x), x
    return (x / old).max(axis=1)
