"""Dispatches at the edges of their rules: transfers between levels of which
only some axes coarsen, and the row residuals of a general permeability on
grids launched dependent on the kernel before and on larger ones."""
import numpy as np
import pytest

import oracle as O
from _cases import random_level, rel_err, unknown_mask

gpu = pytest.mark.gpu


# the last steps of a hierarchy: one axis, or none of two, left to coarsen
@gpu
@pytest.mark.parametrize("n, sc", [((8, 6, 10), (1, 1, 2)), ((6, 8, 10), (1, 2, 1)),
                                   ((10, 6, 8), (2, 1, 1)), ((40, 36, 28), (2, 1, 2))])
@pytest.mark.parametrize("prec", [0, 1])
def test_transfers_of_partial_coarsening_match_oracle(n, sc, prec):
    """Restriction and prolongation against the oracle's: sums of up to 18
    products, so 1e-14 of the norm in FP64 and 2e-6 in complex64."""
    from libemmi_mgfd_gb300 import gpu as G
    n, x, raw, cells, om, u, f = random_level(n, seed=11)
    nc = tuple(a // b for a, b in zip(n, sc))
    xc = [np.asarray(x[e])[::sc[e]].copy() for e in range(3)]
    rng = np.random.default_rng(12)
    sc_n = 3 * (nc[0] + 1) * (nc[1] + 1) * (nc[2] + 1)
    uc = rng.standard_normal(sc_n) + 1j * rng.standard_normal(sc_n)
    tol = 1e-14 if prec == G.PREC_FP64 else 2e-6
    fc_ref = O.restrict(n, x, nc, xc, sc, f)
    fc = G.level_transfer(n, x, sc, f, np.zeros(sc_n, np.complex128), 0, prec)
    assert np.linalg.norm(fc - fc_ref) <= tol * np.linalg.norm(fc_ref)
    up_ref = O.prolong(n, x, nc, xc, sc, uc, u)
    up = G.level_transfer(n, x, sc, uc, u, 1, prec)
    assert np.linalg.norm(up - up_ref) <= tol * np.linalg.norm(up_ref)


# 48^3: level 0 of 3 right-hand sides in 324 blocks a colour, of 25 in 2700
@gpu
@pytest.mark.parametrize("n, nrhs", [((48, 48, 48), 3), ((48, 48, 48), 25)])
def test_rows_of_a_general_permeability_match_the_sweeps_that_factor(n, nrhs):
    """Stored fp32 factors against factoring in every sweep, mu_r != 1: the
    same line systems, two cycles, float rounding: 1e-5 of the field's norm
    in H."""
    from libemmi_mgfd_gb300 import gpu as G
    rng = np.random.default_rng(19)
    x = [np.concatenate([[0.0], np.cumsum(100.0 * 1.05 ** np.abs(np.arange(v) - v // 2))])
         .astype(np.float32) for v in n]
    raw = np.concatenate([10.0 ** rng.uniform(-1, 0.5, (3,) + n[::-1]),
                          1.0 / rng.uniform(1.0, 1.5, (1,) + n[::-1])]).astype(np.float32)
    S = (n[0] + 1) * (n[1] + 1) * (n[2] + 1)
    unk = np.flatnonzero(unknown_mask(n).ravel())
    b = np.zeros((nrhs, 3 * S), np.complex128)
    for r in range(nrhs):
        b[r, rng.choice(unk, 5, replace=False)] = rng.standard_normal(5)
    out = []
    for lf in (1, 0):
        s = G.Solver(n, *x, raw[None], np.full(nrhs, 6.28, np.float32), op=np.zeros(nrhs, np.int32),
                     options=G.Options(precision=G.PREC_MIXED, ncycle=2, tol=0.0, autotune=0,
                                       line_factors=lf))
        out.append(s.solve(b)[1])
        s.close()
    for r in range(nrhs):
        assert rel_err(out[0][r], out[1][r]) < 1e-5, r
