"""The complex64 line relaxation's kernels at the sizes their dispatch splits
at, against the library's general path for the same lines."""
import numpy as np
import pytest

from _cases import rel_err, unknown_mask
from libemmi_mgfd_gb300 import gpu as G

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("n, nrhs", [((4, 8, 16), 1),      # one group an end, tiles of 8
                                     ((20, 36, 12), 2),    # ragged tiles
                                     ((48, 48, 16), 25),   # tiles of 32: rings reused and not
                                     ((12, 40, 44), 70)])  # partial last tiles of 32
@pytest.mark.parametrize("lf", [1, 2])
def test_line_ends_match_the_sweeps_that_factor(n, nrhs, lf):
    """The substitution with stored two-ended factors (complex64) over the
    tile widths, ring lengths and remainders it is dispatched to, against the
    sweep that factors as it goes: the one-ended one (line_factors = 0) for
    fp32 factors, the one-launch sweep with the same fp16 multipliers for
    fp16.  Same line systems, so two cycles differ by float rounding: 1e-5 of
    the field's largest value in H (the curl-free part of E is not fixed by
    complex64)."""
    rng = np.random.default_rng(17)
    x = [np.concatenate([[0.0], np.cumsum(100.0 * 1.1 ** np.abs(np.arange(v) - v // 2))])
         .astype(np.float32) for v in n]
    raw = np.concatenate([10.0 ** rng.uniform(-1, 0.5, (3,) + n[::-1]),
                          np.ones((1,) + n[::-1])]).astype(np.float32)
    S = (n[0] + 1) * (n[1] + 1) * (n[2] + 1)
    unk = unknown_mask(n).ravel()
    b = np.zeros((nrhs, 3 * S), np.complex128)
    for r in range(nrhs):
        b[r, rng.choice(np.flatnonzero(unk), 5, replace=False)] = rng.standard_normal(5)
    out = []
    for o in (dict(line_factors=lf), dict(line_factors=0) if lf == 1 else
              dict(line_factors=2, line_sweep=1)):
        s = G.Solver(n, *x, raw[None], np.full(nrhs, 6.28, np.float32), op=np.zeros(nrhs, np.int32),
                     options=G.Options(precision=G.PREC_MIXED, ncycle=2, tol=0.0, autotune=0, **o))
        out.append(s.solve(b)[1])
        if len(out) == 1:
            assert s.line_factor_format == {1: 0, 2: 1}[lf]
        s.close()
    for r in range(nrhs):
        assert rel_err(out[0][r], out[1][r]) < 1e-5, r


@gpu
@pytest.mark.parametrize("lf", [1, 2])
def test_factors_of_many_groups_match_those_of_few(lf):
    """Line factors of 1216 groups (frequencies) of a 16^3 operator, whose
    level-0 lines are factored a line a thread, against solvers of one group,
    an end a thread.  The factors are the same; the sweeps differ in tiles and
    the residual's kernel, so two cycles differ by float rounding: 1e-5 of the
    field's norm in H."""
    n, nrhs = (16, 16, 16), 1216
    rng = np.random.default_rng(29)
    x = [np.concatenate([[0.0], np.cumsum(100.0 * 1.1 ** np.abs(np.arange(v) - v // 2))])
         .astype(np.float32) for v in n]
    raw = np.concatenate([10.0 ** rng.uniform(-1, 0.5, (3,) + n[::-1]),
                          np.ones((1,) + n[::-1])]).astype(np.float32)
    om = np.linspace(3.0, 12.0, nrhs).astype(np.float32)
    unk = np.flatnonzero(unknown_mask(n).ravel())
    b = np.zeros((nrhs, 3 * 17 ** 3), np.complex128)
    for r in range(nrhs):
        b[r, rng.choice(unk, 5, replace=False)] = rng.standard_normal(5)

    def run(rows):
        s = G.Solver(n, *x, raw[None], om[rows], op=np.zeros(len(rows), np.int32),
                     options=G.Options(precision=G.PREC_MIXED, ncycle=2, tol=0.0, autotune=0,
                                       sigma_floor=1e-3, line_factors=lf))
        h = s.solve(b[rows])[1]
        assert s.line_factor_format == {1: 0, 2: 1}[lf]
        s.close()
        return h
    many = run(np.arange(nrhs))
    for r in (0, 617, nrhs - 1):
        assert rel_err(many[r], run(np.array([r]))[0]) < 1e-5, r


@gpu
def test_shapes_of_wide_tiles_never_change_the_result():
    """Every forced sweep shape on a batch whose level 0 works in tiles of 32
    lines, with rings shorter than the x and y lines (23 groups an end) and
    longer than the z lines (7): the defaults' iterates bit for bit."""
    n, nrhs = (48, 48, 16), 25
    rng = np.random.default_rng(47)
    x = [np.concatenate([[0.0], np.cumsum(100.0 * 1.1 ** np.abs(np.arange(v) - v // 2))])
         .astype(np.float32) for v in n]
    raw = np.concatenate([10.0 ** rng.uniform(-1, 0.5, (3,) + n[::-1]),
                          np.ones((1,) + n[::-1])]).astype(np.float32)
    S = (n[0] + 1) * (n[1] + 1) * (n[2] + 1)
    unk = np.flatnonzero(unknown_mask(n).ravel())
    b = np.zeros((nrhs, 3 * S), np.complex128)
    for r in range(nrhs):
        b[r, rng.choice(unk, 5, replace=False)] = rng.standard_normal(5)

    def run(autotune):
        s = G.Solver(n, *x, raw[None], np.full(nrhs, 6.28, np.float32), op=np.zeros(nrhs, np.int32),
                     options=G.Options(precision=G.PREC_MIXED, ncycle=3, tol=0.0,
                                       autotune=autotune))
        e, h, _ = s.solve(b)
        s.close()
        return e, h
    e0, h0 = run(0)
    for k in range(1, 11):
        e, h = run(-k)
        assert np.array_equal(e, e0) and np.array_equal(h, h0), k
