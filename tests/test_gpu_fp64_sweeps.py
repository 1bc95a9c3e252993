"""complex128 sweeps from stored coefficients and factors, distributed over
lanes where the lines are few, against the sweeps that factor as they go: the
same operations in the same order."""
import numpy as np
import pytest

from _cases import unknown_mask
from libemmi_mgfd_gb300 import gpu as G

gpu = pytest.mark.gpu


def _solve(n, nrhs, prec, **o):
    rng = np.random.default_rng(23)
    x = [np.concatenate([[0.0], np.cumsum(100.0 * 1.1 ** np.abs(np.arange(v) - v // 2))])
         .astype(np.float32) for v in n]
    raw = np.concatenate([10.0 ** rng.uniform(-1, 0.5, (3,) + n[::-1]),
                          np.ones((1,) + n[::-1])]).astype(np.float32)
    S = (n[0] + 1) * (n[1] + 1) * (n[2] + 1)
    unk = np.flatnonzero(unknown_mask(n).ravel())
    b = np.zeros((nrhs, 3 * S), np.complex128)
    for r in range(nrhs):
        b[r, rng.choice(unk, 5, replace=False)] = rng.standard_normal(5)
    s = G.Solver(n, *x, raw[None], np.full(nrhs, 6.28, np.float32), op=np.zeros(nrhs, np.int32),
                 options=G.Options(precision=prec, ncycle=3, tol=0.0, autotune=0, **o))
    out, h, _ = s.solve(b)
    s.close()
    return out, h


# the lanes' lines: odd counts (8 x 8 lines: 9 and 16), a last pair of one;
# (28, 36, 20): a coarsest level that does not fit a block; 130 RHS: one lane a
# line; v1 = 2: both colour orders in the coarsest level's one launch
@gpu
@pytest.mark.parametrize("n, nrhs, more", [((8, 8, 8), 1, {}), ((16, 12, 20), 3, {"v1": 2}),
                                           ((72, 36, 40), 1, {}), ((16, 16, 16), 130, {}),
                                           ((12, 8, 16), 2, {"cycleopt": 3})])
def test_fp64_stored_sweeps_equal_the_factoring_ones(n, nrhs, more):
    """Bit for bit (signed zeros apart) where the stored line factors are also
    the factoring solve's: the lines' LDL^T is the same code in both, so what
    may differ is contraction of its elimination alone; 1e-12 of the largest
    value in H over three cycles."""
    a = _solve(n, nrhs, G.PREC_FP64, **more)[1]
    b = _solve(n, nrhs, G.PREC_FP64, line_factors=0, **more)[1]
    assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


@gpu
@pytest.mark.parametrize("n, nrhs, more", [((8, 8, 8), 1, {}), ((16, 12, 20), 3, {"v1": 2}),
                                           ((72, 36, 40), 2, {}), ((12, 8, 16), 2, {"cycleopt": 3})])
def test_complex64_stored_patches_equal_the_factoring_ones(n, nrhs, more):
    """The coarsest level's patches from stored factors (line_factors = 1)
    against patches factored in every sweep (line_factors = 0) in complex64:
    float rounding over three cycles, 1e-5 of the largest value in H."""
    a = _solve(n, nrhs, G.PREC_MIXED, line_factors=1, **more)[1]
    b = _solve(n, nrhs, G.PREC_MIXED, line_factors=0, **more)[1]
    assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()


# 16^3: a launch of 160 right-hand sides has 10240 lines, past the 7680 up to
# which a line takes 12 lanes; (20, 12, 16): the x lines just reach them, the y
# and z lines pass them
@gpu
@pytest.mark.parametrize("n", [(16, 16, 16), (20, 12, 16)])
def test_fp64_lanes_give_the_bits_of_a_thread_a_line(n):
    """One right-hand side alone (12 lanes a line) and 160 copies of it (a
    thread a line), stored factors both: equal E and H."""
    rng = np.random.default_rng(53)
    x = [np.concatenate([[0.0], np.cumsum(100.0 * 1.1 ** np.abs(np.arange(v) - v // 2))])
         .astype(np.float32) for v in n]
    raw = np.concatenate([10.0 ** rng.uniform(-1, 0.5, (3,) + n[::-1]),
                          np.ones((1,) + n[::-1])]).astype(np.float32)
    b = np.zeros((1, 3 * (n[0] + 1) * (n[1] + 1) * (n[2] + 1)), np.complex128)
    b[0, rng.choice(np.flatnonzero(unknown_mask(n).ravel()), 5, replace=False)] = 1.0
    out = []
    for k in (1, 160):
        s = G.Solver(n, *x, raw[None], np.full(k, 6.28, np.float32), op=np.zeros(k, np.int32),
                     options=G.Options(precision=G.PREC_FP64, ncycle=3, tol=0.0))
        out.append(s.solve(np.repeat(b, k, 0))[:2])
        s.close()
    for one, many in zip(*out):
        assert np.abs(one).max() > 0
        for r in (0, 77, 159):
            assert np.array_equal(one[0], many[r])
