"""The staged residual over the depths of its tiles."""
import numpy as np
import pytest

from _cases import rel_err, unknown_mask

gpu = pytest.mark.gpu


# 64^3 in five tiles of rows: two right-hand sides take tiles of 4 planes, four
# of 8, eight of 16 (a last tile of one plane each), so that the ring of four
# planes is refilled once and several times; (40, 44, 60) x 6: 16 planes a tile
# and 13 in the last.  mu_r != 1 stages the permeability's plane besides.
@gpu
@pytest.mark.parametrize("n, nrhs, mur", [((64, 64, 64), 2, 1.0), ((64, 64, 64), 4, 1.0),
                                          ((64, 64, 64), 8, 1.0), ((40, 44, 60), 6, 1.0),
                                          ((64, 64, 64), 4, 1.6), ((64, 64, 64), 8, 1.6)])
def test_staged_tiles_of_every_depth_match_the_plain_residual(n, nrhs, mur):
    """The same edge equations in another order of summation: two cycles differ
    by float rounding, 1e-5 of the field's norm in H; a plane of another tile
    or an older one in the ring would show at its size."""
    from libemmi_mgfd_gb300 import gpu as G
    rng = np.random.default_rng(37)
    x = [np.concatenate([[0.0], np.cumsum(100.0 * 1.05 ** np.abs(np.arange(v) - v // 2))])
         .astype(np.float32) for v in n]
    raw = np.concatenate([10.0 ** rng.uniform(-1, 0.5, (3,) + n[::-1]),
                          np.full((1,) + n[::-1], 1.0 / mur)]).astype(np.float32)
    S = (n[0] + 1) * (n[1] + 1) * (n[2] + 1)
    unk = np.flatnonzero(unknown_mask(n).ravel())
    b = np.zeros((nrhs, 3 * S), np.complex128)
    for r in range(nrhs):
        b[r, rng.choice(unk, 200, replace=False)] = rng.standard_normal(200)
    out = []
    for staged in (1, 0):
        s = G.Solver(n, *x, raw[None], np.full(nrhs, 6.28, np.float32), op=np.zeros(nrhs, np.int32),
                     options=G.Options(precision=G.PREC_MIXED, ncycle=2, tol=0.0, autotune=0,
                                       staged=staged))
        assert s.staged == bool(staged)
        out.append(s.solve(b)[1])
        s.close()
    for r in range(nrhs):
        assert rel_err(out[0][r], out[1][r]) < 1e-5, r
