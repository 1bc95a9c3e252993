"""The learned correction's input and convolutions at the edges of their
split: chunks of planes of every length with remainders, tiles of 128 slots
that end in a plane, and the permeability read from the cells."""
import numpy as np
import pytest

import oracle as O
from learned_oracle import Net, TAPS, CH, unknown_masks
from _cases import weighted_cells

gpu = pytest.mark.gpu


# few columns of slots: chunks of two planes (n3 = 4), of three and a last one
# of one (7); many: of four with a remainder of none, one and two (16, 13, 14).
# 16 x 8 x 6: 153 slots a plane, a second tile of 25
@gpu
@pytest.mark.parametrize("n, nrhs, mur", [((8, 8, 4), 1, 1.0), ((16, 8, 6), 3, 1.0),
                                          ((16, 8, 7), 2, 1.7), ((64, 64, 16), 5, 1.0),
                                          ((64, 64, 13), 6, 1.0), ((48, 64, 14), 8, 1.7)])
def test_correction_over_chunk_edges_matches_oracle(n, nrhs, mur):
    """u += c against the oracle's network, per right-hand side.  Both round
    the input and the hidden layer to bf16 (2^-9); values on either side of a
    rounding differ by a whole step, a few per cent of them: 2e-3 of the norm."""
    import torch
    from libemmi_mgfd_gb300 import gpu as G
    rng = np.random.default_rng(31)
    x = [np.concatenate([[0.0], np.cumsum(100.0 * 1.1 ** np.abs(np.arange(v) - v // 2).clip(0, 9))])
         .astype(np.float32) for v in n]
    raw = np.concatenate([10.0 ** rng.uniform(-1, 0.5, (3,) + n[::-1]),
                          np.full((1,) + n[::-1], 1.0 / mur)]).astype(np.float32)
    oms = np.where(np.arange(nrhs) % 3 == 2, 3.0, 6.0).astype(np.float32)
    s = G.Solver(n, *x, raw[None], oms, op=np.zeros(nrhs, np.int32),
                 options=G.Options(precision=G.PREC_MIXED, sigma_floor=1e-30, autotune=0))
    W = (0.05 * rng.standard_normal((2, TAPS, CH, CH))).astype(np.float32).reshape(-1)
    s.set_learned(W)
    unk = unknown_masks(n).reshape(-1)
    u, f = np.zeros((2, nrhs, unk.size), np.complex64)
    for v in (u, f):
        v[:, unk] = rng.standard_normal((nrhs, unk.sum())) + 1j * rng.standard_normal((nrhs, unk.sum()))
    du, df = torch.tensor(u, device="cuda"), torch.tensor(f, device="cuda")
    s.learned_apply(df, du)
    got = du.cpu().numpy().astype(np.complex128) - u.astype(np.complex128)
    s.close()
    xs = [v.astype(np.float64) for v in x]
    c = weighted_cells(n, xs, raw)
    for r in range(nrhs):
        lev = O.Level(n, xs, c[:3], c[3], float(oms[r]))
        net = Net(lev, bf16_round=True)
        want, _ = net.forward(W.astype(np.float64),
                              f[r].astype(np.complex128) - lev.apply(u[r].astype(np.complex128)))
        err = np.linalg.norm(got[r] - want) / np.linalg.norm(want)
        assert err < 2e-3, (r, err)
        assert np.all(got[r][~unk] == 0)
