"""What a solver stores to save recomputation, when device memory is short: the
line factors find the room they had without the other stored data, and three
eighths of the memory that was free stay free."""
import numpy as np
import pytest

from _cases import rel_err, unknown_mask

gpu = pytest.mark.gpu


def _solver(n, nop, prec, lf):
    from libemmi_mgfd_gb300 import gpu as G
    rng = np.random.default_rng(41)
    x = [np.concatenate([[0.0], np.cumsum(100.0 * 1.05 ** np.abs(np.arange(v) - v // 2))])
         .astype(np.float32) for v in n]
    raw = np.concatenate([10.0 ** rng.uniform(-1, 0.5, (nop, 3) + n[::-1]),
                          np.ones((nop, 1) + n[::-1])], 1).astype(np.float32)
    return G.Solver(n, *[np.stack([v] * nop) for v in x], raw, np.full(nop, 6.28, np.float32),
                    options=G.Options(precision=prec, ncycle=2, tol=0.0, autotune=0,
                                      line_factors=lf))


def _solve(s, n, nop):
    rng = np.random.default_rng(43)
    S = (n[0] + 1) * (n[1] + 1) * (n[2] + 1)
    unk = np.flatnonzero(unknown_mask(n).ravel())
    b = np.zeros((nop, 3 * S), np.complex128)
    for r in range(nop):
        b[r, rng.choice(unk, 5, replace=False)] = rng.standard_normal(5)
    return s.solve(b)[1]


class _Free:
    """Leaves about `target` bytes of device memory free."""

    def __init__(self, target):
        import torch
        from libemmi_mgfd_gb300 import gpu as G
        torch.cuda.synchronize()
        assert G.lib().emmi_trim_memory() == 0
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        assert free > target, "the device is smaller than this test expects"
        self.hold = torch.empty(free - int(target), dtype=torch.uint8, device="cuda")
        self.free = torch.cuda.mem_get_info()[0]

    def close(self):
        import torch
        self.hold = None
        torch.cuda.empty_cache()


# 62 halves once: level 0's factors are all there are (96 bytes a row in
# complex128, 28 in complex64), and the coarsest levels of 62 x 31 x 31 have
# large patch data
_N62 = (62, 62, 62)


def _factors62(nop, row):
    return nop * 3 * 61 * 61 * (5 * 62 - 4) * row


# room for the factors in half of what is free, for the patch data or the
# coefficients besides, and not for all three within five eighths (32 MB: the
# pool's granularity)
@gpu
def test_stored_data_leaves_three_eighths_of_the_memory_free():
    from libemmi_mgfd_gb300 import gpu as G
    n, nop = _N62, 8
    s = _solver(n, nop, G.PREC_FP64, 0)
    base = s.device_bytes
    s.close()
    s = _solver(n, nop, G.PREC_FP64, 1)
    stored, want = s.device_bytes - base, _solve(s, n, nop)
    s.close()
    room = _Free(base + 2.45 * _factors62(nop, 96))
    try:
        s = _solver(n, nop, G.PREC_FP64, 1)
        kept = s.device_bytes - base
        assert s.line_factor_format == 0
        assert kept <= 0.625 * (room.free - base) + (32 << 20) < stored, (kept, stored)
        got = _solve(s, n, nop)
        s.close()
    finally:
        room.close()
    for r in range(nop):
        assert rel_err(got[r], want[r]) < 1e-10


# the coefficients fit beside factors that take nearly their whole half
@gpu
def test_coefficients_fit_wherever_the_line_factors_do():
    from libemmi_mgfd_gb300 import gpu as G
    n, nop = (32, 32, 32), 8
    s = _solver(n, nop, G.PREC_FP64, 0)
    base = s.device_bytes
    s.close()
    s = _solver(n, nop, G.PREC_FP64, 1)
    stored = s.device_bytes - base
    s.close()
    room = _Free(base + 1.75 * stored)
    try:
        s = _solver(n, nop, G.PREC_FP64, 1)
        assert s.device_bytes - base == stored
        s.close()
    finally:
        room.close()


# the patch data must not push the line factors out of their half
@gpu
@pytest.mark.parametrize("prec, row", [(0, 96), (1, 28)])
def test_patch_data_does_not_displace_the_line_factors(prec, row):
    from libemmi_mgfd_gb300 import gpu as G
    assert (G.PREC_FP64, G.PREC_MIXED) == (0, 1)
    n, nop, lf = _N62, 4, 2 if prec else 1
    factors = _factors62(nop, row)
    s = _solver(n, nop, prec, 0)
    # the complex64 solver's FP64 coefficients of level 0 come after the factors
    base = s.device_bytes - (nop * 240 * 63 ** 3 if prec else 0)
    s.close()
    room = _Free(base + 2.15 * factors)
    try:
        s = _solver(n, nop, prec, lf)
        assert s.line_factor_format == lf - 1
        s.close()
    finally:
        room.close()
