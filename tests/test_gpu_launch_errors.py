"""Launches that the runtime refuses are reported, not left out."""
import numpy as np
import pytest

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("graphs", [1, 0])
def test_a_refused_launch_is_an_error(graphs):
    """65536 right-hand sides ask for one block more along y than a grid has:
    the runtime refuses the cycle's launches, and the solver says so when it
    records them (use_graphs = 1) or at its first solve."""
    from libemmi_mgfd_gb300 import gpu as G
    n, nrhs = (4, 4, 4), 65536
    x = [np.arange(v + 1, dtype=np.float32) * 100.0 for v in n]
    raw = np.ones((1, 4) + n[::-1], np.float32)

    def run():
        s = G.Solver(n, *x, raw, np.full(nrhs, 6.28, np.float32), op=np.zeros(nrhs, np.int32),
                     options=G.Options(precision=G.PREC_FP64, ncycle=1, use_graphs=graphs))
        if not graphs:
            s.solve(np.ones((nrhs, 3 * 125), np.complex128), want_h=False)
        s.close()
    with pytest.raises(RuntimeError, match="refused" if graphs else "invalid"):
        run()
    # the library's next solver is not touched by it
    s = G.Solver(n, *x, raw, np.full(2, 6.28, np.float32), op=np.zeros(2, np.int32),
                 options=G.Options(precision=G.PREC_FP64, ncycle=2, tol=0.0, use_graphs=graphs))
    assert [q["cycles"] for q in s.solve(np.ones((2, 3 * 125), np.complex128))[2]] == [2, 2]
    s.close()
