"""The tuning file across versions of the kernels."""
import json
import os
import subprocess
import sys

import pytest

from test_gpu_solver import _TUNE_CHILD

gpu = pytest.mark.gpu


@gpu
def test_shapes_of_other_kernels_are_timed_anew(tmp_path):
    """A file written before its shapes' numbers meant the present kernels'
    (no version, or another one) is not taken: the set-up times the shapes and
    rewrites the file, which the next process reads."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    path = tmp_path / "tune.json"
    old = [dict(grid=[12, 12, 12], chunk=2, nrhs=2, fmt=1, dir=d, subst=2, rhs_threads=128)
           for d in range(3)]

    def child():
        r = subprocess.run([sys.executable, "-c", _TUNE_CHILD, root], capture_output=True, text=True,
                           env=dict(os.environ, EMMI_TUNE_FILE=str(path)), timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout.strip().splitlines()[-1])
    for doc in (dict(sweep_shapes=old), dict(version=1, sweep_shapes=old)):
        path.write_text(json.dumps(doc))
        shapes, tuned = child()
        assert tuned
        assert json.loads(path.read_text())["version"] == 2
        assert child() == [shapes, False]
