"""The FP32 line solve's write-back, shared by the line's two warps, against the
one-warp form's: the same sums c + d whoever makes them, so the same bits.
Lines of 1 to 9 cells (whole and broken groups of 4), around 57 cells (one
round of both warps' 16 words a lane is 1024 words, 113.8 cells; of one warp's
512), and several rounds."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import sys
import numpy as np
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
import triblocksolve_b200 as tbs
from meshes import ragged_mesh
mesh = ragged_mesh([int(x) for x in sys.argv[3].split(",")], seed=2)
s = tbs.Solver(0)
s.set_mesh(mesh)
s.set_jacobian(tbs.Jacobian.generate(mesh, 4.0, 3))
s.factor(tbs.ALGO_MIXED)
s.set_inner_sweeps(4)
n, h = s.solve(1e-10, 60)
np.savez(sys.argv[2], n=n, h=h, U=s.solution(), dU=s.update())
s.close()
"""


@pytest.mark.parametrize("lens", ["1,2,3,4,5,6,7,8,9", "56,57,58,113,114,115", "300,1,227,228,400"])
def test_forms_agree(tmp_path, lens):
    got = []
    for form in (0, 1):
        out = str(tmp_path / f"form{form}.npz")
        env = dict(os.environ, TBS_THOMAS_WS=str(form))
        subprocess.run([sys.executable, "-c", SCRIPT, ROOT, out, lens], env=env, check=True, timeout=300)
        got.append(np.load(out))
    assert int(got[0]["n"]) >= 1
    for k in got[0].files:
        np.testing.assert_array_equal(got[0][k], got[1][k])
