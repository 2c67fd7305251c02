"""First APGD iterates against the oracle where a solve takes a launch form that the sizes of
test_gpu_iterates.py do not reach.  Same settings, same bounds, derived there: six iterations from a
step size far above 1/L, FP64 to 1e-12 and FP32 to 6e-4 (2-norm)."""
import numpy as np
import pytest

import py_oracle as orc
from scopi_b200 import FRICTION, ScopiBatch
from test_gpu_iterates import DT, bed, settings

pytestmark = pytest.mark.gpu


# more scenes than the SMs hold clusters: several CTAs of 128 (2D, 3D) or 256 (2D) threads on an SM,
# one CTA an SM; chains of the sums shared out over fewer threads than there are chains
@pytest.mark.parametrize("dim,sizes", [(2, [10 + k % 41 for k in range(700)]), (2, [150 + k % 151 for k in range(600)]),
                                       (2, [390 + k % 21 for k in range(148)]), (3, [4 + k % 30 for k in range(600)]),
                                       (3, [190 + k % 21 for k in range(152)])])
def test_many_friction_scenes(dim, sizes):
    scenes = [bed(dim, n, seed=20 + k) for k, n in enumerate(sizes)]
    kw = settings(dim, FRICTION)
    b = ScopiBatch(scenes, **kw)
    b.run(DT, 1)
    for k in range(0, len(scenes), len(scenes) // 16):
        pa = scenes[k]
        o = orc.OracleSolver(pa, **kw).run(DT, 1)
        st, so = b.scene_stats(k), o.stats()
        assert st["contacts"] == so["contacts"]
        assert (st["iterations"], st["backtracks"]) == (so["iterations"], so["backtracks"])
        g = b.scene(k)
        assert np.linalg.norm(g.v - o.pa.v) <= 1e-12 * np.linalg.norm(o.pa.v)
        assert np.linalg.norm(g.omega - o.pa.omega) <= 1e-12 * np.linalg.norm(o.pa.omega)
    b.close()
