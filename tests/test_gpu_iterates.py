"""The first APGD iterates of the persistent kernels against the oracle, at the sizes where a
launch changes shape: one contact, a partly filled block, one more trip than the grid's threads.

max_ite = 6 from a step size far above 1/L: the first iterations backtrack, so candidates that
are thrown away and taken are both on the path.  Six iterations on sums of at most a few tens of
terms amplify rounding by well under 1e4 (the step never exceeds 1/L after backtracking), so FP64
iterates agree to 1e4 * 2^-53 ~ 1e-12 and FP32 ones to 1e4 * 2^-24 ~ 6e-4 (2-norm).
"""
import numpy as np
import pytest

import py_oracle as orc
from scopi_b200 import FP64, FRICTION, MIXED, NOFRICTION, VISCOUS, ScopiBatch, ScopiSolver, configs

pytestmark = pytest.mark.gpu

DT, ITE = 1e-3, 6


def bed(dim, count, seed=7):
    """`count` approaching bodies: a lattice with gaps of a sixth of a diameter, 3 m/s."""
    if dim == 3:
        pa = configs.box_3d(seed=seed, count=count)
    else:
        pa = configs.disks_2d(seed=seed, side=int(np.ceil(np.sqrt(count))))
        n = count
        for k in ("shape", "pos", "q", "v", "omega", "vd", "omega_d", "f", "m", "j", "radius", "length", "axes",
                  "squareness", "worm"):
            setattr(pa, k, np.ascontiguousarray(getattr(pa, k)[:n]))
    rng = np.random.default_rng(seed)
    a = pa.nb_inactive
    pa.v[a:, :dim] = rng.uniform(-3, 3, (pa.n - a, dim))
    if dim == 3:
        pa.omega[a:] = rng.uniform(-50, 50, (pa.n - a, 3))
        q = rng.normal(size=(pa.n - a, 4))
        pa.q[a:] = q / np.linalg.norm(q, axis=1)[:, None]
    else:
        pa.omega[a:, 2] = rng.uniform(-50, 50, pa.n - a)
    return pa


def settings(dim, problem):
    kw = dict(dmax=0.0045 if dim == 3 else 0.01, vap=1, tolerance=1e-12, max_ite=ITE, alpha=1e9, problem=problem)
    if problem == FRICTION:
        kw["mu"] = 0.3
    return kw


def check(dim, count, problem, precision):
    pa = bed(dim, count)
    kw = settings(dim, problem)
    o = orc.OracleSolver(pa, **kw).run(DT, 1)
    more = {}
    if precision == MIXED:
        # the FP32 iterates alone: the reference's first step, no correction solves
        more = dict(initial_step=0, mixed_max_corrections=0, mixed_violation_tol=1e9)
    s = ScopiSolver(pa, precision=precision, **kw, **more)
    s.step(DT, 1)
    g = s.download(pa.copy())
    lam, ref = s.lagrange_multiplier(), o.lagrange_multiplier()
    st, so = s.stats(), o.stats()
    assert st["contacts"] == so["contacts"] > 0
    assert (st["iterations"], st["backtracks"]) == (so["iterations"], so["backtracks"])
    bound = 1e-12 if precision == FP64 else 6e-4
    assert count < 10 or np.linalg.norm(ref) > 0
    assert np.linalg.norm(lam - ref) <= bound * np.linalg.norm(ref)
    assert np.linalg.norm(g.v - o.pa.v) <= bound * np.linalg.norm(o.pa.v)
    assert np.linalg.norm(g.omega - o.pa.omega) <= bound * np.linalg.norm(o.pa.omega)


# FP64 friction: 148 blocks of 256 threads; FP32: 148 of 512.  About 3 contacts a body.
@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("dim,count", [(3, 2), (3, 60), (3, 300), (3, 14001), (3, 30011), (2, 3), (2, 200), (2, 25000)])
def test_friction_iterates(dim, count, precision):
    check(dim, count, FRICTION, precision)


# normal problems: FP64 148 blocks of 512 threads, FP32 148 of 768
@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("problem", [NOFRICTION, VISCOUS])
@pytest.mark.parametrize("dim,count", [(3, 2), (3, 200), (3, 27001), (3, 45007), (2, 3), (2, 300)])
def test_normal_iterates(dim, count, problem, precision):
    check(dim, count, problem, precision)


# Batched friction scenes: clusters of four CTAs (few scenes) and of two (many), the largest
# scenes on a whole cluster, the others one CTA each; 256 chains of contacts in the sums.
@pytest.mark.parametrize("dim,sizes", [(2, [300]), (2, [3, 700, 90, 1500]), (2, [40 + 7 * k for k in range(90)]),
                                       (3, [250, 5, 600]), (3, [20 + k for k in range(80)])])
def test_batch_friction_iterates(dim, sizes):
    scenes = [bed(dim, n, seed=20 + k) for k, n in enumerate(sizes)]
    kw = settings(dim, FRICTION)
    b = ScopiBatch(scenes, **kw)
    b.run(DT, 1)
    for k, pa in enumerate(scenes):
        o = orc.OracleSolver(pa, **kw).run(DT, 1)
        st, so = b.scene_stats(k), o.stats()
        assert st["contacts"] == so["contacts"]
        assert (st["iterations"], st["backtracks"]) == (so["iterations"], so["backtracks"])
        g = b.scene(k)
        assert np.linalg.norm(g.v - o.pa.v) <= 1e-12 * np.linalg.norm(o.pa.v)
        assert np.linalg.norm(g.omega - o.pa.omega) <= 1e-12 * np.linalg.norm(o.pa.omega)
    b.close()
