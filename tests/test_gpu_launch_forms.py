"""First APGD iterates against the oracle where a solve takes a launch form that the sizes of
test_gpu_iterates.py do not reach.  Same settings, same bounds, derived there: six iterations from a
step size far above 1/L, FP64 to 1e-12 and FP32 to 6e-4 (2-norm)."""
import numpy as np
import pytest

import py_oracle as orc
from scopi_b200 import FP64, FRICTION, MIXED, NOFRICTION, VISCOUS, ScopiBatch, ScopiSolver, _abi
from scopi_b200.solver import ScopiGPUError
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


def first_iterates(pa, problem, precision, contacts=None):
    """One step against the oracle; `contacts`: (least, most) that put the solve into its form."""
    kw = settings(pa.dim, problem)
    o = orc.OracleSolver(pa, **kw).run(DT, 1)
    # FP32: the iterates alone, the reference's first step and no correction solves
    more = dict(initial_step=0, mixed_max_corrections=0, mixed_violation_tol=1e9) if precision == MIXED else {}
    s = ScopiSolver(pa, precision=precision, **kw, **more)
    s.step(DT, 1)
    g = s.download(pa.copy())
    lam, ref = s.lagrange_multiplier(), o.lagrange_multiplier()
    st, so = s.stats(), o.stats()
    s.close()
    assert st["contacts"] == so["contacts"]
    if contacts:
        assert contacts[0] <= st["contacts"] <= contacts[1]
    assert (st["iterations"], st["backtracks"]) == (so["iterations"], so["backtracks"])
    bound = 1e-12 if precision == FP64 else 6e-4
    assert np.linalg.norm(ref) > 0
    assert np.linalg.norm(lam - ref) <= bound * np.linalg.norm(ref)
    assert np.linalg.norm(g.v - o.pa.v) <= bound * np.linalg.norm(o.pa.v)
    assert np.linalg.norm(g.omega - o.pa.omega) <= bound * np.linalg.norm(o.pa.omega)
    return o


# friction, one block per 256 contacts: clusters of 8 and 16 CTAs, then 17 blocks of the grid form
@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("dim,count,blocks", [(3, 900, 7), (3, 2050, 16), (3, 2100, 17), (2, 2100, 16), (2, 2200, 17)])
def test_friction_clusters(dim, count, blocks, precision):
    first_iterates(bed(dim, count), FRICTION, precision, (256 * blocks - 255, 256 * blocks))


# normal problems: 512 contacts a block in FP64, 768 in FP32, a cluster up to 16 blocks
@pytest.mark.parametrize("problem", [NOFRICTION, VISCOUS])
@pytest.mark.parametrize("count,precision,contacts", [
    (1950, FP64, (7 * 512 + 1, 8 * 512)), (3500, FP64, (15 * 512 + 1, 16 * 512)), (3550, FP64, (16 * 512 + 1, 17 * 512)),
    (4900, MIXED, (15 * 768 + 1, 16 * 768)), (5000, MIXED, (16 * 768 + 1, 17 * 768))])
def test_normal_clusters(count, problem, precision, contacts):
    first_iterates(bed(3, count), problem, precision, contacts)


# The grid's registers hold two (FP64) or four (FP32) contacts and one body a thread, 148 blocks of
# 512 or 768 threads; past that the records are streamed.
G64, G32 = 148 * 512, 148 * 768


@pytest.mark.parametrize("problem", [NOFRICTION, VISCOUS])
@pytest.mark.parametrize("dim,count,precision,contacts", [
    (3, 90_000, MIXED, (2 * G32 + 1, 4 * G32)), (3, 52_000, FP64, (2 * G64 + 1, 3 * G64)),
    (2, 76_000, FP64, (G64 + 1, 2 * G64)), (3, 120_000, MIXED, (3 * G32 + 1, 4 * G32))])
def test_normal_resident_and_streaming(dim, count, problem, precision, contacts):
    pa = bed(dim, count)
    if count == 76_000 or count == 120_000:
        assert pa.n - pa.nb_inactive > (G64 if precision == FP64 else G32)  # more bodies than threads
    first_iterates(pa, problem, precision, contacts)


def slab_with_a_large_sphere(count=6000, radius=0.06):
    """A sphere of twelve times the others' radius among them: its list of contacts is far longer than
    the mean, so that the incidence records stay in rows."""
    pa = bed(3, count)
    a = pa.nb_inactive
    x = pa.pos[a:]
    i = int(np.argmin(((x - x.mean(0)) ** 2).sum(1)))
    keep = np.linalg.norm(x - x[i], axis=1) >= radius + pa.radius[a:] + 1e-4
    keep[i] = True
    pa.radius[a + i] = radius
    pa.m[a + i] = (radius / 0.005) ** 3
    pa.j[a + i] = 0.4 * pa.m[a + i] * radius ** 2
    keep = np.concatenate([np.ones(a, bool), keep])
    for k in ("shape", "pos", "q", "v", "omega", "vd", "omega_d", "f", "m", "j", "radius", "length", "axes",
              "squareness", "worm"):
        setattr(pa, k, np.ascontiguousarray(getattr(pa, k)[keep]))
    return pa, int(keep[:a + i].sum())


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("problem", [NOFRICTION, VISCOUS, FRICTION])
def test_uneven_incidence_lists(problem, precision):
    pa, large = slab_with_a_large_sphere()
    c = first_iterates(pa, problem, precision).contacts()
    na = pa.n - pa.nb_inactive
    width = int(((c["i"] == large) | (c["j"] == large)).sum())
    # columns as wide as the longest list would not fit the 4 records per contact of capacity
    assert width * 32 * -(-na // 32) > 4 * max(8192, 6 * na + 128 * pa.nb_inactive)


@pytest.mark.parametrize("problem,precision,count", [
    (NOFRICTION, FP64, 27_001), (NOFRICTION, FP64, 60_000), (NOFRICTION, MIXED, 120_000), (VISCOUS, FP64, 60_000),
    (FRICTION, FP64, 14_001), (FRICTION, MIXED, 14_001)])
def test_wait_limit_of_the_grid_forms(problem, precision, count):
    """One block withholds its first arrival (scopi_gpu_test_barrier_stall): every wait ends at the
    limit, the step reports it, and the next one gives a fresh handle's first step (vap_fixed and static
    walls: the failed step moved nothing).  Resident, streaming and friction launches of the whole grid."""
    pa = bed(3, count)
    pa.vd[:] = pa.v
    pa.omega_d[:] = pa.omega
    kw = dict(settings(3, problem), vap=0, precision=precision)
    s = ScopiSolver(pa, barrier_timeout_us=5000, **kw)
    s.step(DT, 0)
    lib = _abi.load()
    assert lib.scopi_gpu_test_barrier_stall(s._h) == 0
    with pytest.raises(ScopiGPUError) as exc:
        s.step(DT, 1)
    assert f"({_abi.ETIMEOUT})" in str(exc.value)
    s.step(DT, 1)
    ref = ScopiSolver(pa, **kw)
    ref.step(DT, 1)
    g, h = s.download(pa.copy()), ref.download(pa.copy())
    assert np.array_equal(g.pos, h.pos) and np.array_equal(g.v, h.v)
    s.close()
    ref.close()
