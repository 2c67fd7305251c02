"""Host code of the engine against a CUDA runtime without a GPU (tests/cpp/fake_cudart.cpp): two
devices, device memory that is host memory, kernels that do nothing, failures on request.

Each test runs in a process of its own, where the runtime of the test takes the place of the
real one before the library is loaded.
"""
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GXX = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else (shutil.which("g++") or "g++")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PRELUDE = """
import ctypes as C
import sys
fake = C.CDLL({so!r}, mode=C.RTLD_GLOBAL)
fake.fake_get.restype = fake.fake_launches_of.restype = C.c_longlong
get = lambda w: fake.fake_get(w.encode())
put = lambda w, v: fake.fake_set(w.encode(), C.c_longlong(v))
sys.path[:0] = [{root!r}, {tests!r}]
import numpy as np
import pytest
from scopi_b200 import FP64, FRICTION, MIXED, NOFRICTION, VISCOUS, ScopiBatch, ScopiSolver, _abi, configs
from scopi_b200.solver import ScopiGPUError
lib = _abi.load()

def rows(fn):
    return ScopiSolver(configs.box_3d(count=fn.pop("count", 60)), vap=1, dmax=0.0045, **fn)
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime_api.h")):
        pytest.skip("CUDA headers unavailable")
    from scopi_b200 import _abi, build
    if not os.path.exists(_abi.LIB_PATH):
        build.build()
    out = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run([GXX, "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(CUDA, "include"),
                    os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), "-o", out], check=True)

    def run(body):
        code = PRELUDE.format(so=out, root=ROOT, tests=os.path.join(ROOT, "tests")) + textwrap.dedent(body)
        r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout

    return run


def test_friction_clusters_on_a_second_device(fake):
    """9 to 16 blocks run as a cluster of 16, which every device has to allow for itself."""
    fake("""
    put("contacts", 4000)
    for dev in (0, 1, 0):
        for precision in (FP64, MIXED):
            s = rows(dict(problem=FRICTION, mu=0.3, precision=precision, device=dev))
            before = get("cluster_launches")
            s.step(1e-3, 1)
            assert get("cluster_launches") > before
            s.close()
    """)


def test_sphere_clusters_on_a_second_device(fake):
    fake("""
    put("contacts", 16 * 512)
    for dev in (0, 1, 0):
        for problem in (NOFRICTION, VISCOUS):
            for precision in (FP64, MIXED):
                s = rows(dict(problem=problem, precision=precision, device=dev))
                before = get("cluster_launches")
                s.step(1e-3, 1)
                assert get("cluster_launches") > before
                s.close()
    """)


def test_streaming_kernel_on_a_second_device(fake):
    """More contacts than the grid's registers hold: the form whose shared memory needs permission."""
    fake("""
    for dev in (0, 1):
        for problem in (NOFRICTION, VISCOUS):
            for precision, contacts in ((FP64, 160_000), (MIXED, 500_000), (MIXED, 2_000_000)):
                put("contacts", contacts)
                s = rows(dict(problem=problem, precision=precision, device=dev))
                s.step(1e-3, 1)
                assert s.stats()["contacts"] == contacts
                s.close()
    """)


def test_superellipsoid_start_kernel_on_a_second_device(fake):
    fake("""
    put("contacts", 100)
    put("superellipsoids", 20)
    for dev in (0, 1):
        s = ScopiSolver(configs.se_pile(20, side=3), vap=1, dmax=0.004, problem=FRICTION, mu=0.3, device=dev)
        s.step(5e-4, 1)
        assert get("launches") > 0 and get("refused") == 0
        s.close()
    """)


def test_refused_cluster_launch_takes_the_cooperative_form(fake):
    fake("""
    put("refuse_clusters", 1)
    put("contacts", 2000)
    for problem in (FRICTION, NOFRICTION, VISCOUS):
        for precision in (FP64, MIXED):
            s = rows(dict(problem=problem, precision=precision))
            s.step(1e-3, 1)
            assert s.stats()["contacts"] == 2000 and get("cluster_launches") == 0
            s.close()
    """)


@pytest.mark.parametrize("problem,precision", [("FRICTION", "FP64"), ("FRICTION", "MIXED"), ("NOFRICTION", "MIXED")])
def test_upload_retried_after_a_failed_allocation(fake, problem, precision):
    """Whichever allocation of an upload fails, the handle has no particles until the next one,
    which allocates everything; the first upload of a handle and one of another size."""
    fake(f"""
    kw = dict(problem={problem}, precision={precision}, vap=1, dmax=0.0045, mu=0.3)
    put("contacts", 100)
    small, large = configs.box_3d(count=30), configs.box_3d(count=60)

    def attempt(k, first):
        s = ScopiSolver(large if first else small, **kw)
        if not first:
            s.step(1e-3, 1)
        else:
            h = C.c_void_p()
            assert lib.scopi_gpu_create(C.byref(s._params), C.byref(h)) == 0
            s._h, s._created = h, True
        before = get("mallocs")
        put("fail_malloc", k)
        try:
            s.upload(large)
            failed = False
        except ScopiGPUError:
            failed = True
        put("fail_malloc", -1)
        if failed:
            with pytest.raises(ScopiGPUError, match="no particles"):
                s.step(1e-3, 1)
            s.upload(large)
        s.step(1e-3, 1)
        got = get("bytes"), get("mallocs") - before
        s.close()
        return failed, got

    for first in (True, False):
        _, (whole, count) = attempt(-1, first)
        assert count > 10
        for k in range(count):
            failed, (held, _) = attempt(k, first)
            assert failed and held == whole, (k, held, whole)
    """)


@pytest.mark.parametrize("problem,precision", [("FRICTION", "FP64"), ("NOFRICTION", "MIXED"), ("VISCOUS", "FP64")])
def test_step_retried_after_a_failed_growth(fake, problem, precision):
    """The contact buffers grow inside a step: after a failure the multipliers and the old list are
    gone, the bodies are not, and the next step allocates again."""
    fake(f"""
    kw = dict(problem={problem}, precision={precision}, vap=1, dmax=0.0045, mu=0.3)
    pa = configs.box_3d(count=30)

    def attempt(k):
        s = ScopiSolver(pa, **kw)
        put("contacts", 100)
        s.step(1e-3, 1)
        put("contacts", 20000)
        before = get("mallocs")
        put("fail_malloc", k)
        try:
            s.step(1e-3, 1)
            failed = False
        except ScopiGPUError:
            failed = True
        put("fail_malloc", -1)
        if failed:
            assert len(s.lagrange_multiplier()) == 0 and len(s.current_contacts()["i"]) == 0
            assert np.array_equal(s.download(pa.copy()).pos, pa.pos)
            s.step(1e-3, 1)
        got = get("bytes"), get("mallocs") - before
        s.close()
        return failed, got

    _, (whole, count) = attempt(-1)
    assert count > 10
    for k in range(count):
        failed, (held, _) = attempt(k)
        assert failed and held == whole, (k, held, whole)
    """)


@pytest.mark.parametrize("problem", ["FRICTION", "NOFRICTION"])
def test_corrections_allocate_nothing(fake, problem):
    """A violation target that is never met: every step ends with the FP64 correction."""
    fake(f"""
    put("contacts", 1000)
    s = rows(dict(problem={problem}, precision=MIXED, mu=0.3, mixed_violation_tol=-1.0, mixed_max_corrections=1))
    s.stream_handle()
    before = get("mallocs"), get("bytes")
    s.step(1e-3, 2)
    assert s.stats()["corrections"] == 2
    assert (get("mallocs"), get("bytes")) == before
    """)


@pytest.mark.parametrize("kw", ["problem=FRICTION, mu=0.3", "block_threads=2048", "block_threads=2048, precision=MIXED"])
def test_batch_step_without_its_solve_fails(fake, kw):
    """A solve that cannot be launched fails the step; nothing is replayed without it, and the batch
    steps again once the launch is possible."""
    fake(f"""
    scenes = [configs.box_3d(seed=k, count=30) for k in range(3)]
    b = ScopiBatch(scenes, vap=1, dmax=0.0045, {kw})
    for _ in range(2):
        put("refuse_clusters", 1)
        for _ in range(2):
            with pytest.raises(ScopiGPUError, match="batch solve"):
                b.run(1e-3, 1)
        put("refuse_clusters", 0)
        b.run(1e-3, 1)
        b.run(2e-3, 1)
        b.run(1e-3, 0)
    b.close()
    """)


# which kernel a friction batch takes: a queue of clusters loses to one small CTA per scene, a few
# large scenes win from clusters (template arguments of the names: dim, cluster or threads, CTAs per SM)
@pytest.mark.parametrize("dim,sizes,kernel", [
    (2, [2000] * 4, "k_fric_batchILi2ELi4"), (3, [250, 5, 600], "k_fric_batchILi3ELi4"),
    (2, [2000, 1900] + [200] * 94, "k_fric_batchILi2ELi4"), (2, [2000 - 20 * k for k in range(90)], "k_fric_batchILi2ELi2"),
    (2, [400] * 148, "k_fric_batchILi2ELi2"), (2, [300] * 600, "k_fric_manyILi2ELi256ELi2"),
    (2, [30] * 600, "k_fric_manyILi2ELi128ELi4"), (3, [30] * 600, "k_fric_manyILi3ELi128ELi2"),
    (3, [200] * 300, "k_fric_batchILi3ELi2")])
def test_friction_batch_form(fake, dim, sizes, kernel):
    fake(f"""
    scenes = []
    for n in {sizes}:
        pa = configs.box_3d(count=n)
        pa.dim = {dim}
        scenes.append(pa)
    b = ScopiBatch(scenes, vap=1, dmax=0.0045, problem=FRICTION, mu=0.3)
    b.run(1e-3, 1)
    assert fake.fake_launches_of(b"k_fric_batchI") + fake.fake_launches_of(b"k_fric_manyI") == 1
    assert fake.fake_launches_of({kernel.encode()}) == 1
    b.close()
    """)


# Device bytes per contact of capacity.  Normal problems and ViscousFriction: at most what they took
# when every handle had its own coefficient array.  Friction keeps packed rows (192 in FP64), incidence
# records (4 x 80) and iterates (96) beside the assembled rows; the generic rows took 832 and 1096.
@pytest.mark.parametrize("problem,precision,limit", [
    ("NOFRICTION", "FP64", 576), ("NOFRICTION", "MIXED", 728), ("VISCOUS", "FP64", 624), ("VISCOUS", "MIXED", 792),
    ("VISCOUS_FRICTION", "FP64", 928), ("VISCOUS_FRICTION", "MIXED", 1212), ("FRICTION", "FP64", 1104),
    ("FRICTION", "MIXED", 1140)])
def test_memory_per_contact(fake, problem, precision, limit):
    fake(f"""
    from scopi_b200 import VISCOUS_FRICTION
    got = []
    for n in (20_000, 60_000):
        put("contacts", n)
        s = rows(dict(problem={problem}, precision={precision}, mu=0.3))
        s.step(1e-3, 1)
        got.append(get("bytes"))
        s.close()
    # the capacity grows to 1.3 times the contacts
    assert got[1] - got[0] <= ({limit} + 0.5) * 1.3 * 40_000, (got[1] - got[0]) / 52_000
    """)


@pytest.mark.parametrize("kw,limit", [("", 748), ("precision=MIXED", 900), ("problem=VISCOUS", 796),
                                      ("problem=FRICTION, mu=0.3", 1192)])
def test_memory_of_a_batch(fake, kw, limit):
    """The bodies' share (about 1030 bytes each) included, per contact of capacity (six a body)."""
    fake(f"""
    got = []
    for n in (3000, 9000):
        b = ScopiBatch([configs.box_3d(count=n)], vap=1, dmax=0.0045, {kw})
        got.append(get("bytes"))
        b.close()
    assert got[1] - got[0] <= ({limit} + 0.5) * 6 * 6000, (got[1] - got[0]) / 36_000
    """)


@pytest.mark.parametrize("dim", [2, 3])
def test_noalloc_loads_its_kernels_at_the_first_call(fake, dim):
    """A kernel's first use loads its code into device memory: a caller that has warmed up on a small
    problem must not meet that on a larger one."""
    fake(f"""
    def call(contacts):
        n = contacts // 4
        i = np.zeros(contacts, np.int32)
        ptr, idx, x = np.zeros(n + 1, np.int32), np.zeros(2 * contacts, np.int32), np.zeros(3 * contacts)
        out, u, it = np.zeros(contacts), np.zeros((n, 3)), C.c_int64()
        p = lambda a: a.ctypes.data
        return lib.scopi_gpu_apgd_noalloc({dim}, n, 0, contacts, p(i), p(i), p(x), p(x), p(x), p(ptr), p(idx), 1e-3, 0.05,
                                          1e-6, 10, 1, p(out), p(u), C.byref(it), None)

    assert call(400) >= 0
    put("late_loads", 0)
    for contacts in (400, 4000, 8192, 8193, 12000, 16384):
        assert call(contacts) >= 0
    assert get("late_loads") == 0
    """)


def test_batch_creation_that_fails_leaves_no_handle(fake):
    fake("""
    scenes = [configs.box_3d(seed=k, count=30) for k in range(3)]
    arr = (_abi.ParticlesC * 3)()
    dp = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    for k, pa in enumerate(scenes):
        arr[k] = _abi.ParticlesC(pa.n, pa.nb_inactive, pa.shape.ctypes.data_as(C.POINTER(C.c_int32)), dp(pa.pos), dp(pa.q),
                                 dp(pa.v), dp(pa.omega), dp(pa.vd), dp(pa.omega_d), dp(pa.f), dp(pa.m), dp(pa.j),
                                 dp(pa.radius), dp(pa.length))
    p = _abi.Params()
    lib.scopi_gpu_default_params(C.byref(p), 3)
    p.problem = FRICTION

    def create(k):
        h = C.c_void_p()
        before = get("mallocs")
        put("fail_malloc", k)
        rc = lib.scopi_gpu_batch_create(C.byref(p), 3, arr, C.byref(h))
        put("fail_malloc", -1)
        return rc, h, get("mallocs") - before

    rc, h, count = create(-1)
    assert rc == 0 and h and count > 60
    lib.scopi_gpu_destroy(h)
    for k in range(count):
        rc, h, _ = create(k)
        assert rc < 0 and not h and get("bytes") == 0, (k, rc, h, get("bytes"))
    """)
