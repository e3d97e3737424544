"""What the host code orders before what, without a GPU: the library's own objects linked
with fake_cudart.cpp, where no kernel runs and device work stays pending until something
waits for it."""
import ctypes as C
import glob
import importlib.util
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sinking-simulator_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def bound(tmp_path_factory):
    """The binding over the library's host code and the fake runtime."""
    subprocess.run(["make", "-s", "-C", PKG, "-j8"], check=True)
    so = str(tmp_path_factory.mktemp("fake") / "libfemstep_fake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-Wl,--no-undefined",
                    "-I", os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "fake_cudart.cpp"),
                    *sorted(glob.glob(os.path.join(PKG, "_build", "*.o"))), "-o", so, "-lpthread"], check=True)
    spec = importlib.util.spec_from_file_location("femstep_fake", os.path.join(PKG, "femstep.py"))
    module = importlib.util.module_from_spec(spec)
    real = C.CDLL
    C.CDLL = lambda path, *a, **k: real(so, *a, **k)
    try:
        spec.loader.exec_module(module)
    finally:
        C.CDLL = real
    return module


@pytest.fixture
def fake(bound):
    bound.lib.fake_reset()
    return bound


def tet_case(fem, mode, adjacency, cells=(4, 2, 2), load=True):
    pos, idx = fem.box_tet_mesh(0.4, 0.1, 0.02, *cells)
    N, T = pos.size // 3, idx.size // 4
    kw = {}
    if mode == "ref32":
        kw = dict(mass=np.ones(N), rest_inv=np.ones((T, 9)), rest_volume=np.ones(T))
    else:
        kw = dict(density=7850.0)
        if load:
            kw["external_force"] = np.ones(N * 3)
    if adjacency:
        kw["adjacency_offset"], kw["adjacency_entry"] = fem.csr(N, idx, 4)
    return pos, idx, dict(kw, mode=mode, fixed=np.zeros(N, np.uint32), velocity=np.zeros(N * 3))


@pytest.mark.parametrize("load", [True, False])
@pytest.mark.parametrize("adjacency", [True, False])
@pytest.mark.parametrize("mode", ["ref32", "f32", "f32k", "f64"])
def test_tet_uploads_land_before_the_solver_reads_them(fake, mode, adjacency, load):
    """A copy from pageable memory and a memset on the legacy stream may return before the
    device has done them, and the solver's stream does not wait for that stream: both are
    waited for before a set-up kernel and before create returns."""
    pos, idx, kw = tet_case(fake, mode, adjacency, load=load)
    s = fake.TetSolver(pos, idx, **kw)
    assert fake.lib.fake_unordered() == 0
    assert fake.lib.fake_pending() == 0
    s.run(40, dt=1e-6)
    assert fake.lib.fake_unordered() == 0
    s.close()


@pytest.mark.parametrize("mode,adjacency,most", [("ref32", True, 51), ("f32k", True, 70), ("f32k", False, 80),
                                                 ("f64", True, 60), ("f64", False, 80)])
def test_tet_create_makes_few_calls(fake, mode, adjacency, most):
    """Every allocation, copy, wait and launch of a create is some 3 us of a small mesh's 250:
    what can share one does."""
    pos, idx, kw = tet_case(fake, mode, adjacency)
    fake.lib.fake_reset()
    s = fake.TetSolver(pos, idx, **kw)
    assert fake.lib.fake_calls() <= most
    s.close()


def shell_zone(fem, nx, ny):
    rest, index, pinned, load = fem.stiffened_panel(nx=nx, ny=ny, lx=0.01 * nx, ly=0.01 * ny, thickness=0.008,
                                                    stiffeners=0, imperfection=2e-4, peak_pressure=4e7, radius=10.0)
    return fem.ShellSolver(rest, index, pinned=pinned, load=load, density=7850.0)


@pytest.mark.parametrize("fibres", [False, True])
def test_shell_step_after_a_graph_waits_for_it(fake, fibres):
    """The last step of a graph renews the order that an element pass reads as soon as it comes
    up: a direct step right after a graph is an ordinary launch."""
    s = shell_zone(fake, 90, 80)
    if fibres:
        s.set_fibers([[0, 8281, 1, 8282]], [[0.5, 0.5]], [1e-4])
    for n in (37, 16, 5):
        s.run(n, dt=1e-7)
        assert fake.lib.fake_early_after_graph() == 0
    s.close()


@pytest.mark.parametrize("mode", ["ref32", "f32", "f32k", "f64"])
def test_refused_cluster_launch_leaves_no_error(fake, mode):
    """Where the launch of a small mesh's cluster is refused, the run takes two kernels a step
    and succeeds."""
    pos, idx, kw = tet_case(fake, mode, mode == "ref32")
    s = fake.TetSolver(pos, idx, **kw)
    fake.lib.fake_refuse_clusters(1)
    s.run(200, dt=1e-6)
    assert s.launches == 400 and fake.lib.fake_last_error() == 0
    s.close()


@pytest.mark.parametrize("mode", ["f32k", "f64"])
def test_failed_create_frees_nothing_that_kernels_still_use(fake, mode):
    """With no memory for the slot runs' scratch, create fails while its adjacency kernels are
    still in flight: they are waited for before their arrays go back to the device's pool."""
    pos, idx, kw = tet_case(fake, mode, False)
    fake.lib.fake_fail_malloc(3)  # the two of the adjacency, then the runs'
    with pytest.raises(fake.FemStepError) as e:
        fake.TetSolver(pos, idx, **kw)
    assert e.value.code == fake.ENOMEM
    assert fake.lib.fake_freed_in_flight() == 0


def test_small_readback_leaves_another_error_alone(fake):
    """An error that another call of this thread has left pending is not this one's to clear."""
    s = shell_zone(fake, 3, 3)
    fake.lib.fake_set_last_error(1)
    s.readback()
    assert fake.lib.fake_last_error() == 1
    s.close()


@pytest.mark.parametrize("mode,cells,most", [("f32", (4, 2, 2), 2), ("f32", (40, 9, 9), 4), ("f32k", (4, 2, 2), 4),
                                             ("f32k", (40, 9, 9), 4)])
def test_tet_readback_takes_no_device_memory(fake, mode, cells, most):
    """The positions formed on the device go through memory that the solver has: a launch, a copy
    and a wait for them, and the velocities' copy.  A small mesh's in the plain mode are one copy."""
    pos, idx, kw = tet_case(fake, mode, False, cells=cells)
    s = fake.TetSolver(pos, idx, **kw)
    for read in (s.readback, s.readback64):
        fake.lib.fake_reset()
        read()
        assert fake.lib.fake_calls() <= most
    s.close()


def test_pool_admission_launches_no_more_than_it_needs(fake):
    """A mesh's admission: its record and arrays, the adjacency, the rest state by tets and by
    nodes."""
    pos, idx = fake.box_tet_mesh(0.4, 0.1, 0.02, 4, 2, 2)
    pool = fake.TetPool(20000, 8000, max_meshes=8, tile=128)
    mesh = dict(position=pos, index=idx, external_force=np.ones(pos.size), dt=1e-8)
    pool.admit_many([mesh], [5])
    fake.lib.fake_reset()
    pool.admit_many([mesh], [5])
    assert fake.lib.fake_calls() <= 25
    pool.close()


def test_shell_create_makes_few_calls(fake):
    """A zone whose groups are taken in an order asks for no memory of its own for it: it is
    created with the calls of the smaller zones, which have none."""
    calls = []
    for nx, ny in ((88, 80), (90, 80)):  # 7,040 elements, one wave; 7,200
        fake.lib.fake_reset()
        s = shell_zone(fake, nx, ny)
        calls.append(fake.lib.fake_calls())
        s.close()
    assert calls[0] == calls[1]


def test_shell_settings_land_before_the_next_run(fake):
    """A punch, a driven edge, fibres and a restored state go up by copies that may return before
    they have landed; the next run's stream does not wait for them, so the calls do."""
    s = shell_zone(fake, 6, 5)
    saved = s.checkpoint()
    prescribed = np.zeros(3 * s.nodes)
    prescribed[:3] = 1e-4
    for setting in (lambda: s.restore(saved), lambda: s.set_punch([1, 3], [0.0, 0.0, -1.0], 1.0),
                    lambda: s.set_punch([1, 3], [0.0, 0.0, -1.0], 1.0, mass=10.0), lambda: s.set_edge(prescribed),
                    lambda: s.set_fibers([[0, 1, 12, 13]], [[0.5, 0.5]], [1e-4], density=7850.0)):
        setting()
        assert fake.lib.fake_pending() == 0
        s.run(3, dt=1e-7)
        assert fake.lib.fake_unordered() == 0
    s.close()
