"""Tet step on the GPU, through the C ABI, against the oracle.

REF32 and J2_F64 must be bit-identical to their CPU counterparts; the FP32 modes are
held to the target tolerance against the FP64 oracle (1e-5 relative displacement,
0.5 % energy-balance drift).
"""
import ctypes as C
import os

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def cantilever(fem, nx=40, ny=4, nz=4, load=20e3):
    """The CPU-runnable cantilever: 1.0 x 0.1 x 0.1 m, 6 Kuhn tets per cell, clamped at x = 0,
    tip load spread equally over the x = 1 face nodes in -z."""
    pos, idx = fem.box_tet_mesh(1.0, 0.1, 0.1, nx, ny, nz)
    fixed = (pos[0::3] < 1e-6).astype(np.uint32)
    tip = pos[0::3] > 1.0 - 1e-6
    fext = np.zeros(pos.size)
    fext[2::3][tip] = -load / tip.sum()
    return pos, idx, fixed, fext


def test_ref32_bit_identical_to_reference_step(fem, port):
    """The fem_spike GPU-vs-CPU case (tools/fem_spike/main.cpp:143-222), where the
    reference accepts 1e-4 after one step: here the GPU matches bit for bit."""
    g = np.load(os.path.join(GOLDEN, "tet32_spike.npz"))
    s = fem.TetSolver(g["start"], g["index"], mode="ref32", mass=g["mass"], fixed=g["fixed"],
                      rest_inv=g["rest_inv"], rest_volume=g["rest_volume"], adjacency_offset=g["adj_offset"],
                      adjacency_entry=g["adj_entry"])
    dt = float(g["dt"])
    done = 0
    for target in (1, 10, 100):
        s.run(target - done, youngs=210e9, poisson=0.3, dt=dt, gravity=9.80665, damping=1.0)
        done = target
        p, v = s.readback()
        assert np.array_equal(p, g[f"position_{target}"]), target
        assert np.array_equal(v, g[f"velocity_{target}"]), target
    # and on to 1000 steps against the restatement (graph-captured chunks)
    m = O.TetMesh32(port, g["start"], g["index"])
    m.fixed[:] = g["fixed"]
    for name in ("mass", "rest_inv", "rest_volume", "adj_offset", "adj_entry"):
        getattr(m, name)[:] = g[name]
    m.step(210e9, 0.3, 7850.0, dt, 9.80665, 1.0, 1000)
    s.run(900, youngs=210e9, poisson=0.3, dt=dt, gravity=9.80665, damping=1.0)
    p, v = s.readback()
    assert np.array_equal(p, m.position) and np.array_equal(v, m.velocity)


def test_f64_bit_identical_to_oracle(fem):
    g = np.load(os.path.join(GOLDEN, "tet64_cantilever.npz"))
    pos, idx, fixed, fext = cantilever(fem)
    s = fem.TetSolver(pos, idx, mode="f64", fixed=fixed, external_force=fext, density=7850.0)
    assert s.critical_dt(210e9, 0.3, 7850.0, 0.9) == float(g["dt"])
    s.run(int(g["steps"]), dt=float(g["dt"]), ramp_steps=2000)
    p, v = s.readback64()
    assert np.array_equal(p, g["position"])
    assert np.array_equal(v, g["velocity"])
    assert np.array_equal(s.plastic().reshape(-1), g["plastic"])
    e = s.energy()
    assert np.allclose(e[:4], g["energy"][:4], rtol=1e-12, atol=1e-18)


def _rel_disp_error(p, ref, rest):
    u, ur = p - rest, ref - rest
    return np.abs(u - ur).max() / np.abs(ur).max()


@pytest.mark.parametrize("mode,tol", [("f32k", 1e-5), ("f32", 1e-3)])
def test_f32_against_fp64_oracle(fem, port, mode, tol):
    """The config-0 cantilever with the tip load scaled to 200 kN (ramped over 1000
    steps) so that ~40 % of the tets yield by step 2000, as the precision study asks."""
    pos, idx, fixed, fext = cantilever(fem, load=200e3)
    ref = O.TetMesh64(port, pos, idx, fixed, fext)
    dt = port.tet64_critical_dt(C.byref(ref._s), 210e9, 0.3, 7850.0, 0.9)
    params = O.tet64_params(dt=dt, ramp_steps=1000)
    ref.step(params, 2000)
    s = fem.TetSolver(pos, idx, mode=mode, fixed=fixed, external_force=fext, density=7850.0)
    s.run(2000, dt=dt, ramp_steps=1000)
    p, _ = s.readback64()
    rest = pos.astype(np.float64)
    err = _rel_disp_error(p, ref.position, rest)
    yielded = (ref.plastic.reshape(-1, 7)[:, 6] > 0).mean()
    assert yielded > 0.3, "the case must exercise plasticity"
    assert err < tol, (mode, err)
    e, er = s.energy(), ref.energy
    # energy account against the oracle's, and its own balance
    assert abs(e[0] - er[0]) / er[0] < 5e-3
    drift = abs(e[0] - (e[1] + e[2] + e[3])) / e[0]
    drift_ref = abs(er[0] - (er[1] + er[2] + er[3])) / er[0]
    assert abs(drift - drift_ref) < 5e-3


def test_graph_replay_is_bit_identical_to_single_launches(fem):
    pos, idx, fixed, fext = cantilever(fem, nx=20, ny=2, nz=2)
    a = fem.TetSolver(pos, idx, mode="f32k", fixed=fixed, external_force=fext, density=7850.0)
    b = fem.TetSolver(pos, idx, mode="f32k", fixed=fixed, external_force=fext, density=7850.0)
    dt = a.critical_dt()
    a.run(96, dt=dt, ramp_steps=200)
    for _ in range(96):
        b.run(1, dt=dt, ramp_steps=200)
    pa, va = a.readback()
    pb, vb = b.readback()
    assert np.array_equal(pa, pb) and np.array_equal(va, vb)
    assert np.array_equal(a.energy(), b.energy())
    assert a.launches == 2 * 96 and b.launches == 2


def test_rest_stays_at_rest(fem):
    """A patch at rest with no load stays at rest (tests/test_zone.cpp:483), in every mode."""
    pos, idx, fixed, _ = cantilever(fem, nx=8, ny=2, nz=2)
    for mode in ("f32", "f32k", "f64"):
        s = fem.TetSolver(pos, idx, mode=mode, fixed=fixed, density=7850.0)
        s.run(200, dt=s.critical_dt())
        p, v = s.readback64()
        # FP32 modes carry the displacement gradient, which is exactly zero at rest;
        # FP64 carries F = Ds Dm^-1, whose rounding residue (~1e-16) may move a node
        # by far less than a femtometre.
        tol = 0.0 if mode != "f64" else 1e-14
        assert np.abs(p - pos).max() <= tol and np.abs(v).max() <= tol * 1e5, mode


@pytest.mark.parametrize("cells", [(1, 1, 1), (2, 1, 1), (5, 3, 1)])
def test_tiny_meshes_in_every_mode(fem, port, cells):
    """Meshes far smaller than a block (6, 12 and 90 tets): the tail threads of the
    element and node passes do nothing.  The FP64 step is bit-identical to the FP64
    oracle; the FP32-compensated one within the target tolerance; REF32 bit-identical
    to the reference's float step restated."""
    nx, ny, nz = cells
    pos, idx = fem.box_tet_mesh(0.1 * nx, 0.1 * ny, 0.1 * nz, nx, ny, nz)
    fixed = (pos[0::3] < 1e-6).astype(np.uint32)
    tip = pos[0::3] > 0.1 * nx - 1e-6
    fext = np.zeros(pos.size)
    fext[2::3][tip] = -2e5 * ny * nz / tip.sum()
    ref = O.TetMesh64(port, pos, idx, fixed, fext)
    dt = port.tet64_critical_dt(C.byref(ref._s), 210e9, 0.3, 7850.0, 0.9)
    ref.step(O.tet64_params(dt=dt, ramp_steps=100), 300)
    g = fem.TetSolver(pos, idx, mode="f64", fixed=fixed, external_force=fext, density=7850.0)
    g.run(300, dt=dt, ramp_steps=100)
    p64, _ = g.readback64()
    assert np.array_equal(p64, ref.position)
    k = fem.TetSolver(pos, idx, mode="f32k", fixed=fixed, external_force=fext, density=7850.0)
    k.run(300, dt=dt, ramp_steps=100)
    pk, _ = k.readback64()
    assert np.abs(ref.position - pos).max() > 1e-7, "the mesh must move"
    assert _rel_disp_error(pk, ref.position, pos.astype(np.float64)) < 1e-5
    # REF32: the reference's float step (elastic, gravity), restated, bit for bit
    m = O.TetMesh32(port, pos, idx)
    m.fixed[:] = fixed
    m.rest_state(210e9, 0.3, 7850.0)
    r = fem.TetSolver(pos, idx, mode="ref32", fixed=fixed, mass=m.mass, rest_inv=m.rest_inv,
                      rest_volume=m.rest_volume, adjacency_offset=m.adj_offset, adjacency_entry=m.adj_entry)
    m.step(210e9, 0.3, 7850.0, 1e-6, 9.80665, 1.0, 50)
    r.run(50, youngs=210e9, poisson=0.3, dt=1e-6, gravity=9.80665, damping=1.0)
    pr, vr = r.readback()
    assert np.array_equal(pr, m.position) and np.array_equal(vr, m.velocity)


@pytest.mark.parametrize("mode", ["f64", "f32k", "f32"])
def test_device_set_up_is_the_host_set_up(fem, mode):
    """A J2 mesh given without an adjacency is set up on the device (CSR, slot map and
    the FP64 rest state); given with one, on the host.  The two must be the same to the
    bit: the same critical step, and the same state after a yielding run."""
    pos, idx, fixed, fext = cantilever(fem, 24, 3, 3, load=300e3)
    offset, entry = fem.csr(pos.size // 3, idx, 4)
    dev = fem.TetSolver(pos, idx, mode=mode, fixed=fixed, external_force=fext, density=7850.0)
    host = fem.TetSolver(pos, idx, mode=mode, fixed=fixed, external_force=fext, density=7850.0,
                         adjacency_offset=offset, adjacency_entry=entry)
    dt = dev.critical_dt(210e9, 0.3, 7850.0, 0.9)
    assert dt == host.critical_dt(210e9, 0.3, 7850.0, 0.9)
    for s in (dev, host):
        s.run(400, dt=dt, ramp_steps=200)
    pd, vd = dev.readback64()
    ph, vh = host.readback64()
    assert np.array_equal(pd, ph) and np.array_equal(vd, vh)
    assert np.array_equal(dev.plastic(), host.plastic())
    assert (host.plastic()[:, 6] > 0).any(), "the case must yield"
    assert np.array_equal(dev.energy(), host.energy())


@pytest.mark.parametrize("cells", [(7, 3, 1), (16, 4, 1), (43, 1, 1), (13, 5, 2)])
@pytest.mark.parametrize("pull", [2e4, 2e7])
def test_f64_at_block_edges_and_large_rotations(fem, port, cells, pull):
    """The FP64 step packs a block's unfinished polar iterations together: meshes of 126
    to 780 tets, around one to six blocks' edges and with ragged last ones, from small
    strains (iterations that cycle or drift in the last bits) to rotations and stretches
    of order one, bit-identical to the FP64 oracle."""
    nx, ny, nz = cells
    pos, idx = fem.box_tet_mesh(0.1 * nx, 0.1 * ny, 0.1 * nz, nx, ny, nz)
    fixed = (pos[0::3] < 1e-6).astype(np.uint32)
    tip = pos[0::3] > 0.1 * nx - 1e-6
    fext = np.zeros(pos.size)
    fext[2::3][tip] = -pull * ny * nz / tip.sum()
    ref = O.TetMesh64(port, pos, idx, fixed, fext)
    dt = 0.5 * port.tet64_critical_dt(C.byref(ref._s), 210e9, 0.3, 7850.0, 0.9)
    ref.step(O.tet64_params(dt=dt, ramp_steps=100), 400)
    assert np.isfinite(ref.position).all()
    g = fem.TetSolver(pos, idx, mode="f64", fixed=fixed, external_force=fext, density=7850.0)
    g.run(400, dt=dt, ramp_steps=100)
    p, v = g.readback64()
    assert np.array_equal(p, ref.position) and np.array_equal(v, ref.velocity)
    assert np.array_equal(g.plastic().reshape(-1), ref.plastic)


@pytest.mark.parametrize("spokes", [1, 7, 8, 9, 31, 300])
def test_uneven_runs_of_slots(fem, port, spokes):
    """A hub shared by every tet beside nodes of at most three: the node pass's runs are
    strided where a group of 32 nodes is even and contiguous where it is not, and their
    loads go in batches of eight.  FP64 and REF32 bit-identical to their oracles."""
    k = np.arange(spokes + 2)
    ring = np.stack([np.cos(2.1 * k), np.sin(2.1 * k), 0.3 * np.cos(0.7 * k)], 1)
    pos = np.vstack([[[0.0, 0.0, 0.9]], ring]).astype(np.float32).reshape(-1)
    idx = np.stack([0 * k[:-2], k[:-2] + 1, k[1:-1] + 1, k[2:] + 1], 1).astype(np.uint32).reshape(-1)
    fixed = np.zeros(pos.size // 3, np.uint32)
    fixed[-1] = 1
    fext = np.zeros(pos.size)
    fext[2] = 1e4
    ref = O.TetMesh64(port, pos, idx, fixed, fext)
    dt = port.tet64_critical_dt(C.byref(ref._s), 210e9, 0.3, 7850.0, 0.5)
    ref.step(O.tet64_params(dt=dt, ramp_steps=10), 60)
    g = fem.TetSolver(pos, idx, mode="f64", fixed=fixed, external_force=fext, density=7850.0)
    g.run(60, dt=dt, ramp_steps=10)
    p, v = g.readback64()
    assert np.array_equal(p, ref.position) and np.array_equal(v, ref.velocity)
    m = O.TetMesh32(port, pos, idx)
    m.fixed[:] = fixed
    m.rest_state(210e9, 0.3, 7850.0)
    r = fem.TetSolver(pos, idx, mode="ref32", fixed=fixed, mass=m.mass, rest_inv=m.rest_inv,
                      rest_volume=m.rest_volume, adjacency_offset=m.adj_offset, adjacency_entry=m.adj_entry)
    m.step(210e9, 0.3, 7850.0, dt, 9.80665, 1.0, 60)
    r.run(60, youngs=210e9, poisson=0.3, dt=dt, gravity=9.80665, damping=1.0)
    pr, vr = r.readback()
    assert np.array_equal(pr, m.position) and np.array_equal(vr, m.velocity)


@pytest.mark.parametrize("mode", ["ref32", "f32", "f32k", "f64"])
@pytest.mark.parametrize("cells", [(1, 1, 1), (7, 3, 1), (43, 1, 1), (13, 9, 5), (11, 10, 6), (682, 1, 1), (21, 13, 5)])
def test_cluster_run_is_the_steps_to_the_bit(fem, mode, cells):
    """A long run of a small mesh is one launch of one cluster of blocks: 6 to 8,190 tets,
    one to sixteen blocks of 128 to 512 threads, ragged last groups (FP64 above 4,096 tets
    takes the two kernels a step).  State and energy account to the bit those of the same
    steps in short runs, before and after it too."""
    nx, ny, nz = cells
    pos, idx = fem.box_tet_mesh(0.05 * nx, 0.05 * ny, 0.05 * nz, nx, ny, nz)
    fixed = (pos[0::3] < 1e-6).astype(np.uint32)
    tip = pos[0::3] > 0.05 * nx - 1e-6
    fext = np.zeros(pos.size)
    fext[2::3][tip] = -3e5 * ny * nz / max(1, tip.sum())  # the longest mesh's tip rounds away: gravity alone
    if mode == "ref32":
        x = pos.reshape(-1, 3).astype(np.float64)[idx.reshape(-1, 4)]
        d = np.transpose(x[:, 1:] - x[:, :1], (0, 2, 1))
        vol = np.abs(np.linalg.det(d)) / 6
        off, ent = fem.csr(pos.size // 3, idx, 4)
        mass = np.bincount(idx, weights=np.repeat(7850 * vol / 4, 4), minlength=pos.size // 3)
        vel = np.zeros(pos.size)
        vel[2::3] = -10.0 * pos[0::3]
        kw = dict(mass=mass, velocity=vel, rest_volume=vol, adjacency_offset=off, adjacency_entry=ent,
                  rest_inv=np.transpose(np.linalg.inv(d), (0, 2, 1)))
    else:
        kw = dict(external_force=fext, density=7850.0)
    a, b = (fem.TetSolver(pos, idx, mode=mode, fixed=fixed, **kw) for _ in range(2))
    run = dict(dt=1.5e-6, gravity=9.80665, damping=0.9999, ramp_steps=100)
    a.run(7, **run)
    a.run(200, **run)
    used = a.launches
    a.run(40, **run)
    for n in (7, 50, 50, 50, 50, 40):
        b.run(n, **run)
    fits = idx.size // 4 <= (4096 if mode == "f64" else 8192)
    assert used == (1 if fits else 400)
    pa, va = a.readback64()
    pb, vb = b.readback64()
    assert np.abs(pa - pos).max() > 1e-7 and np.isfinite(pa).all()
    assert np.array_equal(pa, pb) and np.array_equal(va, vb)
    assert np.array_equal(a.plastic(), b.plastic()) and np.array_equal(a.energy(), b.energy())
    if mode != "ref32" and nx > 10 and tip.any():
        assert (a.plastic()[:, 6] > 0).any(), "the case must yield"


@pytest.mark.parametrize("cells", [(7, 3, 1), (16, 4, 1), (43, 1, 1), (13, 5, 2)])
@pytest.mark.parametrize("pull", [2e4, 2e7])
def test_f64_two_kernel_step_at_block_edges_and_large_rotations(fem, port, cells, pull):
    """The same meshes and loads in runs too short for a cluster: two kernels a step, as every
    large mesh has them, bit-identical to the FP64 oracle."""
    nx, ny, nz = cells
    pos, idx = fem.box_tet_mesh(0.1 * nx, 0.1 * ny, 0.1 * nz, nx, ny, nz)
    fixed = (pos[0::3] < 1e-6).astype(np.uint32)
    tip = pos[0::3] > 0.1 * nx - 1e-6
    fext = np.zeros(pos.size)
    fext[2::3][tip] = -pull * ny * nz / tip.sum()
    ref = O.TetMesh64(port, pos, idx, fixed, fext)
    dt = 0.5 * port.tet64_critical_dt(C.byref(ref._s), 210e9, 0.3, 7850.0, 0.9)
    ref.step(O.tet64_params(dt=dt, ramp_steps=100), 400)
    g = fem.TetSolver(pos, idx, mode="f64", fixed=fixed, external_force=fext, density=7850.0)
    for _ in range(4):
        g.run(100, dt=dt, ramp_steps=100)
        assert g.launches == 200, "two kernels a step"
    p, v = g.readback64()
    assert np.array_equal(p, ref.position) and np.array_equal(v, ref.velocity)
    assert np.array_equal(g.plastic().reshape(-1), ref.plastic)


@pytest.mark.parametrize("mode", ["f32", "f32k"])
@pytest.mark.parametrize("spare", [0, 11, 12, 400])
def test_readback_between_runs_changes_nothing(fem, mode, spare):
    """The FP32 modes' positions are formed on the device in the force slots, or on the host
    where the nodes in no tet (one tet of four nodes and 4 slots, up to 404 nodes) outnumber
    them: the same positions either way, and steps after a readback are those without one."""
    pos = np.concatenate([[0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0, 1], 3.0 + 0.01 * np.arange(3 * spare)]).astype(np.float32)
    idx = np.array([0, 1, 2, 3], np.uint32)
    fixed = np.zeros(pos.size // 3, np.uint32)
    fixed[0] = 1
    ext = np.zeros(pos.size)
    ext[3:6] = 1e5
    a, b = (fem.TetSolver(pos, idx, mode=mode, fixed=fixed, external_force=ext, density=7850.0) for _ in range(2))
    run = dict(dt=2e-5, ramp_steps=10)
    for n in (7, 40, 3):
        a.run(n, **run)
        b.run(n, **run)
        p, v = a.readback64()
        q, w = a.readback()
        assert np.array_equal(p.astype(np.float32), q) and np.array_equal(v, w)
    assert np.abs(p[:12] - pos[:12]).max() > 1e-6
    pb, vb = b.readback64()
    assert np.array_equal(p, pb) and np.array_equal(v, vb) and np.array_equal(a.energy(), b.energy())


@pytest.mark.parametrize("mode", ["f32", "f32k"])
@pytest.mark.parametrize("cells", [(11, 13, 11), (15, 15, 7), (13, 13, 13)])
def test_readback_between_runs_of_a_box(fem, mode, cells):
    """The same for meshes of 2,016, 2,048 and 2,744 nodes, around the line under which the plain
    mode forms its positions on the host."""
    nx, ny, nz = cells
    pos, idx = fem.box_tet_mesh(0.05 * nx, 0.05 * ny, 0.05 * nz, nx, ny, nz)
    fixed = (pos[0::3] < 1e-6).astype(np.uint32)
    a, b = (fem.TetSolver(pos, idx, mode=mode, fixed=fixed, density=7850.0) for _ in range(2))
    run = dict(dt=2e-6, gravity=9.80665)
    for n in (3, 40):
        a.run(n, **run)
        b.run(n, **run)
        p, v = a.readback64()
        q, w = a.readback()
        assert np.array_equal(p.astype(np.float32), q) and np.array_equal(v, w)
    assert np.abs(p - pos).max() > 1e-8
    pb, vb = b.readback64()
    assert np.array_equal(p, pb) and np.array_equal(v, vb) and np.array_equal(a.energy(), b.energy())
