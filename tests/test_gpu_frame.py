"""Whole frames in one persistent launch with mailboxes between the tiles
(xpbd_frame_persistent) against the launch-by-launch path: the same program,
sums of the same corrections in another order.  A frame's differences are FP32
rounding of positions amplified by its iterations: 1e-5 of the scene's
diagonal, the gate of the per-iteration parity tests."""
import numpy as np
import pytest
import torch

from rlmusclev2_b200 import MuscleSim, XpbdSolver
from rlmusclev2_b200 import _capi as capi
from rlmusclev2_b200.batch import BatchSim
from rlmusclev2_b200.meshgen import batched_box_scene, box_muscle, humanv2_scene
from rlmusclev2_b200.mg import MultiGridSim, load_config
from tests._cases import bbox_diag
from tests.test_gpu_parity import _mixed_problem

pytestmark = pytest.mark.gpu

BOX = dict(dts=1.0 / 24.0, num_substeps=10, density=1060.0, veldamping=0.02, gravity=-9.8, relaxation=0.25, device="cuda:0",
           constraint_configs=[{"type": "tetarapsvd", "name": "arap", "compliance": 1e-7},
                               {"type": "volume", "name": "volume", "compliance": 0.0}])


@pytest.mark.parametrize("dims,tile", [((2, 2, 4), None), ((4, 4, 8), 64), ((4, 4, 8), 768), ((5, 7, 9), 100),
                                       ((8, 8, 32), None)])
def test_box_frames_match_launch_by_launch(dims, tile):
    """One tile, a few and many; remainders of the 256-thread loops."""
    m = box_muscle(*dims)
    sims = []
    for use in (True, False):
        s = MuscleSim.from_procedural(m.verts, m.tets, m.fiber_per_tet, stopped=m.stopped, tile_tets=tile, **BOX)
        s.use_persistent = use
        for _ in range(3):
            s.step()
        sims.append(s)
    a, b = sims
    tol = 1e-5 * bbox_diag(m.verts)
    assert a.persistent_status() == 0
    assert np.abs(a.positions_np() - b.positions_np()).max() <= tol
    assert (a.pprev - b.pprev).abs().max() <= tol
    # a velocity is a position difference over dt = 1/240 s
    assert (a.vel - b.vel).abs().max() <= 2 * 240 * tol


@pytest.mark.parametrize("quasi", [False, True])
def test_body_frames_match_launch_by_launch(quasi):
    """Pins, belly attachments with damping, fibres, SDF push-out; frame targets change between frames."""
    cfg = load_config("rlmusclev2_b200/configs/humanv2_synth.json")
    cfg["demo"]["collision"]["sdf_res"] = 64
    cfg["fine_iterations"] = 3
    cfg["quasi_static"] = quasi
    sc = humanv2_scene(seed=2, n_muscles=4, n_bones=4, target_tets=9000, fascia_tets=1500, box=(0.3, 0.3, 0.3))
    out = []
    for use in (True, False):
        s = MultiGridSim(cfg, scene=sc)
        s.use_persistent = use
        for f in (1, 2, 3):
            s.set_fiber_activation(sc.activation(f))
            s.step_frame(f)
        out.append(s.positions_np())
        assert s.persistent_status() == 0
    assert np.abs(out[0] - out[1]).max() <= max(1e-5 * bbox_diag(sc.verts), 1e-4)  # 1e-4 m: the frame gate of the parity tests
    assert np.abs(out[0] - sc.verts).max() > 1e-3


def test_batch_ranges_match_launch_by_launch():
    """Closed tile ranges of whole instances, each vertex's own SDF grid."""
    cfg = load_config("rlmusclev2_b200/configs/batched_256.json")
    sc = batched_box_scene(n_inst=6, seed=4, tets_lo=500, tets_hi=4000, sdf_res=32)
    out = []
    for use in (True, False):
        s = BatchSim(cfg, scene=sc)
        s._build_persist(int(np.bincount(s.layout.tile_group).max()) + 1)
        assert len(s._persist) > 1
        s.use_persistent = use
        for f in (1, 2, 3):
            s.step_frame_inputs(f)
        out.append(s.positions_np())
        assert s.persistent_status() == 0
    assert np.abs(out[0] - out[1]).max() <= 1e-4


@pytest.mark.parametrize("order", [("grid", "exchange", "grid"), ("exchange", "neighbour", "exchange", "grid")])
def test_kinds_of_persistent_launch_may_alternate(order):
    """The accumulator ring and the mailboxes keep their phases through each other's launches."""
    verts, tets, table, mass, vf, act, tendon, deformed, prev = _mixed_problem()
    kw = dict(dt=1.0 / 240.0, contraction_ratio=0.4, fiber_stiffness_scale=3.0, v_fiber=vf, tet_tendonmask=tendon,
              mass=mass, device="cuda:0", tile_tets=64)
    a, b = XpbdSolver(verts, tets, table, **kw), XpbdSolver(verts, tets, table, **kw)
    b.use_persistent = False
    for s in (a, b):
        s.set_activation(act)
        s.set_positions(prev, also_prev=True)
        s.set_positions(deformed)
    ptr, idx = a._tile_neighbours()
    a._t_nbr_ptr, a._t_nbr_idx = torch.from_numpy(ptr).cuda(), torch.from_numpy(idx).cuda()
    for k, kind in enumerate(order):
        a.persistent_sync = kind
        ps = a._persist[0]
        nb = kind == "neighbour"
        ps.nbr_ptr = a._t_nbr_ptr.data_ptr() if nb else None
        ps.nbr_idx = a._t_nbr_idx.data_ptr() if nb else None
        ps.tile_cnt = a._t_cnt.data_ptr() if nb else None
        a._fused_iterations(k + 1)
        b._fused_iterations(k + 1)
    assert a.persistent_status() == 0
    assert np.abs(a.positions_np() - b.positions_np()).max() <= 1e-5 * bbox_diag(verts)


def test_mailbox_wait_gives_up_and_recovers():
    """A tile whose counter is ahead sends iteration numbers nobody waits for:
    the waits run out, the launch ends with the status bit, and after the
    reset the next launch is right again."""
    m = box_muscle(4, 4, 8)
    s = MuscleSim.from_procedural(m.verts, m.tets, m.fiber_per_tet, stopped=m.stopped, tile_tets=64, **BOX)
    ref = MuscleSim.from_procedural(m.verts, m.tets, m.fiber_per_tet, stopped=m.stopped, tile_tets=64, **BOX)
    s.synchronize()
    with torch.cuda.stream(s._stream):
        s._ex_cnt[1] += 4
    s._fused_iterations(2)
    assert s.persistent_status() & capi.STATUS_BARRIER_TIMEOUT
    s.reset()
    s.step()
    ref.step()
    assert s.persistent_status() == 0
    assert np.abs(s.positions_np() - ref.positions_np()).max() <= 1e-5 * bbox_diag(m.verts)


PRE, VEL, PIN = capi.OP_PREDICT, capi.OP_VELOCITY, capi.OP_PIN


def _mixed_solver(tile_tets=64, extra=None, **kw):
    """The mixed problem (ARAP, damped volume and SNH, fibres, damped attachments)
    with gravity and velocities.  extra = (verts, mass, attach rows, pins): vertices in no tet."""
    from rlmusclev2_b200.builder import ConstraintTable
    verts, tets, table, mass, vf, act, tendon, deformed, prev = _mixed_problem()
    pins = None
    if extra is not None:
        ev, em, rows, pins = extra(verts)
        verts, mass = np.concatenate([verts, ev]), np.concatenate([mass, em])
        vf = np.concatenate([vf, np.tile(np.float32([0, 0, 1]), (len(ev), 1))])
        deformed, prev = np.concatenate([deformed, ev]), np.concatenate([prev, ev])
        table = ConstraintTable.concat([table, rows]).sorted_by_type()
    s = XpbdSolver(verts, tets, table, mass=mass, v_fiber=vf, tet_tendonmask=tendon, device="cuda:0", dt=1.0 / 240.0,
                   contraction_ratio=0.4, fiber_stiffness_scale=3.0, tile_tets=tile_tets, gravity=(0.0, -9.8, 0.3),
                   veldamping=0.05, relaxation=0.5, pins=pins, **kw)
    s.set_activation(act)
    s.set_positions(prev, also_prev=True)
    s.set_positions(deformed)
    return s


def _substeps(s, n_sub, n_iters, pin=0):
    """n_sub substeps in one launch, or launch by launch; True: one launch."""
    if s._fused_substeps(n_sub, n_iters, PRE | pin, PRE | pin | VEL, VEL):
        return True
    for k in range(n_sub):
        s._vstep(PRE | pin | (VEL if k else 0))
        for _ in range(n_iters):
            s._fused_iteration()
    s._vstep(VEL)
    return False


def _same_state(a, b, scale):
    """Positions within 1e-5 of the scene's extent, velocities within that over the substep."""
    assert a.persistent_status() == 0 and b.persistent_status() == 0
    tol = 1e-5 * scale
    assert np.abs(a.positions_np() - b.positions_np()).max() <= tol
    assert (a.pprev - b.pprev).abs().max() <= tol
    assert (a.vel - b.vel).abs().max() <= 2 * 240 * tol


@pytest.mark.parametrize("n_sub,n_iters", [(1, 1), (3, 1), (2, 3)])
def test_damped_snh_frames_match_launch_by_launch(n_sub, n_iters):
    """The damped full constraint set with a vertex step between the substeps:
    its constraints read the previous positions that the step has replaced."""
    a, b = _mixed_solver(), _mixed_solver()
    b.use_persistent = False
    assert _substeps(a, n_sub, n_iters) and not _substeps(b, n_sub, n_iters)
    _same_state(a, b, bbox_diag(a.pos0_np))
    assert np.abs(a.positions_np() - a.pos0_np).max() > 1e-4


def _loose_vertices(verts):
    """Eleven vertices in no tet: free ones, attached ones, pinned ones (one pin not active)."""
    from rlmusclev2_b200.builder import create_attach_constraints
    n = verts.shape[0]
    rng = np.random.default_rng(9)
    ev = rng.uniform(-0.02, 0.06, size=(11, 3)).astype(np.float32)
    att = np.arange(n + 4, n + 7)
    rows = create_attach_constraints(att, ev[4:7] + np.float32(0.003), 0.001, 2e5, 0.1)
    has, act = np.zeros(n + 11, bool), np.zeros(n + 11, np.int32)
    has[n + 7:], act[n + 7:] = True, [1, 1, 0, 1]
    has[3], act[3] = True, 1
    tgt = np.concatenate([verts, ev]) + np.float32(0.002)
    return ev, np.full(11, 0.01, np.float32), rows, (has, tgt, act)


@pytest.mark.parametrize("tile", [64, 4096])
def test_vertices_in_no_tet_take_part(tile):
    """Loose vertices fall, follow their attachments and pins in the one-launch frame as launch by launch."""
    a, b = _mixed_solver(tile, _loose_vertices), _mixed_solver(tile, _loose_vertices)
    assert a.layout.orphans.shape[0] == 11
    b.use_persistent = False
    for _ in range(2):
        assert _substeps(a, 3, 2, PIN) and not _substeps(b, 3, 2, PIN)
    _same_state(a, b, bbox_diag(a.pos0_np))
    x, x0 = a.positions_np()[-11:], a.pos0_np[-11:]
    moved = np.abs(x - x0).max(1)
    assert (moved > 1e-4).all()  # every loose vertex falls or is pulled
    np.testing.assert_allclose(x[[7, 8, 10]], x0[[7, 8, 10]] + np.float32(0.002), atol=1e-6)


@pytest.mark.parametrize("kind", ["mixed", "box"])
def test_shared_memory_layouts_are_bit_identical(kind):
    """Compile-time and run-time (tile_variant bit 4) layouts of the shared block."""
    out = []
    for variant in (0, 16):
        if kind == "mixed":
            s = _mixed_solver()
        else:
            m = box_muscle(5, 7, 9)
            s = MuscleSim.from_procedural(m.verts, m.tets, m.fiber_per_tet, stopped=m.stopped, tile_tets=100, **BOX)
        s._prm.tile_variant = variant
        assert _substeps(s, 4, 3)
        assert s.persistent_status() == 0
        out.append((s.positions_np(), s.pprev.numpy(), s.vel.numpy()))
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)


def test_tiles_past_the_compile_time_layout():
    """More than 768 vertices a tile: the run-time layout by necessity."""
    m = box_muscle(10, 10, 20)
    kw = dict(stopped=m.stopped, tile_tets=4096, **BOX)
    a = MuscleSim.from_procedural(m.verts, m.tets, m.fiber_per_tet, **kw)
    b = MuscleSim.from_procedural(m.verts, m.tets, m.fiber_per_tet, **kw)
    assert a.layout.max_tile_verts > 768
    b.use_persistent = False
    assert _substeps(a, 3, 2) and not _substeps(b, 3, 2)
    _same_state(a, b, bbox_diag(m.verts))


def test_iteration_numbers_pass_16_bits():
    """The mailboxes' 16-bit iteration number wraps; the counters go on."""
    a, b = _mixed_solver(), _mixed_solver()
    a.synchronize()
    with torch.cuda.stream(a._stream):
        a._ex_cnt.fill_(65530)
    for _ in range(3):
        assert _substeps(a, 2, 2) and _substeps(b, 2, 2)
    assert a.persistent_status() == 0
    assert int(a._ex_cnt.min()) == int(a._ex_cnt.max()) == 65542
    np.testing.assert_array_equal(a.positions_np(), b.positions_np())
