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
