"""The kinds of persistent iteration launch (XpbdEngine.persistent_sync and the
prefetch instance, tile_variant 4) against the oracle and the per-iteration
launches.

"exchange" runs xpbd_frame_persistent; "grid", and any kind with tile_variant 4,
xpbd_iterate_persistent over the three-slot accumulator ring, which stays the
path where the mailboxes do not fit.  The gates are those of
test_gpu_persistent.py: 1e-5 x bbox diagonal."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from rlmusclev2_b200.engine import XpbdSolver
from rlmusclev2_b200.mg import MultiGridSim, load_config
from rlmusclev2_b200.meshgen import humanv2_scene
from tests._cases import bbox_diag
from tests.test_gpu_parity import _mixed_problem, _oracle_table

pytestmark = pytest.mark.gpu

KINDS = [("exchange", 0), ("grid", 0), ("grid", 4), ("exchange", 4)]


def _launches(sim, monkeypatch):
    """Names of the persistent entry points called from here on."""
    names = []
    lib = sim._lib

    class Lib:
        def __getattr__(self, name):
            fn = getattr(lib, name)
            if name in ("xpbd_frame_persistent", "xpbd_iterate_persistent"):
                names.append(name)
            return fn

    monkeypatch.setattr(sim, "_lib", Lib())
    return names


@pytest.mark.parametrize("sync,variant", KINDS)
@pytest.mark.parametrize("n_iters", [1, 3])
def test_mixed_constraints_vs_oracle(sync, variant, n_iters, monkeypatch):
    verts, tets, table, mass, vf, act, tendon, deformed, prev = _mixed_problem()
    kw = dict(dt=1.0 / 240.0, contraction_ratio=0.4, fiber_stiffness_scale=3.0)
    sim = XpbdSolver(verts, tets, table, mass=mass, v_fiber=vf, tet_tendonmask=tendon, device="cuda:0",
                     tile_tets=64, **kw)
    sim.persistent_sync = sync
    sim._prm.tile_variant = variant
    sim.set_activation(act)
    sim.set_positions(prev, also_prev=True)
    sim.set_positions(deformed)
    names = _launches(sim, monkeypatch)
    _, B, _, _ = O.precompute_rest(verts, tets, 1060.0, "f32")
    o = O.OracleSolver(verts, tets, _oracle_table(table), mass, np.zeros(len(verts), np.int32), B,
                       gravity_vec=(0, 0, 0), v_fiber=vf, activation=act, tendonmask=tendon, prec="f32", **kw)
    o.pos[:] = deformed
    o.pprev[:] = prev
    for _ in range(n_iters):
        o.project()
        o.apply_dP()
    sim._fused_iterations(n_iters)
    got = sim.positions_np()
    assert sim.persistent_status() == 0
    assert set(names) == {"xpbd_frame_persistent" if (sync, variant) == ("exchange", 0) else "xpbd_iterate_persistent"}
    tol = 1e-5 * bbox_diag(verts)
    assert np.abs(o.pos - deformed).max() > 10 * tol
    assert np.abs(got - o.pos).max() <= tol


@pytest.mark.parametrize("sync,variant", KINDS)
def test_humanv2_small_matches_per_iteration_path(sync, variant):
    """20 iterations in launches of 7 and 13; the ring's phase goes on across them."""
    cfg = load_config("rlmusclev2_b200/configs/humanv2_synth.json")
    cfg["demo"]["collision"]["sdf_res"] = 96
    sc = humanv2_scene(seed=1, n_muscles=5, n_bones=4, target_tets=20000, fascia_tets=3000, box=(0.35, 0.35, 0.35))
    sim = MultiGridSim(cfg, scene=sc)
    sim.persistent_sync = sync
    frame = 6
    sim.set_fiber_activation(sc.activation(frame))
    sim.load_frame_targets(frame)
    sim._targets_kernel()
    rng = np.random.default_rng(5)
    x = (sc.verts + rng.normal(scale=0.001, size=sc.verts.shape)).astype(np.float32)
    sim.set_positions(x)
    start = sim._pos4.clone()
    for _ in range(20):
        sim._fused_iteration()
    ref = sim.positions_np()
    with torch.cuda.stream(sim._stream):
        sim._pos4.copy_(start)
    sim._prm.tile_variant = variant
    sim._fused_iterations(7)
    sim._fused_iterations(13)
    got = sim.positions_np()
    assert sim.persistent_status() == 0
    tol = 1e-5 * bbox_diag(sc.verts)
    assert np.abs(ref - x).max() > 10 * tol
    assert np.abs(got - ref).max() <= tol
    if (sync, variant) != ("exchange", 0):
        assert int(sim._psync[2].item()) == 20 % 3


@pytest.mark.parametrize("case", ["tangled", "flat"])
def test_deferred_svd_pass_is_bit_identical_in_the_ring_pass(case):
    """tile_variant bit 6 in xpbd_iterate_persistent ("tangled": many inverted
    tets; "flat": more than the deferred list holds)."""
    verts, tets, table, mass, vf, act, tendon, deformed, prev = _mixed_problem()
    rng = np.random.default_rng(7)
    if case == "tangled":
        deformed = verts + rng.normal(scale=0.004, size=verts.shape).astype(np.float32)
    else:
        deformed = (verts * np.array([1.0, 1.0, 1e-6], np.float32)).astype(np.float32)
    out = []
    for tv in (0, 64):
        sim = XpbdSolver(verts, tets, table, mass=mass, v_fiber=vf, tet_tendonmask=tendon, device="cuda:0",
                         tile_tets=512 if case == "flat" else 64, dt=1.0 / 240.0, contraction_ratio=0.4,
                         fiber_stiffness_scale=3.0)
        sim.persistent_sync = "grid"
        sim._prm.tile_variant = tv
        sim.set_activation(act)
        sim.set_positions(prev, also_prev=True)
        sim.set_positions(deformed)
        sim._fused_iterations(3)
        assert sim.persistent_status() == 0
        out.append(sim.positions_np())
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1])
    assert np.abs(out[0] - deformed).max() > 0
