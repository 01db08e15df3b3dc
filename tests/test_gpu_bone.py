"""Bone-surface binding on the GPU (xpbd_bone_bind, xpbd_bone_slide_targets,
xpbd_bone_surface_pose) against the oracle, through the C-ABI, on three
capsule bones (1,536 faces, more than one shared-memory face chunk) and
6,000 query points 1-20 mm outside the surfaces.  Faces agree except at ties
(closest points on shared edges or corners), where either face is right; the
closest distance agrees to 1e-6 m, offsets (same face) and targets to 1e-5 m."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import oracle as O
from rlmusclev2_b200 import _capi as capi
from rlmusclev2_b200.meshgen import capsule_surface

pytestmark = pytest.mark.gpu


def _bones():
    parts = [capsule_surface([0.0, 0.0, 0.0], [0.0, 0.0, 1.0], 0.12, 0.02, 32, 8),
             capsule_surface([0.05, 0.0, 0.15], [1.0, 0.2, 0.1], 0.08, 0.015, 32, 8),
             capsule_surface([-0.04, 0.05, -0.1], [0.2, 1.0, 0.0], 0.06, 0.018, 32, 8)]
    vs, ts, vb, off = [], [], [], 0
    for b, (v, t) in enumerate(parts):
        vs.append(v)
        ts.append(t + off)
        vb.append(np.full(v.shape[0], b, np.int32))
        off += v.shape[0]
    return np.concatenate(vs), np.concatenate(ts).astype(np.int32), np.concatenate(vb)


def _d(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _p(t):
    return C.c_void_p(t.data_ptr())


def _v4(a):
    out = np.zeros((a.shape[0], 4), np.float32)
    out[:, :3] = a
    return out


def _cp(v, t, face, uv):
    A, B, Cc = v[t[face, 0]], v[t[face, 1]], v[t[face, 2]]
    return uv[:, :1] * A + uv[:, 1:] * B + (1 - uv.sum(1, keepdims=True)) * Cc


def test_bind_slide_and_pose_match_oracle():
    lib = capi.load()
    v, t, vb = _bones()
    assert t.shape[0] > 1024
    rng = np.random.default_rng(3)
    # muscle-like queries: 1-20 mm outside the bone surfaces, where the
    # closest point is well defined except at edge and corner ties
    f0 = rng.integers(0, t.shape[0], 6000)
    w = rng.random((6000, 2))
    w[w.sum(1) > 1] = 1 - w[w.sum(1) > 1]
    A, B, Cc = v[t[f0, 0]], v[t[f0, 1]], v[t[f0, 2]]
    nrm = np.cross(B - A, Cc - A)
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    q = (w[:, :1] * A + w[:, 1:] * B + (1 - w.sum(1, keepdims=True)) * Cc
         + rng.uniform(0.001, 0.02, (6000, 1)) * nrm).astype(np.float32)
    n, nbv, nbt = q.shape[0], v.shape[0], t.shape[0]
    q4, b4, tr_ = _d(_v4(q)), _d(_v4(v)), _d(t)
    face = torch.zeros(n, dtype=torch.int32, device="cuda")
    uv = torch.zeros((n, 2), dtype=torch.float32, device="cuda")
    loc = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    assert lib.xpbd_bone_bind(n, _p(q4), nbv, _p(b4), nbt, _p(tr_), C.c_float(1.0), _p(face), _p(uv), _p(loc),
                              None) == 0
    torch.cuda.synchronize()
    of, ouv, oloc = O.bone_bind(q, v, t, 1.0)
    gf, guv, gloc = face.cpu().numpy(), uv.cpu().numpy(), loc.cpu().numpy()
    same = gf == of
    print(f"bind: faces equal {same.mean():.4%}")
    # ties (closest points on shared edges or corners) let FP32 rounding pick
    # either face; both are right, so compare distances, and offsets where the
    # faces agree
    assert same.mean() > 0.9
    dg = np.linalg.norm(q - _cp(v, t, gf, guv), axis=1)
    do = np.linalg.norm(q - _cp(v, t, of, ouv), axis=1)
    assert np.abs(dg - do).max() < 1e-6
    assert (np.abs(gloc[same] - oloc[same]).max(1) < 1e-5).mean() > 0.999
    back, _, _, _ = O.bone_slide_targets(q, gf, guv, gf, guv, gloc, 0.004, 0, 1.0, v, t)
    assert np.abs(back - q).max() < 1e-5  # the GPU's binding reconstructs the query
    # pose the bones for a frame, then targets without and with re-projection
    T = np.zeros((3, 3, 4), np.float32)
    for b in range(3):
        th = 0.2 * (b + 1)
        T[b, :, :3] = [[np.cos(th), 0.0, np.sin(th)], [0.0, 1.0, 0.0], [-np.sin(th), 0.0, np.cos(th)]]
        T[b, :, 3] = [0.01 * b, 0.02, -0.01]
    posed = torch.zeros_like(b4)
    assert lib.xpbd_bone_surface_pose(nbv, _p(b4), _p(_d(vb)), 3, _p(_d(T.reshape(3, 12))), _p(posed), None) == 0
    torch.cuda.synchronize()
    vp = O.bone_pose(v, vb, T)
    assert np.abs(posed.cpu().numpy()[:, :3] - vp).max() < 1e-6
    moved = q + np.float32(0.003) * rng.normal(size=q.shape).astype(np.float32)
    m4 = _d(_v4(moved))
    for reproject in (0, 1):
        bf, buv, bl = face.clone(), uv.clone(), loc.clone()
        pin = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
        pin[:, 3] = 1.0
        assert lib.xpbd_bone_slide_targets(n, _p(m4), _p(face), _p(uv), _p(bf), _p(buv), _p(bl), C.c_float(0.004),
                                           reproject, C.c_float(1.0), nbv, _p(posed), nbt, _p(tr_), _p(pin), None,
                                           None) == 0
        torch.cuda.synchronize()
        ot, obf, obuv, obl = O.bone_slide_targets(moved, gf, guv, gf, guv, gloc, 0.004, reproject, 1.0, vp, t)
        g = pin.cpu().numpy()
        ok = np.abs(g[:, :3] - ot).max(1) < 1e-5
        print(f"reproject={reproject}: bind faces equal {(bf.cpu().numpy() == obf).mean():.4%}, "
              f"targets within 1e-5: {ok.mean():.4%}")
        assert (g[:, 3] == 1.0).all()
        # a tie can flip a slide at the slide_range boundary; nothing else may differ
        assert ok.mean() > 0.999

def _mesh_sim(sliding=False):
    from rlmusclev2_b200.mg import MultiGridSim, load_config
    from rlmusclev2_b200.meshgen import humanv2_scene
    cfg = load_config("rlmusclev2_b200/configs/humanv2_synth.json")
    cfg["demo"]["collision"]["sdf_res"] = 96
    cfg["target_mode"] = "mesh"
    cfg["use_sliding"] = sliding
    cfg["slide_interval"] = 1
    sc = humanv2_scene(seed=1, n_muscles=5, n_bones=4, target_tets=20000, fascia_tets=3000, box=(0.35, 0.35, 0.35))
    return MultiGridSim(cfg, scene=sc), sc


def test_multigrid_mesh_targets_match_oracle():
    """target_mode="mesh" in MultiGridSim: the start-frame targets reconstruct
    the rest pose, later frames' targets ride the posed capsule surfaces as the
    oracle's bind + follow gives them, and frames step to finite positions."""
    sim, sc = _mesh_sim()
    perm = sim.layout.perm
    sim._targets_kernel()
    sim.synchronize()
    got0 = sim._pin_tgt[:, :3].cpu().numpy()
    assert np.abs(got0 - sim.pos0_np[perm]).max() < 2e-6
    bv, bt, bvb = sc.bone_surface()
    start = O.bone_pose(bv, bvb, sc.bone_transforms(sim.start_frame).reshape(-1, 12))
    face, uv, loc = O.bone_bind(sim.pos0_np, start, bt, sim.slide_range + 1.0)
    for frame in (4, 9):
        sim.load_frame_targets(frame)
        sim._targets_kernel()
        sim.synchronize()
        posed = O.bone_pose(bv, bvb, sc.bone_transforms(frame).reshape(-1, 12))
        tgt, _, _, _ = O.bone_slide_targets(sim.pos0_np, face, uv, face, uv, loc, sim.slide_range, 0, 1.0, posed, bt)
        got = sim._pin_tgt[:, :3].cpu().numpy()
        err = np.abs(got - tgt[perm]).max()
        print(f"frame {frame}: |gpu - oracle| targets {err:.2e}")
        assert err < 2e-5
        np.testing.assert_allclose(sim._attach_tgt[:, :3].cpu().numpy(), got, atol=0)
    for frame in range(1, 4):
        sim.set_fiber_activation(sc.activation(frame))
        sim.step_frame(frame)
    assert np.isfinite(sim.positions_np()).all()


def test_multigrid_mesh_sliding_steps():
    """use_sliding: re-projection every frame on the eager path (no frame graph)."""
    sim, sc = _mesh_sim(sliding=True)
    assert not sim._fusable()
    for frame in range(1, 4):
        sim.set_fiber_activation(sc.activation(frame))
        sim.step_frame(frame)
    assert np.isfinite(sim.positions_np()).all()
    assert np.isfinite(sim._pin_tgt.cpu().numpy()).all()


def test_multigrid_mesh_from_bone_dir_matches_capsule_pose(tmp_path):
    """target_mode="mesh" with a bone_dir of bone_<frame>.geo files (the
    reference's GeoBoneSource): files holding, bit for bit, the capsule
    surfaces the device posed give the same run as the device pose."""
    from rlmusclev2_b200.geo import write_geo
    sim, sc = _mesh_sim()
    bdir = tmp_path / "bone"
    bdir.mkdir()
    tris = sim._bs_tris.cpu().numpy()
    for f in range(1, 5):
        sim.load_frame_targets(f)
        sim._pose_bone_surface()
        sim.synchronize()
        write_geo(bdir / f"bone_{f}.geo", sim._bs_pos4[:, :3].cpu().numpy(), tris=tris)
    sim2, _ = _mesh_sim()
    cfg2 = dict(sim2.cfg, bone_dir=str(bdir))
    from rlmusclev2_b200.mg import MultiGridSim
    sim2 = MultiGridSim(cfg2, scene=sc)
    sim, _ = _mesh_sim()
    assert sim2._bone_dir
    for frame in range(1, 5):
        a = sc.activation(frame)
        for s in (sim, sim2):
            s.set_fiber_activation(a)
            s.step_frame(frame)
    err = np.abs(sim.positions_np() - sim2.positions_np()).max()
    print(f"bone_dir run vs capsule-pose run: max |diff| {err:.2e} m")
    assert err < 1e-6


@pytest.mark.parametrize("n", [1, 9, 33, 6001, 37856, 37857, 151297])
def test_lanes_per_query_agree(n):
    """The lanes that share a query's faces depend on the query count (32 below
    37,857 queries, then 8): both find a closest face.

    Tolerance of the distance: about ten FP32 roundings of coordinates below
    0.5 m on either side, 2 * 10 * 0.5 * 6e-8 = 6e-7, taken as 1e-6."""
    lib = capi.load()
    v, t, _ = _bones()
    v, t = v[:400], t[(t < 400).all(1)][:389]  # a face count that 8 and 32 do not divide, over one chunk
    rng = np.random.default_rng(n)
    q = (v[rng.integers(0, 400, n)] + rng.normal(scale=0.01, size=(n, 3))).astype(np.float32)
    q[0] = v[t[0, 0]]  # on a vertex: several faces at distance zero, the lowest index wins
    reach = 0.01
    face = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    uv = torch.full((n, 2), -7.0, device="cuda")
    loc = torch.full((n, 4), -7.0, device="cuda")
    q4, b4, td = _d(_v4(q)), _d(_v4(v)), _d(t)
    assert lib.xpbd_bone_bind(n, _p(q4), v.shape[0], _p(b4), t.shape[0], _p(td), C.c_float(reach), _p(face), _p(uv),
                              _p(loc), None) == 0
    torch.cuda.synchronize()
    gf, guv, gloc = face.cpu().numpy(), uv.cpu().numpy().astype(np.float64), loc.cpu().numpy()
    v64 = v.astype(np.float64)
    pick = rng.permutation(n)[:2000]
    pick[0] = 0
    of, ouv, _ = O.bone_bind(q[pick], v, t, 1.0)
    d_or = np.linalg.norm(q[pick] - _cp(v64, t, of, ouv.astype(np.float64)), axis=1)
    found = d_or < reach - 1e-6
    d_gpu = np.linalg.norm(q[pick] - _cp(v64, t, gf[pick], guv[pick]), axis=1)
    assert np.abs(d_gpu - d_or)[found].max() <= 1e-6
    none = d_or > reach + 1e-6
    assert (gf[pick][none] == 0).all() and (guv[pick][none] == 0).all() and (gloc[pick][none] == 0).all()
    assert gf[0] == np.nonzero((t == t[0, 0]).any(1))[0][0]


def test_more_queries_than_32_bit_threads():
    """2^29 + 64 queries of one face: eight lanes each are more threads than 32
    bits count, and every query is answered all the same (24 GB of buffers)."""
    lib = capi.load()
    n = 2**29 + 64
    if torch.cuda.get_device_properties(0).total_memory < 40e9:
        pytest.skip("needs 24 GB")
    q4 = torch.zeros((n, 4), device="cuda")
    q4[:, 2] = 0.5
    b4, td = _d(_v4(np.float32([[-1, -1, 0], [3, -1, 0], [-1, 3, 0]]))), _d(np.int32([[0, 1, 2]]))
    face = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    uv = torch.full((n, 2), -7.0, device="cuda")
    loc = torch.full((n, 4), -7.0, device="cuda")
    torch.cuda.synchronize()
    assert lib.xpbd_bone_bind(n, _p(q4), 3, _p(b4), 1, _p(td), C.c_float(1.0), _p(face), _p(uv), _p(loc), None) == 0
    torch.cuda.synchronize()
    assert int((face != 0).sum()) == 0
    for k in (0, 2**28, 2**29 - 1, 2**29, n - 1):
        assert abs(float(loc[k, 2]) - 0.5) < 1e-6 and float(uv[k, 0]) > 0.0
    del q4, face, uv, loc
    torch.cuda.empty_cache()


@pytest.mark.parametrize("n,nf", [(24_000, 24), (24_999, 24), (25_000, 24), (60_000, 59), (60_000, 61)])
def test_few_faces_agree_with_many_lanes(n, nf):
    """One lane per query where the faces are few against the queries: the same
    faces, coordinates and offsets, bit for bit, as the same queries get in
    small calls (32 lanes), in the bindings and in the re-projection."""
    lib = capi.load()
    v, t, _ = _bones()
    t = np.ascontiguousarray(t[:nf])
    rng = np.random.default_rng(nf)
    q4 = _d(_v4((v[t[rng.integers(0, nf, n), 0]] + rng.normal(scale=0.01, size=(n, 3))).astype(np.float32)))
    b4, td = _d(_v4(v)), _d(t)
    nv, far = v.shape[0], C.c_float(0.012)

    def buffers():
        return (torch.full((n,), -7, dtype=torch.int32, device="cuda"), torch.full((n, 2), -7.0, device="cuda"),
                torch.full((n, 4), -7.0, device="cuda"), torch.full((n,), -7.0, device="cuda"),
                torch.full((n,), -7, dtype=torch.int32, device="cuda"))

    def run(step):
        face, uv, loc, gap, ok = buffers()
        sface, suv, pin = torch.empty_like(face), torch.empty_like(uv), torch.zeros_like(loc)
        moved = (q4 + torch.tensor([0.003, -0.002, 0.001, 0.0], device="cuda")).contiguous()
        for k in range(0, n, step):
            m = min(step, n - k)
            assert lib.xpbd_bone_bind(m, _p(q4[k:]), nv, _p(b4), nf, _p(td), far, _p(face[k:]), _p(uv[k:]), _p(loc[k:]),
                                      None) == 0
        bf, buv, bl = face.clone(), uv.clone(), loc.clone()
        for k in range(0, n, step):
            m = min(step, n - k)
            assert lib.xpbd_bone_slide_targets(m, _p(moved[k:]), _p(face[k:]), _p(uv[k:]), _p(bf[k:]), _p(buv[k:]),
                                               _p(bl[k:]), C.c_float(0.004), 1, far, nv, _p(b4), nf, _p(td),
                                               _p(pin[k:]), None, None) == 0
            assert lib.xpbd_surface_bind(m, _p(q4[k:]), nv, _p(b4), nf, _p(td), far, _p(sface[k:]), _p(suv[k:]),
                                         _p(gap[k:]), _p(ok[k:]), None) == 0
        torch.cuda.synchronize()
        return face, uv, loc, bf, buv, bl, pin, sface, suv, gap, ok

    whole, parts = run(n), run(2000)
    assert 0 < int(whole[-1].sum()) < n  # some within reach, some not
    for a, b in zip(whole, parts):
        assert torch.equal(a, b)


def _slide_sim(interval, cls=None, **over):
    from rlmusclev2_b200.mg import MultiGridSim, load_config
    from rlmusclev2_b200.meshgen import humanv2_scene
    cfg = load_config("rlmusclev2_b200/configs/humanv2_synth.json")
    cfg["demo"]["collision"]["sdf_res"] = 64
    cfg.update(target_mode="mesh", use_sliding=True, slide_interval=interval, fine_iterations=3, **over)
    sc = humanv2_scene(seed=2, n_muscles=4, n_bones=4, target_tets=9000, fascia_tets=1500, box=(0.3, 0.3, 0.3))
    return (cls or MultiGridSim)(cfg, scene=sc), sc


def _slide_state(sim):
    sim.synchronize()
    return [sim.positions_np(), sim._bind_face.cpu().numpy(), sim._bind_uv.cpu().numpy(), sim._local4.cpu().numpy(),
            sim._pin_tgt.cpu().numpy()]


@pytest.mark.parametrize("interval", [1, 2, 3])
def test_sliding_graphs_match_eager_launches_and_the_phase_program(interval):
    """Sliding frames replayed from their graphs (two when only some frames
    re-project) against the same launches issued eagerly, bit for bit (the
    sums between tiles are integers), and against the phase program of unfused
    primitives: positions within 1e-4 m, the frame gate of the parity tests
    (sums in another order; the faces are not compared there, since noise of
    3e-8 m on the positions gives one bound vertex in ten another of two faces
    that share its closest point)."""
    graph, sc = _slide_sim(interval)
    eager, _ = _slide_sim(interval)
    phase, _ = _slide_sim(interval)
    eager.use_graphs = False
    phase.build_program()
    moved = 0
    for frame in range(1, 8):
        before = graph._bind_uv.clone()
        for s in (graph, eager, phase):
            s.set_fiber_activation(sc.activation(frame))
            s.step_frame(frame)
        a, b, c = (_slide_state(s) for s in (graph, eager, phase))
        moved += int((graph._bind_uv != before).any())
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)
        assert np.abs(a[0] - c[0]).max() <= 1e-4
    assert set(graph._graphs) == {("frame", True)} | ({("frame", False)} if interval > 1 else set())
    # the re-projecting frames move the binding, the others and frame 1 (the pose it was bound in) do not
    assert moved == len(range(1, 8, interval)) - 1
    assert np.abs(a[0] - sc.verts).max() > 1e-3


def _no_slide(s):
    s.slide_range = 0.0


def _more_iterations(s):
    s.fine_iters = 5


def _fewer_substeps(s):
    s.nsubsteps = 6


def _soft_pin(s):
    s.presubframe_pintotarget = 0.25


def _heavier(s):
    s._prm.gravity[1] = -9.8


def _wide_push_out(s):
    # the muscles lie 31 mm off the bones at least
    s.collision_solvers[0].band = 0.08
    s.collision_solvers[0]._s.contact_offset = 0.04


@pytest.mark.parametrize("change", [_no_slide, _more_iterations, _fewer_substeps, _soft_pin, _heavier,
                                    _wide_push_out])
def test_sliding_frames_follow_their_parameters(change):
    """A parameter set between two sliding frames counts from the next frame
    on, captured or not."""
    graph, sc = _slide_sim(2)
    eager, _ = _slide_sim(2)
    kept, _ = _slide_sim(2)
    eager.use_graphs = False
    for frame in range(1, 7):
        if frame == 4:
            change(graph)
            change(eager)
        for s in (graph, eager, kept):
            s.set_fiber_activation(sc.activation(frame))
            s.step_frame(frame)
        if frame in (1, 2, 4):
            captured = graph._graphs[("frame", frame % 2 == 1)].value
        elif frame == 6:  # captured once per change, not every frame
            assert graph._graphs[("frame", False)].value == captured
    for x, y in zip(_slide_state(graph), _slide_state(eager)):
        np.testing.assert_array_equal(x, y)
    assert np.abs(_slide_state(graph)[0] - _slide_state(kept)[0]).max() > 0


def test_sliding_frames_start_from_empty_sums():
    """Corrections left by an unfused solve do not enter the next captured frame."""
    sims = [_slide_sim(1)[0] for _ in range(2)]
    sc = sims[0].scene
    for s in sims:
        s.use_persistent = False  # tile pass and boundary launch per iteration, through the global accumulator
    noise = np.random.default_rng(0).normal(scale=0.005, size=sc.verts.shape).astype(np.float32)
    for frame in range(1, 4):
        if frame == 3:  # corrections of millimetres, for positions that are put back
            x = sims[0].positions_np()
            sims[0].set_positions(x + noise)
            sims[0].solve_constraints()
            assert float(sims[0].dP.abs().max()) > 1e-3
            sims[0].set_positions(x)
        for s in sims:
            s.set_fiber_activation(sc.activation(frame))
            s.step_frame(frame)
    a, b = (s.positions_np() for s in sims)
    print("difference", np.abs(a - b).max())
    assert np.abs(a - b).max() <= 1e-4  # boundary sums are float atomics here


def test_sliding_frames_run_a_replaced_phase_program():
    """A subclass's own phases run, frame after frame."""
    from rlmusclev2_b200.mg import MultiGridSim

    class Counting(MultiGridSim):
        calls = 0

        def update_velocities(self):
            self.calls += 1
            super().update_velocities()

    sim, sc = _slide_sim(1, cls=Counting)
    for frame in (1, 2):
        sim.set_fiber_activation(sc.activation(frame))
        sim.step_frame(frame)
    assert sim.calls == 2 * sim.nsubsteps


def test_sliding_frames_are_captured_once(monkeypatch):
    """Nothing that frames leave behind counts as a changed parameter."""
    sim, sc = _slide_sim(1)
    released = []
    release = sim.release_graphs
    monkeypatch.setattr(sim, "release_graphs", lambda: released.append(sim.step_cnt) or release())
    for frame in range(1, 6):
        sim.set_fiber_activation(sc.activation(frame))
        sim.step_frame(frame)
        sim.positions_np()
        sim.metrics()
    assert not released


def test_sliding_multigrid_follows_its_switch():
    """use_multigrid set to False between sliding frames leaves the V-cycle out, captured or not."""
    over = dict(use_multigrid=True, mg_coarse_iters=2)
    graph, sc = _slide_sim(1, **over)
    eager, _ = _slide_sim(1, **over)
    kept, _ = _slide_sim(1, **over)
    eager.use_graphs = False
    for frame in range(1, 6):
        if frame == 4:
            graph.use_multigrid = eager.use_multigrid = False
        for s in (graph, eager, kept):
            s.set_fiber_activation(sc.activation(frame))
            s.step_frame(frame)
    a, b, c = (s.positions_np() for s in (graph, eager, kept))
    assert np.isfinite(a).all()
    assert np.abs(a - b).max() <= 1e-4  # the restriction's sums are float atomics
    assert np.abs(a - c).max() > 1e-4
