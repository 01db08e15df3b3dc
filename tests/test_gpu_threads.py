"""Several engines at once: one thread and one stream each."""
import threading

import numpy as np
import pytest
import torch

from rlmusclev2_b200 import MuscleSim
from rlmusclev2_b200.cagenet import CageMLP
from rlmusclev2_b200.meshgen import box_muscle
from tests.test_gpu_frame import BOX

pytestmark = pytest.mark.gpu


def _in_threads(jobs):
    """Run the jobs at the same time; the first exception of any is raised."""
    errors, gate = [], threading.Barrier(len(jobs))

    def go(job):
        try:
            gate.wait(30)
            job()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=go, args=(j,)) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if errors:
        raise errors[0]


def _box(tile_tets=None, dims=(8, 8, 32)):
    m = box_muscle(*dims)
    return MuscleSim.from_procedural(m.verts, m.tets, m.fiber_per_tet, stopped=m.stopped, tile_tets=tile_tets, **BOX)


@pytest.mark.parametrize("sync", ["exchange", "grid"])
def test_threads_with_different_shared_memory(sync):
    """Two engines whose tiles need 60 and 66 KB of shared memory launch the
    same kernel instance from two threads: neither lowers the other's limit."""
    sims = [_box(2048), _box(3000)]
    for s in sims:
        s.use_graphs = False
        s.persistent_sync = sync
        s.synchronize()

    def run(s):
        def job():
            for _ in range(3000):
                s._fused_iterations(1)
        return job

    _in_threads([run(s) for s in sims])
    for s in sims:
        assert s.persistent_status() == 0
        assert np.isfinite(s.positions_np()).all()


def test_network_in_a_fresh_thread():
    """A thread whose first CUDA call is the network's: the launches bring the
    device's context along, for the tensor maps too."""
    net = CageMLP("cuda:0", 200, stream=torch.cuda.Stream())
    target = torch.ones((200, 3), device="cuda")
    torch.cuda.synchronize()
    _in_threads([lambda: net.forward(200, train=False)])
    _in_threads([lambda: net.forward(200)])
    _in_threads([lambda: net.backward(200, target)])
    torch.cuda.synchronize()
    assert int(net.status.item()) == 0
    assert float(net.loss.item()) == 600.0  # features and biases are zero, so are the outputs


@pytest.mark.parametrize("graphs", [True, False])
def test_two_simulators_at_once(graphs):
    """Two engines stepped and read by two threads on their own streams give,
    bit for bit, what each gives alone: the one-launch frames of one do not
    disturb the other's (their tiles wait for one another within a grid only)."""
    dims = [(8, 8, 32), (5, 7, 41)]
    alone = []
    for d in dims:
        s = _box(dims=d)
        s.use_graphs = graphs
        for _ in range(60):
            s.step()
        alone.append(s.positions_np())
    sims = [_box(dims=d) for d in dims]
    reads = [[], []]

    def run(k):
        def job():
            sims[k].use_graphs = graphs
            for f in range(60):
                sims[k].step()
                if f % 3 == 0:
                    reads[k].append(sims[k].positions_np())
        return job

    _in_threads([run(0), run(1)])
    for s, ref, r in zip(sims, alone, reads):
        assert s.persistent_status() == 0
        np.testing.assert_array_equal(s.positions_np(), ref)
        assert len({x.ctypes.data for x in r}) == len(r)  # every read an array of its own


def test_one_engine_read_by_two_threads():
    """positions_np from two threads on one engine: both read the same positions."""
    s = _box()
    for _ in range(3):
        s.step()
    ref = s.positions_np()
    out = [[], []]
    _in_threads([lambda k=k: out[k].extend(s.positions_np() for _ in range(50)) for k in (0, 1)])
    for x in out[0] + out[1]:
        np.testing.assert_array_equal(x, ref)


def test_positions_are_read_on_the_engines_own_device(monkeypatch):
    """The read-back launches its gather with the engine's stream, and so its
    device, current: the caller may have another one selected."""
    s = _box()
    s.step()
    lib, current = s._lib, []

    class Lib:
        def __getattr__(self, name):
            if name == "xpbd_gather":
                current.append(torch.cuda.current_stream() == s._stream)
            return getattr(lib, name)

    monkeypatch.setattr(s, "_lib", Lib())
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):  # what the caller queued on its own stream is waited for
        torch.cuda._sleep(20_000_000)
        s._pos4[:, :3] += 1.0
        x = s.positions_np()
    assert current == [True]
    np.testing.assert_array_equal(x, s._pos4[:, :3].cpu().numpy()[s.layout.inv])
