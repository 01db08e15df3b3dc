"""Host-side handling of the device status words (no GPU needed).

The persistent pass's grid barrier sets XPBD_STATUS_BARRIER_TIMEOUT when a
wait gives up and the bit is sticky: every later barrier of later launches
gives up early too.  The tile passes set XPBD_STATUS_ACC_RANGE when a tet's
corrections leave the fixed-point range (or are not finite).  The engine
copies the words behind every frame and raises at the next frame or
synchronising read; these tests pin which bits are fatal.
"""
from rlmusclev2_b200 import _capi as capi
from rlmusclev2_b200.engine import XpbdEngine, status_error


def test_clean_words_pass():
    assert status_error(0, 0) is None


def test_dcd_overflow_bits_are_warnings_only():
    warn = capi.STATUS_PAIR_OVERFLOW | capi.STATUS_CONTACT_OVERFLOW | capi.STATUS_STACK_OVERFLOW
    assert status_error(0, warn) is None


def test_barrier_timeout_is_fatal():
    msg = status_error(capi.STATUS_BARRIER_TIMEOUT)
    assert msg is not None and "grid barrier" in msg and "cleared" in msg


def test_accumulator_range_is_fatal():
    msg = status_error(capi.STATUS_ACC_RANGE)
    assert msg is not None and "fixed-point" in msg


def test_dcd_sort_timeout_is_fatal():
    msg = status_error(0, capi.STATUS_BARRIER_TIMEOUT)
    assert msg is not None and "DCD" in msg


def test_all_fatal_bits_reported_together():
    msg = status_error(capi.STATUS_BARRIER_TIMEOUT | capi.STATUS_ACC_RANGE, capi.STATUS_BARRIER_TIMEOUT)
    assert msg.count(";") == 2


class _FrameEngine:
    """What _fused_substeps reads of an engine, with a library that counts launches."""
    use_persistent, _persist_fits, persistent_sync, n_cons = True, True, "exchange", 1
    fused_mode = capi.PROJECT_FUSED

    def __init__(self):
        self._prm, self._tiles, self._verts = capi.XpbdParams(), capi.XpbdTiles(), capi.XpbdVerts()
        self._exchange, self._persist, self._sdf, self._sp = capi.XpbdExchange(), [capi.XpbdPersist()] * 2, None, None
        self.launched = []
        self._lib = type("Lib", (), {"xpbd_frame_persistent": lambda _, p, t, v, ps, f, s: self.launched.append(
            (f._obj.n_sub, f._obj.n_iters)) or 0})()


def test_frames_that_one_launch_does_not_take_go_substep_by_substep():
    """No substeps, no iterations, or more iterations in all than one launch
    takes: nothing is launched and the caller runs the substeps one by one, as
    many iterations each as before."""
    for n_sub, n_iters, fits in ((10, 20, True), (1, 1 << 20, True), (0, 20, False), (3, 0, False),
                                 (2, (1 << 19) + 1, False), (10, 1 << 20, False), (1, (1 << 20) + 1, False)):
        e = _FrameEngine()
        assert XpbdEngine._fused_substeps(e, n_sub, n_iters, 0, 0, 0) is fits
        assert e.launched == ([(n_sub, n_iters)] * 2 if fits else [])


def test_few_iterations_by_themselves_take_the_ring():
    """The mailbox launch costs more to start than it saves on a few
    iterations; whoever chose another kind of launch keeps it."""
    from types import SimpleNamespace
    for n_tets, n_tiles, first in ((28_046, 439, 2), (256 * 444, 444, 2), (256 * 444 + 1, 444, 10), (470_478, 444, 10)):
        for sync in ("exchange", "grid", "neighbour"):
            taken = []
            e = SimpleNamespace(layout=SimpleNamespace(n_tets=n_tets, n_tiles=n_tiles), persistent_sync=sync,
                                _ring_iterations=lambda n: taken.append("ring"),
                                _fused_iterations=lambda n: taken.append("fused"))
            for n in (1, first - 1, first, 20):
                XpbdEngine._jacobi_iterations(e, n)
            assert taken == (["ring", "ring", "fused", "fused"] if sync == "exchange" else ["fused"] * 4)
