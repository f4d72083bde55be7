"""Host buffers that kernels read and write in place or through staged copies
(field batches, particle records): what is refused, and that every way gives
the same bytes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")
import test_particle_gb300.workloads as wl  # noqa: E402

DT = 0.02


def _setup(steps=20):
    dom = tp.Domain()
    dom.xmax = dom.ymax = dom.zmax = 1.0
    dom.tmax = (steps + 0.5) * DT
    tp.configure(system_type=tp.SYS_FORCEFREE, dom=dom, abc=(1.0, 0.7, 0.4), lambda0=2 * np.pi)
    tp.set_spectrum(50, 1e-3, 1e2)


def _track(prec, n, p0, p, out, nst=None, steps=20):
    esp, ese, ds, rem = np.zeros(50), np.zeros(50), np.zeros(8), np.zeros(1, np.int32)
    return tp.lib().tp_track_host_to(C.c_int(prec), C.c_int(n), C.c_double(DT), C.c_int(1), C.c_int(50), tp._ptr(p0),
                                     tp._ptr(p), tp._ptr(out), tp._ptr(nst), tp._ptr(esp), tp._ptr(ese), tp._ptr(ds),
                                     tp._ptr(rem), None)


def test_null_buffers_are_refused():
    """Refused on the host, with a message and no error left for the next call."""
    _setup()
    L = tp.lib()
    x, e, f = np.zeros((4, 4)), np.zeros((4, 6)), np.zeros((4, 6), np.float32)
    p = wl.shell_particles(4, 0.5, (0, 0, 0), (1, 1, 1), 1)
    s = tp.Session(4)
    h = C.c_void_p(s.h)
    for call in (lambda: L.tp_get_emf_batch(4, None, tp._ptr(e)), lambda: L.tp_get_emf_batch(4, tp._ptr(x), None),
                 lambda: L.tp_get_emf_mixed_batch(4, None, tp._ptr(f)),
                 lambda: L.tp_get_emf_mixed_batch(4, tp._ptr(x), None),
                 lambda: L.tp_session_load(h, None, tp._ptr(p)), lambda: L.tp_session_load(h, tp._ptr(p), None),
                 lambda: L.tp_session_load(h, None, None), lambda: _track(tp.PREC_FP64, 4, None, None, p),
                 lambda: _track(tp.PREC_FP64, 4, p, None, p), lambda: _track(tp.PREC_FP64, 4, None, p, p)):
        assert call() == -1
        assert b"null" in L.tp_last_error()
        L.tp_clear_status()
    assert np.isfinite(tp.get_emf(x)).all()
    s.load(p)
    assert _track(tp.PREC_FP64, 4, p, p, None) == 0  # no particles wanted back
    assert tp.device_status() == 0


def test_record_arrays_of_other_lengths():
    """Fewer records than particles are refused (the device would read past the
    array); more are returned behind the tracked ones as they came."""
    _setup()
    p = wl.shell_particles(8, 0.5, (0, 0, 0), (1, 1, 1), 1)
    with pytest.raises(ValueError):
        tp.track(p, DT, 1, 50, ptl=p[:7])
    s = tp.Session(8)
    with pytest.raises(ValueError):
        s.load(p[:7])
    with pytest.raises(ValueError):
        s.load(p, p[:7])
    few = tp.track(p[:5], DT, 1, 50, ptl=p)
    assert few["ptl"].shape == (8,) and len(few["nsteps"]) == 5
    assert few["ptl"][5:].tobytes() == p[5:].tobytes()
    assert few["ptl"][:5].tobytes() == tp.track(p[:5], DT, 1, 50)["ptl"].tobytes()


@pytest.mark.parametrize("n", [1, 129, 20000])
@pytest.mark.parametrize("shift", [0, 3])
def test_fields_written_over_their_points(n, shift):
    """A result that overlaps the points is what one in its own buffer is."""
    _setup()
    rng = np.random.default_rng(n)
    pts = rng.random((n, 4))
    want = tp.get_emf(pts)
    for at, to in ((0, shift), (shift, 0)):
        buf = np.zeros(6 * n + 8)
        buf[at:at + 4 * n] = pts.ravel()
        tp.check(tp.lib().tp_get_emf_batch(C.c_int(n), tp._ptr(buf[at:]), tp._ptr(buf[to:])))
        assert buf[to:to + 6 * n].tobytes() == want.tobytes()
    want = tp.get_emf_mixed(pts[:, :3])
    buf = np.zeros(3 * n + 8)
    buf[:3 * n] = pts[:, :3].ravel()
    out = buf.view(np.float32)[shift:shift + 6 * n]
    tp.check(tp.lib().tp_get_emf_mixed_batch(C.c_int(n), tp._ptr(buf), tp._ptr(out)))
    assert out.tobytes() == want.tobytes()


def test_failed_run_leaves_the_outputs():
    """A refused run leaves the records and step counts as they were, and an
    output that lies over part of the inputs is written after they are read
    (its pages are mapped, but not changed, while the run is going)."""
    _setup()
    n = 5000
    p = wl.shell_particles(n, 0.5, (0, 0, 0), (1, 1, 1), 1)
    out = np.frombuffer(np.random.default_rng(1).bytes(88 * n), dtype=tp.PARTICLE_DTYPE).copy()
    nst = np.arange(n, dtype=np.int32) + 1000
    keep = out.copy(), nst.copy()
    assert _track(7, n, p, p, out, nst) == -1  # no such precision
    tp.lib().tp_clear_status()
    assert out.tobytes() == keep[0].tobytes() and nst.tobytes() == keep[1].tobytes()
    # the same outputs over part of the inputs: read before they are written
    both = np.zeros(2 * n, dtype=tp.PARTICLE_DTYPE)
    both[:n] = p
    want = np.zeros(n, dtype=tp.PARTICLE_DTYPE)
    assert _track(tp.PREC_MIXED, n, p, p, want, nst) == 0
    shifted = both[n // 2:n // 2 + n]
    assert _track(tp.PREC_MIXED, n, both, both, shifted, nst) == 0
    assert shifted.tobytes() == want.tobytes()


@pytest.mark.parametrize("n", [87381, 87382])
def test_field_batches_around_the_size_of_results_in_place(n):
    """48 bytes a point: 4 MB of results and one more point."""
    _setup()
    rng = np.random.default_rng(7)
    pts = rng.random((n, 4))
    out = tp.get_emf(pts)
    pick = np.r_[0:300, n - 300:n]
    assert np.array_equal(tp.get_emf(pts[pick]), out[pick])
    mixed = tp.get_emf_mixed(np.r_[pts, pts][:, :3])  # 24 bytes a point
    assert mixed[:n].tobytes() == mixed[n:].tobytes()
    assert np.array_equal(tp.get_emf_mixed(pts[pick, :3]), mixed[pick])


@pytest.mark.parametrize("n", [47662, 47663])
def test_records_around_the_size_of_results_in_place(n):
    """88 bytes a particle, fetched from a session and from a whole run."""
    _setup()
    p = wl.shell_particles(n, 0.5, (0, 0, 0), (1, 1, 1), 1)
    r = tp.track(p, DT, 1, 50, precision=tp.PREC_MIXED)
    s = tp.Session(n)
    s.load(p)
    s.track(DT, 1, 50, tp.PREC_MIXED)
    f = s.fetch(1, 50, 1)
    assert f["ptl"].tobytes() == r["ptl"].tobytes()
    assert np.array_equal(f["nsteps"], r["nsteps"])
    few = tp.track(p[n - 100:], DT, 1, 50, precision=tp.PREC_MIXED)
    assert few["ptl"].tobytes() == r["ptl"][n - 100:].tobytes()


@pytest.mark.parametrize("n", [190650, 190651])
def test_records_around_the_size_of_mapped_results_in_place(n):
    """A run's own result: 16 MB and one more particle."""
    _setup()
    p = wl.shell_particles(n, 0.5, (0, 0, 0), (1, 1, 1), 1)
    r = tp.track(p, DT, 1, 50, precision=tp.PREC_MIXED)
    for a in (0, n - 500):
        assert tp.track(p[a:a + 500], DT, 1, 50, precision=tp.PREC_MIXED)["ptl"].tobytes() == r["ptl"][a:a + 500].tobytes()


def _at(nbytes, off):
    """A byte array of nbytes that starts `off` bytes past a 64-byte boundary."""
    raw = np.zeros(nbytes + 128, np.uint8)
    a = -raw.ctypes.data % 64 + off
    return raw[a:a + nbytes]


@pytest.mark.parametrize("n", [1, 129, 60001])
@pytest.mark.parametrize("src,dst", [(4, 0), (0, 4), (4, 4)])
def test_misaligned_buffers_take_the_copies(n, src, dst):
    """Doubles on 4-byte boundaries (and floats on 2-byte ones), which no kernel
    reads or writes: the same bytes through staged copies."""
    _setup()
    L = tp.lib()
    rng = np.random.default_rng(n)
    pts = rng.random((n, 4))
    x, e = _at(32 * n, src), _at(48 * n, dst)
    x[:] = pts.view(np.uint8).ravel()
    tp.check(L.tp_get_emf_batch(C.c_int(n), tp._ptr(x), tp._ptr(e)))
    assert e.tobytes() == tp.get_emf(pts).tobytes()
    xm, em = _at(24 * n, src), _at(24 * n, dst // 2)
    xm[:] = np.ascontiguousarray(pts[:, :3]).view(np.uint8).ravel()
    tp.check(L.tp_get_emf_mixed_batch(C.c_int(n), tp._ptr(xm), tp._ptr(em)))
    assert em.tobytes() == tp.get_emf_mixed(pts[:, :3]).tobytes()
    p = wl.shell_particles(n, 0.5, (0, 0, 0), (1, 1, 1), 1)
    other = p.copy()
    other["t"] = 0.5
    want = tp.track(p, DT, 1, 50, precision=tp.PREC_MIXED, ptl=other)
    p0, p1, out = _at(88 * n, src), _at(88 * n, src), _at(88 * n, dst)
    p0[:], p1[:] = p.view(np.uint8), other.view(np.uint8)
    assert _track(tp.PREC_MIXED, n, p0, p1, out) == 0
    assert out.tobytes() == want["ptl"].tobytes()
    # one buffer in and out, initial and current records the same
    want = tp.track(p, DT, 1, 50, precision=tp.PREC_MIXED)
    esp, ese, ds, rem, nst = np.zeros(50), np.zeros(50), np.zeros(8), np.zeros(1, np.int32), np.zeros(n, np.int32)
    tp.check(L.tp_track_host(C.c_int(tp.PREC_MIXED), C.c_int(n), C.c_double(DT), C.c_int(1), C.c_int(50), tp._ptr(p0),
                             tp._ptr(p0), tp._ptr(nst), tp._ptr(esp), tp._ptr(ese), tp._ptr(ds), tp._ptr(rem), None))
    assert p0.tobytes() == want["ptl"].tobytes() and np.array_equal(nst, want["nsteps"])
    assert np.array_equal(esp, want["espect"].ravel())
