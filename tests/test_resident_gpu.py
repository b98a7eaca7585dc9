"""The resident kernel: runs of eight steps or more on grids that fit on chip are one launch.

The grid is cut into bricks that trade boundary rows through memory, so the shapes here are those
where a brick, a row of four-cell units or a column of planes ends early, down to one cell per brick
and up to the largest that fit.  Reference: the FP32 oracle, bit for bit.
"""
import numpy as np
import pytest

import oracle
import ptask_gb300 as P

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 2, 2), (1, 5, 3), (3, 1, 9), (4, 4, 4), (5, 160, 1), (31, 3, 152), (32, 32, 32), (33, 31, 29),
          (48, 40, 36), (127, 7, 5), (128, 13, 11), (401, 9, 10), (64, 64, 64), (89, 89, 89), (96, 96, 96), (128, 95, 71)]


def medium(pr, kind, rng):
    """`pr`'s dielectric boxes as they are, conducting, or every coefficient of every cell its own."""
    if kind == "lossy":
        inside = pr.Cb != pr.Cb.max()
        pr.Ca[inside] = np.float32(0.98)
        pr.Da[inside] = np.float32(0.99)
    elif kind == "graded":
        for c, scale in ((pr.Ca, 0.01), (pr.Cb, 0.5), (pr.Da, 0.01), (pr.Db, 0.5)):
            c *= 1 - np.float32(scale) * rng.random(c.shape, dtype=np.float32)
    return pr


@pytest.mark.parametrize("kind", ["boxes", "lossy", "graded"])
@pytest.mark.parametrize("shape", SHAPES)
def test_resident_runs_match_oracle(shape, kind):
    """Split runs (even and odd lengths: results land in either buffer), a waveform that ends mid-run, a launch per run."""
    rng = np.random.default_rng(sum(shape))
    parts = (8, 11, 9)
    pr = medium(P.Problem.generate(*shape, n_boxes=3, eps=(1, 10), box=(2, 20), steps=sum(parts) - 5, source_mode=2,
                                   seed=sum(shape)), kind, rng)
    f = P.random_fields(*shape, seed=90, scale=1e-2)
    ref = oracle.step_ext_f32(f, sum(parts), pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db, pr.src, pr.wave)
    with P.Solver(pr.params) as s:
        s.set_tiles(11, 0, 4, 4)
        s.set_problem(pr)
        s.set_fields(f)
        for n in parts:
            s.run(n)
            assert s.last_launches() == 1
        got = s.get_fields()
    for q in range(6):
        np.testing.assert_array_equal(got[q], ref[q], err_msg=f"{shape} {kind} {P.FIELDS[q]}")


def test_short_runs_resets_and_larger_grids_keep_their_kernel():
    """Runs under eight steps keep the step kernel; mixing both with a clock reset continues the same fields."""
    shape = (40, 33, 21)
    pr = P.Problem.generate(*shape, n_boxes=2, steps=0, seed=5, source_mode=0)
    f = P.random_fields(*shape, seed=91, scale=1e-2)
    ref = oracle.step_ext_f32(f, 3 + 9 + 4 + 8, pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db)
    with P.Solver(pr.params) as s:
        s.set_tiles(11, 5, 4, 4)
        s.set_problem(pr)
        s.set_fields(f)
        for n in (3, 9, 4, 8):
            s.run(n)
            assert (s.last_launches() == 1) == (n >= 8)
            s.reset_clock()
        got = s.get_fields()
    for q in range(6):
        np.testing.assert_array_equal(got[q], ref[q], err_msg=P.FIELDS[q])
    with P.Solver(P.reference_params(160, 160, 120)) as s:   # too large to fit on chip
        s.set_tiles(11, 0, 4, 4)
        s.run(8)
        assert s.last_launches() >= 8


def test_two_solvers_run_resident_launches_from_two_threads():
    """Each solver has its own exchange; runs queued from two threads on two streams stay independent."""
    import threading

    from ptask_gb300.device import Stream
    shape, steps = (60, 50, 40), 60
    out, errs = {}, []

    def work(k):
        try:
            pr = P.Problem.generate(*shape, n_boxes=3, steps=steps, seed=40 + k, source_mode=2)
            f = P.random_fields(*shape, seed=50 + k, scale=1e-2)
            st = Stream()
            with P.Solver(pr.params) as s:
                s.set_tiles(11, 0, 4, 4)
                s.set_problem(pr, stream=st.handle)
                for _ in range(3):
                    s.set_fields(f, stream=st.handle)
                    s.reset_clock()
                    s.run(steps, stream=st.handle)
                out[k] = (pr, f, s.get_fields(stream=st.handle))
            st.close()
        except Exception as e:   # noqa: BLE001 -- reported by the main thread
            errs.append(e)

    th = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errs, errs
    for pr, f, got in out.values():
        ref = oracle.step_ext_f32(f, steps, pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db, pr.src, pr.wave)
        for q in range(6):
            np.testing.assert_array_equal(got[q], ref[q], err_msg=P.FIELDS[q])


@pytest.mark.parametrize("shape,vacuum", [((89, 89, 89), False), ((64, 64, 64), True), ((33, 71, 50), False), ((400, 20, 21), True),
                                          ((700, 31, 31), False), ((1, 1, 1), False)])
def test_static_solve_runs_resident_where_its_scratch_fits(shape, vacuum):
    """ptk_fdtd_solve_static over the resident launch and, where its scratch does not fit ((700, 31, 31)), the step kernel."""
    import ctypes as C

    from ptask_gb300 import _lib
    from ptask_gb300.device import DeviceBuffer
    steps, V = 13, C.c_void_p
    pr = P.Problem.generate(*shape, n_boxes=3, eps=(1, 10), box=(2, 20), steps=9, source_mode=0 if vacuum else 2, seed=7)
    if vacuum:
        pr = P.Problem.vacuum(pr.params)
    else:
        medium(pr, "lossy", None)
    f = P.random_fields(*shape, seed=94, scale=1e-2)
    src = pr.src if pr.has_source else (-1, -1, -1)
    ref = oracle.step_ext_f32(f, steps, pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db, src, pr.wave)
    bufs = [DeviceBuffer.from_array(a) for a in f]
    coefs = [] if vacuum else [DeviceBuffer.from_array(a) for a in (pr.Ca, pr.Cb, pr.Da, pr.Db)]
    wave = DeviceBuffer.from_array(pr.wave) if pr.has_source else None
    for _ in range(2):   # the second call finds the first one's leftovers in the scratch
        for b, a in zip(bufs, f):
            b.upload(a)
        _lib.call("ptk_fdtd_solve_static", C.byref(pr.params), (V * 6)(*[b.ptr for b in bufs]),
                  *([c.ptr for c in coefs] if coefs else [None] * 4), *src, wave.ptr if wave else None,
                  int(pr.wave.size) if wave else 0, steps, None)
        _lib.call("ptk_device_sync")
        got = [b.download(a.shape) for b, a in zip(bufs, f)]
        for q in range(6):
            np.testing.assert_array_equal(got[q], ref[q], err_msg=f"{shape} {P.FIELDS[q]}")
    for b in bufs + coefs + ([wave] if wave else []):
        b.free()


def test_under_capture():
    """An allocation-free solve is captured and replayed; a solver's run is refused, on chip as by replayed graphs."""
    import ctypes as C

    from ptask_gb300 import _lib
    from ptask_gb300.device import DeviceBuffer, Stream
    V = C.c_void_p
    shape, steps = (30, 20, 24), 20
    p = P.reference_params(*shape)
    f = P.random_fields(*shape, seed=1, scale=1e-2)
    st = Stream()

    def solve(bufs):
        _lib.call("ptk_fdtd_solve_static", C.byref(p), (V * 6)(*[b.ptr for b in bufs]), *[None] * 4, -1, -1, -1, None, 0, steps,
                  st.handle)

    first, second = ([DeviceBuffer.from_array(a) for a in f] for _ in range(2))
    solve(first)
    st.sync()
    graph = V()
    _lib.call("ptk_capture_begin", st.handle)
    solve(second)
    _lib.call("ptk_capture_end", st.handle, C.byref(graph))
    _lib.call("ptk_graph_exec_launch", graph, st.handle, 1)
    st.sync()
    for q in range(6):
        np.testing.assert_array_equal(second[q].download(P.field_shape(q, *shape)), first[q].download(P.field_shape(q, *shape)))
    with P.Solver(p) as s:
        s.set_fields(f)
        s.run(steps, st.handle)
        st.sync()
        before = s.get_fields()
        _lib.call("ptk_capture_begin", st.handle)
        with pytest.raises(_lib.PtkError):
            s.run(steps, st.handle)
        _lib.call("ptk_capture_end", st.handle, C.byref(graph))
        for a, b in zip(s.get_fields(), before):
            np.testing.assert_array_equal(a, b)
