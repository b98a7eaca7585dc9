"""What a solver reports, and how it goes on, after a run whose bounded waits ran out.

The error word is raised from the host (`ptk_selftest_solver_expiry`): no kernel waits in vain.
"""
import ctypes as C

import numpy as np
import pytest

import oracle
import ptask_gb300 as P
from ptask_gb300 import _lib
from ptask_gb300.device import DeviceBuffer

pytestmark = pytest.mark.gpu
V = C.c_void_p
# (grid, tiles): register kernel, on-chip runs, two steps per launch
SOLVERS = [((16, 12, 10), (8, 0, 4, 0)), ((40, 33, 21), (11, 0, 4, 4)), ((128, 96, 120), (11, 0, 4, 4))]


def problem(shape, steps):
    return (P.Problem.generate(*shape, n_boxes=2, eps=(1, 6), box=(3, 9), steps=steps, seed=sum(shape)),
            P.random_fields(*shape, seed=97, scale=1e-2))


def fetch_device(s, shape):
    bufs = [DeviceBuffer(4 * int(np.prod(P.field_shape(q, *shape)))) for q in range(6)]
    _lib.call("ptk_solver_get_fields", s.handle, (V * 6)(*[b.ptr for b in bufs]), _lib.PTK_DEVICE, None)
    out = [b.download(P.field_shape(q, *shape)) for q, b in enumerate(bufs)]
    for b in bufs:
        b.free()
    return out


@pytest.mark.parametrize("shape,tiles", SOLVERS)
def test_device_read_back_is_nan_after_an_expired_wait(shape, tiles):
    pr, f = problem(shape, 18)
    with P.Solver(pr.params) as s:
        s.set_tiles(*tiles)
        s.set_problem(pr)
        s.set_fields(f)
        s.run(18)
        ref = oracle.step_ext_f32(f, 18, pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db, pr.src, pr.wave)
        for q, a in enumerate(fetch_device(s, shape)):
            np.testing.assert_array_equal(a, ref[q], err_msg=P.FIELDS[q])
        _lib.call("ptk_selftest_solver_expiry", s.handle, None)
        with pytest.raises(_lib.PtkError) as e:
            s.get_fields()
        assert e.value.code == 5   # PTK_ERR_TIMEOUT
        for q, a in enumerate(fetch_device(s, shape)):
            assert np.isnan(a).all(), P.FIELDS[q]


@pytest.mark.parametrize("where", [_lib.PTK_HOST, _lib.PTK_DEVICE])
@pytest.mark.parametrize("shape,tiles", SOLVERS)
def test_new_fields_after_an_expired_wait_run_as_before(shape, tiles, where):
    """A run that finds the word raised gives up, on chip each block at its own step; the solver goes on with new fields."""
    pr, f = problem(shape, 18)
    ref = oracle.step_ext_f32(f, 18, pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db, pr.src, pr.wave)
    with P.Solver(pr.params) as s:
        s.set_tiles(*tiles)
        s.set_problem(pr)
        s.set_fields(f)
        s.run(18)
        for _ in range(2):
            _lib.call("ptk_selftest_solver_expiry", s.handle, None)
            s.run(17)
            with pytest.raises(_lib.PtkError):
                s.get_fields()
            if where == _lib.PTK_HOST:
                s.set_fields(f)
            else:
                bufs = [DeviceBuffer.from_array(a) for a in f]
                s.set_fields_device([b.value for b in bufs])
                _lib.call("ptk_stream_sync", None)
                for b in bufs:
                    b.free()
            s.reset_clock()
            s.run(18)
            for q, a in enumerate(s.get_fields()):
                np.testing.assert_array_equal(a, ref[q], err_msg=P.FIELDS[q])
