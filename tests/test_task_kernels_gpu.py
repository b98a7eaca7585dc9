"""The task kernels over dense blocks at the ends of their rows, row groups and plane groups, against the oracle, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import oracle
import ptask_gb300 as P
from ptask_gb300 import _lib
from ptask_gb300.device import DeviceBuffer

pytestmark = pytest.mark.gpu
V = C.c_void_p
SHAPES = [(1, 1, 1), (31, 8, 4), (32, 9, 5), (33, 7, 3), (64, 16, 8), (65, 1, 9), (1, 17, 2), (2, 2, 1), (95, 23, 7),
          (97, 41, 70)]   # the last: fields large enough for several planes per warp


def check(bufs, ref, shape, what):
    for q in range(6):
        np.testing.assert_array_equal(bufs[q].download(P.field_shape(q, *shape)), ref[q], err_msg=f"{what} {shape} {P.FIELDS[q]}")


@pytest.mark.parametrize("halves", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_scalar_tasks(shape, halves):
    p, steps = P.reference_params(*shape), 3
    f = P.random_fields(*shape, seed=95)
    cur, nxt = [DeviceBuffer.from_array(a) for a in f], [DeviceBuffer(a.nbytes) for a in f]
    ins = ((0, 4, 5), (1, 3, 5), (2, 3, 4), (3, 1, 2), (4, 0, 2), (5, 0, 1))
    for _ in range(steps):
        if halves:
            _lib.call("ptk_launch_h_half_step", (V * 6)(*[b.ptr for b in cur]), (V * 3)(*[b.ptr for b in nxt[:3]]), C.byref(p), None)
            _lib.call("ptk_launch_e_half_step", (V * 3)(*[b.ptr for b in cur[3:]]), (V * 3)(*[b.ptr for b in nxt[:3]]),
                      (V * 3)(*[b.ptr for b in nxt[3:]]), C.byref(p), None)
        else:
            for q, (a, b, c) in enumerate(ins):
                src = [cur[a], (nxt if q >= 3 else cur)[b], (nxt if q >= 3 else cur)[c]]
                _lib.call("ptk_launch_field_update", q, *[s.ptr for s in src], C.byref(p), nxt[q].ptr, None)
        cur, nxt = nxt, cur
    check(cur, oracle.step_ref_f32(f, steps, p), shape, "halves" if halves else "fields")
    for b in cur + nxt:
        b.free()


@pytest.mark.parametrize("shape,steps", [(n, 4) for n in SHAPES] + [((97, 41, 70), 60)])   # the last: a long chain of launches
def test_coefficient_tasks_in_place(shape, steps):
    pr = P.Problem.generate(*shape, n_boxes=2, eps=(1, 9), box=(1, 20), steps=3, source_mode=2, seed=6)
    rng = np.random.default_rng(7)
    for c in (pr.Ca, pr.Cb, pr.Da, pr.Db):
        c *= 1 - np.float32(0.1) * rng.random(c.shape, dtype=np.float32)
    f = P.random_fields(*shape, seed=96, scale=1e-2)
    src = pr.src if pr.has_source else (-1, -1, -1)
    ref = oracle.step_ext_f32(f, steps, pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db, src, pr.wave)
    cur = [DeviceBuffer.from_array(a) for a in f]
    Ca, Cb, Da, Db, wave = (DeviceBuffer.from_array(a) for a in (pr.Ca, pr.Cb, pr.Da, pr.Db, pr.wave))
    count = DeviceBuffer.from_array(np.zeros(1, np.int32))
    h, e = (V * 3)(*[b.ptr for b in cur[:3]]), (V * 3)(*[b.ptr for b in cur[3:]])
    for _ in range(steps):
        _lib.call("ptk_launch_h_step_coef", h, e, Da.ptr, Db.ptr, C.byref(pr.params), None)
        _lib.call("ptk_launch_e_step_coef", e, h, Ca.ptr, Cb.ptr, C.byref(pr.params), *src, wave.ptr if pr.has_source else None,
                  int(pr.wave.size) if pr.has_source else 0, count.ptr if pr.has_source else None, None)
    check(cur, ref, shape, "in place")
    for b in cur + [Ca, Cb, Da, Db, wave, count]:
        b.free()
