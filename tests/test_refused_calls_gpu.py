"""What the library does when a CUDA call that it can do without is refused.

A preloaded library stands in front of the CUDA runtime in a child process and answers chosen calls with
their error code; nothing reaches the GPU from those.
"""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>

int refused, starved; /* launches and allocations answered with an error so far */
size_t limit = -1;    /* bytes of an allocation at most */

cudaError_t cudaMallocFromPoolAsync(void **p, size_t bytes, cudaMemPool_t pool, cudaStream_t stream)
{
    if (bytes > limit) {
        ++starved;
        return cudaErrorMemoryAllocation;
    }
    cudaError_t (*next)(void **, size_t, cudaMemPool_t, cudaStream_t) = dlsym(RTLD_NEXT, "cudaMallocFromPoolAsync");
    return next(p, bytes, pool, stream);
}

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args)
{
    for (unsigned q = 0; q < c->numAttrs; ++q)
        if (c->attrs[q].id == cudaLaunchAttributeCooperative && c->attrs[q].val.cooperative) {
            ++refused;
            return cudaErrorCooperativeLaunchTooLarge;
        }
    cudaError_t (*next)(const cudaLaunchConfig_t *, const void *, void **) = dlsym(RTLD_NEXT, "cudaLaunchKernelExC");
    return next(c, f, args);
}
"""

PRELUDE = r"""
import ctypes as C, sys
import numpy as np
import oracle, ptask_gb300 as P
from ptask_gb300 import _lib
from ptask_gb300.device import DeviceBuffer
refused, starved = (C.c_int.in_dll(C.CDLL(sys.argv[1]), n) for n in ("refused", "starved"))
limit = C.c_size_t.in_dll(C.CDLL(sys.argv[1]), "limit")
V = C.c_void_p
def problem(shape, steps):
    pr = P.Problem.generate(*shape, n_boxes=2, eps=(1, 8), box=(3, 9), steps=steps, source_mode=2, seed=sum(shape))
    f = P.random_fields(*shape, seed=99, scale=1e-2)
    return pr, f, oracle.step_ext_f32(f, steps, pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db, pr.src, pr.wave)
def same(got, ref):
    for q in range(6):
        np.testing.assert_array_equal(got[q], ref[q], err_msg=P.FIELDS[q])
"""


def child(tmp_path, body):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-I", f"{cuda}/include", str(src), "-o", str(so), "-ldl", "-Wl,--no-as-needed",
                    "-L", f"{cuda}/lib64", "-lcudart", f"-Wl,-rpath,{cuda}/lib64"], check=True)   # the runtime is next to it
    r = subprocess.run([sys.executable, "-c", PRELUDE + body, str(so)], cwd=ROOT, capture_output=True, text=True, timeout=240,
                       env=dict(os.environ, LD_PRELOAD=str(so)))
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("shape", [(40, 33, 21), (30, 12, 16)])
def test_step_kernels_where_an_on_chip_launch_cannot_be_placed(tmp_path, shape):
    child(tmp_path, f"""
shape = {shape}
pr, f, ref = problem(shape, 21)
for tiles in (None, (11, 0, 4, 4), "tuned"):
    with P.Solver(pr.params) as s:
        if tiles:
            s.set_tiles(*(P.tuned_tiles(*shape) if tiles == "tuned" else tiles))
        s.set_problem(pr)
        s.set_fields(f)
        before = refused.value
        for n in (1, 9, 2, 9):
            s.run(n)
            assert s.last_launches() == n + 1
        assert refused.value - before <= 1   # asked once
        same(s.get_fields(), ref)
assert refused.value >= 2
before = refused.value
bufs = [DeviceBuffer.from_array(a) for a in f]
coefs = [DeviceBuffer.from_array(a) for a in (pr.Ca, pr.Cb, pr.Da, pr.Db, pr.wave)]
_lib.call("ptk_fdtd_solve_static", C.byref(pr.params), (V * 6)(*[b.ptr for b in bufs]), *[c.ptr for c in coefs[:4]], *pr.src,
          coefs[4].ptr, int(pr.wave.size), 21, None)
_lib.call("ptk_device_sync")
same([b.download(a.shape) for b, a in zip(bufs, f)], ref)
assert refused.value == before + 1
""")


def test_host_arrays_are_staged_one_by_one_where_there_is_no_room_for_all(tmp_path):
    child(tmp_path, """
shape, steps = (40, 33, 21), 9
pr, f, ref = problem(shape, steps)
with P.Solver(pr.params) as s:
    limit.value = max(a.nbytes for a in f) + 256   # the largest field's slot, and no more
    s.set_problem(pr)
    s.set_fields(f)
    s.run(steps)
    got = s.get_fields()
    assert starved.value == 6, starved.value   # coefficients, fields, fields back: each tried twice
    same(got, ref)
    limit.value = 1000
    for call in (lambda: s.set_fields(f), s.get_fields, lambda: s.set_problem(pr)):
        try:
            call()
            raise SystemExit("no error")
        except _lib.PtkError as e:
            assert e.code == 3, e.code   # PTK_ERR_NOMEM
""")


@pytest.mark.parametrize("shape,steps", [((40, 33, 21), 9), ((128, 96, 120), 19)])
def test_a_solver_in_pieces_where_no_block_holds_it(tmp_path, shape, steps):
    """No allocation larger than one padded array: the solver's arrays come one by one, and go again."""
    child(tmp_path, f"""
shape, steps = {shape}, {steps}
pr, f, ref = problem(shape, steps)
def used():
    _lib.call("ptk_device_sync")
    r, u = C.c_size_t(), C.c_size_t()
    _lib.call("ptk_pool_stats", C.byref(r), C.byref(u))
    return u.value
with P.Solver(pr.params) as s:   # what a first solver sets up once
    s.set_problem(pr)
    s.run(steps)
base = used()
array = 4 * (-(-(shape[0] + 1) // 32) * 32) * (shape[1] + 1) * (shape[2] + 1)
limit.value = -(-array // 256) * 256
with P.Solver(pr.params) as s:
    assert starved.value >= 2
    s.set_problem(pr)
    s.set_fields(f)
    s.run(steps)
    same(s.get_fields(), ref)
    taken = used() - base
    assert s.nbytes() <= taken <= s.nbytes() + 30 * (2 << 20)
assert used() == base
limit.value = limit.value - 256
try:
    P.Solver(pr.params)
    raise SystemExit("no error")
except _lib.PtkError as e:
    assert e.code == 3, e.code   # PTK_ERR_NOMEM
assert used() == base
""")
