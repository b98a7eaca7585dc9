"""The two-step kernel: runs of sixteen steps or more on grids too large for the chip.

Each launch advances frames of the grid by two steps and yields their inner cells, so the shapes
here put frame and tile boundaries everywhere: one tile or many in x, rows and planes left over,
ragged last units, long thin grids.  Reference: the FP32 oracle, bit for bit.
"""
import numpy as np
import pytest

import oracle
import ptask_gb300 as P

pytestmark = pytest.mark.gpu

SHAPES = [(128, 96, 120), (127, 97, 119), (261, 37, 130), (97, 201, 63), (400, 24, 130), (2000, 30, 20), (130, 129, 71),
          (33, 200, 190), (18, 330, 210), (301, 301, 17)]


@pytest.mark.parametrize("lossy", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_two_step_runs_match_oracle(shape, lossy):
    """Odd and even runs (a last single step), a short run between, a waveform that ends on an odd step."""
    parts = (17, 3, 16)
    pr = P.Problem.generate(*shape, n_boxes=5, eps=(1, 10), box=(3, 40), steps=sum(parts) - 5, source_mode=2, seed=sum(shape))
    if lossy:
        inside = pr.Cb != pr.Cb.max()
        pr.Ca[inside] = np.float32(0.98)
        pr.Da[inside] = np.float32(0.99)
    f = P.random_fields(*shape, seed=92, scale=1e-2)
    ref = oracle.step_ext_f32(f, sum(parts), pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db, pr.src, pr.wave)
    with P.Solver(pr.params) as s:
        s.set_tiles(11, 0, 4, 4)
        s.set_problem(pr)
        s.set_fields(f)
        for n in parts:
            s.run(n)
        got = s.get_fields()
    for q in range(6):
        np.testing.assert_array_equal(got[q], ref[q], err_msg=f"{shape} {P.FIELDS[q]}")


@pytest.mark.parametrize("src", [(1, 1, 0), (62, 20, 9), (63, 21, 10), (64, 40, 11), (66, 41, 60), (129, 95, 70)])
def test_source_where_frames_overlap(src):
    """Every frame that holds the source node adds the waveform, in each of its two steps."""
    shape, steps = (130, 96, 101), 18
    p = P.Problem.generate(*shape, n_boxes=0, steps=steps, seed=3)
    pr = P.Problem(p.params, p.Ca, p.Cb, p.Da, p.Db, src, p.wave)
    f = P.zero_fields(*shape)
    ref = oracle.step_ext_f32(f, steps, pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db, pr.src, pr.wave)
    with P.Solver(pr.params) as s:
        s.set_tiles(11, 0, 4, 4)
        s.set_problem(pr)
        s.set_fields(f)
        s.run(steps)
        assert s.last_launches() == steps // 2 + 1
        got = s.get_fields()
    for q in range(6):
        np.testing.assert_array_equal(got[q], ref[q], err_msg=P.FIELDS[q])


def test_clock_reset_after_an_odd_number_of_buffer_flips():
    """A run of 18 steps flips the buffers nine times; the next run continues from the current fields."""
    shape = (128, 96, 120)
    pr = P.Problem.generate(*shape, n_boxes=3, steps=0, seed=8, source_mode=0)
    f = P.random_fields(*shape, seed=93, scale=1e-2)
    ref = oracle.step_ext_f32(f, 18 + 5 + 17, pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db)
    with P.Solver(pr.params) as s:
        s.set_tiles(11, 0, 4, 4)
        s.set_problem(pr)
        s.set_fields(f)
        for n in (18, 5, 17):
            s.run(n)
            s.reset_clock()
        got = s.get_fields()
        s.set_fields(f)      # fields set again land in the buffer the next run reads
        s.run(18 + 5 + 17)
        again = s.get_fields()
    for q in range(6):
        np.testing.assert_array_equal(got[q], ref[q], err_msg=P.FIELDS[q])
        np.testing.assert_array_equal(again[q], ref[q], err_msg=P.FIELDS[q])


@pytest.mark.parametrize("vary", ["permittivity", "one_Ca", "one_Db"])
@pytest.mark.parametrize("shape", SHAPES + [(40, 33, 28)])   # the last fits on chip
def test_permittivity_of_every_cell(shape, vary):
    """More materials than the index holds: Cb from its array while Ca = Da = 1 and Db is one value; one cell
    that breaks that (its last) sends the run to the kernels that read all four arrays."""
    steps = 17
    pr = P.Problem.generate(*shape, n_boxes=0, steps=steps, source_mode=2, seed=sum(shape))
    pr.Cb *= np.random.default_rng(5).uniform(0.2, 1.0, pr.Cb.shape).astype(np.float32)
    if vary == "one_Ca":
        pr.Ca.flat[-1] = np.float32(0.98)
    if vary == "one_Db":
        pr.Db.flat[-1] *= np.float32(0.5)
    f = P.random_fields(*shape, seed=92, scale=1e-2)
    ref = oracle.step_ext_f32(f, steps, pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db, pr.src, pr.wave)
    with P.Solver(pr.params) as s:
        s.set_tiles(11, 0, 4, 4)
        s.set_problem(pr)
        assert s.material_count() == 0
        s.set_fields(f)
        s.run(steps)
        if shape[0] > 40:
            assert s.last_launches() == (steps // 2 + 2 if vary == "permittivity" else steps + 1)
        got = s.get_fields()
    for q in range(6):
        np.testing.assert_array_equal(got[q], ref[q], err_msg=f"{shape} {P.FIELDS[q]}")
