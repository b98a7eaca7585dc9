"""Runs of a few steps: what a solver with the library's own shape takes for them, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
import ptask_gb300 as P

pytestmark = pytest.mark.gpu


def check(s, pr, f, steps, what):
    ref = oracle.step_ext_f32(f, steps, pr.params, pr.Ca, pr.Cb, pr.Da, pr.Db, pr.src, pr.wave)
    for q, a in enumerate(s.get_fields()):
        np.testing.assert_array_equal(a, ref[q], err_msg=f"{what} {P.FIELDS[q]}")


def problem(shape, steps):
    pr = P.Problem.generate(*shape, n_boxes=3, eps=(1, 10), box=(2, 20), steps=steps - 4, source_mode=2, seed=sum(shape))
    return pr, P.random_fields(*shape, seed=98, scale=1e-2)


# one brick or many, rows of one unit, ragged last units and planes, the largest that fit
@pytest.mark.parametrize("shape", [(17, 17, 17), (5, 160, 8), (33, 31, 29), (48, 40, 36), (401, 9, 10), (31, 3, 152), (96, 96, 96)])
def test_every_run_on_chip_is_one_launch(shape):
    """Single steps go to the other buffer, longer ones stay in place; runs by a step kernel between them continue the fields."""
    parts = (1, 1, 2, 1, 3, 7, 8, 1, 4)
    pr, f = problem(shape, sum(parts) + 5)
    with P.Solver(pr.params) as s:
        s.set_problem(pr)
        s.set_fields(f)
        for n in parts:
            s.run(n)
            assert s.last_launches() == 1
        s.set_tiles(11, 3, 4, 4)   # a shape that a caller sets is taken at its word
        s.run(5)
        assert s.last_launches() > 5
        check(s, pr, f, sum(parts) + 5, shape)


@pytest.mark.parametrize("shape", [(24, 24, 24), (64, 40, 30), (96, 96, 96), (8, 400, 300), (70, 130, 120)])
def test_short_runs_with_the_tuned_shape(shape):
    """On chip one launch, but perhaps for a single step; larger grids, narrow ones too, take the tuned step kernels."""
    parts = (2, 1, 7, 1, 3, 17, 4)
    pr, f = problem(shape, sum(parts))
    on_chip = shape[0] * shape[1] * shape[2] < 900000
    with P.Solver(pr.params) as s:
        s.set_tiles(*P.tuned_tiles(*shape))
        tiles = s.tiles()
        s.set_problem(pr)
        s.set_fields(f)
        for n in parts:
            s.run(n)
            if on_chip and n > 1:
                assert s.last_launches() == 1
            assert s.tiles() == tiles
        check(s, pr, f, sum(parts), shape)


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("shape,register", [((8, 400, 300), (1, 5, 15)), ((32, 200, 190), (1, 5, 15)), ((33, 200, 190), ()),
                                            ((40, 160, 200), (1,)), ((49, 150, 150), ()), ((700, 700, 3), (1,)), ((60, 3000, 6), (1,))])
def test_default_shape_of_narrow_and_thin_grids(shape, register, dense):
    """Rows far shorter than a staged tile, and single steps of thin grids, keep the register kernel; long runs go two
    steps per launch but for thin grids and media that vary in every coefficient."""
    parts = (1, 5, 15, 19, 2)
    pr, f = problem(shape, sum(parts))
    if dense:
        rng = np.random.default_rng(3)
        for c in (pr.Ca, pr.Cb, pr.Da, pr.Db):
            c *= 1 - np.float32(0.1) * rng.random(c.shape, dtype=np.float32)
    with P.Solver(pr.params) as s:
        assert s.kernel()[0] == (0 if 15 in register else 4)
        s.set_problem(pr)
        s.set_fields(f)
        for n in parts:
            fused = n == 19 and shape[2] >= 8 and not dense
            staged = fused or not (n in register or 15 in register)   # a launch more, for the walls
            before = P.launch_count()
            s.run(n)
            assert s.last_launches() == (n // 2 + 2 if fused else n + 1)
            assert P.launch_count() - before == s.last_launches() + staged + 2   # two set the run up
        check(s, pr, f, sum(parts), shape)
