"""The public counters against what a run launches."""
import ctypes as C
import gc

import pytest

import ptask_gb300 as P
from ptask_gb300 import _lib
from ptask_gb300.graph import FDTDGraph

pytestmark = pytest.mark.gpu


# on chip: one launch, no graph; shorter loops and larger grids: 32 steps a graph, two steps per launch 64
@pytest.mark.parametrize("shape,steps,graphs", [((30, 22, 17), 70, 0), ((30, 22, 17), 5, 1), ((128, 96, 80), 200, 4),
                                                ((128, 96, 80), 15, 1), ((150, 140, 6), 70, 0), ((700, 700, 3), 70, 3)])
def test_graph_replays_of_a_lowered_loop(shape, steps, graphs):
    f = P.zero_fields(*shape)
    with FDTDGraph(P.reference_params(*shape), "fused") as g:
        g.set_problem(P.Problem.vacuum(P.reference_params(*shape)))
        for done in (1, 2):
            g.solve(f, steps)
            st = g.stats()
            assert st["cycles_lowered"] == done and st["graph_replays"] == done * graphs


def pool_used():
    gc.collect()   # objects of earlier tests
    _lib.call("ptk_device_sync")
    reserved, used = C.c_size_t(), C.c_size_t()
    _lib.call("ptk_pool_stats", C.byref(reserved), C.byref(used))
    return used.value


@pytest.mark.parametrize("shape", [(12, 12, 12), (96, 96, 96), (401, 9, 10), (200, 150, 100)])
def test_solver_bytes_are_what_the_pool_gave(shape):
    """Three allocations at most, each rounded up by the pool to no more than 2 MiB."""
    pr = P.Problem.generate(*shape, n_boxes=1, box=(2, 6), steps=50000, seed=4)
    before = pool_used()
    with P.Solver(pr.params) as s:
        s.set_problem(pr)
        s.run(9)
        taken = pool_used() - before
        assert s.nbytes() <= taken <= s.nbytes() + 3 * (2 << 20)


@pytest.mark.parametrize("tiles,walls", [((8, 0, 4, 0), 0), ((11, 0, 4, 4), 1)])
@pytest.mark.parametrize("shape,steps", [((40, 33, 21), 5), ((128, 96, 120), 40)])
def test_launch_count_of_replayed_graphs(shape, steps, tiles, walls):
    """Steps (two per launch on the larger grid's staged shape), the clock and the staged kernels' walls of each graph,
    and the two launches that set a run up."""
    fused = walls and steps == 40
    graphs, launches = (2, 40) if steps == 40 and not fused else (1, 20 if fused else 5)
    with P.Solver(P.reference_params(*shape)) as s:
        s.set_tiles(*tiles)
        for _ in range(2):
            before = P.launch_count()
            s.run(steps)
            assert s.last_launches() == launches + graphs
            assert P.launch_count() - before == launches + graphs * (1 + walls) + 2
