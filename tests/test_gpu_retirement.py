"""When a bad block is retired: the step that meets it is its last.  A block
whose field is bad when a call begins (marked by the primitives that open the
step) takes one step like every other block and stands still from the second on,
whether the steps come in one call or several, replayed from a graph or not."""
import numpy as np
import pytest

from aerocfd_b200 import grids

pytestmark = pytest.mark.gpu
ST_NEG_DENSITY = 1
BAD = 1


@pytest.fixture(scope="module")
def gpu():
    from aerocfd_b200 import build, solver
    build.build()
    return solver


def run(gpu, calls, retire, graphs):
    """q of every block after steps taken in `calls`, block BAD's field
    uploaded with one negative density."""
    case, params = grids.batch_case([grids.bump_channel(17, 9, 5, h=0.05 + 0.01 * c) for c in range(3)])
    gc = gpu.GpuCase(case, block_params=params)
    try:
        gc.use_graphs(graphs)
        gc.compute_geometry()
        gc.init_flowfield()
        gc.start()
        gc.step(2, history=False)
        gc.sync_to_host(gpu.mask("q"))
        q = case.blocks[BAD].fields["q"]
        q[tuple(n // 2 for n in q.shape[:3]) + (0,)] *= -1.0
        gc.sync_to_device(gpu.mask("q"))
        gc.clear_block_status()
        gc.set_retirement(retire)
        for n in calls:
            gc.step(n, history=False)
        st = gc.block_status()
        assert st[BAD] & ST_NEG_DENSITY and not np.delete(st, BAD).any(), st
        gc.sync_to_host(gpu.mask("q"))
        return [b.fields["q"].copy() for b in case.blocks]
    finally:
        gc.close()


@pytest.mark.parametrize("graphs", [False, True])
def test_a_bad_field_takes_one_step(gpu, graphs):
    one = run(gpu, [1], False, graphs)
    three = run(gpu, [3], False, graphs)
    for calls in ([1], [3], [1, 2], [2, 1], [1, 1, 1]):
        q = run(gpu, calls, True, graphs)
        assert np.array_equal(q[BAD], one[BAD], equal_nan=True), calls
        want = one if calls == [1] else three
        for m in (0, 2):
            assert np.all(np.isfinite(q[m])) and np.array_equal(q[m], want[m]), (calls, m)
