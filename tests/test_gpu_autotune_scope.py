"""aero_autotune changes the shapes of the kernels that run and no others: with
the pipelined sweeps the block-record threads and the sweep stages keep what
aero_set_tuning gave them; with other sweeps selected, those stay selected."""
import re

import pytest

from aerocfd_b200 import grids

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from aerocfd_b200 import build, solver
    build.build()
    return solver


@pytest.mark.parametrize("mats, nst", [(64, 2), (128, 3), (256, 4), (64, 4)])
def test_shapes_of_idle_kernels_stay(gpu, mats, nst):
    gc = gpu.GpuCase(grids.bump_channel(33, 17, 5))
    try:
        gc.set_tuning(64, 256, 128, mats, nst)
        gc.compute_geometry()
        gc.init_flowfield()
        gc.start()
        text = gc.autotune(2)
        assert "sweep_exchange=pipelined" in text
        assert f"mats_threads={mats} " in text and f"sweep_stages<={nst} " in text, text
        gc.set_sweep_cluster(1)
        text = gc.autotune(1)
        assert "pipelined" not in text and re.search(r"sweep_exchange=(l2|shared2?|slab) ", text), text
        assert gc.sweep_pipeline()["ctas"] == 0
        assert gc.status() == 0
    finally:
        gc.close()
