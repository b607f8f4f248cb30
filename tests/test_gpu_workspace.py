"""Device memory of a registered case: the fields and the workspace of the sweeps
that are selected, not of every sweep the library has.  Selecting others
between steps lays the workspace out again and changes no bit of the run."""
import ctypes

import numpy as np
import pytest

from aerocfd_b200 import grids
from aerocfd_b200.case import FIELDS, IFLAG_NSSOLVER, IFLAG_SA, Config

pytestmark = pytest.mark.gpu

# Words a node takes in the fields, the device-only ones among them (radii 3,
# diagonal, viscous fluxes 15, SA scratch 8, face fluxes 15), and bytes an updated node takes
# in the workspace: the pipelined sweeps' records (42 + 14 words) and index, or
# the other sweeps' records (175 + 13 words) and indexes (36 bytes).
FIELD_WORDS = sum(nc for _, nc in FIELDS) + 42
PIPED, OTHER = 56 * 8 + 4, 188 * 8 + 36
SLACK = 32 << 20  # tables by plane and face, allocation granularity


@pytest.fixture(scope="module")
def gpu():
    from aerocfd_b200 import build, solver
    build.build()
    return solver


def free_bytes():
    import torch
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("shape, piped", [((97, 97, 41), False), ((129, 65, 33), True)])
def test_memory_of_a_case(gpu, shape, piped):
    """A block whose planes are too wide for the pipeline holds the other sweeps'
    workspace from the start, another one the pipeline's until others are selected."""
    gpu.GpuCase(grids.bump_channel(9, 9, 9)).close()  # context and modules
    case = grids.bump_channel(*shape)
    b = case.blocks[0]
    size = lambda x: (x[1] - x[0] + 1) * (x[3] - x[2] + 1) * (x[5] - x[4] + 1)
    fields, n1 = size(b.box) * FIELD_WORDS * 8, size(b.box1)
    before = free_bytes()
    gc = gpu.GpuCase(case)
    try:
        gc.L.aero_tuning.restype = ctypes.c_char_p
        assert ("pipelined" in gc.L.aero_tuning().decode()) == piped
        # (the SA pipeline takes the mean flow's order: without it, it is off too)
        assert before - free_bytes() <= fields + n1 * (PIPED if piped else OTHER) + SLACK
        gc.set_sweep_cluster(8)
        gc.set_sa_sweep_cluster(8)
        assert before - free_bytes() <= fields + n1 * OTHER + SLACK
    finally:
        gc.close()


@pytest.mark.parametrize("graphs", [False, True])
def test_other_sweeps_between_steps(gpu, graphs):
    cfg = Config(solver=IFLAG_NSSOLVER, turbulence=IFLAG_SA, ma=0.2, re=5.0e6, cfl=2.0, nutinf=3.0)
    out = []
    for switch in (False, True):
        case = grids.flat_plate(2, 1, 1, ni=41, nj=33, nk=9, dy_wall=1e-4, cfg=cfg)
        gc = gpu.GpuCase(case)
        try:
            gc.use_graphs(graphs)
            gc.compute_geometry()
            gc.init_flowfield()
            gc.start()
            h = [gc.step(2)]
            for select in (lambda: gc.set_sweep_cluster(1), lambda: gc.set_sa_sweep_cluster(4),
                           lambda: gc.set_sweep_cluster(8), lambda: gc.set_sa_sweep_cluster(1)):
                if switch:
                    select()
                h.append(gc.step(2))
            gc.sync_to_host(gpu.mask("q", "nut"))
            assert gc.status() == 0
            out.append([np.concatenate(h)] + [b.fields[k].copy() for b in case.blocks for k in ("q", "nut")])
        finally:
            gc.close()
    for a, b in zip(*out):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)


def test_sweeps_selected_before_set_up(gpu):
    """aero_set_sweep_cluster and aero_set_sa_sweep_cluster before the case is
    registered: set-up lays out what they selected."""
    from aerocfd_b200 import _lib
    cfg = Config(solver=IFLAG_NSSOLVER, turbulence=IFLAG_SA, ma=0.2, re=5.0e6, cfl=2.0, nutinf=3.0)
    out = []
    for sel in ((None, None), (8, None), (None, 4), (1, 1)):
        L = _lib.load()
        _lib.check(L.aero_init(ctypes.c_int(0)), "aero_init")
        if sel[0]:
            _lib.check(L.aero_set_sweep_cluster(ctypes.c_int(sel[0])))
        if sel[1]:
            _lib.check(L.aero_set_sa_sweep_cluster(ctypes.c_int(sel[1])))
        case = grids.flat_plate(2, 1, 1, ni=41, nj=33, nk=9, dy_wall=1e-4, cfg=cfg)
        gc = gpu.GpuCase(case)
        try:
            gc.compute_geometry()
            gc.init_flowfield()
            gc.start()
            h = gc.step(3)
            gc.sync_to_host(gpu.mask("q", "nut"))
            assert gc.status() == 0
            out.append([h] + [b.fields[k].copy() for b in case.blocks for k in ("q", "nut")])
        finally:
            gc.close()
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a, b)
