"""crank2nd with its lines in shared memory: shapes at the edges of a CTA's share
of lines (one line, fewer than four, a remainder), of the line lengths (one
updated node), and past them (a line too long for shared memory, which takes the
path through global memory), against the oracle at the 1e-12 of the other
crank2nd tests; the arithmetic is the oracle's, in its order."""
import ctypes

import numpy as np
import pytest

from aerocfd_b200 import grids
from aerocfd_b200.case import IFLAG_2NDCRANK, IFLAG_NSSOLVER, IFLAG_UNSTEADY, Config
from conftest import relerr
from test_gpu_crank import _d, _i, _p, gpu, prepared  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 4, 3), (9, 5, 3), (3, 40, 3), (70, 6, 7), (450, 4, 3), (4, 4, 90)])
def test_line_shapes(gpu, oracle_mod, shape):  # noqa: F811
    cfg = Config(solver=IFLAG_NSSOLVER, ma=0.5, re=2000.0, cfl=3.0, time=IFLAG_UNSTEADY, timeadvance=IFLAG_2NDCRANK,
                 dt=1.0e-3)
    oc, co, cg = prepared(lambda: grids.bump_channel(*shape, cfg=cfg), oracle_mod, seed=sum(shape))
    gc = gpu.GpuCase(cg)
    try:
        b = co.blocks[0]
        F = b.fields
        rng = np.random.default_rng(1)
        F["rhsi"][...] = rng.standard_normal(F["rhsi"].shape) * 1e-2
        F["rhsv"][...] = rng.standard_normal(F["rhsv"].shape) * 1e-3
        f = {k: v.copy() for k, v in F.items()}
        names = ("q", "q0", "dt", "pri_v", "rhs", "rhsi", "rhsv", "dxidx", "inv_j")
        assert gc.L.aero_crank2nd(*[_p(f[k]) for k in names], *[_i(v) for v in b.box + b.box0 + b.box1],
                                  _d(1.4), _i(1), _i(1)) == 0, gc.L.aero_last_error()
        box18 = np.array(b.box + b.box0 + b.box1, dtype=np.int32)
        oc.L.oracle_crank2nd(*[_p(F[k]) for k in names], box18.ctypes.data_as(ctypes.c_void_p), ctypes.c_double(1.4))
        for k in ("q", "rhs"):
            assert relerr(f[k], F[k]) <= 1e-12, (k, relerr(f[k], F[k]))
    finally:
        gc.close()
