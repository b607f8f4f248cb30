"""aero_set_sweep_pipeline: the way back to the pipelined sweeps, and every
cluster size that fits a set of blocks: whole iterations against the oracle at
1e-12 per field, bit for bit the same on every size and as the sweeps of one
CTA per block, in FP64 and in mixed precision."""
import ctypes

import numpy as np
import pytest

from aerocfd_b200 import _lib, grids
from aerocfd_b200.case import IFLAG_2D, IFLAG_NSSOLVER, IFLAG_SA, Config
from conftest import relerr

pytestmark = pytest.mark.gpu
TOL = 1e-12
SIZES = (1, 2, 4, 8, 16)


@pytest.fixture(scope="module")
def gpu():
    from aerocfd_b200 import build, solver
    build.build()
    return solver


def plate():
    """One block of 25 x 129 x 33: planes of 184 nodes on 4 CTAs, in two turns
    of 15 warps; 713 and 368 on 1 and 2, which fit no CTA."""
    cfg = Config(solver=IFLAG_NSSOLVER, turbulence=IFLAG_SA, ma=0.2, re=5.0e6, cfl=2.0, nutinf=3.0)
    return grids.flat_plate(1, 1, 1, ni=25, nj=129, nk=33, dy_wall=1e-4, cfg=cfg)


def batch():
    """80 channels of 33 x 33 x 7: from 2 CTAs on two CTAs per SM, on 2 with
    planes of 80 nodes in two turns of 7 warps."""
    return grids.batch_case([grids.bump_channel(33, 33, 7, h=0.05 + 0.0005 * c) for c in range(80)])[0]


def naca_2d():
    cfg = Config(solver=IFLAG_NSSOLVER, ma=0.5, re=5000.0, aoa_deg=2.0, cfl=2.0, dimension=IFLAG_2D,
                 turbulence=IFLAG_SA)
    return grids.naca_ogrid(nblk=4, ni=33, nj=17, first=1e-3, cfg=cfg)


# per case: its blocks, the sizes that fit, and what a size must give (CTAs per
# SM, whether a plane takes several turns of the group's warps)
CASES = [(plate, (4, 8, 16), {4: (1, True), 8: (1, False), 16: (1, False)}),
         (batch, SIZES, {1: (1, False), 2: (2, True), 4: (2, False), 8: (2, False), 16: (2, False)}),
         (lambda: grids.bump_channel(33, 17, 5), SIZES, {}),
         (lambda: grids.bump_channel(57, 57, 57), (16,), {16: (1, True)}),
         (naca_2d, SIZES, {})]


@pytest.mark.parametrize("make, fits, shape", CASES)
def test_every_cluster_size(gpu, oracle_mod, make, fits, shape):
    co = make()
    oc = oracle_mod.OracleCase(co)
    oc.geometry()
    oc.init_flowfield()
    oc.start()
    oc.iterate(2)
    names = ["q"] + (["nut"] if co.cfg.turbulence else [])
    for mixed in (False, True):
        ref = None
        for size in (None,) + SIZES:  # None: the sweeps of one CTA per block
            case = make()
            gc = gpu.GpuCase(case)
            try:
                if size is None:
                    gc.set_sweep_cluster(1)
                    gc.set_sa_sweep_cluster(1)
                    assert gc.sweep_pipeline()["ctas"] == 0
                elif size not in fits:
                    was = gc.sweep_pipeline()
                    with pytest.raises(_lib.AeroError):
                        gc.set_sweep_pipeline(size)
                    assert gc.sweep_pipeline() == was
                    continue
                else:
                    gc.set_sweep_pipeline(size)
                    s = gc.sweep_pipeline()
                    assert s["ctas"] == size and s["sa_ctas"] == size, s
                    if size in shape:
                        assert (s["per_sm"], s["plane"] > 10 * s["warps"]) == shape[size], s
                gc.set_precision(mixed)
                gc.compute_geometry()
                gc.init_flowfield()
                gc.start()
                h = gc.step(2)
                gc.sync_to_host(gpu.mask(*names))
                assert gc.status() == 0
                out = [h] + [b.fields[k].copy() for b in case.blocks for k in names]
            finally:
                gc.close()
            if ref is None:
                ref = out
                if not mixed:
                    for x, b in enumerate(co.blocks):
                        for y, k in enumerate(names):
                            assert relerr(out[1 + len(names) * x + y], b.fields[k]) <= TOL, (b.m, k)
                continue
            for a, b in zip(ref, out):
                assert np.all(np.isfinite(a)) and np.array_equal(a, b), (mixed, size)


def test_the_way_back(gpu):
    """After other sweeps, aero_set_sweep_pipeline(0) gives the selection that
    set-up made, before or after registration."""
    out = []
    for early in (False, True):
        if early:
            L = _lib.load()
            _lib.check(L.aero_init(ctypes.c_int(0)))
            _lib.check(L.aero_set_sweep_cluster(ctypes.c_int(8)))
            _lib.check(L.aero_set_sa_sweep_cluster(ctypes.c_int(2)))
            _lib.check(L.aero_set_sweep_pipeline(ctypes.c_int(0)))
        case = naca_2d()
        gc = gpu.GpuCase(case)
        try:
            gc.use_graphs(True)
            gc.L.aero_tuning.restype = ctypes.c_char_p
            text, shape = gc.L.aero_tuning(), gc.sweep_pipeline()
            assert b"pipelined" in text and shape["ctas"] > 0
            gc.compute_geometry()
            gc.init_flowfield()
            gc.start()
            h = [gc.step(2)]
            gc.set_sweep_cluster(8)
            gc.set_sa_sweep_cluster(4)
            assert b"pipelined" not in gc.L.aero_tuning()
            h.append(gc.step(2))
            gc.set_sweep_pipeline()
            assert gc.L.aero_tuning() == text and gc.sweep_pipeline() == shape
            h.append(gc.step(2))
            gc.sync_to_host(gpu.mask("q", "nut"))
            assert gc.status() == 0
            out.append([np.concatenate(h)] + [b.fields[k].copy() for b in case.blocks for k in ("q", "nut")])
        finally:
            gc.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_refused_sizes(gpu):
    L = _lib.load()
    L.aero_finalize()
    _lib.check(L.aero_init(ctypes.c_int(0)))
    assert L.aero_set_sweep_pipeline(ctypes.c_int(3)) == 1  # AERO_ERR_ARG
    assert L.aero_set_sweep_pipeline(ctypes.c_int(8)) == 2  # AERO_ERR_STATE: before set-up
    assert L.aero_set_sweep_pipeline(ctypes.c_int(0)) == 0
    out = (ctypes.c_int * 8)()
    assert L.aero_get_sweep_pipeline(out) == 2
    L.aero_finalize()
