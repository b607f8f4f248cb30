"""The sweeps that aero_set_sweep_cluster selects, which also run where the
pipelined ones do not fit: their launch shapes, their withheld plane, blocks too
wide for the pipeline, and planes smaller than the cluster."""
import ctypes
import time

import numpy as np
import pytest

from aerocfd_b200 import _lib, grids
from aerocfd_b200.case import IFLAG_NSSOLVER, IFLAG_SA, Config
from conftest import relerr

pytestmark = pytest.mark.gpu
TOL = 1e-12
ST_TIMEOUT = 8


@pytest.fixture(scope="module")
def gpu():
    from aerocfd_b200 import build, solver
    build.build()
    return solver


def naca():
    return grids.naca_ogrid(nblk=4, ni=33, nj=17, nk=3)


def plate():
    cfg = Config(solver=IFLAG_NSSOLVER, turbulence=IFLAG_SA, ma=0.2, re=5.0e6, cfl=2.0, nutinf=3.0)
    return grids.flat_plate(2, 1, 1, ni=25, nj=13, nk=7, dy_wall=1e-3, cfg=cfg)


def run(gpu, make, steps, before=lambda gc: None, mixed=False):
    """History, q and nut of every block after `steps`."""
    case = make()
    gc = gpu.GpuCase(case)
    try:
        before(gc)
        gc.set_precision(mixed)
        gc.compute_geometry()
        gc.init_flowfield()
        gc.start()
        h = gc.step(steps)
        gc.sync_to_host(gpu.mask("q", "nut"))
        assert gc.status() == 0
        return [h] + [b.fields[k].copy() for b in case.blocks for k in ("q", "nut")]
    finally:
        gc.close()


@pytest.mark.parametrize("make", [naca, plate])
@pytest.mark.parametrize("mixed", [False, True])
def test_every_record_and_stage_shape(gpu, make, mixed):
    """The block-record threads and the stages of the staged sweep, which only
    these sweeps launch: the bits of the pipelined ones."""
    ref = run(gpu, make, 3, mixed=mixed)
    for mats in (64, 128, 256):
        for nst in (2, 3, 4):
            def before(gc):
                gc.set_sweep_cluster(1)
                gc.set_sa_sweep_cluster(1)
                gc.set_tuning(64, 256, 128, mats, nst)
            for a, b in zip(ref, run(gpu, make, 3, before, mixed)):
                assert np.all(np.isfinite(a)) and np.array_equal(a, b), (mats, nst)


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("plane", [0, 5])
def test_withheld_plane_of_the_staged_sweep(gpu, graphs, plane):
    """A producer that never issues a plane's copies ends the one-CTA staged
    sweep's waits by their poll budget; the next steps run clean."""
    case = naca()
    gc = gpu.GpuCase(case)
    try:
        gc.set_sweep_cluster(1)
        gc.compute_geometry()
        gc.init_flowfield()
        gc.start()
        gc.step(5)
        assert gc.status() == 0
        gc.sync_to_host(gpu.ALL)
        gc.use_graphs(graphs)
        gc.set_poll_budget(4096)
        gc.inject_sweep_stall(plane)
        t0 = time.perf_counter()
        gc.step(1)
        assert time.perf_counter() - t0 < 30.0
        assert gc.sweep_pipeline()["ctas"] == 0
        site = (ctypes.c_int * 5)()
        assert gc.L.aero_timeout_site(site) == 0
        assert gc.status() & ST_TIMEOUT
        assert site[0] == 4 and 0 <= site[1] < len(case.blocks) and list(site)[2:] == [0, plane, 1], list(site)
        gc.inject_sweep_stall(-1)
        gc.set_poll_budget(1 << 20)
        gc.sync_to_device(gpu.mask("q"))
        gc.getpri_all()
        assert np.all(np.isfinite(gc.step(3))) and gc.status() == 0
    finally:
        gc.close()


def test_block_too_wide_for_the_pipeline(gpu, oracle_mod):
    """60 x 60 x 60: planes of 240 nodes on 16 CTAs.  The sweeps of one CTA per
    block run, whole iterations against the oracle, and clusters give their bits."""
    co, cg = grids.bump_channel(60, 60, 60), grids.bump_channel(60, 60, 60)
    oc = oracle_mod.OracleCase(co)
    oc.geometry()
    oc.init_flowfield()
    oc.start()
    oc.iterate(2)
    gc = gpu.GpuCase(cg)
    try:
        assert gc.sweep_pipeline()["ctas"] == 0
        gc.L.aero_tuning.restype = ctypes.c_char_p
        assert b"pipelined" not in gc.L.aero_tuning()
        gc.compute_geometry()
        gc.init_flowfield()
        gc.start()
        h = gc.step(2)
        gc.sync_to_host(gpu.mask("q"))
        assert gc.status() == 0
        q = cg.blocks[0].fields["q"].copy()
        assert relerr(q, co.blocks[0].fields["q"]) <= TOL
    finally:
        gc.close()
    out = run(gpu, lambda: grids.bump_channel(60, 60, 60), 2, lambda gc: gc.set_sweep_cluster(8))
    assert np.array_equal(out[0], h) and np.array_equal(out[1], q)


@pytest.mark.parametrize("shape", [(3, 3, 3), (41, 4, 3), (4, 41, 3), (9, 7, 5), (65, 5, 5)])
@pytest.mark.parametrize("mixed", [False, True])
def test_planes_smaller_than_the_cluster(gpu, shape, mixed):
    """Planes of one to a few nodes on up to 16 CTAs with the bulk exchange, most
    of them without a node of their own: no wait runs out, the bits stay."""
    make = lambda: grids.bump_channel(*shape)
    ref = run(gpu, make, 20, mixed=mixed)
    for ctas in (2, 4, 8, 16):
        for exch in ("shared", "shared2"):
            def before(gc):
                gc.set_sweep_exchange(exch)
                gc.set_sweep_cluster(ctas)
            try:
                out = run(gpu, make, 20, before, mixed)
            except _lib.AeroError:
                assert ctas == 16  # the device holds no such cluster
                continue
            for a, b in zip(ref, out):
                assert np.all(np.isfinite(a)) and np.array_equal(a, b), (ctas, exch)
