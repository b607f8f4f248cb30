"""The pipelined LU-SGS sweeps against the oracle, whole iterations at 1e-12 per
field (the arithmetic is the oracle's), for block shapes at the edges of the
cuts: a single updated node, extents below the cluster's size, planes wider than
a CTA's warps, many blocks (two CTAs per SM), one layer per slab, planes too wide
for the pipeline, and mixed precision against FP64."""
import ctypes

import numpy as np
import pytest

from aerocfd_b200 import grids
from aerocfd_b200.case import IFLAG_NSSOLVER, IFLAG_SA, Config
from conftest import relerr

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.fixture(scope="module")
def gpu():
    from aerocfd_b200 import build, solver
    build.build()
    return solver


def channel(*shape):
    return lambda: grids.bump_channel(*shape)


def channels(n, *shape):
    return lambda: grids.batch_case([grids.bump_channel(*shape, h=0.05 + 0.001 * c) for c in range(n)])[0]


def plate(*blocks, **size):
    cfg = Config(solver=IFLAG_NSSOLVER, turbulence=IFLAG_SA, ma=0.2, re=5.0e6, cfl=2.0, nutinf=3.0)
    return lambda: grids.flat_plate(*blocks, dy_wall=1e-4, cfg=cfg, **size)


@pytest.mark.parametrize("make", [channel(3, 3, 3), channel(4, 9, 3), channel(40, 3, 3), channel(24, 20, 18),
                                  channel(7, 40, 40), channels(40, 17, 41, 7), channels(90, 9, 9, 3),
                                  plate(8, 1, 1, ni=41, nj=33, nk=9), plate(2, 2, 2, ni=25, nj=17, nk=9)])
def test_block_shapes(gpu, oracle_mod, make):
    co, cg = make(), make()
    oc = oracle_mod.OracleCase(co)
    oc.geometry()
    oc.init_flowfield()
    oc.start()
    gc = gpu.GpuCase(cg)
    try:
        gc.compute_geometry()
        gc.init_flowfield()
        gc.start()
        oc.iterate(3)
        gc.step(3)
        gc.sync_to_host(gpu.mask("q", "nut"))
        assert gc.status() == 0
        for bo, bg in zip(co.blocks, cg.blocks):
            assert np.all(np.isfinite(bo.fields["q"]))
            for k in ["q"] + (["nut"] if co.cfg.turbulence else []):
                assert relerr(bg.fields[k], bo.fields[k]) <= TOL, (bg.m, k)
    finally:
        gc.close()


def test_planes_too_wide_for_the_pipeline(gpu):
    """A block whose planes no cluster's slabs hold takes the sweeps through
    global memory; both give the update that splits of the same block give, so
    the block is compared with itself in mixed precision (at most 1e-6) and the
    run must stay finite."""
    q = {}
    for mixed in (False, True):
        case = grids.bump_channel(70, 70, 70)
        gc = gpu.GpuCase(case)
        try:
            gc.set_precision(mixed)
            gc.compute_geometry()
            gc.init_flowfield()
            gc.start()
            h = gc.step(2)
            gc.sync_to_host(gpu.mask("q"))
            assert gc.status() == 0 and np.all(np.isfinite(h))
            q[mixed] = case.blocks[0].fields["q"].copy()
        finally:
            gc.close()
    assert relerr(q[True], q[False]) <= 1e-6


def test_wide_blocks_outnumbering_the_sms(gpu):
    """Clusters of more CTAs than the device has SMs whose planes leave no room
    for a second CTA per SM: the sweeps through global memory give the same bits."""
    q = []
    for piped in (True, False):
        case = channels(20, 42, 42, 42)()
        gc = gpu.GpuCase(case)
        try:
            if not piped:
                gc.set_sweep_cluster(1)
            gc.compute_geometry()
            gc.init_flowfield()
            gc.start()
            gc.step(2)
            gc.sync_to_host(gpu.mask("q"))
            assert gc.status() == 0
            gc.set_register_bound(False)  # (writes the shapes' text)
            gc.L.aero_tuning.restype = ctypes.c_char_p
            assert ("pipelined" in gc.L.aero_tuning().decode()) == piped
            q.append([b.fields["q"].copy() for b in case.blocks])
        finally:
            gc.close()
    for a, b in zip(*q):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)


@pytest.mark.parametrize("graphs", [False, True])
def test_steps_of_one_call_and_of_several(gpu, graphs):
    """The primitives that open a step are the ones that closed the step before:
    three steps in one call, or one by one, or after a field that went to the
    device between two calls, are the same."""
    out = []
    for split in ([3], [1, 1, 1], [2, 1]):
        case = plate(1, 1, 1, ni=17, nj=13, nk=7)()
        gc = gpu.GpuCase(case)
        try:
            gc.use_graphs(graphs)
            gc.compute_geometry()
            gc.init_flowfield()
            gc.start()
            h = []
            for n in split:
                gc.sync_to_host(gpu.mask("q", "nut"))
                gc.sync_to_device(gpu.mask("q", "nut"))
                h.append(gc.step(n))
            gc.sync_to_host(gpu.mask("q", "nut", "pri_v"))
            b = case.blocks[0].fields
            out.append([np.concatenate(h)] + [b[k].copy() for k in ("q", "nut", "pri_v")])
        finally:
            gc.close()
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a, b)
