"""A call that the device has no memory for is refused with AERO_ERR_NOMEM and
leaves the library as it was: later calls that fit run, with the same results."""
import ctypes

import numpy as np
import pytest

from aerocfd_b200 import _lib, grids

pytestmark = pytest.mark.gpu
ERR_NOMEM = 4


@pytest.fixture(scope="module")
def gpu():
    from aerocfd_b200 import build, solver
    build.build()
    return solver


def primitives(L, n, pri, q):
    """aero_get_primitivevariables on unregistered arrays of n^3 nodes."""
    ints = [ctypes.byref(ctypes.c_int(v)) for v in (1, 1, n, 1, n, 1, n)]
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    d = lambda v: ctypes.byref(ctypes.c_double(v))
    return L.aero_get_primitivevariables(ints[0], p(pri), p(q), d(1.4), d(7.0), *ints[1:])


def test_a_box_that_no_device_holds(gpu):
    """4000^3 nodes (64 TB) are refused before any array is read."""
    L = _lib.load()
    L.aero_finalize()
    _lib.check(L.aero_init(ctypes.c_int(0)))
    rng = np.random.default_rng(0)

    def run(n):
        q = rng.uniform(1.0, 2.0, (n, n, n, 5))
        q[..., 4] += 10.0
        pri = np.zeros((n, n, n, 7))
        _lib.check(primitives(L, n, pri, q), "primitives")
        assert np.array_equal(pri[..., 0], q[..., 0]) and np.all(np.isfinite(pri))

    run(24)
    big = np.zeros(8)
    assert primitives(L, 4000, big, big) == ERR_NOMEM
    for n in (8, 24, 32):
        run(n)
    L.aero_finalize()


def test_a_network_that_no_device_holds(gpu):
    """32 layers of 1024 on 20 million rows (5 TB) are refused; the next network
    trains."""
    from aerocfd_b200 import warmstart
    L = _lib.load()
    assert L.aero_mlp_create(5, 4, 1024, 32, 512 * 40000, ctypes.c_ulonglong(1)) == ERR_NOMEM
    net = warmstart.Network(n_in=5, n_out=4, width=128, depth=2, batch=512)
    try:
        rng = np.random.default_rng(0)
        loss = net.train(rng.uniform(-1, 1, (1024, 5)), rng.uniform(-1, 1, (1024, 4)), 4)
        assert np.all(np.isfinite(loss)) and np.all(loss > 0)
    finally:
        net.close()


def test_sweeps_whose_workspace_does_not_fit(gpu):
    """aero_set_sweep_cluster on a full device keeps the sweeps that run, and
    the run goes on to the same bits; with room it is accepted."""
    import torch
    out = []
    for full in (False, True):
        case = grids.bump_channel(129, 65, 33)
        gc = gpu.GpuCase(case)
        try:
            gc.compute_geometry()
            gc.init_flowfield()
            gc.start()
            h = [gc.step(2)]
            if full:
                was = gc.sweep_pipeline()
                block = torch.empty(torch.cuda.mem_get_info()[0] - (160 << 20), dtype=torch.uint8, device="cuda")
                assert gc.L.aero_set_sweep_cluster(ctypes.c_int(8)) == ERR_NOMEM
                assert gc.sweep_pipeline() == was
                h.append(gc.step(2))
                del block
                torch.cuda.empty_cache()
                gc.set_sweep_cluster(8)
                assert gc.sweep_pipeline()["ctas"] == 0
            else:
                h.append(gc.step(2))
            h.append(gc.step(2))
            gc.sync_to_host(gpu.mask("q"))
            assert gc.status() == 0
            out.append([np.concatenate(h), case.blocks[0].fields["q"].copy()])
        finally:
            gc.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
