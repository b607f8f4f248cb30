"""Device memory of a warm-start network: its own arrays and no fixed share."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from aerocfd_b200 import _lib, build
    build.build()
    return _lib.load()


@pytest.mark.parametrize("width, depth, batch", [(128, 1, 512), (128, 3, 1024), (256, 2, 2048)])
def test_memory_of_a_network(lib, width, depth, batch):
    """The activations (BF16 twice, FP32 once and the padded ends), the layers
    (seven FP32 or BF16 copies at most 24 bytes a weight in all), the 32 partial
    tiles of a weight gradient and the allocator's 2 MB pages."""
    import torch
    create = lambda: lib.aero_mlp_create(5, 4, width, depth, batch, ctypes.c_ulonglong(1))
    assert create() == 0 and lib.aero_mlp_destroy() == 0  # context and modules
    free = torch.cuda.mem_get_info()[0]
    assert create() == 0
    used = free - torch.cuda.mem_get_info()[0]
    lib.aero_mlp_destroy()
    arrays = batch * width * (8 * depth + 16) + batch * 128 * 16 + (depth + 1) * width * width * 24 + 32 * width * width * 4
    assert used <= arrays + (4 << 20)
