"""A tensor core product that does not complete within its bounded wait.

The probe runs the hashing kernels' own product and wait code on one CTA and leaves one product out.  Every thread has
to give up on it, and, whatever number of products is called before and after, keep the phase it gave up on: a phase
that moved on would name an earlier product, which has landed, and the tensor memory would be freed at once.
The group has to agree to leave.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = 1024


@pytest.fixture()
def lib(pkg):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pkg.init(0)
    lib = pkg.load()
    yield lib
    lib.b200_tma_wait_errors()


@pytest.mark.parametrize("before", [0, 1, 2])
@pytest.mark.parametrize("after", [0, 1, 2, 5])
def test_threads_give_up_on_the_same_product(pkg, lib, before, after):
    counts = np.full(3, 7, np.uint32)
    assert lib.b200_tma_wait_errors() == 0
    pkg._check(lib.b200_probe_product_wait(before, after, counts.ctypes.data))
    assert counts.tolist() == [THREADS, 0, THREADS]
    assert lib.b200_tma_wait_errors() == 1
    assert lib.b200_tma_wait_errors() == 0
