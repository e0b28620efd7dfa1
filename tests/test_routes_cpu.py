"""Which kernel a call goes to, asked of the library without a GPU."""
import pytest

from qfactory import _native

SIMT, TENSOR = 1, 2


@pytest.fixture
def lib():
    L = _native.lib()
    yield L
    L.qfb_set_tensor_min_batch(0)


@pytest.mark.parametrize("k", [2752, 4096])
def test_the_smallest_batch_of_the_tensor_core_kernel_can_be_set(lib, k):
    lib.qfb_set_tensor_min_batch(100)
    assert [lib.qfb_select_kernel(m, 3000, k, 4, 0) for m in (8, 37, 99, 100)] == [SIMT, SIMT, SIMT, TENSOR]
    assert lib.qfb_select_kernel(37, 3000, k, 4, _native.FLAG_FORCE_TENSOR) == TENSOR
    assert lib.qfb_select_kernel(200, 3000, k, 4, _native.FLAG_FORCE_SIMT) == SIMT
    lib.qfb_set_tensor_min_batch(0)
    assert lib.qfb_select_kernel(37, 3000, k, 4, 0) == TENSOR


def test_odd_multiples_of_64_take_one_pass_of_the_cuda_core_kernel_up_to_8_rows(lib):
    assert [lib.qfb_select_kernel(m, 3000, 2752, 4, 0) for m in (1, 8, 9)] == [SIMT, SIMT, TENSOR]
