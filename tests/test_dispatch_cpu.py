"""The rules by which calls are sent to one kernel or another, as the kernel library and the bindings state them (no GPU needed)."""
import pytest

from mlxcel_b200.ops import _lib


@pytest.fixture(scope="module")
def lib():
    if not _lib.lib_path().exists():
        pytest.skip("the kernel library is not built")
    return _lib.load()


@pytest.mark.parametrize("experts,rows,ahead", [(128, 4, 0), (128, 128, 0), (128, 255, 0), (128, 256, 1), (8, 15, 0), (8, 16, 1), (1, 1, 0),
                                                (1, 2, 1), (1 << 30, 1 << 30, 0)])
def test_expert_weights_are_asked_for_early_only_where_nearly_all_are_used(lib, experts, rows, ahead):
    assert lib.mx_qstream_ahead(experts, rows) == ahead
