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


@pytest.mark.parametrize("seqs,tokens,longest,Hq,Hkv,heads", [
    (1, 128, 128, 32, 8, 1), (1, 512, 512, 32, 8, 1), (1, 513, 513, 32, 8, 2), (1, 1024, 1024, 32, 8, 2), (1, 12001, 2048, 28, 4, 1),
    (8, 8192, 1024, 32, 8, 2), (4, 260, 65, 32, 8, 1), (8, 520, 65, 32, 8, 2), (2, 256, 128, 64, 8, 1), (1, 2048, 2048, 8, 1, 1),
    (1, 2500, 2500, 8, 1, 2), (8, 1032, 1025, 16, 2, 2), (4, 1030, 1025, 8, 2, 1), (64, 64 * 2048, 2048, 16, 16, 1)])
def test_prefill_takes_two_heads_where_single_ones_need_a_second_round(lib, seqs, tokens, longest, Hq, Hkv, heads):
    """148 SMs: tiles of 128 tokens times query heads, by the longest piece or, where pieces differ, by the tokens."""
    assert lib.mx_prefill_heads(seqs, tokens, longest, Hq, Hkv) == heads
