"""The rules by which calls are sent to one kernel or another, as the kernel library and the bindings state them (no GPU needed)."""
import re
from types import SimpleNamespace

import pytest
import torch

from mlxcel_b200 import ops
from mlxcel_b200.models import moe
from mlxcel_b200.ops import _lib, quant


@pytest.fixture(scope="module")
def lib():
    if not _lib.lib_path().exists():
        pytest.skip("the kernel library is not built")
    return _lib.load()


@pytest.mark.parametrize("experts,rows,blocks,ahead", [(128, 4, 45, 0), (128, 128, 45, 0), (128, 255, 45, 0), (128, 256, 45, 1), (8, 15, 56, 0),
                                                       (8, 16, 56, 1), (8, 6, 22, 1), (8, 2, 88, 0), (1, 1, 500, 0), (1 << 30, 1 << 30, 2, 0)])
def test_expert_weights_are_asked_for_early_only_where_nearly_all_are_used(lib, experts, rows, blocks, ahead):
    """... or where all blocks are on the GPU at once (444 of them)."""
    assert lib.mx_qstream_ahead(experts, rows, experts * blocks, 444) == ahead


@pytest.mark.parametrize("seqs,tokens,longest,Hq,Hkv,heads", [
    (1, 128, 128, 32, 8, 1), (1, 512, 512, 32, 8, 1), (1, 513, 513, 32, 8, 2), (1, 1024, 1024, 32, 8, 2), (1, 12001, 2048, 28, 4, 1),
    (8, 8192, 1024, 32, 8, 2), (4, 260, 65, 32, 8, 1), (8, 520, 65, 32, 8, 2), (2, 256, 128, 64, 8, 1), (1, 2048, 2048, 8, 1, 1),
    (1, 2500, 2500, 8, 1, 2), (8, 1032, 1025, 16, 2, 2), (4, 1030, 1025, 8, 2, 1), (64, 64 * 2048, 2048, 16, 16, 1)])
def test_prefill_takes_two_heads_where_single_ones_need_a_second_round(lib, seqs, tokens, longest, Hq, Hkv, heads):
    """148 SMs: tiles of 128 tokens times query heads, by the longest piece or, where pieces differ, by the tokens."""
    assert lib.mx_prefill_heads(seqs, tokens, longest, Hq, Hkv) == heads


@pytest.mark.parametrize("S,max_q,Hq,Hkv,D,keys,coded,tc,packed", [
    # many tiles: the context is read once per 16 rows, against once per 128 rows of one or two heads
    (16, 64, 32, 32, 128, 64, False, True, False), (64, 64, 32, 32, 128, 512, False, True, False), (16, 48, 8, 8, 128, 4096, False, True, False),
    (16, 64, 32, 32, 128, 64, True, False, False), (64, 8, 64, 8, 128, 64, True, False, False),
    (64, 16, 32, 32, 128, 512, False, True, True), (16, 64, 32, 32, 128, 512, True, False, True),
    # few tiles: either side is one round of CTAs, short contexts are over sooner without packing
    (1, 16, 32, 8, 128, 16, False, True, False), (1, 4, 32, 8, 128, 512, False, True, False), (4, 4, 8, 8, 128, 512, False, True, False),
    (1, 4, 32, 8, 128, 8192, False, True, True), (3, 4, 32, 8, 128, 12001, False, True, True), (1, 1, 16, 1, 128, 8192, False, True, True),
    (1, 16, 32, 8, 128, 16, True, False, False), (1, 4, 32, 8, 128, 512, True, False, True),
    # verify rounds
    (16, 4, 64, 8, 128, 4096, False, True, True), (16, 4, 32, 8, 128, 4096, False, True, True), (8, 4, 64, 8, 64, 2048, False, True, True)])
def test_short_pieces_are_packed_where_that_is_faster(S, max_q, Hq, Hkv, D, keys, coded, tc, packed):
    """Calls that were timed on both sides (at least a tenth apart)."""
    assert bool(ops.packed_splits(S, max_q, Hq, Hkv, D, keys, coded, tc)) == packed


def test_key_splits_of_packed_pieces_follow_the_context():
    """No split below 768 keys (merging costs as much as 1000), no more CTAs than two an SM, one split where the tiles fill the GPU."""
    for S in (1, 3, 16, 64):
        for keys in (128, 1024, 4096, 12032, 131072):
            s = ops.packed_splits(S, 4, 32, 8, 128, keys, True, False)
            assert s <= max(1, keys // 768) and s <= 16 and (s <= 1 or s * S * 8 <= 296)


def test_shared_memory_is_allowed_on_every_device():
    """Function attributes are per device: no launcher may keep one flag for all of them (a process that drives two GPUs would get a
    launch error on the second)."""
    for src in sorted((_lib.lib_path().parent.parent / "csrc").glob("*.cu")):
        text = src.read_text()
        if "MaxDynamicSharedMemorySize" in text or "allow_shared(" in text:
            assert not re.search(r"static\s+bool\s+\w+\s*(=|;)", text), src.name


def test_expanded_weights_are_not_read_ahead(monkeypatch):
    """A GEMM asks for its first weights before the kernel ahead of it has ended. Where that kernel expands the weights into a buffer the
    call has to say so: nothing else orders the two."""
    seen = []
    monkeypatch.setattr(ops, "linear", lambda x, w, **kw: seen.append(kw.get("w_fresh", False)))
    monkeypatch.setattr(ops, "glu_linear", lambda x, w, *a, **kw: seen.append(kw.get("w_fresh", False)))
    monkeypatch.setattr(quant, "dequantize", lambda qt, out=None: out)
    monkeypatch.setattr(quant, "_TMP", {})
    monkeypatch.setattr(_lib, "load", lambda: None)
    packed, dense = quant.quantize(torch.randn(32, 64), "affine", 4, 64), torch.randn(32, 64)
    x = SimpleNamespace(is_cuda=True, shape=(300, 64), device=torch.device("cpu"))
    quant.qlinear(x, packed)
    for w in (packed, dense):
        moe._shared_expert(SimpleNamespace(hidden_act="silu"), SimpleNamespace(shared_gate_up=w, shared_down=w, shared_gate=None), x)
    assert seen == [True, True, True, False, False]
    # the re-tiled copy of packed weights: built by the first call
    assert [quant.quant_extras(packed, 1)[1].w_fresh for _ in range(2)] == [1, 0]
    assert _lib.gemm_extras(w_fresh=True).w_fresh == 1 and _lib.gemm_extras() is None


@pytest.mark.parametrize("M,N,glu,pairs", [(256, 4096, 0, 0), (257, 264, 0, 1), (257, 264, 1, 1), (512, 128, 0, 0), (512, 136, 0, 1), (600, 136, 0, 1),
                                           (300, 28672, 0, 0), (543, 28672, 0, 1), (543, 14336, 1, 0), (2048, 14336, 1, 1), (8192, 4096, 0, 1),
                                           (512, 4100, 0, 0)])
def test_gemms_on_pairs_of_sms(lib, M, N, glu, pairs):
    """More than 256 rows, features in 16-byte pieces, and no last wave of tiles that costs more than the pairing gives."""
    assert lib.mx_gemm_on_pairs(M, N, glu) == pairs
