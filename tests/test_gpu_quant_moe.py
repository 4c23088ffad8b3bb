"""Quantized-weight kernels, MoE routing / permutation / grouped GEMM vs PyTorch fp32 references."""
import pytest
import torch

from mlxcel_b200 import ops
from mlxcel_b200.ops import moe as moe_ops, quant

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(got, want, rtol=2e-2, atol=2e-2):
    got, want = got.float(), want.float()
    err = (got - want).abs()
    bad = (~((err <= atol + rtol * want.abs()) | (got == want))).sum().item()          # (a NaN is no match)
    assert bad == 0, f"{bad}/{err.numel()} mismatches, max err {err.max().item():.4g}"


def _qt_to(qt, dev):
    return qt.to(dev)


@pytest.mark.parametrize("mode,bits,group", [("affine", 2, 64), ("affine", 3, 32), ("affine", 4, 64),
                                             ("affine", 5, 64), ("affine", 6, 128), ("affine", 8, 64),
                                             ("mxfp4", 4, 32), ("mxfp8", 8, 32)])
def test_dequantize(mode, bits, group):
    w = torch.randn(96, 512) * 0.1
    qt = quant.quantize(w, mode, bits, group)
    want = quant.dequantize_ref(qt)
    got = quant.dequantize(_qt_to(qt, DEV))
    _close(got.cpu(), want, rtol=1e-2, atol=1e-3)


@pytest.mark.parametrize("mode,bits,group", [("affine", 4, 64), ("affine", 8, 64), ("affine", 4, 32),
                                             ("mxfp4", 4, 32), ("mxfp8", 8, 32), ("affine", 3, 64)])
@pytest.mark.parametrize("M", [1, 3, 8, 40, 300])
def test_qlinear(mode, bits, group, M):
    N, K = 384, 1024
    w = torch.randn(N, K) * 0.05
    qt = quant.quantize(w, mode, bits, group)
    wd = quant.dequantize_ref(qt)
    x = torch.randn(M, K).to(torch.bfloat16)
    res = torch.randn(M, N).to(torch.bfloat16)
    want = x.float() @ wd.t() + res.float()
    got = quant.qlinear(x.to(DEV), _qt_to(qt, DEV), residual=res.to(DEV))
    _close(got.cpu(), want, rtol=2e-2, atol=6e-2)


@pytest.mark.parametrize("N,K,group", [(1, 32, 32), (7, 1056, 32), (33, 2880, 64), (640, 4096, 64), (9475, 1024, 128)])
def test_one_row_affine4(N, K, group):
    """One row against affine 4-bit weights, plain (bias, residual) and gated: odd feature counts, rows of a single piece, a last
    round that only some lanes take part in, both rows-per-warp forms. Everything is summed in fp32 (1e-5 of the sum of magnitudes
    covers any order of it) and rounded once to bf16 (2^-8)."""
    g = torch.Generator().manual_seed(N + K)
    qt = _qt_to(quant.quantize(torch.randn(2 * N, K, generator=g) * 0.05, "affine", 4, group), DEV)
    wd = quant.dequantize_ref(_qt_to(qt, "cpu")).double()
    x = torch.randn(1, K, generator=g).to(torch.bfloat16)
    bias = torch.randn(2 * N, generator=g).to(torch.bfloat16)
    res = torch.randn(1, 2 * N, generator=g).to(torch.bfloat16)
    y, size = x.double() @ wd.t(), x.double().abs() @ wd.abs().t()

    def check(got, want, slack):
        err = (got.cpu().double() - want).abs()
        assert (err <= want.abs() * 2 ** -8 + slack * 1e-5 + 1e-6).all(), err.max().item()
    check(quant.qlinear(x.to(DEV), qt), y, size)
    check(quant.qlinear(x.to(DEV), qt, bias=bias.to(DEV), residual=res.to(DEV)), y + bias.double() + res.double(), size + 4)
    z = y + bias.double()
    want = torch.nn.functional.silu(z[:, :N]) * z[:, N:]
    slack = (1.1 * size[:, :N] + 1) * (z[:, N:].abs() + 1) + z[:, :N].abs() * (size[:, N:] + 1)      # |silu'| < 1.1
    check(quant.qglu_linear(x.to(DEV), qt, N, "silu", bias=bias.to(DEV)), want, slack)


@pytest.mark.parametrize("mode,group", [("mxfp4", 32), ("affine", 32), ("affine", 64), ("affine", 128)])
@pytest.mark.parametrize("counts,n_out,K", [([1], 16, 32), ([0, 9, 1, 40], 130, 2880), ([3, 0, 0, 0, 0, 0, 0, 2], 72, 1152),
                                            ([17, 33, 8, 16], 64, 640)])
@pytest.mark.parametrize("act", [None, "clipped_swiglu"])
def test_expert_streaming_shapes(monkeypatch, mode, group, counts, n_out, K, act):
    """Grouped 4-bit streaming products: scales that start inside a 32-bit word, a last block that is not full, K split over a
    cluster, experts without rows and with several passes, every column-tile form, features that do not fill a warp's tile."""
    if K % group:
        pytest.skip("rows are whole groups")
    monkeypatch.setattr(moe_ops, "_QGEMV_MAX_ROWS", 1 << 20)
    g = torch.Generator().manual_seed(K + n_out)
    E, rows = len(counts), sum(counts)
    w = torch.randn(E, n_out * (2 if act else 1), K, generator=g) * 0.05
    qt = quant.quantize(w, mode, 4, group)
    wd = quant.dequantize_ref(qt)
    xs = torch.randn(rows, K, generator=g).to(torch.bfloat16)
    off = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32)
    b = (torch.randn(E, w.shape[1], generator=g) * 0.1).to(torch.bfloat16)
    got = moe_ops.grouped_linear(xs.to(DEV), _qt_to(qt, DEV), off.to(DEV), n_out, b.to(DEV), act).cpu()
    for e in range(E):
        s = slice(int(off[e]), int(off[e + 1]))
        z = xs[s].float() @ wd[e].t() + b[e].float()
        if act:
            from mlxcel_b200.ops import reference as ref
            z = ref.glu_act(moe_ops._ACT_TO_EPI[act], z[:, :n_out], z[:, n_out:], 1.702, 7.0)
        _close(got[s], z, rtol=1e-2, atol=1e-2)


def test_one_row_of_strided_weights():
    """A gated projection of one row over a window of a wider packed matrix's columns: the rows do not lie back to back, so the
    one-row kernel, which takes them by pointer, must leave the call to the form that re-tiles them."""
    wide = _qt_to(quant.quantize(torch.randn(256, 512, generator=torch.Generator().manual_seed(3)) * 0.05, "affine", 4, 64), DEV)
    parts = [wide.packed[:, 32:], wide.scales[:, 4:], wide.biases[:, 4:]]
    x = torch.randn(1, 256, generator=torch.Generator().manual_seed(4)).to(torch.bfloat16).to(DEV)
    want = quant.qglu_linear(x, quant.QuantizedTensor(*(t.contiguous() for t in parts), 4, 64, "affine"), 128, "silu")
    for i in range(3):                                     # one strided part at a time, then all of them
        some = [t if j == i else t.contiguous() for j, t in enumerate(parts)]
        _close(quant.qglu_linear(x, quant.QuantizedTensor(*some, 4, 64, "affine"), 128, "silu"), want)
    _close(quant.qglu_linear(x, quant.QuantizedTensor(*parts, 4, 64, "affine"), 128, "silu"), want)


@pytest.mark.parametrize("mode,group,K", [("mxfp4", 32, 160), ("mxfp4", 32, 96), ("affine", 32, 160), ("affine", 64, 192)])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_expert_streaming_keeps_rows_apart(mode, group, K, value):
    """A weight row whose scales are not numbers spoils its own feature only. The last block of a row is not full there, so that
    the words its scales are fetched by hold the next row's as well."""
    E, n_out, rows = 3, 24, 5
    g = torch.Generator().manual_seed(K)
    qt = quant.quantize(torch.randn(E, n_out, K, generator=g) * 0.05, mode, 4, group)
    if mode == "mxfp4":
        qt.scales[:, 7] = 255
    else:
        qt.scales[:, 7], qt.biases[:, 7] = value, value
    xs = torch.randn(rows, K, generator=g).to(torch.bfloat16)
    off = torch.tensor([0, 2, 2, 5], dtype=torch.int32)
    got = moe_ops.grouped_linear(xs.to(DEV), _qt_to(qt, DEV), off.to(DEV), n_out).cpu().float()
    wd = quant.dequantize_ref(qt).float()
    want = torch.cat([xs[off[e]:off[e + 1]].float() @ wd[e].t() for e in range(E)])
    fine = torch.arange(n_out) != 7
    assert not got[:, 7].isfinite().any() and got[:, fine].isfinite().all()
    _close(got[:, fine], want[:, fine], rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("mode,bits,group", [("affine", 4, 64), ("affine", 4, 128), ("affine", 8, 32), ("mxfp4", 4, 32)])
@pytest.mark.parametrize("M", [1, 16, 64, 200])
def test_fused_dequant_gemm(monkeypatch, mode, bits, group, M):
    """Packed weights dequantised inside the tcgen05 GEMM (transform warps): plain with bias and
    residual, and the gated projection, for every batch size the path serves (M <= 256)."""
    monkeypatch.setattr(quant, "_QMV_MAX_M", 0)      # also M <= 8 through the GEMM path
    N, K, I = 640, 1536, 384                        # N not a multiple of the 128-row tile
    g = torch.Generator().manual_seed(M)
    w = torch.randn(N, K, generator=g) * 0.05
    qt = quant.quantize(w, mode, bits, group)
    wd = quant.dequantize_ref(qt)
    x = (torch.randn(M, K, generator=g)).to(torch.bfloat16)
    res = torch.randn(M, N, generator=g).to(torch.bfloat16)
    bias = torch.randn(N, generator=g).to(torch.bfloat16)
    assert quant.fused_wq(_qt_to(qt, DEV), M, K) != 0
    got = quant.qlinear(x.to(DEV), _qt_to(qt, DEV), residual=res.to(DEV))
    _close(got.cpu(), x.float() @ wd.t() + res.float(), rtol=2e-2, atol=6e-2)
    got = quant.qlinear(x.to(DEV), _qt_to(qt, DEV), bias=bias.to(DEV))
    _close(got.cpu(), x.float() @ wd.t() + bias.float(), rtol=2e-2, atol=6e-2)
    wg = torch.randn(2 * I, K, generator=g) * 0.05
    qg = quant.quantize(wg, mode, bits, group)
    y = x.float() @ quant.dequantize_ref(qg).t()
    want = torch.nn.functional.silu(y[:, :I]) * y[:, I:]
    got = quant.qglu_linear(x.to(DEV), _qt_to(qg, DEV), I, "silu")
    _close(got.cpu(), want, rtol=3e-2, atol=6e-2)


@pytest.mark.parametrize("mode,norm", [("topk_softmax", True), ("softmax_topk", True), ("softmax_topk", False)])
@pytest.mark.parametrize("E,k", [(8, 2), (128, 4), (60, 8)])
def test_route(mode, norm, E, k):
    lg = torch.randn(77, E, device=DEV).to(torch.bfloat16)
    ids, w = moe_ops.route(lg, k, mode, norm)
    ids_r, w_r = moe_ops.route_ref(lg, k, mode, norm)
    # compare as sets per row: order of equal logits may differ
    assert torch.equal(ids.sort(-1).values, ids_r.sort(-1).values)
    order, order_r = ids.argsort(-1), ids_r.argsort(-1)
    _close(w.gather(1, order), w_r.gather(1, order_r), rtol=1e-3, atol=1e-4)


@pytest.mark.parametrize("T,E,k,H,I,act", [(5, 8, 2, 256, 512, "silu"), (64, 16, 4, 256, 256, "clipped_swiglu"),
                                           (700, 8, 2, 512, 384, "silu"), (128, 32, 4, 2880 // 8 * 8, 256, "clipped_swiglu")])
@pytest.mark.parametrize("local", [False, True])
def test_moe_experts(T, E, k, H, I, act, local):
    g = torch.Generator(device=DEV).manual_seed(T + E)
    r = lambda *s, sc=1.0: (torch.randn(*s, generator=g, device=DEV) * sc).to(torch.bfloat16)  # noqa: E731
    x = r(T, H)
    lg = r(T, E)
    ids, wts = moe_ops.route(lg, k, "topk_softmax", True)
    e0, e1 = (E // 4, E // 2) if local else (0, E)
    wgu, wd = r(e1 - e0, 2 * I, H, sc=0.05), r(e1 - e0, H, I, sc=0.05)
    bias = act == "clipped_swiglu"
    bgu = r(e1 - e0, 2 * I, sc=0.1) if bias else None
    bd = r(e1 - e0, H, sc=0.1) if bias else None
    res = r(T, H)
    want = moe_ops.moe_ref(x, ids, wts, wgu, wd, I, act, bgu, bd, e_begin=e0) + res.float()
    got = moe_ops.moe_experts(x, ids, wts, wgu, wd, I, act, bgu, bd, e_begin=e0, residual=res)
    _close(got, want, rtol=3e-2, atol=5e-2)
    from mlxcel_b200.ops import _lib
    torch.cuda.synchronize()
    assert _lib.read_status(torch.device(DEV)) == 0


@pytest.mark.parametrize("mode,bits,group", [("mxfp4", 4, 32), ("affine", 4, 64)])
@pytest.mark.parametrize("T,E,k,H,I,act", [(5, 8, 2, 256, 512, "silu"), (64, 16, 4, 320, 192, "clipped_swiglu"),
                                           (128, 32, 4, 2880, 384, "clipped_swiglu")])
def test_moe_experts_packed(mode, bits, group, T, E, k, H, I, act):
    """Packed (mxfp4 / affine 4-bit) expert weights through the grouped fused dequant GEMM; hidden
    and expert sizes that are not multiples of the 128-row tile (gpt-oss: 2880)."""
    g = torch.Generator().manual_seed(T + E)
    r = lambda *s, sc=1.0: (torch.randn(*s, generator=g) * sc)  # noqa: E731
    x = r(T, H).to(torch.bfloat16).to(DEV)
    ids, wts = moe_ops.route(r(T, E).to(torch.bfloat16).to(DEV), k, "topk_softmax", True)
    qgu = quant.quantize(r(E, 2 * I, H, sc=0.05), mode, bits, group)
    qd = quant.quantize(r(E, H, I, sc=0.05), mode, bits, group)
    bias = act == "clipped_swiglu"
    bgu = r(E, 2 * I, sc=0.1).to(torch.bfloat16).to(DEV) if bias else None
    bd = r(E, H, sc=0.1).to(torch.bfloat16).to(DEV) if bias else None
    res = r(T, H).to(torch.bfloat16).to(DEV)
    wgu_d = quant.dequantize_ref(qgu).to(torch.bfloat16).to(DEV)
    wd_d = quant.dequantize_ref(qd).to(torch.bfloat16).to(DEV)
    want = moe_ops.moe_ref(x, ids, wts, wgu_d, wd_d, I, act, bgu, bd) + res.float()
    got = moe_ops.moe_experts(x, ids, wts, _qt_to(qgu, DEV), _qt_to(qd, DEV), I, act, bgu, bd, residual=res)
    _close(got, want, rtol=3e-2, atol=6e-2)
    from mlxcel_b200.ops import _lib
    torch.cuda.synchronize()
    assert _lib.read_status(torch.device(DEV)) == 0


@pytest.mark.parametrize("mode,bits,group", [("mxfp4", 4, 32), ("affine", 4, 64), ("affine", 4, 32)])
@pytest.mark.parametrize("T,E,k,H,I,act,skew", [(3, 8, 2, 256, 512, "silu", False), (24, 16, 4, 2880, 352, "clipped_swiglu", False),
                                                (40, 8, 2, 320, 200, "gelu_tanh", True), (128, 128, 4, 2880, 96, "clipped_swiglu", False)])
def test_moe_experts_weight_streaming_gemv(monkeypatch, mode, bits, group, T, E, k, H, I, act, skew):
    """Decode-sized groups take the grouped 4-bit GEMV (packed rows streamed once, activations in
    registers): experts without rows, one row, odd counts and one overloaded expert (several token
    passes), feature counts that do not fill the last block, against the dequantised fp32 reference."""
    monkeypatch.setattr(moe_ops, "_QGEMV_MAX_ROWS", 1 << 20)          # every case through the GEMV
    g = torch.Generator().manual_seed(T * 7 + E)
    r = lambda *s, sc=1.0: (torch.randn(*s, generator=g) * sc)  # noqa: E731
    x = r(T, H).to(torch.bfloat16).to(DEV)
    logits = r(T, E)
    if skew:
        logits[:, 3] += 6.0                                            # most tokens pick expert 3
    ids, wts = moe_ops.route(logits.to(torch.bfloat16).to(DEV), k, "topk_softmax", True)
    qgu = quant.quantize(r(E, 2 * I, H, sc=0.05), mode, bits, group)
    qd = quant.quantize(r(E, H, I, sc=0.05), mode, bits, group) if I % group == 0 and I % 32 == 0 else None
    bias = act == "clipped_swiglu"
    bgu = r(E, 2 * I, sc=0.1).to(torch.bfloat16).to(DEV) if bias else None
    bd = r(E, H, sc=0.1).to(torch.bfloat16).to(DEV) if bias else None
    wgu_d = quant.dequantize_ref(qgu).to(torch.bfloat16).to(DEV)
    wd = r(E, H, I, sc=0.05)
    wd_d = (quant.dequantize_ref(qd) if qd is not None else wd).to(torch.bfloat16).to(DEV)
    res = r(T, H).to(torch.bfloat16).to(DEV)
    want = moe_ops.moe_ref(x, ids, wts, wgu_d, wd_d, I, act, bgu, bd) + res.float()
    from mlxcel_b200.ops import _lib
    n0 = _lib.launches()
    got = moe_ops.moe_experts(x, ids, wts, _qt_to(qgu, DEV), _qt_to(qd, DEV) if qd is not None else wd_d, I, act, bgu, bd,
                              residual=res)
    _close(got, want, rtol=3e-2, atol=6e-2)
    torch.cuda.synchronize()
    assert _lib.read_status(torch.device(DEV)) == 0
    # the same call through the tensor-core path agrees too (both are checked against the reference above)
    monkeypatch.setattr(moe_ops, "_QGEMV_MAX_ROWS", 0)
    other = moe_ops.moe_experts(x, ids, wts, _qt_to(qgu, DEV), _qt_to(qd, DEV) if qd is not None else wd_d, I, act, bgu, bd,
                                residual=res)
    _close(other, want, rtol=3e-2, atol=6e-2)


def test_tiny_moe_models_gpu_vs_cpu_logits():
    from mlxcel_b200.config import preset
    from mlxcel_b200.models.decoder import DecoderModel, StepBatch
    from mlxcel_b200.models.weights import random_weights
    from mlxcel_b200.cache.kv_pool import KVPool
    import copy

    for name in ("tiny-moe", "tiny-gpt-oss", "tiny-qwen3"):
        cfg = preset(name)
        w32 = random_weights(cfg, seed=3, dtype=torch.float32, std=0.05)
        w16 = copy.deepcopy(w32)
        for obj in [w16, *w16.layers]:
            for kname, v in vars(obj).items():
                if isinstance(v, torch.Tensor):
                    setattr(obj, kname, (v.to(torch.bfloat16) if (v.dtype == torch.float32 and kname != "sinks") else v).to(DEV))
        T = 40
        ids = torch.randint(0, cfg.vocab_size, (T,), generator=torch.Generator().manual_seed(0), dtype=torch.int32)

        def one_pass(w, dev, dtype):
            pool = KVPool(cfg, 8, 16, device=dev, dtype=dtype)
            b = StepBatch(token_ids=ids.to(dev), positions=torch.arange(T, dtype=torch.int32, device=dev),
                          slot_mapping=torch.arange(T, dtype=torch.int32, device=dev), num_prefill_seqs=1,
                          pf_block_tables=torch.arange(8, dtype=torch.int32, device=dev)[None],
                          pf_cu_q=torch.tensor([0, T], dtype=torch.int32, device=dev),
                          pf_context_lens=torch.tensor([T], dtype=torch.int32, device=dev), pf_max_q_len=T,
                          logits_rows=torch.tensor([T - 1, T // 2], device=dev))
            return DecoderModel(cfg, w).forward(b, pool.layers).float().cpu()

        lc, lg = one_pass(w32, "cpu", torch.float32), one_pass(w16, DEV, torch.bfloat16)
        assert (lc - lg).abs().max().item() < 0.06 * lc.abs().max().item() + 0.03, name
