"""Numerics of every CUDA kernel against the plain PyTorch fp32 statement of the same op."""
import math

import pytest
import torch

from mlxcel_b200 import ops
from mlxcel_b200.ops import KVLayer, reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _bf(*shape, scale=1.0, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(torch.bfloat16)


def _close(got, want, rtol=2e-2, atol=2e-2):
    got, want = got.float(), want.float()
    err = (got - want).abs()
    tol = atol + rtol * want.abs()
    bad = (~((err <= tol) | (got == want))).sum().item()          # (a NaN is no match)
    assert bad == 0, f"{bad}/{err.numel()} mismatches, max err {err.max().item():.4g}, ref max {want.abs().max().item():.4g}"


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    torch.cuda.synchronize()
    from mlxcel_b200.ops import _lib
    assert _lib.read_status(torch.device(DEV)) == 0


# ----------------------------------------------------------------------------- GEMM
@pytest.mark.parametrize("M,N,K", [
    (1, 128, 64), (16, 256, 128), (17, 384, 512), (64, 4096, 4096), (64, 1024, 1096),
    (128, 6144, 4096), (200, 512, 256), (256, 1000, 512), (257, 512, 512), (300, 768, 1024),
    (1024, 4096, 4096), (1000, 1032, 520), (4096, 256, 8192),
])
def test_gemm_plain(M, N, K):
    x, w = _bf(M, K, seed=1), _bf(N, K, scale=0.05, seed=2)
    got = ops.linear(x, w)
    _close(got, ref.linear(x, w), atol=2e-2 * math.sqrt(K) * 0.05)


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("M", [48, 130])
def test_gemm_forced_modes(mode, M):
    x, w = _bf(M, 512, seed=3), _bf(640, 512, scale=0.05, seed=4)
    got = ops.linear(x, w, force_mode=mode)
    _close(got, ref.linear(x, w))


@pytest.mark.parametrize("splits", [1, 2, 4, 7])
def test_gemm_split_k_deterministic(splits):
    x, w = _bf(32, 4096, seed=5), _bf(512, 4096, scale=0.05, seed=6)
    a = ops.linear(x, w, force_mode=2, force_splits=splits)
    b = ops.linear(x, w, force_mode=2, force_splits=splits)
    _close(a, ref.linear(x, w), atol=5e-2)
    assert torch.equal(a, b)


@pytest.mark.parametrize("M", [8, 64, 512])
def test_gemm_bias_residual_fp32(M):
    x, w = _bf(M, 1024, seed=7), _bf(768, 1024, scale=0.05, seed=8)
    bias, res = _bf(768, seed=9), _bf(M, 768, seed=10)
    _close(ops.linear(x, w, bias=bias), ref.linear(x, w, bias))
    _close(ops.linear(x, w, bias=bias, residual=res), ref.linear(x, w, bias, res))
    _close(ops.linear(x, w, out_fp32=True), ref.linear(x, w, out_dtype=torch.float32))
    # in-place residual accumulate
    h = res.clone()
    ops.linear(x, w, residual=h, out=h)
    _close(h, ref.linear(x, w, None, res))


@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "clipped_swiglu"])
@pytest.mark.parametrize("M", [4, 64, 128, 700])
def test_gemm_glu(act, M):
    I, K = 896, 512
    x, w = _bf(M, K, seed=11), _bf(2 * I, K, scale=0.08, seed=12)
    bias = _bf(2 * I, scale=0.1, seed=13) if act == "clipped_swiglu" else None
    got = ops.glu_linear(x, w, I, act, bias=bias)
    want = ref.glu_linear(x, w, I, ops._ACT_TO_EPI[act], bias)
    _close(got, want)


# ----------------------------------------------------------------------------- norms
@pytest.mark.parametrize("rows,dim", [(1, 256), (64, 4096), (33, 5120), (7, 2880), (3, 16384)])
def test_add_rmsnorm(rows, dim):
    x, r, w = _bf(rows, dim, seed=1), _bf(rows, dim, seed=2), _bf(dim, seed=3)
    y, h = ops.add_rmsnorm(x, r, w, 1e-5)
    yr, hr = ref.add_rmsnorm(x, r, w, 1e-5)
    assert torch.equal(h, hr)
    _close(y, yr, rtol=1e-2, atol=1e-2)
    y2 = ops.rmsnorm(x, w, 1e-6, 1.0)
    _close(y2, ref.add_rmsnorm(x, None, w, 1e-6, 1.0)[0], rtol=1e-2, atol=1e-2)


# ----------------------------------------------------------------------------- rope + append
def _pool(nb, Hkv, bs, D, bits):
    if bits == 16:
        return KVLayer(torch.zeros(nb, Hkv, bs, D, dtype=torch.bfloat16, device=DEV),
                       torch.zeros(nb, Hkv, bs, D, dtype=torch.bfloat16, device=DEV), None, None, bs, 16)
    Dq = D if bits == 8 else D // 2        # 4-bit: two codes per byte
    return KVLayer(torch.zeros(nb, Hkv, bs, Dq, dtype=torch.uint8, device=DEV),
                   torch.zeros(nb, Hkv, bs, Dq, dtype=torch.uint8, device=DEV),
                   torch.zeros(nb, Hkv, bs, D // 64, 2, dtype=torch.bfloat16, device=DEV),
                   torch.zeros(nb, Hkv, bs, D // 64, 2, dtype=torch.bfloat16, device=DEV), bs, bits)


@pytest.mark.parametrize("Hq,Hkv,D,qk", [(64, 8, 64, False), (32, 8, 128, True), (10, 2, 64, True)])
@pytest.mark.parametrize("vec", ["1", "0"])
def test_rope_append_prefill_sized(Hq, Hkv, D, qk, vec):
    """Enough tokens that a warp owns several heads (the launch grows heads-per-warp with T): both
    forms of the register-resident kernel against the fp32 statement."""
    from mlxcel_b200.ops import _lib
    T, bs = 2100, 16
    nb = (T + bs - 1) // bs + 2
    qkv = _bf(T, (Hq + 2 * Hkv) * D, seed=14)
    pos = torch.randint(0, 9000, (T,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(nb * bs, device=DEV)[:T].to(torch.int32)
    slots[::97] = -1
    inv, _ = ref.rope_inv_freq(D, 150000.0, None)
    inv = inv.to(DEV)
    qn = _bf(D, seed=5) if qk else None
    kn = _bf(D, seed=6) if qk else None
    kv = _pool(nb, Hkv, bs, D, 16)
    kv_ref = _clone_pool(kv)
    q_ref = qkv.clone()
    _lib.load().mx_set_rope_vec(int(vec))
    try:
        ops.rope_append(qkv, pos, slots, inv, kv, Hq=Hq, Hkv=Hkv, D=D, rot_dim=D, traditional=False,
                        mscale=1.0, q_norm_w=qn, k_norm_w=kn, norm_eps=1e-6)
    finally:
        _lib.load().mx_set_rope_vec(1)
    ref.rope_append(q_ref, pos, slots, inv, kv_ref, Hq=Hq, Hkv=Hkv, D=D, rot_dim=D, traditional=False,
                    mscale=1.0, q_norm_w=qn, k_norm_w=kn, norm_eps=1e-6)
    _close(qkv[:, : Hq * D], q_ref[:, : Hq * D], rtol=2e-2, atol=3e-2)
    _close(kv.k, kv_ref.k, rtol=2e-2, atol=3e-2)
    assert torch.equal(kv.v, kv_ref.v)


def _clone_pool(kv):
    c = lambda t: None if t is None else t.clone()  # noqa: E731
    return KVLayer(c(kv.k), c(kv.v), c(kv.k_meta), c(kv.v_meta), kv.block_size, kv.kv_bits)


@pytest.mark.parametrize("Hq,Hkv,D,rot,trad,qk", [
    (8, 2, 128, 128, False, False), (4, 4, 64, 64, True, False), (8, 1, 128, 64, False, True),
    (16, 2, 64, 64, False, True), (4, 2, 256, 256, False, False), (4, 1, 256, 0, False, True),
    (8, 2, 64, 64, False, False), (8, 2, 128, 128, False, True), (5, 1, 64, 64, False, True), (3, 1, 128, 128, False, False),
])
@pytest.mark.parametrize("bits", [16, 8, 4])
def test_rope_append(Hq, Hkv, D, rot, trad, qk, bits):
    T, bs, nb = 37, 16, 12
    qkv = _bf(T, (Hq + 2 * Hkv) * D, seed=4)
    pos = torch.randint(0, 5000, (T,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(nb * bs, device=DEV)[:T].to(torch.int32)
    slots[5] = -1
    inv, ms = ref.rope_inv_freq(rot, 500000.0, dict(rope_type="llama3", factor=8.0, low_freq_factor=1.0,
                                                    high_freq_factor=4.0,
                                                    original_max_position_embeddings=8192))
    inv = inv.to(DEV)
    qn = _bf(D, seed=5) if qk else None
    kn = _bf(D, seed=6) if qk else None
    kv = _pool(nb, Hkv, bs, D, bits)
    kv_ref = _clone_pool(kv)
    q_ref = qkv.clone()
    ops.rope_append(qkv, pos, slots, inv, kv, Hq=Hq, Hkv=Hkv, D=D, rot_dim=rot, traditional=trad,
                    mscale=1.1, q_norm_w=qn, k_norm_w=kn, norm_eps=1e-6)
    ref.rope_append(q_ref, pos, slots, inv, kv_ref, Hq=Hq, Hkv=Hkv, D=D, rot_dim=rot, traditional=trad,
                    mscale=1.1, q_norm_w=qn, k_norm_w=kn, norm_eps=1e-6)
    _close(qkv[:, : Hq * D], q_ref[:, : Hq * D], rtol=2e-2, atol=3e-2)
    if bits == 16:
        _close(kv.k, kv_ref.k, rtol=2e-2, atol=3e-2)
        assert torch.equal(kv.v, kv_ref.v)
    else:
        # a value that sits on a rounding boundary may land one code apart: one quantisation step of slack
        dq = ref.dequantize_kv4 if bits == 4 else ref.dequantize_kv8
        step = (kv_ref.k_meta[..., 0].float().abs().max().item() if bits == 4 else 0.0)
        _close(dq(kv.k, kv.k_meta), dq(kv_ref.k, kv_ref.k_meta), rtol=3e-2, atol=6e-2 + step)
        stepv = (kv_ref.v_meta[..., 0].float().abs().max().item() if bits == 4 else 0.0)
        _close(dq(kv.v, kv.v_meta), dq(kv_ref.v, kv_ref.v_meta), rtol=3e-2, atol=6e-2 + stepv)
        if bits == 4:
            # and exact agreement on the vast majority of codes
            assert (kv.v == kv_ref.v).float().mean().item() > 0.99


# ----------------------------------------------------------------------------- attention
def _fill_pool(kv, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    if kv.kv_bits == 16:
        kv.k.copy_(torch.randn(kv.k.shape, generator=g, device=DEV))
        kv.v.copy_(torch.randn(kv.v.shape, generator=g, device=DEV))
    else:
        for t, m in ((kv.k, kv.k_meta), (kv.v, kv.v_meta)):
            shape = t.shape if kv.kv_bits == 8 else (*t.shape[:-1], t.shape[-1] * 2)
            qz = ref.quantize_kv4 if kv.kv_bits == 4 else ref.quantize_kv8
            q, meta = qz(torch.randn(shape, generator=g, device=DEV))
            t.copy_(q)
            m.copy_(meta)


def _tables(lens, bs, nb, width):
    B = len(lens)
    perm = torch.randperm(nb)
    tab = torch.zeros(B, width, dtype=torch.int32)
    o = 0
    for i, n in enumerate(lens):
        k = (n + bs - 1) // bs
        tab[i, :k] = perm[o:o + k].to(torch.int32)
        o += k
    return tab.to(DEV)


@pytest.mark.parametrize("Hq,Hkv,D", [(8, 2, 128), (8, 8, 64), (8, 1, 128), (16, 2, 64), (8, 4, 256), (4, 1, 256)])
@pytest.mark.parametrize("bits,window,sinks,splits", [
    (16, 0, False, 1), (16, 0, False, 4), (16, 48, True, 3), (8, 0, False, 2), (8, 100, True, 1),
    (4, 0, False, 2), (4, 100, True, 1)])
def test_paged_decode(Hq, Hkv, D, bits, window, sinks, splits):
    bs, nb = 16, 256
    lens = [1, 15, 16, 17, 130, 513, 700, 64]
    B = len(lens)
    if bits == 4 and D == 256:
        pytest.skip("4-bit KV is served by the tensor-core kernels (head sizes 64 and 128)")
    kv = _pool(nb, Hkv, bs, D, bits)
    _fill_pool(kv, 3)
    tab = _tables(lens, bs, nb, 48)
    cl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    qkv = _bf(B, (Hq + 2 * Hkv) * D, seed=9)
    q = qkv[:, : Hq * D]
    sk = torch.randn(Hq, device=DEV) if sinks else None
    scale = 1.0 / math.sqrt(D)
    got = ops.paged_decode(q, kv, tab, cl, Hq=Hq, Hkv=Hkv, D=D, scale=scale, window=window,
                           sinks=sk, num_splits=splits)
    cu = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    want = ref.paged_attention(q, kv, tab, cl, cu, Hq=Hq, Hkv=Hkv, D=D, scale=scale, window=window,
                               sinks=sk)
    _close(got, want, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("Hq,Hkv,D", [(8, 2, 128), (4, 4, 64), (8, 1, 128), (16, 2, 64), (8, 4, 256), (4, 1, 256)])
@pytest.mark.parametrize("bits,window,sinks", [(16, 0, False), (16, 40, True), (8, 0, False), (4, 0, False), (4, 40, True)])
def test_paged_prefill(Hq, Hkv, D, bits, window, sinks):
    bs, nb = 16, 256
    ctx = [70, 300, 33, 129]       # total visible tokens per sequence
    qlen = [70, 45, 1, 129]        # the last qlen of them are queries
    S = len(ctx)
    kv = _pool(nb, Hkv, bs, D, bits)
    _fill_pool(kv, 5)
    tab = _tables(ctx, bs, nb, 24)
    cl = torch.tensor(ctx, dtype=torch.int32, device=DEV)
    cu = torch.tensor([0] + list(torch.tensor(qlen).cumsum(0)), dtype=torch.int32, device=DEV)
    T = sum(qlen)
    qkv = _bf(T, (Hq + 2 * Hkv) * D, seed=10)
    q = qkv[:, : Hq * D]
    sk = torch.randn(Hq, device=DEV) if sinks else None
    scale = 1.0 / math.sqrt(D)
    got = ops.paged_prefill(q, kv, tab, cu, cl, Hq=Hq, Hkv=Hkv, D=D, scale=scale, max_q_len=max(qlen),
                            window=window, sinks=sk)
    want = ref.paged_attention(q, kv, tab, cl, cu, Hq=Hq, Hkv=Hkv, D=D, scale=scale, window=window,
                               sinks=sk)
    _close(got, want, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("Hq,Hkv,D", [(8, 1, 128), (8, 2, 64), (4, 4, 64), (16, 1, 128), (12, 4, 128)])
@pytest.mark.parametrize("bits,window,sinks,softcap", [(16, 0, False, 0.0), (16, 40, True, 0.0), (8, 0, True, 0.0), (4, 24, False, 0.0),
                                                       (16, 0, False, 3.0), (8, 30, True, 3.0)])
@pytest.mark.parametrize("ctx,qlen", [([5, 300, 33, 4, 17], [1, 4, 3, 4, 2]), ([1500], [4]), ([2, 16, 640], [2, 1, 7])])
def test_paged_prefill_short_pieces(monkeypatch, Hq, Hkv, D, bits, window, sinks, softcap, ctx, qlen):
    """Pieces of a few tokens share 16-row tiles of the decode kernel: tiles that are full, partly filled and empty, contexts that
    end inside a key group or hold nothing but the piece, windows that begin inside a tile's tokens, key splits that are merged
    (one sequence) and splits without keys."""
    if (bits != 16 or softcap) and Hq // Hkv not in (1, 2, 4, 8):
        pytest.skip("quantized pools and soft caps: 1, 2, 4 or 8 query heads a key head")
    # (the packed form whatever the dispatch would take; key splits as a decode step has them)
    monkeypatch.setattr(ops, "packed_splits", lambda S, max_q, Hq, Hkv, D, keys, coded, tc: ops.decode_splits(
        S * -(-max_q // (16 // (Hq // Hkv))), Hkv, keys))
    bs, nb = 16, 256
    kv = _pool(nb, Hkv, bs, D, bits)
    _fill_pool(kv, 6)
    tab = _tables(ctx, bs, nb, 100)
    cl = torch.tensor(ctx, dtype=torch.int32, device=DEV)
    cu = torch.tensor([0] + list(torch.tensor(qlen).cumsum(0)), dtype=torch.int32, device=DEV)
    q = _bf(sum(qlen), (Hq + 2 * Hkv) * D, seed=12)[:, : Hq * D]
    sk = torch.randn(Hq, device=DEV) if sinks else None
    kw = dict(Hq=Hq, Hkv=Hkv, D=D, scale=1.0 / math.sqrt(D), window=window, sinks=sk, softcap=softcap)
    took, lib = [], ops._lib.load()
    real = lib.mx_paged_verify
    monkeypatch.setattr(lib, "mx_paged_verify", lambda *a: took.append(real(*a)) or took[-1])
    out = torch.full((sum(qlen), Hq * D), float("nan"), dtype=torch.bfloat16, device=DEV)
    got = ops.paged_prefill(q, kv, tab, cu, cl, max_q_len=max(qlen), out=out, **kw)
    _close(got, ref.paged_attention(q, kv, tab, cl, cu, **kw), rtol=2e-2, atol=2e-2)
    assert took == ([0] if max(qlen) <= 4 * (16 // (Hq // Hkv)) else [])
    # the kernels for longer pieces give the same
    monkeypatch.setattr(ops, "packed_splits", lambda *a: 0)
    _close(got, ops.paged_prefill(q, kv, tab, cu, cl, max_q_len=max(qlen), **kw), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("M,N,K", [(257, 264, 8), (512, 512, 512), (600, 136, 200), (1000, 1032, 1000), (2304, 4096, 448)])
@pytest.mark.parametrize("form", ["plain", "bias", "residual", "gated"])
def test_gemm_on_sm_pairs(M, N, K, form):
    """Many-row projections on pairs of SMs: ragged rows, features and K, one k-slice, several tiles a pair, a single pair; against
    64 bits, rounded once to bf16 (2^-8), with 1e-5 of the magnitudes for the order of the sums (gated: and for fast exp)."""
    from mlxcel_b200.ops import _lib
    assert _lib.load().mx_gemm_on_pairs(M, N, form == "gated") == 1
    x, w = _bf(M, K, seed=1), _bf(2 * N if form == "gated" else N, K, seed=2, scale=0.05)
    b = _bf(w.shape[0], seed=3) if form in ("bias", "gated") else None
    res = _bf(M, N, seed=4) if form == "residual" else None
    z = x.double() @ w.double().t() + (0 if b is None else b.double())
    size = x.double().abs() @ w.double().abs().t() + 4
    if form == "gated":
        got = ops.glu_linear(x, w, N, "silu", bias=b)
        size = 1.1 * size[:, :N] * (z[:, N:].abs() + 1) + z[:, :N].abs() * size[:, N:]      # |silu'| < 1.1
        z = torch.nn.functional.silu(z[:, :N]) * z[:, N:]
    else:
        got = ops.linear(x, w, bias=b, residual=res)
        z = z if res is None else z + res.double()
    err = (got.double() - z).abs()
    assert (err <= z.abs() * 2 ** -8 + size * 1e-5 + 1e-6).all(), err.max().item()
    assert _lib.read_status(torch.device(DEV)) == 0


@pytest.mark.parametrize("M", [1, 16, 64, 200, 700])
def test_gemm_deferred_rmsnorm(M):
    """producer GEMM (+residual) leaves per-tile sums of squares; consumer GEMMs (plain and gated)
    fed with the un-normalised stream and norm-folded weights match norm-then-project."""
    H, N2, I = 1024, 768, 512
    eps = 1e-5
    a = _bf(M, 256, seed=1)
    wo = _bf(H, 256, seed=2, scale=0.05)
    res = _bf(M, H, seed=3)
    ln = (1.0 + 0.1 * torch.randn(H, device=DEV)).to(torch.bfloat16)
    w2 = _bf(N2, H, seed=4, scale=0.05)
    wg = _bf(2 * I, H, seed=5, scale=0.05)
    bias = _bf(N2, seed=6)
    ssq = ops.SsqBuffer(1024, H // 128, DEV)
    h = ops.linear(a, wo, residual=res.clone(), ssq_out=ssq)
    want_h = ref.linear(a, wo, None, res)
    _close(h, want_h, rtol=2e-2, atol=2e-2)
    parts = int(ssq.buf[:1].view(torch.int32).item())
    got_ss = ssq.buf[8:8 + parts * ssq.max_tokens].view(parts, ssq.max_tokens)[:, :M].sum(0)
    _close(got_ss, h.float().pow(2).sum(-1), rtol=1e-3, atol=1e-3)
    # consumers
    fold = lambda w: (w.float() * ln.float().unsqueeze(0)).to(torch.bfloat16)
    rn = ops.RowNorm(ssq, eps, H)
    x = ref.add_rmsnorm(h, None, ln, eps, 0.0)[0]
    _close(ops.linear(h, fold(w2), bias=bias, row_norm=rn), ref.linear(x, w2, bias, None), rtol=3e-2, atol=3e-2)
    # gate * up compounds the rounding differences of two dot products (folded weight in bf16,
    # normalised input not rounded to bf16): wider absolute tolerance
    _close(ops.glu_linear(h, fold(wg), I, "silu", row_norm=rn), ref.glu_linear(x, wg, I, ops.EPI_SWIGLU, None, 1.702, 7.0),
           rtol=5e-2, atol=1e-1)
    # a chain started by row_ssq (one partial)
    ops.row_ssq(h, ssq)
    _close(ops.linear(h, fold(w2), row_norm=rn), ref.linear(x, w2, None, None), rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("Hq,Hkv,D", [(2, 1, 128), (8, 2, 128), (4, 2, 64), (16, 1, 64), (6, 1, 128)])
@pytest.mark.parametrize("ctx,qlen,window,sinks", [([128, 129, 700], [128, 129, 257], 0, False), ([1500, 127], [1000, 127], 0, True),
                                                   ([900, 300, 1], [300, 300, 1], 130, True), ([2300], [260], 1, False)])
@pytest.mark.parametrize("heads", [1, 2])
def test_paged_prefill_two_heads(monkeypatch, heads, Hq, Hkv, D, ctx, qlen, window, sinks):
    """Two query heads of a key head per CTA, and one, whatever the dispatch would take: one key tile and many, tiles that end on an
    edge, behind it and inside a row, a single row, windows of one key and across tiles, large logits that move the running maximum
    by more than the rescaling threshold."""
    monkeypatch.setattr(ops, "_PREFILL_HEADS", heads)
    bs, nb = 16, 512
    kv = _pool(nb, Hkv, bs, D, 16)
    _fill_pool(kv, 7)
    tab = _tables(ctx, bs, nb, 160)
    cl = torch.tensor(ctx, dtype=torch.int32, device=DEV)
    cu = torch.tensor([0] + list(torch.tensor(qlen).cumsum(0)), dtype=torch.int32, device=DEV)
    qkv = _bf(sum(qlen), (Hq + 2 * Hkv) * D, seed=11)
    qkv[::37] *= 6.0
    q = qkv[:, : Hq * D]
    kw = dict(Hq=Hq, Hkv=Hkv, D=D, scale=1.0 / math.sqrt(D), window=window, sinks=torch.randn(Hq, device=DEV) if sinks else None)
    out = torch.full((sum(qlen), Hq * D), float("nan"), dtype=torch.bfloat16, device=DEV)
    got = ops.paged_prefill(q, kv, tab, cu, cl, max_q_len=max(qlen), out=out, **kw)
    _close(got, ref.paged_attention(q, kv, tab, cl, cu, **kw), rtol=2e-2, atol=2e-2)
    from mlxcel_b200.ops import _lib
    assert _lib.read_status(torch.device(DEV)) == 0


@pytest.mark.parametrize("tc", [True, False])
@pytest.mark.parametrize("Hq,Hkv,D,window,sinks", [(8, 2, 128, 0, False), (4, 1, 64, 300, True), (4, 4, 128, 130, False)])
def test_paged_prefill_long(monkeypatch, tc, Hq, Hkv, D, window, sinks):
    """Many key tiles per query tile (running-max rescaling, window edges inside tiles, a prefix
    longer than the chunk) on the tensor-core kernel and on the fallback."""
    monkeypatch.setattr(ops, "_PREFILL_TC", tc)
    bs, nb = 16, 512
    ctx = [1500, 700, 257]
    qlen = [900, 700, 130]
    kv = _pool(nb, Hkv, bs, D, 16)
    _fill_pool(kv, 7)
    tab = _tables(ctx, bs, nb, 96)
    cl = torch.tensor(ctx, dtype=torch.int32, device=DEV)
    cu = torch.tensor([0] + list(torch.tensor(qlen).cumsum(0)), dtype=torch.int32, device=DEV)
    T = sum(qlen)
    # a few large logits so that the running maximum moves by more than the rescaling threshold
    qkv = _bf(T, (Hq + 2 * Hkv) * D, seed=11)
    qkv[::37] *= 6.0
    q = qkv[:, : Hq * D]
    sk = torch.randn(Hq, device=DEV) if sinks else None
    scale = 1.0 / math.sqrt(D)
    got = ops.paged_prefill(q, kv, tab, cu, cl, Hq=Hq, Hkv=Hkv, D=D, scale=scale, max_q_len=max(qlen),
                            window=window, sinks=sk)
    want = ref.paged_attention(q, kv, tab, cl, cu, Hq=Hq, Hkv=Hkv, D=D, scale=scale, window=window,
                               sinks=sk)
    _close(got, want, rtol=2e-2, atol=2e-2)
    from mlxcel_b200.ops import _lib
    assert _lib.read_status(torch.device(DEV)) == 0


# ----------------------------------------------------------------------------- misc + sampling
def test_embedding_argmax():
    table = _bf(1000, 256, seed=1)
    ids = torch.tensor([0, 999, 5, -1, 1000, 17], dtype=torch.int32, device=DEV)
    assert torch.equal(ops.embedding(ids, table), ref.embedding(ids, table))
    _close(ops.embedding(ids, table, 16.0), ref.embedding(ids, table, 16.0), rtol=1e-2, atol=1e-2)
    for V in (1000, 128256, 201088 + 3):
        lg = _bf(5, V, seed=V)
        lg[2, V - 1] = 100.0
        lg[3, 0] = float("nan")
        assert torch.equal(ops.argmax(lg), ref.argmax(lg))
        lf = lg.float()
        assert torch.equal(ops.argmax(lf), ref.argmax(lf))


def test_sample_matches_reference_stream():
    B, V = 6, 5000
    lg = (torch.randn(B, V, device=DEV) * 3).float()
    temp = torch.tensor([0.0, 1.0, 0.7, 1.3, 1.0, 0.5], device=DEV)
    tk = torch.tensor([0, 0, 40, 0, 1, 5], dtype=torch.int32, device=DEV)
    tp = torch.tensor([1.0, 1.0, 1.0, 0.9, 1.0, 0.8], device=DEV)
    mp = torch.tensor([0.0, 0.0, 0.0, 0.05, 0.0, 0.0], device=DEV)
    seeds = torch.tensor([1, 2, 3, 4, 5, 6], dtype=torch.int64, device=DEV)
    for step in (0, 1, 77):
        steps = torch.full((B,), step, dtype=torch.int64, device=DEV)
        got, lp = ops.sample(lg, temp, tk, tp, mp, seeds, steps)
        want, lpr = ref.sample(lg, temp, tk, tp, mp, seeds, steps)
        assert got.tolist() == want.tolist()
        _close(lp, lpr, rtol=1e-3, atol=1e-3)


def test_sample_typical_p_and_top_n_sigma_match_reference():
    """The typical-p and top-n-sigma stages of the fused sampler against the PyTorch reference chain:
    the same Philox stream, so the drawn tokens agree unless a token sits on a cut's boundary (the
    kernel evaluates the cuts in fp32, the reference in fp64); every drawn token must lie in the
    reference's kept set for a slightly wider cut."""
    B, V = 8, 5000
    g = torch.Generator().manual_seed(5)
    lg = (torch.randn(B, V, generator=g) * 3).float().to(DEV)
    temp = torch.tensor([1.0, 0.8, 1.2, 1.0, 1.0, 0.7, 1.0, 1.5], device=DEV)
    tk = torch.tensor([0, 0, 50, 0, 0, 0, 200, 0], dtype=torch.int32, device=DEV)
    tp = torch.tensor([1.0, 1.0, 1.0, 0.95, 1.0, 1.0, 1.0, 1.0], device=DEV)
    mp = torch.zeros(B, device=DEV)
    ty = torch.tensor([0.2, 0.5, 0.9, 0.6, 1.0, 1.0, 0.7, 0.95], device=DEV)
    ns = torch.tensor([0.0, 0.0, 0.0, 0.0, 1.0, 2.0, 1.5, 0.0], device=DEV)
    seeds = torch.arange(11, 11 + B, dtype=torch.int64, device=DEV)
    wide = []
    for b in range(B):
        l = lg[b].cpu()
        keep = ref.filter_mask(l, int(tk[b]), float(tp[b]), float(mp[b]))
        if float(ns[b]) > 0:
            keep &= ref.sigma_mask(l, float(ns[b]) * 1.02)
            keep[l.argmax()] = True
        if float(ty[b]) < 1.0:
            keep = ref.typical_mask(l, keep, min(1.0, float(ty[b]) + 0.02))
        wide.append(keep)
    same = total = 0
    for step in range(24):
        steps = torch.full((B,), step, dtype=torch.int64, device=DEV)
        got, lp = ops.sample(lg, temp, tk, tp, mp, seeds, steps, ty, ns)
        want, lpr = ref.sample(lg, temp, tk, tp, mp, seeds, steps, ty, ns)
        got, want = got.cpu().tolist(), want.cpu().tolist()
        for b in range(B):
            assert bool(wide[b][got[b]]), (b, step, got[b])
            same += got[b] == want[b]
            total += 1
    assert same >= 0.9 * total, (same, total)
    # the filters bite: a tight typical-p keeps far fewer tokens than the vocabulary
    assert int(wide[0].sum()) < V // 4


def test_sample_distribution_chi_square():
    V, N = 16, 4000
    probs = torch.softmax(torch.randn(V), 0)
    lg = torch.log(probs).to(DEV)[None].repeat(N, 1).contiguous()
    ones = torch.ones(N, device=DEV)
    got, _ = ops.sample(lg, ones, torch.zeros(N, dtype=torch.int32, device=DEV), ones,
                        torch.zeros(N, device=DEV), torch.arange(N, dtype=torch.int64, device=DEV),
                        torch.zeros(N, dtype=torch.int64, device=DEV))
    counts = torch.bincount(got.cpu().long(), minlength=V).float()
    chi2 = ((counts - N * probs) ** 2 / (N * probs)).sum().item()
    assert chi2 < 45.0, chi2  # 15 dof: P(chi2 > 45) < 1e-4


def test_penalties_and_verify():
    B, V = 3, 300
    lg = torch.randn(B, V, device=DEV)
    hist = torch.tensor([[1, 2, 2, -1], [5, 5, 5, 5], [-1, -1, -1, -1]], dtype=torch.int32, device=DEV)
    rep = torch.tensor([1.3, 1.0, 1.2], device=DEV)
    fr = torch.tensor([0.0, 0.5, 0.0], device=DEV)
    pr = torch.tensor([0.2, 0.0, 0.0], device=DEV)
    want = ref.apply_penalties(lg, hist, rep, fr, pr)
    got = ops.apply_penalties(lg.clone(), hist, rep, fr, pr)
    _close(got, want, rtol=1e-5, atol=1e-5)
    K = 4
    logits = torch.randn(B, K, V, device=DEV)
    tgt = logits.argmax(-1).to(torch.int32)
    draft = tgt[:, : K - 1].clone()
    draft[1, 1] = (draft[1, 1] + 1) % V
    draft[2, 0] = (draft[2, 0] + 1) % V
    t, a, n = ops.spec_verify(logits, draft)
    assert torch.equal(t, tgt) and a.tolist() == [3, 1, 0]
    assert n.tolist() == [int(tgt[0, 3]), int(tgt[1, 1]), int(tgt[2, 0])]


# ----------------------------------------------------------------------------- out-of-bounds canaries
@pytest.mark.parametrize("M,N,K", [(1, 136, 64), (7, 4096, 512), (65, 520, 192), (200, 1032, 256), (300, 264, 128),
                                   (1500, 1000, 320)])
def test_gemm_writes_stay_inside_the_output(M, N, K):
    """No compute-sanitizer on this pool: every kernel writes into a buffer with sentinel rows above
    and below and sentinel columns to the right (row stride > N); the sentinels must survive."""
    pad_r, ld = 3, N + 24
    SENT = -1234.0
    x = _bf(M, K, seed=1)
    w = _bf(N, K, seed=2, scale=0.05)
    res_full = torch.full((M + 2 * pad_r, ld), SENT, dtype=torch.bfloat16, device=DEV)
    out = res_full[pad_r:pad_r + M, :N]
    bias = _bf(N, seed=3)
    got = ops.linear(x, w, bias=bias, out=out)
    assert got.data_ptr() == out.data_ptr()
    _close(out, ref.linear(x, w, bias, None), rtol=2e-2, atol=2e-2)
    assert (res_full[:pad_r] == SENT).all() and (res_full[pad_r + M:] == SENT).all()
    assert (res_full[pad_r:pad_r + M, N:] == SENT).all()
    if N % 16 == 0:
        I = N // 2
        g_full = torch.full((M + 2 * pad_r, I + 8), SENT, dtype=torch.bfloat16, device=DEV)
        go = g_full[pad_r:pad_r + M, :I]
        ops.glu_linear(x, w, I, "silu", out=go)
        _close(go, ref.glu_linear(x, w, I, ops.EPI_SWIGLU, None, 1.702, 7.0), rtol=3e-2, atol=3e-2)
        assert (g_full[:pad_r] == SENT).all() and (g_full[pad_r + M:] == SENT).all()
        assert (g_full[pad_r:pad_r + M, I:] == SENT).all()


def test_attention_and_rope_writes_stay_inside_their_buffers():
    Hq, Hkv, D, bs, nb = 8, 2, 128, 16, 64
    SENT = -77.0
    ctx, qlen = [130, 47], [130, 20]
    kv = _pool(nb, Hkv, bs, D, 16)
    _fill_pool(kv, 3)
    tab = _tables(ctx, bs, nb, 16)
    cl = torch.tensor(ctx, dtype=torch.int32, device=DEV)
    cu = torch.tensor([0, qlen[0], sum(qlen)], dtype=torch.int32, device=DEV)
    T = sum(qlen)
    q = _bf(T, Hq * D, seed=4)
    full = torch.full((T + 6, Hq * D), SENT, dtype=torch.bfloat16, device=DEV)
    out = full[3:3 + T]
    ops.paged_prefill(q, kv, tab, cu, cl, Hq=Hq, Hkv=Hkv, D=D, scale=D ** -0.5, max_q_len=max(qlen), out=out)
    _close(out, ref.paged_attention(q, kv, tab, cl, cu, Hq=Hq, Hkv=Hkv, D=D, scale=D ** -0.5))
    assert (full[:3] == SENT).all() and (full[3 + T:] == SENT).all()
    # decode: B rows
    B = 2
    qd = _bf(B, Hq * D, seed=5)
    fulld = torch.full((B + 4, Hq * D), SENT, dtype=torch.bfloat16, device=DEV)
    ops.paged_decode(qd, kv, tab, cl, Hq=Hq, Hkv=Hkv, D=D, scale=D ** -0.5, out=fulld[2:2 + B])
    assert (fulld[:2] == SENT).all() and (fulld[2 + B:] == SENT).all()
    # rope + append: only the slots named in slot_mapping may change in the pool
    k_before, v_before = kv.k.clone(), kv.v.clone()
    Tn = 5
    qkv = _bf(Tn, (Hq + 2 * Hkv) * D, seed=6)
    slots = torch.tensor([3, 17, 40, 41, 1000], dtype=torch.int32, device=DEV)
    pos = torch.arange(Tn, dtype=torch.int32, device=DEV)
    inv = ref.rope_inv_freq(D, 10000.0, None)[0].to(DEV)
    ops.rope_append(qkv, pos, slots, inv, kv, Hq=Hq, Hkv=Hkv, D=D, rot_dim=D)
    touched = torch.zeros(nb * bs, dtype=torch.bool, device=DEV)
    touched[slots.long()] = True
    kb = (kv.k != k_before).view(nb, Hkv, bs, D).any(-1).any(1).view(-1)     # [nb * bs] slot changed?
    vb = (kv.v != v_before).view(nb, Hkv, bs, D).any(-1).any(1).view(-1)
    assert not (kb & ~touched).any() and not (vb & ~touched).any()
    assert kb[slots.long()].all()


# ----------------------------------------------------------------------------- end to end
@pytest.mark.parametrize("fold", [False, True])
def test_tiny_llama_gpu_matches_cpu_reference(fold):
    """bf16 CUDA executor vs the fp32 CPU executor: greedy tokens on a tiny model agree while the
    top-2 logit margin is not a near tie. ``fold``: RMSNorm weights folded into the projections and
    the norms deferred into the GEMM epilogues."""
    from mlxcel_b200.config import preset
    from mlxcel_b200.engine import Engine, EngineConfig, SamplingParams
    from mlxcel_b200.models.decoder import DecoderModel
    from mlxcel_b200.models.weights import random_weights
    import copy

    cfg = preset("tiny-llama")
    w32 = random_weights(cfg, seed=3, dtype=torch.float32, std=0.05)
    gn = torch.Generator().manual_seed(5)
    for lw in w32.layers:      # non-trivial norm weights
        lw.ln1 = lw.ln1 + 0.2 * torch.randn(lw.ln1.shape, generator=gn)
        lw.ln2 = lw.ln2 + 0.2 * torch.randn(lw.ln2.shape, generator=gn)
    w16 = copy.deepcopy(w32)
    for lw in [w16, *w16.layers]:
        for k, v in vars(lw).items():
            if isinstance(v, torch.Tensor):
                setattr(lw, k, v.to(torch.bfloat16).to(DEV) if v.dtype == torch.float32 and k != "sinks" else v.to(DEV))
    w16.lm_head = w16.embed
    ec = dict(max_batch=4, max_num_batched_tokens=256, num_blocks=64, max_model_len=256)
    cpu = Engine(DecoderModel(cfg, w32), cfg, EngineConfig(cuda_graphs=False, **ec))
    gpu = Engine(DecoderModel(cfg, w16, fold_norms=fold), cfg, EngineConfig(cuda_graphs=True, **ec))
    assert gpu.model.fold_attn == fold and gpu.model.fold_mlp == fold
    g = torch.Generator().manual_seed(1)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (20, 7, 33)]
    sp = SamplingParams(max_tokens=12, ignore_eos=True)
    a = [s.output for s in cpu.generate(prompts, sp)]
    b = [s.output for s in gpu.generate(prompts, sp)]
    agree = sum(x == y for sa, sb in zip(a, b) for x, y in zip(sa, sb))
    total = sum(len(s) for s in a)
    # a bf16 executor may flip a near tie and then diverge: most tokens must agree, and the
    # logits of one prefill pass must be close in absolute terms.
    assert agree >= 0.6 * total, (a, b)

    from mlxcel_b200.models.decoder import StepBatch
    ids = torch.tensor(prompts[0], dtype=torch.int32)
    T = ids.numel()

    def one_pass(eng, dev):
        kv = eng.pool.layers
        batch = StepBatch(token_ids=ids.to(dev), positions=torch.arange(T, dtype=torch.int32, device=dev),
                          slot_mapping=torch.arange(T, dtype=torch.int32, device=dev), num_decode=0,
                          num_prefill_seqs=1,
                          pf_block_tables=torch.arange(8, dtype=torch.int32, device=dev)[None],
                          pf_cu_q=torch.tensor([0, T], dtype=torch.int32, device=dev),
                          pf_context_lens=torch.tensor([T], dtype=torch.int32, device=dev), pf_max_q_len=T,
                          logits_rows=torch.tensor([T - 1], device=dev))
        return eng.model.forward(batch, kv).float().cpu()

    lc, lg = one_pass(cpu, "cpu"), one_pass(gpu, DEV)
    assert (lc - lg).abs().max().item() < 0.05 * lc.abs().max().item() + 0.02


@pytest.mark.parametrize("family,extra", [
    ("starcoder2", {}),                                              # LayerNorm + bias, plain GELU MLP
    ("cohere", {}),                                                  # parallel block, interleaved RoPE, logit scale
    ("olmo2", {}),                                                   # post-norm only, whole-projection q/k norm
    ("nemotron", {}),                                                # LayerNorm1P, partial rotary, relu^2 MLP
    ("apertus", {}),                                                 # xIELU MLP, per-head q/k norm
    ("smollm3", dict(num_hidden_layers=4, no_rope_layer_interval=2)),  # layers without positional encoding
    ("glm4_moe", dict(n_routed_experts=8, num_experts_per_tok=2, moe_intermediate_size=128, n_shared_experts=1,
                      n_group=2, topk_group=1, first_k_dense_replace=1, routed_scaling_factor=1.5, use_qk_norm=True)),
    ("deepseek_v3", dict(n_routed_experts=8, num_experts_per_tok=2, moe_intermediate_size=128, n_shared_experts=1,
                         n_group=2, topk_group=1, first_k_dense_replace=1, routed_scaling_factor=2.5, q_lora_rank=96,
                         kv_lora_rank=64, qk_nope_head_dim=64, qk_rope_head_dim=32, v_head_dim=64,
                         num_key_value_heads=4)),                      # MLA, keys padded 96 -> 128
    ("gemma3_text", dict(sliding_window=16, sliding_window_pattern=2, query_pre_attn_scalar=64,
                         rope_local_base_freq=10000.0, rope_theta=1000000.0)),
])
def test_less_common_layouts_gpu_matches_cpu(family, extra):
    """The layouts outside the main fused path (LayerNorm, plain MLPs, parallel blocks, post-norm only,
    NoPE layers, per-layer RoPE bases): bf16 GPU kernels against the fp32 CPU statement."""
    import copy

    from mlxcel_b200.cache.kv_pool import KVPool
    from mlxcel_b200.config import ModelConfig
    from mlxcel_b200.models.decoder import DecoderModel, StepBatch
    from mlxcel_b200.models.weights import random_weights
    from mlxcel_b200.ops import _lib

    raw = dict(model_type=family, num_hidden_layers=2, hidden_size=256, num_attention_heads=4, num_key_value_heads=2,
               head_dim=64, intermediate_size=512, vocab_size=512, max_position_embeddings=512)
    raw.update(extra)
    cfg = ModelConfig.from_dict(raw)
    w32 = random_weights(cfg, seed=5, dtype=torch.float32, std=0.05)
    w16 = copy.deepcopy(w32)
    for obj in [w16, *w16.layers]:
        for k, v in vars(obj).items():
            if isinstance(v, torch.Tensor):
                setattr(obj, k, (v.to(torch.bfloat16) if v.dtype == torch.float32 and k != "sinks" else v).to(DEV))
        if getattr(obj, "mla", None):
            obj.mla = {k: (None if v is None else v.to(torch.bfloat16).to(DEV)) for k, v in obj.mla.items()}
    if cfg.tie_word_embeddings:
        w16.lm_head = w16.embed
    T = 40
    ids = torch.randint(0, cfg.vocab_size, (T,), generator=torch.Generator().manual_seed(0), dtype=torch.int32)

    def logits(w, dev, dtype):
        pool = KVPool(cfg, 8, 16, device=dev, dtype=dtype)
        b = StepBatch(token_ids=ids.to(dev), positions=torch.arange(T, dtype=torch.int32, device=dev),
                      slot_mapping=torch.arange(T, dtype=torch.int32, device=dev), num_prefill_seqs=1,
                      pf_block_tables=torch.arange(8, dtype=torch.int32, device=dev)[None],
                      pf_cu_q=torch.tensor([0, T], dtype=torch.int32, device=dev),
                      pf_context_lens=torch.tensor([T], dtype=torch.int32, device=dev), pf_max_q_len=T,
                      logits_rows=torch.tensor([T - 1, T // 2], device=dev))
        return DecoderModel(cfg, w).forward(b, pool.layers).float().cpu()

    lc, lg = logits(w32, "cpu", torch.float32), logits(w16, DEV, torch.bfloat16)
    assert (lc - lg).abs().max().item() < 0.06 * lc.abs().max().item() + 0.03, family
    torch.cuda.synchronize()
    assert _lib.read_status(torch.device(DEV)) == 0


def test_layernorm_and_activations():
    from mlxcel_b200.ops import recurrent as R
    x = (torch.randn(37, 520, device=DEV) * 2 + 0.5).to(torch.bfloat16)
    w, b = (torch.randn(520, device=DEV) * 0.2 + 1).to(torch.bfloat16), (torch.randn(520, device=DEV) * 0.2).to(torch.bfloat16)
    for bias in (b, None):
        got = R.layernorm(x, w, bias, 1e-5)
        want = R.layernorm(x.cpu().float(), w.cpu().float(), None if bias is None else bias.cpu().float(), 1e-5)
        assert (got.float().cpu() - want).abs().max().item() < 0.05
    for kind in ("gelu_tanh", "gelu", "relu2", "silu"):
        got = R.activation(x, kind)
        want = R.activation(x.cpu().float(), kind)
        assert (got.float().cpu() - want).abs().max().item() < 0.05 + 0.01 * want.abs().max().item(), kind


@pytest.mark.parametrize("graphs", [True, False])
def test_speculative_rounds_on_gpu_reproduce_plain_decoding(graphs):
    """Verify rounds (draft-model drafter = the target itself, so every draft is accepted) through the
    device accept walk, replayed from a CUDA graph per (rows, K): the text equals plain greedy decoding
    of the same engine, and the rounds were actually graph replays."""
    from mlxcel_b200.config import preset
    from mlxcel_b200.engine import Engine, EngineConfig, SamplingParams
    from mlxcel_b200.models.decoder import DecoderModel
    from mlxcel_b200.models.weights import random_weights
    from mlxcel_b200.speculative import DraftModelDrafter

    cfg = preset("tiny-llama")
    w = random_weights(cfg, seed=3, dtype=torch.bfloat16, device=DEV, std=0.05)
    ec = dict(max_batch=4, max_num_batched_tokens=256, num_blocks=96, max_model_len=256, cuda_graphs=graphs)
    g = torch.Generator().manual_seed(1)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (20, 7, 33)]
    sp = SamplingParams(max_tokens=24, ignore_eos=True)
    plain = Engine(DecoderModel(cfg, w), cfg, EngineConfig(**ec))
    want = [s.output for s in plain.generate(prompts, sp)]
    eng = Engine(DecoderModel(cfg, w), cfg, EngineConfig(**ec))
    eng.drafter = DraftModelDrafter(DecoderModel(cfg, w), cfg, num_blocks=96, max_model_len=256)
    eng.spec_k = 4
    got = [s.output for s in eng.generate(prompts, sp)]
    st = eng.stats
    assert st["spec_rounds"] > 0 and st["spec_accepted"] > 0
    if graphs:
        assert st.get("verify_graph_replays", 0) > 0
    # block and chain passes use different tilings; a near tie may flip late
    agree = sum(x == y for a, b in zip(got, want) for x, y in zip(a, b)) / sum(len(b) for b in want)
    assert [a[:4] for a in got] == [b[:4] for b in want] and agree >= 0.8, (got, want)
    assert ops._lib.read_status(torch.device(DEV)) == 0
