"""bf16 tcgen05 GEMM (C = A @ Bt^T, fp32 accumulation) through the C ABI against an fp64 product of the same
bf16-rounded operands.  Gate: max|got - ref| <= 2^-8 * max|ref| (one bf16 ulp at the largest magnitude) + the
accumulation-order slack of fp32, far below it."""
import numpy as np
import pytest
import torch

from oracle import ref_attention as R

pytestmark = pytest.mark.gpu


def run_case(M, N, K, seed):
    from baranet_bdml_b200 import ops
    rng = np.random.default_rng(seed)
    a = R.round_bf16(rng.standard_normal((M, K), dtype=np.float32))
    bt = R.round_bf16((rng.standard_normal((N, K)) * 0.05).astype(np.float32))
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ops.gemm_bf16_nt(torch.from_numpy(a).cuda().to(torch.bfloat16), torch.from_numpy(bt).cuda().to(torch.bfloat16),
                           error_word=err)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ref = a.astype(np.float64) @ bt.astype(np.float64).T
    return got.float().cpu().numpy(), ref


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 256, 2048), (256, 512, 128), (1, 8, 8), (100, 264, 72),
                                   (129, 257 // 8 * 8, 65 // 8 * 8), (300, 2048, 2048), (1000, 512, 2048),
                                   (4096, 256, 256)])
def test_gemm_matches_fp64_product(lib, M, N, K):
    got, ref = run_case(M, N, K, M + 3 * N + 7 * K)
    scale = max(np.abs(ref).max(), 1e-30)
    assert np.abs(got - ref).max() <= scale * 2.0 ** -8, (M, N, K, np.abs(got - ref).max() / scale)


def test_gemm_projection_shapes_of_the_layer(lib):
    """q_proj / k_proj of TinyLLaMA on 2048 tokens: (2048, 2048) @ (2048, 2048)^T and (2048, 2048) @ (256, 2048)^T;
    linearity in A: gemm(2a) == 2 gemm(a) exactly (a power-of-two scale commutes with every rounding)."""
    from baranet_bdml_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn((2048, 2048), generator=g, device="cuda").to(torch.bfloat16)
    for n_out in (2048, 256):
        w = (torch.randn((n_out, 2048), generator=g, device="cuda") * 0.02).to(torch.bfloat16)
        y = ops.gemm_bf16_nt(x, w)
        y2 = ops.gemm_bf16_nt((x.float() * 2).to(torch.bfloat16), w)
        torch.cuda.synchronize()
        assert torch.equal(y2.float(), y.float() * 2)
        ref = x.double() @ w.double().T
        assert float((y.double() - ref).abs().max()) <= float(ref.abs().max()) * 2.0 ** -8


# more tiles than multiprocessors and a long K: two CTAs share a tile of 256 x 256.  Odd numbers of 128-row tiles, rows and columns
# that fill no tile, K that fills no step, one pair more than run together
PAIRED = [(2569, 2048, 1024), (300, 19000, 1032), (1290, 4616, 1096), (256 * 75, 256, 1024), (4097, 1544, 2040)]


@pytest.mark.parametrize("M,N,K", PAIRED)
def test_paired_tiles_are_the_single_ones(lib, M, N, K):
    """Every epilogue on rows that come in one call (pairs) and in calls of few enough rows for single tiles: the same sums over the
    same k in the same order, so the same bits; and against fp64."""
    from baranet_bdml_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn((M, K), generator=g, device="cuda").bfloat16()
    w, u = ((torch.randn((N, K), generator=g, device="cuda") * K ** -0.5).bfloat16() for _ in "wu")
    bias = torch.randn(N, generator=g, device="cuda")
    mul = torch.randn((M, N), generator=g, device="cuda").bfloat16()
    packed = ops.pack_gate_up(w, u)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream

    def run(kind, r0, r1):
        a, m, rows = x[r0:r1], mul[r0:r1], r1 - r0
        out = torch.full((rows, N), 7.0, dtype=torch.float32 if kind == "f32" else torch.bfloat16, device="cuda")
        head, tail = (a.data_ptr(), w.data_ptr()), (rows, N, K, err.data_ptr(), st)
        if kind == "plain":
            rc = lib.bn_gemm_bf16_nt(*head, out.data_ptr(), *tail)
        elif kind == "f32":
            rc = lib.bn_gemm_bf16_nt_f32(*head, out.data_ptr(), *tail)
        elif kind == "bias":
            rc = lib.bn_gemm_bias_act_bf16_nt(*head, bias.data_ptr(), out.data_ptr(), rows, N, K, _lib.BN_ACT_RELU2, err.data_ptr(), st)
        elif kind == "mul":
            rc = lib.bn_gemm_act_mul_bf16_nt(*head, m.data_ptr(), m.stride(0), out.data_ptr(), rows, N, K, _lib.BN_ACT_SILU, err.data_ptr(), st)
        else:
            act = _lib.BN_ACT_SILU if kind == "silu" else _lib.BN_ACT_GELU_TANH
            rc = lib.bn_gemm_glu_bf16_nt(a.data_ptr(), packed.data_ptr(), out.data_ptr(), rows, N, K, act, err.data_ptr(), st)
        _lib.check(rc)
        return out

    few = max(1, 148 // (-(-2 * N // 256))) * 128
    for kind in ("plain", "f32", "bias", "mul", "silu", "gelu"):
        whole, parts = run(kind, 0, M), torch.cat([run(kind, r, min(M, r + few)) for r in range(0, M, few)])
        if few > 128:                       # (up to 128 rows some of them take other forms)
            assert torch.equal(whole, parts), kind
        if kind == "f32":
            exact = x.double() @ w.double().T
            assert ((whole.double() - exact).abs() <= K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)).all()
        else:
            assert ((whole.double() - parts.double()).abs() <= 2.0 ** -7 * parts.double().abs() + 2.0 ** -8).all(), kind
    assert int(err.item()) == 0


def test_gemm_rejects_bad_arguments(lib):
    from baranet_bdml_b200 import ops
    a = torch.zeros((16, 12), dtype=torch.bfloat16, device="cuda")
    with pytest.raises(RuntimeError, match="multiples of 8"):
        ops.gemm_bf16_nt(a, torch.zeros((8, 12), dtype=torch.bfloat16, device="cuda"))
    with pytest.raises(RuntimeError, match="inner dimensions mismatch"):
        ops.gemm_bf16_nt(torch.zeros((16, 16), dtype=torch.bfloat16, device="cuda"),
                         torch.zeros((8, 8), dtype=torch.bfloat16, device="cuda"))
    with pytest.raises(RuntimeError, match="only GPU implementation available"):
        ops.gemm_bf16_nt(torch.zeros((16, 16), dtype=torch.bfloat16), torch.zeros((8, 16), dtype=torch.bfloat16))


def test_bf16_layer_against_staged_fp64_restatement(lib):
    """The whole attention layer on the bf16 path (4 tcgen05 GEMMs + the fused attention core) against the oracle's
    per-head attention with fp64 arithmetic and a bf16 rounding wherever the kernels round (q, k, v, attention output,
    layer output).  Gate 2e-2 absolute, the bf16 tolerance of the path."""
    import torch
    from baranet_bdml_b200.layers import GroupedQueryAttentionBF16, LLaMAConfig
    cfg = LLaMAConfig(hidden_size=512, num_attention_heads=8, num_key_value_heads=2, intermediate_size=1024,
                      num_hidden_layers=1)
    np.random.seed(5)
    layer = GroupedQueryAttentionBF16(cfg)
    B, S = 2, 300
    rng = np.random.default_rng(8)
    x = R.round_bf16(rng.standard_normal((B, S, cfg.hidden_size), dtype=np.float32))
    got = layer(torch.from_numpy(x).cuda().to(torch.bfloat16), position_offset=2).float().cpu().numpy()
    wq, wk, wv, wo = (w.float().cpu().numpy().astype(np.float64) for w in (layer.q_proj, layer.k_proj, layer.v_proj,
                                                                          layer.o_proj))
    for b in range(B):
        xb = x[b].astype(np.float64)
        q, k, v = (R.round_bf16((xb @ w.T).astype(np.float32)) for w in (wq, wk, wv))
        attn = R.attention_per_head(q, k, v, num_heads=8, num_kv_heads=2, head_dim=64, position_offset=2, causal=True,
                                    dtype=np.float64, round_rope_bf16=True)
        ref = R.round_bf16(attn.astype(np.float32)).astype(np.float64) @ wo.T
        assert np.abs(got[b] - ref).max() <= 2e-2, np.abs(got[b] - ref).max()


@pytest.mark.parametrize("M,inter,K", [(128, 128, 64), (200, 256, 128), (64, 5632, 2048), (300, 136, 72), (1000, 1000, 512)])
def test_swiglu_gemm_against_fp64(lib, M, inter, K):
    """silu(x Wg) * (x Wu) from one launch against fp64 on the same bf16 operands; the kernel applies the activation
    to its fp32 accumulators and rounds once, so the gate is one bf16 ulp at the largest magnitude."""
    from baranet_bdml_b200 import ops
    rng = np.random.default_rng(M + inter + K)
    x = R.round_bf16(rng.standard_normal((M, K), dtype=np.float32))
    wg = R.round_bf16((rng.standard_normal((inter, K)) * 0.05).astype(np.float32))
    wu = R.round_bf16((rng.standard_normal((inter, K)) * 0.05).astype(np.float32))
    tx, tg, tu = (torch.from_numpy(a).cuda().to(torch.bfloat16) for a in (x, wg, wu))
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ops.gemm_swiglu_bf16_nt(tx, ops.pack_gate_up(tg, tu), inter, error_word=err).float().cpu().numpy()
    assert int(err.item()) == 0
    g = x.astype(np.float64) @ wg.astype(np.float64).T
    u = x.astype(np.float64) @ wu.astype(np.float64).T
    ref = g / (1.0 + np.exp(-g)) * u
    assert np.abs(got - ref).max() <= max(np.abs(ref).max(), 1e-30) * 2.0 ** -8


def test_bf16_mlp_against_staged_fp64(lib):
    """MLPBF16 (fused gate/up GEMM + down GEMM) against fp64 with a bf16 rounding of the intermediate, where the
    kernels round."""
    from baranet_bdml_b200.layers import LLaMAConfig, MLPBF16
    cfg = LLaMAConfig(hidden_size=512, num_attention_heads=8, num_key_value_heads=2, intermediate_size=1408,
                      num_hidden_layers=1)
    np.random.seed(2)
    mlp = MLPBF16(cfg)
    rng = np.random.default_rng(4)
    x = R.round_bf16(rng.standard_normal((333, 512), dtype=np.float32))
    got = mlp(torch.from_numpy(x).cuda().to(torch.bfloat16)).float().cpu().numpy()
    wg, wu, wd = (w.float().cpu().numpy().astype(np.float64) for w in (mlp.gate_proj, mlp.up_proj, mlp.down_proj))
    g, u = x.astype(np.float64) @ wg.T, x.astype(np.float64) @ wu.T
    inter = R.round_bf16((g / (1.0 + np.exp(-g)) * u).astype(np.float32)).astype(np.float64)
    ref = inter @ wd.T
    assert np.abs(got - ref).max() <= np.abs(ref).max() * 2.0 ** -7


def test_bf16_decoder_layer_against_staged_fp64(lib):
    """The whole pre-norm decoder block on the bf16 path (norm, attention layer, fused residual add + norm, SwiGLU MLP,
    residual) against fp64 with a bf16 rounding wherever a kernel rounds; and two stacked layers with the deferred
    residual add (`forward_parts(pending=...)`) equal to the plain composition."""
    from baranet_bdml_b200.layers import LLaMAConfig, LLaMADecoderLayerBF16
    cfg = LLaMAConfig(hidden_size=512, num_attention_heads=8, num_key_value_heads=2, intermediate_size=1408,
                      num_hidden_layers=2)
    np.random.seed(12)
    layer = LLaMADecoderLayerBF16(cfg)
    B, S, H = 2, 200, 512
    rng = np.random.default_rng(3)
    x = R.round_bf16(rng.standard_normal((B, S, H), dtype=np.float32))
    tx = torch.from_numpy(x).cuda().to(torch.bfloat16)
    got = layer(tx).float().cpu().numpy()

    rb = lambda a: R.round_bf16(np.asarray(a, dtype=np.float32)).astype(np.float64)
    f64 = lambda t: t.float().cpu().numpy().astype(np.float64)
    at, ml = layer.self_attn, layer.mlp
    wq, wk, wv, wo = f64(at.q_proj), f64(at.k_proj), f64(at.v_proj), f64(at.o_proj)
    wg, wu, wd = f64(ml.gate_proj), f64(ml.up_proj), f64(ml.down_proj)

    def norm(s):
        return rb(s / np.sqrt((s * s).mean(axis=1, keepdims=True) + cfg.rms_norm_eps))

    for b in range(B):
        h0 = x[b].astype(np.float64)
        n1 = norm(h0)
        q, k, v = rb(n1 @ wq.T), rb(n1 @ wk.T), rb(n1 @ wv.T)
        attn = rb(R.attention_per_head(q, k, v, num_heads=8, num_kv_heads=2, head_dim=64, causal=True, dtype=np.float64,
                                       round_rope_bf16=True))
        h1 = rb(h0 + rb(attn @ wo.T))
        n2 = norm(h1)
        g, u = n2 @ wg.T, n2 @ wu.T
        m = rb(rb(g / (1.0 + np.exp(-g)) * u) @ wd.T)
        ref = rb(h1 + m)
        err = np.abs(got[b] - ref).max()
        # the attention path's 2e-2 plus two bf16 ulps at the largest magnitude: a value that sits near a rounding
        # boundary may round the other way in the kernel and its neighbours downstream
        assert err <= 2e-2 + np.abs(ref).max() * 2.0 ** -7, (err, np.abs(ref).max())

    layer2 = LLaMADecoderLayerBF16(cfg)
    plain = layer2(layer(tx))
    res, pend = layer.forward_parts(tx)
    res2, pend2 = layer2.forward_parts(res, pending=pend)
    assert torch.equal(res2 + pend2, plain)


def test_graphed_decoder_layer_equals_eager(lib):
    """The block captured into a CUDA graph returns the bits of the eager block, call after call."""
    from baranet_bdml_b200.layers import GraphedDecoderLayerBF16, LLaMAConfig, LLaMADecoderLayerBF16
    cfg = LLaMAConfig(hidden_size=512, num_attention_heads=8, num_key_value_heads=2, intermediate_size=1408,
                      num_hidden_layers=1)
    np.random.seed(21)
    layer = LLaMADecoderLayerBF16(cfg)
    g = torch.Generator(device="cuda").manual_seed(1)
    xs = [torch.randn((2, 160, 512), generator=g, device="cuda").to(torch.bfloat16) for _ in range(3)]
    graphed = GraphedDecoderLayerBF16(layer, xs[0])
    for x in xs:
        res_e, mlp_e = layer.forward_parts(x)
        res_g, mlp_g = graphed(x)
        torch.cuda.synchronize()
        assert torch.equal(res_e, res_g) and torch.equal(mlp_e, mlp_g)


# rows around the widths of the narrow operand and at the lines of the dispatch; K on both sides of its lines (640, 1280), ragged,
# and of full clusters; columns of one 128-wide tile, of a part of one, and on both sides of the most that clusters of two (17152)
# and gate and up in clusters of four (4224, 8576) are for
@pytest.mark.parametrize("M", [1, 17, 32, 33, 48, 49, 64, 65, 128])
@pytest.mark.parametrize("N,K", [(8, 8), (136, 328), (256, 2120), (2048, 2048), (16896, 128), (8, 632), (136, 648), (264, 1272), (264, 1288),
                                 (17152, 640), (17160, 640), (4224, 1280), (4232, 1280), (8576, 640), (8584, 640)])
def test_small_m_epilogues(lib, M, N, K):
    from baranet_bdml_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(M * 31 + N + K)
    rnd = lambda *s: torch.randn(s, generator=gen, device="cuda")                                # noqa: E731
    x, w, u = rnd(M, K).bfloat16(), (rnd(N, K) * 0.06).bfloat16(), (rnd(N, K) * 0.06).bfloat16()
    bias, mul = rnd(N), rnd(M, N + 8).bfloat16()
    prod, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    up, up_size = x.double() @ u.double().T, x.double().abs() @ u.double().abs().T
    n = int(lib.bn_gemm_bf16_nt_small_m_workspace_bytes(M, N, K))
    ws, word, st = torch.empty(n, dtype=torch.uint8, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), torch.cuda.current_stream().cuda_stream
    tail = (ws.data_ptr(), n, word.data_ptr(), st)
    c, c32 = torch.empty((M, N), dtype=torch.bfloat16, device="cuda"), torch.empty((M, N), device="cuda")
    # fp32 sums of exact products: K roundings (or truncations of 2 units) of at most 2^-24 of the absolute sum
    slack, bf = 2 * K * 2.0 ** -24, 2.0 ** -8
    silu = torch.nn.functional.silu
    _lib.check(lib.bn_gemm_bf16_nt_small_m_f32(x.data_ptr(), w.data_ptr(), c32.data_ptr(), M, N, K, *tail))
    assert ((c32.double() - prod).abs() <= slack * size).all()
    _lib.check(lib.bn_gemm_bf16_nt_small_m(x.data_ptr(), w.data_ptr(), c.data_ptr(), M, N, K, *tail))
    assert torch.equal(c, c32.bfloat16())
    _lib.check(lib.bn_gemm_bias_act_bf16_nt_small_m(x.data_ptr(), w.data_ptr(), bias.data_ptr(), c.data_ptr(), M, N, K, _lib.BN_ACT_RELU2, *tail))
    assert torch.equal(c, (torch.relu(c32 + bias) ** 2).bfloat16())
    # the fast exponential and quotient: within 2^-18 of the factor; the slope of silu is below 1.1
    _lib.check(lib.bn_gemm_act_mul_bf16_nt_small_m(x.data_ptr(), w.data_ptr(), mul.data_ptr(), N + 8, c.data_ptr(), M, N, K, _lib.BN_ACT_SILU, *tail))
    m = mul[:, :N].double()
    assert ((c.double() - silu(prod) * m).abs() <= bf * (silu(prod) * m).abs() + (1.1 * slack * size + 2.0 ** -18 * prod.abs()) * m.abs() + 1e-30).all()
    packed = ops.pack_gate_up(w, u)
    _lib.check(lib.bn_gemm_glu_bf16_nt(x.data_ptr(), packed.data_ptr(), c.data_ptr(), M, N, K, _lib.BN_ACT_SILU, word.data_ptr(), st))
    want = silu(prod) * up
    bound = bf * want.abs() + (1.1 * slack * size + 2.0 ** -18 * prod.abs()) * up.abs() + slack * up_size * (silu(prod).abs() + slack * size) + 1e-30
    assert ((c.double() - want).abs() <= bound).all()
    assert int(word.item()) == 0


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (64, 2048, 2048), (64, 256, 2048), (17, 2048, 5632), (128, 1000, 520),
                                   (64, 32000, 2048), (130, 136, 264)])
def test_small_m_gemm(lib, M, N, K):
    """The split-K form for few rows: against fp64 on the same operands, equal run to run (fixed summation order), and
    within one bf16 ulp of the large-tile kernel."""
    from baranet_bdml_b200 import ops
    rng = np.random.default_rng(M * 3 + N + K)
    a = R.round_bf16(rng.standard_normal((M, K), dtype=np.float32))
    bt = R.round_bf16((rng.standard_normal((N, K)) * 0.05).astype(np.float32))
    ta, tb = torch.from_numpy(a).cuda().to(torch.bfloat16), torch.from_numpy(bt).cuda().to(torch.bfloat16)
    got = ops.gemm_bf16_nt_small_m(ta, tb)
    again = ops.gemm_bf16_nt_small_m(ta, tb)
    big = ops.gemm_bf16_nt(ta, tb)
    torch.cuda.synchronize()
    assert torch.equal(got, again)
    ref = a.astype(np.float64) @ bt.astype(np.float64).T
    scale = max(np.abs(ref).max(), 1e-30)
    assert np.abs(got.float().cpu().numpy() - ref).max() <= scale * 2.0 ** -8
    assert float((got.float() - big.float()).abs().max()) <= scale * 2.0 ** -7


@pytest.mark.parametrize("B,S,off", [(3, 803, 0), (2, 1300, 5)])
def test_fused_qkv_projection_in_paired_tiles(lib, B, S, off):
    """The fused projection where two CTAs share a tile: its parts are those of the plain products, the cache holds what it returns."""
    from baranet_bdml_b200 import ops
    from baranet_bdml_b200.kv_cache import PagedKVCache, PAGE_TOKENS
    Hq, Hkv, D, hidden = 32, 4, 64, 1024
    g = torch.Generator(device="cuda").manual_seed(S)
    x = torch.randn((B * S, hidden), generator=g, device="cuda").bfloat16()
    w = (torch.randn(((Hq + 2 * Hkv) * D, hidden), generator=g, device="cuda") * 0.03).bfloat16()
    pages = -(-(S + off) // PAGE_TOKENS)
    cache = PagedKVCache(B * pages, B, pages, Hkv, D)
    cache.page_table.copy_(torch.arange(B * pages, dtype=torch.int32).view(B, pages).flip(1))
    ws = ops.prefill_workspace(B, S, Hq, Hkv, D)
    ops.prefill_table(ws, B, S, Hkv, D, 10000.0, off)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    q, v = ops.gemm_qkv_rope_bf16(x, w, B, S, Hq, Hkv, D, ws, position_offset=off, cache=cache, error_word=err)
    wq, wk, wv = w.split([Hq * D, Hkv * D, Hkv * D])
    assert torch.equal(q.view(B * S, -1), ops.gemm_bf16_nt(x, wq.contiguous())) and torch.equal(v.view(B * S, -1), ops.gemm_bf16_nt(x, wv.contiguous()))
    rows = cache.pool[cache.page_table.long()].permute(0, 1, 4, 2, 3, 5).reshape(B, pages * PAGE_TOKENS, Hkv, 2, D)[:, off:off + S]
    assert torch.equal(rows[:, :, :, 1], v.view(B, S, Hkv, D))
    k = (x.double() @ wk.double().T).view(B, S, Hkv, D // 2, 2)
    i = torch.arange(D // 2, device="cuda", dtype=torch.float32)
    freq = (1.0 / torch.pow(torch.tensor(10000.0, device="cuda"), 2 * i / D)).float()
    a = ((torch.arange(S, device="cuda", dtype=torch.float32) + off)[:, None] * freq).double()[:, None]
    want = torch.stack([k[..., 0] * a.cos() - k[..., 1] * a.sin(), k[..., 0] * a.sin() + k[..., 1] * a.cos()], -1).flatten(-2)
    assert float((rows[:, :, :, 0].double() - want).abs().max()) <= float(want.abs().max()) * 2.0 ** -8
    out = ops.attn_prefill_bf16(q, None, v, position_offset=off, workspace=ws, reuse_rotated_k=True)
    ref = ops.attn_prefill_bf16(q, ops.gemm_bf16_nt(x, wk.contiguous()).view(B, S, Hkv, D), v, position_offset=off)
    assert float((out.float() - ref.float()).abs().max()) <= 2e-2
    ws.status()
    assert int(err.item()) == 0


@pytest.mark.parametrize("B,S,off", [(2, 200, 0), (1, 128, 0), (3, 77, 5)])
def test_fused_qkv_projection_with_rope_and_cache_append(lib, B, S, off):
    """bn_gemm_qkv_rope_bf16 against the separate launches it replaces: q and v are the bits of the plain GEMM; the
    rotated K (rotated from the fp32 accumulators, one rounding) is within one bf16 ulp of the fp64 rotation of the
    fp64 product; the cache pages hold that same K and V at positions off .. off + S - 1; the per-tile norm maxima
    bound the stored keys; and the attention that follows matches the unfused path within the bf16 gate."""
    from baranet_bdml_b200 import ops
    from baranet_bdml_b200.kv_cache import PagedKVCache, PAGE_TOKENS
    Hq, Hkv, D, hidden = 8, 2, 64, 256
    rng = np.random.default_rng(S + off)
    x = R.round_bf16(rng.standard_normal((B * S, hidden), dtype=np.float32))
    wq = R.round_bf16((rng.standard_normal((Hq * D, hidden)) * 0.06).astype(np.float32))
    wk = R.round_bf16((rng.standard_normal((Hkv * D, hidden)) * 0.06).astype(np.float32))
    wv = R.round_bf16((rng.standard_normal((Hkv * D, hidden)) * 0.06).astype(np.float32))
    tx = torch.from_numpy(x).cuda().to(torch.bfloat16)
    tq, tk, tv = (torch.from_numpy(w).cuda().to(torch.bfloat16) for w in (wq, wk, wv))
    wqkv = torch.cat([tq, tk, tv], 0).contiguous()
    max_pages = (S + off + PAGE_TOKENS - 1) // PAGE_TOKENS
    cache = PagedKVCache(B * max_pages + 3, B, max_pages, Hkv, D)
    perm = rng.permutation(B * max_pages + 3)[: B * max_pages].astype(np.int32).reshape(B, max_pages)
    cache.page_table.copy_(torch.from_numpy(perm))
    ws = ops.prefill_workspace(B, S, Hq, Hkv, D)
    ops.prefill_table(ws, B, S, Hkv, D, 10000.0, off)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    q, v = ops.gemm_qkv_rope_bf16(tx, wqkv, B, S, Hq, Hkv, D, ws, position_offset=off, cache=cache, error_word=err)
    out = ops.attn_prefill_bf16(q, None, v, position_offset=off, workspace=ws, reuse_rotated_k=True)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ws.status()
    # q, v: the plain GEMM's bits
    assert torch.equal(q.view(B * S, -1), ops.gemm_bf16_nt(tx, tq))
    assert torch.equal(v.view(B * S, -1), ops.gemm_bf16_nt(tx, tv))
    # rotated K in the cache pages against fp64
    k64 = x.astype(np.float64) @ wk.astype(np.float64).T                       # (B*S, Hkv*D)
    pool = cache.pool.float().cpu().numpy()
    vq = v.float().cpu().numpy().reshape(B, S, Hkv, D)
    worst = 0.0
    for b in range(B):
        pos = np.arange(S) + off
        i = np.arange(D // 2)
        freq = (1.0 / np.power(np.float32(10000.0), (2 * i).astype(np.float32) / np.float32(D))).astype(np.float32)
        ang = (pos[:, None].astype(np.float32) * freq[None]).astype(np.float64)
        kb = k64[b * S:(b + 1) * S].reshape(S, Hkv, D // 2, 2)
        rot = np.empty_like(kb)
        rot[..., 0] = kb[..., 0] * np.cos(ang)[:, None] - kb[..., 1] * np.sin(ang)[:, None]
        rot[..., 1] = kb[..., 0] * np.sin(ang)[:, None] + kb[..., 1] * np.cos(ang)[:, None]
        rot = rot.reshape(S, Hkv, D)
        pages, slots = perm[b][pos // PAGE_TOKENS], pos % PAGE_TOKENS
        got_k = pool[pages, :, 0, slots, :]                                    # (S, Hkv, D)
        got_v = pool[pages, :, 1, slots, :]
        worst = max(worst, np.abs(got_k - rot).max() / max(np.abs(rot).max(), 1e-30))
        assert np.array_equal(got_v, vq[b])
    assert worst <= 2.0 ** -8
    # the attention that follows, against the unfused path (separate GEMMs, K rotated from its bf16 rounding)
    k_plain = ops.gemm_bf16_nt(tx, tk).view(B, S, Hkv, D)
    ref = ops.attn_prefill_bf16(q, k_plain, v, position_offset=off)
    torch.cuda.synchronize()
    assert float((out.float() - ref.float()).abs().max()) <= 2e-2


@pytest.mark.parametrize("M,N,K", [(1, 8, 256), (16, 2048, 2048), (2, 2560, 2048), (16, 2048, 5632), (5, 32000, 2048),
                                   (13, 264, 512)])
def test_skinny_gemm(lib, M, N, K):
    """The weight-streaming product for at most 16 rows against fp64 on the same operands (one bf16 ulp at the largest
    magnitude), equal run to run, and split into three column ranges equal to the unsplit result."""
    from baranet_bdml_b200 import ops
    rng = np.random.default_rng(M + N + K)
    a = R.round_bf16(rng.standard_normal((M, K), dtype=np.float32))
    bt = R.round_bf16((rng.standard_normal((N, K)) * 0.05).astype(np.float32))
    ta, tb = torch.from_numpy(a).cuda().to(torch.bfloat16), torch.from_numpy(bt).cuda().to(torch.bfloat16)
    got = ops.gemm_bf16_nt_skinny(ta, tb)
    again = ops.gemm_bf16_nt_skinny(ta, tb)
    torch.cuda.synchronize()
    assert torch.equal(got, again)
    ref = a.astype(np.float64) @ bt.astype(np.float64).T
    assert np.abs(got.float().cpu().numpy() - ref).max() <= max(np.abs(ref).max(), 1e-30) * 2.0 ** -8
    if N >= 24:
        n0 = (N // 3) // 8 * 8
        n1 = 8
        parts = ops.gemm_bf16_nt_skinny(ta, tb, (n0, n1, N - n0 - n1))
        torch.cuda.synchronize()
        assert torch.equal(torch.cat(parts, dim=1), got)


# Wide products of few rows: one column group more than three a multiprocessor, a number of groups that the CTAs do not share evenly,
# K of one, two, seven and eight steps a warp, rows in the low half of a fragment and in both; K in two parts, of which the last is one
# step or eight, and in four, the last of five, with groups that follow one another in a CTA (the rows are read again for each)
@pytest.mark.parametrize("N,K", [(3560, 256), (4608, 512), (3704, 1792), (8520, 2048), (3560, 2304), (4616, 4096), (8520, 7424)])
@pytest.mark.parametrize("M", [1, 8, 9, 16])
def test_wide_products_of_few_rows(lib, M, N, K):
    """Every output form against fp64: bf16's rounding (2^-9 of the result) and fp32 sums of K terms"""
    from baranet_bdml_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w, u = ((torch.randn(N, K, generator=g, device="cuda") * 0.05).bfloat16() for _ in range(2))
    bias, mul = torch.randn(N, generator=g, device="cuda"), torch.randn(M, N + 8, generator=g, device="cuda").bfloat16()
    st = torch.cuda.current_stream().cuda_stream
    ref = x.double() @ w.double().T
    up = x.double() @ u.double().T
    terms = 2.0 ** -24 * (K / 16 + 24) * float((x.double().abs() @ w.double().abs().T).max())

    def out(dtype=torch.bfloat16, cols=N):
        return torch.full((M, cols), float("nan"), dtype=dtype, device="cuda")

    def near(got, want, slope=1.0, exact=False):
        err, scale = (got.double() - want).abs(), want.abs()
        assert bool((err <= (0 if exact else 2.0 ** -8) * scale + slope * terms + 1e-30).all()), float(err.max())

    y32 = out(torch.float32)
    _lib.check(lib.bn_gemm_bf16_nt_skinny_f32(x.data_ptr(), w.data_ptr(), M, N, K, y32.data_ptr(), st))
    near(y32, ref, exact=True)
    widened = out(torch.float32)
    _lib.check(lib.bn_gemm_bf16_nt_skinny_widened(x.data_ptr(), w.data_ptr(), M, N, K, widened.data_ptr(), st))
    assert torch.equal(widened, y32.bfloat16().float())
    n0, n1 = 1024, 2504
    parts = [out(cols=n) for n in (n0, n1, N - n0 - n1)]
    _lib.check(lib.bn_gemm_bf16_nt_skinny(x.data_ptr(), w.data_ptr(), M, N, K, parts[0].data_ptr(), n0, parts[1].data_ptr(), n1, parts[2].data_ptr(), st))
    near(torch.cat(parts, 1), ref)
    y = out()
    _lib.check(lib.bn_gemm_bias_act_bf16_nt_skinny(x.data_ptr(), w.data_ptr(), bias.data_ptr(), y.data_ptr(), M, N, K, 3, st))
    near(y, (ref + bias.double()).clamp_min(0).square(), slope=2 * float((ref + bias.double()).abs().max()))
    _lib.check(lib.bn_gemm_act_mul_bf16_nt_skinny(x.data_ptr(), w.data_ptr(), mul.data_ptr(), N + 8, y.data_ptr(), M, N, K, 1, st))
    silu = torch.nn.functional.silu(ref)
    near(y, silu * mul[:, :N].double(), slope=1.1 * float(mul.abs().max()) + 2.0 ** -12)
    _lib.check(lib.bn_gemm_glu_bf16_nt_skinny(x.data_ptr(), w.data_ptr(), u.data_ptr(), y.data_ptr(), M, N, K, 1, st))
    near(y, silu * up, slope=1.1 * float(up.abs().max()) + 1.1 * float(ref.abs().max()))


def test_skinny_swiglu(lib):
    from baranet_bdml_b200 import ops
    rng = np.random.default_rng(77)
    M, K, inter = 16, 2048, 5632
    x = R.round_bf16(rng.standard_normal((M, K), dtype=np.float32))
    wg = R.round_bf16((rng.standard_normal((inter, K)) * 0.03).astype(np.float32))
    wu = R.round_bf16((rng.standard_normal((inter, K)) * 0.03).astype(np.float32))
    tx, tg, tu = (torch.from_numpy(t).cuda().to(torch.bfloat16) for t in (x, wg, wu))
    got = ops.gemm_swiglu_bf16_nt_skinny(tx, tg, tu).float().cpu().numpy()
    g = x.astype(np.float64) @ wg.astype(np.float64).T
    u = x.astype(np.float64) @ wu.astype(np.float64).T
    ref = g / (1.0 + np.exp(-g)) * u
    assert np.abs(got - ref).max() <= max(np.abs(ref).max(), 1e-30) * 2.0 ** -8
    assert lib.bn_gemm_bf16_nt_skinny(tx.data_ptr(), tg.data_ptr(), 17, inter, K, tx.data_ptr(), inter, None, 0, None, None) != 0


@pytest.mark.parametrize("M,Hq,Hkv,D,hidden", [(16, 32, 4, 64, 2048), (3, 4, 2, 64, 256), (7, 6, 3, 32, 512), (16, 32, 4, 64, 2304),
                                               (5, 32, 4, 64, 4096)])
def test_skinny_qkv_with_cache_append(lib, M, Hq, Hkv, D, hidden):
    """One launch for the q, k and v projections of a decode step with RoPE(K) and the cache append against the
    two-launch path (three-output skinny GEMM, then bn_kv_append): q equal, and every page of the cache equal bit for
    bit - including rows whose position is out of the page table's range, which both paths skip."""
    from baranet_bdml_b200 import ops
    from baranet_bdml_b200.kv_cache import PagedKVCache
    rng = np.random.default_rng(M * 1000 + hidden)
    x = torch.from_numpy(R.round_bf16(rng.standard_normal((M, hidden), dtype=np.float32))).cuda().to(torch.bfloat16)
    w = torch.from_numpy(R.round_bf16((rng.standard_normal(((Hq + 2 * Hkv) * D, hidden)) * 0.05).astype(np.float32)))
    w = w.cuda().to(torch.bfloat16)
    pages_per = 6                                                      # 96 positions per sequence
    pos = rng.integers(0, pages_per * 16, (M,)).astype(np.int32)
    if M > 4:
        pos[1] = pages_per * 16 + 5                                    # past the last page: skipped
        pos[2] = -1
    seq = rng.permutation(M).astype(np.int32)
    caches = []
    for _ in range(2):
        c = PagedKVCache(M * pages_per + 2, M, pages_per, Hkv, D)
        c.page_table.copy_(torch.from_numpy(rng.permutation(M * pages_per + 2)[: M * pages_per].astype(np.int32)
                                            .reshape(M, pages_per)))
        c.pool.zero_()
        caches.append(c)
    caches[1].page_table.copy_(caches[0].page_table)
    seq_t, pos_t = torch.from_numpy(seq).cuda(), torch.from_numpy(pos).cuda()
    q1, k1, v1 = ops.gemm_bf16_nt_skinny(x, w, (Hq * D, Hkv * D, Hkv * D))
    caches[0].append(seq_t, pos_t, k1, v1)
    q2 = ops.gemm_qkv_append_bf16_skinny(x, w, caches[1], seq_t, pos_t, Hq)
    torch.cuda.synchronize()
    assert torch.equal(q1, q2)
    assert torch.equal(caches[0].pool, caches[1].pool)
    assert float(caches[1].pool.float().abs().max()) > 0
