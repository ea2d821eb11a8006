"""fp32 path vs the oracle, through the C ABI (TensorF / AGTensor mirror the
reference's bten / mygrad surface, so these read like the reference's own
test_llama.py — with assertions).  Gate (fp32 path): max|d| / max|ref| <= 1e-5."""
import numpy as np
import pytest
import torch

from oracle import ref_attention as R

pytestmark = pytest.mark.gpu

GATE = 1e-5


def nerr(a, b):
    return float(np.abs(a.astype(np.float64) - b.astype(np.float64)).max() / max(np.abs(b).max(), 1e-30))


@pytest.fixture(scope="module")
def T(lib):
    from baranet_bdml_b200 import tensor
    return tensor


@pytest.fixture(scope="module")
def dev_inv_freq(T):
    """The device's own frequency table (CUDA powf), read back through bn_rope_f32:
    rotating (1, 0) pairs at position 1 yields (cos f_i, sin f_i)."""
    out = {}
    for D in (6, 20, 32, 64):
        x = np.zeros((1, D), dtype=np.float32)
        x[0, 0::2] = 1.0
        t = T.TensorF(1, D)
        t.copy_from_numpy(x)
        y = t.rope(1, D, 10000.0).to_numpy()
        out[D] = np.arctan2(y[0, 1::2].astype(np.float64), y[0, 0::2].astype(np.float64))
    return out


def test_inv_freq_matches_cpu_table(dev_inv_freq, cref):
    for D in (32, 64):
        cpu = cref.inv_freq(D).astype(np.float64)
        assert np.abs(dev_inv_freq[D] - cpu).max() / cpu.max() < 1e-6


@pytest.mark.parametrize("M,K,N", [(128, 2048, 256), (4, 128, 64), (33, 70, 65), (1, 64, 1), (130, 16, 200)])
def test_mm_matches_reference_order(T, cref, M, K, N):
    rng = np.random.default_rng(1)
    a = rng.standard_normal((M, K), dtype=np.float32)
    b = rng.standard_normal((K, N), dtype=np.float32)
    ta, tb = T.TensorF(M, K), T.TensorF(K, N)
    ta.copy_from_numpy(a)
    tb.copy_from_numpy(b)
    got = (ta @ tb).to_numpy()
    import ctypes as C
    ref = np.empty((M, N), dtype=np.float32)
    fp = C.POINTER(C.c_float)
    cref.cpu().ref_mm_f32(a.ctypes.data_as(fp), C.c_long(K), C.c_long(1), b.ctypes.data_as(fp), C.c_long(N),
                          C.c_long(1), ref.ctypes.data_as(fp), C.c_int(M), C.c_int(K), C.c_int(N))
    assert np.array_equal(got, ref), nerr(got, ref)   # same FMA chain -> same bits


@pytest.mark.parametrize("M,K,N", [(8, 4, 32), (9, 20, 33), (17, 52, 1000), (33, 68, 4736), (65, 16, 9473), (1151, 24, 2052), (1, 1, 8)])
@pytest.mark.parametrize("layout", ["nn", "nt", "nn_odd", "nt_odd", "a_t"])
def test_mm_tiles_and_copies(T, cref, M, K, N, layout):
    """Every tile size and every way the operands are copied (along K, along N, element by element where a stride or an
    address is odd, a transposed A), with ragged edges: the bits of the chain."""
    rng = np.random.default_rng(M + K + N)
    a, b = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal((K, N), dtype=np.float32)

    def on_gpu(x, odd):
        t = T.TensorF(x.shape[0], x.shape[1] + (3 if odd else 0))
        t.copy_from_numpy(np.pad(x, ((0, 0), (0, 3))) if odd else x)
        return T.TensorF(x.shape[0], x.shape[1], _base=t.base, _stride_h=t.stride_h)
    odd = layout.endswith("odd")
    ta = on_gpu(a.T, False).T if layout == "a_t" else on_gpu(a, odd)
    tb = on_gpu(b.T, odd).T if layout.startswith("nt") else on_gpu(b, odd)
    got = (ta @ tb).to_numpy()
    import ctypes as C
    ref = np.empty((M, N), dtype=np.float32)
    fp = C.POINTER(C.c_float)
    cref.cpu().ref_mm_f32(a.ctypes.data_as(fp), C.c_long(K), C.c_long(1), b.ctypes.data_as(fp), C.c_long(N),
                          C.c_long(1), ref.ctypes.data_as(fp), C.c_int(M), C.c_int(K), C.c_int(N))
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("M,K,N", [(1, 8, 8), (127, 72, 72), (129, 136, 136), (300, 2056, 264), (513, 64, 2056), (1300, 128, 4096)])
@pytest.mark.parametrize("parts", [1, 3])
def test_mm_of_bf16_parts(lib, M, K, N, parts):
    import torch
    from baranet_bdml_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(M + parts)
    x, w, bias = (torch.randn(s, generator=gen, device="cuda") for s in ((M, K), (N, K), (N,)))
    if parts == 1:
        w = w.bfloat16().float()
    xp, wp = ops._bf16_parts(x), ops._bf16_parts(w)
    assert torch.equal(xp.double().sum(0), x.double()) and torch.equal(wp.double().sum(0), w.double())
    assert bool(wp[1:].any()) == (parts == 3)
    # a bad row of x and a bad row of w touch their own results alone, and there the chain decides
    x[M // 2, K // 2], w[N // 2, 0] = float("inf"), float("nan")
    xp, wp = ops._bf16_parts(x), ops._bf16_parts(w)
    L, st = lib, torch.cuda.current_stream().cuda_stream
    chain, word = torch.empty((M, N), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.check(L.bn_mm_f32(x.data_ptr(), K, 1, w.data_ptr(), 1, K, chain.data_ptr(), N, 1, M, K, N, st))
    exact, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    fine = torch.isfinite(chain)
    for b, act in ((None, 0), (bias, 3), (bias, 2)):
        got = torch.empty((M, N), device="cuda")
        _lib.check(L.bn_mm_f32_split(xp.data_ptr(), wp.data_ptr(), parts, x.data_ptr(), K, w.data_ptr(), K,
                                    None if b is None else b.data_ptr(), act, got.data_ptr(), M, N, K, word.data_ptr(), st))
        want = chain.clone()
        if act:
            _lib.check(L.bn_bias_act_f32(want.data_ptr(), N, b.data_ptr(), M, N, act, st))
        assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
        if act == 0:
            # in an accumulator 4 truncations at full size, each of 2 units of 2^-24, beside 8 at 2^-8 of it; K / 64 roundings
            # of the sum; products left out and the bias: 1 more
            bound = (4 * 2 + 1 + K / 64 + 1) * 2.0 ** -24 * size
            assert ((got.double() - exact).abs() <= bound)[fine].all()
        elif act == 2:
            # the activation's slope is below 1.13; the chain itself is off by at most K roundings
            bound = 1.13 * (K + K / 64 + 12) * 2.0 ** -24 * (size + b.double().abs())
            assert ((got.double() - want.double()).abs() <= bound)[fine].all()
    assert int(word.item()) == 0


@pytest.mark.parametrize("shift_x,shift_w", [(1, 0), (0, 3), (2, 1)])
def test_mm_of_bf16_parts_reads_operands_at_any_address(lib, shift_x, shift_w):
    """The operands themselves, which results that are not finite are worked out from, need no alignment."""
    from baranet_bdml_b200 import _lib, ops
    M, K, N = 140, 264, 200
    gen = torch.Generator(device="cuda").manual_seed(shift_x)
    x, w = torch.randn((M, K), generator=gen, device="cuda"), torch.randn((N, K), generator=gen, device="cuda")
    x[3], x[130, 7], w[70, 5] = float("inf"), -float("inf"), float("nan")
    xp, wp = ops._bf16_parts(x), ops._bf16_parts(w)
    xs, ws = (torch.zeros((r, K + s), device="cuda")[:, s:] for r, s in ((M, shift_x), (N, shift_w)))
    xs.copy_(x)
    ws.copy_(w)
    got, chain, word = torch.empty((M, N), device="cuda"), torch.empty((M, N), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.bn_mm_f32(x.data_ptr(), K, 1, w.data_ptr(), 1, K, chain.data_ptr(), N, 1, M, K, N, st))
    _lib.check(lib.bn_mm_f32_split(xp.data_ptr(), wp.data_ptr(), 3, xs.data_ptr(), xs.stride(0), ws.data_ptr(), ws.stride(0), None, 0,
                                   got.data_ptr(), M, N, K, word.data_ptr(), st))
    assert torch.equal(torch.isnan(got), torch.isnan(chain)) and torch.equal(torch.isposinf(got), torch.isposinf(chain))
    fine = torch.isfinite(chain)
    assert ((got - chain).abs()[fine] <= 2e-4).all() and int(word.item()) == 0


@pytest.mark.parametrize("M,K,N", [(1, 8, 8), (127, 72, 72), (129, 136, 136), (300, 2056, 264), (513, 64, 2056), (1300, 128, 4096)])
@pytest.mark.parametrize("weights", ["bf16", "fp32", "mixed"])
def test_linear_f32_cuts_its_operands(lib, M, K, N, weights):
    """Tiles of one part beside tiles of three; what is not written in the scratch is not read."""
    from baranet_bdml_b200 import _lib
    gen = torch.Generator(device="cuda").manual_seed(M + K)
    x, w, bias = (torch.randn(s, generator=gen, device="cuda") for s in ((M, K), (N, K), (N,)))
    if weights == "bf16":
        w = w.bfloat16().float()
    elif weights == "mixed":
        whole = torch.rand(((N + 63) // 64, (K + 63) // 64), generator=gen, device="cuda") < 0.5
        whole = whole.repeat_interleave(64, 0)[:N].repeat_interleave(64, 1)[:, :K]
        w = torch.where(whole, w.bfloat16().float(), w)
    n = lib.bn_linear_f32_workspace_bytes(M, N, K)
    scratch, word = torch.full((n,), 0xff, dtype=torch.uint8, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    got = torch.empty((M, N), device="cuda")
    args = (x.data_ptr(), K, w.data_ptr(), K, bias.data_ptr(), 0, got.data_ptr(), M, N, K, scratch.data_ptr())
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.bn_linear_f32(*args, n, word.data_ptr(), st))
    exact = x.double() @ w.double().T + bias.double()
    # per 64 k: 4 truncations at full size, each of 2 units of 2^-24, beside 8 at 2^-8 of it; K / 64 roundings of the sum; products
    # left out and the bias: 2 more
    bound = (4 * 2 + 1 + K / 64 + 2) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T + bias.double().abs())
    assert ((got.double() - exact).abs() <= bound).all() and int(word.item()) == 0
    assert lib.bn_linear_f32(*args, n - 1, word.data_ptr(), st) != 0


@pytest.mark.parametrize("bad", ["row", "rows", "nan", "weight"])
@pytest.mark.parametrize("act", [0, 1, 2, 3])
def test_linear_f32_of_values_that_are_not_finite(lib, bad, act):
    """Results that are not finite are the chain's and the others stay within their bound; a long K takes a few ms at worst, and
    no wait runs out."""
    from baranet_bdml_b200 import _lib
    M, K, N = 300, 7424, 1032
    gen = torch.Generator(device="cuda").manual_seed(act)
    x, w, bias = (torch.randn(s, generator=gen, device="cuda") for s in ((M, K), (N, K), (N,)))
    if bad == "row":
        x[7, 5], x[129, K - 1] = float("inf"), -float("inf")
    elif bad == "rows":
        x[:, 3] = float("inf")                              # every result infinite, none a NaN
    elif bad == "nan":
        x[40:200, 0] = float("nan")
    else:
        w[1031, 77], w[12] = float("inf"), 3e38
    chain, got = torch.empty((M, N), device="cuda"), torch.empty((M, N), device="cuda")
    st, word = torch.cuda.current_stream().cuda_stream, torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.check(lib.bn_mm_f32(x.data_ptr(), K, 1, w.data_ptr(), 1, K, chain.data_ptr(), N, 1, M, K, N, st))
    fine = torch.isfinite(chain)
    _lib.check(lib.bn_bias_act_f32(chain.data_ptr(), N, bias.data_ptr(), M, N, act, st))
    n = lib.bn_linear_f32_workspace_bytes(M, N, K)
    scratch = torch.empty(n, dtype=torch.uint8, device="cuda")
    times = []
    for _ in range(3):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        _lib.check(lib.bn_linear_f32(x.data_ptr(), K, w.data_ptr(), K, bias.data_ptr(), act, got.data_ptr(), M, N, K, scratch.data_ptr(), n,
                                     word.data_ptr(), st))
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    assert int(word.item()) == 0 and min(times) < 10.0, times
    assert torch.equal(got[~fine].view(torch.int32), chain[~fine].view(torch.int32)) or \
        (torch.equal(torch.isnan(got[~fine]), torch.isnan(chain[~fine])) and torch.equal(got[~fine].nan_to_num(5.0), chain[~fine].nan_to_num(5.0)))
    ok = fine & torch.isfinite(chain)
    xd, wd = x.double().nan_to_num(0.0, 0.0, 0.0), w.double().nan_to_num(0.0, 0.0, 0.0)
    size = xd.abs() @ wd.abs().T + bias.double().abs()
    err = (K + K / 64 + 12) * 2.0 ** -24 * size             # of the chain and of the product, before the activation
    # slopes: 1.1 for SiLU, 1.13 for GELU; a square's 2 z, and the roundings of the square itself
    bound = err if act == 0 else 2 * (size + err) * err + 2.0 ** -22 * size ** 2 if act == 3 else 1.13 * err + 2.0 ** -20 * size
    assert ((got.double() - chain.double()).abs() <= bound)[ok].all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("write", ["data", "in_place", "replaced"])
def test_linear_f32_reads_the_weight_of_the_call(lib, dtype, write):
    """A weight that is written to, by whatever way, is the one that many rows are multiplied with as well as few."""
    from baranet_bdml_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(7)
    N, K, rows = 2048, 2048, 512
    x, w0, w1 = (torch.randn(s, generator=gen, device="cuda") for s in ((rows, K), (N, K), (N, K)))
    lin = ops.Linear(w0.to(dtype), torch.float32)
    assert torch.equal(lin.weight, w0.to(dtype).float())
    lin(x)
    if write == "data":
        lin.weight.data.copy_(w1)
    elif write == "in_place":
        lin.weight.mul_(0).add_(w1)
    else:
        lin.weight = w1.clone()
    many, few = lin(x), torch.cat([lin(x[i:i + 4]) for i in range(0, rows, 4)])
    exact, size = x.double() @ w1.double().T, x.double().abs() @ w1.double().abs().T
    for got in (many, few):
        assert ((got.double() - exact).abs() <= K * 2.0 ** -24 * size).all()
    # the two are two routes; a wide weight takes few rows by the third
    form = lambda r, n: lib.bn_linear_f32_form(r, n, K, lin.parts_hint)                          # noqa: E731
    assert form(rows, N) == _lib.BN_LINEAR_F32_PARTS and form(4, N) == _lib.BN_LINEAR_F32_CHAINS
    assert form(16, 32000) == _lib.BN_LINEAR_F32_SUMS


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16, 17, 40])
@pytest.mark.parametrize("K,N,odd", [(4, 8, 0), (128, 24, 0), (132, 2056, 4), (1028, 4744, 0), (2048, 19000, 0), (7424, 64, 8)])
def test_linear_stream(lib, M, K, N, odd):
    """Every number of rows a warp has sums for, one to four slices of K, rounds that are not full, columns that fill no block."""
    from baranet_bdml_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(M + K + N)
    x, w = (torch.randn((r, K + odd), generator=gen, device="cuda")[:, :K] for r in (M, N))
    bias = torch.randn(N, generator=gen, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    run = lambda x, bias, act, out: _lib.check(lib.bn_linear_f32_stream(                         # noqa: E731
        x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), None if bias is None else bias.data_ptr(), ops.ACTIVATIONS[act],
        out.data_ptr(), out.stride(0), M, N, K, st))
    out = torch.full((M, N + 5), 7.0, device="cuda")
    run(x, None, "none", out)
    exact, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # a lane's links (K in 128 lanes at the least), five additions of lanes, four of slices
    bound = (4 * (K // 128 + 1) + 9) * 2.0 ** -24 * size
    assert ((out[:, :N].double() - exact).abs() <= bound).all() and bool((out[:, N:] == 7.0).all())
    run(x, bias, "relu2", out)
    exact = exact + bias.double()
    size = size + bias.double().abs()
    bound = (4 * (K // 128 + 1) + 10) * 2.0 ** -24 * size
    want = exact.clamp(min=0).square()
    assert ((out[:, :N].double() - want).abs() <= 2 * bound * (exact.abs() + bound) + 2.0 ** -23 * want).all()
    if M > 1:                                      # a row that is not finite stays alone
        y = x.clone()
        y[M - 1, K - 1] = float("inf")
        again = torch.empty((M, N), device="cuda")
        run(y, None, "none", again)
        chain = torch.empty((1, N), device="cuda")
        _lib.check(lib.bn_mm_f32(y[M - 1:].data_ptr(), y.stride(0), 1, w.data_ptr(), 1, w.stride(0), chain.data_ptr(), N, 1, 1, K, N, st))
        run(x, None, "none", out)
        assert torch.equal(again[:M - 1], out[:M - 1, :N]) and torch.equal(again[M - 1].nan_to_num(5.0), chain[0].nan_to_num(5.0))


@pytest.mark.parametrize("M,K,N", [(1, 4, 32), (8, 16, 33), (9, 20, 33), (17, 52, 1000), (33, 144, 4736), (65, 128, 9473), (1151, 272, 2052), (3, 2056, 8)])
@pytest.mark.parametrize("odd", [False, True])
def test_mm_sums(lib, M, K, N, odd):
    """Every tile, both ways the operands are copied, K of less than a step, ragged, and on both sides of eight steps."""
    from baranet_bdml_b200 import _lib
    gen = torch.Generator(device="cuda").manual_seed(M + K + N)
    x, w = (torch.randn((r, K + (3 if odd else 0)), generator=gen, device="cuda")[:, :K] for r in (M, N))
    out = torch.full((M, N + 5), 7.0, device="cuda")
    _lib.check(lib.bn_mm_f32_sums(x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), out.data_ptr(), N + 5, M, N, K,
                                  torch.cuda.current_stream().cuda_stream))
    exact, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # 16 links, 8 additions, and one more for every 128 k
    bound = (min(K, 16) + 8 + K / 128 + 1) * 2.0 ** -24 * size
    assert ((out[:, :N].double() - exact).abs() <= bound).all() and bool((out[:, N:] == 7.0).all())


@pytest.mark.parametrize("M,K,widths", [(128, 64, (2048, 256, 256)), (5, 20, (40, 8, 33)), (33, 16, (64, 1, 65)), (70, 36, (100, 260))])
@pytest.mark.parametrize("transposed", [(), (1,), (0, 1, 2)])
def test_mm_each_is_the_single_products(T, M, K, widths, transposed):
    rng = np.random.default_rng(M + K + len(transposed))

    def tensor(h, w):
        t = T.TensorF(h, w)
        t.copy_from_numpy(rng.standard_normal((h, w), dtype=np.float32))
        return t

    x = tensor(M, K)
    ws = [tensor(n, K).T if i in transposed else tensor(K, n) for i, n in enumerate(widths)]
    for got, w in zip(x.matmul_each(ws), ws):
        assert np.array_equal(got.to_numpy(), (x @ w).to_numpy())
    with pytest.raises(RuntimeError):
        x.matmul_each([ws[0], tensor(K + 1, 4)])


def test_mm_transposed_and_sliced_views(T):
    rng = np.random.default_rng(2)
    a = rng.standard_normal((40, 96), dtype=np.float32)
    b = rng.standard_normal((50, 96), dtype=np.float32)
    ta, tb = T.TensorF(40, 96), T.TensorF(50, 96)
    ta.copy_from_numpy(a)
    tb.copy_from_numpy(b)
    got = (ta[4:36, 32:96] @ tb.T[32:96, 1:50]).to_numpy()
    ref = a[4:36, 32:96].astype(np.float64) @ b.T[32:96, 1:50].astype(np.float64)
    assert nerr(got, ref) < 1e-6


@pytest.mark.parametrize("rows,cols,D,off", [(4, 64, 32, 0), (128, 2048, 64, 0), (128, 256, 64, 7), (3, 128, 64, 2040)])
def test_rope(T, cref, rows, cols, D, off):
    rng = np.random.default_rng(3)
    x = rng.standard_normal((rows, cols), dtype=np.float32)
    t = T.TensorF(rows, cols)
    t.copy_from_numpy(x)
    got = t.rope(off, D, 10000.0).to_numpy()
    ref = cref.rope(x, D, 10000.0, off)
    # angles are fp32 products position*freq; a last-bit difference between CUDA's and glibc's
    # powf moves the angle by position * 2^-24 relative
    tol = 1e-6 + (rows + off) * 2.0 ** -23
    assert nerr(got, ref) < tol


CASES = [  # S, Hq, Hkv, D, offset, causal
    (128, 32, 4, 64, 0, True),     # the layer shape of BASELINE config 1
    (4, 4, 2, 32, 0, True),        # the reference's own test shape (test_llama.py:142-165)
    (2, 4, 2, 32, 0, True),
    (1, 32, 4, 64, 0, True),
    (17, 8, 2, 64, 3, True),
    (65, 8, 8, 32, 0, False),
    (130, 4, 1, 64, 0, True),
    (149, 8, 4, 64, 0, True),      # from here on: other numbers of rows to a block, several key tiles, head sizes that are
    (257, 5, 5, 20, 2, False),     # no multiple of 4, wide results
    (300, 6, 3, 6, 0, True),
    (1300, 4, 4, 64, 0, True),     # scores that do not fit beside the keys: computed twice
]


@pytest.mark.parametrize("S,Hq,Hkv,D,off,causal", CASES)
@pytest.mark.parametrize("mode", ["collapsed", "per_head"])
def test_attention_core_f32(T, cref, dev_inv_freq, S, Hq, Hkv, D, off, causal, mode):
    from baranet_bdml_b200 import _lib
    rng = np.random.default_rng(S * 131 + Hq)
    q = rng.standard_normal((S, Hq * D), dtype=np.float32)
    k = rng.standard_normal((S, Hkv * D), dtype=np.float32)
    v = rng.standard_normal((S, Hkv * D), dtype=np.float32)
    tq, tk, tv = T.TensorF(S, Hq * D), T.TensorF(S, Hkv * D), T.TensorF(S, Hkv * D)
    for t, a in ((tq, q), (tk, k), (tv, v)):
        t.copy_from_numpy(a)
    scale = 1.0 / np.sqrt(D)
    hm = _lib.BN_HEADS_COLLAPSED if mode == "collapsed" else _lib.BN_HEADS_PER_HEAD
    got = tq.attention_fused(tk, tv, scale, causal, off, num_heads=Hq, num_kv_heads=Hkv, head_dim=D,
                             heads_mode=hm).to_numpy()
    inv = dev_inv_freq[D].astype(np.float32)
    if mode == "collapsed":
        ref = cref.attention_collapsed(q, k, v, num_heads=Hq, num_kv_heads=Hkv, head_dim=D, position_offset=off,
                                       causal=causal, inv_freq=inv)
        ref64 = R.attention_collapsed(q, k, v, num_heads=Hq, num_kv_heads=Hkv, head_dim=D, position_offset=off,
                                      causal=causal, dtype=np.float64, inv_freq=inv)
    else:
        ref64 = R.attention_per_head(q, k, v, num_heads=Hq, num_kv_heads=Hkv, head_dim=D, position_offset=off,
                                     causal=causal, dtype=np.float64, inv_freq=inv)
        ref = ref64.astype(np.float32)
    assert nerr(got, ref) < GATE, (nerr(got, ref), nerr(got, ref64))
    assert nerr(got, ref64) < 2e-5


@pytest.mark.parametrize("S,Hq,Hkv,D", [(149, 2, 1, 40), (385, 4, 2, 24), (1, 4, 4, 18), (641, 5, 5, 10)])
def test_attention_core_f32_of_just_under_48_kb(T, S, Hq, Hkv, D):
    """Scores, keys and queries that together with the kernel's own arrays are a few bytes above what needs no asking"""
    import torch
    from baranet_bdml_b200 import _lib
    rng = np.random.default_rng(S)
    q, k, v = (rng.standard_normal((S, h * D), dtype=np.float32) for h in (Hq, Hkv, Hkv))
    tq, tk, tv = (T.TensorF.from_torch(torch.from_numpy(a).cuda()) for a in (q, k, v))
    sizes = dict(num_heads=Hq, num_kv_heads=Hkv, head_dim=D)
    got = tq.attention_fused(tk, tv, D ** -0.5, True, 0, theta=1.0, heads_mode=_lib.BN_HEADS_COLLAPSED, **sizes).to_numpy()
    want = R.attention_collapsed(q, k, v, position_offset=0, causal=True, dtype=np.float64, inv_freq=np.ones(D // 2, np.float32), **sizes)
    assert nerr(got, want) < 2e-5


def test_layer_config1_matches_oracle(T, cref, dev_inv_freq):
    """one TinyLLaMA attention layer, fp32, S=128, through the
    mirrored GroupedQueryAttention API with injected seeded weights."""
    from baranet_bdml_b200.layers import GroupedQueryAttention, LLaMAConfig
    from baranet_bdml_b200.tensor import AGTensor
    cfg = LLaMAConfig()
    rng = np.random.default_rng(0)
    S, hid, Hq, Hkv, D = 128, cfg.hidden_size, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim
    x = rng.standard_normal((S, hid), dtype=np.float32)
    wq = (rng.standard_normal((hid, Hq * D)) * 0.02).astype(np.float32)
    wk = (rng.standard_normal((hid, Hkv * D)) * 0.02).astype(np.float32)
    wv = (rng.standard_normal((hid, Hkv * D)) * 0.02).astype(np.float32)
    wo = (rng.standard_normal((Hq * D, hid)) * 0.02).astype(np.float32)
    attn = GroupedQueryAttention(cfg, is_cuda=True)
    attn.q_proj, attn.k_proj, attn.v_proj, attn.o_proj = (AGTensor(w, is_cuda=True) for w in (wq, wk, wv, wo))
    out = attn(AGTensor(x, is_cuda=True)).numpy()
    assert out.shape == (S, hid)
    inv = dev_inv_freq[D].astype(np.float32)
    ref = cref.gqa_layer(x, wq, wk, wv, wo, num_heads=Hq, num_kv_heads=Hkv, head_dim=D, inv_freq=inv)
    assert nerr(out, ref) < GATE, nerr(out, ref)
    ref64 = R.gqa_layer_collapsed(x, wq, wk, wv, wo, num_heads=Hq, num_kv_heads=Hkv, head_dim=D, dtype=np.float64,
                                  inv_freq=inv)
    assert nerr(out, ref64) < 2e-5


# S, hidden, Hq, Hkv, D, offset, causal: tiles of 64 keys, groups of 1, 2, 3, 5, 8 and 12 heads; rows to a block, on 148 multiprocessors,
# 1, 2, 4 and 8 collapsed (4 and 2 where 8 are wanted and have no room) and 1, 2, 4, 8 and 16 per head
LAYERS = [
    (1, 128, 4, 2, 32, 0, True),
    (16, 2048, 32, 4, 64, 0, True),
    (65, 100, 5, 5, 20, 3, False),
    (129, 192, 12, 4, 16, 0, True),
    (200, 260, 5, 1, 12, 2, True),
    (333, 768, 12, 1, 64, 0, True),
    (512, 256, 32, 4, 64, 0, False),
    (600, 128, 8, 2, 4, 0, True),
    (900, 128, 8, 4, 64, 0, True),
    (2400, 64, 4, 2, 16, 0, True),
    (2400, 128, 8, 4, 64, 0, False),
    (4200, 64, 8, 4, 64, 0, True),
    (300, 192, 12, 4, 16, 3, True),
]


@pytest.mark.parametrize("S,hid,Hq,Hkv,D,off,causal", LAYERS)
@pytest.mark.parametrize("mode", ["collapsed", "per_head"])
def test_layer_in_one_call(T, dev_inv_freq, S, hid, Hq, Hkv, D, off, causal, mode):
    """bn_attn_layer_f32 against 64 bits (the gate of the layer's other tests) and against the single operators; a row that is not
    finite is seen by the rows behind it alone."""
    import torch
    from baranet_bdml_b200 import _lib
    rng = np.random.default_rng(S + Hq)
    x = rng.standard_normal((S, hid), dtype=np.float32)
    ws = [(rng.standard_normal(s) * hid ** -0.5).astype(np.float32) for s in ((hid, Hq * D), (hid, Hkv * D), (hid, Hkv * D), (Hq * D, hid))]
    scale, hm = D ** -0.5, _lib.BN_HEADS_COLLAPSED if mode == "collapsed" else _lib.BN_HEADS_PER_HEAD
    tx, *tw = (T.TensorF.from_torch(torch.from_numpy(a).cuda()) for a in (x, *ws))
    theta = 10000.0 if S <= 1000 else 1.0      # far from the start a frequency's rounding on one side shows; those of theta 1 are exact
    sizes = dict(num_heads=Hq, num_kv_heads=Hkv, head_dim=D, theta=theta, heads_mode=hm)
    layer = lambda t: t.attention_layer(*tw, scale, causal, off, **sizes)                         # noqa: E731
    got = layer(tx).to_numpy()
    inv = np.array([np.float32(1.0 / float(np.float32(10000.0) ** (np.float32(2 * i) / np.float32(D)))) for i in range(D // 2)], dtype=np.float32)
    inv = dev_inv_freq[D].astype(np.float32) if D in dev_inv_freq else inv
    inv = inv if theta > 1.0 else np.ones_like(inv)
    q, k, v = (x.astype(np.float64) @ w.astype(np.float64) for w in ws[:3])
    core = R.attention_collapsed if mode == "collapsed" else R.attention_per_head
    want = core(q, k, v, num_heads=Hq, num_kv_heads=Hkv, head_dim=D, position_offset=off, causal=causal, dtype=np.float64,
                inv_freq=inv) @ ws[3].astype(np.float64)
    single = tx @ tw[0]
    single = single.attention_fused(tx @ tw[1], tx @ tw[2], scale, causal, off, **sizes) @ tw[3]
    assert nerr(got, want) < 2e-5 and nerr(got, single.to_numpy()) < 2 * GATE, (nerr(got, want), nerr(got, single.to_numpy()))
    if causal and S > 2:
        x[S // 2, 0] = np.inf
        bad = layer(T.TensorF.from_torch(torch.from_numpy(x).cuda())).to_numpy()
        before = S // 2 - off
        assert before <= 0 or np.array_equal(bad[:before], got[:before])
        assert not np.isfinite(bad[S // 2:]).any()


def test_layer_in_one_call_from_several_threads(T):
    """A thread's call of less shared memory (both ask for more than 48 KB, of the same kernel) leaves another thread's limit alone"""
    import threading
    import torch
    from baranet_bdml_b200 import _lib

    def layer(S):
        g = torch.Generator(device="cuda").manual_seed(S)
        x, *w = (T.TensorF.from_torch(torch.randn(s, generator=g, device="cuda") * 0.05) for s in ((S, 256), (256, 2048), (256, 256), (256, 256), (2048, 256)))
        return x.attention_layer(*w, 0.125, False, 0, num_heads=32, num_kv_heads=4, head_dim=64, theta=10000.0, heads_mode=_lib.BN_HEADS_PER_HEAD).to_numpy()

    first, other = layer(512), []
    thread = threading.Thread(target=lambda: other.append(layer(200)))
    thread.start()
    thread.join()
    assert np.array_equal(layer(512), first) and len(other) == 1 and np.array_equal(layer(200), other[0])


def test_layer_in_one_call_refuses_what_it_does_not_take(T):
    import torch
    from baranet_bdml_b200 import _lib
    x = torch.randn(8, 64, device="cuda")
    w = [torch.randn(s, device="cuda") for s in ((64, 48), (64, 12), (64, 12), (48, 64))]
    sizes = dict(num_heads=4, num_kv_heads=1, head_dim=12, theta=10000.0, heads_mode=_lib.BN_HEADS_COLLAPSED)
    run = lambda x, w, off=0, **kw: T.TensorF.from_torch(x).attention_layer(*(T.TensorF.from_torch(t) for t in w), 1.0, True, off, **{**sizes, **kw})   # noqa: E731
    assert run(x, w) is not None
    assert run(x, [w[0].t().contiguous().t()] + w[1:]) is None                       # columns that are not contiguous
    assert run(torch.randn(8, 65, device="cuda")[:, 1:], w) is None                  # rows that do not start on 16 bytes
    assert run(x, w, num_heads=2) is None and run(x, w, -1) is None
    assert run(x, [torch.randn(64, 24, device="cuda"), *(torch.randn(64, 6, device="cuda") for _ in "kv"), torch.randn(24, 64, device="cuda")],
               head_dim=6) is None                                                    # heads that are no multiple of 4


def test_layer_matches_reference_cuda_ops(T, cref):
    """Same inputs through the reference's OWN CUDA operators (compiled from the
    reference tree into oracle/_ref) and through the fused layer."""
    if not cref.gpu_available():
        pytest.skip("oracle/_ref not built (needs the reference tree at build time)")
    from baranet_bdml_b200.layers import GroupedQueryAttention, LLaMAConfig
    from baranet_bdml_b200.tensor import AGTensor
    for cfg, S in ((LLaMAConfig(), 128), (LLaMAConfig(vocab_size=1000, hidden_size=128, intermediate_size=256,
                                                     num_hidden_layers=2, num_attention_heads=4,
                                                     num_key_value_heads=2), 4)):
        rng = np.random.default_rng(5)
        hid, Hq, Hkv, D = cfg.hidden_size, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim
        x = rng.standard_normal((S, hid), dtype=np.float32)
        ws = [(rng.standard_normal(s) * 0.02).astype(np.float32)
              for s in ((hid, Hq * D), (hid, Hkv * D), (hid, Hkv * D), (Hq * D, hid))]
        attn = GroupedQueryAttention(cfg, is_cuda=True)
        attn.q_proj, attn.k_proj, attn.v_proj, attn.o_proj = (AGTensor(w, is_cuda=True) for w in ws)
        out = attn(AGTensor(x, is_cuda=True)).numpy()
        ref = cref.gpu_gqa_layer(x, *ws, num_heads=Hq, num_kv_heads=Hkv, head_dim=D)
        assert nerr(out, ref) < GATE, nerr(out, ref)


def test_host_tensor_ops_raise(T):
    a = T.TensorF(4, 4, is_cuda=False)
    with pytest.raises(RuntimeError, match="only GPU implementation available"):
        a @ a
    with pytest.raises(RuntimeError, match="only GPU implementation available"):
        a.rope()
