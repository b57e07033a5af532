"""The specialised kernels against the general ones (bit for bit) and against 64-bit results, at the sizes and values where a
specialised path can go wrong: tile edges, remainders, degenerate blocks, non-finite words."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _no_device_timeout():
    yield
    from latentq_llm_b200 import _lib
    assert _lib.lib.lq_gemm_device_status(1) == 0, "a bounded device-side wait expired"


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


# ---- fused optimizer step -------------------------------------------------------------------------------------------
def _adam_case(wbit, N, K, seed, grad_kind):
    from latentq_llm_b200 import ops
    g = _gen(seed)
    n = N * K
    blocks = n // (2048 if n % 2048 == 0 else 128)
    per = n // blocks
    grad = (torch.randn(N, K, device="cuda", generator=g) * torch.exp(3 * torch.randn(N, 1, device="cuda", generator=g)) * 1e-4).to(torch.bfloat16)
    if grad_kind == "zero":
        grad.zero_()
    elif grad_kind == "tiny":
        grad = (grad.float() * 1e-33).to(torch.bfloat16)
    elif grad_kind == "nonfinite":
        flat = grad.view(-1)
        flat[5], flat[(per + 3) % n], flat[n - 1] = float("inf"), float("nan"), -float("inf")
        flat[2 * per:3 * per] = float("nan")
    st = [torch.randint(0, 256, (N, K), device="cuda", generator=g, dtype=torch.uint8) for _ in range(2)]
    sc = [torch.rand(blocks, 1, device="cuda", generator=g) * 1e-5 + 1e-10 for _ in range(2)]
    tm = [torch.rand(blocks, 1, device="cuda", generator=g) * 1e-3 for _ in range(2)]
    words = torch.randint(-2 ** 31, 2 ** 31, (n // 8,), device="cuda", generator=g, dtype=torch.int64).to(torch.int32)
    hyper = ops.make_adam_hyper(0.9, 0.95, 1e-8, 1e-3)

    def run(has_residual):
        o = ops.make_opts(codec=ops.CODEC_THREEFOLD, dither=ops.DITHER_HASH, has_residual=has_residual, mu_enc=1, mu_dec=0)
        a = [t.clone() for t in (st[0], sc[0], tm[0], st[1], sc[1], tm[1])]
        w = words.clone()
        gg = _gen(seed + 1)
        if wbit == 4:
            codes = torch.randint(-128, 128, (n // 2,), device="cuda", generator=gg, dtype=torch.int8)
            s = (torch.rand(n // 128, device="cuda", generator=gg) * 0.01 + 1e-3).to(torch.bfloat16)
            z = torch.randint(0, 16, (n // 128,), device="cuda", generator=gg).to(torch.bfloat16)
            ops.adam_a16w4_step(codes, w, grad, s, z, *a, hyper, o)
        else:
            codes = torch.randint(-128, 128, (N, K), device="cuda", generator=gg, dtype=torch.int8)
            s = (torch.rand(N, device="cuda", generator=gg) * 0.01 + 1e-4).to(torch.bfloat16)
            ops.adam_a8w8_step(codes, w, grad, s, *a, hyper, o)
        return [codes, w] + a

    return run, torch.isfinite(grad.float()).view(blocks, per).all(1)


@pytest.mark.parametrize("wbit", [4, 8])
@pytest.mark.parametrize("N,K", [(16, 128), (64, 32 * 128), (3, 1152), (1088, 1152), (520, 128)])
@pytest.mark.parametrize("grad_kind", ["normal", "zero", "tiny", "nonfinite"])
def test_fast_optimizer_step_equals_generic_kernel(monkeypatch, wbit, N, K, grad_kind):
    run, finite = _adam_case(wbit, N, K, 7 * N + K, grad_kind)
    for has_residual in (True, False):
        monkeypatch.delenv("LQ_REQUANT_GENERIC", raising=False)
        fast = run(has_residual)
        monkeypatch.setenv("LQ_REQUANT_GENERIC", "1")
        slow = run(has_residual)
        for a, b in zip(fast, slow):
            # state blocks with a non-finite gradient have no defined result; they must not touch the others
            assert torch.equal(a.reshape(finite.numel(), -1)[finite], b.reshape(finite.numel(), -1)[finite])


def test_int8_optimizer_step_captured_before_its_table_exists():
    """The first step at a curve level builds a table, which ends with a synchronisation; under capture the generic kernel steps in."""
    from latentq_llm_b200 import ops
    g = _gen(5)
    N, K = 8, 256
    grad = (torch.randn(N, K, device="cuda", generator=g) * 1e-3).to(torch.bfloat16)
    qs = torch.full((N,), 0.01, device="cuda").to(torch.bfloat16)
    codes0 = torch.randint(-100, 100, (N, K), device="cuda", generator=g, dtype=torch.int8)
    hyper = ops.make_adam_hyper(0.9, 0.95, 1e-8, 1e-3)
    o = ops.make_opts(codec=ops.CODEC_THREEFOLD, dither=ops.DITHER_HASH, has_residual=False, mu_enc=3, v0=0.03125)   # a table of its own

    def state():
        z = torch.zeros(1, 1, device="cuda")
        return [codes0.clone(), torch.zeros(N * K // 8, dtype=torch.int32, device="cuda")] + [
            t for _ in range(2) for t in (torch.zeros(N, K, dtype=torch.uint8, device="cuda"), z + 1e-10, z.clone())]

    a, b = state(), state()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.adam_a8w8_step(a[0], a[1], grad, qs, *a[2:], hyper, o)
    graph.replay()
    ops.adam_a8w8_step(b[0], b[1], grad, qs, *b[2:], hyper, o)
    for x, y in zip(a, b):
        assert torch.equal(x, y)


@pytest.mark.parametrize("kind", ["step4", "step8", "fold4", "fold8"])
@pytest.mark.parametrize("v0", [0.0, 0.125])
def test_captured_launch_keeps_its_hash_offset(monkeypatch, kind, v0):
    """A launch captured with one hash offset replays with it after calls with other offsets have built what they need."""
    from latentq_llm_b200 import ops
    g = _gen(11)
    N, K = 16, 2048
    n, blocks = N * K, N * K // 2048
    codes0 = torch.randint(-128, 128, (N, K) if kind.endswith("8") else (n // 2,), device="cuda", generator=g, dtype=torch.int8)
    words0 = torch.randint(-2 ** 31, 2 ** 31, (n // 8,), device="cuda", generator=g, dtype=torch.int64).to(torch.int32)
    upd = (torch.randn(N, K, device="cuda", generator=g) * 1e-3).to(torch.bfloat16)
    rows = N if kind.endswith("8") else n // 128
    s = (torch.rand(rows, device="cuda", generator=g) * 0.01 + 1e-3).to(torch.bfloat16)
    z = torch.randint(0, 16, (rows,), device="cuda", generator=g).to(torch.bfloat16)
    hyper = ops.make_adam_hyper(0.9, 0.95, 1e-8, 1e-3)

    def launch(offset):
        o = ops.make_opts(codec=ops.CODEC_THREEFOLD, dither=ops.DITHER_HASH, has_residual=True, mu_enc=2, mu_dec=2, v0=offset)
        c, w = codes0.clone(), words0.clone()
        st = [t for _ in range(2) for t in (torch.zeros(N, K, dtype=torch.uint8, device="cuda"), torch.full((blocks, 1), 1e-10, device="cuda"),
                                            torch.zeros(blocks, 1, device="cuda"))]
        if kind == "step4":
            ops.adam_a16w4_step(c, w, upd, s, z, *st, hyper, o)
        elif kind == "step8":
            ops.adam_a8w8_step(c, w, upd, s, *st, hyper, o)
        elif kind == "fold4":
            ops.a16w4_fold_delta(c, w, upd.view(-1), s, z, o)
        else:
            ops.a8w8_fold_delta(c, w, upd, s, o)
        return c, w

    monkeypatch.setenv("LQ_REQUANT_GENERIC", "1")
    want = launch(v0)
    monkeypatch.delenv("LQ_REQUANT_GENERIC")
    launch(v0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = launch(v0)
    for other in (0.0, 0.125, 0.25, 0.375):
        if other != v0:
            launch(other)
    graph.replay()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


# ---- requantize with Philox dither ----------------------------------------------------------------------------------
@pytest.mark.parametrize("seed,step,param", [(0, 0, 0), (1234, 7, 3), (2 ** 64 - 1, 2 ** 32 - 1, 2 ** 32 - 1)])
def test_philox_fold_equals_generic_kernel(monkeypatch, seed, step, param):
    from latentq_llm_b200 import ops
    g = _gen(3)
    n = 1024 * 128
    codes = torch.randint(-128, 128, (n // 2,), device="cuda", generator=g, dtype=torch.int8)
    words = torch.randint(-2 ** 31, 2 ** 31, (n // 8,), device="cuda", generator=g, dtype=torch.int64).to(torch.int32)
    s = (torch.rand(n // 128, device="cuda", generator=g) * 0.01 + 1e-3).to(torch.bfloat16)
    z = torch.randint(0, 16, (n // 128,), device="cuda", generator=g).to(torch.bfloat16)
    delta = (torch.randn(n, device="cuda", generator=g) * 1e-3).to(torch.bfloat16)
    out = []
    for generic in (False, True):
        monkeypatch.setenv("LQ_REQUANT_GENERIC", "1") if generic else monkeypatch.delenv("LQ_REQUANT_GENERIC", raising=False)
        c, w = codes.clone(), words.clone()
        ops.a16w4_fold_delta(c, w, delta, s, z, ops.make_opts(codec=ops.CODEC_THREEFOLD, dither=ops.DITHER_PHILOX, seed=seed, step=step,
                                                              param_id=param))
        out.append((c, w))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


# ---- A16W4 forward and grad-input at the edges of the token tiles ----------------------------------------------------
def _w4(N, K, seed, group=128):
    g = _gen(seed)
    q = torch.randint(0, 16, (N * K // 2, 2), device="cuda", generator=g, dtype=torch.uint8)
    s = (torch.rand(N * K // group, device="cuda", generator=g) * 0.01 + 1e-3).to(torch.bfloat16)
    z = torch.randint(0, 16, (N * K // group,), device="cuda", generator=g).to(torch.bfloat16)
    w = ((q.view(-1, group).double() - z.double()[:, None]) * s.double()[:, None]).view(N, K)
    return ((q[:, 0] << 4) | q[:, 1]).view(torch.int8).contiguous(), s, z, w


# bf16 weight and output roundings (2^-9 each, uncorrelated) leave a relative 2-norm error below 2.5e-3; a misplaced or missing tile,
# group or token is of order 1
@pytest.mark.parametrize("M", [3, 16, 17, 31, 33, 64, 65, 96, 97, 128, 129, 160, 161, 192, 193, 257, 300])
@pytest.mark.parametrize("N,K,group", [(128, 256, 128), (192, 384, 128), (4160, 2176, 128), (320, 512, 64), (256, 1024, 256)])
def test_a16w4_token_tile_edges(M, N, K, group):
    from latentq_llm_b200 import ops
    codes, s, z, w = _w4(N, K, N + K, group)
    g = _gen(M)
    x, bias = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16), torch.randn(N, device="cuda", generator=g).to(torch.bfloat16)
    for b in (None, bias):
        y = ops.gemm_a16w4_fwd(x, codes, s, z, b, N, K, group)
        ref = x.double() @ w.t() + (0 if b is None else b.double())
        assert float((y.double() - ref).norm() / ref.norm()) < 4e-3
    dy = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16)
    dx = ops.gemm_a16w4_dgrad(dy, codes, s, z, N, K, group)
    ref = dy.double() @ w
    assert float((dx.double() - ref).norm() / ref.norm()) < 4e-3


# The grad-input at the token count from which the transposed copy is considered, on both sides of its rule, with the default dispatch.
# Neither route splits the contraction at these shapes, so the bits agree.
@pytest.mark.parametrize("M", [1791, 1792, 1793, 2047, 2560])
@pytest.mark.parametrize("N,K", [(2112, 2048), (4160, 2304), (1088, 2560), (4096, 1536)])
def test_grad_input_routes_agree_bitwise(monkeypatch, M, N, K):
    from latentq_llm_b200 import ops
    codes, s, z, w = _w4(N, K, N + K)
    dy = torch.randn(M, N, device="cuda", generator=_gen(M)).to(torch.bfloat16)
    out = []
    for mode in (None, "0", "1"):
        monkeypatch.delenv("LQ_GEMM_DGRAD_TRANSPOSE", raising=False) if mode is None else monkeypatch.setenv("LQ_GEMM_DGRAD_TRANSPOSE", mode)
        ops._ws_need.clear()
        out.append(ops.gemm_a16w4_dgrad(dy, codes, s, z, N, K))
    ops._ws_need.clear()
    ref = dy.double() @ w
    assert float((out[0].double() - ref).norm() / ref.norm()) < 4e-3
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])


# Every token-tile width with the weight tile in tensor memory and in shared memory: the same bf16 weights in the same order, so the
# same bits.  11008 rows, so that the widest tile without padding is the cheapest (24 tokens: 32 wide ... 250: 256); 1152 = nine groups, whose
# parameters are not staged.
@pytest.mark.parametrize("M", [24, 64, 90, 128, 150, 190, 250])
@pytest.mark.parametrize("N,K", [(11008, 1024), (11008, 1152), (1024, 11008)])
def test_operand_placements_agree_at_every_tile_width(monkeypatch, M, N, K):
    from latentq_llm_b200 import ops
    codes, s, z, w = _w4(N, K, N + K)
    g = _gen(M)
    x, dy = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16), torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16)
    out = {}
    for where in ("tmem", "smem"):
        monkeypatch.setenv("LQ_GEMM_A_OPERAND", where)
        out[where] = (ops.gemm_a16w4_fwd(x, codes, s, z, None, N, K), ops.gemm_a16w4_dgrad(dy, codes, s, z, N, K))
    for a, b, ref in zip(out["tmem"], out["smem"], (x.double() @ w.t(), dy.double() @ w)):
        assert torch.equal(a, b)
        assert float((a.double() - ref).norm() / ref.norm()) < 4e-3


# ---- A8W8 linear ------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("M,N,K", [(5, 64, 128), (130, 200, 256), (2048, 512, 1024), (64, 4096, 2048)])
@pytest.mark.parametrize("with_bias", [True, False])
def test_a8w8_module_launch_equals_the_op_chain(M, N, K, with_bias):
    from latentq_llm_b200 import ops
    g = _gen(M + N)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w8 = torch.randint(-128, 128, (N, K), device="cuda", generator=g, dtype=torch.int8)
    qs = (torch.rand(N, 1, device="cuda", generator=g) * 0.01 + 1e-4).to(torch.bfloat16)
    bias = (torch.randn(N, device="cuda", generator=g) * 0.1).to(torch.bfloat16) if with_bias else None
    x8, clampv = ops.act_quant_per_tensor(x)
    b = ((bias if with_bias else 0 * qs.view(-1)) / (qs.view(-1) if with_bias else 1)).to(torch.bfloat16).contiguous()
    alpha = (clampv.to(torch.bfloat16) / 127.).float().reshape(1).expand(M).contiguous()
    ref = ops.gemm_a8w8(x8, w8, alpha, None, 1.0, b) * qs.view(1, -1)
    assert torch.equal(ops.gemm_a8w8_module(x8, w8, clampv, 1.0, bias, qs), ref)
    static = ops.gemm_a8w8(x8, w8, torch.full((M,), 2.5 / 127., device="cuda"), None, 1.0, b) * qs.view(1, -1)
    assert torch.equal(ops.gemm_a8w8_module(x8, w8, None, 2.5 / 127., bias, qs), static)


@pytest.mark.parametrize("rows,cols", [(1, 16), (7, 48), (33, 1000), (512, 2048)])
def test_i8_dequant_equals_the_op_chain(rows, cols):
    from latentq_llm_b200 import ops
    g = _gen(rows)
    c = torch.randint(-128, 128, (rows, cols), device="cuda", generator=g, dtype=torch.int8)
    qs = (torch.rand(rows, 1, device="cuda", generator=g) * 0.01).to(torch.bfloat16)
    clampv = torch.tensor([3.140625], device="cuda")
    assert torch.equal(ops.i8_dequant(c, row_scales=qs), c.to(torch.bfloat16) * qs)
    assert torch.equal(ops.i8_dequant(c, clampv=clampv), c.to(torch.bfloat16) * (clampv.to(torch.bfloat16) / 127.))


@pytest.mark.parametrize("scale", [1.0, 1e-30, 3e4])
def test_per_tensor_activation_quantizer_equals_the_op_chain(scale):
    from latentq_llm_b200 import ops
    x = (torch.randn(64, 4096, device="cuda", generator=_gen(9)) * scale).to(torch.bfloat16)
    x8, clampv = ops.act_quant_per_tensor(x)
    ref = (x * 127. / x.max()).round_().clamp_(-128, 127).to(torch.int8)
    assert float(clampv) == float(x.max()) and torch.equal(x8, ref)


@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 2040), (5, 2056), (40, 8192)])
def test_gradient_accumulator_with_philox_noise_equals_the_generic_kernel(rows, cols):
    """bf16 gradients with the library's own noise take the packed kernel; the same noise from a buffer takes the generic one, which the
    reference's vectors pin.  Bit for bit, first and later micro-batches, gradients that are not finite and scales whose reciprocal is
    not used included."""
    from latentq_llm_b200 import ops
    g = _gen(cols)
    q = [torch.zeros(rows, cols, dtype=torch.int8, device="cuda") for _ in range(2)]
    sc = [torch.zeros(rows, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    for it in range(4):
        f = (torch.randn(rows, cols, device="cuda", generator=g) * 10.0 ** (it - 3)).to(torch.bfloat16)
        if it == 2:
            f.view(-1)[:4] = torch.tensor([float("nan"), float("inf"), -float("inf"), 1e-40])
        if it == 3:                                   # scales beyond 2^40 and below 2^-40
            for s in sc:
                s[0], s[rows - 1] = 2.0 ** 45, 2.0 ** -45 if rows > 1 else 2.0 ** 45
        noise = ops.philox_dither(7, ((it + 1) << 32) | 11, rows * cols // 8, "cuda")
        ops.gradq_accumulate(f, q[0], sc[0], it == 0, ops.make_opts(dither=ops.DITHER_PHILOX, seed=7, step=it + 1, param_id=11))
        ops.gradq_accumulate(f, q[1], sc[1], it == 0, ops.make_opts(dither=ops.DITHER_EXPLICIT, dither_buf=noise))
        assert torch.equal(q[0], q[1]) and torch.equal(sc[0], sc[1]), it


@pytest.mark.parametrize("n", [8, 8 * 255, 8 * 257, 8 * 148 * 8 * 256 * 2 + 8])
def test_per_tensor_activation_quantizer_sizes_and_special_values(n):
    from latentq_llm_b200 import ops
    x = (torch.randn(n, device="cuda", generator=_gen(n)) * 3).to(torch.bfloat16)
    for case in ("plain", "negative", "nan", "max at the end"):
        y = -x.abs() - 1 if case == "negative" else x.clone()
        if case == "nan":
            y[n // 2] = float("nan")
        if case == "max at the end":
            y[n - 1] = 100.0
        x8, clampv = ops.act_quant_per_tensor(y)
        top = torch.where(torch.isnan(y), torch.full_like(y, -float("inf")), y).max()          # NaN is passed over, and its code is -128
        ref = (y * 127. / top).round_().clamp_(-128, 127)
        ref = torch.where(torch.isnan(y), torch.full_like(y, -128.0), ref).to(torch.int8)
        assert float(clampv) == float(top) and torch.equal(x8, ref), case


@pytest.mark.parametrize("rows,cols", [(1, 16), (3, 11008), (2047, 1040), (1200, 4112)])
def test_i8_dequant_rows_by_multiplication(rows, cols):
    from latentq_llm_b200 import ops
    c = torch.randint(-128, 128, (rows, cols), device="cuda", generator=_gen(cols), dtype=torch.int8)
    qs = (torch.rand(rows, 1, device="cuda", generator=_gen(rows)) * 0.01 + 1e-3).to(torch.bfloat16)
    assert torch.equal(ops.i8_dequant(c, row_scales=qs), c.to(torch.bfloat16) * qs)


# The widths of 48, 80 and 112 tokens, which only the two-block kernel has: one and two tiles, a token to spare and none, with and without
# split-K; the same bits with the weight tile in shared memory, where those launches take the next width, and with group parameters
# that cannot be staged (their address is odd).
@pytest.mark.parametrize("M", [33, 48, 80, 81, 97, 112, 200, 224])
@pytest.mark.parametrize("N,K", [(11008, 1024), (8192, 2048), (2048, 4096)])
def test_token_tiles_between_the_multiples_of_32(monkeypatch, M, N, K):
    from latentq_llm_b200 import ops
    codes, s, z, w = _w4(N, K, N + K)
    x = torch.randn(M, K, device="cuda", generator=_gen(M)).to(torch.bfloat16)
    odd = [torch.cat([t.reshape(-1)[:1], t.reshape(-1)])[1:] for t in (s, z)]
    out = [ops.gemm_a16w4_fwd(x, codes, s, z, None, N, K), ops.gemm_a16w4_fwd(x, codes, *odd, None, N, K)]
    monkeypatch.setenv("LQ_GEMM_A_OPERAND", "smem")
    out.append(ops.gemm_a16w4_fwd(x, codes, s, z, None, N, K))
    ref = x.double() @ w.t()
    assert float((out[0].double() - ref).norm() / ref.norm()) < 4e-3
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])


def test_i8_dequant_beyond_2_to_the_35_codes():
    """There is no size from which the codes are converted one by one (8.6 times slower per code); the last rows take their own scales."""
    from latentq_llm_b200 import ops
    if torch.cuda.mem_get_info()[0] < 125 << 30:
        pytest.skip("needs 103 GB on the device")
    per_code = []
    for rows, cols in ((1 << 15, 32784), ((1 << 20) + 33, 32784)):
        c = torch.full((rows, cols), 3, dtype=torch.int8, device="cuda")
        s = (torch.arange(rows, device="cuda") % 251 + 1).to(torch.bfloat16)
        y, ms = None, []
        for _ in range(4):
            y = None                                                # its memory serves the next call
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            y = ops.i8_dequant(c, row_scales=s)
            b.record()
            b.synchronize()
            ms.append(a.elapsed_time(b))
        per_code.append(min(ms) / c.numel())
        for r in (0, 1, rows // 2, rows - 2, rows - 1):
            assert torch.equal(y[r], c[r].to(torch.bfloat16) * s[r])
        del c, y
        torch.cuda.empty_cache()
    assert per_code[1] < 3 * per_code[0], per_code
