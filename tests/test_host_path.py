"""The native host path (`_lqhost`) serves plain calls and leaves every other to the Python that checks, raises or handles it."""
import pytest
import torch


def test_what_is_not_plain_is_left_to_python():
    from latentq_llm_b200 import _lqhost as h, ops
    x, w, s = torch.zeros(4, 128, dtype=torch.bfloat16), torch.zeros(64 * 64, dtype=torch.int8), torch.zeros(64, dtype=torch.bfloat16)
    x8 = torch.zeros(4, 128, dtype=torch.int8)
    for r in (h.w4_gemm(False, x, w, s, s, None, 64, 128, 128, None, 0), h.w4_gemm(True, None, w, s, s, None, 64, 128, 128, None, 0),
              h.a8w8_gemm(x8, x8, None, None, 1.0, None, None, 0), h.a8w8_module(x8, x8, None, 1.0, None, s, None, 0),
              h.act_quant_per_token(x), h.act_quant_per_tensor(3), h.i8_dequant(x8, None, None)):
        assert r is None                                             # CPU tensors, no tensors
    with pytest.raises(TypeError):
        h.act_quant_per_token()
    with pytest.raises(TypeError):
        h.w4_gemm(False, x)
    for call in (lambda: ops.gemm_a16w4_fwd(x, w, s, s, None, 64, 128), lambda: ops.gemm_a16w4_dgrad(x, w, s, s, 64, 128), lambda: ops.gemm_a8w8(x8, x8),
                 lambda: ops.act_quant_per_token(x), lambda: ops.act_quant_per_tensor(x), lambda: ops.i8_dequant(x8, row_scales=s),
                 lambda: ops.act_quant_per_tensor(None)):
        with pytest.raises(ValueError):
            call()


@pytest.mark.gpu
@pytest.mark.parametrize("M", [0, 1, 17, 300])
def test_native_and_python_paths_agree_and_refuse_alike(M, monkeypatch):
    from latentq_llm_b200 import ops
    N, K = 192, 256
    g = torch.Generator(device="cuda").manual_seed(M)
    x, dy = (torch.randn(M, c, device="cuda", generator=g).to(torch.bfloat16) for c in (K, N))
    w = torch.randint(-128, 128, (N * K // 2,), device="cuda", generator=g, dtype=torch.int8)
    s = (torch.rand(N * K // 128, device="cuda", generator=g) * 0.01).to(torch.bfloat16)
    z = torch.randint(0, 16, s.shape, device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g).to(torch.bfloat16)
    w8 = torch.randint(-128, 128, (N, K), device="cuda", generator=g, dtype=torch.int8)
    x8 = torch.randint(-128, 128, (M, K), device="cuda", generator=g, dtype=torch.int8)
    rs, cs, qs = torch.rand(M, device="cuda", generator=g), torch.rand(N, device="cuda", generator=g), (torch.rand(N, 1, device="cuda", generator=g) + 0.1).to(torch.bfloat16)
    one = torch.full((1,), 2.5, device="cuda")
    good = [lambda: ops.gemm_a16w4_fwd(x, w, s, z, bias, N, K), lambda: ops.gemm_a16w4_fwd(x, w, s.view(-1, 1), z.view(-1, 1), None, N, K),
            lambda: ops.gemm_a16w4_dgrad(dy, w, s, z, N, K), lambda: ops.gemm_a8w8(x8, w8, rs, cs, 0.5, bias), lambda: ops.gemm_a8w8(x8, w8),
            lambda: ops.gemm_a8w8_module(x8, w8, one, 1.0, bias, qs), lambda: ops.gemm_a8w8_module(x8, w8, None, 0.01, None, qs),
            lambda: ops.act_quant_per_token(x), lambda: ops.act_quant_per_tensor(x) if M else (x, x), lambda: ops.i8_dequant(w8, row_scales=qs), lambda: ops.i8_dequant(x8, clampv=one)]
    bad = [lambda: ops.gemm_a16w4_fwd(x.float(), w, s, z, None, N, K), lambda: ops.gemm_a16w4_fwd(x.t().contiguous().t()[:, ::2], w, s, z, None, N, K // 2),
           lambda: ops.gemm_a16w4_fwd(x, w[:-1], s, z, None, N, K), lambda: ops.gemm_a16w4_fwd(x, w, s.float(), z, None, N, K), lambda: ops.gemm_a16w4_fwd(x, w, s, z, bias, N, K, group=96),
           lambda: ops.gemm_a16w4_fwd(x.cpu(), w, s, z, None, N, K), lambda: ops.gemm_a16w4_dgrad(dy, w, s, z, K, N), lambda: ops.gemm_a8w8(x8, w8[:, :128]),
           lambda: ops.gemm_a8w8_module(x8, w8, one.double(), 1.0, None, qs), lambda: ops.gemm_a8w8_module(x8, w8, None, 1.0, bias[:-1], qs),
           lambda: ops.act_quant_per_token(x[:, :100]), lambda: ops.act_quant_per_token(x.half()), lambda: ops.i8_dequant(w8, row_scales=qs[:-1]), lambda: ops.i8_dequant(w8)]

    def outcome(f):
        try:
            r = f()
        except Exception as e:                                       # noqa: BLE001
            return type(e), str(e)
        return r if isinstance(r, tuple) else (r,)

    native = [outcome(f) for f in good + bad]

    class Off:
        def __getattr__(self, name):
            return lambda *a: None
    monkeypatch.setattr(ops, "_host", Off())
    for f, a, n in zip(good + bad, native, range(100)):
        b = outcome(f)
        assert len(a) == len(b), (n, a, b)
        for u, v in zip(a, b):
            if isinstance(u, torch.Tensor):
                assert u.dtype == v.dtype and u.shape == v.shape and torch.equal(u, v), n
            else:
                assert u == v, (n, a, b)
