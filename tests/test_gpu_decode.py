"""GPU parity of the decode-side kernels (residual add + RMSNorm, RoPE + KV store, single-query attention,
silu*up) against the CPU oracle.  Tolerance: one bf16 ulp (2^-8 relative) on at least 99.5 % of the elements and
2^-6 of the largest magnitude on all (reduction order and transcendental implementations differ)."""
import numpy as np
import pytest
import torch

import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from latentq_llm_b200 import ops as _ops
    return _ops


def _close(got, want, frac=0.995):
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    err = np.abs(got - want) / np.maximum(np.abs(want), 1e-6)
    assert (err <= 2.0 ** -8 + 1e-9).mean() >= frac, (err <= 2.0 ** -8).mean()
    assert np.abs(got - want).max() <= 2.0 ** -6 * np.abs(want).max()


def _bf(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().to(torch.bfloat16)


@pytest.mark.parametrize("hf", [True, False])
@pytest.mark.parametrize("M,K", [(1, 4096), (16, 4096), (3, 11008), (64, 2048)])
def test_add_rmsnorm(ops, M, K, hf):
    rng = np.random.default_rng(M * 7 + K)
    h = orc.bf16_round(rng.standard_normal((M, K)).astype(np.float32))
    d = orc.bf16_round(rng.standard_normal((M, K)).astype(np.float32) * 0.5)
    gamma = orc.bf16_round((1 + 0.1 * rng.standard_normal(K)).astype(np.float32))
    for delta in (d, None):
        hd_ = _bf(h)
        y = ops.add_rmsnorm(hd_, None if delta is None else _bf(delta), _bf(gamma), 1e-5, hf_rounding=hf)
        want_h, want_y = orc.rmsnorm(h, gamma, 1e-5, delta=delta, hf_rounding=hf)
        assert np.array_equal(hd_.float().cpu().numpy(), want_h)            # the residual stream is exact
        _close(y.float().cpu().numpy(), want_y)


@pytest.mark.parametrize("hf", [True, False])
@pytest.mark.parametrize("B,Hq,Hkv,hd", [(1, 32, 32, 128), (4, 8, 2, 64)])
def test_rope_kv_store(ops, B, Hq, Hkv, hd, hf):
    rng = np.random.default_rng(B + Hq)
    max_len = 96
    qkv = orc.bf16_round(rng.standard_normal((B, (Hq + 2 * Hkv) * hd)).astype(np.float32))
    pos = rng.integers(0, max_len, B).astype(np.int64)
    inv_freq = (1.0 / (10000.0 ** (np.arange(0, hd, 2, dtype=np.float32) / hd))).astype(np.float32)
    kc = torch.zeros((B, Hkv, max_len, hd), dtype=torch.bfloat16, device="cuda")
    vc = torch.zeros_like(kc)
    t = _bf(qkv)
    ops.rope_kv_store(t, torch.from_numpy(pos).cuda(), torch.from_numpy(inv_freq).cuda(), kc, vc, Hq, Hkv, hd, hf_rounding=hf)
    got = t.float().cpu().numpy()
    q = qkv[:, :Hq * hd].reshape(B, Hq, hd)
    k = qkv[:, Hq * hd:(Hq + Hkv) * hd].reshape(B, Hkv, hd)
    v = qkv[:, (Hq + Hkv) * hd:].reshape(B, Hkv, hd)
    _close(got[:, :Hq * hd].reshape(B, Hq, hd), orc.rope_rotate_half(q, pos[:, None], inv_freq, hf_rounding=hf))
    assert np.array_equal(got[:, Hq * hd:], qkv[:, Hq * hd:])              # k and v columns of the row are left alone
    kr = orc.rope_rotate_half(k, pos[:, None], inv_freq, hf_rounding=hf)
    kcn, vcn = kc.float().cpu().numpy(), vc.float().cpu().numpy()
    for b in range(B):
        _close(kcn[b, :, pos[b]], kr[b])
        assert np.array_equal(vcn[b, :, pos[b]], v[b])
        mask = np.ones(max_len, bool); mask[pos[b]] = False
        assert not kcn[b][:, mask].any() and not vcn[b][:, mask].any()     # nothing else was written


@pytest.mark.parametrize("hf", [True, False])
@pytest.mark.parametrize("B,P,Hq,Hkv,hd", [(2, 200, 32, 32, 128), (16, 1, 64, 16, 64), (19, 1, 64, 16, 64), (3, 67, 5, 5, 16), (1, 1100, 2, 1, 512), (7, 41, 6, 3, 40)])
def test_rope_kv_store_of_many_tokens_equals_the_calls_of_single_tokens(ops, B, P, Hq, Hkv, hd, hf):
    """In large calls a thread serves several heads; a token by itself takes the kernel of one rotation pair per thread.
    The same bits: head sets that do not divide the heads, head sizes that leave threads idle, positions beyond the cache."""
    g = torch.Generator(device="cuda").manual_seed(B + P)
    qkv = torch.randn(B * P, (Hq + 2 * Hkv) * hd, device="cuda", generator=g).to(torch.bfloat16)
    pos = torch.arange(P, device="cuda").repeat(B) + 3
    pos[-1] = P + 40
    inv_freq = 1.0 / (10000.0 ** (torch.arange(0, hd, 2, dtype=torch.float32, device="cuda") / hd))
    caches = [torch.zeros(B, Hkv, P + 8, hd, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    want = qkv.clone()
    for m in range(B * P):
        b = m // P
        ops.rope_kv_store(want[m:m + 1], pos[m:m + 1], inv_freq, caches[0][b:b + 1], caches[1][b:b + 1], Hq, Hkv, hd, hf_rounding=hf)
    ops.rope_kv_store(qkv, pos, inv_freq, caches[2], caches[3], Hq, Hkv, hd, tokens_per_seq=P, hf_rounding=hf)
    assert torch.equal(qkv, want) and torch.equal(caches[2], caches[0]) and torch.equal(caches[3], caches[1])


@pytest.mark.parametrize("P,Hq,Hkv,hd,several", [(18, 32, 32, 128, False), (19, 32, 32, 128, True), (383, 4, 2, 64, False), (384, 4, 2, 64, True),
                                                 (63, 32, 8, 256, False), (64, 32, 8, 256, True), (2047, 1, 1, 128, False), (2048, 1, 1, 128, True),
                                                 (400, 6, 3, 12, False)])
def test_rope_kernel_of_small_and_of_large_calls(ops, kernel_of, P, Hq, Hkv, hd, several):
    """Both sides of each line of the rule: many heads, few, large ones, three; a head size that is not a multiple of eight keeps the general kernel."""
    qkv = torch.zeros(P, (Hq + 2 * Hkv) * hd, device="cuda", dtype=torch.bfloat16)
    cache = [torch.zeros(1, Hkv, P, hd, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    pos, inv_freq = torch.arange(P, device="cuda"), torch.ones(hd // 2, device="cuda")
    ran = kernel_of(lambda: ops.rope_kv_store(qkv, pos, inv_freq, *cache, Hq, Hkv, hd, tokens_per_seq=P))
    assert ran == ("k_rope_kv_store4" if several else "k_rope_kv_store")


@pytest.mark.parametrize("B,Hq,Hkv,hd,max_len", [(1, 32, 32, 128, 1024), (16, 32, 32, 128, 640), (3, 8, 2, 64, 200), (64, 8, 8, 128, 96)])
def test_decode_attention(ops, B, Hq, Hkv, hd, max_len):
    rng = np.random.default_rng(B * 3 + hd)
    qkv = orc.bf16_round(rng.standard_normal((B, (Hq + 2 * Hkv) * hd)).astype(np.float32))
    kc = orc.bf16_round(rng.standard_normal((B, Hkv, max_len, hd)).astype(np.float32))
    vc = orc.bf16_round(rng.standard_normal((B, Hkv, max_len, hd)).astype(np.float32))
    pos = rng.integers(0, max_len, B).astype(np.int64)
    pos[0] = max_len - 1
    if B > 1:
        pos[1] = 0
    for _ in range(2):          # twice: the ticket counters must have been left at zero
        out = ops.decode_attention(_bf(qkv), torch.from_numpy(pos).cuda(), _bf(kc), _bf(vc), Hq, Hkv, hd)
        want = orc.decode_attention(qkv[:, :Hq * hd].reshape(B, Hq, hd), kc, vc, pos, hd ** -0.5)
        got = out.float().cpu().numpy().reshape(B, Hq, hd)
        assert np.abs(got - want).max() <= 2.0 ** -7 * np.abs(want).max()


@pytest.mark.parametrize("hf", [True, False])
def test_silu_mul(ops, hf):
    rng = np.random.default_rng(5)
    gu = orc.bf16_round((rng.standard_normal((7, 2 * 11008)) * 2).astype(np.float32))
    got = ops.silu_mul(_bf(gu), hf_rounding=hf).float().cpu().numpy()
    _close(got, orc.silu_mul(gu, hf_rounding=hf))


@pytest.mark.parametrize("hf", [True, False])
@pytest.mark.parametrize("M,I,K", [(1, 1024, 4096), (2, 544, 4096), (8, 1024, 1024), (16, 288, 2048), (48, 512, 1024)])
def test_fused_gate_up_silu(ops, M, I, K, hf):
    """silu(x·Wgate^T) * (x·Wup^T) from the fused 2I-row weight: one launch at decode sizes (streaming kernel for one
    or two tokens, row-block kernel up to 16), GEMM + silu*up beyond; against the oracle's dequantize-matmul-silu chain
    within two bf16 ulps of the largest magnitude."""
    rng = np.random.default_rng(M + I)
    w = orc.bf16_round((rng.standard_normal((2 * I, K)) * 0.02).astype(np.float32))
    s, z = orc.find_qparams(w, 128, 15, False)
    s, z = orc.bf16_round(s), orc.bf16_round(z)
    codes, _, _ = orc.a16w4_requant(s, z, w=w, codec=orc.CODEC_NONE, math_bf16=True)
    x = orc.bf16_round(rng.standard_normal((M, K)).astype(np.float32))
    got = ops.gemm_a16w4_fwd_silu(_bf(x), torch.from_numpy(codes).cuda(), _bf(s), _bf(z), I, K, hf_rounding=hf).float().cpu().numpy()
    gu = orc.gemm_a16w4(x, codes, s, z, 2 * I, K)
    want = orc.silu_mul(gu, hf_rounding=hf)
    # (both projections are rounded to bf16 before silu and the product: an ulp in either moves the product by up to two)
    assert np.abs(got - want).max() <= 2.0 ** -6 * np.abs(want).max()
    # and exactly what the two separate launches give (same GEMM kernels, same rounding points)
    sep = ops.silu_mul(ops.gemm_a16w4_fwd(_bf(x), torch.from_numpy(codes).cuda(), _bf(s), _bf(z), None, 2 * I, K), hf_rounding=hf)
    if M <= 16:
        assert np.array_equal(got, sep.float().cpu().numpy())


@pytest.mark.parametrize("B,V,D", [(1, 32000, 4096), (16, 32000, 4096), (3, 1027, 256), (64, 50272, 2048), (2, 8, 8)])
def test_argmax_embed(ops, B, V, D):
    """The end of a greedy step in one launch: the first maximum per row (ties, rows of equal values, a NaN, rows that do
    not start on 16-byte boundaries), positions advanced by one, the winners' embedding rows copied."""
    g = torch.Generator(device="cuda").manual_seed(B + V)
    logits = torch.randn(B, V, device="cuda", generator=g).to(torch.bfloat16)
    logits[0, V // 3] = logits[0].max()                  # a tie in the first row: the lower index wins
    logits[0, V - 1] = logits[0].max()
    if B > 1:
        logits[1] = 0.5                                  # all equal: index 0
    if B > 2:
        logits[2, V // 2] = float("nan")                 # NaN counts as the maximum
        logits[2, V // 2 + 3] = float("nan")
    embed = torch.randn(V, D, device="cuda", generator=g).to(torch.bfloat16)
    tok = torch.full((B,), -1, dtype=torch.long, device="cuda")
    pos = torch.arange(B, dtype=torch.long, device="cuda") + 5
    h = torch.zeros(B, D, dtype=torch.bfloat16, device="cuda")
    ops.argmax_embed(logits, tok, pos, embed, h)
    want = logits.float().argmax(-1)
    assert torch.equal(tok, want)
    assert torch.equal(pos, torch.arange(B, device="cuda") + 6)
    assert torch.equal(h, embed[want])
    # argmax alone, on a column slice (row stride != V)
    tok2 = torch.full((B,), -1, dtype=torch.long, device="cuda")
    ops.argmax_embed(logits[:, : V - 1], tok2)
    assert torch.equal(tok2, logits[:, : V - 1].float().argmax(-1))


@pytest.mark.parametrize("B,Hq,Hkv,hd,max_len", [(1, 32, 32, 128, 64), (1, 32, 32, 128, 65), (2, 32, 8, 128, 192), (1, 16, 16, 64, 512), (2, 32, 32, 128, 1500),
                                                 (4, 32, 32, 128, 511), (3, 32, 32, 64, 384), (9, 32, 32, 128, 100), (10, 32, 32, 128, 100), (1, 3, 1, 64, 700)])
def test_decode_attention_split_plans(ops, B, Hq, Hkv, hd, max_len):
    """Clusters of two, four and eight splits, tickets and a single split, next to the context lengths and row counts where the plan
    changes, with sequences that leave splits without a key; inside a decode chain and outside of one the same bits."""
    rng = np.random.default_rng(B * 5 + max_len)
    qkv = orc.bf16_round(rng.standard_normal((B, (Hq + 2 * Hkv) * hd)).astype(np.float32))
    kc = orc.bf16_round(rng.standard_normal((B, Hkv, max_len, hd)).astype(np.float32))
    vc = orc.bf16_round(rng.standard_normal((B, Hkv, max_len, hd)).astype(np.float32))
    for first in (max_len - 1, 0, 5):
        pos = rng.integers(0, max_len, B).astype(np.int64)
        pos[0] = first
        args = (_bf(qkv), torch.from_numpy(pos).cuda(), _bf(kc), _bf(vc), Hq, Hkv, hd)
        out = ops.decode_attention(*args)
        with ops.decode_chain():
            again = ops.decode_attention(*args)
        want = orc.decode_attention(qkv[:, :Hq * hd].reshape(B, Hq, hd), kc, vc, pos, hd ** -0.5)
        got = out.float().cpu().numpy().reshape(B, Hq, hd)
        assert np.abs(got - want).max() <= 2.0 ** -7 * np.abs(want).max()
        assert torch.equal(out, again)


@pytest.mark.parametrize("B,Hq,Hkv,hd,max_len,cluster", [
    (1, 8, 8, 128, 1500, True), (1, 8, 8, 128, 2048, False), (1, 4, 4, 128, 8192, False), (1, 16, 16, 64, 4096, False), (1, 32, 8, 128, 3072, False),
    (1, 32, 32, 128, 1500, True), (1, 32, 32, 128, 16384, False), (2, 32, 32, 128, 1500, True), (4, 16, 16, 64, 4000, True), (7, 8, 8, 128, 1800, True), (8, 8, 8, 128, 2048, False),
    (2, 32, 32, 128, 600, True), (7, 16, 4, 128, 3072, False)])
def test_decode_attention_long_contexts(ops, B, Hq, Hkv, hd, max_len, cluster):
    """Few rows and a long context keep the tickets, whose splits are finer (a cluster has eight at most).  The plan shows in the scratch:
    clusters leave it untouched.  Full caches, against 64-bit arithmetic."""
    from latentq_llm_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(max_len + Hq)
    qkv = torch.randn(B, (Hq + 2 * Hkv) * hd, device="cuda", generator=g).to(torch.bfloat16)
    kc, vc = (torch.randn(B, Hkv, max_len, hd, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    pos, out = torch.full((B,), max_len - 1, device="cuda"), torch.empty(B, Hq * hd, dtype=torch.bfloat16, device="cuda")
    ws = torch.zeros(_lib.lib.lq_decode_attention_workspace_bytes(B, Hq, hd, max_len), dtype=torch.uint8, device="cuda")
    _lib.call("lq_decode_attention", qkv.data_ptr(), qkv.stride(0), kc.data_ptr(), vc.data_ptr(), pos.data_ptr(), out.data_ptr(), B, Hq, Hkv, hd, max_len, hd ** -0.5,
              ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert bool(ws.any()) != cluster
    q = qkv[:, :Hq * hd].double().view(B, Hkv, Hq // Hkv, hd)
    p = torch.softmax(q @ kc.double().transpose(-1, -2) * hd ** -0.5, -1)
    want = (p @ vc.double()).view(B, Hq * hd)
    assert float((out.double() - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max())


@pytest.mark.parametrize("B,V,D", [(2, 16384, 64), (18, 16392, 8), (18, 24584, 8), (3, 100008, 4096), (40, 98304, 264)])
def test_argmax_of_a_large_vocabulary_by_clusters(ops, B, V, D):
    """Eight CTAs per row from 16384 logits on: maxima in the first and last place of a CTA's share, ties across shares, a NaN behind the maximum."""
    logits = torch.randn(B, V, device="cuda", generator=torch.Generator(device="cuda").manual_seed(V)).to(torch.bfloat16)
    share = (V // 8 + 7) // 8 * 8
    logits[0, share - 1] = logits[0, share] = logits[0, V - 1] = 50.0
    logits[1, 7 * share] = 50.0
    if B > 2:
        logits[2, 0], logits[2, V - 1] = 50.0, float("nan")
    embed = torch.randn(V, D, device="cuda").to(torch.bfloat16)
    tok, pos, h = torch.zeros(B, dtype=torch.long, device="cuda"), torch.arange(B, device="cuda"), torch.zeros(B, D, dtype=torch.bfloat16, device="cuda")
    want = logits.float().argmax(-1)
    assert want[:2].tolist() == [share - 1, 7 * share]
    ops.argmax_embed(logits, tok, pos, embed, h)
    assert torch.equal(tok, want) and torch.equal(pos, torch.arange(B, device="cuda") + 1) and torch.equal(h, embed[want])


@pytest.mark.parametrize("B,V,cluster", [(2, 16376, False), (12, 16384, True), (13, 16384, False), (18, 24576, True), (19, 24576, False), (64, 98304, True),
                                         (65, 98304, False), (98, 131072, True), (99, 131072, False), (148, 131072, False), (149, 131072, True), (2, 16390, False)])
def test_argmax_by_clusters_where_they_are_faster(ops, kernel_of, B, V, cluster):
    """Both sides of each line of the rule, on 148 SMs; rows that are not whole vectors keep the single CTA."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the numbers of rows are those of 148 SMs")
    logits = torch.randn(B, V, device="cuda", generator=torch.Generator(device="cuda").manual_seed(V)).to(torch.bfloat16)
    tok = torch.zeros(B, dtype=torch.long, device="cuda")
    assert kernel_of(lambda: ops.argmax_embed(logits, tok)) == ("k_argmax_embed_cluster" if cluster else "k_argmax_embed")
    assert torch.equal(tok, logits.float().argmax(-1))


@pytest.mark.parametrize("M,N,K", [(1, 32000, 4096), (8, 1003, 4096), (2, 16 * 149, 4096), (3, 50, 2048), (5, 50272, 2048), (1, 7, 2048), (9, 100, 4096), (2, 100, 512)])
def test_linear_rows(ops, kernel_of, M, N, K):
    """The head of a decode step against fp32 matmul: row counts that leave a block of 16 incomplete, fewer and more blocks than SMs, all token counts' edges; the
    last two go to torch's linear.  One rounding to bf16, and fp32 sums of K products in any order."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.02).to(torch.bfloat16)
    ref = x.double() @ w.double().t()
    bound = ref.abs() * 2.0 ** -8 + (x.double().abs() @ w.double().abs().t()) * (K * 2.0 ** -24)
    out = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    for y in (ops.linear_rows(x, w), ops.linear_rows(x, w, out=out)):
        if M > 8 or K == 512:                         # (the library may round its partial sums to bf16, which the bound does not hold for)
            assert torch.equal(y, torch.nn.functional.linear(x, w))
        else:
            assert y.shape == (M, N) and bool(((y.double() - ref).abs() <= bound).all())
    ops.silu_mul(torch.zeros(1, 16, device="cuda", dtype=torch.bfloat16))
    assert torch.equal(out, y) and kernel_of(lambda: ops.linear_rows(x, w)) == ("k_linear_rows" if M <= 8 and K != 512 else "k_silu_mul")
    wt = w.t().contiguous().t()                           # strides that the kernel does not have
    assert torch.equal(ops.linear_rows(x, wt), torch.nn.functional.linear(x, wt))
    x8, w8 = x[:1].clone().requires_grad_(True), w.clone()                # gradients at every token count
    ops.linear_rows(x8, w8).sum().backward()
    assert torch.equal(x8.grad, torch.autograd.grad(torch.nn.functional.linear(x8, w8).sum(), x8)[0])
    host = torch.empty(M, N, dtype=torch.bfloat16)
    assert torch.equal(ops.linear_rows(x, w, out=host), torch.nn.functional.linear(x, w).cpu())
    if N >= K:                                            # the result over the tokens
        both = torch.cat([x.reshape(-1), torch.zeros(M * (N - K), dtype=x.dtype, device="cuda")])
        ops.linear_rows(both[:M * K].view(M, K), w, out=both.view(M, N))
        assert torch.equal(both.view(M, N), torch.nn.functional.linear(x, w))
    with pytest.raises(RuntimeError):
        ops.linear_rows(x, w.cpu())
