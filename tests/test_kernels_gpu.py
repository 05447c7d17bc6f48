"""Kernel-level parity: each hand-written CUDA kernel, driven through the C ABI, against the oracle's
primitive of the same name on the same seeded inputs.  Tolerances: bit-exact for integer/bf16-bit
work (synthetic weights, argmax, page writes of v); fp32-accumulation noise (1e-4 of the output scale)
for reductions whose summation order differs; one bf16 ulp where the kernel's output is bf16."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests import _gpu_util as G
from tests._gpu_util import (DEV, check, dev_bf16, dev_f32, dev_i32, host, lib, ptr, rand_bf16, sync)

pytestmark = pytest.mark.gpu
BF16_ULP = 2.0 ** -8  # relative spacing of bf16


def test_synth_bits_match_oracle():
    shape = O.ModelShape(512, 128, 3, 8, 2, 16, 352, 256)
    for kind, layer in [(O.WQ, 1), (O.ATTN_NORM, 0), (O.WDOWN, 2), (O.EMBED, 0)]:
        ref = O.synth_tensor(shape, 99, kind, layer).reshape(-1)
        amp, off = C.c_float(), C.c_float()
        cfg = shape.c()
        O.lib().orc_synth_params(C.byref(cfg), kind, C.byref(amp), C.byref(off))
        out = G.empty(ref.size, dtype=torch.bfloat16, device=DEV)
        check(lib().dis_k_synth_bf16(ptr(out), ref.size, 99, kind, layer if kind in O.PER_LAYER else 0, amp.value,
                                     off.value, None))
        sync()
        assert np.array_equal(host(out), ref)


@pytest.mark.parametrize("T,H", [(1, 128), (7, 512), (33, 4096), (4, 8192)])
def test_add_rmsnorm(T, H):
    rng = np.random.default_rng(T * 1000 + H)
    x = rng.standard_normal((T, H)).astype(np.float32)
    parts = rng.standard_normal((3, T, H)).astype(np.float32)
    gain = O.bf16_round(1 + 0.1 * rng.standard_normal(H).astype(np.float32))
    dx, dp, dg = dev_f32(x), dev_f32(parts), dev_f32(gain)
    xn = G.empty((T, H), dtype=torch.bfloat16, device=DEV)
    check(lib().dis_k_add_rmsnorm(ptr(dx), None, None, ptr(dp), 3, T * H, ptr(dg), ptr(xn), None, T, H, 1e-5, None))
    sync()
    xs = x + parts.sum(0)
    assert np.abs(host(dx) - xs).max() <= 1e-5 * np.abs(xs).max()
    ref = O.rmsnorm(xs, gain, 1e-5, round_out=True)
    assert np.abs(host(xn) - ref).max() <= BF16_ULP * np.abs(ref).max() * 1.01


def test_add_rmsnorm_embedding_and_rowmap():
    rng = np.random.default_rng(5)
    V, H, T = 300, 256, 9
    emb = rand_bf16(rng, (V, H), 0.02)
    toks = rng.integers(0, V, T).astype(np.uint32)
    gain = np.ones(H, np.float32)
    dx = G.zeros((T, H), dtype=torch.float32, device=DEV)
    xn = G.empty((T, H), dtype=torch.bfloat16, device=DEV)
    dt = torch.from_numpy(toks.astype(np.int64)).to(DEV).to(torch.int32)
    check(lib().dis_k_add_rmsnorm(ptr(dx), ptr(dt), ptr(dev_bf16(emb)), None, 0, 0, ptr(dev_f32(gain)), ptr(xn), None,
                                  T, H, 1e-5, None))
    sync()
    assert np.array_equal(host(dx), emb[toks])
    ref = O.rmsnorm(emb[toks], gain, 1e-5, round_out=True)
    assert np.abs(host(xn) - ref).max() <= BF16_ULP * np.abs(ref).max() * 1.01
    # row_map: compact rows, x untouched
    rows = np.array([8, 2, 5], np.int32)
    xn2 = G.empty((3, H), dtype=torch.bfloat16, device=DEV)
    before = host(dx).copy()
    check(lib().dis_k_add_rmsnorm(ptr(dx), None, None, None, 0, 0, ptr(dev_f32(gain)), ptr(xn2), ptr(dev_i32(rows)), 3,
                                  H, 1e-5, None))
    sync()
    assert np.array_equal(host(dx), before)
    assert np.array_equal(host(xn2), host(xn)[rows])


GEMM_SHAPES = [(32, 256, 128), (5, 200, 352), (64, 384, 512), (17, 1000, 1024), (128, 512, 256), (300, 640, 192),
               (32, 4096, 4096),
               # prefill-sized: the persistent, TMEM-double-buffered kernel (>= 2 tiles per SM), ragged T / N / K too
               (1024, 9600, 576), (1000, 9500, 320), (4096, 2500, 128)]


@pytest.mark.parametrize("T,N,K", GEMM_SHAPES)
def test_gemm_tcgen05(T, N, K):
    rng = np.random.default_rng(T + N + K)
    X, W = rand_bf16(rng, (T, K)), rand_bf16(rng, (N, K), 0.05)
    ref = O.linear(X, W)
    dX, dW = dev_bf16(X), dev_bf16(W)
    for split in sorted({1, lib().dis_k_gemm_pick_split(T, N, K)}):
        out = torch.full((split, T, N), float("nan"), dtype=torch.float32, device=DEV)
        check(lib().dis_k_gemm(ptr(dX), ptr(dW), ptr(out), T, N, K, split, None))
        sync()
        got = host(out).sum(0)
        assert np.isfinite(got).all()
        assert np.abs(got - ref).max() <= 1e-4 * np.abs(ref).max() + 1e-6, (split, np.abs(got - ref).max())


@pytest.mark.parametrize("T,N,K,silu", [(8192, 6144, 4096, False), (4096, 4096, 14336, False), (8192, 14336, 4096, True),
                                        (32, 28672 // 2, 4096, True), (512, 6144, 4096, False)])
def test_gemm_full_size_against_torch(T, N, K, silu):
    """BASELINE-sized projections (Llama-3-8B qkv / down / gate-up at an 8192-token prefill chunk, a decode batch, a
    single 512-token request): too large for the CPU oracle in seconds, so the reference is a plain torch fp32 matmul
    of the same bf16 operands on the device (tolerance: fp32 accumulation order only, 2e-4 of max|y|; the SiLU-gate
    output is bf16, one ulp)."""
    g = torch.Generator(device=DEV); g.manual_seed(T + N + K)
    X = (torch.randn((T, K), device=DEV, generator=g)).to(torch.bfloat16)
    W = (torch.randn(((2 if silu else 1) * N, K), device=DEV, generator=g) * 0.02).to(torch.bfloat16)
    if silu:
        act = G.empty((T, N), dtype=torch.bfloat16, device=DEV)
        check(lib().dis_k_gemm_silu(ptr(X), ptr(W), ptr(act), T, N, K, None))
        sync()
        gate, up = X.float() @ W[:N].float().T, X.float() @ W[N:].float().T
        ref = torch.nn.functional.silu(gate) * up
        err = (act.float() - ref).abs().max().item()
        assert err <= BF16_ULP * ref.abs().max().item() * 1.05 + 1e-6, err
    else:
        out = torch.full((1, T, N), float("nan"), dtype=torch.float32, device=DEV)
        check(lib().dis_k_gemm(ptr(X), ptr(W), ptr(out), T, N, K, 1, None))
        sync()
        ref = X.float() @ W.float().T
        assert torch.isfinite(out).all()
        err = (out[0] - ref).abs().max().item()
        assert err <= 2e-4 * ref.abs().max().item(), err


# Sizes at the edges of the pair kernel's tiles (256 tokens x 256, 224 or 192 columns, a K block of 64), rows that are and are not pieces
# of 32 bytes, K slices, several rounds of its 74 pairs (the last three, whose tile widths differ).
@pytest.mark.parametrize("T,N,K,split", [(1030, 131, 72, 1), (1281, 256, 64, 1), (1024, 1000, 200, 2), (1300, 264, 136, 3), (129, 4096, 256, 4),
                                         (1100, 4100, 64, 1), (1300, 8192, 128, 2), (3000, 2504, 64, 1), (2600, 5000, 72, 1)])
def test_gemm_pairs(T, N, K, split):
    """Pairs of CTAs against float64 of the same bf16 operands: the sums are fp32, at most K terms of |x w|."""
    g = torch.Generator(device=DEV); g.manual_seed(T + N + K)
    X, W = (torch.randn(s, device=DEV, generator=g).to(torch.bfloat16) for s in ((T, K), (N, K)))
    out = G.empty((split, T, N), dtype=torch.float32, device=DEV)
    check(lib().dis_k_gemm(ptr(X), ptr(W), ptr(out), T, N, K, split, None))
    sync()
    ref = X.double() @ W.double().T
    bound = K * 2.0 ** -24 * (X.double().abs() @ W.double().abs().T).max().item()
    assert (out.double().sum(0) - ref).abs().max().item() <= bound


@pytest.mark.parametrize("T,I,K", [(129, 40, 72), (256, 128, 64), (257, 131, 136), (700, 1000, 64), (1000, 4104, 64), (1300, 5632, 72), (3000, 2504, 64)])
def test_gemm_silu_pairs(T, I, K):
    """The gate-up product of the same kernel: silu(gate) * up against float64, one bf16 rounding plus the fast exponential and division."""
    g = torch.Generator(device=DEV); g.manual_seed(T + I + K)
    X, W = torch.randn((T, K), device=DEV, generator=g).to(torch.bfloat16), (torch.randn((2 * I, K), device=DEV, generator=g) * K ** -0.5).to(torch.bfloat16)
    act = G.empty((T, I), dtype=torch.bfloat16, device=DEV)
    check(lib().dis_k_gemm_silu(ptr(X), ptr(W), ptr(act), T, I, K, None))
    sync()
    gate, up = X.double() @ W[:I].double().T, X.double() @ W[I:].double().T
    ref = gate * torch.sigmoid(gate) * up
    # rounding to bf16's 8 significant bits is off by at most 2^-8 of the value; the fast functions add a few 1e-6 of it, the sums 1e-6 K
    assert ((act.double() - ref).abs() <= BF16_ULP * ref.abs() * 1.01 + 1e-5).all()


@pytest.mark.parametrize("T,H,I", [(5, 512, 1024), (32, 2048, 5632), (200, 1024, 4096), (1100, 1024, 1024)])
def test_calls_in_a_row_take_what_the_one_before_wrote(T, H, I):
    """A kernel of the C ABI starts while the one in front of it still runs: activations and even a weight that the call before wrote
    have to be seen whole, in plain stream order, on a stream of its own and from a captured graph."""
    g = torch.Generator(device=DEV); g.manual_seed(T + H + I)
    W = (torch.randn((2 * I, H), device=DEV, generator=g) * H ** -0.5).to(torch.bfloat16)
    W2 = (torch.randn((H, I), device=DEV, generator=g) * I ** -0.5).to(torch.bfloat16)
    x0, gain = torch.randn((T, H), device=DEV, generator=g), torch.ones(H, device=DEV)
    S = lib().dis_k_gemm_pick_split(T, H, I)
    St = lib().dis_k_gemm_pick_split(T, T, H)
    act, part = torch.empty((T, I), dtype=torch.bfloat16, device=DEV), torch.empty((S, T, H), device=DEV)
    xn, x, gram = torch.empty((T, H), dtype=torch.bfloat16, device=DEV), torch.empty_like(x0), torch.empty((St, T, T), device=DEV)

    def chain(after=lambda: None):
        s = torch.cuda.current_stream().cuda_stream
        x.copy_(x0)
        part.zero_()
        check(lib().dis_k_add_rmsnorm(ptr(x), None, None, ptr(part), S, T * H, ptr(gain), ptr(xn), None, T, H, 1e-5, s))
        for _ in range(3):
            after()
            check(lib().dis_k_gemm_silu(ptr(xn), ptr(W), ptr(act), T, I, H, s))
            after()
            check(lib().dis_k_gemm(ptr(act), ptr(W2), ptr(part), T, H, I, S, s))
            after()
            check(lib().dis_k_add_rmsnorm(ptr(x), None, None, ptr(part), S, T * H, ptr(gain), ptr(xn), None, T, H, 1e-5, s))
            after()
            check(lib().dis_k_gemm(ptr(xn), ptr(xn), ptr(gram), T, T, H, St, s))  # xn is the weight as well
        return [t.clone() for t in (x, xn, act, gram)]

    want = chain(sync)
    sync()
    side = torch.cuda.Stream()
    for k in range(6):
        for t in (act, part, xn, gram):
            t.fill_(float("nan"))
        sync()
        with torch.cuda.stream(side if k % 2 else torch.cuda.current_stream()):
            got = chain()
        sync()
        assert all(torch.equal(a, b) for a, b in zip(got, want)), k
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain()
    for t in (act, part, xn, gram):
        t.fill_(float("nan"))
    graph.replay()
    sync()
    assert all(torch.equal(a, b) for a, b in zip(out, want))


def test_gemm_rejects_empty_split():
    X, W = dev_bf16(np.zeros((8, 576), np.float32)), dev_bf16(np.zeros((128, 576), np.float32))
    out = G.zeros((4, 8, 128), dtype=torch.float32, device=DEV)
    assert lib().dis_k_gemm(ptr(X), ptr(W), ptr(out), 8, 128, 576, 4, None) != 0  # 9 k-blocks / 4 -> empty slice


@pytest.mark.parametrize("T,I,K", [(32, 256, 128), (9, 200, 320), (64, 512, 256), (128, 384, 128), (32, 14336, 4096),
                                   (1024, 4800, 192), (1000, 4792, 320), (2048, 2432, 64)])  # persistent dual kernel
def test_gemm_silu(T, I, K):
    rng = np.random.default_rng(T + I + K)
    X, Wgu = rand_bf16(rng, (T, K)), rand_bf16(rng, (2 * I, K), 0.05)
    ref = O.silu_mul(O.linear(X, Wgu[:I]), O.linear(X, Wgu[I:]), round_out=False)
    act = G.empty((T, I), dtype=torch.bfloat16, device=DEV)
    check(lib().dis_k_gemm_silu(ptr(dev_bf16(X)), ptr(dev_bf16(Wgu)), ptr(act), T, I, K, None))
    sync()
    assert np.abs(host(act) - ref).max() <= BF16_ULP * np.abs(ref).max() * 1.05 + 1e-6


@pytest.mark.parametrize("T,N,K", [(1, 256, 128), (2, 201, 352), (4, 512, 4096), (7, 64, 256),
                                   # several row groups per persistent CTA, ragged N and K tails
                                   (1, 4096, 4096), (1, 3001, 6152), (2, 1500, 14336), (3, 2501, 520)])
def test_gemv(T, N, K):
    rng = np.random.default_rng(T + N + K)
    X, W = rand_bf16(rng, (T, K)), rand_bf16(rng, (N, K), 0.05)
    ref = O.linear(X, W)
    out = G.empty((T, N), dtype=torch.float32, device=DEV)
    check(lib().dis_k_gemv(ptr(dev_bf16(X)), ptr(dev_bf16(W)), ptr(out), T, N, K, None))
    sync()
    assert np.abs(host(out) - ref).max() <= 1e-4 * np.abs(ref).max() + 1e-6
    Wgu = rand_bf16(rng, (2 * N, K), 0.05)
    refs = O.silu_mul(O.linear(X, Wgu[:N]), O.linear(X, Wgu[N:]))
    act = G.empty((T, N), dtype=torch.bfloat16, device=DEV)
    check(lib().dis_k_gemv_silu(ptr(dev_bf16(X)), ptr(dev_bf16(Wgu)), ptr(act), T, N, K, None))
    sync()
    assert np.abs(host(act) - refs).max() <= BF16_ULP * np.abs(refs).max() * 1.05 + 1e-6


def _paged_setup(rng, n_seq, ctx_lens, n_kv, d, page_size, n_pages):
    max_pages = (max(ctx_lens) + page_size - 1) // page_size + 1
    perm = rng.permutation(n_pages)
    pt = np.zeros((n_seq, max_pages), np.int32)
    k = 0
    for s in range(n_seq):
        for p in range((ctx_lens[s] + page_size - 1) // page_size):
            pt[s, p] = perm[k]; k += 1
    return pt, max_pages


@pytest.mark.parametrize("d,nh,nkv", [(128, 8, 2), (64, 8, 2), (128, 4, 4), (64, 4, 2), (128, 8, 1), (64, 16, 2)])
def test_rope_kv_write_and_attention(d, nh, nkv):
    rng = np.random.default_rng(d + nh + nkv)
    page_size, n_pages, max_ctx = 16, 64, 256
    ctx_lens = [1, 37, 130, 200]
    n_seq = len(ctx_lens)
    pt, max_pages = _paged_setup(rng, n_seq, ctx_lens, nkv, d, page_size, n_pages)
    cs, sn = O.rope_table(max_ctx, d, 500000.0)
    nq, nk = nh * d, nkv * d
    pool = G.zeros((n_pages, 2, nkv, page_size, d), dtype=torch.bfloat16, device=DEV)
    dpt = dev_i32(pt)
    K_hist = [np.zeros((c, nk), np.float32) for c in ctx_lens]
    V_hist = [np.zeros((c, nk), np.float32) for c in ctx_lens]
    q_last = np.zeros((n_seq, nq), np.float32)
    # write every position of every sequence through the kernel, a ragged batch at a time, with 2 split-K slices
    toks = [(s, p) for s in range(n_seq) for p in range(ctx_lens[s])]
    for b0 in range(0, len(toks), 50):
        chunk = toks[b0:b0 + 50]
        T = len(chunk)
        full = (rng.standard_normal((T, nq + 2 * nk))).astype(np.float32)
        part = rng.standard_normal((2, T, nq + 2 * nk)).astype(np.float32)
        part[1] = full - part[0]
        summed = part[0] + part[1]
        pos = np.array([p for _, p in chunk], np.int32)
        row = np.array([s for s, _ in chunk], np.int32)
        dq = G.empty((T, nq), dtype=torch.bfloat16, device=DEV)
        check(lib().dis_k_rope_kv_write(ptr(dev_f32(part)), 2, T * (nq + 2 * nk), ptr(dq), ptr(pool), ptr(dpt), max_pages,
                                        ptr(dev_i32(row)), ptr(dev_i32(pos)), ptr(dev_f32(cs)), ptr(dev_f32(sn)), T, nh,
                                        nkv, d, page_size, None))
        sync()
        q_ref = O.bf16_round(O.rope(summed[:, :nq], pos, nh, d, cs, sn))
        k_ref = O.bf16_round(O.rope(summed[:, nq:nq + nk], pos, nkv, d, cs, sn))
        v_ref = O.bf16_round(summed[:, nq + nk:])
        got_q = host(dq)
        assert np.abs(got_q - q_ref).max() <= BF16_ULP * np.abs(q_ref).max() * 1.01
        for i, (s, p) in enumerate(chunk):
            K_hist[s][p], V_hist[s][p] = k_ref[i], v_ref[i]
            if p == ctx_lens[s] - 1:
                q_last[s] = got_q[i]
    hp = host(pool)
    for s in range(n_seq):
        for p in range(ctx_lens[s]):
            page, slot = pt[s, p // page_size], p % page_size
            got_k = hp[page, 0, :, slot, :].reshape(-1)
            got_v = hp[page, 1, :, slot, :].reshape(-1)
            assert np.abs(got_k - K_hist[s][p]).max() <= BF16_ULP * max(np.abs(K_hist[s][p]).max(), 1e-3) * 1.01
            assert np.array_equal(got_v, V_hist[s][p])
            K_hist[s][p], V_hist[s][p] = got_k, got_v  # attention below is checked on what is in the pages
    # attention of the last token of every sequence, 1 and several splits
    dq = dev_bf16(q_last)
    ref = np.stack([O.attention_one(q_last[s], K_hist[s], V_hist[s], nh, nkv, d) for s in range(n_seq)])
    for splits in (1, 3, 8):
        out = G.empty((n_seq, nq), dtype=torch.bfloat16, device=DEV)
        n_scr = lib().dis_k_attn_scratch_elems(n_seq, nh, d, splits)
        scr = G.empty(max(n_scr, 1), dtype=torch.float32, device=DEV)
        check(lib().dis_k_attn_paged(ptr(dq), ptr(pool), n_pages, ptr(dpt), max_pages, ptr(dev_i32(np.arange(n_seq))),
                                     ptr(dev_i32(ctx_lens)), ptr(out), ptr(scr), splits, n_seq, nh, nkv, d, page_size, None))
        sync()
        got = host(out)
        # P is rounded to bf16 for the P.V tensor-core MMA: allow two bf16 ulps of the output scale
        assert np.abs(got - ref).max() <= 2 * BF16_ULP * np.abs(ref).max() + 1e-5, (splits, np.abs(got - ref).max())


def test_attention_full_size_against_torch():
    """Llama-3-8B geometry (32 query heads, 8 kv heads, d = 128, 64-token pages), batch 32 with contexts from 1 to 8000
    tokens on shuffled pages: decode attention with 1 and 4 history splits against softmax(q K^T / sqrt(d)) V in fp32
    torch on the same bf16 K/V (tolerance: P is rounded to bf16 for the P.V MMA -- two bf16 ulps of the output scale)."""
    g = torch.Generator(device=DEV); g.manual_seed(9)
    d, nh, nkv, ps, B = 128, 32, 8, 64, 32
    rng = np.random.default_rng(9)
    ctx = np.concatenate([[1, 63, 64, 65, 8000], rng.integers(100, 4000, B - 5)]).astype(np.int32)
    pages_per = [(int(c) + ps - 1) // ps for c in ctx]
    n_pages, max_pages = sum(pages_per) + 3, max(pages_per)
    perm = rng.permutation(n_pages)
    pt = np.zeros((B, max_pages), np.int32)
    k0 = 0
    for b in range(B):
        pt[b, :pages_per[b]] = perm[k0:k0 + pages_per[b]]; k0 += pages_per[b]
    pool = torch.randn((n_pages, 2, nkv, ps, d), device=DEV, generator=g).to(torch.bfloat16)
    q = torch.randn((B, nh * d), device=DEV, generator=g).to(torch.bfloat16)
    dpt, dctx, drow = dev_i32(pt), dev_i32(ctx), dev_i32(np.arange(B))
    ref = G.empty((B, nh, d), dtype=torch.float32, device=DEV)
    for b in range(B):
        pages = torch.as_tensor(pt[b, :pages_per[b]].astype(np.int64), device=DEV)
        kv = pool[pages].float()                                   # [pages, 2, nkv, ps, d]
        K = kv[:, 0].permute(1, 0, 2, 3).reshape(nkv, -1, d)[:, :int(ctx[b])]
        V = kv[:, 1].permute(1, 0, 2, 3).reshape(nkv, -1, d)[:, :int(ctx[b])]
        qb = q[b].float().reshape(nkv, nh // nkv, d)
        p = torch.softmax(qb @ K.transpose(1, 2) / d ** 0.5, dim=-1)
        ref[b] = (p @ V).reshape(nh, d)
    for splits in (1, 4):
        out = G.empty((B, nh * d), dtype=torch.bfloat16, device=DEV)
        scr = G.empty(max(lib().dis_k_attn_scratch_elems(B, nh, d, splits), 1), dtype=torch.float32, device=DEV)
        check(lib().dis_k_attn_paged(ptr(q), ptr(pool), n_pages, ptr(dpt), max_pages, ptr(drow), ptr(dctx), ptr(out), ptr(scr),
                                     splits, B, nh, nkv, d, ps, None))
        sync()
        err = (out.float().reshape(B, nh, d) - ref).abs().max().item()
        assert err <= 2 * BF16_ULP * ref.abs().max().item() + 1e-5, (splits, err)


@pytest.mark.parametrize("nh,nkv,d,page_size", [(8, 2, 128, 64), (8, 1, 128, 16), (16, 2, 64, 128), (4, 2, 64, 8), (2, 2, 128, 64)])
@pytest.mark.parametrize("T,n_splits,pattern", [(8, 1, "one-long"), (13, 1, "ragged"), (2, 1, "one-long"), (3, 1, "equal"), (5, 2, "ragged"), (3, 3, "one-long"),
                                                (2, 4, "one-long"), (1, 5, "equal"), (3, 8, "ragged"), (2, 9, "ragged"), (9, 1, "tiles"),
                                                (9, 1, "holes"), (4, 2, "holes"), (2, 9, "holes"), (230, 1, "short")])
def test_attention_of_ragged_histories(nh, nkv, d, page_size, T, n_splits, pattern):
    """Histories that a cluster of CTAs shares (the page table's width says that they may be long): one long beside short ones, tile edges, batches
    that leave a cluster part empty; slices; more CTAs than fit at once, for heads of 64 as many as take eight computing warps each.  Against
    float64 (weights and outputs in bf16: a relative error of 2^-9 each, 8e-3 of the 2-norm is four times that)."""
    rng = np.random.default_rng(T * 100 + n_splits + d)
    ctx = {"one-long": np.where(np.arange(T) == T // 2, 2500, rng.integers(1, 130, T)), "ragged": rng.integers(1, 1800, T), "equal": np.full(T, 1100),
           "tiles": np.array([1, 63, 64, 65, 127, 128, 129, 1024, 1025])[:T], "short": np.random.default_rng(T).integers(1, 300, T),
           "holes": np.array([0, 700, 0, 2200, 0, 0, 65, 1, 0])[:T]}[pattern].astype(np.int32)
    need = [-(-int(c) // page_size) for c in ctx]
    width = max(max(need), 2100 // page_size + 1)
    table = np.zeros((T, width), np.int32)
    order = rng.permutation(sum(need))
    for t, at in enumerate(np.cumsum([0] + need[:-1])):
        table[t, :need[t]] = order[at:at + need[t]]
    g = torch.Generator(device=DEV); g.manual_seed(T + d)
    pool = torch.randn((sum(need), 2, nkv, page_size, d), device=DEV, generator=g).to(torch.bfloat16)
    q = (torch.randn((T, nh * d), device=DEV, generator=g) * 1.5).to(torch.bfloat16)
    rows, dctx, dtab = dev_i32(np.arange(T, dtype=np.int32)), dev_i32(ctx), dev_i32(table)
    scratch = torch.empty(max(1, lib().dis_k_attn_scratch_elems(T, nh, d, n_splits)), device=DEV)
    outs = []
    for _ in range(3):
        out = torch.full((T, nh * d), float("nan"), dtype=torch.bfloat16, device=DEV)
        check(lib().dis_k_attn_paged(ptr(q), ptr(pool), pool.shape[0], ptr(dtab), width, ptr(rows), ptr(dctx), ptr(out), ptr(scratch), n_splits, T, nh, nkv, d,
                                     page_size, None))
        outs.append(out)
    sync()
    some = torch.from_numpy(ctx > 0).to(DEV)
    assert torch.equal(outs[0][some], outs[1][some]) and torch.equal(outs[0][some], outs[2][some])  # the same bits every time
    for t in range(T):
        if ctx[t] == 0:  # no key: no number, and no neighbour's
            assert bool(torch.isnan(outs[0][t]).all())
            continue
        kv = pool[torch.from_numpy(table[t, :need[t]].astype(np.int64)).to(DEV)].double()
        k, v = (kv[:, c].permute(1, 0, 2, 3).reshape(nkv, -1, d)[:, :int(ctx[t])].repeat_interleave(nh // nkv, 0) for c in (0, 1))
        w = torch.softmax((k @ q[t].double().view(nh, d, 1))[..., 0] * d ** -0.5, -1)
        ref = (w[:, None] @ v)[:, 0].flatten()
        err = (outs[0][t].double() - ref).norm() / ref.norm()
        assert err <= 8e-3, (t, int(ctx[t]), float(err))


@pytest.mark.parametrize("nh,nkv,d", [(32, 8, 128), (32, 4, 64)])
@pytest.mark.parametrize("T,n_splits,most", [(2, 4, 900), (1, 8, 1500), (5, 3, 700), (4, 2, 130), (24, 1, 600), (40, 1, 3000), (130, 1, 300)])
def test_attention_is_as_close_as_its_output_s_type(nh, nkv, d, T, n_splits, most):
    """Decode attention's error against 64 bits is that of rounding the result to bf16 (weights go into the product as two halves: in one, the
    error is 10 % larger): slices, whole histories, histories that a cluster shares, more CTAs than fit at once.  The same bits from a graph, where
    a small call's slices are joined by a kernel of its own and not in a cluster."""
    rng = np.random.default_rng(T + d)
    page_size = 64
    ctx = np.exp(rng.uniform(np.log(most / 12), np.log(most), T)).astype(np.int32)
    ctx[T // 2] = most
    need = [-(-int(c) // page_size) for c in ctx]
    table = np.zeros((T, max(need)), np.int32)
    order = rng.permutation(sum(need))
    for t, at in enumerate(np.cumsum([0] + need[:-1])):
        table[t, :need[t]] = order[at:at + need[t]]
    g = torch.Generator(device=DEV); g.manual_seed(T + d)
    pool = torch.randn((sum(need), 2, nkv, page_size, d), device=DEV, generator=g).to(torch.bfloat16)
    q = (torch.randn((T, nh * d), device=DEV, generator=g) * 1.5).to(torch.bfloat16)
    out = torch.empty_like(q)
    scratch = torch.empty(max(1, lib().dis_k_attn_scratch_elems(T, nh, d, n_splits)), device=DEV)
    rows, dctx, dtab = dev_i32(np.arange(T, dtype=np.int32)), dev_i32(ctx), dev_i32(table)

    def run():
        check(lib().dis_k_attn_paged(ptr(q), ptr(pool), pool.shape[0], ptr(dtab), table.shape[1], ptr(rows), ptr(dctx), ptr(out), ptr(scratch), n_splits, T, nh, nkv, d, page_size,
                                     torch.cuda.current_stream().cuda_stream))

    run()
    eager = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    out.fill_(float("nan"))
    graph.replay()
    sync()
    assert torch.equal(eager, out)
    ref = torch.empty(q.shape, dtype=torch.float64, device=DEV)
    for t in range(T):
        kv = pool[torch.from_numpy(table[t, :need[t]].astype(np.int64)).to(DEV)].double()
        k, v = (kv[:, c].permute(1, 0, 2, 3).reshape(nkv, -1, d)[:, :int(ctx[t])].repeat_interleave(nh // nkv, 0) for c in (0, 1))
        w = torch.softmax((k @ q[t].double().view(nh, d, 1))[..., 0] * d ** -0.5, -1)
        ref[t] = (w[:, None] @ v)[:, 0].flatten()
    err, rounding = (out.double() - ref).norm(), (ref.to(torch.bfloat16).double() - ref).norm()
    assert err <= 1.03 * rounding, float(err / rounding)


def test_attention_long_context_tiles():
    rng = np.random.default_rng(3)
    d, nh, nkv, page_size = 128, 4, 1, 64
    ctx = 1500  # several 256-token tiles per split
    n_pages = 32
    pt, max_pages = _paged_setup(rng, 1, [ctx], nkv, d, page_size, n_pages)
    K = rand_bf16(rng, (ctx, d), 1.0)
    V = rand_bf16(rng, (ctx, d), 1.0)
    pool = np.zeros((n_pages, 2, nkv, page_size, d), np.float32)
    for p in range(ctx):
        pool[pt[0, p // page_size], 0, 0, p % page_size] = K[p]
        pool[pt[0, p // page_size], 1, 0, p % page_size] = V[p]
    q = rand_bf16(rng, (1, nh * d), 1.0)
    ref = O.attention_one(q[0], K, V, nh, nkv, d)
    dpool = dev_bf16(pool)
    for splits in (1, 2, 5):
        out = G.empty((1, nh * d), dtype=torch.bfloat16, device=DEV)
        scr = G.empty(max(lib().dis_k_attn_scratch_elems(1, nh, d, splits), 1), dtype=torch.float32, device=DEV)
        check(lib().dis_k_attn_paged(ptr(dev_bf16(q)), ptr(dpool), n_pages, ptr(dev_i32(pt)), max_pages, ptr(dev_i32([0])),
                                     ptr(dev_i32([ctx])), ptr(out), ptr(scr), splits, 1, nh, nkv, d, page_size, None))
        sync()
        assert np.abs(host(out)[0] - ref).max() <= 2 * BF16_ULP * np.abs(ref).max() + 1e-5


@pytest.mark.parametrize("d,nh,nkv,page_size", [(128, 8, 2, 64), (64, 8, 2, 16), (128, 8, 1, 32), (64, 2, 2, 64), (128, 4, 1, 16),
                                                 (128, 16, 2, 32)])
@pytest.mark.parametrize("short_blocks", [False, True], ids=["full-blocks", "short-blocks"])
def test_attention_prefill_blocks(d, nh, nkv, page_size, short_blocks):
    """Causal attention of query blocks over the paged cache vs the oracle, ragged sequences.  Blocks hold up to
    dis_k_attn_prefill_block_tokens tokens: 32 / 16 on the tcgen05 kernel (head_dim 128 with 4 / 8 query heads per kv
    head), 16 on the mma.sync kernel; short-blocks cuts them at 5 tokens (mostly padding rows, as the decode rows of a
    mixed step are)."""
    BT = lib().dis_k_attn_prefill_block_tokens(nh, nkv, d)
    assert BT == (128 // (nh // nkv) if d == 128 and nh // nkv in (4, 8) else 16)
    if short_blocks:
        BT = 5
    rng = np.random.default_rng(d + nh + nkv + page_size)
    seq_lens = [1, 15, 16, 17, 70, 200]
    n_pages = 32
    pt, max_pages = _paged_setup(rng, len(seq_lens), seq_lens, nkv, d, page_size, n_pages)
    pool = np.zeros((n_pages, 2, nkv, page_size, d), np.float32)
    K = [rand_bf16(rng, (n, nkv * d)) for n in seq_lens]
    V = [rand_bf16(rng, (n, nkv * d)) for n in seq_lens]
    Q = [rand_bf16(rng, (n, nh * d)) for n in seq_lens]
    for s, n in enumerate(seq_lens):
        for p in range(n):
            pool[pt[s, p // page_size], 0, :, p % page_size] = K[s][p].reshape(nkv, d)
            pool[pt[s, p // page_size], 1, :, p % page_size] = V[s][p].reshape(nkv, d)
    # the second half of the longest sequence only: blocks need not start at position 0 (chunked prefill)
    starts = [0, 0, 0, 0, 0, 96]
    q_flat, tok0, qlen, pos0, ptrow, ref = [], [], [], [], [], []
    t = 0
    for s, n in enumerate(seq_lens):
        for p0 in range(starts[s], n, BT):
            ln = min(BT, n - p0)
            tok0.append(t); qlen.append(ln); pos0.append(p0); ptrow.append(s)
            for i in range(ln):
                q_flat.append(Q[s][p0 + i])
                ref.append(O.attention_one(Q[s][p0 + i], K[s][:p0 + i + 1], V[s][:p0 + i + 1], nh, nkv, d))
            t += ln
    q_flat, ref = np.stack(q_flat), np.stack(ref)
    out = G.empty((t, nh * d), dtype=torch.bfloat16, device=DEV)
    check(lib().dis_k_attn_prefill(ptr(dev_bf16(q_flat)), ptr(dev_bf16(pool)), n_pages, ptr(dev_i32(pt)), max_pages,
                                   ptr(dev_i32(tok0)), ptr(dev_i32(qlen)), ptr(dev_i32(pos0)), ptr(dev_i32(ptrow)), ptr(out),
                                   len(tok0), nh, nkv, d, page_size, None))
    sync()
    got = host(out)
    assert np.isfinite(got).all()
    assert np.abs(got - ref).max() <= 2 * BF16_ULP * np.abs(ref).max() + 1e-5, np.abs(got - ref).max()


@pytest.mark.parametrize("T,N,ok", [(1024, 9472, True), (600, 12672, True), (1024, 9344, False), (500, 18944, False), (32, 256, False)])
def test_gemm_slice_count_of_zero(T, N, ok):
    """Zero slices: the plain product where 128 x 256 tiles fill the GPU twice from 512 tokens on, an error elsewhere, as ever."""
    g = torch.Generator(device=DEV); g.manual_seed(T)
    X, W = (torch.randn(s, device=DEV, generator=g).to(torch.bfloat16) for s in ((T, 64), (N, 64)))
    a, b = (G.zeros((T, N)) for _ in range(2))
    rc = lib().dis_k_gemm(ptr(X), ptr(W), ptr(a), T, N, 64, 0, None)
    sync()
    assert (rc == 0) == ok
    if ok:
        check(lib().dis_k_gemm(ptr(X), ptr(W), ptr(b), T, N, 64, 1, None))
        sync()
        assert torch.equal(a, b)
    else:
        assert not a.any()


@pytest.mark.parametrize("nh,nkv,d,BT,page_size", [(32, 8, 128, 32, 64), (64, 8, 128, 16, 16), (32, 4, 64, 16, 8), (32, 8, 64, 32, 128), (16, 4, 128, 32, 32)])
@pytest.mark.parametrize("kind", ["short", "long", "odd"])
def test_attention_prefill_of_many_blocks(nh, nkv, d, BT, page_size, kind):
    """Passes with more blocks than SMs, where a CTA takes pairs of blocks: many prompts of one to three blocks (pairs that are not of
    one sequence), few long ones beside a portion far behind its cache, and blocks in odd lengths with empty ones between.
    Eager twice and from a captured graph: the same bits.  Against float64 as in the tests of single blocks."""
    g = torch.Generator(device=DEV); g.manual_seed(nh + d + page_size)
    rng = np.random.default_rng(nh + d)
    per_head = (3 if d == 128 else 6) * 148 // 2 // nkv + 1  # blocks from which pairs are taken
    lens, past = [], []
    while sum(-(-n // BT) for n in lens) < per_head + 3:
        lens.append({"short": int(rng.integers(1, 3 * BT)), "long": int(rng.integers(17 * BT, 30 * BT)), "odd": int(rng.integers(1, 200))}[kind])
        past.append(1500 if kind == "long" and len(lens) == 2 else int(rng.integers(0, 130)) if kind == "odd" else 0)
    total = [a + b for a, b in zip(past, lens)]
    per = [-(-n // page_size) for n in total]
    perm = rng.permutation(sum(per)).astype(np.int32)
    pt = np.zeros((len(lens), max(per)), np.int32)
    for s, at in enumerate(np.cumsum([0] + per[:-1])):
        pt[s, :per[s]] = perm[at:at + per[s]]
    pool = torch.randn((sum(per), 2, nkv, page_size, d), device=DEV, generator=g)
    for s, p in enumerate(per):  # keys grow with their position: the reference has to be raised
        pool[torch.as_tensor(pt[s, :p].astype(np.int64), device=DEV), 0] *= 0.2 + torch.arange(p * page_size, device=DEV).reshape(p, 1, page_size, 1) / 200.0
    pool = pool.to(torch.bfloat16)
    tok0, qlen, pos0, ptrow, t = [], [], [], [], 0
    for s, n in enumerate(lens):
        p0 = 0
        while p0 < n:
            size = min(int(rng.integers(1, BT + 1)) if kind == "odd" else BT, n - p0)
            tok0.append(t); qlen.append(size); pos0.append(past[s] + p0); ptrow.append(s); t += size; p0 += size
            if kind == "odd" and rng.random() < 0.1:
                tok0.append(t); qlen.append(0); pos0.append(past[s] + p0); ptrow.append(s)
    assert len(tok0) * nkv > (3 if d == 128 else 6) * 74
    q = torch.randn((t, nh * d), device=DEV, generator=g).to(torch.bfloat16)
    args = [dev_i32(a) for a in (pt, tok0, qlen, pos0, ptrow)]

    def run():
        out = torch.full((t + 1, nh * d), float("nan"), dtype=torch.bfloat16, device=DEV)
        check(lib().dis_k_attn_prefill(ptr(q), ptr(pool), pool.shape[0], ptr(args[0]), pt.shape[1], ptr(args[1]), ptr(args[2]), ptr(args[3]), ptr(args[4]),
                                       ptr(out), len(tok0), nh, nkv, d, page_size, torch.cuda.current_stream().cuda_stream))
        return out

    outs = [run(), run()]
    sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs.append(run())
    graph.replay()
    sync()
    assert all(torch.equal(o[:t], outs[0][:t]) for o in outs) and bool(torch.isnan(outs[0][t]).all())
    row = 0
    for s, n in enumerate(lens):
        kv = pool[torch.as_tensor(pt[s, :per[s]].astype(np.int64), device=DEV)].double()
        K, V = (kv[:, c].permute(1, 0, 2, 3).reshape(nkv, -1, d)[:, :total[s]] for c in (0, 1))
        qs = q[row:row + n].double().reshape(n, nkv, nh // nkv, d).permute(1, 2, 0, 3)
        sc = qs @ K.transpose(1, 2).unsqueeze(1) / d ** 0.5
        sc = sc.masked_fill(torch.arange(total[s], device=DEV)[None] > torch.arange(past[s], total[s], device=DEV)[:, None], float("-inf"))
        ref = (torch.softmax(sc, dim=-1) @ V.unsqueeze(1)).permute(2, 0, 1, 3).reshape(n, nh * d)
        err = (outs[0][row:row + n].double() - ref).abs().max().item()
        assert err <= 2 * BF16_ULP * V.abs().max().item() + 1e-5, (s, n, err)
        row += n


@pytest.mark.parametrize("nh,nkv,BT", [(32, 8, 32), (32, 4, 16)])
@pytest.mark.parametrize("longest", [2300, 4200])
def test_attention_prefill_heads_of_64_bits_in_pairs_and_alone(nh, nkv, BT, longest):
    """Heads of 64: a query block has the same bits whether it is one of a pair or alone in its CTA, so the number of blocks of a pass does
    not move its error (even and odd key tiles have a maximum of their own in both forms).  Prompts of 1 to 40 tiles, some behind a cache,
    keys that grow with their position, one block of an odd sequence left over.  With the longer prompt a pass of any size keeps its blocks
    alone, more of them than run at once."""
    d, page_size = 64, 64
    g = torch.Generator(device=DEV); g.manual_seed(nh + nkv)
    rng = np.random.default_rng(nkv)
    lens, past = [longest, 65, 700, 1, 1300], [0, 200, 0, 0, 64]
    while sum(-(-n // BT) for n in lens) * nkv <= 6 * 148 // 2 + nkv:
        lens.append(int(rng.integers(1, 900))); past.append(int(rng.choice([0, 100])))
    total = [a + b for a, b in zip(past, lens)]
    per = [-(-n // page_size) for n in total]
    pt = np.zeros((len(lens), max(per)), np.int32)
    perm = rng.permutation(sum(per))
    for s, at in enumerate(np.cumsum([0] + per[:-1])):
        pt[s, :per[s]] = perm[at:at + per[s]]
    pool = torch.randn((sum(per), 2, nkv, page_size, d), device=DEV, generator=g)
    for s, p in enumerate(per):
        pool[torch.as_tensor(pt[s, :p].astype(np.int64), device=DEV), 0] *= 0.3 + torch.arange(p * page_size, device=DEV).reshape(p, 1, page_size, 1) / 600.0
    pool = pool.to(torch.bfloat16)
    tok0, qlen, pos0, ptrow, t = [], [], [], [], 0
    for s, n in enumerate(lens):
        for k in range(0, n, BT):
            tok0.append(t + k); qlen.append(min(BT, n - k)); pos0.append(past[s] + k); ptrow.append(s)
        t += n
    q = torch.randn((t, nh * d), device=DEV, generator=g).to(torch.bfloat16)
    dpt, args = dev_i32(pt), [np.asarray(a, np.int32) for a in (tok0, qlen, pos0, ptrow)]

    def run(step):
        out = torch.full((t, nh * d), float("nan"), dtype=torch.bfloat16, device=DEV)
        for at in range(0, len(tok0), step):
            part = [dev_i32(a[at:at + step]) for a in args]
            check(lib().dis_k_attn_prefill(ptr(q), ptr(pool), pool.shape[0], ptr(dpt), pt.shape[1], *[ptr(p) for p in part], ptr(out), len(tok0[at:at + step]), nh, nkv, d, page_size,
                                           torch.cuda.current_stream().cuda_stream))
        return out

    together, alone = run(len(tok0)), run(6 * 148 // 2 // nkv)
    sync()
    assert len(tok0) * nkv > 6 * 148 // 2 and not bool(torch.isnan(alone.float()).any())
    assert torch.equal(together, alone)


@pytest.mark.parametrize("nh,nkv,page_size,BT", [(8, 1, 8, 16), (8, 2, 64, 16), (8, 2, 64, 32), (16, 2, 128, 16), (16, 4, 16, 32)])
@pytest.mark.parametrize("past", [0, 63, 200])
def test_attention_prefill_heads_of_64(nh, nkv, page_size, past, BT):
    """The tcgen05 kernel for heads of 64 at the edges of its 64-key tiles: one tile (only one of its two softmax groups works), 64 and 65
    keys, an odd number of tiles, portions behind keys already in the cache, and scores that grow along the keys so that the
    softmax reference has to be raised after the first tile.  Blocks of 16 tokens, as the C ABI promises, and of 32 for groups of 4, as
    the engine makes them (all 128 query rows), full and ragged.  Against float64; two bf16 roundings (weights, result) of values up to
    the largest |v|."""
    g = torch.Generator(device=DEV); g.manual_seed(past + nh + page_size)
    d, lens = 64, [1, 16, 17, 31, 32, 33, 64, 65, 129, 330]
    assert lib().dis_k_attn_prefill_block_tokens(nh, nkv, d) == 16
    total = [past + n for n in lens]
    per = [(n + page_size - 1) // page_size for n in total]
    n_pages = sum(per)
    perm = np.random.default_rng(past).permutation(n_pages).astype(np.int32)
    pt = np.zeros((len(lens), max(per)), np.int32)
    at = 0
    for s, p in enumerate(per):
        pt[s, :p] = perm[at:at + p]; at += p
    pool = torch.randn((n_pages, 2, nkv, page_size, d), device=DEV, generator=g)
    for s, p in enumerate(per):  # keys grow with their position: later tiles hold the largest scores
        pos = torch.arange(p * page_size, device=DEV).reshape(p, 1, page_size, 1)
        pool[torch.as_tensor(pt[s, :p].astype(np.int64), device=DEV), 0] *= 0.2 + pos / 64.0
    pool = pool.to(torch.bfloat16)
    tok0, qlen, pos0, ptrow, t = [], [], [], [], 0
    for s, n in enumerate(lens):
        for p0 in range(0, n, BT):
            tok0.append(t); qlen.append(min(BT, n - p0)); pos0.append(past + p0); ptrow.append(s); t += qlen[-1]
    q = torch.randn((t, nh * d), device=DEV, generator=g).to(torch.bfloat16)
    out = G.empty((t, nh * d), dtype=torch.bfloat16, device=DEV)
    check(lib().dis_k_attn_prefill(ptr(q), ptr(pool), n_pages, ptr(dev_i32(pt)), pt.shape[1], ptr(dev_i32(tok0)), ptr(dev_i32(qlen)),
                                   ptr(dev_i32(pos0)), ptr(dev_i32(ptrow)), ptr(out), len(tok0), nh, nkv, d, page_size, None))
    sync()
    row = 0
    for s, n in enumerate(lens):
        kv = pool[torch.as_tensor(pt[s, :per[s]].astype(np.int64), device=DEV)].double()
        K, V = (kv[:, c].permute(1, 0, 2, 3).reshape(nkv, -1, d)[:, :total[s]] for c in (0, 1))
        qs = q[row:row + n].double().reshape(n, nkv, nh // nkv, d).permute(1, 2, 0, 3)
        sc = qs @ K.transpose(1, 2).unsqueeze(1) / d ** 0.5
        sc = sc.masked_fill(torch.arange(total[s], device=DEV)[None] > torch.arange(past, total[s], device=DEV)[:, None], float("-inf"))
        ref = (torch.softmax(sc, dim=-1) @ V.unsqueeze(1)).permute(2, 0, 1, 3).reshape(n, nh * d)
        err = (out[row:row + n].double() - ref).abs().max().item()
        assert err <= 2 * BF16_ULP * V.abs().max().item() + 1e-5, (s, n, err)
        row += n


@pytest.mark.parametrize("nh,nkv,d", [(8, 1, 64), (8, 2, 64), (8, 2, 128), (4, 4, 64)])
def test_attention_prefill_with_empty_blocks(nh, nkv, d):
    """Blocks of no tokens, at position 0 (no key either) and behind keys, beside a block of seven: they write nothing, and the block beside
    them is what it is alone."""
    g = torch.Generator(device=DEV); g.manual_seed(d + nh)
    ps, T = 16, 7
    pool = torch.randn((1, 2, nkv, ps, d), device=DEV, generator=g).to(torch.bfloat16)
    q = torch.randn((T, nh * d), device=DEV, generator=g).to(torch.bfloat16)
    outs = []
    for tok0, ln, pos0 in (([0], [T], [0]), ([0, 0, 7, 0], [0, T, 0, 0], [0, 0, 0, 9])):
        out = G.zeros((T, nh * d), dtype=torch.bfloat16, device=DEV)
        check(lib().dis_k_attn_prefill(ptr(q), ptr(pool), 1, ptr(dev_i32([[0]])), 1, ptr(dev_i32(tok0)), ptr(dev_i32(ln)), ptr(dev_i32(pos0)),
                                       ptr(dev_i32([0] * len(ln))), ptr(out), len(ln), nh, nkv, d, ps, None))
        sync()
        outs.append(out)
    assert torch.isfinite(outs[0]).all() and outs[0].any()
    assert torch.equal(outs[0], outs[1])


def _prefill_call(nh, nkv, d, off_q, off_out, n=50, ps=64):
    """One prompt of n tokens, q and out starting off_* bf16 elements behind a 16-byte boundary -> (return code, q, pool, out)."""
    g = torch.Generator(device=DEV); g.manual_seed(nh)
    BT = lib().dis_k_attn_prefill_block_tokens(nh, nkv, d)
    pool = torch.randn((1, 2, nkv, ps, d), device=DEV, generator=g).to(torch.bfloat16)
    q = torch.randn(n * nh * d + 8, device=DEV, generator=g).to(torch.bfloat16)[off_q:][:n * nh * d]
    out = G.zeros(n * nh * d + 8, dtype=torch.bfloat16, device=DEV)[off_out:][:n * nh * d]
    t0 = list(range(0, n, BT))
    ln = [min(BT, n - t) for t in t0]
    rc = lib().dis_k_attn_prefill(ptr(q), ptr(pool), 1, ptr(dev_i32([[0]])), 1, ptr(dev_i32(t0)), ptr(dev_i32(ln)), ptr(dev_i32(t0)),
                                  ptr(dev_i32([0] * len(t0))), ptr(out), len(t0), nh, nkv, d, ps, None)
    sync()
    return rc, q.view(n, nh * d), pool, out.view(n, nh * d)


@pytest.mark.parametrize("off_q,off_out", [(2, 0), (0, 2), (6, 4), (0, 0)])
@pytest.mark.parametrize("nh,nkv", [(8, 1), (8, 2)])
def test_attention_prefill_heads_of_64_off_a_16_byte_boundary(nh, nkv, off_q, off_out):
    """q or out on 4 or 8 bytes only: against float64, as test_attention_prefill_heads_of_64."""
    rc, q, pool, out = _prefill_call(nh, nkv, 64, off_q, off_out)
    check(rc)
    n, kv = q.shape[0], pool[0].double()
    K, V = kv[0][:, :n], kv[1][:, :n]
    sc = q.double().reshape(n, nkv, nh // nkv, 64).permute(1, 2, 0, 3) @ K.transpose(1, 2).unsqueeze(1) / 8.0
    sc = sc.masked_fill(torch.ones(n, n, device=DEV).triu(1).bool(), float("-inf"))
    ref = (torch.softmax(sc, dim=-1) @ V.unsqueeze(1)).permute(2, 0, 1, 3).reshape(n, nh * 64)
    assert (out.double() - ref).abs().max().item() <= 2 * BF16_ULP * V.abs().max().item() + 1e-5


@pytest.mark.parametrize("off_q,off_out", [(2, 0), (0, 4)])
def test_attention_prefill_heads_of_128_off_a_16_byte_boundary_are_refused(off_q, off_out):
    rc, _, _, out = _prefill_call(8, 2, 128, off_q, off_out)
    assert rc != 0 and b"16 bytes" in lib().dis_last_error()
    assert not out.any()


@pytest.mark.parametrize("nh,nkv", [(32, 4), (16, 4)])
def test_attention_prefill_heads_of_64_rounds_no_more_than_a_running_maximum(nh, nkv):
    """The 2-norm error against float64 is no larger than that of softmax weights rounded to bf16 under the row's own maximum (whose
    weight is then exactly 1), the sum not rounded, the result rounded once.  2 % for the sample: 2.8e6 results or more; a reference
    that is raised lazily was 3.5 % further off."""
    g = torch.Generator(device=DEV); g.manual_seed(nh)
    d, ps, lens = 64, 64, [1400, 500, 900]
    BT = lib().dis_k_attn_prefill_block_tokens(nh, nkv, d)
    per = [(n + ps - 1) // ps for n in lens]
    pt = np.zeros((len(lens), max(per)), np.int32)
    for s, p in enumerate(per):
        pt[s, :p] = sum(per[:s]) + np.arange(p)
    pool = torch.randn((sum(per), 2, nkv, ps, d), device=DEV, generator=g).to(torch.bfloat16)
    tok0, qlen, pos0, ptrow, t = [], [], [], [], 0
    for s, n in enumerate(lens):
        for p0 in range(0, n, BT):
            tok0.append(t); qlen.append(min(BT, n - p0)); pos0.append(p0); ptrow.append(s); t += qlen[-1]
    q = (1.5 * torch.randn((t, nh * d), device=DEV, generator=g)).to(torch.bfloat16)
    out = G.empty((t, nh * d), dtype=torch.bfloat16, device=DEV)
    check(lib().dis_k_attn_prefill(ptr(q), ptr(pool), sum(per), ptr(dev_i32(pt)), pt.shape[1], ptr(dev_i32(tok0)), ptr(dev_i32(qlen)),
                                   ptr(dev_i32(pos0)), ptr(dev_i32(ptrow)), ptr(out), len(tok0), nh, nkv, d, ps, None))
    sync()
    row, err, bound = 0, 0.0, 0.0
    for s, n in enumerate(lens):
        kv = pool[sum(per[:s]):sum(per[:s + 1])].double()
        K, V = (kv[:, c].permute(1, 0, 2, 3).reshape(nkv, -1, d)[:, :n] for c in (0, 1))
        qs = q[row:row + n].double().reshape(n, nkv, nh // nkv, d).permute(1, 2, 0, 3)
        sc = qs @ K.transpose(1, 2).unsqueeze(1) / d ** 0.5
        sc = sc.masked_fill(torch.arange(n, device=DEV)[None] > torch.arange(n, device=DEV)[:, None], float("-inf"))
        w = torch.exp(sc - sc.amax(-1, keepdim=True))
        l = w.sum(-1, keepdim=True)
        flat = lambda o: o.permute(2, 0, 1, 3).reshape(n, nh * d)  # noqa: E731
        ref = flat((w @ V.unsqueeze(1)) / l)
        rounded = flat((w.to(torch.bfloat16).double() @ V.unsqueeze(1)) / l).to(torch.bfloat16).double()
        err += (out[row:row + n].double() - ref).square().sum().item()
        bound += (rounded - ref).square().sum().item()
        row += n
    assert err ** 0.5 <= 1.02 * bound ** 0.5, (err ** 0.5, bound ** 0.5, (err / bound) ** 0.5)


def test_attention_prefill_full_size_against_torch():
    """Llama-3-8B geometry, a 3000-token prompt prefilled from position 0 and the last 1000 tokens of a 4000-token one
    (a later chunk of a chunked prefill), 64-token pages in shuffled order: causal attention against fp32 torch."""
    g = torch.Generator(device=DEV); g.manual_seed(13)
    d, nh, nkv, ps = 128, 32, 8, 64
    lens, starts = [3000, 4000], [0, 3000]
    rng = np.random.default_rng(13)
    pages_per = [(n + ps - 1) // ps for n in lens]
    n_pages, max_pages = sum(pages_per) + 2, max(pages_per)
    perm = rng.permutation(n_pages)
    pt = np.zeros((2, max_pages), np.int32)
    pt[0, :pages_per[0]] = perm[:pages_per[0]]; pt[1, :pages_per[1]] = perm[pages_per[0]:pages_per[0] + pages_per[1]]
    pool = torch.randn((n_pages, 2, nkv, ps, d), device=DEV, generator=g).to(torch.bfloat16)
    tok0, qlen, pos0, ptrow, t = [], [], [], [], 0
    BT = lib().dis_k_attn_prefill_block_tokens(nh, nkv, d)      # 32: the tcgen05 kernel's 128 query rows = 32 tokens x 4 heads
    assert BT == 32
    for s in range(2):
        for p0 in range(starts[s], lens[s], BT):
            ln = min(BT, lens[s] - p0)
            tok0.append(t); qlen.append(ln); pos0.append(p0); ptrow.append(s); t += ln
    q = torch.randn((t, nh * d), device=DEV, generator=g).to(torch.bfloat16)
    out = G.empty((t, nh * d), dtype=torch.bfloat16, device=DEV)
    check(lib().dis_k_attn_prefill(ptr(q), ptr(pool), n_pages, ptr(dev_i32(pt)), max_pages, ptr(dev_i32(tok0)), ptr(dev_i32(qlen)),
                                   ptr(dev_i32(pos0)), ptr(dev_i32(ptrow)), ptr(out), len(tok0), nh, nkv, d, ps, None))
    sync()
    row, worst, scale = 0, 0.0, 0.0
    for s in range(2):
        pages = torch.as_tensor(pt[s, :pages_per[s]].astype(np.int64), device=DEV)
        kv = pool[pages].float()
        K = kv[:, 0].permute(1, 0, 2, 3).reshape(nkv, -1, d)[:, :lens[s]]
        V = kv[:, 1].permute(1, 0, 2, 3).reshape(nkv, -1, d)[:, :lens[s]]
        n_q = lens[s] - starts[s]
        qs = q[row:row + n_q].float().reshape(n_q, nkv, nh // nkv, d).permute(1, 2, 0, 3)       # [nkv, G, n_q, d]
        sc = qs @ K.transpose(1, 2).unsqueeze(1) / d ** 0.5                                     # [nkv, G, n_q, keys]
        keys = torch.arange(lens[s], device=DEV)[None, :]
        qpos = torch.arange(starts[s], lens[s], device=DEV)[:, None]
        sc = sc.masked_fill(keys > qpos, float("-inf"))
        ref = (torch.softmax(sc, dim=-1) @ V.unsqueeze(1)).permute(2, 0, 1, 3).reshape(n_q, nh * d)
        worst = max(worst, (out[row:row + n_q].float() - ref).abs().max().item())
        scale = max(scale, ref.abs().max().item())
        row += n_q
    assert worst <= 2 * BF16_ULP * scale + 1e-5, (worst, scale)


def test_sampler_argmax_and_ties():
    rng = np.random.default_rng(0)
    T, V = 6, 128256
    lg = rng.standard_normal((T, V)).astype(np.float32)
    lg[1, [500, 90000]] = 9.0      # tie -> lowest index
    lg[2, V - 1] = 11.0            # last element
    lg[3, 0] = 11.0                # first element
    out = G.zeros(T, dtype=torch.int32, device=DEV)
    lp = G.zeros(T, dtype=torch.float32, device=DEV)
    check(lib().dis_k_sample(ptr(dev_f32(lg)), V, T, V, None, None, None, None, ptr(out), ptr(lp), None))
    sync()
    ref = [O.argmax(lg[t])[0] for t in range(T)]
    assert out.cpu().tolist() == ref
    assert ref[1] == 500
    # TokenEvent.logprob (models.rs:276): log softmax(logits)[token], against float64 numpy
    z = lg.astype(np.float64)
    want = z[np.arange(T), ref] - (np.log(np.exp(z - z.max(1, keepdims=True)).sum(1)) + z.max(1))
    assert np.abs(lp.cpu().numpy() - want).max() <= 1e-4


@pytest.mark.parametrize("T,V", [(48, 4099), (24, 128256)], ids=["ragged-vocab", "llama3-vocab"])
def test_sampler_top_p_matches_oracle(T, V):
    rng = np.random.default_rng(1)
    lg = (rng.standard_normal((T, V)) * 2.5).astype(np.float32)
    temps = rng.choice([0.0, 0.5, 1.0, 1.7], T).astype(np.float32)
    tps = rng.choice([0.1, 0.5, 0.9, 0.95, 1.0], T).astype(np.float32)
    seeds = rng.integers(0, 2 ** 40, T).astype(np.uint64)
    steps = rng.integers(0, 100, T).astype(np.uint64)
    out = G.zeros(T, dtype=torch.int32, device=DEV)
    ds = torch.from_numpy(seeds.view(np.int64)).to(DEV)
    dst = torch.from_numpy(steps.view(np.int64)).to(DEV)
    lp = G.zeros(T, dtype=torch.float32, device=DEV)
    check(lib().dis_k_sample(ptr(dev_f32(lg)), V, T, V, ptr(dev_f32(temps)), ptr(dev_f32(tps)), ptr(ds), ptr(dst), ptr(out), ptr(lp), None))
    sync()
    got = out.cpu().tolist()
    # log-probability of the drawn token under softmax(logits / temperature) (temperature 0: the plain softmax)
    for t in range(T):
        z = lg[t].astype(np.float64) / (float(temps[t]) if temps[t] > 0 else 1.0)
        want = z[got[t]] - (np.log(np.exp(z - z.max()).sum()) + z.max())
        assert abs(float(lp[t]) - want) <= 1e-3 * max(1.0, abs(want)), (t, float(lp[t]), want)
    mism = 0
    for t in range(T):
        ref, tau, mass = O.sample(lg[t], float(temps[t]), float(tps[t]), int(seeds[t]), int(steps[t]))
        if got[t] != ref:
            mism += 1
            # only a draw that lands within fp32 noise of a bucket edge may differ
            z = lg[t] / temps[t]; p = np.exp(z - z.max()); p /= p.sum()
            kept = p >= tau * (1 - 1e-5)
            assert kept[got[t]], (t, got[t], ref)
    assert mism <= 2, mism
    # greedy rows are exact
    for t in range(T):
        if temps[t] == 0:
            assert got[t] == int(np.argmax(lg[t]))


@pytest.mark.parametrize("V,ld", [(1, 1), (3, 7), (130, 131), (16384, 16384), (16385, 16388), (65536, 65537), (131073, 131076),
                                  (262144, 262144), (262145, 262145)])
def test_sampler_row_sizes(V, ld):
    """Rows at the edges of the cluster sampler's register sizes (16384 logits per float4 of a thread), rows that do not start on 16
    bytes, and one row more than it takes: draws of the oracle, argmax and log-probability against float64; a second call repeats
    the first bit for bit.  A draw may differ where u * kept is within fp32 noise of an edge: at most one of the rows."""
    T = 6
    rng = np.random.default_rng(V)
    full = np.full((T, ld), 1e9, np.float32)  # the padding behind a row must not be read as logits
    lg = (rng.standard_normal((T, V)) * 2.0).astype(np.float32)
    if V > 100:
        lg[:, 17] = -np.inf
    full[:, :V] = lg
    temps = np.array([0.0, 0.7, 1.0, 1.3, 0.9, 0.0], np.float32)
    tps = np.array([0.5, 0.5, 0.9, 1.0, 0.05, 1.0], np.float32)
    seeds, steps = rng.integers(0, 2 ** 40, T).astype(np.uint64), rng.integers(0, 100, T).astype(np.uint64)
    dl, dt, dp = dev_f32(full), dev_f32(temps), dev_f32(tps)
    ds, dst = (torch.from_numpy(a.view(np.int64)).to(DEV) for a in (seeds, steps))
    runs = []
    for _ in range(2):
        out, lp = G.zeros(T, dtype=torch.int32, device=DEV), G.zeros(T, dtype=torch.float32, device=DEV)
        check(lib().dis_k_sample(ptr(dl), ld, T, V, ptr(dt), ptr(dp), ptr(ds), ptr(dst), ptr(out), ptr(lp), None))
        sync()
        runs.append((out.cpu().numpy(), lp.cpu().numpy()))
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
    got, lp = runs[0]
    off = 0
    for t in range(T):
        z = lg[t].astype(np.float64) / (float(temps[t]) if temps[t] > 0 else 1.0)
        want = z[got[t]] - (np.log(np.exp(z - z.max()).sum()) + z.max())
        assert abs(float(lp[t]) - want) <= 1e-4 * max(1.0, abs(want)), (t, float(lp[t]), want)
        if temps[t] == 0:
            assert got[t] == int(np.argmax(lg[t]))
        else:
            off += got[t] != O.sample(lg[t], float(temps[t]), float(tps[t]), int(seeds[t]), int(steps[t]))[0]
    assert off <= 1, off


@pytest.mark.parametrize("V,masked,calls", [(32000, 0.5, 24), (128256, 0.5, 24), (128256, 0.9, 24), (262144, 0.5, 8), (262145, 0.5, 1)])
def test_sampler_never_draws_a_masked_token(V, masked, calls):
    """Rows with most logits at -inf and no nucleus cut (top_p 1), 4096 draws a call under other seeds, in every row size of the sampler
    and in the kernel for longer rows: every drawn token has a finite logit and a finite log-probability.  Rounding at the edges of lanes
    gave masked tokens 1e-4 of the mass (10 of 98304 draws)."""
    T = 4096
    rng = np.random.default_rng(V)
    row = rng.standard_normal(V).astype(np.float32)
    row[rng.random(V) < masked] = -np.inf
    row[-1] = -np.inf
    dl = dev_f32(row)
    ok = torch.isfinite(dl)
    dt = dev_f32(np.ones(T))
    dp = dt
    dst = torch.arange(T, dtype=torch.int64, device=DEV)
    out, lp = G.zeros(T, dtype=torch.int32, device=DEV), G.zeros(T, dtype=torch.float32, device=DEV)
    for c in range(calls):
        ds = torch.full((T,), 1000 + c, dtype=torch.int64, device=DEV)
        check(lib().dis_k_sample(ptr(dl), 0, T, V, ptr(dt), ptr(dp), ptr(ds), ptr(dst), ptr(out), ptr(lp), None))  # (row stride 0: one row)
        sync()
        bad = int((~ok[out.long()]).sum())
        assert bad == 0, (c, bad)
        assert bool(torch.isfinite(lp).all())


@pytest.mark.parametrize("kind,top_p", [("flat", 0.5), ("flat", 0.999), ("below 2^-30", 0.99997), ("below 2^-61", 0.99999988), ("one octave", 0.3), ("steps", 0.0),
                                        ("steps", 1e-9), ("steps", 0.7), ("steps", 0.99999994)])
def test_sampler_threshold_in_any_octave(kind, top_p):
    """The threshold search over rows whose nucleus ends in the first octave, among equal weights, below 2^-30 of the largest weight (a
    second search over the exponents) and nowhere (nothing below carries mass that fp32 sums see).  Draws with u close to 1 fall to the last kept tokens in index
    order: they are compared, as running masses, with float64; what fp32 sums of V weights leave open is V^0.5 2^-24 of the mass, below
    4e-5; where a tail of 7e-5 is looked at, its weights are added to a sum of about 1 and a share of them may be rounded off."""
    V, T = 131072, 64
    rng = np.random.default_rng(11)
    lg = {"flat": np.zeros(V), "one octave": rng.uniform(-0.6, 0.0, V), "steps": -np.floor(np.arange(V) / 1024) * 0.31,
          "below 2^-30": np.full(V, -21.5), "below 2^-61": np.full(V, -45.0)}[kind].astype(np.float32)
    if kind.startswith("below"):
        lg += rng.uniform(-0.5, 0.5, V).astype(np.float32)
        lg[0] = 0.0
    seeds, u = [], []
    k = 0
    while len(seeds) < T:
        h = _draw_u(k)
        if len(seeds) % 2 == 0 or h > 0.9999:
            seeds.append(k)
            u.append(h)
        k += 1
    ones, tps = dev_f32(np.ones(T)), dev_f32(np.full(T, top_p, np.float32))
    ds, dst = torch.tensor(seeds, dtype=torch.int64, device=DEV), torch.zeros(T, dtype=torch.int64, device=DEV)
    out, lp = G.zeros(T, dtype=torch.int32, device=DEV), G.zeros(T, dtype=torch.float32, device=DEV)
    check(lib().dis_k_sample(ptr(dev_f32(lg)), 0, T, V, ptr(ones), ptr(tps), ptr(ds), ptr(dst), ptr(out), ptr(lp), None))  # (row stride 0: one row)
    sync()
    got = out.cpu().numpy()
    p = np.exp(lg.astype(np.float64) - lg.max())
    p /= p.sum()
    order = np.sort(p)[::-1]
    tp = float(np.float32(top_p))
    tau = order[min(int((np.cumsum(order) < tp).sum()), V - 1)]
    run = np.cumsum(np.where(p >= tau * (1 - 1e-6), p, 0.0))
    for t in range(T):
        at = run[got[t]] / run[-1]
        before = (run[got[t]] - p[got[t]]) / run[-1]
        if top_p <= 0:
            assert got[t] == int(np.argmax(lg))
        else:
            assert before - 4e-5 <= u[t] <= at + 4e-5, (t, u[t], before, at)
            assert p[got[t]] >= tau * (1 - 1e-3), (t, p[got[t]], tau)
        assert abs(float(lp[t]) - np.log(p[got[t]])) <= 1e-4 * max(1.0, abs(np.log(p[got[t]])))


def _draw_u(seed):
    m = (1 << 64) - 1
    z = (seed * 0x9E3779B97F4A7C15 + 0xC0FFEE * 0xD1B54A32D192ED03 + 0x632BE59BD9B4E019) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return ((z ^ (z >> 31)) >> 40) / 16777216.0


@pytest.mark.parametrize("tp,T,V", [(1, 48, 4099), (1, 32, 128256), (2, 48, 4100), (3, 20, 4098), (4, 24, 128256), (8, 16, 128256)],
                         ids=["single-rank-ragged-vocab", "single-rank-llama3-vocab", "tp2-small-vocab", "tp3-small-vocab",
                              "tp4-llama3-vocab", "tp8-llama3-vocab"])
def test_vocab_parallel_sampler_matches_the_one_gpu_sampler_and_the_oracle(tp, T, V):
    """The tensor-parallel engines' sampler (k_tp_sample.cu) with its ranks emulated on one GPU: every rank keeps V/tp
    logit columns and exchanges scalars (candidates, 16 partial masses per round of the threshold search, the drawn
    token).  All ranks must write the same token and log-probability; greedy rows are exact; nucleus rows must draw what
    dis_k_sample and the oracle draw, except where the draw lands within fp32 noise of a bucket edge (the partial sums
    are associated per rank).  Two calls on the same exchange area: the second must not see the first one's words."""
    rng = np.random.default_rng(3 + tp)
    rows = T + 3                                                   # area rows > T: the row stride is the area's, not the call's
    n_area = tp * lib().dis_k_sample_vocab_parallel_area_bytes(tp, rows) // 4
    area = G.zeros(n_area, dtype=torch.int32, device=DEV)
    for call_no in (1, 2):
        lg = (rng.standard_normal((T, V)) * 2.5).astype(np.float32)
        lg[0, [V // tp - 1, (V // tp) % V]] = 40.0                 # a tie across a slice boundary: the lower id wins
        temps = rng.choice([0.0, 0.5, 1.0, 1.7], T).astype(np.float32)
        temps[0] = 0.0
        tps = rng.choice([0.1, 0.5, 0.9, 0.95, 1.0], T).astype(np.float32)
        seeds = rng.integers(0, 2 ** 40, T).astype(np.uint64)
        steps = rng.integers(0, 100, T).astype(np.uint64)
        dl, dt, dp = dev_f32(lg), dev_f32(temps), dev_f32(tps)
        ds = torch.from_numpy(seeds.view(np.int64)).to(DEV)
        dst = torch.from_numpy(steps.view(np.int64)).to(DEV)
        out = G.zeros((tp, T), dtype=torch.int32, device=DEV)
        lp = G.zeros((tp, T), dtype=torch.float32, device=DEV)
        check(lib().dis_k_sample_vocab_parallel(ptr(dl), T, V, tp, ptr(dt), ptr(dp), ptr(ds), ptr(dst), call_no, ptr(area), rows,
                                                ptr(out), ptr(lp), None))
        one = G.zeros(T, dtype=torch.int32, device=DEV)
        one_lp = G.zeros(T, dtype=torch.float32, device=DEV)
        check(lib().dis_k_sample(ptr(dl), V, T, V, ptr(dt), ptr(dp), ptr(ds), ptr(dst), ptr(one), ptr(one_lp), None))
        sync()
        got_all, lp_all = out.cpu().numpy(), lp.cpu().numpy()
        for r in range(1, tp):                                     # every rank computes the same bits
            assert np.array_equal(got_all[0], got_all[r]) and np.array_equal(lp_all[0], lp_all[r]), r
        got, single = got_all[0].tolist(), one.cpu().tolist()
        assert got[0] == (V // tp - 1 if tp > 1 else 0)
        mism_single = mism_oracle = 0
        for t in range(T):
            z = lg[t].astype(np.float64) / (float(temps[t]) if temps[t] > 0 else 1.0)
            want_lp = z[got[t]] - (np.log(np.exp(z - z.max()).sum()) + z.max())
            assert abs(float(lp_all[0, t]) - want_lp) <= 1e-3 * max(1.0, abs(want_lp)), (t, float(lp_all[0, t]), want_lp)
            if temps[t] == 0:
                assert got[t] == int(np.argmax(lg[t])) == single[t]
                continue
            ref, tau, mass = O.sample(lg[t], float(temps[t]), float(tps[t]), int(seeds[t]), int(steps[t]))
            if got[t] != ref or got[t] != single[t]:
                mism_oracle += got[t] != ref
                mism_single += got[t] != single[t]
                p = np.exp(z - z.max()); p /= p.sum()
                assert (p >= tau * (1 - 1e-5))[got[t]], (t, got[t], ref, single[t])   # still inside the nucleus
        assert mism_oracle <= 2 and mism_single <= 2, (mism_oracle, mism_single)
