"""Numerics of every sm_100a kernel against the float32 PyTorch restatement of the same op."""
import math

import pytest
import torch

from zml_b200 import ops
from zml_b200.ops import reference as ref
from zml_b200.testing import expect_close

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _randn(*shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device=DEV, dtype=torch.float32) * scale).to(dtype)


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    ops.raise_on_status()


@pytest.mark.parametrize("m,n,k", [
    (1, 256, 128), (7, 384, 64), (5, 256, 320), (16, 1024, 256), (32, 128, 2048), (128, 128, 2048), (16, 4096, 4096), (32, 6144, 4096), (33, 1000 * 8, 512),
    (64, 4096, 14336), (128, 2048, 2048), (128, 5120, 2048), (100, 2048, 4096), (97, 4096, 4096 + 64), (200, 512, 1024), (256, 1024, 4096),
    (257, 1024, 1024), (512, 4096, 4096), (1000, 2048 + 64, 512), (4096, 4096, 4096),
    (3000, 14336 * 2, 4096 // 2),
])
def test_gemm_matches_fp32(m, n, k):
    torch.manual_seed(m * 7 + n)
    a = _randn(m, k)
    w = _randn(n, k, scale=1.0 / math.sqrt(k))
    out = ops.gemm(a, w)
    want = a.float() @ w.float().t()
    expect_close(out.float(), want, atol=2e-2, rtol=2e-2, min_close=0.999)


@pytest.mark.parametrize("m,n,k,splits", [(16, 512, 2048, 4), (64, 1024, 8192, 8), (300, 512, 4096, 3)])
def test_gemm_split_k_and_epilogue(m, n, k, splits):
    torch.manual_seed(0)
    a = _randn(m, k)
    w = _randn(n, k, scale=1.0 / math.sqrt(k))
    res = _randn(m, n)
    bias = _randn(n)
    want = a.float() @ w.float().t() + bias.float() + res.float()
    out = ops.gemm(a, w, residual=res, bias=bias, force_splits=splits)
    expect_close(out.float(), want, atol=3e-2, rtol=2e-2, min_close=0.999)
    # twice: the tile counters must have been left at zero
    out2 = ops.gemm(a, w, residual=res, bias=bias, force_splits=splits)
    assert torch.equal(out, out2)
    # fp32 output and in-place residual
    out32 = ops.gemm(a, w, out_dtype=torch.float32, force_splits=splits)
    expect_close(out32, a.float() @ w.float().t(), atol=1e-2, rtol=1e-2, min_close=0.999)
    inplace = res.clone()
    ops.gemm(a, w, residual=inplace, out=inplace)
    expect_close(inplace.float(), a.float() @ w.float().t() + res.float(), atol=3e-2, rtol=2e-2, min_close=0.999)


# every epilogue path of the GEMM: cluster split-K with 4, 3 (odd band heights) and 8 CTAs, the stream-K fix-up,
# the generic swap-AB path with 128- and 256-token tiles, and whole tiles with tokens as rows
EPI_SHAPES = [(32, 4096, 4096), (32, 6144, 4096), (8, 2048, 8192), (32, 28672, 4096), (64, 512, 1024), (100, 2048, 4096),
              (200, 1024, 2048), (257, 1024, 1024), (512, 4096, 2048), (1000, 2048 + 64, 512)]


@pytest.mark.parametrize("m,n,k", EPI_SHAPES)
def test_gemm_row_scale_and_swiglu_epilogues(m, n, k):
    """rmsnorm(a) @ (w * g)^T as one GEMM with a per-row scale from partial sums of squares, and SwiGLU on
    interleaved gate / up rows, against the unfused float32 chain."""
    torch.manual_seed(m + n + k)
    a = _randn(m, k)
    w = _randn(n, k, scale=1.0 / math.sqrt(k))
    g = (1.0 + 0.2 * torch.randn(k, device=DEV)).bfloat16()
    stats = ops.row_sumsq(a)
    expect_close(stats.total(), a.float().pow(2).sum(-1), atol=1e-2, rtol=1e-3)
    # the partial sums may come in several parts: split the one part in three unequal ones
    parts = torch.stack([stats.parts[0] * 0.5, stats.parts[0] * 0.25, stats.parts[0] * 0.25])
    stats3 = ops.RowStats(parts.contiguous(), 3)
    wf = (w.float() * g.float()[None, :]).bfloat16()
    normed = a.float() * torch.rsqrt(a.float().pow(2).mean(-1, keepdim=True) + 1e-5)
    want = normed @ wf.float().t()
    bias = _randn(n)
    res = _randn(m, n)
    got = ops.gemm(a, wf, row_stats=stats3, eps=1e-5, bias=bias, residual=res)
    expect_close(got.float(), want + bias.float() + res.float(), atol=3e-2, rtol=2e-2, min_close=0.999)
    # SwiGLU on top of the row scale
    want_act = torch.nn.functional.silu(want[:, : n // 2]) * want[:, n // 2:]
    act = ops.gemm(a, ops.interleave_gate_up(wf), row_stats=stats, eps=1e-5, swiglu=True)
    assert act.shape == (m, n // 2)
    expect_close(act.float(), want_act, atol=3e-2, rtol=3e-2, min_close=0.998)
    # SwiGLU alone equals the separate kernel on the rounded GEMM output, up to that rounding
    act2 = ops.gemm(a, ops.interleave_gate_up(w), swiglu=True)
    expect_close(act2.float(), ref.swiglu((a.float() @ w.float().t()).bfloat16()).float(), atol=3e-2, rtol=3e-2, min_close=0.998)


@pytest.mark.parametrize("m,n,k", EPI_SHAPES)
def test_gemm_emits_row_statistics_of_its_output(m, n, k):
    torch.manual_seed(m * 3 + n)
    a = _randn(m, k)
    w = _randn(n, k, scale=1.0 / math.sqrt(k))
    res = _randn(m, n)
    out, stats = ops.gemm(a, w, residual=res, emit_stats=True)
    expect_close(out.float(), a.float() @ w.float().t() + res.float(), atol=3e-2, rtol=2e-2, min_close=0.999)
    # the statistics describe the stored (rounded) output exactly, up to fp32 summation order
    expect_close(stats.total(), out.float().pow(2).sum(-1), atol=1e-2, rtol=1e-4, min_close=1.0)
    # twice: same bits (fixed summation order), also in place on the residual
    out2, stats2 = ops.gemm(a, w, residual=res, emit_stats=True)
    assert torch.equal(out, out2) and stats.n == stats2.n and torch.equal(stats.parts[:stats.n], stats2.parts[:stats2.n])
    inplace = res.clone()
    out3, stats3 = ops.gemm(a, w, residual=inplace, out=inplace, emit_stats=True, prefetch=w)
    assert torch.equal(out3, out) and torch.equal(stats3.total(), stats.total())


ALL = 1 - 1e-9      # every value: the share is a mean on the GPU, a product with 1 / n that may round below one


@pytest.mark.parametrize("m,n,k", [(1, 16, 64), (3, 17, 72), (8, 130, 1032), (5, 4800, 2056), (7, 96, 4096), (9, 17, 72), (12, 4800, 1032), (16, 130, 2056),
                                   (16, 4800, 2056), (13, 1040, 8200)])
def test_gemm_few_tokens(m, n, k):
    """The kernel of up to 16 tokens at the edges of its tiles (16 rows, 1024 columns, more tiles than CTAs), all epilogues, against fp32:
    a bf16 rounding of a result of size one (2^-9), a few of them at size four."""
    torch.manual_seed(m + n)
    a, w, bias = _randn(m, k), _randn(n, k, scale=1.0 / math.sqrt(k)), _randn(n)
    base = a.float() @ w.float().t()
    expect_close(ops.gemm(a, w, out_dtype=torch.float32, static_w=True), base, atol=1e-4, rtol=1e-4, min_close=ALL)
    res = torch.randn(m, (n + 7) // 8 * 8, device=DEV).bfloat16()[:, :n]
    want = torch.relu(base + bias.float() + res.float()).square()
    got = ops.gemm(a, w, bias=bias, residual=res, act="relu2")
    expect_close(got.float(), want, atol=2e-2, rtol=2e-2, min_close=ALL)
    scale = torch.rsqrt(a.float().pow(2).mean(-1, keepdim=True) + 1e-5)
    inplace = res.clone() if n % 8 == 0 else torch.empty_strided(res.shape, res.stride(), dtype=res.dtype, device=DEV).copy_(res)
    out, stats = ops.gemm(a, w, residual=inplace, out=inplace, row_stats=ops.row_sumsq(a), emit_stats=True)
    expect_close(out.float(), base * scale + res.float(), atol=2e-2, rtol=2e-2, min_close=ALL)
    expect_close(stats.total(), out.float().pow(2).sum(-1), atol=1e-2, rtol=1e-4, min_close=ALL)
    if n % 2 == 0:
        act = ops.gemm(a, ops.interleave_gate_up(w), row_stats=ops.row_sumsq(a), swiglu=True)
        sc = base * scale
        expect_close(act.float(), torch.nn.functional.silu(sc[:, :n // 2]) * sc[:, n // 2:], atol=2e-2, rtol=2e-2, min_close=ALL)


@pytest.mark.parametrize("m,n,k", [(100, 5128, 2048), (129, 264, 72), (200, 136, 2048), (257, 264, 64), (512, 2048, 576), (300, 3080, 712), (770, 5128, 1024)])
def test_gemm_pair_tiles(m, n, k):
    """The two-SM kernel's three tile widths with ragged last tiles, from the fewest tokens it takes on (one shape of too few columns for
    it), its statistics and SwiGLU; also behind a kernel that writes its input, with the weights requested early."""
    torch.manual_seed(n)
    a, w, res = _randn(m, k), _randn(n, k, scale=1.0 / math.sqrt(k)), _randn(m, n)
    base = a.float() @ w.float().t()
    out, stats = ops.gemm(a, w, residual=res, emit_stats=True, static_w=True)
    expect_close(out.float(), base + res.float(), atol=3e-2, rtol=2e-2, min_close=ALL)
    expect_close(stats.total(), out.float().pow(2).sum(-1), atol=1e-2, rtol=1e-4, min_close=ALL)
    scale = torch.rsqrt(a.float().pow(2).mean(-1, keepdim=True) + 1e-5)
    b = torch.empty_like(a)
    for _ in range(3):
        b.copy_(a)
        sc = base * scale
        act = ops.gemm(b, ops.interleave_gate_up(w), row_stats=ops.row_sumsq(b), swiglu=True, static_w=True)
        expect_close(act.float(), torch.nn.functional.silu(sc[:, :n // 2]) * sc[:, n // 2:], atol=3e-2, rtol=2e-2, min_close=ALL)
        b.zero_()


@pytest.mark.parametrize("m,n", [(3, 264), (40, 264), (70, 264), (70, 4104), (128, 264), (200, 136), (200, 264), (300, 264), (300, 136), (600, 520)])
def test_gemm_unaligned_output(m, n):
    """Outputs and residuals whose rows do not start on 16 bytes: float32 rows of an odd stride, views that begin 4 bytes into a buffer;
    what lies around them stays as it was."""
    torch.manual_seed(m + n)
    k = 320
    a, w, bias = _randn(m, k), _randn(n, k, scale=1.0 / math.sqrt(k)), _randn(n)
    base = a.float() @ w.float().t() + bias.float()
    buf = torch.full((m, n + 3), 7.0, device=DEV)
    expect_close(ops.gemm(a, w, bias=bias, out=buf[:, 1:n + 1]), base, atol=1e-4, rtol=1e-4, min_close=ALL)
    assert bool((buf[:, 0] == 7).all() and (buf[:, n + 1:] == 7).all())
    flat, rflat = torch.full((m * (n + 8) + 8,), 7.0, dtype=torch.bfloat16, device=DEV), _randn(m * (n + 8) + 8)
    out, res = (f[2:2 + m * (n + 8)].view(m, n + 8)[:, :n] for f in (flat, rflat))
    want = base + res.float()
    expect_close(ops.gemm(a, w, bias=bias, residual=res, out=out).float(), want, atol=3e-2, rtol=2e-2, min_close=ALL)
    assert bool((flat[:2] == 7).all() and (flat[2:2 + m * (n + 8)].view(m, n + 8)[:, n:] == 7).all())
    expect_close(ops.gemm(a, w, bias=bias, residual=res, out=res).float(), want, atol=3e-2, rtol=2e-2, min_close=ALL)
    act = flat[2:2 + m * (n + 8)].view(m, n + 8)[:, :n // 2]
    gu = a.float() @ w.float().t()
    expect_close(ops.gemm(a, ops.interleave_gate_up(w), out=act, swiglu=True).float(), torch.nn.functional.silu(gu[:, :n // 2]) * gu[:, n // 2:], atol=3e-2, rtol=2e-2,
                 min_close=ALL)


@pytest.mark.parametrize("rows,d", [(1, 2048), (33, 4096), (64, 8192), (5, 1024 + 8), (3, 16384)])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm(rows, d, with_res):
    x = _randn(rows, d)
    w = _randn(d)
    r = _randn(rows, d) if with_res else None
    got = ops.rmsnorm(x, w, 1e-5, residual=r, unit_offset=with_res)
    want = ref.rmsnorm(x, w, 1e-5, residual=r, unit_offset=with_res)
    if with_res:
        expect_close(got[0].float(), want[0].float(), atol=2e-2, rtol=2e-2)
        assert torch.equal(got[1], want[1])
    else:
        expect_close(got.float(), want.float(), atol=2e-2, rtol=2e-2)


def test_swiglu_embedding_argmax():
    gu = _randn(37, 2 * 1024)
    expect_close(ops.swiglu(gu).float(), ref.swiglu(gu).float(), atol=1e-2, rtol=2e-2)
    table = _randn(1000, 512)
    ids = torch.randint(0, 1000, (4, 9), device=DEV, dtype=torch.int32)
    assert torch.equal(ops.embedding(ids, table), table[ids.long()])
    logits = torch.randn(17, 128256, device=DEV)
    logits[3, 77] = 100.0
    logits[3, 99] = 100.0   # tie -> lowest index
    got = ops.argmax(logits)
    assert got[3].item() == 77
    assert torch.equal(got.long(), torch.argmax(logits, -1)) or got[3].item() == 77


@pytest.mark.parametrize("k", [1, 8, 50, 128])
def test_topk_sample(k):
    torch.manual_seed(1)
    logits = torch.randn(9, 32000, device=DEV)
    logits[0, :100] = float("-inf")
    tok, vals, idx = ops.topk_sample(logits, k, temperature=0.8, seed=5, step=2, return_topk=True)
    wv, wi = torch.topk(logits, k, dim=-1)
    assert torch.equal(vals, wv)
    assert torch.equal(idx.long(), wi)
    # the drawn token is one of the top-k
    assert all(int(tok[i]) in set(wi[i].tolist()) for i in range(logits.shape[0]))
    if k == 1:
        assert torch.equal(tok.long(), torch.argmax(logits, -1))
    # frequency check of the Gumbel-max draw on a tiny distribution
    if k == 8:
        small = torch.full((1, 64), -30.0, device=DEV)
        small[0, :4] = torch.tensor([2.0, 1.0, 0.0, -1.0], device=DEV)
        counts = torch.zeros(64)
        n = 2000
        for s in range(n):
            counts[int(ops.topk_sample(small, 8, 1.0, seed=11, step=s))] += 1
        p = torch.softmax(small[0].cpu(), -1)
        assert torch.allclose(counts / n, p, atol=0.04)


def test_topk_of_merged_candidates_equals_topk_of_the_whole_row():
    """What vocab-parallel top-k sampling does: every shard ranks its own columns, the k best of the union of the
    shards' k best are the k best of the row, and the draw on the merged candidates is the draw on the whole row."""
    torch.manual_seed(4)
    k, shards, v_per = 4, 2, 500
    logits = torch.randn(6, shards * v_per, device=DEV)
    logits[:, -3:] = float("-inf")                       # padding columns of the last shard
    cand_v, cand_i = [], []
    for r in range(shards):
        v, i = ops.topk(logits[:, r * v_per:(r + 1) * v_per].contiguous(), k)
        cand_v.append(v)
        cand_i.append(i + r * v_per)
    cand_v, cand_i = torch.cat(cand_v, 1).contiguous(), torch.cat(cand_i, 1)
    assert cand_v.shape == (6, shards * k)
    pos, mv, mi = ops.topk_sample(cand_v, k, temperature=0.7, seed=3, step=9, return_topk=True)
    tok, wv, wi = ops.topk_sample(logits, k, temperature=0.7, seed=3, step=9, return_topk=True)
    assert torch.equal(mv, wv) and torch.equal(cand_i.gather(1, mi.long()), wi)
    assert torch.equal(cand_i.gather(1, pos.long()[:, None])[:, 0], tok)


def _make_paged(batch, seq_lens, hkv, hd, page, extra_pages=3):
    """Random paged cache with a shuffled page assignment."""
    max_pages = max((l + page - 1) // page for l in seq_lens) + 1
    total = sum((l + page - 1) // page for l in seq_lens) + extra_pages
    perm = torch.randperm(total)
    bt = torch.zeros(batch, max_pages, dtype=torch.int32)
    nxt = 0
    for i, l in enumerate(seq_lens):
        n = (l + page - 1) // page
        bt[i, :n] = perm[nxt:nxt + n].to(torch.int32)
        nxt += n
    kc = _randn(total, page, hkv, hd)
    vc = _randn(total, page, hkv, hd)
    return kc, vc, bt.to(DEV)


@pytest.mark.parametrize("hq,hkv,hd", [(32, 8, 64), (32, 8, 128), (8, 1, 128), (16, 16, 64), (16, 2, 256)])
@pytest.mark.parametrize("page", [64, 16])
def test_paged_decode(hq, hkv, hd, page):
    torch.manual_seed(3)
    seq_lens = [1, 17, 64, 65, 300, 1000, 2049]
    b = len(seq_lens)
    kc, vc, bt = _make_paged(b, seq_lens, hkv, hd, page)
    q = _randn(b, hq, hd)
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=DEV)
    want = ref.paged_decode(q, kc, vc, bt, seq_lens)
    for splits in (1, 4, None):
        got = ops.paged_decode(q, kc, vc, bt, sl, num_splits=splits)
        expect_close(got.float(), want.float(), atol=2e-2, rtol=2e-2, min_close=0.995)
    got = ops.paged_decode(q, kc, vc, bt, sl, window=128, num_splits=2)
    want_w = ref.paged_decode(q, kc, vc, bt, seq_lens, window=128)
    expect_close(got.float(), want_w.float(), atol=2e-2, rtol=2e-2, min_close=0.995)


@pytest.mark.parametrize("hq,hkv,hd", [(32, 8, 64), (8, 2, 128), (4, 4, 256)])
def test_paged_prefill_mixed_batch(hq, hkv, hd):
    """Mixed batch as in the reference's pagedAttention test: fresh prompts, a chunked
    continuation (context already cached), a single-token row and an empty row."""
    torch.manual_seed(4)
    page = 64
    q_lens = [5, 64, 130, 1, 0, 257]
    ctx = [0, 0, 70, 99, 0, 64]
    seq_lens = [a + c for a, c in zip(q_lens, ctx)]
    b = len(q_lens)
    kc, vc, bt = _make_paged(b, seq_lens, hkv, hd, page)
    qs = [0]
    for l in q_lens:
        qs.append(qs[-1] + l)
    q = _randn(qs[-1], hq, hd)
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=DEV)
    qst = torch.tensor(qs, dtype=torch.int32, device=DEV)
    got = ops.paged_prefill(q, kc, vc, bt, sl, qst)
    want = ref.paged_attention(q, kc, vc, bt, seq_lens, qs)
    expect_close(got.float(), want.float(), atol=2e-2, rtol=2e-2, min_close=0.995)
    got = ops.paged_prefill(q, kc, vc, bt, sl, qst, window=100)
    want = ref.paged_attention(q, kc, vc, bt, seq_lens, qs, window=100)
    expect_close(got.float(), want.float(), atol=2e-2, rtol=2e-2, min_close=0.995)


@pytest.mark.parametrize("hq,hkv,lens", [(8, 2, [(2048, 0), (300, 1700)]), (4, 1, [(129, 0), (64, 64), (7, 500)]), (16, 8, [(1000, 24)])])
def test_paged_prefill_tensor_core_kernel(hq, hkv, lens):
    """The tcgen05 prefill kernel (head_dim 128, 64-token pages, two query heads of a KV group per CTA) against the
    float32 reference and against the mma.sync kernel: long prompts, chunked continuations, ragged tails."""
    torch.manual_seed(6)
    hd, page = 128, 64
    q_lens = [a for a, _ in lens]
    seq_lens = [a + c for a, c in lens]
    kc, vc, bt = _make_paged(len(lens), seq_lens, hkv, hd, page)
    qs = [0]
    for n in q_lens:
        qs.append(qs[-1] + n)
    q = _randn(qs[-1], hq, hd)
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=DEV)
    qst = torch.tensor(qs, dtype=torch.int32, device=DEV)
    for window in (0, 333):
        got = ops.paged_prefill(q, kc, vc, bt, sl, qst, window=window, impl="tc")
        old = ops.paged_prefill(q, kc, vc, bt, sl, qst, window=window, impl="mma")
        want = ref.paged_attention(q, kc, vc, bt, seq_lens, qs, window=window)
        expect_close(got.float(), want.float(), atol=2e-2, rtol=2e-2, min_close=0.995)
        expect_close(got.float(), old.float(), atol=2e-2, rtol=2e-2, min_close=0.995)


@pytest.mark.parametrize("hd,hq,hkv", [(64, 8, 2), (128, 8, 2), (256, 8, 2), (256, 3, 1)])
@pytest.mark.parametrize("lens", [[(1, 0), (63, 0), (64, 1), (65, 63)], [(127, 0), (128, 64), (129, 191)], [(3, 4000), (260, 0)]])
def test_paged_prefill_page_edges(hd, hq, hkv, lens):
    """The tcgen05 prefill kernels at the edges of pages and query blocks, with scores that grow along the keys, so that a row's
    reference moves again and again.  Probabilities and the result round to bf16, 2^-9 of each: at most 2^-8 of the largest value, which is
    below 4.5; a wrong row is off by one and more."""
    torch.manual_seed(9)
    page = 64
    q_lens, seq_lens = [a for a, _ in lens], [a + c for a, c in lens]
    kc, vc, bt = _make_paged(len(lens), seq_lens, hkv, hd, page)
    for i, n in enumerate(seq_lens):                # key t of a sequence is (1 + t / 40) times as large along one direction
        t = torch.arange(n, device=DEV)
        kc[bt[i, t // page].long(), t % page, :, 0] += (1 + t / 40.0).to(torch.bfloat16)[:, None]
    qs = [0]
    for n in q_lens:
        qs.append(qs[-1] + n)
    q = _randn(qs[-1], hq, hd)
    q[:, :, 0] = 4.0
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=DEV)
    qst = torch.tensor(qs, dtype=torch.int32, device=DEV)
    for window in (0, 1, 64, 100):
        got = ops.paged_prefill(q, kc, vc, bt, sl, qst, window=window, impl="tc")
        want = ref.paged_attention(q, kc, vc, bt, seq_lens, qs, window=window)
        expect_close(got.float(), want.float(), atol=2e-2, rtol=2e-2, min_close=ALL)


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("junk", [float("nan"), float("inf"), 3e38])
def test_paged_prefill_ignores_rows_behind_a_sequence(hd, junk):
    """What a page holds behind the end of its sequence, and unused pages, do not reach the result: to the bit that of a clean cache."""
    torch.manual_seed(hd)
    hq, hkv, page = 4, 2, 64
    parts = [(1, 0), (63, 0), (64, 64), (65, 63), (130, 70), (3, 700), (200, 120)]          # tokens, tokens in the cache
    q_lens, seq_lens = [n for n, _ in parts], [n + c for n, c in parts]
    kc, vc, bt = _make_paged(len(parts), seq_lens, hkv, hd, page)
    used = torch.zeros(kc.shape[:2], dtype=torch.bool, device=DEV)
    for i, n in enumerate(seq_lens):
        t = torch.arange(n, device=DEV)
        used[bt[i, t // page].long(), t % page] = True
    q, qs = _randn(sum(q_lens), hq, hd), [0]
    for n in q_lens:
        qs.append(qs[-1] + n)
    sl, qst = torch.tensor(seq_lens, dtype=torch.int32, device=DEV), torch.tensor(qs, dtype=torch.int32, device=DEV)
    for window in (0, 100):
        kc[~used], vc[~used] = 0.0, 0.0
        clean = ops.paged_prefill(q, kc, vc, bt, sl, qst, window=window, impl="tc")
        kc[~used], vc[~used] = junk, -junk
        assert torch.equal(ops.paged_prefill(q, kc, vc, bt, sl, qst, window=window, impl="tc"), clean)
        assert bool(clean.isfinite().all())


@pytest.mark.parametrize("cap", [0.0, 30.0])
@pytest.mark.parametrize("window,keep", [(0, 0), (100, 3)])
def test_paged_prefill_with_extensions_ignores_rows_behind_a_sequence(cap, window, keep):
    """The same for the kernel with a score cap, a sink and kept first keys."""
    from zml_b200.ops import gqa
    torch.manual_seed(3)
    parts = [(1, 0), (64, 64), (65, 63), (130, 70), (200, 120)]
    q_lens, seq_lens = [n for n, _ in parts], [n + c for n, c in parts]
    kc, vc, bt = _make_paged(len(parts), seq_lens, 2, 128, 64)
    used = torch.zeros(kc.shape[:2], dtype=torch.bool, device=DEV)
    for i, n in enumerate(seq_lens):
        t = torch.arange(n, device=DEV)
        used[bt[i, t // 64].long(), t % 64] = True
    q, qs = _randn(sum(q_lens), 4, 128), [0]
    for n in q_lens:
        qs.append(qs[-1] + n)
    sl, qst = torch.tensor(seq_lens, dtype=torch.int32, device=DEV), torch.tensor(qs, dtype=torch.int32, device=DEV)
    ext, res = gqa.AttnExt(keep, cap, 1, 128, None, 0, 0), []
    assert ops.prefill_on_tc(q, kc, ext)
    for junk in (0.0, float("nan"), float("inf")):
        kc[~used], vc[~used] = junk, -junk
        res.append(ops.paged_prefill(q, kc, vc, bt, sl, qst, window=window, out=torch.empty_like(q), ext=ext))
    assert bool(res[0].isfinite().all()) and torch.equal(res[1], res[0]) and torch.equal(res[2], res[0])


@pytest.mark.parametrize("hd,hq,hkv", [(64, 8, 2), (64, 64, 8), (128, 4, 2), (256, 3, 1)])
@pytest.mark.parametrize("seqs,longest", [(1, 1), (3, 128), (9, 129), (40, 64), (60, 100)])
def test_paged_prefill_routes_of_short_prompts(hd, hq, hkv, seqs, longest):
    """Short prompts, few and many, on whichever kernel the rule takes; `max_seq_len` and a wide block table change no more than the kernel."""
    torch.manual_seed(seqs)
    seq_lens = [longest - i * longest // (2 * seqs) for i in range(seqs)]
    qs = [0]
    for n in seq_lens:
        qs.append(qs[-1] + n)
    kc, vc, bt = _make_paged(seqs, seq_lens, hkv, hd, 64)
    sl, qst, q = torch.tensor(seq_lens, dtype=torch.int32, device=DEV), torch.tensor(qs, dtype=torch.int32, device=DEV), _randn(qs[-1], hq, hd)
    want = ref.paged_attention(q, kc, vc, bt, seq_lens, qs).float()
    for kw in (dict(max_seq_len=longest), {}, dict(impl="mma")):
        # probabilities and the result round to bf16: 2 * 2^-9 of a result of size one
        expect_close(ops.paged_prefill(q, kc, vc, bt, sl, qst, **kw).float(), want, atol=2e-2, rtol=2e-2, min_close=ALL)


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("scale", [-0.2, 0.0])
def test_paged_prefill_scale_below_zero(hd, scale):
    torch.manual_seed(hd)
    seq_lens, qs = [70, 200], [0, 70, 200]
    kc, vc, bt = _make_paged(2, seq_lens, 2, hd, 64)
    sl, qst = torch.tensor(seq_lens, dtype=torch.int32, device=DEV), torch.tensor(qs, dtype=torch.int32, device=DEV)
    q = _randn(200, 4, hd)
    want = ref.paged_attention(q, kc, vc, bt, seq_lens, qs, scale)
    expect_close(ops.paged_prefill(q, kc, vc, bt, sl, qst, scale).float(), want.float(), atol=2e-2, rtol=2e-2, min_close=ALL)


@pytest.mark.parametrize("hd", [64, 128, 256])
def test_paged_prefill_alignment(hd):
    """An `out` that does not start on 16 bytes goes to the kernel that stores 4 at a time; inputs that do not are refused."""
    torch.manual_seed(hd)
    seq_lens, qs = [70, 130], [0, 70, 200]
    kc, vc, bt = _make_paged(2, seq_lens, 2, hd, 64)
    sl, qst = torch.tensor(seq_lens, dtype=torch.int32, device=DEV), torch.tensor(qs, dtype=torch.int32, device=DEV)
    q = _randn(200, 4, hd)
    want = ref.paged_attention(q, kc, vc, bt, seq_lens, qs)
    flat = torch.zeros(q.numel() + 8, dtype=torch.bfloat16, device=DEV)
    out = flat[4:4 + q.numel()].view(q.shape)
    expect_close(ops.paged_prefill(q, kc, vc, bt, sl, qst, out=out).float(), want.float(), atol=2e-2, rtol=2e-2, min_close=ALL)
    assert not flat[:4].any() and not flat[4 + q.numel():].any()

    def moved(t):
        return torch.zeros(t.numel() + 8, dtype=t.dtype, device=DEV)[4:4 + t.numel()].view(t.shape)
    for args in ((moved(q), kc, vc), (q, moved(kc), vc), (q, kc, moved(vc))):
        with pytest.raises(ValueError):
            ops.paged_prefill(*args, bt, sl, qst)
    with pytest.raises(ValueError):
        ops.paged_prefill(q, kc, vc, bt, sl, qst, out=out, impl="tc")
    one = torch.tensor([0, 1], dtype=torch.int32, device=DEV)
    row = q[:1].as_strided((1, 4, hd), (4 * hd + 3, hd, 1))            # the stride of a single row says nothing about where rows start
    want = ref.paged_attention(q[:1], kc, vc, bt[:1], [70], [0, 1])
    expect_close(ops.paged_prefill(row, kc, vc, bt[:1], sl[:1], one).float(), want.float(), atol=2e-2, rtol=2e-2, min_close=ALL)


@pytest.mark.parametrize("layout,rot", [(0, None), (1, None), (0, 32), (2, 32)])
@pytest.mark.parametrize("qk_norm", [False, True])
def test_rope_kvwrite(layout, rot, qk_norm):
    torch.manual_seed(5)
    t, hq, hkv, hd, page, pages = 50, 8, 2, 64, 64, 6
    qkv = _randn(t, (hq + 2 * hkv) * hd)
    pos = torch.randint(0, 5000, (t,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(pages * page, device=DEV)[:t].to(torch.int32)
    slots[7] = -1
    half = (rot or hd) // 2
    inv_freq = (1.0 / (10000.0 ** (torch.arange(half, device=DEV).float() / half))).contiguous()
    qn = _randn(hd) if qk_norm else None
    kn = _randn(hd) if qk_norm else None
    kc = torch.zeros(pages, page, hkv, hd, device=DEV, dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    kc2, vc2 = kc.clone(), vc.clone()
    q = ops.rope_kvwrite(qkv, pos, slots, inv_freq, kc, vc, hq, hkv, hd, layout, rot, 1.0, qn, kn, 1e-6, qk_norm)
    q2 = ref.rope_kvwrite(qkv, pos, slots, inv_freq, kc2, vc2, hq, hkv, hd, layout, rot, 1.0, qn, kn, 1e-6, qk_norm)
    expect_close(q.float(), q2.float(), atol=3e-2, rtol=2e-2, min_close=0.995)
    expect_close(kc.float(), kc2.float(), atol=3e-2, rtol=2e-2, min_close=0.995)
    assert torch.equal(vc, vc2)


@pytest.mark.parametrize("hd,rot,hq,hkv,qk_norm", [(64, 64, 5, 1, True), (128, 128, 32, 8, False), (256, 64, 4, 1, True), (128, 48, 3, 3, True), (64, 16, 70, 2, False), (128, 128, 64, 8, True)])
def test_rope_rows(hd, rot, hq, hkv, qk_norm):
    """The 16-byte form: heads that do not fill a warp, more pieces than threads, partial rotation, strided input, padding rows.  Single values
    differ by a rounding of the normalised value (2^-8 of up to twenty); a wrong 16-byte piece is off by one and more in all eight."""
    torch.manual_seed(hd + rot)
    t, page, pages = 9, 64, 3
    qkv = _randn(t, (hq + 2 * hkv) * hd + 16)[:, :(hq + 2 * hkv) * hd]
    pos = torch.randint(0, 5000, (t,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(pages * page, device=DEV)[:t].to(torch.int32)
    slots[4] = -1
    inv_freq = (1.0 / (10000.0 ** (torch.arange(rot // 2, device=DEV).float() / (rot // 2)))).contiguous()
    qn, kn = (_randn(hd), _randn(hd)) if qk_norm else (None, None)
    kc = torch.zeros(pages, page, hkv, hd, device=DEV, dtype=torch.bfloat16)
    vc, kc2, vc2 = kc.clone(), kc.clone(), kc.clone()
    q = ops.rope_kvwrite(qkv, pos, slots, inv_freq, kc, vc, hq, hkv, hd, 0, rot, 1.1, qn, kn, 1e-6, qk_norm)
    q2 = ref.rope_kvwrite(qkv, pos, slots, inv_freq, kc2, vc2, hq, hkv, hd, 0, rot, 1.1, qn, kn, 1e-6, qk_norm)
    for got, want in ((q, q2), (kc, kc2)):
        expect_close(got.float(), want.float(), atol=3e-2, rtol=2e-2, min_close=0.995)
        assert float((got.float() - want.float()).abs().reshape(-1, 8).mean(-1).max()) < 0.1
    assert torch.equal(vc, vc2)


@pytest.mark.parametrize("rows,vocab", [(1, 128256), (40, 32773), (200, 4099), (3, 1000), (2, 40), (5, 24001), (100, 65537)])
def test_topk_and_argmax_over_clusters(rows, vocab):
    """Rows cut over clusters of 8, 4 and 1: random, rising, falling, all equal and lowest logits against a stable sort (equal logits: the
    lower index first)."""
    torch.manual_seed(vocab)
    ramp = torch.arange(vocab, device=DEV).float().expand(rows, vocab).contiguous()
    for lg in (torch.randn(rows, vocab, device=DEV) * 2.5, ramp, -ramp, ramp % 7, torch.full_like(ramp, torch.finfo(torch.float32).min)):
        v, i = torch.sort(lg, dim=1, descending=True, stable=True)
        assert torch.equal(ops.argmax(lg).long(), i[:, 0])
        for k in (1, 33, 40):
            _, got_v, got_i = ops.topk_sample(lg, k, 0.7, seed=1, return_topk=True)
            assert torch.equal(got_v, v[:, :k]) and torch.equal(got_i.long(), i[:, :k])


# ---------------------------------------------------------------------------- MoE
def test_moe_router_topk():
    from zml_b200 import moe
    torch.manual_seed(7)
    for e, k in ((128, 8), (64, 4), (256, 8)):
        logits = torch.randn(77, e, device=DEV)
        ids, w = moe.router_topk(logits, k)
        wv, wi = torch.topk(logits, k, dim=-1)
        assert torch.equal(ids.long(), wi)
        expect_close(w, torch.softmax(wv, -1), atol=1e-5, rtol=1e-4)
        ids2, w2 = moe.router_topk(logits, k, renormalize=False)
        expect_close(w2, torch.softmax(logits, -1).gather(1, wi), atol=1e-6, rtol=1e-4)


@pytest.mark.parametrize("t,e_total,e_local,e0,k,d,f", [
    (128, 128, 16, 32, 8, 512, 256),       # decode-like: ~8 tokens per expert -> swap-AB tiles
    (7, 16, 16, 0, 2, 256, 128),
    (1500, 8, 8, 0, 2, 256, 256),          # prefill-like: token-major tiles
    (640, 32, 8, 8, 4, 384, 128),
])
def test_moe_fused_experts_vs_dense_reference(t, e_total, e_local, e0, k, d, f):
    from zml_b200 import moe
    torch.manual_seed(11)
    x = _randn(t, d)
    gate = _randn(e_local, f, d, scale=1.0 / math.sqrt(d))
    up = _randn(e_local, f, d, scale=1.0 / math.sqrt(d))
    down = _randn(e_local, d, f, scale=1.0 / math.sqrt(f))
    logits = torch.randn(t, e_total, device=DEV)
    ids, w = moe.router_topk(logits, k)
    want = moe.reference_fused_experts(x, ids, w, gate, up, down, e0)
    got = moe.fused_experts(x, ids, w, moe.interleave_gate_up(gate, up), down, e0, e_total)
    expect_close(got.float(), want.float(), atol=3e-2, rtol=3e-2, min_close=0.995)
    # the CPU restatement of the same pipeline agrees as well
    cpu = moe.fused_experts(x.cpu(), ids.cpu(), w.cpu(), moe.interleave_gate_up(gate, up).cpu(), down.cpu(), e0, e_total)
    expect_close(cpu.float(), want.float().cpu(), atol=3e-2, rtol=3e-2, min_close=0.995)


def test_moe_combine_adds_extra_and_residual():
    """One-launch combine == finalize + shared-expert partial + residual."""
    from zml_b200 import moe
    torch.manual_seed(3)
    t, k, d, e = 37, 4, 512, 16
    ids, w = moe.router_topk(torch.randn(t, e, device=DEV), k)
    meta, sorted_pair, pair_pos = moe.moe_align(ids, 4, 8)            # half of the experts are "remote"
    o = _randn(t * k, d)
    extra, res = _randn(t, d), _randn(t, d)
    want = moe.finalize(o, pair_pos, w, t, k).float() + extra.float() + res.float()
    got = moe.combine(o, pair_pos, w, t, k, extra, res)
    expect_close(got.float(), want, atol=3e-2, rtol=2e-2)
    only = moe.combine(o, pair_pos, w, t, k)
    assert torch.equal(only, moe.finalize(o, pair_pos, w, t, k))
    cpu = moe.combine(o.cpu(), pair_pos.cpu(), w.cpu(), t, k, extra.cpu(), res.cpu())
    expect_close(cpu.float(), want.cpu(), atol=3e-2, rtol=2e-2)


@pytest.mark.parametrize("k", [1, 2, 3, 5, 8, 9])
def test_moe_combine_of_any_number_of_experts(k):
    """Two, four or eight rows at a time: the sums are those of `finalize`, to the bit, half of the experts elsewhere."""
    from zml_b200 import moe
    torch.manual_seed(k)
    t, d = 37, 1032
    ids = torch.stack([torch.randperm(16, device=DEV)[:k] for _ in range(t)]).int()
    _, _, pair_pos = moe.moe_align(ids, 4, 8)
    o, w = _randn(t * k, d), torch.rand(t, k, device=DEV)
    assert torch.equal(moe.combine(o, pair_pos, w, t, k), moe.finalize(o, pair_pos, w, t, k))


@pytest.mark.parametrize("t,k,d", [(511, 8, 64), (512, 1, 2056), (515, 9, 1024), (700, 8, 4104)])
def test_moe_gather_by_tokens(t, k, d):
    """The expert rows gathered from the tokens' side (from 512 tokens on) are those of the gather by rows, half of the experts elsewhere."""
    from zml_b200 import moe
    torch.manual_seed(t)
    x, ids = _randn(t, d), torch.stack([torch.randperm(16, device=DEV)[:k] for _ in range(t)]).int()
    meta, sorted_pair, pair_pos = moe.moe_align(ids, 4, 8)
    rows = int(meta[8])
    want = x[sorted_pair[:rows].long() // k]
    assert torch.equal(moe.gather(x, sorted_pair, meta, 8, k, t * k, pair_pos)[:rows], want)
    assert torch.equal(moe.gather(x, sorted_pair, meta, 8, k, t * k)[:rows], want)


@pytest.mark.parametrize("tokens", [1, 333, 1365, 3000])       # up to 8192 pairs: one launch; above: count / prefix / scatter
def test_moe_align_is_a_permutation(tokens):
    from zml_b200 import moe
    torch.manual_seed(tokens)
    ids = torch.randint(0, 64, (tokens, 6), device=DEV, dtype=torch.int32)
    meta, sorted_pair, pair_pos = moe.moe_align(ids, 16, 24)
    flat = ids.reshape(-1).cpu()
    local = (flat >= 16) & (flat < 40)
    n = int(local.sum())
    m = meta.cpu()
    assert int(m[24]) == n
    sp = sorted_pair.cpu()[:n].long()
    assert sorted(sp.tolist()) == local.nonzero()[:, 0].tolist()
    e_of_row = flat[sp] - 16
    assert torch.equal(e_of_row, torch.sort(e_of_row).values)          # grouped by expert
    counts = torch.bincount(e_of_row, minlength=24)
    assert torch.equal(m[1:25] - m[:24], counts.to(torch.int32))
    pp = pair_pos.cpu()
    assert (pp[~local] == -1).all() and torch.equal(pp[sp], torch.arange(n, dtype=torch.int32))


_BOUNDS_WORKER = r"""
import os, sys, torch
sys.path.insert(0, os.environ["ZB_ROOT"])
from zml_b200 import ops
from zml_b200.ops import _lib
assert _lib.bounds_check_build(), "the bounds-checking library is not the one that was loaded"   # nothing below runs otherwise
dev = "cuda"
g = torch.Generator(device=dev).manual_seed(0)
bf = lambda *s: (torch.randn(*s, device=dev, generator=g) * 0.5).to(torch.bfloat16)
i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)

# the small-shape kernel cases run clean under the checks
a, w = bf(8, 256), bf(384, 256)
assert torch.allclose(ops.gemm(a, w).float(), a.float() @ w.float().t(), atol=0.5, rtol=0.05)
x = bf(4, 256)
ops.rmsnorm(x, torch.ones(256, device=dev, dtype=torch.bfloat16))
table = bf(100, 64)
assert torch.equal(ops.embedding(i32([3, 99, 0]), table), table[[3, 99, 0]])
hq, hkv, hd, page, pages = 4, 2, 64, 16, 8
_lib.set_bounds_extents(pages, 0)
kc = torch.zeros(pages, page, hkv, hd, device=dev, dtype=torch.bfloat16)
vc = torch.zeros_like(kc)
inv = torch.rand(hd // 2, device=dev)
qkv = bf(3, (hq + 2 * hkv) * hd)
ops.rope_kvwrite(qkv, i32([0, 1, 2]), i32([16, 17, -1]), inv, kc, vc, hq, hkv, hd)
q = bf(2, hq, hd)
ops.paged_decode(q, kc, vc, i32([[1, 2, 0, 0], [3, 0, 0, 0]]), i32([20, 5]))
ops.raise_on_status()
print("CLEAN", flush=True)

def expect(kernel, index, fn):
    fn()
    try:
        ops.raise_on_status()
    except _lib.BoundsError as e:
        assert e.kernel == kernel and e.index == index, (e.kernel, e.site, e.index)
        print("CAUGHT", kernel, index, flush=True)
        return
    raise AssertionError(f"{kernel}: index {index} was not reported")

# a token id past the vocabulary, a KV slot past the cache, a page number past the pool: reported, not accessed
expect("embedding", 100, lambda: ops.embedding(i32([3, 100]), table))
expect("rope_kvwrite", pages * page + 5, lambda: ops.rope_kvwrite(qkv, i32([0, 1, 2]), i32([16, pages * page + 5, -1]), inv, kc, vc, hq, hkv, hd))
expect("paged_decode", 4000, lambda: ops.paged_decode(q, kc, vc, i32([[1, 4000, 0, 0], [3, 0, 0, 0]]), i32([20, 5])))
# and the context is intact
assert torch.equal(ops.embedding(i32([5]), table), table[[5]])
ops.raise_on_status()
print("BOUNDS_OK", flush=True)
"""


@pytest.mark.gpu
def test_bounds_checking_build_reports_bad_indices(tmp_path):
    """The same sources built with -DZB_BOUNDS_CHECK (libzb_cuda_bc.so): small-shape cases run clean, and an index
    read from memory that lies outside its extent is recorded in the status word (kernel, site, index) and the
    access skipped, where the normal build masks it silently.  Runs in a process of its own, which loads the
    checking library through ZB_CUDA_LIB and verifies that before it feeds any bad index."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    so = os.path.join(root, "zml_b200", "_C", "libzb_cuda_bc.so")
    if not os.path.exists(so):
        from zml_b200 import _build
        _build.build_cuda(extra_flags=["-DZB_BOUNDS_CHECK", "-rdc=true"], variant="bc")
    script = tmp_path / "w.py"
    script.write_text(_BOUNDS_WORKER)
    r = subprocess.run([sys.executable, str(script)], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, ZB_ROOT=root, ZB_CUDA_LIB=so))
    assert r.returncode == 0 and "BOUNDS_OK" in r.stdout, r.stdout[-1500:] + r.stderr[-2500:]
    assert r.stdout.count("CAUGHT") == 3


@pytest.mark.gpu
def test_platform_cuda_options_cap_and_preallocate():
    """`CudaOptions.memory_fraction` caps the process's share of the device, `preallocate` reserves it at start-up."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = r"""
import sys, torch
sys.path.insert(0, %r)
from zml_b200.platform import CreateOptions, CudaOptions, Platform, Target
p = Platform.init(Target.cuda, CreateOptions(cuda=CudaOptions(memory_fraction=0.02, preallocate=True)))
total = torch.cuda.mem_get_info()[1]
assert torch.cuda.memory_reserved() >= 0.01 * total
try:
    torch.empty(int(0.05 * total), dtype=torch.uint8, device="cuda")
    print("NOT CAPPED")
except torch.OutOfMemoryError:
    print("CAPPED")
""" % root
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "CAPPED" in r.stdout and "NOT CAPPED" not in r.stdout, r.stdout + r.stderr[-1500:]
