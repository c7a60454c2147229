"""GPU parity: split-K GQA paged-attention decode against the per-request oracle
(softmax(q k^T / sqrt(D)) v over the request's own cached rows, src/models/llama.zig:231-270).

Tolerance (bf16 outputs): max |diff| / max |ref| <= 2e-2 and cosine >= 0.9995."""
import numpy as np
import pytest
import torch

from oracle import ref_math

pytestmark = pytest.mark.gpu

REL_TOL, COS_TOL = 2e-2, 0.9995


def _close(got, want):
    g, w = got.astype(np.float64).reshape(-1), want.astype(np.float64).reshape(-1)
    rel = np.abs(g - w).max() / max(np.abs(w).max(), 1e-30)
    cos = g @ w / (np.linalg.norm(g) * np.linalg.norm(w) + 1e-30)
    return rel, cos


def _run_case(ctxs, hq, hkv, d, kv_dtype, seed, scatter=True, pages_per_chunk=0, path=0):
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(seed)
    n = len(ctxs)
    pages = sum(-(-c // 32) for c in ctxs)
    n_pages = int(pages * 1.25) + 2
    kv = dev.PagedKVCache(1, hkv, d, n_pages, n, max(-(-max(ctxs) // 32), 1), hq, max_rows=max(sum(ctxs), n, 1),
                          kv_dtype=kv_dtype)
    dev.set_attn_pages_per_chunk(pages_per_chunk)
    dev.set_attn_path(path)
    if scatter:
        kv.set_free_order(rng.permutation(n_pages).tolist())
    k = ref_math.bf16_round(rng.normal(0, 1, (sum(ctxs), hkv, d)).astype(np.float32))
    v = ref_math.bf16_round(rng.normal(0, 1, (sum(ctxs), hkv, d)).astype(np.float32))
    q = ref_math.bf16_round((rng.normal(0, 1, (n, hq, d)) / np.sqrt(d)).astype(np.float32) * np.sqrt(d))
    desc = dev.pack_desc_array([(s, c, 0, -1) for s, c in enumerate(ctxs)]).cuda()
    kv.reserve(desc)
    kv.append(0, torch.tensor(k, device="cuda").bfloat16(), torch.tensor(v, device="cuda").bfloat16())
    row_seq = torch.arange(n, dtype=torch.int32, device="cuda")
    row_ctx = torch.tensor(ctxs, dtype=torch.int32, device="cuda")
    out = kv.attention(0, torch.tensor(q, device="cuda").bfloat16(), row_seq, row_ctx)
    torch.cuda.synchronize()
    assert kv.error_word() == 0
    got = out.float().cpu().numpy()
    if kv_dtype == dev.KV_FP8_E4M3:
        # the oracle for FP8 pools reads what the pool holds: decode(codes) * scale
        kk, vv = [], []
        for s in range(n):
            a, b = kv.gather(0, s)
            kk.append(a.float().cpu().numpy())
            vv.append(b.float().cpu().numpy())
        k_eff, v_eff = np.concatenate(kk) if sum(ctxs) else k, np.concatenate(vv) if sum(ctxs) else v
    else:
        k_eff, v_eff = k, v
    off = 0
    want = np.zeros_like(got)
    for s, c in enumerate(ctxs):
        if c > 0:
            want[s] = ref_math.gqa_attention_decode(q[s], k_eff[off : off + c], v_eff[off : off + c])
        off += c
    kv.close()
    dev.set_attn_path(0)
    dev.set_attn_pages_per_chunk(0)   # back to the automatic choice
    return got, want, (k, v, q)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("kv_dtype,path", [(0, 0), (0, 1), (1, 0), (1, 1)])  # bf16 tensor-core, bf16 CUDA-core, FP8 tensor-core (head_dim 128), FP8 CUDA-core
def test_ragged_contexts(d, kv_dtype, path):
    ctxs = [1, 31, 32, 33, 64, 65, 200, 257, 700, 5, 1023, 96]
    hq, hkv = (8, 2) if d == 64 else (32, 8)
    got, want, _ = _run_case(ctxs, hq, hkv, d, kv_dtype, seed=7 + d + kv_dtype, path=path)
    rel, cos = _close(got, want)
    assert rel <= REL_TOL and cos >= COS_TOL, (rel, cos)
    for s in range(len(ctxs)):  # every row on its own, so a short context cannot hide behind a long one
        r, c = _close(got[s], want[s])
        assert r <= REL_TOL and c >= COS_TOL, (s, ctxs[s], r, c)


def test_fp8_close_to_bf16_oracle():
    """FP8 pools against the bf16 (unquantised) oracle: the quantisation error itself stays inside
    the tolerance the north-star states for bf16 outputs."""
    from dmlx_b200 import device as dev

    ctxs = [300, 1024, 77]
    got, _, (k, v, q) = _run_case(ctxs, 32, 8, 128, dev.KV_FP8_E4M3, seed=99)
    off = 0
    for s, c in enumerate(ctxs):
        want = ref_math.gqa_attention_decode(q[s], k[off : off + c], v[off : off + c])
        rel, cos = _close(got[s], want)
        assert rel <= 6e-2 and cos >= 0.998, (s, rel, cos)  # E4M3 carries 3 mantissa bits
        off += c


@pytest.mark.parametrize("ppc", [4, 8, 32])
@pytest.mark.parametrize("path", [0, 1])
def test_split_sizes_agree(ppc, path):
    got, want, _ = _run_case([2000, 40, 513], 32, 8, 128, 0, seed=5, pages_per_chunk=ppc, path=path)
    rel, cos = _close(got, want)
    assert rel <= REL_TOL and cos >= COS_TOL


def test_gqa_group_sizes_tensor_core_path():
    """The tensor-core kernel takes the group's query heads as MMA rows: groups of 1, 2 and 8."""
    for hq, hkv in ((2, 2), (4, 2), (16, 2)):
        got, want, _ = _run_case([130, 31, 64], hq, hkv, 128, 0, seed=hq)
        rel, cos = _close(got, want)
        assert rel <= REL_TOL and cos >= COS_TOL, (hq, hkv, rel, cos)


def test_empty_context_row_is_zero():
    got, want, _ = _run_case([0, 40], 8, 2, 64, 0, seed=3)
    assert np.all(got[0] == 0)
    rel, cos = _close(got[1], want[1])
    assert rel <= REL_TOL and cos >= COS_TOL


def test_prefill_rows_as_causal_decode_rows():
    """A prefill chunk is served by giving each row its causal context (position + 1): row r of a
    request sees only its first r+1 tokens — the block-diagonal causal mask of
    src/batch_builder.zig:168-177 without materialising it."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(21)
    hq, hkv, d, n_tok = 8, 2, 64, 70
    kv = dev.PagedKVCache(1, hkv, d, 8, 1, 4, hq, max_rows=128, attn_scratch_chunks=256)
    k = ref_math.bf16_round(rng.normal(0, 1, (n_tok, hkv, d)).astype(np.float32))
    v = ref_math.bf16_round(rng.normal(0, 1, (n_tok, hkv, d)).astype(np.float32))
    q = ref_math.bf16_round(rng.normal(0, 1, (n_tok, hq, d)).astype(np.float32))
    kv.reserve(dev.pack_desc_array([(0, n_tok, 0, -1)]).cuda())
    kv.append(0, torch.tensor(k, device="cuda").bfloat16(), torch.tensor(v, device="cuda").bfloat16())
    row_seq = torch.zeros(n_tok, dtype=torch.int32, device="cuda")
    row_ctx = torch.arange(1, n_tok + 1, dtype=torch.int32, device="cuda")
    got = kv.attention(0, torch.tensor(q, device="cuda").bfloat16(), row_seq, row_ctx).float().cpu().numpy()
    assert kv.error_word() == 0
    for r in range(n_tok):
        want = ref_math.gqa_attention_decode(q[r], k[: r + 1], v[: r + 1])
        rel, cos = _close(got[r], want)
        assert rel <= REL_TOL and cos >= COS_TOL, (r, rel, cos)


@pytest.mark.parametrize("hq,hkv,d,kv_dtype", [(8, 2, 64, 0), (32, 8, 128, 0), (16, 2, 128, 0), (4, 4, 64, 0),
                                                (32, 8, 128, 1), (16, 2, 128, 1)])
def test_prefill_groups_match_oracle_and_row_kernel(hq, hkv, d, kv_dtype):
    """b200_paged_attn_prefill on a mixed batch: prefill chunks that start in the middle of a cached
    prefix (src/scheduler.zig:183-186 chunk cursor), chunks of 1..70 rows, and plain decode rows.
    Every row equals the oracle on its causal prefix, and the per-row kernel on the same inputs."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(5 + hq + d)
    # (cached tokens before the chunk, rows in the chunk)
    reqs = [(0, 70), (100, 33), (37, 1), (250, 5), (0, 1), (64, 16), (31, 2), (500, 1)]
    totals = [c + n for c, n in reqs]
    n_pages = sum(-(-t // 32) for t in totals) + 4
    n_rows = sum(n for _, n in reqs)
    kv = dev.PagedKVCache(1, hkv, d, n_pages, len(reqs), max(-(-max(totals) // 32), 1), hq, max_rows=max(totals) + n_rows,
                          attn_scratch_chunks=4096, kv_dtype=kv_dtype)
    kv.set_free_order(rng.permutation(n_pages).tolist())
    ks = [ref_math.bf16_round(rng.normal(0, 1, (t, hkv, d)).astype(np.float32)) for t in totals]
    vs = [ref_math.bf16_round(rng.normal(0, 1, (t, hkv, d)).astype(np.float32)) for t in totals]
    kv.reserve(dev.pack_desc_array([(s, t, 0, -1) for s, t in enumerate(totals)]).cuda())
    kv.append(0, torch.tensor(np.concatenate(ks), device="cuda").bfloat16(), torch.tensor(np.concatenate(vs), device="cuda").bfloat16())
    if kv_dtype != 0:  # the oracle for FP8 pools reads what the pool holds: decode(codes) * scale
        eff = [kv.gather(0, s) for s in range(len(reqs))]
        ks = [a.float().cpu().numpy() for a, _ in eff]
        vs = [b.float().cpu().numpy() for _, b in eff]
    q = ref_math.bf16_round(rng.normal(0, 1, (n_rows, hq, d)).astype(np.float32))
    row_seq = np.concatenate([np.full(n, s, np.int32) for s, (_, n) in enumerate(reqs)])
    row_ctx = np.concatenate([np.arange(c + 1, c + n + 1, dtype=np.int32) for c, n in reqs])
    qd, rs, rc = torch.tensor(q, device="cuda").bfloat16(), torch.tensor(row_seq, device="cuda"), torch.tensor(row_ctx, device="cuda")
    got = kv.attention(0, qd, rs, rc, prefill=True).float().cpu().numpy()
    per_row = kv.attention(0, qd, rs, rc).float().cpu().numpy()
    assert kv.error_word() == 0
    for r in range(n_rows):
        s, c = int(row_seq[r]), int(row_ctx[r])
        want = ref_math.gqa_attention_decode(q[r], ks[s][:c], vs[s][:c])
        rel, cos = _close(got[r], want)
        assert rel <= REL_TOL and cos >= COS_TOL, (r, s, c, rel, cos)
    assert np.abs(got - per_row).max() <= 2e-2 * np.abs(per_row).max()  # both kernels read the same pool
    kv.close()


@pytest.mark.parametrize("hq,hkv,d,kv_dtype", [(32, 8, 128, 0), (32, 8, 128, 1), (8, 2, 64, 0)])
def test_prefill_batches_of_1024_rows_and_more_write_their_rows_directly(hq, hkv, d, kv_dtype):
    """From 1024 rows on b200_paged_attn_prefill gives every group of rows one chunk as long as its context
    and the kernel normalises and writes the rows itself.  Chunks that start inside a cached prefix, contexts
    over more than 32 pages, plus decode rows in the same batch.  A sample of rows against the oracle, every
    row against the chunked path (partials + combine pass) on the same pool."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(91 + hq + d + kv_dtype)
    reqs = [(0, 520), (700, 333), (1500, 1), (64, 200), (2100, 1), (31, 47)]   # 1102 rows
    totals = [c + n for c, n in reqs]
    n_pages = sum(-(-t // 32) for t in totals) + 4
    n_rows = sum(n for _, n in reqs)
    assert n_rows >= 1024
    kv = dev.PagedKVCache(1, hkv, d, n_pages, len(reqs), -(-max(totals) // 32), hq, max_rows=max(totals) + n_rows,
                          attn_scratch_chunks=8192, kv_dtype=kv_dtype)
    kv.set_free_order(rng.permutation(n_pages).tolist())
    ks = [ref_math.bf16_round(rng.normal(0, 1, (t, hkv, d)).astype(np.float32)) for t in totals]
    vs = [ref_math.bf16_round(rng.normal(0, 1, (t, hkv, d)).astype(np.float32)) for t in totals]
    kv.reserve(dev.pack_desc_array([(s, t, 0, -1) for s, t in enumerate(totals)]).cuda())
    kv.append(0, torch.tensor(np.concatenate(ks), device="cuda").bfloat16(), torch.tensor(np.concatenate(vs), device="cuda").bfloat16())
    if kv_dtype != 0:
        eff = [kv.gather(0, s) for s in range(len(reqs))]
        ks = [a.float().cpu().numpy() for a, _ in eff]
        vs = [b.float().cpu().numpy() for _, b in eff]
    q = ref_math.bf16_round(rng.normal(0, 1, (n_rows, hq, d)).astype(np.float32))
    row_seq = np.concatenate([np.full(n, s, np.int32) for s, (_, n) in enumerate(reqs)])
    row_ctx = np.concatenate([np.arange(c + 1, c + n + 1, dtype=np.int32) for c, n in reqs])
    qd, rs, rc = torch.tensor(q, device="cuda").bfloat16(), torch.tensor(row_seq, device="cuda"), torch.tensor(row_ctx, device="cuda")
    launches = dev.launch_count()
    got = kv.attention(0, qd, rs, rc, prefill=True).float().cpu().numpy()
    direct_launches = dev.launch_count() - launches
    assert kv.error_word() == 0
    try:
        dev.set_attn_prefill_direct(False)
        launches = dev.launch_count()
        chunked = kv.attention(0, qd, rs, rc, prefill=True).float().cpu().numpy()
        assert dev.launch_count() - launches == direct_launches + 1   # the combine pass
    finally:
        dev.set_attn_prefill_direct(True)
    assert kv.error_word() == 0
    assert np.abs(got - chunked).max() <= 1e-2 * np.abs(chunked).max()
    for r in list(range(0, n_rows, 37)) + [519, 520, 852, 853, 854, 1053, 1054, n_rows - 1]:
        s, c = int(row_seq[r]), int(row_ctx[r])
        want = ref_math.gqa_attention_decode(q[r], ks[s][:c], vs[s][:c])
        rel, cos = _close(got[r], want)
        assert rel <= REL_TOL and cos >= COS_TOL, (r, s, c, rel, cos)
    kv.close()


@pytest.mark.parametrize("ctxs,forced", [([300, 70, 1500, 33], 8), ([4100, 3900, 4200, 3500], 16), ([9000, 7000, 8100], 32)])
@pytest.mark.parametrize("kv_dtype", [0, 1])
def test_chunk_length_chosen_on_the_device_equals_the_forced_one(ctxs, forced, kv_dtype):
    """With the tuning hook at 0 the plan kernel picks 8, 16 or 32 pages per chunk from the batch's mean context
    (below 96 pages per row, below 192, above).  The outputs must be the bits of a run with that length forced,
    and match the oracle."""
    auto, want, _ = _run_case(ctxs, 32, 8, 128, kv_dtype, seed=7 + forced)
    same, _, _ = _run_case(ctxs, 32, 8, 128, kv_dtype, seed=7 + forced, pages_per_chunk=forced)
    assert np.array_equal(auto, same)
    other, _, _ = _run_case(ctxs, 32, 8, 128, kv_dtype, seed=7 + forced, pages_per_chunk=4)
    assert not np.array_equal(auto, other) or len(ctxs) == 0   # another split order rounds differently somewhere
    for s in range(len(ctxs)):
        r, c = _close(auto[s], want[s])
        assert r <= REL_TOL and c >= COS_TOL, (s, ctxs[s], r, c)


@pytest.mark.parametrize("kv_dtype", [0, 1])  # bf16 pool, FP8-E4M3 pool (tensor-core kernels, head_dim 128)
def test_long_contexts_of_the_attention_microbench(kv_dtype):
    """Three sequences drawn from the attention microbench's range (log-uniform 128..32768 tokens, 32
    query / 8 KV heads, head_dim 128), one of them at the maximum of 32768 tokens = 1024 pages = 128
    split-K chunks, pages scattered over a pool sized to the pages x 1.25.  Per row against the
    per-request oracle; for the FP8 pool the oracle reads what the pool holds (codes x scale)."""
    ctxs = [32768, 4127, 128]
    got, want, _ = _run_case(ctxs, 32, 8, 128, kv_dtype, seed=2048 + kv_dtype)
    for s in range(len(ctxs)):
        r, c = _close(got[s], want[s])
        assert r <= REL_TOL and c >= COS_TOL, (s, ctxs[s], r, c)


@pytest.mark.parametrize("hq,hkv,d", [(32, 8, 128), (8, 1, 128), (4, 4, 64), (8, 4, 64)])
@pytest.mark.parametrize("scratch", [0, 100000])   # partial sums that hardly fit (key ranges stay whole), and room to split them
@pytest.mark.parametrize("rows", [(31, 32, 33), (63, 64, 65, 1, 1), (127, 128, 129, 2), (255, 256, 257, 1), (1, 1, 1), (700, 330, 1, 1)])
def test_portions_at_the_edges_of_the_row_tiles(hq, hkv, d, scratch, rows):
    """Portions of one token less and more than a tile of 128 rows or a pair of them holds (for each size of the GQA group), contexts at the
    borders of a page and of a block of 128 keys, decoding rows among them: every row against the row-by-row kernel on the same pool, some
    against the oracle.  One key is no number in one dimension: it weighs nothing, as in the row-by-row kernel."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(sum(rows) + hq + d)
    before = [0, 1, 95, 127, 128, 1500]
    reqs = [(before[(i + len(rows)) % len(before)], n) for i, n in enumerate(rows)]
    totals = [c + n for c, n in reqs]
    n_pages, n_rows = sum(-(-t // 32) for t in totals) + 4, sum(rows)
    if scratch == 0:
        # the smallest scratch that the row-by-row kernel, and the limit of batches below 1024 rows, accept
        scratch = sum(n * -(-t // 256) for (_, n), t in zip(reqs, totals)) + n_rows + 8
    kv = dev.PagedKVCache(1, hkv, d, n_pages, len(reqs), -(-max(totals) // 32), hq, max_rows=max(totals) + n_rows, attn_scratch_chunks=scratch)
    kv.set_free_order(rng.permutation(n_pages).tolist())
    k = ref_math.bf16_round(rng.normal(0, 1, (sum(totals), hkv, d)).astype(np.float32))
    v = ref_math.bf16_round(rng.normal(0, 1, (sum(totals), hkv, d)).astype(np.float32))
    q = ref_math.bf16_round(rng.normal(0, 1, (n_rows, hq, d)).astype(np.float32))
    nowhere = totals[0] // 2   # of the first request
    kd = torch.tensor(k, device="cuda").bfloat16()
    kd[nowhere, :, 3] = float("nan")
    kv.reserve(dev.pack_desc_array([(s, t, 0, -1) for s, t in enumerate(totals)]).cuda())
    kv.append(0, kd, torch.tensor(v, device="cuda").bfloat16())
    row_seq = np.concatenate([np.full(n, s, np.int32) for s, (_, n) in enumerate(reqs)])
    row_ctx = np.concatenate([np.arange(c + 1, c + n + 1, dtype=np.int32) for c, n in reqs])
    qd, rs, rc = torch.tensor(q, device="cuda").bfloat16(), torch.tensor(row_seq, device="cuda"), torch.tensor(row_ctx, device="cuda")
    got = kv.attention(0, qd, rs, rc, prefill=True).float().cpu().numpy()
    again = kv.attention(0, qd, rs, rc, prefill=True).float().cpu().numpy()
    per_row = kv.attention(0, qd, rs, rc).float().cpu().numpy()
    assert kv.error_word() == 0
    assert np.array_equal(got, again)
    # both round P and the result to bf16: 2^-8 of the largest weight and of the value, twice
    assert np.abs(got - per_row).max() <= 1.6e-2 * np.abs(per_row).max()
    first = np.concatenate([[0], np.cumsum(totals)])
    for r in sorted({0, 1, 2, 30, 31, 32, 33, 63, 64, 65, 126, 127, 128, 255, 256, n_rows - 2, n_rows - 1} & set(range(n_rows))):
        s, c = int(row_seq[r]), int(row_ctx[r])
        keep = np.arange(first[s], first[s] + c)
        want = ref_math.gqa_attention_decode(q[r], *(x[keep[keep != nowhere] if c > 1 or s > 0 else keep] for x in (k, v)))
        if s == 0 and c == 1 and nowhere == 0:
            want = np.zeros_like(want)
        rel, cos = _close(got[r], want)
        assert rel <= REL_TOL and (cos >= COS_TOL or not want.any()), (r, s, c, rel, cos)
    kv.close()


@pytest.mark.parametrize("hq,hkv,d", [(32, 8, 128), (8, 1, 128), (4, 4, 64), (8, 4, 64)])
@pytest.mark.parametrize("portions", [((2000, 300), (1500, 260), (700, 1)), ((1200, 640), (1000, 400), (90, 2))])   # below 1024 rows, and above
def test_values_that_are_not_finite_reach_only_the_rows_that_see_them(hq, hkv, d, portions):
    """Infinities and NaN in V of tokens inside prompt portions and behind the last token of a page: a row that does not see the token is the same
    to the last bit as without them, a row that sees it is not finite in just those columns of just those heads.  Keys of a token that no row
    sees change nothing; a row whose score is +inf has no sum (0 below 1024 rows, as from the row-by-row kernel); rows without context are 0."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(hq + d + len(portions))
    totals, extra = [c + n for c, n in portions], 7    # tokens behind the contexts, in the last page or the one behind it
    held, n_rows = [t + extra for t in totals], sum(n for _, n in portions)
    k = torch.tensor(rng.normal(0, 1, (sum(held), hkv, d)), device="cuda").bfloat16()
    v = torch.tensor(rng.normal(0, 1, (sum(held), hkv, d)), device="cuda").bfloat16()
    q = torch.tensor(rng.normal(0, 1, (n_rows + 2, hq, d)), device="cuda").bfloat16()
    first = np.concatenate([[0], np.cumsum(held)])
    row_seq = np.concatenate([np.full(n, s, np.int32) for s, (_, n) in enumerate(portions)] + [[0, 1]]).astype(np.int32)
    row_ctx = np.concatenate([np.arange(c + 1, c + n + 1, dtype=np.int32) for c, n in portions] + [[0, 0]]).astype(np.int32)
    rs, rc = torch.tensor(row_seq, device="cuda"), torch.tensor(row_ctx, device="cuda")

    def run(kd, vd, prefill=True):
        kv = dev.PagedKVCache(1, hkv, d, sum(-(-t // 32) for t in held) + 4, len(held), -(-max(held) // 32), hq, max_rows=sum(held), attn_scratch_chunks=40 * n_rows)
        kv.reserve(dev.pack_desc_array([(s, t, 0, -1) for s, t in enumerate(held)]).cuda())
        kv.append(0, kd, vd)
        out = kv.attention(0, q, rs, rc, prefill=prefill).float()
        assert kv.error_word() == 0
        kv.close()
        return out

    nan, inf = float("nan"), float("inf")
    # (request, token, head, column, value): in the middle and at the end of portions, twice in one column with either sign, behind the contexts
    c0, n0 = portions[0]
    c1, n1 = portions[1]
    bad = [(0, c0 + n0 // 2, 0, 3, nan), (0, c0 + n0 // 2 + 1, hkv - 1, 5, inf), (0, c0 + n0 - 2, 0, 7, -inf), (0, c0 + n0 - 2, 0, d - 1, inf), (0, c0 + n0 - 1, 0, d - 1, -inf),
           (1, c1 + n1 - 1, hkv - 1, 0, nan), (1, c1 + 130, 0, 9, inf), (2, portions[2][0] + portions[2][1] - 1, 0, 1, nan)]
    bad += [(s, totals[s] + e, h, 2, val) for s in range(3) for e, val in ((0, nan), (extra - 1, inf)) for h in (0, hkv - 1)]
    clean, dirty = v.clone(), v.clone()
    for s, t, h, c, val in bad:
        clean[first[s] + t, h, c], dirty[first[s] + t, h, c] = 0.0, val
    want, got = run(k, clean), run(k, dirty)
    assert torch.isfinite(want).all() and (want[n_rows:] == 0).all() and (got[n_rows:] == 0).all()
    added = torch.zeros_like(want)
    g = hq // hkv
    for s, t, h, c, val in bad:
        sees = (rs == s) & (rc > t)
        added[sees, h * g:(h + 1) * g, c] += val
    hit = ~torch.isfinite(added)
    assert hit.any()
    assert torch.equal(got[~hit], want[~hit])
    assert torch.equal(torch.isnan(got[hit]), torch.isnan(added[hit])) and torch.equal(got[hit & (added == inf)], added[hit & (added == inf)])
    # keys: behind the contexts nothing happens; inside, the rows behind the token whose score is +inf have no sum
    kd = k.clone()
    for s in range(3):
        kd[first[s] + totals[s]:first[s] + held[s], :, 1] = inf
    assert torch.equal(run(kd, clean), want)
    at = c0 + n0 // 2
    kd[first[0] + at, :, 3] = inf
    got, hidden = run(kd, clean), (rs != 0) | (rc <= at)
    assert torch.equal(got[hidden], want[hidden])
    up = ~hidden[:, None] & (q[:, :, 3] > 0)
    if n_rows < 1022:
        assert (got[up] == 0).all() and (run(kd, clean, prefill=False)[up] == 0).all()
    down = ~hidden[:, None] & (q[:, :, 3] < 0)
    assert torch.isfinite(got[down]).all()


@pytest.mark.parametrize("hq,hkv,d", [(32, 8, 128), (8, 2, 64)])
@pytest.mark.parametrize("spread", [1.0, 4.0])   # standard deviation of the scores: even weights, and a few large ones
@pytest.mark.parametrize("portions", [((0, 200),) * 4, ((256, 512),), ((700, 683),), ((3000, 300),) * 2])
def test_prompt_attention_is_as_close_to_64_bits_as_the_groups(hq, hkv, d, spread, portions):
    """Error (2-norm) of the tcgen05 kernel against 64 bits, at most that of the groups of 16 rows on mma.sync for the same inputs: both round P and
    the result to bf16, and weights that are exact there may not be rounded here.  (The ratio of two such errors over 800,000 results and more
    scatters by less than 0.2 %.)"""
    from dmlx_b200 import device as dev

    g = torch.Generator("cuda").manual_seed(len(portions) + d)
    rand = lambda *s: torch.randn(s, device="cuda", generator=g)
    totals, n_rows = [c + n for c, n in portions], sum(n for _, n in portions)
    k, v, q = rand(sum(totals), hkv, d).bfloat16(), rand(sum(totals), hkv, d).bfloat16(), (spread * rand(n_rows, hq, d)).bfloat16()
    kv = dev.PagedKVCache(1, hkv, d, sum(-(-t // 32) for t in totals) + 4, len(totals), -(-max(totals) // 32), hq, max_rows=max(sum(totals), 1024), attn_scratch_chunks=n_rows * 16)
    kv.reserve(dev.pack_desc_array([(s, t, 0, -1) for s, t in enumerate(totals)]).cuda())
    kv.append(0, k, v)
    rs = torch.cat([torch.full((n,), s, dtype=torch.int32) for s, (_, n) in enumerate(portions)]).cuda()
    rc = torch.cat([torch.arange(c + 1, c + n + 1, dtype=torch.int32) for c, n in portions]).cuda()
    want, at, row = torch.empty(n_rows, hq, d, dtype=torch.float64, device="cuda"), 0, 0
    for (c, n), t in zip(portions, totals):
        kk, vv = (x[at:at + t].double().repeat_interleave(hq // hkv, 1) for x in (k, v))
        s = torch.einsum("rhd,khd->hrk", q[row:row + n].double(), kk) * d ** -0.5
        hidden = torch.arange(t, device="cuda")[None] >= rc[row:row + n, None]
        want[row:row + n] = torch.einsum("hrk,khd->rhd", torch.softmax(s.masked_fill(hidden[None], -float("inf")), -1), vv)
        at, row = at + t, row + n
    err = {}
    try:
        for direct in (True, False):
            dev.set_attn_prefill_direct(direct)
            err[direct] = float((kv.attention(0, q, rs, rc, prefill=True).double() - want).norm() / want.norm())
    finally:
        dev.set_attn_prefill_direct(True)
    assert kv.error_word() == 0
    assert err[True] <= 1.002 * err[False], err
    kv.close()
