"""GPU parity of MoE routing, grouping, the ragged grouped matmul and the whole layer against the
oracle (src/moe_router.zig:55-164, src/models/deepseek_v4.zig:546-681,721-848,1010-1056)."""
import numpy as np
import pytest
import torch

from oracle import ref_math

pytestmark = pytest.mark.gpu


def _bits(a):
    return (ref_math.bf16_round(a).view(np.uint32) >> 16).astype(np.uint16)


def _close(got, want):
    g, w = np.asarray(got, np.float64).reshape(-1), np.asarray(want, np.float64).reshape(-1)
    return np.abs(g - w).max() / max(np.abs(w).max(), 1e-30), g @ w / (np.linalg.norm(g) * np.linalg.norm(w) + 1e-30)


@pytest.mark.parametrize("scoring", ["softmax", "sigmoid", "sqrtsoftplus"])
def test_route_matches_gate_forward(scoring):
    """Expert indices equal the oracle's wherever its decision margin is above f32 rounding of the
    scoring function; weights within 1e-5 relative."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(18)
    n, e, k = 512, 256, 6
    logits = rng.normal(0, 1, (n, e)).astype(np.float32)
    bias = rng.normal(0, 0.02, e).astype(np.float32)
    w_ref, i_ref = ref_math.gate_forward(logits, bias, k, route_scale=1.5, scoring=scoring)
    sc = {"softmax": 0, "sigmoid": 1, "sqrtsoftplus": 2}[scoring]
    idx, w, counts = dev.moe_route(torch.tensor(logits, device="cuda"), k, torch.tensor(bias, device="cuda"), sc, 1.5)
    idx, w = idx.cpu().numpy().astype(np.uint32), w.cpu().numpy()
    same = (idx == i_ref).all(axis=1)
    assert same.mean() >= 0.99, same.mean()
    assert np.allclose(w[same], w_ref[same], rtol=2e-5, atol=1e-9)
    assert counts.cpu().numpy().sum() == n * k
    assert np.array_equal(counts.cpu().numpy(), np.bincount(idx.reshape(-1), minlength=e))
    for t in np.where(~same)[0]:  # a disagreement is a swap at a near-tie: same set, or one expert exchanged
        assert len(set(idx[t].tolist()) ^ set(i_ref[t].tolist())) in (0, 2)


def test_route_tie_rule():
    """Equal scores: the larger expert index wins and comes last (ascending stable argsort, last k;
    src/moe_router.zig:59-73)."""
    from dmlx_b200 import device as dev

    logits = torch.zeros((3, 8), dtype=torch.float32, device="cuda")
    idx, w, _ = dev.moe_route(logits, 3)
    assert idx.cpu().numpy().tolist() == [[5, 6, 7]] * 3
    assert ref_math.topk_route(np.zeros((1, 8), np.float32), 3).tolist() == [[5, 6, 7]]
    assert np.allclose(w.cpu().numpy(), 1.0 / 8)


def test_group_bit_exact():
    """order / inv_order / offsets equal a stable host sort (src/models/deepseek_v4.zig:747-784)."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(3)
    for n, e, k, tile in ((4096, 256, 6, 128), (37, 8, 2, 16), (1, 4, 4, 64)):
        p = rng.random(e) ** 3  # skewed load
        idx = np.stack([rng.choice(e, k, replace=False, p=p / p.sum()) for _ in range(n)]).astype(np.int32)
        counts = np.bincount(idx.reshape(-1), minlength=e).astype(np.int32)
        off, order, inv, items, n_items = dev.moe_group(torch.tensor(idx, device="cuda"), torch.tensor(counts, device="cuda"), tile)
        o_ref, i_ref, tok_ref, off_ref = ref_math.group_by_expert(idx, e)
        assert np.array_equal(off.cpu().numpy(), off_ref)
        assert np.array_equal(order.cpu().numpy(), o_ref) and np.array_equal(inv.cpu().numpy(), i_ref)
        ni = int(n_items.cpu()[0])
        it = items.cpu().numpy()[:ni]
        assert ni == sum(-(-c // tile) for c in counts)
        covered = np.zeros(n * k, np.int32)
        for ex, r0, rows, _ in it:
            assert off_ref[ex] <= r0 and r0 + rows <= off_ref[ex + 1] and 0 < rows <= tile
            covered[r0:r0 + rows] += 1
        assert (covered == 1).all()


@pytest.fixture
def _restore_grouped_path():
    yield
    from dmlx_b200 import device as dev

    dev.set_qmm_grouped_block_scaled(True)  # the library default


@pytest.mark.parametrize("mode_name", ["mxfp4", "affine4", "mxfp4_block_scaled"])
def test_moe_layer_matches_oracle(mode_name, _restore_grouped_path):
    from dmlx_b200 import device as dev

    # "mxfp4" runs the grouped matmuls on the dequantising kernel, the third variant on tcgen05.mma
    # kind::mxf8f6f4 (the default for MXFP4 weights)
    dev.set_qmm_grouped_block_scaled(mode_name == "mxfp4_block_scaled")
    mode_name = "mxfp4" if mode_name == "mxfp4_block_scaled" else mode_name
    rng = np.random.default_rng(11)
    n, d, e, inter, k = 70, 256, 8, 128, 2
    x = ref_math.bf16_round(rng.normal(0, 1, (n, d)))
    wg = ref_math.bf16_round(rng.normal(0, 0.3, (e, d)))
    bias = rng.normal(0, 0.01, e).astype(np.float32)

    def make(n_e, rows, cols):
        """-> (QWeight, dequantised [n_e, rows, cols])"""
        if mode_name == "mxfp4":
            packed = rng.integers(0, 256, (n_e * rows, cols // 2), dtype=np.uint8)
            scales = rng.integers(118, 122, (n_e * rows, cols // 32), dtype=np.uint8)
            w = dev.QWeight(dev.Q_MXFP4_G32, packed, scales, None, rows, cols, n_experts=n_e)
            return w, ref_math.dequantize_mxfp4(packed, scales).reshape(n_e, rows, cols)
        wf = rng.normal(0, 0.05, (n_e * rows, cols)).astype(np.float32)
        packed, s, b = ref_math.quantize_affine4(wf)
        w = dev.QWeight(dev.Q_AFFINE4_G64, packed, _bits(s), _bits(b), rows, cols, n_experts=n_e)
        return w, ref_math.dequantize_affine4(packed, s, b).reshape(n_e, rows, cols)

    gu, gu_deq = make(e, 2 * inter, d)      # rows interleaved: 2i = gate_i, 2i+1 = up_i
    down, down_deq = make(e, d, inter)
    sgu, sgu_deq = make(1, 2 * inter, d)
    sdown, sdown_deq = make(1, d, inter)
    gate = dev.QWeight(dev.Q_BF16, _bits(wg), np.zeros(1, np.uint8), None, e, d)
    layer = dev.MoELayer(d, e, inter, k, gate, gu, down, sgu, sdown, bias=bias, route_scale=1.5, swiglu_limit=10.0,
                         tile_rows=32, max_tokens=128)
    got = layer.forward(torch.tensor(x, device="cuda").bfloat16()).float().cpu().numpy()
    assert dev.qmm_error_word() == 0
    idx, wts, off = layer.last_routing(n)
    # routing against the oracle on bf16 logits (the reference's matmul output dtype)
    logits = ref_math.bf16_round(x.astype(np.float64) @ wg.astype(np.float64).T)
    w_ref, i_ref = ref_math.gate_forward(logits, bias, k, route_scale=1.5)
    same = (idx == i_ref).all(axis=1)
    assert same.mean() >= 0.95
    assert np.array_equal(off, ref_math.group_by_expert(idx, e)[3])
    # layer output against the oracle evaluated with the routing the device chose
    routed = ref_math.switch_glu(x, idx, wts, gu_deq[:, 0::2], gu_deq[:, 1::2], down_deq, limit=10.0)
    shared = ref_math.expert_forward(x, sgu_deq[0, 0::2], sgu_deq[0, 1::2], sdown_deq[0], limit=0.0)
    rel, cos = _close(got, routed + shared)
    assert rel <= 2e-2 and cos >= 0.9995, (rel, cos)


@pytest.mark.parametrize("tile_rows", [128, 112])  # 112: two accumulator sets in tensor memory, work items alternate
def test_moe_layer_at_full_size_against_the_oracle_on_sampled_tokens(tile_rows, _restore_grouped_path):
    """The MoE workload's own shape: hidden 4096, 256 routed experts of intermediate 2048 plus a shared
    expert, top-6 softmax routing with a skewed per-expert bias, 4096 tokens in one step, MXFP4 weights
    generated on the device.  Routing and grouping are checked for all tokens; the layer output of 10
    sampled tokens is compared with the oracle, which reads the experts' weights back from the device
    (b200_qweight_export) and evaluates each sampled token through its six experts and the shared one."""
    # (10 tokens x 7 experts: reading a weight back costs more than evaluating it)
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(4)
    n, d, e, inter, k = 4096, 4096, 256, 2048, 6
    x = ref_math.bf16_round(rng.normal(0, 1, (n, d)))
    wg = ref_math.bf16_round(rng.normal(0, 0.02, (e, d)))
    bias = (rng.normal(0, 1, e) * 0.004).astype(np.float32)
    gate = dev.QWeight(dev.Q_BF16, _bits(wg), np.zeros(1, np.uint8), None, e, d)
    gu = dev.QWeight.random(dev.Q_MXFP4_G32, 2 * inter, d, e, seed=21)
    down = dev.QWeight.random(dev.Q_MXFP4_G32, d, inter, e, seed=22)
    sgu = dev.QWeight.random(dev.Q_MXFP4_G32, 2 * inter, d, 1, seed=23)
    sdown = dev.QWeight.random(dev.Q_MXFP4_G32, d, inter, 1, seed=24)
    layer = dev.MoELayer(d, e, inter, k, gate, gu, down, sgu, sdown, bias=bias, route_scale=1.5, swiglu_limit=10.0,
                         tile_rows=tile_rows, max_tokens=n)
    got = layer.forward(torch.tensor(x, device="cuda").bfloat16()).float().cpu().numpy()
    assert dev.qmm_error_word() == 0
    idx, wts, off = layer.last_routing(n)
    logits = ref_math.bf16_round(x.astype(np.float64) @ wg.astype(np.float64).T)
    w_ref, i_ref = ref_math.gate_forward(logits, bias, k, route_scale=1.5)
    same = (idx == i_ref).all(axis=1)
    assert same.mean() >= 0.97, same.mean()   # the rest are swaps at near-ties of bf16 logits
    # the device's gate matmul and the oracle may round a logit to neighbouring bf16 values (one ulp of a
    # logit near 4 is 2^-6, i.e. 1.6 % of its softmax weight): most weights agree closely, all within 5 %
    dev_rel = np.abs(wts[same] - w_ref[same]) / w_ref[same]
    assert np.median(dev_rel) <= 1e-3 and dev_rel.max() <= 5e-2, (float(np.median(dev_rel)), float(dev_rel.max()))
    assert np.array_equal(off, ref_math.group_by_expert(idx, e)[3])
    counts = np.diff(off)
    assert counts.sum() == n * k and counts.max() > 2 * counts.mean()  # the bias skews the load
    # the oracle's matmuls run in its C twin (cross-checked against the numpy oracle in tests/test_oracle_c.py)
    from oracle import ref_c

    def expert_out(xt, gu_w, down_w, ex, limit):
        p, s, _ = gu_w.export(int(ex))
        y = ref_c.qmm_mxfp4(p, s, xt)[0].astype(np.float64)
        a = ref_math.limited_swiglu(y[0::2], y[1::2], limit).astype(np.float32)
        q, t, _ = down_w.export(int(ex))
        return ref_c.qmm_mxfp4(q, t, a[None, :])[0].astype(np.float64)

    for tkn in rng.choice(n, 10, replace=False):
        xt = x[tkn:tkn + 1]
        want = expert_out(xt, sgu, sdown, 0, 0.0)
        for j in range(k):
            want = want + float(wts[tkn, j]) * expert_out(xt, gu, down, idx[tkn, j], 10.0)
        rel, cos = _close(got[tkn], want)
        assert rel <= 2e-2 and cos >= 0.9995, (int(tkn), rel, cos)


def test_ep_plan_groups_only_the_local_experts():
    """b200_ep_plan for every rank of a group of four, on one GPU: of the assignments of all tokens a rank
    keeps those whose expert it holds, grouped by local expert in a stable order; the others are marked -1
    in inv_order.  Against a stable host sort of the same subset (src/models/deepseek_v4.zig:747-784)."""
    import ctypes as C

    from dmlx_b200 import _lib

    rng = np.random.default_rng(8)
    n, e, k, world, tile = 1000, 64, 6, 4, 32
    p = rng.random(e) ** 2
    idx = np.stack([rng.choice(e, k, replace=False, p=p / p.sum()) for _ in range(n)]).astype(np.uint32)
    counts = np.bincount(idx.reshape(-1), minlength=e).astype(np.int32)
    d_idx, d_counts = torch.tensor(idx.astype(np.int64), device="cuda").to(torch.int32), torch.tensor(counts, device="cuda")
    el, a = e // world, n * k
    for rank in range(world):
        local = torch.empty(a, dtype=torch.int32, device="cuda")
        off = torch.empty(el + 1, dtype=torch.int32, device="cuda")
        order = torch.full((a,), -7, dtype=torch.int32, device="cuda")
        inv = torch.empty(a, dtype=torch.int32, device="cuda")
        items = torch.empty((el + a // tile + 1, 4), dtype=torch.int32, device="cuda")
        n_items = torch.zeros(1, dtype=torch.int32, device="cuda")
        _lib.check(_lib.lib.b200_ep_plan(d_idx.data_ptr(), d_counts.data_ptr(), n, k, e, rank, world, tile, local.data_ptr(),
                                         off.data_ptr(), order.data_ptr(), inv.data_ptr(), items.data_ptr(), n_items.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        flat = idx.reshape(-1).astype(np.int64)
        mine = np.nonzero((flat >= rank * el) & (flat < (rank + 1) * el))[0]
        want_order = mine[np.argsort(flat[mine], kind="stable")]
        want_off = np.concatenate([[0], np.cumsum(counts[rank * el:(rank + 1) * el])])
        m = len(mine)
        assert np.array_equal(off.cpu().numpy(), want_off) and want_off[-1] == m
        assert np.array_equal(order.cpu().numpy()[:m], want_order)
        want_inv = np.full(a, -1, np.int64)
        want_inv[want_order] = np.arange(m)
        assert np.array_equal(inv.cpu().numpy(), want_inv)
        ni = int(n_items.cpu()[0])
        covered = np.zeros(m, np.int32)
        for ex, r0, rows, _ in items.cpu().numpy()[:ni]:
            assert want_off[ex] <= r0 and r0 + rows <= want_off[ex + 1] and 0 < rows <= tile
            covered[r0:r0 + rows] += 1
        assert (covered == 1).all()


@pytest.mark.parametrize("mode_name", ["mxfp4", "affine4"])
def test_expert_parallel_layer_with_a_group_of_one_equals_the_plain_layer(mode_name, _restore_grouped_path):
    """The expert-parallel code path (dispatch, replicated routing, plan, grouped matmuls on the rows that
    exist, f32 partial sums, combine, shared expert) with a communicator of one rank, where both
    collectives are identities: its output must equal the plain layer's on the same weights, and the
    watchdog must see the stream finish."""
    import torch.distributed as dist

    from dmlx_b200 import device as dev
    from dmlx_b200 import expert_parallel as ep

    rng = np.random.default_rng(12)
    n, d, e, inter, k = 90, 256, 8, 128, 2
    x = torch.tensor(ref_math.bf16_round(rng.normal(0, 1, (n, d))), device="cuda").bfloat16()
    wg = ref_math.bf16_round(rng.normal(0, 0.3, (e, d)))
    bias = rng.normal(0, 0.01, e).astype(np.float32)
    mode = dev.Q_MXFP4_G32 if mode_name == "mxfp4" else dev.Q_AFFINE4_G64
    gate = dev.QWeight(dev.Q_BF16, _bits(wg), np.zeros(1, np.uint8), None, e, d)
    gu = dev.QWeight.random(mode, 2 * inter, d, e, seed=1)
    down = dev.QWeight.random(mode, d, inter, e, seed=2)
    sgu = dev.QWeight.random(mode, 2 * inter, d, 1, seed=3)
    sdown = dev.QWeight.random(mode, d, inter, 1, seed=4)
    plain = dev.MoELayer(d, e, inter, k, gate, gu, down, sgu, sdown, bias=bias, route_scale=1.5, tile_rows=32, max_tokens=128)
    want = plain.forward(x).float().cpu().numpy()
    comm = ep.Communicator(0, 1)
    layer = ep.ExpertParallelMoE(comm, d, e, inter, k, gate, gu, down, sgu, sdown, bias=bias, route_scale=1.5, tile_rows=32,
                                 max_tokens=128)
    got = layer.forward(x)
    comm.wait(timeout_ms=5000)
    got = got.float().cpu().numpy()
    assert dev.qmm_error_word() == 0
    rel, cos = _close(got, want)
    # same kernels and the same rows; only the sum over k runs in f32 here (and is rounded once)
    assert rel <= 1e-2 and cos >= 0.9999, (rel, cos)
    layer.close()
    comm.close()
    plain.close()


@pytest.mark.parametrize("n,epilogue", [(256, "swiglu"), (384, "swiglu"), (384, "none"), (136, "none"), (132, "none")])
def test_dense_experts_by_pairs_of_weight_tiles(n, epilogue):
    """Grouped matmul of dense bf16 weights with items of up to 256 rows (two weight tiles share an item's rows, which are loaded 64 at a time):
    experts with no row, one, and one more or less than a copy, a half and a whole item; an odd number of weight tiles; outputs that cannot leave
    in 16-byte pieces; row scales.  Every row against an f64 product of the same bf16 operands; results are rounded to bf16 once
    (2^-8 of the value, 2^-7 with the scale and the gate in front)."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(n + len(epilogue))
    k, counts = 192, [0, 1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 255, 256, 257, 300, 0, 40]
    e, rows = len(counts), sum(counts)
    wf = ref_math.bf16_round(rng.normal(0, k ** -0.5, (e, n, k)))
    w = dev.QWeight(dev.Q_BF16, _bits(wf.reshape(e * n, k)), np.zeros(1, np.uint8), None, n, k, n_experts=e)
    x = ref_math.bf16_round(rng.normal(0, 1, (rows, k)))
    scales = rng.uniform(0.5, 2.0, rows).astype(np.float32)
    first = np.concatenate([[0], np.cumsum(counts)])
    items = [(i, first[i] + at, min(256, c - at), 0) for i, c in enumerate(counts) for at in range(0, c, 256)]
    items_d = torch.tensor(items + [(0, 0, 0, 0)] * 5, dtype=torch.int32, device="cuda")
    got = dev.moe_grouped_qmm(w, torch.tensor(x, device="cuda").bfloat16(), items_d, torch.tensor([len(items)], dtype=torch.int32, device="cuda"), 256,
                              epilogue=dev.EPI_SWIGLU if epilogue == "swiglu" else dev.EPI_NONE, row_scales=torch.tensor(scales, device="cuda")).float().cpu().numpy()
    assert dev.qmm_error_word() == 0
    for i in range(e):
        part = slice(first[i], first[i + 1])
        y = x[part].astype(np.float64) @ wf[i].astype(np.float64).T
        if epilogue == "swiglu":
            y = y[:, 0::2] / (1 + np.exp(-y[:, 0::2])) * y[:, 1::2]
        y = y * scales[part, None]
        assert np.all(np.abs(got[part] - y) <= 2.0 ** -7 * np.abs(y) + 1e-4), (i, counts[i], np.abs(got[part] - y).max())


@pytest.mark.parametrize("n,k,epilogue", [(256, 64, "swiglu"), (384, 576, "swiglu"), (132, 192, "none"), (1160, 2176, "none")])
def test_dense_experts_with_few_rows(n, k, epilogue):
    """Grouped matmul of dense bf16 weights with items of up to 16 rows: experts with no row, one, and one more or less than a half and a whole
    item; K in fewer chunks than warps and in a remainder of them.  Bounds as for the items of pairs of tiles."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(n + k)
    tile_rows, counts = 16, [0, 1, 7, 8, 9, 15, 16, 17, 0, 40, 3]
    e, rows = len(counts), sum(counts)
    wf = ref_math.bf16_round(rng.normal(0, k ** -0.5, (e, n, k)))
    w = dev.QWeight(dev.Q_BF16, _bits(wf.reshape(e * n, k)), np.zeros(1, np.uint8), None, n, k, n_experts=e)
    x = ref_math.bf16_round(rng.normal(0, 1, (rows, k)))
    scales = rng.uniform(0.5, 2.0, rows).astype(np.float32)
    first = np.concatenate([[0], np.cumsum(counts)])
    items = [(i, first[i] + at, min(tile_rows, c - at), 0) for i, c in enumerate(counts) for at in range(0, c, tile_rows)]
    items_d = torch.tensor(items + [(0, 0, 0, 0)] * 5, dtype=torch.int32, device="cuda")
    got = dev.moe_grouped_qmm(w, torch.tensor(x, device="cuda").bfloat16(), items_d, torch.tensor([len(items)], dtype=torch.int32, device="cuda"),
                              tile_rows, epilogue=dev.EPI_SWIGLU if epilogue == "swiglu" else dev.EPI_NONE,
                              row_scales=torch.tensor(scales, device="cuda")).float().cpu().numpy()
    assert dev.qmm_error_word() == 0
    for i in range(e):
        part = slice(first[i], first[i + 1])
        y = x[part].astype(np.float64) @ wf[i].astype(np.float64).T
        if epilogue == "swiglu":
            y = y[:, 0::2] / (1 + np.exp(-y[:, 0::2])) * y[:, 1::2]
        y = y * scales[part, None]
        assert np.all(np.abs(got[part] - y) <= 2.0 ** -7 * np.abs(y) + 1e-4), (i, counts[i], np.abs(got[part] - y).max())


@pytest.mark.parametrize("tile_rows", [144, 160, 176, 192, 208, 224, 240, 256])
@pytest.mark.parametrize("epilogue", ["swiglu", "none"])
def test_dense_experts_at_every_item_size_above_128(tile_rows, epilogue):
    """Items of any accepted size above 128 rows, which arrive 64 rows at a time: full ones, a row short of it, a row more than whole copies, and
    K of more chunks than a block has stages.  Bounds as for the items of pairs of tiles."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(tile_rows)
    n, k, counts = 384, 448, [tile_rows, tile_rows - 1, tile_rows - 15, tile_rows - 16, 64, 65, 128, 129, 0, tile_rows + 1, 1, 2 * tile_rows]
    e, rows = len(counts), sum(counts)
    wf = ref_math.bf16_round(rng.normal(0, k ** -0.5, (e, n, k)))
    w = dev.QWeight(dev.Q_BF16, _bits(wf.reshape(e * n, k)), np.zeros(1, np.uint8), None, n, k, n_experts=e)
    x = ref_math.bf16_round(rng.normal(0, 1, (rows, k)))
    first = np.concatenate([[0], np.cumsum(counts)])
    items = [(i, first[i] + at, min(tile_rows, c - at), 0) for i, c in enumerate(counts) for at in range(0, c, tile_rows)]
    got = dev.moe_grouped_qmm(w, torch.tensor(x, device="cuda").bfloat16(), torch.tensor(items, dtype=torch.int32, device="cuda"),
                              torch.tensor([len(items)], dtype=torch.int32, device="cuda"), tile_rows,
                              epilogue=dev.EPI_SWIGLU if epilogue == "swiglu" else dev.EPI_NONE).float().cpu().numpy()
    assert dev.qmm_error_word() == 0
    for i in range(e):
        part = slice(first[i], first[i + 1])
        y = x[part].astype(np.float64) @ wf[i].astype(np.float64).T
        if epilogue == "swiglu":
            y = y[:, 0::2] / (1 + np.exp(-y[:, 0::2])) * y[:, 1::2]
        assert np.all(np.abs(got[part] - y) <= 2.0 ** -7 * np.abs(y) + 1e-4), (i, counts[i], np.abs(got[part] - y).max())


@pytest.mark.parametrize("tile_rows", [208, 256])
def test_layer_of_dense_experts_with_large_items(tile_rows):
    """MoELayer over dense experts whose items hold more than 128 rows: a few popular experts, every token against f64 sums over the routing that
    the layer reports (two matmuls of bf16 operands, the gated rows and the results rounded to bf16)."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(tile_rows)
    hidden, e, inter, k, n = 256, 5, 128, 2, 500
    mats = [ref_math.bf16_round(rng.normal(0, 1, s) * s[-1] ** -0.5) for s in ((e, hidden), (e, 2 * inter, hidden), (e, hidden, inter))]
    wg, wu, wd = mats
    qw = lambda m, ne=1: dev.QWeight(dev.Q_BF16, _bits(m.reshape(-1, m.shape[-1])), np.zeros(1, np.uint8), None, m.shape[-2], m.shape[-1], n_experts=ne)
    bias = np.array([0.3, 0.2, 0.0, -0.1, -0.2], np.float32)
    layer = dev.MoELayer(hidden, e, inter, k, qw(wg), qw(wu, e), qw(wd, e), bias=bias, swiglu_limit=0.0, tile_rows=tile_rows, max_tokens=n)
    x = ref_math.bf16_round(rng.normal(0, 1, (n, hidden)))
    got = layer.forward(torch.tensor(x, device="cuda").bfloat16()).float().cpu().numpy()
    assert dev.qmm_error_word() == 0
    idx, wts, off = layer.last_routing(n)
    assert np.diff(off).max() > tile_rows
    want = np.zeros((n, hidden))
    for j in range(k):
        for ex in range(e):
            t = np.where(idx[:, j] == ex)[0]
            y = x[t].astype(np.float64) @ wu[ex].astype(np.float64).T
            a = y[:, 0::2] / (1 + np.exp(-y[:, 0::2])) * y[:, 1::2] * wts[t, j][:, None]
            want[t] += a @ wd[ex].astype(np.float64).T
    rel, cos = _close(got, want)
    assert rel <= 2e-2 and cos >= 0.9999, (rel, cos)
    layer.close()


@pytest.mark.parametrize("tile_rows", [16, 64, 128, 256])
def test_dense_items_without_rows_write_nothing(tile_rows):
    """Work items of no rows among the others, the first one at row 0: skipped by every kernel that serves dense experts."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(tile_rows)
    n, k, e, count = 256, 128, 3, min(tile_rows, 40)
    wf = ref_math.bf16_round(rng.normal(0, k ** -0.5, (e, n, k)))
    w = dev.QWeight(dev.Q_BF16, _bits(wf.reshape(e * n, k)), np.zeros(1, np.uint8), None, n, k, n_experts=e)
    x = ref_math.bf16_round(rng.normal(0, 1, (2 * count, k)))
    items = [(0, 0, 0, 0), (1, 0, count, 0), (2, count, 0, 0), (2, count, count, 0), (0, 2 * count, 0, 0)]
    got = dev.moe_grouped_qmm(w, torch.tensor(x, device="cuda").bfloat16(), torch.tensor(items, dtype=torch.int32, device="cuda"),
                              torch.tensor([len(items)], dtype=torch.int32, device="cuda"), tile_rows).float().cpu().numpy()
    assert dev.qmm_error_word() == 0
    for ex, part in ((1, slice(0, count)), (2, slice(count, 2 * count))):
        y = x[part].astype(np.float64) @ wf[ex].astype(np.float64).T
        assert np.all(np.abs(got[part] - y) <= 2.0 ** -8 * np.abs(y) + 1e-4)


def test_layer_whose_router_finds_one_number_per_token():
    """Router logits that are no number but for one expert per token: that expert is chosen top_k times, so experts have more rows than the step
    has tokens and more work items than one each.  The layer's item list holds them, and every token gets its expert's output."""
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(3)
    hidden, e, inter, k, n = 128, 6, 64, 6, 16
    pick = np.arange(n) // 3   # three tokens of six choices each: 18 rows for items of 16
    gate = np.zeros((e, hidden), np.float32)
    gate[np.arange(e), np.arange(e)] = np.inf
    x = ref_math.bf16_round(rng.normal(0, 1, (n, hidden)))
    x[:, :e] = np.eye(e, dtype=np.float32)[pick]
    wu, wd = (ref_math.bf16_round(rng.normal(0, 1, s) * s[-1] ** -0.5) for s in ((e, 2 * inter, hidden), (e, hidden, inter)))
    qw = lambda m, ne=1: dev.QWeight(dev.Q_BF16, (np.ascontiguousarray(m, np.float32).reshape(-1, m.shape[-1]).view(np.uint32) >> 16).astype(np.uint16),
                                     np.zeros(1, np.uint8), None, m.shape[-2], m.shape[-1], n_experts=ne)
    layer = dev.MoELayer(hidden, e, inter, k, qw(gate), qw(wu, e), qw(wd, e), scoring=dev.SCORE_SIGMOID, swiglu_limit=0.0, tile_rows=128, max_tokens=n)
    got = layer.forward(torch.tensor(x, device="cuda").bfloat16()).float().cpu().numpy()
    assert dev.qmm_error_word() == 0
    idx, wts, off = layer.last_routing(n)
    assert (idx == pick[:, None]).all() and np.allclose(wts, 1.0 / k)
    assert sum(-(-c // 16) for c in np.diff(off)) > e + 1
    y = np.einsum("nh,nih->ni", x.astype(np.float64), wu[pick].astype(np.float64))
    a = y[:, 0::2] / (1 + np.exp(-y[:, 0::2])) * y[:, 1::2]
    rel, cos = _close(got, np.einsum("ni,nhi->nh", a, wd[pick].astype(np.float64)))
    assert rel <= 2e-2 and cos >= 0.9999, (rel, cos)
    layer.close()
