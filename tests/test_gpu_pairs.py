"""Matmuls on pairs of CTAs (more than 128 rows), on pairs of weight tiles in tensor memory (17 to 128 rows), experts of few rows with both halves
of an activation side by side, and the small kernels of a step's chain, at the sizes where each can go wrong.

Tolerance of a matmul's row, as 2-norms: the result is rounded to bf16 (2^-9 of each value), a quantised weight too (2^-9 of each weight), SwiGLU
multiplies two sums that carry the weights' part: 3 * 2^-9, and the sums' own rounding is far below that."""
import numpy as np
import pytest
import torch

from oracle import ref_math

pytestmark = pytest.mark.gpu
ROW_TOL = 3 * 2.0 ** -9


def _weight(mode, n, k, seed):
    from dmlx_b200 import device as dev

    rng = np.random.default_rng(seed)
    if mode == "bf16":
        w = ref_math.bf16_round(rng.normal(0, k ** -0.5, (n, k)))
        bits = (w.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
        return dev.QWeight(dev.Q_BF16, bits, np.zeros(1, np.uint8), None, n, k), w
    if mode == "mxfp4":
        packed, scales = rng.integers(0, 256, (n, k // 2), dtype=np.uint8), rng.integers(119, 123, (n, k // 32), dtype=np.uint8)
        return dev.QWeight(dev.Q_MXFP4_G32, packed, scales, None, n, k), ref_math.dequantize_mxfp4(packed, scales)
    packed = rng.integers(0, 2 ** 32, (n, k // 8), dtype=np.uint32)
    s = ref_math.bf16_round(rng.uniform(0.6, 1.4, (n, k // 64)) / (4.6 * k ** 0.5)).astype(np.float32)
    b = ref_math.bf16_round(-7.5 * s).astype(np.float32)
    bits = lambda a: (a.view(np.uint32) >> 16).astype(np.uint16)  # noqa: E731
    return dev.QWeight(dev.Q_AFFINE4_G64, packed, bits(s), bits(b), n, k), ref_math.dequantize_affine4(packed, s, b)


def _rows(rows, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((rows, k), generator=g, device="cuda").bfloat16()


def _check(got, want):
    err = (got.double() - want).norm(dim=1) / want.norm(dim=1).clamp_min(1e-30)
    assert float(err.max()) <= ROW_TOL, float(err.max())


def _run(mode, n, k, rows, path=None):
    from dmlx_b200 import device as dev

    w, dense = _weight(mode, n, k, n + k)
    dense = torch.tensor(np.asarray(dense, np.float32), device="cuda").double()
    kw = {} if path is None else {"path": getattr(dev, path)}
    x = _rows(rows, k, rows)
    plain = x.double() @ dense.T
    guard = torch.full((rows + 2, n), 7.0, dtype=torch.bfloat16, device="cuda")  # the rows behind the last one stay as they are
    _check(dev.qmm(w, x, out=guard[:rows], **kw), plain)
    assert bool((guard[rows:] == 7.0).all())
    residual = _rows(rows, n, rows + 1)
    _check(dev.qmm(w, x, dev.EPI_RESIDUAL, residual=residual, **kw), plain + residual.double())
    if n % 2 == 0:
        _check(dev.qmm(w, x, dev.EPI_SWIGLU, **kw), torch.nn.functional.silu(plain[:, 0::2]) * plain[:, 1::2])
    assert dev.qmm_error_word() == 0


# one chunk of K and several, an odd number of weight tiles, outputs that end inside a tile (dense), K so long that it is split
@pytest.mark.parametrize("mode,n,k", [("bf16", 256, 64), ("bf16", 384, 192), ("bf16", 1000, 320), ("bf16", 1004, 128), ("bf16", 256, 8192), ("affine4", 384, 64),
                                      ("affine4", 256, 4096), ("mxfp4", 384, 192)])
@pytest.mark.parametrize("rows", [129, 144, 255, 256, 257, 273, 512, 513, 770])
def test_pairs_of_ctas(mode, n, k, rows):
    _run(mode, n, k, rows, "QMM_TCGEN05_X2")


# Items enough that the rings of raw blocks, of stages and of sums wrap many times in every pair of CTAs; a last pair of weight tiles with and without
# a second one; chunks enough for several ranges of K.
@pytest.mark.parametrize("mode", ["affine4", "mxfp4", "bf16"])
@pytest.mark.parametrize("n,k,rows", [(33 * 128, 1024, 2500), (34 * 128, 1024, 2500), (256, 4096, 4096)])
def test_pairs_of_ctas_repeat_themselves(mode, n, k, rows):
    """A block or a stage that is read before it is complete would differ from run to run."""
    from dmlx_b200 import device as dev

    w = dev.QWeight.random({"affine4": dev.Q_AFFINE4_G64, "mxfp4": dev.Q_MXFP4_G32, "bf16": dev.Q_BF16}[mode], n, k, seed=9)
    x = _rows(rows, k, 1)
    for epilogue in (dev.EPI_NONE, dev.EPI_SWIGLU):
        first = dev.qmm(w, x, epilogue, path=dev.QMM_TCGEN05_X2)
        for _ in range(40):
            assert torch.equal(dev.qmm(w, x, epilogue, path=dev.QMM_TCGEN05_X2), first)
    assert dev.qmm_error_word() == 0


# K in one range and in two, where SwiGLU decides
@pytest.mark.parametrize("mode", ["bf16", "affine4", "mxfp4"])
@pytest.mark.parametrize("n,k,rows", [(1024, 2048, 256), (1024, 2048, 400), (1024, 1024, 300), (512, 3072, 700)])
def test_pairs_of_ctas_of_small_matrices(mode, n, k, rows):
    _run(mode, n, k, rows, "QMM_TCGEN05_X2")


@pytest.mark.parametrize("n", [33, 34, 129, 130])
@pytest.mark.parametrize("rows", [65, 128, 200, 300])
def test_outputs_that_do_not_come_in_fours(n, rows):
    """The finish pass of split or widely tiled products stored four outputs at a time whatever the row's length."""
    _run("bf16", n, 2048, rows)
    _run("bf16", n, 256, rows)


@pytest.mark.parametrize("mode,n,k", [("affine4", 384, 192), ("affine4", 256, 4096), ("mxfp4", 128, 64)])
@pytest.mark.parametrize("rows", [17, 32, 33, 64, 65, 96, 97, 128])
def test_pairs_of_tiles(mode, n, k, rows):
    _run(mode, n, k, rows, "QMM_TCGEN05_TMEM_A")


@pytest.mark.parametrize("mode,k", [("affine4", 128), ("affine4", 192), ("mxfp4", 128)])
@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("rows", [17, 64, 65, 128])
def test_matrices_around_one_wave_of_tile_pairs(mode, k, more, rows):
    """Up to one pair of weight tiles per SM the pairs take a matrix, beyond it the kernel of single tiles, two CTAs an SM."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _run(mode, (2 * sms + more) * 128, k, rows)


def _grouped(mode, e, n, k, sizes, tile, swiglu):
    from dmlx_b200 import device as dev

    w = dev.QWeight.random(getattr(dev, "Q_BF16" if mode == "bf16" else "Q_MXFP4_G32"), n, k, n_experts=e, seed=n)
    x = _rows(sum(sizes), k, e)
    items, first, want = [], 0, []
    for i, s in enumerate(sizes):
        items.append((i % e, first, s, 0))
        packed, scales, _ = w.export(i % e)
        if mode == "bf16":
            dense = torch.tensor(packed.astype(np.int32), device="cuda").to(torch.int32).mul(65536).view(torch.float32).double().reshape(n, k)
        else:
            dense = torch.tensor(np.asarray(ref_math.dequantize_mxfp4(packed, scales), np.float32), device="cuda").double()
        y = x[first:first + s].double() @ dense.T
        want.append(torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2] if swiglu else y)
        first += s
    dev_items = torch.tensor(items + [(0, 0, 9, 0)], dtype=torch.int32, device="cuda")  # (one more than the list says it has)
    count = torch.tensor([len(items)], dtype=torch.int32, device="cuda")
    scale = torch.rand(sum(sizes), device="cuda") + 0.5
    got = dev.moe_grouped_qmm(w, x, dev_items, count, tile, dev.EPI_SWIGLU if swiglu else dev.EPI_NONE, row_scales=scale)
    assert dev.qmm_error_word() == 0
    _check(got, torch.cat(want) * scale.double()[:, None])


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("sizes", [[1, 15, 16, 17, 0, 255, 256], [130, 129, 241, 256, 3, 64, 65, 66], [200] * 80])
def test_dense_experts_on_pairs_of_ctas(sizes, swiglu):
    _grouped("bf16", 4, 384, 192, sizes, 256, swiglu)


@pytest.mark.parametrize("sizes,tile", [([1, 15, 16], 16), ([1, 16, 17, 31, 32], 32), ([2, 16, 17, 32, 33, 47, 48], 48), ([5] * 160, 48), ([49, 64, 3], 64)])
def test_block_scaled_experts_of_few_rows(sizes, tile):
    # (activations as two E4M3 codes: exact for bf16 rows whose values lie within 2^13 of the largest)
    _grouped("mxfp4", 3, 384, 256, sizes, tile, False)


@pytest.mark.parametrize("tokens", [1, 31, 32, 33, 85, 86, 128, 129])  # 6 choices: 510 assignments are routed by one block, 516 are not
@pytest.mark.parametrize("experts", [8, 33, 200])
def test_routing_by_one_block_is_the_routing_by_kernels(tokens, experts):
    from dmlx_b200 import device as dev

    h, inter, top = 256, 128, 6
    gate = torch.eye(experts, h, device="cuda").bfloat16()  # logits are values of x, whichever kernel multiplies
    bits = lambda t: t.cpu().view(torch.int16).numpy().view(np.uint16)  # noqa: E731
    layer = dev.MoELayer(h, experts, inter, top, dev.QWeight(dev.Q_BF16, bits(gate), np.zeros(1, np.uint8), None, experts, h),
                         dev.QWeight.random(dev.Q_MXFP4_G32, 2 * inter, h, n_experts=experts), dev.QWeight.random(dev.Q_MXFP4_G32, h, inter, n_experts=experts),
                         None, None, route_scale=1.5, max_tokens=256)
    x = _rows(256, h, tokens)
    few, many = layer.forward(x[:tokens]).double(), layer.forward(x).double()[:tokens]
    # another row tile adds a row's two halves up in another order; bf16 activations may then round to the other neighbour
    assert float((few - many).norm() / many.norm()) <= 2.0 ** -8
    assert dev.qmm_error_word() == 0


@pytest.mark.parametrize("vocab", [7, 8191, 8192, 32000, 32001, 128256])
@pytest.mark.parametrize("rows", [1, 16, 17, 33, 130])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_argmax_takes_the_first_maximum_wherever_the_row_is_cut(dtype, rows, vocab):
    from dmlx_b200 import device as dev

    x = torch.randn((rows, vocab), generator=torch.Generator(device="cuda").manual_seed(vocab), device="cuda").to(dtype)
    for r in range(rows):  # the maximum twice, on both sides of a cut or at the ends
        at = [0, vocab // 8, vocab // 4 - 1, vocab // 2, vocab - 1][r % 5]
        x[r, max(at, 0)] = 50.0
        x[r, vocab - 1] = 50.0
    if rows > 1:
        x[1] = -float("inf")
    want = np.array([int(np.argmax(row)) for row in x.float().cpu().numpy()])
    assert np.array_equal(dev.argmax(x).cpu().numpy(), want)


@pytest.mark.parametrize("rule", ["gated", "delta"])
@pytest.mark.parametrize("dk,dv", [(33, 40), (64, 64), (96, 17), (128, 100), (160, 64), (256, 33)])
@pytest.mark.parametrize("ctas", [24, 60, 90])
def test_scan_of_channels_split_over_warps(ctas, dk, dv, rule):
    """Few CTAs: four or two warps share a strip of value columns; many: one.  Portions that end inside a chunk, states handed on.
    The factors carry 16 bits, so what is left is the rounding of the outputs: the same bound as for chunks against single tokens, three times it."""
    from tests.test_gpu_lorulix import DeltaCase
    from tests.test_gpu_sotavik import GlaCase, _bf16, _error

    lens = (37, 5, 66)
    heads = ctas // (3 * (-(-dv // 64)))
    case = DeltaCase(lens, heads, heads, dk, dv, 2) if rule == "delta" else GlaCase(list(lens), heads, dk, dv)
    first = case.step([(0, 0, 37), (1, 0, 5), (2, 0, 33)])
    got = [first[0], first[1], np.concatenate([first[2], case.step([(2, 33, 66)])[0]])]
    for s in range(3):
        want, out = case.want(s), np.asarray(got[s])
        want, out = want.reshape(len(want), -1), out.reshape(len(out), -1)
        assert _error(out, want) <= 3 * _error(_bf16(want), want), (rule, s)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("rows", [1, 64, 127, 128, 129])
def test_sampler_parameters_in_the_launch_and_in_memory_draw_alike(rows, dtype):
    """The same kernel reads them from either place: tokens and log probabilities are the same bits."""
    from dmlx_b200 import device as dev
    from dmlx_b200._lib import check, lib

    rng = np.random.default_rng(rows)
    logits = torch.tensor(rng.normal(size=(rows, 4099)) * 3, dtype=getattr(torch, dtype), device="cuda")
    params = [(0.0 if i % 5 == 0 else 0.5 + 0.1 * (i % 7), int(rng.integers(0, 60)), float(rng.uniform(0.3, 1.0)), float(rng.uniform())) for i in range(rows)]
    got, got_lp = dev.sample_rows(logits, params)
    d = torch.from_numpy(dev.sample_params_array(params)).cuda()
    want, want_lp = torch.empty(rows, dtype=torch.int32, device="cuda"), torch.empty(rows, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    check(lib.b200_sample_rows(logits.data_ptr(), int(dtype == "float32"), rows, 4099, d.data_ptr(), None, None, None, want.data_ptr(), want_lp.data_ptr(), None))
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(got_lp, want_lp)
