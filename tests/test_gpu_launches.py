"""Steps whose kernels are launched while the one ahead still runs (launch.cuh) give the bits of the same steps run kernel by kernel.

CUDA_LAUNCH_BLOCKING makes every launch wait until its kernel has ended, so no kernel starts early; it is read when a process starts, so each
side is a process of its own.  Graphs are off: their kernels are not launched one by one (that they change nothing is tested model by model)."""
import os
import subprocess
import sys
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MODELS = ["llama", "llama int4", "tafuvik", "sotavik", "dovorax", "lorulix"]


def _loaded(name, path):
    from dmlx_b200.models import Limits, load_model
    from tests import test_gpu_decoder, test_gpu_dovorax, test_gpu_lorulix, test_gpu_models, test_gpu_sotavik

    if name.startswith("llama"):
        test_gpu_models._folder(os.path.join(path, "m"), name.endswith("int4"))
        return load_model(os.path.join(path, "m"), "bfloat16", Limits(1024, 4, 4)), 512
    module, case = {"tafuvik": (test_gpu_decoder, "wide_head"), "sotavik": (test_gpu_sotavik, "wide"), "dovorax": (test_gpu_dovorax, "wide"),
                    "lorulix": (test_gpu_lorulix, "wide")}[name]
    cfg = module.CASES[case]
    return module._load(path, cfg, 31, "bfloat16", max_rows=1024)[0], cfg["vocab"]


def _logits(name):
    """Prompts of three requests in one step, the next portion of one beside two that decode, and steps of one row each."""
    from dmlx_b200.serving import TokenFeeder

    with tempfile.TemporaryDirectory() as path:
        loaded, vocab = _loaded(name, path)
        loaded.model.enable_graphs(False)
        tokens = [np.random.default_rng(i).integers(0, vocab, 500).tolist() for i in range(3)]
        at, out = [0, 0, 0], []
        feeder = TokenFeeder(loaded, 64)
        for portions in [(290, 33, 150)] + [(140, 1, 1)] + [(1, 1, 1)] * 12:
            out.append(feeder.step([(i, tokens[i][at[i]:at[i] + n], [n - 1]) for i, n in enumerate(portions)]))
            at = [a + n for a, n in zip(at, portions)]
        return np.stack(out)


@pytest.fixture(scope="module")
def runs(tmp_path_factory):
    out = []
    for blocking in ("1", "0"):
        path = str(tmp_path_factory.mktemp("launches") / "logits.npz")
        subprocess.run([sys.executable, "-m", "tests.test_gpu_launches", path], check=True, cwd=ROOT, timeout=600, env={**os.environ, "CUDA_LAUNCH_BLOCKING": blocking})
        out.append(np.load(path))
    return out


@pytest.mark.parametrize("name", MODELS)
def test_steps_of_early_kernels_equal_steps_kernel_by_kernel(runs, name):
    one_by_one, early = runs
    assert np.isfinite(one_by_one[name]).all()
    for again in (f"{name} 0", f"{name} 1"):
        np.testing.assert_array_equal(early[again], one_by_one[name])


@pytest.mark.parametrize("pages", ["bf16", "fp8"])
@pytest.mark.parametrize("heads,rows", [(16, 127), (16, 128), (16, 129), (8, 257), (1, 2500)])
def test_appends_in_few_blocks_and_in_many(pages, heads, rows):
    """Up to 2048 blocks are launched early, more are not.  Rows come out as they went in; of FP8 pages within half a step of the code (2^-4 of its
    magnitude, or 2^-10 of the scale, which is no more than the largest magnitude / 448) and the rounding of what is read back to bf16."""
    import torch

    from dmlx_b200 import device as dev

    kv = dev.PagedKVCache(1, heads, 64, 200, 4, 100, 4 * heads, kv_dtype=dev.KV_FP8_E4M3 if pages == "fp8" else dev.KV_BF16)
    g = torch.Generator(device="cuda").manual_seed(rows)
    k, v = (torch.randn((rows, heads, 64), generator=g, device="cuda").bfloat16() for _ in range(2))
    first = rows // 3
    kv.reserve(dev.pack_desc_array([(0, first, 0, 0), (1, rows - first, 0, first)]).cuda())
    kv.append(0, k, v)
    for seq, a, b in ((0, 0, first), (1, first, rows)):
        for got, want in zip(kv.gather(0, seq), (k, v)):
            got, want = got.float(), want[a:b].float()
            if pages == "bf16":
                assert torch.equal(got, want)
            else:
                assert bool(((got - want).abs() <= want.abs() * (2.0 ** -4 + 2.0 ** -8) + want.abs().max() / 448 * 2.0 ** -9).all())
    assert kv.error_word() == 0


@pytest.mark.parametrize("rows", [1, 2047, 2048, 2049, 5000])
def test_rows_sorted_for_experts_by_few_blocks_and_by_many(rows):
    import torch

    from dmlx_b200 import device as dev

    g = torch.Generator(device="cuda").manual_seed(rows)
    top = 1 if rows % 2 else 2
    x, weights = torch.randn((rows // top, 264), generator=g, device="cuda").bfloat16(), torch.rand(rows, generator=g, device="cuda")
    order = torch.randperm(rows, generator=g, device="cuda").int()
    xs, scales = dev.moe_gather(x, order, weights, top)
    assert torch.equal(xs, x[order.long() // top]) and torch.equal(scales, weights[order.long()])


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("rows", [128, 129, 150, 1000])
@pytest.mark.parametrize("vocab", [1, 4097, 32760, 32768, 50257])
def test_first_maximum_of_rows_by_blocks_and_by_clusters(dtype, rows, vocab):
    import torch

    from dmlx_b200 import device as dev

    g = torch.Generator(device="cuda").manual_seed(rows + vocab)
    x = torch.randint(-40, 41, (rows, vocab), generator=g, device="cuda").to(getattr(torch, dtype))  # (ties in every row)
    first = torch.where(x == x.amax(1, keepdim=True), torch.arange(vocab, device="cuda"), vocab).amin(1)
    assert torch.equal(dev.argmax(x).long(), first)


@pytest.mark.parametrize("experts,top", [(256, 8), (257, 8), (384, 8), (385, 3), (512, 10), (513, 10), (1024, 16)])
@pytest.mark.parametrize("scoring", [0, 1, 2])
def test_routes_at_the_edges_of_what_a_lane_holds(experts, top, scoring):
    """The chosen experts in ascending score, and their weights: f32 arithmetic of a few dozen operations, 2^-18 of the weight."""
    import torch

    from dmlx_b200 import device as dev

    g = torch.Generator(device="cuda").manual_seed(experts)
    logits = torch.stack([torch.randperm(experts, generator=g, device="cuda") for _ in range(40)]).float() * (16.0 / experts) - 8.0  # (no two alike)
    index, weight, counts = dev.moe_route(logits, top, scoring=scoring)
    x = logits.double()
    score = (torch.softmax(x, 1), torch.sigmoid(x), torch.nn.functional.softplus(x).sqrt())[scoring]
    want, place = score.topk(top, dim=1)
    want, place = want.flip(1), place.flip(1)
    if scoring:
        want = want / want.sum(1, keepdim=True)
    assert torch.equal(index.long(), place)
    assert bool(((weight.double() - want).abs() <= 2.0 ** -18 * want).all())
    assert torch.equal(counts.long(), torch.bincount(place.flatten(), minlength=experts))


@pytest.mark.parametrize("rows", [32, 33, 64, 71, 72, 128, 148, 149])
def test_samplers_of_rows_in_clusters_of_every_size(rows):
    """A row's token and log-probability do not depend on how many CTAs share it."""
    import torch

    from dmlx_b200 import device as dev

    g = torch.Generator(device="cuda").manual_seed(rows)
    logits = (3 * torch.randn((rows, 70000), generator=g, device="cuda")).bfloat16()
    kinds = [(0.0, 50, 1.0), (0.8, 50, 1.0), (0.8, 50, 0.9), (0.9, 0, 1.0), (0.8, 0, 0.9)]
    params = [(*kinds[i % 5], (i + 0.5) / rows) for i in range(rows)]
    tokens, lp = dev.sample_rows(logits, params)
    for i in range(0, rows, 7):
        alone, lp_alone = dev.sample_rows(logits[i:i + 1].contiguous(), params[i:i + 1])
        assert int(alone) == int(tokens[i]) and float(lp_alone) == float(lp[i])


if __name__ == "__main__":
    results = {}
    for model in MODELS:
        results[model] = results[f"{model} 0"] = _logits(model)
        results[f"{model} 1"] = _logits(model)
    np.savez(sys.argv[1], **results)
