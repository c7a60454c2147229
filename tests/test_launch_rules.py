"""What the sources have to keep to so that kernels may be launched while the one ahead of them still runs (launch.cuh)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dmlx_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def _source(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_no_kernel_s_input_is_promised_to_stay_as_it_is(path):
    """`const T* __restrict__` says that the object does not change while the function runs.  A kernel that starts early runs while the one ahead
    still writes, so the compiler might load such an input ahead of the wait, or through a cache that the wait does not concern.  (Functions that
    are called after the wait may say so.)"""
    heads = re.findall(r"__global__[^{;]*?\b(\w+)\s*\(([^{;]*?)\)\s*\{", _source(path), re.S)
    assert heads or "__global__" not in _source(path)
    promised = [(name, p) for name, params in heads for p in re.findall(r"const [\w:]+\s*\*\s*__restrict__ \w+", params)]
    assert not promised, promised


@pytest.mark.parametrize("kernel,names", [("rope_kernel", "qk"), ("rope_append_bf16_kernel", ["q"]), ("rope_append_partials_bf16_kernel", ["positions", "row_seq"]),
                                          ("route_kernel", ["counts"])])
def test_neither_is_what_a_kernel_changes_in_place(kernel, names):
    """The same of memory that a kernel reads and writes: what it reads there comes from the kernel ahead."""
    params = re.search(r"__global__[^{;]*?\b%s\(([^{;]*?)\)\s*\{" % kernel, "\n".join(_source(f) for f in FILES), re.S).group(1)
    for name in names:
        assert re.search(r"\*\s*%s\b" % name, params) and not re.search(r"__restrict__ %s\b" % name, params), name


KERNELS = [(os.path.basename(f), m.group(1), m.start(), f) for f in FILES for m in re.finditer(r"__global__[^{;]*?\b(\w+_kernel)\s*\([^{;]*?\)\s*\{", _source(f), re.S)]


@pytest.mark.parametrize("file,name,start,path", KERNELS, ids=[k[1] for k in KERNELS])
def test_a_kernel_waits_for_those_ahead_before_its_bounded_waits_begin(file, name, start, path):
    """A wait that gives up after so many polls, or a word written to memory, belongs behind the wait for the kernels ahead: their time would count."""
    body = _source(path)[start:]
    body = body[:body.index("\n}\n")]
    wait = re.search(r"\b(after|wait)_previous\(\)", body)
    if wait is None:
        pytest.skip("launched plainly")
    early = re.search(r"\bmbar_wait\w*\(|\batomic\w+\(", body[:wait.start()])
    assert early is None, early.group(0)


def test_weights_are_on_the_device_when_they_are_handed_out():
    """Kernels fetch weights before they wait for anything ahead of them, so a weight object may not leave its constructor while its blocks are on
    their way.  (A copy from pageable memory returns when it has been staged.)"""
    source = _source(os.path.join(CSRC, "qmm.cu"))
    makers = re.findall(r"b200_status (b200_qweight_\w+)\([^{;]*\*\* ?out\) \{(.*?)\n\}\n", source, re.S)
    assert {name for name, _ in makers} == {"b200_qweight_create", "b200_qweight_random"}
    for name, body in makers:
        filled = max(body.rfind("cudaMemcpy("), body.rfind("<<<"))
        assert 0 < filled < body.index("Synchronize(", filled) < body.rindex("*out = w"), name


def test_words_between_ctas_have_the_scope_of_the_cluster():
    """A word that one CTA sends to another stands for shared memory that the other's MMAs read: an arrival without a scope releases to its own CTA."""
    source = "\n".join(_source(f) for f in FILES)
    sent = re.findall(r'"mbarrier\.arrive[^"]*shared::cluster[^"]*"', source)
    assert sent and all(".release.cluster." in a or ".relaxed.cluster." in a for a in sent), sent
    ahead = source[:source.index("mbarrier.arrive.relaxed.cluster")]
    assert ahead.rstrip().endswith('asm volatile("') and "fence.release.sync_restrict::shared::cta.cluster" in ahead[-160:]
    assert re.search(r"mbar_wait_cluster\(ready", source) and not re.search(r"mbar_wait_addr\((ready|acc_free)", source)


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_grids_are_sized_by_the_device(path):
    """How many SMs there are, and how many CTAs run on them at once, is asked of the device."""
    assert not re.findall(r"[^\n]*\b(?:148|296)\b[^\n]*", _source(path))
    assert not re.findall(r"rows \* (?:parts|ranks) \* 2 <= \d+", _source(path))


@pytest.mark.parametrize("kernel", ["qmm_f32_kernel", "attn_simt_kernel", "gla_step_kernel", "delta_step_kernel"])
def test_long_kernels_do_not_share_their_sms(kernel):
    """Warps that wait take issue slots from those that work, and blocks that are scheduled before the kernel ahead has ended lie on few SMs: a kernel that
    may take long lets the next one start when its main loop is done, and has a launch of its own for that."""
    bodies = [(_source(path)[start:], path) for file, name, start, path in KERNELS if name == kernel]
    assert len(bodies) == 1
    body, source = bodies[0][0], _source(bodies[0][1])
    body = body[:body.index("\n}\n")]
    assert "after_previous()" not in body and "wait_previous()" in body and "let_next_start()" in body
    assert re.search(r"launch_apart\((?:kernel|%s)\b" % kernel, source)


def test_the_finish_pass_of_few_rows_and_many_outputs_lets_the_next_kernel_start_when_all_it_reads_has_arrived():
    """An epilogue's own loads and arithmetic come behind the sums: only without one may the next stream of weights begin there."""
    body = next(_source(path)[start:] for file, name, start, path in KERNELS if name == "qmm_finish_kernel")
    body = body[:body.index("\n}\n")]
    assert re.findall(r"[^\n]*let_next_start\(\);", body) == ["  if (!late) let_next_start();", "  if (late && a.epilogue == B200_EPI_NONE) let_next_start();"]
    assert body.index("if (!late)") < body.index("v0 = p[") < body.index("if (late")
