"""What no run can show to be missing, read from the sources: the order of accesses to memory that
one part of a launch writes and another reads, and that the known-answer hooks run the functions
that the kernels run."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "axon_b200" / "csrc"


def code(name: str) -> str:
    """A source file without its comments."""
    src = re.sub(r"/\*.*?\*/", "", (CSRC / name).read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", src)


def test_recall_reads_no_threshold_that_the_step_writes():
    """Several groups of warps select the threshold of a split trajectory, starting from its
    previous one, while the group with its first part stores the new one: the select's passes
    (and their barriers) depend on that value, so what a step reads is never what it writes."""
    src = code("batch.cu")
    select = src[src.index("const uint32_t reFloor"):]
    read = {m for m in re.findall(r"__ldcg\(([\w.]+) \+ b\), grp\)", select)} | set(re.findall(r"hist_floor\(([\w.]+) \+ b\)", src))
    written = set(re.findall(r"__stcg\(([\w.]+) \+ b, theta\)", select))
    assert len(read) == len(written) == 1 and read.isdisjoint(written)
    define = {v: re.search(rf"uint32_t\* {v} = d\.thPrev \+ \(size_t\)(\(par \^ 1u\)|par) \* B;", src).group(1) for v in read | written}
    assert define[read.pop()] == "(par ^ 1u)" and define[written.pop()] == "par"


def test_learned_tiles_are_fenced_before_they_are_copied():
    """A learning step stores W3 tiles with ordinary stores that the next step reads by bulk
    copies: between them, on the storing threads before the block barrier and on the copying
    lanes before the copy, a proxy fence that covers global memory."""
    src = code("present.cuh")
    assert "fence.proxy.async;" in code("batch_common.cuh").split("fence_proxy_async_all()")[1].split("}")[0]
    store = src.index("__stcg(d.W3")
    assert "fence_proxy_async_all();" in src[store:src.index("__syncthreads()", store)]
    copy = src.index("bulk_g2s(")
    assert "if (LEARN) fence_proxy_async_all();" in src[src.rindex("if (on)", 0, copy):copy]
    # no other kernel copies in bulk what the launch has stored
    for name in sorted(p.name for p in CSRC.glob("*.cu*")):
        if "bulk_g2s(" in code(name):
            assert name == "present.cuh" or not re.search(r"__stcg\([^;]*\bW3", code(name)), name


def calls(src: str, name: str, function: str) -> bool:
    """Whether the body of the function `name` in src calls `function`."""
    at = re.search(rf"\b{name}\([^;{{]*\)\s*{{", src).end()
    depth, end = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(src[end], 0)
        end += 1
    return re.search(rf"\b{function}[<(]", src[at:end]) is not None


def test_known_answer_hooks_run_the_kernels_functions():
    for f in ("bs_inc", "bs_dec", "band_clip"):
        assert calls(code("learn.cuh"), "learn_word", f) and calls(code("plain.cu"), "k_bstest", f), f
    assert calls(code("plain.cu"), "k_kwtatest", "warp_kwta")
    assert calls(code("planes.cu"), "k_kwtatest_planes", "plane_kwta")
    assert calls(code("planes_kernel.cuh"), "k_recall_planes", "plane_kwta")
    capi = code("capi.cu")
    for hook in ("launch_bstest", "launch_kwtatest", "launch_kwtatest_planes"):
        assert f"{hook}(" in capi, hook
