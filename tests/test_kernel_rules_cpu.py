"""Rules of the kernels that the GPU does not report when they are broken, checked in the sources."""
import os
import re

_CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "soklyn_b200", "csrc")


def _source(name):
    """The file without its comments."""
    with open(os.path.join(_CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_a_warpgroup_changes_its_register_count_in_one_instruction():
    """setmaxnreg is .aligned over the four warps of a warpgroup: they execute the same instruction, so it may stand
    behind a condition on whole warpgroups only."""
    users = {f: re.findall(r"tc::reg_(?:dec|inc)<", _source(f)) for f in os.listdir(_CSRC) if not f.endswith(".so")}
    assert {f: len(u) for f, u in users.items() if u} == {"sk_gemm_tc.cuh": 2}
    src = _source("sk_gemm_tc.cuh")
    assert re.search(r"constexpr int kTcFirstEpi = 4;", src)
    assert re.search(r"\n    if \(warp < kTcFirstEpi\) \{\s*tc::reg_dec<kTcRegsMain>\(\);", src)
    assert re.search(r"\n    \} else \{\s*tc::reg_inc<kTcRegsEpi>\(\);", src)


def test_a_warp_arrives_at_a_cluster_barrier_as_one():
    """barrier.cluster.*.aligned after a divergent loop is undefined: the only place that issues it brings the lanes
    of a warp together first."""
    uses = [(f, m.start()) for f in os.listdir(_CSRC) for m in re.finditer(r"barrier\.cluster\.arrive", _source(f))]
    assert [f for f, _ in uses] == ["sk_tc_ptx.cuh"]
    assert re.search(r"void cluster_sync\(\) \{\s*__syncwarp\(\);\s*asm volatile\(\"barrier\.cluster\.arrive\.release\.aligned;", _source("sk_tc_ptx.cuh"))


def test_launches_overlap_only_where_the_context_allows_it():
    """A block that waits for the preceding kernel holds its SM, also one that SK_OPTION_RESERVE_SMS keeps free: the
    one rule that lets a launch overlap asks for the option, and every launch of a step goes by it."""
    api, simt = _source("sk_api.cu"), _source("sk_gemm_simt.cuh")
    assert re.search(r"bool overlaps\(const sk_ctx \*c\) \{ return sizeof\(T\) == 2 && c->reserve_sms == 0; \}", api)
    asks = re.findall(r"launch_step\(c->stream, (\w+)", api)
    assert asks and set(asks) == {"overlaps"} and len(asks) == len(re.findall(r"launch_step\(", api))
    assert set(re.findall(r"launch_step\(stream, (\w+)", simt)) == {"overlap"}
    assert re.findall(r"launch_gemm_simt<[^;]*?>\(c->stream, (\w+)", api) == ["overlaps"]
