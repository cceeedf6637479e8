"""Rules of the CUDA sources that no run can be trusted to show broken: a race may pass every test for years."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dsa_triton_ascend_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_copied_operands_are_released_to_the_other_cta():
    """The odd CTA's relays announce blocks that other threads copied, its softmax warps rows of P that 32 lanes stored: a
    relaxed arrival of one thread orders nothing of the others."""
    text = _source("sfa_fwd_sm100.cuh")
    arrivals = re.findall(r"mbar_arrive_remote_(\w+)\((\w+)", text)
    for target in ("k_ready_lead", "v_ready_lead"):
        assert [kind for kind, to in arrivals if to == target] == ["release"]
    assert re.search(r"if \(publish\) ptx::mbar_arrive_remote_release\(remote\);", text)
    assert re.findall(r"signal_lead\(&?(\w+)[^;]*?, (true|false)\);", text) == [
        ("s_empty", "false"), ("p_full", "true"), ("o_free", "false")]
    helper = _source("ptx_sm100.cuh").split("void mbar_arrive_remote_release")[1].split("}")[0]
    assert helper.index("fence.release.sync_restrict::shared::cta.cluster") < helper.index("mbarrier.arrive")


def _kernels():
    """Signature and body of every kernel."""
    found = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\(([^{;]*?)\)\s*\{", _source(name), re.S):
                body = _source(name)[m.end():]
                found[m.group(1)] = (m.group(2), body[:body.index("\n}\n")])
    return found


def test_kernels_that_overlap_the_one_before_read_nothing_before_the_wait():
    """A pointer with __restrict__ lets the compiler move its accesses above griddepcontrol.wait."""
    kernels, launched = _kernels(), set()
    for name in os.listdir(CSRC):
        if name.endswith((".cu", ".cuh")):
            for args in re.findall(r"launch_after\((.*?), dim3\(", _source(name), re.S):
                launched.update(re.findall(r"\w+_kernel\b", args))
    assert len(launched) >= 9 and launched <= set(kernels)
    for name in launched:
        signature, body = kernels[name]
        assert "__restrict__" not in signature, name
        assert "grid_dep_wait();" in body, name
