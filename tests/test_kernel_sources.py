"""Rules of the CUDA sources that no run can be trusted to show broken: a race may pass every test for years."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dsa_triton_ascend_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_copied_operands_are_released_to_the_other_cta():
    """The odd CTA's relays announce blocks that other threads copied: a relaxed arrival orders nothing of theirs."""
    text = _source("sfa_fwd_sm100.cuh")
    arrivals = re.findall(r"mbar_arrive_remote_(\w+)\((\w+)", text)
    for target in ("k_ready_lead", "v_ready_lead"):
        assert [kind for kind, to in arrivals if to == target] == ["release"]
    helper = _source("ptx_sm100.cuh").split("void mbar_arrive_remote_release")[1].split("}")[0]
    assert helper.index("fence.release.sync_restrict::shared::cta.cluster") < helper.index("mbarrier.arrive")
