"""Rules of the role-split kernels that their sources have to keep (read from the sources: what breaks them may show only as
a wait that runs into its limit, or not at all)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openbox-llm_b200", "csrc")


def _source(name):
    return open(os.path.join(CSRC, name)).read()


@pytest.mark.parametrize("name", ["tc.cu", "tc_fwdpair_kernel.cu", "tc_bwd.cu", "tc_bwd_wide.cu"])
def test_a_warp_that_issues_as_one_waits_as_one(name):
    """A warp whose elected lane issues the MMAs leaves every wait by a vote.  Lanes that waited each for itself could part, and
    one that fell two phases behind would wait for a parity that has come round.  Barriers of one phase are exempt."""
    roles = [part for part in re.split(r"\n\s*// ---- ", _source(name)) if "mma_ss_by(" in part]
    assert roles
    for role in roles:
        for line in role.splitlines():
            if re.search(r"\bmbar_(try_|test_)?wait\(", line):
                assert "__all_sync(" in line or "bar_kv" in line or "bar_drain" in line, line



@pytest.mark.parametrize("name", ["tc_fwdpair_kernel.cu", "tc_bwd.cu", "tc_bwd_wide.cu"])
def test_every_producer_waits_for_its_own_loads(name):
    """No load is on its way into a CTA's shared memory when the CTA ends: each warp that sends some waits (bounded) until they
    have landed, on its way to the teardown barrier, whoever gives up and whenever."""
    roles = [part for part in re.split(r"\n\s*// ---- ", _source(name)) if part.startswith("producers")]
    assert len(roles) == 1
    assert "mbar_wait_drain(bar_kv, 0);" in roles[0] and roles[0].count("mbar_wait_drain(") == 2
    assert not re.search(r"if \([^\n]*(s_abort|pw == 0)[^\n]*\{\n[^{}]*mbar_wait_drain", roles[0])


READ_ONLY_PATH = r"__ldg\(|ldg_\w+_now\(|ld\.global\.nc|\bconst \w+\s*\* __restrict__"


@pytest.mark.parametrize("name", ["sel_row.cuh", "sel_plan.cu", "tc_score.cu", "tc.cu", "tc_fwdpair.cu", "tc_bwd.cu"])
def test_chained_kernels_read_by_plain_loads(name):
    """A kernel that is on the GPU before the one ahead has ended reads nothing through the read-only path, which takes its data
    not to change meanwhile.  Two kernels of the backward are launched plainly."""
    functions = re.split(r"\n(?=(?:template <[^\n]*>\n)?(?:__global__|__device__) )", _source(name))
    plain = [f for f in functions if re.search(r"^(tc_bwd_kernel|cmp_chunks_kernel)\(", f, re.M)]
    assert len(plain) == (2 if name == "tc_bwd.cu" else 0)
    for f in functions:
        if f not in plain:
            assert not re.search(READ_ONLY_PATH, f), re.search(READ_ONLY_PATH, f).group(0)
