"""Barriers between the CTAs of a cluster: an arrival on another CTA's barrier, and the wait that goes with it, name the cluster
scope (the default is the CTA, which orders nothing for a thread of another one)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "exact_b200", "csrc")


def _instructions(pattern):
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        for m in re.finditer(r'"[^"\n]*\b(%s)[^"\n]*"' % pattern, open(path).read()):
            found.append((os.path.basename(path), m.group(1)))
    return found


def test_arrivals_on_another_cta():
    remote = [(f, i) for f, i in _instructions(r"mbarrier\.arrive[a-z0-9_.:]*") if "shared::cluster" in i]
    assert remote, "the CTA pairs of the dense GEMM signal across CTAs"
    for where, instruction in remote:
        assert re.search(r"\.(release|relaxed)\.cluster\.", instruction), (where, instruction)


def test_relaxed_sides_carry_their_fences():
    text = open(os.path.join(CSRC, "tc.cuh")).read()
    arrive = text[text.index("mbar_arrive_leader(uint32_t bar)"):]
    assert arrive.index("fence.release.sync_restrict::shared::cta.cluster") < arrive.index("mbarrier.arrive.relaxed.cluster")
    wait = text[text.index("mbar_wait_pair(uint32_t bar"):]
    assert wait.index("mbar_try_wait_cluster") < wait.index("fence.acquire.sync_restrict::shared::cluster.cluster")


@pytest.mark.parametrize("barrier", ["s_ready", "s_tempty"])
def test_issuing_thread_waits_at_cluster_scope(barrier):
    text = open(os.path.join(CSRC, "linear_gemm.cu")).read()
    issuer = text[text.index("MMA issuer ----"):text.index("converter: warps")]
    waits = re.findall(r"(\w+)\(smem_u32\(&%s" % barrier, issuer)
    assert waits == ["wait"] and "PAIR ? mbar_wait_pair" in issuer
