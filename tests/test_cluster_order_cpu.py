"""What the kernels may say to another CTA of their cluster, checked in their source on the
CPU: an arrival on another CTA's barrier orders what the arriving thread did (and saw) before
it only if it is a release at cluster scope, the default being the thread's own CTA; a copy
that the other CTA's barrier counts is one.  Whoever waits there acquires at cluster scope."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "whetstone_b200" / "csrc"


def instructions(path, opcode):
    return re.findall(re.escape(opcode) + r"[\w.:]*", path.read_text())


def test_what_is_announced_to_another_cta_is_ordered_at_cluster_scope():
    announcing = 0
    for path in sorted(CSRC.glob("*.cu*")):
        arrivals = [i for i in instructions(path, "mbarrier.arrive") if ".shared::cluster" in i]
        messages = instructions(path, "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx")
        for instr in arrivals:
            assert ".release.cluster." in instr, f"{path.name}: {instr}"
        if arrivals or messages:
            announcing += 1
            waits = instructions(path, "mbarrier.try_wait")
            assert any(".acquire.cluster." in i for i in waits), path.name
    assert announcing, "the two-SM projection tiles announce the second CTA's half to the first"
