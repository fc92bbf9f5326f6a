"""The waits of whole warps in the router's kernels: a bounded wait that some lanes of a warp give up on and others
do not would send the first past a ballot or a shuffle that counts on them, so what the warp does next goes by a
vote on the lanes' answers and never by a lane's own."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "biv_b200", "csrc", "router.cu")


def test_no_lane_of_a_warp_leaves_by_its_own_answer():
    with open(SRC) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    waits = [line.strip() for line in code.split("\n") if re.search(r"\bpf_bar_wait(_long)?\(", line)]
    assert len(waits) >= 3
    for line in waits:
        assert not re.match(r"(if|while|for)\b", line) or "pf_together(" in line, line
    # an answer that is kept goes into a vote
    for name in re.findall(r"\bbool (\w+) = pf_bar_wait", code):
        assert re.search(r"pf_together\(%s\b" % name, code), name
