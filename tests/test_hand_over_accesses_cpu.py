"""The accesses by which thread blocks hand values to each other (no GPU needed): the memory model makes a vector access
one access per ELEMENT, so whatever must be seen together has to be one element of a strong access."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "frac-ssm-kernels_b200", "csrc")


def test_value_and_tag_are_one_access():
    text = open(os.path.join(CSRC, "scan_fused.cu")).read()
    for name in ("ld_tagged", "st_tagged"):
        body = re.search(r"\b%s\([^)]*\) \{(.*?)\n\}" % name, text, re.S).group(1)
        assert re.search(r'"(ld|st)\.relaxed\.gpu\.global\.v2\.b64 ', body), name


def test_no_volatile_vector_access():
    for name in os.listdir(CSRC):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            assert not re.search(r'"(ld|st)\.volatile[.a-z]*\.v\d', text), name


def test_no_vote_inside_a_loop_that_a_lane_leaves_for_itself():
    """After a wait a lane's own `ok` may differ from its neighbours': a vote of the whole warp inside a loop over it
    would wait for lanes that never come."""
    for name in os.listdir(CSRC):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            for head in re.finditer(r"for \([^;)]*;\s*ok\b[^;]*;[^)]*\) \{", text):
                body = text[head.end():text.index("\n              }\n", head.end())]
                assert not re.search(r"_sync\(|arrived\(", body), (name, head.group(0))
