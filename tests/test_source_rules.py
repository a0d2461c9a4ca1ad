"""Rules of the kernels' sources that no run can show to be broken: what they
guard against needs a schedule, or a state of the caches, that a test cannot ask for."""
from __future__ import annotations

import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "beamforming_gb300", "csrc")


def _source(name):
    """The file without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _body(text, name):
    """The body of kernel `name`."""
    at = re.search(r"\b%s\s*\([^;{]*\)\s*\{" % name, text)
    assert at, name
    depth, i = 1, at.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[at.end():i]


@pytest.mark.parametrize("name,kernel", [("bf_tc.cu", "bf_form_beams_tc"), ("bf_tc_pair.cu", "bf_form_beams_pair")])
def test_barriers_are_set_up_before_their_warp_uses_them(name, kernel):
    """The lanes of a producer warp initialise its barriers together and lane 0
    goes on without waiting for another warp, so the warp meets in between."""
    body = _body(_source(name), kernel)
    inits = [m.end() for m in re.finditer(r"\bmbar_init\(", body)]
    fence = body.index("fence_barrier_init();")
    used = min(body.index(x) for x in ("cluster_arrive();", "cta_arrive(") if x in body)
    assert inits and max(inits) < fence < used
    assert "__syncwarp();" in body[fence:used]


def test_overlapped_kernels_use_plain_loads():
    """A launch that overlaps the one before it may be resident while that one
    writes what it reads, so nothing in it may go through the read-only path."""
    for name in ("bf_tc.cu", "bf_tc_pair.cu", "bf_tc_common.cuh", "bf_ptx.cuh"):
        text = _source(name)
        assert "__ldg" not in text and ".nc." not in text, name
        assert not re.search(r"\bconst\s+\w+\s*\*\s*__restrict__", text), name
    launched = set()
    for name in os.listdir(CSRC):
        launched |= set(re.findall(r"launch_overlapped\(\s*(\w+)\s*,", _source(name)))
    assert launched == {"kern", "bf_pad_e", "write_words"}  # `kern`: of the files above
    head = re.search(r"\bwrite_words\(([^)]*)\)\s*\{", _source("bf_adler.cu"))
    assert "__restrict__" not in head.group(1)


@pytest.mark.parametrize("name,kernel", [("bf_tc.cu", "bf_form_beams_tc"), ("bf_tc_pair.cu", "bf_form_beams_pair")])
def test_commits_are_counted_where_they_are_issued(name, kernel):
    """The issuer waits at its end for the commits that it counted.  A wait that gives
    up ends a tile early, so no wait may lie between a commit and its count: the arrival
    that was left out would land in the shared memory of a CTA that has gone."""
    body = _body(_source(name), kernel)
    calls = [m.end() for m in re.finditer(r"\boffset_mma\(\);", body)]
    assert len(calls) == 2
    for at in calls:
        until = re.search(r"\bmbar_wait\(|\bmbar_wait_drain\(", body[at:]).start()
        assert "ndig" in body[at:at + until]
