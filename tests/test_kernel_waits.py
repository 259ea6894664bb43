"""A wait of ``wait_lite`` that runs out only raises the flag of its CTA: every way out of a kernel that waits so has to carry the flag into the
status word first.  No input makes such a wait run out, so this reads the sources."""
import glob
import os
import re

import pytest

import vig_b200

CSRC = os.path.join(os.path.dirname(vig_b200.__file__), "csrc")
REPORT = re.compile(r"if \(tid == \d+ && \*abort_flag && (p\.)?status\) atomicOr\((p\.)?status, 1\);")


def _kernels(what=r"wait_lite\("):
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^{;]*\{", text):
            depth, at = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            body = text[m.end():at]
            if re.search(what, body):
                yield pytest.param(body, id=f"{os.path.basename(path)}:{text[:m.start()].count(chr(10)) + 1}")


@pytest.mark.parametrize("body", list(_kernels()))
def test_every_way_out_reports_waits_that_ran_out(body):
    last = [m.start() for m in re.finditer(r"wait_lite\(", body)]
    exits = [m.start() for m in re.finditer(r"\breturn;", body) if m.start() > last[0]] + [len(body)]
    reports = [m.end() for m in REPORT.finditer(body)]
    for e in exits:
        before = [r for r in reports if r <= e]
        # nothing but the ends of enclosing blocks, fences and what gives tensor memory back stands between a report and its way out
        assert before and "wait_lite(" not in body[before[-1]:e] and "return" not in body[before[-1]:e], body[max(0, e - 300):e]


@pytest.mark.parametrize("body", list(_kernels(r"\bsend\(")))
def test_no_cta_leaves_before_its_peer_has_written_to_it(body):
    """A CTA that gives up waiting for what the other CTA of its cluster sends must not exit while that one may still write into its shared memory:
    behind the last send stands a cluster barrier, and it is passed ahead of every way out, also by a CTA whose own share is void."""
    last = [m.start() for m in re.finditer(r"\bsend\(", body)][-1]
    arrive, wait = body.find("cluster_arrive()", last), body.find("cluster_wait()", last)
    assert last < arrive < wait
    first = body.index("cluster_wait()")
    assert "return" not in body[first:wait] and "mbar_try_wait" not in body[first:wait]
    # passed whenever there is a peer: the blocks around both halves of the barrier ask for nothing else
    for at in (arrive, wait):
        depth, opener = 0, at
        while depth >= 0:
            opener -= 1
            depth += {"}": 1, "{": -1}.get(body[opener], 0)
        assert re.search(r"if \(both\) $", body[:opener]), body[max(0, opener - 60):opener]


def test_scans_read_what_may_still_be_written_coherently():
    """The one-launch scan may begin before the launch that writes what it reads, states included: no load of it goes through the non-coherent path."""
    text = open(os.path.join(CSRC, "bigla_seg.cu")).read()
    assert not re.findall(r"__ldg\(|ld\.global\.nc", re.sub(r"//[^\n]*", "", text))
