"""A wait of ``wait_lite`` that runs out only raises the flag of its CTA: every way out of a kernel that waits so has to carry the flag into the
status word first.  No input makes such a wait run out, so this reads the sources."""
import glob
import os
import re

import pytest

import vig_b200

CSRC = os.path.join(os.path.dirname(vig_b200.__file__), "csrc")
REPORT = re.compile(r"if \(tid == \d+ && \*abort_flag && (p\.)?status\) atomicOr\((p\.)?status, 1\);")


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^{;]*\{", text):
            depth, at = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            body = text[m.end():at]
            if "wait_lite(" in body:
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
