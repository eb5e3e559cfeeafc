"""Every kernel of the library is launched with programmatic stream serialisation (launch_kernel and its
cluster form set the attribute), so it may start while the kernel in front of it still runs, and the kernel
behind it waits for it alone.  A kernel that never executes griddepcontrol.wait therefore reads and writes
next to its predecessor and cuts the order of the stream for its successors.  Read from the sources: the
order cannot be tested by running it wrong."""
import os
import re

import pytest

from tuiskollm_b200 import build

KERNEL = re.compile(r"__global__\s+void\b[^;{]*?(\w+)\s*\(\s*(?:const\b|[A-Z]\w*Params\b|int\b|unsigned\b|float\b|uint)")


def _body(text, start):
    """The brace-balanced block that begins at the first '{' after `start`."""
    begin = text.index("{", start)
    depth = 0
    for i in range(begin, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[begin:i + 1]
    raise AssertionError("unbalanced braces")


def _kernels(source):
    with open(os.path.join(build.CSRC, source)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    found = [(m.group(1), _body(text, m.end())) for m in KERNEL.finditer(text)]
    assert len(found) == len(re.findall(r"__global__", text)), (source, [n for n, _ in found])
    return found


@pytest.mark.parametrize("source", [s for s in build.SOURCES if s.endswith(".cu")])
def test_every_kernel_waits_for_its_predecessor(source):
    for name, body in _kernels(source):
        assert "pdl_wait()" in body, f"{source}: {name} never waits for the kernel in front of it"


def test_a_wait_that_guards_state_has_one_verdict_per_warp():
    """The recurrence updates its state in place, so rows go back only if all of them had arrived.  Each lane
    updates columns of every row of its warp and one lane sends the rows: were the verdict of the bounded wait
    that lane's own, another lane that gave up first would have its columns stored over the state.  Read from
    the source: lanes part only while a wait is running out."""
    body = dict(_kernels("gdn.cu"))["gdn_recurrence_kernel"]
    waits = re.findall(r"mbar_wait\w*\(", body)
    assert waits and len(re.findall(r"__all_sync\(0xffffffffu, mbar_wait\(", body)) == len(waits)
    assert re.search(r"\bok\) \{\s*bulk_store_1d\(", body)
