"""A launch without a stream goes to the default stream of whatever device is
current, which a caller may have set to another one than the engine's: such a
launch needs the engine's device made current (OnDevice). Every other launch
names a stream of the engine or of the caller."""
import os
import re

import pytest

from gbhsolve import build

HOST = sorted(f for f in os.listdir(build.CSRC) if f.endswith((".cu", ".cpp")))


def _split(args):
    out, depth = [""], 0
    for c in args:
        depth += (c in "([{") - (c in ")]}")
        if c == "," and depth == 0:
            out.append("")
        else:
            out[-1] += c
    return [a.strip() for a in out]


@pytest.mark.parametrize("name", HOST)
def test_launches_name_a_stream_or_a_device(name):
    text = open(os.path.join(build.CSRC, name)).read()
    for m in re.finditer(r"<<<(.*?)>>>", text, re.S):
        args = _split(m.group(1))
        function = text[text.rfind("\n}\n", 0, m.start()):m.start()]
        assert len(args) == 4 and args[3] not in ("0", "nullptr") or "OnDevice on(" in function, m.group(0)


def test_buffers_kept_by_a_later_call_are_the_engines_devices():
    """Outside gbh_create, whose device is current throughout, allocations go to
    the caller's current device; the reverse sweep's plan outlives its call."""
    text = open(os.path.join(build.CSRC, "gbh_engine.cu")).read()
    start = text.index("static int adj_plan(")
    body = text[start:text.index("\n}\n", start)]
    assert ".upload(" in body
    assert body.index("OnDevice on(e->opt.device)") < body.index(".upload(")
