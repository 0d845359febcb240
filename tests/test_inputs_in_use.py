"""Kernels read a build's inputs where the caller has them, so a build that fails
after a launch has to wait for its stream before it returns.  Making a launch
fail halfway needs a device without memory; what is checked here is the source:
every function that takes an input in place first declares the guard that waits
(InputsInUse), and calls it off only where the stream has just been waited for."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "heavyrt_gb300" / "csrc"


def _functions(text):
    """(head, body) of every function defined at the start of a line, its braces in column 0."""
    return re.findall(r"^(\w[^\n;{}]*\([^;{}]*\))\s*\n\{\n(.*?)^\}", text, flags=re.M | re.S)


def _users():
    for path in sorted(CSRC.glob("*.cu")):
        for head, body in _functions(path.read_text()):
            if re.search(r"\binput_in_place\(", body):
                yield head, body


def test_builds_that_fail_wait_for_their_inputs():
    users = list(_users())
    assert len(users) >= 3
    for head, body in users:
        guard = body.find("InputsInUse ")
        assert 0 <= guard < body.find("input_in_place("), head


def test_the_wait_is_called_off_only_after_one():
    for head, body in _users():
        lines = [x.strip() for x in body.splitlines()]
        at = [k for k, x in enumerate(lines) if x == "inputs.idle = true;"]
        assert at, head
        for k in at:
            assert "cudaStreamSynchronize(st)" in lines[k - 1], head


def test_the_guard_waits():
    text = (CSRC / "hrt_api.cu").read_text()
    body = text[text.index("struct InputsInUse"):]
    assert "if (!idle) cudaStreamSynchronize(stream);" in body[:body.index("};")]
