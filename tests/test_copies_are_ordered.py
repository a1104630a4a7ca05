"""Every context and network works on a stream of its own that does not wait for the default
stream. A copy to the device on the default stream may return before its last piece has arrived
(from pageable memory), so no kernel on such a stream may follow one: all copies to the device and
all fills are on a stream. Read from the source: no run can show it reliably."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "hidem_b200" / "csrc"


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.c*")))
def test_copies_to_the_device_are_on_a_stream(source):
    text = re.sub(r"//[^\n]*", "", (CSRC / source).read_text())
    for call in re.findall(r"\bcudaMemcpy(?:2D|3D)?\([^;]*;", text):
        assert "DeviceToHost" in call, call
    assert not re.findall(r"\bcudaMemset(?:2D|3D)?\([^;]*;", text)
    # and every kernel launch names its stream
    for launch in re.findall(r"<<<(.*?)>>>", text, re.S):
        stream = launch.rsplit(",", 1)[-1].strip()
        assert stream in ("s", "st", "so", "sl", "stream") or stream.endswith(("->stream", ".stream")), launch
