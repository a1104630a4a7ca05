"""The kernels launched as programmatic dependents are resident while the kernel before them
still writes: what it writes (records, gather layout, forces) must not reach them through the
read-only path, neither by __ldg nor by a `const ... __restrict__` parameter, since both let the
compiler move the load ahead of the wait. Read from the source: no run can show it reliably."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "hidem_b200" / "csrc"
SRC = re.sub(r"//[^\n]*", "", (CSRC / "kernels.cu").read_text())

# what a timestep's kernel or a layout conversion writes and the next one reads
WRITTEN = ("rec", "g", "force", "diffMax")


def body(pattern):
    """Every definition that `pattern` heads: the text from its parameters to its last brace."""
    out = []
    for m in re.finditer(pattern, SRC):
        i = SRC.index("{", m.end())
        depth, j = 1, i + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(SRC[j], 0)
            j += 1
        out.append(SRC[m.start():j])
    assert out, pattern
    return out


def dependents():
    names = set(re.findall(r"launch_dependent\((?:\w+,\s*)?(k_\w+)", SRC))
    assert names >= {"k_force", "k_integrate_gather", "k_step_items", "k_to_gather"}
    return sorted(names)


@pytest.mark.parametrize("kernel", dependents())
def test_kernel_waits_first_and_takes_written_arrays_plainly(kernel):
    text, = body(rf"\b{kernel}\((?=const|int4)")
    params, code = text.split("{", 1)
    assert re.sub(r"extern __shared__[^;]*;", "", code).strip().startswith("dependent_start();")
    for p in params[params.index("(") + 1:].split(","):
        if p.replace(")", " ").split()[-1].lstrip("*") in WRITTEN:
            assert "__restrict__" not in p, p
    assert "load_rec(" not in code and "load_rec_head" not in code


@pytest.mark.parametrize("reader", [r"\bload_rec_written\(const", r"\bload_body\(Body", r"\bgather_rec\(const int4"])
def test_readers_of_written_arrays_use_plain_loads(reader):
    for text in body(reader):
        assert "__ldg" not in text and "__restrict__" not in text and ".nc" not in text


def test_step_bodies_read_records_through_the_plain_readers():
    for pattern, arrays in ((r"\bforce_particle\(const", "gather"), (r"\bstep_items_block\(const", "in"),
                            (r"\bintegrate_gather\(const Consts", "force")):
        text = body(pattern)[0]
        assert not re.search(rf"__ldg\([^;]*\b(a\.)?{arrays}\b", text), pattern
        assert "load_rec(" not in text and "load_rec_head" not in text


# the lists are read through the read-only path: the kernels that read them follow another kernel
# of the chain where they are launched dependent, and never a rebuild or an earlier call's work
def test_list_readers_are_launched_dependent_only_in_a_chain():
    for m in re.finditer(r"launch_dependent\((?:(\w+),\s*)?(k_\w+)", SRC):
        if m.group(2) in ("k_force", "k_step_items"):
            assert m.group(1) == "chained", m.group(0)
    api = re.sub(r"//[^\n]*", "", (CSRC / "api.cu").read_text())
    run = api[api.index("hidem_status run_steps("):]
    run = run[:run.index("\ntemplate <class LP>\nSoaIn")]
    assert "bool chained = false;" in run
    rebuild = run[run.index("do_rebuild(ctx)"):]
    assert "chained = false;" in rebuild[:rebuild.index("}")]
