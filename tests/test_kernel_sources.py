"""Rules of the execution model that a run does not show when they are broken,
checked on the kernels' source."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "gdock_gb300" / "csrc"


def kernels():
    """(file, name, body) of every __global__ function."""
    for f in sorted(CSRC.glob("*.cu")):
        src = re.sub(r"//[^\n]*", "", f.read_text())
        for m in re.finditer(r"__global__\s+void\b", src):
            at = src.index("{", m.end())
            name = re.search(r"(k_\w+)\s*\(", src[m.end():at]).group(1)
            depth, end = 0, at
            while True:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
                if depth == 0:
                    break
            yield f.name, name, src[at:end]


@pytest.mark.parametrize("file,name,body", [k for k in kernels() if "map_shared_rank" in k[2]],
                         ids=lambda v: v if str(v).startswith("k_") else "")
def test_blocks_have_started_before_their_shared_memory_is_touched(file, name, body):
    """A block's shared memory may be accessed by another block of its cluster
    only once it is known to have started: after a barrier of the cluster."""
    # (a lambda's body runs where it is called)
    first = body.index("map_shared_rank")
    for m in re.finditer(r"auto (\w+) = \[&\][^{]*\{", body):
        end, depth = m.end(), 1
        while depth:
            depth += {"{": 1, "}": -1}.get(body[end], 0)
            end += 1
        if m.start() < first < end:
            later = body[end:]
            uses = [end + later.index(s) for s in (m.group(1) + "(", "map_shared_rank") if s in later]
            first = min(uses)
    assert "cluster.sync()" in body[:first], name


def collectives():
    """(file, statement) of every inline assembly statement that all lanes of a
    warp, or threads of a block, take part in."""
    for f in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        src = re.sub(r"//[^\n]*", "", f.read_text())
        for m in re.finditer(r"\basm\b", src):
            stmt = src[m.start():src.index(";\n", m.start())]
            if re.search(r"\.sync\b|\bbar\.|\bbarrier\.", stmt):
                yield f.name, stmt


def test_collective_assembly_stays_where_it_is_written():
    """A statement that is not volatile may be moved, or sunk into a branch that
    some lanes do not take, as if it were a function of its operands alone."""
    found = list(collectives())
    assert found
    for file, stmt in found:
        assert re.match(r"asm\s+volatile\b", stmt), (file, stmt)
