"""CPU: kernels start before the one in front of them in the stream has ended (programmatic launches), so what they load through
the read-only path has to have been there before any launch: the work tables of a plan, by ``blk_ld_table``, and nothing else."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "blockedattention_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def code(name):
    with open(os.path.join(CSRC, name)) as f:
        return [line.split("//")[0] for line in f]


@pytest.mark.parametrize("name", SOURCES)
def test_read_only_loads_are_of_work_tables(name):
    for n, line in enumerate(code(name), 1):
        where = f"{name}:{n}: {line.strip()}"
        assert "ld.global.nc" not in line and "__restrict__" not in line, where
        if "__ldg" in line:
            assert "blk_ld_table(const int4* p)" in line, where
        for arg in re.findall(r"blk_ld_table\(([^;{]*)\);", line):
            assert re.match(r"(src\b|reinterpret_cast<const int4\*>\(p\.items)", arg), where  # (src: p.items or p.pairs, below)
    text = "".join(code(name))
    for src in re.findall(r"const int4\* src = ([^;]*);", text):
        assert re.match(r"reinterpret_cast<const int4\*>\(p\.(items|pairs) \+ ", src), src
