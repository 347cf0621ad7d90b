"""Indexes of the per-particle arrays at the largest calls the library takes (2^30
particles): the octant slots, eight per element, and the coordinates, three per
particle, lie beyond an int."""
import os
import re
import subprocess

import pytest

from hbtplus_gb300 import build

SOURCE = r"""
#include "device_common.cuh"
#include <cstdio>
#include <cstdlib>
int main(int n, char **e)
{
  for (int k = 1; k < n; k++)
    printf("%llu %llu\n", (unsigned long long)hbtu::first_slot(atoi(e[k])),
           (unsigned long long)hbtu::first_coord(atoi(e[k])));
}
"""


def test_first_slot_and_coordinate(tmp_path):
    src, exe = tmp_path / "width.cu", tmp_path / "width"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I" + build.CSRC, "--cudart", "static",
                    "-o", str(exe), str(src)], check=True, capture_output=True)
    at = [0, 1, (1 << 28) - 1, 1 << 28, (1 << 31) // 3 + 1, (1 << 30) - 1]
    out = subprocess.run([str(exe), *map(str, at)], check=True, capture_output=True, text=True).stdout
    assert [tuple(map(int, line.split())) for line in out.splitlines()] == [(8 * e, 3 * e)
                                                                           for e in at]


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(build.CSRC)
                                        if f.endswith((".cu", ".cuh"))))
def test_slots_are_reached_through_it(name):
    text = open(os.path.join(build.CSRC, name)).read()
    for use in re.findall(r"\bcslot\s*[\[+][^;]*;", text):
        assert "first_slot(" in use, use
