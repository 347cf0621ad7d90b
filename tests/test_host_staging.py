"""The host memory a call's input is gathered in: usable, and grown, also where no pinned
memory can be had (as on a host without a GPU)."""
import subprocess

from hbtplus_gb300 import build

SOURCE = r"""
#include "handle.h"
#include <cstdio>
#include <cstring>
int main()
{
  hbtu::HostStaging s;
  for (size_t bytes : {100, 4000, 200, 1 << 20}) {
    char *p = s.reserve(bytes);
    if (!p) return 1;
    memset(p, 7, bytes);
    if (p[bytes - 1] != 7 || (s.pinned && s.size < bytes)) return 2;
  }
  s.release();
  char *p = s.reserve(64);
  memset(p, 1, 64);
  s.release();
  return 0;
}
"""


def test_reserve(tmp_path):
    src, exe = tmp_path / "staging.cu", tmp_path / "staging"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I" + build.CSRC, "--cudart", "static",
                    "-o", str(exe), str(src)], check=True, capture_output=True)
    assert subprocess.run([str(exe)]).returncode == 0
