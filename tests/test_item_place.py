"""Work items of views with more pixels than an int counts, on the CPU: chunk, column and row of an item
against Python's integers."""
import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
SOURCE = """
#include <cuda_runtime.h>
#include <cstdio>
#include "device/dev_types.cuh"
int main() {
  long long local;
  int w, h;
  while (std::scanf("%lld %d %d", &local, &w, &h) == 3) {
    const bn::ItemPlace p = bn::item_place(local, w, h);
    std::printf("%d %d %d\\n", p.chunk, p.x, p.y);
  }
}
"""


def test_items_of_large_views(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    (tmp_path / "p.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", f"{cuda}/include", "-I", str(ROOT / "barnacle_gb300" / "csrc"),
                    str(tmp_path / "p.cpp"), "-o", str(tmp_path / "p")], check=True)
    cases = []
    for w, h in ((1, 1), (97, 61), (65536, 32769), (70001, 70001), (1, 2**31 - 1), (2**31 - 1, 3)):
        n = w * h
        for pix in {0, 1, w - 1, w, n // 2, 2**31 - 1, 2**31, 2**32 - 1, 2**32, n - 1}:
            cases += [(chunk * n + pix, w, h) for chunk in (0, 1, 63) if 0 <= pix < n]
    r = subprocess.run([str(tmp_path / "p")], input="".join("%d %d %d\n" % c for c in cases), capture_output=True, text=True,
                       check=True)
    want = [((a // (w * h)), a % (w * h) % w, a % (w * h) // w) for a, w, h in cases]
    assert [tuple(map(int, line.split())) for line in r.stdout.split("\n") if line] == want
