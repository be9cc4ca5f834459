"""Tile and slab counts over the whole range of int (ls_sizes.h, the arithmetic
that the grouped kernels use on sizes read from device memory)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <stdio.h>
#include "ls_sizes.h"
int main(int argc, char **) {
  int n, d;
  while (scanf("%d %d", &n, &d) == 2) printf("%d %d\n", ls::ceil_div(n, d), ls::slabs(n, d));
  return argc == 0;
}
"""
TOP = 2 ** 31 - 1


def test_counts_up_to_the_end_of_int(tmp_path):
    src, exe = tmp_path / "sizes.cpp", tmp_path / "sizes"
    src.write_text(PROGRAM)
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-ftrapv", "-I",
                    os.path.join(ROOT, "libshalom_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    cases = [(n, d) for d in (16, 32, 64, 128)
             for n in (-TOP - 1, -5, 0, 1, d - 1, d, d + 1, TOP - d, TOP - d + 1, TOP - 1, TOP)]
    out = subprocess.run([str(exe)], input="".join(f"{n} {d}\n" for n, d in cases), check=True,
                         capture_output=True, text=True).stdout.split("\n")
    for (n, d), line in zip(cases, out):
        want = max(0, -(-n // d))
        assert tuple(map(int, line.split())) == (want, max(1, want)), (n, d)
