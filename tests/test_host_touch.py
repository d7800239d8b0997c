"""The host entry points touch every page of an operand before a kernel reads
or writes it where it lies, so that a hole in it faults on the host: the walk
over the pages, compiled by itself."""
import os
import signal
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <stdio.h>
#include <stdlib.h>
#include <sys/mman.h>
#include <unistd.h>

#include <set>

#include "host_touch.h"

// Walks at 4 KiB pages from several starts against the pages of every single byte of the parts.
static int walk() {
  const size_t page = 4096;
  const size_t shapes[][3] = {  // pitch, width, lines
      {8, 8, 1},        {800, 800, 100},   {808, 800, 100},    {4096, 4096, 9},   {4104, 4096, 9},
      {16384, 64, 40},  {20000, 8, 30},    {12288, 4104, 17},  {9000, 8992, 31},  {24, 24, 3},
      {40000, 39992, 5}, {520, 512, 64}};
  int bad = 0;
  for (const auto &s : shapes)
    for (int tri = 0; tri < 3; ++tri)
      for (size_t base : {size_t(4096), size_t(4096 + 8), size_t(8184), size_t(12288 - 16)}) {
        std::set<size_t> want, got;
        for (size_t l = 0; l < s[2]; ++l)
          for (size_t i = 0; i < s[1]; ++i) {
            const size_t e = i / 8;
            if (tri == 0 || (tri == 1 ? e >= l : e <= l)) want.insert((base + l * s[0] + i) / page);
          }
        size_t calls = 0;
        bool inside = true;
        uvt::for_each_page(base, s[0], s[1], s[2], tri, page, [&](uintptr_t a) {
          got.insert(a / page);
          ++calls;
          const size_t l = (a - base) / s[0], i = (a - base) % s[0], e = i / 8;
          inside = inside && l < s[2] && i < s[1] && (tri == 0 || (tri == 1 ? e >= l : e <= l));
        });
        if (want != got || !inside || calls > got.size() + s[2]) {
          printf("pitch %zu width %zu lines %zu tri %d base %zu\n", s[0], s[1], s[2], tri, base);
          ++bad;
        }
      }
  return bad;
}

// A column-major operand of `lines` columns with a page taken out of its middle.
static int hole(int tri) {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE), pitch = 2 * page + 16, width = pitch - 16, lines = 16;
  char *p = (char *)mmap(nullptr, pitch * lines + page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (p == MAP_FAILED) return 3;
  const size_t at = tri == 2 ? 8 * pitch : 8 * pitch + width / 2;  // of column 8, inside its part
  mprotect(p + at / page * page, page, PROT_NONE);
  volatile char sum = 0;
  uvt::for_each_page((uintptr_t)p, pitch, width, lines, tri, page, [&](uintptr_t a) { sum = sum + *(char *)a; });
  return 0;
}

int main(int argc, char **argv) {
  if (argc > 1) return hole(atoi(argv[1]));
  return walk() ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def walker(tmp_path_factory):
    d = tmp_path_factory.mktemp("touch")
    src, exe = d / "walk.cpp", d / "walk"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "uvatrmm_gb300", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    return str(exe)


def test_every_page_of_the_lines_and_no_byte_beside_them(walker):
    r = subprocess.run([walker], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("tri", [0, 1, 2])
def test_a_hole_inside_an_operand_faults_on_the_host(walker, tri):
    assert subprocess.run([walker, str(tri)]).returncode == -signal.SIGSEGV
