"""The entry index arithmetic of csrc/entries.h, compiled for the CPU: what it writes and
where it stops, at the ends of arrays."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

SRC = r"""
#include <stdio.h>
#include <stdlib.h>
#include <vector>
#include "entries.h"

// every chunk of an array of m entries (a thread takes N): only its own entries change
template <int N>
static int fill(uint32_t m) {
  const int32_t mark = 0x5a5a5a5a, x = -7;
  const uint32_t room = 16;
  int32_t *a = static_cast<int32_t *>(aligned_alloc(16, (((m + room) * 4 + 15) / 16) * 16));
  int bad = 0;
  for (uint32_t e0 = 0; e0 < (m + 1023) / 1024 * 1024; e0 += N) {
    const uint32_t e1 = e0 >= m ? e0 : e0 + N < m ? e0 + N : m;
    for (uint32_t e = 0; e < m + room; e++) a[e] = mark;
    accx_fill_chunk<N>(a, e0, e1, x);
    for (uint32_t e = 0; e < m + room; e++) bad += a[e] != (e >= e0 && e < e1 ? x : mark);
  }
  free(a);
  return bad;
}

// slices and strided loops of ranges that end close to 2^32: every position once, in order
static int walk(uint64_t b, uint64_t end, uint32_t len) {
  uint64_t at = b;
  for (uint32_t e = (uint32_t)b; e < (uint32_t)end;) {
    const uint32_t to = accx_slice_end(e, len, (uint32_t)end);
    if (e != at || to <= e || to - e > len || (to < end && to - e != len)) return 1;
    at = to;
    if (accx_entry_step(e, len, (uint32_t)end) != to) return 1;
    e = to;
  }
  return at != end;
}

int main() {
  for (uint32_t len : {1u, 31u, 32u, 128u, 512u, 1024u, 1000000u, 0x80000000u, 0xffffffffu})
    for (uint64_t end : {100ull, 0x80000000ull, (1ull << 32) - 1025, (1ull << 32) - 1024, (1ull << 32) - 65, (1ull << 32) - 1})
      for (uint64_t n : {0ull, 1ull, 31ull, 64ull, 100ull, 3000ull, 5000001ull})
        if (n <= end && walk(end - n, end, len)) return printf("%u at %llu, %llu left\n", len, (unsigned long long)end, (unsigned long long)n), 1;
  for (uint32_t m = 0; m <= 300; m++) {
    if (fill<4>(m)) return printf("fill<4> of %u entries\n", m), 1;
    if (fill<8>(m)) return printf("fill<8> of %u entries\n", m), 1;
  }
  return 0;
}
"""


def test_entries(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "vector_types.h")):
        pytest.skip("no g++ or CUDA headers")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "acctricnt_gb300", "csrc"), "-I" + CUDA,
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
