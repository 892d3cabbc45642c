"""HostPages without memory: whichever host allocation fails while its threads are started,
nothing is thrown and the buffer stays as it was (CPU, compiled with the host compiler)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <new>
#include "host_pages.h"

static long fail_at = -1;  // the allocation that fails from now on (-1: none)
void *operator new(std::size_t n) {
  if (fail_at >= 0 && fail_at-- == 0) throw std::bad_alloc();
  if (void *p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

int main() {
  const long n = 3 << 20;  // 24 MiB
  double *x = static_cast<double *>(std::malloc(n * sizeof(double)));
  for (long i = 0; i < n; i++) x[i] = i;
  for (long f = -1; f < 12; f++) {
    fail_at = f;
    scess::HostPages pages(x, n);
    fail_at = -1;
    pages.wait();
  }
  for (long i = 0; i < n; i++)
    if (x[i] != i) return 1;
  std::puts("fine");
  return 0;
}
"""


def test_failing_allocations_are_not_passed_on(tmp_path):
    cxx = shutil.which('g++')
    if not cxx:
        pytest.skip('no host compiler')
    src, exe = tmp_path / 'pages.cpp', tmp_path / 'pages'
    src.write_text(SOURCE)
    subprocess.run([cxx, '-std=c++17', '-O1', '-pthread', '-I', os.path.join(ROOT, 'scess_gb300', 'csrc'), str(src),
                    '-o', str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and 'fine' in r.stdout, r.stderr
