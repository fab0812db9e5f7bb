"""Loops over host threads (srs_parallel.h): threads that cannot be created are
done without, and an exception reaches the caller instead of ending the process."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# pthread_create that refuses after the first `allowed` calls
PROGRAM = r"""
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include "srs_parallel.h"
static int allowed = 0;
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* p) {
  using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static Fn real = (Fn)dlsym(RTLD_NEXT, "pthread_create");
  return allowed-- > 0 ? real(t, a, f, p) : EAGAIN;
}
int main(int argc, char** argv) {
  allowed = atoi(argv[1]);
  const int n = atoi(argv[2]), bad = atoi(argv[3]);
  std::vector<int> hits(n, 0);
  try {
    srs::host_parallel(n, 8, [&](int i) {
      if (i == bad) throw std::runtime_error("bad item");
      hits[i]++;
    });
  } catch (const std::runtime_error& e) {
    printf("%s\n", e.what());
    return 0;
  }
  for (int h : hits)
    if (h != 1) return 1;
  printf("done\n");
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("parallel")
    src = d / "p.cpp"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "srs_gb300", "csrc"), str(src),
                    "-o", str(d / "p"), "-ldl"], check=True)
    return str(d / "p")


@pytest.mark.parametrize("allowed", [0, 1, 100])
@pytest.mark.parametrize("n", [0, 1, 5, 1000])
def test_every_item_once(program, allowed, n):
    r = subprocess.run([program, str(allowed), str(n), "-1"], capture_output=True, text=True)
    assert (r.returncode, r.stdout) == (0, "done\n"), r.stderr


@pytest.mark.parametrize("allowed", [0, 1, 100])
@pytest.mark.parametrize("bad", [0, 7, 999])
def test_exception_reaches_the_caller(program, allowed, bad):
    r = subprocess.run([program, str(allowed), "1000", str(bad)], capture_output=True, text=True)
    assert (r.returncode, r.stdout) == (0, "bad item\n"), r.stderr
