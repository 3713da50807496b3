"""The host conversions' thread loop (csrc/host_threads.h) where the system refuses threads: the
loop's own header in a small program whose `pthread_create` fails after a given number of starts
(the answer at a process or thread limit). Every value is still taken exactly once and the program
ends normally: no thread is left running, nothing terminates the process."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ptyrs_b200",
                    "csrc")

PROGRAM = r"""
#include "host_threads.h"

#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>

static int allowed = 0, started = 0;

extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
  using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static const Create real = reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"));
  if (started >= allowed) return EAGAIN;
  ++started;
  return real(t, a, f, x);
}

int main(int argc, char** argv) {
  allowed = atoi(argv[1]);
  const size_t n = strtoull(argv[2], nullptr, 10), each = strtoull(argv[3], nullptr, 10);
  std::vector<std::atomic<int>> taken(n);
  ptyb::eng::parallel_range(n, each, 16, [&](size_t b, size_t e) {
    for (size_t i = b; i < e; ++i) ++taken[i];
  });
  for (size_t i = 0; i < n; ++i)
    if (taken[i] != 1) return 1;
  printf("%d", started);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("host_threads")
    src, exe = d / "main.cpp", d / "main"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-D_GNU_SOURCE", "-I", CSRC, str(src), "-o",
                    str(exe), "-pthread", "-ldl"], check=True)
    return str(exe)


# threads allowed; values; values a thread at least (n / each threads, at most one a core)
@pytest.mark.parametrize("allowed", [0, 1, 2, 100])
@pytest.mark.parametrize("n,each", [(0, 1), (1, 2), (1000, 1001), (1001, 10), (100003, 1)])
def test_every_value_once_at_a_thread_limit(program, allowed, n, each):
    res = subprocess.run([program, str(allowed), str(n), str(each)], capture_output=True,
                         text=True, timeout=60)
    assert res.returncode == 0, res.stderr
    assert int(res.stdout) <= min(allowed, 16, n // each)
