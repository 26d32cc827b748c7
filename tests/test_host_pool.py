"""The host threads behind reads and queries: all work is done, by the caller where no thread
(or only some) can be started, since the reads needed none before they were split."""
import os
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "host/host_pool.hpp"
#include <cerrno>
#include <dlfcn.h>
#include <pthread.h>
#include <cstdio>
static int left = ALLOWED;
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
  if (left-- <= 0) return EAGAIN;
  using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  return reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, x);
}
int main() {
  rtg::HostPool pool;
  std::vector<unsigned char> from(5000001), to(from.size(), 0);
  for (std::size_t k = 0; k < from.size(); ++k) from[k] = static_cast<unsigned char>(k * 7 + k / 251);
  for (int round = 0; round < 3; ++round) {
    std::fill(to.begin(), to.end(), 0);
    pool.copy(to.data(), from.data(), from.size());
    if (to != from) return 1;
    std::vector<std::atomic<int>> ran(1000);
    pool.run(ran.size(), [&](std::size_t k) { ran[k].fetch_add(1); });
    for (auto& r : ran)
      if (r.load() != 1) return 2;
  }
  return 0;
}
"""


@pytest.mark.parametrize("allowed", [0, 1, 100])
def test_work_is_done_with_the_threads_there_are(tmp_path, allowed):
    (tmp_path / "pool.cpp").write_text(PROGRAM)
    exe = tmp_path / "pool"
    subprocess.check_call(["g++", "-std=c++20", "-O1", f"-DALLOWED={allowed}", "-D_GNU_SOURCE",
                           "-I" + os.path.join(ROOT, "ray-tracer_b200", "csrc"), str(tmp_path / "pool.cpp"), "-o",
                           str(exe), "-lpthread", "-ldl"])
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
