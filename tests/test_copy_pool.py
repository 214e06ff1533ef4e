"""The host threads that copy rows beside a transfer (csrc/copypool.h), on the
CPU: every task of a job runs once, whatever the number of threads; a job
started with begin() runs while the caller does something else or helps; and a pool whose
threads cannot all be made (here: no address space left for their stacks) works
with those it has, the calling thread at the least."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "amrex_euler_allmach_explicit_imex_b200", "csrc")

DRIVER = r"""
#include "copypool.h"
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <sys/resource.h>

static long vm_bytes()
{
  long pages = 0;
  FILE* f = std::fopen("/proc/self/statm", "r");
  if (!f || std::fscanf(f, "%ld", &pages) != 1) std::abort();
  std::fclose(f);
  return pages * 4096;
}

static int check(CopyPool& pool)
{
  for (int n : {0, 1, 3, 1000}) {
    std::vector<std::atomic<int>> hits(n);
    pool.run(n, [&](int k) { ++hits[k]; });
    for (auto& h : hits)
      if (h != 1) return 1;
    // held back: the threads wait for the caller between begin and finish
    std::atomic<int> open{0}, ran{0};
    const std::function<void(int)> f = [&](int k) {
      while (open <= k) std::this_thread::yield();
      ++ran;
    };
    CopyPool::Job job;
    job.f = &f;
    job.n = n;
    pool.begin(job);
    for (int k = 0; k < n; ++k) {
      open = k + 1;
      if (k % 3 == 0) pool.help(job, open);
    }
    while (pool.help(job, n / 2)) {
    }
    if (pool.help(job, 0)) return 4;
    pool.finish(job);
    if (ran != n) return 2;
  }
  return 0;
}

int main(int, char** argv)
{
  const int workers = std::atoi(argv[1]);
  const long room = std::atol(argv[2]);
  auto hold = std::make_unique<std::vector<char>>(1 << 16);
  if (room > 0) {
    const rlim_t limit = vm_bytes() + room;
    rlimit r{limit, limit};
    if (setrlimit(RLIMIT_AS, &r) != 0) return 3;
  }
  CopyPool pool(workers);
  const int rc = check(pool);
  std::printf("%d", pool.workers());
  return rc;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("pool")
    src, exe = d / "pool.cpp", d / "pool"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("workers", [0, 1, 7])
def test_every_task_runs_once(driver, workers):
    r = subprocess.run([driver, str(workers), "0"], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == str(workers)


@pytest.mark.parametrize("room", [1 << 20, 20 << 20])
def test_threads_that_cannot_be_made(driver, room):
    r = subprocess.run([driver, "12", str(room)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout) < 12
