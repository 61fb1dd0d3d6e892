"""The engine's host-side pools (csrc/host_pools.hpp), compiled without the
kernels: page-locked allocation is a stand-in that counts."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"))),
                            "include")

PRELUDE = r"""
#include "host_pools.hpp"
#include <cstdio>
#include <sys/wait.h>
#include <unistd.h>
#include <cstdlib>
static size_t locks = 0, locked = 0;
extern "C" cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  locks++;
  locked += n;
  *p = std::malloc(n);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
extern "C" cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError(void) { return cudaSuccess; }
#define CHECK(x) if (!(x)) { std::printf("line %d: %s (locks %zu, locked %zu)\n", __LINE__, #x, locks, locked); return 1; }
using namespace sxe;
constexpr size_t MB = 1u << 20;
"""


def _run(tmp_path, body, timeout=60):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.isdir(CUDA_INCLUDE):
        pytest.skip("no C++ compiler or CUDA headers")
    src, exe = tmp_path / "pools.cpp", tmp_path / "pools"
    src.write_text(PRELUDE + "int main() {\n" + body + "\n  return 0;\n}\n")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "sentinel-x_b200", "csrc"), "-I", CUDA_INCLUDE,
                    str(src), "-o", str(exe), "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=timeout)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("mb", [1, 200, 300, 1500])
def test_streamed_target_sets_lock_pages_once(tmp_path, mb):
    """A caller that streams batches of one size through an engine: the first
    batch locks pages, at most a quarter and 16 MB more than it needs."""
    _run(tmp_path, f"""
  HostBytePool pool;
  for (int i = 0; i < 5; i++) {{
    HostBytes v = pool.take({mb} * MB);
    CHECK(v.capacity() >= {mb} * MB);
    pool.give(std::move(v));
  }}
  CHECK(locks == 1);
  CHECK(locked <= {mb} * MB + std::min<size_t>({mb} * MB / 4, 16 * MB) + 64);""")


def test_row_copies_keep_a_bounded_amount(tmp_path):
    """The row copies' pool: buffers of a chunk's size are kept, two at most,
    larger ones (one very long pair) are freed."""
    _run(tmp_path, """
  HostBytePool pool(256 * MB);
  for (int i = 0; i < 4; i++) pool.give(pool.take(128 * MB));
  CHECK(locks == 1);
  pool.give(pool.take(300 * MB));
  pool.give(pool.take(300 * MB));
  CHECK(locks == 3);
  pool.give(pool.take(128 * MB));
  CHECK(locks == 3);""")


def test_workers_in_a_forked_child(tmp_path):
    """A forked child has none of the pool's threads: its loops still run, and
    the pool (freed with the engine when the child's interpreter exits) waits
    for nobody.  The parent's pool goes on as before."""
    _run(tmp_path, r"""
  WorkerPool pool(4);
  std::atomic<int> sum{0};
  pool.run(1000, 4, [&](size_t) { sum++; });
  CHECK(sum == 1000);
  const pid_t child = fork();
  if (child == 0) {
    alarm(20);
    {
      WorkerPool* p = &pool;
      p->run(1000, 4, [&](size_t) { sum++; });
      p->~WorkerPool();
    }
    _exit(sum == 2000 ? 0 : 2);
  }
  int status = 0;
  CHECK(waitpid(child, &status, 0) == child);
  CHECK(WIFEXITED(status) && WEXITSTATUS(status) == 0);
  pool.run(1000, 4, [&](size_t) { sum++; });
  CHECK(sum == 2000);""")


def test_workers_started_after_a_fork(tmp_path):
    """A pool whose threads a child starts itself is the child's own."""
    _run(tmp_path, r"""
  WorkerPool pool(4);
  std::atomic<int> sum{0};
  const pid_t child = fork();
  if (child == 0) {
    alarm(20);
    pool.run(1000, 4, [&](size_t) { sum++; });
    pool.~WorkerPool();
    _exit(sum == 1000 ? 0 : 2);
  }
  int status = 0;
  CHECK(waitpid(child, &status, 0) == child);
  CHECK(WIFEXITED(status) && WEXITSTATUS(status) == 0);""")
