"""The threads that copy host buffers (csrc/sbb_copy_threads.h, host code only), compiled into a small program: every byte
arrives whatever the size and however many threads ask at once, and also when the system gives no or few threads."""
import os
import shutil
import subprocess

import pytest

from conftest import REPO

PROGRAM = r"""
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <dlfcn.h>
#include <pthread.h>
#include "sbb_copy_threads.h"

static std::atomic<int> asked{0};

// The system's limit on threads, in place of the real call: the first THREADS_ALLOWED succeed.
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
  static std::atomic<int> left{std::getenv("THREADS_ALLOWED") ? std::atoi(std::getenv("THREADS_ALLOWED")) : 1 << 20};
  if (left.fetch_sub(1) <= 0) return EAGAIN;
  asked.fetch_add(1);
  typedef int (*Create)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
  static const Create real = reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"));
  return real(t, a, f, arg);
}

static bool copies(unsigned seed) {
  std::vector<unsigned char> src(6 << 20), dst(src.size() + 2);
  for (size_t k = 0; k < src.size(); ++k) src[k] = (unsigned char)((k * 2654435761u + seed) >> 13);
  const size_t sizes[] = {0, 1, 4095, 65536, 65537, 131072, 524287, 524288, 524288 + 32768 + 15, 262143, 262144, 262145, 262144 + 131072, 1000001, 3 << 20, (6 << 20) - 7};
  for (int round = 0; round < 6; ++round)
    for (size_t n : sizes) {
      std::memset(dst.data(), 0xEE, n + 2);
      sbb::CopyThreads::get().copy(dst.data() + 1, src.data(), n, round & 1);
      if (std::memcmp(dst.data() + 1, src.data(), n) != 0 || dst[0] != 0xEE || dst[n + 1] != 0xEE) {
        std::printf("wrong copy of %zu bytes\n", n);
        return false;
      }
    }
  return true;
}
int main(int argc, char **) {
  if (!copies(1)) return 1;   // (the first copy starts the threads)
  if (argc > 1) return std::printf("%d", asked.load()) < 0;
  std::atomic<int> bad{0};
  std::vector<std::thread> callers;
  for (unsigned k = 0; k < 4; ++k) callers.emplace_back([&bad, k] { bad += !copies(k + 2); });
  for (auto &c : callers) c.join();
  return bad.load();
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs a host compiler")
    d = tmp_path_factory.mktemp("copy")
    src, exe = str(d / "copy.cpp"), str(d / "copy")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-D_GNU_SOURCE", "-pthread", "-I" + os.path.join(REPO, "streambrain_b200", "csrc"), src,
                    "-o", exe, "-ldl"], check=True, timeout=300)
    return exe


def test_copies_from_several_callers(program):
    run = subprocess.run([program], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr


@pytest.mark.parametrize("allowed", [0, 1])
def test_copies_without_the_threads_it_asked_for(program, allowed):
    run = subprocess.run([program, "one caller"], capture_output=True, text=True, timeout=120, env=dict(os.environ, THREADS_ALLOWED=str(allowed)))
    assert run.returncode == 0, run.stdout + run.stderr


def test_processes_of_one_machine_share_its_threads(program):
    """With the number of processes that a launcher started here, each takes its part of the threads, down to none."""
    def workers(env):
        run = subprocess.run([program, "one caller"], capture_output=True, text=True, timeout=120, env=env)
        assert run.returncode == 0, run.stdout + run.stderr
        return int(run.stdout)
    env = {k: v for k, v in os.environ.items() if k != "LOCAL_WORLD_SIZE"}
    alone = workers(env)
    cores = os.cpu_count()
    assert alone <= 11 and alone == max(0, min(12, min(cores, len(os.sched_getaffinity(0))) // 4 * 3) - 1)
    assert workers(dict(env, LOCAL_WORLD_SIZE="1")) == alone
    for processes in (2, 8):
        part = workers(dict(env, LOCAL_WORLD_SIZE=str(processes)))
        assert part <= alone and processes * (part + 1) <= max(processes, cores)
    assert workers(dict(env, LOCAL_WORLD_SIZE=str(cores))) == 0
    one = sorted(os.sched_getaffinity(0))[:1]
    run = subprocess.run(["taskset", "-c", str(one[0]), program, "one caller"], capture_output=True, text=True, timeout=120, env=env) \
        if shutil.which("taskset") else None
    assert run is None or (run.returncode == 0 and int(run.stdout) == 0)
