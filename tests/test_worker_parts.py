"""The parts of a solve on the worker pool (run_parts, csrc/worker_pool.hpp): every
part runs once; a part that fails ends the run, and its own thread has drained its
work before the caller goes on, which may free what that work reads; a pool that is
taken runs nothing. Host code, compiled here."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pyqcm_b200", "csrc")

DRIVER = r"""
#include <chrono>
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>
#include "worker_pool.hpp"

// a stand-in for a thread's stream: work under way ends some time after it was started
struct Stream {
  std::chrono::steady_clock::time_point end;
  bool busy() const { return std::chrono::steady_clock::now() < end; }
};
thread_local Stream *mine = nullptr;
std::vector<Stream *> all;
std::mutex all_m;
Stream &stream() {
  if (!mine) {
    mine = new Stream{};
    std::lock_guard<std::mutex> l(all_m);
    all.push_back(mine);
  }
  return *mine;
}

int main() {
  qed::WorkerPool &pool = *new qed::WorkerPool;
  auto drain = [] { while (stream().busy()) std::this_thread::yield(); };
  int wrong = 0, busy = 0, taken = 0;
  for (int r = 0; r < 200; ++r) {
    const int n = 1 + r % 9, bad = r % 3 == 0 ? (r / 3) % n : -1;
    std::vector<std::atomic<int>> ran(n);
    for (auto &x : ran) x = 0;
    auto part = [&](int i) {  // returns with its stream idle, unless it throws
      ran[i]++;
      stream().end = std::chrono::steady_clock::now() + std::chrono::microseconds(500);
      if (i == bad) throw std::runtime_error("part");
      drain();
    };
    const bool ok = qed::run_parts(pool, 1 + r % 5, n, [&](int i) {
      try { part(i); } catch (const std::exception &) { return false; }
      return true;
    }, drain);
    { std::lock_guard<std::mutex> l(all_m); for (Stream *s : all) busy += s->busy(); }
    wrong += ok != (bad < 0);
    for (int i = 0; i < n; ++i) wrong += ok ? ran[i] != 1 : ran[i] > 1;
  }
  // from inside a run the pool is taken: nothing runs
  qed::run_parts(pool, 1, 1, [&](int) {
    std::thread([&] { taken += qed::run_parts(pool, 2, 3, [&](int) { taken += 100; return true; }, drain); }).join();
    return true;
  }, drain);
  printf("%d %d %d\n", wrong, busy, taken);
  fflush(stdout);
  return 0;
}
"""


def test_failed_part_is_drained_before_the_caller_goes_on(tmp_path):
    src, exe = tmp_path / "drv.cpp", tmp_path / "drv"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == ["0", "0", "0"]
