"""The queue of a recurrence's convergence tests (TaskQueue, csrc/worker_pool.hpp):
results and exceptions reach the futures, whichever thread reads them and whether they
are read at all, and the tasks of many callers run on no more threads than it was
given. Host code, compiled here."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pyqcm_b200", "csrc")

DRIVER = r"""
#include <chrono>
#include <cstdio>
#include <set>
#include <stdexcept>
#include <vector>
#include "worker_pool.hpp"
int main() {
  qed::TaskQueue<double> &q = *new qed::TaskQueue<double>(5);
  std::mutex m;
  std::set<std::thread::id> ids;
  std::atomic<int> wrong{0}, ran{0}, now{0}, most{0};
  auto caller = [&](int c) {
    std::vector<std::future<double>> f;
    for (int i = 0; i < 200; ++i) {
      std::vector<double> own(100, c + i);  // goes with the task
      f.push_back(q.submit([&, i, own] {
        const int n = ++now;
        for (int o = most; n > o && !most.compare_exchange_weak(o, n);) {}
        { std::lock_guard<std::mutex> l(m); ids.insert(std::this_thread::get_id()); }
        std::this_thread::sleep_for(std::chrono::microseconds(50));
        --now;
        ++ran;
        if (i % 17 == 3) throw std::runtime_error("task");
        return own[i % 100];
      }));
      if (f.size() > 8 && i % 31 == 0) f.erase(f.begin());  // a result that nobody reads
    }
    for (auto &x : f) {
      try {
        const double v = x.get();
        wrong += !(v >= c && v < c + 200);
      } catch (const std::runtime_error &) {
      }
    }
  };
  std::vector<std::thread> t;
  for (int c = 0; c < 12; ++c) t.emplace_back(caller, 1000 * c);
  for (auto &x : t) x.join();
  while (ran < 12 * 200) std::this_thread::yield();
  qed::TaskQueue<double> &none = *new qed::TaskQueue<double>(0);  // no thread: the caller's own
  auto own = none.submit([] { return 7.0; });
  wrong += own.wait_for(std::chrono::seconds(0)) != std::future_status::ready || own.get() != 7.0;
  printf("%d %d %d\n", wrong.load(), (int)ids.size(), most.load());
  fflush(stdout);
  return 0;
}
"""


def test_tasks_run_once_on_few_threads(tmp_path):
    src, exe = tmp_path / "drv.cpp", tmp_path / "drv"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    wrong, threads, most = map(int, r.stdout.split())
    assert wrong == 0
    assert threads <= 5 and most <= 5
