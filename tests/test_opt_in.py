"""The record of a kernel's granted shared memory (csrc/opt_in.cuh) under threads that ask for different sizes: host code,
compiled here with a stand-in for the runtime's attribute."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sager_b200", "csrc")

PROBE = r"""
#include <chrono>
#include <cstdio>
#include <thread>
#include "opt_in.cuh"

static std::atomic<int> attribute{0};

int main() {
  // the interleaving that hurts: while one thread has set the larger size and not yet recorded it, another asks for less
  sgr::SmemGrant grant;
  std::thread other;
  bool ok = grant.ensure(0, 100, [&](int n) {
    attribute = n;
    other = std::thread([&] { grant.ensure(0, 60, [&](int m) { attribute = m; return true; }); });
    std::this_thread::sleep_for(std::chrono::milliseconds(200));
    return true;
  });
  other.join();
  if (!ok || attribute < 100) { std::printf("attribute %d below the granted 100\n", attribute.load()); return 1; }
  if (!grant.ensure(0, 80, [&](int) { attribute = -1; return true; }) || attribute < 100) { std::printf("lowered\n"); return 1; }
  // many threads, two sizes, several devices: what was granted always holds
  sgr::SmemGrant g2;
  std::atomic<int> attr[4] = {}, bad{0};
  auto work = [&](int bytes) {
    for (int i = 0; i < 20000; ++i) {
      const int dev = i & 3;
      if (!g2.ensure(dev, bytes, [&](int m) { attr[dev] = m; return true; }) || attr[dev] < bytes) ++bad;
    }
  };
  std::thread a(work, 100), b(work, 60), c(work, 80);
  a.join(); b.join(); c.join();
  if (bad != 0) { std::printf("%d requests below their grant\n", bad.load()); return 1; }
  // a refusal is not recorded; ordinals past the table are refused
  sgr::SmemGrant g3;
  if (g3.ensure(0, 10, [](int) { return false; }) || !g3.ensure(0, 10, [](int) { return true; })) { std::printf("refusal kept\n"); return 1; }
  if (g3.ensure(64, 1, [](int) { return true; }) || g3.ensure(-1, 1, [](int) { return true; })) { std::printf("ordinal\n"); return 1; }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_grant_only_grows(tmp_path):
    src = tmp_path / "probe.cpp"
    src.write_text(PROBE)
    exe = str(tmp_path / "probe")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout
