"""A kernel's shared-memory limit is set once on each device (csrc/
once_per_device.h), with a stand-in for the runtime's setter: a second device
gets its own, a failure is tried again, threads may arrive together."""
import glob
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nitroozk-stwo_b200", "csrc")

PROGRAM = r"""
#include "once_per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  gs::OncePerDevice set;
  int calls[70] = {0}, fail = 0;
  auto on = [&](int d) { return set.run(d, [&] { calls[d]++; return fail; }); };
  fail = 3;
  CHECK(on(0) == 3 && on(0) == 3 && calls[0] == 2);
  fail = 0;
  CHECK(on(0) == 0 && on(0) == 0 && calls[0] == 3);
  CHECK(on(1) == 0 && on(1) == 0 && calls[1] == 1 && on(0) == 0 && calls[0] == 3);
  CHECK(on(63) == 0 && on(63) == 0 && calls[63] == 1);
  CHECK(on(64) == 0 && on(64) == 0 && calls[64] == 2);  // past the flags: set every time
  gs::OncePerDevice shared;
  std::atomic<int> made{0};
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; t++)
    threads.emplace_back([&] { for (int d = 0; d < 64; d++) shared.run(d, [&] { made++; return 0; }); });
  for (auto& t : threads) t.join();
  CHECK(made >= 64 && made <= 512);
  made = 0;
  for (int d = 0; d < 64; d++) shared.run(d, [&] { made++; return 0; });
  CHECK(made == 0);
  return 0;
}
"""


def test_once_on_each_device(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(tmp_path / "t")])
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout


def test_every_limit_is_set_through_it():
    uses = {}
    for path in glob.glob(os.path.join(CSRC, "**", "*.c*"), recursive=True):
        n = len(re.findall(r"\bcudaFuncSetAttribute\b", open(path).read()))
        if n:
            uses[os.path.basename(path)] = n
    assert uses == {"runtime.cuh": 1}, uses
