"""Values kept per device (csrc/per_device.h): threads that come for one at the same time, without the interpreter lock, all get the
same complete value."""
import re
import subprocess
from pathlib import Path

import superscaler_b200

CSRC = Path(superscaler_b200.__file__).parent / "csrc"

PROGRAM = r"""
#include "per_device.h"
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
struct Value {
  static std::atomic<int> made, alive;
  int parts[64];
  Value() {
    made++; alive++;
    for (int i = 0; i < 64; ++i) { parts[i] = i; if (i % 16 == 0) std::this_thread::sleep_for(std::chrono::milliseconds(1)); }
  }
  Value(Value&& o) { alive++; for (int i = 0; i < 64; ++i) parts[i] = o.parts[i]; }
  ~Value() { alive--; }
};
std::atomic<int> Value::made{0}, Value::alive{0};
int main() {
  static ssb::PerDevice<Value> values;
  constexpr int kThreads = 16, kDevices = 3;
  Value* got[kThreads][kDevices];
  std::atomic<int> ready{0};
  std::vector<std::thread> threads;
  for (int t = 0; t < kThreads; ++t)
    threads.emplace_back([&, t] {
      ready++;
      while (ready < kThreads) {}
      for (int d = 0; d < kDevices; ++d) {
        Value& v = values.get((d + t) % kDevices, [] { return Value(); });
        for (int i = 0; i < 64; ++i) if (v.parts[i] != i) std::puts("incomplete");
        got[t][(d + t) % kDevices] = &v;
      }
    });
  for (auto& t : threads) t.join();
  for (int t = 0; t < kThreads; ++t)
    for (int d = 0; d < kDevices; ++d)
      if (got[t][d] != got[0][d] || (d && got[t][d] == got[t][d - 1])) std::puts("not one value per device");
  if (Value::alive != kDevices) std::puts("values left over");
  if (Value::made < kDevices) std::puts("too few made");
  std::puts("done");
}
"""


def test_threads_that_come_together_share_one_complete_value(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", f"-I{CSRC}", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    for _ in range(5):
        assert subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True, timeout=60).stdout == "done\n"


def test_lazily_made_device_values_go_through_it():
    """A function-local tensor that is filled in on first use is a race between the forward's and the backward's thread."""
    code = re.sub(r"//[^\n]*", "", (CSRC / "bindings.cpp").read_text())
    for name in ("num_sms", "status_tensor", "ticket_tensor"):
        body = code[code.index(f" {name}() {{"):]
        body = body[:body.index("\n}")]
        assert "PerDevice<" in body and ".get(" in body
    assert not re.search(r"static\s+std::vector<\s*Tensor\s*>", code)
