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


ONCE = r"""
#include "per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
int main() {
  static ssb::OncePerDevice<> once;
  int asked[3] = {}, value = 0;
  auto ask = [&](int device, int rc, int answer) {
    return once.get(device, &value, [&](int* v) { asked[device]++; *v = answer; return rc; });
  };
  if (ask(0, 0, 7) != 0 || value != 7 || ask(0, 0, 9) != 0 || value != 7 || asked[0] != 1) std::puts("not kept");
  if (ask(1, 0, 8) != 0 || value != 8 || asked[1] != 1) std::puts("the other device was not asked");
  if (ask(2, -5, 3) != -5 || ask(2, 0, 4) != 0 || value != 4 || asked[2] != 2) std::puts("an error was kept");
  static ssb::OncePerDevice<> shared;
  std::vector<std::thread> threads;
  for (int t = 0; t < 16; ++t)
    threads.emplace_back([&] {
      for (int d = 0; d < 64; ++d) {
        int v = 0;
        if (shared.get(d, &v, [&](int* x) { *x = d + 1; return 0; }) != 0 || v != d + 1) std::puts("wrong value");
      }
    });
  for (auto& t : threads) t.join();
  std::puts("done");
}
"""


def test_what_is_set_once_is_set_on_every_device(tmp_path):
    (tmp_path / "t.cpp").write_text(ONCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", f"-I{CSRC}", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True, timeout=60).stdout == "done\n"


def test_launchers_keep_no_flag_of_the_process():
    """A function-local number or flag that a launcher sets belongs to the process; what it stands for belongs to a device."""
    for path in sorted(CSRC.glob("*.cu")):
        code = re.sub(r"//[^\n]*", "", path.read_text())
        assert not re.search(r"^\s+static\s+(?:bool|int)\s+\w+\s*=", code, re.M), path.name
