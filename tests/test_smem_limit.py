"""The bookkeeping of raised shared-memory limits (``csrc/atb_smem.hpp``) on a fake
device call: every device is raised for itself, once, never lowered, and again
after a failure; threads that raise it to different sizes leave the largest."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "atb_smem.hpp"
#include <cstdio>
#include <thread>
#include <vector>
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main() {
  size_t limit[3] = {0, 0, 0};
  int calls = 0;
  bool fails = false;
  atb::SmemLimit L;
  auto launch = [&](int dev, size_t bytes) {
    L.raise(dev, bytes, [&] { ++calls; if (fails) return 1; limit[dev] = bytes; return 0; });
    return bytes <= atb::SmemLimit::kDefault || (dev < 3 && bytes <= limit[dev]);
  };
  CHECK(launch(0, 1000) && calls == 0);
  CHECK(launch(0, 60000) && calls == 1);
  CHECK(launch(0, 60000) && launch(0, 50000) && calls == 1);
  CHECK(launch(1, 60000) && calls == 2);  // another device of the same process
  CHECK(launch(0, 90000) && calls == 3 && limit[1] == 60000);
  CHECK(launch(0, 60000) && limit[0] == 90000);
  fails = true;
  CHECK(!launch(2, 60000) && calls == 4);
  fails = false;
  CHECK(launch(2, 60000) && calls == 5);
  size_t shared = 0;
  atb::SmemLimit M;
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; ++t)
    ts.emplace_back([&, t] {
      for (int i = 0; i < 2000; ++i) {
        const size_t b = 50000 + 1000 * ((t * 7 + i) % 97);
        M.raise(0, b, [&] { shared = b; return 0; });
      }
    });
  for (auto& t : ts) t.join();
  CHECK(shared == 50000 + 1000 * 96);
  return 0;
}
"""


def test_limits_per_device(tmp_path):
    src, exe = tmp_path / "smem.cpp", tmp_path / "smem"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(ROOT, "atum.jl_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
