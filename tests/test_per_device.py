"""What the library asks of the CUDA runtime about a kernel belongs to one
device, and contexts of several devices share a process: such answers are kept
per device (zyklop_b200/csrc/per_device.hpp) and never in a function-local
static (CPU only; devices are numbers here)."""
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "zyklop_b200", "csrc")

SRC = r"""
#include <cstdio>
#include <stdexcept>
#include "per_device.hpp"
int made = 0;
int value(int dev, bool fail) {
  static zk::PerDevice<int> known;
  return known.get(dev, [&] {
    made++;
    if (fail) throw std::runtime_error("lookup");
    return 10 * dev;
  });
}
void show(int dev) {
  const int v = value(dev, false);
  printf("%d:%d ", v, made);
}
int main() {
  show(0);
  show(0);  // kept
  show(1);  // another device has its own
  show(0);
  try { value(2, true); } catch (const std::exception&) { printf("threw "); }
  show(2);  // a failed lookup is not kept
}
"""


def test_one_lookup_per_device_and_failures_are_not_kept(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-Wall", "-I", CSRC, "-o", exe,
                           str(tmp_path / "t.cpp")])
    assert subprocess.check_output([exe], text=True) == "0:1 0:1 10:2 0:2 threw 20:4 "


def test_no_runtime_answer_is_kept_in_a_static():
    found = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cpp", ".hpp", ".cuh")):
            continue
        text = open(os.path.join(CSRC, name)).read()
        for m in re.finditer(r"\bstatic\s[^;={(]*=\s*", text):
            rest = text[m.end():]
            # an initialiser, up to the call of its lambda if it is one
            init = rest[: rest.index("}()" if rest.startswith("[") else ";")]
            if re.search(r"\b(cuda[A-Z]|device_sm_count)", init):
                found.append((name, " ".join(m.group(0).split())))
    assert not found, found
