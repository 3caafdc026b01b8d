"""Function attributes are a device's, not a process's: the helper that keeps what was
set or asked for each device, and that nothing keeps it in a plain static beside it."""
import glob
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hwyblas_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "internal.h"
namespace hb {
static Context g_context;
Context& Ctx() { return g_context; }
}  // namespace hb
int main() {
  hb::PerDevice<int> value;
  int calls = 0;
  for (int device : {0, 0, 3, 0, 3, 63, 64, 64, -1, 63}) {
    hb::Ctx().device = device;
    const int v = value.Get([&] { return ++calls, 100 * calls + device; });
    std::printf("%d:%d ", device, v);
  }
  std::printf("calls %d\n", calls);
}
"""


def test_once_for_each_device(tmp_path):
    include = "/usr/local/cuda/include"
    if not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", f"-I{include}", str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    # Devices beyond the table ask every time.
    assert out.split() == ["0:100", "0:100", "3:203", "0:100", "3:203", "63:363", "64:464",
                           "64:564", "-1:599", "63:363", "calls", "6"]


def test_no_attribute_is_kept_for_the_process():
    found = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = open(path).read()
        for use in re.finditer(r"cudaFuncSetAttribute\(|cudaOccupancyMax\w+\(", text):
            head = max(m.start() for m in re.finditer(r"^[A-Za-z].*[({]$|^[A-Za-z].*,$", text, re.M)
                       if m.start() < use.start())
            body = text[head:use.start()]
            statics = [s for s in re.findall(r"\bstatic (?:const |thread_local )?\w+[^;(]*;?", body)
                       if "PerDevice<" not in s and not s.startswith("static void")]
            assert not statics, (os.path.basename(path), statics)
            found += 1
    assert found > 20
