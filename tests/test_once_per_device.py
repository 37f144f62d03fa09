"""Setup that belongs to a device (shared-memory limits of kernels, constant
tables) runs once on every device, not once in the process (CPU: the helper
with made-up device numbers, and that every such setup goes through it)."""
import glob
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dage_b200", "csrc")

PROGRAM = r"""
#include "once_per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
int main() {
  dage::OncePerDevice once;
  int calls[200] = {};
  auto on = [&](int dev, int rc) { return once.run(dev, [&] { ++calls[dev]; return rc; }); };
  if (on(0, 0) || on(0, 0) || calls[0] != 1) return 1;  // once
  if (on(1, 0) || calls[1] != 1) return 2;              // a second device too
  if (on(2, -7) != -7 || on(2, 0) || on(2, 0) || calls[2] != 2) return 3;  // failures are retried
  if (on(130, 0) || on(130, 0) || calls[130] != 1) return 4;
  std::vector<std::thread> ts;
  for (int t = 0; t < 16; ++t) ts.emplace_back([&, t] { on(10 + t % 2, 0); });
  for (auto &t : ts) t.join();
  return calls[10] == 1 && calls[11] == 1 ? 0 : 5;
}
"""


def test_helper(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "once.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "once"
    subprocess.run([cxx, "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def _bodies(text, name):
    """Bodies of the functions in `text` that call `name` (brace matching from
    the last line that starts in column 0 with a function head)."""
    for m in re.finditer(name, text):
        head = [h for h in re.finditer(r"^[A-Za-z].*\{$|^\w.*\n? .*\) \{$", text[:m.start()], re.M)][-1]
        depth, i = 0, text.index("{", head.start())
        for j in range(i, len(text)):
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            if depth == 0:
                yield text[head.start():j + 1]
                break


def test_device_setup_keeps_no_process_wide_flag():
    """No function that sets a kernel attribute or uploads a table decides by
    a static flag of its own whether to do so."""
    seen = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = open(path).read()
        for name in ("cudaFuncSetAttribute", "cudaMemcpyToSymbol"):
            for body in _bodies(text, name):
                seen += 1
                assert not re.search(r"static (bool|int|unsigned|std::once_flag)", body), (path, body[:300])
    assert seen >= 6
