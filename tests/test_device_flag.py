"""CPU: the per-device answers that the LU keeps about its kernels (csrc/qbg_device_flag.cuh),
compiled with the host compiler: every device is asked on its own, yes and no
are both kept, and a device beyond the table is asked each time."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "quantumbilliards.jl_gb300" / "csrc"
MAIN = r"""
#include <cstdio>
#include "qbg_device_flag.cuh"
int main() {
  qbg::DeviceFlag f;
  int asked = 0;
  auto yes = [&] { ++asked; return true; };
  auto no = [&] { ++asked; return false; };
  bool ok = f.get(0, yes) && f.get(0, no) && asked == 1;   // device 0: kept
  ok = ok && !f.get(1, no) && asked == 2 && !f.get(1, yes) && asked == 2;  // device 1 has its own answer
  ok = ok && f.get(63, yes) && f.get(0, no) && !f.get(1, yes) && asked == 3;
  ok = ok && f.get(64, yes) && !f.get(64, no) && f.get(-1, yes) && asked == 6;  // beyond the table
  std::puts(ok ? "ok" : "wrong");
}
"""


def test_every_device_is_asked(tmp_path):
    src = tmp_path / "flag.cpp"
    src.write_text(MAIN)
    exe = tmp_path / "flag"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.strip() == "ok"


def test_the_lu_keeps_no_answer_for_the_process():
    text = (CSRC / "qbg_linalg.cu").read_text()
    kernels = [i for i in range(len(text)) if text.startswith("cudaFuncAttributeMaxDynamicSharedMemorySize", i)]
    assert kernels
    assert "static const bool" not in text and "static std::atomic<bool>" not in text
    assert "static bool panel_attr" not in text
