"""Contracts of the kernels' sources that no run can show to be kept."""
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "eulersr_b200" / "csrc"


def test_stage_kernels_may_run_in_place():
    """A second Runge-Kutta stage is launched with Wbase and Wout on the same
    buffer. A kernel that takes both must not promise that they do not alias,
    and must not read Wbase through the non-coherent path, which is only
    defined for memory that the launch does not write."""
    kernels = 0
    for path in sorted(CSRC.glob("*.cuh")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__[^{;]*?\bk_\w+\(([^)]*\bWbase\b[^)]*)\)\s*\{", text):
            kernels += 1
            for name in ("Wbase", "Wout"):
                decl = re.search(r"[^,(]*\b%s\b" % name, m.group(1)).group(0)
                assert "__restrict__" not in decl, (path.name, decl)
        readers = set(re.findall(r"(\w+)\(\s*Wbase\b", text))
        for name in readers:
            body = re.search(r"void %s\([^)]*\)\s*\{(.*?)\n\}" % name, text, re.S)
            if body:
                assert ".nc" not in body.group(1), (path.name, name)
        assert "__ldg(Wbase" not in text
    assert kernels == 4   # k_stage, k_stage_pair, k_flux, k_flux_patch


def test_kernel_limits_are_raised_on_every_device(tmp_path):
    """esr_per_device.h: set once per device, again after a failure, and no
    kernel of the network keeps a process-wide flag of its own."""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "per_device.cpp"
    src.write_text('''
#include <cstdio>
#include <initializer_list>
#include "esr_per_device.h"
int main() {
  esr::PerDevice limit, other;
  int calls[70] = {0}, fail_once = 1, bad = 0;
  auto set = [&](int d) { ++calls[d]; return d == 2 && fail_once-- > 0 ? 7 : 0; };
  for (int r = 0; r < 3; ++r)
    for (int d : {0, 1, 5, 63}) bad += limit.once(d, set) != 0;
  for (int d : {0, 1, 5, 63}) bad += calls[d] != 1;          // every device, once
  bad += limit.once(2, set) != 7 || limit.once(2, set) != 0 || limit.once(2, set) != 0 || calls[2] != 2;
  bad += limit.once(64, set) != 0 || limit.once(64, set) != 0 || calls[64] != 2;
  bad += other.once(0, set) != 0 || calls[0] != 2;           // another kernel's own record
  std::printf("%d\\n", bad);
  return bad != 0;
}
''')
    exe = tmp_path / "per_device"
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "0", r.stdout
    text = re.sub(r"//[^\n]*", "", (CSRC / "esr_mlp.cu").read_text())
    assert text.count("cudaFuncSetAttribute(") == 1   # in allow_smem, behind PerDevice
    assert not re.search(r"static (const )?(bool|cudaError_t) attr", text)
