"""Contracts of the kernels' sources that no run can show to be kept."""
import re

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
