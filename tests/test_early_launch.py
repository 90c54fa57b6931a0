"""Source check of the kernels that are set up while the work before them on the stream still runs: whatever they
read may still be written when they start, so none of their loads may be one that the compiler takes to be of data
that nothing writes meanwhile (__ldg, ld.global.nc, a __restrict__ pointer)."""

import re

from conftest import ROOT

CSRC = ROOT / "stdgpu_gb300" / "csrc"


def _code(path):
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _with_includes(path, seen):
    """The file and what it includes from this repository."""
    if path in seen or not path.exists():
        return
    seen.add(path)
    for name in re.findall(r'#include "([^"]+)"', path.read_text()):
        for base in (path.parent, CSRC, ROOT / "include"):
            _with_includes(base / name, seen)


def test_early_launched_kernels_use_no_read_only_loads():
    units = [p for p in sorted(CSRC.glob("*.cu")) if "wait_for_stream()" in _code(p)]
    assert units, "no early-launched kernel found"
    files = set()
    for unit in units:
        _with_includes(unit, files)
    bad = [f"{p.relative_to(ROOT)}:{k}: {line.strip()}" for p in sorted(files)
           for k, line in enumerate(_code(p).splitlines(), 1)
           if re.search(r"__ldg\b|ld\.global\.nc|__restrict", line)]
    assert not bad, "\n".join(bad)


def test_every_early_launched_kernel_waits_first():
    """wait_for_stream() is the first statement of each kernel that launch_early starts."""
    for unit in sorted(CSRC.glob("*.cu")):
        code = _code(unit)
        early = set(re.findall(r"launch_early(?:_shared)?\(\s*(\w+)", code))
        early |= set(re.findall(r"cudaLaunchKernelEx\(&cfg, (\w+)", code))
        for name in sorted(early - {"kernel"}):
            body = re.search(r"__launch_bounds__\([^{;]*\)?\s*" + name + r"\([^{;]*\)\s*\{(.*?)\n\}", code, re.S) or \
                re.search(r"__global__[^{;]*\b" + name + r"\([^{;]*\)\s*\{(.*?)\n\}", code, re.S)
            assert body, (unit.name, name)
            assert body.group(1).lstrip().startswith("wait_for_stream();"), (unit.name, name)
