"""Rules of the CUDA sources that no output shows while it happens to be right."""
import glob
import os
import re

import __graft_entry__ as ge

CSRC = os.path.join(ge.PKG_DIR, "csrc")


def _sources():
    """Path -> text of every kernel file, comments taken out."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path, encoding="utf-8") as f:
            out[os.path.basename(path)] = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
    return out


def test_kernels_launched_early_use_no_non_coherent_loads():
    """A kernel under programmatic dependent launch is resident while the call
    before it may still write its source: that memory is not read-only for the
    kernel's lifetime, as ld.global.nc (__ldg) requires."""
    sources = _sources()
    early = [n for n, s in sources.items() if n.endswith(".cuh") or "grid_dependency_wait" in s]
    assert len(early) > 5
    assert [n for n in early if re.search(r"__ldg\s*\(|ld\.global\.nc", sources[n])] == []


def test_asynchronous_copies_are_ordered_for_the_compiler():
    """A copy into a staged slot that is read and refilled: without a "memory"
    clobber the compiler may move the read behind the copy."""
    copies = []
    for name, s in _sources().items():
        copies += [(name, m) for m in re.findall(r'asm volatile\(\s*"cp\.async\.c[ag][^;]*;.*?\);', s, flags=re.S)]
    assert len(copies) >= 6
    assert [c for c in copies if '"memory"' not in c[1]] == []
