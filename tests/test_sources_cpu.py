"""Rules of the kernel sources that no compiler checks."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vmamba_b200", "csrc")


def test_dynamic_shared_memory_declares_its_alignment():
    """Parts of it are read and written as 16-byte vectors: its start has to be aligned by declaration, not by chance."""
    found = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        for line in re.findall(r"extern\s+__shared__[^;]*;", open(path).read()):
            assert re.search(r"__align__\((16|32|64|128|1024)\)", line), (os.path.basename(path), line)
            found += 1
    assert found > 10


def test_limits_of_shared_memory_only_grow():
    """They belong to a kernel and all threads that launch it: one function sets them, under a lock."""
    sets = {os.path.basename(p): open(p).read().count("cudaFuncSetAttribute(") for p in glob.glob(os.path.join(CSRC, "*")) if os.path.isfile(p)}
    assert {p: n for p, n in sets.items() if n} == {"api.cu": 1}


def test_kernels_that_follow_one_another_read_with_ordinary_loads():
    """`launch` lets a kernel start while the one in front of it, of this library or any other, still writes.  What it waits for is
    promised to its ordinary loads alone: not to the read-only path, whose loads may also be moved in front of the wait."""
    kernels = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        src = re.sub(r"#else *\n[^#]*#endif", "", src)          # of host builds
        assert "<<<" not in src and not re.search(r"__ldg|\bld\.global\.nc|ldu", src), os.path.basename(path)
        for k in re.finditer(r"__global__\s+void[^{;]*\{\s*([^;]*;)", src):
            assert k.group(1) == "follow_previous();", (os.path.basename(path), k.group(0)[:200])
            assert "__restrict__" not in k.group(0)                              # a kernel argument that is: read-only by the compiler's own choice
            kernels += 1
    assert kernels > 35
