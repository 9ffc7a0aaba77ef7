"""Kernels that wait on the device for the one ahead (follow_previous) are on
the SMs while it writes, where PTX allows no non-coherent load of what is
written.  No stale read can be provoked for a test, so this one reads the
sources: no explicit non-coherent load, and no read-only kernel parameter but
the tables that nothing writes while a kernel runs."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "opencl-sph_gb300", "csrc")
NEVER_WRITTEN = {("SceneDesc", "scenes"), ("CopySeg", "segs"), ("RigidWork", "work")}  # uploaded by the host


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"/\*.*?\*/", " ", open(path).read(), flags=re.S)
        yield os.path.basename(path), re.sub(r"//[^\n]*", " ", text)


def test_no_noncoherent_loads():
    for name, text in sources():
        assert not re.search(r"__ldg\s*\(|ld\.global(\.\w+)*\.nc|__ld(cs|lu|cv)\s*\(", text), name


def test_read_only_kernel_parameters_are_tables():
    kernels = 0
    for name, text in sources():
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(([^)]*)\)\s*\{", text):
            kernels += 1
            found = set(re.findall(r"const\s+(\w+)\s*\*\s*__restrict__\s+(\w+)", m.group(2)))
            assert found <= NEVER_WRITTEN, (name, m.group(1), found)
    assert kernels > 20
