"""Rules that every kernel source keeps and no run on a GPU can show: what a breach of them does depends on timing."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepgemm_rust_b200", "csrc")


def device_sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            yield os.path.basename(path), re.sub(r"//[^\n]*", "", f.read())


def test_no_non_coherent_loads():
    # kernels overlap the one before them in the stream (programmatic serialisation), so their inputs may still be written while
    # they are resident; the non-coherent load path is defined only for data that is read-only for a kernel's whole lifetime
    for name, text in device_sources():
        assert not re.search(r"ld\.global\.nc|__ldg\s*\(", text), name
