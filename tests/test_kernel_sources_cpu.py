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


def test_overlapped_kernels_declare_no_constant_inputs():
    # through `const T* __restrict__` the compiler may move a load above griddep_wait() or onto the non-coherent path
    overlapped = 0
    for name, text in device_sources():
        for head in re.split(r"__global__", text)[1:]:
            signature, _, body = head.partition(") {")
            if "griddep_wait()" in body:
                overlapped += 1
                assert not re.search(r"\bconst\b[^,(]*\*\s*__restrict__", signature), (name, signature)
    assert overlapped >= 15      # the pattern still finds the kernels


def test_a_wait_that_ran_out_can_be_told_from_every_other():
    # the status record names the wait by its site; 0x700 is the self-test's, as the public header says
    sites = {}
    for name, text in device_sources():
        found = re.findall(r"(?:p\.)?status, (\([^)]*\)|0x[0-9a-f]+)", text)
        codes = [int(c, 16) for f in found for c in re.findall(r"0x[0-9a-f]+", f)]
        assert len(codes) == len(set(codes)), (name, [hex(c) for c in codes])
        sites[name] = codes
    assert [name for name, codes in sites.items() if 0x700 in codes] == ["dg_cast_kernels.cuh"]
    assert sum(map(len, sites.values())) >= 20      # the pattern still finds the waits


def test_loops_over_a_grid_end():
    # work that fits 32 bits may end less than one stride below 2^32: a 32-bit counter that only adds would wrap round and never end
    strided = 0
    for name, text in device_sources():
        loops = re.findall(r"for \((\w+) \w+ = [^;]*blockIdx\.x[^;]*;[^;]*;[^)]*\+=", text)
        assert all(kind == "uint64_t" for kind in loops), (name, loops)
        strided += len(loops)
    assert strided >= 2      # the pattern still finds the loops
