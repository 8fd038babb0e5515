"""The kernels are launched so that a grid may exist while the kernel before it still writes. The non-coherent load path is
only for data that nobody writes for as long as the grid exists, so no kernel uses it, and none gives the compiler leave to."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hipkittens_b200", "csrc")


@pytest.mark.parametrize("name", sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu*"))))
def test_no_load_assumes_that_its_data_is_never_written(name):
    with open(os.path.join(CSRC, name)) as f:
        code = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
    assert not re.findall(r"__ldg\b|__restrict__|\.global\.nc|__builtin_nontemporal_load", code)


def test_the_kernel_that_reads_before_it_waits_reads_past_l1():
    """The dQ kernel may read what kernels before the one in front of it wrote without having waited itself: no cache of an
    SM may answer for the row statistics and the key lengths."""
    with open(os.path.join(CSRC, "attn_bwd_sm100.cuh")) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    code = code[code.index("decode_dq_item(const BwdParams"):]
    for name in ("lse", "delta", "kv_lens"):
        reads = re.findall(rf"[^\n]*\bp\.{name}\b[^\n]*", code)
        assert reads and all(re.search(rf"ld_gpu\(p\.{name} \+", r) for r in reads), reads
        assert not any(re.search(rf"\bp\.{name}\[", r) for r in reads), reads
