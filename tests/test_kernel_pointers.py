"""What the kernels promise the compiler about their pointers, read from their source: a broken promise
need not show in the results of one compiler."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "opencl_fdtd_gb300", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _files():
    return sorted(os.path.basename(p) for ext in ("cu", "cuh") for p in glob.glob(os.path.join(CSRC, "*." + ext)))


def test_pointers_to_the_updated_field_are_not_restrict():
    """The per-update kernels read the updated field through one pointer and write it through another,
    which in place is the same array: neither may be restrict."""
    text = _source("yee_kernels.cu")
    start = text.index("k_bulk_e(const YeeK")
    bodies = text[start:text.index("k_bulk_s(const SK")]
    declared = re.findall(r"[^;{}]*\b(?:[PW][xyz])\b\s*=[^;]*;", bodies)
    declared = [d for d in declared if re.search(r"\bR\s*\*", d)]
    assert len(declared) >= 4                                # P and W of the E and of the H kernel
    for d in declared:
        assert "__restrict__" not in d, d
