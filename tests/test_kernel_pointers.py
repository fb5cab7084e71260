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


def test_dependent_kernels_read_fields_coherently():
    """Kernels launched dependently run beside the one that writes what they read, and the persistent
    batch kernel writes the fields it reads: non-coherent loads (__ldg, const restrict pointers) are left
    to the coefficient tables, which no launch writes."""
    yee = _source("yee_kernels.cu")
    bodies = {"yee_kernels.cu": yee[yee.index("k_bulk_e(const YeeK"):yee.index("k_prepare(const PrepK")]}
    for name in ("hs_fused.cu", "batch.cu", "lbc.cu", "yee_device.cuh"):
        bodies[name] = _source(name)
    for name, text in bodies.items():
        assert "__restrict__" not in text, name
        assert text.count("__ldg") == (1 if name == "yee_device.cuh" else 0), name
        for arg in re.findall(r"(?<!_)\bldg\(([^;]*?)[,;]", text):
            assert "tab[" in arg or arg.startswith("const T *p"), (name, arg)
    assert set(bodies) < set(_files())


def test_a_batch_keeps_its_tiles_until_it_has_new_ones():
    """A refused allocation must leave a batch that can run: a launch without a tile list would read
    address zero. What a batch has is therefore touched after the last step that can fail only."""
    text = _source("batch_abi.cu")
    body = text[text.index("int build_tiles("):text.index("int make_var(")]
    fails = body.index("cudaMemcpyHostToDevice")
    changes = re.findall(r"cudaFree\(b->tiles\)|b->\w+(?:\[\d\])?\s*=[^=]|b->groups\.(?:clear|push_back|swap)", body)
    assert len(changes) >= 6
    for m in re.finditer(r"cudaFree\(b->tiles\)|b->\w+(?:\[\d\])?\s*=[^=]|b->groups\.(?:clear|push_back|swap)", body):
        assert m.start() > fails, m.group()
    tune = text[text.index("int fdtd_batch_tune("):text.index("int fdtd_batch_run(")]
    assert tune.index("b->xchunk =") > tune.index("build_tiles(")
