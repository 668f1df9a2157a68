"""Kernels launched with programmatic stream serialization are resident while their predecessor writes what they read: the library's kernels use
the read-only load path, which no wait orders behind those writes, for weights and tables only (a check of the sources; no GPU)."""
import glob
import os
import re

from yasakani_b200 import build


def _code(path):
    text = open(path).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def test_no_read_only_loads():
    for path in build.sources() + glob.glob(os.path.join(build.CSRC, "*.cuh")):
        code, name = _code(path), os.path.basename(path)
        assert code.count("__ldg(") == (name == "kv4_common.cuh") and not re.search(r"ld\.global(\.\w+)*\.nc\b", code), name
        # ld_table: the norm weights (wn) and rows of the rope table (rr) of the row epilogue
        assert set(re.findall(r"\bld_table\((?:reinterpret_cast<[^>]*>\()?(\w+)", code)) <= {"kvx_codec.cu": {"wn", "rr"}, "kv4_common.cuh": {"const"}}.get(name, set()), name
        # const + __restrict__ lets the compiler choose that path: the sign vector is a table; the copy kernel is launched in plain stream order
        names = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", code))
        assert names <= {"kv4_xform.cu": {"signs"}, "kv4_codec.cu": {"src"}}.get(name, set()), (name, names)


def test_the_position_is_the_only_early_read_of_the_int8_decode_kernel():
    """Ahead of its wait the kernel loads the position once, past L1, for the address of a prefetch; everything else it reads stands behind the wait."""
    code = _code(os.path.join(build.CSRC, "kv8_decode.cu"))
    early = code[code.index("kv8_decode_kernel(const Kv8P P) {"):]
    early = early[:early.index("griddepcontrol.wait")]
    loads = re.findall(r"__ldc[gs]\(|ldg16\(|\bld\.global|ld_table\(|\*A\.\w+|A\.\w+\[", early)
    assert loads == ["__ldcg("] and "__ldcg(A.d_pos)" in early and "prefetch.L2" in early
