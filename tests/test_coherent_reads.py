"""Kernels that are started as programmatic dependents (launch_kernel) are resident while the kernels
queued before them still write: what those may write -- source rows, padded copies, patch coords,
queries -- is not read through the non-coherent path, which asks for data that nobody writes during
a kernel's lifetime.

Checked on the sources: in files with such kernels, and the headers they share, each non-coherent read
(ld.global.nc, __ldg, ld_stream) is of an array listed here: a table's own, which is complete before
the table is handed out, or one that only kernels behind all earlier work (<<<>>>) read.
"""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "opensubdiv_gb300", "csrc")

# arrays that a table owns
OWNED = {
    "patchmap_walk.cuh": ["m.nodes", "m.handles"],
    "stencils_tma.cu": ["a.sliceSlot", "a.idx"],
    "stencils_units.cu": ["own"],
    "unit_eval.cuh": ["far"],
    "unit_ring.cuh": [],
    "patch_basis.cuh": [],
    "patches.cu": [],
    "patchmap.cu": [],
}
# read by kernels that are launched behind all earlier work
PLAIN = {
    "stencils_tma.cu": ["a.offsets", "a.sizes", "a.indices", "a.w[k]"],  # k_stencils_tma
    "stencil_eval.cuh": ["a.w[k]", "a.indices"],  # entries outside a stage: k_stencils_tma, batch
    "stencils_batch.cu": ["j.", "&j", "a.tileBase", "a.jobs", "rowBase",
                         "v.src", "r + u"],  # k_stencils_batch, k_pad_rows
    "tessellation.cu": ["src", "cg", "pcSrc"],  # k_share_emit
}


def _argument(text, at):
    depth, end = 1, at
    while depth:
        depth += {"(": 1, ")": -1}.get(text[end], 0)
        end += 1
    arg = re.sub(r"^\s*(reinterpret_cast<[^>]*>\s*\(|\((const )?(long long|int) ?\*\)\s*)", "",
                 text[at:end - 1])
    return " ".join(arg.split())


def _code(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


def test_non_coherent_reads_are_of_arrays_that_no_queued_work_writes():
    dependent = {os.path.basename(f) for f in glob.glob(CSRC + "/*.cu")
                 if "launch_kernel(" in _code(f)}
    assert dependent >= {"stencils_tma.cu", "stencils_units.cu", "patches.cu", "patchmap.cu",
                         "tessellation.cu", "stencils_batch.cu"}
    found = []
    for name in sorted(dependent | set(OWNED) | {"stencil_eval.cuh"}):
        text = _code(os.path.join(CSRC, name))
        allowed = OWNED.get(name, []) + PLAIN.get(name, [])
        for m in re.finditer(r"\b(__ldg|ld_stream|load_far)\s*\(", text):
            if "__device__" in text[max(0, m.start() - 60):m.start()]:
                continue  # its definition
            arg = _argument(text, m.end())
            if not any(arg.startswith(p) for p in allowed):
                found.append((name, m.group(1), arg))
    assert not found, found


def test_non_coherent_instructions_are_in_the_named_loads_only():
    """ld_stream and the unit layout's weights; every other asm load is coherent."""
    for path in glob.glob(CSRC + "/*.cu*"):
        text, name = _code(path), os.path.basename(path)
        for m in re.finditer(r"asm\s*(volatile)?\s*\((.*?)\);", text, flags=re.S):
            if "ld.global.nc" in m.group(2):
                before = re.findall(r"__device__[^\n]*?(\w+)\(", text[:m.start()])[-1]
                assert (name, before) in {("common.cuh", "ld_stream"), ("unit_eval.cuh", "load_far")}


def test_coherent_loads_stay_behind_the_wait():
    """An asm load is volatile, as the wait is, or one of those whose addresses the dependent kernels
    take from behind_wait: rows of units, EvalPatches' source elements and patch indices."""
    movable = {}
    for path in glob.glob(CSRC + "/*.cu*"):
        text = _code(path)
        for m in re.finditer(r"asm\s*(volatile)?\s*\((.*?)\);", text, flags=re.S):
            if "ld.global" in m.group(2) and ".nc" not in m.group(2) and m.group(1) is None:
                load = re.findall(r"__device__[^\n]*?(\w+)\(", text[:m.start()])[-1]
                movable[load] = os.path.basename(path)
    assert movable == dict.fromkeys(("ld_point", "ld_point4", "ld_point8", "ld_index",
                                     "ld_index4"), "common.cuh")
    for path in glob.glob(CSRC + "/*.cu*"):
        if re.search(r"\b(ld_point[48]?|ld_index4?)\(", _code(path)):
            assert os.path.basename(path) in ("common.cuh", "patch_basis.cuh", "unit_eval.cuh",
                                              "stencil_eval.cuh"), path
    # stencil_eval.cuh's are for the batched kernels, which are not dependents
    for name in ("stencils_tma.cu", "stencils_units.cu"):
        assert not re.search(r"gather_row<0>|true>\(a, id", _code(os.path.join(CSRC, name)))
    assert "launch_kernel(k_stencils_batch" not in _code(os.path.join(CSRC, "stencils_batch.cu"))
    assert "behind_wait(a.src)" in _code(os.path.join(CSRC, "stencils_units.cu"))
    text = _code(os.path.join(CSRC, "patches.cu"))
    assert "behind_wait(a.src)" in text and "behind_wait(a.indices)" in text
    assert text.count("= args_behind_wait<") == len(re.findall(r"\bk_eval_patches\w*\(const", text))
    # the wait itself is volatile too
    common = _code(os.path.join(CSRC, "common.cuh"))
    assert 'asm volatile("griddepcontrol.wait;" ::: "memory")' in common


def test_row_pointers_are_not_restrict():
    """A __restrict__ pointer to const data lets the compiler choose the non-coherent path itself."""
    for name in ("patch_basis.cuh", "patches.cu", "patchmap.cu", "patchmap_walk.cuh",
                 "unit_eval.cuh", "stencil_eval.cuh", "stencils_tma.cu", "stencils_units.cu",
                 "tessellation.cu", "tess_pattern.cuh"):
        assert "__restrict__" not in _code(os.path.join(CSRC, name)), name
