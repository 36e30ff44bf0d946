"""CPU: kernels that may start before the kernel ahead of them is done (those
that wait for it with grid_chain or chain_wait) take pointers to anything that
kernel may have written without __restrict__, which would let the compiler
read it before the wait or through the non-coherent path.  Checked in the
sources, since a compiler that happens not to move the loads hides it: only
arrays of the matrix or its plan and the caller's x may be restrict, and the
gathers of the solver's direction vector go through ld_chain."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rvvlasparse_b200", "csrc")
# written by no kernel of any call (formats and plans); x: by none but the solvers' (see below)
CONSTANT = {"rst", "Rst", "bits", "Col", "Val", "perm", "wrow", "row_map", "colidx", "vals", "cols", "rec", "wb", "thr",
            "co", "cf", "sp", "mk", "val", "col", "los", "row_order", "x"}
# outputs of crs_run_kernel: it only writes them, with values that depend on loads behind its wait (y is read for
# beta, at rows that no kernel ahead of it writes)
WRITTEN = {"crs_run_kernel": {"y", "carry_row", "carry_val", "dot_part"}}


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{}()]*(?:\([^()]*(?:\([^()]*\)[^()]*)*\))?\s*\b(\w+_kernel)\(([^{};]*)\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield m.group(1), m.group(2), text[m.end():i]


def test_chained_kernels_read_behind_their_wait():
    seen = set()
    for name, args, body in _kernels():
        if "grid_chain()" not in body and "chain_wait()" not in body:
            continue
        seen.add(name)
        restrict = set(re.findall(r"__restrict__\s+(\w+)", args))
        assert restrict <= CONSTANT | WRITTEN.get(name, set()), (name, restrict - CONSTANT)
    assert {"crs_run_kernel", "crs_stream_fixup_kernel", "crs_dot_fixup_kernel", "csr5_calibrate_kernel", "csr5_tail_kernel",
            "cvr_spmv_kernel", "lav_fused_kernel", "vhcc_overflow_kernel", "vhcc_out_kernel", "cg_update_kernel",
            "cg_xp_kernel"} <= seen


def test_solver_direction_is_gathered_coherently():
    body = next(b for n, _, b in _kernels() if n == "crs_run_kernel")
    assert "ld_chain(x + yrow(r)" in body and not re.search(r"\bx\[", body)
    assert re.search(r"DOT \? ld_chain\(x \+ cidx\[i\], pl\) : ld_keep\(x \+ cidx\[i\], pl\)", body)
    text = open(os.path.join(CSRC, "rvvla_internal.cuh")).read()
    for asm in re.findall(r"ld_chain\(const \w+\* p.*?\n\}", text, re.S):
        assert "asm volatile" in asm and ".nc" not in asm and '"memory"' in asm
