"""Rules of kernels that are launched early (programmatic dependent launch), read from the sources: nothing on a CPU can show a
load that came before its wait."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "msa_b200", "csrc")
# read-only for as long as kernels run: weights of a model, tables of a bank
CONSTANT = {("moe_topk_kernel", "bias"), ("select_topk_kernel", "doc_ids_table")}


def kernels():
    """(name, parameters, body) of every kernel, comments and asm text left out."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(\w+)\s*\((?=[^()]*(?:\([^()]*\)[^()]*)*\)\s*\{)", text):
            if m.group(1) == "__launch_bounds__":
                continue
            at, depth = m.end(), 1
            while depth:
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            params, start = text[m.end():at - 1], text.index("{", at)
            end, depth = start + 1, 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield m.group(1), params, text[start:end]


def test_the_scan_finds_the_kernels():
    found = {name for name, _, _ in kernels()}
    text = "".join(re.sub(r"//[^\n]*", "", open(p).read()) for p in glob.glob(os.path.join(CSRC, "*.cu*")))
    assert len(found) > 60 and {"pack_rows_kernel", "select_topk_kernel", "merge_partials_kernel", "rows_gemm_kernel", "route_dec_kernel"} <= found
    assert sum("grid_dependency_wait();" in body for _, _, body in kernels()) >= 8
    assert len(re.findall(r"__global__", text)) == len(list(kernels()))


def test_what_earlier_kernels_write_is_read_behind_the_wait():
    """A load through `const __restrict__` may be moved above the wait."""
    early = [f"{name}: {p.strip()}" for name, params, body in kernels() if "grid_dependency_wait()" in body
             for p in params.split(",") if "const" in p and "__restrict__" in p and (name, p.split()[-1]) not in CONSTANT]
    assert not early
    assert not [name for name, _, body in kernels() if "grid_dependency_wait()" in body and "__restrict__" in body]


def test_a_library_product_is_not_let_in_early():
    """Kernels in front of a product let it start while they run only where it is the few-row one, which has weights to fetch; those
    that always let their dependents start stand in front of a kernel of this package."""
    always = {"fold_kernel",                                        # route_dec_kernel (any other waits for its end)
              "live_blocks_kernel",                                  # pack_rows_kernel
              "moe_topk_kernel", "moe_sort_kernel", "moe_gemm_tc_kernel",
              "rows_gemm_kernel"}
    assert {name for name, _, body in kernels() if re.search(r"(?<!\) )grid_launch_dependents\(\);", body)} <= always
    assert "if (rows <= kEarlyRows) grid_launch_dependents();" in open(os.path.join(CSRC, "lm_common.cuh")).read()
