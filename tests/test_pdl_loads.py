"""Kernels launched as programmatic dependents (they begin with pdl_entry())
read what other kernels of their chain write with ordinary loads: the
read-only path (__ldg, const __restrict__ pointers) asks for data that stay as
they are for the kernel's whole life, which begins while its predecessors
still write.  Only the matrix, its pattern, the aggregates and D^-1, complete
before a chain begins, may take it."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "chuanflow_b200" / "csrc"
FIXED = {"val", "dinv", "ms", "mem", "agg", "m", "A.start", "A.col", "L.rs", "L.cols", "L.val", "L.sstart", "L.scol",
         "L.sval"}


def functions(text):
    """(name, parameters, body) of the functions: their braces stand in the first column."""
    for m in re.finditer(r"^\{$(?=(.*?)^\}$)", text, re.M | re.S):
        head = text[:m.start()].rstrip()
        if not head.endswith(")"):
            continue
        i, depth = len(head) - 1, 1
        while depth:
            i -= 1
            depth += {")": 1, "(": -1}.get(head[i], 0)
        name = re.search(r"(\w+)$", head[:i])
        if name:
            yield name.group(1), head[i + 1:-1], m.group(1)


def sources(names):
    return {f[0]: f for n in names for f in functions((CSRC / n).read_text())}


def test_dependent_kernels_read_their_chain_with_ordinary_loads():
    found = sources(["amg.cu", "solvers.cuh", "kernels.cuh"])
    kernels = [f for f in found.values() if "pdl_entry();" in f[2]]
    assert len(kernels) >= 20
    called = [found[n] for n in ("sell_row", "sell_row3", "group_row", "do_restrict", "do_residual", "do_smooth",
                                 "sell32_row", "spmv_row", "spmv_row_gather")]
    for name, params, body in kernels + called:
        for p in params.split(","):
            if "const" in p and "__restrict__" in p:
                assert p.split()[-1] in FIXED, (name, p)
        for arg in re.findall(r"__ldg\(([\w.]+)", body):
            assert arg in FIXED, (name, arg)
