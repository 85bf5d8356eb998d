"""Rules of the CUDA sources that no run can show to hold."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash_moe_b200", "csrc")
TABLES = {"down", "up", "shards", "B0", "B1"}  # weights: no kernel of the library writes them
TABLE_ROWS = {"ra", "rb", "row"}               # pointers into them


def kernels(text):
    """(parameter list, body) of every __global__ function."""
    for m in re.finditer(r"__global__", text):
        brace = text.index("{", text.index(")", text.index("_kernel(", m.end())))
        head = text[m.end():brace]
        depth, i = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield head[head.index("_kernel("):], text[brace:i]


def test_early_kernels_do_not_read_their_predecessors_output_as_constant_memory():
    """A kernel that is made resident before its predecessor has ended waits with pdl_wait(); a load through a
    const __restrict__ parameter or __ldg counts as one of memory that does not change while the kernel runs, and the compiler
    may move it in front of the wait.  Only weights and tables are read that way."""
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for params, body in kernels(text):
            if "pdl_wait()" not in body:
                continue
            seen += 1
            constant = set(re.findall(r"const\s+\w+\s*\*(?:\s*const\s*\*)?\s*__restrict__\s+(\w+)", params))
            assert constant <= TABLES, (os.path.basename(path), params[:60], constant - TABLES)
            through = set(re.findall(r"(?:\bldg16|\bldg32|__ldg)\(\s*(?:reinterpret_cast<[^>]*>\(\s*)?(\w+)", body))
            assert through <= TABLE_ROWS, (os.path.basename(path), params[:60], through - TABLE_ROWS)
    assert seen >= 10
    with open(os.path.join(CSRC, "gemm_epilogue.cuh")) as f:
        assert "ldg" not in re.sub(r"//[^\n]*", "", f.read())  # addend and residual


def test_waits_for_tensor_memory_name_the_registers_that_they_wait_for():
    """To the compiler the registers of a tcgen05.ld are written at the load.  Every wait takes them as operands, so that nothing
    is done with them in front of it, and every load has its wait."""
    loads = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        if path.endswith("ptx_sm100.cuh"):
            waits = re.findall(r'asm volatile\("tcgen05\.wait::ld[^;]*;"(.*?)\);\n', text, re.S)
            assert sorted(w.count('"+r"') for w in waits) == [16, 32]
            continue
        assert not re.search(r"tmem_ld_wait\(\s*\)", text), os.path.basename(path)
        loaded = re.findall(r"tmem_ld_32x\d+\([^;]*,\s*([\w.]+)\);", text)
        waited = re.findall(r"tmem_ld_wait\(([\w.]+)\);", text)
        assert sorted(loaded) == sorted(waited), (os.path.basename(path), loaded, waited)
        loads += len(loaded)
    assert loads >= 10
