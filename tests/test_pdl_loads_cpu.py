"""Kernels that start while their predecessors still run (csrc/pdl.cuh) read global memory with coherent loads only."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "dizo_b200" / "ops" / "csrc"


def _code(path: Path) -> str:
    return re.sub(r"//[^\n]*", "", path.read_text())


def _kernels(src: str):
    """(name, signature, body) of every __global__ function."""
    for m in re.finditer(r"__global__", src):
        brace = src.index("{", m.end())
        depth, end = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(src[end], 0)
            end += 1
        sig = src[m.end():brace]
        name = re.findall(r"(\w+)\s*\(", re.sub(r"__\w+__\s*\([^()]*(?:\([^()]*\))?[^()]*\)", "", sig))[0]
        yield name, sig, src[brace:end]


DEPENDENT = [(p.name, n) for p in sorted(CSRC.glob("*.cu")) for n, _, body in _kernels(_code(p)) if "pdl_wait(" in body]


def test_the_dependent_kernels_are_found():
    names = {n for _, n in DEPENDENT}
    assert names >= {"layernorm_kernel", "rmsnorm_kernel", "gemm_bf16_tn_kernel", "gemm2_bf16_kernel", "skinny_gemm_kernel",
                     "gemv_kernel", "attn_fwd_kernel", "decode_attn_kernel", "zo_sweep_kernel"}, names


@pytest.mark.parametrize("file,name", DEPENDENT)
def test_no_non_coherent_load(file, name):
    src = _code(CSRC / file)
    (sig, body), = [(s, b) for n, s, b in _kernels(src) if n == name]
    assert "__ldg" not in body
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", sig), sig
    # helpers of the file (device functions with inline loads) count too
    assert "ld.global.nc" not in src
