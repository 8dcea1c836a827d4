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


def _bodies(path: Path):
    """Kernel bodies with their role comments (a line of dashes opens each)."""
    src = path.read_text()
    for m in re.finditer(r"__global__", src):
        brace = src.index("{", m.end())
        depth, end = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(src[end], 0)
            end += 1
        yield src[brace:end]


def test_bounded_waits_start_after_the_predecessors():
    """A wait on a barrier gives up after a time limit.  In a kernel that may start early it begins behind pdl_wait(), in
    every role: the run time of the predecessors does not count against it."""
    seen = 0
    for path in sorted(CSRC.glob("*.cu")):
        for body in _bodies(path):
            if "pdl_wait(" not in body or "mbar_wait(" not in body:
                continue
            common, *roles = re.split(r"//\s*-{20,}", body)
            if "pdl_wait(" in common:
                assert common.find("mbar_wait(") in (-1, *range(common.index("pdl_wait("), len(common)))
                seen += 1
                continue
            for role in roles:
                if "mbar_wait(" in role:
                    assert 0 <= role.find("pdl_wait(") < role.index("mbar_wait("), (path.name, role[:60])
                    seen += 1
    assert seen >= 6, seen
