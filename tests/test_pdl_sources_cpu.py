"""Kernels that wait for their predecessor inside (pdl_wait): nothing that an earlier kernel may have written is a `const T* __restrict__`
parameter, whose loads the compiler may move ahead of the wait.  Read from the sources; what carries the qualifier is a constant of the layer."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "basalt_b200" / "csrc"
CONSTANTS = {"gate", "bias", "blobs", "replicated"}          # router weights, tables of blob addresses and of replicated experts
NORM_WEIGHTS = {"norm_pack_kernel", "norm_images_kernel"}    # their `w`


def kernels():
    """(file, name, parameters, body) of every __global__ function"""
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(([^)]*)\)\s*\{", text):
            depth, at = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            yield path.name, m.group(1), m.group(2), text[m.end():at]


def test_no_restrict_on_what_a_predecessor_writes():
    seen = 0
    for file, name, params, body in kernels():
        if "pdl_wait()" not in body:
            continue
        seen += 1
        for p in params.split(","):
            if "__restrict__" in p and re.match(r"\s*const\b", p):
                var = re.findall(r"\w+", p)[-1]
                assert var in CONSTANTS or (name in NORM_WEIGHTS and var == "w"), f"{file}: {name}({p.strip()})"
    assert seen >= 15, seen
