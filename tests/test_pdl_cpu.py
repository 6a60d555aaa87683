"""Kernels that may start while the kernels before them still run (pdl.hpp) read what those wrote
with ordinary loads: checked in the sources, since a breach shows up as stale operands at best now
and then."""
import glob
import os
import re

import pytest

from tests.helpers import ROOT

# complete before the first kernel of such a chain starts: packed codes, the dense matrix, the
# missing-entry index lists
STATIC = {"codes", "A", "idx"}
STATIC_LOADS = {"rowp", "base"}  # pointers into the codes


def closing(text, i, pair):
    """Index past the bracket that closes the one at i."""
    depth = 0
    while True:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return i


def functions(text):
    """(name, parameters, body) of every __global__ and __device__ function of a source text."""
    text = re.sub(r"//[^\n]*", "", text)
    text = re.sub(r"__launch_bounds__\([^()]*\)|__cluster_dims__\([^()]*\)|__forceinline__", "", text)
    for m in re.finditer(r"__(?:global|device)__[\w\s:&*<>]*?\b(\w+)\s*\(", text):
        i = closing(text, m.end() - 1, "()")
        body = re.match(r"\s*(?:const\s*)?\{", text[i:])
        if body:
            yield m.group(1), text[m.end():i - 1], text[i:closing(text, i + body.end() - 1, "{}")]


SOURCES = sorted(f for f in glob.glob(os.path.join(ROOT, "pcaone_b200", "csrc", "*.cu"))
                 if "pdl_begin();" in open(f).read())


def test_every_kernel_launched_early_waits():
    waiting, launched = set(), set()
    for f in SOURCES:
        text = open(f).read()
        waiting |= {name for name, _, body in functions(text) if "pdl_begin();" in body}
        launched |= set(re.findall(r"launch_pdl\(\s*(k_\w+)", text))
    assert {"k_prep", "k_accum", "k_quant", "k_decode_gemm_i8", "k_tall", "k_flip", "k_apply", "k_decode_gemm",
            "k_dense_gemm2"} <= waiting
    assert launched <= waiting


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_chain_results_are_read_with_ordinary_loads(path):
    checked = 0
    funcs = list(functions(open(path).read()))
    # the waiting kernels and the helpers that they call
    inside = {name for name, _, body in funcs if "pdl_begin();" in body}
    while True:
        bodies = " ".join(body for name, _, body in funcs if name in inside)
        more = {name for name, _, _ in funcs if re.search(rf"\b{name}\s*(<[^;()]*>)?\s*\(", bodies)} - inside
        if not more:
            break
        inside |= more
    for name, params, body in funcs:
        if name not in inside:
            continue
        checked += 1
        for p in re.findall(r"const\s+[\w ]+\*\s*__restrict__\s+(\w+)", params):
            assert p in STATIC, f"{name}: const __restrict__ {p}"
        for arg in re.findall(r"__ld(?:g|cs|cg|ca|lu)\(([^;]*)", body):
            assert set(re.findall(r"[A-Za-z_]\w*", arg)) & STATIC_LOADS, f"{name}: non-coherent load of {arg}"
    assert checked
