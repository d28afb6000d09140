"""The rule beside grid_dep_sync (csrc/common.cuh), checked in the sources: a kernel that launch_chained starts is alive while the kernels
before it still write its inputs, so it must not promise the compiler that those inputs are constant (const __restrict__, __ldg)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "so3lr_b200", "csrc")
# the model's weights, and arrays that are complete before the first chained kernel of an evaluation starts
CONSTANT = {"projT", "proj", "projT_u", "proj_u", "img_g", "sph1_k", "sph1_b", "embed", "row_ptr", "nbr_j", "edge_i", "Z", "perm", "graph_start",
            "total_charge"}
SOURCES = {os.path.basename(f): re.sub(r"//[^\n]*", "", open(f).read()) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")))}
CHAINED = sorted({k for s in SOURCES.values() for k in re.findall(r"launch_chained\((\w+)", s)})
KERNEL = re.compile(r"__global__ void (?:__launch_bounds__\([^)]*(?:\([^)]*\))?[^)]*\) )?(\w+)\(([^{]*?)\)\s*\{", re.S)


def _kernels():
    for name, s in SOURCES.items():
        heads = list(KERNEL.finditer(s))
        for m, nxt in zip(heads, heads[1:] + [None]):
            if m.group(1) in CHAINED:
                yield name, m.group(1), m.group(2), s[m.end():nxt.start() if nxt else len(s)]


def test_every_chained_kernel_is_found():
    assert len(CHAINED) > 25 and {k for _, k, _, _ in _kernels()} == set(CHAINED)


@pytest.mark.parametrize("kernel", CHAINED)
def test_inputs_of_chained_kernels_are_not_promised_constant(kernel):
    for _, k, params, body in _kernels():
        if k == kernel:
            assert "grid_dep_sync();" in body
            promised = set(re.findall(r"const [\w ]+\* __restrict__ (\w+)", params))
            assert promised <= CONSTANT, promised - CONSTANT


@pytest.mark.parametrize("source", sorted({f for f, *_ in _kernels()}))
def test_non_coherent_loads_are_of_weights(source):
    for arg in re.findall(r"\b(?:__ldg|ldg4|ldg8)\((?:reinterpret_cast<const float4\*>\()?([A-Za-z_][\w.]*)", SOURCES[source]):
        # members of the weight records, the arguments of the loading helpers themselves, weights passed on under a name
        assert arg.startswith(("L.", "M.")) or arg in {"const", "W", "p", "bias", "fin"}, arg


def test_one_clearing_launch_holds_all_its_arrays():
    """The arrays travel in an object of fixed size that is passed by value: one too many must not be written behind its end."""
    s = SOURCES["engine.cu"]
    room = int(re.search(r"struct ClearArgs \{.*?kMax = (\d+);", s, re.S).group(1))
    assert "if (count < kMax)" in re.search(r"struct ClearArgs \{.*?\n\};", s, re.S).group(0)
    uses = re.findall(r"ClearArgs A;(.*?)if \(int rcc = launch_clear\(st, A\)\) return rcc;", s, re.S)
    assert len(uses) == len(re.findall(r"ClearArgs A;", s)) and all(0 < u.count("A.add(") <= room for u in uses)


def test_statuses_of_the_attention_launches_are_looked_at():
    """They refuse a list that was compacted for other rows; an evaluation that went on would hold no attention sums."""
    calls = re.findall(r"([^;{}]*?)\b((?:launch_attn_\w+_tc\w*|attn_\w+_dispatch)\()", SOURCES["engine.cu"])
    used = [(before.split("\n")[-1].strip(), name) for before, name in calls]
    assert len(used) > 8
    for before, name in used:
        assert before.endswith(("return", "=", "int")), (before, name)
