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
            constant = CONSTANT - {"perm"} if k == "gather_positions_kernel" else CONSTANT      # it stands right behind the sort that makes the order
            assert promised <= constant, promised - constant


@pytest.mark.parametrize("source", sorted({f for f, *_ in _kernels()}))
def test_non_coherent_loads_are_of_weights(source):
    for arg in re.findall(r"\b(?:__ldg|ldg4|ldg8)\((?:reinterpret_cast<const float4\*>\()?([A-Za-z_][\w.]*)", SOURCES[source]):
        # members of the weight records, the arguments of the loading helpers themselves, weights passed on under a name
        assert arg.startswith(("L.", "M.")) or arg in {"const", "W", "p", "bias", "fin"}, arg


def _function(source, name):
    m = re.search(r"\b%s\([^;{]*\)\s*\{" % name, SOURCES[source])
    return SOURCES[source][m.end():SOURCES[source].index("\n}\n", m.end())]


def test_only_the_second_of_two_lists_starts_beside_the_kernel_before_it():
    """Kernels that launch_early starts without a wait at their start: the row kernels of a second list, beside the first list's.  Nothing else may
    take its place while a list is being written, and each of them ends behind its predecessor."""
    everything = SOURCES | {os.path.basename(f): re.sub(r"//[^\n]*", "", open(f).read()) for p in ("*.h", "*.cuh") for f in glob.glob(os.path.join(CSRC, p))}
    assert {f for f, s in everything.items() if "griddepcontrol" in s} == {"common.cuh", "nlist.cu"}
    assert {f: len(re.findall(r"(?<!void )launch_early\(", s)) for f, s in everything.items() if "launch_early(" in s} == {"kernels.h": 1, "nlist.cu": 1}
    s = SOURCES["nlist.cu"]
    rows = set(re.findall(r"launch_rows\(beside, (\w+)", s))
    assert rows == {"build_rows_kernel", "build_rows_graph_kernel"}
    assert len(re.findall(r"let_next_start\(\)", s)) == 1 + len(rows) == 1 + len(re.findall(r"if \(first_of_two\) let_next_start\(\);", s))
    for k in rows:
        assert re.search(r"void (?:__launch_bounds__\(256\) )?%s\([^{]*bool first_of_two\) \{\s*if \(first_of_two\) let_next_start" % k, s)
        body = _function("nlist.cu", k)
        assert body.rstrip().endswith("end_after_previous();") and "return" not in body
    assert "if (beside == RowsBeside::kSecond) launch_early(" in _function("nlist.cu", "launch_rows")
    assert set(re.findall(r"(\w+) \? RowsBeside::k(?:First|Second) : RowsBeside::kNo", SOURCES["engine.cu"])) == {"both", "both_counts"}
    assert len(re.findall(r"RowsBeside::k(?:First|Second)", SOURCES["engine.cu"])) == 4


def test_lists_are_complete_ahead_of_the_first_chained_kernel():
    """An operation launched the ordinary way between the kernels that write a list and the chained kernels that take it as constant."""
    body = _function("engine.cu", "rebuild_lists")
    behind = body[body.rindex("nlist_end("):]
    assert "launch_chained" not in body[body.index("nlist_begin("):] and "cudaMemcpyAsync(S->d_Rref" in behind
    assert "return kOk" not in behind[:behind.index("cudaMemcpyAsync(S->d_Rref")]
    body = _function("engine.cu", "so3lr_b200_dd_begin")
    behind = body[body.rindex("nlist_build("):]
    assert behind.index("fill(st, S->e_zbl, n0, 0.f);") < behind.index("launch_sr_geometry_zbl(")


def test_one_clearing_launch_holds_all_its_arrays():
    """The arrays travel in an object of fixed size that is passed by value: one too many must not be written behind its end."""
    s = SOURCES["engine.cu"]
    room = int(re.search(r"struct ClearArgs \{.*?kMax = (\d+);", s, re.S).group(1))
    assert "if (count < kMax)" in re.search(r"struct ClearArgs \{.*?\n\};", s, re.S).group(0)
    uses = re.findall(r"ClearArgs A;(.*?)if \(int rcc = launch_clear\(st, A\)\) return rcc;", s, re.S)
    assert len(uses) == len(re.findall(r"ClearArgs A;", s)) and all(0 < u.count("A.add(") <= room for u in uses)


def test_cycle_counts_are_divided_by_the_tiles_that_were_walked():
    """Timing builds of the attention kernels: every slot that is printed is written, and the divisors are counted tile by tile."""
    s = SOURCES["attention_tc.cu"]
    printed = _function("attention_tc.cu", "tc_debug_print")
    phases, tiles = {}, {}
    for name in ("attn_fwd_tc_kernel", "attn_bwd_tc_kernel"):
        m = re.search(r"__global__ void (?:__launch_bounds__\([^)]*\) )?%s\(" % name, s)
        body = s[m.end():s.index("tcgen05.dealloc", m.end())]
        (slot,) = re.findall(r"TC_TILE\((\d+)\);", body)
        assert f"dbg[{slot}] = 0" in body and "gridDim.x;" not in "".join(re.findall(r"if \(dbg[^\n]*", body))
        (at,) = re.findall(r"dbg\[(?:(\d+) \+ )?q\] = [tb]ph\[q\]", body)
        tiles[name], phases[name] = int(slot), range(int(at or 0), int(at or 0) + 8)
    for slot in map(int, re.findall(r"(?<!long long )\bh\[(\d+)\]", printed)):
        assert slot in tiles.values() or any(slot in r for r in phases.values()), slot


def test_statuses_of_the_attention_launches_are_looked_at():
    """They refuse a list that was compacted for other rows; an evaluation that went on would hold no attention sums."""
    calls = re.findall(r"([^;{}]*?)\b((?:launch_attn_\w+_tc\w*|attn_\w+_dispatch)\()", SOURCES["engine.cu"])
    used = [(before.split("\n")[-1].strip(), name) for before, name in calls]
    assert len(used) > 8
    for before, name in used:
        assert before.endswith(("return", "=", "int")), (before, name)
