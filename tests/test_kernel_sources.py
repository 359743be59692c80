"""Rules of the kernels' sources that no run shows: operations that are undefined
although today's compiler makes something harmless of them."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sovereign-solver_gb300", "csrc")


def _source(name):
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", src)


def test_node_map_has_its_divisor():
    """k_node64 divides by the nodes of an instance: every launch's arguments come from
    node_args, which sets them."""
    src = _source("gnn.cu")
    assert re.findall(r"Node64 \w+\{\};", src) == ["Node64 a{};"]
    helper = src[src.index("Node64 node_args("):]
    assert "a.n = n;" in helper[:helper.index("return a;")]


def test_gradient_in_place_is_read_with_plain_loads():
    """k_back64 writes dh over dout: __ldg needs memory that the launch does not write."""
    src = _source("gnn.cu")
    body = src[src.index("k_back64(const Back64 a)"):src.index("k_in_back64(const Back64 a)")]
    assert "a.dout)" in body
    assert not re.search(r"__ldg\([^;]*a\.dout", body)


def test_copied_to_shared_memory_is_aligned():
    """16-byte copies and reads (the sliced passes' ring): every dynamic shared array says so."""
    for name in sorted(os.listdir(CSRC)):
        for line in re.findall(r"extern __shared__[^;]*;", _source(name)):
            assert "__align__(16)" in line, (name, line)


def test_epilogue_slots_hold_every_check():
    """A SEGMENT column's slot holds the partials of the PDLP form's check, the most there are (the
    writers assert it at compile time too)."""
    n = {k: int(v) for name in ("engine.cuh", "decide.cuh")
         for k, v in re.findall(r"constexpr int (k\w+) = (\d+);", _source(name))}
    assert n["kMaxEpiPartials"] >= max(n["kColPartials"] + n["kLagPartials"], n["kRowPartials"])
    assert _source("engine.cuh").count("static_assert(Epi::NP <= kMaxEpiPartials") == 2
