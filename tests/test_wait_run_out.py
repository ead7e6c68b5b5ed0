"""A bounded wait that runs out inside a kernel ends the loop the kernel belongs to.

No GPU can be made to lose a copy on purpose, so the sources are read: wherever a kernel records that a
wait ran out, it also sets the flag that the loop's next kernel stops on, and the host turns the record
into an error.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "freefem-sources_gb300", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _body(text, start):
    """The block of braces that opens after ``start``."""
    i = text.index("{", text.index(start))
    depth = 0
    for k in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[i:k + 1]
    raise AssertionError(start)


def test_inner_loop_stops_when_a_copy_does_not_arrive():
    body = _body(_source("ffgpu_mixed.cu"), "ir_ka_ring(SellArgs")
    after = body[body.index("if (!ok) {"):]
    assert re.search(r"ks->fail = 1;\s*ks->done = 1;", after)
    kb = _body(_source("ffgpu_mixed.cu"), "ir_kb(int")
    assert re.search(r"if \(ks->done\) \{\s*if \(in_graph[^;]*ir_graph_stop\(cond\);\s*return;", kb)


def test_every_run_out_is_an_error_on_the_host():
    mixed, solve = _source("ffgpu_mixed.cu"), _source("ffgpu_solve.cu")
    assert "hk.fail" in _body(mixed, "int ffgpu_solve_ir(") and "S.ks->fail" in _body(mixed, "int ir_tune(")
    assert "kWaitRanOut" in _body(solve, "int tune_lanes(")
    one = _body(solve, "int cg_one(")
    assert one.index("cudaMemsetAsync(A->ks, 0") < one.index("FFGPU_CHECK(hk.done != kWaitRanOut")
