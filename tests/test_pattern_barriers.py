"""The phases of pattern_kernel hand shared memory from lane to lane: a warp barrier lies between each
phase that writes an array and the next that reads it (votes and shuffles order no memory).  A missing
one may go unseen on a GPU, so the source is read."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "freefem-sources_gb300", "csrc")


def test_a_warp_barrier_lies_between_the_phases():
    with open(os.path.join(CSRC, "ffgpu_assembly.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    body = text[text.index("pattern_kernel(int nnodes"):]
    body = body[:body.index("\n}\n")]
    # one statement of each phase, in order: table cleared, candidates hashed, distinct nodes listed, ranks
    # back into the table, ranks read per candidate, next row
    phases = ["tab[i] = -1", "atomicCAS(tab + h", "lst[i] = v", "tab[lsl[i]] = r", "tab[sl[p]]"]
    at = [body.index(p) for p in phases] + [len(body)]
    assert at == sorted(at)
    for a, b, name in zip(at, at[1:], phases):
        assert "__syncwarp()" in body[a:b], "no barrier after: " + name
