"""The resident reduction's exchange areas (csrc/zq_resident.cu), read from the source.

The CTAs of a group meet at barriers; between two of them an array that other CTAs
read must not be written (a CTA that runs ahead would overwrite what a later one
has yet to read, and the two would go on with different values).
"""
from __future__ import annotations

import os
import re

SRC = os.path.join(os.path.dirname(__file__), "..", "zquatev_gb300", "csrc", "zq_resident.cu")

READ = re.compile(r"(?:__ldcg|q_ldcg|acc_load|warp_gather<R>)\([^;]*?\bgr\.(\w+)")
WRITE = [re.compile(r"\bgr\.(\w+)\[[^\]]*\] = "),                    # gr.a[i] = v
         re.compile(r"\bgr\.(\w+)\)\[[^\]]*\] = "),                  # reinterpret_cast<R*>(gr.a)[i] = v
         re.compile(r"\b(?:acc_store|q_store)\(gr\.(\w+)"),
         re.compile(r"reinterpret_cast<R\*>\(gr\.(\w+) [^;]*?\)\[k\] = "),
         re.compile(r"R\* o = reinterpret_cast<R\*>\(gr\.(\w+) ")]   # filled through o[...]


def body(text, head):
    """The braces that follow `head`."""
    i = text.index("{", text.index(head))
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise ValueError(head)


def phases():
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    fn = body(text, "__device__ bool reduce_matrix(")
    norms = body(fn, "auto publish_norms = ")
    fn = fn.replace(norms, "{}")
    fn = re.sub(r"publish_norms\([^;]*\);", lambda _: norms, fn)
    loop = body(fn, "for (int j = 0; j + 1 < m; ++j)")
    before = fn[:fn.index(loop)].split("if (!barrier()) return false;")
    inside = loop.split("if (!barrier()) return false;")
    assert len(before) == 3 and len(inside) == 3
    # the loop's end runs on into its next pass, and so does what precedes the loop
    return {"load": before[0], "column 0": before[1], "sweep": before[2] + inside[2] + inside[0], "rows": inside[1]}


def test_no_array_is_written_while_others_read_it():
    seen = {"r": set(), "w": set()}
    for name, code in phases().items():
        reads = set(READ.findall(code))
        writes = set().union(*(w.findall(code) for w in WRITE))
        seen["r"] |= reads
        seen["w"] |= writes
        if name == "rows":
            reads.discard("x")  # of the rows that the same CTA writes, behind a block barrier
        assert not reads & writes, (name, reads & writes)
    # every exchanged array was recognised on both sides
    assert seen["r"] == seen["w"] == {"cpart", "npart", "q2", "x", "y", "col", "part"}
