"""Kernels of a step start before their predecessors complete, so what a kernel writes
must not be read through the read-only path (__ldg), which asks for data that is
constant for the reading kernel's whole life.  Looks over the sources of the cell
kernels for such reads of the arrays that the ballot and the cell passes write."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "physicore_gb300", "csrc")
WRITTEN = ("vox", "foff", "num", "den", "fac", "rnum", "rden", "rfac", "owner", "counts", "role", "shared", "flags", "err",
           "internal", "field", "sums", "rank", "sorted", "pieces", "writers", "steps_left", "recompute", "mc_tot", "mc_out")


def read_only_reads(text):
    """The arguments of every __ldg, with nested parentheses."""
    for m in re.finditer(r"__ldg\(", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        yield text[m.end():k - 1]


def test_no_read_only_loads_of_what_a_step_writes():
    bad = []
    for name in ("cells.cu", "cells_device.cuh", "batch.cu", "field_ops.cu", "field_device.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            for arg in read_only_reads(f.read()):
                if re.search(r"[.>](%s)\b" % "|".join(WRITTEN), arg) or (name.startswith("cells") and re.search(r"\bq\b", arg)):
                    bad.append((name, arg))
    assert not bad
