"""CPU-only source check of the relaxed cluster barrier.

cluster_barrier_relaxed() carries no release fence: a write-after-read hazard is covered only where
every remote read before it has been consumed by a store of this CTA that a CTA barrier follows.  One
place in the kernels meets that (the inverse transform's first pass, whose gathered values are
butterflied and stored locally before the arrive).  An exchange that only accumulates remote values in
registers does not, and takes the ordered barrier.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zinq_b200", "csrc")


def calls():
    """(file, name of the enclosing function) of every use of the relaxed barrier."""
    out = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"\bcluster_barrier_relaxed\(\)", text):
            heads = re.findall(r"__(?:forceinline|noinline)__[^;{}()]*?(\w+)\s*\([^;{}]*\)\s*(?:const\s*)?\{", text[:m.end() + 2])
            out.append((name, heads[-1]))
    return out


def test_the_relaxed_barrier_stands_only_where_reads_are_consumed():
    uses = calls()
    assert ("line_kernel.cuh", "cluster_barrier_relaxed") in uses  # its definition
    assert sorted(set(uses) - {("line_kernel.cuh", "cluster_barrier_relaxed")}) == [("line_solve.cuh", "local_fft")]


def test_an_observation_that_keeps_psi_ends_in_the_ordered_barrier():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "line_solve.cuh")).read())
    m = re.search(r"if \(!prop && alt\(\)\) \{([^}]*)return nullptr;", text)
    assert m and "cl.sync();" in m.group(1), m and m.group(1)
