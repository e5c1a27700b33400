"""CUDA lets a CTA touch another CTA's shared memory only once that CTA is known
to run, which a cluster barrier shows.  That cannot be provoked on a GPU, so
this reads the sources: in every kernel of a cluster a cluster barrier comes
before the first call that reaches into another CTA."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bounce_b200", "csrc")
REACHES = re.compile(r"map_shared_rank|\bresident_solve<|\bbatch_solve<|\brun_cg<")
BARRIER = re.compile(r"\b(?:team\.barrier|cl\.sync|this_cluster\(\)\.sync|Team<T>::sync)\(\)")


def _kernels(text):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__\b", text):
        start = text.index("{", m.end())
        depth, at = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield re.search(r"\b(k_\w+)\s*\(", text[m.end():start]).group(1), text[start:at]


def test_cluster_kernels_start_with_a_barrier():
    seen = set()
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for kernel, body in _kernels(text):
            reach = REACHES.search(body)
            if not reach or "GridScope" in body:  # (the CTAs of a cooperative launch share none)
                continue
            barrier = BARRIER.search(body)
            assert barrier and barrier.start() < reach.start(), f"{name}: {kernel}"
            seen.add(kernel)
    assert seen == {"k_resident_team", "k_batch_resident", "k_batch_cg"}
