"""The on-chip CG's grid form takes a row or a partial from another CTA by its tag
alone, so memory that held an earlier object's tags must not reach it: every
owner of such memory clears the whole allocation before the first solve.  What
a missed clear does is a matter of timing, so the sources are read for it."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bounce_b200", "csrc")


@pytest.mark.parametrize("file,function,clear", [
    ("cloth_api.cu", "realize_cloth", r"cudaMemsetAsync\(A\.base, 0, A\.size, st\)"),
    ("softbody.cu", "ensure_sell", r"cudaMemsetAsync\(b->pcg, 0, bytes, s\)"),
])
def test_owner_clears_its_allocation(file, function, clear):
    with open(os.path.join(CSRC, file)) as f:
        text = f.read()
    body = text[text.index(f"b3g_status {function}("):]
    body = body[:body.index("\n}\n")]
    cleared = re.search(clear, body)
    upload = re.search(r"cudaMemcpyAsync\(d_|\bup\(slice_off", body)
    assert cleared and upload and cleared.start() < upload.start()


@pytest.mark.gpu
def test_softbody_after_memory_full_of_tags(b3g):
    """Bodies made where freed memory held the first reductions' tags in every
    word step like any other."""
    import torch

    scene = b3g.pinned_block_scene(20, 20, 20, 1.0 / 20)
    opts = b3g.SolverOptions.relative(1e-5, 30, 2)
    ends = []
    for tag in (None, 0, 1, 2, 3):
        if tag is not None:
            words = torch.full((1 << 26,), tag - (1 << 22), dtype=torch.int32, device="cuda:0")  # 0xffc00000 | tag
            torch.cuda.synchronize()
            del words
            torch.cuda.empty_cache()
        body = b3g.SoftBody(scene.vertices, scene.tets, scene.sdef).setup(scene, opts)
        for _ in range(3):
            body.step(scene.dt)
        ends.append(body.state()["x"])
        body.close()
    assert all(np.array_equal(ends[0], e) for e in ends[1:])
