"""The path kernel's shared counters: every block reads the pass and the queue
count before the last block to leave rewrites them.  A wrong order loses paths
only in a rare interleaving, so the order is read from the source: the reads,
then a barrier of the block, then a fence, the ticket, a fence and the writes.
On the GPU, waves of few paths (most warps of a block have nothing to do and
pass their end long before the others) give the instrumented wavefront's films
every time."""
import os
import re

import numpy as np
import pytest

from asuna_gb300 import scenes

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "asuna_gb300", "csrc", "path.cu")


def _kernel():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    at = text.index("k_path(KParams P")
    return text[at:text.index("\n}\n", at)]


def test_reads_precede_the_ticket_and_the_writes_follow_it():
    body = _kernel()
    reads = [m.start() for m in re.finditer(r"passOf\(P\)|= W\.cnt->c\[kCntExtend0", body)]
    ticket = body.index("atomicAdd(&W.cnt->c[kCntTicket]")
    writes = [m.start() for m in re.finditer(r"W\.cnt->c\[kCnt(Extend0 \+ pass\.cur|Pass|Ticket)\] = ", body)]
    writes = [w for w in writes if w > ticket]
    reads = [r for r in reads if r < ticket]
    assert len(reads) == 2 and len(writes) == 3
    # (the barrier is outside the `take` branch: every thread reaches it)
    barrier = body.index("__syncthreads()", max(reads))
    assert max(reads) < barrier < body.index("if (take && n)") < ticket
    assert "__threadfence()" in body[body.index("if (take && n)"):ticket]
    assert ticket < body.index("__threadfence()", ticket) < min(writes)


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1, 1), (2, 1), (33, 1), (61, 41)])
def test_few_paths_repeat(ctx, w, h):
    b, shot = scenes.mixed_scene(w, h, frames=1, max_depth=7, n_spheres=6, level=3, seed=3, env_size=(32, 16))
    scene, film = ctx.create_scene(b.desc()), ctx.create_film(w, h)
    images = (0, 1, 2, 3, 8)
    ctx.set_counters(True)  # wavefront passes only
    try:
        ctx.render(scene, shot, film)
        want = np.stack([film.read(k) for k in images])
    finally:
        ctx.set_counters(False)
    for _ in range(200):
        film.clear()
        ctx.render(scene, shot, film)
        assert np.array_equal(np.stack([film.read(k) for k in images]), want)
