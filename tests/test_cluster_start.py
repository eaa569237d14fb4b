"""A CTA may touch the shared memory of another CTA of its cluster only once
that CTA runs, which nothing but a barrier of the whole cluster shows.  A run
cannot show the absence of the barrier (the peers nearly always run by then),
so this reads the batched kernel: on every way to its first store to a peer
there is a barrier of the team.
"""
import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / "pimd-b_gb300" / "csrc" / "batch.cu"


def test_a_barrier_comes_before_the_first_store_to_a_peer():
    text = re.sub(r"//[^\n]*", "", SOURCE.read_text())
    body = text[text.index("k_batch(const BatchRep"):]
    before_loop = body[:body.index("for (;;)")]
    assert "set_peer" not in before_loop and "peer(" not in before_loop
    assert re.search(r"if constexpr \(kCl\)\s+T::sync\(\);", before_loop)
