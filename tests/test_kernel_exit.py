"""What an expert GEMM waits for before a CTA leaves, read from the kernel sources.

tcgen05.commit arrives on an mbarrier in shared memory when the MMAs are done, in a CTA pair on one
in each CTA, and nothing orders the arrivals of two commits.  A CTA that has seen the last
accumulator complete may therefore still be owed the arrivals that free its last slots.  If it left,
they would land in the barriers of whichever CTA gets that shared memory next.  A run cannot be relied on to
show it, so the waits are checked where they are written."""
import re

import pytest

from test_launch_order import kernel_body


@pytest.mark.parametrize("file,name", [
    ("gemm_tc5_ts.cuh", "expert_gemm_ts_kernel"),
    ("gemm_tc5_pair.cuh", "expert_gemm_pair_kernel"),
])
def test_every_slot_is_seen_free_before_exit(file, name):
    body = kernel_body(file, name)
    producer = body[body.index("warp == 1)"):body.index("warp == MMA_WARP)", body.index("warp == 1)"))]
    after_last_copy = producer[max(m.end() for m in re.finditer(r"tma_load_\dd\(", producer)):]
    assert re.search(r"(while|for) \([^{]*\bok &&[^{]*\{[^}]*mbar_wait\(bar_empty\(", after_last_copy)
    # and the other way round: what the issuing thread signals is on no third kind of barrier
    assert set(re.findall(r"commit(?:_both)?\(bar_(\w+)\(", body)) == {"empty", "tmem_full"}
