"""The int8-slice product releases its tensor and shared memory only after the
MMAs it issued have ended, on every way out.  The ways out that need a barrier
to stall cannot be run, so this reads the source: the MMA warp commits each
chunk to the barrier of its outcome (accumulators, or drain after a wait that
gave up) and waits for that last commit before it leaves its role."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "turbid_b200", "csrc", "islice.cu")


def test_last_commit_is_awaited_on_every_way_out():
    src = open(SRC).read()
    role = src[src.index("// ---- MMAs"):src.index("// ---- epilogue")]
    commit = re.search(r"ok \? bar_acc : bar_drain\),\s*\"r\"\(elected\)\);\s*committed = true;", role)
    assert commit
    tail = role[commit.end():]
    # after the chunk loop: no return, and one wait that depends on the commit alone
    assert "return" not in tail
    waits = re.findall(r"(if \(.*?\) )?mbar_wait\((.*)\);", tail)
    assert waits == [("if (committed) ", "ok ? bar_acc : bar_drain, ok ? (nchunks - 1) & 1 : 0")]
    # tensor memory is released behind the block-wide barrier that follows the roles
    end = src[src.index("// ---- epilogue"):]
    assert end.index("__syncthreads();") < end.index("tcgen05.dealloc")
