"""Rules of the execution model that a kernel can break without a wrong result on most runs, read off the sources."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chronicals_b200", "csrc")


def _closing(src, at):
    """Index behind the bracket that closes the one at ``at``."""
    opens, closes, depth = src[at], {"(": ")", "{": "}"}[src[at]], 0
    while True:
        depth += (src[at] == opens) - (src[at] == closes)
        at += 1
        if depth == 0:
            return at


def _kernels():
    """``(file, name, body without comments)`` of every ``__global__`` function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", src):
            at = m.end()
            while True:                                               # past __launch_bounds__(...) and the like
                call = re.compile(r"(\w+)\s*\(").search(src, at)
                at = _closing(src, call.end() - 1)
                if not call.group(1).startswith("__"):
                    break
            body = src.index("{", at)
            yield os.path.basename(path), call.group(1), src[body:_closing(src, body)]


def test_kernels_are_found():
    names = {name for _, name, _ in _kernels()}
    assert {"ce_logits_kernel", "attn_bwd3_kernel", "gemm2sm_kernel", "rmsnorm_bwd_kernel"} <= names


def test_a_cluster_meets_before_one_block_touches_the_memory_of_another():
    """Distributed shared memory belongs to a block that may not have started: a barrier of the whole cluster comes first."""
    access = re.compile(r"map_shared_rank|ld_shared_cluster|mbar_arrive_remote")
    seen = 0
    for path, name, body in _kernels():
        first = access.search(body)
        if first is None:
            continue
        seen += 1
        before = body[:first.start()]
        whole = "cluster_sync_all()" in before or re.search(r"\.sync\(\)", before)
        split = re.search(r"barrier_arrive\(\).*barrier_wait\(", before, re.S)
        assert whole or split, f"{path}: {name}"
    assert seen >= 2


def test_a_warpgroup_changes_its_registers_at_one_place():
    """``setmaxnreg`` is one instruction for all four warps of a warpgroup: no branch inside a warpgroup may lie before it."""
    seen = 0
    for path, name, body in _kernels():
        changes = list(re.finditer(r"reg_(?:inc|dec)<(\w+)>\(\)", body))
        for m in changes:
            seen += 1
            assert sum(c.group(0) == m.group(0) for c in changes) == 1, f"{path}: {name}: {m.group(0)} in more than one branch"
            opened = [c for c in re.finditer(r"if \(warp (\S+) (\w+)\) \{", body[:m.start()])
                      if _closing(body, c.end() - 1) > m.start()]     # the conditions that hold where it stands
            for c in opened:
                bound = int(c.group(2))
                assert c.group(1) in (">=", "<") and bound % 4 == 0, f"{path}: {name}: {c.group(0)}"
    assert seen >= 3
