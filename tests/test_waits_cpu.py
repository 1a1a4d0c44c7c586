"""Waits that run out and arrivals that are counted, read from the sources (a run shows one order of many, and one in which a wait runs out
takes seconds)."""
import re

from test_launch_order_cpu import functions

BARRIER = r"__syncthreads|barrier\.sync|bar\.sync"
EXIT = re.compile(r"if \((?:[^;{}]*\|\| )?(?:[^;{}]*&& )?!(?:__all_sync\([^;{}]*)?(?:mbar_wait\w*|wait_count|wait_equal|grid_counter_wait)\([^;{}]*\)\s*(?:return;|\{[^{}]*return;\s*\})")


def behind(body, at):
    """The code that a warp which does not leave at `at` goes on to: the rest of each enclosing block, up to one that ends by returning."""
    out, depth, start = "", 0, at
    for i in range(at, len(body)):
        depth += {"{": 1, "}": -1}.get(body[i], 0)
        if depth < 0:
            out += body[start:i]
            if re.search(r"[;}]\s*return;\s*$", body[start:i]):
                return out
            depth, start = 0, i + 1
            alternative = re.match(r"\s*else\b[^{;]*\{", body[start:])      # not taken by who was in the block
            while alternative:
                start += alternative.end()
                level = 1
                while level:
                    level += {"{": 1, "}": -1}.get(body[start], 0)
                    start += 1
                alternative = re.match(r"\s*else\b[^{;]*\{", body[start:])
    return out + body[start:]


def test_no_barrier_behind_a_warp_that_leaves():
    """A warp that leaves alone when its wait runs out is missing at a barrier of the CTA that the others come to, where one that waits for
    the cluster's meanwhile would be waited for without an end: such a wait's outcome is made the CTA's, by the barrier itself."""
    seen = set()
    for name, (_, _, body) in functions().items():
        for m in EXIT.finditer(body):
            seen.add(name)
            assert not re.search(BARRIER, behind(body, m.end())), (name, m[0])
    assert {"gemv_stream_kernel", "kv_attn_kernel"} <= seen


def test_all_who_read_behind_a_count_have_met_who_counted():
    """One thread counts an arrival and acquires what the others left.  The threads that read it meet that thread at a barrier of their own first:
    a shuffle or a vote orders no memory."""
    seen = set()
    for name, (kernel, _, body) in functions().items():
        for m in re.finditer(r"count_arrival\(", body) if kernel else ():
            seen.add(name)
            rest = body[m.end():]
            read = re.search(r"__ldcg\(|ld\.global|\bws\b", rest)
            assert read and re.search(r"__syncwarp\(|__syncthreads", rest[:read.start()]), name
    assert seen == {"gemm_tc16_kernel", "kv_attn_kernel"}
