"""A kernel of a wave that finds the error word set returns at its start, and
other kernels of the wave may set the word at that very moment.  The threads of
a block that meet at barriers (or share an array) and the lanes of a warp that
vote must therefore take one answer between them: block_failed or warp_failed
(wave_common.cuh), never each thread its own."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "photon_gb300", "csrc")
BLOCK_WIDE = re.compile(r"__shared__|__syncthreads|begin_grads|block_fetch")


def _kernels():
    """(name, body) of every __global__ function that asks for the error word."""
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = open(os.path.join(CSRC, f)).read()
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            start = text.index("{", m.end())
            depth, end = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
                if depth == 0:
                    break
            body = text[start:end]
            if "_failed(" in body:
                yield m.group(1), body


def test_no_thread_answers_alone():
    found = dict(_kernels())
    assert {"k_trace", "k_shadow", "k_mat_hist", "k_mat_scan", "k_mat_scatter", "k_adj_resolve"} <= set(found)
    alone = [k for k, body in found.items() if "wave_failed(" in body]
    assert not alone, alone


def test_kernels_with_barriers_ask_as_a_block():
    shared_rings = {"k_trace"}  # its shared array is one ring per warp, no barrier of the block
    bad = [k for k, body in _kernels()
           if BLOCK_WIDE.search(body) and "block_failed(" not in body and k not in shared_rings]
    assert not bad, bad
