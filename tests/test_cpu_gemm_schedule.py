"""The dequantising groups of the GEMM core (pie_gemm.cuh) wait for packed chunks by slot parity and skip the chunks they do not
read.  A parity wait is only right if the slot's previous chunk has arrived by then: walked here for every group, chunk size and
tile length, over many tiles."""
import os
import re

import pytest

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "proxy_inference_engine_b200", "csrc", "pie_gemm.cuh")


def constants():
    with open(HEADER) as f:
        text = f.read()
    pick = lambda pattern: int(re.search(pattern, text).group(1))
    return pick(r"int GROUPS = (\d+);"), pick(r"RING = QB \? (\d+) : 0"), pick(r"int S = QB \? (\d+) :")


def unsound_waits(per_chunk, steps, groups, ring, stages, tiles=40):
    """Waits of a group for a chunk whose slot's previous chunk it neither waited for nor knows to have arrived.  Known: when a
    group dequantised its last K step v, the MMA of step v - stages had finished, and with it the chunks of all steps up to it."""
    chunk_of, first_step, base = [], {}, 0
    for _ in range(tiles):
        for k in range(steps):
            first_step.setdefault(base + k // per_chunk, len(chunk_of))
            chunk_of.append(base + k // per_chunk)
        base += -(-steps // per_chunk)
    bad = 0
    for g in range(groups):
        waited, last = set(), None
        for step in range(g, len(chunk_of), groups):
            before = chunk_of[step] - ring
            if before >= 0 and before not in waited:
                bad += last is None or first_step[before] > last - stages
            waited.add(chunk_of[step])
            last = step
    return bad


@pytest.mark.parametrize("per_chunk", [2, 4])      # 8-bit, 4-bit weights: K steps of 64 in 128 packed bytes
def test_no_group_outruns_a_skipped_chunk(per_chunk):
    groups, ring, stages = constants()
    for steps in range(2, 450, 2):                 # K is a multiple of 128; a cluster rank's share of 512
        assert unsound_waits(per_chunk, steps, groups, ring, stages) == 0, steps


def test_the_walk_finds_the_broken_settings():
    assert unsound_waits(4, 64, 3, 1, 6) == 0 < unsound_waits(2, 64, 3, 1, 6)
    assert unsound_waits(2, 64, 4, 3, 5) > 0
