"""The converters' wait for their weights, as a model: converter groups take K blocks in turn, loads land in any order, and a
wait by parity passes whenever the barrier's current phase has the other parity.  It is sound only if a barrier belongs to
one group (the number of barriers is a multiple of the number of groups), whatever the ring's length."""
import random
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mxmoe_b200" / "csrc"


def early_passes(stages: int, groups: int, barriers: int, skips: bool, seed: int, blocks: int = 400) -> int:
    """Waits that passed although their block had not landed.  ``skips``: stages of other tiles between the blocks."""
    rng = random.Random(seed)
    at, pos = [], 0
    for _ in range(blocks):                       # ring position of every converted block
        if skips and rng.random() < 0.1:
            pos += rng.choice((11, 16, 22, 32, 48))
        at.append(pos)
        pos += 1
    phase = [0] * barriers                        # completed phases of each barrier
    nxt = list(range(groups))                     # the block each group waits for
    done, pending, issued, early = set(), [], 0, 0
    while min(nxt) < blocks:
        oldest = min(nxt)                         # MMAs run in order: everything before the oldest open block is consumed
        while issued < blocks and at[issued] < at[oldest] + stages:
            pending.append(issued)
            issued += 1
        if pending and rng.random() < 0.5:
            n = pending.pop(rng.randrange(len(pending)))
            done.add(n)
            phase[n % barriers] += 1
        g = rng.randrange(groups)
        n = nxt[g]
        if n < blocks and phase[n % barriers] % 2 != (n // barriers) % 2:
            if n not in done:
                early += 1
            nxt[g] += groups
    return early


@pytest.mark.parametrize("skips", [False, True])
@pytest.mark.parametrize("stages,groups", [(5, 2), (7, 3), (10, 3)])
def test_a_barrier_belongs_to_one_group(stages, groups, skips):
    barriers = -(-stages // groups) * groups
    assert sum(early_passes(stages, groups, barriers, skips, s) for s in range(20)) == 0
    # a barrier per stage of these rings changes hands: the fault that this arrangement replaces
    assert sum(early_passes(stages, groups, stages, skips, s) for s in range(20)) > 0


def test_the_kernels_have_this_arrangement():
    duo, swap = (CSRC / "gg_duo_kernel.cu").read_text(), (CSRC / "gg_swap_kernel.cu").read_text()
    assert re.search(r"kWBars\s*= \(kStages \+ kCvtGroups - 1\) / kCvtGroups \* kCvtGroups;", duo)
    assert re.search(r"kWBars\s*= 2 \* kStages;", swap) and re.search(r"kCvtWarps\s*= 8;", swap)
    assert "wfull[G::kWBars]" in duo and "wfull[G::kWBars]" in swap
    # every role that walks these barriers wraps at their number, not at the ring's length
    assert "if (++wbar == G::kWBars) wbar = 0;" in duo and duo.count("wb -= G::kWBars; wpar ^= 1u;") == 2
    assert swap.count("if (++wb == G::kWBars) wb = 0;") == 2 and swap.count("if (++wb == G::kWBars) { wb = 0; wphase ^= 1u; }") >= 1


def test_arrivals_release_what_converters_write_to_shared_memory():
    """The CTA-pair kernel's converters signal the leader's MMA warp.  Without release semantics that is good for payloads in
    tensor memory only.  Packed activations are expanded into shared memory: the leader's converters release to their own
    barrier, the second CTA's to theirs, from which forwarders release at cluster scope, and the MMA warp acquires at it, by
    the poll that looks ahead too."""
    duo = (CSRC / "gg_duo_kernel.cu").read_text()
    cvt = duo[duo.index("if (kMode == 2 && ti.scheme == SCH_W4A4) {"):]
    cvt = cvt[:cvt.index("s += kCvtGroups;")]
    assert cvt.index("convert_w4a4<") < cvt.index("fence_proxy_async_smem();") < cvt.index("__syncwarp();")
    assert re.search(r"if \(kMode == 2 && ti\.scheme == SCH_W4A4\)\s+mbar_arrive\(\(rank == 0 \? full0 : smem_base \+ MXB_CTRL\(xdone\)\) \+ 8 \* s\);", cvt)
    fwd = duo[duo.index("void forward_arrivals("):duo.index("gg_duo_kernel(const")]
    assert fwd.index("bar_wait<G>(smem_base, xdone0") < fwd.index("fence_acq_rel_cluster();") < fwd.index("mbar_arrive_leader_relaxed_n(full0")
    mma = duo[duo.index("__device__ __forceinline__ bool mma_tile("):]
    mma = mma[:mma.index("return true;")]
    assert "wwait<G, kAcquire>(" in mma and "mbar_test_wait_cluster(" in mma
    assert re.findall(r"mma_tile<(\d), ([^,]+), G>", duo) == [(str(v), "kMode == 2") for v in range(4)]
