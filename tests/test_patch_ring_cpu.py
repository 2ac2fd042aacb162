"""The filter ring of conv_patch_kernel on the CPU: every interleaving of the warp that copies filter blocks, the issuing warps, the copies in
flight and the summing warps, over the ring sizes and accumulator counts that the kernel has, with the order of an issuing warp's waits read from its
source. No block's UMMAs may be issued before its filter block has landed, and every order must come to its end.

An mbarrier is what it is on the device: a wait for a parity passes once the phase of that parity is not the current one, so a wait that is asked
a whole phase early passes for the phase before.
"""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(__file__), "..", "crusaderbackend_b200", "csrc", "conv_patch.cu")


def waits_in_source():
    text = open(SOURCE).read()
    issuing = text[text.index("if (turn == a) {"):]
    order = re.findall(r"mbar_wait_uniform\(smem_u32\(&b\.(\w+)\[", issuing[:issuing.index("tc_fence_after()")])
    assert sorted(order) == ["ffull", "tempty"]
    return order


def fault(order, slots, accumulators, blocks):
    """None, or the first block whose UMMAs an interleaving issues before its filter block is there ("stuck": one that does not end)."""
    passes = lambda completed, fill: completed % 2 != fill % 2  # try_wait for the phase of a barrier's fill-th use
    # fills asked for; which have landed; per issuing warp: its next block, how many of its waits have passed; blocks computed; blocks summed
    start = (0, frozenset(), tuple((a, 0) for a in range(accumulators)), frozenset(), 0)
    seen, todo = {start}, [start]
    while todo:
        asked, landed, issuers, computed, summed = todo.pop()
        nexts = []
        # the copying warp: slot i % slots is free once the block that was in it has been computed
        if asked < blocks and (asked < slots or asked - slots in computed):
            nexts.append((asked + 1, landed, issuers, computed, summed))
        # a copy lands, in any order
        nexts += [(asked, landed | {i}, issuers, computed, summed) for i in range(asked) if i not in landed]
        for w, (block, passed) in enumerate(issuers):
            if block >= blocks:
                continue
            if passed < len(order):
                if order[passed] == "ffull":
                    completed = sum(1 for i in landed if i % slots == block % slots)
                    ok = passes(completed, block // slots)
                else:  # the accumulator's use before this one has been added up (its barrier counts one phase a use)
                    completed = sum(1 for i in range(summed) if i % accumulators == block % accumulators)
                    ok = passes(completed, block // accumulators - 1)
                if ok:
                    nexts.append((asked, landed, issuers[:w] + ((block, passed + 1),) + issuers[w + 1:], computed, summed))
            else:
                if block not in landed:
                    return block
                # (its UMMAs complete at some time: the order in which two warps' do is that of these steps)
                nexts.append((asked, landed, issuers[:w] + ((block + accumulators, 0),) + issuers[w + 1:], computed | {block}, summed))
        if summed < blocks and summed in computed:
            nexts.append((asked, landed, issuers, computed, summed + 1))
        if not nexts and not (asked == summed == blocks):
            return "stuck"
        for n in nexts:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return None


@pytest.mark.parametrize("accumulators", [1, 2])
@pytest.mark.parametrize("slots", [2, 3, 4])
def test_no_block_is_computed_before_its_filter_has_landed(slots, accumulators):
    text = open(SOURCE).read()
    assert "constexpr int kMaxRing = 4;" in text and "for (int fslots = kMaxRing; fslots >= 2; --fslots)" in text and "kAcc = BN == 32 ? 2 : 1" in text
    assert fault(waits_in_source(), slots, accumulators, 10) is None


def test_the_model_sees_a_phase_that_is_one_behind():
    """The planted order: the filter first. Three slots and two issuing warps let a warp see the other's fill of its slot as its own."""
    assert fault(["ffull", "tempty"], 3, 2, 10) is not None
    assert fault(["ffull", "tempty"], 4, 2, 10) is None and fault(["ffull", "tempty"], 3, 1, 10) is None
