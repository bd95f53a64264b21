"""A host-side model of the rings of stream_linear_kernel and prefill_attention_kernel (csrc): a slot is released by an arrival that the tensor core makes when
the multiplications in front of it are complete, and is waited for before the slot is filled again.  Every such arrival must be waited for: one that is
not can reach shared memory when the CTA has left it.  The condition of a release is read from the kernels."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpuk_b200", "csrc")


def _condition(file):
    text = open(os.path.join(CSRC, file)).read()
    assert len(re.findall(r"tc_commit\(&empty", text)) == 1, "one place that releases a slot"
    m = re.search(r"if \(([^;{}]*)\) tc_commit\(&empty", text)
    assert m, "a release without a condition"
    return m.group(1).replace("p.stages", "stages").replace("kSlots", "stages")


def _outstanding(condition, steps, stages, names):
    """Arrivals on a slot that no refill waits for, and refills that no arrival answers."""
    arrivals, waits = [0] * stages, [0] * stages
    for i in range(steps):
        arrivals[i % stages] += bool(eval(condition, {}, dict(names, i=i, stages=stages)))
        if i >= stages:
            waits[i % stages] += 1
    return [a - w for a, w in zip(arrivals, waits)]


@pytest.mark.parametrize("steps", [0, 1, 2, 3, 4, 5, 6, 7, 11, 16, 64, 65])
def test_every_release_is_waited_for(steps):
    condition = _condition("stream_linear.cu")
    for stages in range(1, 12):
        assert not any(_outstanding(condition, steps, stages, {"nsteps": steps}))


@pytest.mark.parametrize("rounds", list(range(1, 20)) + [64])
def test_every_release_of_the_prefill_s_ring_is_waited_for(rounds):
    text = open(os.path.join(CSRC, "prefill_attention.cu")).read()
    stages = int(re.search(r"constexpr int kSlots = (\d+);", text).group(1))
    assert not any(_outstanding(_condition("prefill_attention.cu"), 2 * rounds, stages, {"rounds": rounds}))
