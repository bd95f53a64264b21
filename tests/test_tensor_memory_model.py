"""A host-side model of how the clusters of stream_linear_kernel (csrc/stream_linear.cu) share tensor memory.  An SM has 512 columns; a CTA takes kAcc * N of
them, waiting without a limit, and meets the other CTAs of its cluster in a barrier.  If it frees its columns only behind the barrier, clusters can wait for one
another in a ring: each has CTAs that hold columns and wait at the barrier, and CTAs that wait for columns which the others' hold.  The order of the
two steps is read from the kernel, and the model lets every order of allocation happen."""
import os
import random
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpuk_b200", "csrc", "stream_linear.cu")
COLUMNS = 512


def _kernel():
    text = open(SRC).read()
    return text[text.index("stream_linear_kernel("):text.index("kernel_for(")]


def _frees_before_waiting():
    body = _kernel()
    waits = [m.start() for m in re.finditer(r"cluster_(?:wait|barrier)\(\)", body)]
    return body.index("tmem_free<") < min(waits)


def _finishes(per_sm, columns, cluster, free_first, rng):
    """Clusters of one CTA on each of `cluster` SMs, `per_sm` of them resident together; True if all get through, whoever is served first."""
    ctas = [(c, s) for c in range(per_sm) for s in range(cluster)]
    free = [COLUMNS] * cluster
    state = dict.fromkeys(ctas, "allocating")
    while any(v != "done" for v in state.values()):
        steps = []
        for c, s in ctas:
            peers = [state[c, p] for p in range(cluster)]
            if state[c, s] == "allocating" and free[s] >= columns:
                steps.append((c, s))
            elif state[c, s] == "holding":       # multiplied: nothing it waits for but itself
                steps.append((c, s))
            elif state[c, s] == "barrier" and not any(p in ("allocating", "holding") for p in peers):
                steps.append((c, s))
        if not steps:
            return False
        c, s = rng.choice(steps)
        if state[c, s] == "allocating":
            free[s] -= columns
            state[c, s] = "holding"
        elif state[c, s] == "holding":
            state[c, s] = "barrier"
            free[s] += columns if free_first else 0
        else:
            state[c, s] = "done"
            free[s] += 0 if free_first else columns
    return True


@pytest.mark.parametrize("cluster", [2, 3, 8])
@pytest.mark.parametrize("columns", [64, 128])
def test_clusters_do_not_wait_for_one_another_s_columns(columns, cluster):
    free_first = _frees_before_waiting()
    for seed in range(25):
        assert _finishes(11, columns, cluster, free_first, random.Random(seed))


def test_the_model_finds_the_ring():
    assert not all(_finishes(11, 128, 8, False, random.Random(seed)) for seed in range(25))
