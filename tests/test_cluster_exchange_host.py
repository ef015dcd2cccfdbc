"""CTAs of a cluster that send partials into one another's shared memory (``csrc/gemm_split_sm100.cu``, ``csrc/qwen3_chain.cu`` and both kernels of
``csrc/qwen3_short.cu``): none may leave while another can still write to it, also where waits run out.  A host model of the roles; no wait is made to run out on a GPU
for it (CPU)."""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ittai_b200", "csrc")


def _leave(rng, n, hold):
    """``n`` CTAs in a random interleaving.  Each waits for its own data (some in vain: they give up late and send all the same), sends a
    partial to every owner, collects what it owns, or, if it gave up or has no patience, stops collecting; what is sent lands some time
    later.  ``hold``: a CTA that gave up leaves once its partials have landed or, its patience at an end again, once all others have
    left; otherwise after some time.  Returns the writes into CTAs that had left and the number of CTAs that gave up."""
    owners = rng.randint(1, n)
    state, gave_up, in_flight, landed, late = ["wait"] * n, [rng.random() < 0.3 for _ in range(n)], [], [0] * n, 0
    slow = [rng.choice([1, 1, 1, 40]) for _ in range(n)]                 # a CTA's turns per step of its own
    while any(s != "left" for s in state) or in_flight:
        c = rng.randrange(n + 1)
        if c == n:
            if in_flight:
                owner = in_flight.pop(rng.randrange(len(in_flight)))
                late += state[owner] == "left"
                landed[owner] += 1
            continue
        if rng.randrange(slow[c]):
            continue
        complete = c >= owners or landed[c] == n
        if state[c] == "wait":
            state[c] = "send"
        elif state[c] == "send":
            in_flight += range(owners)
            state[c] = "collect"
        elif state[c] == "collect":
            if complete and not gave_up[c]:
                state[c] = "left"
            elif gave_up[c] or rng.random() < 0.01:
                gave_up[c], state[c] = True, "gave up"
        elif state[c] == "gave up":
            if not hold or complete:
                state[c] = "left"
            elif rng.random() < 0.05:
                state[c] = "barrier"
        elif state[c] == "barrier" and all(s in ("left", "barrier") for s in state) and not in_flight:
            state[c] = "left"                                            # the time for copies in flight follows the barrier
    return late, sum(gave_up)


@pytest.mark.parametrize("n", [2, 4, 7, 8, 12])
def test_no_cta_leaves_ahead_of_what_is_sent_to_it(n):
    runs = [_leave(random.Random(seed), n, True) for seed in range(300)]
    assert not any(late for late, _ in runs) and sum(gave > 0 for _, gave in runs) > 100
    assert any(_leave(random.Random(seed), n, False)[0] for seed in range(300)), "the model does not show what the barrier is for"


def _block(text, start):
    """The text of the brace block that begins at or after ``start``."""
    i = text.index("{", start)
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == "{") - (text[j] == "}")
        if depth == 0:
            return text[i:j + 1]


@pytest.mark.parametrize("source,failure", [("gemm_split_sm100.cu", "if (*abort_flag) {"), ("qwen3_chain.cu", "if (failed) {"),
                                            ("qwen3_short.cu", "if (!__syncthreads_and(ok && came)) {"), ("qwen3_short.cu", "if (failed) {")])
def test_the_kernels_follow_the_model(source, failure):
    """In the branch of a CTA that gave up: the wait for the bytes, the barrier behind it, and then the time for copies in flight."""
    with open(os.path.join(CSRC, source)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    leaving = _block(text, text.index(failure, text.rindex("st_async_f32x2(&rml" if "chain" in source else "st.async")))
    steps = [re.search(p, leaving) for p in (r"mbar_try_wait_cluster\(&?arrived", r"__syncthreads_and", r"cluster_arrive\(\)|cluster\.arrive",
                                             r"cluster_wait\(\)|cluster\.wait", r"clock64")]
    assert all(steps) and [m.start() for m in steps] == sorted(m.start() for m in steps)
