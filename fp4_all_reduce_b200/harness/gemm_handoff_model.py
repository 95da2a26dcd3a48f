"""A randomised model of the partial-tile hand-off of the stream-K GEMM (no GPU), after csrc/kernels/gemm_fp4.cu.

Unit u + 1 leaves the FP32 partial of a tile it shares with unit u in ITS slot and sets the slot's flag with a
release store; unit u waits for the flag (acquire), adds the partial, and resets the flag with a release store once
every lane has the data in registers.  Slots and flags belong to a workspace, not to a launch, so the next launch of the
workspace reuses them; its producer first waits until the flag is 0.  Every unit of every launch is its own thread of
control and a random scheduler interleaves them.  Between the launches of one stream the model asks less than the kernel
gives: "a unit of the next launch starts after the SAME unit index of the one before has finished" (the kernel touches its
workspace only after the whole launch before it).  Launches of different streams (launch L is on stream L % streams) are
not ordered at all, and every stream has its own workspace.

Checked on every schedule: a producer never overwrites a partial that has not been consumed; a consumer only ever
reads the partial of its own launch, complete; every flag is 0 at the end; nobody waits forever.  `variant` removes
one rule to show that the checker can fail: "no_free_wait" (the producer does not wait for flag == 0),
"early_reset" (the consumer resets the flag before it has read the data) and, with several streams, "one_space" (one
workspace for the device) must all produce violations.
"""
from __future__ import annotations

import random


class Violation(AssertionError):
    pass


def run(units: int, launches: int, seed: int, variant: str = "product", words: int = 3, max_steps: int = 200000,
        streams: int = 1) -> None:
    rng = random.Random(seed)
    space = (lambda L: 0) if variant == "one_space" else (lambda L: L % streams)
    # flag of slot s of a workspace (slot s is written by unit s, read by unit s - 1)
    flag = {(w, s): 0 for w in range(streams) for s in range(units)}
    slot = {k: [None] * words for k in flag}
    # which units share a tile: in a launch unit u consumes from u + 1 iff shared[L][u]; random per launch
    shared = [[rng.random() < 0.7 for _ in range(units - 1)] + [False] for _ in range(launches)]
    # program of (launch, unit): produce (if unit u - 1 consumes from u) FIRST, then consume (if shared) LAST
    pc = {}
    for L in range(launches):
        for u in range(units):
            ops = []
            if u > 0 and shared[L][u - 1]:
                if variant != "no_free_wait":
                    ops.append(("wait_free", u))
                ops += [("write", u, w) for w in range(words)] + [("set", u)]
            ops.append(("work",))
            if shared[L][u]:
                ops.append(("wait_full", u + 1))
                if variant == "early_reset":
                    ops.append(("reset", u + 1))
                ops += [("read", u + 1, w) for w in range(words)]
                if variant != "early_reset":
                    ops.append(("reset", u + 1))
            pc[(L, u)] = [ops, 0]
    done = set()
    steps = 0
    while len(done) < launches * units:
        steps += 1
        if steps > max_steps:
            raise Violation("no progress: a wait never ends")
        ready = [(L, u) for (L, u), (ops, i) in pc.items() if (L, u) not in done and (L < streams or (L - streams, u) in done)]
        L, u = rng.choice(ready)
        ops, i = pc[(L, u)]
        op = ops[i]
        advance = True
        s = (space(L), op[1]) if len(op) > 1 else None
        if op[0] == "wait_free":
            advance = flag[s] == 0
        elif op[0] == "write":
            w = op[2]
            if flag[s] != 0:
                raise Violation(f"launch {L} unit {u} overwrites slot {s} whose partial has not been consumed")
            slot[s][w] = (L, w)
        elif op[0] == "set":
            flag[s] = 1
        elif op[0] == "wait_full":
            advance = flag[s] == 1
        elif op[0] == "read":
            w = op[2]
            if slot[s][w] != (L, w):
                raise Violation(f"launch {L} unit {u} read {slot[s][w]} from slot {s} word {w}")
        elif op[0] == "reset":
            flag[s] = 0
        if advance:
            pc[(L, u)][1] = i + 1
            if i + 1 == len(ops):
                done.add((L, u))
    if any(flag.values()):
        raise Violation("a flag is still set at the end")


def check(units: int, launches: int, seeds: int = 200, variant: str = "product", streams: int = 1) -> int:
    """Number of seeds (out of `seeds`) on which the model found a violation."""
    bad = 0
    for seed in range(seeds):
        try:
            run(units, launches, seed, variant, streams=streams)
        except Violation:
            bad += 1
    return bad
