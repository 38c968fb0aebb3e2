"""The row sums of the FP32 cluster sweeps (jacobi_cluster.cu) under the orders
that the split cluster barrier allows.

In sweep s a thread stores its row sum to slot s % kRowSlots after its arrival at
the barrier and before its wait; the summing threads, after their arrival, read the
slot of sweep s - kRowLag.  The only order between threads is that of the barrier:
what precedes a thread's k-th arrival precedes what follows any thread's k-th wait.
Every read has to follow the store it means, and every later store to that slot has
to follow the read, whichever thread runs ahead."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "picard_b200", "csrc",
                   "jacobi_cluster.cu")


def protocol():
    with open(SRC) as f:
        text = f.read()

    def const(name):
        return int(re.search(rf"constexpr int {name} = (\d+);", text).group(1))

    return const("kRowLag"), const("kRowSlots")


# A point of the program, as (arrivals done, waits done) of its thread.
def ordered(first, second):
    """Whether `first` in one thread precedes `second` in another: some barrier that
    the first thread arrives at afterwards has been waited for by the second."""
    return first[0] + 1 <= second[1]


def violations(lag, slots, m):
    after_arrive = [(s + 1, s) for s in range(m)]  # sweep s: its arrival is done, its wait is not
    after_last = (m, m)
    read = {}
    for s in range(m):
        if s >= lag:
            read[s - lag] = after_arrive[s]
    for s in range(max(0, m - lag), m):
        read[s] = after_last  # behind a block barrier: after every store
    assert sorted(read) == list(range(m)), "every sweep is summed once"
    bad = []
    for s, at in read.items():
        if at != after_last and not ordered(after_arrive[s], at):
            bad.append(("read before the store", s))
        for later in range(s + slots, m, slots):
            if not ordered(at, after_arrive[later]):
                bad.append(("overwritten before the read", s, later))
    return bad


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 16, 64])
def test_rows_are_read_between_their_store_and_the_next(m):
    lag, slots = protocol()
    assert violations(lag, slots, m) == []


def test_the_model_sees_a_missing_barrier():
    assert violations(1, 3, 8) and violations(1, 4, 8) and violations(2, 3, 8)
