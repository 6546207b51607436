"""The arrival counts of cut strips (csrc/arrivals.cuh), which decide who adds up a strip's partial sums: every order in which the
contributors' reads and atomics can fall, whatever lay in the scratch before, and where the counts are kept."""
import itertools
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm-scaler_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
BITS = 10
MAX = (1 << BITS) - 1


def _contributor(word, tag, others, finished, me):
    """arrivals_open, then arrivals_last: one step per access to memory."""
    v = word[0]
    yield
    if (v ^ tag) >> BITS:
        if word[0] == v:
            word[0] = tag
        yield
    word[0] += 1
    if (word[0] - 1) & MAX == others:
        finished.append(me)
        yield
        word[0] = 0
    yield


def _run(order, garbage, tags, contributors):
    """Launches in turn on one word; order: which contributor of a launch moves next."""
    word, results = [garbage], []
    for tag in tags:
        finished = []
        live = {i: _contributor(word, tag, contributors - 1, finished, i) for i in range(contributors)}
        for i in itertools.chain(order, itertools.cycle(range(contributors))):
            if not live:
                break
            if i in live and next(live[i], "end") == "end":
                del live[i]
        results.append((finished, word[0]))
    return results


@pytest.mark.parametrize("garbage", [0, 1, MAX, (5 << BITS) | 3, (7 << BITS) | 2, 2 ** 64 - 1])
def test_one_contributor_finishes_and_leaves_a_zero(garbage):
    """Two launches, and the second one again (a replay); the scratch may hold an earlier launch's count."""
    tags = (8 << BITS, 6 << BITS, 6 << BITS)
    for order in itertools.product(range(3), repeat=8):
        for finished, left in _run(order, garbage, tags, 3):
            assert len(finished) == 1 and left == 0


def test_the_model_sees_a_count_that_two_launches_share():
    """What the counts must not do: a second launch's arrivals on the same word finish the strip of the first one early."""
    word, finished = [0], []
    a = [_contributor(word, 5 << BITS, 1, finished, "a%d" % i) for i in range(2)]
    b = [_contributor(word, 5 << BITS, 1, finished, "b%d" % i) for i in range(2)]
    for c in (a[0], b[0]):
        for _ in c:
            pass
    assert finished == ["b0"]        # and b's second contributor has not written its sums


def test_tags_are_never_handed_out_twice():
    with open(os.path.join(CSRC, "arrivals.cuh")) as f:
        text = f.read()
    factor = int(re.search(r"\* (0x[0-9A-F]+)ull << ARRIVALS_BITS", text).group(1), 16)
    assert factor % 2 == 1 and int(re.search(r"ARRIVALS_BITS = (\d+)", text).group(1)) == BITS
    tags = {n * factor % 2 ** 64 * 2 ** BITS % 2 ** 64 for n in range(1, 100001)}
    assert len(tags) == 100000 and 0 not in tags


@pytest.mark.parametrize("name", SOURCES)
def test_counts_are_in_the_callers_scratch(name):
    """Counts in memory of the library's own are shared by launches that share nothing else, in other streams and graphs."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    assert not re.search(r"__device__\s+(unsigned\s+)?(int|u?int\d+_t|long long)\s+\w*count\w*\s*\[", text)
    if "partials" in text and "__global__" in text:
        assert text.count("arrivals_open(") == 1 and text.count("arrivals_last(") == 1 and "atomicAdd(" not in text
