"""The hand-over of a finished item's accumulators in the fused attention's dK / dV kernel, as a model of
its roles and barriers in which every arrival may come late: whoever reads the last item's accumulators
has waited for that item, whatever the order of the arrivals.  On a GPU a wait that passes a phase early
shows only when an arrival is hundreds of cycles late, so this runs on the CPU."""

import os
import random
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vkgrad_b200", "csrc",
                   "attn_sm100.cu")
SOFTMAX_WARPS = 2      # 16 in the kernel; two show every order that matters


def out_barriers():
    """How many barriers the kernel signals finished items on, and that its three users agree on which."""
    text = open(SRC).read()
    n = int(re.search(r"\bKV_ACC_FREE = (\d+)", text)[1]) - int(re.search(r"\bKV_OUT_FULL = (\d+)", text)[1])
    by_item = re.findall(r"KV_OUT_FULL \+ \((?:last_)?j & 1\)", text)
    assert n == 1 or (n == 2 and len(by_item) == 3), (n, by_item)
    return n


class Barrier:
    def __init__(self, count):
        self.count, self.left, self.phase = count, count, 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1

    def passes(self, parity):      # mbarrier.try_wait.parity
        return self.phase & 1 != parity


def roles(items, n_out, done, read):
    """The roles as generators of ("wait", barrier, parity), ("arrive", barrier) and ("commit", barrier,
    product): a commit arrives some time after its product has retired, each on its own."""
    last = len(items) - 1
    out = lambda j: (("out", j % n_out), (j // n_out) & 1)

    def scores():                  # warp 1
        g = 0
        for steps in items:
            for _ in range(steps):
                yield "wait", "sdp_free", (g & 1) ^ 1
                yield "commit", "sdp_full", None
                g += 1

    def gradients():               # warp 2
        g = 0
        for j, steps in enumerate(items):
            for i in range(steps):
                yield "wait", "pds_full", g & 1
                if i == 0:
                    yield "wait", "acc_free", (j & 1) ^ 1
                yield "commit", "pds_free", (j, i)
                if i == steps - 1:
                    yield "commit", out(j)[0], (j, i)
                g += 1

    def epilogue():                # every item but the last
        for j in range(last):
            yield ("wait",) + out(j)
            read.append((j, (j, items[j] - 1) in done))
            yield "arrive", "acc_free"

    def softmax():
        g = 0
        for steps in items:
            for _ in range(steps):
                yield "wait", "sdp_full", g & 1
                yield "arrive", "sdp_free"
                yield "wait", "pds_free", (g & 1) ^ 1
                yield "arrive", "pds_full"
                g += 1
        yield ("wait",) + out(last)
        read.append((last, (last, items[last] - 1) in done))
    return [scores(), gradients(), epilogue()] + [softmax() for _ in range(SOFTMAX_WARPS)]


def play(items, n_out, rng, late):
    """Runs the roles to their end in an order drawn from rng; arrivals on the barriers `late` names come
    only when nothing else can happen.  Returns [(item read, whether it had been finished)]."""
    done, read, pending = set(), [], []
    bars = {b: Barrier(SOFTMAX_WARPS if b in ("sdp_free", "pds_full") else 1)
            for b in ["sdp_full", "sdp_free", "pds_full", "pds_free", "acc_free"] + [("out", i) for i in range(n_out)]}
    live = {i: [r, op] for i, r in enumerate(roles(items, n_out, done, read)) if (op := next(r, None))}
    while live:
        can = [i for i, (_, op) in live.items() if op[0] != "wait" or bars[op[1]].passes(op[2])]
        ready = [c for c in pending if not late(c[0])] or ([] if can else pending)
        assert can or ready, "the roles wait for one another"
        pick = rng.choice(can + ready)
        if pick in ready:
            pending.remove(pick)
            if pick[1] is not None:
                done.add(pick[1])
            bars[pick[0]].arrive()
            continue
        gen, op = live[pick]
        if op[0] == "arrive":
            bars[op[1]].arrive()
        elif op[0] == "commit":
            pending.append((op[1], op[2]))
        try:
            live[pick][1] = next(gen)
        except StopIteration:
            del live[pick]
    return read


def wrong_reads(items, n_out, seeds=40):
    wrong = []
    for late in (lambda bar: bar[0] == "out", lambda bar: False, lambda bar: bar == "pds_free"):
        for seed in range(seeds):
            wrong += [j for j, ok in play(items, n_out, random.Random(seed), late) if not ok]
    return wrong


@pytest.mark.parametrize("items", [[1], [3], [1, 1], [2, 1], [3, 2, 1], [1, 1, 1, 1], [4, 4, 3, 1, 1], [2, 2, 2]])
def test_nobody_reads_an_item_that_is_not_finished(items):
    assert not wrong_reads(items, out_barriers())


@pytest.mark.parametrize("registers", [0, 72, 79, 80, 85])
def test_kernels_with_too_few_registers_are_refused(registers):
    """The softmax warps ask for 96 registers of the 80 a thread that the block is launched with; that
    request waits without a limit, so fewer must end in an error before the launch."""
    from vkgrad_b200 import _lib
    from vkgrad_b200.vk import VkError, _check
    call = _lib.load().vkg_selftest_attn_registers(registers)
    if registers >= 80:
        assert call == 0
    else:
        with pytest.raises(VkError, match=f"launched with {registers} registers"):
            _check(call, "attn_bwd")


def test_one_barrier_for_all_items_would_be_read_a_phase_early():
    """What the model is for: the last item of one step, with the item before it not signalled yet."""
    assert wrong_reads([2, 1], 1) and not wrong_reads([2, 1], 2)
