"""What the dK/dV kernel's issuing warps wait for (csrc/attn/dkdv_waits.h). The roles of the kernel run as a model on the
CPU, one step of one role, one landing load or one MMA at a time in random order, with the kernel's own wait rule: no
product may read a tile that has not landed or has been replaced. On a GPU: the written gradients, which nothing adds
to, are the same bits on every launch, and blocks of few items match the host path."""
import math
import random
from collections import Counter

import pytest
import torch

from zenyx_b200.ops import _ext
from zenyx_b200.ops.attention import MaskSpec, attn_backward, attn_forward

WARPS = 2   # compute warps per half (eight in the kernel)


class _Kernel:
    """One block with n items. Barriers are those of attn_bwd.cu; a wait on a parity passes as mbarrier.try_wait does."""

    def __init__(self, n, rng, waits):
        self.n, self.rng, self.waits = n, rng, waits
        self.phase, self.arrived = Counter(), Counter()
        self.need = {"p_ready": WARPS, "ds_ready": WARPS, "stat_free": 2 * WARPS, "acc_done": 2}
        self.tile, self.tmem = {}, {}         # shared-memory slot -> landed item; (columns, half, warp) -> (kind, item)
        self.loads, self.queue, self.running = [], ([], []), [None, None]
        self.bad = []

    def arrive(self, bar):
        self.arrived[bar] += 1
        if self.arrived[bar] == self.need.get(bar[0], 1):
            self.arrived[bar] = 0
            self.phase[bar] += 1

    def load(self, buf, slot, item):
        self.tile[buf, slot] = None           # bytes of either tile until it has landed
        self.loads.append((buf, slot, item))

    def producer(self):
        for n in range(self.n):
            yield ("q_empty", n % 3), n // 3 & 1 ^ 1
            self.load("q", n % 3, n)
            yield ("do_empty", n % 2), n // 2 & 1 ^ 1
            self.load("do", n % 2, n)
            yield ("stat_free", n % 2), n // 2 & 1 ^ 1
            self.arrive(("stat_full", n % 2))

    def issuer(self, scores):
        x, y, depth = ("q", "do", 3) if scores else ("do", "q", 2)
        cols, out, ready = ("s", "s_full", "p_ready") if scores else ("dp", "dp_full", "ds_ready")
        q = self.queue[0 if scores else 1]

        def first(h, n):
            q.append(("mma", (x, n % depth, n), None, (cols, h, n)))
            q.append(("commit", (out, h)))

        yield (x + "_full", 0), 0
        first(0, 0)
        first(1, 0)
        for n in range(self.n):
            more = n + 1 < self.n
            for h in range(2):
                mask = self.waits(scores, h, more)
                if mask & 1:
                    yield (ready, h), n & 1
                if mask & 2:
                    yield (x + "_full", (n + 1) % depth), (n + 1) // depth & 1
                if mask & 4:
                    yield ("do_full", n % 2), n // 2 & 1
                q.append(("mma", (y, n % (5 - depth), n), (cols, h, n), None))
                if more:
                    first(h, n + 1)
        q.append(("commit", ("acc_done", 0)))

    def compute(self, half, w):
        lead = half == 1 and w == 0

        def convert(cols, n):
            if self.tmem.get((cols, half, w)) != ("raw", n):
                self.bad.append(("columns", cols, half, n))
            self.tmem[cols, half, w] = ("bf16", n)

        for n in range(self.n):
            yield ("stat_full", n % 2), n // 2 & 1
            yield ("s_full", half), n & 1
            if lead and n:
                self.arrive(("do_empty", (n - 1) % 2))
            convert("s", n)
            self.arrive(("p_ready", half))
            yield ("dp_full", half), n & 1
            if lead and n:
                self.arrive(("q_empty", (n - 1) % 3))
            convert("dp", n)
            self.arrive(("ds_ready", half))
            self.arrive(("stat_free", n % 2))

    def check(self, op):
        buf, slot, item = op[1]
        if self.tile.get((buf, slot)) != item:
            self.bad.append(("tile", buf, item))
        if op[2] is not None:
            cols, h, n = op[2]
            if any(self.tmem.get((cols, h, w)) != ("bf16", n) for w in range(WARPS)):
                self.bad.append(("operand columns", cols, h, n))

    def step_mma(self, i):
        op = self.running[i] or self.queue[i].pop(0)
        if op[0] == "commit":
            self.arrive(op[1])
        elif self.running[i] is None:
            self.check(op)
            self.running[i] = op
        else:                                 # still there when the product ends
            self.check(op)
            if op[3] is not None:
                cols, h, n = op[3]
                self.tmem.update({(cols, h, w): ("raw", n) for w in range(WARPS)})
            self.running[i] = None

    def land(self, k):
        buf, slot, item = self.loads.pop(k)
        self.tile[buf, slot] = item
        self.arrive((buf + "_full", slot))

    def run(self):
        roles = [self.producer(), self.issuer(True), self.issuer(False)]
        roles += [self.compute(h, w) for h in range(2) for w in range(WARPS)]
        waiting = [next(r) for r in roles]
        late = {buf: self.rng.choice((1, 1, 8, 64)) for buf in ("q", "do")}   # how reluctantly that buffer's loads land
        while True:
            moves = [(r,) for r, w in enumerate(waiting) if w is not None and self.phase[w[0]] & 1 != w[1]]
            moves += [("mma", i) for i in range(2) if self.running[i] or self.queue[i]]
            moves += [("land", k) for k in range(len(self.loads))]
            if not moves:
                break
            weight = [1 / late[self.loads[m[1]][0]] if m[0] == "land" else 1 for m in moves]
            m = self.rng.choices(moves, weight)[0]
            if m[0] == "mma":
                self.step_mma(m[1])
            elif m[0] == "land":
                self.land(m[1])
            else:
                waiting[m[0]] = next(roles[m[0]], None)
        if any(w is not None for w in waiting) or not self.phase["acc_done", 0]:
            self.bad.append(("stuck", waiting))
        return self.bad


def _violations(waits, items, seeds):
    return [b for n in items for s in range(seeds) for b in _Kernel(n, random.Random(100 * n + s), waits).run()]


def test_no_product_reads_a_tile_that_has_not_landed():
    assert _violations(_ext.host().dkdv_waits, (1, 2, 3, 7, 12), 40) == []


@pytest.mark.parametrize("scores,bit", [(True, 1), (True, 2), (True, 4), (False, 1), (False, 2)])
def test_the_model_sees_every_wait_that_is_left_out(scores, bit):
    def without(s, h, more):
        waits = _ext.host().dkdv_waits(s, h, more)
        return waits & ~bit if s == scores else waits

    assert _violations(without, (1, 2, 7), 40)


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,Hq,Hkv,causal", [
    (1, 128, 1, 1, True),       # one item per block: no later load to hide behind
    (4, 128, 32, 32, False),    # many such blocks at once
    (2, 384, 8, 2, True),       # 4 to 12 items
    (1, 4096, 32, 8, True),     # many waves, inputs of 100 MB
])
def test_written_gradients_are_the_same_bits_on_every_launch(B, S, Hq, Hkv, causal):
    """No atomics in this form, so a product that reads a tile too early shows as a difference between launches (L2 is
    flushed in front of each, so that the loads are late) and, for the smaller shapes, from the host path. Bound as in
    test_attention_schedule.py: P and dS are rounded to bf16."""
    torch.manual_seed(S + Hq)
    mask, scale = MaskSpec(causal), 1.0 / math.sqrt(128)
    host = [torch.randn(B, S, h, 128).bfloat16() for h in (Hq, Hkv, Hkv, Hq)]
    q, k, v, do = (t.cuda() for t in host)
    o, lse = torch.empty_like(q), torch.empty(B, Hq, S, device="cuda")
    attn_forward(q, k, v, o, lse, scale, mask, [0], [0])
    flush = torch.empty(1 << 28, device="cuda", dtype=torch.uint8)
    runs = []
    for i in range(6):
        grads = [torch.full(t.shape, math.nan, device="cuda") for t in (q, k, v)]
        flush.fill_(i)
        attn_backward(q, k, v, o, do, lse, torch.empty_like(lse), *grads, scale, mask, [0], [0], kv_overwrite=True)
        runs.append(grads)
    _ext.check_status()
    for r in runs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(runs[0], r))
    if S <= 384:
        want = [torch.empty(t.shape) for t in host[:3]]
        attn_backward(*host[:3], o.cpu(), host[3], lse.cpu(), torch.empty(B, Hq, S), *want, scale, mask, [0], [0],
                      kv_overwrite=True)
        for got, ref in zip(runs[0], want):
            assert (got.cpu() - ref).norm() <= 2e-2 * ref.norm()
