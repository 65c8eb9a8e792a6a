"""The rings of the tensor kernel (csrc/tc_gemm.cu) as a discrete-event model on the CPU.

An mbarrier wait names the parity of a phase, not its number: it cannot tell "the phase
asked for is complete" from "the phase before it has not completed yet".  Every wait is
safe only if something else keeps its waiter within one phase of the barrier.  The model
runs the kernel's roles (two TMA producers, two dequant groups per row set, one MMA
issuer per row set) on such barriers with random latencies and checks every slot that is
read for the fill it should hold."""
import heapq
import os
import random
import re

import pytest

SOURCE = os.path.join(os.path.dirname(__file__), "..", "shark_platform_b200", "csrc", "tc_gemm.cu")


def _geometry(nmax):
    """TcCfg<nmax>'s ring constants, evaluated from the source."""
    text = open(SOURCE).read()
    body = text[text.index("struct TcCfg {"):]
    body = body[:body.index("\n};")]
    env = {"NMAX": nmax}
    for name in ("ASLOTS", "HK", "HSLOTS", "WSLOTS", "XSLOTS"):
        expr = re.search(rf"static constexpr int {name} = ([^;]+);", body).group(1).replace("/", "//")
        parts = re.split(r"[?:]", expr)  # c1 ? a : c2 ? b : c
        py = parts[-1]
        for cond, val in reversed(list(zip(parts[0:-1:2], parts[1:-1:2]))):
            py = f"({val}) if ({cond}) else ({py})"
        env[name] = eval(py, {}, env)
    return {k: env[k] for k in ("HK", "HSLOTS", "WSLOTS", "XSLOTS")}


class ModelError(Exception):
    pass


class Barrier:
    def __init__(self, sim, count):
        self.sim, self.count, self.pending, self.loads, self.phase, self.waiters = sim, count, count, 0, 0, []

    def ready(self, parity):
        return (self.phase & 1) != parity

    def arrive(self, loads=0):
        if self.pending == 0:
            raise ModelError("an arrival on a phase that has had all of its arrivals")
        self.pending -= 1
        self.loads += loads
        self._maybe_complete()

    def landed(self):
        self.loads -= 1
        self._maybe_complete()

    def _maybe_complete(self):
        if self.pending == 0 and self.loads == 0:
            self.phase += 1
            self.pending = self.count
            again, self.waiters = self.waiters, []
            for role, parity in again:
                self.sim.wait(role, self, parity)


class Sim:
    """Roles are generators that yield (barrier, parity) to wait or a number to sleep."""

    def __init__(self, seed):
        self.rng, self.queue, self.now, self.order, self.live = random.Random(seed), [], 0.0, 0, 0

    def at(self, delay, fn):
        self.order += 1
        heapq.heappush(self.queue, (self.now + delay, self.order, fn))

    def start(self, role):
        self.live += 1
        self.at(0, lambda: self.step(role))

    def step(self, role):
        try:
            item = next(role)
        except StopIteration:
            self.live -= 1
            return
        if isinstance(item, tuple):
            self.wait(role, *item)
        else:
            self.at(item, lambda: self.step(role))

    def wait(self, role, bar, parity):
        if bar.ready(parity):
            self.at(0.02, lambda: self.step(role))
        else:
            bar.waiters.append((role, parity))

    def run(self):
        while self.queue:
            self.now, _, fn = heapq.heappop(self.queue)
            fn()
        if self.live:
            raise ModelError(f"{self.live} roles wait for ever")


def run_rings(HK, HSLOTS, WSLOTS, XSLOTS, seed, fills=40, late=0.05):
    """One tile of `fills` weight slots (128 k each), two 64-k stages per slot."""
    sim = Sim(seed)
    rng = sim.rng
    dur = lambda lo, hi: rng.uniform(lo, hi)
    latency = lambda: dur(20, 40) if rng.random() < late else dur(0.5, 2.0)
    wfull = [Barrier(sim, 1) for _ in range(WSLOTS)]
    wempty = [Barrier(sim, 2 if HK == 2 else 4) for _ in range(WSLOTS)]  # row sets x groups that read the slot
    xfull = [Barrier(sim, 1) for _ in range(XSLOTS)]
    xempty = [Barrier(sim, 2) for _ in range(XSLOTS)]
    a_ready = [[Barrier(sim, 1) for _ in range(2)] for _ in range(HSLOTS)]
    a_free = [[Barrier(sim, 1) for _ in range(2)] for _ in range(HSLOTS)]
    w_holds, x_holds = [None] * WSLOTS, [None] * XSLOTS
    a_holds = [[None] * 2 for _ in range(HSLOTS)]
    handovers = fills * 2 // HK

    def producer(full, empty, holds, slots, loads):
        for i in range(fills):
            s = i % slots
            yield empty[s], (i // slots & 1) ^ 1
            holds[s] = None
            full[s].arrive(loads)
            lands = sorted(latency() for _ in range(loads))

            def last(s=s, i=i):
                holds[s] = i
                full[s].landed()
            for t in lands[:-1]:
                sim.at(t, full[s].landed)
            sim.at(lands[-1], last)
            yield dur(0.01, 0.1)

    def dequant(grp, rset):
        ws, wph, a, aph = (grp if HK == 2 else 0), 0, grp, 1  # the kernel's counters
        for i in range(grp, handovers, 2):
            fill = i if HK == 2 else i // 2
            yield wfull[ws], wph
            if w_holds[ws] != fill:
                raise ModelError(f"fill {fill} read from a slot that holds {w_holds[ws]}")
            yield dur(0.05, 0.4)
            if w_holds[ws] != fill:
                raise ModelError(f"fill {fill} overwritten while it was read")
            wempty[ws].arrive()
            ws += HK
            if ws >= WSLOTS:
                ws, wph = ws - WSLOTS, wph ^ 1
            yield dur(0.1, 3.0)
            yield a_free[a][rset], aph
            if a_holds[a][rset] is not None:
                raise ModelError("a hand-over into a slot whose products are still running")
            a_holds[a][rset] = i
            yield dur(0.05, 0.3)
            a_ready[a][rset].arrive()
            a += 2
            if a >= HSLOTS:
                a, aph = a - HSLOTS, aph ^ 1

    pipe = [0.0]  # the tensor pipe works through the products in the order they were issued

    def issuer(rset):
        xs = xph = a = aph = 0
        for i in range(handovers):
            last = HK == 2 or i % 2 == 1
            if HK == 2 or i % 2 == 0:
                yield xfull[xs], xph
            yield a_ready[a][rset], aph
            if a_holds[a][rset] != i or x_holds[xs] != (i if HK == 2 else i // 2):
                raise ModelError("products of the wrong operands")
            pipe[0] = max(pipe[0], sim.now) + dur(0.2, 0.8)

            def done(a=a, xs=xs, last=last):
                a_holds[a][rset] = None
                a_free[a][rset].arrive()
                if last:
                    xempty[xs].arrive()
            sim.at(pipe[0] - sim.now, done)
            yield dur(0.02, 0.1)
            if last:
                xs += 1
                if xs == XSLOTS:
                    xs, xph = 0, xph ^ 1
            a += 1
            if a == HSLOTS:
                a, aph = 0, aph ^ 1

    sim.start(producer(wfull, wempty, w_holds, WSLOTS, 2))
    sim.start(producer(xfull, xempty, x_holds, XSLOTS, 2))
    for rset in range(2):
        sim.start(issuer(rset))
        for grp in range(2):
            sim.start(dequant(grp, rset))
    sim.run()


@pytest.mark.parametrize("nmax", [64, 128, 192])
def test_the_kernels_rings_hold_for_every_order_of_events(nmax):
    for seed in range(150):
        run_rings(**_geometry(nmax), seed=seed)


@pytest.mark.parametrize("HSLOTS", [2, 3, 4])
@pytest.mark.parametrize("WSLOTS", [2, 3, 4, 5, 6, 7])
def test_rule_of_the_static_assert(WSLOTS, HSLOTS):
    """With whole slots per group: an even ring keeps each slot with one group; an odd one
    passes slots between the groups, and a group may be a phase early unless its last
    hand-over vouches for the other group's fill of the slot (HSLOTS + 2 <= WSLOTS)."""
    bad = 0
    for seed in range(60):
        try:
            run_rings(2, HSLOTS, WSLOTS, 3, seed)
        except ModelError:
            bad += 1
    safe = WSLOTS % 2 == 0 or HSLOTS + 2 <= WSLOTS
    assert (bad == 0) == safe, bad


@pytest.mark.parametrize("name", ["tc_gemm.cu", "tc_pair_gemm.cu", "stream_gemm.cu"])
def test_no_kernel_leaves_with_copies_in_flight(name):
    """After a wait that ran out, mbar_wait returns at once: a producer's last waits for its
    own copies, and an issuer's for its MMAs, are mbar_drain, which ignores the abort flag."""
    text = open(os.path.join(os.path.dirname(SOURCE), name)).read()
    drains = re.findall(r"for \(uint32_t \w+ = [^;]+; \w+ < \w+; \+\+\w+\)\s*\n\s*(\w+)\(", text)
    assert drains and set(drains) == {"mbar_drain"}
    if name != "stream_gemm.cu":
        assert re.search(r"commit\w*\(mma_done[^\n]*\n(\s*__syncwarp\(\);\n)?\s*mbar_drain\(mma_done", text)
        # a scale slot is filled before the wait for its weights can run out: counted by itself
        assert "++gn;" in text and not re.search(r"gn = n /", text)
