"""A model of the barrier protocol of the kernel that runs all layers of a decode step (csrc/wf_step.cu) when a wait runs out: a cluster
of CTAs with a producer and consumer warps each, copies and sends that land in any order, one wait that gives up early or one
transfer that never lands.  Checked: no barrier is armed while its phase is incomplete, nothing is sent and no cache row written that
is computed from what has not arrived, nothing is on its way into a CTA's shared memory when that goes away, every role runs to its
end.  A model of the protocol, not of the hardware: it guards the bookkeeping against edits."""
import random

import pytest

CTAS, WARPS, LAYERS, STAGES = 3, 2, 3, 2
PHASES = ("qkv", "o", "gu", "down")
COUNT = {"qkv": 2, "o": 1, "gu": 3, "down": 1}  # ring stages of a phase
WAITS = {"qkv": "x_down", "o": "x_attn", "gu": "x_o", "down": "x_act"}
SENDS = {"qkv": "x_qkv", "o": "x_o", "gu": "x_act", "down": "x_down"}


class TxBar:
    """One arrival that announces `tx` transfers, and the transfers themselves."""

    def __init__(self, name):
        self.name, self.pending, self.tx, self.phase = name, 1, 0, 0

    def _check(self):
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 1, 1

    def expect(self, n):
        assert self.pending == 1, f"{self.name}: armed while phase {self.phase} is incomplete"
        self.pending, self.tx = 0, self.tx + n
        self._check()

    def land(self):
        self.tx -= 1
        self._check()

    def done(self, parity):
        return (self.phase & 1) != parity


class CountBar:
    def __init__(self):
        self.pending, self.phase = WARPS, 0

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.phase, self.pending = self.phase + 1, WARPS

    def done(self, parity):
        return (self.phase & 1) != parity


class Cta:
    def __init__(self, r):
        self.x = {n: TxBar(f"cta {r} {n}") for n in ("x_qkv", "x_attn", "x_o", "x_act", "x_down")}
        self.full, self.empty = [TxBar(f"cta {r} full{i}") for i in range(STAGES)], [CountBar() for _ in range(STAGES)]
        self.meta, self.meta_empty = [TxBar(f"cta {r} meta{i}") for i in range(2)], [CountBar() for _ in range(2)]
        self.poisoned, self.sync = False, [0, 0, False, False]  # sync: generation, arrived, any, answer
        self.lost = 1 << 30  # the barrier generation in which a warp's wait failed first: what follows a later barrier lacks its input


def run(seed, fault, mended):
    rnd = random.Random(seed)
    ctas, flying, errors, gone = [Cta(r) for r in range(CTAS)], [], [], []
    victim, at, waits = rnd.randrange(CTAS), rnd.randrange(12, 160), [0]
    transfers = [0]

    def transfer(to, bar):
        transfers[0] += 1
        if not (fault == "transfer" and transfers[0] == 3 * at):
            flying.append((to, bar))

    def wait(c, r, bar, parity):
        waits[0] += r == victim
        limit = rnd.randrange(2, 6) if fault == "wait" and r == victim and waits[0] >= at else 3000
        while not bar.done(parity):
            limit -= 1
            if limit < 0 or c.poisoned:
                c.poisoned = True
                return False
            yield
        return True

    def sync(c, bad=False):
        gen = c.sync[0]
        c.sync[1], c.sync[2] = c.sync[1] + 1, c.sync[2] or bad
        if c.sync[1] == WARPS:
            c.sync[:] = [gen + 1, 0, False, c.sync[2]]
        while c.sync[0] == gen:
            yield
        return c.sync[3]

    def producer(c, r):
        s, lap, norms = 0, 0, [0, 0]
        for layer in range(LAYERS):
            ms = layer & 1
            if layer >= 2:
                yield from wait(c, r, c.meta_empty[ms], ((layer >> 1) - 1) & 1)
            if not c.poisoned:
                c.meta[ms].expect(1)
                norms[ms] += 1
                transfer(r, c.meta[ms])
                for ph in PHASES:
                    for _ in range(COUNT[ph]):
                        if lap > 0:
                            yield from wait(c, r, c.empty[s], (lap - 1) & 1)
                        if c.poisoned:
                            break
                        c.full[s].expect(1)
                        transfer(r, c.full[s])
                        s, lap = (0, lap + 1) if s + 1 == STAGES else (s + 1, lap)
                        yield
        if mended and c.poisoned:  # its own copies land, within a limit
            armed = [(c.full[i], lap + (i < s)) for i in range(STAGES)] + list(zip(c.meta, norms))
            for bar, n in armed:
                limit = 3000
                while n > 0 and not bar.done((n - 1) & 1) and limit > 0:
                    limit -= 1
                    yield

    def consumer(c, r, w):
        s, lap, ok = 0, 0, True
        every = {"x_qkv": CTAS, "x_attn": CTAS, "x_o": CTAS, "x_act": CTAS, "x_down": CTAS}

        def awaited(name, parity):
            nonlocal ok
            here = yield from wait(c, r, c.x[name], parity)
            ok = ok and here
            c.lost = min(c.lost, c.sync[0] if not here else c.lost)
            if w == 0 and (here or not mended):
                c.x[name].expect(every[name])

        def send(name):
            if c.lost < c.sync[0]:
                errors.append(f"cta {r} sends {name} without its input")
            for to in range(w, CTAS, WARPS):
                transfer(to, ctas[to].x[name])

        if w == 0:
            for name in every:
                c.x[name].expect(every[name])
        yield from sync(c)
        for layer in range(LAYERS + 1):
            ms = layer & 1
            if layer < LAYERS:
                here = yield from wait(c, r, c.meta[ms], (layer >> 1) & 1)
                ok = ok and here
                c.lost = min(c.lost, c.sync[0] if not here else c.lost)
            for ph in PHASES:
                if layer or ph != "qkv":
                    yield from awaited(WAITS[ph], (layer - 1 if ph == "qkv" else layer) & 1)
                yield from sync(c)
                if layer == LAYERS:
                    return
                for _ in range(COUNT[ph]):
                    here = yield from wait(c, r, c.full[s], lap & 1)
                    ok = ok and here
                    c.lost = min(c.lost, c.sync[0] if not here else c.lost)
                    if mended and not here:
                        break
                    yield
                    c.empty[s].arrive()
                    s, lap = (0, lap + 1) if s + 1 == STAGES else (s + 1, lap)
                if ph == "down":
                    c.meta_empty[ms].arrive()
                if (yield from sync(c, not ok)) and mended:
                    return
                send(SENDS[ph])
                if ph == "qkv":
                    yield from awaited("x_qkv", layer & 1)
                    if (yield from sync(c, not ok)) and mended:
                        return
                    if c.lost < c.sync[0]:
                        errors.append(f"cta {r} writes its cache without its input")
                    yield from sync(c)
                    send("x_attn")

    live = {}
    for r, c in enumerate(ctas):
        live[r, "p"] = producer(c, r)
        live.update({(r, w): consumer(c, r, w) for w in range(WARPS)})
    for _ in range(400_000):
        if not live or errors:
            break
        if flying and rnd.random() < 0.5:
            to, bar = flying.pop(rnd.randrange(len(flying)))
            bar.land()
            continue
        k = rnd.choice(list(live))
        try:
            next(live[k])
        except StopIteration:
            del live[k]
        except AssertionError as e:
            errors.append(str(e))
    if live and not errors:
        errors.append(f"no progress: {sorted(map(str, live))}")
    if not errors:  # behind the cluster's last barrier: a CTA that has given up waits for what lands, the others leave at once
        gone = [to for to, _ in flying if not (mended and ctas[to].poisoned)]
        if gone:
            errors.append(f"transfers on their way into CTAs {sorted(set(gone))} that have left")
    return errors, any(c.poisoned for c in ctas)


def test_without_a_fault():
    for seed in range(8):
        assert run(seed, None, True) == ([], False), seed


@pytest.mark.parametrize("fault", ["wait", "transfer"])
def test_a_wait_that_runs_out_ends_the_cluster(fault):
    reached = 0
    for seed in range(30):
        errors, poisoned = run(seed, fault, True)
        assert not errors, (seed, errors[:2])
        reached += poisoned
    assert reached > 10
    assert any(run(seed, fault, False)[0] for seed in range(30))  # carrying on as if the data had arrived breaks the rules above
