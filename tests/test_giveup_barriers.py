"""What a CTA does after one of its bounded waits gave up, on a model of its named barriers (no GPU).

Named barriers have no time limit.  An arrival made before the partner has reached its previous call completes the wrong phase, and
`bar.sync` then waits for ever.  The kernels whose roles meet in named barriers therefore keep to two rules: MMA issuers issue and commit
in every trip, whether or not a wait for a load gave up, and waits for those commits do not end early.  The rules are looked for
in the source, together with the list of barrier calls that the model restates; the model runs every warp as a coroutine in random order
while loads stop landing at a random tile."""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "triton_diff_attn_b200", "csrc")
COMMITTED = "s_full|pv_done|o_full|mma_done|acc_full"        # mbarriers that an issuer's commit completes


class _Cta:
    """Warps are generators that yield ("sync" | "arrive", barrier, threads) or ("load" | "commit", predicate): a wait for something
    that may never come, and a wait for an issuer's commit.  `gated`: waits for commits do not give up, as in the kernels."""

    def __init__(self, rng, items, gated=True):
        self.rng, self.items, self.gated, self.aborted, self.arrived = rng, items, gated, False, {}
        self.total = sum(items)
        self.limit = rng.choice((self.total, rng.randrange(self.total + 1)))      # tiles whose loads land

    def tiles(self):
        """(item, index in it, tiles of it, tile number)"""
        n = 0
        for it, count in enumerate(self.items):
            for i in range(count):
                yield it, i, count, n
                n += 1

    def stuck(self):
        """Warps that never end."""
        warps = self.warps()
        state = {name: ("start",) for name in warps}
        while state:
            ready = [n for n, s in state.items() if s[0] in ("start", "go") or (s[0] in ("load", "commit") and s[1]())]
            late = [n for n, s in state.items() if s[0] in (("load",) if self.gated else ("load", "commit")) and not s[1]()]
            value = True
            if late and (not ready or (self.aborted and self.rng.random() < 0.1)):
                name, value, self.aborted = self.rng.choice(late), False, True
            elif ready:
                name = self.rng.choice(ready)
            else:
                return sorted(state)
            try:
                op = warps[name].send(None if state[name] == ("start",) else value)
            except StopIteration:
                del state[name]
                continue
            if op[0] in ("load", "commit"):
                state[name] = op
                continue
            state[name] = ("bar", op[1]) if op[0] == "sync" else ("go",)
            count = self.arrived.get(op[1], 0) + 32
            if count == op[2]:
                state = {n: ("go",) if s == ("bar", op[1]) else s for n, s in state.items()}
            self.arrived[op[1]] = count % op[2]
        return []


class _Fwd64(_Cta):
    """A tile of 128 keys is two sub-tiles per branch."""
    source = ("fwd64.cuh", "diffattn_fwd64_kernel", "else if (warp == WARP_MMA)", [
        "sync NB_KV", "sync NB_O", "sync NB_P + br * 2 + u", "sync NB_KV", "sync NB_STORE + br", "sync NB_M + br * 2 + (u ^ 1)",
        "arrive NB_M + br * 2 + u", "arrive NB_P + br * 2 + u", "sync NB_ALL", "arrive NB_O", "sync NB_ALL", "arrive NB_STORE + br"])

    def warps(self):
        self.s, self.pv, self.o, self.k_next = set(), set(), set(), 0
        w = {"mma": self.mma(), "watch": self.watch(), "store": self.store()}
        w.update({f"softmax{i}": self.softmax(i >> 3, (i >> 2) & 1) for i in range(16)})
        return w

    def mma(self):
        ok = True
        for it, j, count, n in self.tiles():
            if j == 0:
                ok = ok and (yield "load", lambda: n < self.limit)
                self.s |= {(br, 2 * n + u) for br in (0, 1) for u in (0, 1)}
            yield "sync", "KV", 64
            if j == 0 and it > 0:
                yield "sync", "O", 544
            for u in (0, 1):
                for br in (0, 1):
                    yield "sync", ("P", br, u), 160
                    self.pv.add((br, 2 * n + u))
                    if j + 1 < count:
                        self.s.add((br, 2 * n + u + 2))
            if j + 1 == count:
                self.o.add(it)

    def watch(self):
        ok = True
        for it, j, count, n in self.tiles():
            ok = ok and (yield "load", lambda: n < self.limit)
            if j + 1 < count:
                ok = ok and (yield "load", lambda: n + 1 < self.limit)
            yield "sync", "KV", 64

    def store(self):
        for _ in self.items:
            for br in (0, 1):
                yield "sync", ("STORE", br), 288

    def softmax(self, br, u):
        for it, j, count, n in self.tiles():
            t = 2 * n + u
            yield "commit", lambda: (br, t) in self.s
            if j > 0 or u > 0:
                yield "sync", ("M", br, u ^ 1), 256
            if j + 1 < count or u == 0:
                yield "arrive", ("M", br, u), 256
            if (j > 0 or u > 0) and self.rng.random() < 0.3:           # the running maximum was raised
                yield "commit", lambda: (br, t - 1) in self.pv
            yield "arrive", ("P", br, u), 160
            if j + 1 == count:
                yield "commit", lambda: it in self.o
                yield "sync", "ALL", 512
                if it + 1 < len(self.items):
                    yield "arrive", "O", 544
                yield "sync", "ALL", 512
                yield "arrive", ("STORE", br), 288


class _Fwd128(_Cta):
    source = ("fwd128.cuh", "diffattn_fwd128_branch_kernel", "else if (warp == WARP_S)", [
        "sync NB_SF + u", "sync NB_P + u", "sync NB_START", "arrive NB_SF + u", "sync NB_M + (u ^ 1)", "arrive NB_M + u", "arrive NB_START",
        "arrive NB_P + u", "sync 1", "sync NB_OUT + u", "sync 1"])

    def warps(self):
        self.nsub, self.s, self.pv, self.o = 2 * self.items[0], set(), set(), False
        w = {"s": self.issue_s(), "pv": self.issue_pv()}
        w.update({f"softmax{i}": self.softmax(i >> 2) for i in range(8)})
        return w

    def issue_s(self):
        ok = True
        for t in range(self.nsub):
            ok = ok and (yield "load", lambda: t < 2 * self.limit)
            if t >= 2:
                yield "sync", ("SF", t & 1), 160
            self.s.add(t)

    def issue_pv(self):
        ok, limit = True, self.rng.randrange(self.nsub + 1)
        for t in range(self.nsub):
            ok = ok and (yield "load", lambda: t < limit)
            yield "sync", ("P", t & 1), 160
            self.pv.add(t)
        self.o = True

    def softmax(self, u):
        nsub = self.nsub
        if u == 1:
            yield "sync", "START", 256
        for t in range(u, nsub, 2):
            yield "commit", lambda: t in self.s
            if t + 2 < nsub:
                yield "arrive", ("SF", u), 160
            if t > 0:
                yield "sync", ("M", u ^ 1), 256
            if t + 1 < nsub:
                yield "arrive", ("M", u), 256
            if t > 0 and self.rng.random() < 0.3:
                yield "commit", lambda: t - 1 in self.pv
            if t == 0:
                yield "arrive", "START", 256
            if t >= 2:
                yield "commit", lambda: t - 2 in self.pv
            yield "arrive", ("P", u), 160
        yield "commit", lambda: self.o
        yield "sync", "ALL", 256
        yield "sync", ("OUT", u), 128


class _DkDv64(_Cta):
    source = ("bwd.cuh", "diffattn_bwd_dkdv64_kernel", "else if (warp == WARP_MMA || warp == WARP_MMA + 1)", [
        "sync NB_STORE", "sync NB_SFREE", "sync NB_SFREE", "sync NB_ACC", "sync NB_E + (i & 1)", "arrive NB_SFREE", "arrive NB_E + (i & 1)",
        "arrive NB_ACC", "arrive NB_STORE"])

    def __init__(self, rng, items, gated=True):
        super().__init__(rng, [2 * count for count in items], gated)         # 64 query rows: an even number of tiles

    def warps(self):
        self.loaded, self.s, self.done, self.acc = set(), (set(), set()), set(), set()
        w = {"tma": self.tma(), "s": self.scores(0), "dp": self.scores(1), "out": self.outputs()}
        w.update({f"wg{i}": self.elementwise() for i in range(16)})
        return w

    def tma(self):
        ok = True
        for it, i, count, n in self.tiles():
            if it > 0 and i == 0:
                ok = ok and (yield "load", lambda: all(n - 1 in s for s in self.s)) and not self.aborted
            if it > 0 and i == 1:
                yield "sync", "STORE", 544
            ok = ok and (yield "load", lambda: n < 3 or n - 3 in self.done) and not self.aborted
            if ok and n < self.limit:
                self.loaded.add(n)
        yield "sync", "STORE", 544

    def scores(self, which):
        ok = True
        for it, i, count, n in self.tiles():
            ok = ok and (yield "load", lambda: n in self.loaded)
            if n > 0:
                yield "sync", "SFREE", 576
            self.s[which].add(n)
        yield "sync", "SFREE", 576

    def outputs(self):
        for it, i, count, n in self.tiles():
            if it > 0 and i == 0:
                yield "sync", "ACC", 544
            yield "sync", ("E", i & 1), 544
            self.done.add(n)
            if i + 1 == count:
                self.acc.add(it)

    def elementwise(self):
        for it, i, count, n in self.tiles():
            yield "commit", lambda: all(n in s for s in self.s)
            yield "arrive", "SFREE", 576
            if i > 0:
                yield "commit", lambda: n - 1 in self.done
            yield "arrive", ("E", i & 1), 544
            if i + 1 == count:
                yield "commit", lambda: it in self.acc
                if it + 1 < len(self.items):
                    yield "arrive", "ACC", 544
                yield "arrive", "STORE", 544


class _Dq64(_Cta):
    source = ("bwd.cuh", "diffattn_bwd_dq64_kernel", "else if (warp == WARP_MMA)", [
        "sync NB_ACC", "sync NB_DP", "sync NB_DS1", "sync NB_DS2", "sync NB_START", "arrive NB_DP", "arrive NB_START", "arrive NB_DS1",
        "arrive NB_DS2", "arrive NB_ACC"])

    def warps(self):
        self.s, self.acc = (set(), set()), set()
        w = {"mma": self.mma()}
        w.update({f"wg{i}": self.elementwise(i >> 2) for i in range(16)})
        return w

    def mma(self):
        ok = True
        for it, j, count, n in self.tiles():
            if j == 0:
                ok = ok and (yield "load", lambda: n < self.limit)
                self.s[0].add(n)
                self.s[1].add(n)
            more = j + 1 < count
            if more:
                ok = ok and (yield "load", lambda: n + 1 < self.limit)
            if j == 0 and it > 0:
                yield "sync", "ACC", 544
            yield "sync", "DP", 544
            for br in (0, 1):
                yield "sync", ("DS", br), 544
                if more:
                    self.s[br].add(n + 1)
            if not more:
                self.acc.add(it)

    def elementwise(self, g):
        if g >= 2:
            yield "sync", "START", 512
        for it, j, count, n in self.tiles():
            yield "commit", lambda: n in self.s[0]
            yield "arrive", "DP", 544
            if n == 0 and g < 2:
                yield "arrive", "START", 512
            yield "arrive", ("DS", 0), 544
            yield "commit", lambda: n in self.s[1]
            yield "arrive", ("DS", 1), 544
            if j + 1 == count:
                yield "commit", lambda: it in self.acc
                if it + 1 < len(self.items):
                    yield "arrive", "ACC", 544


KERNELS = [_Fwd64, _Fwd128, _DkDv64, _Dq64]


def _draws(kernel, gated):
    for seed in range(200):
        rng = random.Random(seed)
        yield seed, kernel(rng, [rng.randint(1, 4) for _ in range(rng.randint(1, 3))], gated)


@pytest.mark.parametrize("kernel", KERNELS)
def test_source_keeps_the_rules(kernel):
    name, function, issuers, calls = kernel.source
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    text = text[text.index(function + "("):]
    text = text[:text.index("__syncthreads();\n  if (warp ==", text.index("__syncthreads();") + 1)]
    found = [" ".join(m) for m in re.findall(r"named_bar_(sync|arrive)\(([^,;]+),", text)]
    assert found == calls                                        # (the model below restates these)
    assert not re.findall(r"mbar_wait(?:_warp)?\(&misc->(?:%s)\b" % COMMITTED, text)
    text = text[text.index(issuers):]
    assert not re.findall(r"\bok\b[^;{\n]*elect_one\(\)", text) and "break;" not in text


@pytest.mark.parametrize("kernel", KERNELS)
def test_every_warp_ends(kernel):
    gave_up = 0
    for seed, cta in _draws(kernel, gated=True):
        assert not cta.stuck(), seed
        gave_up += cta.aborted
    assert 20 < gave_up < 200


@pytest.mark.parametrize("kernel", KERNELS)
def test_model_sees_waits_that_end_early(kernel):
    assert any(cta.stuck() for _, cta in _draws(kernel, gated=False))
