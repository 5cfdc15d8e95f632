"""Host model of the hand-over between sweeps of the bulge chase (csrc/band_eig.cu).

Sweeps run in CTAs, K of them a cluster; a sweep's results travel in slots, one a task: into the next
CTA's ring of five by a bulk copy that an mbarrier counts, the beta of task s + 2 apart, with credits
coming back; between clusters through global memory behind a flag. The model runs the kernel's roles as
coroutines in random order on real numbers, with copies that land any time after they are issued, and
checks on the CPU what the kernel relies on:
* no slot is overwritten before it is read, nothing deadlocks, and d, e are those of the chase run
  sweep after sweep, for rings, phases, credits, betas, sweeps of one task, and sweeps with one task
  fewer than the one before;
* when waits run out and CTAs leave early, no copy lands in a CTA that has left.
"""
import random

import numpy as np
import pytest

RING = 5


def _ntask(n, b, j):
    return (n - 2 - j) // b + 1


def _house(x):
    sig = float(x[1:] @ x[1:])
    if sig == 0.0:
        return 0.0, x[0], 0.0
    beta = -np.copysign(np.sqrt(x[0] * x[0] + sig), x[0])
    return (beta - x[0]) / beta, beta, 1.0 / (x[0] - beta)


class Bar:
    """mbarrier of one arrival a phase with a transaction count."""

    def __init__(self):
        self.phase, self.pending, self.tx = 0, 1, 0

    def _step(self):
        assert self.pending >= 0, "more arrivals than the phase expects"
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 1, 1

    def arrive(self, tx=0):
        self.tx += tx
        self.pending -= 1
        self._step()

    def complete(self):
        self.tx -= 1
        self._step()

    def test(self, parity):
        return (self.phase & 1) != (parity & 1)


class Slot:
    def __init__(self, b):
        self.d, self.o, self.beta = np.zeros((b, b)), np.zeros((b, b)), 0.0


class Cta:
    def __init__(self, b, first):
        self.raw = [Slot(b) for _ in range(RING)]
        self.stage = [Slot(b) for _ in range(RING)]
        self.xin, self.xout = np.zeros(b), np.zeros(b)
        self.full, self.own, self.credit = ([Bar() for _ in range(RING)] for _ in range(3))
        self.fullx = Bar()
        self.abort = self.left = False
        self.tasks = self.refl = 0
        self.blocks = self.betas = self.firsts = self.sent = self.sentx = 0
        self.expected = 1
        self.at = 0  # CTA-wide barriers passed
        if not first:
            for f in self.full:
                f.arrive(2)
            self.fullx.arrive(1)


class Model:
    def __init__(self, M, b, K, clusters, seed, give_up=0.0, drain=True):
        self.speed = (0.002, 0.05, 0.7)[seed % 3]  # of the copies
        self.n, self.b, self.K, self.rng = M.shape[0], b, K, random.Random(seed)
        n = self.n
        self.give_up, self.drain, self.err, self.late = give_up, drain, False, 0
        self.d, self.e = np.zeros(n), np.zeros(n)
        A = np.zeros((n + 3 * b, n + 3 * b))
        A[:n, :n] = np.tril(M) + np.tril(M, -1).T
        nt = _ntask(n, b, 0)
        self.gx, self.G = A[1:1 + b, 0].copy(), [Slot(b) for _ in range(nt)]
        for s, g in enumerate(self.G):
            r = 1 + s * b
            g.d[:], g.o[:] = A[r:r + b, r:r + b], A[r + b:r + 2 * b, r:r + b]
            g.beta, g.o[b - 1, b - 1] = g.o[b - 1, b - 1], 0.0
        self.d[0] = A[0, 0]
        self.progress = [0] * n
        self.cta = [Cta(b, g % K == 0) for g in range(K * clusters)]
        self.flying = []  # (destination CTA or None, what to do when it lands)
        self.tasks = [self._main(g) for g in range(K * clusters)]

    # ---- coroutines: each yields a condition to wait for
    def _wait(self, c, ready):
        """A bounded wait: ends when ready, when this CTA has given up, or by giving up itself."""
        def over():
            if c.abort or ready():
                return True
            r = self.rng.random()
            if r < self.give_up:
                self.err = c.abort = True
            elif self.err and r < 0.2:
                c.abort = True
            return c.abort
        yield over

    def _fly(self, dst, land):
        self.flying.append((dst, land))

    def _block(self, c, nx, m):
        u = m % RING

        def land():
            nx.raw[u].d[:] = c.stage[u].d
            o, corner = nx.raw[u].o, nx.raw[u].o[-1, -1]
            o[:] = c.stage[u].o
            o[-1, -1] = corner
            nx.full[u].complete()
        self._fly(nx, land)

    def _beta(self, nx, m, v):
        u = m % RING

        def land():
            nx.raw[u].beta = v
            nx.full[u].complete()
        self._fly(nx, land)

    def _first(self, c, nx, last):
        x = np.append(c.xout[:-1], last)

        def land():
            nx.xin[:] = x
            nx.fullx.complete()
        self._fly(nx, land)
        c.firsts += 1

    def _copy_out(self, c, j, s, out0):
        if s < 0:
            self.gx[:] = c.xout
        else:
            u = (out0 + s) % RING
            g, st = self.G[s], c.stage[u]
            g.d[:], g.o[:], g.beta = st.d, st.o, st.beta
            c.credit[u].arrive()
        self.progress[j] = s + 2

    def _give_back(self, c, pv, m):
        c.full[m % RING].arrive(2)
        pv.credit[m % RING].arrive()

    def _load(self, c, j, nt, in0):
        for s in range(-1, nt):
            if j > 0:
                yield from self._wait(c, lambda: self.progress[j - 1] >= s + 2)
            if s < 0:
                c.xin[:] = self.gx
                c.fullx.arrive()
                continue
            m = in0 + s
            u = m % RING
            yield from self._wait(c, lambda: c.own[u].test(((m // RING) & 1) ^ 1))
            if not c.abort:
                c.full[u].arrive(1)
                g = self.G[s]

                def land(u=u, g=g):
                    c.raw[u].d[:], c.raw[u].o[:], c.raw[u].beta = g.d, g.o, g.beta
                    c.full[u].complete()
                self._fly(c, land)
                c.sent = m + 1

    def _credits(self, c, pv, nt, in0):
        for s in range(-1, nt - 1):
            yield lambda: c.tasks >= s + 2 or c.abort
            if c.abort:
                return
            if s < 0:
                c.fullx.arrive(1)
                c.expected += 1
            else:
                self._give_back(c, pv, in0 + s)

    def _send(self, c, nx, j, nt, out0):
        for s in range(0 if nx else -1, nt - 2):
            yield lambda: (c.tasks if nx else c.refl) >= s + 3 or c.abort
            if c.abort:
                return
            if nx:
                self._block(c, nx, out0 + s)
                c.blocks = out0 + s + 1
            else:
                self._copy_out(c, j, s, out0)
            yield lambda: True

    def _scalars(self, c, sh, nx, far, first, nt, in0, out0, j):
        for s in range(nt):
            yield lambda: sh["x"] > s
            c.tasks = s + 1
            tau, beta, sc = _house(sh["col"])
            sh["scal"] = (tau, beta, sc)
            sh["y"] = s + 1
            yield lambda: True
            so2 = out0 + s - 2
            if nx and not c.abort:
                if s == 1:
                    self._first(c, nx, beta)
                if s >= 2:
                    self._beta(nx, so2, beta)
                    c.betas = so2 + 1
            yield lambda: True
            if far:
                if s == 1:
                    c.xout[-1] = beta
                if s >= 2:
                    c.stage[so2 % RING].beta = beta
                c.refl = s + 1
            if first and s > 0 and not c.abort:
                c.own[(in0 + s - 1) % RING].arrive()
            if s == 0:
                self.e[j] = beta
            sh["p1"] = s + 1

    def _blocks(self, c, sh, send, nt, in0, out0, j, sweeps):
        n, b = self.n, self.b
        yield from self._wait(c, lambda: c.fullx.test(sweeps & 1))
        col, bulge = c.xin.copy(), None
        for s in range(nt):
            sh["col"], sh["x"] = col, s + 1  # the barrier: everybody is done with the task before
            m, o = in0 + s, out0 + s
            raw = c.raw[m % RING]
            st, st1 = c.stage[o % RING], c.stage[(o - 1) % RING]
            end, snd = s + 1 == nt, send and not c.abort
            yield from self._wait(c, lambda: c.full[m % RING].test((m // RING) & 1))
            D, O = raw.d.copy(), raw.o.copy()
            O[-1, -1] = raw.beta
            if snd:
                yield from self._wait(c, lambda: c.credit[o % RING].test(((o // RING) & 1) ^ 1))
            yield lambda: sh["y"] > s
            tau, beta, sc = sh["scal"]
            v = np.append(1.0, sc * col[1:])
            O = O - tau * np.outer(O @ v, v)
            w = tau * (D @ v)
            w -= 0.5 * tau * (v @ w) * v
            D = D - np.outer(v, w) - np.outer(w, v)
            if s == 0:
                self.d[j + 1] = D[0, 0]
                if j == n - 3:
                    self.e[n - 2], self.d[n - 1] = D[1, 0], D[1, 1]
            L = bulge - tau * np.outer(v, v @ bulge) if s > 0 else None
            yield lambda: True
            if snd:
                st.d[:-1, :-1] = D[1:, 1:]
                if s == 0:
                    c.xout[:-1] = D[1:, 0]
                else:
                    st1.d[-1, -1], st1.o[:-1, -1] = D[0, 0], D[1:, 0]
                    st1.o[:-1, :-1] = L[1:, 1:]
                    st1.d[-1, :-1] = st1.d[:-1, -1] = L[0, 1:]
                if end:
                    st.d[-1, :] = st.d[:, -1] = 0.0
                    st.o[:-1, :] = 0.0
            bulge, col = O, O[:, 0].copy()
            yield lambda: sh["p1"] > s  # barrier X of the next task

    def _epilogue(self, c, nx, pv, far, first, j, nt, ntp, in0, out0):
        if nx and not c.abort:
            if nt == 1:
                self._first(c, nx, 0.0)
            for s in range(max(0, nt - 2), nt):
                self._block(c, nx, out0 + s)
                self._beta(nx, out0 + s, 0.0)
                c.blocks = c.betas = out0 + s + 1
        if far and not c.abort:
            if nt == 1:
                c.xout[-1] = 0.0
                self._copy_out(c, j, -1, out0)
            for s in range(max(0, nt - 2), nt):
                c.stage[(out0 + s) % RING].beta = 0.0
                self._copy_out(c, j, s, out0)
        if not c.abort:
            if first:
                c.own[(in0 + nt - 1) % RING].arrive()
            else:
                for s in range(nt - 1, ntp):
                    m = in0 + s
                    if s >= nt:
                        yield from self._wait(c, lambda: c.full[m % RING].test((m // RING) & 1))
                        if c.abort:
                            break
                    self._give_back(c, pv, m)

    def _main(self, g):
        n, b, K = self.n, self.b, self.K
        c, rank, base = self.cta[g], g % K, g - g % K
        first, last = rank == 0, rank == K - 1
        nx = None if last else self.cta[g + 1]
        pv = None if first else self.cta[g - 1]
        in0 = out0 = sweeps = 0
        for j in range(g, n - 2, len(self.cta)):
            nt, ntp = _ntask(n, b, j), _ntask(n, b, j - 1) if j > 0 else 0
            send = j + 1 <= n - 3
            near, far = nx if send else None, send and last
            c.refl = c.tasks = 0
            if c.abort:
                break
            sh = {"x": 0, "y": 0, "p1": 0}
            roles = [self._load(c, j, nt, in0) if first else self._credits(c, pv, nt, in0),
                     self._scalars(c, sh, near, far, first, nt, in0, out0, j),
                     self._blocks(c, sh, send, nt, in0, out0, j, sweeps)]
            if send:
                roles.append(self._send(c, near, j, nt, out0))
            done = [0]
            for r in roles:
                self._spawn(r, done)
            yield lambda: done[0] == len(roles)
            yield from self._epilogue(c, near, pv, far, first, j, nt, ntp, in0, out0)
            in0 += nt if first else ntp
            out0 += nt if send else 0
            sweeps += 1
        # leaving: what was begun is made whole and announced, and everybody waits for what comes in
        if self.drain and nx:
            for m in range(min(c.blocks, c.betas), max(c.blocks, c.betas)):
                if m >= c.blocks:
                    self._block(c, nx, m)
                else:
                    self._beta(nx, m, 0.0)
            nx.sent, nx.sentx = max(c.blocks, c.betas), c.firsts
        c.at = 1
        yield lambda: all(p.at >= 1 for p in self.cta[base:base + K])
        if self.drain:
            for m in range(max(0, c.sent - RING), c.sent):
                yield lambda: c.full[m % RING].test((m // RING) & 1)
            if c.sentx > c.expected:
                c.fullx.arrive(1)
            if c.sentx:
                yield lambda: c.fullx.test((c.sentx - 1) & 1)
        c.at = 2
        yield lambda: all(p.at >= 2 for p in self.cta[base:base + K])
        c.left = True

    # ---- scheduler
    def _spawn(self, gen, done):
        self.live.append([gen, next(gen, None), done])

    def run(self):
        self.live = []
        for t in self.tasks:
            self.live.append([t, next(t), [0]])
        idle = 0
        while self.live:
            if self.flying and self.rng.random() < self.speed:
                dst, land = self.flying.pop(self.rng.randrange(len(self.flying)))
                self.late += dst.left
                land()
                idle = 0
                continue
            t = self.rng.choice(self.live)
            if t[1] is not None and not t[1]():
                idle += 1
                assert idle < 200000 or self.flying, "deadlock"
                continue
            idle = 0
            try:
                t[1] = next(t[0])
            except StopIteration:
                t[2][0] += 1
                self.live.remove(t)
        self.late += len(self.flying)
        return self


def _band(n, b, seed):
    M = np.random.default_rng(seed).standard_normal((n, n))
    M = M + M.T
    M[np.abs(np.subtract.outer(np.arange(n), np.arange(n))) > b] = 0.0
    return M


@pytest.mark.parametrize("K,clusters", [(1, 1), (1, 3), (2, 2), (4, 1), (3, 2), (16, 1)])
@pytest.mark.parametrize("n,b", [(3, 2), (5, 4), (13, 2), (19, 3), (26, 4), (40, 32)])
def test_slots_carry_the_chase(n, b, K, clusters):
    M = _band(n, b, 10 * n + b)
    lam = np.linalg.eigvalsh(M)
    for seed in range(3):
        r = Model(M, b, K, clusters, seed).run()
        assert not r.err and r.late == 0
        T = np.diag(r.d) + np.diag(r.e[:-1], 1) + np.diag(r.e[:-1], -1)
        assert np.abs(np.linalg.eigvalsh(T) - lam).max() <= 1e-12 * np.abs(lam).max()


def _late(drain):
    """Copies that landed too late, and runs that gave up, over several sizes and speeds of the copies."""
    late = gave_up = 0
    for n, b, K, clusters, p in [(26, 3, 4, 2, 0.0005), (13, 3, 2, 1, 0.005), (16, 4, 4, 1, 0.01)]:
        for seed in range(60):
            r = Model(_band(n, b, 1), b, K, clusters, seed, give_up=p, drain=drain).run()
            late, gave_up = late + r.late, gave_up + r.err
    return late, gave_up


def test_no_copy_lands_in_a_cta_that_has_left():
    late, gave_up = _late(True)
    assert gave_up >= 100 and late == 0


def test_the_model_sees_copies_that_land_late():
    """The same runs when nobody waits for what is on its way."""
    assert _late(False)[0] > 0
