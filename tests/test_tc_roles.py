"""A CPU model of what the roles of ``k_conv3d_tc`` (pybella_gb300/csrc/bella_cnn.cu) hand to each other
since its input planes come by bulk copies and a warp for each row block issues the MMAs, run under random
interleavings; ``test_tc_protocol.py`` models the same rings with one issuer.

* A producer warp waits until the MMAs of both issuers on the slot's previous plane are complete,
  zeroes its share of the slot's rows outside the plane when a run of another row block first takes
  the slot, and arrives at the slot's ``full`` barrier with the bytes of its copies, which land
  later and in any order; planes outside the grid have no copies.
* An issuer waits for ``full``, takes the accumulators of the outputs that it starts, issues, and commits to
  the plane's completion barrier, of which each issuer is one arrival; its MMAs read the slot
  until they complete, in order for each issuer, the two issuers' apart.
* The epilogue warps of a row block read an output once both issuers' MMAs on its last input plane are
  complete, and the accumulators are free when all of them have.

Checked: no deadlock, no parity alias, the slot holds the plane and the run's zeros from the first to
the last of its MMAs, accumulators are read complete and taken again only after their readers, no
copy is in flight at the end.
"""
import random

import pytest

from test_tc_protocol import D, LIVE, R, S, Bar, _const, _runs, tc_blocks, tc_win

NPROD, NMB = _const("TC_PROD_WARPS"), _const("TC_MB")
NEPI = 4 * NMB


class FullBar(Bar):
    """An mbarrier whose phase also waits for the bytes announced with its arrivals."""

    def __init__(self, count, name):
        super().__init__(count, name)
        self.bytes = 0

    def _end(self):
        if self.pending == 0 and self.bytes == 0:
            self.done += 1
            self.pending = self.count

    def arrive_expect(self, nbytes):
        self.pending -= 1
        assert self.pending >= 0, self.name
        self.bytes += nbytes
        self._end()

    def land(self, nbytes):
        self.bytes -= nbytes
        assert self.bytes >= 0, self.name
        self._end()


def _simulate(nx, xseg, work, cta, nblk, seed):
    rng = random.Random(seed)
    runs = _runs(cta, work, nx, nblk)
    full = [FullBar(NPROD, "full%d" % k) for k in range(S)]
    done = [Bar(NMB, "done%d" % k) for k in range(D)]
    free = [Bar(NEPI, "free%d" % k) for k in range(LIVE)]
    data = {}                                       # (slot, producer): plane, once its copies have landed
    zeros = {(k, w): 0 for k in range(S) for w in range(NPROD)}      # run whose padding rows are zero there
    copies, flight = [], [[] for _ in range(NMB)]   # (slot, producer, plane, pieces left); issued MMAs
    contrib = [{} for _ in range(NMB)]
    owner = [{} for _ in range(NMB)]

    def producer(w):
        i = 0
        for r, (_, ia, ib) in enumerate(runs):
            first = i
            for p in range(ia - 1, ib + 1):
                slot, prev = i % S, i - S
                if prev >= 0:
                    while not done[prev % D].ready(prev // D):
                        yield
                if first > 0 and i - first < S:
                    zeros[(slot, w)] = r
                if 0 <= p < nx and rng.random() < 0.9:       # a warp may have no piece of a short plane
                    n = rng.randint(1, 3)
                    data.pop((slot, w), None)
                    full[slot].arrive_expect(n)
                    copies.append([slot, w, i, n])
                else:
                    data[(slot, w)] = i
                    full[slot].arrive_expect(0)
                i += 1
                yield
        for k in range(max(0, i - S), i):                    # no copy outlives the block
            while not full[k % S].ready(k // S):
                yield

    def mma(mb):
        i = obase = acq = 0
        for r, (_, ia, ib) in enumerate(runs):
            for p in range(ia - 1, ib + 1):
                slot = i % S
                while not full[slot].ready(i // S):
                    yield
                reads = False
                if 0 <= p < nx:
                    s0 = (p // xseg) * xseg
                    qlo, qhi = max(p - 1, ia, s0), min(p + 1, ib - 1, s0 + xseg - 1)
                    if qlo <= qhi:
                        olo, ohi = obase + qlo - ia, obase + qhi - ia
                        while acq <= ohi:
                            if acq >= LIVE:
                                while not free[acq % LIVE].ready(acq // LIVE - 1):
                                    yield
                            acq += 1
                        w = obase + p + 1 - ia
                        assert tc_win(w) + (w - olo) <= R - 1
                        for o in range(olo, ohi + 1):
                            if o not in contrib[mb]:
                                for b in tc_blocks(o):
                                    q = owner[mb].get(b)
                                    assert q is None or contrib[mb][q] == "read", "accumulators taken too early"
                                    owner[mb][b] = o
                                contrib[mb][o] = 0
                            assert owner[mb][tc_win(w) + (w - o)] == o
                        reads = (olo, ohi)
                flight[mb].append((i, r, reads))
                i += 1
                yield
            obase += ib - ia

    def check_slot(i, r):
        assert all(data.get((i % S, w)) == i for w in range(NPROD)), "the slot holds another plane"
        assert all(zeros[(i % S, w)] == r for w in range(NPROD)), "the slot holds another run's padding"

    def epilogue(mb):
        o = ibase = 0
        for (_, ia, ib) in runs:
            for q in range(ia, ib):
                j = ibase + (q - ia + 2)
                while not done[j % D].ready(j // D):
                    yield
                want = sum(1 for pp in (q - 1, q, q + 1) if 0 <= pp < nx and pp // xseg == q // xseg)
                assert contrib[mb][o] in (want, "read"), ("incomplete output", q)
                yield
                readers[mb][o] = readers[mb].get(o, 0) + 1
                if readers[mb][o] == NEPI // NMB:
                    contrib[mb][o] = "read"
                free[o % LIVE].arrive()
                o += 1
            ibase += ib - ia + 2

    readers = [{} for _ in range(NMB)]
    started = [False] * NMB

    def asynchronous():
        while True:
            if copies and rng.random() < 0.6:
                c = rng.choice(copies)                       # in any order
                c[3] -= 1
                if c[3] == 0:
                    copies.remove(c)
                    data[(c[0], c[1])] = c[2]
                full[c[0]].land(1)
            for mb in range(NMB):
                if flight[mb]:
                    i, r, reads = flight[mb][0]
                    if reads and not started[mb]:
                        check_slot(i, r)                     # the first of its MMAs
                        started[mb] = True
                    elif rng.random() < 0.5:
                        flight[mb].pop(0)
                        started[mb] = False
                        if reads:
                            check_slot(i, r)                 # the last
                            for o in range(reads[0], reads[1] + 1):
                                contrib[mb][o] += 1
                        done[i % D].arrive()
            yield

    roles = ("none", "producer", "mma0", "mma1", "epilogue", "async")
    slow = roles[seed % len(roles)]
    weight = {r: 0.05 if r == slow else 1.0 for r in roles}
    actors = [("producer", producer(w)) for w in range(NPROD)] + [("mma%d" % m, mma(m)) for m in range(NMB)] + \
             [("epilogue", epilogue(w // 4)) for w in range(NEPI)]
    bg = ("async", asynchronous())
    steps = 0
    while actors:
        steps += 1
        assert steps < 5_000_000, "deadlock"
        pool = actors + [bg]
        role, a = rng.choices(pool, weights=[weight[r] for r, _ in pool])[0]
        try:
            next(a)
        except StopIteration:
            actors.remove((role, a))
    assert not copies


@pytest.mark.parametrize("nx,xseg,nblk,grid", [(129, 129, 35, 152), (40, 8, 3, 7), (24, 12, 2, 3), (9, 9, 1, 1),
                                               (12, 12, 9, 152), (25, 5, 3, 4), (1, 1, 40, 4), (2, 2, 30, 3)])
def test_roles(nx, xseg, nblk, grid):
    items = nblk * nx
    grid = min(grid, items)
    work = -(-items // grid)
    for cta in (range(grid) if grid <= 8 else (0, 1, grid // 2, grid - 1)):
        if cta * work >= items:
            continue
        for seed in range(6):
            _simulate(nx, xseg, work, cta, nblk, seed)
