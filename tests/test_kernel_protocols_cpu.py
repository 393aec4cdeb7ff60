"""Host model of the barrier protocols of the warp-specialised kernels.

The attention kernels (csrc/attention.cu: ``attn_fwd2_kernel``, ``attn_bwd_dq2_kernel``, ``attn_bwd_dkv2_kernel``, the
same for both head widths) and the persistent GEMMs (csrc/gemm_umma.cu: ``umma_gemm_kernel``, ``umma_gemm_pair_kernel``)
are warp-specialised: a TMA producer, a single-thread MMA issuer and softmax / epilogue warps hand shared-memory stages
and tensor-memory regions to one another through mbarriers that are waited on by phase parity; the GEMM's epilogue hands
staging buffers to TMA stores through bulk groups, and the dK/dV kernel's clusters meet at cluster barriers.  The selective
scan's kernels (csrc/scan.cu) are pairs of warps, one that prepares and finishes chunks and one that carries the
recurrence, which meet at named barriers without a time limit.  This file
restates each role's sequence of waits, arrivals, loads, MMAs and stores, runs the roles under randomly chosen
interleavings (loads, MMAs and stores complete asynchronously, MMAs of a CTA in issue order) and checks for every step
count that

* nothing deadlocks (a parity wait that can never be satisfied would show up as one), and
* every read sees the data it is meant to see: each write tags its buffer with (what, step), each read asserts
  the tag - an MMA that overwrites S before the threads have read it, a load that lands in a stage an MMA still
  needs, or a barrier phase completed by arrivals that belong to two different steps, fails the assertion.

It is a model of the protocol, not of the arithmetic; the kernels themselves are tested on the GPU against fp32
PyTorch (tests/test_gpu_ops.py, tests/test_gpu_gemm.py).
"""
import random

import pytest

WARPS = range(8)      # softmax warps: warp w owns the 32 rows of quarter w % 4 in column half w // 4


class Bar:
    def __init__(self, count):
        self.count, self.pending, self.phase = count, count, 0

    def arrive(self):
        self.pending -= 1
        assert self.pending >= 0, "more arrivals than the barrier expects in one phase"
        if self.pending == 0:
            self.pending, self.phase = self.count, self.phase + 1

    def passed(self, parity):          # mbarrier.try_wait.parity: true once the phase with this parity completed
        return (self.phase & 1) != parity


class Machine:
    """Roles are generators that yield ('wait', bar, parity), ('until', condition) or None (a scheduling point).
    ``pipes`` are the in-order tensor pipes (one per CTA, or per pair), ``loads`` the TMA requests in flight, ``stores``
    the TMA stores of each thread that have not read their buffer yet, oldest first."""

    def __init__(self, seed, pipes=1):
        self.rng = random.Random(seed)
        self.mem = {}
        self.pipes, self.loads, self.stores = [[] for _ in range(pipes)], [], {}

    def write(self, buf, tag):
        self.mem[buf] = tag

    def read(self, buf, tag):
        assert self.mem.get(buf) == tag, f"{buf}: expected {tag}, found {self.mem.get(buf)}"

    def mma(self, reads, writes, pipe=0):
        self.pipes[pipe].append(("mma", reads, writes))

    def commit(self, *bars, pipe=0):
        for b in bars:
            self.pipes[pipe].append(("commit", b))

    def load(self, buf, tag, bar):
        self.loads.append((buf, tag, bar))

    def store(self, thread, buf, tag):
        self.stores.setdefault(thread, []).append((buf, tag))

    def stores_read(self, thread, but):        # cp.async.bulk.wait_group.read `but`
        return ("until", lambda: len(self.stores.get(thread, ())) <= but)

    def run(self, roles):
        roles = [[r, None] for r in roles]
        for r in roles:
            r[1] = next(r[0], "done")
        # uneven speeds: every other seed makes some roles, the tensor pipe or the loads very slow or very fast,
        # so that one warp can run a whole step ahead of another
        skew = self.rng.random() < 0.5
        speed = lambda: self.rng.choice([0.02, 0.2, 1.0, 1.0, 5.0, 50.0]) if skew else 1.0
        w_role = [speed() for _ in roles]
        w_pipe, w_load, w_store = [speed() for _ in self.pipes], speed(), speed()
        steps = 0
        while True:
            steps += 1
            assert steps < 200000, "model did not terminate"
            choices, weights = [], []
            for i, (gen, st) in enumerate(roles):
                if st == "done":
                    continue
                if st is None or (st[0] == "wait" and st[1].passed(st[2])) or (st[0] == "until" and st[1]()):
                    choices.append(("role", i))
                    weights.append(w_role[i])
            for i, pipe in enumerate(self.pipes):
                if pipe:
                    choices.append(("pipe", i))
                    weights.append(w_pipe[i])
            for t, q in self.stores.items():
                if q:
                    choices.append(("store", t))
                    weights.append(w_store)
            for i in range(len(self.loads)):
                choices.append(("load", i))
                weights.append(w_load)
            if not choices:
                assert all(st == "done" for _, st in roles), \
                    "deadlock: " + str([st for _, st in roles if st != "done"][0][2:])
                return
            kind, i = self.rng.choices(choices, weights)[0]
            if kind == "role":
                roles[i][1] = next(roles[i][0], "done")
            elif kind == "pipe":
                item = self.pipes[i].pop(0)
                if item[0] == "mma":
                    for buf, tag in item[1]:
                        self.read(buf, tag)
                    for buf, tag in item[2]:
                        self.write(buf, tag)
                else:
                    item[1].arrive()
            elif kind == "store":
                self.read(*self.stores[i].pop(0))
            else:
                buf, tag, bar = self.loads.pop(i)
                self.write(buf, tag)
                bar.arrive()


def run_dq2(nblk, seed, ds_barriers=2):
    """TMEM: S | dP x 2 | dQ.  K: 3 stages (held until the step's dQ MMAs), V: 2 stages.  ``ds_barriers`` is the
    number of barriers on which the threads announce dS: the kernel has one per dP buffer."""
    m = Machine(seed)
    qdo = Bar(1)
    k_full, k_empty = [Bar(1) for _ in range(3)], [Bar(1) for _ in range(3)]
    v_full, v_empty = [Bar(1) for _ in range(2)], [Bar(1) for _ in range(2)]
    s_full, s_free, dq_full = Bar(1), Bar(8), Bar(1)
    dp_full = [Bar(1), Bar(1)]
    ds_full = [Bar(8) for _ in range(ds_barriers)]
    NB = ds_barriers

    def producer():
        m.load("QdO", ("QdO", 0), qdo)
        for j in range(nblk):
            ks, st = j % 3, j & 1
            yield ("wait", k_empty[ks], ((j // 3) & 1) ^ 1)
            m.load(("K", ks), ("K", j), k_full[ks])
            yield ("wait", v_empty[st], ((j >> 1) & 1) ^ 1)
            m.load(("V", st), ("V", j), v_full[st])

    def issuer():
        yield ("wait", qdo, 0)
        yield ("wait", k_full[0], 0)
        m.mma([("QdO", ("QdO", 0)), (("K", 0), ("K", 0))], [("S", ("S", 0))])
        m.commit(s_full)
        yield ("wait", v_full[0], 0)
        m.mma([("QdO", ("QdO", 0)), (("V", 0), ("V", 0))], [(("dP", 0, w), ("dP", 0)) for w in WARPS])
        m.commit(dp_full[0], v_empty[0])
        for j in range(nblk):
            st, nx, ks, kn = j & 1, (j & 1) ^ 1, j % 3, (j + 1) % 3
            if j + 1 < nblk:
                yield ("wait", k_full[kn], ((j + 1) // 3) & 1)
                yield ("wait", v_full[nx], ((j + 1) >> 1) & 1)
                yield ("wait", s_free, j & 1)
                m.mma([(("K", kn), ("K", j + 1))], [("S", ("S", j + 1))])
                m.commit(s_full)
                m.mma([(("V", nx), ("V", j + 1))], [(("dP", nx, w), ("dP", j + 1)) for w in WARPS])
                m.commit(dp_full[nx], v_empty[nx])
            yield ("wait", ds_full[j % NB], (j // NB) & 1)
            m.mma([(("dP", st, w), ("dS", j)) for w in WARPS] + [(("K", ks), ("K", j))], [("dQ", ("dQ", j))])
            m.commit(k_empty[ks])
        m.commit(dq_full)

    def softmax(h):                                   # warp h owns its rows and column half of every accumulator
        for j in range(nblk):
            yield ("wait", s_full, j & 1)
            m.read("S", ("S", j))
            s_free.arrive()
            yield None
            yield ("wait", dp_full[j & 1], (j >> 1) & 1)
            m.read(("dP", j & 1, h), ("dP", j))
            yield None
            m.write(("dP", j & 1, h), ("dS", j))
            ds_full[j % NB].arrive()
        yield ("wait", dq_full, 0)
        m.read("dQ", ("dQ", nblk - 1))

    m.run([producer(), issuer()] + [softmax(w) for w in WARPS])


def run_dkv2(niter, seed, q_stages=3, split=1):
    """TMEM: S^T | dP^T | dV | dK (single buffers).  Q with its ndelta: ``q_stages`` stages, held until the dK MMAs; dO with
    its nlse: 2, released by the dV MMAs.  A stage's two loads (tile and statistics) credit one barrier.  ``split`` CTAs of
    a cluster share the key block: each lays its sums over its own tiles, all meet, each reads its rows of everybody's, and
    nobody leaves before all have read."""
    m = Machine(seed, pipes=split)
    NQ = q_stages
    meet, leave = Bar(10 * split), Bar(10 * split)      # cluster barriers: eight softmax warps, producer, issuer
    roles = []

    def finish(c, part):
        if split == 1:
            return
        meet.arrive()
        yield ("wait", meet, 0)
        for p in range(split):                         # warps 8 and 9 take their share of the rows as well
            for w in WARPS:
                m.read(("part", p, w), ("part", p))
        yield None
        leave.arrive()
        yield ("wait", leave, 0)
        if part is not None:
            m.write(("part", c, part), "gone")

    def cta(c):
        kv = Bar(2)
        q_full, q_empty = [Bar(2) for _ in range(NQ)], [Bar(1) for _ in range(NQ)]
        do_full, do_empty = [Bar(2), Bar(2)], [Bar(1), Bar(1)]
        st_full, dpt_full, p_full, ds_full, acc_full = Bar(1), Bar(1), Bar(8), Bar(8), Bar(1)
        mma = lambda reads, writes: m.mma([((c, b), t) for b, t in reads], [((c, b), t) for b, t in writes], pipe=c)
        commit = lambda bar: m.commit(bar, pipe=c)
        read = lambda b, t: m.read((c, b), t)
        write = lambda b, t: m.write((c, b), t)

        def load_q(it):
            m.load((c, ("Q", it % NQ)), ("Q", it), q_full[it % NQ])
            m.load((c, ("ndelta", it % NQ)), ("ndelta", it), q_full[it % NQ])

        def load_do(it):
            m.load((c, ("dO", it & 1)), ("dO", it), do_full[it & 1])
            m.load((c, ("nlse", it & 1)), ("nlse", it), do_full[it & 1])

        def producer():
            m.load((c, "K"), "K", kv)
            load_q(0)
            m.load((c, "V"), "V", kv)
            load_do(0)
            for it in range(1, niter):
                yield ("wait", q_empty[it % NQ], ((it // NQ) & 1) ^ 1)
                load_q(it)
                yield ("wait", do_empty[it & 1], ((it >> 1) & 1) ^ 1)
                load_do(it)
            yield from finish(c, None)

        def issuer():
            yield ("wait", kv, 0)
            yield ("wait", q_full[0], 0)
            mma([("K", "K"), (("Q", 0), ("Q", 0))], [(("ST", w), ("ST", 0)) for w in WARPS])
            commit(st_full)
            yield ("wait", do_full[0], 0)
            mma([("V", "V"), (("dO", 0), ("dO", 0))], [(("DPT", w), ("DPT", 0)) for w in WARPS])
            commit(dpt_full)
            for it in range(niter):
                qs, qn, os_, on = it % NQ, (it + 1) % NQ, it & 1, (it & 1) ^ 1
                yield ("wait", p_full, it & 1)
                mma([(("ST", w), ("PT", it)) for w in WARPS] + [(("dO", os_), ("dO", it))], [("dV", ("dV", it))])
                commit(do_empty[os_])
                if it + 1 < niter:
                    yield ("wait", q_full[qn], ((it + 1) // NQ) & 1)
                    mma([("K", "K"), (("Q", qn), ("Q", it + 1))], [(("ST", w), ("ST", it + 1)) for w in WARPS])
                    commit(st_full)
                yield ("wait", ds_full, it & 1)
                mma([(("DPT", w), ("dST", it)) for w in WARPS] + [(("Q", qs), ("Q", it))], [("dK", ("dK", it))])
                commit(q_empty[qs])
                if it + 1 < niter:
                    yield ("wait", do_full[on], ((it + 1) >> 1) & 1)
                    mma([("V", "V"), (("dO", on), ("dO", it + 1))], [(("DPT", w), ("DPT", it + 1)) for w in WARPS])
                    commit(dpt_full)
            commit(acc_full)
            yield from finish(c, None)

        def softmax(h):                               # warp h owns its rows and column half of S^T and dP^T
            for it in range(niter):
                qs, os_ = it % NQ, it & 1
                yield ("wait", do_full[os_], (it >> 1) & 1)
                yield ("wait", st_full, it & 1)
                read(("ST", h), ("ST", it))
                read(("nlse", os_), ("nlse", it))
                yield None
                write(("ST", h), ("PT", it))
                p_full.arrive()
                yield ("wait", q_full[qs], (it // NQ) & 1)
                yield ("wait", dpt_full, it & 1)
                read(("DPT", h), ("DPT", it))
                read(("ndelta", qs), ("ndelta", it))
                yield None
                write(("DPT", h), ("dST", it))
                ds_full.arrive()
            yield ("wait", acc_full, 0)
            read("dV", ("dV", niter - 1))
            read("dK", ("dK", niter - 1))
            if split > 1:                              # the sums go over the tiles: no load may land there any more
                assert not [b for b, _, _ in m.loads if b[0] == c]
                m.write(("part", c, h), ("part", c))
            yield from finish(c, h)

        roles.extend([producer(), issuer()] + [softmax(w) for w in WARPS])

    for c in range(split):
        cta(c)
    m.run(roles)


def run_fwd2(nb, seed):
    """Forward, two 128-query tiles per CTA (``attn_fwd2_kernel``).  TMEM: S_0 | S_1 | O_0 | O_1; K and V: 2 stages
    shared by the tiles.  ``nb[t]`` = key blocks tile t visits (tile 0 may visit fewer).  Warps 4t..4t+3 own tile t."""
    m = Machine(seed)
    nblk = max(nb)
    q_full = Bar(1)
    k_full, k_empty, v_full, v_empty = ([Bar(1), Bar(1)] for _ in range(4))
    s_full, pv_done = [Bar(1), Bar(1)], [Bar(1), Bar(1)]
    p_full = [Bar(4), Bar(4)]
    tile_warps = lambda t: range(4 * t, 4 * t + 4)

    def producer():
        m.load("Q", ("Q", 0), q_full)
        for j in range(nblk):
            st, par = j & 1, ((j >> 1) & 1) ^ 1
            yield ("wait", k_empty[st], par)
            m.load(("K", st), ("K", j), k_full[st])
            yield ("wait", v_empty[st], par)
            m.load(("V", st), ("V", j), v_full[st])

    def issue_s(t, j):
        m.mma([("Q", ("Q", 0)), (("K", j & 1), ("K", j))], [(("S", w), ("S", j)) for w in tile_warps(t)])
        m.commit(s_full[t])

    def issuer():
        yield ("wait", q_full, 0)
        yield ("wait", k_full[0], 0)
        for t in range(2):
            if nb[t] > 0:
                issue_s(t, 0)
        m.commit(k_empty[0])
        for j in range(nblk):
            st = j & 1
            yield ("wait", v_full[st], (j >> 1) & 1)
            if j + 1 < nblk:
                yield ("wait", k_full[(j + 1) & 1], ((j + 1) >> 1) & 1)
            for t in range(2):
                if j >= nb[t]:
                    continue
                yield ("wait", p_full[t], j & 1)
                # O_t += P_t V_j: reads the rows the threads rescaled for this step, leaves O(j)
                reads = [(("S", w), ("P", j)) for w in tile_warps(t)] + [(("V", st), ("V", j))]
                reads += [(("O", w), ("O scaled", j)) for w in tile_warps(t)] if j > 0 else []
                m.mma(reads, [(("O", w), ("O", j)) for w in tile_warps(t)])
                m.commit(pv_done[t])
                if j + 1 < nb[t]:
                    issue_s(t, j + 1)
            if j + 1 < nblk:
                m.commit(k_empty[(j + 1) & 1])
            m.commit(v_empty[st])

    def softmax(w):
        t = w // 4
        for j in range(nb[t]):
            yield ("wait", s_full[t], j & 1)
            m.read(("S", w), ("S", j))
            yield None
            if j > 0:                              # rescale of O: PV(j - 1) must be complete, PV(j) not issued
                m.read(("O", w), ("O", j - 1))
                m.write(("O", w), ("O scaled", j))
                yield None
            m.write(("S", w), ("P", j))
            p_full[t].arrive()
        if nb[t] > 0:
            yield ("wait", pv_done[t], (nb[t] - 1) & 1)
            m.read(("O", w), ("O", nb[t] - 1))

    m.run([producer(), issuer()] + [softmax(w) for w in WARPS])


# ---------------------------------------------------------------- persistent GEMMs (csrc/gemm_umma.cu)
def run_gemm(k_blocks, stages, seed, ctas=1, warps=4, slabs=None, in_flight=None):
    """``umma_gemm_kernel`` (ctas=1) and ``umma_gemm_pair_kernel`` (ctas=2) for the tiles one CTA (pair) works
    through: ``k_blocks[i]`` reduction blocks for tile i (0 = a group without rows in a batched product: the
    epilogue writes zeros / the addend and the issuer arrives by itself).  Ring of ``stages`` shared-memory
    stages, two accumulators.  Of eight epilogue ``warps`` of a CTA (pairs only) two share 32 rows, each with every other
    column slab and one staging buffer; one of four has all slabs of its rows and two buffers in turn.  A warp takes its
    share of the accumulator in ``slabs`` column slabs, hands it back with the last one in registers, and sends each slab
    from a staging buffer by a TMA store that it does not wait for: before it writes the next slab, all but ``in_flight``
    (one less than its buffers) of its stores have been read.  In the pair the ``full`` and ``tmem_empty`` barriers live
    in the leader, ``empty`` and ``tmem_full`` exist in both CTAs and get the leader's commits."""
    m = Machine(seed)
    C = range(ctas)
    W, buffers = range(warps), 8 // warps
    slabs = 16 // warps if slabs is None else slabs
    in_flight = buffers - 1 if in_flight is None else in_flight
    full = [Bar(1 + ctas) for _ in range(stages)]         # the leader's expect_tx + one load group per CTA
    empty = [[Bar(1) for _ in range(stages)] for _ in C]
    tmem_full = [[Bar(1), Bar(1)] for _ in C]
    tmem_empty = [Bar(len(W) * ctas), Bar(len(W) * ctas)]

    def producer(c):
        s, ph, n = 0, 0, 0
        for i, kb_n in enumerate(k_blocks):
            for kb in range(kb_n):
                yield ("wait", empty[c][s], ph ^ 1)
                if c == 0:
                    full[s].arrive()                      # arrive.expect_tx
                m.load(("stage", c, s), ("AB", n), full[s])
                n += 1
                s += 1
                if s == stages:
                    s, ph = 0, ph ^ 1

    def issuer():
        s, ph, n = 0, 0, 0
        for i, kb_n in enumerate(k_blocks):
            acc, acc_ph = i & 1, (i >> 1) & 1
            yield ("wait", tmem_empty[acc], acc_ph ^ 1)
            for kb in range(kb_n):
                yield ("wait", full[s], ph)
                reads = [(("stage", c, s), ("AB", n)) for c in C]
                if kb > 0:
                    reads += [(("acc", c, acc, w), ("acc", i, kb - 1)) for c in C for w in W]
                m.mma(reads, [(("acc", c, acc, w), ("acc", i, kb)) for c in C for w in W])
                m.commit(*[empty[c][s] for c in C])
                n += 1
                s += 1
                if s == stages:
                    s, ph = 0, ph ^ 1
            if kb_n > 0:
                m.commit(*[tmem_full[c][acc] for c in C])
            else:
                for c in C:
                    tmem_full[c][acc].arrive()

    def epilogue(c, w):
        me, n = (c, w), 0
        for i, kb_n in enumerate(k_blocks):
            acc, acc_ph = i & 1, (i >> 1) & 1
            yield ("wait", tmem_full[c][acc], acc_ph)
            for sl in range(slabs):
                if kb_n > 0:
                    m.read(("acc", c, acc, w), ("acc", i, kb_n - 1))
                if sl == slabs - 1:
                    tmem_empty[acc].arrive()
                yield m.stores_read(me, in_flight)
                m.write(("stage out", me, n % buffers), ("out", i, sl))
                yield None
                m.store(me, ("stage out", me, n % buffers), ("out", i, sl))
                n += 1
        yield m.stores_read(me, 0)

    m.run([producer(c) for c in C] + [issuer()] + [epilogue(c, w) for c in C for w in W])


def run_register_split(tiles, seed, hand_back=False):
    """``umma_gemm_pair_kernel`` with eight epilogue warps: registers per thread move between the warps of a CTA through a pool
    (setmaxnreg), from 168 for all to 72 for the four load and MMA warps and 216 for the eight epilogue warps.  ``inc`` waits, without a limit, until
    the pool holds what it takes.  ``hand_back``: everybody takes 168 again at the end, which the kernel must not do."""
    m = Machine(seed)
    pool, done = [0], Bar(12)
    dec = lambda n: pool.__setitem__(0, pool[0] + n)

    def inc(n):
        yield ("until", lambda: pool[0] >= n, "registers")
        pool[0] -= n

    def role():
        dec(168 - 72)
        for _ in range(tiles):
            yield None
        if hand_back:
            yield from inc(168 - 72)
        done.arrive()
        yield ("wait", done, 0)

    def epilogue():
        yield None
        yield from inc(216 - 168)
        for _ in range(tiles):
            yield None
        if hand_back:
            dec(216 - 168)
        done.arrive()
        yield ("wait", done, 0)

    m.run([role() for _ in range(4)] + [epilogue() for _ in range(8)])


@pytest.mark.parametrize("tiles", [0, 1, 5])
def test_registers_reach_the_epilogue(tiles):
    for seed in range(100):
        run_register_split(tiles, seed)


@pytest.mark.parametrize("tiles", [0, 1])
def test_registers_handed_back_without_order_can_block(tiles):
    """A CTA with little to do: the load and MMA warps take back what the epilogue warps have not got yet."""
    with pytest.raises(AssertionError, match="deadlock"):
        for seed in range(200):
            run_register_split(tiles, seed, hand_back=True)


# ---------------------------------------------------------------- selective scan (csrc/scan.cu)
class NamedBar:
    """bar.sync / bar.arrive of two warps: a phase ends when both have come."""

    def __init__(self):
        self.here, self.phase = set(), 0

    def arrive(self, warp):
        assert warp not in self.here, "a warp arrives twice in one phase"
        self.here.add(warp)
        if len(self.here) == 2:
            self.here, self.phase = set(), self.phase + 1

    def sync(self, warp):
        p = self.phase
        self.arrive(warp)
        return ("until", lambda: self.phase > p, "named barrier")


class Copies:
    """cp.async groups of the helper warp: stage(j) brings chunk j and, in the backward pass, its checkpoint."""

    def __init__(self, m, ntiles, ck_buffers=0):
        self.m, self.ntiles, self.ck_buffers, self.groups = m, ntiles, ck_buffers, []

    def stage(self, j):
        done = Bar(2 if self.ck_buffers else 1)
        if j < self.ntiles:
            self.m.load(("raw", j & 1), ("raw", j), done)
            if self.ck_buffers:
                self.m.load(("ck", j % self.ck_buffers), ("ck", j), done)
        else:
            done.phase = 1                       # an empty group
        self.groups.append(done)

    def wait_but_one(self):
        older = self.groups[:-1]
        return ("until", lambda: all(g.phase >= 1 for g in older), "copies")


def run_scan_fwd(ntiles, seed):
    """``scan_fwd_kernel``, pass with outputs: both warps meet after every chunk."""
    m = Machine(seed)
    step, copies = NamedBar(), Copies(m, ntiles)

    def prepare(j):
        m.read(("raw", j & 1), ("raw", j))
        m.write(("prep", j & 1), ("prep", j))

    def helper():
        copies.stage(0)
        copies.stage(1)
        yield copies.wait_but_one()
        if ntiles > 0:
            prepare(0)
        yield step.sync("helper")
        for j in range(ntiles):
            if j > 0:
                m.read(("part", (j - 1) & 1), ("part", j - 1))
            yield None
            copies.stage(j + 2)
            yield copies.wait_but_one()
            if j + 1 < ntiles:
                prepare(j + 1)
            yield step.sync("helper")
        m.read(("part", (ntiles - 1) & 1), ("part", ntiles - 1))

    def recurrence():
        yield step.sync("recurrence")
        for j in range(ntiles):
            m.read(("prep", j & 1), ("prep", j))
            yield None
            m.read(("prep", j & 1), ("prep", j))
            m.write(("part", j & 1), ("part", j))
            yield step.sync("recurrence")

    m.run([helper(), recurrence()])


def run_scan_carry(ntiles, seed, empty=True):
    """``scan_bwd_carry_kernel``: the helper is up to two chunks ahead.  ``empty=False`` leaves its wait for a free buffer out."""
    m = Machine(seed)
    ready, free, copies = [NamedBar(), NamedBar()], [NamedBar(), NamedBar()], Copies(m, ntiles)

    def prepare(j):
        m.read(("raw", j & 1), ("raw", j))
        m.write(("prep", j & 1), ("prep", j))

    def helper():
        copies.stage(0)
        copies.stage(1)
        yield copies.wait_but_one()
        prepare(0)
        ready[0].arrive("helper")
        for j in range(ntiles - 1):
            copies.stage(j + 2)
            yield copies.wait_but_one()
            if j > 0 and empty:
                yield free[(j + 1) & 1].sync("helper")
            prepare(j + 1)
            ready[(j + 1) & 1].arrive("helper")

    def recurrence():
        for j in range(ntiles):
            yield ready[j & 1].sync("recurrence")
            m.read(("prep", j & 1), ("prep", j))
            yield None
            m.read(("prep", j & 1), ("prep", j))
            if j + 2 < ntiles and empty:
                free[j & 1].arrive("recurrence")

    m.run([helper(), recurrence()])


def run_scan_bwd(ntiles, seed, ck_buffers=3, empty=True):
    """``scan_bwd_kernel``: chunks in halves, the later one first; results of half h lie in buffer h."""
    m = Machine(seed)
    ready, full, free = ([NamedBar(), NamedBar()] for _ in range(3))
    copies = Copies(m, ntiles, ck_buffers)

    def prepare(j):
        m.read(("raw", j & 1), ("raw", j))
        m.write(("prep", j & 1), ("prep", j))

    def finish(j, half):
        m.read(("sums", half), ("sums", j))

    def helper():
        copies.stage(0)
        copies.stage(1)
        yield copies.wait_but_one()
        if ntiles > 0:
            prepare(0)
        ready[0].arrive("helper")
        for j in range(ntiles):
            if j > 0:
                yield full[0].sync("helper")
                finish(j - 1, 0)
                yield None
                finish(j - 1, 0)
                if empty:
                    free[0].arrive("helper")
            copies.stage(j + 2)
            yield copies.wait_but_one()
            if j + 1 < ntiles:
                prepare(j + 1)
                ready[(j + 1) & 1].arrive("helper")
            yield full[1].sync("helper")
            finish(j, 1)
            yield None
            finish(j, 1)
            if j + 1 < ntiles and empty:
                free[1].arrive("helper")
        yield full[0].sync("helper")
        finish(ntiles - 1, 0)

    def recurrence():
        for j in range(ntiles):
            yield ready[j & 1].sync("recurrence")
            for half in (1, 0):
                m.read(("ck", j % ck_buffers), ("ck", j))
                m.read(("prep", j & 1), ("prep", j))
                yield None
                if j > 0 and empty:
                    yield free[half].sync("recurrence")
                m.read(("prep", j & 1), ("prep", j))
                m.write(("sums", half), ("sums", j))
                full[half].arrive("recurrence")

    m.run([helper(), recurrence()])


@pytest.mark.parametrize("ntiles", list(range(1, 9)) + [33])
@pytest.mark.parametrize("kernel", [run_scan_fwd, run_scan_carry, run_scan_bwd])
def test_scan_warps_hand_chunks_over(kernel, ntiles):
    for seed in range(30):
        kernel(ntiles, seed)


@pytest.mark.parametrize("kernel", [run_scan_fwd, run_scan_bwd])
def test_the_scan_needs_a_chunk(kernel):
    """Without one the helper finishes what was never begun (forward) or waits for it (backward): the host does not launch."""
    with pytest.raises(AssertionError):
        kernel(0, 0)


@pytest.mark.parametrize("run", [lambda s: run_scan_bwd(5, s, ck_buffers=2), lambda s: run_scan_bwd(5, s, empty=False),
                                 lambda s: run_scan_carry(5, s, empty=False)])
def test_the_model_notices_a_missing_scan_buffer_or_wait(run):
    with pytest.raises(AssertionError):
        for seed in range(200):
            run(seed)


@pytest.mark.parametrize("nblk", list(range(1, 10)) + [16])
def test_dq_kernel_protocol_has_no_deadlock_and_no_stale_read(nblk):
    for seed in range(40):
        run_dq2(nblk, seed)


@pytest.mark.parametrize("niter", list(range(1, 10)) + [16, 64])
def test_dkv_kernel_protocol_has_no_deadlock_and_no_stale_read(niter):
    for seed in range(40):
        run_dkv2(niter, seed)


@pytest.mark.parametrize("split", [2, 4])
@pytest.mark.parametrize("niter", [1, 2, 3, 4, 7])
def test_dkv_clusters_meet_and_leave(niter, split):
    for seed in range(12):
        run_dkv2(niter, seed, split=split)


@pytest.mark.parametrize("nb1", list(range(1, 10)) + [17])
def test_forward_kernel_protocol_has_no_deadlock_and_no_stale_read(nb1):
    for nb0 in sorted({max(nb1 - 1, 0), nb1}):     # tile 0 ends one key block earlier, or the sequence end cuts both
        for seed in range(25):
            run_fwd2((nb0, nb1), seed)
    for seed in range(25):                         # the sequence ends inside tile 0: tile 1 has no rows
        run_fwd2((nb1, 0), seed)


@pytest.mark.parametrize("ctas,warps", [(1, 4), (2, 4), (2, 8)])
@pytest.mark.parametrize("stages", [2, 4, 6])
def test_gemm_ring_and_accumulator_hand_off(ctas, warps, stages):
    rng = random.Random(stages * 10 + ctas)
    shapes = [[1], [3], [1, 1, 1, 1, 1], [2, 0, 5, 0, 0, 1], [0], [0, 0, 0], [32, 2, 32], [7] * 9]
    shapes += [[rng.choice([0, 1, 2, 3, 9]) for _ in range(rng.randint(1, 8))] for _ in range(6)]
    for kbs in shapes:
        for seed in range(12):
            run_gemm(kbs, stages, seed, ctas=ctas, warps=warps)


def test_one_ds_barrier_for_two_dp_buffers_would_mix_phases():
    """Why the dQ kernel has a dS barrier per dP buffer: dS(j + 1) depends only on the threads having read S(j), so
    a fast warpgroup can announce dS(j + 1) before a slow one has announced dS(j).  On a single barrier the two
    arrivals complete one phase and the dQ MMAs would read a half of dS(j) that is not written yet."""
    with pytest.raises(AssertionError):
        for seed in range(200):
            run_dq2(4, seed, ds_barriers=1)


def test_the_model_notices_a_missing_stage():
    """Sanity of the model itself: one Q stage cannot hold the next step's tile for S^T while this step's is still needed
    for dK, so nothing can proceed."""
    with pytest.raises(AssertionError):
        for seed in range(200):
            run_dkv2(6, seed, q_stages=1)


@pytest.mark.parametrize("ctas,warps", [(1, 4), (2, 4), (2, 8)])
def test_the_model_notices_a_reused_staging_buffer(ctas, warps):
    """With one more store in flight it would be reading what the next slab overwrites."""
    with pytest.raises(AssertionError):
        for seed in range(50):
            run_gemm([2, 2, 2], 4, seed, ctas=ctas, warps=warps, in_flight=8 // warps)
