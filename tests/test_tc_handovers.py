"""Hand-overs of the tensor-core kernels, checked on the CPU from their source (a missing wait or fence rarely shows in an output)."""
import pathlib
import random
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "lfm2-ampere_b200" / "csrc"

# a wait, the fence that orders tcgen05 operations behind it, and the operations themselves
TOKEN = re.compile(r"(?P<open>\{)|(?P<close>\})|(?P<wait>\btc_wait(?:<\w+>)?\()|(?P<fence>\btc_fence_after\()"
                   r"|(?P<op>\btc_(?:ld\d*(?:<[^>]*>)?|st8|mma_\w+)\()")


def unfenced(text):
    """Lines of tcgen05 operations that some path reaches from a barrier wait without tcgen05.fence::after_thread_sync between
    the two.  A fence inside a block counts for that block alone: the block may be skipped."""
    text = re.sub(r"//[^\n]*", "", text)
    bad, due, blocks, before = [], False, [], False
    for t in TOKEN.finditer(text):
        if t["open"]:                                    # (state on entry, state at the end of the branches before this one)
            blocks.append((due, before))
            before = False
        elif t["close"]:
            entry, earlier = blocks.pop()
            if text[t.end():t.end() + 8].lstrip().startswith("else"):
                before, due = earlier or due, entry
            else:
                due = due or entry or earlier
        elif t["wait"]:
            due = True
        elif t["fence"]:
            due = False
        elif due:
            bad.append(text.count("\n", 0, t.start()) + 1)
    return bad


def test_checker_sees_a_fence_that_may_be_skipped():
    assert unfenced("f() { tc_wait(b); if (grown) { tc_fence_after(); tc_ld8(o); } tc_st8(p); }") == [1]
    assert unfenced("f() { tc_wait(b); tc_fence_after(); if (grown) { tc_ld8(o); } tc_st8(p); }") == []
    assert unfenced("f() { if (producer) { tc_wait(b); } else { tc_ld8(o); } tc_st8(p); }") == [1]


@pytest.mark.parametrize("name", ["lkb_pfattn.cu", "lkb_gemm_tc.cu"])
def test_every_tmem_access_is_fenced_behind_its_wait(name):
    assert unfenced((CSRC / name).read_text()) == []


# ---- the GEMM's rings: the roles of one block as generators over barriers with phases, run in random order ------------------
GEMM = (CSRC / "lkb_gemm_tc.cu").read_text()


def _const(name):
    return int(re.search(rf"#define {name}\s+(\d+)", GEMM).group(1))


NS, AU, SC_RING, WS_RING, AHEAD = (_const(n) for n in ("TC_NS", "TC_AUNITS", "TC_SC_RING", "TC_WS_RING", "TC_SC_AHEAD"))
ISSUERS = GEMM[GEMM.index("// ============================ MMA issuers"):GEMM.index("// ============================ expansion")]


class Barrier:
    """An mbarrier.  What an arriving thread knows (releases) goes to whoever waits for that phase; the arrival of a
    tcgen05.commit tells that the MMAs are done and nothing about other threads' writes."""
    def __init__(self, count):
        self.count, self.left, self.phase, self.gathered, self.known = count, count, 0, {}, {}

    def arrive(self, knows):
        for k, v in knows.items():
            self.gathered[k] = max(v, self.gathered.get(k, -1))
        self.left -= 1
        assert self.left >= 0, "more arrivals than the phase takes"
        if self.left == 0:
            self.left, self.phase, self.known, self.gathered = self.count, self.phase + 1, self.gathered, {}

    def done(self, parity):
        return (self.phase & 1) != parity


def _run_roles(rng, stages, free, tells, wcopy):
    full, empty = [Barrier(1) for _ in range(NS)], [Barrier(2) for _ in range(NS)]
    afull, aempty = [Barrier(1) for _ in range(AU)], [Barrier(2) for _ in range(AU)]
    tfull = [[Barrier(1 + tells) for _ in range(2)] for _ in range(2)]         # [column half (free form)][buffer]
    tempty = [[Barrier(1 if free else 2) for _ in range(2)] for _ in range(2)]
    raw, dk, wsc = {}, {}, {}
    read = {0: -1, 1: -1, "expansion": -1}                                     # the last stage a reader has finished

    def wait(b, parity, knows):
        while not b.done(parity):
            yield
        for k, v in b.known.items():
            knows[k] = max(v, knows.get(k, -1))

    def producer():
        knows = {}
        for it in range(stages):
            yield from wait(empty[it % NS], ((it // NS) & 1) ^ 1, knows)
            assert read["expansion"] >= it - NS, "nibbles overwritten before they were read"
            raw[it % NS] = it
            if wcopy:
                put_scales(it)
            full[it % NS].arrive({"raw": it, "wsc": it} if wcopy else {"raw": it})

    def put_scales(it):                                                        # of two stages
        if it % 2 == 0 and it < stages:
            assert min(read[0], read[1]) >= it - WS_RING + 1, "weight scales overwritten before they were read"
            wsc[it // 2 % (WS_RING // 2)] = it

    def expansion():
        knows = {}
        for it in range(AHEAD if not wcopy else 0):
            put_scales(it)
        for it in range(stages):
            yield from wait(full[it % NS], (it // NS) & 1, knows)
            assert raw[it % NS] == it and knows["raw"] >= it
            assert min(read[0], read[1]) >= it - SC_RING, "constants overwritten before they were read"
            dk[it % SC_RING] = it
            yield
            yield from wait(aempty[it % AU], ((it // AU) & 1) ^ 1, knows)
            read["expansion"] = it
            afull[it % AU].arrive({**knows, "dk": it} if wcopy else {**knows, "dk": it, "wsc": it})
            if not wcopy:
                put_scales(it + AHEAD)

    def issuer(q):
        knows = {}
        for it in range(stages):
            yield from wait(full[it % NS], (it // NS) & 1, knows)
            yield from wait(afull[it % AU], (it // AU) & 1, knows)
            for i in range(4 if free else 2):
                h = i & 1 if free else q
                yield from wait(tempty[q if free else 0][h], i >> 1 if free else i, knows)
                if tells:
                    tfull[q if free else 0][h].arrive(knows)                   # the thread itself
                    yield
                tfull[q if free else 0][h].arrive({})                          # a commit
                yield
            aempty[it % AU].arrive({})
            empty[it % NS].arrive({})

    def epilogue(half):
        knows, own = {}, half if free else 0
        for b in tempty[own]:
            b.arrive({})
        for it in range(stages):
            for j in range(4):
                yield from wait(tfull[own][j & 1], j >> 1, knows)
                if j == 0:
                    assert wsc[it // 2 % (WS_RING // 2)] == it // 2 * 2 and knows.get("wsc", -1) >= it // 2 * 2, "weight scales not acquired"
                assert dk[it % SC_RING] == it and knows.get("dk", -1) >= it, "constants not acquired"
                yield
                if j == 3:
                    read[half] = it
                tempty[own][j & 1].arrive(knows)
    roles = [producer(), expansion(), issuer(0), issuer(1), epilogue(0), epilogue(1)]
    weight = [rng.random() ** 3 + 0.01 for _ in roles]                         # every run has slow and fast roles
    idle, before = 0, None
    while roles:
        i = rng.choices(range(len(roles)), weight)[0]
        try:
            next(roles[i])
        except StopIteration:
            del roles[i], weight[i]
        now = [b.phase for b in full + afull + tfull[0] + tfull[1]]
        idle, before = (0 if now != before else idle + 1), now
        assert idle < 20000, "the roles wait for one another"


@pytest.mark.parametrize("wcopy", [True, False], ids=["tensor-copy", "cp-async"])
@pytest.mark.parametrize("free", [False, True], ids=["plain", "swiglu"])
def test_epilogue_acquires_what_it_reads(free, wcopy):
    """Weight scales (written by a tensor copy or the expansion warps) and constants (by the expansion warps) reach the epilogue by releases and
    acquires of threads, a commit not counted, and no ring is overwritten early."""
    for seed in range(40):
        _run_roles(random.Random(seed), stages=60, free=free, tells="tc_mbar_arrive(&tfull[" in ISSUERS, wcopy=wcopy)
