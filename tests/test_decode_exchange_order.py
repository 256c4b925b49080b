"""The exchange of the persistent decode kernel, checked on the CPU from its source (a missing order rarely shows in an output).
Words travel without a release; what keeps a reader from a word's previous content is that its making due is ordered before the
arrival that the reader waits for: due store, CTA barrier, a fence of the arriving thread (or a releasing arrival), arrival.  And a
word is made due only when a barrier is through that every reader arrived at behind its read."""
import itertools
import pathlib
import re

import pytest

SRC = (pathlib.Path(__file__).resolve().parent.parent / "lfm2-ampere_b200" / "csrc" / "lkb_fused.cu").read_text()
TOKEN = re.compile(r"(?P<release>\bgrid_arrive\()|(?P<arrive>\bgrid_arrive<!XCH>\()|(?P<one>\bgrid_arrive_one<!XCH>\()|(?P<wait>\bgrid_wait\()"
                   r"|(?P<sync>__syncthreads\(\))|(?P<fence>tid == 0\) xch_fence\(\))|\bxch_due\((?P<due>[\w.]+)"
                   r"|\bxch_put<XCH>\((?P<put>[\w.]+)|(?:\bxch_get4?<XCH>|\bxch_ld4)\((?P<get>[\w.]+)|\bfused_load_u<XCH>\(S, (?P<load>[\w.]+)")
NAMES = {"qh": "a.mxbuf", "kh": "a.mxbuf", "vh": "a.mxbuf"}


def _body():
    text = re.sub(r"//[^\n]*", "", SRC[SRC.index("for (int l = 0; l < a.n_layers; ++l) {"):])
    return _block(text, 0)[1]


def _block(text, at):
    """(offset behind the block that opens at or after `at`, its text)."""
    start, depth = text.index("{", at), 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return i + 1, text[start:i + 1]


def _without(text, head):
    at = text.index(head)
    return text[:at] + text[_block(text, at)[0]:]


def events(layers):
    """(kind, word) in program order for consecutive layers, each "moe" (the stack), "conv" or "attn"."""
    out = []
    for n, kind in enumerate(layers):
        text = _body()
        if kind == "moe":
            text = _without(text, "if constexpr (MIX) {")
        elif kind == "conv":
            text = re.sub(r"if \(is_attn\) xch_put<XCH>\([^;]*;\s*else", "", _without(text, "if (is_attn) {"))
            text = re.sub(r"if \(slice\)[^;]*;", "", text)
        else:
            text = _without(text, "if (!is_attn) {")
        for t in TOKEN.finditer(text):
            if t["sync"] or t["wait"]:
                out += [("sync", "")] + ([("wait", "")] if t["wait"] else [])
            elif t["release"]:
                out += [("sync", ""), ("fence", ""), ("arrive", "")]
            elif t["arrive"] or t["one"]:
                out += ([("sync", "")] if t["arrive"] else []) + [("arrive", "")]
            elif t["fence"]:
                out.append(("fence", ""))
            else:
                name = t["due"] or t["put"] or t["get"] or t["load"]
                name = NAMES.get(name, name)
                if kind == "moe" and name == "x_mid":
                    name = "a.x"
                if name in ("lg", "lg_old"):                            # the two sets of logit words, by the layer's parity
                    name = f"logits {(n + (name == 'lg_old')) % 2}"
                out.append(("due" if t["due"] else "put" if t["put"] else "get", name))
    return out


def _next(ev, i, kinds, word=None):
    return next((j for j in range(i + 1, len(ev)) if ev[j][0] in kinds and (word is None or ev[j][1] == word)), None)


def _chain(ev, i, end, kinds):
    """Whether events of these kinds follow one another in this order between i and end."""
    for k in kinds:
        i = _next(ev, i, (k,))
        if i is None or i >= end:
            return False
    return True


def faults(ev):
    bad = []
    for i, (kind, word) in enumerate(ev):
        if kind == "due":
            put = _next(ev, i, ("put",), word)
            if put is not None and not _chain(ev, i, _next(ev, put, ("arrive",)), ("sync", "fence")):
                bad.append(f"{word}: due words are not ordered before the arrival that publishes the next ones")
        if kind == "get":
            due = _next(ev, i, ("due",), word)
            if due is not None and not _chain(ev, i, due, ("arrive", "wait")):
                bad.append(f"{word}: made due before every reader is known to have read")
        if kind == "put":
            put = _next(ev, i, ("put",), word)
            if put is not None and not any(e == ("due", word) for e in ev[i:put]):
                bad.append(f"{word}: published twice without being due in between")
    return sorted(set(bad))


def test_checker_sees_what_it_is_for():
    chain = [("due", "w"), ("sync", ""), ("fence", ""), ("put", "w"), ("arrive", ""), ("wait", ""), ("get", "w"), ("arrive", ""), ("wait", ""), ("due", "w")]
    assert faults(chain + chain) == []
    assert len(faults([e for e in chain if e[0] != "fence"] * 2)) == 1
    assert len(faults([chain[0], chain[2], chain[1]] + chain[3:])) == 1                     # a fence ahead of the CTA barrier
    assert len(faults(chain[:7] + [("due", "w")])) == 1


@pytest.mark.parametrize("layers", [("moe",) * 4] + [k for k in itertools.product(("conv", "attn"), repeat=4)], ids="-".join)
def test_words_are_due_before_the_next_ones_are_published(layers):
    ev = events(layers)
    words = {w for _, w in ev if w}
    assert {"a.gu", "a.x"} <= words and ("moe" in layers or {"x_mid", "m_out"} <= words) and sum(k == "put" for k, _ in ev) >= 3 * len(layers)
    assert faults(ev) == []


def _function(head):
    return _block(re.sub(r"//[^\n]*", "", SRC[SRC.index(head):]), 0)[1]


def test_every_way_out_waits_for_the_copies_in_flight():
    """A CTA that leaves early has no copy into its shared memory under way: every `return` of the kernel follows a barrier wait that gave up,
    which drains, or a drain of its own; the one exception leaves before anything is requested.  The drain knows the phases that
    copies were requested for from the one function that announces their bytes."""
    kernel = _function("k_moe_ffn_stack(const FusedArgs a) {")
    requests = kernel.index("mbar_expect_tx(")
    for t in re.finditer(r"\breturn;", kernel):
        before = kernel[:t.start()].rstrip()
        assert before.endswith("fused_drain(S);") or re.search(r"if \(!grid_wait\([^;]*\)$", before) or t.start() < requests, before[-120:]
    assert re.search(r"if \(S\.abort == 0\) return true;\s*fused_drain\(S\);\s*return false;\s*}$", _function("bool grid_wait("))
    announce = _function("void mbar_expect_tx(")
    assert "++b->issued;" in announce and SRC.count("mbarrier.arrive.expect_tx") == announce.count("mbarrier.arrive.expect_tx") == 1
    drain = _function("void fused_drain(")
    assert "cp.async.wait_all" in drain
    assert "if (i >= N_BARS) return;" in drain and "&S.mbar[i]" in drain and "FusedBar mbar[N_BARS];" in SRC and SRC.count("FusedBar mbar") == 1
