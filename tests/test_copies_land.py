"""No block leaves with a copy in flight into its shared memory, whichever role's bounded wait gave up: the roles of a block that copies through a
ring, run in random order on the CPU, and the source's own way out of its copying warps."""
import pathlib
import random
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "lfm2-ampere_b200" / "csrc"
# file, what names the copying warps' code, what follows it
COPIERS = {"few": ("lkb_gemm_few.cu", "producers (three warps)", "token constants (one warp)"),
           "tensor-core GEMM": ("lkb_gemm_tc.cu", "producer (one warp)", "MMA issuers (two warps)"),
           "attention": ("lkb_pfattn.cu", "if (warp == C::TMA_WARP) {", "} else if (warp == C::MMA_WARP) {"),
           "output projection": ("lkb_lmhead.cu", "if (warp == LM_WARPS) {", "// consumers: the activation"),
           "router": ("lkb_prefill.cu", "if (warp == NW) {\n", "} else for (int tile")}


def _drains(name):
    """'always', 'own' (only when the copying warp's own wait gave up) or 'never'."""
    file, a, b = COPIERS[name]
    text = (CSRC / file).read_text()
    part = text[text.index(a):text.index(b, text.index(a))]
    part = re.sub(r"//[^\n]*", "", part)
    d = re.search(r"tc_drain|tc_mbar_try|\blm_try", part)
    if not d:
        return "never"
    return "own" if re.search(r"if \((?:!ok|tile < NTILES)\)", part[:d.start()]) else "always"


def _leave(rng, drains, stages=9, ring=4, quits=None):
    """Copies still in flight when every role has left.  quits: a role and the stage at which its wait runs out (the copy is late, or the consumer)."""
    landed, issued, freed, abort = [0], [0], [0], [False]          # copies land in order; stages freed by the consumer

    def copier():
        for it in range(stages):
            while freed[0] <= it - ring:
                if abort[0] or quits == ("copier", it):
                    abort[0] = True
                    if drains != "never":
                        while landed[0] < issued[0]:
                            yield
                    return
                yield
            issued[0] += 1
            yield
        if drains == "always":
            while landed[0] < issued[0]:
                yield

    def consumer():
        for it in range(stages):
            while landed[0] <= it:
                if abort[0] or quits == ("consumer", it):
                    abort[0] = True
                    return
                yield
            yield
            freed[0] += 1

    roles, slow = [copier(), consumer()], rng.random() ** 2 + 0.02
    while roles:
        if landed[0] < issued[0] and rng.random() < slow:          # memory
            landed[0] += 1
        role = rng.choice(roles)
        try:
            next(role)
        except StopIteration:
            roles.remove(role)
    return issued[0] - landed[0]


def _worst(drains):
    rng = random.Random(3)
    return max(_leave(rng, drains, quits=(role, it)) for role in ("copier", "consumer") for it in range(9) for _ in range(60))


def test_model_sees_what_is_left_behind():
    assert _worst("never") > 0 and _worst("own") > 0 and _worst("always") == 0
    assert _leave(random.Random(1), "never") == 0                  # nobody gives up: the consumer has waited for every copy


@pytest.mark.parametrize("name", COPIERS)
def test_copies_land_before_the_block_leaves(name):
    assert _worst(_drains(name)) == 0, f"{name}: drains {_drains(name)}"
