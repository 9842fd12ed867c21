"""The hand-over protocol of the tensor-memory tile kernel (it_matmul_tc.cu), without a GPU.

A wait on an mbarrier sees one bit, the parity of the phase: a role that has not yet seen phase q complete must be sure that phase
q + 1 of the same barrier cannot complete first, or it waits for good, and that phase q - 1 is complete, or it goes on too early.  The model below has the kernel's roles as step counters and
walks every order in which they can proceed; how many barriers the steps commit to in turn is read from the source.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "irontimber_b200", "csrc")
STEPS = 14


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def commit_barriers(acc):
    """Barriers the steps commit to in turn: every wait for a step's commit goes through the same ring."""
    src = source("it_matmul_tc.cu")
    rings = set(re.findall(r"if \(\+\+(?:k0|k|kc) == (\w+)\)", src)) | set(re.findall(r"if \(dp >= (\w+)\)", src)) | set(re.findall(r"k < (\w+); k\+\+\) mbar_init\(dfull0", src))
    assert len(rings) == 1, rings                  # the one ring of issuer, producer, expanders, epilogue and set-up
    return acc if rings == {"TC_ND"} else int(re.search(rings.pop() + r" = (\d+)", src).group(1))


def most_pairs():
    """Pairs of expanded tiles where they fit; else two."""
    src = source("it_matmul_tc.cu")
    assert re.search(r"if \(gp >= na\) ok = ok && mbar_wait\(dfull0 \+ 8 \* dp", src) and re.search(r"\bdp = TC_NC - na\b", src)      # step n waits for the commit of step n - na
    assert re.search(r"if \(\+\+pair == na\) pair = 0;", src) and re.search(r"na = TC_NA_MAX;\s*if \(!fits\(2, 2\)\) na = 2;", src)
    return int(re.search(r"TC_NA_MAX = (\d+)", src).group(1))


def overtaken(acc, boxes, commits, pairs):
    """(role, step) of a wait whose barrier can be two phases on; None when there is no such order.  acc: steps of accumulators, boxes:
    slots of the activation ring, commits: barriers the steps commit to in turn, pairs: pairs of expanded tiles, which both sets of
    expanders fill in turn."""
    seen, todo = set(), [(0, 0, 0, 0, 0, 0)]
    while todo:
        st = todo.pop()
        if st in seen:
            continue
        seen.add(st)
        x, e0, e1, m, c, p = st                     # boxes issued, steps expanded by either set, MMAs issued, committed, steps folded
        for role, q in (("producer", x - boxes), ("expanders 0", 2 * e0 - pairs), ("expanders 1", 2 * e1 + 1 - pairs), ("epilogue", p)):
            if q >= 0 and (c > q + commits or c <= q - commits):       # the phase after is complete, or the one before is not: either is taken for phase q
                return role, q
        if x < STEPS and (x < boxes or c > x - boxes):
            todo.append((x + 1, e0, e1, m, c, p))
        if 2 * e0 < STEPS and c > 2 * e0 - pairs:
            todo.append((x, e0 + 1, e1, m, c, p))
        if 2 * e1 + 1 < STEPS and c > 2 * e1 + 1 - pairs:
            todo.append((x, e0, e1 + 1, m, c, p))
        if m < x and (e1 if m & 1 else e0) > m // 2 and p > m - acc:
            todo.append((x, e0, e1, m + 1, c, p))
        if c < m:
            todo.append((x, e0, e1, m, c + 1, p))
        if p < c:
            todo.append((x, e0, e1, m, c, p + 1))
    assert (STEPS, STEPS // 2, STEPS // 2, STEPS, STEPS, STEPS) in seen           # the model can run to its end
    return None


@pytest.mark.parametrize("acc,boxes", [(4, 2), (4, 3), (2, 2), (2, 3)])      # 64- and 128-row tiles, with two and three steps of boxes
def test_no_wait_can_be_overtaken(acc, boxes):
    for pairs in range(2, most_pairs() + 1):
        assert overtaken(acc, boxes, commit_barriers(acc), pairs) is None


def test_the_model_sees_an_overtaken_wait():
    """A barrier per accumulator, two of them, and three slots of boxes: box n - 1 is in place while the producer waits for step n - 3, and
    both commit to one barrier."""
    assert overtaken(2, 3, 2, 2) == ("producer", 0)


@pytest.mark.parametrize("acc,boxes", [(4, 2), (4, 3), (2, 2), (2, 3)])
def test_more_pairs_than_commit_barriers_are_too_many(acc, boxes):
    """As many pairs as barriers are the limit that the kernel asserts: step n, which commits to the barrier of step n - 4, waits for its
    expanders.  With a fifth pair step n - 1 commits to the barrier of step n - 5, which a late set of expanders is still to see."""
    assert overtaken(acc, boxes, 4, 4) is None
    assert overtaken(acc, boxes, 4, 5)[0].startswith("expanders")
    assert "static_assert(TC_NA_MAX <= TC_NC" in source("it_matmul_tc.cu")


def warp_statements(src, pattern):
    """Statements of `src` in which `pattern` occurs and that no enclosing condition gives to one lane."""
    out, scopes = [], []
    for m in re.finditer(r"[{}]|" + pattern, src):
        head = re.split(r"[;{}]", src[:m.start()])[-1]
        if m.group() == "{":
            scopes.append(head)
        elif m.group() == "}":
            scopes.pop()
        elif not any("lane == 0" in s or "tid == 0" in s for s in scopes + [head]):
            out.append(head + re.split(r"[;{}]", src[m.start():])[0])
    return out


def test_a_warp_gives_up_as_one():
    """The roles of whole warps go on to warp-wide instructions: a lane that leaves alone after a wait that ran out, or after a look of its
    own at the abort flag, leaves its siblings there without a limit.  A lane's wait may only be remembered; what leaves is voted on."""
    src = re.sub(r"//(?! -{16})[^\n]*|\"[^\"\n]*\"", "", source("it_matmul_tc.cu"))
    kernel = src[src.index("k_matmul_tc("):src.index("it_shard_finish")]
    assert [s for s in warp_statements(kernel, r"mbar_wait\(") if "ok = ok && mbar_wait(" not in s] == []
    assert [s for s in warp_statements(kernel, r"\*abort_flag\b") if "_sync(" not in s and "lane == 0" not in s and "volatile int* abort_flag" not in s] == []
    roles = {r.split()[0].strip(":"): r for r in kernel.split("// ---------------- ")[1:]}
    for role in ("activation", "expanders", "epilogue"):          # "activation": the scales, the later of the two roles of that name
        leaves = warp_statements("{" + roles[role], r"\bbreak;")
        assert [s for s in leaves if "__all_sync(" not in s and "mbar_wait_warp(" not in s] == [], role
        assert not re.search(r"for \([^;]*;[^;]*\bok\b", roles[role]), role
