"""The hand-overs between CTAs of the decode step kernel (it_step.cu), without a GPU.

The kernel has no barrier across the grid: values travel with the tag of the phase that made them, and the next layer's values take
the place of this layer's.  A reader looks for one tag, so a value that is overwritten before its last reader has seen it leaves that
reader waiting for good.  The model below has every read and every write of a step as an event of the CTA and role that performs it, ordered by
nothing but what the kernel guarantees: the order of a role's own work, hand-overs inside a CTA, and a read after the write whose tag it
waits for.  Any CTA may be arbitrarily late; a write is safe only if every read of what it overwrites comes before it in that order.  The cuts of the
matrices and the halves of the quantised row come from the kernel's own plan (it_step_plan.h).
"""
import ctypes as C
import graphlib
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "irontimber_b200", "csrc")
SM = 148
PHASES = "ABCDEFGHI"
KINDS = ("in_gdn", "in_att", "out_gdn", "out_att", "gate_up", "down", "head")
SPAN = ("n", "hl", "tl", "lead", "uh", "uf", "ut", "nb", "cpr", "parts", "units")


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, lib = d / "plan.cpp", d / "plan.so"
    src.write_text('#include "it_step_plan.h"\n'
                   'extern "C" int codes_half(int ph) { return step_codes_half(ph); }\n'
                   'extern "C" void spans(int grid, int rows, int cols, int parts, int* out) {\n'
                   '  std::vector<StepSpan> v((size_t)grid * SP_KINDS); step_spans(v, 0, grid, rows, cols, parts);\n'
                   '  for (int b = 0; b < grid; b++) { const StepSpan& s = v[(size_t)b * SP_KINDS]; const int f[11] = { s.n, s.hl, s.tl, s.lead, s.uh, s.uf, s.ut, s.nb, s.cpr, s.parts, s.units }; memcpy(out + 11 * b, f, sizeof f); } }\n'
                   'extern "C" int ring_slots(const it_model_config* c, int sm) { return step_ring_slots(*c, step_attn_split(*c, sm)); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    return C.CDLL(str(lib))


class Geometry:
    def __init__(self, layers=4, e=5120, ff=17408, vocab=4096, nh=24, nkv=4, hd=256, attn_g=4, nv=48, nk=16, interval=4, grouped=1, grid=SM):
        self.__dict__.update(locals())
        self.inner, self.att, self.qk = 128 * nv, nh * hd, 128 * nk
        self.cd = 2 * self.qk + self.inner
        self.widest = max(e, ff, self.inner, self.att)
        self.attn_base = nv if nv + attn_g * nh <= grid else 0

    def recurrent(self, il):
        return (il + 1) % self.interval != 0

    def matrix(self, kind):
        """rows, columns, matrices of a pair"""
        return {"in_gdn": (self.cd + self.inner, self.e, 1), "in_att": ((2 * self.nh + 2 * self.nkv) * self.hd, self.e, 1), "out_gdn": (self.e, self.inner, 1),
                "out_att": (self.e, self.att, 1), "gate_up": (2 * self.ff, self.e, 2), "down": (self.e, self.ff, 1), "head": (self.vocab, self.e, 1)}[kind]


def spans(plan, g, kind):
    rows, cols, parts = g.matrix(kind)
    buf = (C.c_int * (11 * g.grid))()
    plan.spans(g.grid, rows, cols, parts, buf)
    return [dict(zip(SPAN, buf[11 * b:11 * b + 11])) for b in range(g.grid)]


def units_of(s):
    """The row groups of a CTA's run in its order: (row group, part) with part 'first' (begun, handed on), 'whole' or 'last' (finished)."""
    out, i, unit = [], 0, s["uf"]
    while i < s["n"]:
        if i < s["hl"]:
            out.append((s["uh"], "first")); i += s["hl"]
        elif i >= s["n"] - s["tl"]:
            out.append((s["ut"], "last")); i += s["tl"]
        else:
            out.append((unit, "whole")); unit += 1; i += s["cpr"] * s["parts"]
    return out


class Step:
    """One launch: events with the set of events that surely come before them (a bit each), and per buffer place its writes with their reads."""

    def __init__(self, plan, g, half):
        self.g, self.before, self.places, self.label, self.current = g, [], {}, [], {}
        self.spans = {k: spans(plan, g, k) for k in KINDS}
        self.half = half
        self.cons = [self.event("start %d" % c, []) for c in range(g.grid)]          # a CTA's consumer warps: the event they come from
        self.sums = [[c, c] for c in self.cons]                                      # its two sum warps
        self.start = list(self.cons)
        self.score_events = []                                                       # (CTAs of the head, event that makes the first of them known to the others)
        for il in range(g.layers):
            self.layer(il)
        self.tail()

    def event(self, label, after, reads=(), writes=()):
        m = 0
        for p in after:
            m |= self.before[p] | 1 << p
        for place in reads:                                  # waits for the write that the place has last had when the schedule comes here
            w = self.places[place][-1][0]
            m |= self.before[w] | 1 << w
        k = len(self.before)
        self.before.append(m); self.label.append(label)
        for place in reads:
            self.places[place][-1][1].append(k)
        for place in writes:
            self.places.setdefault(place, []).append((k, []))
        return k

    def transform(self, name, ph, blocks, reads_of, dense=()):
        """The owners of the row's blocks bring in what `reads_of` says and publish their block; `dense`: CTAs that want the row for a dense row."""
        g = self.g
        step = g.grid // (g.widest // 1024)
        owner = {b * step: b for b in range(blocks)}
        for c in sorted(set(owner) | set(dense)):
            rd = self.event("%s: row read by %d" % (name, c), [self.cons[c]], reads=reads_of(owner.get(c)))
            if c in owner:
                rd = self.event("%s: block %d published" % (name, owner[c]), [rd], writes=[("codes", self.half(PHASES.index(ph)), k * blocks + owner[c]) for k in range(4)])
            self.cons[c] = rd

    def matrix(self, name, ph, kind, blocks, dst, old=None, gates=()):
        g, begun = self.g, []
        for c, s in enumerate(self.spans[kind]):
            st = self.event("%s: begun by %d" % (name, c), [self.cons[c]])           # every CTA lets its sum warps in
            if s["n"]:
                st = self.event("%s: codes read by %d" % (name, c), [st], reads=[("codes", self.half(PHASES.index(ph)), c % 4 * blocks + b) for b in range(blocks)])
            self.cons[c] = st
            begun.append(st)
            self.sums[c] = [self.event("", [w, st]) for w in self.sums[c]]
        for r, c in enumerate(gates):                        # dense rows: sum warp 1 of their CTAs
            self.sums[c][1] = self.event("%s: gate %d" % (name, r), [self.sums[c][1]], writes=[("gate", r)])
        rows = [units_of(s) for s in self.spans[kind]]
        for part in ("first", None):                         # nobody waits for anything in front of its first part
            for c, us in enumerate(rows):
                for o, (u, p) in enumerate(us):
                    if (p == "first") != (part == "first"):
                        continue
                    reads = ([(old, u)] if old and p != "first" else []) + ([("prefix", c - 1)] if p == "last" else [])
                    self.sums[c][o & 1] = self.event("%s: row group %d by %d" % (name, u, c), [self.sums[c][o & 1]], reads=[x for x in reads if x in self.places or x[0] != old],
                                                     writes=[("prefix", c)] if p == "first" else [(dst, u)] if dst else [])
        if dst is None:
            for c in range(g.grid):
                for w in (0, 1):
                    self.sums[c][w] = self.event("%s: pick" % name, [self.sums[c][w]], writes=[("partials", c, w)])
        else:                                                # consumers go on when both sum warps are through
            self.cons = [self.event("", [self.cons[c]] + self.sums[c]) for c in range(g.grid)]

    def heads(self, name, recurrent):
        g = self.g
        if recurrent:
            for h in range(g.nv):
                kh = h % g.nk
                rows = [("rows", (at + r) // 32) for at in (kh * 128, g.qk + kh * 128, 2 * g.qk + h * 128, g.cd + h * 128) for r in range(0, 128, 32)]
                rd = self.event("%s: rows read by head %d" % (name, h), [self.cons[h]], reads=rows + [("gate", h), ("gate", g.nv + h)])
                at = (h // g.nk + g.nv // g.nk * kh if g.grouped else h) * 4
                self.cons[h] = self.event("%s: head %d" % (name, h), [rd], writes=[("o", at + i) for i in range(4)])
            return
        for h in range(g.nh):
            kh = h // (g.nh // g.nkv)
            ctas = [g.attn_base + h * g.attn_g + k for k in range(g.attn_g)]
            runs = ((2 * h) * g.hd, (2 * h + 1) * g.hd, 2 * g.nh * g.hd + kh * g.hd, 2 * g.nh * g.hd + g.nkv * g.hd + kh * g.hd)
            sc = []
            for k, c in enumerate(ctas):
                rd = self.event("%s: rows read by head %d, %d" % (name, h, k), [self.cons[c]], reads=[("rows", (at + r) // 32) for at in runs for r in range(0, g.hd, 32)])
                sc.append(self.event("%s: scores of head %d, %d" % (name, h, k), [rd], writes=[("scores", h, k)]))
                self.score_events.append((ctas, c, sc[-1]))
            for k, c in enumerate(ctas):
                rd = self.event("%s: scores read by head %d, %d" % (name, h, k), [sc[k]], reads=[("scores", h, j) for j in range(g.attn_g) if j != k])
                per = g.hd // g.attn_g
                self.cons[c] = self.event("%s: head %d, %d" % (name, h, k), [rd], writes=[("o", (h * g.hd + k * per + r) // 32) for r in range(0, per, 32)])

    def layer(self, il):
        g, rec, n = self.g, self.g.recurrent(il), "layer %d " % il
        eb, ob, fb = g.e // 1024, (g.inner if rec else g.att) // 1024, g.ff // 1024
        row = lambda buf: [(buf, u) for u in range(g.e // 32)]
        block = lambda buf: lambda b: [(buf, 32 * b + i) for i in range(32)]
        gates = [g.grid - 1 - r % g.grid for r in range(2 * g.nv)] if rec else []
        self.transform(n + "A", "A", eb, lambda b: row("xi") if il else [], gates)
        self.matrix(n + "B", "B", "in_gdn" if rec else "in_att", eb, "rows", gates=gates)
        self.heads(n + "C", rec)
        self.transform(n + "D", "D", ob, block("o"))
        self.matrix(n + "E", "E", "out_gdn" if rec else "out_att", ob, "xe", old="xi")
        self.transform(n + "F", "F", eb, lambda b: row("xe"))
        self.matrix(n + "G", "G", "gate_up", eb, "act")
        self.transform(n + "H", "H", fb, block("act"))
        self.matrix(n + "I", "I", "down", fb, "xi", old="xe")

    def tail(self):
        g = self.g
        self.transform("tail A", "A", g.e // 1024, lambda b: [("xi", u) for u in range(g.e // 32)])
        self.matrix("tail B", "B", "head", g.e // 1024, None)
        self.end = self.event("end", [self.cons[0]] + [w for c in range(g.grid) for w in self.sums[c]], reads=[("partials", c, w) for c in range(g.grid) for w in (0, 1)])

    def overwritten_early(self):
        """(read, write that may come before it) pairs; a write to a place after a write that nobody is sure to have read counts as well."""
        out = []
        for place, writes in self.places.items():
            for (w1, reads), (w2, _) in zip(writes, writes[1:]):
                for r in reads or [w1]:
                    if not self.before[w2] >> r & 1:
                        out.append((self.label[r], self.label[w2]))
        return out


GEOMETRIES = {
    "27B": dict(),
    "attention only": dict(interval=1, layers=2),
    "interval 2, widths of 5120 / 1024": dict(ff=1024, interval=2, vocab=64),
    "one block a row": dict(e=1024, ff=2048, nh=4, nkv=2, nv=8, nk=2, vocab=1000),
    "cut gate / up pairs": dict(e=3072, ff=5120, nv=16, nk=4, nh=8, nkv=2, hd=128, attn_g=2, grouped=0, vocab=5000),
    "149 row groups of the head": dict(e=2048, ff=5120, nv=24, nk=8, nh=16, nkv=4, hd=64, attn_g=1, vocab=4767),
    "two dense rows for some CTAs": dict(e=1024, ff=2048, nh=4, nkv=2, nv=80, nk=8, vocab=1000),
    "as many value heads as CTAs allow": dict(e=1024, ff=2048, nh=4, nkv=2, nv=144, nk=16, vocab=1000, interval=2),
    "8192 wide": dict(e=8192, ff=2048, nh=4, nkv=2, nv=8, nk=2, vocab=200),
}


@pytest.mark.parametrize("name", GEOMETRIES)
def test_nothing_is_overwritten_before_its_last_reader(plan, name):
    step = Step(plan, Geometry(**GEOMETRIES[name]), plan.codes_half)
    assert step.overwritten_early() == []
    assert all(step.before[step.end] >> s & 1 for s in step.start)      # the words a launch begins with are read by all before the next launch's are written


def test_the_model_sees_an_early_overwrite(plan):
    """All rows but the activation's in one half: a block of D needs a few heads, whose rows come from some of the CTAs that read A's row."""
    step = Step(plan, Geometry(), lambda ph: int(PHASES[ph] in "HI"))
    early = step.overwritten_early()
    assert early and all(re.match(r"layer \d B: codes read by", r) and re.match(r"layer \d D: block", w) for r, w in early)
    late = {r.rsplit(" ", 1)[1] for r, w in early if r.startswith("layer 0") and w == "layer 0 D: block 0 published"}
    assert len(late) > SM // 2                                          # most CTAs give block 0 nothing


def test_a_count_read_at_the_start_can_come_late(plan):
    """Why the CTAs of an attention head exchange nothing but tagged scores: a count that a CTA reads at its own start may already hold a
    sibling's arrival when layer 0 is an attention layer, or when nobody needs anything of the late CTA's."""
    def late(g):
        step = Step(plan, g, plan.codes_half)
        return [(c, d) for ctas, c, ev in step.score_events for d in ctas if d != c and not step.before[ev] >> step.start[d] & 1]
    assert late(Geometry()) == []
    assert late(Geometry(interval=1, layers=1))
    assert late(Geometry(**dict(GEOMETRIES["one block a row"], attn_g=4)))            # CTAs without row groups
    with open(os.path.join(CSRC, "it_step.cu")) as f:
        phase = re.search(r"void attn_phase\(.*?\n}\n", f.read(), re.S).group()
    assert "st_tagged(shared_sc" in phase and "ld_tagged(P, shared_sc" in phase and "count_up" not in phase and "count_wait" not in phase


def test_the_kernel_uses_the_plan():
    """Both sides of the quantised row take their half from the plan."""
    with open(os.path.join(CSRC, "it_step.cu")) as f:
        src = f.read()
    uses = re.findall(r"P\.codes \+ ([^;]*?)P\.codes_half", src)
    assert uses == ["step_codes_half(ph) * "] * 2, uses


class Ring:
    """One CTA's ring over the matrices of its spans: chunks are issued in order, land in any order, are multiplied by one of three groups of
    warps and summed by one of two warps.  A wait sees the parity of its barrier only, so when it begins the phase before must surely be
    complete, and the phase after must not complete before it has ended."""

    GROUPS, SUMS = 3, 2

    def __init__(self, spans, slots, gated):
        self.after, self.slots = {}, slots
        edge = lambda e, *before: self.after.setdefault(e, set()).update(b for b in before if b is not None)
        group, sums, phase, q0 = [None] * self.GROUPS, [None] * self.SUMS, None, 0
        self.chunks = sum(s["n"] for s in spans)
        for q in range(self.chunks):
            edge(("issue", q), ("issue", q - 1) if q else None, ("free", q - slots) if q >= slots else None)
            edge(("land", q), ("issue", q))
        for p, s in enumerate(spans):
            edge(("phase", p), phase, *sums)
            for i in range(s["n"]):                          # consumer groups
                q, g = q0 + i, i % self.GROUPS
                edge(("full wait", q), group[g], ("phase", p), ("issue", q) if gated and i >= slots else None)
                edge(("use", q), ("full wait", q), ("land", q))
                group[g] = ("use", q)
            i, sums = 0, [("phase", p)] * self.SUMS
            for o, (u, part) in enumerate(units_of(s)):
                n, w = {"first": s["hl"], "last": s["tl"], "whole": s["cpr"] * s["parts"]}[part], o % self.SUMS
                if gated and i + min(n, slots) > slots:      # one look a row group: its first `slots` chunks have been issued
                    edge(("group", p, o), sums[w], ("issue", q0 + i + min(n, slots) - 1))
                    sums[w] = ("group", p, o)
                for k in range(0, n, 2):
                    turn = [q0 + i + k + d for d in range(min(2, n - k))]
                    for q in turn:
                        edge(("sum wait", q), sums[w])
                        edge(("sum", q), ("sum wait", q), ("use", q))
                        sums[w] = ("sum", q)
                    for q in turn:
                        edge(("free", q), sums[w])
                i += n
            assert i == s["n"]
            q0 += s["n"]
        self.before, order = {}, list(graphlib.TopologicalSorter(self.after).static_order())
        bit = {e: 1 << k for k, e in enumerate(order)}
        for e in order:
            m = 0
            for b in self.after.get(e, ()):
                m |= self.before[b] | bit[b]
            self.before[e] = m
        self.bit = bit

    def surely(self, a, b):
        return self.before[b] & self.bit[a]

    def aliased(self):
        out = []
        for q in range(self.chunks):
            if q >= self.slots:
                out += [(w, q) for w, done in (("full wait", "land"), ("sum wait", "use")) if not self.surely((done, q - self.slots), (w, q))]
            if q + self.slots < self.chunks:
                assert self.surely(("use", q), ("land", q + self.slots)) and self.surely(("sum", q), ("use", q + self.slots))
        return out


def ring_spans(plan, g, cta, layers=2):
    kinds = sum(([("in_gdn" if g.recurrent(il) else "in_att"), "out_gdn" if g.recurrent(il) else "out_att", "gate_up", "down"] for il in range(layers)), []) + ["head"]
    return [spans(plan, g, k)[cta] for k in kinds]


@pytest.mark.parametrize("slots", [16, 8, 4])
@pytest.mark.parametrize("name", GEOMETRIES)
def test_no_chunk_wait_takes_another_phase_for_its_own(plan, name, slots):
    g = Geometry(**GEOMETRIES[name])
    for cta in (0, 1, 20, 86, g.grid - 1):
        assert Ring(ring_spans(plan, g, cta), slots, True).aliased() == []


def test_the_model_sees_a_wait_a_phase_early(plan):
    """A row of the down projection is 17 chunks: the sum warp that has the row group behind it waits on a slot of the ring of 16 whose chunk
    the other one may not have summed; and a group's chunk may have been preceded in its slot by one of another group's that has yet to land."""
    g = Geometry()
    found = Ring(ring_spans(plan, g, 86), 16, False).aliased()
    down = sum(s["n"] for s in ring_spans(plan, g, 86)[:3])
    assert ("sum wait", down + 17) in found and any(w == "full wait" for w, _ in found)
    with open(os.path.join(CSRC, "it_step.cu")) as f:
        src = f.read()
    loops = re.search(r"void matvec_phase\(.*?\n}\n.*?void sum_warps\(.*?\n}\n", src, re.S).group()
    assert len(re.findall(r"chunk_wait\(c\.bars \+ 8 \* cs,", loops)) == 1 and not re.findall(r"mbar_wait\w*\(c\.bars", loops)
    gate, tf = re.search(r"want = q \+ \(unsigned\)min\(len, P\.slots\);\s*if \(ok && \(int\)\(want - issued\) > 0\) { issued = issued_past\(c\.issued, want - 1u,", loops), [m.start() for m in re.finditer(r"mbar_wait\(c\.tf", loops)]
    assert len(tf) == 2 and gate.start() < tf[0]
    producer = re.search(r"void producer\(.*?\n}\n", src, re.S).group()
    assert loops.count("unsigned issued = c.q + (unsigned)P.slots;") == 2              # the first chunks of a phase follow a phase that is through
    assert producer.index("mbar_wait(") < producer.index("st_issued(c.issued, (unsigned)issued + 1u)") < producer.index("issued++")


def test_copies_are_waited_for_on_every_way_out():
    """A CTA that leaves with copies in flight lets them land in the shared memory of the next one: whoever starts bulk copies drains its
    rings at its end, and the consumer warps have one way out, behind a wait for their asynchronous copies."""
    with open(os.path.join(CSRC, "it_step.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    producer = re.search(r"void producer\(.*?\n}\n", src, re.S).group()
    assert producer.count("bulk_load(") == 1 and re.search(r"drain_copies\(c\.bars, [^;]*;\s*}\n$", producer) and "return" not in producer
    attn = re.search(r"void attn_phase\(.*?\n}\n", src, re.S).group()
    loader = attn[attn.index("warp == ST_AT_LOADER"):]
    loader = loader[:loader.index("return;")]
    assert attn.count("bulk_load(") == loader.count("bulk_load(") == loader.count("drain_copies(") == 2
    consumers = src[src.index("c.base = *reinterpret_cast<volatile unsigned*>(P.sync + 3)"):]
    consumers = consumers[:consumers.index("leave:")]
    assert not re.search(r"\breturn;", consumers)
    assert re.search(r"leave:\s*asm volatile\(\"cp\.async\.wait_all;", src)


@pytest.mark.parametrize("ctx,slots", [(8192, 16), (9900, 16), (9988, 16), (9989, 8), (16384, 8), (27000, 8), (32768, 4)])
def test_ring_depth_by_context(plan, ctx, slots):
    """The 27B widths: the scores of an attention CTA share its shared memory with the ring."""
    from irontimber_b200.engine import config_27b
    assert plan.ring_slots(C.byref(config_27b(ctx_len=ctx)), SM) == slots


def test_ring_depth_by_widths(plan):
    """Wide rows at a short context: a norm's weights and a dense row come in beside the widest matrix's terms."""
    from irontimber_b200.engine import config_27b
    def depth(**over):
        cfg = config_27b(ctx_len=1024)
        for k, v in over.items():
            setattr(cfg, k, v)
        return plan.ring_slots(C.byref(cfg), SM)
    assert depth(n_head=32, n_head_kv=8, head_dim=128, n_embd=4096, n_ff=12288, ssm_inner=4096, ssm_vheads=32, ctx_len=16384) == 16
    assert depth(n_ff=22528) == 16 and depth(n_ff=32768) == 8 and depth(n_embd=8192, n_ff=40960) == 8
