"""The work that users of this library have it do, as cases that can be timed and compared.

Two kinds of user.  A host with its own schedule calls the operations of `CudaBackend` one by one: the Hadamard rotation with
q8k quantisation in front of a ternary product, the int8-group product with the greedy pick behind it.  A serving program
calls `CudaEngine`: prompts, plain greedy decoding, decoding with its own sampler on the logits, speculative decoding.

Weights, prompts and activations are random, as in this repository's benchmark and tests: ternary codes uniform over
{-1, 0, +1} with f16 block scales in [0.01, 0.05], int8 groups, activations N(0, 1), token ids uniform over the vocabulary;
all of them follow from the seed.  The engine is the 27B architecture (`config_27b`) at context 8192.

Results are compared exactly: the library's contract is the reference's own order of rounded additions (exact integers
inside a block of 128, every f32 product and sum rounded in block, position or index order), so token histories, logits
and products have one right answer at this precision, and the tests hold them to it bit for bit.
"""
import math
import weakref

import numpy as np
import torch

from irontimber_b200.backend import CudaBackend
from irontimber_b200.engine import CudaEngine, config_27b

CTX = 8192
VOCAB = 248320


def listed():
    return [
        # ---- operations -----------------------------------------------------------------------------------
        # one projection of a decoded token, issued call by call: the smallest unit a host schedules (attention output width)
        {"name": "project-1", "kind": "project", "rows": 5120, "cols": 6144, "ntok": 1, "mats": 1, "acc": False, "graph": False},
        # a decoded token's gate projections of twelve layers (285 MB: weights come from HBM as in a real step), recorded once
        # and replayed, which is how a host runs its decode schedule
        {"name": "project-1-sweep", "kind": "project", "rows": 17408, "cols": 5120, "ntok": 1, "mats": 12, "acc": False, "graph": True},
        # the stacked gate/up projection of a long prompt, the largest product of the architecture
        {"name": "project-512", "kind": "project", "rows": 34816, "cols": 5120, "ntok": 512, "mats": 1, "acc": False, "graph": False},
        # an int8 LM head over the whole vocabulary and the greedy pick
        {"name": "head-q8", "kind": "head", "rows": VOCAB, "cols": 5120, "ntok": 1},
        # ---- engine ---------------------------------------------------------------------------------------
        # a short question and a short answer: latency of a request with next to no context
        {"name": "chat-9", "kind": "chat", "layers": 64, "prompt": 9, "new": 48},
        # the benchmark's request: a 512-token prompt, then greedy decoding
        {"name": "chat-512", "kind": "chat", "layers": 64, "prompt": 512, "new": 64},
        # a server that samples on the host: every token's logits cross to the host
        {"name": "sampled-133", "kind": "sampled", "layers": 64, "prompt": 133, "new": 16},
        # prompts alone (time to the first token, scoring): short and ragged, ordinary and ragged, long
        {"name": "prompt-61", "kind": "prompt", "layers": 64, "prompt": 61},
        {"name": "prompt-777", "kind": "prompt", "layers": 64, "prompt": 777},
        {"name": "prompt-4096", "kind": "prompt", "layers": 64, "prompt": 4096},
        # speculative decoding, the reference's draft length and the longest one
        {"name": "mtp-1", "kind": "mtp", "layers": 64, "prompt": 128, "new": 32, "k": 1},
        {"name": "mtp-3", "kind": "mtp", "layers": 64, "prompt": 128, "new": 32, "k": 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("project", "project", "project", "head", "chat", "sampled", "prompt", "prompt", "mtp"))
    if kind == "project":
        ntok = _log(rng, 1, 512)
        mats = rng.choice((1, 4)) if ntok <= 8 else 1
        acc = rng.random() < 0.3
        return {"kind": kind, "rows": _log(rng, 500, 69632 if ntok <= 64 else 34816), "cols": 1024 * rng.randint(1, 17), "ntok": ntok, "mats": mats,
                "acc": acc, "graph": not acc and rng.random() < 0.5}
    if kind == "head":
        return {"kind": kind, "rows": _log(rng, 4096, VOCAB), "cols": 1024 * rng.randint(1, 10), "ntok": rng.randint(1, 4)}
    layers = rng.choice((8, 64))
    if kind == "chat":
        return {"kind": kind, "layers": layers, "prompt": _log(rng, 1, 2048), "new": rng.randint(8, 64)}
    if kind == "sampled":
        return {"kind": kind, "layers": layers, "prompt": _log(rng, 1, 1024), "new": rng.randint(4, 24)}
    if kind == "prompt":
        return {"kind": kind, "layers": layers, "prompt": _log(rng, 9, 4096)}
    return {"kind": kind, "layers": layers, "prompt": _log(rng, 16, 1024), "new": rng.randint(8, 32), "k": rng.randint(1, 3)}


class _Handles:
    """Native handles, closed in order when the state that made them and the views into its arena are gone."""

    def __init__(self, *handles):
        weakref.finalize(self, _close, handles)


def _close(handles):
    for h in handles:
        h.close()


class _Graph:
    def __init__(self, backend, handle):
        self.backend, self.handle = backend, handle

    def close(self):
        self.backend.graph_destroy(self.handle)


class _Floats:
    """A run of arena elements, for torch to see without a copy; keeps the arena alive."""

    def __init__(self, backend, off, shape, handles):
        self.handles = handles
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f4", "data": (backend.arena_ptr + 4 * off, False), "version": 3}


def _view(backend, off, shape, handles):
    return torch.as_tensor(_Floats(backend, off, shape, handles), device="cuda:%d" % backend.device)


class _State:
    """What the caller keeps between calls."""


def _up(n):
    return (n + 63) // 64 * 64


def _prepare_project(s, c, seed):
    rng = np.random.default_rng(seed)
    rows, cols, ntok, mats = c["rows"], c["cols"], c["ntok"], c["mats"]
    ys = (rows + 3) // 4 * 4                                     # output row stride
    xo, yo = 0, _up(ntok * cols)
    ylen = _up(ntok * ys)
    be = CudaBackend(0, arena_floats=yo + ylen * (1 if c["acc"] else mats))
    ws = [be.mat_synth(1000003 * seed + i, rows, cols) for i in range(mats)]
    q = be.q8_rows(cols, ntok)
    be.set_signs(np.where(rng.integers(0, 2, cols) == 1, 1.0, -1.0).astype(np.float32))
    be.upload(xo, rng.standard_normal((ntok, cols), dtype=np.float32))
    s.be, s.ws, s.q, s.ys = be, ws, q, ys
    s.yo = [yo if c["acc"] else yo + i * ylen for i in range(mats)]
    s.ylen = ylen
    handles = [q, *ws, be]
    s.graph = None
    if c["graph"]:
        _project(s)                                              # once outside the recording, as a host's warm-up does
        be.sync()
        be.capture_begin()
        _project(s)
        s.graph = be.capture_end()
        handles.insert(0, _Graph(be, s.graph))
    s.handles = _Handles(*handles)
    s.y = _view(be, yo, (1 if c["acc"] else mats, ylen), s.handles)
    be.sync()


def _project(s):
    c, be = s.case, s.be
    cols, ntok = c["cols"], c["ntok"]
    if c["acc"]:
        be.zero(s.yo[0], s.ylen)                            # a residual that the products accumulate into
    for w, yo in zip(s.ws, s.yo):
        be.had_q8(cols, ntok, 0, cols, s.q)
        be.mv(w, ntok, s.q, yo, s.ys, acc=c["acc"])


def _prepare_head(s, c, seed):
    rng = np.random.default_rng(seed)
    rows, cols, ntok = c["rows"], c["cols"], c["ntok"]
    ys = (rows + 3) // 4 * 4
    yo = _up(ntok * cols)
    po = yo + _up(ntok * ys)
    be = CudaBackend(0, arena_floats=po + 64)
    w = be.qmat_synth(seed, rows, cols)
    be.upload(0, rng.standard_normal((ntok, cols), dtype=np.float32))
    s.be, s.w, s.yo, s.ys, s.po = be, w, yo, ys, po
    s.handles = _Handles(w, be)
    s.y = _view(be, yo, (ntok, ys), s.handles)
    s.pick = _view(be, po, (ntok,), s.handles).view(torch.int32)
    be.sync()


def prepare(case, seed):
    s = _State()
    s.case = case
    if case["kind"] == "project":
        _prepare_project(s, case, seed)
    elif case["kind"] == "head":
        _prepare_head(s, case, seed)
    else:
        rng = np.random.default_rng(seed)
        s.eng = CudaEngine(config_27b(n_layer=case["layers"], ctx_len=CTX, n_vocab=VOCAB), seed=seed, with_mtp=case["kind"] == "mtp")
        s.prompt = rng.integers(0, VOCAB, case["prompt"]).astype(np.uint32)
        s.handles = _Handles(s.eng)
    return s


def run(s):
    c = s.case
    kind = c["kind"]
    if kind == "project":
        if s.graph is not None:
            s.be.graph_launch(s.graph)
        else:
            _project(s)
        return s.y
    if kind == "head":
        s.be.mvq(s.w, c["ntok"], 0, c["cols"], s.yo, s.ys)
        for t in range(c["ntok"]):
            s.be.argmax(s.yo + t * s.ys, c["rows"], s.po + t)
        return {"logits": s.y, "pick": s.pick}
    eng = s.eng
    if kind == "prompt":
        eng.reset()
        return eng.eval(s.prompt)
    if kind == "chat":
        eng.reset()
        toks = eng.generate(s.prompt, c["new"])
        return {"tokens": np.array(toks, np.int64), "logits": eng.eval(toks[-1:])}      # the logits a caller continues from
    if kind == "sampled":
        eng.reset()
        logits = eng.eval(s.prompt)
        toks = []
        for _ in range(c["new"]):
            toks.append(int(logits.argmax()))                    # stands for the caller's sampler
            logits = eng.eval(toks[-1:])
        return {"tokens": np.array(toks, np.int64), "logits": logits}
    toks, stats = eng.generate_mtp(s.prompt, c["new"]) if c["k"] == 1 else eng.generate_mtp_k(s.prompt, c["new"], c["k"])
    return {"tokens": np.array(toks, np.int64), "stats": np.array([stats[k] for k in sorted(stats)], np.int64), "logits": eng.eval(toks[-1:])}


# ---- what a pass cannot do without ---------------------------------------------------------------------------
def _trunk(layers):
    """(weights of the layers, weights of the LM head, bytes of recurrent state, attention layers)."""
    cfg = config_27b(n_layer=layers, ctx_len=CTX, n_vocab=VOCAB)
    e, ff, inner = cfg.n_embd, cfg.n_ff, cfg.ssm_inner
    cd = 2 * cfg.ssm_state * cfg.ssm_groups + inner
    att = sum(1 for il in range(layers) if not cfg.is_recurrent(il))
    gdn = layers - att
    w = gdn * (cd + 2 * inner) * e + att * (2 * cfg.n_head + 2 * cfg.n_head_kv + cfg.n_head) * cfg.head_dim * e + layers * 3 * ff * e
    state = gdn * 4 * (cfg.ssm_vheads * cfg.ssm_state ** 2 + (cfg.conv_k - 1) * cd)
    return cfg, w, VOCAB * e, state, att


def _pass_work(layers, rows, pos, heads):
    """One pass over `rows` tokens from position `pos` on, logits of `heads` of them: (bytes, flops)."""
    cfg, w, head, state, att = _trunk(layers)
    kvd = cfg.n_head_kv * cfg.head_dim
    kv = att * 2 * 2 * kvd * (pos + 2 * rows)                    # the cache read once, the new entries written once
    seen = rows * pos + rows * (rows + 1) // 2
    b = (w + (head if heads else 0)) / 128 * 34 + 2 * state + kv + 4 * rows * cfg.n_embd + 4 * heads * VOCAB
    f = 2 * w * rows + 2 * head * heads + att * 4 * cfg.n_head * cfg.head_dim * seen + (layers - att) * 8 * cfg.ssm_vheads * cfg.ssm_state ** 2 * rows
    return b, f


def _head_work(rows, ntok):
    """The NextN head over `rows` tokens: int8 groups with an f16 scale per 32."""
    cfg = config_27b(n_layer=4)
    e, kvd, qf = cfg.n_embd, cfg.n_head_kv * cfg.head_dim, 2 * cfg.n_head * cfg.head_dim
    w = e * (2 * e + qf + 2 * kvd + cfg.n_head * cfg.head_dim + 3 * cfg.n_ff)
    return w * 34 / 32 + VOCAB * e / 128 * 34 + 4 * VOCAB, 2 * w * rows + 2 * VOCAB * e


def work(case):
    kind = case["kind"]
    if kind == "project":
        r, k, t, m = case["rows"], case["cols"], case["ntok"], case["mats"]
        y = 4 * t * r * (1 if case["acc"] else m)
        return {"bytes": m * r * k / 128 * 34 + 4 * t * k + y, "flops": 2 * m * r * k * t}
    if kind == "head":
        r, k, t = case["rows"], case["cols"], case["ntok"]
        return {"bytes": r * k / 32 * 34 + 4 * t * k + 4 * t * r, "flops": 2 * r * k * t}
    layers, p = case["layers"], case["prompt"]
    b, f = _pass_work(layers, p, 0, 1)
    if kind in ("chat", "sampled"):
        for i in range(case["new"]):                              # the prompt gives the first token; the last token's logits close the request
            x, y = _pass_work(layers, 1, p + i, 1)
            b, f = b + x, f + y
    elif kind == "mtp":
        # random weights: every draft is rejected, so a token costs a verification pass of k + 1 rows and k draft steps
        hb, hf = _head_work(p, 1)
        b, f = b + hb, f + hf
        for i in range(case["new"] - 1):
            x, y = _pass_work(layers, case["k"] + 1, p + i, case["k"] + 1)
            b, f = b + x, f + y
            for _ in range(case["k"]):
                x, y = _head_work(1, 1)
                b, f = b + x, f + y
        x, y = _pass_work(layers, 1, p + case["new"], 1)
        b, f = b + x, f + y
    return {"bytes": b, "flops": f}


def tolerance(case):
    return "exact"
