"""What the speed of this framework is measured on: passes of its models and two of its operators, through the calls that a user's
program makes.

Block-quantised decoders (the shapes of `config_tiny`, `config_8b_target` and `config_8b_draft`), one pass at a time:

- a decoded token, a chain of proposals or a tree of proposals of one or more streams over a filled context, whose logits come back, and
  the rollback that follows when nothing is accepted;
- a whole prompt, then the logits of the token after it.

Plain-weight decoders (the Nigenex design in the smaller of its benchmark's widths): a prompt, one token of each of many streams, and a
prompt's portion beside the tokens of other streams, as a continuously batched server brings them.

Operators: acceptance of a round's proposals, and the routed feed-forward.

The cached rows of the block-quantised models are the library's seeded synthetic ones; `exact` makes the same numbers again.
"""
import math

import numpy as np
import torch

import turbospark_b200 as tsb
from turbospark_b200 import capi, nigenex, plain
from turbospark_b200.model import N_ATTN, N_FFN, N_OUT, W_DOWN, W_EMBED, W_GATE, W_K, W_LM_HEAD, W_O, W_Q, W_UP, W_V

# layers, width, query heads, key heads, head size, feed-forward, vocabulary, norm epsilon, rotation base
SHAPES = {"tiny": (4, 512, 8, 2, 64, 1536, 8192, 1e-6, 1e4), "2b": (16, 2048, 32, 8, 64, 8192, 128256, 1e-5, 5e5),
          "8b": (32, 4096, 32, 8, 128, 14336, 128256, 1e-5, 5e5)}
TYPES = {"q4_k": (capi.Q4_K, 256, 144), "q6_k": (capi.Q6_K, 256, 210), "q8_0": (capi.Q8_0, 32, 34), "mxfp4": (capi.MXFP4, 32, 17)}
LAYERS = 8  # layers of a block-quantised model with tensors of their own (a gigabyte at the largest shape); the ones behind them use these again
# a Nigenex model: layers, width, query heads, key heads, head size, window, feed-forward, vocabulary
PLAIN = (8, 2048, 32, 8, 64, 1024, 8192, 32000)


def listed():
    return [
        # the smallest call: one token of a small model, where the launches are what counts
        dict(name="decode_tiny", kind="pass", shape="tiny", blocks="q4_k", streams=1, rows=1, tree=False, context=200),
        # one user's next token on the target and on the drafter of the speculative pair
        dict(name="decode_8b", kind="pass", shape="8b", blocks="q4_k", streams=1, rows=1, tree=False, context=4093),
        dict(name="decode_2b", kind="pass", shape="2b", blocks="q4_k", streams=1, rows=1, tree=False, context=4093),
        # the verify pass of the speculative round: five proposals and the confirmed token
        dict(name="verify_8b", kind="pass", shape="8b", blocks="q4_k", streams=1, rows=6, tree=False, context=4093),
        # the verify pass of a tree round
        dict(name="tree_8b", kind="pass", shape="8b", blocks="q4_k", streams=1, rows=65, tree=True, context=8191),
        # the verify pass of a server's round
        dict(name="verify_8b_streams", kind="pass", shape="8b", blocks="q4_k", streams=16, rows=6, tree=False, context=1500),
        # another block format
        dict(name="verify_2b_q6_k", kind="pass", shape="2b", blocks="q6_k", streams=2, rows=5, tree=False, context=1021),
        # a prompt
        dict(name="prefill_8b", kind="prefill", shape="8b", blocks="q4_k", tokens=1000),
        # acceptance of a server's round, shaped as chat services shape
        dict(name="accept", kind="accept", batch=32, k=5, vocab=128256, temperature=0.8, top_k=0, top_p=0.95, min_p=0.0),
        # the routed feed-forward of the mixture-of-experts benchmark, eight streams of five rows
        dict(name="experts", kind="experts", blocks="mxfp4", tokens=40, experts=128, top=8, width=2048, ffn=768),
        # plain weights: a prompt, and one token of each of many streams
        dict(name="plain_prefill", kind="plain", streams=1, rows=2000, context=0, mixed=False),
        dict(name="plain_decode", kind="plain", streams=16, rows=1, context=900, mixed=False),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["pass", "pass", "pass", "pass", "prefill", "accept", "experts", "plain"])
    if kind == "pass":
        shape = rng.choice(["tiny", "2b", "2b", "8b"])
        blocks = rng.choice(["q4_k", "q4_k", "q4_k", "q6_k", "q8_0"])
        what = rng.choice(["decode", "verify", "tree"])
        streams = rng.choice([1, 1, _log(rng, 2, 16)])
        rows = 1 if what == "decode" else rng.randint(2, 9) if what == "verify" else rng.randint(17, 65)
        if what == "tree":
            streams = 1
        return dict(kind=kind, shape=shape, blocks=blocks, streams=streams, rows=rows, tree=what == "tree", context=_log(rng, 16, 4093 if streams == 1 else 1500))
    if kind == "prefill":
        return dict(kind=kind, shape=rng.choice(["tiny", "2b", "8b"]), blocks="q4_k", tokens=_log(rng, 20, 1000))
    if kind == "accept":
        temperature = rng.choice([0.0, 0.6, 0.8, 1.0, 1.0])
        return dict(kind=kind, batch=_log(rng, 1, 32), k=rng.randint(1, 8), vocab=rng.choice([8192, 32003, 128256, 151936]), temperature=temperature,
                    top_k=rng.choice([0, 0, 40]) if temperature else 0, top_p=rng.choice([0.0, 0.9, 0.95]) if temperature else 0.0,
                    min_p=rng.choice([0.0, 0.0, 0.05]) if temperature else 0.0)
    if kind == "experts":
        experts = rng.choice([8, 32, 128])
        return dict(kind=kind, blocks=rng.choice(["mxfp4", "mxfp4", "q4_k"]), tokens=_log(rng, 1, 64), experts=experts, top=rng.choice([2, 4, 8]),
                    width=rng.choice([1024, 2048]), ffn=rng.choice([256, 768]))
    what = rng.choice(["prefill", "decode", "mixed"])
    if what == "prefill":
        return dict(kind=kind, streams=1, rows=_log(rng, 33, 2000), context=0, mixed=False)
    return dict(kind=kind, streams=_log(rng, 2, 24), rows=1 if what == "decode" else _log(rng, 17, 120), context=_log(rng, 100, 1200), mixed=what == "mixed")


class Opened:
    """Handles that are closed, the last one first, when the state goes."""

    def __init__(self):
        self.ctx = tsb.Ctx(0)
        self.handles = [self.ctx]

    def own(self, h):
        self.handles.append(h)
        return h

    def __del__(self):
        try:
            while self.handles:
                self.handles.pop().close()
        except Exception:
            pass


def _seeds(seed, *more):
    return np.random.default_rng([int(seed)] + list(more))


def _tree_parents(rows):
    return [-1] + [(j - 1) // 3 for j in range(1, rows)]


def _feed(case, seed):
    rng, v = _seeds(seed, 1), SHAPES[case["shape"]][6]
    return rng.integers(0, v, size=(case["streams"], case["rows"])).astype(np.int32)


def _prompt(case, seed):
    rng, v = _seeds(seed, 2), SHAPES[case["shape"]][6]
    return rng.integers(0, v, size=case["tokens"] + 1).astype(np.int32)


def _blocks(blocks, count, g):
    """[count, bytes of a block]: any bytes, with scales that make zero-mean weights of standard deviation 0.02."""
    size = TYPES[blocks][2]
    p = torch.randint(0, 256, (count, size), device="cuda", generator=g, dtype=torch.uint8)
    u = torch.rand(count, device="cuda", generator=g) + 0.5

    def put(at, v):
        p[:, at:at + 2] = v.half().view(torch.uint8).view(-1, 2)
    if blocks == "q4_k":
        put(0, u * 7.7e-5)
        put(2, u * 5.8e-4)
    elif blocks == "q6_k":
        put(208, u * 1.46e-5)
    elif blocks == "q8_0":
        put(0, u * 2.7e-4)
    else:
        p[:, 0] = 119 + (p[:, 0] & 1)
    return p


def _matrices(case, seed):
    """(layer, [(which, rows, columns, blocks), ...]) of a model's layers, then (-1, [embedding, head])."""
    layers, d, nq, nkv, hd, ff, vocab, _, _ = SHAPES[case["shape"]]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 6700417 + 7)
    per = TYPES[case["blocks"]][1]
    make = lambda which, rows, cols: (which, rows, cols, _blocks(case["blocks"], rows * cols // per, g))  # noqa: E731
    for l in range(min(layers, LAYERS)):
        yield l, [make(*m) for m in ((W_Q, nq * hd, d), (W_K, nkv * hd, d), (W_V, nkv * hd, d), (W_O, d, nq * hd), (W_GATE, ff, d), (W_UP, ff, d), (W_DOWN, d, ff))]
    yield -1, [make(W_EMBED, vocab, d), make(W_LM_HEAD, vocab, d)]


_pinned = None


def _on_host(p):
    """The bytes of p in page-locked memory, valid until the next call."""
    global _pinned
    if _pinned is None or _pinned.numel() < p.numel():
        _pinned = torch.empty(p.numel(), dtype=torch.uint8, pin_memory=True)
    v = _pinned[:p.numel()]
    v.copy_(p.view(-1))
    return v.numpy()


def _open_model(s, case, seed, max_context):
    layers, d, nq, nkv, hd, ff, vocab, eps, theta = SHAPES[case["shape"]]
    m = s.own(tsb.Model(s.ctx, tsb.ModelConfig(layers, d, nq, nkv, hd, ff, vocab, max_context, eps, theta)))
    ones = np.full(d, 0x3F80, dtype=np.uint16)
    for l, mats in _matrices(case, seed):
        for which, rows, cols, p in mats:
            m.set_matrix(l, which, TYPES[case["blocks"]][0], _on_host(p), rows, cols)
        for which in (N_ATTN, N_FFN) if l >= 0 else (N_OUT,):
            m.set_norm(l, which, ones)
    for l in range(LAYERS, layers):
        m.share(l, m, l % LAYERS)
    return m


# ------------------------------------------------------------------ inputs
def _prepare_pass(case, seed):
    s = Opened()
    n, c = case["rows"], case["context"]
    m = _open_model(s, case, seed, c + n + 32)
    s.sess = s.own(tsb.Session(s.ctx, m, None, case["streams"], n))
    s.sess.fill_context(c, seed=2000 + seed)
    s.feed, s.parents, s.context, s.tree, s.streams = _feed(case, seed), _tree_parents(n) if case["tree"] else list(range(-1, n - 1)), c, case["tree"], case["streams"]
    return s


def _run_pass(s):
    sess, c = s.sess, s.context
    if s.streams > 1:
        logits = sess.verify_tree_streams(s.feed, s.parents)
    elif s.tree:
        logits = sess.verify_tree(s.feed[0], s.parents, c)
    elif s.feed.shape[1] > 1:
        logits = sess.verify(s.feed[0], c)
    else:
        logits = sess.produce(int(s.feed[0, 0]), c)
    for q in range(s.streams):
        sess.rollback_retaining(c, 0, stream=q)
    return logits.view(np.float16)


def _prepare_prefill(case, seed):
    s = Opened()
    n = case["tokens"]
    m = _open_model(s, case, seed, n + 32)
    s.sess = s.own(tsb.Session(s.ctx, m, None, 1, 128))
    s.tokens = _prompt(case, seed)
    s.once = tsb.run_config(tsb.shaping(temperature=0.0), 1, 1)
    return s


def _run_prefill(s):
    n = len(s.tokens) - 1
    s.sess.sequential_run(s.tokens[:n], s.once)
    return s.sess.produce(int(s.tokens[n]), n).view(np.float16)


def _accept_inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7919 + 3)
    b, k, v = case["batch"], case["k"], case["vocab"]
    t = torch.randn(b, k + 1, v, device="cuda", generator=g) * 3.0
    d = t[:, :k] + torch.randn(b, k, v, device="cuda", generator=g) * 0.7
    target, draft = t.half(), d.half()
    warm = case["temperature"] or 1.0
    props = torch.multinomial(torch.softmax(draft.float().reshape(b * k, v) / warm, -1), 1, generator=g).to(torch.int32).reshape(b, k)
    uniforms = torch.randint(-(1 << 63), (1 << 63) - 1, (b, 2 * k + 1), device="cuda", generator=g, dtype=torch.int64)
    return target, draft, props, uniforms


def _prepare_accept(case, seed):
    s = Opened()
    b, k, v = case["batch"], case["k"], case["vocab"]
    s.inputs = _accept_inputs(case, seed)
    s.out = torch.zeros(b, 96, device="cuda", dtype=torch.uint8)
    s.scratch = s.ctx.alloc(s.ctx.accept_scratch_bytes(b, k, v))
    s.cfg = tsb.shaping(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], min_p=case["min_p"])
    s.sizes = (b, k, v)
    return s


def _run_accept(s):
    t, d, p, u = s.inputs
    s.ctx.accept(t.data_ptr(), d.data_ptr(), p.data_ptr(), u.data_ptr(), *s.sizes, s.cfg, s.out.data_ptr(), s.scratch)
    return {"decided": s.out.view(torch.int32)[:, :19], "margins": s.out.view(torch.float64)[:, 10:]}


def _experts_inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 104729 + 5)
    e, d, f, n, top = case["experts"], case["width"], case["ffn"], case["tokens"], case["top"]
    per = TYPES[case["blocks"]][1]

    def blocks(rows, cols):  # the bytes behind the last block are what the calls may read too much
        p = _blocks(case["blocks"], e * rows * cols // per, g).view(-1)
        return torch.cat([p, torch.zeros(256, device="cuda", dtype=torch.uint8)])

    x = torch.randn(n, d, device="cuda", generator=g).half()
    residual = torch.randn(n, d, device="cuda", generator=g).half()
    score, ids = torch.topk(torch.randn(n, e, device="cuda", generator=g) * 2.0, top, dim=1)
    return blocks(2 * f, d), blocks(d, f), x, residual, ids.to(torch.int32), torch.softmax(score, 1).half()


def _prepare_experts(case, seed):
    s = Opened()
    s.inputs = _experts_inputs(case, seed)
    s.y = torch.empty_like(s.inputs[2])
    s.case = case
    return s


def _run_experts(s):
    c, (gu, dn, x, residual, ids, w) = s.case, s.inputs
    s.ctx.moe_ffn(TYPES[c["blocks"]][0], gu.data_ptr(), dn.data_ptr(), c["experts"], c["width"], c["ffn"], x.data_ptr(), residual.data_ptr(), ids.data_ptr(), w.data_ptr(),
                  c["tokens"], c["top"], s.y.data_ptr())
    return s.y


def _plain_config():
    layers, d, nq, nkv, hd, window, ff, vocab = PLAIN
    layer = {"type": "attention", "mixer": {"heads": nq, "kv_heads": nkv, "dim": hd, "vdim": hd, "mask": {"size": window}, "scale": hd ** -0.5, "softcap": 50.0},
             "mlp": {"kind": "dense", "ff": ff}}
    return {"architecture": "Nigenex", "width": d, "vocab": vocab, "norm": {"eps": 1e-6}, "logit_softcap": 30.0, "layers": [layer] * layers}


def _plain_weights(seed):
    """name -> tensor on the GPU, values that are bfloat16 numbers."""
    layers, d, nq, nkv, hd, _, ff, vocab = PLAIN
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 15485863 + 11)

    def normal(*shape, std):
        return (torch.randn(*shape, device="cuda", generator=g) * std).bfloat16()

    def uniform(n, lo, hi):
        return (torch.rand(n, device="cuda", generator=g) * (hi - lo) + lo).bfloat16()

    w = {"embed": normal(vocab, d, std=1.0), "head": normal(vocab, d, std=d ** -0.5), "final.norm": uniform(1, 0.9, 1.1)}
    for i in range(layers):
        p = "l%d." % i
        w[p + "norm1"], w[p + "shift"] = uniform(1, 0.9, 1.1), uniform(d, 0.1, 0.9)
        w[p + "mix.q"], w[p + "mix.k"], w[p + "mix.g"] = normal(nq * hd, d, std=d ** -0.5), normal(nkv * hd, d, std=d ** -0.5), normal(nq, d, std=d ** -0.5)
        w[p + "mix.r1"], w[p + "mix.r2"] = uniform(nq, 0.5, 1.5), uniform(nq, 0.1, 0.5)
        w[p + "mix.o"] = normal(d, nq * hd, std=0.5 * (nq * hd) ** -0.5)
        w[p + "mlp.gate"], w[p + "mlp.up"], w[p + "mlp.down"] = normal(ff, d, std=d ** -0.5), normal(ff, d, std=d ** -0.5), normal(d, ff, std=0.5 * ff ** -0.5)
    return w


def _plain_tokens(case, seed):
    """(tokens before the pass, tokens of the pass) of every stream."""
    rng, vocab = _seeds(seed, 3), PLAIN[7]
    got = []
    for q in range(case["streams"]):
        rows = case["rows"] if q == 0 or not case["mixed"] else 1
        got.append((rng.integers(0, vocab, size=case["context"]).tolist(), rng.integers(0, vocab, size=rows).tolist()))
    return got


def _prepare_plain(case, seed):
    s = Opened()
    streams, rows, c = case["streams"], case["rows"], case["context"]
    w = _plain_weights(seed)
    m = s.own(nigenex.build(s.ctx, _plain_config(), lambda name: w[name].view(torch.int16).cpu().numpy().view(np.uint16), c + rows + 16, plain.BF16))
    s.tokens = _plain_tokens(case, seed)
    s.sess = s.own(tsb.Session(s.ctx, m, None, streams, min(rows, 128), step_rows=max(c, streams + rows)))
    for q, (before, _) in enumerate(s.tokens):
        if before:
            s.sess.step([(q, before, [len(before) - 1])])
    s.context = c
    return s


def _run_plain(s):
    logits = s.sess.step([(q, now, [len(now) - 1]) for q, (_, now) in enumerate(s.tokens)])
    for q in range(len(s.tokens)):
        if s.context:
            s.sess.rollback_retaining(s.context, 0, stream=q)
        else:
            s.sess.reset(q)
    return logits


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, int(seed))


def run(state):
    return state.run(state)


def _with_run(kind):
    make, go = globals()["_prepare_" + kind], globals()["_run_" + kind]

    def made(case, seed):
        s = make(case, seed)
        s.run = go
        return s
    return made


for _kind in ("pass", "prefill", "accept", "experts", "plain"):
    globals()["_prepare_" + _kind] = _with_run(_kind)


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    if case["kind"] in ("pass", "prefill"):
        layers, d, nq, nkv, hd, ff, vocab, _, _ = SHAPES[case["shape"]]
        _, per, size = TYPES[case["blocks"]]
        body = layers * d * (hd * (2 * nq + 2 * nkv) + 3 * ff)
        if case["kind"] == "pass":
            n, c, heads = case["streams"] * case["rows"], case["context"], case["streams"] * case["rows"]
            cached = case["streams"] * c * layers * 2 * nkv * hd * 2
            seen = n * c
        else:
            n, heads, cached = case["tokens"] + 1, 2, 0
            seen = n * n / 2
        return {"bytes": (body + vocab * d) / per * size + cached + n * (layers * 2 * nkv * hd * 2 + d / per * size) + heads * vocab * 2,
                "flops": 2.0 * body * n + 2.0 * vocab * d * heads + 4.0 * layers * nq * hd * seen}
    if case["kind"] == "accept":
        rows = case["batch"] * (2 * case["k"] + 1)
        return {"bytes": rows * case["vocab"] * 2.0, "flops": rows * case["vocab"] * (2.0 if case["temperature"] else 1.0)}
    if case["kind"] == "experts":
        e, d, f, n, top = case["experts"], case["width"], case["ffn"], case["tokens"], case["top"]
        met = e * (1 - (1 - top / e) ** n)
        _, per, size = TYPES[case["blocks"]]
        return {"bytes": met * 3 * d * f / per * size + n * d * 6, "flops": 6.0 * n * top * d * f}
    layers, d, nq, nkv, hd, window, ff, vocab = PLAIN
    streams, c = case["streams"], case["context"]
    portions = [case["rows"] if q == 0 or not case["mixed"] else 1 for q in range(streams)]
    body = layers * d * (hd * (2 * nq + nkv) + nq + 3 * ff)
    seen = sum(sum(min(window, c + j + 1) for j in range(r)) for r in portions)
    keys = sum(min(c, window) for _ in portions)
    return {"bytes": 2.0 * (body + vocab * d) + layers * nkv * hd * 2.0 * (keys + sum(portions)) + 4.0 * streams * vocab,
            "flops": 2.0 * body * sum(portions) + 2.0 * vocab * d * streams + 4.0 * layers * nq * hd * seen}


def tolerance(case):
    if case["kind"] == "accept":
        return {"rel": 1e-6, "differ": 0.0}  # sums of f64 in any order; tokens stay
    if case["kind"] == "experts":
        return {"rel": 1e-3, "max": 2e-2}  # f16 activations between two matmuls, f16 results
    if case["kind"] == "plain":
        return {"rel": 1.2e-2, "max": 0.1}  # bfloat16 operands
    return {"rel": 2e-2, "max": 0.15}  # f16 activations and stored sums through all layers


# ------------------------------------------------------------------ the same in 64 bits
_M = 0xFFFFFFFF


def _mix(x):
    x = x ^ (x >> 16)
    x = (x * 0x7FEB352D) & _M
    x = x ^ (x >> 15)
    x = (x * 0x846CA68B) & _M
    return x ^ (x >> 16)


def _half_at(p, at):
    return p[:, at:at + 2].contiguous().view(torch.float16).double()


def _dequantise(blocks, p):
    """[n, bytes] -> [n, values of a block] in 64 bits."""
    n, q = p.shape[0], p.to(torch.int16)
    if blocks == "q4_k":
        s = q[:, 4:16]
        lo, hi = s[:, 0:4], s[:, 4:8]
        sc = torch.cat([lo & 63, (s[:, 8:12] & 15) | ((lo >> 6) << 4)], 1)
        mn = torch.cat([hi & 63, (s[:, 8:12] >> 4) | ((hi >> 6) << 4)], 1)
        w = q[:, 16:].reshape(n, 4, 1, 32)
        v = torch.cat([w & 15, w >> 4], 2).reshape(n, 8, 32).double()
        return (_half_at(p, 0)[:, :, None] * sc.double()[:, :, None] * v - (_half_at(p, 2) * mn.double())[:, :, None]).reshape(n, 256)
    if blocks == "q6_k":
        ql, qh = q[:, :128].reshape(n, 2, 2, 32), q[:, 128:192].reshape(n, 2, 32)
        v = torch.stack([(ql[:, :, 0] & 15) | ((qh & 3) << 4), (ql[:, :, 1] & 15) | (((qh >> 2) & 3) << 4), (ql[:, :, 0] >> 4) | (((qh >> 4) & 3) << 4),
                         (ql[:, :, 1] >> 4) | (((qh >> 6) & 3) << 4)], 2).double() - 32
        sc = p[:, 192:208].view(torch.int8).double().reshape(n, 2, 4, 2, 1)
        return (v.reshape(n, 2, 4, 2, 16) * sc).reshape(n, 256) * _half_at(p, 208)
    if blocks == "q8_0":
        return p[:, 2:].contiguous().view(torch.int8).double() * _half_at(p, 0)
    table = torch.tensor([0, 1, 2, 3, 4, 6, 8, 12, 0, -1, -2, -3, -4, -6, -8, -12], device="cuda", dtype=torch.float64)
    v = torch.cat([q[:, 1:] & 15, q[:, 1:] >> 4], 1).long()
    return table[v] * torch.pow(2.0, q[:, :1].double() - 128.0)


def _times(case, x, rows, p):
    """x [n, columns] times the transposed matrix of blocks p, some rows at a time."""
    cols, size = x.shape[1], p.shape[1]
    step = max(1, (1 << 28) // cols)
    p = p.view(rows, -1)
    return torch.cat([x @ _dequantise(case["blocks"], p[r:r + step].reshape(-1, size)).view(-1, cols).T for r in range(0, rows, step)], 1)


def _cached(layer, which, tokens, width, seed):
    """Row by row what fill_context leaves of a layer's keys (0) or values (1)."""
    i = torch.arange(tokens * width, device="cuda", dtype=torch.int64) + (2 * layer + which) * tokens * width
    zero = torch.zeros(1, device="cuda", dtype=torch.int64)
    h = _mix((i & _M) ^ ((seed * 0x9E3779B9) & _M)) ^ _mix(((i >> 32) + (seed >> 32) + zero) & _M)
    acc = torch.zeros(i.numel(), device="cuda", dtype=torch.float32)
    for k in range(4):
        h = _mix((h + 0x9E3779B9 * (k + 1)) & _M)
        acc += (h >> 8).to(torch.float32) * (1.0 / 16777216.0)
    return ((acc - 2.0) * float(np.float32(1.7320508))).half().double().view(tokens, width)


def _norm(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, positions, theta):
    half = x.shape[-1] // 2
    f = theta ** (-torch.arange(half, device="cuda", dtype=torch.float64) / half)
    a = positions.double()[:, None] * f
    c, s = a.cos()[:, None], a.sin()[:, None]
    lo, hi = x[..., :half], x[..., half:]
    return torch.cat([lo * c - hi * s, hi * c + lo * s], -1)


def _decoder(case, seed, tokens, parents, context, wanted):
    """Logits of the wanted rows: tokens [streams, n] behind `context` filled positions; row j of a stream sees row parents[j] and what
    that one sees."""
    layers, d, nq, nkv, hd, ff, vocab, eps, theta = SHAPES[case["shape"]]
    streams, n = tokens.shape
    mats = {l: {which: (rows, p) for which, rows, _, p in m} for l, m in _matrices(case, int(seed))}
    times = lambda l, which, x: _times(case, x, *mats[l][which])  # noqa: E731
    ids = torch.from_numpy(tokens.reshape(-1).astype(np.int64)).cuda()
    x = _dequantise(case["blocks"], mats[-1][W_EMBED][1].view(vocab, -1)[ids].reshape(-1, TYPES[case["blocks"]][2])).view(-1, d)
    see = torch.zeros(n, n, dtype=torch.bool, device="cuda")
    depth = np.zeros(n, dtype=np.int64)
    for j, p in enumerate(parents):
        if p >= 0:
            see[j], depth[j] = see[p], depth[p] + 1
        see[j, j] = True
    pos = torch.from_numpy(np.tile(context + depth, streams)).cuda()
    mask = torch.cat([torch.ones(n, context, dtype=torch.bool, device="cuda"), see], 1)
    for l in range(layers):
        h, w = _norm(x, eps), l % LAYERS
        q, k, v = (times(w, which, h).view(-1, heads, hd) for which, heads in ((W_Q, nq), (W_K, nkv), (W_V, nkv)))
        q, k = _rotate(q, pos, theta), _rotate(k, pos, theta)
        out = []
        for s in range(streams):
            rows = slice(s * n, (s + 1) * n)
            ks, vs = k[rows], v[rows]
            if context:
                ks, vs = (torch.cat([_cached(l, i, context, nkv * hd, 2000 + int(seed) + 2 * s).view(context, nkv, hd), t]) for i, t in ((0, ks), (1, vs)))
            qs = q[rows].view(n, nkv, nq // nkv, hd)
            score = torch.einsum("ngrd,mgd->grnm", qs, ks) * hd ** -0.5
            prob = torch.softmax(score.masked_fill(~mask, -math.inf), -1)
            out.append(torch.einsum("grnm,mgd->ngrd", prob, vs).reshape(n, nq * hd))
        x = x + times(w, W_O, torch.cat(out))
        h = _norm(x, eps)
        x = x + times(w, W_DOWN, torch.nn.functional.silu(times(w, W_GATE, h)) * times(w, W_UP, h))
    return times(-1, W_LM_HEAD, _norm(x[wanted], eps))


def _exact_pass(case, seed):
    n = case["rows"]
    parents = _tree_parents(n) if case["tree"] else list(range(-1, n - 1))
    y = _decoder(case, seed, _feed(case, seed), parents, case["context"], slice(None))
    if case["streams"] > 1:
        return y.view(case["streams"], n, -1)
    return y if case["tree"] or n > 1 else y[0]


def _exact_prefill(case, seed):
    n = case["tokens"] + 1
    return _decoder(case, seed, _prompt(case, seed)[None], list(range(-1, n - 1)), 0, slice(n - 1, n))[0]


def _shaped(row, case):
    """(probabilities, tokens in rank order) of a row of logits after truncation."""
    x = row.double()
    e = torch.exp(x - x.max())
    order = torch.sort(x, descending=True, stable=True)[1]
    keep = torch.ones_like(order, dtype=torch.bool)
    if 0 < case["top_k"] < x.numel():
        keep[case["top_k"]:] = False
    if case["top_p"] > 0:
        c = torch.cumsum(e[order] / e.sum(), 0)
        keep &= torch.cat([torch.ones(1, dtype=torch.bool, device="cuda"), c[:-1] < case["top_p"]])
    if case["min_p"] > 0:
        keep &= e[order] >= case["min_p"]
    support = order[keep]
    w = torch.zeros_like(e)
    w[support] = e[support] ** (1.0 / case["temperature"])
    return w / w.sum(), support


def _drawn(p, support, u):
    """(token, distance to the nearer bound) of the draw of u in [0, 1) over p's tokens in rank order."""
    c = torch.cumsum(p[support], 0)
    i = min(int((c <= u).sum()), support.numel() - 1)
    lo = float(c[i - 1]) if i else 0.0
    return int(support[i]), min(u - lo, float(c[i]) - u)


def _exact_accept(case, seed):
    target, draft, props, uniforms = _accept_inputs(case, seed)
    b, k = case["batch"], case["k"]
    decided, margins = np.zeros((b, 19), dtype=np.int32), np.zeros((b, 2))
    unit = ((uniforms.cpu().numpy().view(np.uint64) >> np.uint64(11)).astype(np.float64)) * 2.0 ** -53
    props = props.cpu().numpy()
    for s in range(b):
        accepted, draws, close, rejected, bound = 0, 0, math.inf, False, 16.0
        for i in range(k):
            x = int(props[s, i])
            if case["temperature"] == 0:
                if int(target[s, i].float().argmax()) != x:
                    break
                accepted += 1
                continue
            p, q = _shaped(target[s, i], case), _shaped(draft[s, i], case)
            r = unit[s, draws]
            draws += 1
            close = min(close, abs(r * float(q[0][x]) - float(p[0][x])))
            if r * float(q[0][x]) <= float(p[0][x]):
                accepted += 1
            else:
                rejected = True
                break
        if case["temperature"] == 0:
            token = int(target[s, accepted].float().argmax())
        else:
            p = _shaped(target[s, accepted], case)
            if rejected:
                left = torch.clamp(p[0] - q[0], min=0.0)
                if float(left.sum()) >= 1e-12:
                    p = (left / left.sum(), p[1][left[p[1]] > 0])
            token, bound = _drawn(*p, unit[s, draws])
            draws += 1
        tokens = props[s, :accepted].tolist() + [token]
        decided[s, :2], decided[s, 2:18], decided[s, 18] = (accepted, draws), tokens + [-1] * (16 - len(tokens)), 0
        margins[s] = close, bound
    return {"decided": decided, "margins": margins}


def _exact_experts(case, seed):
    gu, dn, x, residual, ids, w = _experts_inputs(case, seed)
    e, d, f = case["experts"], case["width"], case["ffn"]
    size = TYPES[case["blocks"]][2]
    gu, dn = gu[:-256].view(e, -1, size), dn[:-256].view(e, -1, size)
    y = residual.double()
    for i in range(e):
        at, slot = torch.nonzero(ids == i, as_tuple=True)
        if at.numel() == 0:
            continue
        h = x[at].double() @ _dequantise(case["blocks"], gu[i]).view(2 * f, d).T
        a = torch.nn.functional.silu(h[:, :f]) * h[:, f:]
        y.index_add_(0, at, (a @ _dequantise(case["blocks"], dn[i]).view(d, f).T) * w[at, slot].double()[:, None])
    return y


def _exact_plain(case, seed):
    layers, d, nq, nkv, hd, window, ff, vocab = PLAIN
    w = {k: v.double() for k, v in _plain_weights(seed).items()}
    got = []
    for before, now in _plain_tokens(case, seed):
        t = before + now
        n = len(t)
        x = w["embed"][torch.tensor(t, device="cuda")]
        dist = torch.arange(n, device="cuda")[:, None] - torch.arange(n, device="cuda")[None]
        mask, far = (dist >= 0) & (dist < window), dist.clamp(min=0).double()
        for i in range(layers):
            p = "l%d." % i
            h = _norm(x, 1e-6) * w[p + "norm1"]
            m = h + (torch.cat([torch.zeros_like(h[:1]), h[:-1]]) - h) * w[p + "shift"]
            q, k = (m @ w[p + "mix.q"].T).view(n, nq, hd), (m @ w[p + "mix.k"].T).view(n, nkv, hd)
            out = torch.empty_like(q)
            for j in range(nq):
                kj = k[:, j // (nq // nkv)]
                s = 50.0 * torch.tanh(q[:, j] @ kj.T * hd ** -0.5 / 50.0) - w[p + "mix.r1"][j] * torch.log(1.0 + w[p + "mix.r2"][j] * far)
                out[:, j] = torch.softmax(s.masked_fill(~mask, -math.inf), -1) @ kj
            out = out * torch.sigmoid(m @ w[p + "mix.g"].T)[:, :, None]
            a = torch.nn.functional.gelu(h @ w[p + "mlp.gate"].T, approximate="tanh") * (h @ w[p + "mlp.up"].T)
            x = x + out.reshape(n, -1) @ w[p + "mix.o"].T + a @ w[p + "mlp.down"].T
        h = _norm(x[-1:], 1e-6) * w["final.norm"]
        got.append(30.0 * torch.tanh(h @ w["head"].T / 30.0))
    return torch.cat(got)


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, int(seed))
