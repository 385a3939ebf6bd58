"""Workloads of the attention path that its speed is judged on.

One pass is what an engine does for its attention layers: the prologue (RMSNorm, RoPE, K and V into the cache)
and then the attention over the cache. Decode steps write 1 to 4 new tokens of one sequence, or of a batch over a
page pool; prefill passes write a chunk of up to 2,048 tokens. The model's shape is 24 query heads over 4 KV heads
of dimension 256, 17 caches; with 2 KV heads and 12 query heads it is one card's half, with 1 and 6 one GPU's quarter.
"""
import importlib
import math
import random

import torch

q27 = importlib.import_module("qwen27-engine_b200")

AD, GQA, PAGE = 256, 6, 256
KQ_SCALE = 1.0 / 16.0
EPS = 1e-6
THETA_SCALE = 10000000.0 ** (-2.0 / 64)


def decode(name, T, n, nkvh=4, q8=True, layers=1, graph=False, q8_1=False):
    """n positions, the T new ones included. graph: the step of all layers is replayed from a CUDA graph, which is
    how an engine issues it; otherwise call by call. q8_1: the output quantised for the next matrix product."""
    c = {"kind": "decode", "T": T, "n": n, "nkvh": nkvh, "q8": q8, "layers": layers, "graph": graph, "q8_1": q8_1}
    return dict(c, name=name) if name else c


def batch(name, B, T, lo, hi, order):
    """B sequences of lo to hi positions, drawn by `order`, over 256-position pages in random order."""
    c = {"kind": "batch", "B": B, "T": T, "lo": lo, "hi": hi, "order": order}
    return dict(c, name=name) if name else c


def prefill(name, M, pos0, nkvh=4, q8=True, f16_qk=False):
    """M query tokens behind pos0 earlier ones. f16_qk: on a q8_0 cache, the f16 form of Q K^T (Q27_ATTN_I8=0)."""
    c = {"kind": "prefill", "M": M, "pos0": pos0, "nkvh": nkvh, "q8": q8, "f16_qk": f16_qk}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the first generated token behind a short prompt, one layer, plain calls: launches and host time are all of it
        decode("first_token", 1, 257),
        # speculative verification early in a chat, all layers as one graph, output quantised for the next GEMV
        decode("verify_1k", 4, 1024, layers=17, graph=True, q8_1=True),
        # the same behind a long document, the ordinary length of the headline range
        decode("verify_32k", 4, 32768, layers=17, graph=True),
        # f16 cache, one card's half of the heads, an odd length and three tokens
        decode("verify_30k_f16", 3, 30011, nkvh=2, q8=False, layers=17, graph=True),
        # the longest context, one layer, plain calls
        decode("verify_150k", 4, 150000),
        # a batch of short chats, one token each
        batch("batch_small", 8, 1, 64, 8192, 1),
        # a full batch of 64 long sequences with verification
        batch("batch_64", 64, 4, 1024, 131072, 2),
        # the first chunk of a prompt
        prefill("prefill_start", 2048, 0),
        # a user's next turn, a short odd-sized message behind a long conversation
        prefill("prefill_turn", 131, 30011),
        # a chunk in the middle of a document with the f16 form of Q K^T
        prefill("prefill_32k_f16qk", 2048, 32768, f16_qk=True),
        # a chunk in the middle of a document on an f16 cache, the last and partly filled one
        prefill("prefill_20k_f16", 1537, 20011, q8=False),
        # the last chunk of the longest prompt
        prefill("prefill_148k", 2048, 148000),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "batch", "prefill", "prefill"])
    nkvh = rng.choice([4, 4, 2, 1])
    if kind == "decode":
        n, q8 = _log(rng, 64, 150000), rng.random() < 0.75
        layers = 17 if n < 40000 else 4
        graph = rng.random() < 0.5
        return decode(None, rng.randint(1, 4), n, nkvh, q8, layers if graph else 1, graph, rng.random() < 0.25)
    if kind == "batch":
        B, hi = _log(rng, 1, 64), _log(rng, 512, 131072)
        return batch(None, B, rng.randint(1, 4), max(16, hi // rng.choice([4, 32, 128])), hi, rng.randrange(1 << 20))
    q8 = rng.random() < 0.75
    pos0 = 0 if rng.random() < 0.15 else _log(rng, 100, 148000)
    return prefill(None, _log(rng, 16, 2048), pos0, nkvh, q8, q8 and rng.random() < 0.3)


def _lengths(case):
    """Sequence lengths of a batch, spread evenly between lo and hi (they belong to the case, not to the seed)."""
    r = random.Random(case["order"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["B"])]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _fill(values, scales, gen):
    """values int8 [rows][256], scales f16 [rows][8]: N(0, 1) rows as q8_0 (d = amax / 127 per 32 values)."""
    step = 1 << 18
    for a in range(0, values.shape[0], step):
        b = min(values.shape[0], a + step)
        x = torch.randn((b - a, 8, 32), generator=gen, device="cuda")
        d = x.abs().amax(-1, keepdim=True) / 127.0
        values[a:b] = (x / d).round_().to(torch.int8).view(b - a, AD)
        scales[a:b] = d.view(b - a, 8).half()


def _parts(buf, outer, nkvh, rows):
    """The values [outer][nkvh][rows][256] and scales [..][8] of a q8_0 cache (outer = 1) or page pool."""
    nv = outer * nkvh * rows * AD
    return buf[:nv].view(torch.int8).view(outer, nkvh, rows, AD), buf[nv:].view(torch.float16).view(outer, nkvh, rows, 8)


def _cache(nkvh, n_ctx, q8, gen):
    c = torch.empty(q27.kv_cache_bytes(nkvh, n_ctx, q8), dtype=torch.uint8, device="cuda")
    if q8:
        v, s = _parts(c, 1, nkvh, n_ctx)
        _fill(v.view(-1, AD), s.view(-1, 8), gen)
    else:
        c.view(torch.float16).copy_(torch.randn(c.numel() // 2, generator=gen, device="cuda"))
    return c


def _new_rows(c, nkvh, n_ctx, q8, a, b):
    """Views of the cache rows that a pass writes."""
    if q8:
        v, s = _parts(c, 1, nkvh, n_ctx)
        return [v[0, :, a:b], s[0, :, a:b]]
    return [c.view(torch.float16).view(nkvh, n_ctx, AD)[:, a:b]]


def _tokens(lead, nkvh, gen):
    """Query + gate, K and V of new tokens, and buffers for the results."""
    nqh = nkvh * GQA
    rn = lambda *shape: torch.randn(shape, generator=gen, device="cuda")  # noqa: E731
    return {"qg": rn(*lead, nqh, 2 * AD), "k": rn(*lead, nkvh, AD), "v": rn(*lead, nkvh, AD),
            "q_norm": 1 + 0.1 * rn(AD), "k_norm": 1 + 0.1 * rn(AD),
            "qn": torch.empty((*lead, nqh, AD), device="cuda"), "o": torch.empty((*lead, nqh, AD), device="cuda")}


def prepare(case, seed):
    s = _state(case, seed)
    if case.get("graph"):
        _decode_layers(s)  # once before the capture: workspace and one-time set-up
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            _decode_layers(s)
    return s


def _state(case, seed):
    gen = _gen(seed)
    if case["kind"] == "batch":
        return _prepare_batch(case, gen)
    nkvh, q8 = case["nkvh"], case["q8"]
    n = case["n"] if case["kind"] == "decode" else case["pos0"] + case["M"]
    T = case["T"] if case["kind"] == "decode" else case["M"]
    n_ctx = -(-n // 256) * 256 + 256
    layers = []
    for _ in range(case.get("layers", 1)):
        w = _tokens((T,), nkvh, gen)
        w["kc"], w["vc"] = _cache(nkvh, n_ctx, q8, gen), _cache(nkvh, n_ctx, q8, gen)
        w["xq"] = w["xd"] = None
        if case.get("q8_1"):
            w["xq"] = torch.empty(w["o"].shape, dtype=torch.int8, device="cuda")
            w["xd"] = torch.empty(w["o"].numel() // 32, device="cuda")
            w["o"] = None
        layers.append(w)
    s = {"case": case, "layers": layers, "T": T, "nqh": nkvh * GQA, "nkvh": nkvh, "n_ctx": n_ctx, "q8": q8,
         "pos": torch.tensor([n - T], dtype=torch.int32, device="cuda")}
    outs = {"result": [w[k] for w in layers for k in ("o", "xq", "xd") if w[k] is not None]}
    if len(layers) == 1:  # of many layers the attention outputs alone: each depends on its qn and new rows
        outs["qn"] = layers[0]["qn"]
        outs["rows"] = [r for c in (layers[0]["kc"], layers[0]["vc"]) for r in _new_rows(c, nkvh, n_ctx, q8, n - T, n)]
    s["outs"] = outs
    return s


def _prepare_batch(case, gen):
    B, T, nkvh = case["B"], case["T"], 4
    lens = _lengths(case)
    pages = [-(-n // PAGE) for n in lens]
    n_pages, max_pages = sum(pages), max(pages)
    s = {"case": case, "nkvh": nkvh, "nqh": nkvh * GQA, "n_pages": n_pages, "max_pages": max_pages, "max_len": max(lens)}
    # pages in random order; the pages handed out last, which receive the new rows, are the last B of the pool
    order = (torch.randperm(n_pages - B, generator=gen, device="cuda").tolist() if n_pages > B else []) + list(range(n_pages - B, n_pages))
    table, at = torch.full((B, max_pages), -1, dtype=torch.int32), 0
    for b, p in enumerate(pages):
        table[b, :p] = torch.tensor(order[at:at + p - 1] + [n_pages - B + b], dtype=torch.int32)
        at += p - 1
    s["table"], s["lens"] = table.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")
    outs = {}
    for which in ("kpool", "vpool"):
        pool = torch.empty(q27.kv_pool_bytes(nkvh, n_pages), dtype=torch.uint8, device="cuda")
        v, d = _parts(pool, n_pages, nkvh, PAGE)
        _fill(v.view(-1, AD), d.view(-1, 8), gen)
        s[which] = pool
        outs[which] = [v[n_pages - B:], d[n_pages - B:]]
    s.update(_tokens((B, T), nkvh, gen))
    s["outs"] = dict(outs, o=s["o"], qn=s["qn"])
    return s


def _decode_layers(s):
    for w in s["layers"]:
        q27.attn_prep(w["qg"], w["k"], w["v"], w["q_norm"], w["k_norm"], w["qn"], w["kc"], w["vc"], s["pos"], s["T"], EPS,
                      THETA_SCALE, s["nqh"], s["nkvh"], s["n_ctx"], s["q8"])
        q27.attn_decode(w["qn"], w["qg"], w["kc"], w["vc"], w["o"], w["xq"], w["xd"], s["pos"], s["T"], KQ_SCALE, s["nqh"],
                        s["nkvh"], s["n_ctx"], s["q8"])


def run(s):
    c = s["case"]
    if c["kind"] == "decode":
        if c["graph"]:
            s["graph"].replay()
        else:
            _decode_layers(s)
    elif c["kind"] == "batch":
        q27.attn_prep_paged(s["qg"], s["k"], s["v"], s["q_norm"], s["k_norm"], s["qn"], s["kpool"], s["vpool"], s["table"],
                            s["lens"], c["B"], c["T"], EPS, THETA_SCALE, s["nqh"], s["nkvh"], s["n_pages"], s["max_pages"])
        q27.attn_decode_paged(s["qn"], s["qg"], s["kpool"], s["vpool"], s["table"], s["lens"], s["o"], c["B"], c["T"],
                              KQ_SCALE, s["nqh"], s["nkvh"], s["n_pages"], s["max_pages"], s["max_len"])
    else:
        w = s["layers"][0]
        q27.attn_prep(w["qg"], w["k"], w["v"], w["q_norm"], w["k_norm"], w["qn"], w["kc"], w["vc"], s["pos"], s["T"], EPS,
                      THETA_SCALE, s["nqh"], s["nkvh"], s["n_ctx"], s["q8"])
        if c["f16_qk"]:  # a process-wide choice: put back, since other workloads share the process
            q27.set_prefill_kernel(2)
        try:
            q27.attn_prefill(w["qn"], w["qg"], w["kc"], w["vc"], w["o"], s["pos"], c["M"], KQ_SCALE, s["nqh"], s["nkvh"],
                             s["n_ctx"], s["q8"], c["pos0"])
        finally:
            if c["f16_qk"]:
                q27.set_prefill_kernel(0)
    return s["outs"]


def _norm_rope(x, w, pos):
    """RMSNorm and rotary embedding of rows [token][head][256] at positions [token]; pairs (j, j + 32), j < 32."""
    x = x.double()
    x = x / (x.square().mean(-1, keepdim=True) + EPS).sqrt() * w.double()
    theta = pos.double()[:, None, None] * THETA_SCALE ** torch.arange(32, dtype=torch.float64, device=x.device)
    a, b = x[..., :32], x[..., 32:64]
    return torch.cat([a * theta.cos() - b * theta.sin(), a * theta.sin() + b * theta.cos(), x[..., 64:]], -1)


def _stored(x, q8):
    """Rows as the cache gives them back: f16, or q8_0 with scales amax / 127 in f16 (and these scales)."""
    if not q8:
        return x.half().double(), None
    b = x.reshape(*x.shape[:-1], 8, 32)
    d = b.abs().amax(-1, keepdim=True) / 127.0
    return (torch.round(b / d) * d.half().double()).reshape(x.shape), d[..., 0]


def _attend(qn, qg, k, v, pos):
    """One sequence: qn [T][nqh][256], k and v [nkvh][n][256] (the new rows included), pos [T]; the gated output."""
    T, nkvh, n = qn.shape[0], k.shape[0], k.shape[1]
    o = torch.empty((T, nkvh * GQA, AD), dtype=torch.float64, device=qn.device)
    step = max(1, min(T, (1 << 28) // (GQA * n)))  # scores of at most 2 GB at a time
    at = torch.arange(n, device=qn.device)
    for h in range(nkvh):
        for a in range(0, T, step):
            q = qn[a:a + step, h * GQA:(h + 1) * GQA]
            sc = (q.reshape(-1, AD) @ k[h].T).view(q.shape[0], GQA, n).mul_(KQ_SCALE)
            sc.masked_fill_(at > pos[a:a + step, None, None], -math.inf)
            o[a:a + step, h * GQA:(h + 1) * GQA] = (torch.softmax(sc, -1).view(-1, n) @ v[h]).view(q.shape)
    return o * torch.sigmoid(qg[..., AD:].double())


def _dequant(values, scales):
    return (values.double().view(*values.shape[:-1], 8, 32) * scales.double()[..., None]).view(values.shape)


def exact(case, seed):
    """What run returns, in float64 from the same inputs (RoPE angles too). No value for whole numbers."""
    s = _state(case, seed)
    return _exact_batch(s) if case["kind"] == "batch" else _exact_one(s)


def _exact_one(s):
    T, nkvh, n_ctx, q8 = s["T"], s["nkvh"], s["n_ctx"], s["q8"]
    first = int(s["pos"][0])
    pos = torch.arange(first, first + T, device="cuda")
    outs = {"result": []}
    for w in s["layers"]:
        qn, rows, kv = _norm_rope(w["qg"][..., :AD], w["q_norm"], pos), [], []
        for c, x in ((w["kc"], _norm_rope(w["k"], w["k_norm"], pos)), (w["vc"], w["v"].double())):
            x = x.transpose(0, 1)  # [nkvh][T][256], the cache's order
            back, d = _stored(x, q8)
            old = _dequant(*_parts(c, 1, nkvh, n_ctx))[0] if q8 else c.view(torch.float16).view(nkvh, n_ctx, AD).double()
            old[:, first:first + T] = back
            kv.append(old[:, :first + T])
            rows += [None, d] if q8 else [x]
        o = _attend(qn, w["qg"], *kv, pos)
        if s["case"].get("q8_1"):
            outs["result"] += [None, o.reshape(-1, 32).abs().amax(-1) / 127.0]
        else:
            outs["result"].append(o)
        outs["qn"], outs["rows"] = qn, rows
    return outs if len(s["layers"]) == 1 else {"result": outs["result"]}


def _exact_batch(s):
    B, T, nkvh = s["case"]["B"], s["case"]["T"], s["nkvh"]
    pools = [_parts(s[which], s["n_pages"], nkvh, PAGE) for which in ("kpool", "vpool")]
    o, qns = torch.empty(s["o"].shape, dtype=torch.float64, device="cuda"), torch.empty(s["qn"].shape, dtype=torch.float64, device="cuda")
    for b, n in enumerate(s["lens"].tolist()):
        pos = torch.arange(n - T, n, device="cuda")
        qns[b] = _norm_rope(s["qg"][b][..., :AD], s["q_norm"], pos)
        pg, kv = s["table"][b, :-(-n // PAGE)].long(), []
        for (vals, scales), x in zip(pools, (_norm_rope(s["k"][b], s["k_norm"], pos), s["v"][b].double())):
            whole = _dequant(vals[pg], scales[pg]).transpose(0, 1).reshape(nkvh, -1, AD)
            whole[:, n - T:n] = _stored(x.transpose(0, 1), True)[0]
            kv.append(whole[:, :n])
        o[b] = _attend(qns[b], s["qg"][b], *kv, pos)
    return {"kpool": [None, None], "vpool": [None, None], "o": o, "qn": qns}


def work(case):
    """Each K and V row read once, the new ones written once; per token and head 512 query, gate and 256 output values in
    and out, the normalised query written and read. 4 * 256 operations per (query row, visible position)."""
    nkvh = 4 if case["kind"] == "batch" else case["nkvh"]
    row = 2 * nkvh * (2 * AD if not case.get("q8", True) else AD + 16)
    if case["kind"] == "batch":
        lens, T = _lengths(case), case["T"]
        positions, tokens, layers = sum(lens), case["B"] * T, 1
        pairs = sum(sum(n - T + t + 1 for t in range(T)) for n in lens)
    else:
        T = case["T"] if case["kind"] == "decode" else case["M"]
        n = case["n"] if case["kind"] == "decode" else case["pos0"] + T
        positions, tokens, layers = n, T, case.get("layers", 1)
        pairs = T * (n - T) + T * (T + 1) // 2
    nqh = nkvh * GQA
    per_token = nqh * AD * (2 + 2 + 1) * 4 + 2 * nkvh * AD * 4 + row
    return {"bytes": layers * (positions * row + tokens * per_token), "flops": layers * pairs * nqh * 4 * AD}


def tolerance(case):
    """Against a float64 statement of the same operator on the same cache bytes the path is off by 2.5e-4 to 4.2e-4 in
    the 2-norm and by up to 5e-3 of the RMS in single values: P and the dequantised V are rounded to f16 (2^-11 of a
    value), P against a running maximum that moves with the order of the tiles. Four times that is stated. Whole values
    are q8_0 / q8_1 bytes: a value near a rounding tie may fall either way, in q8_1 outputs (steps of 1/127 of the
    largest of 32 values, each off by some 1e-4 of it) in up to one of a hundred."""
    return {"rel": 1.6e-3, "max": 1.6e-2, "differ": 1e-2 if case.get("q8_1") else 1e-4}
