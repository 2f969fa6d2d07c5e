"""Serving iterations that a user of the engines runs: one call of ``Engine.run`` on a batch in the scheduler's layout.

A case names a model whose sizes the package ships, the dense batch the engine is configured for, and what the batch
holds: ``decode`` requests that add one token to ``ctx_lo`` ... ``ctx_hi`` cached ones, and ``prompts`` portions of
about ``prompt`` tokens, the first of them behind ``past`` tokens that earlier iterations have cached (chunked prefill).
Models keep their widths, heads, vocabulary and options and run their first ``LAYERS`` layers. Weights and cached
keys are random; the output head is tied to the embedding, so that logits have a clear winner like a trained model's.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

LAYERS = 4
PAGE = 16
LLAMA = {   # width, feed-forward, query heads, KV heads, vocabulary, rotary base, norm epsilon, bias of the QKV projection
    "llama3-8B": (4096, 14336, 32, 8, 128256, 500000.0, 1e-5, False),
    "llama2-70B": (8192, 28672, 64, 8, 32000, 10000.0, 1e-5, False),
    "qwen2-72B": (8192, 29568, 64, 8, 152064, 1000000.0, 1e-6, True),
}
HEAD_DIM = 128
VOLARAX = dict(width=4096, ff=14336, vocab=128256, heads=32, dim=128, rank=512, window=1024, m_heads=8, m_dim=256, m_vdim=512,
               cap=15.0, eps=1e-5)


# ---- cases -------------------------------------------------------------------------------------------------------
def _case(name, model, dense, decode=0, ctx=(0, 0), prompts=0, prompt=0, past=0):
    return dict(name=name, model=model, dense=dense, decode=decode, ctx_lo=ctx[0], ctx_hi=ctx[1], prompts=prompts,
                prompt=prompt, past=past)


def listed():
    return [
        # one user's chat: a single token, everything is launches and the weights' way through the chip
        _case("8B decode 1", "llama3-8B", 2048, decode=1, ctx=(900, 900)),
        # light online traffic, contexts of very different length
        _case("8B decode 24", "llama3-8B", 2048, decode=24, ctx=(100, 6000)),
        # offline generation without new prompts
        _case("8B decode 256", "llama3-8B", 2048, decode=256, ctx=(200, 2000)),
        # the first token of one short question
        _case("8B prompt 333", "llama3-8B", 2048, prompts=1, prompt=333),
        # a full dense batch of 1024-token prompts and 512-token answers: the shipped configuration's steady state
        _case("8B steady 2048", "llama3-8B", 2048, decode=683, ctx=(1024, 1536), prompts=2, prompt=682),
        # a long document: the second 4096 tokens of a prompt
        _case("8B long prompt", "llama3-8B", 4096, prompts=1, prompt=4096, past=4096),
        # the headline workload on one GPU, dense batch 256
        _case("70B steady 256", "llama2-70B", 256, decode=170, ctx=(1024, 1536), prompts=1, prompt=86, past=512),
        # prompts of a batch job on a large model
        _case("70B prompts", "llama2-70B", 2048, prompts=2, prompt=1000),
        # a large model with biases under moderate traffic
        _case("72B decode 48", "qwen2-72B", 1024, decode=48, ctx=(200, 3000)),
        # the layer-list family: latent attention with a window beside a recurrence
        _case("volarax decode 96", "volarax-8B", 2048, decode=96, ctx=(200, 4000)),
        _case("volarax mixed", "volarax-8B", 2048, decode=40, ctx=(100, 2000), prompts=3, prompt=600),
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model = rng.choice(["llama3-8B", "llama3-8B", "llama2-70B", "qwen2-72B", "volarax-8B"])
    dense = rng.choice([1024, 2048, 4096] if model == "llama3-8B" else [256, 1024, 2048] if model != "volarax-8B" else [2048])
    kind = rng.choice(["decode", "prompt", "mixed"])
    decode = prompts = prompt = past = lo = hi = 0
    if kind != "prompt":
        decode = log(1, min(512, dense) if model != "volarax-8B" else 200)
        lo = log(50, 1500)
        hi = max(lo, log(100, 3000))
    if kind != "decode":
        prompts = rng.choice([1, 1, 2, 3])
        prompt = log(17 if model != "volarax-8B" else 150, max(18, (dense - decode) // (2 if prompts > 1 else 1)))
        most = dense if model == "llama3-8B" else min(dense, 1800)
        prompt = max(2, min(prompt, (most - decode) // prompts))
        past = log(16, 4000) if model != "volarax-8B" and rng.random() < 0.4 else 0
    c = _case("", model, dense, decode, (lo, hi), prompts, prompt, past)
    del c["name"]
    return c


def _spans(case):
    """[(cached tokens, new tokens)] of the batch's requests."""
    r = random.Random("%d %d %d %d %d" % (case["decode"], case["ctx_lo"], case["ctx_hi"], case["prompts"], case["prompt"]))
    lo, hi = case["ctx_lo"], case["ctx_hi"]
    spans = [(int(round(math.exp(r.uniform(math.log(lo), math.log(hi))))), 1) for _ in range(case["decode"])]
    left = min(case["prompts"] * case["prompt"], case["dense"] - case["decode"])
    for i in range(case["prompts"]):
        last = i + 1 == case["prompts"]
        n = left if last else max(2, min(int(case["prompt"] * r.uniform(0.6, 1.4)), left - 2 * (case["prompts"] - 1 - i)))
        spans.append((case["past"] if i == 0 else 0, n))
        left -= n
    return spans


def _tokens(case, seed, vocab):
    g = np.random.default_rng(seed)
    return [g.integers(0, vocab, n).astype(np.int32) for _, n in _spans(case)]


# ---- weights and cached tokens -------------------------------------------------------------------------------------
class _Random:
    """Tensors on the GPU, in the order they are asked for."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def __call__(self, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        return torch.empty(*shape, dtype=dtype, device="cuda").normal_(mean, std, generator=self.g)


def _llama_tensors(model, seed):
    W, F, H, G, V, _, _, bias = LLAMA[model]
    rn = _Random(seed)
    mat = lambda rows, cols: rn(rows, cols, std=cols ** -0.5)
    layers = [dict(wqkv=mat((H + 2 * G) * HEAD_DIM, W),                              # rows: keys, values, queries
                   wo=mat(W, H * HEAD_DIM), wg=mat(F, W), wu=mat(F, W), wd=mat(W, F),
                   ln_attn=rn(W, std=0.05, mean=1.0), ln_ffn=rn(W, std=0.05, mean=1.0),
                   bqkv=rn((H + 2 * G) * HEAD_DIM, std=0.1) if bias else None) for _ in range(LAYERS)]
    embed = rn(V, W)
    return layers, embed, embed * 0.02, rn(W, std=0.05, mean=1.0)


def _volarax_shapes():
    v = VOLARAX
    W, H, d, r, F = v["width"], v["heads"], v["dim"], v["rank"], v["ff"]
    mk, mv = v["m_heads"] * v["m_dim"], v["m_heads"] * v["m_vdim"]
    out = {"embed": (v["vocab"], W)}
    for n in ("embed.norm", "final.norm"):
        out.update({n: (W,), n + ".b": (W,)})
    for i in range(LAYERS):
        p = "l%d." % i
        for n in ("norm1", "norm1b", "norm2", "norm2b"):
            out.update({p + n: (W,), p + n + ".b": (W,)})
        out.update({p + "mlp.gate": (F, W), p + "mlp.up": (F, W), p + "mlp.down": (W, F)})
        if i % 2 == 0:
            mix = dict(q=(H * d, W), dkv=(r, W), uk=(H * d, r), uv=(H * d, r), sink=(H,), o=(W, H * d))
            mix["dkv.norm"] = (r,)
        else:
            mix = dict(q=(mk, W), k=(mk, W), v=(mv, W), g=(mv, W), o=(W, mv), norm=(mv,), i=(v["m_heads"], W), f=(v["m_heads"], W))
            mix.update({"i.b": (v["m_heads"],), "f.b": (v["m_heads"],)})
        out.update({p + "mix." + n: s for n, s in mix.items()})
    return out


def _volarax_tensors(seed):
    rn, out = _Random(seed), {}
    for name, shape in _volarax_shapes().items():
        if name == "embed":
            out[name] = rn(*shape)
        elif len(shape) == 2:
            out[name] = rn(*shape, std=shape[1] ** -0.5)
        elif name.endswith(".f.b"):                      # forget gates that let the state live for a while
            out[name] = rn(*shape, std=1.0, mean=3.0)
        else:                                            # norms around one; biases and sinks around zero
            out[name] = rn(*shape, std=0.1, mean=0.0 if name.endswith(".b") or "sink" in name else 1.0)
    out["head"] = out["embed"] * 0.02
    return out


def _pages(n):
    return (n + PAGE - 1) // PAGE


def _context(seed, layer, shape):
    """What a layer's cache holds of all requests, page by page in their order."""
    return _Random(1000 * seed + layer)(*shape)


def _recurrent(seed, layer, requests):
    """State of an mLSTM layer that requests with earlier tokens go on from: (S, n); its scale m is zero."""
    rn, v = _Random(1000 * seed + 500 + layer), VOLARAX
    return [rn(requests, v["m_heads"], *tail, std=2.0, dtype=torch.float32) for tail in ((v["m_dim"], v["m_vdim"]), (v["m_dim"],))]


# ---- the framework's part ------------------------------------------------------------------------------------------
def prepare(case, seed):
    """An engine with its weights and filled cache, and the batch that the scheduler has formed."""
    from nanoflow_b200.config import make_config, parse_config
    from nanoflow_b200.models.registry import family_of
    from nanoflow_b200.serving import DistKVCache, DistKVPool, Portion, StateSlotPool, plan_portions

    spans, llama = _spans(case), case["model"] in LLAMA
    pages = sum(_pages(c + n) for c, n in spans) + 16
    raw = make_config(case["model"], global_batch_size=case["dense"], num_pages=pages, pipeline_type="NON_OVERLAP_LOCAL")
    if llama:
        raw["model"]["num_hidden_layers"] = raw["model_configs"]["run_layer"] = LAYERS
    else:
        raw["model"]["layers"] = raw["model"]["layers"][:LAYERS]
        raw["model_configs"]["max_batch_size"] = 256
    cfg = parse_config(raw)
    device = torch.device("cuda", torch.cuda.current_device())
    if llama:
        from nanoflow_b200.models.llama import LayerWeights, RankWeights
        layers, embed, head, norm = _llama_tensors(case["model"], seed)
        weights = RankWeights(embed=embed, norm=norm, lm_head=head, layers=[LayerWeights(**t) for t in layers])
    else:
        from nanoflow_b200.models.volarax import weights_from_tensors
        weights = weights_from_tensors(cfg.model, _volarax_tensors(seed).__getitem__, device)
    engine = family_of(raw["model"]).engine(cfg, weights, device=device, executor="graph")

    m = engine.model
    pool = DistKVPool(m.run_layers, m.num_kv_heads, m.head_dim, pages, PAGE, 1)
    slots = None if llama else StateSlotPool(256)
    portions, held, at = [], [], 0
    for (ctx, n), ids in zip(spans, _tokens(case, seed, m.vocab_size)):
        kv = DistKVCache(pool, slots)
        kv.allocate_tokens(ctx + n)
        held.append(np.array(kv.indices))
        portions.append(Portion(kv, ids, [n - 1]))
    where = torch.from_numpy(np.concatenate(held)).long().to(device)
    for layer, cache in enumerate(engine.bufs.kv_pool if llama else engine.pools):
        if cache is not None:
            cache[where] = _context(seed, layer, (len(where), *cache.shape[1:]))
        else:
            S, n = _recurrent(seed, layer, len(spans))
            engine.state[layer][0][:len(spans)], engine.state[layer][1][:len(spans)] = S, n[:, :, None]
    if not llama:
        for p in portions:                               # pages that no window reaches are given back
            p.kv.trim(m.first_seen(p.kv.seqlen - len(p.tokens)))
    plan = plan_portions(portions, tile_tokens=max(1, 128 // m.group_size))
    torch.cuda.synchronize()
    return dict(engine=engine, plan=plan, rows=len(spans), kv=engine.bufs.kv_pool[-1] if llama else None)


def run(state):
    """One iteration: logits of every request's last token, the tokens sampled from them, and for the Llama models the last
    layer's cache with the new keys and values."""
    engine = state["engine"]
    tokens = engine.run(state["plan"])
    out = dict(logits=engine.bufs.logits[:state["rows"], :engine.model.vocab_size], tokens=tokens)
    if state["kv"] is not None:
        out["kv"] = state["kv"]
    return out


def _pairs(spans, window=0):
    """(query, key) pairs that attention looks at, and keys that some query sees."""
    if not window:
        return sum(n * c + n * (n + 1) // 2 for c, n in spans), sum(c + n for c, n in spans)
    return (sum(sum(min(c + t + 1, window) for t in range(n)) for c, n in spans), sum(min(c + n, window + n - 1) for c, n in spans))


def work(case):
    spans = _spans(case)
    T, B = sum(n for _, n in spans), len(spans)
    if case["model"] in LLAMA:
        W, F, H, G, V, _, _, _ = LLAMA[case["model"]]
        matrices = LAYERS * (W * (2 * H + 2 * G) * HEAD_DIM + 3 * W * F)
        pairs, keys = _pairs(spans)
        flops = 2.0 * T * matrices + 2.0 * B * W * V + 4.0 * LAYERS * pairs * H * HEAD_DIM
        cache = LAYERS * 2 * G * HEAD_DIM * 2 * (keys + T)
        return dict(bytes=2.0 * matrices + 2.0 * V * W + 2.0 * T * W + cache + 2.0 * B * V, flops=flops)
    v = VOLARAX
    W, H, d, r = v["width"], v["heads"], v["dim"], v["rank"]
    mk, mv, half = v["m_heads"] * v["m_dim"], v["m_heads"] * v["m_vdim"], LAYERS // 2
    attn, mlstm, ff = W * (2 * H * d + r) + 2 * H * d * r, W * (2 * mk + 3 * mv + 2 * v["m_heads"]), 3 * W * v["ff"]
    pairs, keys = _pairs(spans, v["window"])
    matrices = half * (attn + mlstm) + LAYERS * ff
    flops = 2.0 * T * matrices + 2.0 * B * W * v["vocab"] + half * (4.0 * pairs * H * d + 4.0 * T * mk * v["m_vdim"])
    state = half * B * mk * v["m_vdim"] * 4 * 2
    return dict(bytes=2.0 * matrices + 2.0 * v["vocab"] * W + 2.0 * T * W + half * (keys + T) * r * 2 + state + 4.0 * B * v["vocab"],
                flops=flops)


def tolerance(case):
    """bf16 activations through ``LAYERS`` layers; tokens have a winner by a wide margin."""
    return {"rel": 0.02, "max": 0.15, "differ": 0.0}


# ---- the same in 64 bits -------------------------------------------------------------------------------------------
def _attend(q, k, v, offset, scale, window=0, sink=None):
    """q [n, H, d] of positions offset ..., k and v [S, G, d] of positions 0 ... (or the last S up to the last query's)."""
    n, H, _ = q.shape
    S, G = k.shape[0], k.shape[1]
    first = offset + n - S
    out = torch.empty_like(q)
    kt, vt = k.transpose(0, 1), v.transpose(0, 1)
    step = max(1, (1 << 28) // (H * S))
    j = first + torch.arange(S, device=q.device)
    for a in range(0, n, step):
        b = min(n, a + step)
        s = torch.matmul(q[a:b].reshape(b - a, G, H // G, -1).permute(1, 2, 0, 3).reshape(G, -1, q.shape[2]), kt.transpose(1, 2)) * scale
        i = offset + torch.arange(a, b, device=q.device)
        seen = j[None, :] <= i[:, None]
        if window:
            seen &= j[None, :] > i[:, None] - window
        s = s.view(G, H // G, b - a, S).masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.view(G, H // G, 1, 1).expand(-1, -1, b - a, 1)], dim=-1)
        p = torch.softmax(s, dim=-1)[..., :S]
        o = torch.matmul(p.reshape(G, -1, S), vt).view(G, H // G, b - a, -1)
        out[a:b] = o.permute(2, 0, 1, 3).reshape(b - a, H, -1)
    return out


def _exact_llama(case, seed):
    W, F, H, G, V, theta, eps, bias = LLAMA[case["model"]]
    spans = _spans(case)
    layers, embed, head, norm = _llama_tensors(case["model"], seed)
    ids = torch.from_numpy(np.concatenate(_tokens(case, seed, V))).long().cuda()
    pos = torch.cat([torch.arange(c, c + n) for c, n in spans]).cuda()
    angle = pos[:, None].double() * theta ** (-torch.arange(0, HEAD_DIM, 2, device="cuda").double() / HEAD_DIM)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def turn(t):
        lo, hi = t.chunk(2, dim=-1)
        return torch.cat([lo * cos - hi * sin, hi * cos + lo * sin], dim=-1)

    rms = lambda x, w: x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()
    x = embed[ids].double()
    pages = sum(_pages(c + n) for c, n in spans)
    for l, t in enumerate(layers):
        qkv = rms(x, t["ln_attn"]) @ t["wqkv"].double().T + (t["bqkv"].double() if bias else 0.0)
        k, v, q = qkv.view(-1, H + 2 * G, HEAD_DIM).split([G, G, H], dim=1)
        k, q = turn(k), turn(q)
        cache = _context(seed, l, (pages, 2, G, PAGE, HEAD_DIM))
        last = l + 1 == LAYERS
        kv = torch.cat([cache, torch.zeros_like(cache[:16])]).double() if last else None      # the pool has 16 spare pages
        o, page, row = torch.empty_like(q), 0, 0
        for c, n in spans:
            held = cache[page:page + _pages(c + n)]
            old = held.permute(1, 0, 3, 2, 4).reshape(2, -1, G, HEAD_DIM)[:, :c].double()
            new = slice(row, row + n)
            o[new] = _attend(q[new], torch.cat([old[0], k[new]]), torch.cat([old[1], v[new]]), c, HEAD_DIM ** -0.5)
            if last:
                p = torch.arange(c, c + n, device="cuda")
                kv[page + p // PAGE, 0, :, p % PAGE] = k[new]
                kv[page + p // PAGE, 1, :, p % PAGE] = v[new]
            page, row = page + _pages(c + n), row + n
        x = x + o.reshape(len(x), -1) @ t["wo"].double().T
        h = rms(x, t["ln_ffn"])
        x = x + (torch.nn.functional.silu(h @ t["wg"].double().T) * (h @ t["wu"].double().T)) @ t["wd"].double().T
    ends = torch.cumsum(torch.tensor([n for _, n in spans]), 0).cuda() - 1
    return dict(logits=rms(x[ends], norm) @ head.double().T, tokens=None, kv=kv)


def _exact_volarax(case, seed):
    v, spans = VOLARAX, _spans(case)
    eps, H, d = v["eps"], v["heads"], v["dim"]
    w = _volarax_tensors(seed)
    get = lambda n: w[n].double()
    ids = torch.from_numpy(np.concatenate(_tokens(case, seed, v["vocab"]))).long().cuda()

    def norm(x, name):
        y = x - x.mean(-1, keepdim=True)
        return y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps) * get(name) + get(name + ".b")

    rms = lambda x: x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    pages = sum(_pages(c + n) for c, n in spans)

    def attention(h, p, layer):
        q = (h @ get(p + "q").T).view(-1, H, d)
        new = rms(h @ get(p + "dkv").T) * get(p + "dkv.norm")
        # cached pages are stored in tiles of 8 rows by 64 columns
        rows = _context(seed, layer, (pages, PAGE, v["rank"])).view(pages, 2, v["rank"] // 64, 8, 64).permute(0, 1, 3, 2, 4)
        rows = rows.reshape(pages * PAGE, v["rank"])
        o, page, row = torch.empty_like(q), 0, 0
        for c, n in spans:
            first = max(0, c - v["window"] + 1)
            lat = torch.cat([rows[page * PAGE + first:page * PAGE + c].double(), new[row:row + n]])
            k, u = ((lat @ get(p + part).T).view(-1, H, d) for part in ("uk", "uv"))
            o[row:row + n] = _attend(q[row:row + n], k, u, c, d ** -0.5, v["window"], get(p + "sink"))
            page, row = page + _pages(c + n), row + n
        return o.reshape(len(h), -1) @ get(p + "o").T

    def mlstm(h, p, layer):
        M, dk, dv = v["m_heads"], v["m_dim"], v["m_vdim"]
        q, k = (h @ get(p + "q").T).view(-1, M, dk) * dk ** -0.5, (h @ get(p + "k").T).view(-1, M, dk)
        val = (h @ get(p + "v").T).view(-1, M, dv)
        capped = lambda n: v["cap"] * torch.tanh((h @ get(p + n).T + get(p + n + ".b")) / v["cap"])
        log_i, log_f = capped("i"), torch.nn.functional.logsigmoid(capped("f"))
        o = torch.empty_like(val)
        starts = np.cumsum([0] + [n for _, n in spans])
        for t in range(max(n for _, n in spans)):        # all requests that have a token t
            live = [i for i, (_, n) in enumerate(spans) if n > t]
            at = torch.tensor([starts[i] + t for i in live], device="cuda")
            if t == 0:
                S, nn = (z.double() for z in _recurrent(seed, layer, len(spans)))
                mm = torch.zeros(len(spans), M, dtype=torch.float64, device="cuda")
                for i, (c, _) in enumerate(spans):
                    if c == 0:
                        S[i], nn[i] = 0.0, 0.0
            elif len(live) < len(was):
                keep = torch.tensor([was.index(i) for i in live], device="cuda")
                S, nn, mm = S[keep], nn[keep], mm[keep]
            was = live
            top = torch.maximum(log_f[at] + mm, log_i[at])
            old, new = torch.exp(log_f[at] + mm - top), torch.exp(log_i[at] - top)
            S = old[..., None, None] * S + (new[..., None] * k[at])[..., None] * val[at][:, :, None]
            nn, mm = old[..., None] * nn + new[..., None] * k[at], top
            den = torch.maximum((nn * q[at]).sum(-1).abs(), torch.exp(-mm)) + 1e-6
            o[at] = (S * q[at][..., None]).sum(2) / den[..., None]
        return (rms(o).reshape(len(h), -1) * get(p + "norm") * torch.sigmoid(h @ get(p + "g").T)) @ get(p + "o").T

    x = norm(w["embed"][ids].double(), "embed.norm")
    for i in range(LAYERS):
        p = "l%d." % i
        h = norm(x, p + "norm1")
        x = x + norm(attention(h, p + "mix.", i) if i % 2 == 0 else mlstm(h, p + "mix.", i), p + "norm1b")
        h = norm(x, p + "norm2")
        x = x + norm((torch.relu(h @ get(p + "mlp.gate").T) * (h @ get(p + "mlp.up").T)) @ get(p + "mlp.down").T, p + "norm2b")
    ends = torch.cumsum(torch.tensor([n for _, n in spans]), 0).cuda() - 1
    return dict(logits=norm(x[ends], "final.norm") @ get("head").T, tokens=None)


def exact(case, seed):
    with torch.no_grad():
        return _exact_llama(case, seed) if case["model"] in LLAMA else _exact_volarax(case, seed)
