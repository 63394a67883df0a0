"""What this framework is timed on: the work its users have it do, over the public Python API, from one projected row to a
2048-token prompt.

Kinds of case
  projection  one weight matrix applied to a batch of rows that is on the device (a host that keeps its own model code)
  generate    one request alone: prompt, greedy tokens on the device, the logits of the last token
  decode      one engine step of a batch of sequences: a token each, the ids of all and the logits of the sampled ones
  prefill     one prompt in chunks, the logits behind it
  layered     a layered design in bf16: a ragged batch of prompts in one step, then steps of one given token per sequence

Sizes are those of the repository's benchmark and tests; depths are cut where a layer more only repeats the others.  Weights are
random; int8 matrices have codes and scales as the quantiser leaves them for normal weights.
"""
import math

import numpy as np
import torch

from paged_infer_b200 import api
from paged_infer_b200 import loader as ld

BLOCK = 16
ARCHS = {
    "tinyllama": dict(hidden=2048, heads=32, kv_heads=4, inter=5632, vocab=32000, theta=10000.0),
    "llama3_8b": dict(hidden=4096, heads=32, kv_heads=8, inter=14336, vocab=128256, theta=500000.0),
}
EPS = 1e-5
WIDTH, VOCAB, FF, WINDOW = 2048, 32000, 5632, 1024          # of the layered cases
EXPERTS, TOP, GROUPS, KEEP, EXPERT_FF, SHARED_FF = 64, 6, 8, 4, 704, 1408


def listed():
    return [
        # one row through one matrix: what a launch and its latency cost
        dict(name="projection_row", kind="projection", weights="int8", rows=5632, cols=2048, batch=1),
        # a batch of rows through the largest matrix of a small model
        dict(name="projection_head_128", kind="projection", weights="int8", rows=32000, cols=2048, batch=128),
        # one user, interactive: the prompt and the greedy continuation of the smallest whole workload
        dict(name="generate_alone", kind="generate", arch="tinyllama", layers=22, weights="int8", head="int8", prompt=128, chunk=128, steps=32),
        # a lightly loaded server, the head left in its checkpoint's precision as the loader's int8 mode does
        dict(name="decode_8", kind="decode", arch="tinyllama", layers=11, weights="int8", head="bf16", batch=8, lo=100, hi=1000, shared=0, logits=2),
        # the loaded server: 64 sequences, half of them behind one common prompt
        dict(name="decode_64", kind="decode", arch="tinyllama", layers=11, weights="int8", head="int8", batch=64, lo=256, hi=2048, shared=512, logits=4),
        # a larger model's layers and head size over long contexts
        dict(name="decode_long_16", kind="decode", arch="llama3_8b", layers=2, weights="int8", head="int8", batch=16, lo=3000, hi=4096, shared=0, logits=2),
        # long prompts, small and larger model; the second is no multiple of the chunk
        dict(name="prefill_2048", kind="prefill", arch="tinyllama", layers=11, weights="int8", head="int8", prompt=2048, chunk=512),
        dict(name="prefill_wide_1500", kind="prefill", arch="llama3_8b", layers=4, weights="int8", head="int8", prompt=1500, chunk=512),
        # an unquantised checkpoint, the loader's default
        dict(name="prefill_bf16_weights", kind="prefill", arch="tinyllama", layers=6, weights="bf16", head="bf16", prompt=400, chunk=256),
        # layered designs: a long prompt; many short ones with some tokens each; routed experts and latent attention
        dict(name="sumosun_prompt", kind="layered", design="sumosun", layers=6, batch=1, lo=2048, hi=2048, steps=0),
        dict(name="sumosun_batch", kind="layered", design="sumosun", layers=6, batch=32, lo=20, hi=60, steps=6),
        dict(name="lilosun_batch", kind="layered", design="lilosun", layers=3, batch=16, lo=30, hi=120, steps=4),
    ]


def _between(rng, lo, hi):
    """A whole number, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["projection", "projection", "generate", "decode", "decode", "prefill", "prefill", "layered"])
    if kind == "projection":
        weights = rng.choice(["int8", "int8", "int8", "bf16"])
        cols = 128 * _between(rng, 8, 64) if weights == "int8" else 8 * _between(rng, 100, 700)
        return dict(kind=kind, weights=weights, rows=_between(rng, 250, 24000), cols=cols, batch=_between(rng, 1, 512 if weights == "int8" else 64))
    if kind == "generate":
        return dict(kind=kind, arch="tinyllama", layers=rng.randint(6, 16), weights="int8", head=rng.choice(["int8", "bf16"]), prompt=_between(rng, 5, 300),
                    chunk=rng.choice([64, 128, 512]), steps=_between(rng, 8, 32))
    if kind == "decode":
        big = rng.random() < 0.3
        batch = _between(rng, 2, 16 if big else 64)
        lo = _between(rng, 20, 1000)
        return dict(kind=kind, arch="llama3_8b" if big else "tinyllama", layers=rng.randint(1, 2) if big else rng.randint(4, 10), weights="int8",
                    head=rng.choice(["int8", "int8", "bf16"]) if not big else "int8", batch=batch, lo=lo, hi=lo + _between(rng, 10, 1000),
                    shared=rng.choice([0, 256]), logits=min(batch, 2))
    if kind == "prefill":
        big = rng.random() < 0.4
        weights = "int8" if big else rng.choice(["int8", "int8", "bf16"])
        return dict(kind=kind, arch="llama3_8b" if big else "tinyllama", layers=rng.randint(1, 3) if big else rng.randint(3, 6), weights=weights,
                    head="int8" if weights == "int8" else "bf16", prompt=_between(rng, 17, 400 if weights == "bf16" else 1500), chunk=rng.choice([128, 256, 512]))
    batch = _between(rng, 1, 32)
    lo = _between(rng, 4, max(5, 1200 // batch))
    return dict(kind=kind, design=rng.choice(["sumosun", "lilosun"]), layers=3, batch=batch, lo=lo, hi=lo + rng.randint(0, max(1, 700 // batch)), steps=rng.randint(0, 4))


# ---- inputs -----------------------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)


def _int8_matrix(g, rows, cols):
    """Codes and row scales as the quantiser leaves them for N(0, 0.02) weights."""
    codes = (_normal(g, rows, cols) * 35).round_().clamp_(-127, 127).to(torch.int8)
    scales = (0.02 / 35) * (1 + 0.05 * _normal(g, rows).clamp_(-3, 3))
    return codes, scales


def _matrix(g, kind, rows, cols):
    return _int8_matrix(g, rows, cols) if kind == "int8" else (_normal(g, rows, cols) * 0.02).bfloat16()


def _host(m):
    """What the library's constructors take: (codes, scales), or bf16 bits."""
    if isinstance(m, tuple):
        return m[0].cpu().numpy(), m[1].cpu().numpy()
    return m.view(torch.int16).cpu().numpy().view(np.uint16)


def _wide(m):
    """The matrix in 64 bits."""
    return m[0].double() * m[1].double()[:, None] if isinstance(m, tuple) else m.double()


NAMES = ("wq", "wk", "wv", "wo", "w1", "w2", "w3")


def _llama_weights(case, seed):
    a = ARCHS[case["arch"]]
    H, I, V, KV = a["hidden"], a["inter"], a["vocab"], a["kv_heads"] * (a["hidden"] // a["heads"])
    shapes = dict(wq=(H, H), wk=(KV, H), wv=(KV, H), wo=(H, H), w1=(I, H), w2=(H, I), w3=(I, H))
    g = _generator(seed)
    w = dict(embed=(_normal(g, V, H) * 0.02).bfloat16(), final=1 + 0.1 * _normal(g, H))
    w["norms"] = [(1 + 0.1 * _normal(g, H), 1 + 0.1 * _normal(g, H)) for _ in range(case["layers"])]
    w["layers"] = [{n: _matrix(g, case["weights"], *shapes[n]) for n in NAMES} for _ in range(case["layers"])]
    w["head"] = _matrix(g, case["head"], V, H)
    return w


def _llama(case, seed, max_batch):
    a = ARCHS[case["arch"]]
    w = _llama_weights(case, seed)
    cfg = ld.LlamaConfig(hidden_size=a["hidden"], num_hidden_layers=case["layers"], num_attention_heads=a["heads"], num_key_value_heads=a["kv_heads"],
                         intermediate_size=a["inter"], vocab_size=a["vocab"], rms_norm_eps=EPS, rope_theta=a["theta"])
    hw = ld.HostWeights(token_embeddings=_host(w["embed"]), final_norm=w["final"].cpu().numpy(), attention_norm=[n[0].cpu().numpy() for n in w["norms"]],
                        ffn_norm=[n[1].cpu().numpy() for n in w["norms"]], projections=[{n: _host(l[n]) for n in NAMES} for l in w["layers"]],
                        lm_head=None)
    ctx = api.Context(0)
    return ctx, api.LlamaWeights(ctx, cfg, hw, max_batch=max_batch, max_positions=4608, lm_head=_host(w["head"]))


def _tokens(case, seed):
    """The prompts of a case, from numpy's generator: {lengths, shared part and tokens} for decode, else one prompt."""
    rng = np.random.default_rng(int(seed) + 17)
    vocab = ARCHS[case["arch"]]["vocab"]
    if case["kind"] != "decode":
        return rng.integers(0, vocab, case["prompt"]).astype(np.uint32)
    B = case["batch"]
    lengths = rng.integers(case["lo"], case["hi"] + 1, B)
    shared = np.zeros(B, np.int64)
    if case["shared"]:
        half = max(B // 2, 1)
        lengths[0] = max(case["hi"], case["shared"] + 1)
        shared[1:half] = np.minimum(case["shared"], (lengths[1:half] - 1) // BLOCK * BLOCK)
    prompts = [rng.integers(0, vocab, n).astype(np.uint32) for n in lengths]
    for b in range(B):
        prompts[b][:shared[b]] = prompts[0][:shared[b]]
    return prompts, shared, rng.integers(0, vocab, B).astype(np.uint32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "projection":
        g = _generator(seed)
        ctx = api.Context(0)
        w = _host(_matrix(g, case["weights"], case["rows"], case["cols"]))
        p = api.Projection.int8(ctx, *w) if case["weights"] == "int8" else api.Projection.f32(ctx, w)
        x = _normal(g, case["batch"], case["cols"])
        y = torch.empty(case["batch"], case["rows"], device="cuda")
        torch.cuda.synchronize()
        return dict(kind=kind, ctx=ctx, p=p, x=x, y=y, batch=case["batch"])
    if kind == "layered":
        return _prepare_layered(case, seed)
    rng = np.random.default_rng(int(seed) + 23)
    if kind != "decode":
        ctx, model = _llama(case, seed, case["chunk"])
        n = case["prompt"] + case.get("steps", 0) + 1
        blocks = -(-n // BLOCK)
        kv = api.KvCache(ctx, model.kv_layout(blocks + 3, BLOCK))
        table = api.BlockTable(rng.permutation(blocks + 3)[:blocks])
        return dict(kind=kind, ctx=ctx, model=model, kv=kv, table=table, tokens=_tokens(case, seed), chunk=case["chunk"], steps=case.get("steps", 0))
    prompts, shared, nexts = _tokens(case, seed)
    ctx, model = _llama(case, seed, 512)
    need = [(len(p) // BLOCK + 1) - s // BLOCK for p, s in zip(prompts, shared)]
    free = list(rng.permutation(sum(need) + 3))
    kv = api.KvCache(ctx, model.kv_layout(len(free), BLOCK))
    tables = api.PackedBlockTables(len(prompts), max(len(p) for p in prompts) // BLOCK + 1)
    rows = []
    for b, p in enumerate(prompts):
        rows.append((rows[0][:shared[b] // BLOCK] if b else []) + [int(free.pop()) for _ in range(need[b])])
        tables.set_row(b, rows[b])
        model.prefill_batched(p[shared[b]:], int(shared[b]), api.BlockTable(rows[b]), kv, 512)
    return dict(kind=kind, ctx=ctx, model=model, kv=kv, tables=tables, tokens=nexts, positions=np.array([len(p) for p in prompts], np.int32),
                logits=list(range(case["logits"])))


def run(s):
    if s["kind"] == "projection":
        s["p"].apply_device(s["x"], s["y"], s["batch"])
        return s["y"]
    if s["kind"] == "prefill":
        return s["model"].prefill_batched(s["tokens"], 0, s["table"], s["kv"], s["chunk"])
    if s["kind"] == "generate":
        n = len(s["tokens"])
        first, t = s["model"].prefill_batched(s["tokens"], 0, s["table"], s["kv"], s["chunk"], want_argmax=True)
        ids = s["model"].decode_multi([t], [n], [s["table"]], s["kv"], s["steps"])
        return {"prompt": first, "tokens": ids, "last": s["model"].forward(int(ids[-1, 0]), n + s["steps"], s["table"], s["kv"])}
    if s["kind"] == "decode":
        logits, ids = s["model"].decode_batch_rows(s["tokens"], s["positions"], s["tables"], s["kv"], s["logits"])
        return {"logits": logits, "ids": ids}
    out = [s["model"].step(s["prompts"], s["zeros"], s["tables"], s["kv"], s["state"], s["slots"])]
    for i, t in enumerate(s["given"]):
        out.append(s["model"].step(t, s["lengths"] + i, s["tables"], s["kv"], s["state"], s["slots"]))
    return out


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    size = {"int8": 1, "bf16": 2}
    if kind == "projection":
        n, k, m = case["rows"], case["cols"], case["batch"]
        return {"bytes": n * k * size[case["weights"]] + 4 * m * (n + k), "flops": 2 * m * n * k}
    if kind == "layered":
        return _layered_work(case)
    a = ARCHS[case["arch"]]
    hd = a["hidden"] // a["heads"]
    per_layer = a["hidden"] * (2 * a["hidden"] + 2 * a["kv_heads"] * hd + 3 * a["inter"])
    weights = per_layer * case["layers"] * size[case["weights"]]
    head = a["vocab"] * a["hidden"]
    token = case["layers"] * 2 * a["kv_heads"] * hd * 4            # cache bytes of a token
    attend = case["layers"] * 4 * a["hidden"]                      # operations per query and key
    if kind == "decode":
        n = case["batch"] * (case["lo"] + case["hi"]) / 2
        seen = n - (max(case["batch"] // 2 - 1, 0) * min(case["shared"], (case["lo"] + case["hi"]) / 2) if case["shared"] else 0)
        return {"bytes": weights + head * size[case["head"]] + token * (seen + case["batch"]),
                "flops": 2 * case["batch"] * (per_layer * case["layers"] + head) + attend * n}
    n, steps = case["prompt"], case.get("steps", 0)
    passes = 1 + (steps + 1 if kind == "generate" else 0)
    total = n + passes - 1
    return {"bytes": passes * (weights + head * size[case["head"]]) + token * (total + (passes - 1) * n),
            "flops": 2 * total * per_layer * case["layers"] + 2 * passes * head + attend * total * total / 2}


def tolerance(case):
    # about four times what the path is off the 64-bit result on these inputs: 32-bit sums of one product; through the layers, where the
    # difference grows with depth and length; bf16 activations through the layers
    rel = {"projection": 2e-6, "generate": 2e-5, "decode": 3e-5, "prefill": 1e-4, "layered": 0.02}[case["kind"]]
    return {"rel": rel, "max": 10 * rel}


# ---- 64 bits --------------------------------------------------------------------------------------------------------------------
def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


class _Llama64:
    """The model token by token or in chunks, with its own cache; the rotary table is the 32-bit one that the model is defined with."""

    def __init__(self, case, seed):
        a = self.a = ARCHS[case["arch"]]
        w = _llama_weights(case, seed)
        self.embed, self.final, self.head = w["embed"], w["final"].double(), w["head"]
        self.norms = [(x.double(), y.double()) for x, y in w["norms"]]
        self.layers = [{n: _wide(m) for n, m in l.items()} for l in w["layers"]]
        self.hd = a["hidden"] // a["heads"]
        part = (np.arange(0, self.hd, 2, dtype=np.float32) / np.float32(self.hd)).astype(np.float64)
        self.freq = np.float32(1) / (a["theta"] ** part).astype(np.float32)

    def rotate(self, x, pos):
        angle = torch.from_numpy((np.asarray(pos, np.float32)[:, None] * self.freq).astype(np.float64)).cuda()[:, None]
        c, s = torch.cos(angle).float().double(), torch.sin(angle).float().double()
        u, v = x.chunk(2, -1)
        return torch.cat([u * c - v * s, v * c + u * s], -1)

    def forward(self, tokens, start, cache):
        """The last token's hidden row; cache: one [k, v] per layer, appended to."""
        a, T = self.a, len(tokens)
        x = self.embed[torch.as_tensor(np.asarray(tokens, np.int64)).cuda()].double()
        pos = np.arange(start, start + T)
        q_pos, group = torch.arange(start, start + T, device="cuda"), a["heads"] // a["kv_heads"]
        for l, w in enumerate(self.layers):
            h = _rms(x, self.norms[l][0], EPS)
            q = self.rotate((h @ w["wq"].T).view(T, a["heads"], self.hd), pos)
            k = self.rotate((h @ w["wk"].T).view(T, a["kv_heads"], self.hd), pos)
            v = (h @ w["wv"].T).view(T, a["kv_heads"], self.hd)
            if len(cache) <= l:
                cache.append([k, v])
            else:
                cache[l] = [torch.cat([cache[l][0], k]), torch.cat([cache[l][1], v])]
            K, V = cache[l]
            hide = torch.arange(len(K), device="cuda")[None] > q_pos[:, None]
            o = torch.empty_like(q)
            for n in range(a["kv_heads"]):
                s = torch.einsum("tgd,sd->gts", q[:, n * group:(n + 1) * group], K[:, n]) / math.sqrt(self.hd)
                o[:, n * group:(n + 1) * group] = torch.einsum("gts,sd->tgd", s.masked_fill(hide, -math.inf).softmax(-1), V[:, n])
            x = x + o.reshape(T, -1) @ w["wo"].T
            h = _rms(x, self.norms[l][1], EPS)
            x = x + (torch.nn.functional.silu(h @ w["w1"].T) * (h @ w["w3"].T)) @ w["w2"].T
        return x[-1]

    def prompt(self, tokens, cache):
        for c in range(0, len(tokens), 512):
            x = self.forward(tokens[c:c + 512], c, cache)
        return x

    def logits(self, x):
        h = _rms(x, self.final, EPS)
        if not isinstance(self.head, tuple):
            return torch.cat([part.double() @ h for part in self.head.split(16000)])
        return torch.cat([part.double() @ h for part in self.head[0].split(16000)]) * self.head[1].double()


def exact(case, seed):
    kind = case["kind"]
    if kind == "projection":
        g = _generator(seed)
        w = _matrix(g, case["weights"], case["rows"], case["cols"])
        return _normal(g, case["batch"], case["cols"]).double() @ _wide(w).T
    if kind == "layered":
        return _layered_exact(case, seed)
    m = _Llama64(case, seed)
    if kind == "decode":
        prompts, _, nexts = _tokens(case, seed)
        rows = []
        for b in range(case["logits"]):
            cache = []
            m.prompt(prompts[b], cache)
            rows.append(m.logits(m.forward(nexts[b:b + 1], len(prompts[b]), cache)))
        return {"logits": torch.stack(rows), "ids": None}
    tokens, cache = _tokens(case, seed), []
    first = m.logits(m.prompt(tokens, cache))
    if kind == "prefill":
        return first
    ids, t = [], int(first.argmax())
    for i in range(case["steps"]):
        t = int(m.logits(m.forward([t], len(tokens) + i, cache)).argmax())
        ids.append([t])
    return {"prompt": first, "tokens": torch.tensor(ids), "last": m.logits(m.forward([t], len(tokens) + case["steps"], cache))}


# ---- layered designs --------------------------------------------------------------------------------------------------------------
SUMOSUN = dict(attention=dict(heads=16, kv_heads=4, dim=64, vdim=128), gla=dict(heads=16, dim=64, vdim=128), mlstm=dict(heads=8, dim=128, vdim=256))
TAU, CAP, DIFF, ROT_BASE, RANK = 16.0, 15.0, 0.5, 500000.0, 16
LATENT = dict(heads=16, dim=128, rot=64, vdim=128, rank=512)
SSD = dict(heads=64, vdim=64, state=128, conv=4)
YARN = dict(factor=8.0, original=4096, fast=32.0, slow=1.0)
LIMIT, LAYER_EPS = 7.0, 1e-6


def _layered_config(case):
    layers = []
    for i in range(case["layers"]):
        if case["design"] == "sumosun":
            kinds = [ld.LayerConfig(ld.MIXER_ATTENTION, maps=2, window=WINDOW, rot_dims=64, rot_base=ROT_BASE, scale=0.125, diff=DIFF, ff=FF, **SUMOSUN["attention"]),
                     ld.LayerConfig(ld.MIXER_GLA, tau=TAU, ff=FF, **SUMOSUN["gla"]), ld.LayerConfig(ld.MIXER_MLSTM, gate_cap=CAP, ff=FF, **SUMOSUN["mlstm"])]
        else:
            experts = dict(ff_kind=ld.FF_EXPERTS, ff=EXPERT_FF, experts=EXPERTS, top=TOP, expert_groups=GROUPS, keep_groups=KEEP, shared_ff=SHARED_FF, limit=LIMIT,
                           shared_limit=LIMIT)
            ssd = dict(heads=SSD["heads"], vdim=SSD["vdim"], dim=SSD["state"], groups=1, norm_groups=1, conv=SSD["conv"])
            kinds = [ld.LayerConfig(ld.MIXER_LATENT, heads=LATENT["heads"], dim=LATENT["dim"], vdim=LATENT["vdim"], rank=LATENT["rank"], window=WINDOW,
                                    rot_dims=LATENT["rot"], rot_base=10000.0, rot_factor=YARN["factor"], rot_original=YARN["original"], rot_fast=YARN["fast"],
                                    rot_slow=YARN["slow"], scale=192 ** -0.5, **experts),
                     ld.LayerConfig(ld.MIXER_SSD, ff_kind=ld.FF_SILU, ff=FF, **ssd), ld.LayerConfig(ld.MIXER_SSD, **ssd, **experts)]
        layers.append(kinds[i % 3])
    if case["design"] == "sumosun":
        return ld.LayeredConfig(WIDTH, VOCAB, LAYER_EPS, layers)
    return ld.LayeredConfig(WIDTH, VOCAB, LAYER_EPS, layers, norm=ld.NORM_LAYER, tied=False)


def _layered_tensors(case, seed):
    g, W = _generator(seed), WIDTH
    t = {}

    def put(name, *shape, std=None, mean=0.0):
        t[name] = (_normal(g, *shape) * (shape[-1] ** -0.5 if std is None else std) + mean).bfloat16()

    if case["design"] == "sumosun":
        def norm(name, alpha):
            put(name, W, std=0.2, mean=1.0)
            put(name + ".b", W, std=0.1)
            t[name + ".alpha"] = torch.tensor(alpha, device="cuda").bfloat16()

        put("embed", VOCAB, W, std=1.0)
        for i in range(case["layers"]):
            p, kind = f"l{i}.mix.", ("attention", "gla", "mlstm")[i % 3]
            m = SUMOSUN[kind]
            H, D, E = m["heads"], m["dim"], m["vdim"]
            norm(f"l{i}.norm1", 0.7)
            norm(f"l{i}.norm1b", 0.9)
            if kind == "attention":
                put(p + "q", H * 2 * D, W)
                put(p + "k", m["kv_heads"] * 2 * D, W)
                put(p + "v", m["kv_heads"] * E, W)
                for n in ("lq1", "lk1", "lq2", "lk2"):
                    put(p + n, D, std=0.1)
            else:
                put(p + "q", H * D, W)
                put(p + "k", H * D, W)
                put(p + "v", H * E, W)
                put(p + "g", H * E, W)
                if kind == "gla":
                    put(p + "a1", RANK, W)
                    put(p + "a2", H * D, RANK, std=1.0)
                    put(p + "a2.b", H * D, std=1.5, mean=1.0)
                    put(p + "norm", E, std=0.2, mean=1.0)
                else:
                    for n, b in (("i", 0.0), ("f", 3.0)):
                        put(p + n, H, W)
                        put(p + n + ".b", H, std=1.0, mean=b)
                    put(p + "norm", H * E, std=0.2, mean=1.0)
            put(p + "o", W, H * E)
            norm(f"l{i}.norm2", 0.8)
            norm(f"l{i}.norm2b", 1.1)
            put(f"l{i}.mlp.gate", FF, W)
            put(f"l{i}.mlp.up", FF, W)
            put(f"l{i}.mlp.down", W, FF)
        norm("final.norm", 0.6)
        return t

    # A trained router is decided about most tokens.  Here every token names its experts in leading channels that no sublayer writes
    # and the routers read: TOP experts in TOP / 2 groups, clearly ahead of the rest.
    def gated(p, F):
        put(p + "gate", F, W)
        put(p + "up", F, W)
        put(p + "down", W, F)

    put("embed", VOCAB, W, std=1.0)
    n = EXPERTS // GROUPS
    lead = torch.rand(VOCAB, GROUPS, generator=g, device="cuda").argsort(-1)[:, :TOP // 2]
    pick = torch.rand(VOCAB, TOP // 2, n, generator=g, device="cuda").argsort(-1)[:, :, :2]
    chosen = torch.zeros(VOCAB, EXPERTS, device="cuda").scatter_(1, (lead[:, :, None] * n + pick).reshape(VOCAB, -1), 1.0)
    t["embed"][:, :EXPERTS] = (chosen * 4 - 1.5 + 0.4 * torch.rand(VOCAB, EXPERTS, generator=g, device="cuda")).bfloat16()
    for i in range(case["layers"]):
        l, p = f"l{i}.", f"l{i}.mix."
        for k in (1, 2):
            put(l + f"norm{k}", W, std=0.2, mean=1.0)
            put(l + f"ls{k}", W, std=0.2, mean=0.5)
            t[l + f"norm{k}"][:EXPERTS] = 1
            t[l + f"ls{k}"][:EXPERTS] = 0
        if i % 3 == 0:
            H, D, R, E, K = (LATENT[x] for x in ("heads", "dim", "rot", "vdim", "rank"))
            put(p + "q", H * (D + R), W)
            put(p + "dkv", K + R, W)
            put(p + "dkv.norm", K, std=0.2, mean=1.0)
            put(p + "uk", H * D, K)
            put(p + "uv", H * E, K)
            put(p + "g", H * E, W)
        else:
            H, E, N = SSD["heads"], SSD["vdim"], SSD["state"]
            put(p + "in", 2 * H * E + 2 * N + H, W)
            put(p + "conv", H * E + 2 * N, SSD["conv"], std=0.4)
            put(p + "conv.b", H * E + 2 * N, std=0.2)
            put(p + "dt_bias", H, std=1.0, mean=-2.0)
            put(p + "A_log", H, std=1.0)
            put(p + "D", H, std=0.5, mean=0.5)
            put(p + "norm", H * E, std=0.2, mean=1.0)
        put(p + "o", W, H * E)
        p = l + "mlp."
        if i % 3 == 1:
            gated(p, FF)
        else:
            t[p + "router"] = torch.zeros(EXPERTS, W, device="cuda").bfloat16()
            t[p + "router"][:, :EXPERTS] = torch.eye(EXPERTS, device="cuda").bfloat16()
            put(p + "correction", EXPERTS, std=0.01)
            for e in range(EXPERTS):
                gated(f"{p}e{e}.", EXPERT_FF)
            gated(p + "shared.", SHARED_FF)
            put(p + "shared.sg", 1, W)
    put("final.norm", W, std=0.2, mean=1.0)
    put("head", VOCAB, W)
    return t


def _layered_inputs(case, seed):
    rng = np.random.default_rng(int(seed) + 29)
    lengths = rng.integers(case["lo"], case["hi"] + 1, case["batch"])
    return [rng.integers(0, VOCAB, n + case["steps"]).astype(np.uint32) for n in lengths], lengths


def _prepare_layered(case, seed):
    ctx = api.Context(0)
    tokens, lengths = _layered_inputs(case, seed)
    tensors = {}
    for name, a in _layered_tensors(case, seed).items():
        tensors[name] = _host(a.reshape(-1) if a.dim() == 0 else a)
    model = api.LayeredModel(ctx, _layered_config(case), tensors, "bfloat16", int(max(lengths.sum(), 64)))
    need = [-(-len(t) // BLOCK) for t in tokens]
    free = np.random.default_rng(int(seed) + 31).permutation(sum(need) + 2)
    tables, at = api.PackedBlockTables(len(tokens), max(need)), 0
    for b, n in enumerate(need):
        tables.set_row(b, free[at:at + n])
        at += n
    B = len(tokens)
    return dict(kind="layered", ctx=ctx, model=model, kv=model.kv_pool(len(free), BLOCK), state=model.state_pool(B), slots=list(range(B)), tables=tables,
                prompts=[t[:n] for t, n in zip(tokens, lengths)], zeros=np.zeros(B, np.int32), lengths=lengths.astype(np.int32),
                given=[[t[n + i:n + i + 1] for t, n in zip(tokens, lengths)] for i in range(case["steps"])])


def _layered_work(case):
    W, B, L = WIDTH, case["batch"], case["layers"]
    n = B * (case["lo"] + case["hi"]) / 2
    seen = lambda m: m * min(m, WINDOW) - min(m, WINDOW) ** 2 / 2            # query and key pairs of a prompt of m tokens
    pairs = B * seen((case["lo"] + case["hi"]) / 2)
    fixed = 0.0                                                             # weights that every token meets
    routed = state = attend = 0.0
    layers_with_experts = 0
    for i in range(L):
        if case["design"] == "sumosun":
            m = SUMOSUN[("attention", "gla", "mlstm")[i % 3]]
            H, D, E = m["heads"], m["dim"], m["vdim"]
            fixed += W * (H * E * (1 if i % 3 == 0 else 2) + 3 * FF)
            fixed += W * (2 * D * (H + m["kv_heads"]) + m["kv_heads"] * E) if i % 3 == 0 else W * (2 * H * D + H * E)
            attend += 2 * H * (2 * D + 2 * E) * (i % 3 == 0)
            state += 4 * H * D * E * (i % 3 != 0)
        else:
            if i % 3 == 0:
                m = LATENT
                fixed += W * (m["heads"] * (m["dim"] + m["rot"]) + m["rank"] + m["rot"] + 2 * m["heads"] * m["vdim"])
                attend += 2 * m["heads"] * (m["dim"] + m["rot"] + m["vdim"])
            else:
                fixed += W * (3 * SSD["heads"] * SSD["vdim"] + 2 * SSD["state"] + SSD["heads"])
                state += 4 * SSD["heads"] * SSD["vdim"] * SSD["state"]
            if i % 3 == 1:
                fixed += 3 * W * FF
            else:
                fixed += W * (3 * SHARED_FF + EXPERTS + 1)
                routed += TOP * 3 * W * EXPERT_FF
                layers_with_experts += 1
    head = VOCAB * W
    met = lambda tokens: layers_with_experts * 3 * W * EXPERT_FF * EXPERTS * (1 - (1 - TOP / EXPERTS) ** tokens)
    steps = case["steps"]
    return {"bytes": 2 * (fixed + met(n) + head) + steps * 2 * (fixed + met(B) + head) + (2 * steps + 1) * B * state + 4 * B * VOCAB * (steps + 1),
            "flops": 2 * (n + steps * B) * (fixed + routed) + 2 * B * (steps + 1) * head + attend * (pairs + steps * n)}


def _turn(x, freq, gain):
    """Pairs of neighbouring channels of x [T, heads, d] turn with the position."""
    a = torch.arange(x.shape[0], device="cuda", dtype=torch.float64)[:, None, None] * freq
    c, s = torch.cos(a) * gain, torch.sin(a) * gain
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)


def _attend(q, k, v, scale):
    """q, k [T, d], v [T, e]: softmax over the window."""
    T = q.shape[0]
    d = torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]
    return (q @ k.T * scale).masked_fill((d < 0) | (d >= WINDOW), -math.inf).softmax(-1) @ v


def _unit(x, eps=LAYER_EPS):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _sumosun_mixer(w, kind, h):
    m, T = SUMOSUN[kind], h.shape[0]
    H, D, E = m["heads"], m["dim"], m["vdim"]
    lin = lambda n: h @ w(n).T
    if kind == "attention":
        G = m["kv_heads"]
        f = ROT_BASE ** (-torch.arange(0, 64, 2, device="cuda", dtype=torch.float64) / 64)
        q, k = _turn(lin("q").view(T, 2 * H, D), f, 1.0), _turn(lin("k").view(T, 2 * G, D), f, 1.0)
        v = lin("v").view(T, G, E)
        lam = torch.exp((w("lq1") * w("lk1")).sum()) - torch.exp((w("lq2") * w("lk2")).sum()) + DIFF
        o = torch.empty(T, H, E, device="cuda", dtype=torch.float64)
        for n in range(H):
            j = n // (H // G)
            o[:, n] = _unit(_attend(q[:, 2 * n], k[:, 2 * j], v[:, j], 0.125) - lam * _attend(q[:, 2 * n + 1], k[:, 2 * j + 1], v[:, j], 0.125)) * (1 - DIFF)
        return o.reshape(T, -1) @ w("o").T
    q, k, v = lin("q").view(T, H, D) * D ** -0.5, lin("k").view(T, H, D), lin("v").view(T, H, E)
    S = torch.zeros(H, D, E, device="cuda", dtype=torch.float64)
    o = torch.empty(T, H, E, device="cuda", dtype=torch.float64)
    if kind == "gla":
        keep = torch.exp(torch.nn.functional.logsigmoid(lin("a1") @ w("a2").T + w("a2.b")) / TAU).view(T, H, D, 1)
        for t in range(T):
            S = torch.baddbmm(S * keep[t], k[t, :, :, None], v[t, :, None])
            o[t] = (q[t, :, None] @ S)[:, 0]
        return (_unit(o) * w("norm")).reshape(T, -1).mul(torch.nn.functional.silu(lin("g"))) @ w("o").T
    log_i = CAP * torch.tanh((lin("i") + w("i.b")) / CAP)
    log_f = torch.nn.functional.logsigmoid(CAP * torch.tanh((lin("f") + w("f.b")) / CAP))
    N, top = torch.zeros(H, D, device="cuda", dtype=torch.float64), torch.zeros(H, device="cuda", dtype=torch.float64)
    for t in range(T):
        new = torch.maximum(log_f[t] + top, log_i[t])
        keep, add = torch.exp(log_f[t] + top - new), torch.exp(log_i[t] - new)
        S = S * keep[:, None, None] + (add[:, None] * k[t])[:, :, None] * v[t, :, None]
        N = N * keep[:, None] + add[:, None] * k[t]
        top = new
        o[t] = (q[t, :, None] @ S)[:, 0] / (torch.maximum((N * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6)[:, None]
    return _unit(o).reshape(T, -1).mul(w("norm")).mul(torch.sigmoid(lin("g"))) @ w("o").T


def _lilosun_mixer(w, latent, h):
    T = h.shape[0]
    lin = lambda n: h @ w(n).T
    if latent:
        H, D, R, E, K = (LATENT[x] for x in ("heads", "dim", "rot", "vdim", "rank"))
        i = torch.arange(R // 2, device="cuda", dtype=torch.float64)
        f = 10000.0 ** (-2 * i / R)
        at = lambda turns: R * math.log(YARN["original"] / (2 * math.pi * turns)) / (2 * math.log(10000.0))
        lo, hi = max(math.floor(at(YARN["fast"])), 0), min(math.ceil(at(YARN["slow"])), R - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f, gain = f / YARN["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(YARN["factor"]) + 1
        q, down = lin("q").view(T, H, D + R), lin("dkv")
        c = _unit(down[:, :K]) * w("dkv.norm")
        k, v = (c @ w("uk").T).view(T, H, D), (c @ w("uv").T).view(T, H, E)
        q_rot, k_rot = _turn(q[:, :, D:], f, gain), _turn(down[:, None, K:], f, gain)[:, 0]
        o = torch.stack([_attend(torch.cat([q[:, n, :D], q_rot[:, n]], -1), torch.cat([k[:, n], k_rot], -1), v[:, n], 192 ** -0.5) for n in range(H)], 1)
        return o.reshape(T, -1).mul(torch.sigmoid(lin("g"))) @ w("o").T
    H, E, N, taps = (SSD[x] for x in ("heads", "vdim", "state", "conv"))
    p, inner = lin("in"), H * E
    z, x, dt = p[:, :inner], p[:, inner:2 * inner + 2 * N], torch.nn.functional.softplus(p[:, 2 * inner + 2 * N:] + w("dt_bias"))
    past = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    x = torch.nn.functional.silu(w("conv.b") + sum(w("conv")[:, j] * past[j:j + T] for j in range(taps)))
    x, Bm, Cm = x[:, :inner].view(T, H, E), x[:, inner:inner + N], x[:, inner + N:]
    keep = torch.exp(-torch.exp(w("A_log")) * dt)
    S, y = x.new_zeros(H, N, E), torch.empty_like(x)
    for t in range(T):
        S = S * keep[t][:, None, None] + Bm[t][None, :, None] * (dt[t][:, None] * x[t])[:, None]
        y[t] = Cm[t] @ S + w("D")[:, None] * x[t]
    return (_unit(y.reshape(T, inner) * torch.nn.functional.silu(z)) * w("norm")) @ w("o").T


def _clamped(h, gate, up, down):
    g, u = (h @ gate.T).clamp(max=LIMIT), (h @ up.T).clamp(-LIMIT, LIMIT)
    return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ down.T


def _experts(w, h):
    s = torch.sigmoid(h @ w("router").T)
    choice = s + w("correction")
    best = choice.view(-1, GROUPS, EXPERTS // GROUPS).topk(2, -1).values.sum(-1)
    kept = torch.zeros_like(best).scatter_(1, best.topk(KEEP, -1).indices, 1.0).repeat_interleave(EXPERTS // GROUPS, 1)
    ids = choice.masked_fill(kept == 0, -math.inf).topk(TOP, -1).indices
    p = torch.zeros_like(s).scatter_(1, ids, s.gather(1, ids))
    p = p / (p.sum(-1, keepdim=True) + 1e-20)
    out = torch.sigmoid(h @ w("shared.sg").T) * _clamped(h, w("shared.gate"), w("shared.up"), w("shared.down"))
    for e in range(EXPERTS):
        rows = p[:, e].nonzero()[:, 0]
        if len(rows):
            out[rows] += p[rows, e, None] * _clamped(h[rows], w(f"e{e}.gate"), w(f"e{e}.up"), w(f"e{e}.down"))
    return out


def _layered_exact(case, seed):
    t = _layered_tensors(case, seed)
    tokens, lengths = _layered_inputs(case, seed)
    ends = np.cumsum([len(x) for x in tokens])
    parts = [slice(int(e - len(x)), int(e)) for e, x in zip(ends, tokens)]
    wide = lambda prefix: lambda n: t[prefix + n].double()
    x = t["embed"][torch.as_tensor(np.concatenate(tokens).astype(np.int64)).cuda()].double()

    def dyt(name, v):
        w = wide("")
        return torch.tanh(w(name + ".alpha") * v) * w(name) + w(name + ".b")

    def layer_norm(name, v):
        d = v - v.mean(-1, keepdim=True)
        return _unit(d) * t[name].double()

    for i in range(case["layers"]):
        l, mix, mlp = f"l{i}.", wide(f"l{i}.mix."), wide(f"l{i}.mlp.")
        if case["design"] == "sumosun":
            h = dyt(l + "norm1", x)
            kind = ("attention", "gla", "mlstm")[i % 3]
            x = x + dyt(l + "norm1b", torch.cat([_sumosun_mixer(mix, kind, h[p]) for p in parts]))
            h = dyt(l + "norm2", x)
            x = x + dyt(l + "norm2b", (torch.nn.functional.gelu(h @ mlp("gate").T, approximate="tanh") * (h @ mlp("up").T)) @ mlp("down").T)
        else:
            h = layer_norm(l + "norm1", x)
            x = x + t[l + "ls1"].double() * torch.cat([_lilosun_mixer(mix, i % 3 == 0, h[p]) for p in parts])
            h = layer_norm(l + "norm2", x)
            y = (torch.nn.functional.silu(h @ mlp("gate").T) * (h @ mlp("up").T)) @ mlp("down").T if i % 3 == 1 else _experts(mlp, h)
            x = x + t[l + "ls2"].double() * y
    x = dyt("final.norm", x) if case["design"] == "sumosun" else layer_norm("final.norm", x)
    head = t["embed" if case["design"] == "sumosun" else "head"].double()
    last = np.array([p.start for p in parts]) + lengths - 1
    return [x[torch.as_tensor(last + i).cuda()] @ head.T for i in range(case["steps"] + 1)]
