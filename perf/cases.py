"""The work by which this framework's speed is judged, as cases that can be prepared, run and checked.

A case is what a program around the framework has it do: prompts of unequal lengths taken in one step, a long prompt in
portions, one decode step of a batch that is under way, or a whole short request.  The model sizes are the presets of the
dense decoder (``config/presets``) and the sizes at which ``bench.py`` compares the Revelix design; batch sizes, prompt lengths and
contexts lie in the ranges of the benchmark's configurations (prompts up to 2,048 tokens, contexts up to 4,096, batches of
1, 8 and 64, cache blocks of 16 and of the library's own 64 tokens) and below, where requests are short.

Weights are drawn once per model, as a server loads its checkpoint once; a state has its own cache, sequences and captured
decode graph, made from the seed.  Decode steps are fed given tokens (a state's own), so that one step does not depend on
how a near-tie among the last step's logits was decided; the sampled tokens are read back all the same, because a program
looks for its stop tokens.  In bfloat16 only logits are compared: over a vocabulary of 150,000 the largest two are often
closer than the rounding.  In float32 the tokens are compared too.
"""

import math

import torch

import flashdecode_cuda_b200 as fd
from flashdecode_cuda_b200.config import config_from_dict, preset_dict
from flashdecode_cuda_b200.engine.decode import GraphDecoder

WEIGHT_SEED = 7
GIVEN = 256                      # tokens given to every decoding sequence, used round and round
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}

REVELIX = {                      # the sizes of the Revelix comparison in bench.py
    "revelix-w1024": dict(width=1024, heads=8, kv=2, dim=128, window=1024, keep=64, taps=3, rot=64, rec_heads=4, rec_dim=128,
                          rec_vdim=128, ret_heads=8, ret_dim=128, ret_vdim=128, ff=4096),
    "revelix-w2048": dict(width=2048, heads=16, kv=4, dim=128, window=1024, keep=64, taps=3, rot=64, rec_heads=8, rec_dim=128,
                          rec_vdim=128, ret_heads=16, ret_dim=128, ret_vdim=128, ff=8192),
}


def _case(name, kind, model, dtype, block, batch, shortest, longest, portion=0, new=0, temperature=0.0):
    return dict(name=name, kind=kind, model=model, dtype=dtype, block=block, batch=batch, shortest=shortest, longest=longest,
                portion=portion, new=new, temperature=temperature)


def listed():
    small, mid, large = "qwen2.5-1.5b", "qwen2.5-7b", "qwen2.5-14b"
    return [
        # the smallest call: one short question; the host's launches and the kernels' start-up times show
        _case("prompt-19", "prompt", small, "bf16", 64, 1, 19, 19),
        # the benchmark's prompt step
        _case("prompt-2048", "prompt", small, "bf16", 16, 1, 2048, 2048),
        # a batch that starts together, prompts of unequal lengths packed into one step
        _case("prompts-8", "prompt", small, "bf16", 64, 8, 253, 2048),
        # a long document taken in portions, as servers do that decode other sequences in between; odd lengths
        _case("prompt-portions", "prompt", small, "bf16", 64, 1, 3001, 3001, portion=384),
        # one user waiting for each token
        _case("decode-1", "decode", small, "bf16", 64, 1, 1300, 1300),
        # the benchmark's decode step
        _case("decode-8", "decode", small, "bf16", 16, 8, 1500, 3000),
        # a full server, sampling
        _case("decode-64", "decode", small, "bf16", 16, 64, 700, 1400, temperature=0.8),
        # the larger presets: a small batch, and prompts of questions' and short documents' length
        _case("7b-decode-8", "decode", mid, "bf16", 64, 8, 1100, 2600),
        _case("14b-prompts-3", "prompt", large, "bf16", 64, 3, 101, 700),
        # the true 32-bit path, by which a deployment checks its bfloat16 results
        _case("fp32-decode-8", "decode", small, "fp32", 16, 8, 150, 1200, temperature=0.8),
        _case("fp32-prompts-3", "prompt", small, "fp32", 16, 3, 17, 250),
        # a design with recurrent state, a whole request: prompts, then tokens one by one, then the slots are given back
        _case("revelix-request-4", "request", "revelix-w1024", "bf16", 64, 4, 150, 900, new=24),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["prompt", "prompt", "decode", "decode", "decode", "request"])
    dtype = rng.choice(["bf16"] * 5 + ["fp32"] * 2)
    model = "qwen2.5-1.5b"
    if dtype == "bf16":
        model = rng.choice(["qwen2.5-1.5b"] * 4 + ["qwen2.5-7b", "qwen2.5-14b", "revelix-w1024", "revelix-w2048"])
    size = {"qwen2.5-7b": 5, "qwen2.5-14b": 10}.get(model, 1)     # about the larger presets' work per token
    block = rng.choice([16, 64])
    temperature = rng.choice([0.0, 0.0, 0.8])
    if kind == "decode":
        batch = log_int(1, 64 if dtype == "bf16" else 16)
        longest = log_int(40, 3200 if dtype == "bf16" else 1200)
        bound = max(1024, 1 << (longest - 1).bit_length())       # a graph serves lengths up to a power of two: stay clear of the
        longest = min(longest, bound - 800)                      # next capture for the steps that are timed
        return _drawn(kind, model, dtype, block, batch, log_int(max(8, longest // 4), longest), longest, temperature=temperature)
    total = log_int(5, (7000 if dtype == "bf16" else 400) // size)
    batch = rng.randint(1, max(1, min(8, total // 4)))
    longest = max(2, min(3300, total * 2 // (batch + 1) if batch > 1 else total))
    portion = log_int(64, 700) if kind == "prompt" and longest > 800 and rng.random() < 0.4 else 0
    shortest = longest if batch == 1 else rng.randint(1, longest)
    return _drawn(kind, model, dtype, block, batch, shortest, longest, portion, rng.randint(3, max(4, 40 // size)) if kind == "request" else 0,
                  temperature if kind == "request" else 0.0)


def _drawn(*a, **kw):
    c = _case("", *a, **kw)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# sizes
# ---------------------------------------------------------------------------

def _config(name):
    """The config.json dictionary of a model."""
    if name not in REVELIX:
        return preset_dict(name)
    z = REVELIX[name]
    left = {"conv": z["taps"], "dim": z["dim"], "heads": z["heads"], "kv_heads": z["kv"], "scale": z["dim"] ** -0.5, "softcap": 30.0,
            "mask": {"size": z["window"], "keep_first": z["keep"]}, "vdim": z["dim"],
            "rot": {"base": 1000000.0, "dims": z["rot"], "scaling": {"factor": 8.0, "original": 1024, "fast": 32.0, "slow": 1.0}}}
    right = {"dim": z["rec_dim"], "heads": z["rec_heads"], "vdim": z["rec_vdim"]}
    n = z["ret_heads"]
    ret = {"decay": [1.0 - 2.0 ** (-5 - 5 * i / (n - 1)) for i in range(n)], "dim": z["ret_dim"], "heads": n, "vdim": z["ret_vdim"],
           "rot": {"base": 10000.0, "dims": z["ret_dim"]}}
    par = {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0}
    return {"architecture": "Revelix", "vocab": 32768, "width": z["width"], "norm": {"eps": 1e-5}, "logit_scale": 1.0,
            "layers": [{"type": t, "mixer": m, "mlp": {"ff": z["ff"], "kind": "dense"}}
                       for t, m in (("retention", ret), ("parallel", par)) * 4]}


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def _lengths(case):
    """Prompt length of every sequence: unequal, the longest first, the others spread evenly down to the shortest."""
    n, lo, hi = case["batch"], case["shortest"], case["longest"]
    return [hi - (hi - lo) * i // max(1, n - 1) for i in range(n)]


def _tokens(case, seed):
    """(prompts, given tokens [batch, GIVEN]) on the host, as a tokenizer leaves them."""
    g = torch.Generator().manual_seed(seed)
    vocab = _vocab(_config(case["model"]))
    prompts = [torch.randint(0, vocab, (n,), generator=g).tolist() for n in _lengths(case)]
    return prompts, torch.randint(0, vocab, (case["batch"], GIVEN), generator=g).tolist()


# ---------------------------------------------------------------------------
# the passes
# ---------------------------------------------------------------------------

_loaded = {}                     # the one model that is loaded


def _weights(model, dtype):
    """Seeded weights of which the residual stream is made up as in a trained model: about as much of the embedding as of what
    the layers add, each a little.  (With every matrix drawn alike, the first layer drowns the embedding, 48 layers amplify one
    rounding a hundredfold, and no two implementations agree on the logits.)"""
    cfg, L = model.config, len(model.blocks)
    W = fd.random_weights(model, WEIGHT_SEED, dtype, device="cuda")
    if hasattr(cfg, "hidden_size"):
        # N(0, 0.02) throughout: the projections' outputs have the size g, the gated product about 0.35 g^2
        g = 0.02 * cfg.hidden_size ** 0.5
        add = 1.5 / (2 * L) ** 0.5
        down, out = add / (0.35 * g * g * cfg.intermediate_size ** 0.5), add / (g * (cfg.num_attention_heads * cfg.head_dim) ** 0.5)
        for name, w in W.items():
            if name.endswith(("down_proj.weight", "o_proj.weight")):
                w.mul_(down if name.endswith("down_proj.weight") else out)
    else:
        for name, w in W.items():
            if name == "embed":
                w.mul_(50.0)     # rows of unit size: this design's norms do not rescale their input
            elif name.endswith((".o", ".down")):
                w.mul_((2 * L) ** -0.5)
    return W


def _engine(case):
    key = (case["model"], case["dtype"])
    if key not in _loaded:
        _loaded.clear()
        torch.cuda.empty_cache()
        dtype = DTYPES[case["dtype"]]
        model = fd.Model.from_config(config_from_dict(_config(case["model"])), dtype, "cuda")
        _loaded[key] = fd.Engine(model.bind(_weights(model, dtype)))
    return _loaded[key]


class _State:
    def __init__(self, case, seed):
        self.case, self.seed = case, seed
        self.engine = _engine(case)
        self.prompts, self.given = _tokens(case, seed)
        self.n, self.at = case["batch"], 0
        self.ids = list(range(self.n))
        self.temps = [case["temperature"]] * self.n
        room = {"prompt": 0, "decode": 1024, "request": case["new"]}[case["kind"]]
        self.cache = self.engine.new_paged_cache(self.n, case["longest"] + room, case["block"])
        self.decoder = GraphDecoder(self.engine.model, self.cache) if room else None
        self.slots = []

    def start(self, want):
        """Slots for the sequences, and their prompts into the cache: in one step, or in portions."""
        self.slots = [self.cache.admit() for _ in self.prompts]
        portion = self.case["portion"] or self.case["longest"]
        for at in range(0, self.case["longest"], portion):
            live = [i for i, p in enumerate(self.prompts) if len(p) > at]
            ends = at + portion >= self.case["longest"]
            logits = self.engine.step(self.cache, [self.slots[i] for i in live], [self.prompts[i][at:at + portion] for i in live],
                                      want if ends else None)
        self.at = 0
        return logits

    def token(self):
        """One decode step over given tokens: (sampled tokens, logits)."""
        j = self.at
        self.decoder.run(self.slots, [t[j % GIVEN] for t in self.given], self.temps, self.ids, [j] * self.n, self.seed)
        self.at += 1
        return self.decoder.read_tokens(self.n), self.decoder.last_logits(self.n)

    def end(self):
        for s in self.slots:
            self.cache.release(s)
        self.slots = []


def prepare(case, seed):
    state = _State(case, seed)
    if case["kind"] == "decode":
        # the sequences are under way: prompts in the cache (a few at a time, which bounds the scratch memory), one token decoded
        state.slots = [state.cache.admit() for _ in state.prompts]
        for i in range(0, state.n, 8):
            state.engine.step(state.cache, state.slots[i:i + 8], state.prompts[i:i + 8], None)
        state.token()
    elif case["kind"] == "request":
        state.start(None)
        state.token()            # the server has its graph of this batch size
        state.end()
    return state


def run(state):
    kind, exact_tokens = state.case["kind"], state.case["dtype"] == "fp32"
    if kind == "prompt":
        logits = state.start("last")
        state.end()
        return {"logits": logits}
    if kind == "decode":
        if state.at >= 1024:     # the cache's longest sequence: a program would end them here
            state.end()
            state.start(None)
        tokens, logits = state.token()
        return {"logits": logits, "tokens": torch.tensor(tokens)} if exact_tokens else {"logits": logits}
    first = state.start("last")
    sampled = []
    for _ in range(state.case["new"]):
        tokens, logits = state.token()
        sampled.append(tokens)
    state.end()
    return {"first": first, "logits": logits, "tokens": torch.tensor(sampled)} if exact_tokens else {"first": first, "logits": logits}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _dense_sizes(cfg):
    """(layers, matrix elements per layer, query heads x head size, key/value elements per token and layer, head elements)."""
    H, I, d = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    q, kv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
    return cfg["num_hidden_layers"], H * (q + 2 * kv) + q * H + 3 * H * I, q, 2 * kv, H * cfg["vocab_size"]


def work(case):
    cfg, lens = _config(case["model"]), _lengths(case)
    e = 2 if case["dtype"] == "bf16" else 4
    n, new = len(lens), case["new"]
    vocab = _vocab(cfg)
    # per step: (new tokens, of each sequence: (tokens cached before, new tokens), logits wanted)
    if case["kind"] == "decode":
        steps = [([(l + 1, 1) for l in lens], n)]
    else:
        portion = case["portion"] or case["longest"]
        steps = []
        for at in range(0, case["longest"], portion):
            live = [(at, min(portion, l - at)) for l in lens if l > at]
            steps.append((live, len(live) if at + portion >= case["longest"] else 0))
        steps += [([(l + j, 1) for l in lens], n) for j in range(new)]
    total = {"bytes": 0.0, "flops": 0.0}
    for rows, wanted in steps:
        T = sum(k for _, k in rows)
        if "hidden_size" in cfg:
            L, mats, q, kv, head = _dense_sizes(cfg)
            H = cfg["hidden_size"]
            read = sum(c for c, _ in rows) * L * kv
            flops = 2.0 * T * L * mats + L * 4.0 * q * sum(k * (c + (k + 1) / 2) for c, k in rows)
            write = T * L * kv
        else:
            H, head, read, write, mats, flops, L = cfg["width"], cfg["width"] * vocab, 0.0, 0.0, 0.0, 0.0, 1
            for layer in cfg["layers"]:
                m = layer["mixer"]
                mats += 2 * H * layer["mlp"]["ff"]
                rec = m if layer["type"] == "retention" else m["right"]
                qk, v = rec["heads"] * rec["dim"], rec["heads"] * rec["vdim"]
                mats += H * (2 * qk + 2 * v) + v * H if layer["type"] == "retention" else H * (2 * qk + v) + v * H
                flops += 4.0 * T * qk * rec["vdim"]
                read += len(rows) * 2 * qk * rec["vdim"] * 4 / e / 2          # the state: float32, read
                write += len(rows) * 2 * qk * rec["vdim"] * 4 / e / 2         # and written
                if layer["type"] != "retention":
                    a, size = m["left"], m["left"]["mask"]["size"] + m["left"]["mask"]["keep_first"]
                    q, kv = a["heads"] * a["dim"], 2 * a["kv_heads"] * a["dim"]
                    mats += H * (q + kv) + q * H
                    flops += 4.0 * q * sum(min(c + i + 1, size) for c, k in rows for i in range(k))
                    read += sum(min(c, size) for c, _ in rows) * kv
                    write += T * kv
            flops += 2.0 * T * mats
        total["bytes"] += e * (L * mats + read + write + T * H + (head if wanted else 0)) + 4.0 * wanted * vocab
        total["flops"] += flops + 2.0 * wanted * head
    return total


def tolerance(case):
    # About four times what the path differs from ``exact`` by.  Measured: bfloat16 activations through 28 and 48 dense layers
    # rel 0.005 to 0.008 (largest 0.023 to 0.043), through the 8 layers of the design with recurrences 0.003 (0.016); float32
    # 3.5e-6 (1.9e-5).  Float32 tokens: drawn from logits that agree to five digits, over 150,000 of them.
    if case["dtype"] == "fp32":
        return {"rel": 1.4e-5, "max": 8e-5, "differ": 0.0}
    return {"rel": 0.012, "max": 0.065} if case["model"] in REVELIX else {"rel": 0.028, "max": 0.16}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------

F64 = torch.float64


def _turn(x, pos, freqs, mag=1.0, interleaved=False):
    """x [B, S, heads, d]: the first 2 * len(freqs) dimensions of every head turned by position * frequency."""
    half = freqs.numel()
    a = pos.to(F64)[:, None] * freqs
    c, s = (a.cos() * mag)[None, :, None, :], (a.sin() * mag)[None, :, None, :]
    out = x.clone()
    iu, iv = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if interleaved else (slice(0, half), slice(half, 2 * half))
    u, v = x[..., iu], x[..., iv]
    out[..., iu], out[..., iv] = u * c - v * s, v * c + u * s
    return out


def _frequencies(dims, base, scaling=None):
    f = torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=F64)
    if not scaling:
        return f.cuda(), 1.0

    def pair(turns):
        return dims * math.log(scaling["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(pair(scaling["fast"])), 0), min(math.ceil(pair(scaling["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return (f / scaling["factor"] * ramp + f * (1.0 - ramp)).cuda(), 0.1 * math.log(scaling["factor"]) + 1.0


def _dense_exact(cfg, W, seqs, at):
    """Logits of sequence i at its positions at[i]; the sequences' tokens are packed into one batch for the products."""
    nq, nkv, d, H = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["hidden_size"]
    eps, lens = cfg["rms_norm_eps"], [len(s) for s in seqs]

    def mat(name):
        return W[name].to(F64).t()

    def norm(x, name):
        return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps) * W[name].to(F64)
    freqs, _ = _frequencies(d, cfg["rope_theta"])
    x = W["model.embed_tokens.weight"][torch.tensor([t for s in seqs for t in s], device="cuda")].to(F64)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}"
        h = norm(x, f"{p}.input_layernorm.weight")
        q, k, v = (h @ mat(f"{p}.self_attn.{n}_proj.weight") + W[f"{p}.self_attn.{n}_proj.bias"].to(F64) for n in "qkv")
        out = []
        for qs, ks, vs in zip(q.split(lens), k.split(lens), v.split(lens)):
            S = qs.shape[0]
            pos = torch.arange(S, device="cuda")
            qs, ks = _turn(qs.view(1, S, nq, d), pos, freqs)[0], _turn(ks.view(1, S, nkv, d), pos, freqs)[0]
            vs = vs.view(S, nkv, d)
            rows = torch.empty(S, nq, d, dtype=F64, device="cuda")
            hidden = pos[None, :] > pos[:, None]
            for g in range(nkv):
                heads = slice(g * nq // nkv, (g + 1) * nq // nkv)
                s = torch.einsum("ihd,jd->hij", qs[:, heads], ks[:, g]) / math.sqrt(d)
                rows[:, heads] = torch.einsum("hij,jd->ihd", s.masked_fill_(hidden, -math.inf).softmax(-1), vs[:, g])
            out.append(rows.reshape(S, nq * d))
        x = x + torch.cat(out) @ mat(f"{p}.self_attn.o_proj.weight")
        h = norm(x, f"{p}.post_attention_layernorm.weight")
        gate = h @ mat(f"{p}.mlp.gate_proj.weight")
        x = x + (gate * torch.sigmoid(gate) * (h @ mat(f"{p}.mlp.up_proj.weight"))) @ mat(f"{p}.mlp.down_proj.weight")
    starts = [sum(lens[:i]) for i in range(len(lens))]
    x = norm(x[[s + p for s, places in zip(starts, at) for p in places]], "model.norm.weight")
    return x @ mat("model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight")


def _revelix_exact(cfg, W, seqs, at):
    """The same for the Revelix design; sequences are padded at their ends, which no earlier position sees."""
    eps, S = cfg["norm"]["eps"], max(len(s) for s in seqs)
    W = {n: w.to(F64) for n, w in W.items()}
    pos = torch.arange(S, device="cuda")
    tokens = torch.tensor([s + [0] * (S - len(s)) for s in seqs], device="cuda")
    x = W["embed"][tokens]
    B = x.shape[0]

    def norm(x, n):
        return torch.tanh(W[n + ".alpha"] * x) * W[n] + W[n + ".b"]

    def lin(h, n, bias=False):
        return h @ W[n].t() + (W[n + ".b"] if bias else 0.0)

    def unit(o):
        return o / torch.sqrt(o.pow(2).mean(-1, keepdim=True) + eps)

    def conv(u, w):
        taps = w.shape[1]
        y = torch.zeros_like(u)
        for j in range(taps):
            back = taps - 1 - j
            if back < S:
                y[:, back:] += w[:, j] * u[:, :S - back]
        return y

    def retention(h, p, m):
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = (lin(h, f"{p}.{n}").view(B, S, H, -1) for n in "qkv")
        freqs, mag = _frequencies(m["rot"]["dims"], m["rot"]["base"])
        q, k = _turn(q, pos, freqs, mag), _turn(k, pos, freqs, mag) * d ** -0.5
        gap = (pos[:, None] - pos[None, :]).to(F64)
        out = torch.empty(B, S, H, dv, dtype=F64, device="cuda")
        for n in range(H):
            fade = torch.where(gap >= 0, m["decay"][n] ** gap.clamp(min=0), 0.0)
            out[:, :, n] = (q[:, :, n] @ k[:, :, n].transpose(1, 2) * fade) @ v[:, :, n]
        g = lin(h, f"{p}.g")
        return lin(unit(out).reshape(B, S, H * dv) * g * torch.sigmoid(g), f"{p}.o")

    def attention(h, p, m):
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (conv(lin(h, f"{p}.{n}", True), W[f"{p}.{n}.conv"]) for n in "qkv")
        freqs, mag = _frequencies(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"])
        q, k = _turn(q.view(B, S, H, d), pos, freqs, mag, True), _turn(k.view(B, S, G, d), pos, freqs, mag, True)
        v = v.view(B, S, G, dv)
        gap, mask, cap = pos[:, None] - pos[None, :], m["mask"], m["softcap"]
        seen = (gap >= 0) & ((gap < mask["size"]) | (pos[None, :] < mask["keep_first"]))
        sink = W[f"{p}.sink"][:, None, None]
        out = torch.empty(B, S, H, dv, dtype=F64, device="cuda")
        for b in range(B):
            s = torch.einsum("ihd,jhd->hij", q[b], k[b].repeat_interleave(H // G, 1)) * m["scale"]
            s = (cap * torch.tanh(s / cap)).masked_fill(~seen, -math.inf)
            w = torch.softmax(torch.cat([s, sink.expand(H, S, 1)], -1), -1)[:, :, :S]
            w = torch.einsum("hg,gij->hij", W[f"{p}.talk"], w)
            out[b] = torch.einsum("hij,jhv->ihv", w, v[b].repeat_interleave(H // G, 1))
        return lin(out.reshape(B, S, H * dv), f"{p}.o")

    def recurrence(h, p, m):
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        q = lin(h, f"{p}.q")
        q = (q * torch.sigmoid(q)).view(B, S, H, d)
        low = W[f"{p}.lower"]
        f = (low + (1.0 - low) * torch.sigmoid(lin(h, f"{p}.f", True))).view(B, S, H, d)
        v = lin(h, f"{p}.v").view(B, S, H, dv)
        state = torch.zeros(B, H, d, dv, dtype=F64, device="cuda")
        out = torch.empty(B, S, H, dv, dtype=F64, device="cuda")
        for t in range(S):
            state = f[:, t, :, :, None] * state + (1.0 - f[:, t])[..., None] * v[:, t, :, None, :]
            out[:, t] = (q[:, t, :, None, :] @ state)[:, :, 0]
        return lin((unit(out) * W[f"{p}.norm"]).reshape(B, S, H * dv), f"{p}.o")

    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}", layer["mixer"]
        h = norm(x, f"{p}.norm1")
        if layer["type"] == "retention":
            x = x + retention(h, f"{p}.mix", m)
        else:
            x = (x + m["left_scale"] * attention(h, f"{p}.mix.left", m["left"])
                 + m["right_scale"] * recurrence(h, f"{p}.mix.right", m["right"]))
        z = lin(norm(x, f"{p}.norm2"), f"{p}.mlp.up")
        a, b = torch.nn.functional.softplus(W[f"{p}.mlp.act"])
        act = torch.where(z > 0, a * z * z, (0.5 + b) * (torch.expm1(z.clamp(max=0.0)) - z)) + 0.5 * z
        x = x + lin(act, f"{p}.mlp.down")
    x = norm(torch.cat([x[b, places] for b, places in enumerate(at)]), "final.norm")
    return x @ W["embed"].t() * cfg["logit_scale"]


def exact(case, seed):
    cfg, (prompts, given) = _config(case["model"]), _tokens(case, seed)
    # tokens decoded when run() returns: a decode state has one token more than its prompt when the pass begins
    new = {"prompt": 0, "decode": 2, "request": case["new"]}[case["kind"]]
    seqs = [p + [g[j % GIVEN] for j in range(new)] for p, g in zip(prompts, given)]
    if work(dict(case, kind="prompt", portion=0, new=0))["flops"] > 3.5e14:
        return None              # over about 20 seconds at the rate of 64-bit products
    model = fd.Model.from_config(config_from_dict(cfg), torch.float32, "cpu")
    _loaded.clear()
    W = _weights(model, DTYPES[case["dtype"]])
    forward = _dense_exact if "hidden_size" in cfg else _revelix_exact
    with torch.no_grad():
        if case["kind"] == "request":
            both = forward(cfg, W, seqs, [[len(p) - 1, len(s) - 1] for p, s in zip(prompts, seqs)])
            out = {"first": both[0::2].contiguous(), "logits": both[1::2].contiguous()}
        else:
            last = [[len(s) - 1] for s in seqs]
            if case["portion"]:  # sequences that ended in an earlier portion have no logits in the last step
                live = [i for i, p in enumerate(prompts) if len(p) > (case["longest"] - 1) // case["portion"] * case["portion"]]
                seqs, last = [seqs[i] for i in live], [last[i] for i in live]
            out = {"logits": forward(cfg, W, seqs, last)}
    if case["dtype"] == "fp32" and case["kind"] != "prompt":
        out["tokens"] = None     # drawn with the library's own noise
    return out
