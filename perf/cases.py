"""The work that a user of this framework has it do, as cases that can be timed and compared: whole speculative and
autoregressive requests, prompts, and the verify forward as a caller of the reference's own functions drives it.

Weights are random but for two planted things, so that requests run as they do with a trained pair: the base model's most
likely next token is decided by a clear margin (token t is followed by t + 1), and the drafter guesses it for about three
tokens in four.  Steps then accept 0 .. L-1 drafted tokens, and the tokens do not hang on the last bit of a sum."""
import math
import os
import sys
import zlib

import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ml-recurrent-drafter_b200"))

import recurrent_drafting as rd  # noqa: E402

EPS = 1e-6
ROPE_BASE = 10000.0
EMBED_STD = 2.0
HEAD_SCALE = 0.02
DRAFT_LOGIT = 14.0  # of the token that the drafter guesses

# Sizes of this repository's benchmark: the decoders of its decode workloads and of its comparison of base models.
SHAPES = {
    "tiny": dict(width=256, heads=4, kv=4, ff=688, vocab=1000, draft_layers=1, dtype="float32"),
    "2k": dict(width=2048, heads=16, kv=4, ff=5632, vocab=32000, draft_layers=2, dtype="bfloat16", mem=(4, 256, 512),
               latent=(16, 128, 64, 128, 512)),
    "4k": dict(width=4096, heads=32, kv=8, ff=11008, vocab=32000, draft_layers=2, dtype="bfloat16", mem=(8, 256, 512),
               latent=(32, 128, 64, 128, 512)),
    "7b": dict(width=4096, heads=32, kv=32, ff=11008, vocab=32000, draft_layers=2, dtype="bfloat16"),
}
WINDOW, KEEP_FIRST, GLU_LIMIT, GLU_ALPHA, GATE_CAP, GROUPS = 1024, 4, 7.0, 1.702, 15.0, 8


def listed():
    return [
        # the smallest models and calls: 32-bit, a few short launches per step, the host in between
        dict(name="speculative tiny fp32", kind="speculative", shape="tiny", layers=2, batch=2, prompt=32, new=64, beams=4, length=3,
             temperature=0.0),
        # one user of a 7B model, wide beams: latency of a step
        dict(name="speculative 7b batch 1", kind="speculative", shape="7b", layers=32, batch=1, prompt=200, new=48, beams=45, length=5,
             temperature=0.0),
        # the headline workload: eight requests with prompts of up to 500 tokens
        dict(name="speculative 7b batch 8", kind="speculative", shape="7b", layers=32, batch=8, prompt=500, new=40, beams=45, length=5,
             temperature=0.0),
        # speculative sampling, sixteen requests, narrow beams
        dict(name="sampling 7b batch 16", kind="speculative", shape="7b", layers=32, batch=16, prompt=256, new=24, beams=16, length=5,
             temperature=1.0),
        # the plain decode loop: one user, then a small server's batch that samples
        dict(name="autoregressive 7b batch 1", kind="autoregressive", design="llama", shape="7b", layers=32, batch=1, prompt=120, new=28,
             temperature=0.0),
        dict(name="autoregressive llama batch 24", kind="autoregressive", design="llama", shape="4k", layers=8, batch=24, prompt=333, new=24,
             temperature=1.0),
        # the two hybrid decoders generating for a few users
        dict(name="autoregressive dilavik batch 6", kind="autoregressive", design="dilavik", shape="4k", layers=8, batch=6, prompt=300, new=40,
             temperature=0.0),
        dict(name="autoregressive nulunex batch 8", kind="autoregressive", design="nulunex", shape="4k", layers=4, batch=8, prompt=1100, new=40,
             temperature=0.0),
        # prompts: one long document; many of different lengths; a long one that comes in portions beside short ones
        dict(name="prompt llama long", kind="prompt", design="llama", shape="4k", layers=8, lengths="8192", portion=0),
        dict(name="prompt dilavik ragged", kind="prompt", design="dilavik", shape="4k", layers=8, lengths="17,700,2048,3001,333", portion=0),
        dict(name="prompt nulunex portions", kind="prompt", design="nulunex", shape="4k", layers=4, lengths="5000,900,1536", portion=1024),
        # a caller who keeps the reference's own verify code: pack, dense mask, forward, unpack
        dict(name="verify forward", kind="verify", shape="7b", layers=4, batch=4, prompt=450, beams=24, length=5),
    ]


def draw(rng):
    def spread(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["speculative", "speculative", "autoregressive", "autoregressive", "prompt", "prompt", "verify"])
    if kind == "speculative":
        if rng.random() < 0.25:
            return dict(kind=kind, shape="tiny", layers=2, batch=spread(1, 8), prompt=spread(8, 96), new=spread(16, 96), beams=spread(2, 16),
                        length=rng.randint(2, 5), temperature=0.0)
        batch = spread(1, 16)
        return dict(kind=kind, shape=rng.choice(["2k", "4k", "7b"]), layers=rng.choice([4, 8, 16]), batch=batch,
                    prompt=spread(16, min(1000, 8000 // batch)), new=spread(12, 48), beams=spread(4, min(50, 400 // batch)),
                    length=rng.randint(3, 7), temperature=rng.choice([0.0, 0.0, 1.0]))
    if kind == "autoregressive":
        design, batch = rng.choice(["llama", "dilavik", "nulunex"]), spread(1, 32)
        return dict(kind=kind, design=design, shape=rng.choice(["2k", "4k"]), layers=rng.choice([4, 8]), batch=batch,
                    prompt=spread(8, min(2000, 8000 // batch)), new=spread(8, 40), temperature=rng.choice([0.0, 0.0, 1.0]))
    if kind == "prompt":
        rows, left = rng.randint(1, 6), 8000
        lengths = []
        for _ in range(rows):
            lengths.append(max(1, spread(1, max(2, left - 1))))
            left -= lengths[-1]
        return dict(kind=kind, design=rng.choice(["llama", "dilavik", "nulunex"]), shape=rng.choice(["2k", "4k"]), layers=rng.choice([4, 8]),
                    lengths=",".join(str(v) for v in lengths if v > 0), portion=rng.choice([0, 0, spread(100, 2000)]))
    return dict(kind=kind, shape=rng.choice(["2k", "4k", "7b"]), layers=rng.choice([2, 4]), batch=spread(1, 8), prompt=spread(16, 900),
                beams=spread(2, 32), length=rng.randint(2, 6))


# ------------------------------------------------------------------------------------------------------------ weights
def _generator(seed, name):
    return torch.Generator("cuda").manual_seed((seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))


def _dtype(z):
    return getattr(torch, z["dtype"])


class Weights:
    """Tensors by name, made from the seed alone; matrices are normal with 1.25 over the root of the input width."""

    def __init__(self, seed, dtype):
        self.seed, self.dtype = seed, dtype

    def normal(self, name, shape, std, mean=0.0):
        t = torch.randn(shape, generator=_generator(self.seed, name), device="cuda", dtype=self.dtype)
        return t.mul_(std).add_(mean) if mean else t.mul_(std)

    def matrix(self, name, rows, cols):
        return self.normal(name, (rows, cols), 1.25 / math.sqrt(cols))

    def gain(self, name, n):
        return self.normal(name, (n,), 0.1, 1.0)

    def embedding(self, z):
        return self.normal("embed", (z["vocab"], z["width"]), EMBED_STD)

    def head(self, z):
        return torch.roll(self.embedding(z), 1, dims=0).mul_(HEAD_SCALE)  # token t is followed by t + 1


def _llama_layer(w, z, i):
    H, hd, n = z["width"], z["width"] // z["heads"], f"model.layers.{i}."
    rows = {"self_attn.q_proj": (z["heads"] * hd, H), "self_attn.k_proj": (z["kv"] * hd, H), "self_attn.v_proj": (z["kv"] * hd, H),
            "self_attn.o_proj": (H, H), "mlp.gate_proj": (z["ff"], H), "mlp.up_proj": (z["ff"], H), "mlp.down_proj": (H, z["ff"])}
    out = {f"{n}{k}.weight": w.matrix(n + k, *s) for k, s in rows.items()}
    for k in ("self_attn.o_proj", "mlp.down_proj"):  # a deep stack's layers each add a part of what the stream holds
        out[f"{n}{k}.weight"].mul_(0.25)
    out.update({f"{n}{k}.weight": w.gain(n + k, H) for k in ("input_layernorm", "post_attention_layernorm")})
    return out


def _design(case, z):
    """config.json of the two hybrid decoders, laid out as the benchmark's comparison of base models lays them out."""
    if case["design"] == "dilavik":
        att = {"type": "attention", "mlp": {"kind": "dense", "ff": z["ff"] * 3 // 2},
               "mixer": {"heads": z["heads"], "kv_heads": z["kv"], "dim": 128, "vdim": 128, "rot": {"dims": 64, "base": ROPE_BASE},
                         "scale": 128 ** -0.5, "mask": {"size": WINDOW, "keep_first": KEEP_FIRST}}}
        mem = {"type": "mlstm", "mlp": None, "mixer": dict(zip(("heads", "dim", "vdim"), z["mem"]), gate_cap=GATE_CAP)}
        layers = ([att, mem, mem, att] * case["layers"])[: case["layers"]]
        return {"architecture": "Dilavik", "embedding": {"scale": 1.0}, "norm": {"eps": EPS, "groups": GROUPS}, "layers": layers,
                "vocab": z["vocab"], "width": z["width"]}
    mlp = {"kind": "dense", "ff": z["ff"], "limit": GLU_LIMIT}
    att = {"type": "attention", "mlp": mlp, "mixer": {"heads": z["heads"], "kv_heads": z["kv"], "dim": 128, "vdim": 128,
           "rot": {"dims": 128, "base": ROPE_BASE}, "scale": 128 ** -0.5, "mask": {"size": WINDOW}}}
    lat = {"type": "latent_attention", "mlp": mlp, "mixer": dict(zip(("heads", "dim", "rot_dim", "vdim", "kv_rank"), z["latent"]),
           rot={"dims": 64, "base": ROPE_BASE}, scale=192 ** -0.5, mask={"size": WINDOW})}
    return {"architecture": "Nulunex", "norm": {"eps": EPS}, "layers": ([att, lat] * case["layers"])[: case["layers"]],
            "vocab": z["vocab"], "width": z["width"]}


def _hybrid_layer(w, cfg, i):
    H, layer = cfg["width"], cfg["layers"][i]
    c, p = layer["mixer"], f"l{i}."
    mat = {}
    if layer["type"] == "attention":
        mat = {"q": (c["heads"] * c["dim"], H), "k": (c["kv_heads"] * c["dim"], H), "o": (H, c["heads"] * c["vdim"])}
        if cfg["architecture"] == "Dilavik":
            mat.update(v=(c["kv_heads"] * c["vdim"], H), g=(c["heads"], H))
    elif layer["type"] == "mlstm":
        mat = {"q": (c["heads"] * c["dim"], H), "k": (c["heads"] * c["dim"], H), "v": (c["heads"] * c["vdim"], H), "g": (c["heads"] * c["vdim"], H),
               "i": (c["heads"], H), "f": (c["heads"], H), "o": (H, c["heads"] * c["vdim"])}
    else:
        mat = {"q": (c["heads"] * (c["dim"] + c["rot_dim"]), H), "dkv": (c["kv_rank"] + c["rot_dim"], H), "uk": (c["heads"] * c["dim"], c["kv_rank"]),
               "uv": (c["heads"] * c["vdim"], c["kv_rank"]), "o": (H, c["heads"] * c["vdim"])}
    out = {f"{p}mix.{k}": w.matrix(f"{p}mix.{k}", *s) for k, s in mat.items()}
    if layer["type"] == "mlstm":
        out[p + "mix.norm"] = w.gain(p + "mix.norm", c["heads"] * c["vdim"])
        out[p + "mix.i.b"] = w.normal(p + "mix.i.b", (c["heads"],), 0.5)
        out[p + "mix.f.b"] = w.normal(p + "mix.f.b", (c["heads"],), 1.0, 4.0)  # gates that remember
    if layer["type"] == "latent_attention":
        out[p + "mix.dkv.norm"] = w.gain(p + "mix.dkv.norm", c["kv_rank"])
        out[p + "mix.sink"] = w.normal(p + "mix.sink", (c["heads"],), 1.0)
    out[p + "norm1"] = w.gain(p + "norm1", H)
    if layer["mlp"] is not None:
        ff = layer["mlp"]["ff"]
        for k in ("up",) if cfg["architecture"] == "Dilavik" else ("gate", "up"):
            out[f"{p}mlp.{k}"] = w.matrix(f"{p}mlp.{k}", ff, H)
        out[p + "mlp.down"] = w.matrix(p + "mlp.down", H, ff)
        out[p + "norm2"] = w.gain(p + "norm2", H)
        if cfg["architecture"] == "Dilavik":
            out[p + "mlp.act"] = w.normal(p + "mlp.act", (2,), 0.5)
    if cfg["architecture"] == "Dilavik":  # mostly the layer's own result goes on
        out[p + "dwa"] = w.normal(p + "dwa", (i + 2,), 0.1)
        out[p + "dwa"][-1] += 1.0
    return out


def _is_wrong(t):
    """Tokens after which the drafter guesses wrongly."""
    return (t * 40503 >> 4) % 4 == 0


def _drafter_weights(w, z):
    H, R, V = z["width"], z["draft_layers"], z["vocab"]
    E = 2 * H
    out = {"rnn_w.weight": w.matrix("rnn_w", H, H), "rnn_u.weight": w.matrix("rnn_u", H, H).mul_(0.2), "rnn_u.bias": w.normal("rnn_u.b", (H,), 0.1)}
    for r in range(R):
        out[f"lm_head.{r}.linear.weight"] = w.matrix(f"res{r}", E, E).mul_(0.3)
        out[f"lm_head.{r}.linear.bias"] = w.normal(f"res{r}.b", (E,), 0.1)
    # the state after reading token t, roughly; its row in the vocabulary layer is that of t + 1, or of t + 2 where the guess is wrong
    state = F.silu((w.embedding(z) @ out["rnn_w.weight"].T).float())
    mark = state - state.mean(dim=0)
    mark *= DRAFT_LOGIT / mark.square().sum(dim=1).mean()
    wrong = _is_wrong(torch.arange(V, device="cuda"))[:, None]
    rows = torch.roll(torch.where(wrong, -mark, mark), 1, dims=0) + torch.roll(torch.where(wrong, mark, torch.zeros_like(mark)), 2, dims=0)
    vocab = w.matrix("vocab", V, E).mul_(0.1)
    vocab[:, H:] += rows.to(w.dtype)
    out[f"lm_head.{R}.weight"] = vocab
    return out


def _llama(case, seed):
    from transformers.models.llama.configuration_llama import LlamaConfig

    z = SHAPES[case["shape"]]
    cfg = LlamaConfig(hidden_size=z["width"], num_attention_heads=z["heads"], num_key_value_heads=z["kv"], num_hidden_layers=case["layers"],
                      intermediate_size=z["ff"], vocab_size=z["vocab"], rms_norm_eps=EPS, hidden_act="silu", pad_token_id=0)
    cfg.rope_theta = ROPE_BASE
    w = Weights(seed, _dtype(z))
    sd = {"model.embed_tokens.weight": w.embedding(z), "lm_head.weight": w.head(z), "model.norm.weight": w.gain("norm", z["width"])}
    for i in range(case["layers"]):
        sd.update(_llama_layer(w, z, i))
    with torch.device("cuda"):
        llm = rd.modeling_llama.LlamaForCausalLM(cfg).to(w.dtype)
    llm.load_state_dict(sd)
    return llm


def _model(case, seed):
    if case.get("design", "llama") == "llama":
        return _llama(case, seed)
    z = SHAPES[case["shape"]]
    cfg, w = _design(case, z), Weights(seed, _dtype(z))
    sd = {"embed": w.embedding(z), "head": w.head(z), "final.norm": w.gain("final.norm", z["width"])}
    for i in range(case["layers"]):
        sd.update(_hybrid_layer(w, cfg, i))
    llm = rd.registry.new_model(cfg, w.dtype, "cuda")
    llm.load_state_dict(sd)
    return llm


def _prompts(case, seed):
    """Left-padded token ids: the first row fills the width, the others are shorter."""
    z, B, L = SHAPES[case["shape"]], case["batch"], case["prompt"]
    g = torch.Generator().manual_seed(seed * 7919 + B)
    ids = torch.randint(1, z["vocab"], (B, L), generator=g)
    for b in range(1, B):
        ids[b, : int(torch.randint(0, L // 2 + 1, (1,), generator=g))] = 0
    return ids


def _beams(case, seed):
    """Draft beams that share their first token and many of their prefixes, as beam search leaves them."""
    z, B, W, L = SHAPES[case["shape"]], case["batch"], case["beams"], case["length"]
    g = torch.Generator().manual_seed(seed * 104729 + W)
    first = torch.randint(1, z["vocab"], (B, 1, 1), generator=g)
    branch = torch.randint(0, 1 << 30, (B, W, L), generator=g).float().div_(1 << 30).pow_(3).mul_(max(3, 2 * W // L)).long()
    branch[:, :, 0] = 0
    path = branch.cumsum(-1) * 7919 % (z["vocab"] - 1)  # a child's id hangs on its branch
    return (first + path) % (z["vocab"] - 1) + 1


# ------------------------------------------------------------------------------------------------------- prepare, run
def prepare(case, seed):
    z = SHAPES[case["shape"]]
    s = dict(case, seed=seed)
    with torch.no_grad():
        s["llm"] = llm = _model(case, seed)
        if case["kind"] == "speculative":
            E = 2 * z["width"]
            with torch.device("cuda"):
                drafter = rd.modeling_drafter.Drafter(rd.configuration_drafter.DrafterConfig(
                    vocab_size=z["vocab"], hidden_size=z["width"], exit_dim=E, num_draft_layers=z["draft_layers"], rnn=True)).to(_dtype(z))
            drafter.load_state_dict(_drafter_weights(Weights(seed, _dtype(z)), z))
            s["model"] = rd.RecurrentDrafting(llm, drafter)
        if case["kind"] in ("speculative", "autoregressive"):
            s["ids"] = _prompts(case, seed).cuda()
            s["sampling"] = rd.SamplingArgs(case["temperature"] or 1.0, not case["temperature"])
        if case["kind"] == "prompt":
            s["counts"] = [int(v) for v in case["lengths"].split(",")]
            g = torch.Generator().manual_seed(seed * 7919)
            s["tokens"] = [torch.randint(1, z["vocab"], (n,), generator=g).cuda() for n in s["counts"]]
            s["session"] = rd.session.Session(llm, len(s["counts"]), max(s["counts"]) + 1)
        if case["kind"] == "verify":
            B, S = case["batch"], case["prompt"]
            s["beams"] = _beams(case, seed).cuda()
            s["padding_mask"] = torch.ones(B, S, dtype=torch.int64, device="cuda")
            s["cache"] = cache = llm.new_cache(B, S + case["beams"] * case["length"])
            g = torch.Generator().manual_seed(seed * 7919 + B)
            ids = torch.randint(1, z["vocab"], (B, S), generator=g).cuda()
            llm.forward(ids, rd.attention.causal_mask(s["padding_mask"], S, ids.device), torch.arange(S, device="cuda").expand(B, S), cache.sliced)
    return s


def run(s):
    return {"speculative": _run_speculative, "autoregressive": _run_autoregressive, "prompt": _run_prompt, "verify": _run_verify}[s["kind"]](s)


def _run_speculative(s):
    torch.manual_seed(s["seed"])
    model, tokens = s["model"], None
    for tokens in model.generate(rd.stats.Ledger(), s["ids"], s["prompt"] + s["new"], rd.modeling_drafter.BeamShape(s["beams"], s["length"]),
                                 s["sampling"], rd.SpecialTokens(0, None)):
        pass
    rows = model.last_state.ctx  # hidden states that the next tokens are chosen from
    with torch.no_grad():
        logits = s["llm"].lm_logits(rows, torch.empty(rows.shape[0], SHAPES[s["shape"]]["vocab"], dtype=torch.float32, device="cuda"))
    return {"tokens": tokens, "hidden": rows, "logits": logits}


def _run_autoregressive(s):
    torch.manual_seed(s["seed"])
    llm, tokens, B = s["llm"], None, s["batch"]
    for tokens in rd.autoregressive.generate(llm, s["ids"], s["prompt"] + s["new"], rd.SpecialTokens(0, None), s["sampling"]):
        pass
    rows = llm.workspace(B, B)["hidden"]  # of the step that chose the last tokens
    with torch.no_grad():
        logits = llm.lm_logits(rows, torch.empty(B, SHAPES[s["shape"]]["vocab"], dtype=torch.float32, device="cuda"))
    return {"tokens": tokens, "hidden": rows, "logits": logits}


def _portions(counts, portion):
    """Lists of (from, to) per row: everything at once, or `portion` tokens of every row that still has some."""
    if not portion:
        yield [(0, n) for n in counts]
        return
    for at in range(0, max(counts), portion):
        yield [(min(at, n), min(at + portion, n)) for n in counts]


def _run_prompt(s):
    session, counts = s["session"], s["counts"]
    for b in range(len(counts)):
        session.release(b)
    hidden, last = [], [None] * len(counts)
    for spans in _portions(counts, s["portion"]):
        ids = torch.cat([t[a:b] for t, (a, b) in zip(s["tokens"], spans)])
        rows = session.extend(ids, [b - a for a, b in spans])
        if s["portion"]:
            rows = rows.clone()  # the next portion uses the same buffer
        hidden.append(rows)
        end = 0
        for r, (a, b) in enumerate(spans):
            end += b - a
            if b > a and b == counts[r]:
                last[r] = rows[end - 1]
    out = {f"hidden{i}": h for i, h in enumerate(hidden)}
    out["logits"] = session.logits(torch.stack(last))
    return out


def _run_verify(s):
    llm, cache, S = s["llm"], s["cache"], s["prompt"]
    cache.set_length(S)
    packed, unpacker, mask, offsets = rd.tree_attention.pack(s["beams"], s["padding_mask"])
    got = llm.forward(packed, mask, offsets + S, cache.sliced)
    return {"unpacker": unpacker, "logits": rd.tree_attention.unpack(got.logits, unpacker),
            "hidden": rd.tree_attention.unpack(got.hidden_states, unpacker)}


# --------------------------------------------------------------------------------------------------------------- work
def _matrix_sizes(case):
    """(weights of the layers' matrices, of the LM head, key/value bytes that a token leaves, state bytes of a row)."""
    z = SHAPES[case["shape"]]
    H, ff, e = z["width"], z["ff"], 4 if z["dtype"] == "float32" else 2
    hd = H // z["heads"]
    head, design = z["vocab"] * H, case.get("design", "llama")
    if design == "llama":
        return case["layers"] * (2 * H * H + 2 * z["kv"] * hd * H + 3 * H * ff), head, case["layers"] * 2 * z["kv"] * hd * e, 0
    w = kv = state = 0
    for layer in _design(case, z)["layers"]:
        c = layer["mixer"]
        if layer["type"] == "attention":
            w += H * (2 * c["heads"] + (2 if design == "dilavik" else 1) * c["kv_heads"]) * 128
            kv += 2 * c["kv_heads"] * 128 * e
        elif layer["type"] == "mlstm":
            w += H * c["heads"] * (2 * c["dim"] + 3 * c["vdim"])
            state += 4 * c["heads"] * c["dim"] * (c["vdim"] + 1)
        else:
            w += H * (c["heads"] * (c["dim"] + c["rot_dim"] + c["vdim"]) + c["kv_rank"] + c["rot_dim"]) + c["heads"] * 256 * c["kv_rank"]
            kv += (c["kv_rank"] + c["rot_dim"]) * e
        if layer["mlp"] is not None:
            w += H * layer["mlp"]["ff"] * (2 if design == "dilavik" else 3)
    return w, head, kv, state


def work(case):
    z = SHAPES[case["shape"]]
    H, V, e = z["width"], z["vocab"], 4 if z["dtype"] == "float32" else 2
    layers, head, kv, state = _matrix_sizes(case)
    reach = WINDOW if case.get("design", "llama") != "llama" else 1 << 30  # keys that a token looks back on

    def attention(queries, keys):
        return 4.0 * case["layers"] * H * queries * min(keys, reach)

    if case["kind"] == "prompt":
        counts = [int(v) for v in case["lengths"].split(",")]
        M = sum(counts)
        return {"bytes": layers * e + head * e + M * (2 * H * e + kv) + len(counts) * (V * 4 + state),
                "flops": 2.0 * layers * M + 2.0 * head * len(counts) + sum(attention(n, n / 2) for n in counts)}
    B, S = case["batch"], case["prompt"]
    if case["kind"] == "verify":
        M = B * case["beams"] * (case["length"] + 1) // 2  # distinct prefixes, about
        return {"bytes": (layers + head) * e + B * S * kv + M * H * e + B * case["beams"] * case["length"] * (V * 4 + H * e),
                "flops": 2.0 * (layers + head) * M + attention(M, S)}
    tokens = B * S * 0.75 + B * S * 0.25 / B  # the first row is full, the others three quarters on average
    prompt = {"bytes": layers * e + tokens * kv, "flops": 2.0 * layers * tokens + attention(tokens, S / 2)}
    if case["kind"] == "autoregressive":
        n = case["new"]
        each = (layers + head) * e + B * (min(S, reach) * kv + 2 * state + V * 4)
        return {"bytes": prompt["bytes"] + n * each, "flops": prompt["flops"] + n * (2.0 * (layers + head) * B + attention(B, S))}
    W, L = case["beams"], case["length"]
    steps = max(1, round(case["new"] / min(L, 3.05)))  # three guesses in four are right
    E = 2 * H
    draft = 2 * H * H + z["draft_layers"] * E * E + E * V
    M = B * 2 * W
    each = (layers + head) * e + (L - 1) * draft * e + B * S * kv
    return {"bytes": prompt["bytes"] + steps * each,
            "flops": prompt["flops"] + steps * (2.0 * (layers + head) * M + 2.0 * (L - 2) * draft * B * W + 2.0 * draft * B + attention(M, S))}


def tolerance(case):
    """Relative error of bf16 activations through the stack (32-bit for the small model); tokens are decided by a margin."""
    if SHAPES[case["shape"]]["dtype"] == "float32":
        return {"rel": 4e-6, "max": 2e-5}
    if case.get("design", "llama") == "llama":  # the residual stream is bf16 too
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 0.02, "max": 0.2}


# -------------------------------------------------------------------------------------------------------------- exact
def _rms(x, eps=EPS):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _rotate(x, pos, dims, neighbours=False):
    """x [T, heads, d] turned by position: feature i with i + dims/2, or 2i with 2i + 1."""
    a = pos.double()[:, None] * ROPE_BASE ** (-2.0 * torch.arange(dims // 2, device=x.device, dtype=torch.float64) / dims)
    c, s, y = a.cos()[:, None], a.sin()[:, None], x.clone()
    u, v = (x[..., 0:dims:2], x[..., 1:dims:2]) if neighbours else (x[..., : dims // 2], x[..., dims // 2 : dims])
    at = (slice(0, dims, 2), slice(1, dims, 2)) if neighbours else (slice(0, dims // 2), slice(dims // 2, dims))
    y[..., at[0]], y[..., at[1]] = u * c - v * s, v * c + u * s
    return y


def _attend(q, k, v, visible, scale, sink=None):
    """q [T, heads, d], k and v [T, kv heads, d]; visible(queries) -> [len(queries), T] bool; sink [heads]."""
    T, nh, group = q.shape[0], q.shape[1], q.shape[1] // k.shape[1]
    out = torch.empty(T, nh, v.shape[2], dtype=torch.float64, device=q.device)
    for at in range(0, T, 1024):
        rows = torch.arange(at, min(at + 1024, T), device=q.device)
        see = visible(rows)
        for h in range(nh):
            s = (q[rows, h] @ k[:, h // group].T * scale).masked_fill(~see, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(len(rows), 1)], dim=1)
            p = torch.softmax(s, dim=-1)
            out[rows, h] = p[:, :T] @ v[:, h // group]
    return out


def _causal(T):
    j = torch.arange(T, device="cuda")
    return lambda i: j[None] <= i[:, None]


def _llama_exact(case, seed, rows):
    """Final hidden states of every (token ids, positions, visible) in rows."""
    z = SHAPES[case["shape"]]
    w, hd = Weights(seed, _dtype(z)), z["width"] // z["heads"]
    embed = w.embedding(z)
    xs = [embed[ids].double() for ids, _, _ in rows]
    for i in range(case["layers"]):
        m = {k.split(".", 3)[3][: -len(".weight")]: v.double() for k, v in _llama_layer(w, z, i).items()}
        for r, (_, pos, visible) in enumerate(rows):
            x = xs[r]
            h = _rms(x) * m["input_layernorm"]
            q, k, v = ((h @ m[f"self_attn.{n}_proj"].T).unflatten(1, (-1, hd)) for n in "qkv")
            o = _attend(_rotate(q, pos, hd), _rotate(k, pos, hd), v, visible, hd ** -0.5)
            x = x + o.flatten(1) @ m["self_attn.o_proj"].T
            h = _rms(x) * m["post_attention_layernorm"]
            xs[r] = x + (F.silu(h @ m["mlp.gate_proj"].T) * (h @ m["mlp.up_proj"].T)) @ m["mlp.down_proj"].T
    return [_rms(x) * w.gain("norm", z["width"]).double() for x in xs]


def _memory_exact(h, m, c):
    """The matrix memory, token by token."""
    T, nh, d, dv = h.shape[0], c["heads"], c["dim"], c["vdim"]
    q, k = (h @ m["q"].T).view(T, nh, d) * d ** -0.5, (h @ m["k"].T).view(T, nh, d)
    v = (h @ m["v"].T).view(T, nh, dv)
    i = GATE_CAP * torch.tanh((h @ m["i"].T + m["i.b"]) / GATE_CAP)
    f = F.logsigmoid(GATE_CAP * torch.tanh((h @ m["f.w"].T + m["f.b"]) / GATE_CAP))
    top = torch.empty_like(i)
    cur = torch.zeros_like(i[0])
    for t in range(T):
        cur = top[t] = torch.maximum(f[t] + cur, i[t])
    before = torch.cat([torch.zeros_like(top[:1]), top[:-1]])
    keep, take = torch.exp(f + before - top), torch.exp(i - top)
    S = torch.zeros(nh, d, dv + 1, dtype=torch.float64, device=h.device)  # the last column is the normaliser
    v1 = torch.cat([v, torch.ones_like(v[..., :1])], dim=-1) * take[..., None]
    o = torch.empty(T, nh, dv + 1, dtype=torch.float64, device=h.device)
    for t in range(T):
        S.mul_(keep[t, :, None, None]).baddbmm_(k[t, :, :, None], v1[t, :, None, :])
        o[t] = torch.bmm(q[t, :, None, :], S)[:, 0]
    den = torch.maximum(o[..., dv].abs(), torch.exp(-top)) + 1e-6
    return _rms(o[..., :dv] / den[..., None]).flatten(1) * m["norm"] * torch.sigmoid(h @ m["g"].T) @ m["o"].T


def _mix_exact(h, m, layer, pos, dilavik):
    c, T = layer["mixer"], h.shape[0]
    j = torch.arange(T, device=h.device)
    if layer["type"] == "mlstm":
        return _memory_exact(h, dict(m, **{"f.w": m["f"]}), c)
    if layer["type"] == "attention":
        q, k = (h @ m["q"].T).unflatten(1, (-1, 128)), (h @ m["k"].T).unflatten(1, (-1, 128))
        qr, kr = _rotate(q, pos, c["rot"]["dims"]), _rotate(k, pos, c["rot"]["dims"])
        if dilavik:
            o = _attend(qr, kr, (h @ m["v"].T).unflatten(1, (-1, 128)),
                        lambda i: (j <= i[:, None]) & ((i[:, None] - j < WINDOW) | (j < KEEP_FIRST)), c["scale"])
            o = o * torch.sigmoid(h @ m["g"].T)[:, :, None]
        else:
            zero = torch.zeros(c["heads"], dtype=torch.float64, device=h.device)
            o = _attend(_rms(qr), _rms(kr), k, lambda i: (j <= i[:, None]) & (i[:, None] // WINDOW == j // WINDOW), c["scale"], zero)
        return o.flatten(1) @ m["o"].T
    d, r = c["dim"], c["kv_rank"]
    q = (h @ m["q"].T).unflatten(1, (-1, d + c["rot_dim"]))
    q = torch.cat([q[..., :d], _rotate(q[..., d:], pos, c["rot"]["dims"], True)], dim=-1)
    y = h @ m["dkv"].T
    lat, kr = _rms(y[:, :r]) * m["dkv.norm"], _rotate(y[:, None, r:], pos, c["rot"]["dims"], True)
    k = torch.cat([(lat @ m["uk"].T).unflatten(1, (-1, d)), kr.expand(-1, c["heads"], -1)], dim=-1)
    o = _attend(q, k, (lat @ m["uv"].T).unflatten(1, (-1, c["vdim"])), lambda i: (j <= i[:, None]) & (i[:, None] - j < WINDOW), c["scale"], m["sink"])
    return o.flatten(1) @ m["o"].T


def _group_norm(x, groups):
    return _rms(x.unflatten(-1, (groups, -1))).flatten(-2)


def _hybrid_exact(case, seed, rows):
    z = SHAPES[case["shape"]]
    cfg, w = _design(case, z), Weights(seed, _dtype(z))
    dilavik = cfg["architecture"] == "Dilavik"
    groups, embed = GROUPS if dilavik else 1, w.embedding(z)
    xs = [embed[ids].double() for ids, _, _ in rows]
    history = [[x] for x in xs]
    for i, layer in enumerate(cfg["layers"]):
        m = {k.split(".", 1)[1]: v.double() for k, v in _hybrid_layer(w, cfg, i).items()}
        mix = {k[4:]: v for k, v in m.items() if k.startswith("mix.")}
        for r, (_, pos, _) in enumerate(rows):
            x = xs[r] + _mix_exact(_group_norm(xs[r], groups) * m["norm1"], mix, layer, pos, dilavik)
            if layer["mlp"] is not None:
                h = _group_norm(x, groups) * m["norm2"]
                u = h @ m["mlp.up"].T
                if dilavik:
                    p, q = F.softplus(m["mlp.act"])
                    low = u.clamp(max=0.0)
                    a = torch.where(u > 0, p * u * u, (0.5 + q) * (torch.expm1(low) - low)) + u / 2
                else:
                    g = (h @ m["mlp.gate"].T).clamp(max=GLU_LIMIT)
                    a = g * torch.sigmoid(GLU_ALPHA * g) * (u.clamp(-GLU_LIMIT, GLU_LIMIT) + 1.0)
                x = x + a @ m["mlp.down"].T
            if dilavik:
                history[r].append(x)
                x = sum(c * y for c, y in zip(m["dwa"], history[r]))
            xs[r] = x
    return [_group_norm(x, groups) * w.gain("final.norm", z["width"]).double() for x in xs]


def _hidden_exact(case, seed, sequences):
    rows = [(ids, torch.arange(len(ids), device="cuda"), _causal(len(ids))) for ids in (s.cuda() for s in sequences)]
    return (_llama_exact if case.get("design", "llama") == "llama" else _hybrid_exact)(case, seed, rows)


def _follow(t, n, vocab):
    """n tokens after t."""
    return (t + 1 + torch.arange(n)) % vocab


def _speculative_exact(case, seed):
    """Tokens and lengths as the planted pair leaves them."""
    V, L = SHAPES[case["shape"]]["vocab"], case["length"]
    rows = [r[r != 0] for r in _prompts(case, seed)]
    most = case["prompt"] + case["new"]
    while True:
        for b, r in enumerate(rows):
            new = [(int(r[-1]) + 1) % V]
            while len(new) < L and not _is_wrong(new[-1]):
                new.append((new[-1] + 1) % V)
            rows[b] = torch.cat([r, torch.tensor(new)])
        longest = max(len(r) for r in rows)
        if longest + 1 >= most:
            break
    out = torch.zeros(len(rows), longest + 1, dtype=torch.int64)
    for b, r in enumerate(rows):
        out[b, longest - len(r) : longest], out[b, longest] = r, (int(r[-1]) + 1) % V
    return rows, out[:, :most]


def exact(case, seed):
    with torch.no_grad():
        z, w = SHAPES[case["shape"]], Weights(seed, _dtype(SHAPES[case["shape"]]))
        head = w.head(z)
        if case["kind"] == "prompt":
            g = torch.Generator().manual_seed(seed * 7919)
            counts = [int(v) for v in case["lengths"].split(",")]
            hidden = _hidden_exact(case, seed, [torch.randint(1, z["vocab"], (n,), generator=g) for n in counts])
            out = {f"hidden{i}": torch.cat([h[a:b] for h, (a, b) in zip(hidden, spans)]) for i, spans in enumerate(_portions(counts, case["portion"]))}
            out["logits"] = torch.stack([h[-1] for h in hidden]) @ head.double().T
            return out
        if case["kind"] == "verify":
            B, S, W, L = case["batch"], case["prompt"], case["beams"], case["length"]
            g = torch.Generator().manual_seed(seed * 7919 + B)
            ids, beams = torch.randint(1, z["vocab"], (B, S), generator=g), _beams(case, seed)
            j = torch.arange(S + W * L, device="cuda")
            beam, place = torch.where(j < S, -1, (j - S) // L), torch.where(j < S, j, S + (j - S) % L)
            see = ((beam[None] == -1) | (beam[None] == beam[:, None])) & (place[None] <= place[:, None])
            rows = [(torch.cat([ids[b], beams[b].flatten()]).cuda(), place, lambda i: see[i]) for b in range(B)]
            hidden = torch.stack([h[S:] for h in _llama_exact(case, seed, rows)]).view(B, W, L, -1)
            return {"unpacker": None, "logits": hidden @ head.double().T, "hidden": hidden}
        if case["kind"] == "speculative":
            rows, tokens = _speculative_exact(case, seed)
        else:
            ids = _prompts(case, seed)
            new = torch.stack([_follow(int(r[-1]), case["new"], z["vocab"]) for r in ids])
            tokens = torch.cat([ids, new], dim=1)
            rows = [t[t[: case["prompt"]].eq(0).sum() : -1] for t in tokens]
        hidden = torch.stack([h[-1] for h in _hidden_exact(case, seed, rows)])
        return {"tokens": tokens, "hidden": hidden, "logits": hidden @ head.double().T}
