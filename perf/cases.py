"""The calls this package is timed on: quantized LLaMA inference (one token of a running generation, a prompt, the feed-forward at
batch and prompt sizes in int4 and llm.int8) and the layers of the folder-loaded families (latent attention, rotary softmax
attention, mixture of experts, matrix memory), each through the module a program calls.

A case names a ``kind`` and its sizes.  ``prepare`` makes what a program holds before the call, ``run`` is the call, ``exact`` the
same result in 64 bits from plain torch.  Weights and inputs come from the seed alone, on the GPU."""
import math
import sys
from pathlib import Path

import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "lit-llama-ja_b200"))

from lit_llama.latent_attention import LatentAttention, LatentAttentionSpec  # noqa: E402
from lit_llama.model import MLP, LLaMA, LLaMAConfig  # noqa: E402
from lit_llama.moe import MoE, MoESpec  # noqa: E402
from lit_llama.quantization import ColBlockQuantizedLinear  # noqa: E402
from lit_llama.recurrence import MatrixMemoryMixer, MatrixMemorySpec  # noqa: E402
from lit_llama.rotary import RotarySpec  # noqa: E402
from lit_llama.softmax_attention import SoftmaxAttention, SoftmaxAttentionSpec  # noqa: E402
from lit_llama.utils import EmptyInitOnDevice, quantization  # noqa: E402

DEV, BF = "cuda", torch.bfloat16
EPS = 1e-5


def listed():
    return [
        # one token of a running batch-1 generation after a 512-token prompt: four blocks of the 7B model, replayed as one graph
        dict(name="llama_int4_token", kind="llama_token", width=4096, heads=32, layers=4, vocab=32000, group=128, prompt=512, seq=768),
        # the prompt of such a request
        dict(name="llama_int4_prompt", kind="llama_prompt", width=4096, heads=32, layers=2, vocab=32000, group=128, batch=1, prompt=512,
             seq=768),
        # feed-forward of the 13B model over eight prompts of 2048 tokens
        dict(name="int4_mlp_prompts", kind="int4_mlp", width=5120, group=128, rows=16384),
        # feed-forward of the 7B model in a batch of 32 single tokens
        dict(name="int4_mlp_batch", kind="int4_mlp", width=4096, group=128, rows=32),
        # the same under llm.int8, and a 512-token prompt under llm.int8
        dict(name="int8_mlp_batch", kind="int8_mlp", width=4096, rows=32, outliers=6),
        dict(name="int8_mlp_prompt", kind="int8_mlp", width=4096, rows=512, outliers=6),
        # latent attention: a prompt, and one token over a filled cache
        dict(name="latent_prompt", kind="latent", width=2048, heads=16, nope=128, rot=64, v=128, rank=512, window=1024, batch=1,
             past=0, tokens=2048),
        dict(name="latent_token", kind="latent", width=2048, heads=16, nope=128, rot=64, v=128, rank=512, window=1024, batch=1,
             past=2048, tokens=1),
        # mixture of experts with a shared expert: a prompt, and one token
        dict(name="moe_prompt", kind="moe", width=2048, experts=32, top=4, ff=1024, shared=1536, tokens=2048),
        dict(name="moe_token", kind="moe", width=2048, experts=32, top=4, ff=1024, shared=1536, tokens=1),
        # rotary softmax attention over the whole past, capped scores and a gate: a prompt
        dict(name="softmax_prompt", kind="softmax", width=2048, heads=16, kv_heads=4, dim=128, cap=50.0, window=0, chunk=0, sink=False,
             norm=False, batch=1, past=0, tokens=2048),
        # matrix memory with exponential gates: a prompt
        dict(name="matrix_memory_prompt", kind="matrix_memory", width=2048, heads=8, dim=128, vdim=256, batch=1, tokens=2048),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["llama_token", "llama_prompt", "int4_mlp", "int4_mlp", "int8_mlp", "latent", "latent", "moe", "softmax", "softmax",
                       "matrix_memory"])
    if kind in ("llama_token", "llama_prompt"):
        width, heads = rng.choice([(2048, 16), (4096, 32), (5120, 40)])
        c = dict(kind=kind, width=width, heads=heads, layers=rng.randint(1, 3), vocab=32000, group=rng.choice([128, 128, -1]))
        if kind == "llama_token":
            c["prompt"] = _log_int(rng, 2, 1500)
        else:
            c["batch"] = rng.randint(1, 3)
            c["prompt"] = _log_int(rng, 17, 2048 // c["batch"])
        c["seq"] = min(2048, c["prompt"] + _log_int(rng, 16, 512))
        return c
    if kind == "int4_mlp":
        return dict(kind=kind, width=rng.choice([2048, 4096, 5120]), group=rng.choice([128, 128, -1]), rows=_log_int(rng, 1, 16000))
    if kind == "int8_mlp":
        return dict(kind=kind, width=rng.choice([2048, 4096, 5120]), rows=_log_int(rng, 1, 2048), outliers=rng.randint(0, 12))
    width, heads = rng.choice([(1024, 8), (2048, 16), (4096, 32)])
    step = rng.random() < 0.3
    batch, tokens = rng.randint(1, 4 if step else 2), 1 if step else _log_int(rng, 2, 2048)
    past = _log_int(rng, 1, 2048) if step else rng.choice([0, 0, rng.randint(1, 700)])
    if kind == "latent":
        return dict(kind=kind, width=width, heads=heads, nope=rng.choice([64, 128]), rot=rng.choice([32, 64]), v=rng.choice([64, 128]),
                    rank=rng.choice([256, 512]), window=rng.choice([0, 512, 1024, 1500]), batch=batch, past=past, tokens=tokens)
    if kind == "moe":
        return dict(kind=kind, width=width, experts=rng.choice([16, 32]), top=rng.choice([2, 4]), ff=rng.choice([768, 1024, 2048]),
                    shared=rng.choice([0, 1280, 1536]), tokens=batch if step else _log_int(rng, 2, 3000))
    if kind == "softmax":
        window, chunk = rng.choice([(0, 0), (0, 0), (rng.randint(100, 1500), 0), (0, rng.choice([512, 1024]))])
        return dict(kind=kind, width=width, heads=heads, kv_heads=heads // rng.choice([1, 2, 4]), dim=rng.choice([64, 96, 128]),
                    cap=rng.choice([0.0, 50.0]), window=window, chunk=chunk, sink=rng.random() < 0.4, norm=rng.random() < 0.4, batch=batch,
                    past=past, tokens=tokens)
    return dict(kind=kind, width=width, heads=rng.choice([4, 8]), dim=rng.choice([64, 128]), vdim=rng.choice([128, 256]), batch=rng.randint(1, 2),
                tokens=_log_int(rng, 2, 2048))


# ------------------------------------------------------------------------------------------------------------------ tensors of a case
class _Rand:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, scale=1.0, dtype=BF):
        return (torch.randn(shape, generator=self.g, device=DEV) * scale).to(dtype)

    def rows(self, n, k):
        """A weight ``[n, k]`` that keeps the size of what passes through it."""
        return self.normal(n, k, scale=k ** -0.5)

    def ids(self, vocab, *shape):
        return torch.randint(0, vocab, shape, generator=self.g, device=DEV)

    def int4(self, n, k, group):
        """(codes [n, k], scales, zeros [n, groups]): round-to-nearest 4-bit weights of standard deviation 0.02, per group of columns."""
        t = k if group == -1 else group
        w = (torch.randn((n, k), generator=self.g, device=DEV) * 0.02).view(n, k // t, t)
        lo, hi = w.amin(-1), w.amax(-1)
        scales = ((hi - lo) / 15.0).to(BF)
        zeros = torch.round(-lo / ((hi - lo) / 15.0)).to(BF)
        codes = torch.clamp(torch.round(w / scales.float()[..., None]) + zeros.float()[..., None], 0, 15).to(torch.uint8)
        return codes.view(n, k), scales, zeros


def _hidden(width):
    return LLaMAConfig(n_embd=width).n_hidden


def _int4_names(width):
    h = _hidden(width)
    return [("mlp.c_fc1", h, width), ("mlp.c_fc2", h, width), ("mlp.c_proj", width, h)]


def _llama_tensors(c, r):
    E, V = c["width"], c["vocab"]
    t = {"wte": r.normal(V, E, scale=2.0)}
    for i in range(c["layers"]):
        for name, n, k in [("attn.c_attn", 3 * E, E), ("attn.c_proj", E, E)] + _int4_names(E):
            t[f"h.{i}.{name}"] = r.int4(n, k, c["group"])
        t[f"h.{i}.rms_1"], t[f"h.{i}.rms_2"] = 1.0 + r.normal(E, scale=0.1), 1.0 + r.normal(E, scale=0.1)
    t["ln_f"] = 1.0 + r.normal(E, scale=0.1)
    t["lm_head"] = r.int4(V, E, c["group"])
    n = c["prompt"] + (1 if c["kind"] == "llama_token" else 0)
    t["idx"] = r.ids(V, c.get("batch", 1), n)
    return t


def _latent_tensors(c, r):
    E, H = c["width"], c["heads"]
    w = {"q": r.rows(H * (c["nope"] + c["rot"]), E), "g": r.rows(H, E), "dkv": r.rows(c["rank"] + c["rot"], E),
         "dkv.norm": (1.0 + r.normal(c["rank"], scale=0.1)).float(), "uk": r.rows(H * c["nope"], c["rank"]),
         "uv": r.rows(H * c["v"], c["rank"]), "o": r.rows(E, H * c["v"])}
    x = r.normal(c["batch"] * c["tokens"], E)
    return w, x, r.normal(c["batch"], c["past"] + c["tokens"], c["rank"] + c["rot"])


def _softmax_tensors(c, r):
    E, H, G, D = c["width"], c["heads"], c["kv_heads"], c["dim"]
    w = {"q": r.rows(H * D, E), "k": r.rows(G * D, E), "v": r.rows(G * D, E), "g": r.rows(H * D, E), "o": r.rows(E, H * D)}
    if c["norm"]:
        w["q.norm"], w["k.norm"] = (1.0 + r.normal(H * D, scale=0.1)).float(), (1.0 + r.normal(G * D, scale=0.1)).float()
    if c["sink"]:
        w["sink"] = r.normal(H).float()
    x = r.normal(c["batch"] * c["tokens"], E)
    n = c["past"] + c["tokens"]
    return w, x, r.normal(c["batch"], n, G * D), r.normal(c["batch"], n, G * D)


def _moe_tensors(c, r):
    E, X, F = c["width"], c["experts"], c["ff"]
    w = {"router": r.rows(X, E).float(), "router.b": r.normal(X, scale=0.1).float()}
    for e in range(X):
        w[f"e{e}.gate"], w[f"e{e}.up"], w[f"e{e}.down"] = r.rows(F, E), r.rows(F, E), r.rows(E, F)
    if c["shared"]:
        w["shared.gate"], w["shared.up"], w["shared.down"] = r.rows(c["shared"], E), r.rows(c["shared"], E), r.rows(E, c["shared"])
        w["shared.sg"] = r.rows(1, E)
    return w, r.normal(c["tokens"], E)


def _memory_tensors(c, r):
    E, H = c["width"], c["heads"]
    hd, hv = H * c["dim"], H * c["vdim"]
    w = {"q": r.rows(hd, E), "k": r.rows(hd, E), "v": r.rows(hv, E), "g": r.rows(hv, E), "i": r.rows(H, E), "f": r.rows(H, E),
         "i.b": r.normal(H, scale=0.1).float(), "f.b": 3.0 + r.normal(H, scale=0.5).float(),
         "norm": (1.0 + r.normal(hv, scale=0.1)).float(), "o": r.rows(E, hv)}
    return w, r.normal(c["batch"] * c["tokens"], E)


def _int8_tensors(c, r):
    E, h = c["width"], _hidden(c["width"])
    w = {"c_fc1.weight": r.normal(h, E, scale=0.02), "c_fc2.weight": r.normal(h, E, scale=0.02), "c_proj.weight": r.normal(E, h, scale=0.02)}
    x = r.normal(c["rows"], E, scale=0.5, dtype=torch.float32)
    cols = torch.randperm(E, generator=r.g, device=DEV)[: c["outliers"]]       # the features that stand out in every token
    big = torch.randn((c["rows"], c["outliers"]), generator=r.g, device=DEV)
    x[:, cols] = torch.sign(big) * (8.0 + 2.0 * big.abs())
    return w, x.to(BF)


# ------------------------------------------------------------------------------------------------------------------ prepare and run
def _fill_int4(lin: ColBlockQuantizedLinear, codes, scales, zeros):
    lin.quant_weight.copy_(codes[:, 0::2] | (codes[:, 1::2] << 4))             # even columns in the low half of a byte
    lin.scales.copy_(scales)
    lin.zeros.copy_(zeros)


def _llama(c, t):
    cfg = LLaMAConfig(block_size=2048, vocab_size=c["vocab"], n_layer=c["layers"], n_head=c["heads"], n_embd=c["width"])
    with EmptyInitOnDevice(device=DEV, dtype=BF), quantization("gptq.int4", groupsize=c["group"]):
        m = LLaMA(cfg).eval()
    m.transformer.wte.weight.copy_(t["wte"])
    m.transformer.ln_f.scale.copy_(t["ln_f"])
    _fill_int4(m.lm_head, *t["lm_head"])
    for i, b in enumerate(m.transformer.h):
        b.rms_1.scale.copy_(t[f"h.{i}.rms_1"])
        b.rms_2.scale.copy_(t[f"h.{i}.rms_2"])
        for name in ("attn.c_attn", "attn.c_proj", "mlp.c_fc1", "mlp.c_fc2", "mlp.c_proj"):
            _fill_int4(b.get_submodule(name), *t[f"h.{i}.{name}"])
    return m


def _sms():
    return torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count


@torch.no_grad()
def prepare(case, seed):
    c, r = case, _Rand(seed)
    s = dict(c=c)
    if c["kind"].startswith("llama"):
        t = _llama_tensors(c, r)
        s["model"], s["idx"] = _llama(c, t), t["idx"]
        s["pos"] = torch.arange(c["prompt"], device=DEV)
        if c["kind"] == "llama_token":              # mid-generation: the prompt is in the cache and a token has been made
            s["model"](s["idx"][:, :-1], c["seq"], s["pos"])
            s["one"], s["at"] = s["idx"][:, -1:].contiguous(), torch.tensor([c["prompt"]], device=DEV)
            s["model"](s["one"], c["seq"], s["at"])
    elif c["kind"] == "int4_mlp":
        with EmptyInitOnDevice(device=DEV, dtype=BF), quantization("gptq.int4", groupsize=c["group"]):
            s["mlp"] = MLP(LLaMAConfig(n_embd=c["width"], n_head=c["width"] // 128)).eval()
        for name, n, k in _int4_names(c["width"]):
            _fill_int4(getattr(s["mlp"], name[4:]), *r.int4(n, k, c["group"]))
        s["x"] = r.normal(c["rows"], c["width"])
    elif c["kind"] == "int8_mlp":
        w, s["x"] = _int8_tensors(c, r)
        with EmptyInitOnDevice(device=DEV, dtype=BF), quantization("llm.int8"):
            s["mlp"] = MLP(LLaMAConfig(n_embd=c["width"], n_head=c["width"] // 128)).eval()
        s["mlp"].load_state_dict(w)
    else:
        s["pos"] = torch.arange(c.get("past", 0), c.get("past", 0) + c["tokens"], dtype=torch.int32, device=DEV)
        s["splits"] = 1
    if c["kind"] == "latent":
        w, s["x"], s["cache"] = _latent_tensors(c, r)
        spec = LatentAttentionSpec(width=c["width"], heads=c["heads"], nope_dim=c["nope"], rot_dim=c["rot"], v_dim=c["v"], kv_rank=c["rank"],
                                   window=c["window"] or None, scale=(c["nope"] + c["rot"]) ** -0.5, eps=EPS)
        n = c["past"] + c["tokens"]
        if c["tokens"] == 1:                        # few queries: the models share the window among blocks
            s["splits"] = max(1, min(16, (2 * _sms()) // (c["batch"] * ((c["heads"] + 31) // 32)), (min(c["window"] or n, n) + 63) // 64))
        s["mix"], s["rope"] = LatentAttention(spec, BF, DEV), spec.rope_table(n, DEV)
        s["mix"].load(w.__getitem__)
    elif c["kind"] == "softmax":
        w, s["x"], k, v = _softmax_tensors(c, r)
        s["caches"] = (k, v)
        spec = SoftmaxAttentionSpec(width=c["width"], heads=c["heads"], kv_heads=c["kv_heads"], dim=c["dim"], vdim=c["dim"],
                                    scale=c["dim"] ** -0.5, eps=EPS, rotary=RotarySpec(c["dim"] // 2), softcap=c["cap"],
                                    window=c["window"] or None, chunk=c["chunk"] or None, sink=c["sink"], qk_norm=c["norm"])
        n = c["past"] + c["tokens"]
        if c["tokens"] == 1:
            s["splits"] = max(1, min(64, (2 * _sms()) // ((c["batch"] * c["heads"] + 3) // 4), (min(spec.reach or n, n) + 127) // 128))
        s["mix"] = SoftmaxAttention(spec, BF, DEV)
        s["mix"].load(w.__getitem__)
    elif c["kind"] == "moe":
        w, s["x"] = _moe_tensors(c, r)
        s["mix"] = MoE(MoESpec(c["width"], c["experts"], c["top"], c["ff"], 7.0, c["shared"] or None, 7.0), BF, DEV)
        s["mix"].load(w.__getitem__)
    elif c["kind"] == "matrix_memory":
        w, s["x"] = _memory_tensors(c, r)
        s["mix"] = MatrixMemoryMixer(MatrixMemorySpec(c["width"], c["heads"], c["dim"], c["vdim"], 15.0, EPS), BF, DEV)
        s["mix"].load(w.__getitem__)
        s["states"] = [torch.zeros(n, dtype=torch.float32, device=DEV) for n in s["mix"].state_shapes(c["batch"])]
    return s


@torch.no_grad()
def run(state):
    s, c = state, state["c"]
    if c["kind"] == "llama_token":
        logits = s["model"](s["one"], c["seq"], s["at"])
        return {"logits": logits, "kv": [t for kv in s["model"].kv_caches for t in kv]}
    if c["kind"] == "llama_prompt":
        s["model"].reset_cache()
        logits = s["model"](s["idx"], c["seq"], s["pos"])
        return {"logits": logits, "kv": [t for kv in s["model"].kv_caches for t in kv]}
    if c["kind"] in ("int4_mlp", "int8_mlp"):
        return s["mlp"](s["x"])
    if c["kind"] == "latent":
        return s["mix"](s["x"], c["batch"], c["tokens"], s["pos"], s["rope"], s["cache"], s["splits"]), s["cache"]
    if c["kind"] == "softmax":
        return s["mix"](s["x"], c["batch"], c["tokens"], s["pos"], s["caches"], None, s["splits"]), s["caches"]
    if c["kind"] == "moe":
        return s["mix"](s["x"])
    return s["mix"](s["x"], c["batch"], c["tokens"], s["pos"], s["states"]), s["states"]


# ------------------------------------------------------------------------------------------------------------------ least work
def _pairs(c):
    """(query, visible key) pairs of one sequence."""
    w, n = c.get("window") or 1 << 30, 0
    for p in range(c["past"], c["past"] + c["tokens"]):
        n += min(w, p + 1 if not c.get("chunk") else p % c["chunk"] + 1)
    return n


def work(case):
    c = case
    E = c["width"]
    if c["kind"] in ("llama_token", "llama_prompt"):
        H, n = _hidden(E), 1 if c["kind"] == "llama_token" else c["prompt"]
        B, L, V = c.get("batch", 1), c["layers"], c["vocab"]
        w = L * (4 * E * E + 3 * E * H) + V * E
        groups = w / (128 if c["group"] == 128 else E)
        pairs = c["prompt"] + 1 if c["kind"] == "llama_token" else n * (n + 1) // 2
        kv = (c["prompt"] + 1 if c["kind"] == "llama_token" else n) * B * L * 2 * E * 2
        return {"bytes": w / 2 + groups * 4 + kv + 2 * B * n * (E + V), "flops": 2 * B * n * w + 4 * B * L * pairs * E}
    if c["kind"] in ("int4_mlp", "int8_mlp"):
        w = 3 * E * _hidden(E)
        wb = w if c["kind"] == "int8_mlp" else w / 2 + 4 * w / (128 if c["group"] == 128 else E)
        return {"bytes": wb + 4 * c["rows"] * E, "flops": 2 * c["rows"] * w}
    if c["kind"] == "latent":
        M, H, n = c["batch"] * c["tokens"], c["heads"], c["past"] + c["tokens"]
        n_seen = min(n, (c["window"] or n) + c["tokens"] - 1)
        q, row = c["nope"] + c["rot"], c["rank"] + c["rot"]
        w = E * (H * q + H + row) + H * c["rank"] * (c["nope"] + c["v"]) + H * c["v"] * E
        pairs = c["batch"] * _pairs(c)
        absorbed = 2 * M * H * c["rank"] * (c["nope"] + c["v"]) + 2 * pairs * H * (row + c["rank"])
        expanded = 2 * c["batch"] * n_seen * H * c["rank"] * (c["nope"] + c["v"]) + 2 * pairs * H * (q + c["v"])
        return {"bytes": 2 * (w + 2 * M * E + c["batch"] * (n_seen + c["tokens"]) * row),
                "flops": 2 * M * E * (H * q + H + row + H * c["v"]) + min(absorbed, expanded)}
    if c["kind"] == "softmax":
        M, H, G, D = c["batch"] * c["tokens"], c["heads"], c["kv_heads"], c["dim"]
        n = c["past"] + c["tokens"]
        n_seen = min(n, min(c["window"] or n, c["chunk"] or n) + c["tokens"] - 1)
        w = E * (3 * H * D + 2 * G * D)
        return {"bytes": 2 * (w + 2 * M * E + 2 * c["batch"] * (n_seen + c["tokens"]) * G * D),
                "flops": 2 * M * w + 4 * c["batch"] * _pairs(c) * H * D}
    if c["kind"] == "moe":
        rows, branch = c["tokens"] * c["top"], 3 * c["ff"] * E
        used = c["experts"] * (1 - (1 - c["top"] / c["experts"]) ** c["tokens"])      # experts that some token chooses
        return {"bytes": 2 * (used * branch + 3 * c["shared"] * E + 2 * c["tokens"] * E) + 4 * c["experts"] * E,
                "flops": 2 * rows * branch + 6 * c["tokens"] * c["shared"] * E + 2 * c["tokens"] * c["experts"] * E}
    M, H, d, e = c["batch"] * c["tokens"], c["heads"], c["dim"], c["vdim"]
    w = E * (2 * H * d + 3 * H * e + 2 * H)
    return {"bytes": 2 * (w + 2 * M * E) + 4 * c["batch"] * H * d * (e + 1), "flops": 2 * M * w + 4 * M * H * d * (e + 1)}


def tolerance(case):
    """bf16 activations between the steps of a layer; a whole model adds its layers up, and where scores or weights are small beside
    the sums they come from (llm.int8: codes that turn over with the last bit of the activation) somewhat more."""
    kind = case["kind"]
    if kind in ("llama_token", "llama_prompt"):
        return {"rel": 0.03}
    return {"rel": 0.02 if kind == "int8_mlp" else 0.012, "max": 0.3}


# ------------------------------------------------------------------------------------------------------------------ 64 bits
def _silu(x):
    return x * torch.sigmoid(x)


def _w4(codes, scales, zeros):
    n, k = codes.shape
    g = scales.shape[1]
    return ((codes.view(n, g, k // g).double() - zeros.double()[..., None]) * scales.double()[..., None]).view(n, k)


def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * w.double()


def _turn(x, pos, dims, pair):
    """The first ``dims`` of the last dimension turn by position; ``pair``: "next" (2i with 2i + 1) or "half" (i with i + dims/2).
    ``x [B, T, heads, dim]``."""
    f = 10000.0 ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=x.device) / dims)
    ang = pos.double()[:, None] * f
    co, si = ang.cos()[:, None], ang.sin()[:, None]
    y = x.clone()
    a, b = (x[..., 0:dims:2], x[..., 1:dims:2]) if pair == "next" else (x[..., : dims // 2], x[..., dims // 2: dims])
    u, v = a * co - b * si, a * si + b * co
    if pair == "next":
        y[..., 0:dims:2], y[..., 1:dims:2] = u, v
    else:
        y[..., : dims // 2], y[..., dims // 2: dims] = u, v
    return y


def _attend(q, k, v, scale, q_pos, window=0, chunk=0, cap=0.0, sink=None):
    """``q [B, T, H, d]``, ``k [B, n, G, d]``, ``v [B, n, G, e]`` -> ``[B, T, H * e]``; key j is at position j."""
    B, T, H, _ = q.shape
    G = k.shape[2]
    j, i = torch.arange(k.shape[1], device=q.device)[None], q_pos[:, None].long()
    seen = j <= i
    if window:
        seen &= i - j < window
    if chunk:
        seen &= torch.div(j, chunk, rounding_mode="floor") == torch.div(i, chunk, rounding_mode="floor")
    out = torch.empty((B, T, H, v.shape[3]), dtype=torch.float64, device=q.device)
    for b in range(B):
        for h in range(H):
            g = h // (H // G)
            s = q[b, :, h] @ k[b, :, g].t() * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill(~seen, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].double().expand(T, 1)], dim=1)
            out[b, :, h] = torch.softmax(s, dim=1)[:, : k.shape[1]] @ v[b, :, g]
    return out.reshape(B, T, -1)


def _exact_llama(c, r):
    t = _llama_tensors(c, r)
    E, H = c["width"], c["heads"]
    B, n = t["idx"].shape
    pos = torch.arange(n, device=DEV)
    x, kv = t["wte"][t["idx"]].double(), []
    for i in range(c["layers"]):
        p = f"h.{i}."
        qkv = (_rms(x, t[p + "rms_1"]) @ _w4(*t[p + "attn.c_attn"]).t()).view(B, n, 3, H, E // H)
        q, k, v = (_turn(qkv[:, :, 0], pos, E // H, "next"), _turn(qkv[:, :, 1], pos, E // H, "next"), qkv[:, :, 2])
        x = x + _attend(q, k, v, (E // H) ** -0.5, pos) @ _w4(*t[p + "attn.c_proj"]).t()
        h = _rms(x, t[p + "rms_2"])
        h = _silu(h @ _w4(*t[p + "mlp.c_fc1"]).t()) * (h @ _w4(*t[p + "mlp.c_fc2"]).t())
        x = x + h @ _w4(*t[p + "mlp.c_proj"]).t()
        for u in (k, v):
            full = torch.zeros((B, H, c["seq"], E // H), dtype=torch.float64, device=DEV)
            full[:, :, :n] = u.transpose(1, 2)
            kv.append(full)
    if c["kind"] == "llama_token":
        x = x[:, -1:]
    return {"logits": _rms(x, t["ln_f"]) @ _w4(*t["lm_head"]).t(), "kv": kv}


def _exact_int8(x, w):
    """Vector-wise int8 product with the features that reach 6 kept apart in 16 bits."""
    a, wh = x.half().double(), w.half().double()
    scb = wh.abs().amax(1)
    cb = torch.clamp(torch.round(wh * (127.0 / scb)[:, None]), -127, 127)
    big = a.abs() >= 6.0
    cols = big.any(0)
    rest = a.masked_fill(big, 0.0)
    sca = rest.abs().amax(1)
    ca = torch.round(rest * (127.0 / sca.clamp_min(1e-30))[:, None]).masked_fill(cols[None], 0.0)
    return (ca @ cb.t()) * sca[:, None] * scb[None] / 127.0 ** 2 + a[:, cols] @ (cb[:, cols] * scb[:, None] / 127.0).t()


@torch.no_grad()
def exact(case, seed):
    c, r = case, _Rand(seed)
    if c["kind"].startswith("llama"):
        return _exact_llama(c, r)
    if c["kind"] == "int4_mlp":
        w = [r.int4(n, k, c["group"]) for _, n, k in _int4_names(c["width"])]
        x = r.normal(c["rows"], c["width"]).double()
        return (_silu(x @ _w4(*w[0]).t()) * (x @ _w4(*w[1]).t())) @ _w4(*w[2]).t()
    if c["kind"] == "int8_mlp":
        w, x = _int8_tensors(c, r)
        h = _silu(_exact_int8(x, w["c_fc1.weight"])) * _exact_int8(x, w["c_fc2.weight"])
        return _exact_int8(h, w["c_proj.weight"])
    pos = torch.arange(c.get("past", 0), c.get("past", 0) + c["tokens"], device=DEV)
    if c["kind"] == "latent":
        w, x, cache = _latent_tensors(c, r)
        w, x, cache = {n: t.double() for n, t in w.items()}, x.double(), cache.double()
        B, T, H, R = c["batch"], c["tokens"], c["heads"], c["rank"]
        q = (x @ w["q"].t()).view(B, T, H, -1)
        q = torch.cat([q[..., : c["nope"]], _turn(q[..., c["nope"]:], pos, c["rot"], "next")], dim=-1)
        d = (x @ w["dkv"].t()).view(B, T, 1, -1)
        row = torch.cat([_rms(d[..., :R], w["dkv.norm"]), _turn(d[..., R:], pos, c["rot"], "next")], dim=-1)
        cache[:, c["past"]:] = row[:, :, 0]
        n = cache.shape[1]
        k = torch.cat([(cache[..., :R] @ w["uk"].t()).view(B, n, H, -1), cache[:, :, None, R:].expand(B, n, H, c["rot"])], dim=-1)
        v = (cache[..., :R] @ w["uv"].t()).view(B, n, H, -1)
        o = _attend(q, k, v, (c["nope"] + c["rot"]) ** -0.5, pos, window=c["window"]).view(B * T, H, -1)
        return (o * torch.sigmoid(x @ w["g"].t())[..., None]).reshape(B * T, -1) @ w["o"].t(), cache
    if c["kind"] == "softmax":
        w, x, kc, vc = _softmax_tensors(c, r)
        w, x, kc, vc = {n: t.double() for n, t in w.items()}, x.double(), kc.double(), vc.double()
        B, T, H, G, D = c["batch"], c["tokens"], c["heads"], c["kv_heads"], c["dim"]
        q, k = x @ w["q"].t(), x @ w["k"].t()
        if c["norm"]:
            q, k = _rms(q, w["q.norm"]), _rms(k, w["k.norm"])
        kc[:, c["past"]:] = _turn(k.view(B, T, G, D), pos, D // 2, "half").reshape(B, T, -1)
        vc[:, c["past"]:] = (x @ w["v"].t()).view(B, T, -1)
        n = kc.shape[1]
        o = _attend(_turn(q.view(B, T, H, D), pos, D // 2, "half"), kc.view(B, n, G, D), vc.view(B, n, G, D), D ** -0.5, pos,
                    window=c["window"], chunk=c["chunk"], cap=c["cap"], sink=w.get("sink"))
        return (o.view(B * T, -1) * torch.sigmoid(x @ w["g"].t())) @ w["o"].t(), (kc, vc)
    if c["kind"] == "moe":
        w, x = _moe_tensors(c, r)
        w, x = {n: t.double() for n, t in w.items()}, x.double()

        def unit(gate, up):
            g, u = gate.clamp(max=7.0), up.clamp(-7.0, 7.0)
            return g * torch.sigmoid(1.702 * g) * (u + 1.0)

        z, chosen = torch.topk(x @ w["router"].t() + w["router.b"], c["top"], dim=1)
        weight = torch.softmax(z, dim=1)
        y = torch.zeros_like(x)
        for e in range(c["experts"]):
            rows, slot = torch.nonzero(chosen == e, as_tuple=True)
            h = unit(x[rows] @ w[f"e{e}.gate"].t(), x[rows] @ w[f"e{e}.up"].t()) @ w[f"e{e}.down"].t()
            y.index_add_(0, rows, h * weight[rows, slot][:, None])
        if c["shared"]:
            h = unit(x @ w["shared.gate"].t(), x @ w["shared.up"].t()) @ w["shared.down"].t()
            y += torch.sigmoid(x @ w["shared.sg"].t()) * h
        return y
    w, x = _memory_tensors(c, r)
    w, x = {n: t.double() for n, t in w.items()}, x.double()
    B, T, H, d, e = c["batch"], c["tokens"], c["heads"], c["dim"], c["vdim"]
    q, k = (x @ w["q"].t()).view(B, T, H, d) * d ** -0.5, (x @ w["k"].t()).view(B, T, H, d)
    v = torch.cat([(x @ w["v"].t()).view(B, T, H, e), torch.ones((B, T, H, 1), dtype=torch.float64, device=DEV)], dim=-1)
    li = (15.0 * torch.tanh((x @ w["i"].t() + w["i.b"]) / 15.0)).view(B, T, H)
    lf = torch.nn.functional.logsigmoid(15.0 * torch.tanh((x @ w["f"].t() + w["f.b"]) / 15.0)).view(B, T, H)
    run_f = lf.cumsum(1)
    top = run_f + torch.cummax(li - run_f, dim=1).values.clamp_min(0.0)          # the running stabiliser, which starts at 0
    o = torch.empty((B, T, H, e), dtype=torch.float64, device=DEV)
    memory = torch.empty((B, H, d, e + 1), dtype=torch.float64, device=DEV)
    keep = torch.ones((T, T), dtype=torch.bool, device=DEV).tril()
    for b in range(B):
        for h in range(H):
            mass = (run_f[b, :, None, h] - run_f[b, None, :, h] + li[b, None, :, h] - top[b, :, None, h]).masked_fill(~keep, -math.inf).exp()
            a = (q[b, :, h] @ k[b, :, h].t() * mass) @ v[b, :, h]
            o[b, :, h] = a[:, :e] / (torch.maximum(a[:, e:].abs(), torch.exp(-top[b, :, h, None])) + 1e-6)
            memory[b, h] = (k[b, :, h] * mass[-1][:, None]).t() @ v[b, :, h]
    o = (o / torch.sqrt((o * o).mean(-1, keepdim=True) + EPS)).reshape(B * T, -1) * w["norm"] * torch.sigmoid(x @ w["g"].t())
    return o @ w["o"].t(), [memory, top[:, -1]]
