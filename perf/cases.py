"""What a user of the engine has it do, as cases that can be timed and compared: decoding and prompts of GGUF models (F16, Q8_0, Q4_K_M; dense
and with routed experts), a prompt of a layer-list model with recurrent and latent-attention layers, and a mixed serving step of one with
windowed attention and experts.

A case is a dict: `model` and `storage` name the shapes (public sizes of the presets in models/config.py and of `bench.py --layers`), `layers`
how many of them (models in blocks are cut to a part of their layers, which repeat the same work: 8-bit activations of small batches add up
over the depth until two correct paths differ by as much as a mistake would show), `do` the call:
  decode   `tokens` steps of one token for each of `batch` sequences with up to `cached` tokens in the cache (lengths spread below it)
  prefill  one sequence with `cached` tokens in the cache takes a prompt of `tokens` tokens
  step     one forward for `batch` generating sequences beside a new prompt of `tokens` tokens
Weights, cached keys and values and token ids are random, made from the seed alone.  Sequences are cut back to `cached` behind each pass, so
that a pass can be repeated.
"""
import math
import zlib

import torch

PAGE = 64
F64 = torch.float64

# vocab, width, layers, query heads, key / value heads, head size, ff, rotation base, experts, experts per token
GGUF = {
    "tinyllama-1.1b": dict(vocab=32000, width=2048, layers=22, heads=32, kv=4, dim=64, ff=5632, base=10000.0, experts=0, top=0),
    "llama-3-8b": dict(vocab=128256, width=4096, layers=32, heads=32, kv=8, dim=128, ff=14336, base=500000.0, experts=0, top=0),
    "mixtral-8x7b": dict(vocab=32000, width=4096, layers=32, heads=32, kv=8, dim=128, ff=14336, base=1000000.0, experts=8, top=2),
}
# three recurrent layers to one of latent attention, a gated feed-forward in each
TALIZEN = dict(vocab=32000, width=2048, heads=16, dim=128, rank=512, ff=5632, groups=4)
# windowed grouped-query attention and routed experts in every layer
VOZINEX = dict(vocab=32000, width=2048, heads=32, kv=4, dim=128, ff=768, experts=64, top=8, window=1984, keep=64, base=1e6)
EPS = 1e-5
BITS = {"F16": 2.0, "Q8_0": 34 / 32, "Q4_K": 144 / 256, "Q6_K": 210 / 256, "bf16": 2.0}       # bytes per weight


def listed():
    def case(name, model, storage, layers, do, batch, cached, tokens):
        return dict(name=name, model=model, storage=storage, layers=layers, do=do, batch=batch, cached=cached, tokens=tokens)
    return [
        # a small model answering one user: launches and latency count
        case("tinyllama q8_0 decode", "tinyllama-1.1b", "Q8_0", 8, "decode", 1, 100, 4),
        # single-stream decoding of the benchmark's model
        case("llama-8b f16 decode", "llama-3-8b", "F16", 32, "decode", 1, 512, 4),
        # the same far into a long document
        case("llama-8b f16 decode 32k", "llama-3-8b", "F16", 32, "decode", 1, 32000, 4),
        # a server with 32 busy slots, conversations of different lengths
        case("llama-8b f16 decode batch 32", "llama-3-8b", "F16", 32, "decode", 32, 2000, 4),
        # the common download format, one user
        case("llama-8b q4_k_m decode", "llama-3-8b", "Q4_K_M", 8, "decode", 1, 700, 4),
        # a handful of users on 8-bit weights
        case("llama-8b q8_0 decode batch 7", "llama-3-8b", "Q8_0", 8, "decode", 7, 900, 4),
        # the benchmark's prompt
        case("llama-8b f16 prompt 512", "llama-3-8b", "F16", 32, "prefill", 1, 0, 512),
        # a long prompt on top of a conversation, in several chunks of the engine's batch
        case("llama-8b f16 prompt 3001 at 4096", "llama-3-8b", "F16", 32, "prefill", 1, 4096, 3001),
        # a prompt on 4-bit weights
        case("llama-8b q4_k_m prompt 1021", "llama-3-8b", "Q4_K_M", 8, "prefill", 1, 0, 1021),
        # concurrent requests on a mixture of experts
        case("mixtral q4_k_m decode batch 16", "mixtral-8x7b", "Q4_K_M", 4, "decode", 16, 1000, 4),
        # a prompt of a layer-list model: chunked recurrence and latent attention
        case("talizen bf16 prompt 1999", "talizen", "bf16", 8, "prefill", 1, 0, 1999),
        # a serving step of a layer-list model: a new prompt beside generating requests
        case("vozinex bf16 step 15 + 300", "vozinex", "bf16", 4, "step", 15, 2500, 300),
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))
    kind = rng.choice(["decode", "decode", "decode", "decode", "prefill", "prefill", "prefill", "talizen", "vozinex"])
    if kind == "talizen":
        return dict(model="talizen", storage="bf16", layers=8, do="prefill", batch=1, cached=0, tokens=log(5, 6000))
    if kind == "vozinex":
        return dict(model="vozinex", storage="bf16", layers=4, do="step", batch=log(1, 31), cached=log(16, 8000), tokens=log(5, 1900))
    model, storage, layers = rng.choice([("tinyllama-1.1b", "Q8_0", 8), ("tinyllama-1.1b", "F16", 22), ("llama-3-8b", "F16", 32), ("llama-3-8b", "F16", 32),
                                         ("llama-3-8b", "Q8_0", 8), ("llama-3-8b", "Q4_K_M", 8), ("mixtral-8x7b", "Q4_K_M", 4)])
    if kind == "decode":
        batch = log(1, 32)
        return dict(model=model, storage=storage, layers=layers, do="decode", batch=batch, cached=log(16, min(32000, 64000 // batch)), tokens=4)
    return dict(model=model, storage=storage, layers=layers, do="prefill", batch=1, cached=rng.choice([0, log(16, 4000)]), tokens=log(5, 3000))


# ---- inputs: every tensor from (seed, name), on the GPU -------------------------------------------------------------------------------
def generator(seed, name):
    return torch.Generator("cuda").manual_seed((zlib.crc32(name.encode()) << 20) + seed)


def normal(seed, name, shape, std, dtype):
    t = torch.empty(shape, dtype=dtype, device="cuda")
    t.view(-1).normal_(0.0, std, generator=generator(seed, name))
    return t


def matrix(seed, name, n, k, kind, quiet=0):
    """A weight [n, k] of variance 1 / k: fp16 / bf16 values, or the bytes [n, row] of GGUF blocks; the first `quiet` rows are zero."""
    if kind in ("F16", "bf16"):
        t = normal(seed, name, (n, k), k ** -0.5, torch.float16 if kind == "F16" else torch.bfloat16)
        t[:quiet] = 0
        return t
    per, size = {"Q8_0": (32, 34), "Q4_K": (256, 144), "Q6_K": (256, 210)}[kind]
    words = n * (k // per) * size
    raw = torch.randint(-2 ** 63, 2 ** 63 - 1, ((words + 7) // 8,), dtype=torch.int64, device="cuda", generator=generator(seed, name)).view(torch.uint8)[:words]
    raw = raw.view(n, k // per, size)

    def half(col, value):
        d = (value * (0.75 + 0.5 * torch.rand(n, k // per, device="cuda", generator=generator(seed, name + ".d")))).to(torch.float16)
        d[:quiet] = 0
        raw[:, :, col:col + 2] = d.view(torch.uint8).view(n, k // per, 2)
    if kind == "Q8_0":            # d | 32 x int8
        half(0, k ** -0.5 / 73.9)
    elif kind == "Q4_K":          # d | dmin | 12 bytes of 6-bit scales and mins | 128 bytes of nibbles: mins that centre the values, as quantised weights have
        half(0, k ** -0.5 / 168)
        half(2, 7.5 * k ** -0.5 / 168)
        raw[:, :, 8:12] = raw[:, :, 4:8]
        low = raw[:, :, 12:16] & 15
        raw[:, :, 12:16] = low | (low << 4)
    else:                         # 128 low nibbles | 64 high bits | 16 x int8 scales | d
        raw[:, :, 192:208] &= 63
        half(208, k ** -0.5 / 675)
    return raw.view(n, -1)


def values(t, kind):
    """The weights that `matrix` stands for, in 64 bits."""
    if kind in ("F16", "bf16"):
        return t.to(F64)
    n = t.shape[0]
    if kind == "Q8_0":
        b = t.view(n, -1, 34)
        return (b[..., :2].contiguous().view(torch.float16).to(F64) * b[..., 2:].contiguous().view(torch.int8).to(F64)).view(n, -1)
    if kind == "Q4_K":
        b = t.view(n, -1, 144)
        d, m = (b[..., i:i + 2].contiguous().view(torch.float16).to(F64)[..., None] for i in (0, 2))
        s = b[..., 4:16].to(torch.int64)
        scale = torch.cat([s[..., :4] & 63, (s[..., 8:] & 15) | (s[..., :4] >> 6 << 4)], -1)
        least = torch.cat([s[..., 4:8] & 63, (s[..., 8:] >> 4) | (s[..., 4:8] >> 6 << 4)], -1)
        q = b[..., 16:].reshape(n, -1, 4, 32)
        q = torch.stack([q & 15, q >> 4], 3).view(n, -1, 8, 32).to(F64)
        return (q * (d * scale[..., None]) - m * least[..., None]).view(n, -1)
    b = t.view(n, -1, 210)
    low, high = b[..., :128].reshape(n, -1, 2, 64), b[..., 128:192].reshape(n, -1, 2, 1, 32)
    low = torch.stack([low & 15, low >> 4], 3).view(n, -1, 2, 4, 32)
    q = low | (torch.cat([high >> (2 * i) & 3 for i in range(4)], 3) << 4)
    scale = b[..., 192:208].contiguous().view(torch.int8).to(F64).view(n, -1, 16, 1)
    return ((q.to(F64) - 32).view(n, -1, 16, 16) * scale * b[..., 208:].contiguous().view(torch.float16).to(F64)[..., None]).view(n, -1)


def more_bits(i, n):
    """Layers whose value and down matrices a Q4_K_M file keeps in Q6_K."""
    return i < n // 8 or i >= 7 * n // 8 or (i - n // 8) % 3 == 2


def kinds(case, m, il):
    """Storage of a layer's matrices: q|k|v, output, gate / up, down.  (A file of mixed types: q, k and v are decoded to fp16 together at load.)"""
    if case["storage"] != "Q4_K_M":
        return (case["storage"],) * 4
    more = more_bits(il, case["layers"])
    return "F16" if more else "Q4_K", "Q4_K", "Q4_K", "Q6_K" if more else "Q4_K"


def lengths(case):
    """Cached tokens of every sequence: spread up to `cached`."""
    return [max(1, case["cached"] * (i + 1) // case["batch"]) if case["cached"] else 0 for i in range(case["batch"])]


def vector(seed, name, n):
    return 1 + 0.1 * normal(seed, name, (n,), 1.0, torch.float32)


def table(seed, m, kind):
    """Token embeddings.  With experts the first columns hold every token's preferences, which no layer writes to: the best `top` stand clear of
    the rest, as a trained router's choices do."""
    t = normal(seed, "embed", (m["vocab"], m["width"]), 1.0, torch.float16 if kind == "F16" else torch.bfloat16)
    n = m.get("experts", 0)
    if n:
        rank = torch.rand(m["vocab"], n, device="cuda", generator=generator(seed, "prefer")).argsort(-1).argsort(-1).float()
        t[:, :n] = torch.where(rank >= n - m["top"], 4 + 0.25 * (rank - n), -1 + rank / n).to(t.dtype)
    return t


def router(seed, il, m):
    """[experts, width]: layer il reads the preferences in an order of its own."""
    t = torch.zeros(m["experts"], m["width"], device="cuda")
    t[torch.arange(m["experts"], device="cuda"), torch.randperm(m["experts"], device="cuda", generator=generator(seed, f"l{il}.order"))] = 1.5
    return t


def kept(seed, il, name, n, heads, dim, dtype):
    """Keys or values of the cached tokens of all sequences, one after the other."""
    return normal(seed, f"l{il}.{name}.cache", (n, heads, dim), 1.5 if name == "k" else 1.0, dtype)


def ids(case, seed, vocab):
    n = case["tokens"] * (1 if case["do"] == "prefill" else case["batch"]) + (case["tokens"] if case["do"] == "step" else 0)
    return torch.randint(3, vocab, (n,), generator=torch.Generator().manual_seed(seed), dtype=torch.int32)


# ---- models in device memory ----------------------------------------------------------------------------------------------------------
_staging = []


def weight(t, kind, k):
    from distributed_llm_pipeline_b200.gguf.constants import GGMLType
    from distributed_llm_pipeline_b200.ops.weights import DeviceWeight
    if kind == "F16":
        return DeviceWeight(GGMLType.F16, t.shape[0], k, [t])
    if not _staging or _staging[0].numel() < t.numel():        # a file's bytes, as the loader reads them
        _staging[:] = [torch.empty(t.numel(), dtype=torch.uint8, pin_memory=True)]
    raw = _staging[0][:t.numel()].view(t.shape)
    raw.copy_(t)
    return DeviceWeight.from_raw(raw.numpy(), GGMLType[kind], (t.shape[0], k), "cuda:0")


def gguf_matrix(seed, m, case, il, name):
    """(values or bytes, storage, columns) of one matrix of layer il (None: of the model)."""
    hd, kd, w, f = m["heads"] * m["dim"], m["kv"] * m["dim"], m["width"], m["ff"]
    if name == "head":
        kind = {"Q4_K_M": "Q6_K"}.get(case["storage"], case["storage"])
        return matrix(seed, "head", m["vocab"], w, kind), kind, w
    qkv, o, up, down = kinds(case, m, il)
    n, k, kind, quiet = {"qkv": (hd + 2 * kd, w, qkv, 0), "o": (w, hd, o, m["experts"]), "gate": (f * max(1, m["experts"]), w, up, 0),
                         "up": (f * max(1, m["experts"]), w, up, 0), "down": (w, f, down, m["experts"])}[name.split(".")[0]]
    return matrix(seed, f"l{il}.{name}", n, k, kind, quiet), kind, k


def gguf_weights(case, seed):
    from distributed_llm_pipeline_b200.gguf.constants import GGMLType
    from distributed_llm_pipeline_b200.models.config import preset
    from distributed_llm_pipeline_b200.models.weights import LayerWeights, ModelWeights
    from distributed_llm_pipeline_b200.ops.weights import DeviceWeight, stack_rows
    m = GGUF[case["model"]]
    cfg = preset(case["model"], n_layer=case["layers"])
    layers = {}
    for il in range(case["layers"]):
        def mat(name):
            return weight(*gguf_matrix(seed, m, case, il, name))
        lw = LayerWeights(attn_norm=vector(seed, f"l{il}.norm1", m["width"]), wqkv=mat("qkv"), wo=mat("o"), ffn_norm=vector(seed, f"l{il}.norm2", m["width"]))
        if m["experts"]:
            n = m["experts"]
            lw.router = router(seed, il, m)
            lw.e_gate_s, lw.e_up_s, lw.e_down_s = mat("gate"), mat("up"), stack_rows([mat(f"down.{e}") for e in range(n)])
            for stack, one in ((lw.e_gate_s, lw.e_gate), (lw.e_up_s, lw.e_up), (lw.e_down_s, lw.e_down)):
                rows = stack.N // n
                one += [DeviceWeight(stack.wtype, rows, stack.K, [p.view(stack.N, -1)[e * rows:(e + 1) * rows] for p in stack.planes]) for e in range(n)]
            r16 = torch.zeros(128, m["width"], dtype=torch.float16, device="cuda")
            r16[:n] = lw.router
            lw.router_w = DeviceWeight(GGMLType.F16, n, m["width"], [r16[:n].contiguous()])
            lw.router_wp = DeviceWeight(GGMLType.F16, 128, m["width"], [r16])
        else:
            lw.w_gate, lw.w_up, lw.w_down = mat("gate"), mat("up"), mat("down")
        layers[il] = lw
    embed = DeviceWeight(GGMLType.F16, m["vocab"], m["width"], [table(seed, m, "F16")])
    return ModelWeights(cfg, layers, range(case["layers"]), 0, 1, embed, vector(seed, "norm", m["width"]), weight(*gguf_matrix(seed, m, case, None, "head")),
                        (0, m["vocab"]), None, n_head_local=m["heads"], n_head_kv_local=m["kv"], n_ff_local=m["ff"])


def talizen_tensors(seed, il):
    t = TALIZEN
    hd, w, r, f = t["heads"] * t["dim"], t["width"], t["rank"], t["ff"]
    shapes = {"gate": (f, w), "up": (f, w), "down": (w, f), "o": (w, hd), "q": (hd, w)}
    shapes |= {"dkv": (r, w), "g": (t["heads"], w), "uk": (hd, r), "uv": (hd, r)} if il % 4 == 3 else {"f": (hd, w), "v": (hd, w)}
    out = {n: matrix(seed, f"l{il}.{n}", *s, "bf16") for n, s in shapes.items()}
    if il % 4 == 3:
        out["dkv.norm"] = vector(seed, f"l{il}.dkv.norm", r)
    else:
        out |= {"f.b": 3 + normal(seed, f"l{il}.f.b", (hd,), 0.5, torch.float32), "norm": vector(seed, f"l{il}.norm", t["dim"]),
                "lower": 0.9 * torch.rand(hd, device="cuda", generator=generator(seed, f"l{il}.lower"))}
    return out


def talizen_layer(il):
    t = TALIZEN
    if il % 4 == 3:
        return {"type": "latent_attention", "mixer": {"heads": t["heads"], "dim": t["dim"], "vdim": t["dim"], "kv_rank": t["rank"], "scale": t["dim"] ** -0.5},
                "mlp": {"kind": "dense", "ff": t["ff"]}}
    return {"type": "hgrn2", "mixer": {"heads": t["heads"], "dim": t["dim"], "vdim": t["dim"]}, "mlp": {"kind": "dense", "ff": t["ff"]}}


def vozinex_tensors(seed, il):
    v = VOZINEX
    hd, kd, w, n, f = v["heads"] * v["dim"], v["kv"] * v["dim"], v["width"], v["experts"], v["ff"]
    down = matrix(seed, f"l{il}.down", n * w, f, "bf16").view(n, w, f)
    down[:, :n] = 0
    return {"q": matrix(seed, f"l{il}.q", hd, w, "bf16"), "k": matrix(seed, f"l{il}.k", kd, w, "bf16"), "v": matrix(seed, f"l{il}.v", kd, w, "bf16"),
            "o": matrix(seed, f"l{il}.o", w, hd, "bf16", n), "q.norm": vector(seed, f"l{il}.q.norm", hd), "k.norm": vector(seed, f"l{il}.k.norm", kd),
            "up": matrix(seed, f"l{il}.up", n * f, w, "bf16").view(n, f, w), "down": down, "router": router(seed, il, v).to(torch.bfloat16),
            "router.b": torch.zeros(n, device="cuda")}


def layered_weights(case, seed):
    from distributed_llm_pipeline_b200.gguf.constants import GGMLType
    from distributed_llm_pipeline_b200.models.layered import LayeredLayer, LayeredWeights, Norm
    from distributed_llm_pipeline_b200.models.mixers import MIXERS, MLPS
    from distributed_llm_pipeline_b200.models.modeldir import talizen_config, vozinex_config
    from distributed_llm_pipeline_b200.ops.weights import DeviceWeight
    if case["model"] == "talizen":
        m = TALIZEN
        cfg = talizen_config({"width": m["width"], "vocab": m["vocab"], "norm": {"groups": m["groups"], "eps": EPS}, "layers": [talizen_layer(i) for i in range(case["layers"])]})
    else:
        m = VOZINEX
        spec = {"type": "attention", "mixer": {"heads": m["heads"], "kv_heads": m["kv"], "dim": m["dim"], "vdim": m["dim"], "scale": m["dim"] ** -0.5,
                                               "rot": {"dims": m["dim"], "base": m["base"]}, "mask": {"size": m["window"], "keep_first": m["keep"]}},
                "mlp": {"kind": "moe", "expert": {"ff": m["ff"]}, "router": {"experts": m["experts"], "top": m["top"]}}}
        cfg = vozinex_config({"width": m["width"], "vocab": m["vocab"], "norm": {"eps": EPS}, "layers": [spec] * case["layers"]})

    def norm(name):
        w = vector(seed, name, m["width"])
        return Norm(w) if case["model"] == "talizen" else Norm(w, 0.1 * normal(seed, name + ".b", (m["width"],), 1.0, torch.float32))
    layers = {}
    for i, s in enumerate(cfg.layers):
        t = talizen_tensors(seed, i) if case["model"] == "talizen" else vozinex_tensors(seed, i)

        def get(name):
            if name.startswith("e") and "." in name and name[1].isdigit():
                e, part = name[1:].split(".")
                return t[part][int(e)]
            return t[name]
        layers[i] = LayeredLayer(MIXERS[s.type](s.mixer, get, "cuda:0", torch.bfloat16, EPS), norm(f"l{i}.norm1"),
                                 MLPS[s.mlp["kind"]](s.mlp, get, "cuda:0", torch.bfloat16, m["width"]), norm(f"l{i}.norm2"))
    embed, head = table(seed, m, "bf16"), matrix(seed, "head", m["vocab"], m["width"], "bf16")
    last = norm("norm")
    return LayeredWeights(cfg, layers, range(case["layers"]), 0, 1, DeviceWeight(GGMLType.BF16, m["vocab"], m["width"], [embed]), last.w,
                          DeviceWeight(GGMLType.BF16, m["vocab"], m["width"], [head]), (0, m["vocab"]), None, out_norm_b=last.b)


def prepare(case, seed):
    """The engine with its weights, sequences with their cached tokens, and the next token ids."""
    from distributed_llm_pipeline_b200.models.layered import LayeredEngine
    from distributed_llm_pipeline_b200.models.llama import LlamaEngine
    gguf = case["model"] in GGUF
    m = GGUF[case["model"]] if gguf else TALIZEN if case["model"] == "talizen" else VOZINEX
    n_ctx = (max(case["cached"], 0) + case["tokens"] + 2 * PAGE) // PAGE * PAGE
    seqs = case["batch"] + (case["do"] == "step")
    with torch.no_grad():
        w = gguf_weights(case, seed) if gguf else layered_weights(case, seed)
        eng = (LlamaEngine if gguf else LayeredEngine)(w, n_ctx=n_ctx, max_seqs=seqs, page_size=PAGE)
        sids, lens = [eng.alloc_seq() for _ in range(case["batch"])], lengths(case)
        where = []
        for sid, n in zip(sids, lens):
            seq = eng.seqs[sid]
            eng.kv.ensure(seq, n)
            seq.length = n
            eng.seq_len_dev[sid] = n
            where += [p * PAGE + i for p in seq.pages for i in range(PAGE)][:n]
        if where:
            slot = torch.tensor(where, device="cuda")
            for il in range(case["layers"]):
                for name in ("k", "v"):
                    plane = eng.kv.planes[name][il]
                    plane[slot // PAGE, :, slot % PAGE] = kept(seed, il, name, len(where), m["kv"], m["dim"], plane.dtype)
    tok = ids(case, seed, m["vocab"])
    state = dict(case=case, eng=eng, sids=sids, lens=lens, last=case["layers"] - 1)
    if case["do"] == "decode":
        state["tokens"] = list(tok.view(case["tokens"], case["batch"]).cuda())
    elif case["do"] == "prefill":
        state["tokens"] = tok
    else:
        state["tokens"] = tok[:case["batch"]].tolist(), tok[-case["tokens"]:].tolist()
    return state


def run(state):
    """One pass; returns the logits and what the last layer left in the cache (or in its recurrent state)."""
    eng, sids, lens, tok, case = (state[k] for k in ("eng", "sids", "lens", "tokens", "case"))
    out = {}
    if case["do"] == "decode":
        out["logits"] = [eng.decode(sids, t, sample=False).clone() for t in tok]
    elif case["model"] == "talizen":        # (a recurrent state cannot be cut back: a new sequence)
        eng.free_seq(sids[0])
        sids[0] = eng.alloc_seq()
        out["logits"] = eng.prefill(sids[0], tok)
    elif case["do"] == "prefill":
        out["logits"] = eng.prefill(sids[0], tok)
    else:
        new = eng.alloc_seq()
        out["logits"] = eng.step([(s, [t]) for s, t in zip(sids, tok[0])] + [(new, tok[1])])
        eng.free_seq(new)
    if case["model"] == "talizen":
        out["state"] = [t for _, _, t in eng.rstate.each()][-1]
        out["latents"] = eng.kv.planes["c"][max(eng.kv.planes["c"])] if "c" in eng.kv.planes else None
    else:
        for sid, n in zip(sids, lens):
            eng.truncate_seq(sid, n)
        out["k"], out["v"] = (eng.kv.planes[p][state["last"]] for p in ("k", "v"))
    return out


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------------------
def work(case):
    B, T = case["batch"], case["tokens"]
    steps = T if case["do"] == "decode" else 1
    rows = B if case["do"] == "decode" else T + (B if case["do"] == "step" else 0)        # of one forward
    n_logits = {"decode": B, "prefill": 1, "step": B + 1}[case["do"]]
    lens = lengths(case)
    if case["model"] == "talizen":
        t = TALIZEN
        hd, w, f, r = t["heads"] * t["dim"], t["width"], t["ff"], t["rank"]
        weights = flops = moved = 0
        for il in range(case["layers"]):
            n = 3 * w * f + (2 * w * hd + w * (r + t["heads"]) + 2 * hd * r if il % 4 == 3 else 4 * w * hd)
            weights, flops = weights + 2 * n, flops + 2 * rows * n
            flops += 2 * T * T * hd if il % 4 == 3 else 6 * T * hd * t["dim"]
            moved += 2 * T * r if il % 4 == 3 else 4 * hd * t["dim"]
        head = t["vocab"] * w
        return {"bytes": weights + moved + 2 * head + 2 * T * w + 4 * t["vocab"], "flops": flops + 2 * head}
    if case["model"] == "vozinex":
        v = VOZINEX
        hd, kd, w, f = v["heads"] * v["dim"], v["kv"] * v["dim"], v["width"], v["ff"]
        seen = [min(n + 1, v["window"] + v["keep"]) for n in lens]
        used = v["experts"] * (1 - (1 - v["top"] / v["experts"]) ** rows)
        per = 2 * w * hd + 2 * w * kd + v["experts"] * w
        head = v["vocab"] * w
        prompt = sum(min(i + 1, v["window"] + v["keep"]) for i in range(T))
        flops = case["layers"] * (2 * rows * (per + v["top"] * 2 * w * f) + 4 * hd * (sum(seen) + prompt))
        moved = case["layers"] * (2 * (per + used * 2 * w * f) + 4 * kd * (sum(seen) + rows))
        return {"bytes": moved + 2 * head + 4 * n_logits * v["vocab"], "flops": flops + 2 * n_logits * head}
    m = GGUF[case["model"]]
    hd, kd, w, f = m["heads"] * m["dim"], m["kv"] * m["dim"], m["width"], m["ff"]
    bytes_, flops = 0.0, 0.0
    used = m["experts"] * (1 - (1 - m["top"] / m["experts"]) ** rows) if m["experts"] else 1
    for il in range(case["layers"]):
        qkv, o, up, down = (BITS[k] for k in kinds(case, m, il))
        bytes_ += (hd + 2 * kd) * w * qkv + w * hd * o + used * w * f * (2 * up + down)
        flops += 2 * rows * ((hd + 2 * kd) * w + w * hd + (m["top"] or 1) * 3 * w * f)
    kind = {"Q4_K_M": "Q6_K"}.get(case["storage"], case["storage"])
    bytes_ += m["vocab"] * w * BITS[kind] + 4 * n_logits * m["vocab"]
    flops += 2 * n_logits * m["vocab"] * w
    bytes_, flops = bytes_ * steps, flops * steps
    per_token = 4 * kd * case["layers"]              # keys and values in 16 bits
    if case["do"] == "decode":
        keys = sum(n + s + 1 for n in lens for s in range(steps))
        bytes_ += per_token * keys
    else:
        keys = sum(lens[0] + i + 1 for i in range(T))
        bytes_ += per_token * (lens[0] + T)
    return {"bytes": bytes_, "flops": flops + 4 * hd * case["layers"] * keys}


def tolerance(case):
    """About four times what the path is from 64 bits: 16-bit activations, and for block formats in small batches 8-bit ones."""
    return {"rel": 0.02} if case["storage"] in ("F16",) else {"rel": 0.03}


# ---- the same in 64 bits, plainly -----------------------------------------------------------------------------------------------------
def rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def silu(x):
    return x * torch.sigmoid(x)


def attend(q, k, v, n, seen):
    """q [T, H, D] at positions n .. n+T-1 over k, v [n + T, G, D]; seen(i, j): whether the query at i sees the key at j."""
    T, H, D = q.shape
    G = k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=F64, device="cuda")
    i, j = torch.arange(n, n + T, device="cuda")[:, None], torch.arange(k.shape[0], device="cuda")[None]
    mask = ~seen(i, j)
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T).masked_fill_(mask, -math.inf)
        out[:, h] = torch.softmax(s, -1) @ v[:, h * G // H]
    return out.reshape(T, -1)


def turn(x, pos, base, half):
    """Rotation of x [T, H, D]: pairs (2i, 2i + 1), or (i, i + D / 2)."""
    d = x.shape[-1]
    a = pos.to(F64)[:, None, None] * base ** (-2 * torch.arange(d // 2, dtype=F64, device="cuda") / d)
    c, s = torch.cos(a), torch.sin(a)
    if half:
        u, v = x[..., :d // 2], x[..., d // 2:]
        return torch.cat([u * c - v * s, v * c + u * s], -1)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)


def choose(z, top):
    """[T, experts]: the softmax over the best `top`, zero elsewhere."""
    best = z.topk(top, -1)
    return torch.zeros_like(z).scatter_(-1, best.indices, torch.softmax(best.values, -1))


def exact(case, seed):
    with torch.no_grad():
        return {"talizen": exact_talizen, "vozinex": exact_vozinex}.get(case["model"], exact_gguf)(case, seed)


def exact_gguf(case, seed):
    m = GGUF[case["model"]]
    H, G, D, n = m["heads"], m["kv"], m["dim"], m["experts"]
    lens, tok = lengths(case), ids(case, seed, m["vocab"]).cuda().long()
    per = case["tokens"]
    if case["do"] == "decode":          # rows by sequence, then by step
        tok = tok.view(per, case["batch"]).T.reshape(-1)
    pos = torch.cat([torch.arange(c, c + per, device="cuda") for c in lens])

    def mat(il, name):
        t, kind, _ = gguf_matrix(seed, m, case, il, name)
        return values(t, kind)
    h = table(seed, m, "F16")[tok].to(F64)
    for il in range(case["layers"]):
        x = rms(h) * vector(seed, f"l{il}.norm1", m["width"]).to(F64)
        q, k, v = (x @ mat(il, "qkv").T).split([H * D, G * D, G * D], -1)
        q, k = turn(q.view(-1, H, D), pos, m["base"], False) * D ** -0.5, turn(k.view(-1, G, D), pos, m["base"], False)
        v = v.reshape(-1, G, D)
        ck, cv = (kept(seed, il, c, sum(lens), G, D, torch.float16) for c in ("k", "v"))
        att, at = [], 0
        for i, c in enumerate(lens):
            rows = slice(i * per, (i + 1) * per)
            att.append(attend(q[rows], torch.cat([ck[at:at + c].to(F64), k[rows]]), torch.cat([cv[at:at + c].to(F64), v[rows]]), c, lambda a, b: b <= a))
            at += c
        h = h + torch.cat(att) @ mat(il, "o").T
        x = rms(h) * vector(seed, f"l{il}.norm2", m["width"]).to(F64)
        if not n:
            h = h + (silu(x @ mat(il, "gate").T) * (x @ mat(il, "up").T)) @ mat(il, "down").T
            continue
        p = choose(x @ router(seed, il, m).to(F64).T, m["top"])
        gate, up = (gguf_matrix(seed, m, case, il, c) for c in ("gate", "up"))
        for e in range(n):
            g, u = (values(t[e * m["ff"]:(e + 1) * m["ff"]].contiguous(), kind) for t, kind, _ in (gate, up))
            h = h + p[:, e, None] * ((silu(x @ g.T) * (x @ u.T)) @ mat(il, f"down.{e}").T)
    if case["do"] == "prefill":
        h = h[-1:]
    logits = (rms(h) * vector(seed, "norm", m["width"]).to(F64)) @ mat(None, "head").T
    return {"logits": list(logits.view(case["batch"], per, -1).transpose(0, 1)) if case["do"] == "decode" else logits[0], "k": None, "v": None}


def exact_talizen(case, seed):
    t = TALIZEN
    H, D, T, R = t["heads"], t["dim"], case["tokens"], t["rank"]

    def behind(x, name):
        return rms(x.view(T, t["groups"], -1)).view(T, -1) * vector(seed, name, t["width"]).to(F64)
    h = table(seed, t, "bf16")[ids(case, seed, t["vocab"]).cuda().long()].to(F64)
    state = latents = None
    for il in range(case["layers"]):
        w = {k: v.to(F64) for k, v in talizen_tensors(seed, il).items()}
        if il % 4 == 3:
            c = rms(h @ w["dkv"].T) * w["dkv.norm"]
            q, k, v = (x.view(T, H, D) for x in (h @ w["q"].T, c @ w["uk"].T, c @ w["uv"].T))
            o = attend(q * D ** -0.5, k, v, 0, lambda a, b: b <= a).view(T, H, D) * torch.sigmoid(h @ w["g"].T)[..., None]
        else:
            q = silu(h @ w["q"].T).view(T, H, D)
            f = (w["lower"] + (1 - w["lower"]) * torch.sigmoid(h @ w["f"].T + w["f.b"])).view(T, H, D, 1)
            v, S, o = (h @ w["v"].T).view(T, H, 1, D), torch.zeros(H, D, D, dtype=F64, device="cuda"), torch.empty(T, H, D, dtype=F64, device="cuda")
            for i in range(T):
                S = f[i] * S + (1 - f[i]) * v[i]
                o[i] = torch.einsum("hdv,hd->hv", S, q[i])
            o, state = rms(o) * w["norm"], S
        h = h + behind(o.reshape(T, -1) @ w["o"].T, f"l{il}.norm1")
        g = h @ w["gate"].T
        h = h + behind((torch.nn.functional.gelu(g, approximate="tanh") * (h @ w["up"].T)) @ w["down"].T, f"l{il}.norm2")
    x = rms(h[-1].view(t["groups"], -1)).view(-1) * vector(seed, "norm", t["width"]).to(F64)
    return {"logits": matrix(seed, "head", t["vocab"], t["width"], "bf16").to(F64) @ x, "state": state[None], "latents": latents}


def exact_vozinex(case, seed):
    v = VOZINEX
    H, G, D, B, T, n = v["heads"], v["kv"], v["dim"], case["batch"], case["tokens"], v["experts"]
    lens = lengths(case)

    def norm(x, name):
        d = x - x.mean(-1, keepdim=True)
        return d / torch.sqrt((d * d).mean(-1, keepdim=True) + EPS) * vector(seed, name, v["width"]).to(F64) + 0.1 * normal(seed, name + ".b", (v["width"],), 1.0, torch.float32).to(F64)
    tok = ids(case, seed, v["vocab"]).cuda().long()
    h = table(seed, v, "bf16")[torch.cat([tok[:B], tok[-T:]])].to(F64)
    parts = [(i, i + 1, c) for i, c in enumerate(lens)] + [(B, B + T, 0)]
    pos = torch.cat([torch.tensor(lens, device="cuda"), torch.arange(T, device="cuda")])

    def seen(i, j):
        return (j <= i) & ((i - j < v["window"]) | (j < v["keep"]))
    for il in range(case["layers"]):
        w = {k: t.to(F64) for k, t in vozinex_tensors(seed, il).items()}
        x = norm(h, f"l{il}.norm1")
        q, k = rms(x @ w["q"].T) * w["q.norm"], rms(x @ w["k"].T) * w["k.norm"]
        q, k, val = turn(q.view(-1, H, D), pos, v["base"], True) * D ** -0.5, turn(k.view(-1, G, D), pos, v["base"], True), (x @ w["v"].T).view(-1, G, D)
        ck, cv = (kept(seed, il, c, sum(lens), G, D, torch.bfloat16) for c in ("k", "v"))
        att, at = [], 0
        for lo, hi, c in parts:
            att.append(attend(q[lo:hi], torch.cat([ck[at:at + c].to(F64), k[lo:hi]]), torch.cat([cv[at:at + c].to(F64), val[lo:hi]]), c, seen))
            at += c
        h = h + torch.cat(att) @ w["o"].T
        x = norm(h, f"l{il}.norm2")
        p = choose(x @ w["router"].T, v["top"])
        for e in range(n):
            h = h + p[:, e, None] * (torch.clamp(x @ w["up"][e].T, min=0) ** 2 @ w["down"][e].T)
    rows = norm(h[list(range(B)) + [B + T - 1]], "norm")
    return {"logits": rows @ matrix(seed, "head", v["vocab"], v["width"], "bf16").to(F64).T, "k": None, "v": None}
