"""The work that users of the framework have it do, as cases to time: operators called on their own (as a host runtime calls the library
behind its custom calls) and steps of the three decoders (as the engine runs them).

A case is a dict of plain values.  `listed()` gives the named ones, `draw(rng)` more of the same ranges; `prepare` makes what a program
holds before the call, `run` is one pass, `exact` the same outputs in 64 bits from plain torch.

    attention    paged attention over a block-table cache: `rows` sequences with lengths spread from context / 8 to context
    projection   the int8 weight-only projection of `rows` rows
    llama, latent, mixed   one step of a decoder: `decoding` sequences take one token each (contexts spread like the lengths above), and a
                 prompt portion of `prompt` tokens follows `start` tokens of its sequence that are in the cache already

The decoders' layers have the sizes of the benchmark's workloads; a case takes a few of them, so that the vocabulary's projection keeps about
the share it has in a whole model.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

from tlaloc_b200 import ops
from tlaloc_b200.decoder import LLAMA3_8B, LLAMA3_70B, TINY, Decoder, DecoderConfig
from tlaloc_b200.latent_decoder import LatentDecoder, LatentDecoderConfig
from tlaloc_b200.mixed_decoder import MixedDecoder, MixedDecoderConfig
from tlaloc_b200.paging import PADDING_PAGE, Sequence, stage_ragged

DEVICE = "cuda:0"
VOCAB, WINDOW, KEEP, EPS = 32768, 4096, 64, 1e-5
TYPES = {"bf16": torch.bfloat16, "f32": torch.float32, "f8": torch.float8_e4m3fn}
LLAMA = {"tiny": TINY, "8b": LLAMA3_8B, "70b": LLAMA3_70B}
LATENT = {
    4096: dict(heads=32, dim=128, rot_dim=64, vdim=128, q_rank=1536, kv_rank=512, ff=21504),
    2560: dict(heads=40, dim=64, rot_dim=32, vdim=64, q_rank=768, kv_rank=256, ff=9600),
    2048: dict(heads=16, dim=128, rot_dim=64, vdim=128, q_rank=768, kv_rank=512, ff=8256),
}
MIXED = {
    4096: dict(attention=dict(heads=16, kv_heads=4, dim=128, vdim=256), retention=dict(heads=16, dim=128, vdim=256), ff=14336),
    2560: dict(attention=dict(heads=20, kv_heads=5, dim=64, vdim=128), retention=dict(heads=20, dim=64, vdim=128), ff=6400),
    2048: dict(attention=dict(heads=16, kv_heads=4, dim=64, vdim=128), retention=dict(heads=8, dim=256, vdim=512), ff=1408,
               experts=64, top=6, shared=2816),
}


# ------------------------------------------------------------------------------------------------ the cases

def listed() -> list[dict]:
    return [
        # a single user's decoding through the custom call: one short sequence, latency is all
        dict(name="attention one sequence", kind="attention", rows=1, heads=32, kv_heads=8, dim=128, block=16, context=701, query="f32", pool="bf16", window=0),
        # the operator's usual batch, grouped heads, lengths 512 .. 8192 with a remainder
        dict(name="attention 32 sequences", kind="attention", rows=32, heads=32, kv_heads=8, dim=128, block=16, context=8191, query="bf16", pool="bf16", window=0),
        # the same over the cache that is half the size
        dict(name="attention 8-bit cache", kind="attention", rows=32, heads=32, kv_heads=8, dim=128, block=16, context=8191, query="bf16", pool="f8", window=0),
        # a batch's down projection through the custom call: f32 rows, residual, the default form
        dict(name="projection 40 rows", kind="projection", rows=40, k=14336, n=4096, x="f32", residual=True, swiglu=False, i8=False),
        # one user on a model of 8 billion parameters' layers: a chain of row-vector projections
        dict(name="llama 1 sequence", kind="llama", size="8b", layers=4, pool="bf16", decoding=1, context=1500, prompt=0, start=0),
        # the serving batch on the 70 billion parameters' layers
        dict(name="llama 128 sequences", kind="llama", size="70b", layers=2, pool="bf16", decoding=128, context=8192, prompt=0, start=0),
        # serving the latent-attention decoder: a full decode batch whose longer sequences are past the window
        dict(name="latent decode", kind="latent", width=2560, type="bf16", layers=4, decoding=64, context=8000, prompt=0, start=0),
        # reading a long prompt beside decoding sequences: a portion after the first
        dict(name="latent prompt", kind="latent", width=4096, type="bf16", layers=4, decoding=7, context=4000, prompt=2000, start=2048),
        # checking a model in f32: a short portion beside decoding sequences
        dict(name="latent f32", kind="latent", width=2048, type="f32", layers=2, decoding=3, context=1000, prompt=200, start=300),
        # serving differential attention and retention, a batch that is no power of two
        dict(name="mixed decode", kind="mixed", width=4096, type="bf16", layers=4, decoding=45, context=8000, prompt=0, start=0),
        # its prompts: a portion of a prompt that is past the window already
        dict(name="mixed prompt", kind="mixed", width=2560, type="bf16", layers=4, decoding=0, context=0, prompt=2048, start=5000),
        # its experts with a small decode batch and the beginning of a prompt
        dict(name="mixed experts", kind="mixed", width=2048, type="bf16", layers=4, decoding=15, context=6000, prompt=150, start=0),
    ]


def draw(rng) -> dict:
    """One more case of the ranges above; one that would cost more than the largest of them is drawn again."""
    most = max(_cost(c) for c in listed())
    most_f32 = max(_cost(c) for c in listed() if c.get("type") == "f32")
    while True:
        c = _drawn(rng)
        if _cost(c) <= (most_f32 if c.get("type") == "f32" else most):
            return c


def _cost(case) -> float:
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def _spread(rng, lo: int, hi: int) -> int:
    """A whole number from lo to hi, its logarithm uniform."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _drawn(rng) -> dict:
    kind = rng.choice(["attention", "projection", "llama", "latent", "mixed"])
    if kind == "attention":
        heads, kv_heads = rng.choice([(32, 8), (64, 8), (8, 1), (16, 16), (20, 5), (24, 8)])
        return dict(kind=kind, rows=_spread(rng, 1, 128), heads=heads, kv_heads=kv_heads, dim=rng.choice([64, 128, 128]), block=rng.choice([16, 16, 32, 64]),
                    context=_spread(rng, 16, 16384), query=rng.choice(["f32", "bf16"]), pool=rng.choice(["bf16", "bf16", "f8"]),
                    window=rng.choice([0, 0, 0, 1000, 4096]))
    if kind == "projection":
        swiglu = rng.random() < 0.25
        rows = _spread(rng, 17 if swiglu else 1, 256)
        n = rng.choice([256, 1024, 4096, 5120, 6144, 8192, 11008, 14336, 28672])
        return dict(kind=kind, rows=rows, k=rng.choice([256, 688, 1024, 2048, 2560, 4096, 5120, 8192, 11008, 14336, 28672]), n=2 * n if swiglu else n,
                    x=rng.choice(["bf16", "f32"]), residual=not swiglu and rng.random() < 0.5, swiglu=swiglu, i8=rng.random() < 0.5)
    if kind == "llama":
        case = dict(kind=kind, size=rng.choice(["tiny", "8b", "8b"]), layers=rng.randint(1, 4), pool=rng.choice(["bf16", "bf16", "f8"]))
        most = 128
    elif kind == "latent":
        case = dict(kind=kind, width=rng.choice(sorted(LATENT)), type=rng.choice(["bf16", "bf16", "bf16", "f32"]), layers=rng.randint(1, 4))
        most = 2048 if case["type"] == "bf16" else 256
    else:
        case = dict(kind=kind, width=rng.choice(sorted(MIXED)), type=rng.choice(["bf16", "bf16", "bf16", "f32"]), layers=rng.randint(1, 4))
        most = 2048 if case["type"] == "bf16" else 256
    shape = rng.choice(["decode", "decode", "prompt", "both"])
    decoding = _spread(rng, 1, 64 if shape == "decode" else 63) if shape != "prompt" else 0
    prompt = _spread(rng, 2, most - decoding) if shape != "decode" else 0
    start = rng.choice([0, _spread(rng, 16, 6000)]) if prompt else 0
    return dict(case, decoding=decoding, context=_spread(rng, 16, 8192) if decoding else 0, prompt=prompt, start=start)


def tolerance(case) -> dict:
    """About four times the widest distance from 64 bits that was measured over these ranges."""
    if case["kind"] == "attention":
        return {"rel": 7e-3} if case["query"] == "bf16" else {"rel": 1.5e-5}  # the result is rounded to bf16, or f32 throughout
    if case["kind"] == "projection":
        return {"rel": 7e-3} if case["x"] == "f32" or case["swiglu"] else {"rel": 2e-5}  # rows or results rounded to bf16; exact products, f32 sums
    if case.get("type") == "f32":
        return {"rel": 1.5e-5 if case["kind"] == "latent" else 3e-5}
    out = {"rel": {"llama": 1.5e-2, "latent": 2e-2, "mixed": 3e-2}[case["kind"]], "max": 0.9}  # rounded to bf16 between the projections
    if case.get("pool") == "f8":
        out["differ"] = 0.01  # the new rows of an 8-bit cache
    return out


# ------------------------------------------------------------------------------------------------ what a pass cannot do without

def _lengths(count: int, context: int) -> list[int]:
    """Cached positions of the decoding sequences."""
    return [int(round(v)) for v in np.linspace(max(1, context // 8), max(1, context), count)] if count else []


def _live(length: int, window: int | None, keep: int = 0) -> int:
    """Positions that a token at position length - 1 sees."""
    return length if not window or length <= window else window + min(keep, length - window)


def _portion(case, window, keep=0) -> tuple[int, int]:
    """(positions the prompt portion's tokens see in all, cached positions that any of them sees)"""
    n, start = case["prompt"], case["start"]
    if not n:
        return 0, 0
    seen = sum(_live(start + i + 1, window, keep) for i in range(n))
    return seen, min(start, _live(start + 1, window, keep) - 1)


def _latent_params(width: int) -> dict:
    s = LATENT[width]
    row, qd = s["kv_rank"] + s["rot_dim"], s["dim"] + s["rot_dim"]
    return dict(row=row, each=s["heads"] * 2 * (qd + s["vdim"]),
                weights=width * (s["q_rank"] + row + s["heads"] * s["vdim"] + 2 * s["ff"]) + s["heads"] * (qd * s["q_rank"] + (s["dim"] + s["vdim"]) * s["kv_rank"]))


def work(case) -> dict:
    kind = case["kind"]
    if kind == "attention":
        live = sum(_live(n, case["window"]) for n in _lengths(case["rows"], case["context"]))
        q = case["rows"] * case["heads"] * case["dim"]
        return {"bytes": 2 * live * case["kv_heads"] * case["dim"] * (1 if case["pool"] == "f8" else 2) + 2 * q * (4 if case["query"] == "f32" else 2),
                "flops": 4.0 * live * case["heads"] * case["dim"]}
    if kind == "projection":
        m, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": k * n + 4 * n + m * k * (4 if case["x"] == "f32" else 2) + m * n * (1 if case["swiglu"] else 8 if case["residual"] else 4),
                "flops": 2.0 * m * k * n}
    tokens, want = case["decoding"] + case["prompt"], case["decoding"] + (1 if case["prompt"] else 0)
    contexts = _lengths(case["decoding"], case["context"])
    if kind == "llama":
        c = LLAMA[case["size"]]
        d, hd, vocab = c["d_model"], c["head_dim"], _llama_vocab(case)
        weights = d * (2 * c["num_heads"] + 2 * c["num_kv_heads"]) * hd + 3 * d * c["ffn"]
        seen, cached = _portion(case, None)
        seen += sum(n + 1 for n in contexts)
        kv = (sum(contexts) + cached + tokens) * 2 * c["num_kv_heads"] * hd * (1 if case["pool"] == "f8" else 2)
        return {"bytes": case["layers"] * (weights + kv) + d * vocab + want * 4 * vocab,
                "flops": case["layers"] * (2.0 * tokens * weights + 4.0 * seen * c["num_heads"] * hd) + 2.0 * want * d * vocab}
    e, width = (2 if case["type"] == "bf16" else 4), case["width"]
    head = {"bytes": VOCAB * width * e + want * 4 * VOCAB, "flops": 2.0 * want * width * VOCAB}
    if kind == "latent":
        p = _latent_params(width)
        seen, cached = _portion(case, WINDOW)
        rows = cached + tokens + sum(_live(n + 1, WINDOW) - 1 for n in contexts)
        seen += sum(_live(n + 1, WINDOW) for n in contexts)
        return {"bytes": case["layers"] * e * (p["weights"] + p["row"] * rows) + head["bytes"],
                "flops": case["layers"] * (2.0 * tokens * p["weights"] + seen * p["each"]) + head["flops"]}
    bytes_, flops, s = head["bytes"], head["flops"], MIXED[width]
    seen, cached = _portion(case, WINDOW, KEEP)
    seen += sum(_live(n + 1, WINDOW, KEEP) for n in contexts)
    rows = cached + tokens + sum(_live(n + 1, WINDOW, KEEP) - 1 for n in contexts)
    for layer in _mixed_config(case)["layers"]:
        m = layer["mixer"]
        if layer["type"] == "attention":
            weights = width * (m["heads"] * (2 * m["dim"] + 1 + m["vdim"]) + m["kv_heads"] * (2 * m["dim"] + m["vdim"]))
            bytes_ += e * rows * m["kv_heads"] * (2 * m["dim"] + m["vdim"])
            flops += seen * m["heads"] * 4.0 * (m["dim"] + m["vdim"])
        else:
            weights = width * m["heads"] * (2 * m["dim"] + 3 * m["vdim"])
            bytes_ += 8 * want * m["heads"] * m["dim"] * m["vdim"]
            flops += 4.0 * tokens * m["heads"] * m["dim"] * m["vdim"]
        used = weights = weights + 3 * width * s.get("shared", s["ff"] if "experts" not in s else 0)
        if "experts" in s:
            one = 3 * width * s["ff"]
            weights += width * (s["experts"] + 1) + one * s["experts"] * (1 - (1 - s["top"] / s["experts"]) ** tokens)
            used += width * (s["experts"] + 1) + one * s["top"]
        bytes_ += e * weights
        flops += 2.0 * tokens * used
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------------------------------------------ inputs

def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _normal(g, *shape, kind=torch.bfloat16) -> torch.Tensor:
    """Standard normal values that the type can hold."""
    return torch.randn(shape, device=DEVICE, generator=g, dtype=torch.float32 if kind == torch.float32 else torch.bfloat16).to(kind)


def _codes(g, k: int, n: int):
    """An int8 projection whose results are about as large as its inputs."""
    return (torch.randint(-127, 128, (k, n), dtype=torch.int8, device=DEVICE, generator=g),
            torch.empty((n,), device=DEVICE).uniform_(0.5, 1.5, generator=g) / (73.0 * k ** 0.5))


def _tables(lengths, block: int, rng):
    """Block tables over pages of any order, and the number of pages."""
    need = [-(-n // block) for n in lengths]
    pages, tables, at = 1 + rng.permutation(sum(need)), np.zeros((len(need), max(need)), np.int32), 0
    for r, n in enumerate(need):
        tables[r, :n] = pages[at:at + n]
        at += n
    return tables, at + 1


def _attention_inputs(case, seed):
    g, rng = _generator(seed), np.random.default_rng(seed)
    lengths = rng.permutation(_lengths(case["rows"], case["context"]))
    tables, blocks = _tables(lengths, case["block"], rng)
    pool = lambda: _normal(g, blocks, case["block"], case["kv_heads"], case["dim"], kind=TYPES[case["pool"]])
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.int32)).to(DEVICE)
    return dict(query=_normal(g, case["rows"], case["heads"], case["dim"], kind=TYPES[case["query"]]), keys=pool(), values=pool(), tables=to(tables),
                lengths=to(lengths), scale=case["dim"] ** -0.5)


def _projection_inputs(case, seed):
    g = _generator(seed)
    codes, scales = _codes(g, case["k"], case["n"])
    return dict(x=_normal(g, case["rows"], case["k"], kind=TYPES[case["x"]]), codes=codes, scales=scales,
                residual=_normal(g, case["rows"], case["n"], kind=torch.float32) if case["residual"] else None)


def _llama_vocab(case) -> int:
    return min(VOCAB, LLAMA[case["size"]]["vocab"])


def _llama_weights(case, seed):
    c, g = LLAMA[case["size"]], _generator(seed)
    d, hd, vocab = c["d_model"], c["head_dim"], _llama_vocab(case)
    gain = lambda: 1.0 + 0.1 * _normal(g, d, kind=torch.float32)
    layers = [dict(q=_codes(g, d, c["num_heads"] * hd), k=_codes(g, d, c["num_kv_heads"] * hd), v=_codes(g, d, c["num_kv_heads"] * hd),
                   o=_codes(g, c["num_heads"] * hd, d), gate=_codes(g, d, c["ffn"]), up=_codes(g, d, c["ffn"]), down=_codes(g, c["ffn"], d),
                   ln1=gain(), ln2=gain()) for _ in range(case["layers"])]
    return SimpleNamespace(embed=_normal(g, vocab, d).float(), layers=layers, final_norm=gain(), head=_codes(g, d, vocab))


def _latent_config(case) -> dict:
    s = LATENT[case["width"]]
    mixer = {k: s[k] for k in ("heads", "dim", "rot_dim", "vdim", "q_rank", "kv_rank")}
    mixer.update(scale=(s["dim"] + s["rot_dim"]) ** -0.5, mask={"size": WINDOW},
                 rot={"base": 10000.0, "dims": s["rot_dim"], "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}})
    layer = {"type": "latent_attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": s["ff"]}}
    return {"architecture": "Marotar", "width": case["width"], "vocab": VOCAB, "norm": {"eps": EPS}, "layers": [layer] * case["layers"]}


def _mixed_config(case) -> dict:
    """Three layers of retention to one of attention, which is the second of each four."""
    s = MIXED[case["width"]]
    rot = lambda d: {"base": 10000.0, "dims": d}
    a, r = s["attention"], s["retention"]
    attention = dict(a, rot=rot(a["dim"]), scale=a["dim"] ** -0.5, diff=0.3, mask={"size": WINDOW, "keep_first": KEEP})
    retention = dict(r, rot=rot(r["dim"]), decay=[1 - 0.5 ** (5 + 4 * h / r["heads"]) for h in range(r["heads"])])
    mlp = {"kind": "dense", "ff": s["ff"]}
    if "experts" in s:
        mlp = {"kind": "moe", "expert": {"ff": s["ff"]}, "router": {"experts": s["experts"], "top": s["top"]}, "shared": {"ff": s["shared"]}}
    layers = [{"type": "attention" if i % 4 == 1 else "retention", "mixer": attention if i % 4 == 1 else retention, "mlp": mlp} for i in range(case["layers"])]
    return {"architecture": "Videdra", "width": case["width"], "vocab": VOCAB, "norm": {"eps": EPS}, "layers": layers}


def _checkpoint(cfg, seed) -> dict:
    """Random tensors of a checkpoint, sized so that activations stay about one through the layers; a router's as a trained one's, whose first
    choices stand out."""
    g, out = _generator(seed), {}
    around_zero = isinstance(cfg, LatentDecoderConfig)  # the design stores these gains so
    for name, shape in cfg.tensor_shapes().items():
        t = _normal(g, *shape)
        if len(shape) == 1:
            gain = ("norm" in name or ".ls" in name) and not (around_zero and not name.endswith((".dq.norm", ".dkv.norm")))
            out[name] = 0.1 * t + 1.0 if gain else 0.1 * t
        else:
            out[name] = t if name == "embed" and not around_zero else t * ((3.0 if name.endswith("router") else 1.0) * shape[1] ** -0.5)
    return out


def _sequences(case, seed, *, block: int, window=None, keep: int = 0):
    """([(sequence, its next tokens)], pages of the pool): the sequences hold pages in any order, none where no window reaches any more."""
    rng = np.random.default_rng(seed)
    counts = [(int(n), 1) for n in rng.permutation(_lengths(case["decoding"], case["context"]))]
    if case["prompt"]:
        counts.append((case["start"], case["prompt"]))
    held = []
    for length, n in counts:
        dropped = max(0, length - window + 1) // block if window else 0
        held.append([b < -(-keep // block) or b >= dropped for b in range(-(-(length + n) // block))])
    pages = iter(1 + rng.permutation(sum(sum(h) for h in held)))
    vocab = _llama_vocab(case) if case["kind"] == "llama" else VOCAB
    work = [(Sequence(pages=[int(next(pages)) if here else PADDING_PAGE for here in h], length=length, state=s + 1), rng.integers(0, vocab, size=n).tolist())
            for s, (h, (length, n)) in enumerate(zip(held, counts))]
    return work, 1 + sum(sum(h) for h in held)


def _wanted(work) -> list[int]:
    """The rows whose logits the engine reads: the last of every sequence."""
    return [int(r) for r in np.cumsum([len(tokens) for _, tokens in work]) - 1]


def _fill(g, tensors, spread=1.0) -> None:
    for t in tensors:
        if t.dtype == torch.float8_e4m3fn:
            t.copy_(_normal(g, *t.shape))
        else:
            t.normal_(0.0, spread, generator=g)


def _caches(model) -> tuple[list, list]:
    """(what the model keeps in pages, what it keeps in state slots), each buffer once"""
    if isinstance(model, Decoder):
        return model.key_pools + model.value_pools, []
    return [p for p in model.pools if p is not None], [s for s in getattr(model, "states", []) if s is not None]


def _model(case, seed):
    """(model, its sequences and tokens): what a server holds before a step."""
    block = 16 if case["kind"] == "llama" else 64
    work, blocks = _sequences(case, seed, block=block, **({} if case["kind"] == "llama" else {"window": WINDOW, "keep": KEEP if case["kind"] == "mixed" else 0}))
    max_len = max(s.length + len(t) for s, t in work)
    if case["kind"] == "llama":
        tokens = sum(len(t) for _, t in work)
        c = dict(LLAMA[case["size"]], num_layers=case["layers"], vocab=_llama_vocab(case))
        model = Decoder(DecoderConfig(**c, kv_dtype=TYPES[case["pool"]], max_positions=max_len), tokens, blocks, -(-max_len // block), device=DEVICE)
        w, host = _llama_weights(case, seed), lambda v: tuple(t.cpu().numpy() for t in v) if isinstance(v, tuple) else v.cpu().numpy()
        model.load_host_weights(SimpleNamespace(embed=host(w.embed), final_norm=host(w.final_norm), head=host(w.head),
                                                layers=[{k: host(v) for k, v in lw.items()} for lw in w.layers]))
    else:
        cls, cfg = (LatentDecoder, LatentDecoderConfig.from_config(_latent_config(case))) if case["kind"] == "latent" else \
            (MixedDecoder, MixedDecoderConfig.from_config(_mixed_config(case)))
        model = cls(cfg, num_blocks=blocks, max_len=max_len, dtype=TYPES[case["type"]], device=DEVICE)  # up to 2048 tokens of 64 sequences a step
        model.load_tensors(_checkpoint(cfg, seed))
    pools, states = _caches(model)
    g = _generator(seed + 1)
    _fill(g, pools)
    _fill(g, states, 2.0)
    return model, work


def prepare(case, seed) -> dict:
    ops.init()
    if case["kind"] == "attention":
        return dict(case=case, **_attention_inputs(case, seed))
    if case["kind"] == "projection":
        return dict(case=case, **_projection_inputs(case, seed))
    model, work = _model(case, seed)
    if case["kind"] == "llama":
        model.capture()  # the step of a server: one graph for its batch (the other models capture the decode batches that come again themselves)
    return dict(case=case, model=model, step=stage_ragged(work, max_blocks=model.max_blocks, block_size=model.block_size), want=_wanted(work))


# ------------------------------------------------------------------------------------------------ a pass

def run(state):
    case = state["case"]
    if case["kind"] == "attention":
        return ops.paged_attention(state["query"], state["keys"], state["values"], state["tables"], state["lengths"], scale=state["scale"],
                                   sliding_window=case["window"] or None)
    if case["kind"] == "projection":
        if case["swiglu"]:
            return ops.int8_gemm_swiglu(state["x"], state["codes"], state["scales"], i8_mma=case["i8"])
        return ops.int8_gemm(state["x"], state["codes"], state["scales"], residual=state["residual"], i8_mma=case["i8"])
    # one step as the engine runs it: the rows' logits, and the next tokens from them.  The tokens themselves are not among the outputs:
    # wherever the two largest logits are within rounding of one another, two correct implementations choose differently.
    model = state["model"]
    logits = model.run(state["step"], state["want"])
    model.greedy(logits)
    pools, states = _caches(model)
    return {"logits": logits, "cache": [p.view(torch.int8) if p.dtype == torch.float8_e4m3fn else p for p in pools], "states": [s[1:] for s in states]}  # slot 0 is padding's


# ------------------------------------------------------------------------------------------------ the same in 64 bits

def exact(case, seed):
    with torch.no_grad():
        return {"attention": _exact_attention, "projection": _exact_projection, "llama": _exact_llama, "latent": _exact_latent, "mixed": _exact_mixed}[case["kind"]](case, seed)


def _exact_attention(case, seed):
    s = _attention_inputs(case, seed)
    out = torch.empty(s["query"].shape, dtype=torch.float64, device=DEVICE)
    group = case["heads"] // case["kv_heads"]
    for r, n in enumerate(s["lengths"].tolist()):
        first = max(0, n - case["window"]) if case["window"] else 0
        k, v = (_paged(p, s["tables"][r], torch.arange(first, n, device=DEVICE)) for p in (s["keys"], s["values"]))
        q = s["query"][r].double().view(case["kv_heads"], group, case["dim"])
        p = torch.softmax(torch.einsum("gqd,ngd->gqn", q, k) * s["scale"], -1)
        out[r] = torch.einsum("gqn,ngd->gqd", p, v).reshape(case["heads"], case["dim"])
    return out


def _paged(pool, table, positions):
    """The pool's rows of those positions, in 64 bits."""
    blocks = pool.shape[1]
    slots = table.long()[positions // blocks] * blocks + positions % blocks
    flat = pool.view(-1, *pool.shape[2:])
    if flat.dtype == torch.float8_e4m3fn:
        return flat.view(torch.int8)[slots].view(torch.float8_e4m3fn).double()
    return flat[slots].double()


def _silu(z):
    return z / (1 + torch.exp(-z))


def _times(x, codes, scales):
    """x @ (codes * scales), some columns at a time"""
    return torch.cat([(x @ codes[:, c:c + 8192].double()) * scales[c:c + 8192].double() for c in range(0, codes.shape[1], 8192)], 1)


def _exact_projection(case, seed):
    s = _projection_inputs(case, seed)
    y = _times(s["x"].double(), s["codes"], s["scales"])
    if case["swiglu"]:
        y = y.view(case["rows"], -1, 2, 128)
        return (_silu(y[:, :, 0]) * y[:, :, 1]).reshape(case["rows"], -1)
    return y + s["residual"].double() if case["residual"] else y


def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _turn(x, positions, freqs, magnitude=1.0, interleaved=False):
    """x [tokens, heads, 2 * len(freqs)] with its pairs turned: (2i, 2i + 1), or (i, i + half)."""
    a = positions.double()[:, None] * freqs[None]
    c, s = (torch.cos(a) * magnitude)[:, None], (torch.sin(a) * magnitude)[:, None]
    u, v = (x[..., 0::2], x[..., 1::2]) if interleaved else x.chunk(2, -1)
    pair = (u * c - v * s, v * c + u * s)
    return torch.stack(pair, -1).flatten(-2) if interleaved else torch.cat(pair, -1)


def _freqs(dims: int, base: float = 10000.0):
    return base ** (-2.0 * torch.arange(dims // 2, device=DEVICE, dtype=torch.float64) / dims)


class _Cache:
    """The paged rows of a layer, those in the pool at the start and the step's own in 64 bits."""

    def __init__(self, pool, step, work):
        self.pool, self.step, self.work = pool, step, work
        self.slots = torch.from_numpy(step.slot_mapping).to(DEVICE).long()
        self.tables = torch.from_numpy(step.block_tables).to(DEVICE)

    def rows(self, s: int, new, window=None, keep: int = 0):
        """(rows, their positions) that the tokens of sequence s see, its new ones last"""
        n = self.work[s][0].length
        p = torch.arange(n, device=DEVICE)
        if window:
            p = p[(p > n - window) | (p < keep)]
        return torch.cat([_paged(self.pool, self.tables[s], p), new]), torch.cat([p, n + torch.arange(new.shape[0], device=DEVICE)])

    def after(self, new):
        """The pool after the step, in 64 bits."""
        out = self.pool.double()
        out.view(-1, *self.pool.shape[2:])[self.slots] = new
        return out


def _seen(positions, keys, window=None, keep: int = 0):
    d = positions[:, None] - keys[None]
    return (d >= 0) & ((d < window) | (keys[None] < keep)) if window else d >= 0


def _attend(q, k, v, mask, scale):
    """One head: q [n, d], k [l, d], v [l, e]."""
    return torch.softmax((q @ k.T * scale).masked_fill(~mask, -math.inf), -1) @ v


def _staged(case, seed):
    model, work = _model(case, seed)  # for the cache's first contents alone
    step = stage_ragged(work, max_blocks=model.max_blocks, block_size=model.block_size)
    to = lambda a: torch.from_numpy(a).to(DEVICE).long()
    return model, work, step, to(step.token_ids), to(step.positions), torch.tensor(_wanted(work), device=DEVICE)


def _exact_llama(case, seed):
    model, work, step, ids, positions, want = _staged(case, seed)
    w, c = _llama_weights(case, seed), LLAMA[case["size"]]
    heads, kvh, hd, n = c["num_heads"], c["num_kv_heads"], c["head_dim"], len(step.token_ids)
    freqs, x, keys, values = _freqs(hd), w.embed[ids].double(), [], []
    for l, lw in enumerate(w.layers):
        h = _rms(x) * lw["ln1"].double()
        q = _turn(_times(h, *lw["q"]).view(n, heads, hd), positions, freqs)
        k = _turn(_times(h, *lw["k"]).view(n, kvh, hd), positions, freqs)
        v = _times(h, *lw["v"]).view(n, kvh, hd)
        ck, cv = _Cache(model.key_pools[l], step, work), _Cache(model.value_pools[l], step, work)
        o = torch.empty((n, heads, hd), dtype=torch.float64, device=DEVICE)
        for s, (a, b) in enumerate(zip(step.starts[:-1], step.starts[1:])):
            (ks, at), (vs, _) = ck.rows(s, k[a:b]), cv.rows(s, v[a:b])
            mask = _seen(positions[a:b], at)
            for i in range(heads):
                o[a:b, i] = _attend(q[a:b, i], ks[:, i * kvh // heads], vs[:, i * kvh // heads], mask, hd ** -0.5)
        x = x + _times(o.view(n, -1), *lw["o"])
        h = _rms(x) * lw["ln2"].double()
        x = x + _times(_silu(_times(h, *lw["gate"])) * _times(h, *lw["up"]), *lw["down"])
        keys.append(ck.after(k) if case["pool"] != "f8" else None)
        values.append(cv.after(v) if case["pool"] != "f8" else None)
    return {"logits": _times(_rms(x[want]) * w.final_norm.double(), *w.head), "cache": keys + values, "states": []}


def _exact_latent(case, seed):
    model, work, step, ids, positions, want = _staged(case, seed)
    config = _latent_config(case)
    t = _checkpoint(LatentDecoderConfig.from_config(config), seed)
    n, x, cache = len(step.token_ids), t["embed"].double()[ids], []
    for i, layer in enumerate(config["layers"]):
        m, w = layer["mixer"], lambda name: t[f"l{i}.{name}"].double()
        heads, rank, rot = m["heads"], m["kv_rank"], m["rot"]
        freqs, s = _freqs(rot["dims"], rot["base"]), rot["scaling"]
        turns = lambda k: rot["dims"] * math.log(s["original"] / (2.0 * math.pi * k)) / (2.0 * math.log(rot["base"]))
        lo, hi = max(math.floor(turns(s["fast"])), 0), min(math.ceil(turns(s["slow"])), rot["dims"] - 1)
        ramp = ((torch.arange(len(freqs), device=DEVICE, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        turned = lambda v: _turn(v, positions, freqs / s["factor"] * ramp + freqs * (1 - ramp), 0.1 * math.log(s["factor"]) + 1.0, interleaved=True)
        h = _rms(x) * (1 + w("norm1"))
        q = ((_rms(h @ w("mix.dq").T) * w("mix.dq.norm")) @ w("mix.uq").T).view(n, heads, -1)
        q = torch.cat([q[..., :m["dim"]], turned(q[..., m["dim"]:])], -1)
        down = h @ w("mix.dkv").T
        new = torch.cat([_rms(down[:, :rank]) * w("mix.dkv.norm"), turned(down[:, None, rank:])[:, 0]], 1)
        held = _Cache(model.pools[i], step, work)
        o = torch.empty((n, heads, m["vdim"]), dtype=torch.float64, device=DEVICE)
        for s_, (a, b) in enumerate(zip(step.starts[:-1], step.starts[1:])):
            rows, at = held.rows(s_, new[a:b], m["mask"]["size"])
            k = (rows[:, :rank] @ w("mix.uk").T).view(-1, heads, m["dim"])
            v = (rows[:, :rank] @ w("mix.uv").T).view(-1, heads, m["vdim"])
            mask = _seen(positions[a:b], at, m["mask"]["size"])
            for j in range(heads):
                o[a:b, j] = _attend(q[a:b, j], torch.cat([k[:, j], rows[:, rank:]], 1), v[:, j], mask, m["scale"])
        y = o.view(n, -1) @ w("mix.o").T
        h = _rms(x) * (1 + w("norm2"))
        x = x + y + (h @ w("mlp.up").T + w("mlp.up.b")).clamp_min(0).square() @ w("mlp.down").T + w("mlp.down.b")
        cache.append(held.after(new))
    return {"logits": _rms(x[want]) * (1 + t["final.norm"].double()) @ t["embed"].double().T, "cache": cache, "states": []}


def _exact_retention(q, k, v, decay, state):
    """q, k [n, d], v [n, e] of one head, its state before: outputs and the state after."""
    n = q.shape[0]
    i = torch.arange(n, device=DEVICE, dtype=torch.float64)
    weight = torch.where(i[:, None] >= i[None], decay ** (i[:, None] - i[None]).clamp_min(0), 0.0)
    o = (q @ k.T * weight) @ v + decay ** (i + 1)[:, None] * (q @ state)
    return o, decay ** n * state + (k * decay ** (n - 1 - i)[:, None]).T @ v


def _exact_experts(h, w, mlp):
    z = h @ w("mlp.router").T
    top = torch.topk(z, mlp["router"]["top"], -1)
    weights = torch.zeros_like(z).scatter_(1, top.indices, torch.softmax(top.values, -1))
    gated = lambda rows, p: (_silu(rows @ w(p + "gate").T) * (rows @ w(p + "up").T)) @ w(p + "down").T
    y = torch.sigmoid(h @ w("mlp.shared.sg").T) * gated(h, "mlp.shared.")
    for e in range(mlp["router"]["experts"]):
        rows = weights[:, e].nonzero()[:, 0]
        if len(rows):
            y[rows] += weights[rows, e, None] * gated(h[rows], f"mlp.e{e}.")
    return y


def _exact_mixed(case, seed):
    model, work, step, ids, positions, want = _staged(case, seed)
    config = _mixed_config(case)
    t = _checkpoint(MixedDecoderConfig.from_config(config), seed)
    n, x, cache, states = len(step.token_ids), t["embed"].double()[ids], [], []
    for i, layer in enumerate(config["layers"]):
        m, mlp, w = layer["mixer"], layer["mlp"], lambda name: t[f"l{i}.{name}"].double()
        heads, dim, vdim = m["heads"], m["dim"], m["vdim"]
        freqs, h = _freqs(dim, m["rot"]["base"]), _rms(x) * w("norm1")
        o = torch.empty((n, heads, vdim), dtype=torch.float64, device=DEVICE)
        spans = list(enumerate(zip(step.starts[:-1], step.starts[1:])))
        if layer["type"] == "attention":
            groups, mask = m["kv_heads"], m["mask"]
            q = _turn((h @ w("mix.q").T).view(n, heads * 2, dim), positions, freqs)
            k = _turn((h @ w("mix.k").T).view(n, groups * 2, dim), positions, freqs)
            new = torch.cat([k.reshape(n, -1), h @ w("mix.v").T], 1)
            held = _Cache(model.pools[i], step, work)
            factor = torch.exp((w("mix.lq1") * w("mix.lk1")).sum()) - torch.exp((w("mix.lq2") * w("mix.lk2")).sum()) + m["diff"]
            for s, (a, b) in spans:
                rows, at = held.rows(s, new[a:b], mask["size"], mask["keep_first"])
                ks, vs = rows[:, :groups * 2 * dim].view(-1, groups, 2, dim), rows[:, groups * 2 * dim:].view(-1, groups, vdim)
                seen = _seen(positions[a:b], at, mask["size"], mask["keep_first"])
                for j in range(heads):
                    u = j // (heads // groups)
                    one, two = (_attend(q[a:b, 2 * j + p], ks[:, u, p], vs[:, u], seen, m["scale"]) for p in (0, 1))
                    o[a:b, j] = one - factor * two
            y = (_rms(o) * (1 - m["diff"]) * torch.sigmoid(h @ w("mix.g").T)[:, :, None]).reshape(n, -1)
            cache.append(held.after(new))
        else:
            q = _turn((h @ w("mix.q").T).view(n, heads, dim), positions, freqs)
            k = _turn((h @ w("mix.k").T).view(n, heads, dim), positions, freqs) * dim ** -0.5
            v, state = (h @ w("mix.v").T).view(n, heads, vdim), model.states[i].double()
            for s, (a, b) in spans:
                slot = work[s][0].state
                before = state[slot] if work[s][0].length else torch.zeros_like(state[slot])
                for j in range(heads):
                    o[a:b, j], state[slot, j] = _exact_retention(q[a:b, j], k[a:b, j], v[a:b, j], m["decay"][j], before[j])
            y = _rms(o).reshape(n, -1) * _silu(h @ w("mix.g").T)
            states.append(state[1:])
        x = x + _rms(y @ w("mix.o").T) * w("norm1b") * w("ls1")
        h = _rms(x) * w("norm2")
        if mlp["kind"] == "dense":
            z = h @ w("mlp.gate").T
            y = (0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3))) * (h @ w("mlp.up").T)) @ w("mlp.down").T
        else:
            y = _exact_experts(h, w, mlp)
        x = x + _rms(y) * w("norm2b") * w("ls2")
    return {"logits": (_rms(x[want]) * t["final.norm"].double()) @ t["head"].double().T, "cache": cache, "states": states}
