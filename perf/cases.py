"""The work that programs have this framework do, as cases that can be timed and checked.

A case is a dict of plain values; `prepare` makes what a program holds before the call, `run` is one pass through the public
entry points, `exact` is the same from plain torch in 64 bits.  Eight kinds of work:

  token    `ops.gqa_decode_attention`: one decoded token of one sequence over a contiguous cache, the reference's own operator
           and (in fp32) its own type
  layer    `ops.qkv_decode_step_paged`: the decode step of one layer over a paged cache of a batch, from the output of the QKV
           projection (head norms, rotation, append, attention), as every layer of a step after the first calls it
  prompt   `ops.scaled_dot_product_attention` over a whole prompt (causal) or over an image's patches (not causal)
  tower    `TextTower.decode_step`, the 28-layer step of the text tower, as a CUDA graph
  nuderax_decode, rigozen_decode   a decode step of the language models, as a CUDA graph like the serving engine's
  nuderax_prompt, rigozen_prompt   `ModelRunner.step`: a prompt brought whole or in portions of a step's token budget
"""
import math
import zlib

import numpy as np
import torch

from axono_b200 import models, ops
from axono_b200.cuda_graph import CUDAGraph
from axono_b200.decode import TextTower, TextTowerConfig
from axono_b200.kv_cache import PagedKVCache
from axono_b200.models.layers import Rows
from axono_b200.models.nuderax import tensor_shapes as nuderax_shapes
from axono_b200.models.rigozen import tensor_shapes as rigozen_shapes
from axono_b200.serving import ModelRunner

DEV = "cuda"
DTYPES = {"f32": torch.float32, "f16": torch.float16}
EPS = 1e-6       # of the tower's norms
LM_EPS = 1e-5    # of the language models' norms
THETA = 1e6
VOCAB = 32768    # of the language models


# ---- the cases ------------------------------------------------------------------------------------------------------------

def listed():
    return [
        # a chat's first answer through the reference's operator, one sequence in the reference's type: latency
        dict(name="token_f32", kind="token", dtype="f32", hq=16, hkv=8, d=128, keys=1000),
        # a long document and a model with heads of 64, same operator
        dict(name="token_f32_d64_long", kind="token", dtype="f32", hq=16, hkv=8, d=64, keys=16001),
        # the fused decode block's batch: few sequences, one wave of work
        dict(name="layer_b8", kind="layer", batch=8, context=8192, hq=16, hkv=8, d=128),
        # the long-context batch: 64 sequences of 16 K to 32 K tokens
        dict(name="layer_b64_ragged", kind="layer", batch=64, context=32768, hq=16, hkv=8, d=128),
        # the multimodal prompt (1024 image and 512 text tokens) in the type that the reference's operator takes
        dict(name="prompt_f32", kind="prompt", dtype="f32", hq=16, hkv=8, d=128, tokens=1536, causal=True),
        # a long prompt in half precision
        dict(name="prompt_f16", kind="prompt", dtype="f16", hq=16, hkv=8, d=128, tokens=8192, causal=True),
        # patches of an image (60 x 45) through a vision encoder's attention: heads of 64, every patch sees all
        dict(name="patches_f16_d64", kind="prompt", dtype="f16", hq=16, hkv=16, d=64, tokens=2700, causal=False),
        # the reference's own model, a small batch at short context: weights weigh as much as the cache
        dict(name="tower_decode", kind="tower", batch=8, context=2048),
        # serving of the language models: a batch in the middle of its answers, and prompts
        dict(name="nuderax_decode", kind="nuderax_decode", size="4k", layers=2, batch=32, context=16384),
        dict(name="rigozen_decode", kind="rigozen_decode", size="2k", layers=4, batch=32, context=16384),
        dict(name="nuderax_prompt", kind="nuderax_prompt", size="2k", layers=4, tokens=2000, portion=2048),
        dict(name="rigozen_prompt", kind="rigozen_prompt", size="2k", layers=4, tokens=8192, portion=2048),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["token", "layer", "prompt", "tower", "nuderax_decode", "rigozen_decode", "nuderax_prompt", "rigozen_prompt"])
    hkv, group = rng.choice([2, 4, 8]), rng.choice([1, 2, 4, 8])
    heads = dict(hq=min(32, hkv * group), hkv=min(hkv, min(32, hkv * group)))
    if kind == "token":
        return dict(kind=kind, dtype=rng.choice(["f32", "f32", "f16"]), **heads, d=rng.choice([64, 80, 96, 128]), keys=log_int(64, 32768))
    if kind == "layer":
        batch = log_int(1, 64)
        return dict(kind=kind, batch=batch, context=min(log_int(256, 32768), 32768 * 64 // batch), **heads, d=rng.choice([64, 128, 128]))
    if kind == "prompt":
        dtype = rng.choice(["f32", "f16"])
        return dict(kind=kind, dtype=dtype, **heads, d=rng.choice([64, 80, 128, 128]),
                    tokens=log_int(16, 4096 if dtype == "f32" else 8192), causal=rng.random() < 0.7)
    if kind == "tower":
        batch = log_int(1, 32)
        return dict(kind=kind, batch=batch, context=min(log_int(128, 8192), 32768 // batch))
    size = rng.choice(["2k", "4k"])
    layers = 4 if kind.startswith("rigozen") or size == "2k" else 2
    if kind.endswith("decode"):
        return dict(kind=kind, size=size, layers=layers, batch=log_int(1, 64), context=log_int(256, 8192))
    most = {"nuderax_prompt": {"2k": 4600, "4k": 3300}, "rigozen_prompt": {"2k": 8192, "4k": 2200}}[kind][size]  # like costs
    tokens = log_int(48, most)
    return dict(kind=kind, size=size, layers=layers, tokens=tokens, portion=rng.choice([2048, 8192]))


def lengths(case):
    """Tokens cached per sequence: one sequence holds the whole context, the others between half of it and all."""
    draw_ = np.random.RandomState(7).randint((case["context"] + 1) // 2, case["context"] + 1, case["batch"])
    draw_[0] = case["context"]
    return [int(n) for n in draw_]


# ---- what the inputs are made with ------------------------------------------------------------------------------------------

def generator(seed, *parts):
    return torch.Generator(device=DEV).manual_seed(zlib.crc32(repr((seed, parts)).encode()))


def normal(shape, dtype, seed, *parts):
    """N(0, 1) values of one tensor, which its seed and its name determine."""
    return torch.randn(shape, generator=generator(seed, *parts), device=DEV, dtype=dtype)


def some_ids(n, vocab, seed, *parts):
    return torch.randint(0, vocab, (n,), generator=generator(seed, *parts), device=DEV)


class Weights:
    """A model's tensors by name, bf16, each made from the seed and its name when it is asked for."""

    AROUND_ZERO = {"nuderax": ("correction",), "rigozen": ("norm1", "norm2", "final.norm")}

    def __init__(self, design, shapes, seed):
        self.design, self.shapes, self.seed = design, shapes, seed

    def __getitem__(self, name):
        shape = self.shapes[name]
        w = normal(shape, torch.float32, self.seed, name)
        if name.endswith("A_log"):
            w = w - 1.5
        elif name.endswith("dt_bias"):
            w = 0.5 * w - 1.0
        elif name.endswith("sink"):
            w = w + 1.5
        elif len(shape) == 1:
            w = 0.1 * w + (0.0 if name.endswith(self.AROUND_ZERO[self.design]) else 2.0 if name.endswith("q.norm") else 1.0)
        elif name.endswith("conv"):
            w = 0.7 * w
        elif name != "embed":  # queries that single out a few keys; Nuderax: updates that are small beside the residual
            gain = 2.0 if name.endswith("uq") or (name.endswith("mix.q") and f"{name[:-1]}uk" in self.shapes) else 1.0
            if self.design == "nuderax":
                gain = 0.5 if name.endswith("mix.o") else 0.03 if name.endswith("down") else gain
            w = w * (gain * shape[1] ** -0.5)
        return w.to(torch.bfloat16)


NUDERAX = {
    "2k": dict(width=2048, heads=16, q_rank=1536, ff=1408, shared_ff=2816, experts=64, top=6, groups=8, keep=3),
    "4k": dict(width=4096, heads=32, q_rank=1536, ff=2048, shared_ff=2048, experts=64, top=8, groups=8, keep=4),
}
RIGOZEN = {
    "2k": dict(width=2048, ff=6144, delta=(16, 8), latent=16, attn=(16, 8), window=4096),
    "4k": dict(width=4096, ff=12288, delta=(32, 16), latent=32, attn=(32, 8), window=4096),
}


def model_config(case):
    """config.json of a case's model: Nuderax layers alternate direct and low-rank queries; Rigozen layers go delta, delta,
    latent attention, attention."""
    layers = []
    if case["kind"].startswith("nuderax"):
        z = NUDERAX[case["size"]]
        mlp = {"kind": "moe", "expert": {"ff": z["ff"], "limit": 7.0}, "shared": {"ff": z["shared_ff"], "limit": 7.0},
               "router": {"experts": z["experts"], "top": z["top"], "scale": 1.5, "groups": {"count": z["groups"], "keep": z["keep"]}}}
        for i in range(case["layers"]):
            m = {"heads": z["heads"], "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
                 "rot": {"base": 10000.0, "dims": 64}}
            if i % 2:
                m["q_rank"] = z["q_rank"]
            layers.append({"type": "latent_attention_2" if i % 2 else "latent_attention", "mixer": m, "mlp": mlp})
        name = "Nuderax"
    else:
        z = RIGOZEN[case["size"]]
        mask, scale = {"size": z["window"]}, 128 ** -0.5
        kinds = [("delta", dict(heads=z["delta"][0], kv_heads=z["delta"][1], dim=128, vdim=128, conv=4))] * 2 + [
            ("latent_attention", dict(heads=z["latent"], dim=128, vdim=128, kv_rank=512, scale=scale, mask=mask)),
            ("attention", dict(heads=z["attn"][0], kv_heads=z["attn"][1], dim=128, vdim=128, scale=scale, mask=mask))]
        layers = [dict(type=kinds[i % 4][0], mixer=kinds[i % 4][1], mlp=dict(kind="dense", ff=z["ff"])) for i in range(case["layers"])]
        name = "Rigozen"
    return {"architecture": name, "vocab": VOCAB, "width": z["width"], "norm": {"eps": LM_EPS}, "layers": layers}


def model_weights(case, seed):
    cfg = model_config(case)
    shapes = (nuderax_shapes if cfg["architecture"] == "Nuderax" else rigozen_shapes)(models.config_of(cfg))
    return cfg, Weights(cfg["architecture"].lower(), dict(shapes), seed)


TOWER_PARTS = {"input_ln": None, "post_ln": None, "q_norm": None, "k_norm": None, "qkv": 1.0, "o": 0.3, "gate_up": 1.0, "down": 0.3}


def tower_weight(name, shape, seed, *parts):
    w = normal(shape, torch.float16, seed, name, *parts)
    return 1 + 0.02 * w if TOWER_PARTS.get(name, 1.0) is None else w * (TOWER_PARTS.get(name, 1.0) * shape[1] ** -0.5)


# ---- prepare ----------------------------------------------------------------------------------------------------------------

class Held:
    """A program's model, cache and step; gives the cache's memory back when nothing refers to it or its outputs."""

    def __init__(self, runner):
        self.runner, self.graph, self.views, self.inputs = runner, None, [], None

    def outputs(self, *first):
        """`first` and the cache and state, which keep this object alive as long as they are."""
        views = []
        for t in self.views:
            v = t.detach()
            v.held = self
            views.append(v)
        return [*first, *views]

    def close(self):
        torch.cuda.synchronize()
        if self.graph is not None:
            self.graph.reset()
        self.runner.arena.close()

    def __del__(self):
        if torch is not None and torch.cuda is not None:  # not while the interpreter ends
            self.close()


def cache_views(runner, cfg):
    """Tensors of everything a runner keeps: latent rows, raw keys and their factors, recurrent state."""
    views, at = [], 0
    for layer in cfg["layers"]:
        if layer["type"] == "delta":
            continue
        pool, m = runner.pages[at], layer["mixer"]
        at += 1
        if layer["type"] == "attention":
            rows = pool.shape[1] * m["kv_heads"] * m["dim"]
            views += [pool.view(pool.shape[0], -1)[:, :rows], ops.shared_kv_factors(pool)]
        else:
            views.append(pool)
    return views + [t for layer in runner.states for t in layer]


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"].split("_")[-1]](case, seed)


def _prepare_token(case, seed):
    dt, sh = DTYPES[case["dtype"]], (case["keys"], case["hkv"], case["d"])
    return {"kind": "token", "args": (normal((1, case["hq"], case["d"]), dt, seed, "q"), normal(sh, dt, seed, "k"), normal(sh, dt, seed, "v"))}


def _prompt_tensors(case, seed):
    dt, n, d = DTYPES[case["dtype"]], case["tokens"], case["d"]
    return [normal((n, h, d), dt, seed, name) for name, h in (("q", case["hq"]), ("k", case["hkv"]), ("v", case["hkv"]))]


def _layer_tensors(case, seed):
    """qkv, head norms' weights, and the cache: keys and values (batch, tokens, hkv, d), scaled so that scores stay moderate."""
    b, hq, hkv, d, n = case["batch"], case["hq"], case["hkv"], case["d"], case["context"]
    half = torch.float16
    qkv = normal((b, (hq + 2 * hkv) * d), half, seed, "qkv")
    norms = [1 + 0.02 * normal((d,), half, seed, name) for name in ("q_norm", "k_norm")]
    kv = [normal((b, n, hkv, d), half, seed, name).mul_(0.5) for name in ("k", "v")]
    return qkv, norms, kv


def _prepare_layer(case, seed):
    qkv, norms, (k, v) = _layer_tensors(case, seed)
    lens = lengths(case)
    blocks = -(-(case["context"] + 1) // 64)
    order = torch.randperm(case["batch"] * blocks, generator=torch.Generator().manual_seed(5)).to(torch.int32)
    cache = PagedKVCache(1, case["batch"], case["hkv"], case["d"], case["context"] + 1, dtype=torch.float16, device=DEV, page_order=order)
    cache.fill(0, k, v, lens)
    cache.seq_lens.add_(1)  # the layers after the first find the token counted
    pos = torch.tensor(lens, dtype=torch.int64, device=DEV)
    return {"kind": "layer", "hq": case["hq"], "qkv": qkv, "norms": norms, "cache": cache, "pos": pos, "longest": case["context"] + 1}


def _prepare_prompt(case, seed):
    if case["kind"] != "prompt":
        return _prepare_model_prompt(case, seed)
    return {"kind": "prompt", "args": (*_prompt_tensors(case, seed), case["causal"])}


def _tower_cache(case, seed, layer):
    cfg = TextTowerConfig()
    shape = (case["batch"], case["context"], cfg.n_kv_heads, cfg.head_dim)
    return [normal(shape, torch.float16, seed, name, layer) for name in ("k", "v")]


def _prepare_tower(case, seed):
    cfg, lens = TextTowerConfig(), lengths(case)
    tower = TextTower(cfg, case["batch"], case["context"] + 64, device=DEV)
    tower.embed.copy_(normal(tower.embed.shape, torch.float16, seed, "embed") * 0.1)
    tower.final_ln.copy_(1 + 0.02 * normal(tower.final_ln.shape, torch.float16, seed, "final"))
    for i, layer in enumerate(tower.layers):
        for name, t in layer.items():
            t.copy_(tower_weight(name, t.shape, seed, i))
        tower.cache.fill(i, *_tower_cache(case, seed, i), lens)
    ids = some_ids(case["batch"], cfg.vocab, seed, "ids")
    tower.set_state(ids, lens)
    start = [t.clone() for t in (tower.token_ids, tower.pos3, tower.cache.seq_lens)]

    def step():  # from a kept point: the step itself moves on by a token
        for t, saved in zip((tower.token_ids, tower.pos3, tower.cache.seq_lens), start):
            t.copy_(saved)
        tower.decode_step()
        return tower.last_logits

    graph = CUDAGraph().capture(step)
    return {"kind": "tower", "graph": graph, "tower": tower, "start": start, "outputs": [graph.output, tower.token_ids, *tower.cache.k_pages[:4], *tower.cache.v_pages[:4]]}


def _cached_input(case, seed, layer, b, n):
    """What the projection gave for the tokens that a sequence has in a layer's cache: latents or raw keys."""
    m = model_config(case)["layers"][layer]["mixer"]
    cols = m["kv_heads"] * m["dim"] if "kv_heads" in m else m["kv_rank"] + m.get("rot_dim", 0)
    return normal((n, cols), torch.bfloat16, seed, "cached", layer, b)


def _states(case, seed, layer):
    """Matrices and convolution inputs (slot p % 4 holds position p) that the sequences have in a recurrent layer."""
    m, b = model_config(case)["layers"][layer]["mixer"], case["batch"]
    channels = 2 * m["kv_heads"] * m["dim"] + m["heads"] * m["vdim"]
    return (0.3 * normal((b, m["heads"], m["dim"], m["vdim"]), torch.float32, seed, "state", layer),
            normal((b, m["conv"], channels), torch.bfloat16, seed, "ring", layer))


def _prepare_decode(case, seed):
    cfg, w = model_weights(case, seed)
    model = models.create(cfg, w, torch.bfloat16)
    lens, b = lengths(case), case["batch"]
    runner = ModelRunner(model, b * (case["context"] + 64), max_seqs=b, max_seq_len=case["context"] + 64, shuffle_pages=1)
    held = Held(runner)
    seqs = [runner.open() for _ in range(b)]
    for s, n in zip(seqs, lens):
        runner.lengths[s] = n
        runner.arena.reserve(s, n + 1)
    runner.arena.sync()
    at, state_at = 0, 0
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}.mix."
        if layer["type"] == "delta":
            for pool, values in zip(runner.states[state_at], _states(case, seed, i)):
                pool[torch.tensor(seqs, device=DEV)] = values
            state_at += 1
            continue
        pool = runner.pages[at]
        at += 1
        for s, n in zip(seqs, lens):
            x = _cached_input(case, seed, i, s, n)
            rows = Rows(torch.full((n,), s, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV),
                        runner.block_table, n, n)
            if layer["type"] == "attention":
                q = torch.zeros((n, m["heads"] * m["dim"]), dtype=torch.bfloat16, device=DEV)
                ops.shared_kv_prepare(q, w[p + "q.norm"], x, w[p + "k.norm"], pool, rows,
                                      m["heads"], m["kv_heads"], m["dim"], LM_EPS)
            else:
                rot = m.get("rot_dim", 0)
                freq = torch.tensor([10000.0 ** (-2 * j / max(1, rot)) for j in range(rot // 2)], dtype=torch.float64, device=DEV)
                ops.latent_prepare(rows, freq, rot, dkv=x, dkv_weight=w[p + "dkv.norm"], pages=pool, eps=LM_EPS)
    ids = some_ids(b, VOCAB, seed, "ids")
    rows = Rows(torch.tensor(seqs, dtype=torch.int32, device=DEV), torch.tensor(lens, dtype=torch.int32, device=DEV),
                runner.block_table, max(lens) + 1, b, singles=b)
    held.inputs = ids, rows
    saved = runner.copy_state(seqs)
    held.graph = CUDAGraph().capture(lambda: model.forward(ids, rows, runner.cache, None))  # runs once before it records
    runner.put_state(saved)
    held.views = cache_views(runner, cfg)
    return {"kind": "decode", "held": held}


def _prepare_model_prompt(case, seed):
    cfg, w = model_weights(case, seed)
    runner = ModelRunner(models.create(cfg, w, torch.bfloat16), case["tokens"] + 64, max_seqs=1)
    held = Held(runner)
    held.views = cache_views(runner, cfg)
    prompt = some_ids(case["tokens"], VOCAB, seed, "prompt").tolist()
    return {"kind": "model_prompt", "held": held, "prompt": prompt, "portion": case["portion"]}


def scored(n):
    """The places of a prompt whose logits are asked for: its last 32, as a program does that rates an answer's tokens."""
    return list(range(max(0, n - 32), n))


# ---- run --------------------------------------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "token":
        return ops.gqa_decode_attention(*state["args"])
    if kind == "layer":
        cache = state["cache"]
        k_pages, v_pages, table, lens = cache.get(0)
        out = ops.qkv_decode_step_paged(state["qkv"], state["hq"], *state["norms"], EPS, k_pages, v_pages, table, lens, state["longest"],
                                        pos=state["pos"], theta=THETA, advance=False, slot_delta=-1)
        return out, k_pages, v_pages
    if kind == "prompt":
        return ops.scaled_dot_product_attention(*state["args"])
    if kind == "tower":
        state["graph"].replay_async()
        return state["outputs"]
    held = state["held"]
    if kind == "decode":
        held.graph.replay_async()
        return held.outputs(held.graph.output)
    prompt, portion, logits = state["prompt"], state["portion"], []
    n, wanted = len(prompt), scored(len(prompt))
    seq = held.runner.open()
    for at in range(0, n, portion):
        part = prompt[at:at + portion]
        want = [p - at for p in wanted if at <= p < at + len(part)]
        got = held.runner.step([(seq, part, want)])
        if want:
            logits.append(got)
    held.runner.close(seq)
    return held.outputs(logits[0] if len(logits) == 1 else torch.cat(logits))


# ---- work and tolerance -----------------------------------------------------------------------------------------------------

def _model_work(case, rows, keys, head_rows, cached):
    """Bytes and flops of one step: rows new tokens, `keys(window)` pairs of row and visible key, `cached(window)` cached
    tokens that are read, head_rows rows of logits."""
    cfg = model_config(case)
    width = cfg["width"]
    weights, flops, other = VOCAB * width, 2 * head_rows * VOCAB * width, 0
    for layer in cfg["layers"]:
        m = layer["mixer"]
        window = m["mask"]["size"] if "mask" in m else 0
        if layer["type"] == "delta":
            channels = 2 * m["kv_heads"] * m["dim"] + m["heads"] * m["vdim"]
            n = width * (channels + 2 * m["heads"] * m["vdim"] + 2 * m["heads"])
            flops += 8 * rows * m["heads"] * m["dim"] * m["vdim"]
            other += 2 * 4 * m["heads"] * m["dim"] * m["vdim"] * case.get("batch", 1)
        elif layer["type"] == "attention":
            n = width * m["dim"] * (2 * m["heads"] + m["kv_heads"])
            flops += 4 * m["heads"] * m["dim"] * keys(window)
            other += 2 * m["kv_heads"] * m["dim"] * cached(window)
        else:
            dim, rot, vdim, rank, h = m["dim"], m.get("rot_dim", 0), m["vdim"], m["kv_rank"], m["heads"]
            q = m.get("q_rank")
            n = q * (width + h * (dim + rot)) if q else width * h * (dim + rot)
            n += width * (rank + rot) + h * (dim + vdim) * rank + width * h * vdim
            # per pair: through the cached latents, or expanded keys and values (whose making is counted in n, once per token)
            per = 2 * rank + rot if case["kind"].endswith("decode") else dim + rot + vdim
            flops += 2 * h * per * keys(window)
            other += 2 * (rank + rot) * cached(window)
        weights += n
        flops += 2 * rows * n
        mlp = layer["mlp"]
        if mlp["kind"] == "dense":
            weights += 3 * width * mlp["ff"]
            flops += 6 * rows * width * mlp["ff"]
        else:
            r, ff, sff = mlp["router"], mlp["expert"]["ff"], mlp["shared"]["ff"]
            used = r["experts"] * (1 - (1 - r["top"] / r["experts"]) ** rows)
            weights += 3 * width * (ff * used + sff) + r["experts"] * width
            flops += 6 * rows * width * (ff * r["top"] + sff) + 2 * rows * r["experts"] * width
    return {"bytes": 2 * weights + other + 4 * head_rows * VOCAB, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind in ("token", "layer", "prompt"):
        hq, hkv, d = case["hq"], case["hkv"], case["d"]
        e = 4 if case.get("dtype") == "f32" else 2
        if kind == "prompt":
            n = case["tokens"]
            pairs = n * (n + 1) / 2 if case["causal"] else n * n
            return {"bytes": 2 * n * (hq + hkv) * d * e, "flops": 4 * hq * d * pairs}
        keys, rows = (case["keys"], 1) if kind == "token" else (sum(lengths(case)) + case["batch"], case["batch"])
        extra = 4 * rows * hkv if kind == "layer" else 0  # new keys and values: read from the projection, written to the cache
        return {"bytes": (2 * keys * hkv + 2 * rows * hq + extra) * d * e, "flops": 4 * hq * d * keys}
    if kind == "tower":
        c, keys, b = TextTowerConfig(), sum(lengths(case)) + case["batch"], case["batch"]
        per = c.hidden * c.head_dim * (2 * c.n_q_heads + 2 * c.n_kv_heads) + 3 * c.hidden * c.intermediate
        weights = c.n_layers * per + c.vocab * c.hidden
        return {"bytes": 2 * weights + 4 * c.n_layers * keys * c.n_kv_heads * c.head_dim + 2 * b * c.vocab,
                "flops": 2 * b * weights + 4 * c.n_layers * c.n_q_heads * c.head_dim * keys}
    if kind.endswith("decode"):
        def visible(window):
            return sum(min(n + 1, window) if window else n + 1 for n in lengths(case))

        return _model_work(case, case["batch"], visible, case["batch"], visible)
    n = case["tokens"]

    def pairs(window):
        w = min(window or n, n)
        return w * (w + 1) / 2 + (n - w) * w

    return _model_work(case, n, pairs, min(n, 32), lambda window: n)


def tolerance(case):
    kind = case["kind"]
    if kind in ("token", "prompt") and case["dtype"] == "f32":
        return {"rel": 2e-6, "max": 2e-5}  # 32-bit sums in another order
    if kind in ("token", "layer", "prompt"):
        return {"rel": 2e-3, "max": 2e-2}  # rounding of weights and results to half precision
    return {"rel": 2e-2, "max": 0.9, "differ": 0.01}  # sixteen-bit activations through the layers; a near tie among experts or tokens may fall the other way


# ---- exact ------------------------------------------------------------------------------------------------------------------

def exact(case, seed):
    with torch.no_grad():
        return globals()["_exact_" + case["kind"]](case, seed)


def _softmax_attention(q, k, v, scale, causal=False, window=0, sink=None):
    """One head: q (n, d), k and v (m, .); rows are the last n of the m positions when causal."""
    n, m = q.shape[0], k.shape[0]
    s = (q @ k.T) * scale
    if causal:
        i = torch.arange(m - n, m, device=DEV)[:, None]
        j = torch.arange(m, device=DEV)[None, :]
        hidden = j > i
        if window:
            hidden |= j <= i - window
        s = s.masked_fill_(hidden, -math.inf)
    top = s.amax(-1, keepdim=True)
    if sink is not None:
        top = torch.clamp(top, min=float(sink))
    e = torch.exp(s - top)
    total = e.sum(-1, keepdim=True)
    if sink is not None:
        total = total + torch.exp(sink - top)
    return (e / total) @ v


def _exact_token(case, seed):
    q, k, v = (t.double() for t in _prepare_token(case, seed)["args"])
    group = case["hq"] // case["hkv"]
    out = [_softmax_attention(q[:, h], k[:, h // group], v[:, h // group], case["d"] ** -0.5) for h in range(case["hq"])]
    return torch.stack(out, 1)


def _exact_prompt(case, seed):
    q, k, v = _prompt_tensors(case, seed)
    group, out = case["hq"] // case["hkv"], torch.empty(q.shape, dtype=torch.float64, device=DEV)
    for h in range(case["hq"]):
        out[:, h] = _softmax_attention(q[:, h].double(), k[:, h // group].double(), v[:, h // group].double(), case["d"] ** -0.5, case["causal"])
    return out


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate_halves(x, pos, theta):
    """x (rows, heads, d): pairs (i, i + d/2) turned by pos * theta^(-2i/d)."""
    half = x.shape[-1] // 2
    a = pos.double()[:, None, None] * theta ** (-torch.arange(half, device=DEV, dtype=torch.float64) / half)
    lo, hi = x[..., :half], x[..., half:]
    return torch.cat([lo * torch.cos(a) - hi * torch.sin(a), hi * torch.cos(a) + lo * torch.sin(a)], -1)


def _attend_cache(q, k_new, v_new, k, v, lens):
    """q (rows, hq, d) over each row's first lens[b] cached keys and its new one."""
    group, scale, out = q.shape[1] // k_new.shape[1], q.shape[2] ** -0.5, torch.empty_like(q)
    for b, n in enumerate(lens):
        kb = torch.cat([k[b, :n].double(), k_new[b:b + 1]])
        vb = torch.cat([v[b, :n].double(), v_new[b:b + 1]])
        qb = q[b].view(-1, group, q.shape[2])
        s = torch.einsum("hgd,nhd->hgn", qb, kb) * scale
        out[b] = torch.einsum("hgn,nhd->hgd", torch.softmax(s, -1), vb).reshape(q.shape[1], -1)
    return out


def _qkv_attention(qkv, norms, hq, hkv, d, lens, k, v):
    qkv = qkv.view(qkv.shape[0], hq + 2 * hkv, d)
    pos = torch.tensor(lens, device=DEV)
    q = _rotate_halves(_rms(qkv[:, :hq], EPS) * norms[0].double(), pos, THETA)
    k_new = _rotate_halves(_rms(qkv[:, hq:hq + hkv], EPS) * norms[1].double(), pos, THETA)
    return _attend_cache(q, k_new, qkv[:, hq + hkv:], k, v, lens)


def _exact_layer(case, seed):
    qkv, norms, (k, v) = _layer_tensors(case, seed)
    return _qkv_attention(qkv.double(), norms, case["hq"], case["hkv"], case["d"], lengths(case), k, v), None, None


def _exact_tower(case, seed):
    c, lens = TextTowerConfig(), lengths(case)
    q, kv, d = c.n_q_heads, c.n_kv_heads, c.head_dim
    shapes = {"input_ln": (c.hidden,), "post_ln": (c.hidden,), "q_norm": (d,), "k_norm": (d,), "qkv": ((q + 2 * kv) * d, c.hidden),
              "o": (c.hidden, q * d), "gate_up": (2 * c.intermediate, c.hidden), "down": (c.hidden, c.intermediate)}
    embed = normal((c.vocab, c.hidden), torch.float16, seed, "embed") * 0.1
    final = 1 + 0.02 * normal((c.hidden,), torch.float16, seed, "final")
    x = embed[some_ids(case["batch"], c.vocab, seed, "ids")].double()
    for i in range(c.n_layers):
        w = {name: tower_weight(name, shape, seed, i).double() for name, shape in shapes.items()}
        qkv = (_rms(x, c.eps) * w["input_ln"]) @ w["qkv"].T
        a = _qkv_attention(qkv, (w["q_norm"], w["k_norm"]), q, kv, d, lens, *_tower_cache(case, seed, i))
        x = x + a.reshape(case["batch"], -1) @ w["o"].T
        gate, up = ((_rms(x, c.eps) * w["post_ln"]) @ w["gate_up"].T).chunk(2, -1)
        x = x + (gate * torch.sigmoid(gate) * up) @ w["down"].T
    logits = torch.cat([(_rms(x, c.eps) * final.double()) @ part.double().T for part in embed.split(16384)], -1)
    return [logits, None] + [None] * 8


def _rotate_pairs(x, pos, base):
    """x (rows, ..., n): pairs (2i, 2i + 1) turned by pos * base^(-2i/n)."""
    n = x.shape[-1]
    a = pos.double()[:, None] * base ** (-2.0 * torch.arange(n // 2, device=DEV, dtype=torch.float64) / n)
    a = a.view(a.shape[0], *([1] * (x.dim() - 2)), n // 2)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * torch.cos(a) - v * torch.sin(a), v * torch.cos(a) + u * torch.sin(a)], -1).flatten(-2)


def _latents(w, p, m, down, pos):
    """Normed latent and rotated key part of the rows `down`."""
    rank = m["kv_rank"]
    c = _rms(down[:, :rank], LM_EPS) * w[p + "dkv.norm"].double()
    return c, _rotate_pairs(down[:, rank:], pos, 10000.0) if "rot_dim" in m else down[:, rank:]


def _latent_rows(w, p, m, q, keys_of):
    """Attention through the latents: q (rows, heads, dim + rot) each over what keys_of gives; -> (rows, heads * vdim)."""
    h, dim, vdim, rank = m["heads"], m["dim"], m["vdim"], m["kv_rank"]
    uk, uv = w[p + "uk"].double().view(h, dim, rank), w[p + "uv"].double().view(h, vdim, rank)
    q_lat, q_rot = torch.einsum("rhd,hdk->rhk", q[..., :dim], uk), q[..., dim:]
    sink = w[p + "sink"].double() if "mask" in m else None
    out = []
    for b in range(q.shape[0]):
        c, kr = keys_of(b)
        s = (q_lat[b] @ c.T + q_rot[b] @ kr.T) * m["scale"]
        if sink is not None:
            s = torch.cat([s, sink[:, None]], -1)
        a = torch.softmax(s, -1)[:, :c.shape[0]]
        out.append(torch.einsum("hk,hvk->hv", a @ c, uv).reshape(-1))
    return torch.stack(out)


def _queries(w, p, m, h, pos):
    if "q_rank" in m:
        q = (_rms(h @ w[p + "dq"].double().T, LM_EPS) * w[p + "dq.norm"].double()) @ w[p + "uq"].double().T
    else:
        q = h @ w[p + "q"].double().T
    q = q.view(h.shape[0], m["heads"], -1)
    return torch.cat([q[..., :m["dim"]], _rotate_pairs(q[..., m["dim"]:], pos, 10000.0)], -1) if "rot_dim" in m else q


def _layer_norm(x, w):
    c = x - x.mean(-1, keepdim=True)
    return c / torch.sqrt((c * c).mean(-1, keepdim=True) + LM_EPS) * w.double()


def _mixture(w, p, h, mlp):
    r = mlp["router"]
    n, groups = r["experts"], r["groups"]["count"]
    s = torch.sigmoid(h @ w[p + "router"].double().T)
    choice = s + w[p + "correction"].double()
    per_group = choice.view(-1, groups, n // groups).topk(2, -1).values.sum(-1)
    open_ = torch.zeros_like(per_group).scatter_(1, per_group.topk(r["groups"]["keep"], -1).indices, 1.0)
    closed = open_.repeat_interleave(n // groups, -1) == 0
    ids = choice.masked_fill(closed, -math.inf).topk(r["top"], -1).indices

    def expert(name, x, limit):
        g = torch.clamp(x @ w[f"{p}{name}.gate"].double().T, max=limit)
        u = torch.clamp(x @ w[f"{p}{name}.up"].double().T, min=-limit, max=limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[f"{p}{name}.down"].double().T

    y = expert("shared", h, mlp["shared"]["limit"])
    for e in range(n):
        rows = (ids == e).any(-1).nonzero()[:, 0]
        if rows.numel():
            y[rows] += r["scale"] * s[rows, e][:, None] * expert(f"e{e}", h[rows], mlp["expert"]["limit"])
    return y


def _expanded(w, p, m, q, c, kr):
    """Causal attention of a whole prompt, head by head."""
    h, dim, vdim, rank = m["heads"], m["dim"], m["vdim"], m["kv_rank"]
    uk, uv = w[p + "uk"].double().view(h, dim, rank), w[p + "uv"].double().view(h, vdim, rank)
    sink = w[p + "sink"].double() if "mask" in m else [None] * h
    return torch.cat([_softmax_attention(q[:, i], torch.cat([c @ uk[i].T, kr], -1), c @ uv[i].T, m["scale"], True,
                                         m["mask"]["size"] if "mask" in m else 0, sink[i]) for i in range(h)], -1)


def _no_cache(cfg):
    """The cache and state among the outputs, which have no value here."""
    count = {"delta": 2, "attention": 2}
    return [None] * sum(count.get(layer["type"], 1) for layer in cfg["layers"])


def _nuderax(case, seed, ids, attend):
    """attend(w, i, layer, h): output of layer i's attention, before its last product."""
    cfg, w = model_weights(case, seed)
    x = _layer_norm(w["embed"][ids].double(), w["embed.norm"])
    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}."
        h = _layer_norm(x, w[p + "norm1"])
        y = attend(w, i, layer, h) @ w[p + "mix.o"].double().T
        x = x + y + _mixture(w, p + "mlp.", _layer_norm(x, w[p + "norm2"]), layer["mlp"])
    return cfg, w, x


def _latent_decode(case, seed, lens, pos):
    def attend(w, i, layer, h):
        m, p = layer["mixer"], f"l{i}.mix."
        c_new, kr_new = _latents(w, p, m, h @ w[p + "dkv"].double().T, pos)
        window = m["mask"]["size"] if "mask" in m else 0

        def keys_of(b):
            n = lens[b]
            c, kr = _latents(w, p, m, _cached_input(case, seed, i, b, n).double(), torch.arange(n, device=DEV))
            c, kr = torch.cat([c, c_new[b:b + 1]]), torch.cat([kr, kr_new[b:b + 1]])
            return (c[-window:], kr[-window:]) if window else (c, kr)

        return _latent_rows(w, p, m, _queries(w, p, m, h, pos), keys_of)

    return attend


def _exact_nuderax_decode(case, seed):
    lens = lengths(case)
    pos = torch.tensor(lens, device=DEV)
    cfg, w, x = _nuderax(case, seed, some_ids(case["batch"], VOCAB, seed, "ids"), _latent_decode(case, seed, lens, pos))
    return [_layer_norm(x, w["final.norm"]) @ w["embed"].double().T, *_no_cache(cfg)]


def _latent_prompt(pos):
    def attend(w, i, layer, h):
        m, p = layer["mixer"], f"l{i}.mix."
        return _expanded(w, p, m, _queries(w, p, m, h, pos), *_latents(w, p, m, h @ w[p + "dkv"].double().T, pos))

    return attend


def _exact_nuderax_prompt(case, seed):
    pos = torch.arange(case["tokens"], device=DEV)
    cfg, w, x = _nuderax(case, seed, some_ids(case["tokens"], VOCAB, seed, "prompt"), _latent_prompt(pos))
    return [_layer_norm(x[scored(case["tokens"])], w["final.norm"]) @ w["embed"].double().T, *_no_cache(cfg)]


def _delta_inputs(w, p, m, h, before):
    """Unit queries and keys, values, decays, steps and gates of the rows h; before(channels) gives conv - 1 earlier inputs of
    each row's sequence, (rows, conv - 1, channels), or None where the rows are one sequence from its start."""
    n, groups, heads, dim, vdim, taps = h.shape[0], m["kv_heads"], m["heads"], m["dim"], m["vdim"], m["conv"]
    x = torch.cat([h @ w[p + name].double().T for name in "qkv"], -1)
    conv = torch.cat([w[p + f"{name}.conv"].double() for name in "qkv"])
    if before is None:
        padded = torch.cat([x.new_zeros((taps - 1, x.shape[1])), x])
        x = sum(conv[:, j] * padded[j:j + n] for j in range(taps))
    else:
        x = conv[:, -1] * x + sum(conv[:, j] * before[:, j] for j in range(taps - 1))
    x = x * torch.sigmoid(x)
    q, k, v = x.split([groups * dim, groups * dim, heads * vdim], -1)

    def unit(t):
        t = t.reshape(n, groups, dim)
        return (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(heads // groups, 1)

    beta = torch.sigmoid(h @ w[p + "b"].double().T)
    z = h @ w[p + "a"].double().T + w[p + "dt_bias"].double()
    decay = torch.exp(-torch.exp(w[p + "A_log"].double()) * torch.nn.functional.softplus(z, threshold=50.0))
    gate = h @ w[p + "g"].double().T
    return unit(q) * dim ** -0.5, unit(k), v.reshape(n, heads, vdim), decay, beta, gate * torch.sigmoid(gate)


def _delta_out(w, p, m, o, gate):
    o = _rms(o, LM_EPS) * w[p + "norm"].double()
    return o.reshape(o.shape[0], -1) * gate


def _exact_rigozen(case, seed, ids, mixers, rows=None):
    cfg, w = model_weights(case, seed)
    x = w["embed"][ids].double()

    def post(x, y, name):
        return x + _rms(y, LM_EPS) * (1 + w[name].double())

    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}."
        x = post(x, mixers[layer["type"]](w, i, layer, x) @ w[p + "mix.o"].double().T, p + "norm1")
        g, u = x @ w[p + "mlp.gate"].double().T, x @ w[p + "mlp.up"].double().T
        x = post(x, (g * torch.sigmoid(g) * u) @ w[p + "mlp.down"].double().T, p + "norm2")
    x = x if rows is None else x[rows]
    return (_rms(x, LM_EPS) * (1 + w["final.norm"].double())) @ w["embed"].double().T, _no_cache(cfg)


def _raw_key_inputs(w, p, m, h):
    q = _rms(h @ w[p + "q"].double().T, LM_EPS) * w[p + "q.norm"].double()
    return q.view(h.shape[0], m["heads"], m["dim"]), h @ w[p + "k"].double().T


def _raw_keys(w, p, m, raw):
    k = _rms(raw, LM_EPS) * w[p + "k.norm"].double()
    return k.view(-1, m["kv_heads"], m["dim"]), raw.view(-1, m["kv_heads"], m["dim"])


def _exact_rigozen_decode(case, seed):
    lens = lengths(case)
    pos = torch.tensor(lens, device=DEV)
    states = {}

    def delta(w, i, layer, h):
        m, p = layer["mixer"], f"l{i}.mix."
        state, ring = (t.double() for t in _states(case, seed, i))
        slots = (pos[:, None] + torch.arange(1 - m["conv"], 0, device=DEV)) % m["conv"]
        before = torch.gather(ring, 1, slots[:, :, None].expand(-1, -1, ring.shape[2]))
        q, k, v, decay, beta, gate = _delta_inputs(w, p, m, h, before)
        state = state * decay[..., None, None]
        u = beta[..., None] * (v - torch.einsum("bhdv,bhd->bhv", state, k))
        state = state + k[..., None] * u[..., None, :]
        states[i] = state
        return _delta_out(w, p, m, torch.einsum("bhdv,bhd->bhv", state, q), gate)

    def attention(w, i, layer, h):
        m, p = layer["mixer"], f"l{i}.mix."
        q, raw = _raw_key_inputs(w, p, m, h)
        out = []
        for b, n in enumerate(lens):
            k, v = _raw_keys(w, p, m, torch.cat([_cached_input(case, seed, i, b, n).double(), raw[b:b + 1]])[-m["mask"]["size"]:])
            s = torch.einsum("hgd,nhd->hgn", q[b].view(m["kv_heads"], -1, m["dim"]), k) * m["scale"]
            out.append(torch.einsum("hgn,nhd->hgd", torch.softmax(s, -1), v).reshape(-1))
        return torch.stack(out)

    mixers = {"delta": delta, "latent_attention": _latent_decode(case, seed, lens, pos), "attention": attention}
    logits, rest = _exact_rigozen(case, seed, some_ids(case["batch"], VOCAB, seed, "ids"), mixers)
    order = [t for i in sorted(states) for t in (states[i], None)]
    return [logits, *rest[:len(rest) - len(order)], *order]


def _exact_rigozen_prompt(case, seed):
    pos, states = torch.arange(case["tokens"], device=DEV), {}

    def delta(w, i, layer, h):
        m, p = layer["mixer"], f"l{i}.mix."
        q, k, v, decay, beta, gate = _delta_inputs(w, p, m, h, None)
        state = torch.zeros((m["heads"], m["dim"], m["vdim"]), dtype=torch.float64, device=DEV)
        out = torch.empty_like(v)
        for t in range(h.shape[0]):
            state = state * decay[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], state)[:, 0])
            state = torch.baddbmm(state, k[t][..., None], u[:, None])
            out[t] = torch.bmm(q[t][:, None], state)[:, 0]
        states[i] = state[None]
        return _delta_out(w, p, m, out, gate)

    def attention(w, i, layer, h):
        m, p = layer["mixer"], f"l{i}.mix."
        q, raw = _raw_key_inputs(w, p, m, h)
        k, v = _raw_keys(w, p, m, raw)
        group = m["heads"] // m["kv_heads"]
        return torch.cat([_softmax_attention(q[:, j], k[:, j // group], v[:, j // group], m["scale"], True, m["mask"]["size"])
                          for j in range(m["heads"])], -1)

    mixers = {"delta": delta, "latent_attention": _latent_prompt(pos), "attention": attention}
    logits, rest = _exact_rigozen(case, seed, some_ids(case["tokens"], VOCAB, seed, "prompt"), mixers, scored(case["tokens"]))
    order = [t for i in sorted(states) for t in (states[i], None)]
    return [logits, *rest[:len(rest) - len(order)], *order]
