"""The work whose speed this repository answers for: calls through its public entry points at the sizes its configurations,
tests and benchmark use.

``listed()`` are the cases themselves, ``draw`` gives more of the same ranges, ``prepare`` makes what a program has in hand before
the call, ``run`` is one call, ``exact`` the same outputs in float64 torch without this package, ``work`` what the call cannot do
without, ``tolerance`` how far another correct implementation at the same precision may be.

Two families.  The fixed-batch Llama path: a whole decode step of a small model, the decode attention of an 8B shape, the same
over a long shared prefix, and the prefill -> decode hand-off of a sequence's pages.  The ragged model classes: their sequence
mixers and routed experts as modules, over packed steps of prompt portions or of one token per sequence, and the step engine
with a whole model.  ``width`` fixes the head layout as in the benchmark's model sizes: width / 128 query heads of 128, a quarter
as many key/value heads, width / 128 recurrent heads of 64 x 128.
"""
import math

import torch

import dgi_b200  # noqa: F401
from dgi_b200 import ops
from dgi_b200.fibirax_layer import ParallelMixer
from dgi_b200.paged_layer import PagedBatchState, PagedLayerKV, RaggedBatchState, RaggedLayerCache
from dgi_b200.petipel_layer import (BiasedPagedAttention, GatedLinearRecurrence, PetipelConfig, SigmoidTopKMoE, build_shards,
                                    random_checkpoint)
from dgi_b200.ragged_engine import RaggedStepEngine
from dgi_b200.sanesun_layer import ChannelDeltaMixer
from dgi_b200.testing import LlamaShapeConfig, build_product_shards
from dgi_b200.vatazen_layer import LatentRotaryAttention
from dgi_b200.worker.distributed.kv_cache import KVCachePool

DEV = "cuda:0"
F64 = torch.float64
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
PAGE = 16
EPS = 1e-6
MIXERS = ("petipel_attention", "petipel_recurrence", "sanesun_delta", "latent_attention", "fibirax_mixer")


def listed():
    return [
        # the smallest call: one decode step of the 4-layer model of the CPU comparison, through ModelShard.forward
        dict(name="llama_small_step", kind="llama_step", layers=4, width=512, heads=8, kv_heads=2, ff=1408, vocab=1024, batch=4,
             context=160, dtype="bf16"),
        # one layer's attention in a decode step of the headline workload: 8B shape, 64 sequences at 2k
        dict(name="llama_decode_attention", kind="decode_attention", heads=32, kv_heads=8, dim=128, batch=64, context=2048, prefix=0,
             ragged=False, dtype="bf16"),
        # long-context serving: 8 sequences at 32k, three quarters of it one shared prefix
        dict(name="llama_shared_prefix", kind="decode_attention", heads=32, kv_heads=8, dim=128, batch=8, context=32768,
             prefix=24576, ragged=True, dtype="bf16"),
        # a 4k prompt leaves a prefill GPU and arrives on a decode GPU: gather of its pages, scatter into other pages
        dict(name="kv_handoff", kind="kv_handoff", layers=32, kv_heads=8, dim=128, tokens=4096, dtype="bf16"),
        # Petipel's two mixers over prompts, and its attention over one decoded token per sequence at uneven contexts
        dict(name="petipel_attention_prompt", kind="petipel_attention", width=2048, seqs=8, tokens=2048, past=0, ragged=False,
             dtype="bf16"),
        dict(name="petipel_attention_decode", kind="petipel_attention", width=2048, seqs=48, tokens=1, past=3000, ragged=True,
             dtype="fp16"),
        dict(name="petipel_recurrence_prompt", kind="petipel_recurrence", width=2048, seqs=6, tokens=1900, past=0, ragged=True,
             dtype="bf16"),
        # routed experts of a prompt step of odd length
        dict(name="petipel_experts", kind="petipel_experts", width=1024, tokens=4099, dtype="bf16"),
        # Sanesun's delta rule behind its short convolutions, prompts
        dict(name="sanesun_delta_prompt", kind="sanesun_delta", width=1024, seqs=8, tokens=2048, past=0, ragged=False,
             dtype="bf16"),
        # the latent attention that Vatazen and Zuderax layers run, prompt portions behind cached tokens
        dict(name="latent_prompt", kind="latent_attention", width=2048, seqs=4, tokens=1500, past=700, ragged=True, dtype="bf16"),
        # Fibirax: windowed attention beside retention, medium prompts
        dict(name="fibirax_mixer_prompt", kind="fibirax_mixer", width=2048, seqs=5, tokens=1024, past=0, ragged=True, dtype="bf16"),
        # a whole model on the step engine: uneven prompts admitted, run in one step, finished
        dict(name="petipel_engine_step", kind="engine_step", width=1024, seqs=6, tokens=700, dtype="bf16"),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    kind = rng.choice(("llama_step", "decode_attention", "decode_attention", "kv_handoff", "petipel_experts", "engine_step") + MIXERS * 2)
    if kind == "llama_step":
        kv = rng.choice((1, 2, 4))
        return dict(kind=kind, layers=rng.choice((1, 2, 4)), width=256 * kv, heads=4 * kv, kv_heads=kv, ff=rng.choice((704, 1408)),
                    vocab=1024, batch=_spread(rng, 1, 32), context=_spread(rng, 20, 1500), dtype=dtype)
    if kind == "decode_attention":
        kv, batch = rng.choice((1, 2, 8)), _spread(rng, 1, 64)
        context = _spread(rng, 30, max(64, min(32768, 131072 * 8 // (kv * batch))))
        prefix = rng.choice((0, context * 3 // 4 // PAGE * PAGE)) if batch > 1 else 0
        return dict(kind=kind, heads=4 * kv, kv_heads=kv, dim=rng.choice((64, 128)), batch=batch, context=context, prefix=prefix,
                    ragged=rng.random() < 0.7, dtype=dtype)
    if kind == "kv_handoff":
        return dict(kind=kind, layers=rng.choice((1, 8, 16, 32)), kv_heads=rng.choice((2, 8)), dim=rng.choice((64, 128)),
                    tokens=_spread(rng, 20, 4096), dtype=dtype)
    if kind == "engine_step":
        return dict(kind=kind, width=rng.choice((512, 1024)), seqs=rng.randint(1, 8), tokens=_spread(rng, 5, 700), dtype=dtype)
    width = rng.choice((512, 1024, 2048))
    if kind == "petipel_experts":
        return dict(kind=kind, width=width, tokens=_spread(rng, 1, 6000), dtype=dtype)
    if rng.random() < 0.35:     # one decoded token per sequence
        return dict(kind=kind, width=width, seqs=_spread(rng, 1, 64), tokens=1, past=_spread(rng, 10, 4000), ragged=True, dtype=dtype)
    seqs = rng.randint(1, 8)
    return dict(kind=kind, width=width, seqs=seqs, tokens=_spread(rng, 8, 2048), past=rng.choice((0, 0, _spread(rng, 5, 1500))),
                ragged=rng.random() < 0.7, dtype=dtype)


def tolerance(case):
    """About four times the distance from ``exact`` that was measured: 16-bit roundings of projections and activations."""
    kind, half = case["kind"], case["dtype"] == "fp16"
    if kind == "kv_handoff":
        return "exact"
    if kind == "llama_step":        # four layers in the storage dtype, the residual among it (0.008 in bf16)
        return {"rel": 0.004 if half else 0.034}
    if kind == "decode_attention":  # 0.0032
        return {"rel": 0.0016 if half else 0.013}
    if kind in ("latent_attention", "fibirax_mixer"):   # 0.0073
        return {"rel": 0.0036 if half else 0.03}
    return {"rel": 0.002 if half else 0.016}            # 0.004, also through four layers with an fp32 residual


# ---- inputs: plain tensors made from the seed ---------------------------------------------------------------------------


class _Draw:
    """Random tensors on the device from one seeded generator."""

    def __init__(self, seed, dtype):
        self.gen = torch.Generator(device=DEV).manual_seed(seed)
        self.dtype = dtype

    def normal(self, *shape, s=1.0, mean=0.0, dtype=None):
        return (torch.randn(*shape, generator=self.gen, device=DEV) * s + mean).to(dtype or self.dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=None):
        return (torch.rand(*shape, generator=self.gen, device=DEV) * (hi - lo) + lo).to(dtype or self.dtype)

    def lin(self, out, inp, gain=1.0):
        return self.normal(out, inp, s=gain / math.sqrt(inp))

    def perm(self, n):
        return torch.randperm(n, generator=self.gen, device=DEV)


def _portions(case):
    """(new tokens, tokens before) per sequence; uneven when the case says so."""
    out = []
    for i in range(case["seqs"]):
        cut = (0.618 * (i + 1)) % 1.0 * 0.7 if case.get("ragged") else 0.0
        new = max(1, int(case["tokens"] * (1.0 - cut)))
        past = case.get("past", 0)
        out.append((new, int(past * (1.0 - 0.5 * cut)) if case.get("ragged") else past))
    return out


def _heads(width):
    h = width // 128
    return dict(H=h, G=max(1, h // 4), dk=128, dv=128, RH=h, rdk=64, rdv=128)


def _pages(d, lens):
    """Block tables over shuffled pages for sequences of these lengths: (int32 tables, pages in the pool)."""
    need = [(n + PAGE - 1) // PAGE for n in lens]
    total = sum(need)
    order = d.perm(total).to(torch.int32)
    tables = torch.zeros((len(lens), max(need)), dtype=torch.int32, device=DEV)
    lo = 0
    for b, n in enumerate(need):
        tables[b, :n] = order[lo:lo + n]
        lo += n
    return tables, total


def _mixer_inputs(case, seed):
    """Everything of a mixer case as plain tensors: weights ``t``, the module's spec, packed input rows, pools, states."""
    d = _Draw(seed, DTYPES[case["dtype"]])
    W, kind = case["width"], case["kind"]
    hd = _heads(W)
    H, G, dk, dv, RH, rdk, rdv = (hd[k] for k in ("H", "G", "dk", "dv", "RH", "rdk", "rdv"))
    por = _portions(case)
    N = sum(n for n, _ in por)
    m = dict(hd, W=W, por=por, N=N, h=d.normal(N, W), kv=None, state=None, tail=None, freqs_base=10000.0)
    t = m["t"] = {}
    if kind == "petipel_attention":
        m["spec"] = {"heads": H, "kv_heads": G, "dim": dk, "vdim": dv, "scale": dk ** -0.5, "bias_max": 4096, "v_mix": True,
                     "q_temp": {"coef": 0.1, "every": 512}}
        t.update(q=d.lin(H * dk, W), k=d.lin(G * dk, W), v=d.lin(G * dv, W), g=d.lin(H, W), rel=d.normal(32, H, s=0.5),
                 o=d.lin(W, H * dv), vmix=torch.tensor(0.3, dtype=d.dtype, device=DEV))
        m["kv"] = (G, dk, dv)
    elif kind == "petipel_recurrence":
        m["spec"] = {"heads": RH, "dim": rdk, "vdim": rdv}
        t.update({"q": d.lin(RH * rdk, W), "f": d.lin(RH * rdk, W, 2.0), "v": d.lin(RH * rdv, W), "f.b": d.normal(RH * rdk),
                  "lower": d.uniform(RH * rdk, hi=0.9), "norm": d.normal(rdv, s=0.1, mean=1.0), "o": d.lin(W, RH * rdv)})
    elif kind == "sanesun_delta":
        ra = max(8, W // 16)
        m["spec"] = {"heads": RH, "kv_heads": RH, "dim": rdk, "vdim": rdv, "conv": 4}
        for name, rows in (("q", RH * rdk), ("k", RH * rdk), ("v", RH * rdv)):
            t[name], t[name + ".conv"] = d.lin(rows, W, 1.5), d.normal(rows, 4, s=0.5)
        t.update({"b": d.lin(RH, W), "A_log": d.uniform(RH, lo=-1.5, hi=0.5), "a1": d.lin(ra, W), "a2": d.lin(RH * rdk, ra, 2.0),
                  "dt_bias": d.normal(RH * rdk, mean=-1.0), "g1": d.lin(ra, W), "g2": d.lin(RH * rdv, ra, 2.0),
                  "norm": d.normal(rdv, s=0.1, mean=1.0), "o": d.lin(W, RH * rdv)})
        m["tail"] = d.normal(len(por), 3, RH * (2 * rdk + rdv), dtype=torch.float32)
    elif kind == "latent_attention":
        r, dr = 256, 64
        m.update(rank=r, dr=dr)
        m["spec"] = {"heads": H, "dim": dk, "rot_dim": dr, "vdim": dv, "kv_rank": r, "scale": (dk + dr) ** -0.5,
                     "mask": {"size": 512}, "rot": {"dims": dr, "base": m["freqs_base"]}}
        t.update({"q": d.lin(H * (dk + dr), W, 2.0), "dkv": d.lin(r + dr, W, 2.0), "dkv.norm": d.normal(r, s=0.1, mean=1.0),
                  "uk": d.lin(H * dk, r, 1.5), "uv": d.lin(H * dv, r), "sink": d.normal(H), "o": d.lin(W, H * dv)})
        m["kv"] = (1, r + dr, 0)
    else:
        decay = [1.0 - 2.0 ** (-5.0 - 7.0 * i / max(1, RH - 1)) for i in range(RH)]
        m["spec"] = {"left_scale": 1.0, "right_scale": 0.5,
                     "left": {"heads": H, "kv_heads": G, "dim": dk, "vdim": dv, "scale": dk ** -0.5, "softcap": 30.0,
                              "mask": {"size": 512}, "rot": {"dims": dk // 2, "base": m["freqs_base"]}},
                     "right": {"heads": RH, "dim": rdk, "vdim": rdv, "decay": decay}}
        t.update({"left.q": d.lin(H * dk, W, 2.0), "left.k": d.lin(G * dk, W, 2.0), "left.v": d.lin(G * dv, W),
                  "left.o": d.lin(W, H * dv), "left.q.norm": d.normal(dk, s=0.3, mean=1.0),
                  "left.k.norm": d.normal(dk, s=0.3, mean=1.0), "right.q": d.lin(RH * rdk, W), "right.k": d.lin(RH * rdk, W),
                  "right.v": d.lin(RH * rdv, W), "right.g": d.lin(RH * rdv, W, 2.0), "right.o": d.lin(W, RH * rdv)})
        m["kv"] = (G, dk, dv)
    if kind in ("petipel_recurrence", "sanesun_delta", "fibirax_mixer"):   # what earlier tokens left: read where past > 0
        m["state"] = d.normal(len(por), RH, rdk, rdv, s=0.3, dtype=torch.float32)
    if m["kv"]:
        g, a, b = m["kv"]
        m["tables"], total = _pages(d, [n + p for n, p in por])
        m["k_pool"] = d.normal(total, g, PAGE, a)
        m["v_pool"] = d.normal(total, g, PAGE, b) if b else None
    else:
        m["tables"] = torch.zeros((len(por), 1), dtype=torch.int32, device=DEV)
    return m


def _packed_state(m):
    """The step's description that every layer of a step shares, as the step engine builds it."""
    pos, slots, spans, scans, first = [], [], [], [], 0
    tables = m["tables"].cpu().to(torch.int64)
    for b, (n, past) in enumerate(m["por"]):
        p = torch.arange(past, past + n)
        pos.append(p)
        slots.append(tables[b][p // PAGE] * PAGE + p % PAGE if m["kv"] else p)
        spans.append((first, n, b, past))
        scans.append((first, n, b, 1 if past == 0 else 0))
        first += n
    rows = torch.repeat_interleave(torch.arange(len(spans)), torch.tensor([s[1] for s in spans]))
    return RaggedBatchState(tok_pos=torch.cat(pos).to(torch.int32).to(DEV), slot_mapping=torch.cat(slots).to(DEV),
                            block_tables=m["tables"], scan_seqs=torch.tensor(scans, dtype=torch.int32).to(DEV), spans=spans,
                            tok_row=rows.to(torch.int32).to(DEV), scan_host=scans)


def _llama_config(case):
    return LlamaShapeConfig(hidden_size=case["width"], num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"],
                            intermediate_size=case["ff"], vocab_size=case["vocab"], num_hidden_layers=case["layers"])


def _llama_inputs(case, seed):
    d = _Draw(seed, DTYPES[case["dtype"]])
    W, D, B = case["width"], case["width"] // case["heads"], case["batch"]
    q, kv, ff = case["heads"] * D, case["kv_heads"] * D, case["ff"]
    sd = {"model.embed_tokens.weight": d.normal(case["vocab"], W), "model.norm.weight": d.normal(W, s=0.1, mean=1.0),
          "lm_head.weight": d.lin(case["vocab"], W)}
    for i in range(case["layers"]):
        pre = f"model.layers.{i}."
        for name, out, inp in (("self_attn.q_proj", q, W), ("self_attn.k_proj", kv, W), ("self_attn.v_proj", kv, W),
                               ("self_attn.o_proj", W, q), ("mlp.gate_proj", ff, W), ("mlp.up_proj", ff, W), ("mlp.down_proj", W, ff)):
            sd[pre + name + ".weight"] = d.lin(out, inp)
        for name in ("input_layernorm", "post_attention_layernorm"):
            sd[pre + name + ".weight"] = d.normal(W, s=0.1, mean=1.0)
    lens = [max(1, case["context"] - (37 * b) % max(1, case["context"] // 3)) for b in range(B)]
    tables, total = _pages(d, lens)
    pools = [(d.normal(total, case["kv_heads"], PAGE, D), d.normal(total, case["kv_heads"], PAGE, D)) for _ in range(case["layers"])]
    ids = torch.randint(0, case["vocab"], (B, 1), generator=d.gen, device=DEV)
    return dict(sd=sd, lens=lens, tables=tables, pools=pools, ids=ids, D=D)


def _decode_inputs(case, seed):
    d = _Draw(seed, DTYPES[case["dtype"]])
    B, Hq, G, D, ctx, prefix = (case[k] for k in ("batch", "heads", "kv_heads", "dim", "context", "prefix"))
    own = ctx - prefix
    lens = [prefix + (max(1, own - (own * 3 // 7 * b) % max(1, own // 2)) if case["ragged"] else own) for b in range(B)]
    tables, total = _pages(d, [n - prefix for n in lens])
    if prefix:      # every sequence starts with the same pages
        head = torch.arange(total, total + prefix // PAGE, dtype=torch.int32, device=DEV)
        tables = torch.cat([head.expand(B, -1), tables], dim=1).contiguous()
        total += prefix // PAGE
    pos = torch.tensor([n - 1 for n in lens], device=DEV)
    inv = 500000.0 ** (-torch.arange(0, D, 2, device=DEV, dtype=torch.float32) / D)
    ang = pos.to(torch.float32)[:, None] * inv[None, :]
    ang = torch.cat([ang, ang], dim=1)
    return dict(q=d.normal(B, Hq, D), k=d.normal(B, G, D), v=d.normal(B, G, D), cos=ang.cos().to(d.dtype), sin=ang.sin().to(d.dtype),
                k_pool=d.normal(total, G, PAGE, D), v_pool=d.normal(total, G, PAGE, D), tables=tables, lens=lens,
                ctx=torch.tensor(lens, dtype=torch.int32, device=DEV))


def _handoff_inputs(case, seed):
    d = _Draw(seed, DTYPES[case["dtype"]])
    n = (case["tokens"] + PAGE - 1) // PAGE
    blocks = n + 16
    backing = d.normal(case["layers"], 2, blocks, case["kv_heads"], PAGE, case["dim"])
    return dict(backing=backing, src=d.perm(blocks)[:n].to(torch.int32), dst=d.perm(blocks)[:n].to(torch.int32), blocks=blocks)


def _expert_inputs(case, seed):
    d = _Draw(seed, DTYPES[case["dtype"]])
    W, E = case["width"], 8
    t = {"router": d.lin(E, W, 2.0)}
    for e in range(E):
        t[f"e{e}.gate"], t[f"e{e}.up"], t[f"e{e}.down"] = d.lin(W, W, 2.0), d.lin(W, W, 2.0), d.lin(W, W)
    return dict(t=t, h=d.normal(case["tokens"], W), spec={"expert": {"ff": W, "limit": 7.0}, "router": {"experts": E, "top": 2}})


def _engine_inputs(case, seed):
    W = case["width"]
    hd = _heads(W)
    att = {"type": "attention", "mixer": {"heads": hd["H"], "kv_heads": hd["G"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                          "bias_max": 4096, "v_mix": True, "q_temp": {"coef": 0.1, "every": 512}}}
    rec = {"type": "hgrn2", "mixer": {"heads": hd["RH"], "dim": 64, "vdim": 128}}
    raw = {"architecture": "Petipel", "width": W, "vocab": 2048, "residual_mult": 0.5, "norm": {"eps": EPS},
           "layers": [dict(m, mlp={"kind": "dense", "ff": 4 * W}) for m in (rec, att, rec, att)]}
    lens = [n for n, _ in _portions(dict(case, ragged=True))]
    gen = torch.Generator().manual_seed(seed + 1)
    prompts = [torch.randint(0, raw["vocab"], (n,), generator=gen).tolist() for n in lens]
    return dict(raw=raw, prompts=prompts, t=random_checkpoint(PetipelConfig.from_dict(raw), seed=seed, dtype=DTYPES[case["dtype"]]),
                want=[list(range(max(0, n - 8), n)) for n in lens])


# ---- what a program keeps, and the call -----------------------------------------------------------------------------------


def _prepare_mixer(case, seed):
    m, dtype = _mixer_inputs(case, seed), DTYPES[case["dtype"]]
    kind, spec, t = case["kind"], m["spec"], m["t"]
    if kind == "petipel_attention":
        mod = BiasedPagedAttention(spec, t, EPS, True, DEV, dtype)
    elif kind == "petipel_recurrence":
        mod = GatedLinearRecurrence(spec, t, EPS, DEV, dtype)
    elif kind == "sanesun_delta":
        mod = ChannelDeltaMixer(spec, t, EPS, DEV, dtype)
    elif kind == "latent_attention":
        mod = LatentRotaryAttention(spec, t, EPS, DEV, dtype)
    else:
        mod = ParallelMixer(spec, t, EPS, DEV, dtype)
    state = (m["state"], m["tail"]) if m["tail"] is not None else m["state"]
    cache = RaggedLayerCache(m.get("k_pool"), m.get("v_pool"), state, _packed_state(m))
    return dict(mod=mod, h=m["h"], cache=cache)


def prepare(case, seed):
    kind, dtype = case["kind"], DTYPES[case["dtype"]]
    with torch.no_grad():
        if kind in MIXERS:
            return dict(_prepare_mixer(case, seed), kind=kind)
        if kind == "petipel_experts":
            m = _expert_inputs(case, seed)
            return dict(kind=kind, mod=SigmoidTopKMoE(m["spec"], m["t"], DEV, dtype), h=m["h"])
        if kind == "engine_step":
            m = _engine_inputs(case, seed)
            shards = build_shards(PetipelConfig.from_dict(m["raw"]), m["t"], [(0, 4)], DEV, dtype)
            eng = RaggedStepEngine(shards, max_tokens=sum(len(p) + PAGE for p in m["prompts"]), max_seqs=len(m["prompts"]))
            return dict(kind=kind, eng=eng, entries=[(i, p, w) for i, (p, w) in enumerate(zip(m["prompts"], m["want"]))])
        if kind == "decode_attention":
            m = _decode_inputs(case, seed)
            return dict(m, kind=kind, most=max(m["lens"]), prefix=case["prefix"] // PAGE)
        if kind == "kv_handoff":
            m = _handoff_inputs(case, seed)
            L, shape = case["layers"], (m["blocks"], case["kv_heads"], PAGE, case["dim"])
            pool = KVCachePool(L, case["kv_heads"], case["dim"], PAGE, m["blocks"], DEV, dtype, backing=m["backing"])
            to = KVCachePool(L, case["kv_heads"], case["dim"], PAGE, m["blocks"], DEV, dtype)
            ptrs = [ops.pool_pointer_array([getattr(p.layer(i), w) for i in range(L)]) for p in (pool, to) for w in ("key_pool", "value_pool")]
            return dict(m, kind=kind, pool=pool, to=to, ptrs=ptrs, shape=shape, dtype=dtype)
        m = _llama_inputs(case, seed)
        shard = build_product_shards(_llama_config(case), m["sd"], [(0, case["layers"])], DEV, dtype)[0]
        lens = torch.tensor(m["lens"], device=DEV)
        blk = m["tables"].gather(1, ((lens - 1) // PAGE)[:, None]).squeeze(1).to(torch.int64)
        st = PagedBatchState(block_tables=m["tables"], context_lens=lens.to(torch.int32), slot_mapping=blk * PAGE + (lens - 1) % PAGE,
                             max_context_len=max(m["lens"]))
        return dict(kind=kind, shard=shard, ids=m["ids"], pos=(lens - 1)[:, None], handles=[PagedLayerKV(k, v, st) for k, v in m["pools"]])


def run(s):
    kind = s["kind"]
    with torch.no_grad():
        if kind in MIXERS:
            c = s["cache"]
            out = {"out": s["mod"](s["h"], c), "k_pool": c.k_pool, "v_pool": c.v_pool}
            out["state"], out["tail"] = c.rstate if isinstance(c.rstate, tuple) else (c.rstate, None)
            return out
        if kind == "petipel_experts":
            return s["mod"](s["h"])
        if kind == "engine_step":
            logits = s["eng"].step(s["entries"])
            for rid, _toks, _want in s["entries"]:
                s["eng"].finish(rid)
            return logits
        if kind == "decode_attention":
            args = (s["q"], s["k"], s["v"], s["cos"], s["sin"], s["k_pool"], s["v_pool"], s["tables"], s["ctx"], s["most"])
            out = ops.rope_append_decode_attention_prefix(*args, s["prefix"]) if s["prefix"] else ops.rope_append_decode_attention(*args)
            return [out, s["k_pool"], s["v_pool"]]
        if kind == "kv_handoff":
            packed = ops.kv_pack_layers(s["ptrs"][0], s["ptrs"][1], s["shape"], s["dtype"], s["src"])
            ops.kv_unpack_layers(packed, s["ptrs"][2], s["ptrs"][3], s["shape"], s["dst"])
            return [packed, s["to"].backing]
        h, _ = s["shard"].forward(s["ids"], position_ids=s["pos"], past_key_values=s["handles"])
        return [s["shard"].get_logits(h)] + [p for x in s["handles"] for p in (x.k_pool, x.v_pool)]


# ---- what a call cannot do without -----------------------------------------------------------------------------------------


def _pairs(por, window=0):
    """(query, key) pairs a causal (windowed) mask lets through, and keys that have to be read at all."""
    pairs = keys = 0
    for n, past in por:
        if window:
            pairs += sum(min(p + 1, window) for p in range(past, past + n))
            keys += n + min(past, window - 1)
        else:
            pairs += n * past + n * (n + 1) // 2
            keys += n + past
    return pairs, keys


def work(case):
    kind = case["kind"]
    if kind == "decode_attention":
        B, Hq, G, D = case["batch"], case["heads"], case["kv_heads"], case["dim"]
        own = case["context"] - case["prefix"]
        lens = [max(1, own - (own * 3 // 7 * b) % max(1, own // 2)) if case["ragged"] else own for b in range(B)]
        unique = case["prefix"] + sum(lens)
        return {"bytes": 2 * (unique * G * D * 2 + B * (2 * Hq + 2 * G) * D), "flops": 4 * Hq * D * (sum(lens) + B * case["prefix"])}
    if kind == "kv_handoff":
        payload = case["layers"] * 2 * ((case["tokens"] + PAGE - 1) // PAGE) * case["kv_heads"] * PAGE * case["dim"] * 2
        return {"bytes": 4 * payload, "flops": 0}
    if kind == "llama_step":
        W, D, B = case["width"], case["width"] // case["heads"], case["batch"]
        weights = case["layers"] * (2 * W * case["heads"] * D + 2 * W * case["kv_heads"] * D + 3 * W * case["ff"]) + W * case["vocab"]
        return {"bytes": 2 * (weights + case["layers"] * B * case["context"] * case["kv_heads"] * D * 2), "flops": 2 * B * weights}
    if kind == "petipel_experts":
        n, W = case["tokens"], case["width"]
        return {"bytes": 2 * (min(8, 2 * n) * 3 * W * W + 2 * n * W), "flops": 2 * n * 2 * 3 * W * W}
    W, hd = case["width"], _heads(case["width"])
    H, G, RH = hd["H"], hd["G"], hd["RH"]
    por = _portions(dict(case, ragged=True) if kind == "engine_step" else case)
    N, S = sum(n for n, _ in por), len(por)
    pairs, keys = _pairs(por)
    att_w, rec_w = W * 128 * (2 * H + 2 * G) + H * W, W * RH * (2 * 64 + 2 * 128)
    rec_flops, state = N * RH * 64 * 128 * 6, S * RH * 64 * 128 * 4 * 2
    if kind == "engine_step":
        weights = 2 * (att_w + rec_w) + 4 * 8 * W * W
        return {"bytes": 2 * (weights + 2048 * W) + 2 * state, "flops": 2 * N * weights + 2 * (4 * H * 128 * pairs + rec_flops)}
    io = 4 * N * W
    if kind == "petipel_attention":
        return {"bytes": 2 * att_w + io + keys * G * 256 * 2, "flops": 2 * N * att_w + 4 * H * 128 * pairs}
    if kind == "petipel_recurrence":
        return {"bytes": 2 * rec_w + io + state, "flops": 2 * N * rec_w + rec_flops}
    if kind == "sanesun_delta":
        ra = max(8, W // 16)
        w = rec_w + RH * W + 2 * ra * W + ra * RH * 192
        return {"bytes": 2 * w + io + state, "flops": 2 * N * w + N * RH * 64 * 128 * 8}
    if kind == "latent_attention":
        pairs, keys = _pairs(por, 512)
        w = W * (H * 192 + 320) + H * 256 * 256 + H * 128 * W
        return {"bytes": 2 * w + io + keys * 320 * 2, "flops": 2 * N * w + 2 * H * (320 + 256) * pairs}
    pairs, keys = _pairs(por, 512)
    w = att_w + W * RH * (2 * 64 + 3 * 128)
    return {"bytes": 2 * w + io + state + keys * G * 256 * 2, "flops": 2 * N * w + 4 * H * 128 * pairs + rec_flops}


# ---- the same outputs in float64 ---------------------------------------------------------------------------------------------


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _bucket(n, rows, far):
    half = rows // 2
    if n < half:
        return n
    return min(rows - 1, half + int(math.floor(math.log(n / half) / math.log(far / half) * (rows - half))))


def _turn(x, pos, dims, base, interleaved):
    """x [n, heads, d]: the first ``dims`` entries turned pairwise by the position."""
    f = base ** (-2.0 * torch.arange(dims // 2, device=x.device, dtype=F64) / dims)
    ang = (pos.to(F64)[:, None] * f)[:, None, :]
    c, s, out = ang.cos(), ang.sin(), x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, dims // 2), slice(dims // 2, dims))
    out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return out


def _gather(pool, table, n):
    """The first n rows of a sequence out of its pages: [n, heads, d]."""
    need = (n + PAGE - 1) // PAGE
    p = pool[table[:need].to(torch.int64)].to(F64)
    return p.transpose(1, 2).reshape(need * PAGE, pool.shape[1], pool.shape[3])[:n]


def _store(pool, table, first, rows):
    pos = torch.arange(first, first + rows.shape[0], device=rows.device)
    pool[table[pos // PAGE].to(torch.int64), :, pos % PAGE] = rows


def _attend(q, k, v, first, add=None, window=0, cap=0.0, sink=None):
    """q [n, H, dk] (scaled) of positions first .. over k, v [T, G, d]; ``add(distance, head)``, one head at a time."""
    n, H, T = q.shape[0], q.shape[1], k.shape[0]
    dist = torch.arange(first, first + n, device=q.device)[:, None] - torch.arange(T, device=q.device)[None, :]
    hide = (dist < 0) | (dist >= window) if window else dist < 0
    out = torch.empty(n, H, v.shape[2], dtype=F64, device=q.device)
    for h in range(H):
        g = h // (H // k.shape[1])
        s = q[:, h] @ k[:, g].T
        if cap:
            s = cap * torch.tanh(s / cap)
        if add is not None:
            s = s + add(dist.clamp(min=0), h)
        s = s.masked_fill(hide, float("-inf"))
        m = s.amax(dim=1, keepdim=True)
        m = torch.maximum(m, sink[h]) if sink is not None else m
        e = torch.exp(s - m)
        out[:, h] = (e @ v[:, g]) / (e.sum(1, keepdim=True) + (torch.exp(sink[h] - m) if sink is not None else 0.0))
    return out


def _exact_petipel_attention(t, h, spec, por, tables, kp, vp, v_prev=None):
    """(outputs, the values stored for the step's tokens); the pools are written."""
    H, G, dk, dv = spec["heads"], spec["kv_heads"], spec["dim"], spec["vdim"]
    n_all = h.shape[0]
    q, k, v = (h @ t["q"].T).view(n_all, H, dk), (h @ t["k"].T).view(n_all, G, dk), _unit((h @ t["v"].T).view(n_all, G, dv), EPS)
    if v_prev is not None:
        v = (1.0 - t["vmix"]) * v + t["vmix"] * v_prev
    rows = t["rel"].shape[0]
    most = max(n + p for n, p in por)
    idx = torch.tensor([_bucket(d, rows, spec["bias_max"]) for d in range(most)], device=h.device)
    bias = t["rel"][idx].T.contiguous()
    out, lo = torch.empty(n_all, H, dv, dtype=F64, device=h.device), 0
    for b, (n, past) in enumerate(por):
        _store(kp, tables[b], past, k[lo:lo + n])
        _store(vp, tables[b], past, v[lo:lo + n])
        pos = torch.arange(past, past + n, device=h.device)
        temp = 1.0 + spec["q_temp"]["coef"] * torch.log(((pos + 1) // spec["q_temp"]["every"] + 1).to(F64))
        out[lo:lo + n] = _attend(q[lo:lo + n] * (temp * spec["scale"])[:, None, None], _gather(kp, tables[b], past + n),
                                 _gather(vp, tables[b], past + n), past, add=lambda d, hd: bias[hd][d])
        lo += n
    out = out * torch.sigmoid(h @ t["g"].T)[:, :, None]
    return out.reshape(n_all, H * dv) @ t["o"].T, v


def _scan(por, state, step):
    """Runs ``step(S, token) -> (S, read-out)`` over every sequence; returns the read-outs and writes the states."""
    outs, lo = [], 0
    for b, (n, past) in enumerate(por):
        S = state[b] if past else torch.zeros_like(state[b])
        for i in range(lo, lo + n):
            S, o = step(S, i)
            outs.append(o)
        state[b] = S
        lo += n
    return torch.stack(outs)


def _exact_recurrence(t, h, spec, por, state):
    n, H, dk, dv = h.shape[0], spec["heads"], spec["dim"], spec["vdim"]
    q, v = (h @ t["q"].T).view(n, H, dk), (h @ t["v"].T).view(n, H, dv)
    q, low = q * torch.sigmoid(q), t["lower"].view(H, dk)
    f = low + (1.0 - low) * torch.sigmoid(h @ t["f"].T + t["f.b"]).view(n, H, dk)

    def step(S, i):
        S = f[i][:, :, None] * S + (1.0 - f[i])[:, :, None] * v[i][:, None, :]
        return S, (q[i][:, None, :] @ S).squeeze(1)

    o = _unit(_scan(por, state, step), EPS) * t["norm"]
    return o.reshape(n, H * dv) @ t["o"].T


def _exact_delta(t, h, spec, por, state, tail):
    n, H, dk, dv = h.shape[0], spec["heads"], spec["dim"], spec["vdim"]
    x = h @ torch.cat([t["q"], t["k"], t["v"]]).T
    w = torch.cat([t["q.conv"], t["k.conv"], t["v.conv"]])
    y, lo = torch.empty_like(x), 0
    for b, (m, past) in enumerate(por):
        row = torch.cat([tail[b] if past else torch.zeros_like(tail[b]), x[lo:lo + m]])
        y[lo:lo + m] = sum(row[i:i + m] * w[:, i] for i in range(4))
        tail[b] = row[-3:]
        lo += m
    y = y * torch.sigmoid(y)
    q, k, v = y[:, :H * dk].view(n, H, dk), y[:, H * dk:2 * H * dk].view(n, H, dk), y[:, 2 * H * dk:].view(n, H, dv)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    beta = torch.sigmoid(h @ t["b"].T)
    a = ((h @ t["a1"].T) @ t["a2"].T + t["dt_bias"]).view(n, H, dk)
    g = torch.exp(-torch.exp(t["A_log"])[None, :, None] * torch.nn.functional.softplus(a, threshold=50))

    def step(S, i):
        S = g[i][:, :, None] * S
        u = beta[i][:, None] * (v[i] - (k[i][:, None, :] @ S).squeeze(1))
        S = S + k[i][:, :, None] * u[:, None, :]
        return S, (q[i][:, None, :] @ S).squeeze(1)

    o = _unit(_scan(por, state, step), EPS) * t["norm"] * torch.sigmoid((h @ t["g1"].T) @ t["g2"].T).view(n, H, dv)
    return o.reshape(n, H * dv) @ t["o"].T


def _exact_latent(t, h, m, kp):
    spec, n_all = m["spec"], h.shape[0]
    H, dk, dr, dv, r, base = spec["heads"], spec["dim"], m["dr"], spec["vdim"], m["rank"], m["freqs_base"]
    pos = torch.cat([torch.arange(p, p + n, device=h.device) for n, p in m["por"]])
    q, down = (h @ t["q"].T).view(n_all, H, dk + dr), h @ t["dkv"].T
    q = torch.cat([q[..., :dk], _turn(q[..., dk:], pos, dr, base, True)], dim=-1) * spec["scale"]
    row = torch.cat([(_unit(down[:, :r], EPS) * t["dkv.norm"])[:, None], _turn(down[:, None, r:], pos, dr, base, True)], dim=-1)
    out, lo = torch.empty(n_all, H, dv, dtype=F64, device=h.device), 0
    for b, (n, past) in enumerate(m["por"]):
        _store(kp, m["tables"][b], past, row[lo:lo + n])
        c = _gather(kp, m["tables"][b], past + n)[:, 0]
        k = torch.cat([(c[:, :r] @ t["uk"].T).view(-1, H, dk), c[:, None, r:].expand(-1, H, -1)], dim=-1)
        out[lo:lo + n] = _attend(q[lo:lo + n], k, (c[:, :r] @ t["uv"].T).view(-1, H, dv), past, window=spec["mask"]["size"], sink=t["sink"])
        lo += n
    return out.reshape(n_all, H * dv) @ t["o"].T


def _exact_fibirax(t, h, m, kp, vp, state):
    spec, n_all = m["spec"], h.shape[0]
    L, R = spec["left"], spec["right"]
    H, G, dk, dv, RH, rdk, rdv = (m[k] for k in ("H", "G", "dk", "dv", "RH", "rdk", "rdv"))
    pos = torch.cat([torch.arange(p, p + n, device=h.device) for n, p in m["por"]])
    q = _unit((h @ t["left.q"].T).view(n_all, H, dk), EPS) * t["left.q.norm"]
    k = _unit((h @ t["left.k"].T).view(n_all, G, dk), EPS) * t["left.k.norm"]
    v = (h @ t["left.v"].T).view(n_all, G, dv)
    q, k = (_turn(x, pos, L["rot"]["dims"], L["rot"]["base"], True) for x in (q, k))
    left, lo = torch.empty(n_all, H, dv, dtype=F64, device=h.device), 0
    zero = torch.zeros(H, dtype=F64, device=h.device)
    for b, (n, past) in enumerate(m["por"]):
        _store(kp, m["tables"][b], past, k[lo:lo + n])
        _store(vp, m["tables"][b], past, v[lo:lo + n])
        left[lo:lo + n] = _attend(q[lo:lo + n] * L["scale"], _gather(kp, m["tables"][b], past + n), _gather(vp, m["tables"][b], past + n),
                                  past, window=L["mask"]["size"], cap=L["softcap"], sink=zero)
        lo += n
    rq, rk, rv = (h @ t["right.q"].T).view(n_all, RH, rdk), (h @ t["right.k"].T).view(n_all, RH, rdk) * rdk ** -0.5, (h @ t["right.v"].T).view(n_all, RH, rdv)
    decay = torch.tensor(R["decay"], dtype=torch.float32, device=h.device).to(F64)[:, None, None]

    def step(S, i):
        S = decay * S + rk[i][:, :, None] * rv[i][:, None, :]
        return S, (rq[i][:, None, :] @ S).squeeze(1)

    g = h @ t["right.g"].T
    right = _unit(_scan(m["por"], state, step), EPS).reshape(n_all, RH * rdv) * (g * torch.sigmoid(g))
    return spec["left_scale"] * (left.reshape(n_all, H * dv) @ t["left.o"].T) + spec["right_scale"] * (right @ t["right.o"].T)


def _exact_engine(case, seed):
    m = _engine_inputs(case, seed)
    t = {k: v.to(DEV).to(F64) for k, v in m["t"].items()}
    por = [(len(p), 0) for p in m["prompts"]]
    tables, total = _pages(_Draw(0, F64), [n for n, _ in por])
    x = t["embed"][torch.tensor(sum(m["prompts"], []), device=DEV)]
    v_first = None
    for i, layer in enumerate(m["raw"]["layers"]):
        w = {k[len(f"l{i}."):]: v for k, v in t.items() if k.startswith(f"l{i}.")}
        mix, spec = {k[4:]: v for k, v in w.items() if k.startswith("mix.")}, layer["mixer"]
        h = _unit(x, EPS) * (1.0 + w["norm1"])
        if layer["type"] == "attention":
            kp, vp = (torch.zeros(total, spec["kv_heads"], PAGE, 128, dtype=F64, device=DEV) for _ in range(2))
            y, v = _exact_petipel_attention(mix, h, spec, por, tables, kp, vp, v_first)
            v_first = v if v_first is None else v_first
        else:
            y = _exact_recurrence(mix, h, spec, por, torch.zeros(len(por), spec["heads"], 64, 128, dtype=F64, device=DEV))
        x = x + 0.5 * _unit(y, EPS) * (1.0 + w["norm1b"])
        z = (_unit(x, EPS) * (1.0 + w["norm2"])) @ w["mlp.up"].T
        a, b, c, e = w["mlp.act"]
        y = (a * _unit(z, EPS) + b * _unit(z * z, EPS) + c * _unit(z ** 3, EPS) + e) @ w["mlp.down"].T
        x = x + 0.5 * _unit(y, EPS) * (1.0 + w["norm2b"])
    rows, lo = [], 0
    for (n, _), want in zip(por, m["want"]):
        rows += [lo + i for i in want]
        lo += n
    return (_unit(x[rows], EPS) * (1.0 + t["final.norm"])) @ t["head"].T


def _exact_llama(case, seed):
    m = _llama_inputs(case, seed)
    sd, D, B = {k: v.to(F64) for k, v in m["sd"].items()}, m["D"], case["batch"]
    eps, H, G = 1e-5, case["heads"], case["kv_heads"]
    pos = torch.tensor([n - 1 for n in m["lens"]], device=DEV)
    x, pools = sd["model.embed_tokens.weight"][m["ids"][:, 0]], []
    for i in range(case["layers"]):
        w = lambda n: sd[f"model.layers.{i}.{n}.weight"]  # noqa: E731
        h = _unit(x, eps) * w("input_layernorm")
        q, k, v = ((h @ w(f"self_attn.{n}_proj").T).view(B, -1, D) for n in "qkv")
        q, k = _turn(q, pos, D, 500000.0, False) * D ** -0.5, _turn(k, pos, D, 500000.0, False)
        kp, vp = (p.to(F64) for p in m["pools"][i])
        o = torch.empty(B, H, D, dtype=F64, device=DEV)
        for b, n in enumerate(m["lens"]):
            _store(kp, m["tables"][b], n - 1, k[b:b + 1])
            _store(vp, m["tables"][b], n - 1, v[b:b + 1])
            o[b:b + 1] = _attend(q[b:b + 1], _gather(kp, m["tables"][b], n), _gather(vp, m["tables"][b], n), n - 1)
        x = x + o.view(B, H * D) @ w("self_attn.o_proj").T
        h = _unit(x, eps) * w("post_attention_layernorm")
        g = h @ w("mlp.gate_proj").T
        x = x + (g * torch.sigmoid(g) * (h @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T
        pools += [kp, vp]
    return [((_unit(x, eps) * sd["model.norm.weight"]) @ sd["lm_head.weight"].T)[:, None]] + pools


def _exact_decode(case, seed):
    m = _decode_inputs(case, seed)
    D = case["dim"]
    cos, sin = m["cos"].to(F64)[:, None], m["sin"].to(F64)[:, None]
    half = lambda x: torch.cat([-x[..., D // 2:], x[..., :D // 2]], dim=-1)  # noqa: E731
    q, k = (x.to(F64) * cos + half(x.to(F64)) * sin for x in (m["q"], m["k"]))
    kp, vp, out = m["k_pool"].to(F64), m["v_pool"].to(F64), torch.empty(m["q"].shape, dtype=F64, device=DEV)
    for b, n in enumerate(m["lens"]):
        _store(kp, m["tables"][b], n - 1, k[b:b + 1])
        _store(vp, m["tables"][b], n - 1, m["v"][b:b + 1].to(F64))
        out[b:b + 1] = _attend(q[b:b + 1] * D ** -0.5, _gather(kp, m["tables"][b], n), _gather(vp, m["tables"][b], n), n - 1)
    return [out, kp, vp]


def _exact_experts(case, seed):
    m = _expert_inputs(case, seed)
    t, h = {k: v.to(F64) for k, v in m["t"].items()}, m["h"].to(F64)
    s, limit = torch.sigmoid(h @ t["router"].T), m["spec"]["expert"]["limit"]
    out, ids = torch.zeros_like(h), torch.topk(s, 2, dim=1).indices
    for e in range(8):
        rows = (ids == e).any(1).nonzero().squeeze(1)
        x = s[rows, e][:, None] * h[rows]
        g, u = (x @ t[f"e{e}.gate"].T).clamp(max=limit), (x @ t[f"e{e}.up"].T).clamp(-limit, limit)
        out[rows] += (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ t[f"e{e}.down"].T
    return out


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "kv_handoff":
            return None      # bytes are moved, nothing is computed
        if kind == "engine_step":
            return _exact_engine(case, seed)
        if kind == "llama_step":
            return _exact_llama(case, seed)
        if kind == "decode_attention":
            return _exact_decode(case, seed)
        if kind == "petipel_experts":
            return _exact_experts(case, seed)
        m = _mixer_inputs(case, seed)
        t, h = {k: v.to(F64) for k, v in m["t"].items()}, m["h"].to(F64)
        kp, vp, state, tail = (m.get(k).to(F64) if m.get(k) is not None else None for k in ("k_pool", "v_pool", "state", "tail"))
        if kind == "petipel_attention":
            out, _ = _exact_petipel_attention(t, h, m["spec"], m["por"], m["tables"], kp, vp)
        elif kind == "petipel_recurrence":
            out = _exact_recurrence(t, h, m["spec"], m["por"], state)
        elif kind == "sanesun_delta":
            out = _exact_delta(t, h, m["spec"], m["por"], state, tail)
        elif kind == "latent_attention":
            out = _exact_latent(t, h, m, kp)
        else:
            out = _exact_fibirax(t, h, m, kp, vp, state)
        return {"out": out, "k_pool": kp, "v_pool": vp, "state": state, "tail": tail}
