"""What the engine is measured on: passes of its step function over the seven designs it serves.

A pass is what a server does with a batch.  Every request of the batch has ``context`` tokens in its cache; ONE step
brings the next tokens of all of them (``portion`` tokens for the first ``portions`` requests, a single token for the
others) and ``steps`` further steps bring one token each.  With no context that is a prompt and its first decoded
tokens; with a portion of one it is decoding; with both kinds of request it is the step of a server that batches
continuously.  The logits at the last token of every request and step come back.  Afterwards the requests are cut back
to where they were (designs whose caches can be), or they were forks of the held requests and are given back.

Sizes: the benchmark's shapes (width 2048 and 4096 of its workloads, Qwen3-1.7B and Qwen3-8B, contexts of 1,024 and
4,096, prompts of 2,048, batches of 8 and 64) and the three-layer shape of the tests.
"""
import functools
import json
import math

import torch

import airun_b200
from airun_b200 import Engine, EngineOptions, StepEntry
from airun_b200.config.base import lookup_architecture
from airun_b200.weights.loader import DictSource

VOCAB = 32768
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


def _case(name, design, width, portion, requests=1, portions=None, context=0, steps=1, dtype="bf16", layers=6, ff=None, heads=None,
          kv_heads=8, vocab=VOCAB, ragged=0.0):
    """``ragged``: request i of n is shorter by the share ragged * i / n, in its context and in its portion."""
    return dict(name=name, design=design, dtype=dtype, width=width, layers=layers, ff=ff or 3 * width, heads=heads or width // 128,
                kv_heads=kv_heads, vocab=vocab, requests=requests, portions=requests if portions is None else portions,
                portion=portion, context=context, steps=steps, ragged=ragged)


def listed():
    return [
        # the smallest call: a single request decoding on a small model, where launches and latency count
        _case("small decode 1", "qwen3", 1024, 1, context=100, steps=3, layers=3, ff=2816, heads=16, kv_heads=4, vocab=20000),
        # the benchmark's headline: Qwen3-8B, eight requests at a context of 4,096 tokens
        _case("qwen3 8b decode 8", "qwen3", 4096, 1, requests=8, context=4090, steps=3, layers=36, vocab=151936),
        # ... and its prompt of 2,048 tokens: the time to the first tokens
        _case("qwen3 8b prompt 2048", "qwen3", 4096, 2048, layers=36, vocab=151936),
        # a step of a server that batches continuously (Qwen3-1.7B): 24 requests decoding beside two portions
        _case("qwen3 1.7b serving", "qwen3", 2048, 243, requests=26, portions=2, context=900, steps=0, layers=28, vocab=151936, ragged=0.8),
        # the true 32-bit path, as used to check a model: three prompts of unequal length and their first tokens
        _case("qwen3 fp32 prompts", "qwen3", 1024, 257, requests=3, steps=2, layers=3, ff=2816, heads=16, kv_heads=4, vocab=20000,
              dtype="fp32", ragged=0.5),
        # prompts of the other designs at the benchmark's width, one long or several of odd lengths
        _case("vedizen prompt 2048", "vedizen", 2048, 2048),
        _case("pogarax prompts", "pogarax", 2048, 811, requests=3, ragged=0.5),
        _case("gamanex prompt 2048", "gamanex", 2048, 2048),
        _case("tagulix prompt 2048", "tagulix", 2048, 2048),
        _case("pirerax prompt 1536", "pirerax", 2048, 1536),
        # decoding with recurrent states and routed experts, a small batch and a large one
        _case("pirerax decode 8", "pirerax", 2048, 1, requests=8, context=1024, steps=15),
        _case("losalorn decode 64", "losalorn", 2048, 1, requests=64, context=1000, steps=15, ragged=0.5),
    ]


DESIGNS = ("qwen3", "vedizen", "pogarax", "gamanex", "tagulix", "losalorn", "pirerax")


def draw(rng):
    def size(lo, hi):                                   # evenly over the logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    design, kind = rng.choice(DESIGNS), rng.choice(("prompt", "decode", "both"))
    fp32 = rng.random() < 0.12
    width = 1024 if fp32 else rng.choice((1024, 2048, 2048))
    requests = size(1, 6) if kind == "prompt" else size(1, 8 if fp32 else 64) if kind == "decode" else size(2, 8 if fp32 else 32)
    portion = 1 if kind == "decode" else size(2, 600 if fp32 else 1980) // requests + 1
    context = 0 if kind == "prompt" else size(16, 400 if fp32 else 1500)
    portions = 0 if kind == "decode" else requests if kind == "prompt" else rng.randint(1, requests)
    case = _case("", design, width, portion, requests=requests, portions=portions, context=context,
                 steps={"prompt": rng.randint(0, 2), "decode": rng.randint(3, 15), "both": rng.randint(0, 2)}[kind],
                 dtype="fp32" if fp32 else "bf16", layers=rng.randint(3, 16) if design == "qwen3" else 6,
                 kv_heads=rng.choice((4, 8)), ragged=round(rng.uniform(0.0, 0.9), 2))
    del case["name"]
    return case


# ----------------------------------------------------------------------------- requests
def _lengths(case):
    """[(context, tokens of the first step)] of every request."""
    out = []
    for i in range(case["requests"]):
        cut = 1.0 - case["ragged"] * i / case["requests"]
        out.append((int(case["context"] * cut), max(1, int(case["portion"] * cut)) if i < case["portions"] else 1))
    return out


def _tokens(case, seed):
    """Every request's tokens: context, first step, further steps."""
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, case["vocab"], (c + p + case["steps"],), generator=g).tolist() for c, p in _lengths(case)]


# ----------------------------------------------------------------------------- the designs' configurations
def config_of(case):
    """config.json of the case's model: for the designs other than Qwen3 six layer runs of the benchmark's make."""
    W, F, H, G, V = case["width"], case["ff"], case["heads"], case["kv_heads"], case["vocab"]
    base = dict(vocab=V, width=W, norm=dict(eps=1e-5))
    design = case["design"]
    if design == "qwen3":
        return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=V, hidden_size=W, num_hidden_layers=case["layers"],
                    num_attention_heads=H, num_key_value_heads=G, head_dim=128, intermediate_size=F, max_position_embeddings=40960,
                    rms_norm_eps=1e-6, rope_theta=1000000.0, tie_word_embeddings=False)
    if design == "vedizen":
        mlp = dict(kind="dense", ff=F, limit=7.0)
        gla = dict(type="gla", mixer=dict(heads=H, dim=64, vdim=128, tau=16.0), mlp=mlp)
        att = dict(type="attention", mixer=dict(heads=H, kv_heads=G, dim=64, vdim=128, scale=0.125, softcap=50.0, diff=0.5,
                                                mask=dict(size=2048)), mlp=mlp)
        return dict(base, architecture="Vedizen", embedding=dict(scale=1.0), layers=[gla, att, att, gla], loop=dict(start=0, stop=2, times=2))
    if design == "pogarax":
        dense = dict(kind="dense", ff=F)
        moe = dict(kind="moe", expert=dict(ff=F // 2), router=dict(experts=16, top=2))
        delta = dict(type="channel_delta", mixer=dict(heads=H, kv_heads=H // 2, dim=64, vdim=128, conv=4), mlp=dense)
        lat = dict(heads=H, dim=128, rot_dim=64, vdim=128, q_rank=W // 2, kv_rank=512, scale=192 ** -0.5, mask=dict(size=2048),
                   rot=dict(dims=64, base=1e6, scaling=dict(factor=4.0, original=4096, fast=32.0, slow=1.0)))
        return dict(base, architecture="Pogarax", residual_mult=0.7, layers=[
            delta, dict(type="latent_attention", mixer=lat, mlp=moe), delta, dict(type="latent_attention", mixer=dict(lat, kv_from=1), mlp=moe),
            delta, dict(type="wkv", mixer=dict(heads=W // 64, dim=64), mlp=moe)])
    if design == "gamanex":
        dense = dict(kind="dense", ff=3 * F // 2)
        moe = dict(kind="moe", expert=dict(ff=F // 2), router=dict(experts=16, top=2))
        mix = dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, q_temp=dict(coef=0.3, every=512))
        return dict(base, architecture="Gamanex", logit_scale=0.5, layers=[
            dict(type="attention", mixer=m, mlp=f) for m, f in ((mix, dense), (dict(mix, kv_from=0), moe), (mix, dense),
                                                                (dict(mix, kv_from=2), moe), (mix, dense), (mix, moe))])
    if design == "tagulix":
        moe = dict(kind="moe", expert=dict(ff=F // 4), router=dict(experts=16, top=4, identity=4, scale=1.5, groups=dict(count=4, keep=2)))
        att = dict(type="attention", mixer=dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=0.1, mask=dict(size=1024),
                                                rot=dict(dims=64, base=10000.0)), mlp=moe)
        par = dict(type="parallel", mixer=dict(
            left=dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, bias_max=2048, q_temp=dict(coef=0.3, every=512)),
            right=dict(heads=H // 2, dim=64, vdim=128, decay=[1.0 - 2.0 ** -(3 + i % 6) for i in range(H // 2)]),
            left_scale=1.0, right_scale=1.0), mlp=moe)
        return dict(base, architecture="Tagulix", residual_mult=0.6, streams=4,
                    layers=[att, par, dict(att, weights_of=0), par, dict(att, weights_of=0), dict(par, weights_of=1)])
    if design == "losalorn":
        mlp = dict(kind="dense", ff=F, limit=7.0)
        delta = dict(type="delta", mixer=dict(heads=H, kv_heads=H // 2, dim=64, vdim=128, conv=4), mlp=mlp)
        att = dict(type="attention", mixer=dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=1024),
                                                rot=dict(dims=64, base=500000.0, scaling=dict(factor=8.0, low=1.0, high=4.0, original=8192))), mlp=mlp)
        return dict(base, architecture="Losalorn", embedding=dict(scale=W ** 0.5), logit_softcap=30.0, loop=dict(start=1, stop=3, times=2),
                    layers=[delta, att, delta, att])
    mlp = dict(kind="moe", expert=dict(ff=F // 4, limit=7.0), router=dict(experts=16, top=4, groups=dict(count=4, keep=2)))
    att = dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5)
    lat = dict(type="latent_attention", mixer=dict(heads=H, dim=128, rot_dim=64, vdim=128, kv_rank=512, scale=192 ** -0.5,
                                                   rot=dict(dims=64, base=10000.0)), mlp=mlp)
    par = dict(type="parallel", mixer=dict(left=dict(att, rot=dict(dims=64, base=10000.0)),
                                           right=dict(heads=H, kv_heads=H // 2, dim=64, vdim=128, conv=4)), mlp=mlp)
    layer = dict(type="attention", mixer=dict(att, q_temp=dict(coef=0.3, every=512)), mlp=mlp)
    return dict(base, architecture="Pirerax", layers=[lat, layer, par] * 2)


def _runs(cfg):
    """[(layer, whether a pass of the loop begins with it, the pass)] in the order of execution."""
    loop = cfg.get("loop") or dict(start=0, stop=0, times=0)
    order = [(i, False, 0) for i in range(loop["start"])]
    for t in range(loop["times"]):
        order += [(i, i == loop["start"], t) for i in range(loop["start"], loop["stop"])]
    return order + [(i, False, 0) for i in range(loop["stop"], len(cfg["layers"]))]


# ----------------------------------------------------------------------------- weights
RANK = 16                                               # of every low-rank pair; REL rows of a distance table
REL = 32


def shapes_of(case):
    """name -> shape of every tensor."""
    cfg, d = config_of(case), case["design"]
    V, W = case["vocab"], case["width"]
    s = {}
    if d == "qwen3":
        H, G, F = case["heads"] * 128, case["kv_heads"] * 128, case["ff"]
        s.update({"model.embed_tokens.weight": (V, W), "lm_head.weight": (V, W), "model.norm.weight": (W,)})
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            s.update({p + "input_layernorm.weight": (W,), p + "post_attention_layernorm.weight": (W,), p + "self_attn.q_proj.weight": (H, W),
                      p + "self_attn.k_proj.weight": (G, W), p + "self_attn.v_proj.weight": (G, W), p + "self_attn.o_proj.weight": (W, H),
                      p + "self_attn.q_norm.weight": (128,), p + "self_attn.k_norm.weight": (128,), p + "mlp.gate_proj.weight": (F, W),
                      p + "mlp.up_proj.weight": (F, W), p + "mlp.down_proj.weight": (W, F)})
        return s
    s.update({"embed": (V, W), "final.norm": (W,)})
    if d != "losalorn":
        s["head"] = (V, W)
    if d == "vedizen":
        s.update({"loop.step": (cfg["loop"]["times"], W), "final.norm.b": (W,), "final.norm.alpha": ()})
    if d == "losalorn":
        s["loop.in"] = (W, 2 * W)

    def add(p, **more):
        s.update({p + n.replace("_", "."): v for n, v in more.items()})

    def delta(p, m):
        kd, vd = m["kv_heads"] * m["dim"], m["heads"] * m["vdim"]
        add(p, q=(kd, W), k=(kd, W), v=(vd, W), q_conv=(kd, m["conv"]), k_conv=(kd, m["conv"]), v_conv=(vd, m["conv"]), b=(m["heads"], W),
            norm=(m["vdim"],), o=(W, vd))
        s[p + "A_log"] = (m["heads"],)
        if d == "pogarax":
            add(p, a1=(RANK, W), a2=(m["heads"] * m["dim"], RANK), g1=(RANK, W), g2=(vd, RANK))
            s[p + "dt_bias"] = (m["heads"] * m["dim"],)
        else:
            add(p, a=(m["heads"], W), g=(vd, W))
            s[p + "dt_bias"] = (m["heads"],)

    for i, l in enumerate(cfg["layers"]):
        if "weights_of" in l:
            continue
        m, p, x, mlp = l["mixer"], f"l{i}.", f"l{i}.mix.", l["mlp"]
        add(p, norm1=(W,), norm2=(W,))
        H, G, D, Dv = (m.get(n, 0) for n in ("heads", "kv_heads", "dim", "vdim"))
        if d == "vedizen":
            del s[p + "norm2"]
            add(p, norm1_b=(W,), norm1_alpha=())
            if l["type"] == "gla":
                add(x, q=(H * D, W), k=(H * D, W), v=(H * Dv, W), g=(H * Dv, W), o=(W, H * Dv), norm=(Dv,), a1=(RANK, W), a2=(H * D, RANK), a2_b=(H * D,))
            else:
                add(x, q=(2 * H * D, W), q_b=(2 * H * D,), k=(2 * G * D, W), k_b=(2 * G * D,), v=(G * Dv, W), v_b=(G * Dv,), o=(W, H * Dv),
                    lq1=(D,), lk1=(D,), lq2=(D,), lk2=(D,))
        elif l["type"] in ("delta", "channel_delta"):
            delta(x, m)
        elif l["type"] == "latent_attention":
            R, rd = m["kv_rank"], m["rot_dim"]
            add(x, uk=(H * D, R), uv=(H * Dv, R), sink=(H,), o=(W, H * Dv))
            if "q_rank" in m:
                add(x, dq=(m["q_rank"], W), dq_norm=(m["q_rank"],), uq=(H * (D + rd), m["q_rank"]))
            else:
                add(x, q=(H * (D + rd), W), g=(H, W))
            if "kv_from" not in m:
                add(x, dkv=(R + rd, W), dkv_norm=(R,))
        elif l["type"] == "wkv":
            n = H * D
            add(x, mu_r=(W,), mu_k=(W,), mu_v=(W,), mu_g=(W,), mu_w=(W,), r=(n, W), k=(n, W), v=(n, W), g=(n, W), w1=(RANK, W), w2=(n, RANK),
                w0=(n,), u=(H, D), norm=(n,), o=(W, n))
        elif d == "gamanex":
            add(x, q=(H * D, W), q_norm=(H * D,), r1=(H,), r2=(H,), pb=(H,), o=(W, H * Dv))
            add(p, ls1=(W,), rg1=(W, W), rg1_b=(W,), ls2=(W,), rg2=(W, W), rg2_b=(W,))
            if "kv_from" not in m:
                add(x, k=(G * D, W), v=(G * Dv, W), k_norm=(G * D,))
        elif d == "losalorn":
            add(x, q=(H * D, W), k=(G * D, W), o=(W, H * D))
        elif d == "tagulix" and l["type"] == "attention":
            add(x, q=(H * D, W), q_b=(H * D,), k=(G * D, W), k_b=(G * D,), v=(G * Dv, W), v_b=(G * Dv,), o=(W, H * Dv), o_b=(W,))
        elif d == "tagulix":
            a, r = m["left"], m["right"]
            H, G, D, Dv = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
            add(x + "left.", q=(H * D, W), k=(G * D, W), v=(G * Dv, W), o=(W, H * Dv), q_norm=(D,), k_norm=(D,), rel=(REL, H), sink=(H,))
            n, v = r["heads"] * r["dim"], r["heads"] * r["vdim"]
            add(x + "right.", q=(n, W), k=(n, W), v=(v, W), g=(v, W), o=(W, v), norm=(v,))
        else:                                           # Pirerax
            y, a = (x, m) if l["type"] == "attention" else (x + "left.", m["left"])
            H, G, D, Dv = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
            add(y, q=(H * D, W), k=(G * D, W), v=(G * Dv, W), q_norm=(H * D,), k_norm=(G * D,), g=(H * Dv, W), o=(W, H * Dv))
            if l["type"] == "attention":
                add(x, sink=(H,))
            else:
                delta(x + "right.", m["right"])
                add(x, left_out=(W,), right_out=(W,))
        if d == "tagulix":
            S = cfg["streams"]
            for q in ("hc1", "hc2"):
                add(p + q + ".", **{"in": (S,), "out": (S,), "mix": (S, S)})
        if d == "losalorn":
            add(p, norm1b=(W,), norm2b=(W,))
        if mlp["kind"] == "dense":
            add(p + "mlp.", up=(mlp["ff"], W), down=(W, mlp["ff"]))
            if d != "gamanex":
                add(p + "mlp.", gate=(mlp["ff"], W))
            continue
        r, ff = mlp["router"], mlp["expert"]["ff"]
        n = r["experts"] + r.get("identity", 0)
        add(p + "mlp.", router=(n, W))
        if d == "gamanex":
            add(p + "mlp.", router_b=(n,))
        if d == "tagulix":
            add(p + "mlp.", correction=(n,))
        for e in range(r["experts"]):
            add(f"{p}mlp.e{e}.", up=(ff, W), down=(W, ff))
            if d != "tagulix":
                add(f"{p}mlp.e{e}.", gate=(ff, W))
    return s


def _routing_codes(case, outputs, groups, g):
    """[vocab, outputs]: every token's own order of the router's outputs as evenly spaced levels.  Trained routers are
    sure of most tokens; random ones are not, and a choice that a rounding can tip says nothing about a kernel.  The
    levels are dealt to the groups in turn, so groups are as clearly ordered as their members."""
    V, per = case["vocab"], outputs // groups
    group = torch.rand((V, groups), generator=g, device="cuda").argsort(dim=1)
    inside = torch.rand((V, groups, per), generator=g, device="cuda").argsort(dim=2)
    rank = inside * groups + group[:, :, None]
    return 1.7 - 3.4 / (outputs - 1) * rank.reshape(V, outputs).float()


def weights_of(case, seed):
    """Tensors on the GPU in bfloat16, large enough that every mechanism moves the logits: matrices N(0, 1 / fan in),
    norm weights near 1.  Where experts are routed, the first channels of the residual carry each token's preferences
    (nothing else writes there) and the routers read them."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    d, cfg = case["design"], config_of(case)
    routers = [l["mlp"]["router"] for l in cfg.get("layers", ()) if l["mlp"]["kind"] == "moe"]
    n = routers[0]["experts"] + routers[0].get("identity", 0) if routers else 0
    out = {}
    for name, shape in shapes_of(case).items():
        leaf = name.rsplit(".", 1)[-1]
        t = torch.empty(shape, device="cuda", dtype=torch.float32 if len(shape) < 2 else torch.bfloat16)

        def normal(std, mean=0.0, t=t):
            return t.normal_(mean, std, generator=g)

        if leaf == "conv":
            normal(0.6)
        elif leaf == "mix":
            normal(0.1)
            t += 0.6 * torch.eye(shape[0], device="cuda") + 0.4 * torch.roll(torch.eye(shape[0], device="cuda"), 1, 1)
        elif leaf == "rel":
            normal(1.5)
        elif leaf == "u":
            normal(0.5)
        elif leaf == "router":
            t.zero_()
            t[range(n), range(n)] = 2.0
        elif name in ("embed", "model.embed_tokens.weight"):
            normal(case["width"] ** -0.5 if d == "losalorn" else 1.0)       # Losalorn's table is its head as well
            if n:
                t[:, :n] = _routing_codes(case, n, (routers[0].get("groups") or dict(count=1))["count"], g)
        elif len(shape) == 2 and leaf != "step":
            normal(shape[1] ** -0.5)
            if n and leaf in ("o", "down"):
                t[:n] = 0.0
        elif leaf in ("in", "out") and shape == (cfg.get("streams"),):
            normal(0.3, shape[0] ** -0.5)
        elif leaf == "alpha":
            normal(0.05, 0.6)
        elif leaf.startswith("mu") or ".mu." in name:
            t.uniform_(0.0, 1.0, generator=g)
        elif leaf in ("r1", "r2"):
            t.uniform_(0.2, 0.8, generator=g)
        elif leaf in ("ls1", "ls2"):
            normal(0.2, 0.8)
        elif leaf in ("pb", "w0"):
            normal(0.7, -2.0)
        elif leaf == "A_log":
            normal(1.0, -1.0)
        elif leaf == "sink":
            normal(1.0, 1.0)
        elif leaf == "correction" or name.endswith("router.b"):
            t.zero_()
        elif leaf in ("b", "dt_bias", "lq1", "lk1", "lq2", "lk2", "step"):
            normal(0.3)
        else:                                           # norm weights
            normal(0.2, 1.0)
        if n and shape == (case["width"],):             # what is added to, or scales, the channels of the preferences
            if d in ("gamanex", "tagulix", "pirerax") and leaf in ("norm1", "norm2"):
                t[:n] = 1.0
            elif leaf != "norm" and not leaf.startswith("mu") and ".mu." not in name:
                t[:n] = 0.0
        out[name] = t.to(torch.bfloat16)
    return out


# ----------------------------------------------------------------------------- what is measured
def prepare(case, seed):
    cfg = config_of(case)
    config_cls, builder = lookup_architecture(airun_b200.config.base.architecture_name(cfg))
    config = config_cls.from_dict(json.loads(json.dumps(cfg)))
    tensors = weights_of(case, seed)
    if hasattr(config, "with_tensor_shapes"):
        config = config.with_tensor_shapes({n: tuple(t.shape) for n, t in tensors.items()})
    model = builder(config, DTYPES[case["dtype"]], "cuda:0")
    model.load(DictSource(tensors))
    del tensors
    lengths = _lengths(case)
    longest = max(c + p for c, p in lengths) + case["steps"] + 1
    engine = Engine(config, model, EngineOptions(
        dtype=DTYPES[case["dtype"]], page_size=16, max_requests=2 * case["requests"], max_batch_tokens=2048,
        max_context=max(2048, -(-longest // 1024) * 1024),
        cache_tokens=sum(c + 2 * (p + case["steps"]) + 64 for c, p in lengths) + 4096))
    tokens = _tokens(case, seed)
    for i, (c, _) in enumerate(lengths):                # the contexts, in portions as a server would bring them
        for at in range(0, c, 2048):
            if at == 0:
                engine.manager.add_request(i)
            engine.runner.step([StepEntry(i, tokens[i][at:min(c, at + 2048)])])
    state = dict(engine=engine, lengths=lengths, tokens=_tokens(case, seed + 1_000_003), steps=case["steps"])
    for _ in range(3):                                  # a server that has met steps of these shapes before
        run(state)
    state["tokens"] = tokens
    return state


def run(state):
    engine, steps = state["engine"], state["steps"]
    runner, manager = engine.runner, engine.manager
    rids = []
    for i, (c, _) in enumerate(state["lengths"]):
        rid = i
        if c == 0:
            manager.add_request(i)
        elif not manager.can_rewind:
            rid = ("fork", i)
            engine.storage.run_copies(manager.fork(i, rid))
        rids.append(rid)
    out = []
    for k in range(steps + 1):
        entries = []
        for rid, (c, p), t in zip(rids, state["lengths"], state["tokens"]):
            new = t[c:c + p] if k == 0 else t[c + p + k - 1:c + p + k]
            entries.append(StepEntry(rid, new, (len(new) - 1,)))
        out.append(runner.step(entries).clone())        # the step's own buffer holds until the next step
    for rid, (c, _) in zip(rids, state["lengths"]):
        if c == 0 or not manager.can_rewind:
            manager.free_request(rid)
        else:
            engine.storage.run_copies(manager.truncate(rid, c))
    logits = torch.stack(out, 1)                        # [requests, steps, vocabulary]
    return {"first": logits[0], "others": logits[1:]} if len(rids) > 1 else {"first": logits[0]}


def work(case):
    """Bytes: the weights a step needs (of the experts those its tokens can reach), once for every step, the cached rows its
    tokens see and the logits.  Operations: the products with the weights, and the attention's and the recurrences'."""
    cfg, shapes, esz = config_of(case), shapes_of(case), 2 if case["dtype"] == "bf16" else 4
    layers = cfg.get("layers") or [None] * case["layers"]
    runs = {}
    for i, _, _ in _runs(dict(cfg, layers=layers)):
        src = (layers[i] or {}).get("weights_of", i)
        runs[src] = runs.get(src, 0) + 1
    sizes = [(c, p) for c, p in _lengths(case)]
    count, bytes_, flops = len(sizes), 0.0, 0.0
    for k in range(case["steps"] + 1):
        new = [p if k == 0 else 1 for _, p in sizes]
        T = sum(new)
        for name, shape in shapes.items():
            if len(shape) != 2 or name in ("embed", "model.embed_tokens.weight") and case["design"] != "losalorn":
                continue
            n, parts = shape[0] * shape[1], name.split(".")
            if "head" in name or name == "embed":
                bytes_, flops = bytes_ + n * esz, flops + 2.0 * n * count
                continue
            i = int(parts[2]) if parts[0] == "model" else int(parts[0][1:]) if parts[0][1:].isdigit() else None
            times = runs.get(i, 1)
            if i is not None and len(parts) == 4 and parts[2][0] == "e" and parts[2][1:].isdigit():
                r = layers[i]["mlp"]["router"]
                flops += 2.0 * n * T * r["top"] / (r["experts"] + r.get("identity", 0)) * times
                bytes_ += n * esz * times * min(1.0, T * r["top"] / r["experts"])
            else:
                flops += 2.0 * n * T * times
                bytes_ += n * esz * times
        for i, _, _ in _runs(dict(cfg, layers=layers)):
            for kind, m in _mixers(case, layers[i]):
                for (c, p), q in zip(sizes, new):
                    first = c if k == 0 else c + p + k - 1
                    if kind == "state":
                        flops += 4.0 * q * m[0]
                        bytes_ += 8.0 * m[0]
                    else:                               # key and value elements of a token over all heads, cached row, window
                        pairs = q * first + q * (q + 1) / 2.0
                        if m[2]:
                            pairs = min(pairs, q * float(m[2]))
                        flops += 2.0 * m[0] * pairs
                        bytes_ += (min(first, m[2] or first) + q) * m[1] * esz
        bytes_ += 4.0 * count * case["vocab"]
    return {"bytes": bytes_, "flops": flops}


def _mixers(case, layer):
    """[("state", (elements,)) or ("pages", (multiply-adds of a query-key pair, cached elements of a token, window))]"""
    if layer is None:
        return [("pages", (256 * case["heads"], 256 * case["kv_heads"], 0))]
    m = layer["mixer"]
    if "left" in m:
        return _mixers(case, dict(mixer=m["left"])) + [("state", (m["right"]["heads"] * m["right"]["dim"] * m["right"]["vdim"],))]
    window = (m.get("mask") or {}).get("size", 0)
    if "kv_rank" in m:
        return [("pages", (m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), m["kv_rank"] + m["rot_dim"], window))]
    if layer.get("type") in ("gla", "delta", "channel_delta", "wkv"):
        return [("state", (m["heads"] * m["dim"] * m.get("vdim", m["dim"]),))]
    maps = 2 if "diff" in m else 1
    return [("pages", (m["heads"] * maps * (m["dim"] + m["vdim"]), m["kv_heads"] * (maps * m["dim"] + m["vdim"]), window))]


def tolerance(case):
    """About four times what is seen: logits in bfloat16 stand 0.002 to 0.008 off the 64-bit result (their roundings go
    through up to 36 layers), and two correct ones differ by up to 1.4 times that; 32-bit sums stand 1.4e-6 off it."""
    if case["dtype"] == "fp32":
        return {"rel": 8e-6, "max": 1e-4}
    return {"rel": 0.03, "max": 0.3}


# ----------------------------------------------------------------------------- the same in 64 bits
EXACT_FLOPS = 1.2e14                                    # of plain 64-bit products: about ten seconds on the GPU


def exact(case, seed):
    """All requests, or the first alone where all of them would take too long."""
    lengths, tokens = _lengths(case), _tokens(case, seed)
    one = work(dict(case, context=0, portion=1, portions=0, requests=1, steps=0))["flops"]
    cost = [len(t) * (one + 12.0 * case["width"] * len(t) * len(config_of(case).get("layers", range(case["layers"])))) for t in tokens]
    take = len(tokens) if sum(cost) < EXACT_FLOPS else 1
    if cost[0] > EXACT_FLOPS:
        return None
    ids = torch.zeros((take, max(len(t) for t in tokens[:take])), dtype=torch.long)
    for i, t in enumerate(tokens[:take]):
        ids[i, :len(t)] = torch.tensor(t)               # the places behind a shorter request's tokens are never read
    last = torch.tensor([c + p - 1 for c, p in lengths[:take]], device="cuda")
    x, head = Plain(config_of(case), case, weights_of(case, seed)).forward(ids.cuda(), last[:, None] + torch.arange(case["steps"] + 1, device="cuda"))
    logits = head(x)
    out = {"first": logits[0]}
    if len(tokens) > 1:
        out["others"] = logits[1:] if take > 1 else None
    return out


def _rms(x, eps, w=None):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _silu(z):
    return z * torch.sigmoid(z)


def _clamped(g, u, limit):
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


class Plain:
    """The seven decoders on whole sequences [requests, tokens], without a cache, in 64 bits."""

    def __init__(self, cfg, case, W):
        self.cfg, self.case, self.W = cfg, case, W
        self.eps = cfg["rms_norm_eps"] if "rms_norm_eps" in cfg else cfg["norm"]["eps"]

    def w(self, name):
        return self.W[name].double()

    def lin(self, x, name):
        return x @ self.w(name).T

    def heads(self, x, name, n):
        y = self.lin(x, name)
        if name + ".b" in self.W:
            y = y + self.w(name + ".b")
        return y.unflatten(-1, (n, -1))

    def forward(self, ids, places):
        """Returns (the normed stream at ``places`` [requests, n], the head)."""
        self.pos = torch.arange(ids.shape[1], device="cuda", dtype=torch.float64)
        self.behind = self.pos[:, None] - self.pos[None, :]
        self.ids, self.places = ids, places[..., None]
        return getattr(self, "_" + self.case["design"])()

    def at(self, x):
        return x.gather(1, self.places.expand(-1, -1, x.shape[-1]))

    # ---- pieces
    def angles(self, freqs, mult=1.0):
        a = self.pos[:, None] * torch.tensor(freqs, device="cuda", dtype=torch.float64)
        return torch.cos(a) * mult, torch.sin(a) * mult

    def turn(self, x, tables, near=False):
        """x [.., tokens, heads, n]: the pairs (i, i + half), or neighbours, of the first dimensions turned."""
        c, s = (t[:, None, :] for t in tables)
        n = c.shape[-1]
        a, b = (x[..., 0:2 * n:2], x[..., 1:2 * n:2]) if near else (x[..., :n], x[..., n:2 * n])
        u, v = a * c - b * s, b * c + a * s
        turned = torch.stack((u, v), -1).flatten(-2) if near else torch.cat((u, v), -1)
        return torch.cat((turned, x[..., 2 * n:]), -1)

    def temperature(self, m):
        t = m.get("q_temp")
        return 1.0 if not t else (1.0 + t["coef"] * torch.log(torch.floor((self.pos + 1.0) / t["every"]) + 1.0))[:, None, None]

    def seen(self, window=0, chunk=0):
        ok = self.behind >= 0
        if window:
            ok = ok & (self.behind < window)
        if chunk:
            ok = ok & (torch.floor(self.pos[:, None] / chunk) == torch.floor(self.pos[None, :] / chunk))
        return ok

    def attend(self, q, k, v, scale, ok, bias=None, sink=None, cap=0.0):
        """q [B, T, heads, D], k and v [B, T, KV heads, ..]; ``sink`` [heads]: one more term exp(sink) in the denominator."""
        H, G = q.shape[2], k.shape[2]
        out = q.new_empty(q.shape[:3] + (v.shape[-1],))
        for h in range(H):
            s = (q[:, :, h] @ k[:, :, h * G // H].transpose(1, 2)) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            if bias is not None:
                s = s + bias(h)
            s = s.masked_fill(~ok, -math.inf)
            top = s.amax(-1, keepdim=True)
            if sink is not None:
                top = top.clamp(min=float(sink[h]))
            e = torch.exp(s - top)
            den = e.sum(-1, keepdim=True)
            if sink is not None:
                den = den + torch.exp(sink[h] - top)
            out[:, :, h] = (e / den) @ v[:, :, h * G // H]
        return out

    def walk(self, q, k, v, step):
        """A recurrence over the tokens: ``step(S, t)`` returns the new state and what is read, S [B, heads, D, Dv]."""
        S = q.new_zeros((q.shape[0], q.shape[2], k.shape[-1], v.shape[-1]))
        out = v.new_empty(q.shape[:3] + (v.shape[-1],))
        for t in range(q.shape[1]):
            S, out[:, t] = step(S, t)
        return out

    @staticmethod
    def read(S, q):
        return (S * q[..., None]).sum(-2)

    def conv(self, x, name):
        w, y = self.w(name), torch.zeros_like(x)
        taps = w.shape[1]
        for j in range(taps):
            back = taps - 1 - j
            y[:, back:] += w[:, j] * x[:, :x.shape[1] - back]
        return _silu(y)

    def delta(self, h, p, m, per_channel):
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        q, k, v = (self.conv(self.lin(h, p + n), p + n + ".conv") for n in "qkv")
        unit = lambda x: (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 2)   # noqa: E731
        q, k, v = unit(q.unflatten(-1, (G, D))) * D ** -0.5, unit(k.unflatten(-1, (G, D))), v.unflatten(-1, (H, -1))
        beta = torch.sigmoid(self.lin(h, p + "b"))[..., None]
        z = self.lin(self.lin(h, p + "a1"), p + "a2") if per_channel else self.lin(h, p + "a")
        soft = torch.nn.functional.softplus(z + self.w(p + "dt_bias")).unflatten(-1, (H, -1))
        g = torch.exp(-torch.exp(self.w(p + "A_log"))[:, None] * soft)[..., None]       # [B, T, H, D or 1, 1]

        def step(S, t):
            S = g[:, t] * S
            u = beta[:, t] * (v[:, t] - self.read(S, k[:, t]))
            S = S + k[:, t, :, :, None] * u[:, :, None, :]
            return S, self.read(S, q[:, t])

        o = _rms(self.walk(q, k, v, step), self.eps, self.w(p + "norm"))
        gate = torch.sigmoid(self.lin(self.lin(h, p + "g1"), p + "g2")) if per_channel else _silu(self.lin(h, p + "g"))
        return self.lin(o.flatten(2) * gate, p + "o")

    def latent(self, h, p, m, rows, tables, near):
        H, D, R = m["heads"], m["dim"], m["kv_rank"]
        q = (self.heads(_rms(self.lin(h, p + "dq"), self.eps, self.w(p + "dq.norm")), p + "uq", H) if "q_rank" in m else self.heads(h, p + "q", H))
        c, kr = rows
        q = torch.cat((q[..., :D], self.turn(q[..., D:], tables, near)), -1)
        k = torch.cat((self.heads(c, p + "uk", H), kr.expand(-1, -1, H, -1)), -1)
        o = self.attend(q, k, self.heads(c, p + "uv", H), m["scale"], self.seen((m.get("mask") or {}).get("size", 0)), sink=self.w(p + "sink"))
        if p + "g" in self.W:
            o = o * torch.sigmoid(self.lin(h, p + "g"))[..., None]
        return self.lin(o.flatten(2), p + "o")

    def latent_rows(self, h, p, m, tables, near):
        d = self.lin(h, p + "dkv")
        return _rms(d[..., :m["kv_rank"]], self.eps, self.w(p + "dkv.norm")), self.turn(d[..., None, m["kv_rank"]:], tables, near)

    def experts(self, h, p, r, weights, ids, unit):
        """``weights``, ``ids`` [B, T, top]; ``unit(rows, expert, weight)`` is what an expert returns for its rows."""
        out, flat = torch.zeros_like(h), h.flatten(0, 1)
        acc = out.flatten(0, 1)
        for e in range(r["experts"]):
            rows, slot = (ids.flatten(0, 1) == e).nonzero(as_tuple=True)
            if len(rows):
                acc.index_add_(0, rows, unit(flat[rows], f"{p}e{e}.", weights.flatten(0, 1)[rows, slot][:, None]))
        return out

    def best(self, scores, value, top, groups, strength):
        """The ``top`` outputs of the best groups by ``value``."""
        n, keep = groups["count"], groups["keep"]
        kept = strength(scores.unflatten(-1, (n, -1))).topk(keep, -1).indices
        ok = torch.zeros(scores.shape[:-1] + (n,), device="cuda", dtype=torch.bool).scatter_(-1, kept, True)
        return value.masked_fill(~ok.repeat_interleave(scores.shape[-1] // n, -1), -math.inf).topk(top, -1).indices

    # ---- the designs
    def _qwen3(self):
        c, H, G = self.case, self.case["heads"], self.case["kv_heads"]
        tables = self.angles([1e6 ** (-2.0 * i / 128) for i in range(64)])
        x, ok = self.w("model.embed_tokens.weight")[self.ids], self.seen()
        for i in range(c["layers"]):
            p = f"model.layers.{i}."
            a = p + "self_attn."
            h = _rms(x, self.eps, self.w(p + "input_layernorm.weight"))
            q = self.turn(_rms(self.heads(h, a + "q_proj.weight", H), self.eps, self.w(a + "q_norm.weight")), tables)
            k = self.turn(_rms(self.heads(h, a + "k_proj.weight", G), self.eps, self.w(a + "k_norm.weight")), tables)
            o = self.attend(q, k, self.heads(h, a + "v_proj.weight", G), 128 ** -0.5, ok)
            x = x + self.lin(o.flatten(2), a + "o_proj.weight")
            h = _rms(x, self.eps, self.w(p + "post_attention_layernorm.weight"))
            x = x + self.lin(_silu(self.lin(h, p + "mlp.gate_proj.weight")) * self.lin(h, p + "mlp.up_proj.weight"), p + "mlp.down_proj.weight")
        return _rms(self.at(x), self.eps, self.w("model.norm.weight")), lambda y: self.lin(y, "lm_head.weight")

    def _vedizen(self):
        squash = lambda x, p: torch.tanh(self.w(p + ".alpha") * x) * self.w(p) + self.w(p + ".b")   # noqa: E731
        x = self.w("embed")[self.ids]
        for i, begins, t in _runs(self.cfg):
            l, p = self.cfg["layers"][i], f"l{i}.mix."
            m, f = l["mixer"], f"l{i}.mlp."
            if begins:
                x = x + self.w("loop.step")[t]
            h, H, D = squash(x, f"l{i}.norm1"), m["heads"], m["dim"]
            if l["type"] == "gla":
                q, k, v = self.heads(h, p + "q", H) * D ** -0.5, self.heads(h, p + "k", H), self.heads(h, p + "v", H)
                z = self.lin(self.lin(h, p + "a1"), p + "a2") + self.w(p + "a2.b")
                a = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).unflatten(-1, (H, D))[..., None]

                def step(S, t, q=q, k=k, v=v, a=a):
                    S = a[:, t] * S + k[:, t, :, :, None] * v[:, t, :, None, :]
                    return S, self.read(S, q[:, t])

                o = _rms(self.walk(q, k, v, step), self.eps, self.w(p + "norm"))
                y = self.lin(o.flatten(2) * _silu(self.lin(h, p + "g")), p + "o")
            else:
                dot = lambda n: math.exp(float((self.w(p + "lq" + n) * self.w(p + "lk" + n)).sum()))   # noqa: E731
                q, k, v = self.heads(h, p + "q", 2 * H), self.heads(h, p + "k", 2 * m["kv_heads"]), self.heads(h, p + "v", m["kv_heads"])
                one, two = (self.attend(q[:, :, n::2], k[:, :, n::2], v, m["scale"], self.seen(chunk=m["mask"]["size"]), cap=m["softcap"])
                            for n in (0, 1))
                o = _rms(one - (dot("1") - dot("2") + m["diff"]) * two, self.eps) * (1.0 - m["diff"])
                y = self.lin(o.flatten(2), p + "o")
            x = x + y + self.lin(_clamped(self.lin(h, f + "gate"), self.lin(h, f + "up"), l["mlp"]["limit"]), f + "down")
        return squash(self.at(x), "final.norm"), lambda y: self.lin(y, "head")

    def _pogarax(self):
        mult, rows = self.cfg["residual_mult"], {}
        x = self.w("embed")[self.ids]
        for i, l in enumerate(self.cfg["layers"]):
            m, p, f = l["mixer"], f"l{i}.mix.", f"l{i}.mlp."
            if l["type"] == "channel_delta":
                y = self.delta(x, p, m, True)
            elif l["type"] == "latent_attention":
                r = m["rot"]
                tables = self.angles(*_stretched(r["dims"], r["base"], **r["scaling"]))
                if "kv_from" not in m:
                    rows[i] = self.latent_rows(x, p, m, tables, True)
                y = self.latent(x, p, m, rows[m.get("kv_from", i)], tables, True)
            else:
                H = m["heads"]
                before = torch.cat((torch.zeros_like(x[:, :1]), x[:, :-1]), 1)
                mix = {n: x + (before - x) * self.w(p + "mu." + n) for n in "rkvgw"}
                r, k, v = (self.heads(mix[n], p + n, H) for n in "rkv")
                w = torch.exp(-torch.exp(self.lin(torch.tanh(self.lin(mix["w"], p + "w1")), p + "w2") + self.w(p + "w0"))).unflatten(-1, (H, -1))
                u = self.w(p + "u")[..., None]

                def step(S, t, r=r, k=k, v=v, w=w, u=u):
                    kv = k[:, t, :, :, None] * v[:, t, :, None, :]
                    return w[:, t, :, :, None] * S + kv, self.read(S + u * kv, r[:, t])

                o = _rms(self.walk(r, k, v, step), self.eps).flatten(2) * self.w(p + "norm") * _silu(self.lin(mix["g"], p + "g"))
                y = self.lin(o, p + "o")
            x = x + mult * _rms(y, self.eps, self.w(f"l{i}.norm1"))
            unit = lambda h, e: self.lin(_silu(self.lin(h, e + "gate")) * self.lin(h, e + "up"), e + "down")   # noqa: E731
            if l["mlp"]["kind"] == "dense":
                y = unit(x, f)
            else:
                r = l["mlp"]["router"]
                val, ids = torch.sigmoid(self.lin(x, f + "router")).topk(r["top"], -1)
                y = self.experts(x, f, r, val, ids, lambda h, e, s: unit(s * h, e))
            x = x + mult * _rms(y, self.eps, self.w(f"l{i}.norm2"))
        return _rms(self.at(x), self.eps, self.w("final.norm")), lambda y: self.lin(y, "head")

    def _gamanex(self):
        x, kept, ok = self.w("embed")[self.ids], {}, self.seen()
        for i, l in enumerate(self.cfg["layers"]):
            m, p, f = l["mixer"], f"l{i}.mix.", f"l{i}.mlp."
            H, G = m["heads"], m["kv_heads"]
            h, h2 = (_rms(x, self.eps, self.w(f"l{i}.norm{n}")) for n in (1, 2))
            if "kv_from" not in m:
                kept[i] = _rms(self.lin(h, p + "k"), self.eps, self.w(p + "k.norm")).unflatten(-1, (G, -1)), self.heads(h, p + "v", G)
            k, v = kept[m.get("kv_from", i)]
            q = _rms(self.lin(h, p + "q"), self.eps, self.w(p + "q.norm")).unflatten(-1, (H, -1)) * self.temperature(m)
            a, b, c = (self.w(p + n) for n in ("r1", "r2", "pb"))
            o = torch.empty_like(q)
            for n in range(H):
                s = (q[:, :, n] @ k[:, :, n * G // H].transpose(1, 2)) * m["scale"] - a[n] * torch.log1p(b[n] * self.behind.clamp(min=0)) + c[n]
                o[:, :, n] = (torch.sigmoid(s) * ok) @ v[:, :, n * G // H]
            y = self.lin(o.flatten(2), p + "o")
            if l["mlp"]["kind"] == "dense":
                z = self.lin(torch.relu(self.lin(h2, f + "up")) ** 2, f + "down")
            else:
                r = l["mlp"]["router"]
                val, ids = (self.lin(h2, f + "router") + self.w(f + "router.b")).topk(r["top"], -1)
                z = self.experts(h2, f, r, torch.softmax(val, -1), ids, lambda g, e, s: s * self.lin(
                    _silu(self.lin(g, e + "gate")) * self.lin(g, e + "up"), e + "down"))
            gate = lambda g, n: self.w(f"l{i}.ls{n}") * torch.sigmoid(self.lin(g, f"l{i}.rg{n}") + self.w(f"l{i}.rg{n}.b"))   # noqa: E731
            x = x + gate(h, 1) * y + gate(h2, 2) * z
        return _rms(self.at(x), self.eps, self.w("final.norm")), lambda y: self.lin(y, "head") * self.cfg["logit_scale"]

    def _tagulix(self):
        cfg = self.cfg
        S, mult = cfg["streams"], cfg["residual_mult"]
        xs = self.w("embed")[self.ids][None].repeat(S, 1, 1, 1)
        for i, l in enumerate(cfg["layers"]):
            b = f"l{l.get('weights_of', i)}."
            for n, sub in ((1, self._tagulix_mixer), (2, self._tagulix_experts)):
                u = torch.einsum("s,sbtw->btw", self.w(f"{b}hc{n}.in"), xs)
                y = sub(_rms(u, self.eps, self.w(f"{b}norm{n}")), b, l)
                xs = torch.einsum("st,sbjw->tbjw", self.w(f"{b}hc{n}.mix"), xs) + mult * self.w(f"{b}hc{n}.out")[:, None, None, None] * y
        return _rms(self.at(xs.sum(0)), self.eps, self.w("final.norm")), lambda y: self.lin(y, "head")

    def _tagulix_mixer(self, h, b, l):
        m, p = l["mixer"], b + "mix."
        if l["type"] == "attention":
            H, G, r = m["heads"], m["kv_heads"], m["rot"]
            tables = self.angles([r["base"] ** (-2.0 * i / r["dims"]) for i in range(r["dims"] // 2)])
            q, k = (_rms(self.turn(self.heads(h, p + n, k), tables, True), self.eps) for n, k in (("q", H), ("k", G)))
            o = self.attend(q, k, self.heads(h, p + "v", G), m["scale"], self.seen(m["mask"]["size"]))
            return self.lin(o.flatten(2), p + "o") + self.w(p + "o.b")
        m, y, p = m["left"], p + "left.", p + "right."
        H, G = m["heads"], m["kv_heads"]
        q, k = (_rms(self.heads(h, y + n, k), self.eps, self.w(f"{y}{n}.norm")) for n, k in (("q", H), ("k", G)))
        rel, far = self.w(y + "rel"), m["bias_max"]
        half = rel.shape[0] // 2
        bucket = [n if n < half else min(rel.shape[0] - 1, half + int(math.floor(math.log(n / half) / math.log(far / half) * (rel.shape[0] - half))))
                  for n in range(self.ids.shape[1])]
        table = rel[torch.tensor(bucket, device="cuda")]                                # [distance, heads]
        near = self.behind.clamp(min=0).long()
        o = self.attend(q * self.temperature(m), k, self.heads(h, y + "v", G), m["scale"], self.seen(), bias=lambda n: table[:, n][near],
                        sink=self.w(y + "sink"))
        left = self.lin(o.flatten(2), y + "o")
        m = l["mixer"]["right"]
        q, k, v = (_silu(self.heads(h, p + n, m["heads"])) for n in "qkv")
        d = torch.tensor(m["decay"], device="cuda", dtype=torch.float64)[:, None, None]

        def step(S, t):
            S = d * S + k[:, t, :, :, None] * v[:, t, :, None, :]
            return S, self.read(S, q[:, t])

        o = _rms(self.walk(q, k, v, step).flatten(2), self.eps, self.w(p + "norm")) * torch.sigmoid(self.lin(h, p + "g"))
        return left + self.lin(o, p + "o")

    def _tagulix_experts(self, h, b, l):
        r, p = l["mlp"]["router"], b + "mlp."
        s = torch.softmax(self.lin(h, p + "router"), -1)
        c = s + self.w(p + "correction")
        ids = self.best(c, c, r["top"], r["groups"], lambda g: g.amax(-1))
        val = s.gather(-1, ids)
        val = val / (val.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        y = self.experts(h, p, r, val, ids, lambda g, e, w: w * self.lin(torch.nn.functional.gelu(self.lin(g, e + "up")), e + "down"))
        return y + (val * (ids >= r["experts"])).sum(-1, keepdim=True) * h

    def _losalorn(self):
        x0 = self.w("embed")[self.ids] * self.cfg["embedding"]["scale"]
        x = x0
        for i, begins, _ in _runs(self.cfg):
            l, p, f = self.cfg["layers"][i], f"l{i}.mix.", f"l{i}.mlp."
            m = l["mixer"]
            if begins:
                x = self.lin(torch.cat((x, x0), -1), "loop.in")
            h = _rms(x, self.eps, self.w(f"l{i}.norm1"))
            if l["type"] == "delta":
                y = self.delta(h, p, m, False)
            else:
                r, s = m["rot"], m["rot"]["scaling"]
                freqs = []
                for n in range(r["dims"] // 2):
                    q = r["base"] ** (-2.0 * n / r["dims"])
                    wave = 2.0 * math.pi / q
                    share = min(1.0, max(0.0, (s["original"] / wave - s["low"]) / (s["high"] - s["low"])))
                    freqs.append((1.0 - share) * q / s["factor"] + share * q)
                tables = self.angles(freqs)
                q, k = self.heads(h, p + "q", m["heads"]), self.heads(h, p + "k", m["kv_heads"])
                o = self.attend(self.turn(q, tables), self.turn(k, tables), k, m["scale"], self.seen(m["mask"]["size"]),
                                sink=torch.zeros(m["heads"], device="cuda", dtype=torch.float64))
                y = self.lin(o.flatten(2), p + "o")
            x = x + _rms(y, self.eps, self.w(f"l{i}.norm1b"))
            h = _rms(x, self.eps, self.w(f"l{i}.norm2"))
            y = self.lin(_clamped(self.lin(h, f + "gate"), self.lin(h, f + "up"), l["mlp"]["limit"]), f + "down")
            x = x + _rms(y, self.eps, self.w(f"l{i}.norm2b"))
        cap = self.cfg["logit_softcap"]
        return _rms(self.at(x), self.eps, self.w("final.norm")), lambda y: cap * torch.tanh(self.lin(y, "embed") / cap)

    def _pirerax(self):
        x = self.w("embed")[self.ids]
        for i, l in enumerate(self.cfg["layers"]):
            m, p, f = l["mixer"], f"l{i}.mix.", f"l{i}.mlp."
            h = _rms(x, self.eps, self.w(f"l{i}.norm1"))
            if l["type"] == "latent_attention":
                tables = self._plain_angles(m["rot"])
                y = self.latent(h, p, m, self.latent_rows(h, p, m, tables, False), tables, False)
            elif l["type"] == "attention":
                y = self._gated(h, p, m, self.w(p + "sink"))
            else:
                y = 0.5 * (_rms(self._gated(h, p + "left.", m["left"], None), self.eps, self.w(p + "left.out"))
                           + _rms(self.delta(h, p + "right.", m["right"], False), self.eps, self.w(p + "right.out")))
            x = x + y
            h, r = _rms(x, self.eps, self.w(f"l{i}.norm2")), l["mlp"]["router"]
            z = self.lin(h, f + "router")
            s = torch.sigmoid(z)
            ids = self.best(s, z, r["top"], r["groups"], lambda g: g.topk(2, -1).values.sum(-1))
            x = x + self.experts(h, f, r, s.gather(-1, ids), ids, lambda g, e, w: w * self.lin(
                _clamped(self.lin(g, e + "gate"), self.lin(g, e + "up"), l["mlp"]["expert"]["limit"]), e + "down"))
        return _rms(self.at(x), self.eps, self.w("final.norm")), lambda y: self.lin(y, "head")

    def _plain_angles(self, rot):
        return self.angles([rot["base"] ** (-2.0 * i / rot["dims"]) for i in range(rot["dims"] // 2)])

    def _gated(self, h, p, m, sink):
        H, G = m["heads"], m["kv_heads"]
        q, k = (_rms(self.lin(h, p + n), self.eps, self.w(f"{p}{n}.norm")).unflatten(-1, (c, -1)) for n, c in (("q", H), ("k", G)))
        if "rot" in m:
            tables = self._plain_angles(m["rot"])
            q, k = self.turn(q, tables), self.turn(k, tables)
        o = self.attend(q * self.temperature(m), k, self.heads(h, p + "v", G), m["scale"], self.seen(), sink=sink)
        return self.lin(o.flatten(2) * torch.sigmoid(self.lin(h, p + "g")), p + "o")


@functools.lru_cache(maxsize=8)
def _stretched(dims, base, factor, original, fast, slow):
    """(frequencies, factor of the tables): slow pairs turn ``factor`` times slower, a ramp over the pairs between."""
    def at(turns):
        return dims * math.log(original / (2 * math.pi * turns)) / (2 * math.log(base))

    lo, hi = max(math.floor(at(fast)), 0), min(math.ceil(at(slow)), dims - 1)
    out = []
    for i in range(dims // 2):
        f, ramp = base ** (-2.0 * i / dims), min(1.0, max(0.0, (i - lo) / max(hi - lo, 0.001)))
        out.append(f / factor * ramp + f * (1.0 - ramp))
    return out, 0.1 * math.log(factor) + 1.0
