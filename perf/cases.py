"""What the library's speed is measured on: the work that a program has it do, through the calls
that a program makes (``Engine.step`` for whole models, a part's ``forward`` for single layers,
``DeviceSampler.pick`` for the choice of tokens).

``listed`` names the cases, ``draw`` gives more of the same ranges, ``prepare`` makes what a
program has in hand before the call, ``run`` is one pass, ``work`` the bytes and operations that a
pass cannot do without, ``tolerance`` how far two right answers may lie apart, ``exact`` the
answer in 64 bits by plain torch.
"""
import math
import random

import torch

from mormot2_ai_b200 import DecoderModel, Engine, Entry, PartSpec, Qwen3Config, Runtime, Sampling
from mormot2_ai_b200.cache.pages import PAGE, CacheBook, pages_for, plan_groups
from mormot2_ai_b200.cache.storage import CacheStorage
from mormot2_ai_b200.engine.batch import StepBuffers
from mormot2_ai_b200.parts import FEED_FORWARDS, MIXERS, POSITIONS
from mormot2_ai_b200.parts.block import settle
from mormot2_ai_b200.sampling import DeviceSampler

DEV = "cuda:0"
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}

# Qwen3 shapes: width, heads, KV heads, head size, feed-forward size, tied head
MODELS = {"0.6B": (1024, 16, 8, 128, 3072, True),
          "8B": (4096, 32, 8, 128, 12288, False),
          "32B": (5120, 64, 8, 128, 25600, False)}
VOCAB, THETA, EPS = 151936, 1e6, 1e-6
RESIDUAL = 0.02           # spread of the residual that a single layer adds to: an embedding's rows

# mixers with a state per head, at the layer sizes of the two measured models of their families:
# width, heads, q/k heads, key size, value size
STATES = {"delta": {"small": (1024, 8, 4, 64, 128), "mid": (2048, 16, 8, 128, 128)},
          "gla": {"small": (1024, 8, 8, 64, 128), "mid": (2048, 16, 16, 128, 128)},
          "mlstm": {"small": (1024, 4, 4, 64, 64), "mid": (2048, 8, 8, 128, 128)},
          "wkv": {"small": (1024, 16, 16, 64, 64), "mid": (2048, 32, 32, 64, 64)}}
TAPS, TAU, GLA_RANK, WKV_RANK, CAP = 4, 16.0, 32, 64, 15.0

# routed experts: width, experts, chosen, feed-forward of an expert, of the shared one
EXPERTS = {"small": (1024, 16, 2, 1024, 1024), "mid": (2048, 64, 6, 1408, 2816)}

# latent attention: width, heads, key size, rotated part, value size, KV rank, q rank
LATENTS = {"small": (1024, 8, 64, 32, 64, 256, 384), "mid": (2048, 16, 128, 64, 128, 512, 768)}

SAMPLERS = {"greedy": {}, "temperature": {"temperature": 0.7},
            "top_k": {"temperature": 1.0, "top_k": 50},
            "top_p": {"temperature": 0.7, "top_p": 0.9},
            "min_p": {"temperature": 1.0, "min_p": 0.05}}


# ---------------------------------------------------------------------------- the cases
def listed():
    return [
        # one user who chats with an 8B model: every token of the answer is such a step
        dict(name="decode_8b_b1", kind="decode", model="8B", layers=2, dtype="bfloat16",
             count=1, lo=511, hi=511),
        # a server's full batch in the middle of its answers, every sequence at a length of its own
        dict(name="decode_8b_b64", kind="decode", model="8B", layers=2, dtype="bfloat16",
             count=64, lo=300, hi=2303),
        # the true 32-bit path decoding a small batch (checks of a trace against a reference)
        dict(name="decode_f32_b8", kind="decode", model="0.6B", layers=4, dtype="float32",
             count=8, lo=200, hi=1500),
        # the first step of a few short questions: latency and launches are all of it
        dict(name="prefill_short", kind="prefill", model="8B", layers=4, dtype="bfloat16",
             count=3, lo=5, hi=17),
        # a layer's share of the headline prefill, one prompt of 2,048 tokens
        dict(name="layer_8b_2048", kind="layer", model="8B", dtype="bfloat16",
             count=1, lo=2048, hi=2048),
        # a layer's share of a batch of 64 unequal prompts on the 0.6B model, in one step
        dict(name="layer_0p6b_ragged", kind="layer", model="0.6B", dtype="bfloat16",
             count=64, lo=16, hi=1887),
        # a layer of the 32-bit path over a few unequal prompts
        dict(name="layer_f32_ragged", kind="layer", model="0.6B", dtype="float32",
             count=3, lo=129, hi=1023),
        # the choice of the next token of eight sequences among the 8B model's vocabulary
        dict(name="sample_top_p", kind="sample", how="top_p", rows=8, vocab=VOCAB),
        # the gated delta rule with its convolutions over one long prompt
        dict(name="delta_2048", kind="state", mixer="delta", size="mid", count=1, lo=2048, hi=2048),
        # the matrix memory with exponential gates over four unequal prompts
        dict(name="mlstm_ragged", kind="state", mixer="mlstm", size="mid", count=4, lo=111, hi=900),
        # routed experts in a decode step of eight sequences
        dict(name="experts_8", kind="experts", size="mid", tokens=8),
        # latent attention over one long prompt
        dict(name="latent_2048", kind="latent", size="mid", count=1, lo=2048, hi=2048),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode_f32", "prefill", "layer", "layer", "layer_f32",
                       "sample", "state", "state", "experts", "latent"))
    if kind == "decode":
        model = rng.choice(("0.6B", "8B", "32B"))
        count = _log_int(rng, 1, 64)
        hi = _log_int(rng, 40, min(4000, 80000 // count))
        return dict(kind="decode", model=model, layers=rng.randint(1, 2 if model == "32B" else 3),
                    dtype="bfloat16", count=count, lo=rng.randint(max(1, hi // 4), hi), hi=hi)
    if kind == "decode_f32":
        hi = _log_int(rng, 40, 1500)
        return dict(kind="decode", model="0.6B", layers=rng.randint(1, 4), dtype="float32",
                    count=_log_int(rng, 1, 8), lo=rng.randint(max(1, hi // 4), hi), hi=hi)
    if kind == "prefill":
        hi = _log_int(rng, 2, 300)
        return dict(kind="prefill", model=rng.choice(("0.6B", "8B")), layers=rng.randint(1, 4),
                    dtype="bfloat16", count=_log_int(rng, 1, 8), lo=rng.randint(1, hi), hi=hi)
    if kind == "layer":
        model = rng.choice(("0.6B", "8B", "32B"))
        most = {"0.6B": 32768, "8B": 6000, "32B": 2500}[model]
        hi = _log_int(rng, 60, min(4000, most))
        count = _log_int(rng, 1, max(1, min(64, most // hi)))
        return dict(kind="layer", model=model, dtype="bfloat16", count=count,
                    lo=rng.randint(max(2, hi // 8), hi), hi=hi)
    if kind == "layer_f32":
        hi = _log_int(rng, 20, 1000)
        return dict(kind="layer", model="0.6B", dtype="float32", count=rng.randint(1, 3),
                    lo=rng.randint(max(2, hi // 8), hi), hi=hi)
    if kind == "sample":
        return dict(kind="sample", how=rng.choice(sorted(SAMPLERS)), rows=_log_int(rng, 1, 64),
                    vocab=rng.choice((VOCAB, 32768, _log_int(rng, 1000, VOCAB))))
    if kind == "state":
        hi = _log_int(rng, 20, 2048)
        return dict(kind="state", mixer=rng.choice(sorted(STATES)),
                    size=rng.choice(("small", "mid")), count=_log_int(rng, 1, 8),
                    lo=rng.randint(max(1, hi // 8), hi), hi=hi)
    if kind == "experts":
        return dict(kind="experts", size=rng.choice(("small", "mid")), tokens=_log_int(rng, 1, 2048))
    hi = _log_int(rng, 100, 2048)
    return dict(kind="latent", size=rng.choice(("small", "mid")), count=_log_int(rng, 1, 4),
                lo=rng.randint(hi // 4, hi), hi=hi)


def lengths(case):
    """The sequences' lengths: from ``lo`` to ``hi`` in even steps, in an order of no account."""
    n, lo, hi = case["count"], case["lo"], case["hi"]
    out = [hi if n == 1 else lo + (hi - lo) * i // (n - 1) for i in range(n)]
    random.Random(n).shuffle(out)
    return out


# ---------------------------------------------------------------------------- inputs
class Values:
    """Seeded values on the device, drawn in the order in which they are asked for."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(seed)

    def normal(self, shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        t = torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, 1.0, generator=self.gen)
        return t.mul_(std).add_(mean)

    def uniform(self, shape, lo, hi, dtype=torch.float32):
        return torch.empty(shape, dtype=dtype, device=DEV).uniform_(lo, hi, generator=self.gen)

    def ids(self, n, below):
        return torch.randint(0, below, (n,), generator=self.gen, device=DEV).tolist()


def _qwen3_weights(v, model, layers, vocab, dtype):
    """A Qwen3 checkpoint's tensors by their names."""
    w, nh, nkv, hd, ff, tied = MODELS[model]
    out = {"model.embed_tokens.weight": v.normal((vocab, w), 0.02, dtype=dtype),
           "model.norm.weight": v.normal((w,), 0.1, 1.0, dtype)}
    if not tied:
        out["lm_head.weight"] = v.normal((vocab, w), 0.02, dtype=dtype)
    for i in range(layers):
        p = f"model.layers.{i}."
        for name, shape in (("self_attn.q_proj", (nh * hd, w)), ("self_attn.k_proj", (nkv * hd, w)),
                            ("self_attn.v_proj", (nkv * hd, w)), ("self_attn.o_proj", (w, nh * hd)),
                            ("mlp.gate_proj", (ff, w)), ("mlp.up_proj", (ff, w)),
                            ("mlp.down_proj", (w, ff))):
            out[p + name + ".weight"] = v.normal(shape, 0.02, dtype=dtype)
        for name, size in (("self_attn.q_norm", hd), ("self_attn.k_norm", hd),
                           ("input_layernorm", w), ("post_attention_layernorm", w)):
            out[p + name + ".weight"] = v.normal((size,), 0.1, 1.0, dtype)
    return out


def _qwen3_config(model, layers, vocab):
    w, nh, nkv, hd, ff, tied = MODELS[model]
    return Qwen3Config(vocab_size=vocab, hidden_size=w, num_hidden_layers=layers,
                       num_attention_heads=nh, num_key_value_heads=nkv, head_dim=hd,
                       intermediate_size=ff, max_position_embeddings=40960, rms_norm_eps=EPS,
                       rope_theta=THETA, tie_word_embeddings=tied)


def _model_inputs(case, seed):
    """Weights, prompts and each sequence's next token of a decode or prefill case."""
    v = Values(seed)
    weights = _qwen3_weights(v, case["model"], case["layers"], VOCAB, DTYPES[case["dtype"]])
    prompts = [v.ids(n, VOCAB) for n in lengths(case)]
    return weights, prompts, v.ids(case["count"], VOCAB)


def _layer_inputs(case, seed):
    v = Values(seed)
    weights = _qwen3_weights(v, case["model"], 1, 256, DTYPES[case["dtype"]])
    T = sum(lengths(case))
    return weights, v.normal((T, MODELS[case["model"]][0]), RESIDUAL, dtype=torch.float32)


def _state_inputs(case, seed):
    """A mixer's weights by the names of ``_state_spec``, the normed rows it reads, the residual."""
    v = Values(seed)
    w, nh, nkv, d, dv = STATES[case["mixer"]][case["size"]]
    m, kind = {}, case["mixer"]
    mat = lambda name, *shape: m.__setitem__(name, v.normal(shape, 0.02))
    if kind == "wkv":
        for s in ("r", "k", "v", "g"):
            mat(s, nh * d, w)
        mat("w1", WKV_RANK, w)
        mat("w2", nh * d, WKV_RANK)
        for s in ("r", "k", "v", "g", "w"):
            m["mu_" + s] = v.uniform((w,), 0.0, 1.0).to(torch.bfloat16)
        m["w0"] = v.uniform((nh * d,), -6.0, -1.0).to(torch.bfloat16)   # decays of 0.69 to 0.998
        m["u"] = v.normal((nh, d), 0.3)
        m["norm"] = v.normal((nh * d,), 0.1, 1.0)
        mat("o", w, nh * d)
    else:
        mat("q", nkv * d, w)
        mat("k", nkv * d, w)
        mat("v", nh * dv, w)
        mat("g", nh * dv, w)
        mat("o", w, nh * dv)
        if kind == "mlstm":
            mat("i", nh, w)
            mat("f", nh, w)
            m["i_bias"] = v.normal((nh,), 0.1)
            m["f_bias"] = v.uniform((nh,), 3.0, 6.0).to(torch.bfloat16)
            m["norm"] = v.normal((nh * dv,), 0.1, 1.0)
        else:
            m["norm"] = v.normal((dv,), 0.1, 1.0)
        if kind == "gla":
            mat("a1", GLA_RANK, w)
            mat("a2", nh * d, GLA_RANK)
            m["a2_bias"] = v.normal((nh * d,), 0.5)
        if kind == "delta":
            mat("b", nh, w)
            mat("a", nh, w)
            m["A_log"] = v.uniform((nh,), 1.0, 16.0).log().to(torch.bfloat16)
            dt = v.uniform((nh,), math.log(1e-3), math.log(0.1)).exp()
            m["dt_bias"] = (dt + torch.log(-torch.expm1(-dt))).to(torch.bfloat16)
            for s, n in (("q_conv", nkv * d), ("k_conv", nkv * d), ("v_conv", nh * dv)):
                m[s] = v.normal((n, TAPS), 0.5)
    T = sum(lengths(case))
    return m, v.normal((T, w)), v.normal((T, w), RESIDUAL, dtype=torch.float32)


def _state_spec(case):
    w, nh, nkv, d, dv = STATES[case["mixer"]][case["size"]]
    kind = case["mixer"]
    names = {"wkv": "r k v g w1 w2 mu_r mu_k mu_v mu_g mu_w w0 u norm o",
             "mlstm": "q k v g i f i_bias f_bias norm o", "gla": "q k v g a1 a2 a2_bias norm o",
             "delta": "q k v g b a A_log dt_bias q_conv k_conv v_conv norm o"}[kind].split()
    p = {"hidden_size": w, "heads": nh, "dim": d, "eps": EPS, "names": {n: n for n in names}}
    if kind != "wkv":
        p["vdim"] = dv
    p.update({"wkv": {"decay_rank": WKV_RANK}, "mlstm": {"gate_cap": CAP},
              "gla": {"tau": TAU, "decay_rank": GLA_RANK},
              "delta": {"kv_heads": nkv, "taps": TAPS, "unit_eps": EPS}}[kind])
    return PartSpec({"wkv": "wkv", "mlstm": "mlstm", "gla": "gated_linear_attention",
                     "delta": "gated_delta"}[kind], p)


def _experts_inputs(case, seed):
    v = Values(seed)
    w, ne, top, ff, sff = EXPERTS[case["size"]]
    m = {"router": v.normal((ne, w), 0.02), "shared.sg": v.normal((1, w), 0.02)}
    for e, size in [(f"e{e}.", ff) for e in range(ne)] + [("shared.", sff)]:
        m[e + "gate"] = v.normal((size, w), 0.02)
        m[e + "up"] = v.normal((size, w), 0.02)
        m[e + "down"] = v.normal((w, size), 0.02)
    T = case["tokens"]
    return m, v.normal((T, w)), v.normal((T, w), RESIDUAL, dtype=torch.float32)


def _latent_inputs(case, seed):
    v = Values(seed)
    w, nh, d, rd, vd, kvr, qr = LATENTS[case["size"]]
    m = {"dq": v.normal((qr, w), 0.02), "dq_norm": v.normal((qr,), 0.1, 1.0),
         "uq": v.normal((nh * (d + rd), qr), 0.02), "dkv": v.normal((kvr + rd, w), 0.02),
         "dkv_norm": v.normal((kvr,), 0.1, 1.0), "uk": v.normal((nh * d, kvr), 0.02),
         "uv": v.normal((nh * vd, kvr), 0.02), "g": v.normal((nh * vd, w), 0.02),
         "o": v.normal((w, nh * vd), 0.02)}
    T = sum(lengths(case))
    return m, v.normal((T, w)), v.normal((T, w), RESIDUAL, dtype=torch.float32)


def _sample_inputs(case, seed):
    """Logits as a trained model gives them: a broad bell and a few tokens far above it."""
    v = Values(seed)
    rows, vocab = case["rows"], case["vocab"]
    logits = v.normal((rows, vocab), 2.2, dtype=torch.float32)
    n = min(40, vocab // 4)
    at = torch.rand((rows, vocab), generator=v.gen, device=DEV).topk(n, dim=1).indices
    boost = v.uniform((rows, n), 2.0, 14.0)
    return logits.scatter_add_(1, at, boost)


# ---------------------------------------------------------------------------- prepare
def _context(rt, lens):
    """The step of a part that is run by itself: new sequences of these lengths."""
    buffers = StepBuffers(sum(lens), len(lens), rt.device)
    return buffers.fill([(i, 0, [0] * n, [n - 1]) for i, n in enumerate(lens)])


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("decode", "prefill"):
        weights, prompts, nexts = _model_inputs(case, seed)
        rt = Runtime(DTYPES[case["dtype"]], DEV)
        rt.consume_weights = True
        longest = max(len(p) for p in prompts)
        engine = Engine(_qwen3_config(case["model"], case["layers"], VOCAB), weights, rt,
                        max_tokens=sum(pages_for(len(p) + 1) * PAGE for p in prompts),
                        max_context=pages_for(longest + 1) * PAGE, max_slots=len(prompts))
        s.update(engine=engine, prompts=prompts)
        if kind == "decode":
            s["slots"] = [engine.open() for _ in prompts]
            for slot, p in zip(s["slots"], prompts):
                engine.step([Entry(slot, p)])
            s["entries"] = [Entry(slot, [t]) for slot, t in zip(s["slots"], nexts)]
        return s
    if kind == "sample":
        s["logits"] = _sample_inputs(case, seed)
        s["sampler"] = DeviceSampler(torch.device(DEV), case["rows"], case["vocab"])
        s["slots"] = torch.arange(case["rows"], dtype=torch.int32, device=DEV)
        s["sampling"] = Sampling(seed=seed, **SAMPLERS[case["how"]])
        for slot in range(case["rows"]):
            s["sampler"].start(slot, seed * 1000003 + slot)
        return s
    if kind == "layer":
        weights, s["x0"] = _layer_inputs(case, seed)
        lens = lengths(case)
        rt = Runtime(DTYPES[case["dtype"]], DEV)
        rt.consume_weights = True
        s["model"] = model = DecoderModel(_qwen3_config(case["model"], 1, 256).to_model_spec())
        model.bind(weights, rt)
        need = model.line_needs[0]
        plans = plan_groups({0: (need.kv_heads, need.head_dim, need.window, need.planes,
                                 need.v_dim)},
                            sum(pages_for(n) * PAGE for n in lens), pages_for(max(lens)) * PAGE,
                            len(lens), max(lens))
    elif kind == "latent":
        weights, s["h"], s["x0"] = _latent_inputs(case, seed)
        lens = lengths(case)
        w, nh, d, rd, vd, kvr, qr = LATENTS[case["size"]]
        rt = Runtime(torch.bfloat16, DEV)
        spec = PartSpec("latent_attention", {
            "hidden_size": w, "heads": nh, "dim": d, "rot_dim": rd, "vdim": vd, "kv_rank": kvr,
            "q_rank": qr, "scale": (d + rd) ** -0.5, "latent_norm_eps": EPS, "gate": True,
            "position": "rot", "names": {n: n for n in weights}})
        rot = POSITIONS.build(PartSpec("rope_half", {"theta": 1e4, "rot_dim": rd}))
        rot.bind({}, rt)
        s["part"] = MIXERS.build(spec, "", positions={"rot": rot})
        s["part"].bind(weights, rt)
        plans = plan_groups({0: (1, kvr + rd, 0, 1, 0)},
                            sum(pages_for(n) * PAGE for n in lens), pages_for(max(lens)) * PAGE,
                            len(lens), max(lens))
    elif kind == "state":
        weights, s["h"], s["x0"] = _state_inputs(case, seed)
        lens = lengths(case)
        rt = Runtime(torch.bfloat16, DEV)
        s["part"] = MIXERS.build(_state_spec(case), "", positions={})
        s["part"].bind(weights, rt)
        need = s["part"].state_need()
        s["state"] = torch.zeros((len(lens),) + need.shape, dtype=torch.float32, device=DEV)
    else:
        weights, s["h"], s["x0"] = _experts_inputs(case, seed)
        w, ne, top, ff, sff = EXPERTS[case["size"]]
        lens = [1] * case["tokens"]
        rt = Runtime(torch.bfloat16, DEV)
        spec = PartSpec("routed_experts", {
            "hidden_size": w, "experts": ne, "top": top, "intermediate_size": ff,
            "shared_size": sff, "activation": "silu", "weights": "softmax_of_chosen",
            "names": {"router": "router", "expert": "e{}.", "shared": "shared.",
                      "shared_gate": "shared.sg", "gate": "gate", "up": "up", "down": "down"}})
        s["part"] = FEED_FORWARDS.build(spec, "")
        rt.consume_weights = True
        s["part"].bind(weights, rt)
    if kind in ("layer", "latent"):
        book = CacheBook(plans, len(lens), pages_for(max(lens)) * PAGE)
        cache = CacheStorage(plans, len(lens), rt.dtype, rt.device, {})
        cache.map_pages(book.reserve([(book.open(), n) for n in lens]))
        s["line"] = cache.lines[0]
        s["cache"] = cache
    s["step"] = _context(rt, lens)
    s["x"] = torch.empty_like(s["x0"])
    return s


# ---------------------------------------------------------------------------- run
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "decode":
        engine = s["engine"]
        logits = engine.step(s["entries"])
        for slot, prompt in zip(s["slots"], s["prompts"]):     # back, for another try
            engine.truncate(slot, len(prompt))
        return logits
    if kind == "prefill":
        engine = s["engine"]
        slots = [engine.open() for _ in s["prompts"]]
        logits = engine.step([Entry(slot, p) for slot, p in zip(slots, s["prompts"])])
        for slot in slots:
            engine.close(slot)
        return logits
    if kind == "sample":
        return s["sampler"].pick(s["logits"], s["slots"], s["sampling"])
    x = s["x"]
    x.copy_(s["x0"])           # the residual as the layer before leaves it
    s["step"].memo = {}
    if kind == "layer":
        pending = s["model"].layers[0].block.forward(x, s["step"], s["line"], None, True)
    elif kind == "latent":
        pending = s["part"].forward(s["h"], x, s["step"], s["line"], None, True)
    elif kind == "state":
        s["state"].zero_()     # the sequences are new
        pending = s["part"].forward(s["h"], x, s["step"], None, s["state"], True)
    else:
        pending = s["part"].forward(s["h"], x, s["step"])
    if pending is not None:
        settle(x, pending)
    return (x, s["state"]) if kind == "state" else x


# ---------------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": 4 * n + 4 * case["rows"], "flops": 4 * n}
    if kind == "experts":
        w, ne, top, ff, sff = EXPERTS[case["size"]]
        T = case["tokens"]
        read = ne * (1 - (1 - top / ne) ** T)          # experts that some token chooses
        return {"bytes": 2 * (read * 3 * ff * w + 3 * sff * w + (ne + 1) * w) + T * w * (2 + 8),
                "flops": 2 * T * (top * 3 * ff * w + 3 * sff * w + (ne + 1) * w)}
    lens = lengths(case)
    T = sum(lens)
    pairs = sum(n * (n + 1) // 2 for n in lens)
    if kind in ("decode", "prefill", "layer"):
        w, nh, nkv, hd, ff, _ = MODELS[case["model"]]
        size = 2 if case["dtype"] == "bfloat16" else 4
        matrices = (nh + 2 * nkv) * hd * w + nh * hd * w + 3 * ff * w
        if kind == "layer":
            return {"bytes": size * (matrices + 2 * nkv * hd * T) + 8 * T * w,
                    "flops": 2 * matrices * T + 4 * nh * hd * pairs}
        L, B = case["layers"], case["count"]
        weights, rows = size * (L * matrices + VOCAB * w), B * (size * w + 4 * VOCAB)
        if kind == "decode":
            held = T + B
            return {"bytes": weights + rows + L * size * 2 * nkv * hd * held,
                    "flops": 2 * B * (L * matrices + VOCAB * w) + L * 4 * nh * hd * held}
        return {"bytes": weights + rows + T * size * (w + L * 2 * nkv * hd),
                "flops": 2 * (T * L * matrices + B * VOCAB * w) + L * 4 * nh * hd * pairs}
    if kind == "latent":
        w, nh, d, rd, vd, kvr, qr = LATENTS[case["size"]]
        down = (qr + kvr + rd + nh * vd) * w
        params = down + nh * (d + rd) * qr + nh * (d + vd) * kvr + nh * vd * w
        return {"bytes": 2 * params + T * (2 * w + 8 * w + 2 * (kvr + rd)),
                "flops": 2 * T * params + 2 * nh * (d + rd + vd) * pairs}
    w, nh, nkv, d, dv = STATES[case["mixer"]][case["size"]]
    if case["mixer"] == "wkv":
        params = (4 * nh * d + WKV_RANK) * w + nh * d * WKV_RANK + nh * d * w
    else:
        params = (2 * nkv * d + 2 * nh * dv) * w + nh * dv * w
        if case["mixer"] == "gla":
            params += GLA_RANK * (w + nh * d)
        else:
            params += 2 * nh * w
    state = case["count"] * nh * d * dv
    return {"bytes": 2 * params + 10 * T * w + 8 * state, "flops": 2 * T * params + 4 * T * nh * d * dv}


def tolerance(case):
    """About four times what the answers lie from ``exact``: a 16-bit rounding travels through all
    that follows it in a layer (0.7 per cent), less in a part that is added to its residual (0.2)."""
    if case["kind"] == "sample":
        return "exact"
    if case.get("dtype") == "float32":
        return {"rel": 3e-5}
    return {"rel": 3e-2 if case["kind"] in ("decode", "prefill", "layer") else 1e-2}


# ---------------------------------------------------------------------------- exact
def _rms(x, w=None, eps=EPS):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * w.double()


def _mm(x, w):
    return x @ w.double().t()


def _turn(x, theta, n):
    """x [n, heads, rot]: the rotate-half pairing; the angle is the float32 product of the float32
    frequency and the position, which is how the design states it."""
    rot = x.shape[-1]
    inv = torch.tensor([1.0 / theta ** (2 * i / rot) for i in range(rot // 2)],
                       dtype=torch.float32, device=x.device)
    ang = (torch.arange(n, device=x.device, dtype=torch.float32)[:, None] * inv).double()[:, None]
    a, b = x[..., :rot // 2], x[..., rot // 2:]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], dim=-1)


def _attend(q, k, v, scale):
    """Causal attention of one sequence: q, k, v [n, heads, size]."""
    n = q.shape[0]
    out = torch.empty((n, q.shape[1], v.shape[2]), dtype=q.dtype, device=q.device)
    mask = torch.ones((n, n), dtype=torch.bool, device=q.device).triu(1)
    for h in range(q.shape[1]):
        p = (q[:, h] @ k[:, h].t() * scale).masked_fill_(mask, -math.inf).softmax(-1)
        out[:, h] = p @ v[:, h]
    return out.reshape(n, -1)


def _qwen3_layer(x, lens, m, i, model):
    """x [T, width] float64 of sequences of ``lens`` rows, changed in place."""
    w, nh, nkv, hd, ff, _ = MODELS[model]
    g = {k[len(f"model.layers.{i}."):-len(".weight")]: t.double() for k, t in m.items()
         if k.startswith(f"model.layers.{i}.")}
    at = 0
    for n in lens:
        r = x[at:at + n]
        h = _rms(r, g["input_layernorm"])
        q = _rms((h @ g["self_attn.q_proj"].t()).view(n, nh, hd), g["self_attn.q_norm"])
        k = _rms((h @ g["self_attn.k_proj"].t()).view(n, nkv, hd), g["self_attn.k_norm"])
        v = (h @ g["self_attn.v_proj"].t()).view(n, nkv, hd)
        q, k = _turn(q, THETA, n), _turn(k, THETA, n)
        rep = lambda t: t.repeat_interleave(nh // nkv, dim=1)
        r += _attend(q, rep(k), rep(v), hd ** -0.5) @ g["self_attn.o_proj"].t()
        h = _rms(r, g["post_attention_layernorm"])
        a = torch.nn.functional.silu(h @ g["mlp.gate_proj"].t()) * (h @ g["mlp.up_proj"].t())
        r += a @ g["mlp.down_proj"].t()
        at += n


def _exact_model(case, seed):
    m, prompts, nexts = _model_inputs(case, seed)
    if case["kind"] == "decode":
        prompts = [p + [t] for p, t in zip(prompts, nexts)]
    lens = [len(p) for p in prompts]
    ids = torch.tensor([t for p in prompts for t in p], device=DEV)
    x = m["model.embed_tokens.weight"][ids].double()
    for i in range(case["layers"]):
        _qwen3_layer(x, lens, m, i, case["model"])
    last = torch.tensor(lens, device=DEV).cumsum(0) - 1
    h = _rms(x[last], m["model.norm.weight"])
    head = m["model.embed_tokens.weight" if MODELS[case["model"]][5] else "lm_head.weight"]
    return torch.cat([_mm(h, part) for part in head.split(16384)], dim=1)


def _walk(S, steps):
    """Runs ``steps(t, S) -> (S, o)`` over the tokens; returns the outputs and the last state."""
    outs, t = [], 0
    while True:
        got = steps(t, S)
        if got is None:
            return torch.stack(outs), S
        S, o = got
        outs.append(o)
        t += 1


def _exact_state(case, seed):
    m, h, x = _state_inputs(case, seed)
    m, h, x = {k: t.double() for k, t in m.items()}, h.double(), x.double()
    w, nh, nkv, d, dv = STATES[case["mixer"]][case["size"]]
    kind, at, states = case["mixer"], 0, []
    silu, sig = torch.nn.functional.silu, torch.sigmoid
    f64 = dict(dtype=torch.float64, device=DEV)
    for n in lengths(case):
        r = h[at:at + n]
        S0 = torch.zeros((nh, d, dv), **f64)
        if kind == "wkv":
            prev = torch.cat([torch.zeros((1, w), **f64), r[:-1]])
            mix = lambda s: r + (prev - r) * m["mu_" + s]
            rr, k, v = (_mm(mix(s), m[s]).view(n, nh, d) for s in ("r", "k", "v"))
            dec = torch.exp(-torch.exp(_mm(torch.tanh(_mm(mix("w"), m["w1"])), m["w2"]) + m["w0"]))
            dec, u = dec.view(n, nh, d), m["u"].view(nh, d)

            def walk(t, S):
                if t == n:
                    return None
                kv = k[t][:, :, None] * v[t][:, None, :]
                o = torch.einsum("hdv,hd->hv", S + u[:, :, None] * kv, rr[t])
                return dec[t][:, :, None] * S + kv, o
            o, S = _walk(S0, walk)
            y = _rms(o).reshape(n, -1) * m["norm"] * silu(_mm(mix("g"), m["g"]))
            states.append(torch.cat([r[-1], S.reshape(-1)]))
        elif kind == "gla":
            q, k = ((r @ m[s].t()).view(n, nh, d) for s in ("q", "k"))
            v = (r @ m["v"].t()).view(n, nh, dv)
            a = sig(_mm(_mm(r, m["a1"]), m["a2"]) + m["a2_bias"]).pow(1 / TAU).view(n, nh, d)

            def walk(t, S):
                if t == n:
                    return None
                S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
                return S, torch.einsum("hdv,hd->hv", S, q[t] * d ** -0.5)
            o, S = _walk(S0, walk)
            y = (_rms(o, m["norm"])).reshape(n, -1) * silu(_mm(r, m["g"]))
            states.append(S.reshape(-1))
        elif kind == "mlstm":
            q, k = ((r @ m[s].t()).view(n, nh, d) for s in ("q", "k"))
            v = (r @ m["v"].t()).view(n, nh, dv)
            cap = lambda z: CAP * torch.tanh(z / CAP)
            gi = cap(_mm(r, m["i"]) + m["i_bias"])
            gf = torch.nn.functional.logsigmoid(cap(_mm(r, m["f"]) + m["f_bias"]))

            def walk(t, S):
                if t == n:
                    return None
                S, nv, mx = S
                m2 = torch.maximum(gf[t] + mx, gi[t])
                a, b = torch.exp(gf[t] + mx - m2)[:, None], torch.exp(gi[t] - m2)[:, None]
                S = a[:, :, None] * S + b[:, :, None] * k[t][:, :, None] * v[t][:, None, :]
                nv = a * nv + b * k[t]
                qs = q[t] * d ** -0.5
                den = torch.maximum((nv * qs).sum(-1).abs(), torch.exp(-m2)) + 1e-6
                return (S, nv, m2), torch.einsum("hdv,hd->hv", S, qs) / den[:, None]
            o, S = _walk((S0, torch.zeros((nh, d), **f64), torch.zeros((nh,), **f64)), walk)
            y = _rms(o).reshape(n, -1) * m["norm"] * sig(_mm(r, m["g"]))
            states.append(torch.cat([S[0].reshape(nh, -1), S[1], S[2][:, None]], 1).reshape(-1))
        else:
            z = torch.cat([_mm(r, m[s]) for s in ("q", "k", "v")], dim=1)
            taps = torch.cat([m[s] for s in ("q_conv", "k_conv", "v_conv")])
            past = torch.cat([torch.zeros((TAPS - 1, z.shape[1]), **f64), z])
            c = silu(sum(past[j:j + n] * taps[:, j] for j in range(TAPS)))
            unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + EPS)
            rep = lambda t: unit(t.view(n, nkv, d)).repeat_interleave(nh // nkv, dim=1)
            q, k = rep(c[:, :nkv * d]) * d ** -0.5, rep(c[:, nkv * d:2 * nkv * d])
            v = c[:, 2 * nkv * d:].view(n, nh, dv)
            beta = sig(_mm(r, m["b"]))
            dec = torch.exp(-torch.exp(m["A_log"])
                            * torch.nn.functional.softplus(_mm(r, m["a"]) + m["dt_bias"]))

            def walk(t, S):
                if t == n:
                    return None
                S = dec[t][:, None, None] * S
                u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
                S = S + k[t][:, :, None] * u[:, None, :]
                return S, torch.einsum("hdv,hd->hv", S, q[t])
            o, S = _walk(S0, walk)
            y = (_rms(o, m["norm"])).reshape(n, -1) * silu(_mm(r, m["g"]))
            states.append(torch.cat([S.reshape(-1), past[n:].reshape(-1)]))
        x[at:at + n] += _mm(y, m["o"])
        at += n
    return x, torch.stack(states)


def _exact_experts(case, seed):
    m, h, x = _experts_inputs(case, seed)
    h, x = h.double(), x.double()
    w, ne, top, ff, sff = EXPERTS[case["size"]]
    silu = torch.nn.functional.silu
    mlp = lambda e, r: _mm(silu(_mm(r, m[e + "gate"])) * _mm(r, m[e + "up"]), m[e + "down"])
    z, ids = _mm(h, m["router"]).topk(top, dim=1)
    p = z.softmax(-1)
    for e in range(ne):
        rows, k = (ids == e).nonzero(as_tuple=True)
        if rows.numel():
            x.index_add_(0, rows, p[rows, k][:, None] * mlp(f"e{e}.", h[rows]))
    return x + torch.sigmoid(_mm(h, m["shared.sg"])) * mlp("shared.", h)


def _exact_latent(case, seed):
    m, h, x = _latent_inputs(case, seed)
    h, x = h.double(), x.double()
    w, nh, d, rd, vd, kvr, qr = LATENTS[case["size"]]
    at = 0
    for n in lengths(case):
        r = h[at:at + n]
        q = _mm(_rms(_mm(r, m["dq"]), m["dq_norm"]), m["uq"]).view(n, nh, d + rd)
        kv = _mm(r, m["dkv"])
        c, rot = _rms(kv[:, :kvr], m["dkv_norm"]), _turn(kv[:, None, kvr:], 1e4, n)
        q = torch.cat([q[..., :d], _turn(q[..., d:], 1e4, n)], dim=-1)
        k = torch.cat([_mm(c, m["uk"]).view(n, nh, d), rot.expand(n, nh, rd)], dim=-1)
        o = _attend(q, k, _mm(c, m["uv"]).view(n, nh, vd), (d + rd) ** -0.5)
        x[at:at + n] += _mm(o * torch.sigmoid(_mm(r, m["g"])), m["o"])
        at += n
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return None            # ids of tokens, no computed numbers
    if kind in ("decode", "prefill"):
        return _exact_model(case, seed)
    if kind == "layer":
        weights, x = _layer_inputs(case, seed)
        x = x.double()
        _qwen3_layer(x, lengths(case), weights, 0, case["model"])
        return x
    return {"state": _exact_state, "experts": _exact_experts, "latent": _exact_latent}[kind](case, seed)
