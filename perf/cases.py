"""Workloads of the framework for timing and comparing two builds of it, each through the entry point that a program calls.

``listed()`` names twelve of them; ``draw(rng)`` makes more of the same ranges.  A case is a dict of plain values:

  talker        one decode step of the 1.7B talker (28 layers and the codec head) for ``streams`` sequences, replayed by its runner
  predictor     one decode pass of the code predictor (5 layers and an LM head); a codec frame runs 14 of them per talker step
  talker_layer  one talker layer over whole prompts (voice-clone prompts are thousands of tokens long)
  experts       one mixture-of-experts feed-forward: a prompt step of thousands of tokens, or a decode step of a few
  lm_prompt     one engine step over new prompts of a 4-layer Bokenex model, with the logits of every prompt's last token
  sink_prompt   one softmax attention layer (preparation, cache write, attention, gate) over prompt portions, some of them with
                cached tokens in front, in the three forms that the model families have
  sink_decode   the same layer for one new token of each of ``streams`` sequences
  latent        one latent attention mixer over prompt portions or single tokens
  state_space   one state-space memory (convolution, recurrence, gated norm) over new prompts
  delta_rule    one delta-rule memory over new prompts

``portions`` is "cached+new,cached+new,...": a sequence with ``cached`` tokens behind it runs ``new`` tokens.  Sizes are those of the
shipped 1.7B model and of the 2048-wide layers that ``bench_lm.py`` measures; activations are bfloat16, what serving uses.
Every case can be run again on the same state and gives the same answer: caches are rewritten in place and recurrences start at
position 0."""
import dataclasses
import math

import torch
import torch.nn.functional as F

DEV = "cuda:0"
BF = torch.bfloat16
F64 = torch.float64
EPS = 1e-6
WIDTH, HEADS, KV_HEADS, DIM, PAGE, WINDOW = 2048, 16, 8, 128, 256, 1024
TALKER = dict(hidden=2048, inter=6144, layers=28, vocab=3072, theta=1e6)
PREDICTOR = dict(hidden=1024, inter=3072, layers=5, vocab=2048, theta=1e6, in_hidden=2048)
EXPERTS, TOP, EXPERT_FF, LIMIT, GROUPS = 16, 2, 3072, 7.0, 4
LM = dict(layers=4, vocab=3072, ff=9216, taps=4, mult=0.5, positions=4096)
LATENT = dict(rank=512, rot=64, theta=5e5)
SSM = dict(heads=64, vdim=64, state=128, taps=4)


def listed():
    return [
        # one listener, a short prompt: the latency of a frame, hundreds of dependent launches on one row
        dict(name="talker_1_stream", kind="talker", streams=1, context=97),
        # the serving point of the frame benchmark
        dict(name="talker_64_streams", kind="talker", streams=64, context=200),
        # code predictor of a well-filled GPU, an odd batch
        dict(name="predictor_201_streams", kind="predictor", streams=201, step=7),
        # voice clone: two prompts with reference audio, one of them ragged
        dict(name="talker_layer_clone_prompts", kind="talker_layer", portions="0+4096,0+1531"),
        # mixture of experts: a full prompt step, and a decode step that streams every expert
        dict(name="experts_8192_tokens", kind="experts", tokens=8192, form="silu"),
        dict(name="experts_64_tokens", kind="experts", tokens=64, form="clamped"),
        # a whole token model on a burst of new prompts of unequal length
        dict(name="lm_ragged_prompts", kind="lm_prompt", portions="0+2048,0+1333,0+700,0+57"),
        # attention layers over prompts: windows with kept first keys; capped causal scores on long portions with a cached prefix
        dict(name="window_attention_prompts", kind="sink_prompt", form="window", portions="0+2048,0+2048,0+1999,0+2048"),
        # a decode step of 64 long conversations
        dict(name="attention_64_decoding", kind="sink_decode", form="capped", streams=64, context=1100),
        # latent attention over a full prompt step
        dict(name="latent_prompts", kind="latent", portions="0+2048,0+2048,512+1001,0+2048", window=0),
        # recurrences over a full prompt step and over ragged ones
        dict(name="state_space_prompts", kind="state_space", portions="0+2048,0+2048,0+2048,0+2048"),
        dict(name="delta_rule_ragged_prompts", kind="delta_rule", portions="0+2048,0+1777,0+900,0+131"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _portions(rng, total, cached):
    """Up to six portions of together at most ``total`` tokens."""
    left, out = _log(rng, 24, total), []
    for _ in range(rng.randint(1, 6)):
        n = min(left, 2048, max(1, int(left * rng.uniform(0.3, 1.0))))
        if n:
            out.append(f"{rng.choice([0, 0, rng.randint(1, 1500)]) if cached else 0}+{n}")
        left -= n
    return ",".join(out)


def draw(rng):
    kind = rng.choice(["talker", "predictor", "talker_layer", "experts", "lm_prompt", "sink_prompt", "sink_decode", "latent",
                       "state_space", "delta_rule"])
    c = dict(kind=kind)
    if kind == "talker":
        c.update(streams=_log(rng, 1, 128), context=_log(rng, 16, 400))
    elif kind == "predictor":
        c.update(streams=_log(rng, 1, 512), step=rng.randint(1, 14))
    elif kind == "talker_layer":
        c.update(portions=f"0+{_log(rng, 20, 4096)},0+{_log(rng, 20, 1500)}")
    elif kind == "experts":
        c.update(tokens=_log(rng, 1, 8192), form=rng.choice(["silu", "clamped"]))
    elif kind == "lm_prompt":
        c.update(portions=_portions(rng, 6000, False))
    elif kind == "sink_prompt":
        c.update(form=rng.choice(["window", "chunk", "capped"]), portions=_portions(rng, 8192, True))
    elif kind == "sink_decode":
        c.update(form=rng.choice(["window", "chunk", "capped"]), streams=_log(rng, 1, 128), context=_log(rng, 30, 2000))
    elif kind == "latent":
        c.update(portions=_portions(rng, 7000, True), window=rng.choice([0, WINDOW]))
    else:
        c.update(portions=_portions(rng, 8192, False))
    return c


# ------------------------------------------------------------------------------------------------ inputs
class _Rand:
    """Numbers from a seed, made on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))

    def __call__(self, *shape, std=1.0, mean=0.0, dtype=BF):
        return torch.randn(shape, generator=self.g, device=DEV).mul_(std).add_(mean).to(dtype)

    def ints(self, hi, n):
        return torch.randint(0, hi, (n,), generator=self.g, device=DEV)


def _seqs(case):
    if "portions" in case:
        return [tuple(int(v) for v in p.split("+")) for p in case["portions"].split(",")]
    b = case["streams"]
    return [(c - 1, 1) for c in _contexts(case["context"], b)]


def _contexts(context, b):
    """Context lengths of ``b`` sequences, spread from half to one and a half of ``context``."""
    return [max(2, context // 2 + (context * (2 * i + 1)) // (2 * b)) for i in range(b)]


def _tables(seqs, seed):
    """Pages of every sequence, in a random order: (tables, pages in all)."""
    need = [-(-(c + n) // PAGE) for c, n in seqs]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(seed)).tolist()
    out, o = [], 0
    for n in need:
        out.append(order[o:o + n])
        o += n
    return out, sum(need)


def _sequences(seqs, tables, tokens=None):
    from nano_qwen3tts_vllm_b200.engine.sequence import Sequence
    out, o = [], 0
    for b, ((c, n), bt) in enumerate(zip(seqs, tables)):
        ids = [0] * c + (tokens[o:o + n] if tokens is not None else [0] * n)
        s = Sequence(ids)
        s.num_cached_tokens, s.block_table, s.state_slot = c, bt, b
        out.append(s)
        o += n
    return out


def _layout(seqs, tables):
    from nano_qwen3tts_vllm_b200.engine.step_layout import MixedStepLayout
    lay = MixedStepLayout(sum(n for _, n in seqs), len(seqs), max(len(t) for t in tables), torch.device(DEV))
    lay.fill([(s, n) for s, (_, n) in zip(_sequences(seqs, tables), seqs)], PAGE)
    return lay


def _slots(seqs, tables):
    """Cache slots of each sequence's tokens, cached ones first (for the plain restatements)."""
    return [torch.tensor([bt[p // PAGE] * PAGE + p % PAGE for p in range(c + n)], device=DEV) for (c, n), bt in zip(seqs, tables)]


def _module(make, dtype=BF):
    prev = torch.get_default_dtype()
    torch.set_default_dtype(dtype)
    try:
        with torch.device(DEV):
            return make()
    finally:
        torch.set_default_dtype(prev)


def _fill(pairs):
    with torch.no_grad():
        for p, v in pairs:
            p.copy_(v)


def _talker_weights(seed, s, layers=None):
    """The stack's tensors under the checkpoint's names, drawn as the configurations say: N(0, 0.02^2), norms around 1."""
    r, out, D, I = _Rand(seed), {}, s["hidden"], s["inter"]
    q, kv = HEADS * DIM, KV_HEADS * DIM
    for i in range(layers or s["layers"]):
        p = f"model.layers.{i}."
        for name, rows, cols in (("self_attn.q_proj", q, D), ("self_attn.k_proj", kv, D), ("self_attn.v_proj", kv, D),
                                 ("self_attn.o_proj", D, q), ("mlp.gate_proj", I, D), ("mlp.up_proj", I, D), ("mlp.down_proj", D, I)):
            out[f"{p}{name}.weight"] = r(rows, cols, std=0.02)
        for name, n in (("self_attn.q_norm", DIM), ("self_attn.k_norm", DIM), ("input_layernorm", D), ("post_attention_layernorm", D)):
            out[f"{p}{name}.weight"] = r(n, std=0.02, mean=1.0)
    out["model.norm.weight"] = r(D, std=0.02, mean=1.0)
    return out


def _stack_inputs(case, seed):
    """(weights, input rows, KV pool [2, layers, pages, page, kv heads, dim], sequences, tables) of a decode step."""
    s = TALKER if case["kind"] == "talker" else PREDICTOR
    seqs = _seqs(case) if case["kind"] == "talker" else [(case["step"] + 1, 1)] * case["streams"]
    tables, pages = _tables(seqs, seed)
    w, r = _talker_weights(seed, s), _Rand(seed + 1)
    if case["kind"] == "talker":
        w["model.codec_embedding.weight"] = r(s["vocab"], s["hidden"], std=0.02)
        w["codec_head.weight"] = r(s["vocab"], s["hidden"], std=0.02)
        x = r(case["streams"], s["hidden"], std=0.05)
    else:
        for g in range(15):
            w[f"model.codec_embedding.{g}"] = r(s["vocab"], s["in_hidden"], std=0.02)
            w[f"lm_head.{g}"] = r(s["vocab"], s["hidden"], std=0.02)
        w["small_to_mtp_projection.weight"] = r(s["hidden"], s["in_hidden"], std=0.02)
        w["small_to_mtp_projection.bias"] = r(s["hidden"], std=0.01)
        x = r.ints(s["vocab"], case["streams"])
    kv = torch.empty(2, s["layers"], pages, PAGE, KV_HEADS, DIM, dtype=BF, device=DEV)
    for i in range(s["layers"]):
        for side, std in enumerate((1.0, 0.5)):                                 # normed keys have unit size
            kv[side, i] = r(pages, PAGE, KV_HEADS, DIM, std=std)
    return w, x, kv, seqs, tables


def _expert_inputs(case, seed):
    r, n = _Rand(seed), case["tokens"]
    std = WIDTH ** -0.5
    d = dict(h=r(n, WIDTH), router=r(EXPERTS, WIDTH, std=1.5 * std).float(), up=r(EXPERTS, 2 * EXPERT_FF, WIDTH, std=std),
             down=r(EXPERTS, WIDTH, EXPERT_FF, std=EXPERT_FF ** -0.5))
    if case["form"] == "silu":
        d["bias"] = r(EXPERTS, std=0.1).float()
    else:
        d["shared_gate_up"], d["shared_down"] = r(2 * EXPERT_FF, WIDTH, std=std), r(WIDTH, EXPERT_FF, std=EXPERT_FF ** -0.5)
    return d


def _lm_inputs(case, seed):
    r, D, q, kv = _Rand(seed), WIDTH, HEADS * DIM, KV_HEADS * DIM
    sd = {"embed": r(LM["vocab"], D), "pos": r(LM["positions"], D, std=0.5), "final.norm": r(std=0.05, mean=1.0),
          "head": r(LM["vocab"], D, std=D ** -0.5)}
    for i in range(LM["layers"]):
        p = f"l{i}."
        sd[p + "norm1"] = r(std=0.05, mean=1.0)
        for c, rows in (("q", q), ("k", kv), ("v", kv)):
            sd[f"{p}mix.{c}"], sd[f"{p}mix.{c}.conv"] = r(rows, D, std=D ** -0.5), r(rows, LM["taps"], std=0.5)
        sd[p + "mix.q.norm"], sd[p + "mix.k.norm"] = r(DIM, std=0.1, mean=1.0), r(DIM, std=0.1, mean=1.0)
        sd[p + "mix.r1"], sd[p + "mix.r2"] = r(HEADS, std=0.2, mean=0.5), r(HEADS, std=0.1, mean=0.5).abs()
        sd[p + "mix.pb"], sd[p + "mix.o"] = r(HEADS, std=0.5, mean=-2.0), r(D, q, std=q ** -0.5)
        sd[p + "mlp.up"], sd[p + "mlp.down"] = r(LM["ff"], D, std=D ** -0.5), r(D, LM["ff"], std=LM["ff"] ** -0.5)
    seqs = _seqs(case)
    return sd, r.ints(LM["vocab"], sum(n for _, n in seqs)).tolist(), seqs


def _sink_inputs(case, seed):
    r, seqs = _Rand(seed), _seqs(case)
    tables, pages = _tables(seqs, seed)
    n, nq, nk, form = sum(m for _, m in seqs), HEADS * DIM, KV_HEADS * DIM, case["form"]
    gates = {"window": nq, "chunk": HEADS, "capped": 0}[form]
    d = dict(seqs=seqs, tables=tables, u=r(n, nq + 2 * nk + gates), k=r(pages, PAGE, nk), v=r(pages, PAGE, nk, std=1.0),
             qb=r(nq, std=0.3).float(), kb=r(nk, std=0.3).float(), vb=r(nk, std=0.3).float())
    if form == "window":
        d["qn"], d["kn"] = r(DIM, std=0.1, mean=1.0).float(), r(DIM, std=0.1, mean=1.0).float()
    if form == "chunk":
        d["sink"] = r(HEADS).float()
    return d


def _latent_inputs(case, seed):
    r, seqs, R, dr = _Rand(seed), _seqs(case), LATENT["rank"], LATENT["rot"]
    tables, pages = _tables(seqs, seed)
    n = sum(m for _, m in seqs)
    return dict(seqs=seqs, tables=tables, h=r(n, WIDTH), w_in=r(HEADS * (DIM + dr) + R + dr, WIDTH, std=WIDTH ** -0.5),
                norm=r(R, std=0.1, mean=1.0).float(), uk=r(HEADS, DIM, R, std=R ** -0.5), uv=r(HEADS, DIM, R, std=R ** -0.5),
                sink=r(HEADS).float(), o=r(WIDTH, HEADS * DIM, std=(HEADS * DIM) ** -0.5), cache=r(pages, PAGE, R + dr))


def _ssm_inputs(case, seed):
    r, seqs, H, P, N = _Rand(seed), _seqs(case), SSM["heads"], SSM["vdim"], SSM["state"]
    ch = H * P + 2 * N
    return dict(seqs=seqs, u=r(sum(n for _, n in seqs), H * P + ch + H), conv=r(ch, SSM["taps"], std=0.5).float(), conv_b=r(ch, std=0.2).float(),
                dt_bias=r(H, std=0.5).float(), A_log=r(H, std=0.5, mean=-0.5).float(), D=r(H, std=0.5).float(), norm=r(H * P, std=0.1, mean=1.0).float())


def _delta_inputs(case, seed):
    r, seqs, nk, nv = _Rand(seed), _seqs(case), KV_HEADS * DIM, HEADS * DIM
    return dict(seqs=seqs, u=r(sum(n for _, n in seqs), 2 * nk + 2 * nv + 2 * HEADS), conv=r(2 * nk + nv, 4, std=0.5).float(),
                A_log=r(HEADS, std=0.5, mean=-0.5).float(), dt_bias=r(HEADS, std=0.5).float(), norm=r(DIM, std=0.1, mean=1.0).float())


# ------------------------------------------------------------------------------------------------ what a program keeps, and one pass
class _State:
    """What a program holds between calls; ``close`` gives back what the package keeps for it beyond the tensors."""

    def __init__(self, call, close=None):
        self.call, self.close = call, close

    def __del__(self):
        if self.close is not None:
            self.close()


def _prepare_stack(case, seed):
    from nano_qwen3tts_vllm_b200.config import ModelConfig, qwen3_tts_config
    from nano_qwen3tts_vllm_b200.engine.model_runner.predictor_model_runner import PredictorSequence
    from nano_qwen3tts_vllm_b200.engine.sequence import Sequence
    from nano_qwen3tts_vllm_b200.llm import PredictorLLM, TalkerLLM
    w, x, kv, seqs, tables = _stack_inputs(case, seed)
    mc = qwen3_tts_config("1.7B")
    mc = ModelConfig(dataclasses.replace(mc.talker, text_vocab_size=0), mc.predictor)
    width = max(len(t) for t in tables)
    talker = case["kind"] == "talker"
    eng = (TalkerLLM if talker else PredictorLLM)(
        mc, state_dict=w, num_kvcache_blocks=kv.shape[2], max_num_seqs=max(case["streams"], 2), max_model_len=width * PAGE,
        max_num_batched_tokens=max(16384, width * PAGE), graph_batch_sizes=[case["streams"]], device=DEV)
    runner = eng.model_runner
    runner.kv_cache.copy_(kv)
    out = []
    for i, ((c, _), bt) in enumerate(zip(seqs, tables)):
        if talker:
            s = Sequence(None, input_embeds=x[:1].view(1, 1, -1))
            s.decode_input_embeds, s.num_tokens = x[i].view(1, 1, -1), c + 1
        else:
            s = PredictorSequence(None, input_embeds=x.new_zeros(1, 2, 1), generation_steps=case["step"])
            s.last_token, s.num_tokens = int(x[i]), c + 1
        s.block_table = bt
        out.append(s)
    return _State(lambda: (runner.run_model(out, False), runner.kv_cache), eng.exit)


def _prepare_layer(case, seed):
    from nano_qwen3tts_vllm_b200.config import qwen3_tts_config
    from nano_qwen3tts_vllm_b200.layers.linear import release_packed
    from nano_qwen3tts_vllm_b200.models.qwen3_tts_share import Qwen3TTSDecoderLayer, load_reference_weights
    from nano_qwen3tts_vllm_b200.utils.context import set_context
    layer = _module(lambda: Qwen3TTSDecoderLayer(qwen3_tts_config("1.7B").talker))
    w = {k[len("model.layers.0."):]: v for k, v in _talker_weights(seed, TALKER, 1).items() if "layers" in k}
    load_reference_weights(torch.nn.ModuleDict({"l": layer}), {"l." + k: v for k, v in w.items()})
    seqs = _seqs(case)
    tables, pages = _tables(seqs, seed)
    r = _Rand(seed + 1)
    n, lens = sum(m for _, m in seqs), [m for _, m in seqs]
    x, res = r(n, TALKER["hidden"], std=0.5), r(n, TALKER["hidden"], std=0.5)
    a = layer.self_attn.attn
    a.k_cache, a.v_cache = (torch.zeros(pages, PAGE, KV_HEADS, DIM, dtype=BF, device=DEV) for _ in range(2))
    pos = torch.cat([torch.arange(m, device=DEV) for m in lens])
    slots = torch.cat(_slots(seqs, tables)).to(torch.int32)
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)

    def call():
        set_context(True, cu, cu, max(lens), max(lens), slots)
        with torch.inference_mode():
            y, out = layer(pos, x, res)
        return y, out, a.k_cache, a.v_cache
    return _State(call, lambda: release_packed(layer))


def _prepare_experts(case, seed):
    from nano_qwen3tts_vllm_b200.layers.linear import release_packed
    from nano_qwen3tts_vllm_b200.layers.moe import SharedClampedMoE, SoftmaxTopKGatedMoE
    d = _expert_inputs(case, seed)
    if case["form"] == "silu":
        m = _module(lambda: SoftmaxTopKGatedMoE(WIDTH, EXPERT_FF, EXPERTS, TOP))
        _fill([(m.router_bias, d["bias"])])
    else:
        m = _module(lambda: SharedClampedMoE(WIDTH, EXPERT_FF, EXPERTS, TOP, LIMIT, GROUPS, 1, EXPERT_FF, LIMIT))
        _fill([(m.shared.gate_up.weight, d["shared_gate_up"]), (m.shared.down.weight, d["shared_down"])])
    _fill([(m.router, d["router"]), (m.up, d["up"]), (m.down, d["down"])])
    h = d["h"]

    def call():
        with torch.inference_mode():
            return m(h)
    return _State(call, lambda: release_packed(m))


def _prepare_lm(case, seed):
    from nano_qwen3tts_vllm_b200.config import BokenexConfig
    from nano_qwen3tts_vllm_b200.engine.llm_engine.lm_engine import CausalLMEngine
    sd, tokens, seqs = _lm_inputs(case, seed)
    tables, pages = _tables(seqs, seed)
    layer = {"type": "attention", "mlp": {"kind": "dense", "ff": LM["ff"]},
             "mixer": {"heads": HEADS, "kv_heads": KV_HEADS, "dim": DIM, "vdim": DIM, "conv": LM["taps"], "mask": {"size": WINDOW},
                       "scale": DIM ** -0.5}}
    cfg = BokenexConfig.from_dict({"architecture": "Bokenex", "vocab": LM["vocab"], "width": WIDTH, "max_positions": LM["positions"],
                                   "norm": {"eps": EPS}, "residual_mult": LM["mult"], "layers": [layer] * LM["layers"]})
    eng = CausalLMEngine(cfg, state_dict=sd, kvcache_block_size=PAGE, num_kvcache_blocks=pages, max_num_seqs=max(len(seqs), 2),
                         max_model_len=LM["positions"], max_num_batched_tokens=16384, enforce_eager=True, device=DEV)
    items = [(s, n) for s, (_, n) in zip(_sequences(seqs, tables, tokens), seqs)]
    rows = [sum(n for _, n in seqs[:i + 1]) - 1 for i in range(len(seqs))]
    return _State(lambda: eng.model_runner.run_step(items, rows), eng.exit)


def _prepare_sink(case, seed):
    from nano_qwen3tts_vllm_b200.layers.attention import SinkSoftmaxAttention
    from nano_qwen3tts_vllm_b200.layers.rotary_embedding import PairRotary, PairRotaryTable
    from nano_qwen3tts_vllm_b200.utils.context import set_context
    d, form = _sink_inputs(case, seed), case["form"]
    rot = _module(lambda: {"window": lambda: PairRotaryTable(DIM, 1e6), "chunk": lambda: None,
                           "capped": lambda: PairRotary(DIM // 2, 1e4, {"factor": 2.0})}[form](), torch.float32)
    kw = {"window": dict(sink="none", keep_first=4, head_norm=True, element_gate=True), "chunk": dict(),
          "capped": dict(sink="zero", softcap=50.0)}[form]
    mask = {"window": ("window", WINDOW), "chunk": ("chunk", WINDOW), "capped": ("window", 0)}[form]
    m = _module(lambda: SinkSoftmaxAttention(HEADS, KV_HEADS, DIM, DIM, *mask, DIM ** -0.5, bias=True, rotary=rot, eps=EPS, **kw))
    _fill([(m.q_bias, d["qb"]), (m.k_bias, d["kb"]), (m.v_bias, d["vb"])])
    if form == "window":
        _fill([(m.q_norm, d["qn"]), (m.k_norm, d["kn"])])
    if form == "chunk":
        _fill([(m.sink, d["sink"])])
    m.k_cache, m.v_cache = d["k"], d["v"]
    lay, u = _layout(d["seqs"], d["tables"]), d["u"]
    nq, nk = HEADS * DIM, KV_HEADS * DIM
    gate = u[:, nq + 2 * nk:] if form != "capped" else None
    if form == "window":
        rot.fill(lay.positions)                                                  # once per step, shared by its layers

    def call():
        set_context(False, step_layout=lay)
        with torch.inference_mode():
            o = m(m.prepare(u, 0, nq, nq + nk), gate)
        return o, m.k_cache, m.v_cache
    return _State(call)


def _prepare_latent(case, seed):
    from nano_qwen3tts_vllm_b200.config import LatentMixerSpec, RotarySpec
    from nano_qwen3tts_vllm_b200.layers.linear import release_packed
    from nano_qwen3tts_vllm_b200.models.ridevik import LatentAttentionMixer
    from nano_qwen3tts_vllm_b200.utils.context import set_context
    d, R, dr = _latent_inputs(case, seed), LATENT["rank"], LATENT["rot"]
    spec = LatentMixerSpec(HEADS, DIM, dr, DIM, R, 0, case["window"], (DIM + dr) ** -0.5, RotarySpec(dr, LATENT["theta"]), False)
    m = _module(lambda: LatentAttentionMixer(WIDTH, spec, EPS))
    _fill([(m.in_proj.weight, d["w_in"]), (m.kv_norm, d["norm"]), (m.uk, d["uk"]), (m.uv, d["uv"]), (m.attn.sink, d["sink"]),
           (m.o_proj.weight, d["o"])])
    lay, h, cache = _layout(d["seqs"], d["tables"]), d["h"], d["cache"]

    def call():
        set_context(False, step_layout=lay)
        with torch.inference_mode():
            return m(h, cache), cache
    return _State(call, lambda: release_packed(m))


def _prepare_ssm(case, seed):
    from nano_qwen3tts_vllm_b200.config import StateSpaceSpec
    from nano_qwen3tts_vllm_b200.layers.recurrent import StateSpaceMemory
    d, H, P, N = _ssm_inputs(case, seed), SSM["heads"], SSM["vdim"], SSM["state"]
    m = _module(lambda: StateSpaceMemory(StateSpaceSpec(H, P, N, 1, SSM["taps"], 1), EPS))
    _fill([(m.conv.weight, d["conv"]), (m.conv.bias, d["conv_b"]), (m.dt_bias, d["dt_bias"]), (m.A_log, d["A_log"]), (m.D, d["D"]),
           (m.norm, d["norm"])])
    return _prepare_memory(m, d, {"in": 0})


def _prepare_delta(case, seed):
    from nano_qwen3tts_vllm_b200.config import DeltaRuleSpec
    from nano_qwen3tts_vllm_b200.layers.recurrent import DeltaRuleMemory
    d, nk, nv = _delta_inputs(case, seed), KV_HEADS * DIM, HEADS * DIM
    m = _module(lambda: DeltaRuleMemory(DeltaRuleSpec(HEADS, KV_HEADS, DIM, DIM, 4), EPS))
    _fill([(m.conv.weight, d["conv"]), (m.A_log, d["A_log"]), (m.dt_bias, d["dt_bias"]), (m.norm, d["norm"])])
    return _prepare_memory(m, d, {"q": 0, "k": nk, "v": 2 * nk, "g": 2 * nk + nv, "b": 2 * nk + 2 * nv, "a": 2 * nk + 2 * nv + HEADS})


def _prepare_memory(m, d, cols):
    from nano_qwen3tts_vllm_b200.utils.context import set_context
    state = [torch.zeros(len(d["seqs"]), *shape, dtype=dt or BF, device=DEV) for shape, dt in m.state_plan()]
    m.bind(state)
    lay, u = _layout(d["seqs"], _tables(d["seqs"], 0)[0]), d["u"]

    def call():
        set_context(False, step_layout=lay)
        with torch.inference_mode():
            return m(u, cols), state
    return _State(call)


_PREPARE = {"talker": _prepare_stack, "predictor": _prepare_stack, "talker_layer": _prepare_layer, "experts": _prepare_experts,
            "lm_prompt": _prepare_lm, "sink_prompt": _prepare_sink, "sink_decode": _prepare_sink, "latent": _prepare_latent,
            "state_space": _prepare_ssm, "delta_rule": _prepare_delta}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state.call()


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _pairs(seqs, window=0, chunk=0, keep=0):
    """(query, key) pairs that the mask lets through, and the distinct keys read."""
    pairs = keys = 0
    for c, n in seqs:
        lo_first = 0
        for i in (range(c, c + n) if window or chunk else ()):
            lo = max(0, i - window + 1) if window else i // chunk * chunk
            pairs += i - lo + 1 + min(keep, lo)
        if not (window or chunk):
            pairs += n * c + n * (n + 1) // 2
        else:
            lo_first = max(0, c - window + 1) if window else c // chunk * chunk
        keys += c + n - lo_first + min(keep, lo_first)
    return pairs, keys


def work(case):
    k = case["kind"]
    if k in ("talker", "predictor"):
        s = TALKER if k == "talker" else PREDICTOR
        D, I, q, kv = s["hidden"], s["inter"], HEADS * DIM, KV_HEADS * DIM
        params = s["layers"] * (D * (2 * q + 2 * kv) + 3 * D * I) + s["vocab"] * D + (s["in_hidden"] * D if k == "predictor" else 0)
        lens = _contexts(case["context"], case["streams"]) if k == "talker" else [case["step"] + 2] * case["streams"]
        b = case["streams"]
        return {"bytes": 2.0 * params + 4.0 * kv * s["layers"] * sum(lens) + b * (4.0 * D + 2 * s["vocab"]),
                "flops": 2.0 * params * b + 4.0 * q * s["layers"] * sum(lens)}
    if k == "experts":
        n, mats = case["tokens"], 3 * WIDTH * EXPERT_FF
        extra = 1 if case["form"] == "clamped" else 0
        used = min(EXPERTS, n * TOP) + extra
        return {"bytes": 2.0 * mats * used + 2.0 * WIDTH * n * (1 + TOP + extra), "flops": 2.0 * mats * n * (TOP + extra)}
    seqs = _seqs(case)
    n = sum(m for _, m in seqs)
    if k == "talker_layer":
        D, I, q, kv = TALKER["hidden"], TALKER["inter"], HEADS * DIM, KV_HEADS * DIM
        params = D * (2 * q + 2 * kv) + 3 * D * I
        return {"bytes": 2.0 * params + n * (8.0 * D + 4 * kv), "flops": 2.0 * params * n + 4.0 * q * _pairs(seqs)[0]}
    if k == "lm_prompt":
        q, kv = HEADS * DIM, KV_HEADS * DIM
        params = LM["layers"] * (WIDTH * (2 * q + 2 * kv) + 2 * WIDTH * LM["ff"])
        head = LM["vocab"] * WIDTH
        return {"bytes": 2.0 * (params + head) + n * (2.0 * WIDTH + 4 * kv * LM["layers"]) + len(seqs) * 4.0 * LM["vocab"],
                "flops": 2.0 * params * n + 2.0 * head * len(seqs) + 4.0 * q * LM["layers"] * _pairs(seqs, WINDOW)[0]}
    if k in ("sink_prompt", "sink_decode"):
        form, nq, nk = case["form"], HEADS * DIM, KV_HEADS * DIM
        pairs, keys = _pairs(seqs, WINDOW if form == "window" else 0, WINDOW if form == "chunk" else 0, 4 if form == "window" else 0)
        gates = {"window": nq, "chunk": HEADS, "capped": 0}[form]
        return {"bytes": n * 2.0 * (nq + 2 * nk + gates + nq + 2 * nk) + 4.0 * nk * (keys - n), "flops": 4.0 * nq * pairs}
    if k == "latent":
        R, dr = LATENT["rank"], LATENT["rot"]
        pairs, keys = _pairs(seqs, case["window"])
        params = WIDTH * (HEADS * (DIM + dr) + R + dr) + HEADS * DIM * WIDTH + 2 * HEADS * DIM * R
        expand = 2.0 * HEADS * (2 * DIM + dr) * pairs + 4.0 * HEADS * DIM * R * keys      # keys and values of every head formed once
        absorb = 2.0 * HEADS * (2 * R + dr) * pairs + 4.0 * HEADS * DIM * R * n           # or the queries taken into the latent space
        return {"bytes": 2.0 * params + n * 2.0 * (2 * WIDTH + R + dr) + 2.0 * (R + dr) * (keys - n),
                "flops": 2.0 * n * (params - 2 * HEADS * DIM * R) + min(expand, absorb)}
    if k == "state_space":
        H, P, N = SSM["heads"], SSM["vdim"], SSM["state"]
        return {"bytes": n * 2.0 * (3 * H * P + 2 * N + H) + len(seqs) * 4.0 * H * P * N, "flops": n * H * P * N * 6.0}
    return {"bytes": n * 2.0 * (2 * KV_HEADS * DIM + 3 * HEADS * DIM + 2 * HEADS) + len(seqs) * 4.0 * HEADS * DIM * DIM,
            "flops": n * HEADS * DIM * DIM * 8.0}


def tolerance(case):
    """About four times the distance from ``exact`` that bfloat16 activations were seen to cause; 28 layers of random weights
    multiply it (4e-2 seen), so the whole talker gets somewhat less."""
    return {"talker": {"rel": 1e-1}, "predictor": {"rel": 5e-2}, "talker_layer": {"rel": 2.5e-2}, "experts": {"rel": 1.5e-2},
            "lm_prompt": {"rel": 2.5e-2}, "sink_prompt": {"rel": 1e-2}, "sink_decode": {"rel": 1e-2}, "latent": {"rel": 2e-2},
            "state_space": {"rel": 1e-2}, "delta_rule": {"rel": 1e-2}}[case["kind"]]


# ------------------------------------------------------------------------------------------------ the same answers in 64 bits
def _rms(x, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _rope_half(v, pos, theta):
    """v [n, heads, d]: coordinate i with i + d/2."""
    d = v.shape[-1]
    ang = pos.double()[:, None] * theta ** (-torch.arange(0, d, 2, device=DEV, dtype=F64) / d)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = v[..., :d // 2], v[..., d // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _rope_pairs(v, pos, dims, theta, factor=1.0):
    """v [n, heads, d]: coordinate 2i with 2i + 1, the first ``dims`` of them."""
    ang = pos.double()[:, None] * theta ** (-torch.arange(0, dims, 2, device=DEV, dtype=F64) / dims) / factor
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = v[..., 0:dims:2], v[..., 1:dims:2]
    return torch.cat([torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2), v[..., dims:]], -1)


def _attend(q, k, v, first, see, score=lambda s: s, sink=None, weights=None):
    """q [n, H, d] at positions first .. first + n - 1 over k, v [T, G, .]; ``see(i, j)`` the mask, ``score`` on the products,
    ``sink`` [H] (or None) joins the denominator, ``weights(h, scores, distance)`` replaces the softmax."""
    n, H, rep = q.shape[0], q.shape[1], q.shape[1] // k.shape[1]
    i = torch.arange(first, first + n, device=DEV)[:, None]
    j = torch.arange(k.shape[0], device=DEV)[None]
    ok, out = (j <= i) & see(i, j), []
    for h in range(H):
        s = score(q[:, h] @ k[:, h // rep].T)
        if weights is not None:
            p = weights(h, s, (i - j).clamp(min=0).double()) * ok
        else:
            s = s.masked_fill(~ok, -math.inf)
            m = s.amax(-1, keepdim=True) if sink is None else torch.maximum(s.amax(-1, keepdim=True), sink[h])
            e = torch.exp(s - m)
            p = e / (e.sum(-1, keepdim=True) + (0 if sink is None else torch.exp(sink[h] - m)))
        out.append(p @ v[:, h // rep])
    return torch.stack(out, 1)


def _everything(i, j):
    return torch.ones_like(i + j, dtype=torch.bool)


def _conv(u, w, bias=None):
    """u [n, C], w [C, taps]: causal, the last tap on the row itself."""
    t = w.shape[1]
    pad = torch.cat([u.new_zeros(t - 1, u.shape[1]), u])
    y = sum(pad[j:j + u.shape[0]] * w[:, j] for j in range(t))
    return y if bias is None else y + bias


def _exact_layer(w, p, y, pos, attend):
    """One talker or predictor layer on the residual stream ``y`` [n, D]."""
    W = lambda name: w[f"{p}{name}.weight"].double()
    n = y.shape[0]
    h = _rms(y, W("input_layernorm"))
    q = _rms((h @ W("self_attn.q_proj").T).view(n, HEADS, DIM), W("self_attn.q_norm"))
    k = _rms((h @ W("self_attn.k_proj").T).view(n, KV_HEADS, DIM), W("self_attn.k_norm"))
    v = (h @ W("self_attn.v_proj").T).view(n, KV_HEADS, DIM)
    o = attend(_rope_half(q, pos, 1e6), _rope_half(k, pos, 1e6), v)
    y = y + o.reshape(n, -1) @ W("self_attn.o_proj").T
    h = _rms(y, W("post_attention_layernorm"))
    return y, (F.silu(h @ W("mlp.gate_proj").T) * (h @ W("mlp.up_proj").T)) @ W("mlp.down_proj").T


def _exact_stack(case, seed):
    w, x, kv, seqs, tables = _stack_inputs(case, seed)
    talker = case["kind"] == "talker"
    if talker:
        y, pos, rest = x.double(), torch.tensor([c + 1 for c, _ in seqs], device=DEV), "codec_head.weight"   # its decode positions are the lengths
    else:
        e = w[f"model.codec_embedding.{case['step'] - 1}"].double()[x]
        y = e @ w["small_to_mtp_projection.weight"].double().T + w["small_to_mtp_projection.bias"].double()
        pos, rest = torch.tensor([c for c, _ in seqs], device=DEV), f"lm_head.{case['step']}"
    slots, kv = _slots(seqs, tables), kv.double()
    last = torch.stack([s[-1] for s in slots])
    for i in range(kv.shape[1]):
        rows = kv[:, i].view(2, -1, KV_HEADS, DIM)

        def attend(q, k, v):
            out = []
            rows[0, last], rows[1, last] = k, v
            for b, s in enumerate(slots):
                kk, vv = rows[0, s], rows[1, s]
                sc = torch.einsum("grd,tgd->grt", q[b].view(KV_HEADS, -1, DIM), kk) * DIM ** -0.5
                out.append(torch.einsum("grt,tgd->grd", sc.softmax(-1), vv).reshape(HEADS, DIM))
            return torch.stack(out)
        y, m = _exact_layer(w, f"model.layers.{i}.", y, pos, attend)
        y = y + m
    h = _rms(y, w["model.norm.weight"].double())
    logits = h @ w[rest].double().T
    return ((logits, h) if talker else logits), kv


def _exact_prompt_layer(case, seed):
    w, seqs = _talker_weights(seed, TALKER, 1), _seqs(case)
    tables, pages = _tables(seqs, seed)
    r, n = _Rand(seed + 1), sum(m for _, m in seqs)
    x, res = r(n, TALKER["hidden"], std=0.5), r(n, TALKER["hidden"], std=0.5)
    pos = torch.cat([torch.arange(m, device=DEV) for _, m in seqs])
    kc, vc = (torch.zeros(pages * PAGE, KV_HEADS, DIM, dtype=F64, device=DEV) for _ in range(2))

    def attend(q, k, v):
        out, o = [], 0
        for (_, m), s in zip(seqs, _slots(seqs, tables)):
            kc[s], vc[s] = k[o:o + m], v[o:o + m]
            out.append(_attend(q[o:o + m], k[o:o + m], v[o:o + m], 0, _everything, lambda t: t * DIM ** -0.5))
            o += m
        return torch.cat(out)
    y, m = _exact_layer(w, "model.layers.0.", x.double() + res.double(), pos, attend)
    return m, y, kc, vc


def _exact_experts(case, seed):
    d = {k: v.double() for k, v in _expert_inputs(case, seed).items()}
    h, n = d["h"], case["tokens"]
    silu = case["form"] == "silu"

    def inner(gu):
        g, u = gu[:, :EXPERT_FF], gu[:, EXPERT_FF:]
        if silu:
            return F.silu(g) * u
        g, u = g.clamp(max=LIMIT), u.clamp(-LIMIT, LIMIT)
        return g * torch.sigmoid(1.702 * g) * (u + 1)
    s = h @ d["router"].T
    if silu:
        val, idx = torch.topk(s + d["bias"], TOP, -1)
        wt = val.softmax(-1)
    else:
        s = s.softmax(-1)
        best = s.view(n, GROUPS, -1).amax(-1).argmax(-1)
        kept = torch.zeros(n, GROUPS, dtype=torch.bool, device=DEV).scatter_(1, best[:, None], True).repeat_interleave(EXPERTS // GROUPS, 1)
        idx = torch.topk(s.masked_fill(~kept, -1.0), TOP, -1).indices
        wt = s.gather(1, idx)
    z = torch.zeros(n * TOP, WIDTH, dtype=F64, device=DEV)
    flat = idx.reshape(-1)
    for e in range(EXPERTS):
        p = (flat == e).nonzero()[:, 0]
        z[p] = inner(h[p // TOP] @ d["up"][e].T) @ d["down"][e].T
    return (z, wt) if silu else (z, wt, inner(h @ d["shared_gate_up"].T) @ d["shared_down"].T)


def _exact_lm(case, seed):
    sd, tokens, seqs = _lm_inputs(case, seed)
    sd = {k: v.double() for k, v in sd.items()}
    tok, out, o = torch.tensor(tokens, device=DEV), [], 0
    for _, n in seqs:
        x = sd["embed"][tok[o:o + n]] + sd["pos"][:n]
        o += n
        for i in range(LM["layers"]):
            p = lambda name: sd[f"l{i}.{name}"]
            h = _rms(x) * p("norm1")
            q, k, v = (_conv(h @ p(f"mix.{c}").T, p(f"mix.{c}.conv")).view(n, -1, DIM) for c in "qkv")
            wt = lambda hh, s, dist: torch.sigmoid(s - p("mix.r1")[hh] * torch.log1p(p("mix.r2")[hh] * dist) + p("mix.pb")[hh])
            a = _attend(_rms(q, p("mix.q.norm")), _rms(k, p("mix.k.norm")), v, 0, lambda i_, j: i_ - j < WINDOW, lambda s: s * DIM ** -0.5, weights=wt)
            ff = torch.relu(h @ p("mlp.up").T) ** 2 @ p("mlp.down").T
            x = x + LM["mult"] * (a.reshape(n, -1) @ p("mix.o").T + ff)
        out.append((_rms(x[-1:]) * sd["final.norm"]) @ sd["head"].T)
    return torch.cat(out)


def _exact_sink(case, seed):
    d, form = _sink_inputs(case, seed), case["form"]
    u, nq, nk = d["u"].double(), HEADS * DIM, KV_HEADS * DIM
    kc, vc = d["k"].double().view(-1, KV_HEADS, DIM), d["v"].double().view(-1, KV_HEADS, DIM)
    see = {"window": lambda i, j: (i - j < WINDOW) | (j < 4), "chunk": lambda i, j: i // WINDOW == j // WINDOW, "capped": _everything}[form]
    score = (lambda s: 50.0 * torch.tanh(s * DIM ** -0.5 / 50.0)) if form == "capped" else (lambda s: s * DIM ** -0.5)
    sink = {"window": None, "chunk": d["sink"].double() if "sink" in d else None, "capped": torch.zeros(HEADS, dtype=F64, device=DEV)}[form]
    out, o = [], 0
    for (c, n), s in zip(d["seqs"], _slots(d["seqs"], d["tables"])):
        x, pos = u[o:o + n], torch.arange(c, c + n, device=DEV)
        q = (x[:, :nq] + d["qb"].double()).view(n, HEADS, DIM)
        k = (x[:, nq:nq + nk] + d["kb"].double()).view(n, KV_HEADS, DIM)
        if form == "window":
            q, k = (_rope_pairs(_rms(t, d[w].double()), pos, DIM, 1e6) for t, w in ((q, "qn"), (k, "kn")))
        elif form == "capped":
            q, k = (_rope_pairs(t, pos, DIM // 2, 1e4, 2.0) for t in (q, k))
        kc[s[c:]], vc[s[c:]] = k, (x[:, nq + nk:nq + 2 * nk] + d["vb"].double()).view(n, KV_HEADS, DIM)
        a = _attend(q, kc[s], vc[s], c, see, score, sink)
        if form == "window":
            a = a * torch.sigmoid(x[:, nq + 2 * nk:]).view(n, HEADS, DIM)
        elif form == "chunk":
            a = a * torch.sigmoid(x[:, nq + 2 * nk:])[:, :, None]
        out.append(a.reshape(n, -1))
        o += n
    return torch.cat(out), kc.view(-1, PAGE, nk), vc.view(-1, PAGE, nk)


def _exact_latent(case, seed):
    d, R, dr = _latent_inputs(case, seed), LATENT["rank"], LATENT["rot"]
    u = d["h"].double() @ d["w_in"].double().T
    qs = HEADS * (DIM + dr)
    cache = d["cache"].double().view(-1, R + dr)
    see = (lambda i, j: i - j < case["window"]) if case["window"] else _everything
    scale, uk, uv, sink = (DIM + dr) ** -0.5, d["uk"].double(), d["uv"].double(), d["sink"].double()
    out, o = [], 0
    for (c, n), s in zip(d["seqs"], _slots(d["seqs"], d["tables"])):
        x, pos = u[o:o + n], torch.arange(c, c + n, device=DEV)
        q = x[:, :qs].view(n, HEADS, DIM + dr)
        q = torch.cat([q[..., :DIM], _rope_pairs(q[..., DIM:], pos, dr, LATENT["theta"])], -1)
        cache[s[c:]] = torch.cat([_rms(x[:, qs:qs + R], d["norm"].double()), _rope_pairs(x[:, None, qs + R:], pos, dr, LATENT["theta"])[:, 0]], -1)
        lat, kr = cache[s, :R], cache[s, None, R:].expand(-1, HEADS, dr)
        k = torch.cat([torch.einsum("tr,hdr->thd", lat, uk), kr], -1)
        out.append(_attend(q, k, torch.einsum("tr,hdr->thd", lat, uv), c, see, lambda t: t * scale, sink).reshape(n, -1))
        o += n
    return torch.cat(out) @ d["o"].double().T, cache.view(-1, PAGE, R + dr)


def _exact_ssm(case, seed):
    d, H, P, N = _ssm_inputs(case, seed), SSM["heads"], SSM["vdim"], SSM["state"]
    D = {k: v.double() for k, v in d.items() if torch.is_tensor(v)}
    inner, ch = H * P, H * P + 2 * N
    outs, convs, states, o = [], [], [], 0
    for _, n in d["seqs"]:
        u = D["u"][o:o + n]
        o += n
        xbc = F.silu(_conv(u[:, inner:inner + ch], D["conv"], D["conv_b"]))
        x, B, C = xbc[:, :inner].view(n, H, P), xbc[:, inner:inner + N], xbc[:, inner + N:]
        dt = F.softplus(u[:, inner + ch:] + D["dt_bias"])
        la, S, ys = -torch.exp(D["A_log"]) * dt, u.new_zeros(H, N, P), []
        for a in range(0, n, 128):                                               # the recurrence in blocks: decays inside a block by differences of sums
            e = slice(a, min(a + 128, n))
            cum = la[e].cumsum(0)                                                # [L, H]
            L = cum.shape[0]
            G = torch.exp((cum[:, None] - cum[None]).clamp(max=0)) * torch.ones(L, L, device=DEV, dtype=F64).tril()[..., None]
            M = (C[e] @ B[e].T)[..., None] * G * dt[e][None]
            ys.append(torch.einsum("ijh,jhp->ihp", M, x[e]) + torch.einsum("in,hnp->ihp", C[e], S) * cum.exp()[..., None])
            S = S * cum[-1].exp()[:, None, None] + torch.einsum("jn,jh,jhp->hnp", B[e], torch.exp(cum[-1] - cum) * dt[e], x[e])
        y = (torch.cat(ys) + D["D"][:, None] * x).reshape(n, inner) * F.silu(u[:, :inner])
        outs.append(_rms(y, D["norm"]))
        convs.append(_last_rows(u[:, inner:inner + ch], SSM["taps"] - 1))
        states.append(S)
    return torch.cat(outs), [torch.stack(convs), torch.stack(states)]


def _last_rows(u, k):
    return torch.cat([u.new_zeros(k, u.shape[1]), u])[-k:]


def _exact_delta(case, seed):
    d = _delta_inputs(case, seed)
    D = {k: v.double() for k, v in d.items() if torch.is_tensor(v)}
    nk, nv = KV_HEADS * DIM, HEADS * DIM
    rep = HEADS // KV_HEADS
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    outs, convs, states, o = [], [], [], 0
    for _, n in d["seqs"]:
        u = D["u"][o:o + n]
        o += n
        qkv = F.silu(_conv(u[:, :2 * nk + nv], D["conv"]))
        q = (unit(qkv[:, :nk].view(n, KV_HEADS, DIM)) * DIM ** -0.5).repeat_interleave(rep, 1).transpose(0, 1)
        k = unit(qkv[:, nk:2 * nk].view(n, KV_HEADS, DIM)).repeat_interleave(rep, 1).transpose(0, 1)
        v = qkv[:, 2 * nk:].view(n, HEADS, DIM).transpose(0, 1)
        ba = u[:, 2 * nk + 2 * nv:]
        beta = torch.sigmoid(ba[:, :HEADS]).T
        la = (-torch.exp(D["A_log"]) * F.softplus(ba[:, HEADS:] + D["dt_bias"])).T
        S, ys = u.new_zeros(HEADS, DIM, DIM), []
        for a in range(0, n, 64):                                                # written values of a block by one triangular solve
            e = slice(a, min(a + 64, n))
            cum = la[:, e].cumsum(1)
            L = cum.shape[1]
            G = torch.exp((cum[:, :, None] - cum[:, None]).clamp(max=0))
            K, Q, b = k[:, e], q[:, e], beta[:, e, None]
            A = torch.eye(L, device=DEV, dtype=F64) + ((K @ K.transpose(1, 2)) * G * b).tril(-1)
            U = torch.linalg.solve_triangular(A, b * (v[:, e] - cum.exp()[..., None] * (K @ S)), upper=False)
            ys.append(((Q @ K.transpose(1, 2)) * G).tril() @ U + cum.exp()[..., None] * (Q @ S))
            S = S * cum[:, -1].exp()[:, None, None] + (K * torch.exp(cum[:, -1:] - cum)[..., None]).transpose(1, 2) @ U
        y = _rms(torch.cat(ys, 1).transpose(0, 1), D["norm"]).reshape(n, nv)
        outs.append(y * F.silu(u[:, 2 * nk + nv:2 * nk + 2 * nv]))
        convs.append(_last_rows(u[:, :2 * nk + nv], 3))
        states.append(S)
    return torch.cat(outs), [torch.stack(convs), torch.stack(states)]


_EXACT = {"talker": _exact_stack, "predictor": _exact_stack, "talker_layer": _exact_prompt_layer, "experts": _exact_experts,
          "lm_prompt": _exact_lm, "sink_prompt": _exact_sink, "sink_decode": _exact_sink, "latent": _exact_latent,
          "state_space": _exact_ssm, "delta_rule": _exact_delta}


@torch.no_grad()
def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)
