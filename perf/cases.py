"""The work whose speed this framework is judged by: generation (bf16, int8 and int4 weights; one row
to large batches; short and long prompts; many and few kv heads), scoring of given sequences,
training steps, and the hybrid decoders, each through the entry point that a user's program calls.

A model here is a slice of a configured one: the layer shapes, head counts and vocabulary are those of
``transformer_configs`` and of ``bench/hybrid_shapes.py``, the number of layers is a few. Weights are
random, scaled like a trained model's: residual branches add to the stream without drowning the
embedding, and the head is confident about the next token (a fixed successor of the current one), so
that a greedy choice or a draw at the usual temperatures does not hang on the last bit of a logit.
Of the experts of a hybrid layer all are chosen, with unequal weights, for the same reason.
"""
import math

import torch

# width, heads, kv heads, feed-forward, vocabulary, RoPE base of the configured models
SHAPES = {
    "tiny-llama": (256, 4, 4, 688, 1024, 10000.0),
    "7B": (4096, 32, 32, 11008, 32016, 1000000.0),
    "13B": (5120, 40, 40, 13824, 32000, 10000.0),
    "34B": (8192, 64, 8, 22016, 32000, 1000000.0),
}
EPS = 1e-5
# width, heads, kv heads, window, GLA heads, dense ff, expert ff, latent expert ff, shared ff
HYBRID = {"2k": (2048, 16, 4, 1024, 8, 8192, 2752, 3440, 1376)}
HYBRID_VOCAB, EXPERTS = 32000, 4
GLA_DIM, GLA_VDIM, GLA_TAU, GLA_RANK = 128, 256, 16.0, 16
YARN = dict(factor=4.0, original=4096, fast=32.0, slow=1.0)
RANK, LATENT_DIM, LATENT_ROT, LATENT_VDIM = 512, 128, 64, 128


def _gen(name, shape, layers, batch, prompt, new, weights="bf16", padded=False, temperature=0.7,
         top_k=50):
    return dict(name=name, kind="generate", shape=shape, layers=layers, batch=batch, prompt=prompt,
                new=new, weights=weights, padded=padded, temperature=temperature, top_k=top_k)


def listed():
    return [
        # the plumbing configuration, four short prompts: nothing but latency and launches
        _gen("tiny_generate", "tiny-llama", 2, 4, 32, 16),
        # one user at a prompt (the interactive program's sampling): the weight stream at one row
        _gen("chat_one_row", "7B", 8, 1, 61, 48, temperature=0.8, top_k=200),
        # the headline workload: 64 prompts of unequal length, left padded, then many decode steps
        _gen("batch64_decode", "7B", 8, 64, 256, 96, padded=True),
        # the same with weight-only int8, as rollouts and large evaluations run it
        _gen("int8_batch64", "7B", 8, 64, 128, 64, weights="int8"),
        # weight-only int4 (groups of 128) for a handful of rows
        _gen("int4_batch8", "7B", 8, 8, 203, 64, weights="int4", padded=True),
        # eight query heads per kv head, few long samples (best-of-N on the largest model)
        _gen("gqa_34b_batch32", "34B", 3, 32, 701, 48),
        # prompts near the context limit and a short answer: prefill
        _gen("long_prompt", "7B", 4, 4, 4000, 8, padded=True),
        # process-reward scoring of 64 samples of one problem (256 + 512 tokens), right padded
        dict(name="reward_scoring", kind="score", shape="7B", layers=4, batch=64, seq=768),
        # full-parameter fine-tuning step: 16 sequences of 768 tokens, loss on the responses
        dict(name="sft_step", kind="train", loss="sft", shape="7B", layers=2, batch=16, seq=768),
        # process-reward training step of the next size up, a short ragged batch
        dict(name="prm_step", kind="train", loss="prm", shape="13B", layers=1, batch=5, seq=1003),
        # hybrid decoders: prompts and decode steps of attention, gated linear attention, latent
        # attention, dense and expert feed-forwards
        dict(name="bovinex_generate", kind="hybrid", design="Bovinex", shape="2k", layers=4,
             batch=32, prompt=512, new=48, padded=True),
        dict(name="ruralorn_generate", kind="hybrid", design="Ruralorn", shape="2k", layers=4,
             batch=32, prompt=512, new=48, padded=True),
    ]


def draw(rng):
    """One more case of the same ranges: batch, prompt, new tokens, layers and sequence length vary
    (log-uniformly), odd values among them, bounded so that no case outgrows the listed ones."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["generate"] * 7 + ["score", "train", "train", "hybrid", "hybrid"])
    while True:
        if kind == "generate":
            shape = rng.choice(["tiny-llama", "7B", "7B", "7B", "13B", "34B"])
            weights = "bf16" if shape == "tiny-llama" else rng.choice(["bf16", "bf16", "int8", "int4"])
            hi = {"tiny-llama": 2, "7B": 8, "13B": 5, "34B": 3}[shape]
            c = _gen("", shape, rng.randint(max(1, hi // 2), hi), log(1, 64),
                     log(24, 120 if shape == "tiny-llama" else 4000), log(8, 96), weights=weights,
                     padded=rng.random() < 0.5, temperature=rng.choice([0.7, 0.8, 1.0]),
                     top_k=rng.choice([20, 50, 200]))
            fits = c["batch"] * c["prompt"] <= 16384
        elif kind == "score":
            c = dict(kind="score", shape=rng.choice(["7B", "13B"]), layers=rng.randint(1, 4),
                     batch=log(2, 64), seq=log(100, 2048))
            fits = c["batch"] * c["seq"] <= 32768
        elif kind == "train":
            c = dict(kind="train", loss=rng.choice(["sft", "prm"]), shape=rng.choice(["7B", "13B"]),
                     layers=1, batch=log(1, 16), seq=log(128, 1024))
            fits = True
        else:
            c = dict(kind="hybrid", design=rng.choice(["Bovinex", "Ruralorn"]), shape="2k",
                     layers=rng.randint(2, 4), batch=log(1, 48), prompt=log(32, 1500),
                     new=log(8, 64), padded=rng.random() < 0.5)
            fits = c["batch"] * c["prompt"] <= 16384
        if fits:
            c.pop("name", None)
            return c


# ------------------------------------------------------------------------------ inputs and weights

def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, rows, cols, std):
    return torch.empty(rows, cols, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=g)


def _successor(vocab):
    """The token that follows each token with near certainty."""
    return (torch.arange(vocab, device="cuda") * 7 + 3) % vocab


def _confident_head(g, embed, std, share):
    """Head rows: noise, plus the embedding of the token before; ``share``: how much of a normed
    hidden state is the current token's embedding."""
    vocab, dim = embed.shape
    head = _normal(g, vocab, dim, std)
    e = embed.float()
    e = e * (25.0 / (share * dim)) / e.pow(2).mean().sqrt()
    head[_successor(vocab)] += e.to(torch.bfloat16)
    return head


class _Quantised:
    """Codes [out, in] with per-row (int8) or per-group (int4) scales; ``dense`` in 64 bits."""

    def __init__(self, g, rows, cols, std, bits):
        noise = torch.empty(rows, cols, device="cuda").normal_(generator=g)
        spread = torch.empty(rows, max(1, cols // 128), device="cuda").uniform_(0.8, 1.2, generator=g)
        self.bits = bits
        if bits == 8:
            self.codes = (noise * 32).round_().clamp_(-127, 127).to(torch.int8)
            self.scales = (spread[:, 0] * std / 32).to(torch.bfloat16)
        else:
            self.codes = (noise * 2.7 + 7.5).round_().clamp_(0, 15).to(torch.int32)
            self.scales = (spread * std / 2.7).to(torch.bfloat16)
            self.zeros = (self.scales.float() * 0.5).to(torch.bfloat16)

    def dense(self):
        if self.bits == 8:
            return self.codes.double() * self.scales.double()[:, None]
        rows, cols = self.codes.shape
        q = self.codes.double().view(rows, cols // 128, 128) - 8
        return (q * self.scales.double()[..., None] + self.zeros.double()[..., None]).view(rows, cols)


def _llama_weights(case, seed):
    """name -> bf16 tensor, or codes with scales."""
    W, H, G, ff, V, _ = SHAPES[case["shape"]]
    g, L = _rng(seed), case["layers"]
    bits = {"bf16": 16, "int8": 8, "int4": 4}[case.get("weights", "bf16")]

    def linear(rows, cols, std):
        return _normal(g, rows, cols, std) if bits == 16 else _Quantised(g, rows, cols, std, bits)
    w = {"embed": _normal(g, V, W, 1.0)}
    a, down = 1.28 / math.sqrt(W), 1.28 / math.sqrt(2 * L)
    for i in range(L):
        w[f"{i}.wqkv"] = linear((H + 2 * G) * (W // H), W, a)
        w[f"{i}.wo"] = linear(W, W, down / math.sqrt(W))
        w[f"{i}.w1"] = linear(ff, W, a)
        w[f"{i}.w3"] = linear(ff, W, a)
        w[f"{i}.w2"] = linear(W, ff, down / math.sqrt(ff))
        for n in ("n1", "n2"):
            w[f"{i}.{n}"] = (1 + 0.1 * _normal(g, 1, W, 1.0))[0]
    w["norm"] = (1 + 0.1 * _normal(g, 1, W, 1.0))[0]
    w["head"] = _confident_head(g, w["embed"], 1.28 / math.sqrt(W), 0.7)
    return w


def _tokens(case, seed, rows, cols, vocab):
    """Random ids [rows, cols], none 0, and the left-pad counts of the rows (up to half a row)."""
    g = _rng(seed + 7919)
    ids = torch.randint(1, vocab, (rows, cols), generator=g, device="cuda", dtype=torch.int32)
    pads = torch.randint(0, cols // 2 + 1, (rows,), generator=g, device="cuda", dtype=torch.int32)
    pads[0] = 0
    if not case.get("padded"):
        return ids, None
    ids[torch.arange(cols, device="cuda")[None] < pads[:, None]] = 0
    return ids, pads


def _assign(module, name, value):
    """Put ``value`` in the place of a parameter or buffer."""
    old = module._parameters.get(name)
    if old is not None:
        module._parameters[name] = torch.nn.Parameter(value, requires_grad=old.requires_grad)
    else:
        module._buffers[name] = value


def _fill_llama(model, w):
    _assign(model.tok_embeddings, "weight", w["embed"])
    _assign(model.norm, "weight", w["norm"])
    _assign(model.output, "weight", w["head"])
    for i, blk in enumerate(model.layers):
        _assign(blk.attention_norm, "weight", w[f"{i}.n1"])
        _assign(blk.ffn_norm, "weight", w[f"{i}.n2"])
        for part, names in ((blk.attention, ("wqkv", "wo")), (blk.feed_forward, ("w1", "w3", "w2"))):
            for n in names:
                lin, v = getattr(part, n), w[f"{i}.{n}"]
                if isinstance(v, torch.Tensor):
                    _assign(lin, "weight", v)
                elif v.bits == 8:
                    _assign(lin, "weight", v.codes)
                    _assign(lin, "scales", v.scales)
                else:
                    from easy_to_hard_b200.models import quantize as qz
                    _assign(lin, "weight", qz.pack_int4_tinygemm(v.codes, lin.inner_k_tiles))
                    _assign(lin, "scales_and_zeros", qz.pack_scales_and_zeros(v.scales, v.zeros))


def _model_args(case):
    from easy_to_hard_b200.models.model import ModelArgs
    W, H, G, ff, V, base = SHAPES[case["shape"]]
    return ModelArgs(block_size=8192, vocab_size=V, n_layer=case["layers"], n_head=H, dim=W,
                     intermediate_size=ff, n_local_heads=G, rope_base=base, norm_eps=EPS)


def _prepare_generate(case, seed):
    from easy_to_hard_b200.models.engine import get_engine
    from easy_to_hard_b200.models.model import Transformer
    from easy_to_hard_b200.models.quantize import (WeightOnlyInt4QuantHandler,
                                                   WeightOnlyInt8QuantHandler)
    with torch.device("meta"):
        model = Transformer(_model_args(case), freeze_tok_embeddings=True, freeze_output=True,
                            freeze_norm=True).to(torch.bfloat16)
        if case["weights"] == "int8":
            model = WeightOnlyInt8QuantHandler(model).convert_for_runtime()
        elif case["weights"] == "int4":
            model = WeightOnlyInt4QuantHandler(model, 128).convert_for_runtime()
    _fill_llama(model, _llama_weights(case, seed))
    return _generation_state(case, seed, model.eval(), SHAPES[case["shape"]][4], get_engine)


def _generation_state(case, seed, model, vocab, get_engine):
    B, T = case["batch"], case["prompt"]
    ids, pads = _tokens(case, seed, B, T, vocab)
    s = dict(kind="generate", model=model, ids=ids, pads=pads, new=case["new"], seed=seed % 1000,
             temperature=case.get("temperature", 0.7), top_k=case.get("top_k", 50), vocab=vocab)
    # a serving program has its engine, caches and captured step before the first prompt comes
    s["engine"] = get_engine(model, B, T + case["new"])
    warm = torch.ones(B, 8, dtype=torch.int32, device="cuda")
    s["engine"].generate(warm, None, 2, s["temperature"], s["top_k"])
    return s


def _prepare_score(case, seed):
    from easy_to_hard_b200.models.reward_model import (RewardArgs, RewardModel,
                                                       apply_reward_modeling_head)
    with torch.device("meta"):
        model = RewardModel(RewardArgs(backbone_args=_model_args(case)), freeze_tok_embeddings=True,
                            freeze_output=True, freeze_norm=True).to(torch.bfloat16)
    w = _llama_weights(case, seed)
    _fill_llama(model.backbone_model, w)
    apply_reward_modeling_head(model.backbone_model)
    model.backbone_model.output.weight.data.copy_(_reward_head(case, seed))
    return dict(kind="score", model=model.eval(), ids=_score_tokens(case, seed))


def _score_tokens(case, seed):
    """Right-padded samples, half to all of the row long."""
    ids, _ = _tokens({}, seed, case["batch"], case["seq"], SHAPES[case["shape"]][4])
    lengths = torch.randint(case["seq"] // 2, case["seq"] + 1, (case["batch"], 1),
                            generator=_rng(seed + 31), device="cuda")
    ids[torch.arange(case["seq"], device="cuda")[None] >= lengths] = 0
    return ids


def _reward_head(case, seed):
    W = SHAPES[case["shape"]][0]
    return _normal(_rng(seed + 5), 2, W, 1.28 / math.sqrt(W))


def _train_batch(case, seed):
    B, S = case["batch"], case["seq"]
    g = _rng(seed + 104729)
    ids = torch.randint(1, SHAPES[case["shape"]][4], (B, S), generator=g, device="cuda")
    if case["loss"] == "sft":
        start = torch.randint(min(64, S // 4), S // 2, (B, 1), generator=g, device="cuda")
        labels = ids.masked_fill(torch.arange(S, device="cuda")[None] < start, -100)
        return ids, labels
    labels = torch.randint(0, 2, (B, S), generator=g, device="cuda").float()
    weights = (torch.rand(B, S, generator=g, device="cuda") < 1 / 24).float()
    weights[:, -1] = 1.0
    return ids, labels, weights


TRAIN_LR, TRAIN_BETAS = 2e-5, (0.9, 0.95)


def _prepare_train(case, seed):
    from easy_to_hard_b200.models.model import Transformer
    from easy_to_hard_b200.models.reward_model import (RewardArgs, RewardModel,
                                                       apply_reward_modeling_head)
    from easy_to_hard_b200.parallel.fsdp import ShardedDataParallel
    from easy_to_hard_b200.training import SFTStepper, TrainStepper, pointwise_reward_loss
    from easy_to_hard_b200.utils.memory_efficient_adam import MemoryEfficientAdamW
    frozen = dict(freeze_tok_embeddings=True, freeze_output=True, freeze_norm=True)
    w = _llama_weights(case, seed)
    with torch.device("meta"):
        if case["loss"] == "sft":
            model = backbone = Transformer(_model_args(case), **frozen)
        else:
            model = RewardModel(RewardArgs(backbone_args=_model_args(case)), **frozen)
            backbone = model.backbone_model
    _fill_llama(backbone, w)
    if case["loss"] == "prm":
        apply_reward_modeling_head(backbone, requires_grad=True)
        backbone.output.weight.data.copy_(_reward_head(case, seed))
    sharded = ShardedDataParallel(model, process_group=None, param_dtype=torch.float32,
                                  compute_dtype=torch.bfloat16, reduce_dtype=torch.bfloat16)
    sharded.train()
    opt = MemoryEfficientAdamW(list(sharded.optimizer_parameters()), lr=TRAIN_LR,
                               betas=TRAIN_BETAS, weight_decay=0.0, optim_dtype=torch.float32,
                               optim_device=torch.device("cuda"))
    stepper = SFTStepper(sharded, opt) if case["loss"] == "sft" else \
        TrainStepper(sharded, opt, None, pointwise_reward_loss, 1.0)
    return dict(kind="train", stepper=stepper, model=sharded, batch=_train_batch(case, seed))


def _hybrid_description(case):
    """The checkpoint folder's ``config.json`` of the design, as a dict."""
    W, H, G, win, gh, ff, eff, leff, shared = HYBRID[case["shape"]]
    moe = dict(kind="moe", router=dict(experts=EXPERTS, top=EXPERTS), expert=dict(ff=eff))
    dense = dict(kind="dense", ff=ff)
    if case["design"] == "Bovinex":
        att = dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5,
                   rot=dict(dims=128, base=1e6, scaling=YARN), mask=dict(size=win, keep_first=4))
        gla = dict(heads=gh, dim=GLA_DIM, vdim=GLA_VDIM, tau=GLA_TAU)
        kinds = [("attention", att, dense), ("gla", gla, moe), ("gla", gla, dense),
                 ("attention", att, moe)]
        layers = [dict(type=t, mixer=m, mlp=f) for t, m, f in kinds]
        return dict(architecture="Bovinex", vocab=HYBRID_VOCAB, width=W, norm=dict(eps=EPS),
                    embedding=dict(scale=W ** 0.5), layers=layers[: case["layers"]])
    m = dict(heads=H, dim=LATENT_DIM, rot_dim=LATENT_ROT, vdim=LATENT_VDIM, kv_rank=RANK,
             scale=(LATENT_DIM + LATENT_ROT) ** -0.5, rot=dict(dims=LATENT_ROT, base=1e6),
             mask=dict(size=win))
    f = dict(moe, expert=dict(ff=leff), shared=dict(ff=shared))
    return dict(architecture="Ruralorn", vocab=HYBRID_VOCAB, width=W, norm=dict(eps=EPS),
                embedding=dict(scale=W ** 0.5), logit_scale=0.5, logit_softcap=30.0,
                layers=[dict(type="latent_attention", mixer=m, mlp=f)] * case["layers"])


def _hybrid_weights(case, seed):
    d, g, w = _hybrid_description(case), _rng(seed), {}
    W, L = d["width"], len(d["layers"])
    down = 1.0 / math.sqrt(2 * L)

    def lin(name, rows, cols, gain=1.0):
        w[name] = _normal(g, rows, cols, gain / math.sqrt(cols))

    def vec(name, n, mean=0.0, std=0.1):
        w[name] = (mean + std * torch.randn(n, generator=g, device="cuda")).to(torch.bfloat16)
    bov = d["architecture"] == "Bovinex"
    norm_mean = 0.0 if bov else 1.0
    w["embed"] = _normal(g, d["vocab"], W, W ** -0.5)
    for i, layer in enumerate(d["layers"]):
        p, m, f = f"l{i}.", layer["mixer"], layer["mlp"]
        H = m["heads"]
        vec(p + "norm1", W, norm_mean)
        if bov:
            kv = m.get("kv_heads", H)
            for n, rows in (("q", H * m["dim"]), ("k", kv * m["dim"]), ("v", kv * m["vdim"])):
                lin(p + "mix." + n, rows, W)
                if layer["type"] == "attention":
                    vec(p + f"mix.{n}.b", rows)
            if layer["type"] == "attention":
                vec(p + "mix.q.norm", H * m["dim"], 1.2)
                vec(p + "mix.k.norm", kv * m["dim"], 1.2)
            else:
                vec(p + "mix.norm", m["vdim"], 1.0)
                lin(p + "mix.a1", GLA_RANK, W)
                lin(p + "mix.a2", H * m["dim"], GLA_RANK, 2.0)
                vec(p + "mix.a2.b", H * m["dim"], 1.0, 1.0)
        else:
            lin(p + "mix.q", H * (m["dim"] + m["rot_dim"]), W, 1.2)
            lin(p + "mix.dkv", m["kv_rank"] + m["rot_dim"], W)
            vec(p + "mix.dkv.norm", m["kv_rank"], 1.0)
            lin(p + "mix.uk", H * m["dim"], m["kv_rank"])
            lin(p + "mix.uv", H * m["vdim"], m["kv_rank"])
            vec(p + "norm2", W, norm_mean)
        lin(p + "mix.g", H * m["vdim"], W)
        lin(p + "mix.o", W, H * m["vdim"], down * 2)
        if f["kind"] == "dense":
            lin(p + "mlp.up", f["ff"], W)
            lin(p + "mlp.down", W, f["ff"], down)
            continue
        lin(p + "mlp.router", f["router"]["experts"], W)
        if bov:
            vec(p + "mlp.router.b", f["router"]["experts"])
        for e in range(f["router"]["experts"]):
            for n in ("gate", "up") if bov else ("up",):
                lin(p + f"mlp.e{e}.{n}", f["expert"]["ff"], W)
            lin(p + f"mlp.e{e}.down", W, f["expert"]["ff"], down)
        if f.get("shared"):
            lin(p + "mlp.shared.up", f["shared"]["ff"], W)
            lin(p + "mlp.shared.down", W, f["shared"]["ff"], down)
    vec("final.norm", W, norm_mean)
    head = _confident_head(g, w["embed"], 1.28 / math.sqrt(W), 0.7)
    w["head"] = head if bov else (head.float() * 2).to(torch.bfloat16)   # logits are halved
    return w


def _prepare_hybrid(case, seed):
    from easy_to_hard_b200.models.engine import get_engine
    from easy_to_hard_b200.models.hybrid import HybridLM, hybrid_config
    model = HybridLM.from_tensors(hybrid_config(_hybrid_description(case)),
                                  _hybrid_weights(case, seed), device="cuda", dtype=torch.bfloat16)
    return _generation_state(case, seed, model, HYBRID_VOCAB, get_engine)


def prepare(case, seed):
    return {"generate": _prepare_generate, "score": _prepare_score, "train": _prepare_train,
            "hybrid": _prepare_hybrid}[case["kind"]](case, seed)


# ------------------------------------------------------------------------------ one pass

def run(s):
    if s["kind"] == "generate":
        import inference_generate
        seq, _ = inference_generate.generate(s["model"], s["ids"], s["pads"], s["new"],
                                             temperature=s["temperature"], top_k=s["top_k"],
                                             seed=s["seed"])
        return {"tokens": seq, "logits": s["engine"].logits[:, : s["vocab"]]}
    if s["kind"] == "score":
        import inference_reward
        return {"rewards": inference_reward.model_score(s["model"], s["ids"])}
    loss, norm = s["stepper"].step(*s["batch"])
    return {"loss": loss, "grad_norm": norm, "grads": list(s["model"].grad_shards()),
            "weights": [p.data for p in s["model"].optimizer_parameters()]}


# ------------------------------------------------------------------------------ bounds

def _hybrid_counts(case):
    """(weight elements of the layers, key and value columns read per position, state elements)."""
    d = _hybrid_description(case)
    W, params, kv, state = d["width"], 0, 0, 0
    for layer in d["layers"]:
        m, f = layer["mixer"], layer["mlp"]
        H = m["heads"]
        if layer["type"] == "attention":
            kv += m["kv_heads"] * (m["dim"] + m["vdim"])
            params += W * (H * (m["dim"] + 2 * m["vdim"]) + m["kv_heads"] * (m["dim"] + m["vdim"]))
        elif layer["type"] == "gla":
            state += H * m["dim"] * m["vdim"]
            params += W * H * (2 * m["dim"] + 3 * m["vdim"])
        else:
            kv += m["kv_rank"] + m["rot_dim"]
            params += W * (H * (m["dim"] + m["rot_dim"] + 2 * m["vdim"]) + m["kv_rank"] + m["rot_dim"])
            params += m["kv_rank"] * H * (m["dim"] + m["vdim"])
        if f["kind"] == "dense":
            params += 2 * W * f["ff"]
        else:
            n = 3 if d["architecture"] == "Bovinex" else 2
            params += n * W * f["expert"]["ff"] * f["router"]["experts"]
            params += 2 * W * (f.get("shared") or {"ff": 0})["ff"]
    return params, kv, state


def work(case):
    kind = case["kind"]
    if kind in ("generate", "hybrid"):
        B, T, N = case["batch"], case["prompt"], case["new"]
        if kind == "hybrid":
            W, win = HYBRID[case["shape"]][0], HYBRID[case["shape"]][3]
            params, kv, state = _hybrid_counts(case)
            wb, V = 2.0 * params, HYBRID_VOCAB
            heads = 2 * HYBRID[case["shape"]][1] * 128 * sum(
                x["type"] != "gla" for x in _hybrid_description(case)["layers"])
        else:
            W, H, G, ff, V, _ = SHAPES[case["shape"]]
            D, L = W // H, case["layers"]
            params = L * (W * (H + 2 * G) * D + W * W + 3 * W * ff)
            wb = params * {"bf16": 2.0, "int8": 1.0, "int4": 0.53}[case["weights"]]
            kv, state, win, heads = L * 2 * G * D, 0, 1 << 30, L * 2 * W
        live = T * (0.75 if case.get("padded") else 1.0)        # mean tokens of a row
        seen = min(win, live + N / 2)
        reads = N * (wb + 2.0 * V * W)                          # the prompt pass and N - 1 steps
        cache = 2.0 * B * kv * (live + (N - 1) * seen) + (N - 1) * 8.0 * B * state
        flops = 2.0 * params * B * (live + N - 1) + 2.0 * V * W * B * N
        flops += 2.0 * heads * B * (live * min(win, live) / 2 + (N - 1) * seen)
        return {"bytes": reads + cache, "flops": flops}
    W, H, G, ff, V, _ = SHAPES[case["shape"]]
    L, n = case["layers"], case["batch"] * case["seq"]
    params = L * (2 * W * W + 2 * W * G * (W // H) + 3 * W * ff)
    attn = 2.0 * L * n * case["seq"] * W                        # causal: half of 4 n S W
    if kind == "score":
        return {"bytes": 2.0 * params + 4.0 * n, "flops": 2.0 * params * n + attn}
    head = 2.0 * V * W * n * 2 if case["loss"] == "sft" else 0.0   # the frozen head: no weight grad
    # Adam: master weights and two moments read and written, the gradient written once
    return {"bytes": params * (4 * 7 + 2.0), "flops": 6.0 * params * n + 3.5 * attn + head}


def tolerance(case):
    """bf16 activations and gradients through a few layers: logits, rewards and gradients are about
    0.01 off 64 bits (the hybrids 0.004), so that two correct roundings of the same sums differ by
    about as much; stated three to four times as wide. Tokens are whole numbers: a draw near a tie
    may fall the other way."""
    if case["kind"] == "train":
        return {"rel": 0.03, "max": 0.5}
    if case["kind"] == "score":
        return {"rel": 0.03, "max": 0.3}
    if case["kind"] == "hybrid":
        return {"rel": 0.015, "max": 0.15, "differ": 0.005}
    return {"rel": 0.03, "max": 0.3, "differ": 0.005}


# ------------------------------------------------------------------------------ 64 bits

def _rms(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w.double()


def _softmax_rows(q, k, v, scale, ok):
    """q [H, T, d], k [H, T, d], v [H, T, e], a few heads at a time; ok [T, T]."""
    out = []
    for a in range(0, q.shape[0], 8):
        s = torch.matmul(q[a:a + 8], k[a:a + 8].transpose(1, 2)) * scale
        s = s.masked_fill(~ok, float("-inf"))
        out.append(torch.matmul(torch.softmax(s, -1), v[a:a + 8]))
    return torch.cat(out)


def _dense64(w):
    return w.double() if isinstance(w, torch.Tensor) else w.dense()


def _rope_table(T, dims, base):
    """The bf16 table of the model (cos and sin are constants of the design, rounded once)."""
    f = 1.0 / base ** (torch.arange(0, dims, 2, device="cuda").float() / dims)
    ang = torch.outer(torch.arange(T, device="cuda"), f)
    return torch.cos(ang).bfloat16().double(), torch.sin(ang).bfloat16().double()


def _turn_pairs(x, c, s):
    """x [B, T, heads, dim]: neighbours (2i, 2i + 1) turn."""
    u, v = x[..., 0::2], x[..., 1::2]
    c, s = c[:, None], s[:, None]
    return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)


def _visible(T, pad, win=None, keep=0):
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None]
    ok = (j <= i) & ((j >= pad) | (i == j))
    return ok if not win else ok & ((i - j < win) | (j - pad < keep))


def _llama64(case, w, ids, pads, get=None):
    """Final-norm hidden states [B, T, W] of token ids [B, T]."""
    W, H, G, ff, V, base = SHAPES[case["shape"]]
    get = get or (lambda name: _dense64(w[name]))
    D, (B, T) = W // H, ids.shape
    c, s = _rope_table(T, D, base)
    x = w["embed"].double()[ids.long()]
    causal = _visible(T, 0)
    for i in range(case["layers"]):
        qkv = (_rms(x, w[f"{i}.n1"]) @ get(f"{i}.wqkv").t()).view(B, T, H + 2 * G, D)
        q = _turn_pairs(qkv[:, :, :H], c, s)
        k = _turn_pairs(qkv[:, :, H:H + G], c, s).repeat_interleave(H // G, 2)
        v = qkv[:, :, H + G:].repeat_interleave(H // G, 2)
        rows = []
        for b in range(B):
            ok = causal if pads is None else _visible(T, pads[b])
            o = _softmax_rows(*(t[b].transpose(0, 1) for t in (q, k, v)), D ** -0.5, ok)
            rows.append(o.transpose(0, 1).reshape(T, W))
        x = x + torch.stack(rows) @ get(f"{i}.wo").t()
        del qkv, q, k, v, rows
        h = _rms(x, w[f"{i}.n2"])
        a = torch.nn.functional.silu(h @ get(f"{i}.w1").t()) * (h @ get(f"{i}.w3").t())
        x = x + a @ get(f"{i}.w2").t()
    return _rms(x, w["norm"])


def _chain(ids, new, vocab):
    """The prompt followed by the successors of its last token."""
    nxt, out = _successor(vocab), [ids.long()]
    for _ in range(new):
        out.append(nxt[out[-1][:, -1:]])
    return torch.cat(out, 1)


def _generated(case, hidden, head, ids, vocab, last):
    """Tokens (the greedy choice at every position of the answer) and the last step's logits."""
    T, N = case["prompt"], case["new"]
    logits = hidden[:, T - 1:T - 1 + N] @ head.double().t()
    choice = logits.argmax(-1)
    return {"tokens": torch.cat([ids, choice.to(ids.dtype)], 1), "logits": last(logits[:, -1])}


@torch.no_grad()
def _exact_generate(case, seed):
    V = SHAPES[case["shape"]][4]
    w = _llama_weights(case, seed)
    ids, pads = _tokens(case, seed, case["batch"], case["prompt"], V)
    hidden = _llama64(case, w, _chain(ids, case["new"], V)[:, :-1], pads)
    return _generated(case, hidden, w["head"], ids, V, lambda z: z)


@torch.no_grad()
def _exact_score(case, seed):
    s = _score_tokens(case, seed)
    w, out = _llama_weights(case, seed), []
    for a in range(0, case["batch"], 16):
        h = _llama64(case, w, s[a:a + 16], None)
        out.append((h @ _reward_head(case, seed).double().t()).mean(-1))
    return {"rewards": torch.cat(out)}


PARTS = ("wqkv", "wo", "w1", "w3", "w2")


def _exact_train(case, seed):
    w = _llama_weights(case, seed)
    leaf = {f"{i}.{n}": w[f"{i}.{n}"].double().requires_grad_(True)
            for i in range(case["layers"]) for n in PARTS}
    batch, B = _train_batch(case, seed), case["batch"]
    head = (w["head"] if case["loss"] == "sft" else _reward_head(case, seed)).double()
    if case["loss"] == "prm":
        head.requires_grad_(True)
    if case["loss"] == "sft":
        total = (batch[1][:, 1:] != -100).sum().clamp_min(1)
    else:
        total = batch[2].sum() + 1e-6
    loss = 0.0
    step = max(1, 4096 // case["seq"])
    for a in range(0, B, step):                     # a few sequences at a time
        rows = [t[a:a + step] for t in batch]
        h = _llama64(case, w, rows[0], None, get=leaf.__getitem__)
        z = h @ head.t()
        if case["loss"] == "sft":
            part = torch.nn.functional.cross_entropy(z[:, :-1].flatten(0, 1), rows[1][:, 1:].flatten(),
                                                     ignore_index=-100, reduction="sum")
        else:
            bce = torch.nn.functional.binary_cross_entropy_with_logits(
                z.mean(-1), rows[1].double(), reduction="none")
            part = (bce * rows[2]).sum()
        part = part / total
        part.backward()
        loss += float(part.detach())
        del h, z, part
    params = [[leaf[f"{i}.{n}"] for n in PARTS] for i in range(case["layers"])]
    if case["loss"] == "prm":
        params.append([head])
    with torch.no_grad():
        grads = [torch.cat([p.grad.flatten() for p in ps]) for ps in params]
        flat = [torch.cat([p.flatten() for p in ps]) for ps in params]
        norm = torch.sqrt(sum(x.pow(2).sum() for x in grads))
        clip = float((1.0 / (norm + 1e-6)).clamp(max=1.0))
        # the first Adam step: both bias corrections cancel the decay rates
        new = [p - TRAIN_LR * (x * clip) / ((x * clip).abs() + 1e-8) for p, x in zip(flat, grads)]
    return {"loss": torch.tensor(loss, dtype=torch.float64), "grad_norm": norm.reshape(1),
            "grads": grads, "weights": new}


def _hybrid_angles(T, rot):
    n = rot["dims"]
    i = torch.arange(n // 2, dtype=torch.float64, device="cuda")
    freq, amp, sc = float(rot["base"]) ** (-2.0 * i / n), 1.0, rot.get("scaling")
    if sc:
        def at(turns):
            return n * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), n - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        freq, amp = freq / sc["factor"] * ramp + freq * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1
    ang = torch.arange(T, dtype=torch.float64, device="cuda")[:, None] * freq
    return amp * torch.cos(ang), amp * torch.sin(ang)


def _bovinex_mixer(layer, w, p, h):
    """One sequence h [T, W] -> gated heads [T, H * vdim]."""
    m, T = layer["mixer"], h.shape[0]
    H, d, e = m["heads"], m["dim"], m["vdim"]
    z = h @ w[p + "g"].t()
    if layer["type"] == "attention":
        G, half = m["kv_heads"], m["rot"]["dims"] // 2
        q, k, v = (h @ w[p + n].t() + w[p + n + ".b"] for n in "qkv")
        q, k = (_rms(t, w[p + n]) for t, n in ((q, "q.norm"), (k, "k.norm")))
        c, s = (t[:, None] for t in _hybrid_angles(T, m["rot"]))

        def turn(x):
            u, y = x[..., :half], x[..., half:]
            return torch.cat([u * c - y * s, y * c + u * s], -1)
        q, k = turn(q.view(T, H, d)), turn(k.view(T, G, d)).repeat_interleave(H // G, 1)
        v = v.view(T, G, e).repeat_interleave(H // G, 1)
        ok = _visible(T, 0, m["mask"]["size"], m["mask"]["keep_first"])
        o = _softmax_rows(*(t.transpose(0, 1) for t in (q, k, v)), m["scale"], ok)
        return o.transpose(0, 1).reshape(T, H * e) * torch.sigmoid(z)
    raise ValueError(layer["type"])


def _gla_rows(m, w, p, h):
    """Gated linear attention of rows h [B, T, W] (step by step, all rows at once)."""
    B, T, _ = h.shape
    H, d, e = m["heads"], m["dim"], m["vdim"]
    q = (h @ w[p + "q"].t()).view(B, T, H, d) * d ** -0.5
    k, v = (h @ w[p + "k"].t()).view(B, T, H, d), (h @ w[p + "v"].t()).view(B, T, H, e)
    a = torch.sigmoid((h @ w[p + "a1"].t()) @ w[p + "a2"].t() + w[p + "a2.b"])
    a = a.pow(1.0 / m["tau"]).view(B, T, H, d)
    S = torch.zeros(B, H, d, e, dtype=torch.float64, device="cuda")
    o = torch.empty(B, T, H, e, dtype=torch.float64, device="cuda")
    for t in range(T):
        S.mul_(a[:, t, :, :, None]).addcmul_(k[:, t, :, :, None], v[:, t, :, None, :])
        o[:, t] = torch.matmul(q[:, t, :, None], S)[:, :, 0]
    z = h @ w[p + "g"].t()
    return (_rms(o, w[p + "norm"]).flatten(2)) * (z * torch.sigmoid(z))


def _latent_mixer(m, w, p, h):
    T, H, d, r = h.shape[0], m["heads"], m["dim"], m["kv_rank"]
    c, s = (t[:, None] for t in _hybrid_angles(T, m["rot"]))

    def turn(x):
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    y = h @ w[p + "dkv"].t()
    lat, kr = _rms(y[:, :r], w[p + "dkv.norm"]), turn(y[:, None, r:])
    k = torch.cat([(lat @ w[p + "uk"].t()).view(T, H, d), kr.expand(T, H, -1)], -1)
    v = (lat @ w[p + "uv"].t()).view(T, H, m["vdim"])
    q = (h @ w[p + "q"].t()).view(T, H, d + m["rot_dim"])
    q = torch.cat([q[..., :d], turn(q[..., d:])], -1)
    o = _softmax_rows(*(t.transpose(0, 1) for t in (q, k, v)), m["scale"],
                      _visible(T, 0, m["mask"]["size"]))
    return o.transpose(0, 1).reshape(T, -1) * torch.sigmoid(h @ w[p + "g"].t())


def _feed_forward64(f, w, p, h, bov):
    def gelu(x):
        return 0.5 * x * (1 + torch.erf(x / math.sqrt(2)))
    if f["kind"] == "dense":
        return torch.relu(h @ w[p + "up"].t()).square() @ w[p + "down"].t()
    z = h @ w[p + "router"].t()
    score = torch.softmax(z + w[p + "router.b"], -1) if bov else torch.sigmoid(z)
    out = 0.0 if bov else gelu(h @ w[p + "shared.up"].t()) @ w[p + "shared.down"].t()
    for e in range(f["router"]["experts"]):
        a, down = score[..., e:e + 1], w[p + f"e{e}.down"].t()
        if bov:
            gate = h @ w[p + f"e{e}.gate"].t()
            out = out + a * ((gate * torch.sigmoid(gate) * (h @ w[p + f"e{e}.up"].t())) @ down)
        else:
            out = out + gelu((a * h) @ w[p + f"e{e}.up"].t()) @ down
    return out


@torch.no_grad()
def _exact_hybrid(case, seed):
    d, (B, T, N) = _hybrid_description(case), (case["batch"], case["prompt"], case["new"])
    bov = d["architecture"] == "Bovinex"
    w = {k: v.double() for k, v in _hybrid_weights(case, seed).items()}
    one = 1.0 if bov else 0.0                           # Bovinex norms multiply by 1 + weight
    ids, pads = _tokens(case, seed, B, T, HYBRID_VOCAB)
    pads = [0] * B if pads is None else pads.tolist()
    full = _chain(ids, N, HYBRID_VOCAB)[:, :-1]
    # a row's tokens start at position 0: pads go behind (causal: they change nothing before them)
    full = torch.stack([torch.roll(full[b], -pads[b]) for b in range(B)])
    x = w["embed"][full] * d["embedding"]["scale"]
    for i, layer in enumerate(d["layers"]):
        p, m, f = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        h = _rms(x, one + w[f"l{i}.norm1"])
        if layer["type"] == "gla":
            o = _gla_rows(m, w, p, h)
        elif bov:
            o = torch.stack([_bovinex_mixer(layer, w, p, h[b]) for b in range(B)])
        else:
            o = torch.stack([_latent_mixer(m, w, p, h[b]) for b in range(B)])
        mix = o @ w[p + "o"].t()
        if bov:
            x = x + mix + _feed_forward64(f, w, f"l{i}.mlp.", h, True)
        else:
            x = x + mix
            x = x + _feed_forward64(f, w, f"l{i}.mlp.", _rms(x, w[f"l{i}.norm2"]), False)
    hidden = _rms(x, one + w["final.norm"])
    hidden = torch.stack([torch.roll(hidden[b], pads[b], 0) for b in range(B)])

    def last(z):
        return z if bov else 30.0 * torch.tanh(z * 0.5 / 30.0)
    return _generated(case, hidden, w["head"], ids, HYBRID_VOCAB, last)


def exact(case, seed):
    return {"generate": _exact_generate, "score": _exact_score, "train": _exact_train,
            "hybrid": _exact_hybrid}[case["kind"]](case, seed)
