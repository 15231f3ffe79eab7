"""The work whose speed this repository watches: what users of the framework have it do on one GPU.

Four kinds of pass, through the objects that the trainer and the training service drive (``Zero3Engine``,
``build_optimizer``, the fused lm-head losses) and the model's own modules:

* ``train``  one optimizer step: zero_grad, forward and backward of every micro-batch, gradient norm and
  clipping, AdamW with fp32 master weights and moments;
* ``lora``   the same step with frozen base weights and rank-r adapters on all projections;
* ``score``  log-probabilities of the label tokens without gradients (what the service's ``forward`` runs
  for a rollout), final hidden states included;
* ``moe_block``  one mixture-of-experts block with block-scaled fp8 experts, forward and backward, on given
  hidden states.

Models are slices of the architectures that the presets, examples, benchmark and tests name: their layers
at full width, a few of them, with a 32,000-token vocabulary so that the layers keep about the share of a
step that they have in the full depth.  Rows are packed documents, as every example configures them.  MoE
steps replay given expert choices (rollout routing replay): with free top-k choices a rounding difference
in a near tie moves whole tokens between experts and no two correct runs could be compared.  For the same
reason fp8 experts are measured on given hidden states: e4m3 codes turn a bf16 rounding difference before
them into several percent of every gradient behind them.
"""
import torch

from xorl_b200.adapters.fp8 import inject_fp8_training
from xorl_b200.adapters.lora import inject_lora
from xorl_b200.arguments import LoRAArguments, TrainingArguments
from xorl_b200.models import ModelConfig
from xorl_b200.models.context import StepContext
from xorl_b200.models.decoder import DecoderLM
from xorl_b200.ops.fp8_grouped import invalidate_weight_cache
from xorl_b200.ops.loss import fused_linear_token_loss
from xorl_b200.optim import build_optimizer
from xorl_b200.parallel.state import init_parallel_state, reset_parallel_state
from xorl_b200.parallel.zero import Zero3Engine

# layer shapes by what names them in this repository
SHAPES = {
    # tests and smoke runs: the small presets
    "small": dict(hidden=512, inter=1024, heads=4, kv_heads=2, head_dim=128),
    # the family of small models with 64-wide heads
    "hd64": dict(hidden=1024, inter=3072, heads=16, kv_heads=4, head_dim=64),
    # the smoke model
    "1k": dict(hidden=1024, inter=3072, heads=8, kv_heads=2, head_dim=128),
    # qwen3-8b and llama3-8b (the latter without qk-norm)
    "8b": dict(hidden=4096, inter=12288, heads=32, kv_heads=8, head_dim=128),
    "8b-llama": dict(hidden=4096, inter=14336, heads=32, kv_heads=8, head_dim=128),
    # qwen3-30b-a3b
    "30b-a3b": dict(hidden=2048, inter=768, heads=32, kv_heads=4, head_dim=128),
}


def _case(name, kind, shape, layers, tokens, doc_min, doc_max, vocab=32000, micro=1, recompute=False, qk_norm=True,
          experts=0, top_k=0, fp8=False, rank=0):
    return dict(name=name, kind=kind, **SHAPES[shape], layers=layers, vocab=vocab, tokens=tokens, doc_min=doc_min,
                doc_max=doc_max, micro=micro, recompute=recompute, qk_norm=qk_norm, experts=experts, top_k=top_k,
                fp8=fp8, rank=rank)


def listed():
    return [
        # a step of a toy model on a toy batch: the first thing every user runs, and what tests run all day
        _case("train_small", "train", "small", 2, 256, 40, 200, vocab=4096),
        # its mixture-of-experts sibling
        _case("train_small_moe", "train", "small", 2, 512, 64, 300, vocab=4096, experts=8, top_k=2),
        # a small model with 64-wide heads on a row whose length is no multiple of anything
        _case("train_hd64_2045", "train", "hd64", 2, 2045, 128, 1024),
        # the headline: qwen3-8b layers, 4096 packed tokens, documents U[256, 4096], activations kept
        _case("train_8b_4096", "train", "8b", 2, 4096, 256, 4096),
        # llama3-8b layers, four micro-batches per step with recomputation, ragged rows
        _case("train_llama_accum", "train", "8b-llama", 1, 1999, 64, 1999, micro=4, recompute=True, qk_norm=False),
        # long context: one document of 16,384 tokens, recomputation on
        _case("train_8b_16384", "train", "8b", 1, 16384, 16384, 16384, recompute=True),
        # qwen3-30b-a3b: all 128 experts on one GPU, 256 rows per expert on average
        _case("train_moe_128e", "train", "30b-a3b", 1, 4096, 256, 4096, recompute=True, experts=128, top_k=8),
        # the share of one rank under expert parallelism 8: 16 experts of the same layers
        _case("train_moe_16e", "train", "30b-a3b", 2, 4096, 256, 4096, recompute=True, experts=16, top_k=8),
        # the mixture-of-experts block alone with fp8 experts, routing included
        _case("moe_block_fp8_8192", "moe_block", "30b-a3b", 1, 8192, 8192, 8192, experts=16, top_k=8, fp8=True),
        # adapters of rank 16 on every projection, as the service trains them
        _case("lora_8b_4096", "lora", "8b", 1, 4096, 256, 4096, rank=16),
        # scoring a batch of short rollouts
        _case("score_8b_8192", "score", "8b", 2, 8192, 100, 1200),
        # scoring one short answer: the smallest call at full width
        _case("score_8b_61", "score", "8b", 2, 61, 61, 61),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "moe", "moe", "moe_block", "lora", "score", "score"])
    micro, recompute, qk_norm, rank, experts, top_k = 1, rng.random() < 0.5, True, 0, 0, 0
    if kind in ("moe", "moe_block"):
        shape = rng.choice(["small", "30b-a3b", "30b-a3b"])
        layers = 1 if kind == "moe_block" else rng.choice([1, 2])
        tokens = _log_uniform(rng, 256, 8192 if kind == "moe_block" else 6000)
        experts, top_k = (8, 2) if shape == "small" else rng.choice([(16, 8), (32, 8), (64, 8)])
        kind = "train" if kind == "moe" else kind
    else:
        shape = rng.choice(["small", "hd64", "1k", "8b", "8b", "8b-llama"])
        big = shape.startswith("8b")
        layers = 1 if big and kind != "score" else rng.choice([1, 2])
        qk_norm = shape != "8b-llama"
        tokens = _log_uniform(rng, 48 if kind == "score" else 192, 8192 if kind == "score" else 6000)
        if kind == "train" and tokens < 2048:
            micro = rng.choice([1, 1, 2, 3])
        if kind == "lora":
            rank = rng.choice([8, 16, 32, 64])
    doc_max = min(tokens, _log_uniform(rng, 128, 6000))
    doc_min = max(1, min(doc_max, _log_uniform(rng, 32, 256)))
    c = _case("", kind, shape, layers, tokens, doc_min, doc_max, vocab=rng.choice([4096, 32000]), micro=micro,
              recompute=recompute and kind in ("train", "lora"), qk_norm=qk_norm, experts=experts, top_k=top_k,
              fp8=kind == "moe_block", rank=rank)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------
def _config(c):
    d = dict(model_type="qwen3_moe" if c["experts"] else "qwen3" if c["qk_norm"] else "llama",
             vocab_size=c["vocab"], hidden_size=c["hidden"], num_hidden_layers=c["layers"],
             num_attention_heads=c["heads"], num_key_value_heads=c["kv_heads"], head_dim=c["head_dim"],
             intermediate_size=c["inter"], rope_theta=1e6, tie_word_embeddings=False)
    if c["experts"]:
        d.update(num_experts=c["experts"], num_experts_per_tok=c["top_k"], moe_intermediate_size=c["inter"],
                 norm_topk_prob=True, router_aux_loss_coef=1e-3)
    return ModelConfig.from_dict(d)


def _row(c, seed):
    """One packed row on the GPU: tokens uniform over the vocabulary, document lengths uniform in
    [doc_min, doc_max] (the last one cut), next-token labels with the last target of a document ignored."""
    cpu = torch.Generator().manual_seed(seed)
    T = c["tokens"]
    cu = [0]
    while cu[-1] < T:
        cu.append(min(T, cu[-1] + int(torch.randint(c["doc_min"], c["doc_max"] + 1, (1,), generator=cpu))))
    gpu = torch.Generator(device="cuda").manual_seed(seed)
    ids = torch.randint(0, c["vocab"], (T + 1,), generator=gpu, device="cuda")
    labels = ids[1:].clone()
    starts = torch.tensor(cu, device="cuda")
    labels[starts[1:] - 1] = -100
    lengths = starts[1:] - starts[:-1]
    pos = torch.arange(T, device="cuda") - torch.repeat_interleave(starts[:-1], lengths)
    row = dict(input_ids=ids[:-1].clone(), labels=labels, position_ids=pos, cu_seqlens=starts.to(torch.int32))
    if c["experts"]:
        # recorded expert choices, some experts more popular than others
        E = c["experts"]
        popular = 0.5 * torch.randn(c["layers"], E, generator=gpu, device="cuda")
        noise = torch.rand(T, c["layers"], E, generator=gpu, device="cuda").clamp_min_(1e-9)
        row["routed"] = (popular - torch.log(-torch.log(noise))).topk(c["top_k"], dim=-1)[1]
    return row


def _prepare_block(c, seed):
    model = DecoderLM(_config(c), device="meta")
    inject_fp8_training(model, TrainingArguments(enable_fp8_training=True, fp8_training_allow_blackwell=True,
                                                 fp8_training_target_modules=["experts"]))
    block = model.layers["0"].mlp.to(torch.bfloat16).to_empty(device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(seed)
    for p in block.parameters():
        torch.nn.init.normal_(p, 0.0, 0.02, generator=gen)
    # hidden states as a norm leaves them; output gradients of a mean loss
    x = torch.randn(c["tokens"], c["hidden"], generator=gen, device="cuda").bfloat16().requires_grad_()
    dy = (torch.randn(c["tokens"], c["hidden"], generator=gen, device="cuda") * 1e-4).bfloat16()
    pos = torch.arange(c["tokens"], device="cuda")
    cu = torch.tensor([0, c["tokens"]], device="cuda", dtype=torch.int32)
    return dict(kind="moe_block", block=block, x=x, dy=dy, pos=pos, cu=cu)


def prepare(case, seed):
    """Model, engine, optimizer and the step's packed rows on the GPU."""
    c = case
    reset_parallel_state()
    ps = init_parallel_state(device_type="cuda")
    if c["kind"] == "moe_block":
        return _prepare_block(c, seed)
    model = DecoderLM(_config(c), device="meta")
    if c["kind"] == "lora":
        # B away from zero, as after the first steps: every factor has a gradient
        inject_lora(model, LoRAArguments(enable_lora=True, lora_rank=c["rank"], lora_alpha=2 * c["rank"],
                                         lora_b_init_std=0.02, lora_b_init_seed=seed))
    model.aux_loss_enabled = bool(c["experts"])
    engine = Zero3Engine(model, ps, compute_dtype=torch.bfloat16, device=torch.device("cuda", torch.cuda.current_device()),
                         recompute=c["recompute"], seed=seed)
    rows = [_row(c, seed * 16 + i) for i in range(c["micro"])]
    if c["kind"] == "score":
        return dict(kind="score", engine=engine, row=rows[0])
    optimizer = build_optimizer(engine, lr=1e-5, weight_decay=0.01)
    groups = [g for g in engine.all_groups() if g.grad_shard is not None]
    return dict(kind=c["kind"], engine=engine, optimizer=optimizer, rows=rows,
                scale=1.0 / (c["micro"] * c["tokens"]),
                # the state's own buffers, returned by every step
                grads=[v for g in groups for v in g.param_views(g.grad_shard)],
                weights=[g.master for g in groups],
                moments=[s[id(g)] for s in optimizer.state.values() for g in groups])


def _train_step(s):
    engine, optimizer, rows = s["engine"], s["optimizer"], s["rows"]
    optimizer.zero_grad()
    total = None
    for i, r in enumerate(rows):
        engine.final_micro_batch = i == len(rows) - 1
        extra = {"routing_replay_all": r["routed"]} if "routed" in r else None
        loss = engine.forward_backward(r["input_ids"], r["labels"], position_ids=r["position_ids"],
                                       cu_seqlens=r["cu_seqlens"], grad_scale=s["scale"], extra=extra)
        total = loss if total is None else total + loss
    engine.finish_grad_sync()
    norm, coef = engine.grad_norm_and_clip_coef(1.0)
    optimizer.step(clip_coef=coef)
    return dict(loss=total, norm=norm, grads=s["grads"], weights=s["weights"], moments=s["moments"])


@torch.no_grad()
def _score(s):
    engine, r = s["engine"], s["row"]
    hidden = engine.forward_only(r["input_ids"], position_ids=r["position_ids"], cu_seqlens=r["cu_seqlens"])
    _, logprobs, _ = fused_linear_token_loss(hidden, engine.model.lm_head.weight, r["labels"],
                                             lambda lp, mask: (lp.sum() * 0, {}), 1.0)
    return dict(hidden=hidden, logprobs=logprobs)


def _moe_block(s):
    block, x = s["block"], s["x"]
    # a training step sees new weights: the quantised copies of the last step's are not used
    invalidate_weight_cache()
    x.grad = None
    for p in block.parameters():
        p.grad = None
    ctx = StepContext(cu_seqlens=s["cu"], position_ids=s["pos"], causal=True, training=True)
    y = block(x, ctx)
    y.backward(s["dy"])
    return dict(y=y.detach(), dx=x.grad, grads=[p.grad for p in block.parameters()])


def run(state):
    if state["kind"] == "score":
        return _score(state)
    return _moe_block(state) if state["kind"] == "moe_block" else _train_step(state)


# ------------------------------------------------------------------------------------------------
def work(case):
    c = case
    H, T, V, L = c["hidden"], c["tokens"], c["vocab"], c["layers"]
    q, kv = c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"]
    if c["kind"] == "moe_block":
        weights = c["experts"] * (3 * H * c["inter"] + H)
        used = c["top_k"] * 3 * H * c["inter"] + c["experts"] * H
        # bf16 weights in, bf16 gradients out; hidden states, output and their two gradients
        return {"bytes": 4.0 * weights + 8.0 * T * H, "flops": 6.0 * T * used}
    attn = H * (q + 2 * kv) + q * H
    norms = 2 * H + (2 * c["head_dim"] if c["qk_norm"] else 0)
    mlp = 3 * H * c["inter"]
    if c["experts"]:
        held, used = attn + c["experts"] * (mlp + H), attn + c["top_k"] * mlp + c["experts"] * H
    else:
        held = used = attn + mlp
    matmul = L * used + V * H                       # weights that a token meets
    params = L * (held + norms) + 2 * V * H + H
    mean_doc = (c["doc_min"] + min(c["doc_max"], T)) / 2
    pairs = T * min(mean_doc, T) / 2                # (query, key) pairs under the causal mask, about
    attn_fwd = 4.0 * pairs * q * L
    if c["kind"] == "score":
        return {"bytes": 2.0 * (params - V * H) + 2.0 * T * H * 2 + 20.0 * T, "flops": 2.0 * T * matmul + attn_fwd}
    n = c["micro"]
    if c["kind"] == "lora":
        r = c["rank"]
        adapters = L * r * (3 * H + q + 2 * kv + (q + H) + 2 * H + 2 * c["inter"] + (c["inter"] + H))
        # frozen weights: forward and input gradient only
        return {"bytes": 2.0 * params + 32.0 * adapters + 28.0 * T * n,
                "flops": n * (4.0 * T * matmul + 6.0 * T * adapters + 3.5 * attn_fwd)}
    # fp32 master and two moments in and out, bf16 weights in and out, fp32 gradient out
    return {"bytes": 32.0 * params + 28.0 * T * n, "flops": n * (6.0 * T * matmul + 3.5 * attn_fwd)}


def tolerance(case):
    """bf16 activations rounded at the same places.  Runs whose attention outputs and gradients were jittered
    by half a unit in the last place differed by 0.7 % to 2.3 % in the worst tensor (the qk-norm gradients, the
    second moments) and by up to 0.58 of a tensor's root mean square in single values (second moments of
    embedding rows, which most rows of the table do not have); final hidden states by 0.8 %, the gradients of a
    mixture-of-experts block with a jittered activation by 0.34 %."""
    if case["kind"] == "score":
        return {"rel": 0.03, "max": 0.2}
    if case["kind"] == "moe_block":
        return {"rel": 0.013, "max": 0.35}
    return {"rel": 0.03, "max": 0.95}
