"""The work a user has this package do, as measurable cases.

Six kinds, each through the entry points a training program calls:

  head    fused_head_loss forward and backward (or forward alone, an evaluation pass) on packed
          hidden states against a tied fp16 head weight
  step    one captured QLoRA training step (CapturedStep.load + run) of the Qwen2.5-1.5B
          architecture on a new host batch
  eager   the same training step through the patched model without a graph (qlora_step), what a
          trainer that calls `apply()` runs
  attn    causal attention inside the segments of a packed row, forward and backward
  nf4     dequantisation of the projection weights of decoder blocks
  ops     the per-op functions of a decoder block at one token count: RMSNorm, RoPE, SwiGLU and the
          LoRA branch, forward and backward

Sizes are the benchmark's (hidden 1536, 12 / 2 heads of 128, intermediate 8960, vocabulary 151936,
batches of right-padded rows of 64 to 512 tokens packed to one row) and ranges around them.
"""

import math

import torch

import claudemaxing_b200 as solution
from claudemaxing_b200 import qlora
from claudemaxing_b200.attention import segment_attention
from claudemaxing_b200.lora import LoRABranch
from claudemaxing_b200.nf4 import dequantize_nf4_batch

DEV = "cuda"
LOSS_SCALE = 4096.0     # what a trainer's GradScaler multiplies the loss with: fp16 gradients stay normal
HIDDEN, INTER, VOCAB, LAYERS = 1536, 8960, 151936, 28
HEADS, KV_HEADS, HEAD_DIM = 12, 2, 128
# out x in of q, k, v, o, gate, up, down of one decoder block
PROJECTIONS = ((HIDDEN, HIDDEN), (256, HIDDEN), (256, HIDDEN), (HIDDEN, HIDDEN),
               (INTER, HIDDEN), (INTER, HIDDEN), (HIDDEN, INTER))
BLOCK_WEIGHTS = sum(o * i for o, i in PROJECTIONS)
RANK = 16


def listed():
    return [
        # one short conversation (a batch of one row), where launches and latency count
        dict(name="head_128", kind="head", tokens=128, hidden=HIDDEN, vocab=VOCAB, grad=True),
        # the packed row of an ordinary batch: 4 rows of 64 to 512 tokens, 1168 real ones
        dict(name="head_1168", kind="head", tokens=1168, hidden=HIDDEN, vocab=VOCAB, grad=True),
        # the benchmark's 4 full rows of 512
        dict(name="head_2048", kind="head", tokens=2048, hidden=HIDDEN, vocab=VOCAB, grad=True),
        # a large batch (gradient accumulation folded into one pass)
        dict(name="head_8192", kind="head", tokens=8192, hidden=HIDDEN, vocab=VOCAB, grad=True),
        # the benchmark's training step
        dict(name="step_4_rows", kind="step", rows=4, layers=LAYERS),
        # the same model with a batch that uses the card's memory
        dict(name="step_16_rows", kind="step", rows=16, layers=LAYERS),
        # the step as the trainer launches it, operation by operation
        dict(name="eager_4_rows", kind="eager", rows=4, layers=LAYERS),
        # one layer's attention in the benchmark's packed row (row lengths uniform in 64..512)
        dict(name="attn_short", kind="attn", rows=4, longest=512),
        # long documents in one packed row
        dict(name="attn_long", kind="attn", rows=4, longest=4096),
        # eight decoder blocks' weights, one call per block
        dict(name="nf4_blocks", kind="nf4", blocks=8, dtype="float16", nested=True),
        # the 4-bit model's per-op functions (fp32 hidden states, frozen norms) at a short batch
        dict(name="ops_512", kind="ops", tokens=512, model="4bit"),
        # an fp16 model with trainable norms at a long batch
        dict(name="ops_16384", kind="ops", tokens=16384, model="float16"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["head", "head", "head", "step", "eager", "attn", "attn", "nf4", "ops", "ops"])
    if kind == "head":
        # other widths and vocabularies of the same model families' sizes; every third an evaluation
        return dict(kind=kind, tokens=_log_uniform(rng, 24, 8192), hidden=rng.choice([896, HIDDEN, HIDDEN, 2048]),
                    vocab=rng.choice([VOCAB, VOCAB, 32000, 50257]), grad=rng.random() < 0.7)
    if kind == "step":
        return dict(kind=kind, rows=rng.randint(1, 16), layers=LAYERS)
    if kind == "eager":
        return dict(kind=kind, rows=rng.randint(1, 12), layers=LAYERS)
    if kind == "attn":
        return dict(kind=kind, rows=rng.randint(1, 8), longest=_log_uniform(rng, 64, 3000))
    if kind == "nf4":
        return dict(kind=kind, blocks=rng.randint(1, 8), dtype=rng.choice(["float16", "float16", "float32"]),
                    nested=rng.random() < 0.75)
    return dict(kind=kind, tokens=_log_uniform(rng, 64, 16384), model=rng.choice(["4bit", "4bit", "float16", "bfloat16"]))


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(gen, *shape, dtype=torch.float16, std=1.0):
    return torch.randn(*shape, generator=gen, device=DEV, dtype=torch.float32).mul_(std).to(dtype)


# ------------------------------------------------------------------------------------------ head
def _prepare_head(case, seed):
    gen, n = _gen(seed), case["tokens"]
    weight = torch.empty(case["vocab"], case["hidden"], dtype=torch.float16, device=DEV)
    for r0 in range(0, case["vocab"], 16384):
        rows = weight[r0:r0 + 16384]
        rows.copy_(torch.randn(rows.shape, generator=gen, device=DEV).mul_(0.02))
    target = torch.randint(0, case["vocab"], (1, n), generator=gen, device=DEV)
    target.masked_fill_(torch.rand(1, n, generator=gen, device=DEV) < 0.1, -100)
    target[0, 0] = 5                                   # at least one labelled position
    hidden = _randn(gen, 1, n, case["hidden"]).requires_grad_(case["grad"])
    return dict(case=case, hidden=hidden, weight=weight, target=target)


def _run_head(s):
    h = s["hidden"]
    if not s["case"]["grad"]:
        with torch.no_grad():
            loss, terms = solution.fused_head_loss(h, s["weight"], None, target=s["target"])
        return [loss, terms.token_loss, terms.token_entropy, terms.correct, terms.labelled]
    h.grad = None
    loss, terms = solution.fused_head_loss(h, s["weight"], None, target=s["target"])
    (loss * LOSS_SCALE).backward()
    return [loss.detach(), terms.token_loss, terms.token_entropy, terms.correct, terms.labelled, h.grad]


def _work_head(case):
    n, h, v = case["tokens"], case["hidden"], case["vocab"]
    products = 2 if case["grad"] else 1
    return dict(flops=2.0 * products * n * h * v,
                bytes=2.0 * v * h + 2.0 * n * h * products + 8.0 * n + 8.0 * n)


# --------------------------------------------------------------------------- step and eager step
def _model(case, seed):
    solution.apply()
    model, lora = qlora.build_qlora_model(DEV, config={"num_hidden_layers": case["layers"]}, seed=seed)
    gen = _gen(seed + 1)
    with torch.no_grad():                              # adapters in the middle of a run: B is not zero any more
        for name, p in model.named_parameters():
            if "lora_B" in name:
                p.copy_(_randn(gen, *p.shape, dtype=torch.float32, std=0.01))
    return model, lora


def _prepare_step(case, seed):
    model, lora = _model(case, seed)
    batch = qlora.synthetic_batch(batch=case["rows"], seed=seed)     # as a data loader hands it over
    for key in ("input_ids", "attention_mask", "labels"):
        batch[key] = batch[key].pin_memory()
    optimizer = torch.optim.AdamW(lora, lr=1e-4, fused=True, capturable=True)
    scaler = torch.amp.GradScaler("cuda", init_scale=LOSS_SCALE)
    step = qlora.CapturedStep(model, lora, optimizer, batch, scaler=scaler)
    torch.cuda.manual_seed(seed)                       # the dropout masks of the steps that follow
    return dict(case=case, step=step, batch=batch)


def _run_step(s):
    s["step"].load(s["batch"])
    loss = s["step"].run()
    return [loss, s["step"].flat_grad]                 # the gradient of every adapter weight


def _prepare_eager(case, seed):
    model, lora = _model(case, seed)
    batch = qlora.synthetic_batch(batch=case["rows"], seed=seed, device=DEV)
    # the patched forward settles the tied embedding's storage on its first training call
    qlora.qlora_step(model, batch)
    torch.cuda.manual_seed(seed)
    return dict(case=case, model=model, lora=lora, batch=batch)


class _Scaled:
    """The part of a GradScaler that takes part in backward."""

    @staticmethod
    def scale(loss):
        return loss * LOSS_SCALE


def _run_eager(s):
    for p in s["lora"]:
        p.grad = None
    loss = qlora.qlora_step(s["model"], s["batch"], None, _Scaled)
    return [loss, torch.cat([p.grad.reshape(-1) for p in s["lora"]])]


def _work_step(case):
    rows = case["rows"]
    tokens, pairs = 288.0 * rows, rows * 50000.0       # means over lengths uniform in 64..512
    layers = case["layers"]
    gemm = 4.0 * tokens * (layers * BLOCK_WEIGHTS + HIDDEN * VOCAB)       # forward and input gradient
    adapters = 6.0 * tokens * layers * RANK * (HIDDEN + HIDDEN + HIDDEN + 256)
    attention = 14.0 * layers * pairs * HEADS * HEAD_DIM
    return dict(flops=gemm + adapters + attention,
                bytes=0.52 * layers * BLOCK_WEIGHTS + 2.0 * HIDDEN * VOCAB
                + 4.0 * 3 * layers * RANK * (HIDDEN + HIDDEN + HIDDEN + 256))


# ------------------------------------------------------------------------------------- attention
def _lengths(case):
    """Row lengths from an eighth of the longest to the longest, odd ones among them; the first is
    the longest."""
    rows, longest = case["rows"], case["longest"]
    return [max(1, longest - (i * 7 * longest) // (8 * max(rows - 1, 1)) - (i & 1)) for i in range(rows)]


def _prepare_attn(case, seed):
    gen, lens = _gen(seed), _lengths(case)
    n = sum(lens)
    q = _randn(gen, n, HEADS, HEAD_DIM).requires_grad_(True)
    k = _randn(gen, n, KV_HEADS, HEAD_DIM).requires_grad_(True)
    v = _randn(gen, n, KV_HEADS, HEAD_DIM).requires_grad_(True)
    grad = _randn(gen, 1, n, HEADS, HEAD_DIM)
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    return dict(case=case, q=q, k=k, v=v, grad=grad, cu=cu, longest=max(lens))


def _run_attn(s):
    q, k, v = s["q"], s["k"], s["v"]
    q.grad = k.grad = v.grad = None
    # as a decoder block calls it: [1, heads, tokens, head_dim] views of token-major tensors
    out = segment_attention(*(t.unsqueeze(0).transpose(1, 2) for t in (q, k, v)), s["cu"], s["longest"],
                            HEAD_DIM ** -0.5)
    out.backward(s["grad"])
    return [out.detach(), q.grad, k.grad, v.grad]


def _work_attn(case):
    lens = _lengths(case)
    n, pairs = sum(lens), sum(0.5 * L * (L + 1) for L in lens)
    return dict(flops=14.0 * pairs * HEADS * HEAD_DIM,                    # 2 products forward, 5 backward
                bytes=2.0 * n * HEAD_DIM * (4 * HEADS + 4 * KV_HEADS) + 4.0 * n * HEADS)


# ------------------------------------------------------------------------------------------- nf4
def _prepare_nf4(case, seed):
    gen = _gen(seed)
    blocks = []
    for _ in range(case["blocks"]):
        block = []
        for o, i in PROJECTIONS:
            block.append(qlora.quantize_nf4(_randn(gen, o, i, std=0.02), nested=case["nested"]))
        blocks.append(block)
    return dict(case=case, blocks=blocks, dtype=getattr(torch, case["dtype"]))


def _run_nf4(s):
    out = []
    for block in s["blocks"]:
        out += dequantize_nf4_batch(block, s["dtype"])
    return out


def _work_nf4(case):
    n = case["blocks"] * BLOCK_WEIGHTS
    absmax = n / 64 + 4.0 * n / 16384 if case["nested"] else 4.0 * n / 64
    return dict(flops=0.0, bytes=0.5 * n + absmax + n * (2.0 if case["dtype"] == "float16" else 4.0))


# ------------------------------------------------------------------------------------------- ops
def _prepare_ops(case, seed):
    gen, n = _gen(seed), case["tokens"]
    low = torch.float16 if case["model"] == "4bit" else getattr(torch, case["model"])
    wide = torch.float32 if case["model"] == "4bit" else low               # hidden states, q and k
    weight = torch.rand(HIDDEN, generator=gen, device=DEV).add_(0.5)
    weight[torch.randperm(HIDDEN, generator=gen, device=DEV)[:16]] *= 1e-4  # a few nearly dead channels
    positions = torch.arange(n, device=DEV).remainder(512).float()          # restart in every row
    freq = positions[:, None] * (1e6 ** (-torch.arange(0, HEAD_DIM, 2, device=DEV).float() / HEAD_DIM))[None]
    angle = torch.cat([freq, freq], -1)[None]
    s = dict(case=case,
             x=_randn(gen, 1, n, HIDDEN, dtype=wide).requires_grad_(True),
             weight=weight.to(wide).requires_grad_(case["model"] != "4bit"),
             q=_randn(gen, 1, n, HEADS * HEAD_DIM, dtype=wide).requires_grad_(True),
             k=_randn(gen, 1, n, KV_HEADS * HEAD_DIM, dtype=wide).requires_grad_(True),
             cos=angle.cos().to(wide), sin=angle.sin().to(wide),
             gate=_randn(gen, 1, n, INTER, dtype=low).requires_grad_(True),
             up=_randn(gen, 1, n, INTER, dtype=low).requires_grad_(True),
             xl=_randn(gen, 1, n, HIDDEN, dtype=torch.float32).requires_grad_(True),
             a=_randn(gen, RANK, HIDDEN, dtype=torch.float32, std=0.015).requires_grad_(True),
             b=_randn(gen, HIDDEN, RANK, dtype=torch.float32, std=0.01).requires_grad_(True),
             dx=_randn(gen, 1, n, HIDDEN, dtype=wide),
             dq=_randn(gen, 1, HEADS, n, HEAD_DIM, dtype=wide), dk=_randn(gen, 1, KV_HEADS, n, HEAD_DIM, dtype=wide),
             dact=_randn(gen, 1, n, INTER, dtype=low),
             dlora=_randn(gen, 1, n, HIDDEN, dtype=torch.float16))
    s["xl16"] = s["xl"].detach().half()
    torch.cuda.manual_seed(seed)                       # the LoRA branch's dropout masks
    return s


def _run_ops(s):
    leaves = [s[name] for name in ("x", "weight", "q", "k", "gate", "up", "xl", "a", "b")]
    for t in leaves:
        t.grad = None
    n = s["case"]["tokens"]
    y = solution.rmsnorm(s["x"], s["weight"], 1e-6)
    q, k = solution.rope(s["q"].view(1, n, HEADS, HEAD_DIM).transpose(1, 2),
                         s["k"].view(1, n, KV_HEADS, HEAD_DIM).transpose(1, 2), s["cos"], s["sin"])
    act = solution.swiglu_recompute(s["gate"], s["up"])
    branch = LoRABranch.apply(s["xl"], s["xl16"], s["a"], s["b"], 0.05, 2.0)
    torch.autograd.backward([y, q, k, act, branch], [s["dx"], s["dq"], s["dk"], s["dact"], s["dlora"]])
    return [y.detach(), q.detach(), k.detach(), act.detach(), branch.detach()] + [
        t.grad for t in leaves if t.requires_grad]


def _work_ops(case):
    n = case["tokens"]
    wide = 4.0 if case["model"] == "4bit" else 2.0
    norm = 5 * n * HIDDEN * wide
    rope = 4 * n * (HEADS + KV_HEADS) * HEAD_DIM * wide + 2 * n * HEAD_DIM * wide
    swiglu = 8 * n * INTER * 2.0
    lora = n * HIDDEN * (4.0 + 4.0 + 2.0 + 2.0)
    return dict(bytes=norm + rope + swiglu + lora, flops=12.0 * n * HIDDEN * RANK)


_PREPARE = dict(head=_prepare_head, step=_prepare_step, eager=_prepare_eager, attn=_prepare_attn,
                nf4=_prepare_nf4, ops=_prepare_ops)
_RUN = dict(head=_run_head, step=_run_step, eager=_run_eager, attn=_run_attn, nf4=_run_nf4, ops=_run_ops)
_WORK = dict(head=_work_head, step=_work_step, eager=_work_step, attn=_work_attn, nf4=_work_nf4, ops=_work_ops)
# About four times what was measured between two correct ways to the same numbers: the head and the
# attention against float64 (2.1e-4 and 3.4e-4), the step between its own and torch's attention and
# between the fused chain and the per-op patches (4.1e-3: fp16 activations through 28 layers), the
# per-op functions against float64 (2.9e-4 in fp16, 2.4e-3 in bf16).
_TOLERANCE = dict(
    head={"rel": 1e-3, "max": 5e-3, "differ": 1e-3},
    step={"rel": 1.6e-2, "max": 0.9},
    eager={"rel": 1.6e-2, "max": 0.9},
    attn={"rel": 1.5e-3, "max": 3e-2},
    ops={"rel": 1.5e-3, "max": 2e-2},
)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


def work(case):
    return _WORK[case["kind"]](case)


def tolerance(case):
    if case["kind"] == "nf4":
        return "exact"
    if case.get("model") == "bfloat16":
        return {"rel": 1e-2, "max": 5e-2}
    return _TOLERANCE[case["kind"]]
