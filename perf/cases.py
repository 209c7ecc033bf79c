"""What is timed of this framework: its blocks, its heads and its serving calls, through the entry points a program calls.

A case is a dict of plain values; ``kind`` says which part it is:

* ``core``     one block (`WarpStateCore`) under BF16 autocast: a scoring pass, or forward and backward into an arena;
* ``mixer``    the chunk attention + matrix memory of a block on packed projections, forward and backward;
* ``head``     the tied LM head with cross-entropy, forward and backward: every position labelled (pretraining), or only
               the response of each padded sequence (post-training; DPO takes one log-probability per sequence);
* ``model``    a whole model's micro-batch: loss and every gradient;
* ``prefill``  `DecodeEngine.prefill` of a batch of prompts: the logits after the prompt and the state it leaves;
* ``decode``   a prompt, then teacher-forced single-token steps; the logits of every step.

Widths are those of the production configuration (d 2048, 32 heads, FFN 7168), the default one (1280, 20, 4480) and the
smoke one (256, 4, 688).  Training lengths are whole 128-token chunks, as the blocks demand; prompts have any length.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from warpstate_ai_b200 import WarpStateConfig, WarpStateLM
from warpstate_ai_b200.models.warpstate import WarpStateCore
from warpstate_ai_b200.ops import attention, lmhead
from warpstate_ai_b200.optim import ParamArena
from warpstate_ai_b200.serve.engine import DecodeEngine

DEVICE = "cuda"
VOCAB = 32768
CHUNK = 128
EPS = 1e-5
WIDTHS = {2048: (32, 7168), 1280: (20, 4480), 256: (4, 688)}      # d_model -> (heads, FFN width)


def listed():
    return [
        # a short text scored by one production block (evaluation, frozen DPO reference): latency of few rows
        dict(name="core_score_short", kind="core", d=2048, batch=1, tokens=128, train=False),
        # a validation batch through one production block
        dict(name="core_score_batch", kind="core", d=2048, batch=3, tokens=1152, train=False),
        # the default configuration's block in a small training run
        dict(name="core_train_default", kind="core", d=1280, batch=2, tokens=896, train=True),
        # the headline micro-batch, 8 x 2048 tokens, through one production block
        dict(name="core_train_headline", kind="core", d=2048, batch=8, tokens=2048, train=True),
        # attention and memory alone, at the length and head count of a DPO micro-batch (two pairs)
        dict(name="mixer_train", kind="mixer", d=2048, batch=4, tokens=2048),
        # loss head of the headline micro-batch
        dict(name="head_pretrain", kind="head", d=2048, batch=8, tokens=2048, labels="all"),
        # two DPO pairs padded to 2048: labels on the responses only
        dict(name="head_dpo", kind="head", d=2048, batch=4, tokens=2048, labels="response"),
        # the smoke configuration's whole micro-batch: launches and host work count
        dict(name="model_train_smoke", kind="model", d=256, cores=2, depth=4, batch=2, tokens=512),
        # a chat prompt of the production model, one sequence, not a whole number of chunks
        dict(name="prefill_chat", kind="prefill", d=2048, layers=28, batch=1, tokens=300),
        # a batch of long prompts, eight of the production model's layers
        dict(name="prefill_batch", kind="prefill", d=2048, layers=8, batch=16, tokens=1000),
        # streaming answer to one user, production model, over the end of a chunk
        dict(name="decode_single", kind="decode", d=2048, layers=28, batch=1, tokens=100, steps=48),
        # 64 streams in lock-step, eight of the production model's layers
        dict(name="decode_batch", kind="decode", d=2048, layers=8, batch=64, tokens=128, steps=40),
    ]


def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["core", "core", "core", "mixer", "head", "head", "model", "prefill", "prefill", "decode", "decode"])
    d = rng.choice([1280, 2048, 2048])
    if kind in ("core", "mixer"):
        rows = _log_int(rng, 1, 128 if kind == "core" else 96)     # chunks in all
        batch = _log_int(rng, 1, min(rows, 8))
        case = dict(kind=kind, d=d, batch=batch, tokens=CHUNK * max(1, min(16, rows // batch)))
        if kind == "core":
            case["train"] = rng.random() < 0.6
        return case
    if kind == "head":
        return dict(kind="head", d=d, batch=_log_int(rng, 1, 8), tokens=CHUNK * rng.randint(2, 16),
                    labels=rng.choice(["all", "response"]))
    if kind == "model":
        cores = rng.randint(1, 4)
        return dict(kind="model", d=rng.choice([256, 1280]), cores=cores, depth=cores * rng.randint(1, 2),
                    batch=_log_int(rng, 1, 4), tokens=CHUNK * rng.randint(1, 8))
    layers = rng.choice([4, 8, 28 if d == 2048 else 16])
    if kind == "prefill":
        return dict(kind="prefill", d=d, layers=layers, batch=_log_int(rng, 1, 16 if layers <= 8 else 4),
                    tokens=_log_int(rng, 5, 1000))
    return dict(kind="decode", d=d, layers=layers, batch=_log_int(rng, 1, 64 if layers <= 8 else 16),
                tokens=_log_int(rng, 5, 400), steps=rng.randint(8, 48))


# ------------------------------------------------------------------------------------------------- inputs from the seed
class Draws:
    """Random tensors in a fixed order from one seed."""

    def __init__(self, seed):
        self.generator = torch.Generator(device=DEVICE)
        self.generator.manual_seed(int(seed) * 7919 + 17)

    def normal(self, *shape, std=1.0, mean=0.0):
        return torch.empty(shape, device=DEVICE).normal_(mean, std, generator=self.generator)

    def tokens(self, *shape):
        return torch.randint(0, VOCAB, shape, device=DEVICE, generator=self.generator)


def _core_weights(draws, d, depth):
    """One block's parameters: the framework's initial distributions, norms and decays moved off their starting points."""
    heads, ffn = WIDTHS[d]
    narrow = 0.02 / math.sqrt(2.0 * depth)
    logit = lambda p: math.log(p / (1.0 - p))
    return {"fast_decay_logit": draws.normal(heads, std=0.3, mean=logit(0.90)),
            "slow_decay_logit": draws.normal(heads, std=0.3, mean=logit(0.99)),
            "memory_mix_logit": draws.normal(heads, std=0.3),
            "norm1.weight": draws.normal(d, std=0.1, mean=1.0),
            "in_proj.weight": draws.normal(5 * d, d, std=0.02),
            "out_proj.weight": draws.normal(d, d, std=narrow),
            "norm2.weight": draws.normal(d, std=0.1, mean=1.0),
            "ffn.up_gate.weight": draws.normal(2 * ffn, d, std=0.02),
            "ffn.down.weight": draws.normal(d, ffn, std=narrow)}


def _model_weights(draws, d, cores, depth):
    weights = {"depth_scale": draws.normal(depth, d, std=0.05), "depth_bias": draws.normal(depth, d, std=0.01),
               "embed.weight": draws.normal(VOCAB, d, std=0.02)}
    for index in range(cores):
        weights.update({f"cores.{index}.{name}": w for name, w in _core_weights(draws, d, depth).items()})
    weights["final_norm.weight"] = draws.normal(d, std=0.1, mean=1.0)
    return weights


def _config(d, cores, depth, ffn=None):
    heads, width = WIDTHS[d]
    return WarpStateConfig(vocab_size=VOCAB, d_model=d, n_heads=heads, n_cores=cores, logical_depth=depth,
                           ffn_hidden=ffn or width, chunk_size=CHUNK, rms_eps=EPS, gradient_checkpointing=False,
                           parallel_memory=True)


def _module(make, weights):
    with torch.device("meta"):
        module = make()
    module.load_state_dict(weights, assign=True)
    return module.to(DEVICE)


def _label_spans(case):
    """[start, stop) of the labelled positions of each sequence: prompts of an eighth to a half of the padded length,
    responses of a sixteenth to a half, spread evenly over the batch."""
    batch, length = case["batch"], case["tokens"]
    if case["labels"] == "all":
        return [(0, length)] * batch
    spans = []
    for index in range(batch):
        prompt = length // 8 + (length * 3 // 8) * (2 * index + 1) // (2 * batch)
        response = length // 16 + (length * 7 // 16) * ((2 * index * 3) % (2 * batch) + 1) // (2 * batch)
        spans.append((prompt, min(prompt + response, length)))
    return spans


def _inputs(case, seed):
    """Everything random of a case: what `prepare` loads into the framework and `exact` computes with."""
    draws, kind, d = Draws(seed), case["kind"], case["d"]
    heads, _ = WIDTHS[d]
    if kind == "core":
        shape = (case["batch"], case["tokens"], d)
        return dict(weights=_core_weights(draws, d, 28), x=draws.normal(*shape, std=0.2), dy=draws.normal(*shape, std=0.01),
                    scale=draws.normal(d, std=0.05), bias=draws.normal(d, std=0.01))
    if kind == "mixer":
        rows = case["batch"] * case["tokens"]
        logits = _core_weights(draws, 256, 28)
        return dict(qkvgu=draws.normal(rows, 5 * d, std=0.9).bfloat16(), dy=draws.normal(rows, d, std=0.01).bfloat16(),
                    weights={name: draws.normal(heads, std=0.3, mean=float(logits[name].mean()))
                             for name in ("fast_decay_logit", "slow_decay_logit", "memory_mix_logit")})
    if kind == "head":
        batch, length = case["batch"], case["tokens"]
        labels = torch.full((batch, length), -100, device=DEVICE, dtype=torch.long)
        for row, (start, stop) in enumerate(_label_spans(case)):
            labels[row, start:stop] = draws.tokens(stop - start)
        return dict(weight=draws.normal(VOCAB, d, std=0.02), hidden=draws.normal(batch, length, d).bfloat16(),
                    labels=labels, coef=draws.normal(batch, std=0.05))
    if kind == "model":
        return dict(weights=_model_weights(draws, d, case["cores"], case["depth"]),
                    ids=draws.tokens(case["batch"], case["tokens"]), targets=draws.tokens(case["batch"], case["tokens"]))
    return dict(weights=_model_weights(draws, d, case["layers"], case["layers"]),
                ids=draws.tokens(case["batch"], case["tokens"] + case.get("steps", 0)))


# ------------------------------------------------------------------------------------------------- the framework's side
def prepare(case, seed):
    data, kind, d = _inputs(case, seed), case["kind"], case["d"]
    state = dict(case=dict(case), kind=kind)
    if kind == "core":
        core = _module(lambda: WarpStateCore(_config(d, 1, 28)), data["weights"])
        state.update(core=core, x=data["x"], scale=data["scale"], bias=data["bias"])
        if case["train"]:
            state.update(arena=ParamArena(core), dy=data["dy"])
            for name in ("x", "scale", "bias"):
                state[name].requires_grad_(True)
    elif kind == "mixer":
        core = _module(lambda: WarpStateCore(_config(d, 1, 28, ffn=64)),
                       {**_thin_core(d), **data["weights"]})
        state.update(core=core, qkvgu=data["qkvgu"], dy=data["dy"])
    elif kind == "head":
        model = _module(lambda: WarpStateLM(_config(d, 1, 1, ffn=64)),
                        {"embed.weight": data["weight"], "depth_scale": torch.zeros(1, d, device=DEVICE),
                         "depth_bias": torch.zeros(1, d, device=DEVICE), "final_norm.weight": torch.ones(d, device=DEVICE),
                         **{f"cores.0.{name}": w for name, w in _thin_core(d).items()}}).train()
        state.update(model=model, arena=ParamArena(model), hidden=data["hidden"].requires_grad_(True),
                     labels=data["labels"], coef=data["coef"])
    elif kind == "model":
        model = _module(lambda: WarpStateLM(_config(d, case["cores"], case["depth"])), data["weights"]).train()
        state.update(model=model, arena=ParamArena(model), ids=data["ids"], targets=data["targets"])
    else:
        model = _module(lambda: WarpStateLM(_config(d, case["layers"], case["layers"])), data["weights"]).eval()
        state.update(engine=DecodeEngine(model), ids=data["ids"])
    return state


def _thin_core(d):
    """A block that is built but not run (its FFN is 64 wide)."""
    heads, _ = WIDTHS[d]
    zeros = lambda *shape: torch.zeros(shape, device=DEVICE)
    return {"fast_decay_logit": zeros(heads), "slow_decay_logit": zeros(heads), "memory_mix_logit": zeros(heads),
            "norm1.weight": zeros(d), "norm2.weight": zeros(d), "in_proj.weight": zeros(5 * d, d),
            "out_proj.weight": zeros(d, d), "ffn.up_gate.weight": zeros(128, d), "ffn.down.weight": zeros(d, 64)}


def _autocast():
    return torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False)


def _grads(module):
    return {name: p.grad for name, p in module.named_parameters()}


def run(state):
    return _RUN[state["kind"]](state)


def _run_core(s):
    core = s["core"]
    if "arena" not in s:
        with torch.no_grad(), _autocast():
            return core(s["x"], s["scale"], s["bias"])
    s["arena"].zero_grad()
    for name in ("x", "scale", "bias"):
        s[name].grad = None
    with _autocast():
        y = core(s["x"], s["scale"], s["bias"])
    y.backward(s["dy"])
    return dict(y=y.detach(), dx=s["x"].grad, dscale=s["scale"].grad, dbias=s["bias"].grad, grads=_grads(core))


def _run_mixer(s):
    case, core = s["case"], s["core"]
    y, saved = attention.forward(s["qkvgu"], core, case["batch"], case["tokens"])
    dqkvgu, fast, slow, mix = attention.backward(s["dy"], s["qkvgu"], saved, core, case["batch"], case["tokens"])
    return dict(y=y, dqkvgu=dqkvgu, fast=fast, slow=slow, mix=mix)


def _run_head(s):
    model, hidden = s["model"], s["hidden"]
    s["arena"].zero_grad()
    hidden.grad = None
    batch, length, d = hidden.shape
    with _autocast():
        if s["case"]["labels"] == "all":
            value = model.loss_from_hidden(hidden, s["labels"])
            loss = value
        else:
            rows = lmhead.token_logps(hidden.view(batch * length, d), model.embed.weight, s["labels"].view(-1))
            value = rows.view(batch, length).sum(dim=1)
            loss = (value * s["coef"]).sum()
    loss.backward()
    return dict(value=value.detach(), dhidden=hidden.grad, dweight=model.embed.weight.grad)


def _run_model(s):
    s["arena"].zero_grad()
    with _autocast():
        _, loss = s["model"](s["ids"], s["targets"], return_logits=False)
    loss.backward()
    return dict(loss=loss.detach(), grads=_grads(s["model"]))


def _run_prefill(s):
    engine = s["engine"]
    logits = engine.prefill(s["ids"])
    kept = {"logits": logits}
    for index in sorted({0, len(engine.states) - 1}):        # the first and the last layer's state
        layer = engine.states[index]
        kept[f"layer{index}"] = dict(fast=layer.fast, slow=layer.slow, k=layer.k, v=layer.v, u=layer.u)
    return kept


def _run_decode(s):
    engine, ids, prompt = s["engine"], s["ids"], s["case"]["tokens"]
    logits = [engine.prefill(ids[:, :prompt]).clone()]
    for position in range(prompt, ids.shape[1]):
        logits.append(engine.step(ids[:, position]).clone())
    return torch.stack(logits, dim=1)


_RUN = {"core": _run_core, "mixer": _run_mixer, "head": _run_head, "model": _run_model, "prefill": _run_prefill,
        "decode": _run_decode}


# ------------------------------------------------------------------------------------------------- work and tolerance
def _core_elements(d):
    _, ffn = WIDTHS[d]
    return 6 * d * d + 3 * d * ffn


def _mixer_flops(rows, d, backward):
    """Causal scores and values (half of 128 x 128), memory read and write (64 x 64), per head and position."""
    heads = WIDTHS[d][0]
    forward = rows * heads * (2 * 2 * 64 * 64 + 2 * 2 * 64 * 64)
    return forward * (3.5 if backward else 1.0)


def _decode_state_bytes(case, d, position):
    """Mixed memories and the chunk's keys and values of one layer and step, BF16."""
    heads = WIDTHS[d][0]
    return case["batch"] * heads * (64 * 64 * 2 + 2 * 64 * 2 * (position % CHUNK + 1))


def work(case):
    kind, d = case["kind"], case["d"]
    rows = case["batch"] * case["tokens"]
    if kind == "core":
        elements = _core_elements(d)
        if not case["train"]:
            return dict(bytes=2 * elements + rows * d * 8, flops=2 * elements * rows + _mixer_flops(rows, d, False))
        return dict(bytes=(2 + 4) * elements + rows * d * 16,
                    flops=6 * elements * rows + _mixer_flops(rows, d, True))
    if kind == "mixer":
        return dict(bytes=rows * d * 2 * (5 + 1 + 1 + 5), flops=_mixer_flops(rows, d, True))
    if kind == "head":
        labelled = sum(stop - start for start, stop in _label_spans(case))
        return dict(bytes=VOCAB * d * (2 + 4) + labelled * d * 2 + rows * d * 2, flops=6.0 * labelled * d * VOCAB)
    if kind == "model":
        elements = _core_elements(d)
        flops = case["depth"] * (6 * elements * rows + _mixer_flops(rows, d, True)) + 6.0 * rows * d * VOCAB
        return dict(bytes=(2 + 4) * (case["cores"] * elements + VOCAB * d), flops=flops)
    layers, elements = case["layers"], _core_elements(d)
    heads = WIDTHS[d][0]
    prompt = dict(bytes=2 * layers * elements + 2 * VOCAB * d + layers * case["batch"] * heads * 64 * 64 * 8,
                  flops=layers * (2 * elements * rows + _mixer_flops(rows, d, False)) + 2 * case["batch"] * VOCAB * d)
    if kind == "prefill":
        return prompt
    steps = case["steps"]
    state = sum(_decode_state_bytes(case, d, case["tokens"] + step) for step in range(steps))
    return dict(bytes=prompt["bytes"] + steps * (2 * layers * elements + 2 * VOCAB * d + case["batch"] * VOCAB * 4)
                + layers * state,
                flops=prompt["flops"] + steps * 2 * case["batch"] * (layers * elements + VOCAB * d))


def tolerance(case):
    kind = case["kind"]
    if kind == "core":
        return {"rel": 0.03}
    if kind == "mixer":
        return {"rel": 0.02}
    if kind == "head":
        return {"rel": 0.02}
    return {"rel": 0.06}


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def _norm64(x, weight):
    return x * torch.rsqrt(x.square().mean(dim=-1, keepdim=True) + EPS) * weight


def _rope64(x):
    """``x [..., 128, 64]``: pairs (2i, 2i + 1) turned by position * 10000 ** (-2i / 64)."""
    angle = torch.outer(torch.arange(CHUNK, device=x.device, dtype=torch.float64),
                        10000.0 ** (-torch.arange(0, 64, 2, device=x.device, dtype=torch.float64) / 64))
    cos, sin = angle.cos(), angle.sin()
    even, odd = x[..., 0::2], x[..., 1::2]
    return torch.stack((even * cos - odd * sin, odd * cos + even * sin), dim=-1).flatten(-2)


def _mixer64(packed, logits, heads, complete=None):
    """``packed [B, T, 5d]`` -> (output ``[B, T, d]``, fast and slow state after ``complete`` chunks, roped K, V, U)."""
    batch, length, _ = packed.shape
    chunks = length // CHUNK
    q, k, v, gate, u = packed.view(batch, chunks, CHUNK, 5, heads, 64).permute(3, 0, 1, 4, 2, 5)
    q, k = _rope64(q), _rope64(k)
    scores = q @ k.transpose(-1, -2) / 8.0
    future = torch.ones(CHUNK, CHUNK, dtype=torch.bool, device=packed.device).triu(1)
    local = torch.softmax(scores.masked_fill(future, -math.inf), dim=-1) @ v
    writes = torch.tanh(k).transpose(-1, -2) @ torch.tanh(u) / CHUNK
    fast_keep, slow_keep, mix = (torch.sigmoid(t).view(1, heads, 1, 1) for t in logits)
    fast = slow = torch.zeros_like(writes[:, 0])
    seen, complete = [], chunks if complete is None else complete
    last = (fast, slow)
    for index in range(chunks):
        seen.append(mix * fast + (1.0 - mix) * slow)
        fast = fast_keep * fast + (1.0 - fast_keep) * writes[:, index]
        slow = slow_keep * slow + (1.0 - slow_keep) * writes[:, index]
        if index + 1 == complete:
            last = (fast, slow)
    memory = q @ torch.stack(seen, dim=1) / 8.0
    gate = torch.sigmoid(gate)
    y = gate * local + (1.0 - gate) * memory
    return y.permute(0, 1, 3, 2, 4).reshape(batch, length, heads * 64), last, (k, v, u)


def _core64(x, w, scale, bias, complete=None):
    heads = w["fast_decay_logit"].shape[0]
    x = x * (1.0 + scale) + bias
    packed = _norm64(x, w["norm1.weight"]) @ w["in_proj.weight"].t()
    y, last, kvu = _mixer64(packed, (w["fast_decay_logit"], w["slow_decay_logit"], w["memory_mix_logit"]), heads, complete)
    x = x + y @ w["out_proj.weight"].t()
    up, gate = (_norm64(x, w["norm2.weight"]) @ w["ffn.up_gate.weight"].t()).chunk(2, dim=-1)
    return x + (F.silu(gate) * up) @ w["ffn.down.weight"].t(), last, kvu


def _wide(values, grad=False):
    return {name: t.double().requires_grad_(grad) for name, t in values.items()}


def exact(case, seed):
    data = _inputs(case, seed)
    with torch.no_grad() if case["kind"] in ("prefill", "decode", "head") else torch.enable_grad():
        return _EXACT[case["kind"]](case, data)


def _exact_core(case, data):
    train = case["train"]
    w = _wide(data["weights"], train)
    x, scale, bias = (data[name].double().requires_grad_(train) for name in ("x", "scale", "bias"))
    with torch.set_grad_enabled(train):
        y, _, _ = _core64(x, w, scale, bias)
    if not train:
        return y
    y.backward(data["dy"].double())
    return dict(y=y.detach(), dx=x.grad, dscale=scale.grad, dbias=bias.grad, grads={name: t.grad for name, t in w.items()})


def _exact_mixer(case, data):
    w = _wide(data["weights"], True)
    rows, width = data["dy"].shape
    packed = data["qkvgu"].double().view(case["batch"], case["tokens"], 5 * width).requires_grad_(True)
    y, _, _ = _mixer64(packed, (w["fast_decay_logit"], w["slow_decay_logit"], w["memory_mix_logit"]), width // 64)
    y.backward(data["dy"].double().view_as(y))
    return dict(y=y.detach().view(rows, width), dqkvgu=packed.grad.view(rows, 5 * width), fast=w["fast_decay_logit"].grad,
                slow=w["slow_decay_logit"].grad, mix=w["memory_mix_logit"].grad)


def _head64(hidden, weight, labels, row_weight):
    """Label log-probabilities of ``hidden [rows, d]`` and the gradients of ``sum(row_weight * logp)``."""
    logp = torch.zeros(hidden.shape[0], dtype=torch.float64, device=hidden.device)
    dhidden, dweight = torch.zeros_like(hidden), torch.zeros_like(weight)
    rows = torch.nonzero(labels != -100)[:, 0]
    for part in rows.split(2048):
        h, label = hidden[part], labels[part, None]
        p = torch.log_softmax(h @ weight.t(), dim=-1)
        logp[part] = p.gather(1, label)[:, 0]
        p = p.exp_().neg_()
        p.scatter_add_(1, label, torch.ones_like(label, dtype=torch.float64))
        p *= row_weight[part, None]
        dhidden[part] = p @ weight
        dweight += p.t() @ h
    return logp, dhidden, dweight


def _exact_head(case, data):
    batch, length, d = data["hidden"].shape
    labels = data["labels"].view(-1)
    counted = int((labels != -100).sum())
    if case["labels"] == "all":
        row_weight = torch.full((batch * length,), -1.0 / counted, dtype=torch.float64, device=DEVICE)
    else:
        row_weight = data["coef"].double().repeat_interleave(length)
    logp, dhidden, dweight = _head64(data["hidden"].double().view(-1, d), data["weight"].double(), labels, row_weight)
    value = -logp.sum() / counted if case["labels"] == "all" else logp.view(batch, length).sum(dim=1)
    return dict(value=value, dhidden=dhidden.view(batch, length, d), dweight=dweight)


def _exact_model(case, data):
    w = _wide(data["weights"], True)
    x = w["embed.weight"][data["ids"]]
    for depth in range(case["depth"]):
        prefix = f"cores.{depth % case['cores']}."
        core = {name[len(prefix):]: t for name, t in w.items() if name.startswith(prefix)}
        x, _, _ = _core64(x, core, w["depth_scale"][depth], w["depth_bias"][depth])
    hidden = _norm64(x, w["final_norm.weight"])
    loss = F.cross_entropy((hidden @ w["embed.weight"].t()).flatten(0, 1), data["targets"].flatten())
    loss.backward()
    return dict(loss=loss.detach(), grads={name: t.grad for name, t in w.items()})


def _trunk64(case, w, ids):
    """Final-norm hidden states of ``ids``, and per layer the state left behind, as `DecodeEngine` keeps it."""
    batch, length = ids.shape
    complete = length // CHUNK
    padded = F.pad(ids, (0, -length % CHUNK))
    x = w["embed.weight"][padded].double()
    states = []
    for depth in range(case["layers"]):
        prefix = f"cores.{depth}."
        core = _wide({name[len(prefix):]: t for name, t in w.items() if name.startswith(prefix)})
        x, (fast, slow), kvu = _core64(x, core, w["depth_scale"][depth].double(), w["depth_bias"][depth].double(), complete)
        if depth in (0, case["layers"] - 1):
            open_chunk = [torch.zeros_like(t[:, 0]) for t in kvu]
            for cleared, t in zip(open_chunk, kvu):
                if length % CHUNK:
                    cleared[:, :, :length % CHUNK] = t[:, -1, :, :length % CHUNK]
            states.append((depth, dict(fast=fast, slow=slow, k=open_chunk[0], v=open_chunk[1], u=open_chunk[2])))
    return _norm64(x[:, :length], w["final_norm.weight"].double()), states


def _exact_prefill(case, data):
    hidden, states = _trunk64(case, data["weights"], data["ids"])
    kept = {"logits": hidden[:, -1] @ data["weights"]["embed.weight"].double().t()}
    kept.update({f"layer{depth}": state for depth, state in states})
    return kept


def _exact_decode(case, data):
    hidden, _ = _trunk64(case, data["weights"], data["ids"])
    return hidden[:, case["tokens"] - 1:] @ data["weights"]["embed.weight"].double().t()


_EXACT = {"core": _exact_core, "mixer": _exact_mixer, "head": _exact_head, "model": _exact_model,
          "prefill": _exact_prefill, "decode": _exact_decode}
