"""Prompts of any length in one pass: the logits and the state a decode continues from, against the FP32 model."""
import pytest
import torch

from warpstate_ai_b200 import WarpStateConfig, WarpStateLM
from warpstate_ai_b200.ops import reference as R
from warpstate_ai_b200.ops.gemm import check_device_errors
from warpstate_ai_b200.serve.engine import DecodeEngine

pytestmark = pytest.mark.gpu


def model_of(heads, ffn, depth=3):
    torch.manual_seed(heads)
    cfg = WarpStateConfig(vocab_size=512, d_model=64 * heads, n_heads=heads, n_cores=2, logical_depth=depth, ffn_hidden=ffn,
                          chunk_size=128, gradient_checkpointing=False, parallel_memory=True)
    with torch.device("cuda"):
        model = WarpStateLM(cfg).eval().requires_grad_(False)
        for core in model.cores:
            core.fast_decay_logit.normal_(1.0, 0.5)
            core.memory_mix_logit.normal_(0.0, 0.5)
    return model


def expected_state(model, ids):
    """(logits at the last position, fast, slow, roped K, V, U of the open chunk) of layer 0 and of the last, FP32."""
    batch, length = ids.shape
    complete, rest = divmod(length, 128)
    padded = torch.nn.functional.pad(ids, (0, -length % 128))
    x, kept = model.embed(padded), []
    for depth, core in model._depths():
        x = x * (1.0 + model.depth_scale[depth]) + model.depth_bias[depth]
        packed = core.in_proj(core.norm1(x))
        _, k, v, _, u = R.split_heads(packed, core.h, 128)
        k = R.apply_rope(k, core.rope_cos, core.rope_sin)
        if complete:
            _, memories = R.attention_memory(packed[:, :complete * 128], *core._memory_arguments(), return_state=True)
        else:
            memories = (torch.zeros(batch, core.h, 64, 64, device="cuda"),) * 2
        caches = [torch.zeros(batch, core.h, 128, 64, device="cuda") for _ in range(3)]
        for cache, t in zip(caches, (k, v, u)):
            cache[:, :, :rest] = t[:, complete, :, :rest] if rest else 0.0
        kept.append((*memories, *caches))
        x = core(x)
    return model.logits_from_hidden(model.final_norm(x))[:, length - 1], kept[0], kept[-1]


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-9))


@pytest.mark.parametrize("batch,heads,ffn,use_kernels", [(1, 4, 512, True), (3, 2, 192, True), (70, 2, 192, True), (2, 4, 512, False)])
@pytest.mark.parametrize("length", [1, 31, 127, 128, 129, 300, 1153])
def test_prompt_of_any_length_in_one_pass(batch, heads, ffn, use_kernels, length):
    # BF16 inputs to every product and three layers: 2^-8 per rounding, about ten of them on the way to a logit or a
    # state of the last layer, adding as a random walk -> 2 % at most; layer 0's K, V, U see three roundings
    model = model_of(heads, ffn)
    ids = torch.randint(0, 512, (batch, length + 3), device="cuda")
    engine = DecodeEngine(model, dtype=torch.bfloat16, use_kernels=use_kernels)
    engine.prefill(ids[:, :1])                                       # leaves values of another prompt in the state
    engine.step(ids[:, 1])
    logits = engine.prefill(ids[:, :length]).clone()
    check_device_errors()
    want, first, last = expected_state(model, ids[:, :length])
    assert engine.pos == length % 128
    assert rel(logits, want) < 0.02
    for state, expected, bound in ((engine.states[0], first, 0.01), (engine.states[-1], last, 0.02)):
        for name, value in zip(("fast", "slow", "k", "v", "u"), expected):
            assert rel(getattr(state, name), value) < bound, (name, bound)
            if name in ("k", "v", "u"):
                assert torch.count_nonzero(getattr(state, name)[:, :, length % 128:]) == 0, name
    for position in range(length, length + 3):                        # a decode continues from it
        stepped = engine.step(ids[:, position])
    check_device_errors()
    assert rel(stepped, expected_state(model, ids[:, :length + 3])[0]) < 0.02


def test_a_prefilled_state_equals_a_stepped_one():
    """The same prompt through the step kernels: what the two leave behind differs by BF16 roundings only."""
    model = model_of(4, 512)
    ids = torch.randint(0, 512, (3, 200), device="cuda")
    whole, stepped = DecodeEngine(model), DecodeEngine(model)
    logits = whole.prefill(ids)
    for position in range(200):
        last = stepped.step(ids[:, position])
    assert rel(logits, last) < 0.02 and whole.pos == stepped.pos
    for a, b in zip(whole.states, stepped.states):
        for name in ("fast", "slow", "mixed"):
            assert rel(getattr(a, name), getattr(b, name)) < 0.02, name
        for name in ("k", "v", "u"):
            assert rel(getattr(a, name)[:, :, :72], getattr(b, name)[:, :, :72]) < 0.02, name


@pytest.mark.parametrize("stream_form", [0, 1])
@pytest.mark.parametrize("batch,heads,length", [(1, 2, 100), (2, 3, 255), (16, 4, 128 * 3 + 44)])
def test_open_chunk_keeps_its_softmax_weights(batch, heads, length, stream_form):
    """A decode step weighs the values in FP32, so the positions of the chunk a prompt ends in do, too: next to the BF16
    rounding of the output itself nothing is lost.  (Weights rounded to BF16 would be of its size, 1.4 times in all.)"""
    from warpstate_ai_b200.ops import _ext, attention
    _ext.require()
    torch.manual_seed(length)
    d, rest = 64 * heads, length % 128
    packed = torch.randn(batch, length, 5, heads, 64, device="cuda").bfloat16()
    packed[:, :, 3] = 40.0                                            # the gate: local attention alone
    logits = [torch.zeros(heads, device="cuda") for _ in range(3)]
    fast, slow = (torch.empty(batch, heads, 64, 64, device="cuda") for _ in range(2))
    mixed = torch.empty(batch, heads, 64, 64, device="cuda", dtype=torch.bfloat16)
    caches = [torch.empty(batch, heads, 128, 64, device="cuda", dtype=torch.bfloat16) for _ in range(3)]
    lib = _ext.cdll()
    try:
        lib.ws_attn_set_stream_mode(stream_form)
        y = torch.ops.ws_b200.attn_prefill(packed.view(batch * length, 5 * d), attention.rope_table(packed.device, pair_major=True),
                                           *logits, batch, length, heads, fast, slow, mixed, *caches,
                                           attention.error_flag(packed.device))
    finally:
        lib.ws_attn_set_stream_mode(-1)
    check_device_errors()
    cos, sin = attention.rope_table(packed.device).double()[:rest].unsqueeze(1).unbind(-1)

    def turned(x):                                                    # rounded to BF16, as a decode step caches it
        even, odd = x.double()[..., 0::2], x.double()[..., 1::2]
        return torch.stack((even * cos - odd * sin, odd * cos + even * sin), dim=-1).flatten(-2).bfloat16().double()

    q, k, v = packed[:, length - rest:, :3].unbind(2)
    scores = torch.einsum("brhi,bchi->bhrc", turned(q), turned(k)) / 8.0
    future = torch.ones(rest, rest, dtype=torch.bool, device="cuda").triu(1)
    want = torch.einsum("bhrc,bchi->brhi", torch.softmax(scores.masked_fill(future, float("-inf")), dim=-1), v.double())
    got = y.view(batch, length, heads, 64)[:, length - rest:]
    assert rel(got, want) < 1.1 * rel(want.bfloat16(), want)


@pytest.mark.parametrize("rows", [1, 44, 95, 300, 1000])
@pytest.mark.parametrize("d,ffn", [(256, 688), (2048, 512)])
def test_activation_of_a_prompt_is_rounded_once(rows, d, ffn):
    """As in a decode step, up and gate stay FP32 until the activation: next to its own BF16 rounding nothing is lost (with
    rounded factors it would be 1.5 times that).  The sigmoid's 2^-11 is a sixth of the rounding at most."""
    from warpstate_ai_b200.ops import _ext, gemm as G
    _ext.require()
    torch.manual_seed(rows + d)
    x, w = torch.randn(rows, d, device="cuda").bfloat16(), (torch.randn(2 * ffn, d, device="cuda") / d ** 0.5).bfloat16()
    up, gate = (x.double() @ w.double().t()).chunk(2, dim=-1)
    want = up * gate * torch.sigmoid(gate)
    packed, act = G.linear_swiglu(x, w, want_packed=False, wide=True)
    check_device_errors()
    assert packed is None and rel(act, want) < 1.1 * rel(want.bfloat16(), want)
    packed, rounded = G.linear_swiglu(x, w)                           # training: from the values its backward pass reads
    u, g = packed.double().chunk(2, dim=-1)
    want = u * g * torch.sigmoid(g)
    assert rel(rounded, want) < 1.1 * rel(want.bfloat16(), want)


@pytest.mark.parametrize("heads,ffn,dtype,use_kernels", [(3, 192, torch.float32, True), (1, 64, torch.float32, True),
                                                         (2, 100, torch.float32, False), (2, 192, torch.float16, False)])
def test_short_prompts_of_models_outside_the_tile_kernels(heads, ffn, dtype, use_kernels):
    """Widths that are no multiple of 128, an FFN that is none of 8, half-precision weights: stepped, as ever."""
    model = model_of(heads, ffn).to(dtype)
    ids = torch.randint(0, 512, (2, 21), device="cuda")
    engine = DecodeEngine(model, use_kernels=use_kernels)
    logits = engine.prefill(ids[:, :20]).clone()
    after = engine.step(ids[:, 20])
    check_device_errors()
    wide = model.float()
    assert rel(logits, expected_state(wide, ids[:, :20])[0]) < 0.02 and rel(after, expected_state(wide, ids)[0]) < 0.02
