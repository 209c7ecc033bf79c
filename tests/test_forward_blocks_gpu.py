"""Blocks that nothing differentiates run as one native chain over one allocation: the same bits as launch by launch, the kernels that add
the pieces of a cut product do the next norm, and the first chunk has no memories to read."""
import pytest
import torch

from warpstate_ai_b200 import WarpStateConfig, WarpStateLM
from warpstate_ai_b200.models.warpstate import WarpStateCore
from warpstate_ai_b200.ops import _ext, attention, fused, gemm
from warpstate_ai_b200.serve.engine import DecodeEngine


def config(d, ffn, depth=1, cores=1):
    return WarpStateConfig(vocab_size=512, d_model=d, n_heads=d // 64, n_cores=cores, logical_depth=depth, ffn_hidden=ffn, chunk_size=128,
                           gradient_checkpointing=False, parallel_memory=True)


# one chunk and several; rows whose products are cut along k (out_proj, down, both) and rows whose are not; wider than the norm of pieces
@pytest.mark.gpu
@pytest.mark.parametrize("batch,tokens,d,ffn", [(1, 128, 2048, 192), (1, 128, 256, 2048), (2, 256, 1024, 704), (9, 256, 384, 128), (1, 384, 2176, 4096)])
@pytest.mark.parametrize("modulated", [True, False])
def test_scoring_equals_the_launches_one_by_one(monkeypatch, batch, tokens, d, ffn, modulated):
    torch.manual_seed(d + ffn)
    with torch.device("cuda"):
        core = WarpStateCore(config(d, ffn))
        x = torch.randn(batch, tokens, d)
        mod = torch.randn(2, d).mul_(0.1).unbind(0) if modulated else (None, None)
        for norm in (core.norm1, core.norm2):
            norm.weight.data.normal_(1, 0.2)
    kept = x.clone()
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        one = core(x, *mod)
        monkeypatch.setattr(gemm, "_policy", {"fwd:0x0x0": {"kernel": "pair", "sm_limit": 0}})   # launch by launch, from Python
        many = fused.core_forward(core, x, *mod)
    gemm.check_device_errors()
    assert torch.equal(one, many) and torch.equal(x, kept)


@pytest.mark.gpu
@pytest.mark.parametrize("stream_form", [0, 1])
def test_the_first_chunk_reads_zero_memories(stream_form):
    torch.manual_seed(0)
    batch, heads = 3, 4
    with torch.device("cuda"):
        core = WarpStateCore(config(64 * heads, 128))
        qkvgu = (torch.randn(batch * 128, 5 * 64 * heads) * 1.5).bfloat16()
    lib = _ext.cdll()
    try:
        lib.ws_attn_set_stream_mode(stream_form)
        with_memories = attention.forward_only(qkvgu, core, batch, 128)[0]
        without = attention.forward_first_chunk(qkvgu, core, batch)
    finally:
        lib.ws_attn_set_stream_mode(-1)
    gemm.check_device_errors()
    assert torch.equal(without, with_memories)
    with pytest.raises(RuntimeError, match="states"):
        torch.ops.ws_b200.attn_fwd(qkvgu[:256].contiguous(), None, attention.rope_table(qkvgu.device, pair_major=True), 1, 256, heads,
                                   gemm.error_flag(qkvgu.device))


# prompts below a chunk, of whole chunks and with an open one; few rows, whose products are cut, and many; shared cores; parameters that
# are not FP32 come as copies
@pytest.mark.gpu
@pytest.mark.parametrize("batch,length,d,ffn,half", [(1, 5, 256, 704, False), (2, 128, 512, 2048, False), (1, 300, 2048, 1024, False),
                                                     (5, 700, 256, 704, False), (2, 200, 256, 704, True)])
def test_all_blocks_of_a_prompt_equal_the_blocks_one_by_one(monkeypatch, batch, length, d, ffn, half):
    torch.manual_seed(length)
    with torch.device("cuda"):
        model = WarpStateLM(config(d, ffn, depth=5, cores=2))
    with torch.no_grad():
        model.depth_scale.normal_(0, 0.1)
        model.depth_bias.normal_(0, 0.1)
    model.eval().requires_grad_(False)
    if half:
        for core in model.cores:
            core.norm1.weight.data, core.fast_decay_logit.data = core.norm1.weight.data.bfloat16(), core.fast_decay_logit.data.bfloat16()
    ids = torch.randint(0, 512, (batch, length), device="cuda")
    together, apart = DecodeEngine(model), DecodeEngine(model)
    got = together.prefill(ids).clone()
    assert fused.cores_prefill_state(list(model.cores), torch.zeros(batch * length, d, device="cuda"), model.depth_scale[:2], model.depth_bias[:2],
                                     batch, length, apart.states or together.states[:2]) is not None
    want_engine_state = [[t.clone() for t in (st.fast, st.slow, st.mixed, st.k, st.v, st.u)] for st in together.states[2:]]
    monkeypatch.setattr(fused, "cores_prefill_state", lambda *a: None)
    want = apart.prefill(ids)
    gemm.check_device_errors()
    assert torch.equal(got, want)
    for mine, theirs in zip(want_engine_state, apart.states[2:]):
        assert all(torch.equal(a, getattr(theirs, name)) for a, name in zip(mine, ("fast", "slow", "mixed", "k", "v", "u")))


# the widths that rows are padded to and one row past each; several sequences, whole chunks among them; ragged contractions
@pytest.mark.gpu
@pytest.mark.parametrize("batch,length,d,ffn", [(1, 1, 512, 704), (1, 16, 1280, 4480), (1, 17, 512, 704), (3, 11, 640, 1088), (1, 49, 512, 704),
                                                (13, 5, 1280, 4480), (1, 96, 512, 704), (1, 97, 640, 704), (1, 128, 2048, 1024)])
def test_a_short_prompt_streams_its_weights(monkeypatch, batch, length, d, ffn):
    """In other kernels than longer prompts: the same BF16 products added in FP32 in another order, so both are as far from the FP32 forward
    pass, and no further from each other than roundings to BF16 that a changed ulp flips."""
    torch.manual_seed(length + d)
    with torch.device("cuda"):
        model = WarpStateLM(config(d, ffn, depth=4, cores=2))
    with torch.no_grad():
        model.depth_scale.normal_(0, 0.1)
        model.depth_bias.normal_(0, 0.1)
    model.eval().requires_grad_(False)
    ids = torch.randint(0, 512, (batch, length), device="cuda")
    streamed, tiled = DecodeEngine(model), DecodeEngine(model)
    got = streamed.prefill(ids).clone()
    monkeypatch.setattr(fused, "cores_prefill_state", lambda *a: None)
    want = tiled.prefill(ids)
    gemm.check_device_errors()
    exact = model(torch.nn.functional.pad(ids, (0, -length % 128)))[:, length - 1].float()
    assert float((got - want).norm()) < 0.01 * float(want.norm())
    assert float((got - exact).norm()) < 1.2 * float((want - exact).norm()) + 1e-3 * float(exact.norm())
    for mine, theirs in zip(streamed.states, tiled.states):
        for name in ("fast", "slow", "mixed", "k", "v", "u"):
            a, b = getattr(mine, name).float(), getattr(theirs, name).float()
            assert float((a - b).norm()) <= 0.01 * float(b.norm()), name


# fewer rows than the decode projections take, which read the norms ahead of the launches in front of them; few heads, so that a vector of
# logits is shorter than 16 bytes
@pytest.mark.gpu
@pytest.mark.parametrize("batch,length,d", [(1, 5, 512), (2, 60, 640), (1, 128, 512), (1, 200, 128)])
def test_vectors_that_are_not_fp32_are_copied_once_and_before_the_chain(batch, length, d):
    """The chain refuses to copy one once it has begun.  Norms and logits of values that BF16 holds: the same bits as in FP32."""
    torch.manual_seed(d)
    with torch.device("cuda"):
        model = WarpStateLM(config(d, 704, depth=6, cores=2)).eval().requires_grad_(False)
    vectors = [(core.norm1, "weight") for core in model.cores] + [(core.norm2, "weight") for core in model.cores]
    vectors += [(core, name) for core in model.cores for name in ("fast_decay_logit", "slow_decay_logit", "memory_mix_logit")]
    for owner, name in vectors:
        getattr(owner, name).data = (torch.randn_like(getattr(owner, name)) * 0.2 + 1).bfloat16().float()
    ids = torch.randint(0, 512, (batch, length), device="cuda")
    want = DecodeEngine(model).prefill(ids).clone()
    for owner, name in vectors:
        getattr(owner, name).data = getattr(owner, name).data.bfloat16()
    got = DecodeEngine(model).prefill(ids)
    gemm.check_device_errors()
    assert torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("which", [0, 1])
def test_a_modulation_of_another_device_is_refused(train, which):
    with torch.device("cuda"):
        core = WarpStateCore(config(256, 192)).requires_grad_(train)
        x, mod = torch.randn(1, 128, 256), [torch.zeros(256), torch.zeros(256)]
    mod[which] = mod[which].cpu()
    with pytest.raises(RuntimeError, match="device"), torch.autocast("cuda", dtype=torch.bfloat16):
        core(x, *mod)


# the first length past those that stream at every width, and the last that would; one sequence and several
@pytest.mark.gpu
@pytest.mark.parametrize("batch,length,d,ffn", [(1, 97, 640, 704), (1, 128, 1280, 4480), (8, 16, 512, 704), (1, 128, 1920, 1024)])
def test_past_96_tokens_only_the_widest_stream(monkeypatch, batch, length, d, ffn):
    """The products' own kernels: the same bits as launch by launch."""
    torch.manual_seed(length + d)
    with torch.device("cuda"):
        model = WarpStateLM(config(d, ffn, depth=4, cores=2)).eval().requires_grad_(False)
    ids = torch.randint(0, 512, (batch, length), device="cuda")
    together, apart = DecodeEngine(model), DecodeEngine(model)
    got = together.prefill(ids).clone()
    monkeypatch.setattr(fused, "cores_prefill_state", lambda *a: None)
    want = apart.prefill(ids)
    gemm.check_device_errors()
    assert torch.equal(got, want)
