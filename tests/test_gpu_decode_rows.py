"""The persistent decode step of a few rows (csrc/decode_rows.cu) gives the bits of the separate launches that it replaces: both widths, 1 to 8 rows (both
instances and the rows around their edge), contexts around a tile of 8 tokens, a page, a split and a CTA's part, padding rows, sectioned rotary positions, both
roundings."""
import pytest
import torch

from tests.test_gpu_decoder_stack import _layout

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
PAGE = 256
_STACKS = {}


def _stack(hidden, inter, layers, mrope, rounding):
    from nano_qwen3tts_vllm_b200.config import StackConfig
    from nano_qwen3tts_vllm_b200.models.qwen3_tts_share import DecoderStack, random_init_
    key = (hidden, inter, layers, mrope, rounding)
    if key not in _STACKS:
        _STACKS.clear()
        scaling = {"mrope_section": [24, 20, 20], "interleaved": True} if mrope else None
        cfg = StackConfig(hidden_size=hidden, intermediate_size=inter, num_hidden_layers=layers, num_attention_heads=16, num_key_value_heads=8,
                          head_dim=128, vocab_size=2048, rope_scaling=scaling)
        torch.set_default_dtype(BF16)
        try:
            with torch.device("cuda"):
                _STACKS[key] = DecoderStack(cfg, rounding)
        finally:
            torch.set_default_dtype(torch.float32)
        random_init_(_STACKS[key], 77)
    return _STACKS[key]


def _case(stack, b, max_len, seed, pad_rows=0, lens=None):
    """A run of the stack on fresh copies of the caches: run(rows kernel?, rows or None) -> (hidden, [(k, v)])."""
    from nano_qwen3tts_vllm_b200 import _native as nat
    from nano_qwen3tts_vllm_b200.utils.context import reset_context, set_context
    c = stack.config
    ctx, bt, slots, pos, npages, width = _layout(b, max_len, seed, pad_rows)
    if lens is not None:
        ctx = torch.tensor(lens, dtype=torch.int32, device="cuda")
        slots = (bt.gather(1, ((ctx - 1) // PAGE).long().view(b, 1)).view(-1) * PAGE + (ctx - 1) % PAGE).to(torch.int32)
        pos = (ctx.long() - 1).contiguous()
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    base = [(r(npages, PAGE, 8, 128).to(BF16), r(npages, PAGE, 8, 128).to(BF16)) for _ in stack.layers]
    x = (0.5 * r(b, c.hidden_size)).to(BF16)
    if stack.layers[0].self_attn.rotary_emb.modality is not None:
        pos = torch.stack([pos, pos // 2, pos // 3 + 1]).contiguous()
    ws = nat.fused_decode_attn_workspace(b, 16, 128, width * PAGE, "cuda")

    def run(rows, keep=None):
        sel = slice(None) if keep is None else keep
        caches = [(k.clone(), v.clone()) for k, v in base]
        for layer, (k, v) in zip(stack.layers, caches):
            a = layer.self_attn.attn
            a.k_cache, a.v_cache, a.fused_workspace = k, v, ws
        if rows and getattr(stack, "_rows_ws", None) is None:
            stack.bind_decode_rows()
        kept, stack._rows_ws = getattr(stack, "_rows_ws", None), getattr(stack, "_rows_ws", None) if rows else None
        set_context(False, slot_mapping=slots[sel].contiguous(), context_lens=ctx[sel].contiguous(), block_tables=bt[sel].contiguous(),
                    max_context_len=width * PAGE)
        try:
            assert stack._takes_rows(x[sel]) == rows
            before = x.clone()
            out = stack.run_layers(x[sel], pos[..., sel].contiguous())
            torch.cuda.synchronize()
            assert torch.equal(x, before)
        finally:
            stack._rows_ws = kept
            reset_context()
        nat.check_waits()
        return out, caches
    return run


def _same(run, live):
    (want, wc), (got, gc), (again, ac) = run(False), run(True), run(True)
    for (k1, v1), (k2, v2), (k3, v3) in zip(wc, gc, ac):
        assert torch.equal(k1, k2) and torch.equal(v1, v2) and torch.equal(k2, k3) and torch.equal(v2, v3)
    assert torch.equal(got[:live], want[:live]) and torch.equal(got, again)
    assert torch.isfinite(got).all()


@pytest.mark.parametrize("hidden,inter,layers,mrope,rounding", [(2048, 6144, 3, True, 0), (2048, 6144, 2, False, 1), (1024, 3072, 5, False, 0),
                                                               (1024, 3072, 3, True, 1)])
@pytest.mark.parametrize("b,max_len,pad", [(1, 1, 0), (1, 97, 0), (2, 33, 0), (2, 250, 1), (3, 257, 1), (5, 128, 0), (8, 300, 2), (8, 17, 0), (1, 1300, 0),
                                           (1, 4000, 0), (4, 2100, 0), (8, 1100, 1)])
def test_the_bits_of_separate_launches(hidden, inter, layers, mrope, rounding, b, max_len, pad):
    if hidden == 2048 and b > 4:
        b, pad = b - 4, min(pad, b - 5)                          # wider stacks leave more than 4 rows to the separate launches
    _same(_case(_stack(hidden, inter, layers, mrope, rounding), b, max_len, seed=b * 1000 + max_len, pad_rows=pad), b - pad)


@pytest.mark.parametrize("lens", [[255, 256, 257, 511], [512, 513, 1, 2], [7, 8, 9, 64], [1024, 1025, 1535, 1536]])
def test_contexts_around_tiles_splits_and_parts(lens):
    _same(_case(_stack(1024, 3072, 3, True, 1), 4, max(lens) + 8, seed=9, lens=lens), 4)


def test_replayed_from_a_graph():
    """Captured once with one workspace: every replay gives the eager result, and launches of other row counts between them do no harm.  All of them are the
    persistent step, with the results of the separate launches."""
    from nano_qwen3tts_vllm_b200 import _native as nat
    from nano_qwen3tts_vllm_b200.utils.context import reset_context, set_context
    stack = _stack(1024, 3072, 5, False, 0)
    ctx, bt, slots, pos, npages, width = _layout(8, 120, 3)
    for layer in stack.layers:
        a = layer.self_attn.attn
        a.k_cache, a.v_cache = (torch.randn(npages, PAGE, 8, 128, device="cuda").to(BF16) for _ in range(2))
    stack.bind_decode_rows()
    x = torch.randn(8, 1024, device="cuda").to(BF16)

    def step(n, rows=True):
        set_context(False, slot_mapping=slots[:n], context_lens=ctx[:n], block_tables=bt[:n], max_context_len=width * PAGE)
        assert stack._takes_rows(x[:n]) == rows
        return stack.run_layers(x[:n], pos[:n])
    try:
        kept, stack._rows_ws = stack._rows_ws, None
        for layer in stack.layers:
            layer.self_attn.attn.fused_workspace = nat.fused_decode_attn_workspace(8, 16, 128, width * PAGE, "cuda")
        separate = {n: step(n, False).clone() for n in (1, 2, 3, 8)}
        stack._rows_ws = kept
        eager = step(8).clone()
        assert torch.equal(eager, separate[8])
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = step(8)
        for n in (1, 3, 8, 2):
            assert torch.equal(step(n), separate[n])
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(out, eager)
    finally:
        reset_context()
