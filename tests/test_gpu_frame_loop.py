"""GPU parity of the device-resident frame loop: greedy (top_k = 1) codec
frames of DeviceFrameLoop / StepApiFrameLoop against the CPU oracle's run_frames on the
same random-init weights and prompts (greedy codec-token sequences are identical).

A greedy sequence can only be required to be identical while the oracle's own arg-max is decided by more
than the arithmetic noise between two correct bf16 pipelines: where the oracle's top-2 logit margin is below
one bf16 ulp of the top logit the choice is a coin flip of GEMM accumulation order (fp32 sums are formed in a
different order on the tensor cores than in the CPU's blocked GEMM).  The test therefore demands identity up to the
first frame whose oracle margin is under that ulp, and demands that any divergence sits exactly on such a
near-tie."""
import pytest
import torch

from oracle import model as OM
from oracle import ops as O
from tests.test_gpu_models import small_model_config, small_weights

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
NFRAMES = 24
B = 4


def _prompts(td, b):
    g = torch.Generator().manual_seed(1000)
    prompts = [(torch.randn(n, td.hidden_size, generator=g) * 0.05).to(BF16) for n in ([9, 14, 5, 11] * 4)[:b]]
    pad = (torch.randn(1, td.hidden_size, generator=torch.Generator().manual_seed(999)) * 0.05).to(BF16)
    return prompts, pad


@pytest.fixture(scope="module")
def setup():
    from nano_qwen3tts_vllm_b200.llm import PredictorLLM, TalkerLLM
    td, pd, tw, pw = small_weights()
    prompts, pad = _prompts(td, B)
    margins = []

    def greedy(logits, temps):
        top2 = logits.float().topk(2, dim=-1).values
        margins.append((top2[:, 0] - top2[:, 1], top2[:, 0]))
        return O.topk_sample(logits, temps, torch.ones(logits.shape), top_k=1)

    ot = OM.Talker(td, tw, B * 2)
    op = OM.Predictor(pd, pw, B, td.hidden_size)
    want = torch.tensor(OM.run_frames(ot, op, prompts, NFRAMES, pad, greedy).frames)      # [frames, B, 16]
    mc = small_model_config()
    kw = dict(num_kvcache_blocks=4 * B, max_num_seqs=max(B, 2), max_model_len=512, enforce_eager=True)
    talker = TalkerLLM(mc, state_dict=tw, **kw)
    predictor = PredictorLLM(mc, state_dict=pw, **kw)
    yield dict(td=td, pd=pd, prompts=prompts, pad=pad, want=want, margins=margins, talker=talker, predictor=predictor)
    talker.exit()
    predictor.exit()


def _margin_ulp(margins, f, c, s, ncb=16):
    m, top = margins[ncb * f + c]
    ulp = 2.0 ** (torch.tensor(float(top[s])).abs().log2().floor().item() - 7)
    return float(m[s]) / ulp


def _check_against_oracle(got, want, margins, min_exact=0):
    """Free-running comparison: identity per stream up to its first near-tie; every divergence must sit on a
    near-tie of the ORACLE's logits (<= 2 bf16 ulp between its two best logits; exact ties - margin 0 - are common
    with random-init weights).  Prints the first divergence per stream.  What happens AFTER a divergence is checked
    by the teacher-forced tests, which compare every decision on the oracle's own history."""
    assert got.shape == want.shape
    nframes, b, ncb = want.shape
    exact, report = 0, []
    for s in range(b):
        ne = (got[:, s] != want[:, s]).nonzero()
        if ne.numel() == 0:
            exact += 1
            report.append((s, nframes, None))
            continue
        f, c = ne[0].tolist()
        mu = _margin_ulp(margins, f, c, s, ncb)
        report.append((s, f, round(mu, 2)))
        assert mu <= 2, (f"stream {s} diverges at frame {f} codebook {c} where the oracle's top-2 margin is "
                         f"{mu:.2f} bf16 ulp")
    print("free-running: (stream, identical frames, margin ulp at first divergence) =", report)
    assert exact >= min_exact, f"only {exact} of {b} streams identical over {nframes} frames: {report}"
    return exact


def _check_teacher_forced(sampled, want, margins, max_flip_frac=0.02):
    """Every decision taken on the oracle's history: choices may differ only where the oracle's own top-2 margin
    is <= 2 bf16 ulp, and only rarely."""
    nframes, b, ncb = want.shape
    diff = (sampled != want).nonzero().tolist()
    worst = 0.0
    for f, s, c in diff:
        mu = _margin_ulp(margins, f, c, s, ncb)
        worst = max(worst, mu)
        assert mu <= 2, f"teacher-forced: stream {s} frame {f} codebook {c} differs at a decisive margin ({mu:.2f} ulp)"
    frac = len(diff) / want.numel()
    print(f"teacher-forced: {len(diff)} of {want.numel()} decisions differ (worst margin {worst:.2f} ulp)")
    assert frac <= max_flip_frac, f"{frac:.3%} of the decisions differ"


def test_device_frame_loop_greedy_vs_oracle(setup):
    from nano_qwen3tts_vllm_b200.engine.frame_loop import DeviceFrameLoop
    t, p = setup["talker"].model_runner, setup["predictor"].model_runner
    t.kv_cache.zero_(); p.kv_cache.zero_()
    loop = DeviceFrameLoop(t, p, B, NFRAMES, 16, top_k=1, scatter_pages=True)
    loop.unit_noise = True
    loop.start([x.cuda() for x in setup["prompts"]], setup["pad"].cuda())
    loop.capture()
    loop.run(NFRAMES)
    got = loop.result()
    _check_against_oracle(got, setup["want"], setup["margins"])
    with pytest.raises(RuntimeError, match="frame budget"):          # frames buffer / block tables are sized for NFRAMES
        loop.step()


def test_device_frame_loop_teacher_forced(setup):
    """All NFRAMES x 16 x B decisions compared on the oracle's own history (no drift can hide a later error)."""
    from nano_qwen3tts_vllm_b200.engine.frame_loop import DeviceFrameLoop
    t, p = setup["talker"].model_runner, setup["predictor"].model_runner
    t.kv_cache.zero_(); p.kv_cache.zero_()
    loop = DeviceFrameLoop(t, p, B, NFRAMES, 16, top_k=1, scatter_pages=True)
    loop.unit_noise = True
    loop.force(setup["want"])
    loop.start([x.cuda() for x in setup["prompts"]], setup["pad"].cuda())
    loop.capture()
    loop.run(NFRAMES)
    assert torch.equal(loop.result(), setup["want"])
    sampled = loop.sampled[:NFRAMES].permute(0, 2, 1).cpu()
    _check_teacher_forced(sampled, setup["want"], setup["margins"])


def test_eos_and_trailing_text_vs_oracle(setup):
    """interface.py:1233-1239 (code0 == codec EOS ends the stream before its frame) and :1282-1285 (per-stream
    trailing_text_hiddens[:, step], then tts_pad_embed) on the device, against the oracle's run_frames with the same
    EOS id and trailing rows.  Teacher-forced with the oracle's codes so that every decision is compared: the frame
    COUNT of every stream must equal the oracle's, and the sampler's choices on the oracle's history must agree
    except on rare near-ties (a wrong trailing row or a missed EOS makes them disagree everywhere)."""
    from nano_qwen3tts_vllm_b200.engine.frame_loop import DeviceFrameLoop
    td, prompts, pad = setup["td"], setup["prompts"], setup["pad"]
    g = torch.Generator().manual_seed(4321)
    trailing = [None if n == 0 else (torch.randn(n, td.hidden_size, generator=g) * 0.05).to(BF16) for n in (0, 3, 7, 2)]
    _, _, tw, pw = small_weights()

    def greedy(logits, temps):
        return O.topk_sample(logits, temps, torch.ones(logits.shape), top_k=1)

    def oracle_run(eos):
        ot, op = OM.Talker(td, tw, B * 2), OM.Predictor(setup["pd"], pw, B, td.hidden_size)
        return OM.run_frames(ot, op, prompts, NFRAMES, pad, greedy, trailing=trailing, codec_eos=eos).per_stream
    free = oracle_run(None)
    eos = free[1][6][0]                       # stream 1 stops before its 7th frame (others too if they emit it earlier)
    want = oracle_run(eos)
    counts = [len(w) for w in want]
    assert counts[1] <= 6 and max(counts) > 6
    forced = torch.zeros(NFRAMES, B, 16, dtype=torch.int64)
    for s_, w in enumerate(want):
        if w:
            forced[:len(w), s_] = torch.tensor(w)
        if len(w) < NFRAMES:
            forced[len(w), s_, 0] = eos       # the code0 that ends the stream (sampled at the end of its last frame)
    t, p = setup["talker"].model_runner, setup["predictor"].model_runner
    t.kv_cache.zero_(); p.kv_cache.zero_()
    loop = DeviceFrameLoop(t, p, B, NFRAMES, 16, top_k=1, ignore_eos=False, codec_eos=eos, max_trailing=7)
    loop.unit_noise = True
    loop.force(forced)
    loop.start([x.cuda() for x in prompts], pad.cuda(), trailing=[None if x is None else x.cuda() for x in trailing])
    loop.capture()
    loop.run(NFRAMES)
    assert loop.frame_counts() == counts, f"frames per stream {loop.frame_counts()}, the oracle stops after {counts}"
    got = loop.result_per_stream()
    sampled = loop.sampled[:NFRAMES].permute(0, 2, 1).cpu()          # [F, B, 16]
    total = flips = 0
    for s_, w in enumerate(want):
        assert torch.equal(got[s_], torch.tensor(w, dtype=torch.int64).view(-1, 16))
        n = len(w)
        if n:
            d = sampled[:n, s_] != torch.tensor(w)
            total += d.numel(); flips += int(d.sum())
        if n < NFRAMES:                                               # the EOS itself must be the sampler's choice
            total += 1; flips += int(sampled[n, s_, 0] != eos)
    assert flips <= max(2, 0.03 * total), f"{flips} of {total} decisions differ from the oracle (EOS {eos})"


def test_graph_replay_equals_eager_frames(setup):
    """The captured frame graph and the same frame launched eagerly produce the same codes."""
    from nano_qwen3tts_vllm_b200.engine.frame_loop import DeviceFrameLoop
    t, p = setup["talker"].model_runner, setup["predictor"].model_runner
    outs = []
    for capture in (False, True):
        t.kv_cache.zero_(); p.kv_cache.zero_()
        loop = DeviceFrameLoop(t, p, B, 6, 16, top_k=1, scatter_pages=False)
        loop.unit_noise = True       # exact bf16 logit ties are broken by the sampler's noise otherwise
        loop.start([x.cuda() for x in setup["prompts"]], setup["pad"].cuda())
        if capture:
            loop.capture()
        loop.run(6)
        outs.append(loop.result())
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("batched", [True, False])
def test_step_api_frame_loop_greedy_vs_oracle(setup, batched):
    """The reference's per-frame protocol with host buffers (StepApiFrameLoop) gives the oracle's frames: one
    add_request per stream and one engine step per codebook (the reference's call pattern), and the batched form
    (one add_requests per engine per frame, the predictor's whole burst as one captured graph)."""
    from nano_qwen3tts_vllm_b200.engine.frame_loop import StepApiFrameLoop
    talker, predictor = setup["talker"], setup["predictor"]
    if batched:                 # graphs on: decode graphs + the predictor's burst graphs (the fixture's engines are eager)
        from nano_qwen3tts_vllm_b200.llm import PredictorLLM, TalkerLLM
        _, _, tw, pw = small_weights()
        kw = dict(num_kvcache_blocks=4 * B, max_num_seqs=max(B, 2), max_model_len=512, graph_batch_sizes=[B])
        talker, predictor = TalkerLLM(small_model_config(), state_dict=tw, **kw), PredictorLLM(small_model_config(), state_dict=pw, **kw)
    talker.model_runner.kv_cache.zero_(); predictor.model_runner.kv_cache.zero_()
    old = talker.model_runner.top_k, predictor.model_runner.top_k, predictor.burst
    talker.model_runner.top_k = predictor.model_runner.top_k = 1
    predictor.burst = batched
    try:
        api = StepApiFrameLoop(talker, predictor, setup["pad"], batched=batched)
        api.add_streams([x.unsqueeze(0).pin_memory() for x in setup["prompts"]])
        for _ in range(NFRAMES):
            api.step_frame()
        got = torch.tensor([api.frames[f"s{i}"] for i in range(B)]).permute(1, 0, 2)
        api.close()
    finally:
        talker.model_runner.top_k, predictor.model_runner.top_k, predictor.burst = old
    if batched:
        assert predictor.model_runner.burst_top_k == 1           # the burst graphs were re-captured for greedy and used
        talker.exit(); predictor.exit()
    _check_against_oracle(got, setup["want"], setup["margins"])


def test_step_api_device_glue_and_pipelining_equal_host_glue(setup):
    """The batched step-API loop (a) packs the predictor input and sums the next talker input from the engines' DEVICE
    results (hooks queued before each step's synchronisation) and (b) queues the next engine's step before waiting for
    the previous one (step_launch / step_collect).  Starting every piece of glue from the host values, in the
    reference's order of operations, must give the same frames - and, without the run-ahead, the same pinned buffers."""
    from nano_qwen3tts_vllm_b200.engine.frame_loop import StepApiFrameLoop
    from nano_qwen3tts_vllm_b200.llm import PredictorLLM, TalkerLLM
    _, _, tw, pw = small_weights()
    kw = dict(num_kvcache_blocks=4 * B, max_num_seqs=max(B, 2), max_model_len=512, graph_batch_sizes=[B])
    got = []
    for glue, piped in ((True, True), (True, False), (False, False)):
        talker, predictor = TalkerLLM(small_model_config(), state_dict=tw, **kw), PredictorLLM(small_model_config(), state_dict=pw, **kw)
        talker.model_runner.top_k = predictor.model_runner.top_k = 1
        torch.manual_seed(4321)                     # exact ties at the top are kept by top-k and decided by the noise
        api = StepApiFrameLoop(talker, predictor, setup["pad"], batched=True, device_glue=glue, pipelined=piped)
        assert api.pipelined == piped
        api.add_streams([x.unsqueeze(0).pin_memory() for x in setup["prompts"]])
        for _ in range(8):
            assert api.step_frame() == B
        torch.cuda.synchronize()
        got.append((torch.tensor([api.frames[f"s{i}"] for i in range(B)]), api._pins["pred_in"].clone(), api._pins["next_in"].clone(),
                    api.h2d_bytes, api.d2h_bytes))
        api.close()
        assert getattr(talker.model_runner, "post_sample_hook", None) is None and getattr(predictor, "burst_hook", None) is None
        talker.exit(); predictor.exit()
    assert torch.equal(got[0][0], got[2][0]) and torch.equal(got[1][0], got[2][0])
    assert torch.equal(got[1][1], got[2][1]) and torch.equal(got[1][2], got[2][2])
    assert all(g[3] > 0 and g[4] > 0 for g in got)


def test_step_api_pipelined_retires_streams_on_codec_eos(setup):
    """ignore_eos=False with the run-ahead: a stream whose code0 is the codec EOS leaves without a frame although its
    predictor burst was already queued; the survivors' frames equal the sequential loop's."""
    from nano_qwen3tts_vllm_b200.engine.frame_loop import StepApiFrameLoop
    from nano_qwen3tts_vllm_b200.llm import PredictorLLM, TalkerLLM
    _, _, tw, pw = small_weights()
    kw = dict(num_kvcache_blocks=4 * B, max_num_seqs=max(B, 2), max_model_len=512, graph_batch_sizes=[1, 2, B])
    res, eos = [], -1
    for piped in (None, True, False):           # None: a first run that ignores EOS, to pick a code0 that really comes up
        talker, predictor = TalkerLLM(small_model_config(), state_dict=tw, **kw), PredictorLLM(small_model_config(), state_dict=pw, **kw)
        talker.model_runner.top_k = predictor.model_runner.top_k = 1
        torch.manual_seed(99)
        api = StepApiFrameLoop(talker, predictor, setup["pad"], ignore_eos=piped is None, codec_eos=eos, batched=True,
                               pipelined=bool(piped))
        api.add_streams([x.unsqueeze(0).pin_memory() for x in setup["prompts"]])
        counts = [api.step_frame() for _ in range(6)]
        torch.cuda.synchronize()
        if piped is None:
            eos = api.frames["s1"][2][0]        # stream 1 retires in frame 2 (any other stream emitting it earlier too)
        else:
            res.append((counts, {k: list(v) for k, v in api.frames.items()}, list(api.active)))
        api.close()
        talker.exit(); predictor.exit()
    assert res[0] == res[1]
    assert min(res[0][0]) < B, "the chosen EOS code never came up: the test retired no stream"
    for rid, fr in res[0][1].items():
        assert all(row[0] != eos for row in fr)
