"""Grouped products on the tensor cores against 64-bit sums: group sizes, columns and inner sizes around the edges of the tiles,
scattered rows, every activation."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def nat():
    import nano_qwen3tts_vllm_b200._native as n
    n.lib()
    return n


def _groups(sizes, top, seed):
    """offsets and a random assignment of (token, choice) pairs to groups of these sizes."""
    n = sum(sizes)
    g = torch.Generator().manual_seed(seed)
    pair = torch.randperm(n, generator=g).to(torch.int32)
    off = torch.tensor([sum(sizes[:i]) for i in range(len(sizes) + 1)], dtype=torch.int32)
    return off.to(DEV), pair.to(DEV), n


def _close(got, ref, inner):
    """bf16 storage rounds to 2^-9 of the value (2^-8 allowed); the float sums of ``inner`` products err by at most inner * 2^-24 of
    their absolute sum, which is below sqrt(inner) * 6 here (operands of unit size, six sigma), and the activations used have
    slopes of at most about 2 |z| + 2."""
    err = (got.double() - ref).abs()
    assert bool((err <= ref.abs() * 2.0 ** -8 + inner * 2.0 ** -24 * 6 * inner ** 0.5 * (2 * ref.abs().sqrt() + 2)).all()), err.max().item()


@pytest.mark.parametrize("sizes", [(129, 0, 1, 127, 128), (600, 33), (1, 1, 1, 700), (40, 40, 40)])
@pytest.mark.parametrize("n,k", [(8, 8), (264, 200), (512, 64), (136, 72), (1032, 328)])
def test_group_column_and_inner_edges(nat, sizes, n, k):
    top, E = 2, len(sizes)
    off, pair, pairs = _groups(sizes, top, n + k)
    if pairs % top:
        sizes = sizes[:-1] + (sizes[-1] + 1,)
        off, pair, pairs = _groups(sizes, top, n + k)
    g = torch.Generator(device=DEV).manual_seed(k)
    r = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    tok, w = r(pairs // top, k), r(E, n, k)
    for act in (0, 1):
        c = torch.full((pairs, n), 7.0, device=DEV, dtype=torch.bfloat16)
        nat.grouped_gemm(tok, w, c, off, pair, pairs, top, in_by_token=True, out_by_pair=False, act=act)
        for e in range(E):
            rows = slice(off[e].item(), off[e + 1].item())
            ref = tok[(pair[rows] // top).long()].double() @ w[e].double().T
            _close(c[rows], ref.clamp(min=0) ** 2 if act else ref, k)
    y = r(pairs, k)
    c = torch.full((pairs, n), 7.0, device=DEV, dtype=torch.bfloat16)
    nat.grouped_gemm(y, w, c, off, pair, pairs, top, in_by_token=False, out_by_pair=True, act=0)
    for e in range(E):
        rows = slice(off[e].item(), off[e + 1].item())
        _close(c[pair[rows].long()], y[rows].double() @ w[e].double().T, k)
    assert nat.grouped_gemm_timeouts() == 0


@pytest.mark.parametrize("sizes", [(129, 0, 1, 128), (5, 3, 2), (400, 77)])         # the middle one: the decode-sized kernel
@pytest.mark.parametrize("ff,k", [(8, 64), (136, 200), (128, 8), (264, 136)])
def test_gated_activations(nat, sizes, ff, k):
    top, E = 1, len(sizes)
    off, pair, pairs = _groups(sizes, top, ff + k)
    g = torch.Generator(device=DEV).manual_seed(ff)
    r = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    h, w = r(pairs, k), (r(E, 2 * ff, k) * k ** -0.5).to(torch.bfloat16)
    got = {"silu": torch.empty(pairs, ff, device=DEV, dtype=torch.bfloat16), "clamped": torch.empty(pairs, ff, device=DEV, dtype=torch.bfloat16)}
    nat.grouped_gemm_silu(h, w, got["silu"], off, pair, pairs, top)
    nat.grouped_gemm_gated(h, w, got["clamped"], off, pair, pairs, top, 1.5)
    for e in range(E):
        rows = slice(off[e].item(), off[e + 1].item())
        gu = h[pair[rows].long()].double() @ w[e].double().T
        gate, up = gu[:, :ff], gu[:, ff:]
        _close(got["silu"][rows], torch.nn.functional.silu(gate) * up, k)
        gate, up = gate.clamp(max=1.5), up.clamp(-1.5, 1.5)
        _close(got["clamped"][rows], gate * torch.sigmoid(1.702 * gate) * (up + 1), k)
    nat.check_waits()


@pytest.mark.parametrize("k", [64, 72, 192, 256, 320])               # slices of K: 1, 2, 3, 4, 5, so the ring stands elsewhere at each tile
def test_several_tiles_per_cta(nat, k):
    """More than five tiles for every CTA of the persistent kernel: both accumulators in turn, the ring carried over tile borders, empty
    groups between full ones; scattered rows, consecutive rows and gated products."""
    sizes, top = (2600, 0, 1, 4100, 129, 0, 9000, 4170), 2
    E, n, ff = len(sizes), 1032, 520
    off, pair, pairs = _groups(sizes, top, k)
    blocks = sum((s + 127) // 128 for s in sizes)
    assert blocks * ((n + 255) // 256) > 5 * 148 and blocks * ((ff + 127) // 128) > 5 * 148
    g = torch.Generator(device=DEV).manual_seed(k)
    r = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    tok, w, y = r(pairs // top, k), r(E, n, k), r(pairs, k)
    wg = (r(E, 2 * ff, k) * k ** -0.5).to(torch.bfloat16)
    new = lambda cols: torch.full((pairs, cols), 7.0, device=DEV, dtype=torch.bfloat16)
    gathered, boxed, silu, clamped = new(n), new(n), new(ff), new(ff)
    nat.grouped_gemm(tok, w, gathered, off, pair, pairs, top, in_by_token=True, out_by_pair=False, act=1)
    nat.grouped_gemm(y, w, boxed, off, pair, pairs, top, in_by_token=False, out_by_pair=True, act=0)
    nat.grouped_gemm_silu(tok, wg, silu, off, pair, pairs, top)
    nat.grouped_gemm_gated(tok, wg, clamped, off, pair, pairs, top, 1.5)
    for e in range(E):
        rows = slice(off[e].item(), off[e + 1].item())
        if rows.start == rows.stop:
            continue
        x = tok[(pair[rows] // top).long()].double()
        _close(gathered[rows], (x @ w[e].double().T).clamp(min=0) ** 2, k)
        _close(boxed[pair[rows].long()], y[rows].double() @ w[e].double().T, k)
        gu = x @ wg[e].double().T
        gate, up = gu[:, :ff], gu[:, ff:]
        _close(silu[rows], torch.nn.functional.silu(gate) * up, k)
        gate, up = gate.clamp(max=1.5), up.clamp(-1.5, 1.5)
        _close(clamped[rows], gate * torch.sigmoid(1.702 * gate) * (up + 1), k)
    nat.check_waits()
    assert nat.grouped_gemm_timeouts() == 0


@pytest.mark.parametrize("sizes", [(129, 0, 1, 127, 128), (600, 33), (1, 1, 1, 700)])
@pytest.mark.parametrize("n,k", [(8, 192), (264, 200), (136, 712)])
@pytest.mark.parametrize("ff,kg", [(8, 768), (136, 776), (264, 840), (32, 72)])
def test_edges_at_the_inner_sizes_of_the_tensor_core_kernel(nat, sizes, n, k, ff, kg):
    """The same edges of rows and columns with K long enough (and gated rows of W few enough) for that kernel to be chosen."""
    top, E = 2, len(sizes)
    if sum(sizes) % top:
        sizes = sizes[:-1] + (sizes[-1] + 1,)
    off, pair, pairs = _groups(sizes, top, n + k)
    g = torch.Generator(device=DEV).manual_seed(k)
    r = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    tok, w, y, tg = r(pairs // top, k), r(E, n, k), r(pairs, k), r(pairs // top, kg)
    wg = (r(E, 2 * ff, kg) * kg ** -0.5).to(torch.bfloat16)
    new = lambda cols: torch.full((pairs, cols), 7.0, device=DEV, dtype=torch.bfloat16)
    gathered, boxed, silu, clamped = new(n), new(n), new(ff), new(ff)
    nat.grouped_gemm(tok, w, gathered, off, pair, pairs, top, in_by_token=True, out_by_pair=False, act=1)
    nat.grouped_gemm(y, w, boxed, off, pair, pairs, top, in_by_token=False, out_by_pair=True, act=0)
    nat.grouped_gemm_silu(tg, wg, silu, off, pair, pairs, top)
    nat.grouped_gemm_gated(tg, wg, clamped, off, pair, pairs, top, 1.5)
    for e in range(E):
        rows = slice(off[e].item(), off[e + 1].item())
        token = (pair[rows] // top).long()
        _close(gathered[rows], (tok[token].double() @ w[e].double().T).clamp(min=0) ** 2, k)
        _close(boxed[pair[rows].long()], y[rows].double() @ w[e].double().T, k)
        gu = tg[token].double() @ wg[e].double().T
        gate, up = gu[:, :ff], gu[:, ff:]
        _close(silu[rows], torch.nn.functional.silu(gate) * up, kg)
        gate, up = gate.clamp(max=1.5), up.clamp(-1.5, 1.5)
        _close(clamped[rows], gate * torch.sigmoid(1.702 * gate) * (up + 1), kg)
    nat.check_waits()


@pytest.mark.parametrize("rows", [12, 13, 16, 17, 24, 25])
@pytest.mark.parametrize("n,k", [(64, 64), (64, 184), (64, 192), (256, 648), (1032, 640), (520, 768)])
def test_both_sides_of_the_choice_of_kernel(nat, rows, n, k):
    """Rows an expert and inner sizes on either side of each line of the rule, gathered, in order and gated."""
    E, top, pairs = 6, 2, 6 * rows
    off, pair, _ = _groups((rows,) * E, top, rows)
    g = torch.Generator(device=DEV).manual_seed(n + k)
    r = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    tok, w, y = r(pairs // top, k), (r(E, n, k) * k ** -0.5).to(torch.bfloat16), r(pairs, k)
    a, b, c = (torch.empty(pairs, m, device=DEV, dtype=torch.bfloat16) for m in (n, n, n // 2))
    nat.grouped_gemm(tok, w, a, off, pair, pairs, top, in_by_token=True, out_by_pair=False, act=0)
    nat.grouped_gemm(y, w, b, off, pair, pairs, top, in_by_token=False, out_by_pair=True, act=0)
    nat.grouped_gemm_silu(tok, w, c, off, pair, pairs, top) if n % 16 == 0 else None
    for e in range(E):
        s = slice(e * rows, (e + 1) * rows)
        x = tok[(pair[s] // top).long()].double() @ w[e].double().T
        _close(a[s], x, k)
        _close(b[pair[s].long()], y[s].double() @ w[e].double().T, k)
        if n % 16 == 0:
            _close(c[s], torch.nn.functional.silu(x[:, :n // 2]) * x[:, n // 2:], k)


def test_not_finite_values_stay_in_their_rows(nat):
    """A NaN in one row of the input reaches that row's outputs only, activation included."""
    off, pair, pairs = _groups((150, 90), 1, 3)
    g = torch.Generator(device=DEV).manual_seed(1)
    h = torch.randn(pairs, 64, generator=g, device=DEV).to(torch.bfloat16)
    w = torch.randn(2, 32, 64, generator=g, device=DEV).to(torch.bfloat16)
    h[11, 5] = float("nan")
    c = torch.empty(pairs, 16, device=DEV, dtype=torch.bfloat16)
    nat.grouped_gemm_silu(h, w, c, off, pair, pairs, 1)
    bad = torch.isnan(c).all(1)
    nat.check_waits()
    assert bad.sum() == 1 and pair[bad.nonzero()[0, 0]] == 11 and torch.isfinite(c[~bad]).all()


def test_a_wait_that_ran_out_is_an_error(nat):
    """The next grouped product refuses once, and so does the check that an engine makes; the next call after that runs again."""
    off, pair, pairs = _groups((40, 20), 1, 3)
    h, w = torch.ones(pairs, 64, device=DEV, dtype=torch.bfloat16), torch.ones(2, 32, 64, device=DEV, dtype=torch.bfloat16)
    c = torch.empty(pairs, 32, device=DEV, dtype=torch.bfloat16)
    product = lambda: nat.grouped_gemm(h, w, c, off, pair, pairs, 1, in_by_token=True, out_by_pair=False, act=0)
    before = nat.grouped_gemm_timeouts()
    for consumer in (product, nat.check_waits):
        assert nat.lib().b2tts_grouped_gemm_lose_wait(None) == 0
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match="ran out"):
            consumer()
        nat.check_waits()
        product()
        assert bool((c == 64).all())
    assert nat.grouped_gemm_timeouts() == before + 2


def test_more_rows_of_weights_than_a_copy_can_name(nat):
    """2^31 rows of W and more are beyond a tensor map's coordinates and stay on the general kernel.  Two experts of 2^30 rows of which
    the second is not used (and not there); rows of W repeat every 2^20, so do the outputs, and gate and up rows are the same."""
    free, _ = torch.cuda.mem_get_info()
    rows, k, pairs, period = 1 << 30, 8, 25, 1 << 20
    if free < 60 << 30:
        pytest.skip("needs 45 GB")
    g = torch.Generator(device=DEV).manual_seed(1)
    block = torch.randn(period, k, generator=g, device=DEV).to(torch.bfloat16)
    w = torch.empty(rows, k, device=DEV, dtype=torch.bfloat16)
    w.view(-1, period, k).copy_(block)
    h = torch.randn(pairs, k, generator=g, device=DEV).to(torch.bfloat16)
    off, pair = torch.tensor([0, pairs, pairs], dtype=torch.int32, device=DEV), torch.arange(pairs, dtype=torch.int32, device=DEV)
    c = torch.empty(pairs, rows // 2, device=DEV, dtype=torch.bfloat16)
    rc = nat.lib().b2tts_grouped_gemm_silu(h.data_ptr(), k, w.data_ptr(), c.data_ptr(), rows // 2, off.data_ptr(), pair.data_ptr(), pairs, 2,
                                           rows // 2, k, 1, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    x = h.double() @ block.double().T
    _close(c[:, :period], torch.nn.functional.silu(x) * x, k)
    assert all(torch.equal(c[i].view(-1, period), c[i, :period].expand(rows // 2 // period, period)) for i in range(pairs))
