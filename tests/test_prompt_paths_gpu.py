"""Prompt kernels that a rule on sizes and types chooses, against the general kernels that take every size, over the forms the rule lets in."""
import pytest
import torch

from tests.test_kernels_gpu import DEV, make_meta, ops          # noqa: F401  (ops: fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 300, 2200), (33, 131, 2085), (70, 2560, 4096), (129, 64, 130), (1030, 96, 2048), (17, 40, 16)])
def test_gemm_f32_tiles_give_the_same_bits(ops, M, N, K):       # noqa: F811
    """K cut into segments (K >= 2,048) or not, more rows than one pass over the workspace takes, remainders of every tile."""
    g = torch.Generator().manual_seed(M + N)
    x = torch.randn(M, K, generator=g).to(DEV)
    w = torch.randn(N, K, generator=g).to(DEV)
    want = x.double() @ w.double().T
    got = ops.linear(x, w)
    # a sum of n terms in float32 is off by a few eps sqrt(n) of the terms' norm: K <= 4,096, eps = 6e-8
    assert ((got.double() - want).norm() / want.norm()).item() < 4e-6
    for tile in range(5):
        out = torch.empty_like(got)
        ops._gemm_f32(x, K, w, out, N, M, N, K, tile)
        assert torch.equal(out, got), tile
    assert torch.equal(ops.linear(x[:1], w), got[:1])


@pytest.mark.parametrize("M,N,K", [(1, 2048, 512), (32, 1030, 1020), (33, 128, 8192), (65, 2500, 700), (129, 4096, 1100), (257, 300, 4000), (1030, 1100, 964)])
def test_gemm_f32_on_tensor_cores(ops, M, N, K):                # noqa: F811
    """Products cut into bfloat16 parts: remainders of a tile's rows of W, tokens and 64 of K, one segment of K and several, strided rows, every tile, and
    rows that bfloat16 parts cannot hold (infinities, NaN, the ends of float32's range), which must not touch any other row."""
    g = torch.Generator().manual_seed(M + N)
    x = torch.randn(M, K + 3, generator=g).to(DEV)[:, :K]
    w = torch.randn(N, K, generator=g).to(DEV)
    want = x.double() @ w.double().T
    got = ops.linear(x, w)
    # K / 64 sums are added up in float32, rounded to nearest (half of 2^-23 of the sum so far), behind sums of 64 cut off after 2^-23
    assert ((got.double() - want).norm() / want.norm()).item() < 6e-8 * (K / 64) ** 0.5 + 6e-8
    for tile in range(5):
        out = torch.empty_like(got)
        ops._gemm_f32(x, x.stride(0), w, out, N, M, N, K, tile)
        assert torch.equal(out, got), tile
    assert torch.equal(ops.linear(x[-1:], w), got[-1:])
    x, w = x.contiguous(), w.clone()
    rows = {0: lambda r: r.fill_(0), M // 2: lambda r: r.mul_(1e-30), M // 3: lambda r: r[7:8].fill_(float("inf")), M // 4: lambda r: r[K - 1:].fill_(float("nan")), M - 1: lambda r: r[3:4].fill_(1e36)}
    for m, change in rows.items():
        change(x[m])
    w[N - 1, 5], w[17, K - 2], w[40] = float("-inf"), 1e30, w[40] * 1e-28
    got2, want2 = ops.linear(x, w), x.double() @ w.double().T
    plain_rows = [m for m in range(M) if m not in rows]
    plain_cols = [n for n in range(N) if n not in (N - 1, 17, 40)]
    assert torch.equal(got2[plain_rows][:, plain_cols], got[plain_rows][:, plain_cols])
    assert torch.equal(got2.isnan(), want2.isnan()) and torch.equal(got2.isinf(), want2.isinf())
    for m in range(M):
        ok = want2[m].isfinite()
        if ok.any() and (M < 100 or m in rows):
            size = x[m].double().norm() * w[ok].double().norm(dim=1)        # what a float32 sum's error goes with
            assert ((got2[m][ok].double() - want2[m][ok]).abs() <= 2e-6 * size + 1e-37).all(), m


@pytest.mark.parametrize("M,N,K", [(652, 896, 4100), (700, 896, 4160), (768, 2048, 4100), (1030, 1152, 4132)])
def test_gemm_f32_whose_last_segment_is_short(ops, M, N, K):    # noqa: F811
    """K whose last 512th would be one or two stages, and blocks with several such items in a row: rows of infinities, NaN and 1e30 in every other tile, in the
    last segment's columns, are handed from warp to warp as fast as it gets."""
    g = torch.Generator().manual_seed(M + K)
    x, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    plain = ops.linear(x, w)
    odd = {n: v for n, v in zip(range(5, N, 256), [float("nan"), float("inf"), 1e30] * N)}
    for n, v in odd.items():
        w[n, K - 1] = v
    rest = [n for n in range(N) if n not in odd]
    for _ in range(5):
        got = ops.linear(x, w)
        ops.check_errors()
        want = x.double() @ w.double().T
        assert torch.equal(got[:, rest], plain[:, rest])
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
        big = [n for n, v in odd.items() if v == 1e30]
        if big:                                                  # the sums that a float32 product of 1e30 is added to are lost beside it
            assert ((got[:, big].double() - want[:, big]).abs() <= 2e-6 * x.double().norm(dim=1, keepdim=True) * 1e30).all()


FORMS = ["causal", "window", "blocks_sink", "learned_sink_bias", "slopes", "slopes_bias_window", "cap_keep_gate", "window_keep_narrow"]


def form_arguments(form, H, D, T, dtype):
    g = torch.Generator().manual_seed(5)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)         # noqa: E731
    base = dict(block_size=None, window=None, sink=False)
    return {"causal": base, "window": dict(base, window=70), "blocks_sink": dict(base, block_size=96, sink=True),
            "learned_sink_bias": dict(base, sink=True, sink_values=r(H), distance_bias=r(41, H)),
            "slopes": dict(base, distance_slopes=r(H).abs() * 0.1),
            "slopes_bias_window": dict(base, window=100, distance_slopes=r(H).abs() * 0.1, distance_bias=r(130, H)),
            "cap_keep_gate": dict(base, window=77, softcap=3.0, keep_first=5, gate=r(T, H * D).to(dtype)),
            "window_keep_narrow": dict(base, window=20, keep_first=130)}[form]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,KV,D,page", [(4, 2, 128, 16), (3, 1, 64, 8), (2, 2, 128, 24)])
@pytest.mark.parametrize("form", FORMS)
def test_prompt_attention_forms(ops, dtype, H, KV, D, page, form):      # noqa: F811
    """Portions that start at 0 and behind earlier keys, of one more than a tile's rows, of an odd few, and beside a decoded token."""
    segs = [(0, 129), (200, 65), (31, 3), (0, 300), (77, 1)]
    meta, T = make_meta(page, segs, 120, 3, indirect=True), sum(n for _, n in segs)
    g = torch.Generator().manual_seed(1)
    q = torch.randn(T, (H + 1) * D, generator=g).to(dtype).to(DEV)[:, :H * D]           # rows of a wider tensor
    k, v = (torch.randn(121, KV, page, D, generator=g).to(dtype).to(DEV) for _ in range(2))
    for i, (pos0, n) in enumerate(segs[:4]):                    # what a page holds behind a prompt's last key must not matter
        last = pos0 + n - 1
        page_id = meta.block_table[meta.rows[i], last // page].long()
        k[page_id, :, last % page + 1:], v[page_id, :, last % page + 1:] = float("nan"), float("inf")
    args = form_arguments(form, H, D, T, dtype)
    got = ops.masked_attention(q, k, v, meta, H, KV, D, D, D ** -0.5, **args)
    ops.check_errors()
    saved, ops.fast_attention = ops.fast_attention, False
    try:
        want = ops.masked_attention(q, k, v, meta, H, KV, D, D, D ** -0.5, **args)
    finally:
        ops.fast_attention = saved
    # float32: sums of up to 365 products in another order.  bfloat16: the output's own rounding, half of 2^-8 of the value, may fall differently
    err, limit = (got.float() - want.float()).abs().max().item(), want.float().abs().max().item()
    assert err < (4e-6 if dtype == torch.float32 else 2 ** -8) * limit, (form, err / limit)


@pytest.mark.parametrize("H,KV,D,page", [(4, 2, 128, 16), (3, 1, 64, 8)])
@pytest.mark.parametrize("form", FORMS)
def test_prompt_attention_forms_on_tcgen05(ops, monkeypatch, H, KV, D, page, form):      # noqa: F811
    """The same portions on the kernel that steps of more keys or tokens take."""
    monkeypatch.setattr(ops, "SPLIT_TC_MASKED", (0, 0))
    test_prompt_attention_forms(ops, torch.bfloat16, H, KV, D, page, form)


@pytest.mark.parametrize("behind", [0, 1300])
@pytest.mark.parametrize("n", [2, 64, 65, 128, 200])
def test_values_behind_the_last_key_do_not_count(ops, n, behind):       # noqa: F811
    """Plain tcgen05 attention (Qwen3): a last tile of keys that is whole or not, one tile or many; what its pages hold behind the last key is no number."""
    H, KV, D, page, segs = 4, 2, 128, 16, [(behind, n), (behind + 5, n)]
    meta, g = make_meta(page, segs, 220, 8), torch.Generator().manual_seed(n)
    q = torch.randn(2 * n, H * D, generator=g).to(torch.bfloat16).to(DEV)
    k, v = (torch.randn(221, KV, page, D, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    want = ops.paged_attention(q, k, v, meta, H, KV, D, D ** -0.5, None)
    for i, (pos0, m) in enumerate(segs):
        last = pos0 + m - 1
        at = meta.block_table[i, last // page].long()
        k[at, :, last % page + 1:], v[at, :, last % page + 1:] = float("nan"), float("inf")
    k[0], v[0] = float("nan"), float("inf")                      # the null page, which the loads of a tile's missing pages read
    got = ops.paged_attention(q, k, v, meta, H, KV, D, D ** -0.5, None)
    ops.check_errors()
    assert got.isfinite().all() and torch.equal(got, want)


@pytest.mark.parametrize("D,page", [(128, 16), (64, 24)])
@pytest.mark.parametrize("form", ["plain", "causal", "window", "blocks_sink", "cap_keep_gate", "window_keep_narrow"])
def test_float32_prompt_attention_reads_visible_keys_only(ops, D, page, form):      # noqa: F811
    """A key or value that is no number is met by the rows that see it and by no other, although their tiles of keys hold it as well."""
    H, KV, segs, at = 2, 1, [(40, 300), (0, 70)], 133            # key 133 of the first request, which feeds the positions 40 .. 339
    T = sum(n for _, n in segs)
    meta, g = make_meta(page, segs, 60, 4), torch.Generator().manual_seed(2)
    q = torch.randn(T, H * D, generator=g).to(DEV)
    k, v = (torch.randn(61, KV, page, D, generator=g).to(DEV) for _ in range(2))
    args = None if form == "plain" else form_arguments(form, H, D, T, torch.float32)

    def call(k, v):
        return ops.paged_attention(q, k, v, meta, H, KV, D, D ** -0.5, None) if args is None else ops.masked_attention(q, k, v, meta, H, KV, D, D, D ** -0.5, **args)

    want, bad_k, bad_v, place = call(k, v), k.clone(), v.clone(), (meta.block_table[0, at // page].long(), 0, at % page)
    bad_v[place], bad_k[place] = float("inf"), float("nan")
    pos = torch.arange(40, 340)
    mask = args or {}
    lo = torch.zeros_like(pos) if not mask.get("block_size") else pos // mask["block_size"] * mask["block_size"]
    lo = torch.maximum(lo, pos - mask["window"] + 1) if mask.get("window") else lo
    sees = (pos >= at) & ((lo <= at) | (at < mask.get("keep_first", 0)))
    sees = torch.cat([sees, torch.zeros(70, dtype=torch.bool)]).to(DEV)
    assert sees.any() and not sees.all()
    for got in (call(k, bad_v), call(bad_k, v)):
        assert torch.equal(got[~sees], want[~sees]), form
        assert not got[sees].isfinite().any(), form


@pytest.mark.parametrize("D,page", [(128, 16), (64, 24)])
@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("form", ["plain"] + FORMS)
def test_float32_decoded_tokens(ops, form, group, D, page):     # noqa: F811
    """Eight keys at a time over the warps of a block, one piece of the keys and several: against the general kernel (which takes rows that do not
    start on 16 bytes), with pages that hold no numbers behind the last key."""
    KV, lens = 2, (1, 7, 33, 256, 1000, 65)
    H, T = KV * group, len(lens)
    meta, g = make_meta(page, [(n - 1, 1) for n in lens], 110, group + D, indirect=True), torch.Generator().manual_seed(group)
    q = torch.randn(T, H * D + 1, generator=g).to(DEV)
    k, v = (torch.randn(111, KV, page, D, generator=g).to(DEV) for _ in range(2))
    for i, n in enumerate(lens):
        at = meta.block_table[meta.table_rows[i], (n - 1) // page].long()
        k[at, :, (n - 1) % page + 1:], v[at, :, (n - 1) % page + 1:] = float("nan"), float("inf")
    args = None if form == "plain" else form_arguments(form, H, D, T, torch.float32)

    def call(q):
        return ops.paged_attention(q, k, v, meta, H, KV, D, D ** -0.5, None) if args is None else ops.masked_attention(q, k, v, meta, H, KV, D, D, D ** -0.5, **args)

    want = call(q[:, :H * D])
    try:
        for splits in (None, 1, 5):
            ops.force_splits = splits
            # float32 sums of up to 1,000 weights and 128 products in another order
            assert rows_error(call(q[:, :H * D].contiguous()), want) < 2e-6, (form, splits)
    finally:
        ops.force_splits = None


class Entries:
    """A step's entries as the recurrences see them."""

    def __init__(self, lens):
        q = [0]
        for n in lens:
            q.append(q[-1] + n)
        self.num_segs = len(lens)
        self.seg_q_start = torch.tensor(q, dtype=torch.int32, device=DEV)
        self.seg_slot = torch.arange(len(lens), 0, -1, dtype=torch.int32, device=DEV)


def rows_error(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


@pytest.mark.parametrize("lens", [(9, 1, 8, 120), (129,), (7, 63, 58), (1, 1, 16, 1, 111)])
@pytest.mark.parametrize("H,KV,D,V", [(4, 2, 128, 48), (3, 3, 64, 32), (5, 1, 128, 128)])
def test_recurrences_eight_tokens_at_a_time(ops, lens, H, KV, D, V):        # noqa: F811
    """The delta rule with channel decays and the constant decay against their token-by-token kernels: whole octets, remainders, single tokens
    beside prompts, decays down to 0, states that start non-zero, slots out of order."""
    T, batch, g = sum(lens), Entries(lens), torch.Generator().manual_seed(sum(lens) + D)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)         # noqa: E731
    C = 2 * KV * D + H * V
    prep = torch.zeros(T, (C + H * D + H + 3) // 4 * 4, device=DEV)
    qk = r(T, 2 * KV, D)
    prep[:, :2 * KV * D] = (qk / qk.norm(dim=-1, keepdim=True)).reshape(T, -1)
    prep[:, 2 * KV * D:C] = r(T, H * V)
    decay = torch.rand(T, H * D, generator=g).to(DEV) ** 0.2
    decay[:, ::7], decay[:, 1::7] = 1.0, 0.0
    prep[:, C:C + H * D] = decay
    prep[:, C + H * D:C + H * D + H] = torch.rand(T, H, generator=g).to(DEV)
    state = r(len(lens) + 1, H * D * V + 6)
    p = r(T, 2 * H * D + H * V + 8).to(torch.bfloat16)
    batch.positions = torch.arange(T, dtype=torch.int32, device=DEV)
    freq = torch.rand(D // 4, generator=g).to(DEV)
    constant = torch.tensor([1.0 - 2.0 ** -(1 + 2 * h) for h in range(H)], device=DEV)
    runs = {"delta": lambda s: ops.delta_scan(prep, H, KV, D, V, s, batch), "constant": lambda s: ops.lightning_scan(p, H, D, V, constant, s, batch),
            "rotated": lambda s: ops.retention_scan(p, H, D, V, freq, D ** -0.5, constant, s, batch)}
    for name, run in runs.items():
        a, b = state.clone(), state.clone()
        taken = ops._takes_octets
        assert taken(prep, batch, D, V, a)
        for delta in (0, 1):
            assert ops.lib.mi_octet_floats(T, len(lens), H, D, V, delta) == ops._octet_scratch(T, batch, H, D, V, delta).numel()
        got = run(a)
        ops._takes_octets = lambda *args: False
        try:
            want = run(b)
        finally:
            del ops._takes_octets
        ops.check_errors()
        # two float32 orders of sums over up to 129 tokens and 128 rows
        assert rows_error(got, want) < 3e-6 and rows_error(a, b) < 3e-6, name
        assert torch.equal(a[:, H * D * V:], state[:, H * D * V:]) and torch.equal(a[0], state[0])


def chunk_inputs(lens, H, V, seed):
    T, D, g = sum(lens), 128, torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)         # noqa: E731
    batch = Entries(lens)
    batch.max_q_len, batch.positions = max(lens), torch.arange(T, dtype=torch.int32, device=DEV)
    decay = torch.tensor([1.0 - 2.0 ** -(1 + 3 * h % 20) for h in range(H)], device=DEV)
    return batch, r(T, 2 * H * D + H * V + 8).to(torch.bfloat16), r(len(lens) + 1, H * D * V + 6), decay, torch.rand(D // 4, generator=g).to(DEV)


def chunk_runs(ops, H, V, decay, freq, batch):
    return {"constant": lambda p, s: ops.lightning_scan(p, H, 128, V, decay, s, batch),
            "rotated": lambda p, s: ops.retention_scan(p, H, 128, V, freq, 128 ** -0.5, decay, s, batch)}


@pytest.mark.parametrize("lens,H,V", [((320,), 16, 128), ((384,), 3, 256), ((129, 640, 3, 127), 2, 128), ((700, 1, 1, 1, 513), 5, 128)])
def test_constant_decay_in_chunks(ops, lens, H, V):             # noqa: F811
    """128 tokens at a time against the token-by-token kernels: whole chunks, remainders, short entries beside long ones, two blocks of columns."""
    batch, p, state, decay, freq = chunk_inputs(lens, H, V, sum(lens))
    for name, run in chunk_runs(ops, H, V, decay, freq, batch).items():
        a, b = state.clone(), state.clone()
        assert ops._takes_octets(p, batch, 128, V, a) and ops._takes_chunks(batch, sum(lens), 128, V, H)
        got = run(p, a)
        ops._takes_octets = lambda *args: False
        try:
            want = run(p, b)
        finally:
            del ops._takes_octets
        ops.check_errors()
        # two float32 orders of sums over up to 700 decayed tokens and 128 rows
        assert rows_error(got, want) < 3e-6 and rows_error(a, b) < 3e-6, name
        assert torch.equal(a[:, H * 128 * V:], state[:, H * 128 * V:]) and torch.equal(a[0], state[0])


@pytest.mark.parametrize("what", ["q", "k", "v", "state", "huge k", "all tiny"])
def test_chunks_keep_odd_numbers_in_their_place(ops, what):     # noqa: F811
    """Numbers that three bfloat16 parts do not hold: the outputs are those of the token-by-token kernel, tokens before the number, other entries and
    other heads have the bits they have without it."""
    lens, H, V, at = (330, 320), 2, 128, 150                     # token 150: the 23rd of the first entry's second chunk
    batch, p, state, decay, freq = chunk_inputs(lens, H, V, 3)
    for name, run in chunk_runs(ops, H, V, decay, freq, batch).items():
        spoiled, odd_state = p.clone(), state.clone()
        if what in "qkv":
            spoiled[at, {"q": 5, "k": 128 * H + 7, "v": 256 * H + 9}[what]] = float("inf") if what != "k" else float("nan")
        elif what == "state":
            odd_state[batch.seg_slot[0].item(), 128 * 30 + 4] = float("inf")
        elif what == "huge k":
            spoiled[at, 128 * H + 7] = 1e30
        else:
            spoiled[at:at + 9, 128 * H:128 * H + 128] = -90.0 if name == "constant" else 1e-35
        a, b, c = state.clone(), odd_state.clone(), odd_state.clone()
        want, got = run(p, a), run(spoiled, b)
        ops._takes_octets = lambda *args: False
        try:
            plain = run(spoiled, c)
        finally:
            del ops._takes_octets
        first = 0 if what == "state" else at
        assert torch.equal(got[:first], want[:first]) and torch.equal(got[330:], want[330:]) and torch.equal(got[:, V:], want[:, V:]), name
        assert torch.equal(got.isnan(), plain.isnan()) and torch.equal(got.isinf(), plain.isinf()) and torch.equal(b.isnan(), c.isnan()), name
        ok = plain.isfinite()
        ok[at + 30 if what == "huge k" else len(ok):] = False    # what 1e30 has swallowed does not come back when it has decayed
        assert rows_error(torch.where(ok, got, 0.), torch.where(ok, plain, 0.)) < 3e-6, name


@pytest.mark.parametrize("q,k,v", [(-49, -49, 34), (34, 34, 34), (-85, -80, 40), (-60, -60, 30), (45, 50, 8), (-88, 20, 30), (30, -88, 38), (0, -30, -80), (-49, 34, -60)])
def test_chunks_near_the_ends_of_the_parts(ops, q, k, v):       # noqa: F811
    """Queries, keys and values near the ends of what bfloat16 parts hold, and beyond, together: powers of two, against float64."""
    lens, H, V, D = (330, 320), 2, 128, 128
    batch, p, state, decay, _ = chunk_inputs(lens, H, V, 5)
    decay = torch.tensor([0.5, 0.99], device=DEV)
    sizes = torch.cat([torch.full((H * D,), 2.0 ** q), torch.full((H * D,), 2.0 ** k), torch.full((H * V,), 2.0 ** v), torch.ones(8)]).to(DEV)
    p = (p * sizes).to(torch.bfloat16)
    state = state * 2.0 ** (k + v)
    a = state.clone()
    assert ops._takes_chunks(batch, sum(lens), D, V, H)
    got = ops.retention_scan(p, H, D, V, None, 1.0, decay, a, batch).view(-1, H, V)
    ops.check_errors()
    first = 0
    for i, n in enumerate(lens):
        x = (p[first:first + n, :3 * H * D].double() / sizes[:3 * H * D]).view(n, 3, H, D)
        slot = batch.seg_slot[i].item()
        S = (state[slot, :H * D * V].double() / 2.0 ** (k + v)).view(H, D, V)
        want = torch.empty(n, H, V, dtype=torch.float64, device=DEV)
        for t in range(n):
            S = decay.double()[:, None, None] * S + x[t, 1][:, :, None] * x[t, 2][:, None, :]
            want[t] = torch.einsum("hd,hdv->hv", x[t, 0], S)
        # float32 sums over up to 330 decayed tokens and 128 rows
        assert rows_error(got[first:first + n].double() / 2.0 ** (q + k + v), want) < 3e-6
        assert rows_error(a[slot, :H * D * V].double() / 2.0 ** (k + v), S.reshape(-1)) < 3e-6
        first += n


def test_silu_of_the_chunks(ops):                               # noqa: F811
    """The activation alone, over every bfloat16 from -88 to 2^36: with a decay of 0 and queries and keys of one entry of 64 (silu: 64) a token's output is
    4,096 times its activated values, without a rounding.  Against the division of the same float32 exponential, and against 64 bits."""
    D = V = 128
    x = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).float()
    x = x[(x.abs() >= 2.0 ** -89) & (x >= -60) & (x <= 2.0 ** 36)]      # silu down to 2^-81, which the parts hold
    far = torch.linspace(-88, -60, 513)[:512].to(torch.bfloat16).float()       # beyond -60 pieces of eight are told apart by their size
    g = torch.Generator().manual_seed(1)
    x = torch.cat([x[torch.randperm(x.numel(), generator=g)] for _ in range(2)])       # beside other neighbours each time
    x = torch.cat([x, far, torch.ones((-(x.numel() + 512)) % V)])
    T = x.numel() // V
    p = torch.zeros(T, 3 * D, dtype=torch.bfloat16)
    p[:, 0] = p[:, D] = 64.0
    p[:, 2 * D:] = x.view(T, V)
    batch = Entries((T,))
    batch.max_q_len = T
    state = torch.zeros(2, D * V, device=DEV)
    assert ops._takes_chunks(batch, T, D, V, 1)
    got = (ops.lightning_scan(p.to(DEV), 1, D, V, torch.zeros(1, device=DEV), state, batch).double() / 4096).view(-1)
    ops.check_errors()
    x = x.to(DEV)
    want = x.double() / (1 + (-x.double()).exp())
    division = (x / (1 + torch.exp(-x))).double()
    ulp = 2.0 ** (want.abs().log2().floor() - 23)
    # expf is within 1 unit (2 where the quotient's unit is half of it), the sum and the quotient half a unit each, the latter once more where it is not rounded
    # to nearest
    assert ((got - want).abs() / ulp).max().item() <= 4 and ((got - division).abs() / ulp).max().item() <= 1
    assert ((got - want).abs() / ulp).mean().item() <= 1.02 * ((division - want).abs() / ulp).mean().item()


def delta_inputs(lens, H, KV, V, seed):
    T, D, g = sum(lens), 128, torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)         # noqa: E731
    batch, C = Entries(lens), 2 * KV * D + H * V
    batch.max_q_len = max(lens)
    prep = torch.zeros(T, (C + H * D + H + 3) // 4 * 4, device=DEV)
    qk = r(T, 2 * KV, D)
    prep[:, :2 * KV * D] = (qk / qk.norm(dim=-1, keepdim=True)).reshape(T, -1)
    prep[:, 2 * KV * D:C] = r(T, H * V)
    decay = torch.rand(T, H * D, generator=g).to(DEV) ** 0.2
    decay[:, ::7], decay[:, 1::7] = 1.0, 0.0
    prep[:, C:C + H * D] = decay
    prep[:, C + H * D:C + H * D + H] = torch.rand(T, H, generator=g).to(DEV)
    return batch, prep, r(len(lens) + 1, H * D * V + 6)


@pytest.mark.parametrize("heads_at_once", [False, True])
@pytest.mark.parametrize("lens,H,KV,V", [((192,), 16, 8, 128), ((193, 31), 3, 3, 16), ((1, 256, 33, 7), 4, 2, 144), ((223, 1, 64, 32, 1), 5, 1, 256), ((64, 33, 96, 192), 8, 4, 128)])
def test_channel_decays_in_chunks(ops, monkeypatch, lens, H, KV, V, heads_at_once):     # noqa: F811
    """32 tokens at a time against the token-by-token kernel: whole chunks, remainders, single tokens beside prompts, more than 128 columns, a block
    and two blocks an SM (the last), decays down to 0, with scratch for all heads and for one at a time."""
    batch, prep, state = delta_inputs(lens, H, KV, V, sum(lens))
    if heads_at_once:
        monkeypatch.setattr(ops, "channel_work_bytes", 0)
    a, b = state.clone(), state.clone()
    assert ops._takes_octets(prep, batch, 128, V, a) and ops._takes_delta_chunks(batch, sum(lens), 128, V, H)
    got, want = ops.delta_scan(prep, H, KV, 128, V, a, batch), ops.delta_scan(prep, H, KV, 128, V, b, batch, exact=True)
    ops.check_errors()
    # two float32 orders of sums over up to 256 decayed tokens and 128 rows
    assert rows_error(got, want) < 3e-6 and rows_error(a, b) < 3e-6
    assert torch.equal(a[:, H * 128 * V:], state[:, H * 128 * V:]) and torch.equal(a[0], state[0])


@pytest.mark.parametrize("H", [2, 40])
@pytest.mark.parametrize("what", ["q", "k", "v", "decay", "beta", "state", "huge v", "tiny v"])
def test_channel_chunks_keep_odd_numbers_in_their_place(ops, monkeypatch, what, H):     # noqa: F811
    """Numbers that three bfloat16 parts do not hold: the outputs are those of the token-by-token kernel, tokens before the number, other entries and
    other heads have the bits they have without it."""
    lens, V, at = (200, 192), 32, 83                              # token 83: the 20th of the first entry's third chunk
    batch, prep, state = delta_inputs(lens, H, H, V, 3)
    C = 2 * H * 128 + H * V
    spoiled, odd_state = prep.clone(), state.clone()
    if what == "state":
        odd_state[batch.seg_slot[0].item(), V * 30 + 4] = float("inf")
    elif what == "huge v":
        spoiled[at, 256 * H + 3] = 1e30
    elif what == "tiny v":                                       # a head that holds nothing but numbers at the lower end
        spoiled[:200, 256 * H:256 * H + V] *= 1e-36
        odd_state[batch.seg_slot[0].item(), :128 * V] *= 1e-36
    else:
        spoiled[at, {"q": 5, "k": 128 * H + 7, "v": 256 * H + 9, "decay": C + 11, "beta": C + H * 128}[what]] = float("nan") if what in ("k", "decay", "beta") else float("inf")
    a, b, c = state.clone(), odd_state.clone(), odd_state.clone()
    monkeypatch.setattr(ops, "_takes_delta_chunks", lambda *args: True)         # also with so many heads of so few columns, for a ring of its own
    want, got = ops.delta_scan(prep, H, H, 128, V, a, batch), ops.delta_scan(spoiled, H, H, 128, V, b, batch)
    plain = ops.delta_scan(spoiled, H, H, 128, V, c, batch, exact=True)
    first = 0 if what in ("state", "tiny v") else at
    assert torch.equal(got[:first], want[:first]) and torch.equal(got[200:], want[200:]) and torch.equal(got[:, V:], want[:, V:])
    assert torch.equal(got.isnan(), plain.isnan()) and torch.equal(got.isinf(), plain.isinf()) and torch.equal(b.isnan(), c.isnan())
    ok = plain.isfinite()
    if what == "huge v":                                         # what 1e30 has swallowed does not come back when it has decayed
        ok[at:200] = False
        assert rows_error(got[at:at + 8, :V], plain[at:at + 8, :V]) < 3e-6
    scale = 1e36 if what == "tiny v" else 1.0
    if what == "tiny v":
        ok[:, V:] = False
        ok[200:] = False
    assert rows_error(torch.where(ok, got, 0.) * scale, torch.where(ok, plain, 0.) * scale) < 3e-6


@pytest.mark.parametrize("q,k,v", [(-49, -45, 30), (-85, -60, 40), (-60, -60, 20), (-80, 0, 20), (0, 0, -95), (30, 0, 28), (0, -70, 0), (-45, -3, -40)])
def test_channel_chunks_near_the_ends_of_the_parts(ops, monkeypatch, q, k, v):       # noqa: F811
    """Queries, keys and values near the ends of what bfloat16 parts hold, and beyond, together: powers of two, against float64."""
    lens, H, V, D = (200, 192), 2, 32, 128
    batch, prep, state = delta_inputs(lens, H, H, V, 6)
    C = 2 * H * D + H * V
    sizes = torch.cat([torch.full((H * D,), 2.0 ** q), torch.full((H * D,), 2.0 ** k), torch.full((H * V,), 2.0 ** v)]).to(DEV)
    prep[:, :C] *= sizes
    state = state * 2.0 ** (k + v)
    a = state.clone()
    monkeypatch.setattr(ops, "_takes_delta_chunks", lambda *args: True)
    got = ops.delta_scan(prep, H, H, D, V, a, batch).view(-1, H, V)
    ops.check_errors()
    first = 0
    for i, n in enumerate(lens):
        rows, slot = prep[first:first + n].double(), batch.seg_slot[i].item()
        part = lambda at, heads, w: rows[:, at:at + heads * w].view(n, heads, w)         # noqa: E731
        Q, K, U, g, beta = part(0, H, D), part(H * D, H, D), part(2 * H * D, H, V), part(C, H, D), rows[:, C + H * D:C + H * D + H]
        S, want = state[slot, :H * D * V].double().view(H, D, V), torch.empty(n, H, V, dtype=torch.float64, device=DEV)
        for t in range(n):
            S = g[t][:, :, None] * S
            u = beta[t][:, None] * (U[t] - torch.einsum("hdv,hd->hv", S, K[t]))
            S = S + K[t][:, :, None] * u[:, None, :]
            want[t] = torch.einsum("hd,hdv->hv", Q[t], S)
        # float32 sums over up to 200 decayed tokens and 128 rows
        assert rows_error(got[first:first + n].double() / 2.0 ** (q + k + v), want / 2.0 ** (q + k + v)) < 3e-6
        assert rows_error(a[slot, :H * D * V].double() / 2.0 ** (k + v), S.reshape(-1) / 2.0 ** (k + v)) < 3e-6
        first += n


def test_a_later_value_does_not_say_how_tiny_ones_are_computed(ops):    # noqa: F811
    """Values too small for their parts, with and without an ordinary one behind them in the same eight tokens: the same bits before it."""
    lens, H, V = (200, 192), 2, 128
    batch, prep, state = delta_inputs(lens, H, H, V, 8)
    first = 256 * H
    prep[:8, first:first + H * V] *= 2.0 ** -116
    state[batch.seg_slot[0].item()] = 0
    outs = []
    for size in (1.0, 2.0 ** 116):
        rows = prep.clone()
        rows[7, first:first + H * V] *= size
        outs.append(ops.delta_scan(rows, H, H, 128, V, state.clone(), batch))
    assert ops._takes_delta_chunks(batch, sum(lens), 128, V, H)
    assert torch.equal(outs[0][:7], outs[1][:7]) and not torch.equal(outs[0][7], outs[1][7])


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_octets_keep_later_tokens_out(ops, value):              # noqa: F811
    """A value that is no number reaches its own token and the ones after it; the tokens before it in its octet give the bits they give without it."""
    lens, H, D, V, at = (140, 133), 2, 128, 32, 13               # token 13: the sixth of the first entry's second octet
    T, batch, g = sum(lens), Entries(lens), torch.Generator().manual_seed(7)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)         # noqa: E731
    batch.positions = torch.arange(T, dtype=torch.int32, device=DEV)
    C, constant, state = 2 * H * D + H * V, torch.tensor([0.9, 0.99], device=DEV), r(3, H * D * V)
    prep = torch.cat([0.05 * r(T, 2 * H * D), r(T, H * V), torch.rand(T, H * D + 4, generator=g).to(DEV)], dim=1)
    p = r(T, C).to(torch.bfloat16)
    runs = {"delta": (prep, lambda x, s: ops.delta_scan(x, H, H, D, V, s, batch)), "constant": (p, lambda x, s: ops.lightning_scan(x, H, D, V, constant, s, batch)),
            "rotated": (p, lambda x, s: ops.retention_scan(x, H, D, V, None, 1.0, constant, s, batch))}
    for name, (rows, run) in runs.items():
        assert ops._takes_octets(rows, batch, D, V, state), name
        spoiled = rows.clone()
        spoiled[at, 2 * H * D + 3] = value                       # one value of head 0
        want, got = run(rows, state.clone()), run(spoiled, state.clone())
        assert torch.equal(got[:at], want[:at]) and torch.equal(got[lens[0]:], want[lens[0]:]), name
        assert not got[at, 3].isfinite() and torch.equal(got[:, V:], want[:, V:]), name


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens,inner,N", [((33, 1, 64), 40, 16), ((5, 100), 96, 8), ((31, 2), 33, 32), ((70,), 64, 16)])
def test_selective_scan_of_prompts(ops, dtype, lens, inner, N):         # noqa: F811
    """Chunks of 32 tokens and channels with remainders, against the same tokens one at a time (decode steps take the other kernel)."""
    T, g = sum(lens), torch.Generator().manual_seed(sum(lens))
    r = lambda *s: torch.randn(*s, generator=g)                 # noqa: E731
    x, z, B, C = (r(T, w).to(dtype).to(DEV) for w in (inner, inner, N, N))
    dt, dt_b, Dv = r(T, inner).to(DEV), r(inner).to(DEV), r(inner).to(DEV)
    A = -torch.exp(r(inner, N)).to(DEV)
    A[:, 0] = -300.0                                             # decays of e^-87 and less: 2e-38 at most in the one kernel, down to 0 in the other
    state = r(len(lens) + 1, inner * N + 4).to(DEV)
    a, b = state.clone(), state.clone()
    batch = Entries(lens)
    got = ops.selective_scan(x, dt, dt_b, A, B, C, Dv, z, a, batch, dtype)
    want = torch.empty_like(got)
    starts = batch.seg_q_start.tolist()
    for i, n in enumerate(lens):
        one = Entries((1,))
        one.seg_slot = batch.seg_slot[i:i + 1]
        for t in range(starts[i], starts[i] + n):
            row = slice(t, t + 1)
            want[row] = ops.selective_scan(x[row].contiguous(), dt[row].contiguous(), dt_b, A, B[row], C[row], Dv, z[row], b, one, dtype)
    assert rows_error(a, b) < 3e-6
    assert rows_error(got, want) < (3e-6 if dtype == torch.float32 else 4e-3)        # bfloat16: the output's own rounding may fall differently


def recurrent_part(kind):
    """One recurrent mixer of a design, float32, with seeded weights, and the context of a step of [(slot, tokens)] over given states."""
    import types
    from mini_inference_b200.config.spec import PartSpec
    from mini_inference_b200.parts.base import build_part
    base = dict(hidden_size=96, num_heads=2, key_dim=64, value_dim=64, out_norm_eps=1e-6)
    spec = {"lightning": PartSpec.of("lightning", decay=(0.9, 0.99), **base), "retention": PartSpec.of("retention", decay=(0.9, 0.99), **base),
            "channel_delta": PartSpec.of("channel_delta", num_kv_heads=1, conv_taps=4, unit_eps=1e-6, decay_rank=16, gate_rank=16, **base),
            "selective_scan": PartSpec.of("selective_scan", hidden_size=96, inner=64, state=16, dt_rank=8, conv_taps=4)}[kind]
    part, g = build_part("mixer", spec), torch.Generator().manual_seed(11)
    part.load({w.name: (torch.randn(w.shape, generator=g) * (0.3 if len(w.shape) > 1 else 0.5)).to(DEV) for w in part.weight_specs()}, torch.float32, DEV)
    return part, types.SimpleNamespace(rotary_inv_freq=lambda: None)


@pytest.mark.parametrize("kind", ["lightning", "retention", "channel_delta", "selective_scan"])
def test_float32_recurrences_do_not_see_the_batch(ops, kind):   # noqa: F811
    """A float32 run's outputs and states are the same bits whether a prompt comes whole or in two portions, alone or beside others.  (Steps of
    more than four tokens an entry: below that the matrix recurrences' scan sums over eight lanes instead of sixteen.)"""
    import types
    part, position = recurrent_part(kind)
    floats = part.cache_need().shape[0]
    g = torch.Generator().manual_seed(12)
    h, other = torch.randn(600, 96, generator=g).to(DEV), torch.randn(700, 96, generator=g).to(DEV)

    def step(state, lens, slots, rows, pos0):
        batch = Entries(lens)
        batch.seg_slot = torch.tensor(slots, dtype=torch.int32, device=DEV)
        batch.token_seg = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).int().to(DEV)
        batch.positions = torch.cat([torch.arange(p, p + n) for p, n in zip(pos0, lens)]).int().to(DEV)
        batch.max_q_len = max(lens)
        ctx = types.SimpleNamespace(ops=ops, batch=batch, dtype=torch.float32)
        return part.forward(rows, ctx, types.SimpleNamespace(state=state), position)

    whole = torch.zeros(4, floats, device=DEV)
    want = step(whole, (600,), (1,), h, (0,))
    cut = torch.zeros(4, floats, device=DEV)
    got = [step(cut, (45,), (1,), h[:45], (0,)), step(cut, (97, 700, 1), (1, 3, 2), torch.cat([h[45:142], other, h[:1]]), (45, 0, 0))[:97],
           step(cut, (458, 1), (1, 2), torch.cat([h[142:], h[:1]]), (142, 1))[:458]]
    assert torch.equal(torch.cat(got), want)
    assert torch.equal(cut[1], whole[1])


def test_silu_keeps_its_float32(ops):                           # noqa: F811
    """The filter's activation and the scan's gate of bfloat16 prompts are float32's silu rounded once, down to inputs where 1 + e^-x is nearly
    the largest float32: the fast exponential is 4e-4 off at -80 (a tenth of a bfloat16 step) and the fast quotient 0 from -87.4 on."""
    T, inner, N = 512, 64, 16
    grid = torch.cat([torch.linspace(-88.5, -60, 220), torch.linspace(-20, 20, 292)]).to(torch.bfloat16).to(DEV)
    want = (grid.double() / (1 + (-grid.double()).exp())).float().to(torch.bfloat16)
    rows = grid[:, None].expand(T, inner).contiguous()
    batch = Entries((T,))
    batch.token_seg = torch.zeros(T, dtype=torch.int32, device=DEV)
    conv = ops.short_conv(rows, torch.ones(inner, 1, device=DEV), None, 1, None, 0, batch, act="silu")
    one, zero = torch.ones(T, inner, dtype=torch.bfloat16, device=DEV), torch.zeros(inner, device=DEV)
    bc = torch.zeros(T, N, dtype=torch.bfloat16, device=DEV)
    gate = ops.selective_scan(one, torch.zeros(T, inner, device=DEV), zero, -torch.ones(inner, N, device=DEV), bc, bc, zero + 1, rows,
                              torch.zeros(2, inner * N, device=DEV), batch, torch.bfloat16)           # (0 + 1 * 1) * silu(z)
    for got in (conv, gate):
        # a double rounding may fall the other way where the float32 value lies within its own error of the middle: 2e-7 / 2^-8 of the values
        assert (got != want[:, None]).float().mean().item() < 5e-3
        assert ((got.double() / want.double()[:, None] - 1).abs().nan_to_num() <= 2 ** -7).all()


def states_after_one_decay(ops, A, step, N=16):
    """What a prompt leaves of states that were 1: its first token has the given step, the other 47 a step of 0, and no token adds anything."""
    T, inner = 48, A.shape[0]
    dt = torch.full((T, inner), -200.0, device=DEV)              # softplus: 0
    dt[0] = step                                                # softplus of more than 20: itself
    z = torch.zeros(T, inner, dtype=torch.bfloat16, device=DEV)
    bc, zero, state = torch.zeros(T, N, dtype=torch.bfloat16, device=DEV), torch.zeros(inner, device=DEV), torch.ones(2, inner * N, device=DEV)
    ops.selective_scan(z, dt, zero, A.contiguous(), bc, bc, zero, z, state, Entries((T,)), torch.bfloat16)
    return state[1].view(inner, N)


@pytest.mark.parametrize("step", [32.0, 21.7])
def test_decays_of_the_selective_scan(ops, step):               # noqa: F811
    """e^(step A) over its whole range against 64 bits: no worse than expf of the rounded product, which is within 2 units in the last place."""
    g = torch.Generator().manual_seed(1)
    for lo, hi in ((1e-4, 1e-2), (1e-2, 0.1), (0.1, 1), (1, 5), (5, 20), (20, 50), (50, 86)):
        A = (-(torch.rand(2048, 16, generator=g, dtype=torch.float64) * (hi - lo) + lo) / step).float().to(DEV)
        product = A.double() * torch.tensor(step, device=DEV).float().double()
        got = (states_after_one_decay(ops, A, step).double() / product.exp() - 1).abs()
        expf = ((A * step).exp().double() / product.exp() - 1).abs()
        # half a unit of the result (6e-8 above a power of two) and of the sum before it; expf's own mean is 2.7e-8 to 3.2e-8
        assert got.max().item() < max(1.0e-7, expf.max().item()) and got.mean().item() <= 1.02 * expf.mean().item(), (lo, hi)
    far = states_after_one_decay(ops, torch.full((32, 16), -200.0 / step, device=DEV), step)
    assert 0 <= far.min().item() and far.max().item() < 1e-37


def test_unusual_decays_of_the_selective_scan(ops):             # noqa: F811
    """Rates that are no number, not negative or huge, and steps beyond any softplus of a sane input, go where expf takes them."""
    nan = float("nan")
    A = torch.full((96, 16), -0.5, device=DEV)
    A[3, 2], A[40, 1], A[41, 5], A[70, 0], A[70, 1], A[71, 9] = nan, 1.5, -3e38, 0.0, -1e30, 3.0e3
    for step in (24.0, 1e9):
        want = (step * A).exp()
        got = states_after_one_decay(ops, A, step)
        assert got[3, 2].isnan() and got[~A.isnan()].allclose(want[~A.isnan()], rtol=3e-7, atol=1e-37)
    small = torch.full((32, 16), -1e-9, device=DEV)             # a huge step times a tiny rate
    assert states_after_one_decay(ops, small, 1e9).allclose((small * 1e9).exp(), rtol=3e-7)


@pytest.mark.parametrize("lens,inner,N", [((61, 40), 33, 32), ((70, 1, 33), 40, 8)])
def test_selective_scan_of_prompts_with_other_states(ops, lens, inner, N):      # noqa: F811
    """The same with 8 and 32 states a channel, in steps whose portions are long enough for the prompt kernel."""
    assert ops._takes_prompt_scan(sum(lens), Entries(lens))
    test_selective_scan_of_prompts(ops, torch.bfloat16, lens, inner, N)


@pytest.mark.parametrize("H,KV,D", [(16, 8, 128), (3, 1, 64), (5, 5, 128)])
@pytest.mark.parametrize("form", ["unit", "weights_rotated", "all_rotated", "temperature_keys", "blend", "plain"])
def test_unit_heads_of_prompts(ops, H, KV, D, form):            # noqa: F811
    """Normed, rotated and cached heads of 300 tokens at once, against the same tokens in pieces that the other kernel takes."""
    T, page, g = 300, 16, torch.Generator().manual_seed(H + D)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)         # noqa: E731
    keys = form == "temperature_keys"
    p = r(T, (H + KV) * D + (0 if keys else KV * D)).to(torch.bfloat16)
    qw, kw = (r(D).abs() + 0.5 for _ in range(2))
    freq = torch.rand(D // 2, generator=g).to(DEV) * 0.1
    args = {"unit": {}, "plain": {}, "weights_rotated": dict(q_weight=qw, k_weight=kw, inv_freq=freq[:D // 4].contiguous()), "all_rotated": dict(inv_freq=freq),
            "temperature_keys": dict(q_weight=qw, k_weight=kw, q_temp=(0.1, 64), values_are_keys=True), "blend": {}}[form]
    source = r(T, 2 * KV * D).to(torch.bfloat16)[:, KV * D:] if form == "blend" else None
    lam = torch.tensor([0.3], device=DEV) if form == "blend" else None
    slots = torch.randperm(T, generator=g).to(torch.int32).to(DEV) + page
    positions = torch.arange(7, 7 + T, dtype=torch.int32, device=DEV)
    results = []
    for piece in (T, 100):
        rows, k = p.clone(), torch.zeros((T + page) // page + 2, KV, page, D, dtype=torch.bfloat16, device=DEV)
        v = torch.zeros_like(k)
        for a in range(0, T, piece):
            meta = type("Meta", (), dict(slots=slots[a:a + piece].contiguous(), positions=positions[a:a + piece].contiguous(), page_size=page))
            part = rows[a:a + piece]
            ops.unit_qk_cache(part, H, KV, D, D, None if form == "plain" else 1e-6, lam, None if source is None else source[a:a + piece], meta, k, v, **args)
        results.append((rows, k, v))
    for a, b in zip(*results):                                  # one bfloat16 rounding of values that differ in their last float32 bits
        assert (a.float() - b.float()).abs().max().item() <= 2 ** -8 * b.float().abs().max().item()
        assert (a != b).float().mean().item() < 1e-2


# ---------------------------------------------------------------- kernels that a rule on sizes picks, against the plain statements (tests/ref_ops.py)
def both_batches(lens, slots):
    import types
    qs = [0]
    for n in lens:
        qs.append(qs[-1] + n)
    dev = Entries(lens)
    dev.seg_slot = torch.tensor(slots, dtype=torch.int32, device=DEV)
    dev.token_seg = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).int().to(DEV)
    dev.max_q_len = max(lens)
    return types.SimpleNamespace(host={"seg_q_start": qs, "seg_slot": slots}, num_segs=len(lens)), dev


@pytest.mark.parametrize("D,V", [(64, 64), (64, 128), (128, 64), (128, 128)])
def test_one_token_per_entry_of_matrix_states(ops, D, V):       # noqa: F811
    """Decode steps: states in registers, key heads shared by value heads, slots out of order, rows and slots with padding behind them."""
    from tests.ref_ops import TorchRefOps
    ref, H, KV, lens = TorchRefOps(), 6, 2, (1,) * 7
    host, dev = both_batches(lens, [3, 1, 8, 2, 7, 5, 4])
    g = torch.Generator().manual_seed(D + V)
    C = 2 * KV * D + H * V
    prep = torch.randn(7, C + H * D + H + 6, generator=g)
    prep[:, :2 * KV * D] *= D ** -0.5
    prep[:, C:] = torch.rand(7, H * D + H + 6, generator=g)
    state = torch.randn(9, H * D * V + 12, generator=g)
    p, decay = torch.randn(7, 2 * H * D + H * V + 5, generator=g).to(torch.bfloat16), torch.rand(H, generator=g)
    runs = {"delta": lambda o, s, b, x: o.delta_scan(x[0], H, KV, D, V, s, b), "constant": lambda o, s, b, x: o.lightning_scan(x[1], H, D, V, x[2], s, b)}
    for name, run in runs.items():
        a, b = state.clone().to(DEV), state.clone()
        assert ops._takes_step(7, dev, D, V, a), name
        got = run(ops, a, dev, (prep.to(DEV), p.to(DEV), decay.to(DEV)))
        want = run(ref, b[:, :H * D * V] if name == "constant" else b, host, (prep, p, decay))
        # float32 sums of up to 128 products in another order
        assert rows_error(got.cpu(), want) < 2e-6 and rows_error(a[1:].cpu(), b[1:]) < 2e-6, name
        assert torch.equal(a[:, H * D * V:].cpu(), state[:, H * D * V:]) and torch.equal(a[6].cpu(), state[6]), name


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("H,KV,D,V", [(4, 2, 128, 128), (3, 1, 64, 48), (2, 2, 12, 20)])
def test_delta_prologue_of_prompts(ops, taps, H, KV, D, V):     # noqa: F811
    """A warp takes eight neighbouring tokens: entries that begin and end among them, entries shorter than the taps, the slots' earlier inputs."""
    from tests.ref_ops import TorchRefOps
    ref, lens = TorchRefOps(), (5, 1, 2, 97, 60, 35)
    host, dev = both_batches(lens, [2, 6, 1, 4, 3, 5])
    T, C, g = sum(lens), 2 * KV * D + H * V, torch.Generator().manual_seed(taps)
    assert T >= 192                                              # where the kernel's range begins
    p = torch.randn(T, (C + H + 9) // 4 * 4 + 4, generator=g).to(torch.bfloat16)
    a = torch.randn(T, 2 * H * D, generator=g).to(torch.bfloat16)
    conv, A_log, bias = torch.randn(C, taps, generator=g), torch.randn(H, generator=g) * 0.3, torch.randn(H * D, generator=g)
    state = torch.randn(7, H * D * V + (taps - 1) * C, generator=g)
    sa, sb = state.clone().to(DEV), state.clone()
    got = ops.delta_prepare(p.to(DEV), a.to(DEV)[:, :H * D], conv.to(DEV), A_log.to(DEV), bias.to(DEV), H, KV, D, V, taps, 1e-6, sa, dev)
    want = ref.delta_prepare(p, a[:, :H * D], conv, A_log, bias, H, KV, D, V, taps, 1e-6, sb, host)
    n = C + H * D + H
    assert (got[:, :n].cpu() - want[:, :n]).abs().max().item() < 4e-6 * want.abs().max().item()
    assert torch.equal(sa.cpu(), sb)                             # the newest inputs, copied


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("groups,gs", [(1, 516), (2, 1024), (1, 2052), (3, 4096)])
def test_wide_group_norms(ops, dtype, groups, gs):              # noqa: F811
    """A group in a block's registers: one to four quads a thread, whole and not; a weight per group, per row or none; a gate that is a view."""
    from tests.ref_ops import TorchRefOps
    ref, g, T, n = TorchRefOps(), torch.Generator().manual_seed(gs), 5, groups * gs
    o, gate = torch.randn(T, n, generator=g), torch.randn(T, n + 10, generator=g).to(dtype)
    for weight in (None, torch.randn(gs, generator=g), torch.randn(n, generator=g)):
        for act in ("sigmoid", "silu"):
            got = ops.group_rmsnorm_gate(o.to(DEV), None if weight is None else weight.to(DEV), gate.to(DEV)[:, 6:6 + n], 1e-6, groups, gs, dtype, act=act).cpu()
            want = ref.group_rmsnorm_gate(o, weight, gate[:, 6:6 + n], 1e-6, groups, gs, dtype, act=act)
            limit = 2e-6 if dtype == torch.float32 else 2 ** -7     # bfloat16: the output may round to the neighbouring number
            assert ((got.float() - want.float()).abs() <= limit * want.float().abs().clamp_min(0.1)).all(), (act, weight is None)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [255, 257])
@pytest.mark.parametrize("H,V", [(5, 64), (16, 8), (3, 136)])
def test_head_gates_of_prompts(ops, dtype, T, H, V):            # noqa: F811
    from tests.ref_ops import TorchRefOps
    ref, g = TorchRefOps(), torch.Generator().manual_seed(T + V)
    o, gate = torch.randn(H, T, V, generator=g).to(dtype), torch.randn(T, H + 7, generator=g).to(dtype)
    for w in (gate[:, 3:3 + H], None):
        got, want = ops.head_gate(o.to(DEV), None if w is None else gate.to(DEV)[:, 3:3 + H], dtype).cpu(), ref.head_gate(o, w, dtype)
        limit = 3e-7 if dtype == torch.float32 else 2 ** -7
        assert ((got.float() - want.float()).abs() <= limit * want.float().abs()).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,hidden", [(127, 264), (128, 264), (128, 2050), (600, 2048)])
def test_weighted_sum_of_experts(ops, dtype, T, hidden):        # noqa: F811
    """128 tokens or more in 16-byte pieces where rows allow, fewer an entry a thread; with and without weights, a shared expert and its gate."""
    g, top = torch.Generator().manual_seed(T), 3
    rows, shared = torch.randn(T * top, hidden, generator=g).to(dtype).to(DEV), torch.randn(T, hidden, generator=g).to(dtype).to(DEV)
    weights, gate = torch.rand(T, top, generator=g).to(DEV), torch.randn(T, generator=g).to(DEV)
    for w, s, sg in ((weights, shared, gate), (weights, shared, None), (None, None, None)):
        out = torch.empty(T, hidden, dtype=dtype, device=DEV)
        assert ops.lib.mi_moe_combine(rows, w, s, sg, out, T, hidden, top, int(dtype == torch.bfloat16), ops._stream()) == 0
        want = (rows.double().view(T, top, hidden) * (1.0 if w is None else w.double()[:, :, None])).sum(1)
        if s is not None:
            want += s.double() * (1.0 if sg is None else torch.sigmoid(sg.double())[:, None])
        limit = 1e-6 if dtype == torch.float32 else 2 ** -7
        assert ((out.double() - want).abs() <= limit * want.abs().clamp_min(0.5)).all()


@pytest.mark.parametrize("form", ["causal", "sink", "bias", "gate", "latent"])
def test_both_halves_of_a_softmax_weight_count(ops, form):      # noqa: F811
    """Every weight but the first is e^-0.0021, which bfloat16 rounds down by 0.18 %: with the first half alone all outputs are that much too
    small, far more than their own roundings' mean, which the other half must take away."""
    H, KV, D, T, page = 2, (1 if form == "latent" else 2), 128, 1200, 16        # as many keys as the tcgen05 forms want
    meta, g = make_meta(page, [(0, T)], 80, 6), torch.Generator().manual_seed(3)
    assert ops._takes_split_tc(T, meta, ops.SPLIT_TC_LATENT)
    q, k = torch.zeros(T, H * D), torch.zeros(T, KV, D)
    q[:, ::D], k[1:, :, 0] = 1.0, -0.0021
    v = (0.5 + torch.rand(T, KV, D, generator=g)) * (1 + torch.rand(D, generator=g))
    if form == "latent":                                        # keys are the values: the scores read a column that is no value
        v[:, :, 0] = k[:, :, 0]
    q, k, v = (x.to(torch.bfloat16) for x in (q, k, v))
    pools = [torch.zeros(81, KV, page, D, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    where = meta.slots.long()
    for pool, x in zip(pools, (k, v)):
        pool[where // page, :, where % page] = x.to(DEV)
    if form == "latent":
        got = ops.paged_attention(q.to(DEV), pools[1], pools[1], meta, H, KV, D, 1.0, None, split_weights=True)
    else:
        args = {"causal": {}, "sink": dict(sink_values=torch.zeros(H, device=DEV)), "bias": dict(distance_bias=torch.zeros(9, H, device=DEV)),
                "gate": dict(gate=torch.full((T, H * D), 40.0, dtype=torch.bfloat16, device=DEV))}[form]
        got = ops.masked_attention(q.to(DEV), *pools, meta, H, KV, D, D, 1.0, None, None, form == "sink", **args)
    ops.check_errors()
    w = k[:, 0, 0].double().exp().expand(T, T).tril()
    total = w.sum(1, keepdim=True) + (form == "sink")
    sums = lambda w: torch.einsum("tk,khd->thd", w, v.double()) / total[:, :, None]      # noqa: E731
    want, first_half = sums(w), sums(w.float().to(torch.bfloat16).double())
    pick = lambda x: x[100:, :, 1:]                             # noqa: E731  (rows of many keys)
    got = got.cpu().double().view(T, H, D)
    want, first_half = (x.repeat_interleave(H // KV, dim=1) for x in (want, first_half))
    assert pick(first_half / want - 1).mean().item() < -1.5e-3
    assert abs(pick(got / want - 1).mean().item()) < 1.5e-4


def test_sampler_forms_agree(ops):                              # noqa: F811
    """Few scores: eight a thread, fetched together; 4.5 million and more: sixteen, one after the other.  The choices are the same whole numbers."""
    R, V = 40, 120001
    g = torch.Generator().manual_seed(0)
    logits = torch.randn(R, V, generator=g).to(DEV)
    temps = torch.tensor([0.0, 0.7] * (R // 2), device=DEV)
    seeds, counters = torch.arange(R, dtype=torch.int32, device=DEV), torch.arange(5, 5 + R, dtype=torch.int32, device=DEV)
    got = ops.sample(logits, temps, seeds, counters)
    parts = [ops.sample(logits[a:a + 8], temps[a:a + 8].contiguous(), seeds[a:a + 8].contiguous(), counters[a:a + 8].contiguous()) for a in range(0, R, 8)]
    assert torch.equal(got, torch.cat(parts))
    assert torch.equal(got[::2].long(), logits[::2].argmax(-1))


def expert_rows(ops, counts, seed):
    """chosen [T, 1] with counts[e] tokens of expert e, in a random order."""
    g = torch.Generator().manual_seed(seed)
    chosen = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts))
    return chosen[torch.randperm(len(chosen), generator=g)].to(torch.int32).to(DEV)[:, None].contiguous(), g


@pytest.mark.parametrize("counts", [(1, 31, 0, 32, 33), (255, 256, 257, 0), (512, 513, 7), (0, 0, 700), (3, 16500, 0, 520, 4)])
def test_plan_of_expert_tiles(ops, counts):                     # noqa: F811
    """Every pair once, among its expert's rows; an expert's tiles cover its rows in steps of 32, at most 256 each."""
    chosen, _ = expert_rows(ops, counts, sum(counts))
    P, E = chosen.shape[0], len(counts)
    cap = ops.lib.mi_moe_plan_rows(P, E)
    pairs, plan = torch.full((cap,), -7, dtype=torch.int32, device=DEV), torch.zeros(ops.lib.mi_moe_plan_ints(P, E), dtype=torch.int32, device=DEV)
    assert ops.lib.mi_moe_plan(chosen, P, E, pairs, cap, plan, ops._stream()) == 0
    pairs, plan, chosen = pairs.cpu(), plan.cpu(), chosen.cpu()[:, 0]
    tiles = plan[4:4 + 4 * plan[0].item()].view(-1, 4)
    assert sorted(pairs[pairs >= 0].tolist()) == list(range(P)) and int(pairs.min()) >= -1
    end = 0
    for first, rows, e, _ in tiles.tolist():
        assert first == end and rows % 32 == 0 and 0 < rows <= 256
        end = first + rows
        here = pairs[first:end]
        assert (chosen[here[here >= 0].long()] == e).all()
    assert end == sum(-(-n // 32) * 32 for n in counts) and (pairs[end:] == -1).all()
    assert [sum(t[2] == e for t in tiles.tolist()) for e in range(E)] == [-(-n // 256) for n in counts]


@pytest.mark.parametrize("counts,K,F,hidden", [((1, 31, 32, 33, 200), 64, 64, 8), ((255, 257, 0), 192, 192, 264), ((512, 513), 320, 128, 520), ((0, 60, 420, 96), 1088, 704, 1032)])
def test_expert_products_in_pairs_of_blocks(ops, counts, K, F, hidden):     # noqa: F811
    """The grouped products against float64, with the activated rows and the rows rounded to bfloat16 where the kernels round them: tiles of 32 to 256
    rows, experts without rows, outputs and K that are no multiple of a tile's."""
    chosen, g = expert_rows(ops, counts, K)
    T, E = chosen.shape[0], len(counts)
    r = lambda *s, std=1.0: (std * torch.randn(*s, generator=g)).to(torch.bfloat16).to(DEV)      # noqa: E731
    h, w_in, w_out = r(T, K), r(E, 2 * F, K, std=K ** -0.5), r(E, hidden, F, std=F ** -0.5)
    weights = torch.rand(T, 1, generator=g).to(DEV)
    assert T > 48 * E and ops.moe_tcgen05
    got = ops.expert_ffn(h, chosen, weights, w_in, w_out, 2.0, 1.7, None)
    ops.check_errors()
    want = torch.zeros(T, hidden, dtype=torch.float64, device=DEV)
    for e in range(E):
        t = (chosen[:, 0] == e).nonzero()[:, 0]
        x = h[t].double() @ w_in[e].double().T
        gate, up = x[:, :F].clamp(max=2.0), x[:, F:].clamp(-2.0, 2.0)
        y = (gate * torch.sigmoid(1.7 * gate) * (up + 1.0)).to(torch.bfloat16).double()
        want[t] = (y @ w_out[e].double().T).to(torch.bfloat16).double() * weights[t].double()
    # three roundings to bfloat16 (activated rows and rows on either side of a tie, the sum), each at most 2^-9 of a number
    assert rows_error(got, want) < 3 * 2.0 ** -9


@pytest.mark.parametrize("M,N,K,want", [(5, 4096, 2560, 3), (1030, 4096, 2560, 6), (40, 20480, 1024, 2), (3000, 64, 130, 1), (1030, 96, 2048, 4)])
def test_launches_of_float32_products_are_counted(ops, M, N, K, want):  # noqa: F811
    """Splitting, product and sum of the segments, per 1,024 rows."""
    x, w, before = torch.zeros(M, K, device=DEV), torch.zeros(N, K, device=DEV), ops.launches
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        ops.linear(x, w)
        torch.cuda.synchronize()
    assert ops.launches - before == want
    assert sum(e.count for e in prof.key_averages() if "gemm_f32" in e.key or "split_rows" in e.key or "add_segments" in e.key) == want
