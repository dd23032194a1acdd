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
