"""The rules that choose between kernels, on the CPU: what a faster kernel cannot take stays with the general one."""
import types

import torch

from mini_inference_b200.ops import CudaOps


def off_by(floats, *shape):
    """A contiguous float32 tensor that starts `floats` floats behind a 64-byte boundary."""
    n = torch.Size(shape).numel()
    buf = torch.zeros(n + 32)
    start = (-buf.data_ptr() // 4) % 16 + floats
    return buf[start:start + n].view(*shape)


def step(lens):
    return types.SimpleNamespace(num_segs=len(lens), max_q_len=max(lens))


def test_float32_attention_in_tiles_wants_caches_on_16_bytes():
    """Its 16-byte copies fault on other addresses; the kernel for any head size loads such keys and values as well."""
    me, meta = types.SimpleNamespace(fast_attention=True), types.SimpleNamespace(tile=64)
    q, k, v = off_by(0, 8, 128), off_by(0, 2, 1, 16, 128), off_by(4, 2, 1, 16, 128)
    assert CudaOps._f32_tiles(me, q, 128, 128, meta, k, v)
    for floats in (1, 2, 3):
        odd = off_by(floats, 2, 1, 16, 128)
        assert not CudaOps._f32_tiles(me, q, 128, 128, meta, odd, v)
        assert not CudaOps._f32_tiles(me, q, 128, 128, meta, k, odd)
        assert not CudaOps._f32_tiles(me, off_by(floats, 8, 128), 128, 128, meta, k, v)


def test_states_that_start_anywhere_keep_the_general_scan():
    """The eight-token scan moves states eight bytes at a time (and refuses others); the token-by-token scan takes every start."""
    rows, one = off_by(0, 600, 3 * 128), step((600,))
    assert CudaOps._takes_octets(rows, one, 64, 64, off_by(2, 2, 64 * 64))
    assert not CudaOps._takes_octets(rows, one, 64, 64, off_by(1, 2, 64 * 64))
    assert not CudaOps._takes_octets(rows, one, 64, 64, off_by(0, 2, 64 * 64 + 1))


def test_as_many_tokens_as_entries_is_not_one_each():
    """The kernel for one token per entry reads an entry's first token only."""
    state = off_by(0, 3, 64 * 64)
    assert CudaOps._takes_step(2, step((1, 1)), 64, 64, state)
    assert not CudaOps._takes_step(2, step((2, 0)), 64, 64, state)


def test_line_of_the_eight_token_scans():
    """A prompt of 192 tokens or 512 tokens in all; shorter steps wait for the host, and this way has one launch more."""
    rows, state = off_by(0, 600, 3 * 128), off_by(0, 2, 64 * 64)
    takes = lambda *lens: CudaOps._takes_octets(rows[:sum(lens)], step(lens), 64, 64, state)      # noqa: E731
    assert takes(192) and takes(192, *[1] * 40) and not takes(191) and not takes(64, 64, 64)
    assert takes(*[64] * 8) and not takes(*[63] * 8)


def test_lines_of_recurrences_in_chunks():
    """By tokens, entries and heads: short entries take whole chunks, which many heads feel and few do not."""
    takes = lambda H, V, *lens: CudaOps._takes_chunks(step(lens), sum(lens), 128, V, H)       # noqa: E731
    for H in (1, 2, 16, 64):
        assert takes(H, 128, 320) and takes(H, 128, 2048) and takes(H, 128, *[512] * 4) and not takes(H, 128, 319) and not takes(H, 128, 330, *[1] * 4)
    assert takes(16, 128, 700, 1, 1, 1) and takes(32, 128, 700, 1, 1, 1) and takes(16, 128, 330, 1, 1) and takes(16, 128, 2048, *[1] * 18)
    assert not takes(32, 128, 330, 1, 1) and not takes(64, 128, 1024, *[1] * 8) and not takes(16, 512, 1024, *[1] * 8) and not takes(48, 128, 330, 1)
    delta = lambda H, V, *lens: CudaOps._takes_delta_chunks(step(lens), sum(lens), 128, V, H)    # noqa: E731
    for H in (2, 16, 64):
        assert delta(H, 128, 192) and delta(H, 128, 2048) and delta(H, 128, *[512] * 4) and not delta(H, 128, 192, *[1] * 10)
    assert delta(16, 128, 300, *[1] * 10) and delta(32, 128, *[64] * 16) and delta(16, 256, *[64] * 16) and delta(4, 16, 192)
    assert not delta(32, 128, 300, *[1] * 10) and not delta(2, 128, *[64] * 8) and not delta(64, 16, *[512] * 4) and not delta(64, 16, 192)


def test_line_of_the_selective_scan():
    """An entry costs the kernel for prompts about the same however short it is, the other one walks the longest entry at a quarter of the speed."""
    takes = lambda *lens: CudaOps._takes_prompt_scan(sum(lens), step(lens))      # noqa: E731
    assert takes(18) and not takes(17) and not takes(1) and not takes(1, 1)
    assert takes(40, 1) and takes(130, *[1] * 5) and not takes(74, *[1] * 5) and not takes(2, *[1] * 63)
    assert takes(*[140] * 4) and not takes(*[100] * 4) and not takes(*[24] * 16) and takes(2048, *[1] * 63)


def test_lines_of_split_attention_on_tcgen05():
    """By keys and by tokens: a step that waits for the host anyway keeps the form that costs the host less."""
    takes = lambda T, keys, line: CudaOps._takes_split_tc(T, types.SimpleNamespace(max_kv_len=keys), line)      # noqa: E731
    masked, latent = CudaOps.SPLIT_TC_MASKED, CudaOps.SPLIT_TC_LATENT
    assert takes(2, 520, masked) and takes(780, 260, masked) and not takes(260, 260, masked) and not takes(2000, 200, masked)
    assert takes(2, 1500, latent) and takes(2048, 512, latent) and not takes(2, 1000, latent) and not takes(500, 700, latent)


def test_a_decoded_tokens_keys_do_not_count_for_prompt_attention():
    """Beside a decoded token of 3,000 keys a portion of two tokens behind 500 is a short one."""
    from mini_inference_b200.engine.batch import BatchLayout, StepBatch, StepFacts
    fields = [(n, 8) for n in ("token_ids", "positions", "token_seg", "seg_q_start", "seg_pos0", "seg_kv_len", "seg_slot", "logit_rows")]
    layout = BatchLayout(fields)

    def batch(lens, pos0):
        facts = StepFacts(lens, pos0, list(range(1, len(lens) + 1)), 64)
        return StepBatch(layout, torch.zeros(layout.size, dtype=torch.int32), None, facts, {}, 1, int(facts.kv_len.max()), False)

    mixed, decode = batch([2, 1], [500, 3000]), batch([1, 1], [3000, 20])
    assert mixed.max_kv_len == 3001 and mixed.max_prompt_kv_len == 502 and decode.max_prompt_kv_len == 0
    assert not CudaOps._takes_split_tc(3, mixed, CudaOps.SPLIT_TC_MASKED)
    assert CudaOps._takes_split_tc(3, batch([2, 1], [600, 3000]), CudaOps.SPLIT_TC_MASKED)
