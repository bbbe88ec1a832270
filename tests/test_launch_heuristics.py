"""Host-side launch decisions of the kernel library (no GPU needed: the functions only
compute): into how many runs of keys the attention kernels cut a step."""
import os
import re

import pytest

from inferx_b200.kernels import library, ops


@pytest.fixture(scope="module")
def lib():
    return ops._lib()


def test_prompt_attention_is_cut_only_for_few_queries_over_a_long_context(lib):
    f = lib.ix_attn_prefill_tc_splits          # (tokens, sequences, heads, keys, window)
    assert f(2048, 1, 16, 2048, 0) == 1        # 256 (query tile, head) items fill the device
    assert f(512, 1, 16, 1500, 0) == 1         # few items, but the context is short
    assert f(512, 1, 16, 8192, 0) == 4         # 64 items over 8,192 keys
    assert f(128, 1, 16, 32768, 0) == 16       # never more than 16 runs
    assert f(512, 1, 16, 32768, 4096) == 2     # a window bounds the keys a query sees
    assert f(0, 1, 16, 8192, 0) == 1 and f(512, 1, 16, 0, 0) == 1
    for tokens in (2, 70, 128, 300, 512, 1024, 4096):
        for heads in (1, 4, 16, 28, 64):
            for keys in (64, 1000, 4096, 20000, 131072):
                n = f(tokens, 1, heads, keys, 0)
                assert 1 <= n <= 16
                assert n == 1 or keys // n >= 2048          # a run keeps at least 2,048 keys
                assert n == 1 or n * heads * ((tokens + 127) // 128) <= 2 * 148


def test_decode_attention_splits_are_bounded_and_follow_the_context(lib):
    for pick in (lib.ix_attn_decode_tma_splits, lib.ix_attn_decode_splits):
        for batch in (1, 2, 8, 22, 64, 256):
            last = 0
            for ctx in (1, 64, 500, 4096, 32768, 262144):
                n = pick(batch, 16, 16, ctx)                # (sequences, heads, kv heads, keys)
                assert 1 <= n <= 256
                assert n == 1 or n * 64 <= max(ctx, 64) * 2  # no run much shorter than a tile
                assert n >= last or batch >= 20             # more keys, not fewer runs
                last = n
        # one sequence needs many runs to fill the device, 64 sequences hardly any
        assert pick(1, 16, 16, 32768) >= 8 > pick(64, 16, 16, 32768)


def test_recurrence_is_cut_into_segments_only_for_long_portions():
    f = ops.recurrence_segments                # (longest portion, sequences, heads, value size)
    assert f(1, 64, 32, 64) == (0, 1) and f(127, 1, 4, 64) == (0, 1)      # walked end to end
    assert f(2048, 1, 32, 64) == (128, 16)     # 64 (head, value tile) items x 16 segments
    assert f(4096, 1, 32, 64) == (256, 16)
    assert f(300, 64, 32, 64) == (0, 1)        # many sequences fill the device themselves
    for tokens in (128, 129, 500, 1119, 5000, 100000):
        for seqs in (1, 3, 16):
            for heads in (1, 4, 32):
                seg_len, nseg = f(tokens, seqs, heads, 64)
                if nseg == 1:
                    assert seg_len == 0
                    continue
                assert seg_len >= 64 and seg_len % 16 == 0 and 2 <= nseg <= 64
                assert (nseg - 1) * seg_len < tokens <= nseg * seg_len    # the segments cover it


def test_no_kernel_reads_per_request_state_ahead_of_its_wait():
    """A kernel that may come onto the device while its predecessor still computes reads no state,
    and no table that says whose it is, before it has waited: the predecessor may be what writes it."""
    seen = 0
    for path in library.sources() + library._headers():
        with open(path) as f:
            text = re.sub(r"//[^\n]*|__launch_bounds__\([^)]*\)", "", f.read())
        for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\(([^{}]*?)\)\s*\{", text):
            body = text[m.end():]
            wait = body.find("IX_PDL_WAIT();")
            following = body.find("__global__")
            if wait < 0 or (0 <= following < wait):
                continue                                   # launched the ordinary way
            seen += 1
            ahead = re.findall(r"\b(?:state|state_slot|cu_q|st)\b\s*\[|\bstate\s*\+", body[:wait])
            assert not ahead, f"{os.path.basename(path)}: {m.group(1)} reads {ahead}"
    assert seen > 80


def test_one_block_routes_no_more_than_one_block_dispatches(lib):
    """Selection and tables by one block only where the tables alone are one block's too."""
    f = lib.ix_router_dispatch_applies                     # (tokens, experts, chosen)
    assert f(1, 60, 4) and f(32, 60, 4) and f(32, 256, 8) and f(16, 300, 32) and not f(32, 32, 16)
    assert not f(17, 300, 32) and not f(32, 64, 32) and not f(33, 60, 4) and not f(0, 60, 4)
    for tokens in range(1, 33):
        for experts in (8, 60, 300, 384):
            for chosen in (1, 2, 8, 17, 32):
                if f(tokens, experts, chosen):
                    assert lib.ix_moe_dispatch_scratch_ints(tokens, experts, chosen) == 0


def test_widened_attention_gives_a_block_one_query_tile_while_sms_are_free(lib):
    f = lib.ix_widened_attention_tiles          # (tokens, sequences, heads, rows a sequence, window)
    assert f(2048, 1, 16, 2048, 0) == 1 and f(300, 1, 16, 2304, 0) == 1 and f(3000, 1, 8, 3008, 1024) == 1
    assert f(1500, 1, 32, 1536, 0) == 2         # one round of long walks either way
    assert f(1200, 4, 16, 512, 0) == 2          # 192 blocks would be two rounds
    assert f(60000, 8, 128, 8192, 0) == 2 and f(1 << 30, 1, 128, 1 << 20, 0) == 2
    for tokens in (1, 100, 128, 129, 1000, 4096):
        for seqs in (1, 3, 200):
            for window in (0, 1, 512):
                assert f(max(tokens, seqs), seqs, 16, 4096, window) in (1, 2)
