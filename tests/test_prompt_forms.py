"""Rules by which prompts take the forms made for them: what they promise the kernels, over shapes
drawn at random (no device)."""
import ctypes
import random

import pytest

from inferx_b200.kernels import library, ops


def test_widened_rows_hold_every_visible_key():
    rng = random.Random(1)
    taken = 0
    for _ in range(3000):
        S = rng.randint(1, 6)
        q_lens = [rng.choice([2, 33, 64, 200, 1000, 3000]) for _ in range(S)]
        starts = [rng.randint(0, 6000) for _ in range(S)]
        window = rng.choice([0, 0, 1, 64, 100, 4096])
        slack = rng.choice([0, 17, 4000])             # a recorded step's bound lies above
        heads, rank = rng.choice([(8, 256), (16, 512), (32, 512), (128, 512)])
        bound = max(a + n for a, n in zip(starts, q_lens)) + slack
        rows = ops.widened_latent_rows(q_lens, bound, window, heads, rank, 64, 320,
                                       mixed=rng.random() < 0.3)
        if not rows:
            continue
        taken += 1
        assert rows % 64 == 0 and S * rows * heads * 320 * 2 <= ops.WIDENED_MAX_BYTES
        for n, a in zip(q_lens, starts):
            base = max(0, a - window + 1) // 64 * 64 if window else 0
            assert rows >= a + n - base
    assert taken > 500


def test_widened_form_is_for_many_queries():
    rows = lambda q, kv, **k: ops.widened_latent_rows(q, kv, 0, 16, 512, 64, 320, **k)
    assert rows([3000], 3000) and rows([1500], 9692) and rows([128], 640)
    assert not rows([33], 8225) and not rows([2], 4098) and not rows([], 100)
    assert not rows([3000], 3000000)                  # more than the buffer may take


@pytest.mark.parametrize("new,before,bound,mixed,widened", [
    # a recorded step's bound is a table width rounded up to a power of two: just above an edge the
    # folded form walks half of it, while the widened form pays for all of it
    (128, 1000, 2048, False, False), (128, 2020, 4096, False, False),
    (128, 4000, 8192, False, False), (128, 8192, 16384, False, False),
    (128, 16380, 32768, False, False), (64, 4200, 8192, False, False),
    (256, 2020, 4096, False, False), (256, 8192, 16384, False, False),
    # the bound is a decoding sequence's
    (256, 1000, 2048, True, False), (128, 0, 4096, True, False), (64, 0, 8192, True, False),
    # and where the widened form is far ahead it stays
    (700, 0, 1024, False, True), (700, 2020, 4096, False, True), (700, 16380, 32768, False, True),
    (3000, 0, 4096, False, True), (1024, 8192, 16384, False, True)])
def test_a_bound_is_not_taken_for_a_length(new, before, bound, mixed, widened):
    """16 heads of 128 + 64 over a latent of 512, measured in recorded steps both ways."""
    assert new + before <= bound
    rows = ops.widened_latent_rows([new], bound, 0, 16, 512, 64, 320, mixed=mixed, bound=True)
    assert rows == (bound if widened else 0)


def test_exact_lengths_decide_where_they_are_known():
    rows = lambda own: ops.widened_latent_rows([200, 200], 8192, 0, 16, 512, 64, 320, kv_lens=own)
    assert rows([8192, 8192]) and not rows([8192, 200])


@pytest.mark.parametrize("delta", [True, False])
@pytest.mark.parametrize("K", [16, 64, 65, 128, 129, 256, 257, 512])
def test_segments_fill_the_device_once(delta, K):
    """Blocks of the pass that the segments are counted for stay within what 148 SMs hold: five an SM
    by registers up to keys of 64, beyond that by two stages of 16 tokens in 228 KB."""
    f = getattr(library.load(), "ix_delta_recurrence_segments" if delta
                else "ix_linear_recurrence_segments")
    pitch = next(p for p in (32, 64, 128, 256, 512) if K <= p)
    cols = 16 * (4 if K <= 128 else 2 if K <= 256 else 1)
    smem = 2 * 4 * (3 * 16 * pitch + 16 * cols + (32 if delta else 0))
    most = 148 * min(5 if K <= 64 else 3, 228 * 1024 // (smem + 1024))
    taken = 0
    for H in (1, 2, 3, 5, 8, 16, 30):
        for V in (8, 64, 128, 256):
            seg = ctypes.c_int(0)
            n = f(1, H, K, V, 20000, 128, 64, ctypes.byref(seg))
            tiles = -(-V // cols) + (-(-K // cols) if delta else 0)
            taken += n > 1
            if K > 256 and not delta and n == 2:
                continue                # (two segments whatever the device holds: next test)
            assert n == 1 or (n - 1 if delta else n) * H * tiles <= most
    assert taken


def test_segments_where_they_pay():
    def count(entry, S, H, K, V, longest):
        return getattr(library.load(), entry)(S, H, K, V, longest, 128, 64,
                                              ctypes.byref(ctypes.c_int(0)))
    # two segments of a few dozen tokens on a full device: one pass from end to end
    assert count("ix_delta_recurrence_segments", 1, 64, 128, 128, 200) == 1
    assert count("ix_delta_recurrence_segments", 4, 16, 96, 128, 128) == 1
    assert count("ix_delta_recurrence_segments", 1, 64, 128, 128, 256) == 2
    assert count("ix_delta_recurrence_segments", 4, 16, 64, 128, 128) == 2
    # large keys: the walk from end to end of the linear recurrence is the slower one
    assert count("ix_linear_recurrence_segments", 1, 16, 384, 128, 3000) == 2
    assert count("ix_linear_recurrence_segments", 4, 64, 512, 256, 128) == 2


@pytest.mark.parametrize("q_lens,first,seqs,busy", [
    ([1024] + [8] * 32, 0, 33, 2), ([128] * 4, 0, 4, 4), ([1] * 32 + [256], 32, 1, 1),
    ([1] * 200 + [2000, 100], 200, 2, 2), ([1, 1, 300, 2], 0, 4, 2), ([700], 0, 1, 1)])
def test_segments_are_counted_by_the_tokens_there_are(q_lens, first, seqs, busy):
    """One long prompt among short ones is not one of as many."""
    from types import SimpleNamespace
    step = SimpleNamespace(num_seqs=len(q_lens), max_q_len=max(q_lens), cu_q_prompt=object(),
                           num_decode_seqs=sum(n == 1 for n in q_lens))
    assert ops._segmented_part(step, sum(q_lens)) == (first, seqs, busy, max(q_lens))


def test_segments_do_not_share_scratch():
    """Cells of scratch as the segmented recurrences number them."""
    rng = random.Random(4)
    for _ in range(1000):
        L = 16 * rng.randint(4, 40)
        q = [rng.choice([1, 2, L, rng.randint(1, 3000)]) for _ in range(rng.randint(1, 40))]
        begin, cells = 0, []
        for s, n in enumerate(q):
            cells += [begin // L + s + e for e in range(-(-n // L))]
            begin += n
        assert len(set(cells)) == len(cells) and max(cells) < begin // L + len(q) + 1


def test_chunked_state_space_leaves_what_it_cannot_hold_to_the_walk():
    pay = lambda q, heads=64, K=128, V=64: ops._ssd_chunks_pay(sum(q), len(q), heads, K, V, q)
    assert pay([64]) and pay([2048]) and pay([65, 128]) and pay([129, 2, 15], 4) and pay([64] * 100)
    # heads x portions beyond a grid's 65,535
    assert pay([64] * 511, 128, 8, 8) and not pay([64] * 512, 128, 8, 8)
    # scratch beyond its bound: 32 KB of state a head and chunk
    assert pay([16384]) and not pay([65536]) and not pay([64] * 1000)
    # many portions of a few tokens beside one long enough
    assert not pay([64] + [8] * 32) and not pay([256] + [8] * 128) and pay([64] + [32] * 32)


def test_chunked_state_space_scratch_stays_below_its_bound():
    rng = random.Random(3)
    for _ in range(2000):
        q = [rng.choice([2, 30, 64, 300, 5000, 60000]) for _ in range(rng.choice([1, 4, 300]))]
        heads, N, V = rng.choice([(16, 128, 64), (64, 128, 64), (128, 256, 128), (3, 8, 8)])
        if not ops._ssd_chunks_pay(sum(q), len(q), heads, N, V, q):
            continue
        cells = sum(-(-n // 64) for n in q)
        assert cells * heads * N * V * 4 <= ops.SSD_MAX_SCRATCH_BYTES and heads * len(q) <= 65535


@pytest.mark.parametrize("dim,rot,vdim,rank,takes", [
    (128, 64, 128, 512, True), (96, 32, 128, 256, True), (48, 16, 64, 64, True),
    (128, 0, 128, 128, True),
    # latents and rotated parts of the general form: it keeps what it computes in 32 bits
    (128, 64, 128, 384, False), (128, 64, 128, 96, False), (128, 64, 128, 1024, False),
    (120, 8, 128, 512, False), (104, 24, 64, 256, False),
    (100, 64, 128, 512, False)])                      # no width of the kernel's
def test_widened_form_leaves_the_general_forms_sizes_alone(dim, rot, vdim, rank, takes):
    import torch
    assert ops.widened_latent_applies(torch.bfloat16, dim, rot, vdim, rank, (512, 1024)) is takes
    assert not ops.widened_latent_applies(torch.float32, dim, rot, vdim, rank, (512, 1024))


@pytest.mark.parametrize("M,N,K", [(17, 8, 8), (600, 2048, 5632), (40, 1024, 2048), (1, 1, 8),
                                   (800, 22016, 4096), (65, 3, 4096), (333, 1000, 1032)])
def test_fp32_runs_are_never_empty(M, N, K):
    splits = library.load().ix_gemm_fp32_tc_splits(M, N, K)
    steps = -(-K // 64)
    per = -(-steps // splits)
    assert 1 <= splits <= 16 and per * (splits - 1) < steps


@pytest.mark.parametrize("rows,cols,k,pays", [
    (17, 2048, 2048, True), (600, 11264, 2048, True), (64, 4096, 192, True), (600, 4096, 128, True),
    # the tiles on the CUDA cores are ahead
    (64, 64, 64, False), (64, 4096, 128, False), (600, 4096, 96, False), (2048, 11264, 64, False),
    (17, 8, 8, False),
    (17, 65535 * 128 + 1, 2048, False)])              # columns beyond its grid
def test_fp32_products_take_the_faster_form(rows, cols, k, pays):
    assert ops._fp32_tc_pays(rows, cols, k) is pays


@pytest.mark.parametrize("entry", ["ix_delta_recurrence_segments", "ix_linear_recurrence_segments"])
def test_segments_cover_the_longest_sequence(entry):
    f = getattr(library.load(), entry)
    rng = random.Random(2)
    for _ in range(2000):
        S, H = rng.randint(1, 40), rng.choice([1, 8, 16, 64])
        K, V = rng.choice([7, 16, 64, 100, 128, 256, 512]), rng.choice([8, 64, 128, 333])
        longest, most = rng.randint(1, 20000), rng.choice([2, 64])
        seg = ctypes.c_int(-1)
        n = f(S, H, K, V, longest, 128, most, ctypes.byref(seg))
        if n == 1:
            assert seg.value == 0
            continue
        assert longest >= 128 and 2 <= n <= most and seg.value >= 64 and seg.value % 16 == 0
        assert (n - 1) * seg.value < longest <= n * seg.value
