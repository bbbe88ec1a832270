"""fp32 attention of prompts in bfloat16 terms against 64 bits, beside the CUDA-core kernel."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops():
    from inferx_b200.kernels import ops
    return ops


def _case(q_lens, starts, heads, kvh, hd, vd, page, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    need = [-(-(a + n) // page) for a, n in zip(starts, q_lens)]
    P, T = sum(need) + 2, sum(q_lens)
    perm = torch.randperm(P, generator=torch.Generator().manual_seed(seed)).to(torch.int32)
    bt = torch.full((len(q_lens), max(need) + 1), -1, dtype=torch.int32)
    at = 0
    for s, n in enumerate(need):
        bt[s, :n] = perm[at:at + n]
        at += n
    rand = lambda *shape: torch.randn(shape, generator=g, device="cuda")
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32)
    seq = torch.repeat_interleave(torch.arange(len(q_lens)), torch.tensor(q_lens)).to(torch.int32)
    pos = torch.cat([torch.arange(a, a + n) for a, n in zip(starts, q_lens)]).to(torch.int32)
    return dict(q=rand(T, heads, hd), k=rand(P, kvh, page, hd), v=rand(P, kvh, page, vd),
                bt=bt.cuda(), cu=cu.cuda(), pos0=torch.tensor(starts, dtype=torch.int32).cuda(),
                seq=seq.cuda(), pos=pos.cuda(), q_lens=q_lens, starts=starts)


def _exact(c, window, scale, softcap, keep, sink):
    out, t = [], 0
    group = c["q"].shape[1] // c["k"].shape[1]
    for s, (n, a) in enumerate(zip(c["q_lens"], c["starts"])):
        rows = lambda x: x.double()[c["bt"][s].clamp(min=0).long()].transpose(1, 2).reshape(
            -1, x.shape[1], x.shape[3])[:a + n].repeat_interleave(group, 1)
        sc = torch.einsum("qhd,khd->hqk", c["q"][t:t + n].double(), rows(c["k"])) * scale
        if softcap > 0:
            sc = softcap * torch.tanh(sc / softcap)
        qp = torch.arange(a, a + n, device="cuda")[:, None]
        kp = torch.arange(a + n, device="cuda")[None]
        seen = kp <= qp
        if window > 0:
            seen &= (kp > qp - window) | (kp < keep)
        sc = sc.masked_fill(~seen, -math.inf)
        if sink is not None:
            sc = torch.cat([sc, sink.double()[:, None, None].expand(-1, n, 1)], 2)
        p = torch.softmax(sc, 2)[:, :, :a + n]
        out.append(torch.einsum("hqk,khd->qhd", p, rows(c["v"])))
        t += n
    return torch.cat(out)


def _off(a, ref):
    return float((a.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("hd,vd", [(128, 128), (64, 64), (128, 64), (64, 128)])
@pytest.mark.parametrize("q_lens,starts,heads,kvh,page,window,softcap,keep,sunk", [
    ([1, 64, 130], [70, 0, 31], 4, 2, 16, 0, 0.0, 0, False),       # edges of query and key tiles
    ([600], [0], 4, 1, 16, 0, 0.0, 0, False),
    ([200, 33], [150, 5], 2, 2, 5, 40, 0.0, 0, False),             # a window shorter than a tile
    ([257], [300], 2, 1, 64, 128, 0.0, 70, True),                  # kept first keys, a sink
    ([90], [0], 3, 3, 8, 1, 20.0, 0, False),                       # one key, squashed scores
])
def test_against_64_bits(hd, vd, q_lens, starts, heads, kvh, page, window, softcap, keep, sunk):
    ops = _ops()
    c = _case(q_lens, starts, heads, kvh, hd, vd, page, hd + vd + window)
    c["q"] *= 4.0                                       # attention that is sharp in places
    sink = torch.randn(heads, device="cuda") if sunk else None
    args = (window, hd ** -0.5, softcap, keep, sink)
    ref = _exact(c, *args)
    got = ops.paged_attention_tiled(c["q"], c["k"], c["v"], c["bt"], c["cu"], c["pos0"], *args)
    plain = ops.paged_attention_generic(c["q"], c["k"], c["v"], c["bt"], c["seq"], c["pos"], *args)
    # a score's rounding is some 2^-24 of sum |q k| in either; 2^-22 covers a walk of few keys
    assert _off(got, ref) <= max(1.1 * _off(plain, ref), 2.0 ** -22)


def test_a_query_does_not_depend_on_the_cut():
    ops = _ops()
    c = _case([300], [0], 2, 1, 128, 128, 16, 3)
    args = (0, 0.09)
    whole = ops.paged_attention_tiled(c["q"], c["k"], c["v"], c["bt"], c["cu"], c["pos0"], *args)
    for cut in (1, 37, 64, 200):
        i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
        rest = ops.paged_attention_tiled(c["q"][cut:].contiguous(), c["k"], c["v"], c["bt"],
                                         i32(0, 300 - cut), i32(cut), *args)
        assert torch.equal(rest, whole[cut:])


def test_infinities_nan_and_numbers_without_a_third_term():
    """Where a query sees a key or a value that is not finite its result is what fp32 arithmetic
    gives; the others are untouched, and results below 2^-64 keep their precision."""
    ops = _ops()
    c = _case([200], [0], 2, 2, 64, 64, 16, 9)

    def put(name, key, head, dim, value):
        c[name][int(c["bt"][0, key // 16]), head, key % 16, dim] = value
    put("k", 150, 0, 3, math.inf)
    put("v", 190, 1, 5, math.nan)
    put("v", 180, 1, 7, -math.inf)
    put("v", 100, 1, 9, 3.4e38)                          # its first term rounds up to infinity
    args = (0, 0.125)
    got = ops.paged_attention_tiled(c["q"], c["k"], c["v"], c["bt"], c["cu"], c["pos0"], *args)
    plain = ops.paged_attention_generic(c["q"], c["k"], c["v"], c["bt"], c["seq"], c["pos"], *args)
    assert torch.equal(got.isnan(), plain.isnan()) and torch.equal(got.isinf(), plain.isinf())
    fine = plain.isfinite()
    torch.testing.assert_close(got[fine], plain[fine], rtol=1e-4, atol=1e-5)
    c = _case([100], [0], 1, 1, 128, 128, 16, 10)
    c["v"] *= 1e-36
    got = ops.paged_attention_tiled(c["q"], c["k"], c["v"], c["bt"], c["cu"], c["pos0"], *args)
    plain = ops.paged_attention_generic(c["q"], c["k"], c["v"], c["bt"], c["seq"], c["pos"], *args)
    assert float((got - plain).double().norm()) <= 1e-5 * float(plain.double().norm())


@pytest.mark.parametrize("hd,vd", [(64, 64), (128, 128)])
@pytest.mark.parametrize("what", ["queries", "keys", "weights"])
def test_operands_without_three_terms_that_meet_great_ones(what, hd, vd):
    """Queries or keys below 2^-102 against great partners, weights of e^-87 on great values: scores
    and results of ordinary size keep fp32's precision, what a chain of hd multiply-adds has (a
    weight's relative error is that of its score of 87)."""
    ops = _ops()
    c = _case([150], [20], 2, 1, hd, vd, 16, hd)
    bound = hd ** 0.5 * 2.0 ** -24
    if what == "weights":             # the first key's score is 87, the others' nearly 0
        first = int(c["bt"][0, 0])
        u = c["q"][0, 0].clone()
        c["q"] = u.expand_as(c["q"]).contiguous()
        c["k"] *= 1e-3
        c["k"][first, :, 0] = 87.0 * u / u.square().sum() * hd ** 0.5
        c["v"] *= 2.0 ** 118
        c["v"][first, :, 0] = 0.0
        bound *= 87.0
    else:
        small, great = ("q", "k") if what == "queries" else ("k", "q")
        c[small] *= 2.0 ** -122
        c[great] *= 2.0 ** 122
    args = (0, hd ** -0.5, 0.0, 0, None)
    got = ops.paged_attention_tiled(c["q"], c["k"], c["v"], c["bt"], c["cu"], c["pos0"], *args)
    assert _off(got, _exact(c, *args)) <= bound


def test_a_row_is_made_again_by_what_it_sees():
    """Great entries change no bit of a row that does not see them."""
    ops = _ops()
    c = _case([200], [0], 2, 2, 64, 128, 16, 4)
    call = lambda: ops.paged_attention_tiled(c["q"], c["k"], c["v"], c["bt"], c["cu"], c["pos0"],
                                             40, 0.125)
    before = call()
    c["k"][int(c["bt"][0, 90 // 16]), 0, 90 % 16, 5] = 2.0 ** 90
    c["v"][int(c["bt"][0, 120 // 16]), 1, 120 % 16, 7] = 2.0 ** 40
    c["q"][170, 1, 3] = 2.0 ** 90
    after = call()
    seen = torch.zeros(200, 2, dtype=torch.bool)
    seen[90:130, 0] = seen[120:160, 1] = seen[170, 1] = True
    assert torch.equal(after.cpu()[~seen], before.cpu()[~seen])
    assert not torch.equal(after.cpu()[seen], before.cpu()[seen])
    plain = ops.paged_attention_generic(c["q"], c["k"], c["v"], c["bt"], c["seq"], c["pos"], 40, 0.125)
    torch.testing.assert_close(after, plain, rtol=1e-4, atol=1e-5)
