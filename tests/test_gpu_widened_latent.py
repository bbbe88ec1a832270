"""Latent attention over widened keys and values: the kernels alone against plain statements,
and the mixer's widened form against its folded one and against 32-bit arithmetic."""
import math
from types import SimpleNamespace

import pytest
import torch

import host_ops
from inferx_b200.kernels import library
from test_gpu_dominex import _cuda, _step

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _ops():
    from inferx_b200.kernels import ops
    return ops


def _pages(lens, page, g):
    maxb = max(-(-n // page) for n in lens)
    bt = torch.full((len(lens), maxb), -1, dtype=torch.int32)
    perm, k = torch.randperm(sum(-(-n // page) for n in lens) + 2, generator=g), 0
    for s, n in enumerate(lens):
        for b in range(-(-n // page)):
            bt[s, b] = perm[k]
            k += 1
    return bt, perm.numel()


@pytest.mark.parametrize("page,window,width", [(4, 0, 72), (16, 100, 576), (8, 64, 40)])
def test_collect(page, window, width):
    g = torch.Generator().manual_seed(width)
    q_lens, starts = [3, 70, 200], [0, 130, 5]
    st = _step(q_lens, starts)
    bt, P = _pages([a + n for a, n in zip(starts, q_lens)], page, g)
    cache = torch.randn(P, 1, page, width, generator=g).to(BF)
    rows = 320
    base = [max(0, a - window + 1) // 64 * 64 if window else 0 for a in starts]
    for s, b in enumerate(base):               # pages the window has passed may be gone
        bt[s, :b // page] = -1
    got = _ops().latent_collect(cache.cuda(), bt.cuda(), st.q_pos0.cuda(), st.kv_len.cuda(), rows,
                                window).cpu().view(len(q_lens), rows, width)
    want = torch.zeros_like(got)
    for s in range(len(q_lens)):
        for r in range(rows):
            p = base[s] + r
            if p < int(st.kv_len[s]):
                want[s, r] = cache[bt[s, p // page], 0, p % page]
    assert torch.equal(got, want)


@pytest.mark.parametrize("H,dn,dr,rot_dims,rank", [(3, 24, 16, 16, 40), (16, 128, 64, 64, 512),
                                                  (2, 64, 0, 0, 24), (5, 8, 24, 8, 64)])
def test_front_in_place(H, dn, dr, rot_dims, rank):
    g = torch.Generator().manual_seed(rank)
    T, page, P = 9, 4, 30
    pos = torch.tensor([0, 1, 2, 3, 900, 61, 62, 63, 7], dtype=torch.int32)
    kv_off = H * (dn + dr)
    proj = torch.randn(T, kv_off + rank + dr + 8, generator=g).to(BF)
    freq, gain = torch.rand(rot_dims // 2, generator=g), 1.0 + 0.2 * torch.randn(rank, generator=g)
    slots = torch.randperm(P * page, generator=g)[:T].to(torch.int32)
    cache = torch.zeros(P, 1, page, rank + dr, dtype=BF)
    want = cache.clone()
    rot, plain = host_ops.latent_prepare(proj, 0, kv_off, pos, freq, 1.3, gain, 1e-5, H, dn, dr,
                                         rot_dims, rank, want, slots)
    p, c = proj.cuda(), cache.cuda()
    _ops().latent_front_inplace(p.view(-1), p.shape[1], p.view(-1)[kv_off:], p.shape[1], pos.cuda(),
                                freq.cuda(), 1.3, gain.cuda(), 1e-5, H, dn, dr, rot_dims, rank, c,
                                slots.cuda())
    q = p.cpu()[:, :kv_off].view(T, H, dn + dr)
    tol = dict(rtol=1.6e-2, atol=1.6e-2)
    assert torch.equal(q[..., :dn].transpose(0, 1), plain)
    torch.testing.assert_close(q[..., dn:].float(), rot.float(), **tol)
    assert torch.equal(p.cpu()[:, kv_off:], proj[:, kv_off:])
    torch.testing.assert_close(c.cpu().float(), want.float(), **tol)


# edges: of the 64-key tile, of the 128-query tile, of the 256 queries a block owns; windows
# that cut a tile; several sequences behind contexts; more key tiles than ring stages
@pytest.mark.parametrize("dk,dv", [(64, 64), (64, 128), (128, 64), (128, 128), (192, 64),
                                   (192, 128)])
@pytest.mark.parametrize("q_lens,starts,window", [
    ([2], [0], 0), ([64], [0], 0), ([65, 127], [63, 0], 0), ([128, 129], [0, 200], 0),
    ([256, 257], [1, 511], 0), ([300, 33], [100, 700], 90), ([513], [0], 64), ([70], [640], 1)])
def test_attention(dk, dv, q_lens, starts, window):
    g = torch.Generator().manual_seed(dk + dv + sum(q_lens))
    H, T, S = 3, sum(q_lens), len(q_lens)
    st = _step(q_lens, starts)
    need = max(a + n for a, n in zip(starts, q_lens))
    if window:
        need = min(need, window + max(q_lens) + 63)
    rows = -(-need // 64) * 64
    q = torch.randn(T, H * dk + 8, generator=g).to(BF)
    kv = torch.randn(S * rows, H * (dk + dv), generator=g).to(BF)
    gate = torch.randn(T, H * dv, generator=g).to(BF)
    scale = 2.0 / math.sqrt(dk)
    want = torch.zeros(T, H, dv)
    t0 = 0
    for s, (n, a) in enumerate(zip(q_lens, starts)):
        base = max(0, a - window + 1) // 64 * 64 if window else 0
        m = a + n - base
        k = kv[s * rows:s * rows + m, :H * dk].float().view(m, H, dk)
        v = kv[s * rows:s * rows + m, H * dk:].float().view(m, H, dv)
        sc = torch.einsum("thd,mhd->htm", q[t0:t0 + n, :H * dk].float().view(n, H, dk), k) * scale
        i, j = torch.arange(a, a + n)[:, None], torch.arange(base, a + n)[None]
        seen = (j <= i) & ((i - j < window) if window else torch.ones_like(j <= i))
        want[t0:t0 + n] = torch.einsum("htm,mhd->thd", sc.masked_fill(~seen, -math.inf).softmax(-1),
                                       v)
        t0 += n
    most = float(kv.float().abs().max())
    for gt in (None, gate):
        out = _ops().widened_attention(
            q.cuda().view(-1), q.shape[1], kv.cuda(), st.cu_q.cuda(), st.q_pos0.cuda(), T, H, dk, dv,
            rows, window, scale, None if gt is None else gt.cuda().view(-1), H * dv)
        _ops().check_async_errors()
        ref = want if gt is None else want * torch.sigmoid(gt.float().view(T, H, dv))
        # weights of 16 bits move a mean of values by at most 2^-17 of the largest one, the
        # result's own rounding by 2^-9; scores of some tens of units are fp32 sums, exp2 is
        # good to 2^-22 of them
        bound = most * (2.0 ** -9 + 2.0 ** -17 + 2.0 ** -15)
        assert float((out.cpu().float().view(T, H, dv) - ref).abs().max()) <= bound


@pytest.mark.parametrize("dim,rot,vdim,rank,heads", [(96, 32, 128, 64, 4), (128, 64, 128, 128, 3)])
@pytest.mark.parametrize("q_rank,own,gated,exact", [(0, True, True, False), (40, True, False, True),
                                                    (48, False, False, False)])
@pytest.mark.parametrize("window", [0, 150])
def test_mixer_forms_agree(dim, rot, vdim, rank, heads, q_rank, own, gated, exact, window):
    """The same mixed batch (single tokens far into their sequences, portions behind contexts)
    through the folded and the widened form, both against 32-bit arithmetic."""
    from inferx_b200.parts.latent_attention import LatentAttentionMixer
    from inferx_b200.parts.specs import LatentAttentionSpec
    ops = _ops()
    g = torch.Generator().manual_seed(rank + window + q_rank)
    hidden, page = 64, 16
    spec = LatentAttentionSpec(hidden=hidden, heads=heads, dim=dim, rot_dim=rot, vdim=vdim,
                               kv_rank=rank, scale=1.0 / math.sqrt(dim + rot), window=window,
                               position=None, latent_eps=1e-6, output_gate=gated, q_rank=q_rank,
                               own_records=own, fp32_weights=exact)
    q_lens, starts = [1, 1, 90, 300], [500, 3, 250, 0]
    st = _step(q_lens, starts)
    lens = [a + n for a, n in zip(starts, q_lens)]
    bt, P = _pages(lens, page, g)
    slots = torch.tensor([int(bt[s, p // page]) * page + p % page
                          for s, (n, a) in enumerate(zip(q_lens, starts)) for p in range(a, a + n)],
                         dtype=torch.int32)
    x = torch.randn(st.num_tokens, hidden, generator=g)
    cache = torch.randn(P, 1, page, rank + rot, generator=g)

    def run(dtype, widened):
        mixer = LatentAttentionMixer(spec, SimpleNamespace(ops=ops, dtype=dtype), "m")
        gw = torch.Generator().manual_seed(5)
        w = {d.name: (torch.randn(d.shape, generator=gw) * d.shape[-1] ** -0.5 if len(d.shape) == 2
                      else 1 + 0.1 * torch.randn(d.shape, generator=gw)) for d in mixer.tensors()}
        w = {k: (v.to(BF).to(dtype) if v.dim() == 2 else v).cuda() for k, v in w.items()}
        mixer.bind(w)
        if not widened:
            mixer.kv_w = None
        elif mixer.kv_w is None:
            pytest.fail("the widened form does not take these sizes")
        records = cache.to(BF).to(dtype).cuda()
        step = _cuda(st)
        step.groups = [SimpleNamespace(block_table=bt.cuda(), slots=slots.cuda())]
        before = ops.widened_latent_rows
        if widened:
            need = max(lens) if not window else min(max(lens), window + max(q_lens) + 63)
            ops.widened_latent_rows = lambda *a, **k: -(-need // 64) * 64
        try:
            out = mixer.forward(x.to(BF).to(dtype).cuda(), step,
                                SimpleNamespace(group=0, pages={"latent": records}, writes=True))
        finally:
            ops.widened_latent_rows = before
        ops.check_async_errors()
        return out.float().cpu(), records.float().cpu()

    exact32, rec32 = run(torch.float32, False)
    folded, rec_f = run(BF, False)
    widened, rec_w = run(BF, True)
    scale = float(exact32.norm())
    off_f, off_w = float((folded - exact32).norm()) / scale, float((widened - exact32).norm()) / scale
    # either form rounds every stored value once to 8 bits; the widened one is held to what
    # the folded one shows here (two roundings of a quarter more each would still pass)
    assert off_w <= 1.25 * off_f and off_f < 0.02, (off_f, off_w)
    assert torch.equal(rec_f, rec_w)


def test_a_scale_that_is_not_positive_keeps_the_folded_form():
    from inferx_b200.parts.latent_attention import LatentAttentionMixer
    from inferx_b200.parts.specs import LatentAttentionSpec
    for scale, widened in ((0.1, True), (0.0, False), (-0.1, False)):
        spec = LatentAttentionSpec(hidden=64, heads=2, dim=64, rot_dim=64, vdim=64, kv_rank=64,
                                   scale=scale, window=0, position=None, latent_eps=1e-6)
        mixer = LatentAttentionMixer(spec, SimpleNamespace(ops=_ops(), dtype=BF), "m")
        mixer.bind({d.name: torch.ones(d.shape, device="cuda",
                                       dtype=BF if len(d.shape) == 2 else torch.float32)
                    for d in mixer.tensors()})
        assert (mixer.kv_w is not None) == widened


@pytest.mark.parametrize("H,dn,dr,rank,vdim", [(3, 48, 16, 64, 64), (16, 128, 64, 512, 128),
                                               (5, 96, 32, 128, 128), (2, 64, 0, 64, 64)])
def test_keys_are_two_terms(H, dn, dr, rank, vdim):
    g = torch.Generator().manual_seed(dn + rank)
    rows, lo = 130, {64: 64, 128: 128, 192: 128}[dn + dr]
    rec = torch.randn(rows, rank + dr, generator=g).to(BF).cuda()
    rec[100:] = 0                               # rows past a sequence's end
    uk = (torch.randn(H * dn, rank, generator=g) * rank ** -0.5).to(BF).cuda()
    uv = (torch.randn(H, vdim, rank, generator=g) * rank ** -0.5).to(BF).cuda()
    kv = _ops().latent_widen(rec, rank, uk, uv, H, dn)
    hi, second, v = kv.split([H * (dn + dr), H * lo, H * vdim], dim=1)
    hi, second = hi.view(rows, H, dn + dr), second.view(rows, H, lo)
    want = (rec[:, :rank].double() @ uk.double().T).view(rows, H, dn)
    got = hi[..., :dn].double() + second[..., :dn].double()
    # two roundings to 8 bits, and the product's own fp32 sums
    assert float((got - want).norm() / want.norm()) <= 2.0 ** -16
    assert float((hi[..., :dn].double() - want).norm() / want.norm()) >= 2.0 ** -11
    assert torch.equal(hi[..., dn:], rec[:, None, rank:].expand(rows, H, dr))
    assert not second[..., dn:].any() and not kv[100:].any()
    want_v = (rec[:, :rank].double() @ uv.double().view(H * vdim, rank).T)
    assert float((v.double() - want_v).norm() / want_v.norm()) <= 2.0 ** -8


@pytest.mark.parametrize("dk,dv,second", [(64, 64, 48), (128, 128, 96), (128, 64, 128),
                                          (192, 128, 128), (192, 64, 176)])
@pytest.mark.parametrize("exact", [True, False])
def test_second_key_terms_reach_the_scores(dk, dv, second, exact):
    """Keys whose first terms are all alike: the second ones alone tell them apart."""
    g = torch.Generator().manual_seed(dk + second)
    H, q_lens, starts = 2, [3, 140, 300], [500, 70, 0]
    st = _step(q_lens, starts)
    rows, T, lo = 512, sum(q_lens), dk if dk < 192 or second > 128 else 128
    q = (4.0 * torch.randn(T, H * dk, generator=g)).to(BF)
    k1 = torch.ones(3 * rows, H, dk).to(BF)
    k2 = torch.zeros(3 * rows, H, lo)
    k2[..., :second] = torch.randn(3 * rows, H, second, generator=g)
    v = torch.randn(3 * rows, H, dv, generator=g).to(BF)
    k2 = k2.to(BF)
    kv = torch.cat([t.reshape(3 * rows, -1) for t in (k1, k2, v)], 1).contiguous()
    scale = 1.0 / math.sqrt(dk)
    out = _ops().widened_attention(q.cuda().view(-1), H * dk, kv.cuda(), st.cu_q.cuda(),
                                   st.q_pos0.cuda(), T, H, dk, dv, rows, 0, scale, second=second,
                                   fp32_weights=exact).cpu().double().view(T, H, dv)
    _ops().check_async_errors()
    key = k1.double()
    key[..., :second] += k2.double()[..., :second]
    t0 = 0
    for s, (n, a) in enumerate(zip(q_lens, starts)):
        sl = slice(s * rows, s * rows + a + n)
        sc = torch.einsum("thd,mhd->htm", q[t0:t0 + n].double().view(n, H, dk), key[sl]) * scale
        seen = torch.arange(a + n)[None] <= torch.arange(a, a + n)[:, None]
        want = torch.einsum("htm,mhd->thd", sc.masked_fill(~seen, -math.inf).softmax(-1),
                            v.double()[sl])
        # a result is a mean of values: rounded once, its weights to 8 or to 16 bits, its scores
        # of some tens in fp32
        most = float(v.double().abs().max())
        bound = most * (2.0 ** -9 + 2.0 ** (-16 if exact else -8) + 2.0 ** -15)
        assert float((out[t0:t0 + n] - want).abs().max()) <= bound
        t0 += n


@pytest.mark.parametrize("heads,dim,rot,rank,q_rank,gated,exact", [
    (4, 128, 64, 512, 0, False, False), (4, 128, 64, 512, 96, False, True),
    (8, 96, 32, 256, 0, True, False)])
@pytest.mark.parametrize("sharp", [1.0, 4.0, 8.0])
@pytest.mark.parametrize("n,before", [(70, 0), (400, 0), (90, 700)])
def test_widened_is_no_further_from_exact_than_folded(heads, dim, rot, rank, q_rank, gated, exact,
                                                      sharp, n, before):
    """However decisive the scores are: rounded keys would weigh most where they are."""
    from inferx_b200.parts.latent_attention import LatentAttentionMixer
    from inferx_b200.parts.specs import LatentAttentionSpec
    ops = _ops()
    hidden, page, L = 256, 16, n + before
    spec = LatentAttentionSpec(hidden=hidden, heads=heads, dim=dim, rot_dim=rot, vdim=128,
                               kv_rank=rank, scale=sharp / math.sqrt(dim + rot), window=0,
                               position=None, latent_eps=1e-6, output_gate=gated, q_rank=q_rank,
                               own_records=True, fp32_weights=exact)
    st = _cuda(_step([n], [before]))
    pages = -(-L // page)
    st.groups = [SimpleNamespace(
        block_table=torch.arange(pages, dtype=torch.int32).view(1, -1).cuda(),
        slots=torch.arange(before, L, dtype=torch.int32).cuda())]
    g = torch.Generator().manual_seed(rank + n)
    x = torch.randn(n, hidden, generator=g).to(BF).cuda()
    cache = torch.randn(pages, 1, page, rank + rot, generator=g).to(BF).cuda()

    def run(dtype, rows):
        mixer = LatentAttentionMixer(spec, SimpleNamespace(ops=ops, dtype=dtype), "m")
        gw = torch.Generator().manual_seed(5)
        w = {d.name: (torch.randn(d.shape, generator=gw) * d.shape[-1] ** -0.5 if len(d.shape) == 2
                      else 1 + 0.1 * torch.randn(d.shape, generator=gw)) for d in mixer.tensors()}
        mixer.bind({k: (v.to(BF).to(dtype) if v.dim() == 2 else v).cuda() for k, v in w.items()})
        before_rule, ops.widened_latent_rows = ops.widened_latent_rows, lambda *a, **k: rows
        try:
            return mixer.forward(x.to(dtype), st, SimpleNamespace(
                group=0, pages={"latent": cache.to(dtype)}, writes=True)).double()
        finally:
            ops.widened_latent_rows = before_rule

    want = run(torch.float32, 0)
    off = [float((run(BF, rows) - want).norm() / want.norm()) for rows in (0, -(-L // 64) * 64)]
    ops.check_async_errors()
    assert off[1] <= off[0], off


@pytest.mark.parametrize("n", [300, 1290])          # (few tiles; walks longer than an SM's share)
@pytest.mark.parametrize("window", [0, 90, 700])
def test_a_row_does_not_depend_on_its_neighbours(window, n):
    """The same query in another company, in a portion that begins elsewhere, beside another
    sequence and with more rows a sequence: the same bits."""
    g = torch.Generator().manual_seed(window)
    H, dk, dv = 2, 128, 128
    rows = -(-n // 64) * 64
    q = torch.randn(n, H * dk, generator=g).to(BF)
    kv = torch.randn(rows, H * (dk + dv), generator=g).to(BF)

    def run(q, start, beside=(), more=0):
        st = _step([q.shape[0], *beside], [start] + [0] * len(beside))
        base = max(0, start - window + 1) // 64 * 64 if window else 0
        own = torch.zeros((1 + len(beside)) * (rows + more), kv.shape[1], dtype=BF)
        own[:rows - base] = kv[base:]
        both = torch.cat([q, q.new_ones(sum(beside), q.shape[1])])
        out = _ops().widened_attention(both.cuda().view(-1), H * dk, own.cuda(), st.cu_q.cuda(),
                                       st.q_pos0.cuda(), both.shape[0], H, dk, dv, rows + more,
                                       window, 0.3)
        _ops().check_async_errors()
        return out.cpu()[:q.shape[0]]

    whole = run(q, 0)
    loud = q.clone()
    loud[::2] *= 30.0                            # every other row's maxima grow all along its keys
    assert torch.equal(run(loud, 0)[1::2], whole[1::2])
    for cut in (1, 64, 129, 200, n - 30):
        assert torch.equal(run(q[cut:].contiguous(), cut), whole[cut:])
    assert torch.equal(run(q, 0, beside=(40,)), whole)
    # as many others as make a block own two query tiles instead of one
    lib, many = library.load(), (3,) * 31 + (1500,) * 64
    assert lib.ix_widened_attention_tiles(n, 1, H, rows, window) == 1
    assert lib.ix_widened_attention_tiles(n + sum(many), 1 + len(many), H, 1536, window) == 2
    assert torch.equal(run(q, 0, beside=many, more=1536 - rows), whole)
    assert torch.equal(run(q[n - 30:].contiguous(), n - 30, beside=(n - 200, 7), more=128),
                       whole[n - 30:])
