"""The state-space recurrence in chunks: against 64 bits beside the walk, at the edges of a
chunk, of the padding and of the batch."""
import pytest
import torch

from test_gpu_dominex import _cuda, _step

pytestmark = pytest.mark.gpu


def _ops():
    from inferx_b200.kernels import ops
    return ops


def _plain64(xbc, dt_raw, dt_bias, a_log, d_skip, state, q_lens, slots, H, V, N, G):
    x, dt_raw, st = xbc.double(), dt_raw.double(), state.double().clone()
    dt = torch.nn.functional.softplus(dt_raw + dt_bias.double(), threshold=1000.0)
    a = torch.exp(-torch.exp(a_log.double()) * dt)
    out, t = torch.zeros(x.shape[0], H, V, dtype=torch.float64, device=x.device), 0
    for n, slot in zip(q_lens, slots):
        S = st[slot]
        for _ in range(n):
            xv = x[t, :H * V].view(H, V)
            B = x[t, H * V:H * V + G * N].view(G, N).repeat_interleave(H // G, 0)
            C = x[t, H * V + G * N:].view(G, N).repeat_interleave(H // G, 0)
            S = a[t][:, None, None] * S + (dt[t][:, None] * B)[:, :, None] * xv[:, None]
            out[t] = torch.einsum("hnv,hn->hv", S, C) + d_skip.double()[:, None] * xv
            t += 1
        st[slot] = S
    return out.view(x.shape[0], H * V), st


def _off(a, ref):
    return float((a.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("H,V,N,G", [(4, 64, 128, 2), (2, 40, 24, 1), (6, 8, 8, 3), (1, 136, 256, 1)])
@pytest.mark.parametrize("q_lens", [[64], [65, 128], [1, 1, 63, 200], [129, 2, 15]])
@pytest.mark.parametrize("spread", [0.5, 3.0])     # of the decays' exponents: near 1, and some at 0
def test_against_64_bits(H, V, N, G, q_lens, spread):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(H + V + sum(q_lens))
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    q_lens = sorted(q_lens, key=lambda n: n != 1)
    S, T = len(q_lens), sum(q_lens)
    step = _cuda(_step(q_lens, [5] * S, slots=list(range(S))[::-1]))
    slots = step.state_slot.tolist()
    xbc, dt = rnd(T, H * V + 2 * G * N).bfloat16(), rnd(T, H).bfloat16()
    bias, a_log, d = rnd(H) - 2.0, spread * rnd(H), rnd(H)
    state = rnd(S + 1, H, N, V)
    ref, st_ref = _plain64(xbc, dt, bias, a_log, d, state, q_lens, slots, H, V, N, G)
    res = {}
    for form in ("chunks", "walk"):
        ops.USE_SSD_CHUNKS = form == "chunks"
        try:
            st = state.clone()
            assert ops._ssd_in_chunks(xbc, xbc.shape[1], st, max(q_lens), N, V) == (
                form == "chunks" and max(q_lens) >= ops.SSD_CHUNK_MIN_TOKENS)
            out = ops.ssd_recurrence(xbc, dt, bias, a_log, d, st, step, H, V, N, G)
        finally:
            ops.USE_SSD_CHUNKS = True
        res[form] = _off(out, ref), _off(st, st_ref)
        assert torch.equal(st[S], state[S])          # a slot of no sequence is untouched
    # 24-bit terms into fp32 sums: no further off than 32-bit arithmetic token by token, or a
    # few units in the last place of a sum of a hundred products
    for c, w in zip(res["chunks"], res["walk"]):
        assert c <= max(w, 4e-7), res


def test_decays_of_zero_and_infinite_rates():
    ops = _ops()
    H, V, N, T = 2, 16, 16, 100
    g = torch.Generator(device="cuda").manual_seed(3)
    xbc = torch.randn(T, H * V + 2 * N, generator=g, device="cuda").bfloat16()
    dt = torch.randn(T, H, generator=g, device="cuda").bfloat16()
    step = _cuda(_step([T], [0]))
    par = (torch.zeros(H, device="cuda"), torch.tensor([20.0, 95.0], device="cuda"),
           torch.ones(H, device="cuda"))
    a, b = (torch.randn(1, H, N, V, generator=torch.Generator(device="cuda").manual_seed(5),
                        device="cuda") for _ in range(2))
    got = ops.ssd_recurrence(xbc, dt, *par, a, step, H, V, N, 1)
    ops.USE_SSD_CHUNKS = False
    try:
        ref = ops.ssd_recurrence(xbc, dt, *par, b, step, H, V, N, 1)
    finally:
        ops.USE_SSD_CHUNKS = True
    torch.testing.assert_close(got, ref, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("H,q_lens", [(2048, [2] * 31 + [64]), (2, [64] + [8] * 40)])
def test_steps_that_are_left_to_the_walk(H, q_lens):
    """Heads x portions beyond one dimension of a grid; portions of a few tokens each."""
    ops = _ops()
    V = N = 8
    g = torch.Generator(device="cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    S, T = len(q_lens), sum(q_lens)
    step = _cuda(_step(q_lens, [5] * S))
    xbc, dt = rnd(T, H * V + 2 * N).bfloat16(), rnd(T, H).bfloat16()
    bias, a_log, d = rnd(H) - 2.0, 0.5 * rnd(H), rnd(H)
    state = rnd(S, H, N, V)
    before = ops.LAUNCHES[0]
    got = state.clone()
    out = ops.ssd_recurrence(xbc, dt, bias, a_log, d, got, step, H, V, N, 1)
    assert ops.LAUNCHES[0] == before + 1                  # one pass: the walk
    ops.USE_SSD_CHUNKS = False
    try:
        want = ops.ssd_recurrence(xbc, dt, bias, a_log, d, state, step, H, V, N, 1)
    finally:
        ops.USE_SSD_CHUNKS = True
    assert torch.equal(out, want) and torch.equal(got, state)


@pytest.mark.parametrize("T", [100, 300])
@pytest.mark.parametrize("what", ["nan in x", "inf in x", "inf in B", "inf in C", "nan in dt",
                                  "inf in the state", "products beyond range"])
def test_infinities_and_nan_stay_where_the_walk_has_them(T, what):
    """Tokens ahead of one keep their results, those after it and the state are infinite or not a
    number where the walk's are."""
    ops = _ops()
    H, V, N = 2, 72, 40
    inner = H * V
    g = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    xbc, dt = rnd(T, inner + 2 * N).bfloat16(), rnd(T, H).bfloat16()
    state = rnd(2, H, N, V)
    t, slot = 70, 1
    if what == "nan in x":
        xbc[t, 5] = float("nan")
    elif what == "inf in x":
        xbc[t, 5], xbc[t + 3, inner - 1] = float("inf"), -float("inf")
    elif what == "inf in B":
        xbc[t, inner + 7] = float("inf")
    elif what == "inf in C":
        xbc[t, inner + N + 7] = -float("inf")
    elif what == "nan in dt":
        dt[t, 1] = float("nan")
    elif what == "inf in the state":
        state[slot, 1, 3, 8] = float("inf")
    else:                                    # x of 1e38 against B of 1e-20: finite in the walk
        xbc[t:, :inner], xbc[t:, inner:inner + N] = 1e38, 1e-20
    step = _cuda(_step([T], [0], slots=[slot]))
    par = (rnd(H) + 1.0, torch.tensor([-3.0, -2.0], device="cuda"), torch.ones(H, device="cuda"))
    a, b = state.clone(), state.clone()
    got = ops.ssd_recurrence(xbc, dt, *par, a, step, H, V, N, 1)
    ops.USE_SSD_CHUNKS = False
    try:
        ref = ops.ssd_recurrence(xbc, dt, *par, b, step, H, V, N, 1)
    finally:
        ops.USE_SSD_CHUNKS = True
    for x, y in ((got, ref), (a, b)):
        assert torch.equal(x.isnan(), y.isnan()) and torch.equal(x.isinf(), y.isinf())
        # a few 2^-24 of the sums either way, of the largest term in them
        fine = y.isfinite()
        torch.testing.assert_close(x[fine], y[fine], rtol=2e-4, atol=2e-5)
    if what.endswith(("x", "B", "C", "dt")):
        assert got[:t].isfinite().all()
