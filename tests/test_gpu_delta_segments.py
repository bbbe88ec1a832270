"""The delta rule in segments at every width of key that has a form of its own, at the edges of a
segment and of the batch, against the plain statement."""
import ctypes

import numpy as np
import pytest
import torch

import host_ops
from test_gpu_dominex import _cuda, _step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,HK,K,V", [(2, 2, 16, 40), (2, 1, 20, 33), (2, 2, 64, 128), (2, 1, 66, 8),
                                      (1, 1, 128, 64), (1, 1, 130, 9), (1, 1, 260, 17)])
@pytest.mark.parametrize("q_lens", [[128], [129, 64], [1, 1, 300, 2]])
def test_segments(dtype, H, HK, K, V, q_lens):
    from inferx_b200.kernels import ops
    g = torch.Generator().manual_seed(K + V + sum(q_lens))
    q_lens = sorted(q_lens, key=lambda n: n != 1)
    S, T = len(q_lens), sum(q_lens)
    st = _step(q_lens, [3] * S, slots=list(range(S))[::-1])
    q, k = (torch.randn(T, HK * K, generator=g).to(dtype) for _ in range(2))
    v, beta = torch.randn(T, H * V, generator=g).to(dtype), torch.randn(T, H, generator=g).to(dtype)
    decay = torch.rand(T, H * K, generator=g) * 0.3 + 0.7
    state = torch.randn(S + 1, H, K, V, generator=g)
    st_ref = state.clone()
    ref = host_ops.delta_recurrence(q, k, v, beta, decay, st_ref, st, H, HK, K, V, 1e-6, K ** -0.5)
    before = ops.LAUNCHES[0]
    got = state.cuda()
    out = ops.delta_recurrence(q.cuda(), k.cuda(), v.cuda(), beta.cuda(), decay.cuda(), got,
                               _cuda(st), H, HK, K, V, 1e-6, K ** -0.5)
    assert ops.LAUNCHES[0] == before + 4                  # the four passes
    off = lambda a, b: float((a.cpu() - b.view(a.shape)).norm() / b.norm())
    assert off(out, ref) <= 2e-5 and off(got, st_ref) <= 2e-5
    assert torch.equal(got[S].cpu(), state[S])


@pytest.mark.parametrize("q_lens,launches", [([1] * 9 + [300, 2], 5), ([3] * 20 + [700], 4)])
def test_long_prompts_among_many_short_sequences(q_lens, launches):
    """Single tokens are walked by a launch of their own, the rest in segments; scratch holds one
    long sequence beside many short ones."""
    from inferx_b200.kernels import ops
    g = torch.Generator().manual_seed(len(q_lens))
    H, HK, K, V, S, T = 4, 2, 24, 40, len(q_lens), sum(q_lens)
    st = _step(q_lens, [3] * S, slots=list(range(S))[::-1])
    q, k = (torch.randn(T, HK * K, generator=g) for _ in range(2))
    v, beta = torch.randn(T, H * V, generator=g), torch.randn(T, H, generator=g)
    decay = torch.rand(T, H * K, generator=g) * 0.3 + 0.7
    state = torch.randn(S + 1, H, K, V, generator=g)
    st_ref, got = state.clone(), state.cuda()
    ref = host_ops.delta_recurrence(q, k, v, beta, decay, st_ref, st, H, HK, K, V, 1e-6, K ** -0.5)
    before = ops.LAUNCHES[0]
    out = ops.delta_recurrence(q.cuda(), k.cuda(), v.cuda(), beta.cuda(), decay.cuda(), got,
                               _cuda(st), H, HK, K, V, 1e-6, K ** -0.5)
    assert ops.LAUNCHES[0] == before + launches
    off = lambda a, b: float((a.cpu() - b.view(a.shape)).norm() / b.norm())
    assert off(out, ref) <= 2e-5 and off(got, st_ref) <= 2e-5
    assert torch.equal(got[S].cpu(), state[S])


def _fma32(a, b, c):
    """fp32 a * b + c rounded once: the product is exact in 64 bits, the sum is rounded to odd there."""
    p, c = a.astype(np.float64) * b.astype(np.float64), c.astype(np.float64)
    s = p + c
    back = s - p
    rest = (p - (s - back)) + (c - back)
    even = (s.view(np.int64) & 1) == 0
    return np.where((rest != 0) & even, np.nextafter(s, np.copysign(np.inf, rest)), s).astype(np.float32)


@pytest.mark.parametrize("K,V", [(64, 128), (128, 32), (28, 17), (96, 64), (100, 20), (30, 16), (132, 24)])
def test_start_states_are_chains_in_the_key_s_order(K, V):
    """The second segment's start state, from the first one's own state on (what it leaves behind a
    state of zeros), entry by entry over the key: the bits of that chain, however the join is made."""
    from inferx_b200.kernels import library, ops
    lib, H, T, seg = library.load(), 2, 200, 64
    g = torch.Generator().manual_seed(K + V)
    q, k = (torch.randn(T, H * K, generator=g).cuda() for _ in range(2))
    v, beta = torch.randn(T, H * V, generator=g).cuda(), torch.randn(T, H, generator=g).cuda()
    decay = (torch.rand(T, H * K, generator=g) * 0.1 + 0.9).cuda()
    cu, slot = (torch.tensor(x, dtype=torch.int32).cuda() for x in ([0, T], [0]))
    size = lib.ix_delta_segments_scratch_floats
    size.restype = ctypes.c_longlong

    def scratch_of(state):
        scratch = torch.zeros(size(T, 1, H, H, K, V, seg), device="cuda")
        out = torch.empty(T, H, V, device="cuda")
        long = ctypes.c_longlong
        ops._check(lib.ix_delta_segments(
            ops._ptr(q), long(H * K), ops._ptr(k), long(H * K), ops._ptr(v), long(H * V),
            ops._ptr(beta), long(H), ops._dtype_code(q), ops._ptr(decay), ops._ptr(state),
            ops._ptr(cu), ops._ptr(slot), ops._ptr(out), T, 1, H, H, K, V, ctypes.c_float(1e-6),
            ctypes.c_float(K ** -0.5), seg, 4, ops._ptr(scratch), ops._stream()), "delta_segments")
        return scratch.cpu().numpy()

    cells = (T // seg + 2) * H                     # segments.cuh: ds_cells
    starts = lambda scr: scr[:cells * K * V].reshape(cells // H, H, K, V)
    state = torch.randn(1, H, K, V, generator=g)
    scr = scratch_of(state.cuda())
    at = (cells * K * V + 3) & ~3
    A = scr[at:at + cells * K * K].reshape(cells // H, H, K, K)[0]
    want = starts(scratch_of(torch.zeros(1, H, K, V).cuda()))[1].copy()
    x = state[0].numpy()
    assert np.array_equal(starts(scr)[0], x)
    for i in range(K):
        want = _fma32(A[:, :, i, None], x[:, None, i, :], want)
    assert np.array_equal(starts(scr)[1], want)
