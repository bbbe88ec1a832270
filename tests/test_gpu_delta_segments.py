"""The delta rule in segments at every width of key that has a form of its own, at the edges of a
segment and of the batch, against the plain statement."""
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
