"""Memory that a step's mixers take beside its activations is left free when the cache is sized."""
from types import SimpleNamespace

import pytest
import torch

from inferx_b200.engine.engine import EngineConfig, graph_reserve_bytes, step_scratch_bytes
from inferx_b200.kernels import ops
from inferx_b200.parts.latent_attention import LatentAttentionMixer
from inferx_b200.parts.specs import LatentAttentionSpec
from inferx_b200.parts.state_space import GatedDeltaMixer, StateSpaceMixer

CTX = SimpleNamespace(ops=ops, dtype=torch.bfloat16)


def _model(*mixers):
    return SimpleNamespace(spec=SimpleNamespace(hidden=1024, vocab_size=1000),
                           blocks=[SimpleNamespace(parts=lambda m=m: [m]) for m in mixers])


def _state_space():
    spec = SimpleNamespace(heads=64, groups=1, vdim=64, state=128, norm_groups=1, names=(), conv=4)
    return StateSpaceMixer(spec, CTX, "m")


def _delta():
    return GatedDeltaMixer(SimpleNamespace(heads=16, kv_heads=16, dim=64, vdim=128), CTX, "m")


def _latent():
    m = LatentAttentionMixer(LatentAttentionSpec(
        hidden=1024, heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512, scale=0.1, window=0,
        position=None, latent_eps=1e-6), CTX, "m")
    m.kv_w = object()                       # as bound on a device
    return m


@pytest.mark.parametrize("make,least", [
    # 4,096 tokens: 64 chunks or segments of 32 KB a head; 4,096 rows of 16 x (192 + 128 + 128) x 2
    (_state_space, 64 * 64 * 32768), (_delta, 64 * 16 * 32768), (_latent, 4096 * 16 * 896)])
def test_a_mixers_scratch_is_reserved(make, least):
    cfg = EngineConfig(max_num_seqs=4, max_model_len=4096, max_num_batched_tokens=4096)
    without = graph_reserve_bytes(cfg, _model())
    got = graph_reserve_bytes(cfg, _model(make())) - without
    assert got == step_scratch_bytes(cfg, _model(make())) >= least
    # they take it in turn, and mixers made of two count too
    pair = SimpleNamespace(left=make(), right=make())
    assert step_scratch_bytes(cfg, _model(make(), make(), pair)) == got


def test_scratch_of_long_steps_is_bounded():
    cfg = EngineConfig(max_num_seqs=64, max_model_len=131072, max_num_batched_tokens=131072)
    assert step_scratch_bytes(cfg, _model(_state_space())) <= ops.SSD_MAX_SCRATCH_BYTES
    assert step_scratch_bytes(cfg, _model(_latent())) <= 1.3 * ops.WIDENED_MAX_BYTES


def test_steps_stay_within_what_is_reserved():
    """What the forms allocate for a prompt against what is set aside for it."""
    import ctypes
    lib = ops._lib()
    for T in (200, 2048, 16384):
        seg = ctypes.c_int(0)
        for name, delta in (("ix_delta_recurrence_segments", True),
                            ("ix_linear_recurrence_segments", False)):
            n = getattr(lib, name)(1, 16, 64, 128, T, 128, 64, ctypes.byref(seg))
            assert n > 1
            size = lib.ix_delta_segments_scratch_floats if delta \
                else lib.ix_linear_segments_scratch_floats
            size.restype = ctypes.c_longlong
            took = 4 * (size(T, 1, 16, 16, 64, 128, seg.value) if delta
                        else size(T, 1, 16, 64, 128, seg.value))
            assert took <= ops.segments_scratch_bytes(T, 1, 16, 16, 64, 128, delta)
        rows = ops.widened_latent_rows([T], T, 0, 16, 512, 64, 320)
        took = rows * (16 * 896 + 1152) + min(rows * 16 * 512, ops.WIDENED_FP32_BYTES)
        assert took <= ops.widened_scratch_bytes(T, 1, T, 0, 16, 512, 64, 128, 128)
