"""The norm over whole projections with rotation and store: rows of odd and even sizes, heads whose angles do not fit beside the row, and
(on the CPU) the shared memory that the launch asks for."""
import ctypes

import pytest
import torch

DEV = "cuda:0"


@pytest.mark.parametrize("channels,pairs", [(99, 16), (98, 16), (1, 0), (3, 1), (51200, 64), (51200, 12800), (51199, 3712)])
def test_the_angles_lie_inside_the_shared_memory_asked_for(channels, pairs):
    from llm_b200.csrc import ops
    lib, row = ops.load(), ctypes.c_longlong()
    lib.llmk_norm_rope_smem.restype = ctypes.c_longlong
    asked = lib.llmk_norm_rope_smem(channels, pairs, ctypes.byref(row))
    assert row.value % 8 == 0 and row.value >= 4 * channels and asked <= 226 * 1024
    # the whole table, or none where it does not fit
    assert asked == row.value + 8 * pairs or (asked == row.value and row.value + 8 * pairs > 226 * 1024)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("halves", [True, False])
@pytest.mark.parametrize("H,G,D,V,pairs,T,from_k", [(2, 1, 33, 20, 16, 5, False), (2, 1, 33, 33, 5, 130, True), (16, 4, 128, 128, 32, 8, False),
                                                    (3, 2, 20, 12, 10, 3, False), (1, 1, 25600, 8, 12800, 2, False), (4, 0, 64, 64, 8, 3, False)])
def test_norm_rotation_and_store(dtype, halves, H, G, D, V, pairs, T, from_k):
    from llm_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(D + T)
    R = lambda *s: torch.randn(*s, device=DEV, generator=g)
    page, eps, amp = 8, 1e-5, 1.25
    qkv = R(T, (H + G) * D + (0 if from_k else G * V)).to(dtype)
    gq, gk = R(H * D), R(G * D) if G else None
    freqs = torch.logspace(0, -3, pairs, device=DEV)
    pos = torch.randint(0, 64, (T,), device=DEV, dtype=torch.int32, generator=g)
    slots = torch.randperm(2 * T, device=DEV, generator=g)[:T].to(torch.int32)
    n_pages = -(-2 * T // page)
    kp, vp = torch.zeros(n_pages, max(1, G), page, D, device=DEV, dtype=dtype), torch.zeros(n_pages, max(1, G), page, V, device=DEV, dtype=dtype)
    q = torch.empty(T, H * D, device=DEV, dtype=dtype)
    ops.norm_rope_kv_write(qkv, gq, gk, eps, freqs, halves, pos, slots, kp if G else None, vp if G else None, T, H, G, D, V, q_out=q, amp=amp,
                           v_from_k=from_k)
    angle = (pos.float()[:, None] * freqs).double()
    c, s = angle.cos()[:, None] * amp, angle.sin()[:, None] * amp

    def turned(x, gain, n):
        x = x.double()
        y = (x / (x.pow(2).mean(-1, keepdim=True) + eps).sqrt() * gain.double()).view(T, n, D).clone()
        lo, hi = (slice(0, pairs), slice(pairs, 2 * pairs)) if halves else (slice(0, 2 * pairs, 2), slice(1, 2 * pairs, 2))
        a, b = y[..., lo].clone(), y[..., hi].clone()
        y[..., lo], y[..., hi] = a * c - b * s, b * c + a * s
        return y
    # float32 arithmetic of a few terms (a turned value is a sum of two that may cancel), rounded once to the kind of the result
    near = lambda got, want: bool(((got.double() - want).abs() <= want.abs() * (2 ** -8 if dtype == torch.bfloat16 else 4e-6) + 2e-5).all())
    assert near(q.view(T, H, D), turned(qkv[:, :H * D], gq, H))
    if G:
        k, at = turned(qkv[:, H * D:(H + G) * D], gk, G), slots.long()
        assert near(kp[at // page, :, at % page], k)
        values = qkv[:, H * D:(H + G) * D] if from_k else qkv[:, (H + G) * D:]
        assert torch.equal(vp[at // page, :, at % page], values.reshape(T, G, V))
        assert int((kp != 0).any(-1).sum()) <= T * G
