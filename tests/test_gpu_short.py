"""The single-key-tile kernel (csrc/fwd_short.cu) on a B200: edges of its strips of 16 rows, its steps of 32
keys and its ring plan, every head dimension it takes, against the fp32 oracle; storage orders against the
general mma.sync kernel."""
import ctypes
import math

import pytest
import torch

from oracle.attention_ref import attention_fp32, make_inputs

pytestmark = pytest.mark.gpu

UNIT = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}   # unit roundoff


@pytest.fixture(scope="module")
def fa(cuda_device):
    import ascend_rsfa.flash_attention_forward as mod

    return mod


def bound(v, dtype):
    # every weight and every result is rounded once to 16 bits, the weights sum to one:
    # |error| <= u * max|v| + u * |o|, plus fp32 sums of at most 128 terms
    return 2 * UNIT[dtype] * float(v.float().abs().max()) + 1e-4


@pytest.mark.parametrize("D", [16, 32, 64, 128])
@pytest.mark.parametrize("heads", [(1, 1), (3, 5), (37, 33)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_lengths_at_the_edges_of_strips_and_steps(fa, cuda_device, D, heads, dtype):
    B, H = heads
    for S in (1, 15, 16, 17, 31, 32, 33, 63, 64) + ((65, 95, 96, 97, 112, 113, 127, 128) if D <= 64 else ()):
        q, k, v = make_inputs(B, H, S, D, seed=S + D, dtype=dtype)
        for causal in (False, True):
            n0 = fa.launch_count()
            o, lse = fa.attention_with_lse(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), causal,
                                           1.0 / math.sqrt(D))
            torch.cuda.synchronize()
            fa.device_status()
            assert fa.launch_count() - n0 == 1
            ref, lse_ref = attention_fp32(q, k, v, causal, 1.0 / math.sqrt(D), return_lse=True)
            assert float((o.cpu().float() - ref).abs().max()) <= bound(v, dtype), (S, causal)
            assert torch.allclose(lse.cpu(), lse_ref, atol=1e-4, rtol=1e-4), (S, causal)


@pytest.mark.parametrize("D,S,heads", [(16, 16, 40000), (16, 32, 40000), (16, 100, 12000), (16, 128, 12000), (32, 16, 40000),
                                       (32, 30, 20000), (32, 64, 20000), (32, 128, 4000), (64, 16, 20000), (64, 30, 20000),
                                       (64, 64, 6000), (128, 16, 8000)])
def test_ring_slots_used_again_and_again(fa, cuda_device, D, S, heads):
    # at least twice as many rounds as a ring has slots, one to eight warps per team: the last reader's refill, the phase
    # of the slot and the count of its readers; every head against the general kernel, three rounds' against the oracle
    strips = -(-S // 16)
    tile = -(-S // 32) * 32 * D * 2
    teams = min(8 // strips, 98304 // (3 * tile))
    stages = min(8, 98304 // (teams * 3 * tile))
    assert -(-heads // (2 * torch.cuda.get_device_properties(0).multi_processor_count * teams)) >= 2 * stages + 1
    g = torch.Generator(device=cuda_device).manual_seed(D + S)
    q, k, v = [torch.randn(heads // 4, 4, S, D, generator=g, device=cuda_device).half() for _ in range(3)]
    scale = 1.0 / math.sqrt(D)
    for causal in (False, True):
        o = fa.attention(q, k, v, causal, scale, 64, 64)
        fa.set_option("force_path", 0)
        try:
            general = fa.attention(q, k, v, causal, scale, 64, 64)
        finally:
            fa.set_option("force_path", -1)
        assert float((o.float() - general.float()).abs().max()) <= 2 * bound(v, torch.float16), causal
        for b in (0, heads // 8, heads // 4 - 1):
            ref = attention_fp32(*(t[b:b + 1].cpu() for t in (q, k, v)), causal, scale)
            assert float((o[b:b + 1].cpu().float() - ref).abs().max()) <= bound(v[b:b + 1], torch.float16), (b, causal)


@pytest.mark.parametrize("S,D", [(64, 64), (50, 128), (100, 32), (128, 16), (23, 64)])
def test_storage_orders_agree_with_the_general_kernel(fa, cuda_device, S, D):
    B, H = 5, 6
    g = torch.Generator(device=cuda_device).manual_seed(S)
    rand = lambda *shape: torch.randn(shape, generator=g, device=cuda_device).half()  # noqa: E731
    forms = {
        "bshd": [rand(B, S, H, D).transpose(1, 2) for _ in range(3)],
        "hbsd": [rand(H, B, S, D).transpose(0, 1) for _ in range(3)],
        "packed qkv": list(rand(B, S, 3, H, D).permute(2, 0, 3, 1, 4).unbind(0)),
        "padded rows": [rand(B, H, S, D + 8)[..., :D] for _ in range(3)],
        "sliced heads": [rand(B, 2 * H, S + 3, D)[:, 1::2, 2:S + 2] for _ in range(3)],
        "one batch, odd stride": [rand(3 * H * S * D + 24)[:H * S * D].view(1, H, S, D) for _ in range(3)],
    }
    for name, (q, k, v) in forms.items():
        for causal in (False, True):
            o = fa.attention(q, k, v, causal, 0.2, 64, 64)
            fa.set_option("force_path", 0)
            try:
                general = fa.attention(q, k, v, causal, 0.2, 64, 64)
            finally:
                fa.set_option("force_path", -1)
            torch.cuda.synchronize()
            assert o.stride() == general.stride(), name
            assert float((o.float() - general.float()).abs().max()) <= bound(v, torch.float16), (name, causal)


def test_rows_with_infinite_scores_and_nan_stay_where_they_are(fa, cuda_device):
    # a NaN or an infinity in one query row reaches that row only; in a key or a value, every row that sees it
    q, k, v = make_inputs(2, 3, 40, 64, seed=3)
    q[0, 0, 5, 0] = float("nan")
    q[1, 2, 7, 3] = float("inf")
    o = fa.attention(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), False, 0.125, 64, 64).cpu().float()
    ref = attention_fp32(q, k, v, False, 0.125)
    bad = torch.isnan(ref).any(-1)
    assert torch.equal(torch.isnan(o).any(-1), bad) and bool(bad[0, 0, 5]) and int(bad.sum()) <= 2
    assert float((o - ref)[~bad].abs().max()) <= bound(v, torch.float16)


def hidden_keys(S, D, dtype, hide, scale):
    """Keys that a program hides with the type's lowest value (or -inf) in a column in which every query has a one,
    or, `hide` = "none", scores of some 2^32 times the scale."""
    q, k, v = make_inputs(2, 3, S, D, seed=S + D, dtype=dtype)
    if hide == "none":
        f = 2.0 ** 16 / scale ** 0.5
        return (q.float() * f).to(dtype), (k.float() * f).to(dtype), v
    q[..., 0] = 1.0
    k[..., 0] = 0.0
    first = {"front": S // 2, "all": S, "all, -inf": S}[hide]
    k[:, :, :first, 0] = -math.inf if "inf" in hide else torch.finfo(dtype).min
    return q, k, v


@pytest.mark.parametrize("D", [16, 32, 64, 128])
@pytest.mark.parametrize("hide", ["front", "all", "all, -inf", "none"])
def test_scores_of_any_size(fa, cuda_device, D, hide):
    # with the mask the first rows see hidden keys only; their softmax is over equal scores, not over nothing
    for S in (20, 40, 64) + ((90, 128) if D <= 64 else ()):
        scale = 1.0 / math.sqrt(D)
        q, k, v = hidden_keys(S, D, torch.bfloat16, hide, scale)
        for causal in (False, True):
            o, lse = fa.attention_with_lse(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), causal, scale)
            ref, lse_ref = attention_fp32(q, k, v, causal, scale, return_lse=True)
            if "inf" in hide:   # a softmax over nothing
                assert bool(torch.isnan(o).all()) and bool(torch.isneginf(lse).all())
            else:
                assert torch.allclose(lse.cpu(), lse_ref, atol=1e-4, rtol=1e-4), (S, causal)
                assert float((o.cpu().float() - ref).abs().max()) <= bound(v, torch.bfloat16), (S, causal)


@pytest.mark.parametrize("B,H,S,D,head", [(5, 6, 100, 64, 7), (400, 4, 64, 128, 500), (3000, 4, 16, 16, 9000)])
def test_a_wait_that_runs_out_is_reported(fa, cuda_device, B, H, S, D, head):
    """Of the first loads, those of the heads from one on and the arrivals that announce them are left out ("test_drop_load"): nothing is in
    flight and no address is touched, the waits of the teams that own them run out and the kernel returns by itself."""
    from ascend_rsfa import _capi

    lib = _capi.load()
    q, k, v = [t.to(cuda_device) for t in make_inputs(B, H, S, D, seed=8)]
    whole = fa.attention(q, k, v, False, 0.2, 64, 64)
    fa.device_status()
    fa.set_option("wait_limit_ms", 1)
    fa.set_option("test_drop_load", head)     # from the first slots of the rings, and from their last ones
    try:
        fa.attention(q, k, v, False, 0.2, 64, 64)
        torch.cuda.synchronize()
    finally:
        fa.set_option("test_drop_load", -1)
        fa.set_option("wait_limit_ms", 2000)
    raw = ctypes.c_int(0)
    assert lib.rsfa_device_status(0, ctypes.byref(raw)) == _capi.RSFA_ERR_DEVICE_STATUS
    assert raw.value == (1 << 16) | 4, hex(raw.value)     # the wait for K/V
    for _ in range(2):
        o = fa.attention(q, k, v, False, 0.2, 64, 64)
        torch.cuda.synchronize()
        assert torch.equal(o, whole)
    fa.device_status()
