"""The forms of the tcgen05 kernels for launches that pairs of Q tiles do not suit, on a B200 at the sizes where their
bookkeeping can go wrong: the two of the D = 128 kernel in which each Q tile of a CTA has K/V tiles of its own - two
heads per work item (S <= 128), and the keys of one block of rows dealt out to both tiles - and one Q tile per CTA at
D <= 64.  Against the fp32 oracle, the pair kernels and the general kernel."""
import math

import pytest
import torch

from oracle.attention_ref import attention_fp32, make_inputs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fa(cuda_device):
    import ascend_rsfa.flash_attention_forward as mod

    return mod


def agree(fa, dev, q, k, v, causal, scale):
    u = 2.0 ** -11 if q.dtype == torch.float16 else 2.0 ** -8
    n0 = fa.launch_count()
    o, lse = fa.attention_with_lse(q.to(dev), k.to(dev), v.to(dev), causal, scale)
    torch.cuda.synchronize()
    fa.device_status()
    assert fa.launch_count() - n0 == 1
    ref, lse_ref = attention_fp32(q, k, v, causal, scale, return_lse=True)
    # a weight and a result are each rounded once to 16 bits; fp16 weights below 2^-14 of the tile's range
    # (2^-8 of the row's largest) keep an absolute error of 2^-19 of it: 2^-19 * S in the worst sum
    assert float((o.cpu().float() - ref).abs().max()) <= (2 * u + q.shape[2] * 2.0 ** -19) * float(v.float().abs().max())
    assert torch.allclose(lse.cpu(), lse_ref, atol=1e-4, rtol=1e-4)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("S", [129, 256, 257, 384, 385, 640, 1000, 2048])
def test_split_keys(fa, cuda_device, S, causal):
    # one to sixteen key tiles, odd numbers of them, a tile without any (the first causal block), ragged ends
    for B, H, dtype in ((1, 1, torch.float16), (2, 3, torch.bfloat16)):
        q, k, v = make_inputs(B, H, S, 128, seed=S, dtype=dtype)
        agree(fa, cuda_device, q, k, v, causal, 1.0 / math.sqrt(128))


@pytest.mark.parametrize("causal", [False, True])
def test_split_keys_with_several_items_per_cta(fa, cuda_device, causal):
    # causal: more items than CTAs, light ones last; else a launch of 1.35 waves of pairs, three of split items
    B, H, S = (1, 18, 1280) if causal else (1, 25, 2048)
    q, k, v = make_inputs(B, H, S, 128, seed=7)
    agree(fa, cuda_device, q, k, v, causal, 1.0 / math.sqrt(128))


@pytest.mark.parametrize("order", ["growing", "falling"])
def test_split_keys_when_the_two_halves_have_far_apart_maxima(fa, cuda_device, order):
    # |k| grows or falls with the key index, every second key tile a hundred times smaller: references move,
    # tiles are redone, and the merge weighs one half with next to nothing
    g = torch.Generator().manual_seed(5)
    S = 1024
    ramp = torch.linspace(0.05, 2.0, S) if order == "growing" else torch.linspace(2.0, 0.05, S)
    ramp = ramp * torch.where((torch.arange(S) // 128) % 2 == 0, 1.0, 0.01)
    k = (torch.randn(1, 2, S, 128, generator=g).sign() * ramp.view(1, 1, S, 1)).half()
    q = torch.randn(1, 2, S, 128, generator=g).sign().half()
    v = torch.randn(1, 2, S, 128, generator=g).half()
    for causal in (False, True):
        agree(fa, cuda_device, q, k, v, causal, 1.0)


def test_split_keys_keeps_a_nan_in_its_row(fa, cuda_device):
    q, k, v = make_inputs(1, 2, 512, 128, seed=9)
    q[0, 1, 300, 5] = float("nan")
    o = fa.attention(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), False, 0.1, 128, 128).cpu().float()
    ref = attention_fp32(q, k, v, False, 0.1)
    assert bool(torch.isnan(o[0, 1, 300]).all()) and int(torch.isnan(o).any(-1).sum()) == 1
    keep = ~torch.isnan(ref)
    assert float((o - ref)[keep].abs().max()) < 5e-3


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("S,heads", [(65, 149), (100, 301), (128, 300), (127, 597)])
def test_two_heads_per_item(fa, cuda_device, S, heads, causal):
    # odd numbers of heads: the last item has one; more items than CTAs
    for dtype in (torch.float16, torch.bfloat16):
        q, k, v = make_inputs(1, heads, S, 128, seed=S, dtype=dtype)
        agree(fa, cuda_device, q, k, v, causal, 1.0 / math.sqrt(128))
    q, k, v = make_inputs(heads // 7, 7, S, 128, seed=S + 1)
    agree(fa, cuda_device, q, k, v, causal, 0.5)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("S", [129, 191, 256, 257, 320, 512, 513, 1000, 1024])
def test_single_q_tiles_at_small_head_dimensions(fa, cuda_device, S, causal):
    # one tile per CTA, two CTAs per SM: odd and even numbers of 64-key tiles, a last tile of one row, more items
    # than places; D below 64 reads zero columns
    for B, H, D, dtype in ((1, 1, 64, torch.float16), (2, 3, 32, torch.bfloat16), (1, 5, 16, torch.float16)):
        q, k, v = make_inputs(B, H, S, D, seed=S + D, dtype=dtype)
        agree(fa, cuda_device, q, k, v, causal, 1.0 / math.sqrt(D))
    if S in (257, 512):
        q, k, v = make_inputs(8, 33, S, 64, seed=S)
        agree(fa, cuda_device, q, k, v, causal, 0.125)


def test_single_q_tiles_follow_a_growing_maximum(fa, cuda_device):
    g = torch.Generator().manual_seed(6)
    S = 1024
    k = (torch.randn(1, 2, S, 64, generator=g).sign() * torch.linspace(0.05, 3.0, S).view(1, 1, S, 1)).half()
    q = torch.randn(1, 2, S, 64, generator=g).sign().half()
    v = torch.randn(1, 2, S, 64, generator=g).half()
    for causal in (False, True):
        agree(fa, cuda_device, q, k, v, causal, 1.0)


@pytest.mark.parametrize("B,H,S,D", [(2, 3, 640, 128), (30, 8, 100, 128), (3, 5, 300, 64), (2, 3, 520, 32)])
def test_storage_orders_agree_with_the_pair_kernel(fa, cuda_device, B, H, S, D):
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
    u = 2.0 ** -11
    for name, (q, k, v) in forms.items():
        for causal in (False, True):
            o = fa.attention(q, k, v, causal, 0.15, 128, 128)
            fa.set_option("tcgen05_variant", 0)
            try:
                pair = fa.attention(q, k, v, causal, 0.15, 128, 128)
            finally:
                fa.set_option("tcgen05_variant", -1)
            torch.cuda.synchronize()
            fa.device_status()
            assert o.stride() == pair.stride(), name
            # each is within (2 u + S 2^-19) max|v| of the exact result (see agree)
            limit = 2 * (2 * u + S * 2.0 ** -19) * float(v.float().abs().max())
            assert float((o.float() - pair.float()).abs().max()) <= limit, (name, causal)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("hidden", ["lowest", "-inf"])
@pytest.mark.parametrize("D,S,first,last", [(128, 640, 0, 128), (128, 640, 128, 256), (128, 640, 0, 256), (64, 384, 0, 64),
                                            (64, 1000, 0, 128), (32, 300, 0, 64)])
def test_a_first_key_tile_of_hidden_keys(fa, cuda_device, dtype, hidden, D, S, first, last):
    # keys first .. last - 1 carry the type's lowest value (or -inf) in a column in which every query has a one; the
    # visible scores lie around -8000 times the scale.  The first tile of a form's own keys may be hidden whole.
    q, k, v = make_inputs(1, 3, S, D, seed=S + first, dtype=dtype)
    q[..., :2] = 1.0
    k[..., 0], k[..., 1] = 0.0, -8000.0
    k[:, :, first:last, 0] = -math.inf if hidden == "-inf" else torch.finfo(dtype).min
    scale = 1.0 / math.sqrt(D)
    for causal in (False, True):
        o, lse = fa.attention_with_lse(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), causal, scale)
        torch.cuda.synchronize()
        fa.device_status()
        ref, lse_ref = attention_fp32(q, k, v, causal, scale, return_lse=True)
        seen = slice(last if causal and first == 0 else 0, S)   # rows that see a visible key
        u = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
        # as in agree(), and scores of 8000 are sums in fp32 whose order differs: 2 units of 2^-11 times the scale
        limit = (2 * u + S * 2.0 ** -19 + 2.0 ** -10 * scale) * float(v.float().abs().max())
        assert float((o.cpu().float() - ref)[:, :, seen].abs().max()) <= limit, causal
        assert torch.allclose(lse.cpu()[:, :, seen], lse_ref[:, :, seen], atol=1e-3, rtol=1e-4), causal


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D,S,heads", [(256, 64, 700), (256, 130, 400), (256, 256, 300), (256, 640, 70), (128, 320, 300),
                                       (128, 640, 120), (64, 200, 500), (64, 641, 160)])
def test_work_items_of_one_to_eleven_key_tiles_on_the_64_key_kernels(fa, cuda_device, D, S, heads, causal):
    # where the producer claims its next item: items of up to four tiles, and the last ones of a short-row launch
    g = torch.Generator(device=cuda_device).manual_seed(S)
    q, k, v = [torch.randn(heads, 1, S, D, generator=g, device=cuda_device).half() for _ in range(3)]
    o = fa.attention(q, k, v, causal, 1.0 / math.sqrt(D), 128, 64)
    fa.set_option("force_path", 0)
    try:
        general = fa.attention(q, k, v, causal, 1.0 / math.sqrt(D), 128, 64)
    finally:
        fa.set_option("force_path", -1)
    torch.cuda.synchronize()
    fa.device_status()
    # each is within (2 u + S 2^-19) max|v| of the exact result (see agree)
    limit = 2 * (2 * 2.0 ** -11 + S * 2.0 ** -19) * float(v.float().abs().max())
    assert float((o.float() - general.float()).abs().max()) <= limit


@pytest.mark.parametrize("S,scale,dtype", [(132, 0.125, torch.float16), (143, 0.125, torch.bfloat16), (192, 0.125, torch.float16),
                                           (384, 0.25, torch.bfloat16)])
def test_single_q_tiles_are_as_exact_as_pairs(fa, cuda_device, S, scale, dtype):
    # peaked rows, for which it matters that the row's largest weight is exact: the reference comes from as many keys as
    # in the kernel of the requested tile, so the errors against 64-bit sums differ by their order only (under 0.3 %,
    # measured over 91 sizes; from 64 keys only they were 5 to 17 % larger here)
    g = torch.Generator(device=cuda_device).manual_seed(S)
    q, k, v = [2 * torch.randn(8, 12, S, 64, generator=g, device=cuda_device).to(dtype) for _ in range(3)]
    s = (q.double() @ k.double().transpose(-1, -2)) * scale
    o, lse = torch.softmax(s, -1) @ v.double(), torch.logsumexp(s, -1)
    errors = []
    for variant in (-1, 2):
        fa.set_option("tcgen05_variant", variant)
        try:
            got = fa.attention_with_lse(q, k, v, False, scale, 128, 128)
        finally:
            fa.set_option("tcgen05_variant", -1)
        errors.append([float((a.double() - b).norm()) for a, b in zip(got, (o, lse))])
    assert errors[0][0] <= 1.02 * errors[1][0] and errors[0][1] <= 1.1 * errors[1][1], errors
