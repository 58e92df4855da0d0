"""The native form of the ordinary attention() call (csrc/torch_binding.cpp) answers exactly where the Python
code would have done the same, and hands everything else to it."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

import ascend_rsfa.flash_attention_forward as fa

native = fa._rsfa_torch.forward


def test_declines_what_it_must_not_answer_without_a_device():
    q = torch.zeros(1, 2, 16, 64, dtype=torch.float16)
    assert native(q, q, q, True, 0.5, 128, 128, False) is None            # not on a GPU
    assert native(q, q, None, True, 0.5, 128, 128, False) is None         # not a tensor
    assert native(q, q, q, True, 0.5) is None                             # not its arguments
    with pytest.raises(RuntimeError, match="no CPU path"):
        fa.attention(q, q, q, True, 0.5, 128, 128)


def python_only(monkeypatch):
    monkeypatch.setattr(fa._rsfa_torch, "forward", lambda *a: None)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_same_result_as_the_python_code_for_every_storage_order(cuda_device, monkeypatch, dtype):
    B, H, S, D = 2, 3, 40, 64
    g = torch.Generator(device=cuda_device).manual_seed(1)
    rand = lambda *s: torch.randn(s, generator=g, device=cuda_device).to(dtype)  # noqa: E731
    forms = {
        "dense": ([rand(B, H, S, D) for _ in range(3)], True),
        "bshd": ([rand(B, S, H, D).transpose(1, 2) for _ in range(3)], True),
        "packed qkv": (list(rand(B, S, 3, H, D).permute(2, 0, 3, 1, 4).unbind(0)), True),
        "padded rows": ([rand(B, H, S, D + 8)[..., :D] for _ in range(3)], True),
        "one batch": ([rand(H * S * D + 8)[:H * S * D].view(1, H, S, D) for _ in range(3)], True),
        "requires grad": ([rand(B, H, S, D).requires_grad_() for _ in range(3)], True),
        "parameter": ([torch.nn.Parameter(rand(B, H, S, D)) for _ in range(3)], True),
        "odd row stride": ([rand(B, H, S, D + 4)[..., :D] for _ in range(3)], False),
        "shared heads": ([rand(B, H, S, D)] + [rand(B, 1, S, D).expand(B, H, S, D) for _ in range(2)], False),
        "columns apart": ([rand(B, H, D, S).transpose(2, 3) for _ in range(3)], False),
        "empty": ([rand(B, 0, S, D) for _ in range(3)], False),
    }
    got = {}
    for name, (qkv, ordinary) in forms.items():
        assert (native(*qkv, True, 0.25, 64, 64, True) is not None) == ordinary, name
        got[name] = (fa.attention(*qkv, True, 0.25, 64, 64), *fa.attention_with_lse(*qkv, False, 0.25, 64, 64))
    python_only(monkeypatch)
    for name, (qkv, _) in forms.items():
        want = (fa.attention(*qkv, True, 0.25, 64, 64), *fa.attention_with_lse(*qkv, False, 0.25, 64, 64))
        for a, b in zip(got[name], want):
            assert torch.equal(a, b) and a.stride() == b.stride() and a.dtype == b.dtype, name
            assert a.requires_grad == b.requires_grad, name


@pytest.mark.gpu
def test_refusals_modes_and_argument_types_reach_the_python_code(cuda_device, monkeypatch):
    q = torch.zeros(1, 2, 16, 64, dtype=torch.float16, device=cuda_device)

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Sub(torch.Tensor):
        pass

    off = torch.zeros(2 * 16 * 64 + 1, dtype=torch.float16, device=cuda_device)[1:].view(1, 2, 16, 64)   # unaligned base
    bad = [(off, off, off, True, 0.5, 64, 64), (q, q, q[..., :32], True, 0.5, 64, 64), (q, q, q.bfloat16(), True, 0.5, 64, 64), (q[0], q[0], q[0], True, 0.5, 64, 64),
           (q, q, q.cpu(), True, 0.5, 64, 64), (q.float(),) * 3 + (True, 0.5, 64, 64), (q, q, q, True, float("nan"), 64, 64),
           (q, q, q, True, 0.5, 0, 64), (q[..., :48],) * 3 + (True, 0.5, 64, 64)]

    def raised(args):
        with pytest.raises(Exception) as e:
            fa.attention(*args)
        return type(e.value), str(e.value)

    first = [raised(a) for a in bad]
    assert native(q, q, q, 1, 0.5, 64, 64, False) is None and native(q, q, q, True, 1, 64, 64, False) is None
    assert native(q.as_subclass(Sub), q, q, True, 0.5, 64, 64, False) is None
    with Mode():
        assert native(q, q, q, True, 0.5, 64, 64, False) is None
    with torch.device("cuda"):
        assert native(q, q, q, True, 0.5, 64, 64, False) is None
    assert torch.vmap(lambda x: torch.zeros_like(x) if native(x, x, x, True, 0.5, 64, 64, False) is None else x)(
        q.expand(3, 1, 2, 16, 64)).shape == (3, 1, 2, 16, 64)
    python_only(monkeypatch)
    assert first == [raised(a) for a in bad]
