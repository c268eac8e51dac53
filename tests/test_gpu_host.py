"""What the host path of the operators owes their callers: tensors that saved-tensor hooks replace, arguments that are
refused before a launch, error types, concurrency."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _span_tokens(B, T):
    """Token rows with a [MASK], and two spans of 3 and of T // 4 tokens."""
    x = torch.full((B, T), 50, dtype=torch.int64)
    x[:, 2] = 2
    for start, end in ((5, 9), (T // 2, T // 2 + T // 4 + 1)):
        x[:, start], x[:, end] = 3, 4
    return x.to(DEV)


def test_cocktail_gradient_when_hooks_replace_the_saved_tensors():
    """The saved tensors leave the device between forward and backward, and their memory is overwritten: the gradient
    has to come from what the hooks give back."""
    from kerneldev_b200 import cocktail_scores
    B, T, C = 3, 130, 24
    tokens = _span_tokens(B, T)
    g = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn((B, T, C), generator=g, device=DEV).requires_grad_()
    ds = torch.randn((B, 2), generator=g, device=DEV)
    (want,) = torch.autograd.grad(cocktail_scores(x, tokens), x, ds)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.to(DEV)):
        scores = cocktail_scores(x, tokens)
    rubbish = [torch.full((2 * B * T + 3 * B,), -1, dtype=torch.int32, device=DEV) for _ in range(8)]
    (got,) = torch.autograd.grad(scores, x, ds)
    del rubbish
    assert torch.equal(got, want)


def test_lens_on_another_device_is_refused():
    """The kernels read lens on the device: an address of host memory must not reach them."""
    from kerneldev_b200 import flash_attention
    q = torch.zeros((1, 1, 128, 64), device=DEV, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="lens must live on"):
        flash_attention(q, q, q, lens=torch.tensor([100], dtype=torch.int32))
