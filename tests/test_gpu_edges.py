"""Kernels at the sizes where their tiles, rings and dispatch rules begin and end, against the oracle."""
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
from cocktail_inputs import cocktail_rows, embeddings  # noqa: E402
from oracle import attention_oracle as ao  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# T: one warp's 128 tokens, a chunk of 4096 with and without a remainder, the gradient's 32-token blocks; C: 16-byte
# accesses (8 or 4 elements), element by element (12 in 16 bits), more columns than threads share a row (2056, 4100)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,C", [(1, 127, 8), (2, 129, 12), (3, 4096, 40), (2, 4099, 72), (2, 200, 2056), (1, 96, 4100)])
def test_cocktail_scores_and_gradient(B, T, C, dtype):
    from kerneldev_b200 import cocktail_scores
    x = cocktail_rows(7, B, T, unbalanced=T > 128)
    e = embeddings(7, B, T, C).to(dtype)
    e_dev = e.to(DEV).requires_grad_()
    e_ref = e.double().requires_grad_()
    scores = cocktail_scores(e_dev, x.to(DEV))
    want, h = ao.cocktail_scores(e_ref, x)
    ds = torch.randn(want.shape, generator=torch.Generator().manual_seed(1)).to(dtype)
    # sums in fp32, one rounding to the output type. A score sums C products of a mean over at most T tokens: T + C fp32
    # roundings against the sum of the magnitudes, which |x_mask|_1 max|h| bounds
    eps = {torch.float32: 2.0**-24, torch.bfloat16: 2.0**-9, torch.float16: 2.0**-12}[dtype]
    size = float(e_ref.detach().abs().sum(-1).max() * h.detach().abs().max()) if h.numel() else 0.0
    err = (scores.detach().double().cpu() - want.detach()).abs()
    assert scores.shape == want.shape and bool((err <= 2 * eps * want.detach().abs() + (T + C) * 2.0**-24 * size).all())
    if want.numel() == 0:
        return
    scores.backward(ds.to(DEV))
    want.backward(ds.double())
    # a token's gradient sums at most S products, each of a few fp32 roundings, then one rounding to the output type
    S = want.shape[1]
    top = float(ds.abs().double().sum(1).max() * max(h.detach().abs().max(), e_ref.detach().abs().max()))
    err = (e_dev.grad.double().cpu() - e_ref.grad).abs()
    assert bool((err <= 2 * eps * e_ref.grad.abs() + (S + T + 8) * 2.0**-24 * top).all())
