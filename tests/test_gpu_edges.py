"""Kernels at the sizes where their tiles, rings and dispatch rules begin and end, against the oracle."""
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
from cocktail_inputs import cocktail_rows, embeddings  # noqa: E402
sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
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


# Rows of padding are left alone by the delta and conversion kernels: garbage in every buffer they are given must not come through. T and lens at the
# edges of their blocks (96 rows at head dims up to 64, 48 above) and of tiles
@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (16, torch.float16), (128, torch.bfloat16), (80, torch.float16)])
@pytest.mark.parametrize("T,lens", [(95, (95, 0, 1)), (97, (96, 97, 48)), (300, (47, 289, 128)), (192, (192, 191, 129))])
def test_padding_is_left_out_of_delta_and_conversion(T, lens, D, dtype):
    from tests.helpers import assert_close, rand_inputs
    from kerneldev_b200.original_kernel import _backward, _forward
    from kerneldev_b200.plan import AttentionPlan
    B, H = len(lens), 3
    q, k, v, do = rand_inputs(B, H, T, D, dtype, T + D)
    lens = torch.tensor(lens, dtype=torch.int32)
    plan = AttentionPlan(B, T, DEV, lens=lens.to(DEV), causal=True)
    dev = [x.to(DEV) for x in (q, k, v, do)]
    o, lse = _forward(*dev[:3], plan, D ** -0.5)
    bufs = [torch.full_like(dev[0], float("nan")) for _ in range(3)]
    bufs += [torch.full((B, H, T, *w), float("nan"), device=DEV) for w in ((), (64 if D <= 64 else 128,))]
    got = _backward(*dev[:3], o, lse, dev[3], plan, D ** -0.5, 0, bufs)
    mask = ao.dense_mask(T, lens=lens, causal=True)
    ref = ao.attention_fwd_bwd(*(x.float() for x in (q, k, v, do)), mask, D ** -0.5)[2:]
    beyond = torch.arange(T)[None, None, :, None] >= lens[:, None, None, None]
    for name, g, want in zip(("dQ", "dK", "dV"), got, ref):
        assert_close(name, g, want)
        assert not g.cpu()[beyond.expand_as(g)].any()


# Key tiles that no query sees: their dK and dV are written from a box of 32 zeroed rows. Every element of theirs and nothing beside it: ragged last
# boxes and widths below the tile's, in gradients that are slices of a wider tensor
@pytest.mark.parametrize("D", [16, 48, 64])
@pytest.mark.parametrize("T,lens", [(129, (128, 1)), (161, (0, 100)), (287, (129, 60)), (384, (3, 256))])
def test_empty_key_tiles_are_written_as_zeros(T, lens, D):
    from tests.helpers import rand_inputs
    from kerneldev_b200 import flash_attention
    from kerneldev_b200.original_kernel import _backward, _forward
    from kerneldev_b200.plan import AttentionPlan
    B, H = len(lens), 3
    q, k, v, do = rand_inputs(B, H, T, D, torch.bfloat16, T + D, DEV)
    lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    beyond = (torch.arange(T, device=DEV)[None, None, :, None] >= (lens[:, None, None, None] + 127) // 128 * 128).expand(B, H, T, D)
    plan = AttentionPlan(B, T, DEV, lens=lens, causal=True)
    o, lse = _forward(q, k, v, plan, D ** -0.5)
    wide = [torch.full((B, T, H, D + 16), float("nan"), device=DEV, dtype=q.dtype) for _ in range(3)]
    bufs = [w[..., 8:8 + D].transpose(1, 2) for w in wide]
    bufs += [torch.full((B, H, T, *w), float("nan"), device=DEV) for w in ((), (64,))]
    got = _backward(q, k, v, o, lse, do, plan, D ** -0.5, 0, bufs)
    for g, w in zip(got, wide):
        assert g.data_ptr() == w[..., 8:].data_ptr() and not g[beyond].any()
        assert bool(w[..., :8].isnan().all()) and bool(w[..., 8 + D:].isnan().all())
    # a float32 call, whose boxes are of 32 columns: freed memory that its gradients are likely to be made in holds no zeros
    x32 = [x.float().requires_grad_() for x in (q, k, v)]
    out = flash_attention(*x32, lens=lens)
    spoilt = [torch.full((B, H, T, D), float("nan"), device=DEV) for _ in range(8)]
    del spoilt
    for g in torch.autograd.grad(out, x32, do.float()):
        assert not g[beyond].any() and not g.isnan().any()


# dK and dV of the deterministic backward come from the fused kernel without its dQ: the same sums in the same order. T at the edges of tiles, and lengths at
# which the rows of a head do not begin on 16 bytes; calls behind one another, whose kernels overlap
@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (48, torch.float32), (128, torch.float16), (80, torch.float32)])
@pytest.mark.parametrize("T,lens", [(64, (64, 1)), (128, (128, 70)), (131, (131, 129)), (385, (0, 385)), (1022, (900, 257))])
def test_both_backwards_give_the_same_dk_and_dv(T, lens, D, dtype):
    from tests.helpers import rand_inputs
    from kerneldev_b200 import flash_attention
    B, H = len(lens), 5
    lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    for seed in range(3):
        q, k, v, do = (x.to(dtype) for x in rand_inputs(B, H, T, D, torch.float16, T + D + seed, DEV))
        x = [t.requires_grad_() for t in (q, k, v)]
        want = torch.autograd.grad(flash_attention(*x, lens=lens), x, do)
        got = torch.autograd.grad(flash_attention(*x, lens=lens, deterministic=True), x, do)
        again = torch.autograd.grad(flash_attention(*x, lens=lens, deterministic=True), x, do)
        assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
        assert all(torch.equal(a, b) for a, b in zip(got, again))


# dQ and dK of transformed Q and K, transformed back by the last pass of the fused backward, against the transform's own backward. T and lens at the
# edges of its blocks (128 rows at head dim 16, 64 above)
@pytest.mark.parametrize("D,dtype", [(16, torch.bfloat16), (32, torch.float16), (64, torch.bfloat16), (128, torch.float16)])
@pytest.mark.parametrize("T,lens", [(63, (63, 1, 0)), (129, (64, 129, 65)), (200, (128, 127, 193))])
def test_gradients_of_transformed_tensors(T, lens, D, dtype):
    from tests.helpers import rand_inputs
    from kerneldev_b200 import flash_attention, generate_hadamard_signs, hadamard_transform
    B, H = len(lens), 3
    q, k, v, do = rand_inputs(B, H, T, D, dtype, T + D, DEV)
    lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    signs = torch.cat([torch.ones(1, device=DEV), generate_hadamard_signs(H, D).flatten()])[1:].view(H, D)   # not on 16 bytes
    for x in (q, k, v):
        x.requires_grad_()
    got = torch.autograd.grad(flash_attention(q, k, v, lens=lens, hadamard_signs=signs), (q, k, v), do)
    qt, kt = hadamard_transform(q, signs), hadamard_transform(k, signs)
    o = flash_attention(qt, kt, v, lens=lens)
    dqt, = torch.autograd.grad(o, qt, do, retain_graph=True)
    want = torch.autograd.grad(o, (q, k, v), do)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    # A rounding to p bits moves a number by u = 2^-p of it at most (bfloat16 p = 8, float16 p = 11). The second path rounds dQ before the
    # transform as well, which is orthogonal: the elements' errors move a result by u times the row's 2-norm at most. Both round the result, by u
    # of it each; 1.01 for the products of these, and for the sums of up to two key tiles, which may come in another order (1e-6)
    u = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-11
    bound = 1.01 * u * (dqt.float().norm(dim=-1, keepdim=True) + 2 * want[0].float().abs()) + 1e-6
    assert bool(((got[0].float() - want[0].float()).abs() <= bound).all())


# 33 sequences of 64 tiles are more than a plan holds the bits of PARTIAL tiles for: the kernels form them, and the results are those of
# two calls on parts of the batch, whose plans have them. Rules with spans, prefix and [MASKQ] strewn over all tiles; causal
@pytest.mark.parametrize("rules", [True, False])
@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (48, torch.float32), (128, torch.float16), (80, torch.float32)])
def test_batches_without_mask_bits_in_the_plan(D, dtype, rules):
    from kerneldev_b200 import _capi, clear_plan_cache, flash_attention
    B, H, T, half = 33, 1, 8100, 17
    assert _capi.plan_layout(B, T).total < 8 << 20 < 128 << 20 < _capi.plan_layout(half, T).total
    g = torch.Generator(device=DEV).manual_seed(D)
    q, k, v, do = (torch.randn((B, H, T, D), generator=g, device=DEV).to(dtype) for _ in range(4))
    options = {"lens": torch.randint(1, T + 1, (B,), generator=g, device=DEV).to(torch.int32)}
    if rules:   # runs of 1 to 400 tokens: prefix, context or one of four spans; a [MASKQ] in every tile
        t = torch.arange(T, device=DEV)
        run = t // torch.randint(1, 401, (B, 1), generator=g, device=DEV)
        kind = torch.randint(-3, 5, (B, T), generator=g, device=DEV).gather(1, run)
        options.update(in_span=kind > 0, span_id=torch.where(t % 128 == 77, -1, kind.clamp_min(0)), is_prefix=kind == 0)

    def call(lo, hi, deterministic):
        x = [y[lo:hi].detach().requires_grad_() for y in (q, k, v)]
        o, lse = flash_attention(*x, return_lse=True, deterministic=deterministic, **{n: y[lo:hi] for n, y in options.items()})
        return (o.detach(), lse, *torch.autograd.grad(o, x, do[lo:hi]))

    for deterministic in (False, True):
        whole, parts = call(0, B, deterministic), zip(call(0, half, deterministic), call(half, B, deterministic))
        for n, (got, want) in enumerate(zip(whole, map(torch.cat, parts))):
            # fused dQ: fp32 sums in no fixed order, then a rounding to the type (2^-8 covers bf16's, of any element)
            assert torch.equal(got, want) or (n == 2 and not deterministic and float((got - want).norm()) <= 2.0**-8 * float(want.norm()))
    clear_plan_cache()
    del q, k, v, do, options, whole, parts, got, want
    torch.cuda.empty_cache()   # later tests' plans would hold on to segments of this size


# More items than SMs, so that CTAs take several one after the other; chunks of heads of equal and (at T = 1280) unequal size. `lens` makes runs of empty items longer than the ring of
# item headers between items with work (both tile widths; an odd number of query tiles; a last tile of 1 and of 127 tokens)
@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (128, torch.float16), (80, torch.bfloat16)])
@pytest.mark.parametrize("T,n_full", [(513, 1), (895, 2), (1280, 5)])
def test_many_items_per_cta_with_empty_ones_between(T, n_full, D, dtype, deterministic):
    from tests.helpers import assert_close, random_meta
    from kerneldev_b200 import flash_attention
    B, H = 12, 23
    ins, sid, pre = random_meta(T + D, B, T)
    lens = np.array([T if b % (B // n_full) == 0 else (0, 3, 129)[b % 3] for b in range(B)], np.int32)
    meta = {"in_span": torch.as_tensor(ins, device=DEV), "span_id": torch.as_tensor(sid, device=DEV),
            "is_prefix": torch.as_tensor(pre, device=DEV), "lens": torch.as_tensor(lens, device=DEV)}
    g = torch.Generator(device=DEV).manual_seed(T)
    q, k, v, do = (torch.randn((B, H, T, D), generator=g, device=DEV).to(dtype) for _ in range(4))
    for x in (q, k, v):
        x.requires_grad_()
    o = flash_attention(q, k, v, deterministic=deterministic, **meta)
    grads = torch.autograd.grad(o, (q, k, v), do)
    mask = torch.as_tensor(ao.dense_mask(T, ins, sid, pre, lens))
    for b, h in [(0, 0), (0, H - 1), (1, 3), (2, 5), (B - 1, H - 1), (B - B // n_full, 7)]:
        sl = lambda x: x.detach()[b:b + 1, h:h + 1].float().cpu()
        want = ao.attention_fwd_bwd(sl(q), sl(k), sl(v), sl(do), mask[b:b + 1])
        # the operands P and dS are rounded to 16 bits before their products: the repository's tolerance for that
        assert_close("O", sl(o), want[0])
        for name, got, ref in zip(("dQ", "dK", "dV"), grads, want[-3:]):
            assert_close(name, sl(got), ref)


# Forward above head dim 64: an issuing warp per query tile walks a common list. A tile of prefix tokens in the middle of the
# sequence sees the prefix only, its pair's other tile nearly everything: runs of entries of one tile, longer than the rings of
# K and V tiles, for tile 1 of a pair (tile 8) and for tile 0 (tile 13); a tile beyond the sequence length; an odd number of tiles;
# scores whose maximum grows from tile to tile (O is rescaled). With six heads a call has 84 or 96 pairs, which are its items; with three, 42 or
# 48, whose tiles are items of their own
@pytest.mark.parametrize("H", [6, 3])
@pytest.mark.parametrize("D,dtype", [(128, torch.bfloat16), (80, torch.float16)])
@pytest.mark.parametrize("T,length", [(128 * 14, 128 * 14), (128 * 15 - 127, 128 * 14 + 1), (128 * 14 + 5, 128 * 12)])
def test_forward_wide_unequal_lists_of_a_pair(T, length, D, dtype, H):
    from tests.helpers import assert_close, assert_lse_close
    from kerneldev_b200 import flash_attention
    B = 2
    ins, sid, pre = np.zeros((B, T), bool), np.zeros((B, T), np.int64), np.zeros((B, T), bool)
    for tile in (0, 8, 13):
        pre[:, tile * 128:(tile + 1) * 128] = True
    lens = np.array([length, T], np.int32)
    g = torch.Generator(device=DEV).manual_seed(T + D)
    q, k, v = (torch.randn((B, H, T, D), generator=g, device=DEV) for _ in range(3))
    k *= torch.linspace(0.2, 4.0, T, device=DEV)[:, None]
    q, k, v = (x.to(dtype) for x in (q, k, v))
    with torch.no_grad():
        o, lse = flash_attention(q, k, v, return_lse=True, in_span=torch.as_tensor(ins, device=DEV), span_id=torch.as_tensor(sid, device=DEV),
                                 is_prefix=torch.as_tensor(pre, device=DEV), lens=torch.as_tensor(lens, device=DEV))
    want_o, want_lse = ao.attention_forward(q.float().cpu(), k.float().cpu(), v.float().cpu(), torch.as_tensor(ao.dense_mask(T, ins, sid, pre, lens)))[:2]
    assert_close("O", o, want_o)   # P is rounded to 16 bits before its product: the repository's tolerance for that
    assert_lse_close(lse, want_lse)


# Forward above head dim 64 with more items than SMs, whose lists hold 0, 1 or 2 entries (T = 256) or up to 3 (T = 300: a pair without a second
# tile) and whose tile 1 often has none: the ring of Q tiles passes from one query tile's issuing warp to the other's. Repeats give the same bits
@pytest.mark.parametrize("D,dtype", [(128, torch.bfloat16), (80, torch.float16)])
@pytest.mark.parametrize("T", [256, 300])
def test_forward_wide_ring_of_query_tiles(T, D, dtype):
    from tests.helpers import assert_close, assert_lse_close
    from kerneldev_b200 import flash_attention
    B, H = 40, 37
    lens = np.array([(T, 100, 0, 129)[b % 4] for b in range(B)], np.int32)
    g = torch.Generator(device=DEV).manual_seed(T + D)
    q, k, v = (torch.randn((B, H, T, D), generator=g, device=DEV).to(dtype) for _ in range(3))
    call = lambda: flash_attention(q, k, v, return_lse=True, lens=torch.as_tensor(lens, device=DEV))
    with torch.no_grad():
        o, lse = call()
        for _ in range(20):
            o2, lse2 = call()
            assert torch.equal(o, o2) and torch.equal(lse, lse2)
    pick = [(b, h) for b in range(4) for h in (0, 18, H - 1)] + [(B - 1, H - 1)]
    sel = lambda x: torch.stack([x[b, h] for b, h in pick])[:, None].float().cpu()
    mask = torch.as_tensor(ao.dense_mask(T, lens=lens, causal=True))
    want_o, want_lse = ao.attention_forward(sel(q), sel(k), sel(v), torch.stack([mask[b] for b, _ in pick]))
    assert_close("O", sel(o), want_o)   # P is rounded to 16 bits before its product: the repository's tolerance for that
    assert_lse_close(sel(lse), want_lse)


# Forward items of one query tile (up to 37 pairs of tiles in a call, from five tiles per head on up to 74) and of two (38; 75): pairs with a
# second tile, without one (T = 300, 640), and with entries of the list that are EMPTY for one of them; rows beyond the sequence length; one tile
# per head is not split
@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (112, torch.float16)])
@pytest.mark.parametrize("B,H,T", [(1, 37, 200), (2, 19, 200), (2, 37, 200), (3, 25, 200), (1, 18, 300), (1, 37, 300), (4, 6, 640), (2, 7, 128 * 9 + 1),
                                   (3, 5, 128 * 9 + 1), (2, 2, 128 * 9 + 1), (74, 1, 100)])
def test_forward_items_of_one_tile(B, H, T, D, dtype):
    from tests.helpers import assert_close, assert_lse_close, random_meta, rand_inputs
    from kerneldev_b200 import flash_attention
    ins, sid, pre = random_meta(T + D, B, T)
    ins[:, 128:256], pre[:, 128:256], sid[:, 128:256] = False, True, 0   # a tile of prefix tokens: sees few others
    lens = np.array([T if b % 2 == 0 else T // 2 for b in range(B)], np.int32)
    q, k, v, _ = rand_inputs(B, H, T, D, dtype, T + H)
    with torch.no_grad():
        o, lse = flash_attention(q.to(DEV), k.to(DEV), v.to(DEV), return_lse=True, in_span=torch.as_tensor(ins, device=DEV),
                                 span_id=torch.as_tensor(sid, device=DEV), is_prefix=torch.as_tensor(pre, device=DEV),
                                 lens=torch.as_tensor(lens, device=DEV))
    want_o, want_lse = ao.attention_forward(q, k, v, torch.as_tensor(ao.dense_mask(T, ins, sid, pre, lens)))
    assert_close("O", o, want_o)   # P is rounded to 16 bits before its product: the repository's tolerance for that
    assert_lse_close(lse, want_lse)


# deterministic backward: 738 and 740 items, some five for each SM, of lists of one and two tiles
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H", [(9, 41), (10, 37)])
def test_deterministic_backward_five_items_per_sm(B, H, D):
    from tests.helpers import assert_close, rand_inputs, random_meta
    from kerneldev_b200 import flash_attention
    T = 200
    ins, sid, pre = random_meta(D, B, T)
    q, k, v, do = rand_inputs(B, H, T, D, torch.bfloat16, D + B)
    dev = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    o = flash_attention(*dev, deterministic=True, in_span=torch.as_tensor(ins, device=DEV), span_id=torch.as_tensor(sid, device=DEV),
                        is_prefix=torch.as_tensor(pre, device=DEV))
    grads = torch.autograd.grad(o, dev, do.to(DEV))
    mask = torch.as_tensor(ao.dense_mask(T, ins, sid, pre))
    for b, h in [(0, 0), (1, H - 1), (B - 1, 1), (B - 1, H - 1)]:
        want = ao.attention_fwd_bwd(*(x[b:b + 1, h:h + 1].float() for x in (q, k, v, do)), mask[b:b + 1])
        for name, got, ref in zip(("dQ", "dK", "dV"), grads, want[-3:]):
            assert_close(name, got[b:b + 1, h:h + 1], ref)   # P and dS are rounded to 16 bits: the repository's tolerance for that


# a row of exactly one chunk of 4096 tokens, one more, and several: first [CLS] in the first, a later, or no chunk
@pytest.mark.parametrize("T", [1, 127, 4096, 4097, 12289])
def test_metadata_chunks(T):
    from kerneldev_b200 import metadata_from_tokens
    rng = np.random.default_rng(T)
    x = rng.integers(6, 300, size=(4, T))
    marks = rng.random((4, T)) < 0.05
    x[marks] = rng.integers(2, 6, size=int(marks.sum()))
    x[0, T - 1] = x[1, T // 2] = x[2, 0] = 1
    got = [t.cpu().numpy() for t in metadata_from_tokens(torch.as_tensor(x, device=DEV))]
    for g, w in zip(got, ao.metadata_from_tokens(x)):
        assert np.array_equal(g, w)


def test_host_thread_without_a_cuda_context():
    """A forward and backward whose every allocation comes from the cache, in a host thread that has not used CUDA before."""
    import threading
    from kerneldev_b200 import flash_attention
    q, k, v, do = (torch.randn(1, 2, 200, 64, device=DEV, dtype=torch.bfloat16) for _ in range(4))
    out = []

    def run():
        a, b, c = (x.detach().requires_grad_() for x in (q, k, v))
        o = flash_attention(a, b, c)
        out.append((o.detach(), *torch.autograd.grad(o, (a, b, c), do)))

    run()
    first = out.pop()
    worker = threading.Thread(target=run)
    worker.start()
    worker.join()
    assert len(out) == 1
    for x, y in zip(first, out[0]):
        assert torch.allclose(x.float(), y.float(), atol=1e-2, rtol=1e-2)


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("B,H,T,D,layout", [(1, 1, 1, 16, "bhtd"), (2, 3, 129, 48, "bthd"), (1, 2, 300, 80, "bhtd"), (2, 2, 257, 64, "bthd"), (1, 3, 640, 128, "bthd"), (1, 2, 383, 112, "bhtd")])
def test_float32_results_are_not_rounded_to_16_bits(B, H, T, D, layout, deterministic):
    """float32 O, dQ, dK and dV are written by the attention kernels: rows and columns at the edges of tiles and boxes, memory orders,
    sequences that end early (rows without keys, key tiles without queries). Errors are those of the float16 operands alone."""
    from tests.helpers import rand_inputs
    from kerneldev_b200 import flash_attention
    q, k, v, do = (x.to(DEV) for x in rand_inputs(B, H, T, D, torch.float32, seed=T + D))
    if layout == "bthd":
        q, k, v, do = (x.transpose(1, 2).contiguous().transpose(1, 2) for x in (q, k, v, do))
    lens = torch.tensor([T] + [T // 2] * (B - 1), dtype=torch.int32, device=DEV)
    qg, kg, vg = (x.detach().clone(memory_format=torch.preserve_format).requires_grad_() for x in (q, k, v))
    o = flash_attention(qg, kg, vg, lens=lens, causal=True, out_layout="input", deterministic=deterministic)
    grads = torch.autograd.grad(o, (qg, kg, vg), do, retain_graph=True)
    mask = ao.dense_mask(T, None, None, None, lens.cpu().numpy(), causal=True, B=B)
    half = [x.half().float().cpu() for x in (q, k, v, do)]
    ro, _, *rg = ao.attention_fwd_bwd(*half, mask)
    for got, ref, like in zip((o, *grads), (ro, *rg), (q, q, k, v)):
        assert got.dtype == torch.float32 and got.stride() == like.stride()
        # P, dS and O inside delta are float16 (2^-11 relative each); a handful of such terms of the size of the result. With one
        # token dQ and dK are the difference of two equal fp32 sums of products of size 1 (2^-24 each).
        assert float((got.detach().cpu() - ref).norm()) <= 4 * 2.0**-11 * float(ref.norm()) + D * 2.0**-22
        if T > 1:
            assert not torch.equal(got.half().float(), got)
    # O is not what the backward reads, so it may be written to; dO may have any strides
    with torch.no_grad():
        o.zero_()
    again = torch.autograd.grad(o, (qg, kg, vg), do.transpose(1, 2).contiguous().transpose(1, 2), retain_graph=True)
    expanded = torch.autograd.grad(o, (qg, kg, vg), torch.ones((1, 1, 1, 1), device=DEV).expand(B, H, T, D), retain_graph=True)
    ones = torch.autograd.grad(o, (qg, kg, vg), torch.ones((B, H, T, D), device=DEV))
    for x, y in list(zip(grads, again)) + list(zip(expanded, ones)):
        assert float((x - y).norm()) <= (0.0 if deterministic else 1e-5) * float(y.norm())   # dQ's sums have no fixed order


@pytest.mark.parametrize("B,H,T,D", [(6, 40, 300, 64), (6, 40, 300, 128), (40, 9, 129, 48), (3, 50, 513, 112)])
def test_deterministic_backward_takes_further_items(B, H, T, D):
    """More tiles than SMs, so that CTAs of both kernels run on into other heads, tiles and sequences; runs of tiles without entries
    (sequences of no or few tokens) between those with some, longer than the ring of item headers. Twice the same bits."""
    from tests.helpers import assert_close, rand_inputs
    from kerneldev_b200 import flash_attention
    q, k, v, do = (x.to(DEV) for x in rand_inputs(B, H, T, D, torch.bfloat16, seed=T + D))
    lens = torch.tensor([(T, 0, 1, T // 2, T - 1, 128)[b % 6] for b in range(B)], dtype=torch.int32, device=DEV)
    qg, kg, vg = (x.detach().requires_grad_() for x in (q, k, v))
    o = flash_attention(qg, kg, vg, lens=lens, causal=True, deterministic=True)
    one = torch.autograd.grad(o, (qg, kg, vg), do, retain_graph=True)
    two = torch.autograd.grad(o, (qg, kg, vg), do)
    assert all(torch.equal(x, y) for x, y in zip(one, two))
    mask = ao.dense_mask(T, None, None, None, lens.cpu().numpy(), causal=True, B=B)
    heads = [0, H // 2, H - 1]
    _, _, *ref = ao.attention_fwd_bwd(*(x[:, heads].cpu() for x in (q, k, v, do)), mask)
    for name, got, want in zip(("dQ", "dK", "dV"), one, ref):
        assert_close(name, got[:, heads], want)


# more items than SMs: O leaves through boxes of 32 rows and 32 columns (head dims that end inside the first or the second box, last rows
# of a tile of 1, 31, 32 and 97); 148 items and fewer: by the threads themselves
@pytest.mark.parametrize("layout", ["bhtd", "bthd"])
@pytest.mark.parametrize("B,H,T,D", [(15, 10, 129, 16), (15, 10, 159, 48), (19, 8, 160, 32), (38, 4, 225, 64), (37, 4, 225, 64)])
def test_forward_output_boxes(B, H, T, D, layout):
    from tests.helpers import assert_close, rand_inputs
    from kerneldev_b200 import flash_attention
    q, k, v, _ = (x.to(DEV) for x in rand_inputs(B, H, T, D, torch.float16, seed=D + T))
    if layout == "bthd":
        q, k, v = (x.transpose(1, 2).contiguous().transpose(1, 2) for x in (q, k, v))
    lens = torch.tensor([(T, T // 3, 0)[b % 3] for b in range(B)], dtype=torch.int32, device=DEV)
    o = flash_attention(q, k, v, lens=lens, causal=True, out_layout="input" if layout == "bthd" else "contiguous")
    mask = ao.dense_mask(T, None, None, None, lens.cpu().numpy(), causal=True, B=B)
    assert_close("O", o, ao.attention_forward(q.float().cpu(), k.float().cpu(), v.float().cpu(), mask)[0])


@pytest.mark.parametrize("B,H,T,D,dtype", [(1, 4, 300, 64, torch.bfloat16), (1, 8, 173, 128, torch.float16), (1, 3, 513, 64, torch.float32), (2, 2, 257, 128, torch.float32)])
def test_deterministic_backward_behind_one_another(monkeypatch, B, H, T, D, dtype):
    """The dK/dV kernel starts beside the end of the dQ kernel and reads what the delta kernel of the same call has written. Calls without
    a pause between them, whose scratch is the memory of earlier calls with other gradients, give the bits of calls one by one."""
    monkeypatch.setenv("KD_CHECK_STATUS", "0")   # a check waits for the device
    from tests.helpers import assert_close, rand_inputs
    from kerneldev_b200 import flash_attention
    q, k, v, _ = (x.to(DEV).requires_grad_() for x in rand_inputs(B, H, T, D, dtype, seed=T + D))
    g = torch.Generator(device=DEV).manual_seed(D)
    dos = [(torch.randn((B, H, T, D), generator=g, device=DEV) * 2.0 ** (i % 5 - 2)).to(dtype) for i in range(24)]
    o = flash_attention(q, k, v, deterministic=True)
    torch.cuda.synchronize()
    together = [torch.autograd.grad(o, (q, k, v), do, retain_graph=True) for do in dos]
    torch.cuda.synchronize()
    for i, do in enumerate(dos):
        alone = torch.autograd.grad(o, (q, k, v), do, retain_graph=True)
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(together[i], alone)), i
    mask = ao.dense_mask(T, None, None, None, None, causal=True, B=B)
    for i in (1, 13, 23):
        _, _, *ref = ao.attention_fwd_bwd(*(x.detach().float().cpu() for x in (q, k, v, dos[i])), mask)
        for name, got, want in zip(("dQ", "dK", "dV"), together[i], ref):
            assert_close(name, got, want)   # P and dS are rounded to 16 bits: the repository's tolerance for that


@pytest.mark.parametrize("D", [64, 80])
def test_forward_into_rows_in_descending_order(D):
    """O with a negative time stride, which no tensor map describes, in a call with more items than SMs: written row by row, and the
    call, which succeeds, leaves no message of a refused map behind."""
    import ctypes
    from tests.helpers import rand_inputs
    from kerneldev_b200 import _capi
    from kerneldev_b200.original_kernel import _forward, _kd_tensor, _params
    from kerneldev_b200.plan import AttentionPlan
    B, H, T = 15, 10, 159
    q, k, v, _ = (x.to(DEV) for x in rand_inputs(B, H, T, D, torch.bfloat16, seed=D))
    plan = AttentionPlan(B, T, torch.device(DEV))
    want, lse = _forward(q, k, v, plan, 0.125)
    back = torch.empty_like(want)
    lib = _capi.load()
    p = _params(q, k, v, back, torch.empty_like(lse), plan, 0.125)
    p.D = 7
    assert lib.kd_attn_fwd(ctypes.byref(p), None) != 0
    message = lib.kd_last_error()
    p.D = D
    p.o = _capi.KdTensor(back.data_ptr() + (T - 1) * D * 2, H * T * D, T * D, -D)
    torch.cuda.synchronize()
    assert lib.kd_attn_fwd(ctypes.byref(p), torch.cuda.current_stream().cuda_stream) == 0
    assert message and lib.kd_last_error() == message
    assert torch.equal(back.flip(2), want)


# dK and dV of the deterministic backward with strides that no tensor map describes: written row by row, key tiles that no query sees too
@pytest.mark.parametrize("T,lens", [(159, (159, 100)), (385, (385, 129))])
@pytest.mark.parametrize("D", [48, 64, 80])
def test_deterministic_backward_into_rows_in_descending_order(T, lens, D):
    import ctypes
    from tests.helpers import rand_inputs
    from kerneldev_b200 import _capi
    from kerneldev_b200.original_kernel import _backward, _forward, _kd_tensor, _params
    from kerneldev_b200.plan import AttentionPlan
    B, H = 2, 7
    q, k, v, do = (x.to(DEV) for x in rand_inputs(B, H, T, D, torch.bfloat16, seed=T + D))
    plan = AttentionPlan(B, T, torch.device(DEV), lens=torch.tensor(lens, dtype=torch.int32, device=DEV), causal=True)
    o, lse = _forward(q, k, v, plan, 0.125)
    want = _backward(q, k, v, o, lse, do, plan, 0.125, deterministic=True)
    dq, dk, dv = (torch.full_like(q, float("nan")) for _ in range(3))
    delta = torch.empty_like(lse)
    p = _params(q, k, v, o, lse, plan, 0.125)
    p.d_o, p.dq, p.delta, p.bwd_mode = _kd_tensor(do), _kd_tensor(dq), delta.data_ptr(), 0
    p.dk, p.dv = (_capi.KdTensor(x.data_ptr() + (T - 1) * D * 2, H * T * D, T * D, -D) for x in (dk, dv))
    lib = _capi.load()
    torch.cuda.synchronize()
    assert lib.kd_attn_bwd(ctypes.byref(p), torch.cuda.current_stream().cuda_stream) == 0, lib.kd_last_error()
    for got, ref in zip((dq, dk.flip(2), dv.flip(2)), want):
        assert torch.equal(got, ref)


# 312 pairs of query tiles and 468 key tiles (odd: 780 tiles, some of 1 token), more than SMs: CTAs of all float32 kernels run on into further items, among them runs
# of tiles without keys or queries. O leaves as float32 beside the 16-bit O of the boxes, dK and dV through both staging boxes between dQ tiles
@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("B,H,T,D", [(12, 13, 300, 48), (12, 13, 300, 64), (12, 13, 300, 80), (12, 13, 300, 128), (12, 13, 513, 64), (12, 13, 513, 128)])
def test_float32_calls_with_many_items(B, H, T, D, deterministic):
    from tests.helpers import rand_inputs
    from kerneldev_b200 import flash_attention
    q, k, v, do = (x.to(DEV) for x in rand_inputs(B, H, T, D, torch.float32, seed=T + D))
    lens = torch.tensor([(T, 0, 0, 1, T // 2, T - 1)[b % 6] for b in range(B)], dtype=torch.int32, device=DEV)
    qg, kg, vg = (x.detach().requires_grad_() for x in (q, k, v))
    o = flash_attention(qg, kg, vg, lens=lens, causal=True, deterministic=deterministic)
    got = (o.detach(), *torch.autograd.grad(o, (qg, kg, vg), do))
    with torch.no_grad():   # no backward to come: no 16-bit O
        assert torch.equal(flash_attention(q, k, v, lens=lens, causal=True), got[0])
    heads = [0, 6, H - 1]
    mask = ao.dense_mask(T, None, None, None, lens.cpu().numpy(), causal=True, B=B)
    ro, _, *rg = ao.attention_fwd_bwd(*(x[:, heads].half().float().cpu() for x in (q, k, v, do)), mask)
    for x, ref in zip(got, (ro, *rg)):
        x = x[:, heads].cpu()
        for b in range(B):   # the bound of test_float32_results_are_not_rounded_to_16_bits, sequence by sequence
            assert float((x[b] - ref[b]).norm()) <= 4 * 2.0**-11 * float(ref[b].norm()) + D * 2.0**-22


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("B,H,T,D,dtype", [(1, 4, 300, 64, torch.bfloat16), (2, 40, 257, 128, torch.float16), (1, 3, 300, 64, torch.float32), (2, 40, 257, 128, torch.float32)])
def test_captured_forward_and_backward(monkeypatch, B, H, T, D, dtype, deterministic):
    """A graph of a forward and backward, replayed without a pause on inputs that change in place, gives what the calls give."""
    monkeypatch.setenv("KD_CHECK_STATUS", "0")   # a check waits for the device
    from tests.helpers import rand_inputs
    from kerneldev_b200 import flash_attention
    sets = [[x.to(DEV) for x in rand_inputs(B, H, T, D, dtype, seed=T + D + i)] for i in range(4)]
    q, k, v, do = (x.clone() for x in sets[0])
    lens = torch.tensor([T] + [T // 2] * (B - 1), dtype=torch.int32, device=DEV)

    def call(q, k, v, do):   # the node by hand: the engine's own streams have no place in a capture
        o = flash_attention(*(x.detach().requires_grad_() for x in (q, k, v)), lens=lens, deterministic=deterministic)
        return (o.detach(), *o.grad_fn(do))

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call(q, k, v, do)   # builds the plan
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            outs = call(q, k, v, do)
        replayed = []
        for xs in sets:
            for x, y in zip((q, k, v, do), xs):
                x.copy_(y)
            graph.replay()
            replayed.append([x.clone() for x in outs])
        torch.cuda.synchronize()
        for xs, got in zip(sets, replayed):
            for x, y in zip(got, call(*xs)):
                # fused dQ: fp32 sums in no fixed order, then a rounding to the type (2^-8 covers bf16's, of any element)
                assert torch.equal(x, y) or (not deterministic and float((x - y).norm()) <= 2.0**-8 * float(y.norm()))
