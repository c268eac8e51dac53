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


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("lse_off,delta_off", [(1, 0), (0, 2), (3, 1)])
def test_fused_backward_with_scalars_off_16_bytes(D, lse_off, delta_off):
    """LSE and delta need no alignment beyond a float's: their rows are copied 16 bytes at a time only where they begin on
    16 bytes. Bit-equal dK and dV (fixed order of sums), dQ within the rounding of its unordered fp32 sums."""
    from kerneldev_b200.original_kernel import _backward, _forward
    from kerneldev_b200.plan import AttentionPlan
    B, H, T = 2, 3, 388
    g = torch.Generator(device=DEV).manual_seed(D)
    q, k, v, do = (torch.randn((B, H, T, D), generator=g, device=DEV).to(torch.bfloat16) for _ in range(4))
    plan = AttentionPlan(B, T, DEV)
    o, lse = _forward(q, k, v, plan, D ** -0.5)
    want = _backward(q, k, v, o, lse, do, plan, D ** -0.5)
    n = B * H * T
    shifted = torch.empty(n + 4, device=DEV)[lse_off:lse_off + n].view(B, H, T).copy_(lse)
    delta = torch.empty(n + 4, device=DEV)[delta_off:delta_off + n].view(B, H, T)
    assert shifted.data_ptr() % 16 == 4 * lse_off and delta.data_ptr() % 16 == 4 * delta_off
    bufs = [torch.empty_like(q), torch.empty_like(q), torch.empty_like(q), delta, torch.empty((B, H, T, 64 if D <= 64 else 128), device=DEV)]
    got = _backward(q, k, v, o, shifted, do, plan, D ** -0.5, 0, bufs)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    # at most four key tiles add up in another order, then one rounding to bf16, whose neighbours differ by 2^-7 of the value at most
    assert torch.allclose(got[0].float(), want[0].float(), rtol=2.0**-7, atol=1e-4)


def test_deterministic_backward_with_plans_at_reused_addresses(monkeypatch):
    """Plans of very different masks one after the other in the same memory, without a synchronisation between: each launch
    has to see the plan of its own call, whatever an SM may hold of the one before."""
    from kerneldev_b200 import clear_plan_cache, flash_attention
    monkeypatch.setenv("KD_CHECK_STATUS", "0")
    B, H, T, D = 2, 4, 1024, 64
    g = torch.Generator(device=DEV).manual_seed(5)
    q, k, v, do = (torch.randn((B, H, T, D), generator=g, device=DEV).to(torch.bfloat16) for _ in range(4))
    for x in (q, k, v):
        x.requires_grad_()
    spans = torch.zeros((B, T), dtype=torch.bool, device=DEV)
    spans[:, 300:900] = True
    ids = (torch.arange(T, device=DEV) // 96 + 1).expand(B, T) * spans
    masks = [dict(causal=True), dict(causal=False), dict(in_span=spans, span_id=ids), dict(lens=torch.tensor([130, T], dtype=torch.int32, device=DEV))]

    def run(m):
        clear_plan_cache()   # the plan of the call before goes back to the allocator
        o = flash_attention(q, k, v, deterministic=True, **m)
        return torch.autograd.grad(o, (q, k, v), do)

    want = []
    for m in masks:
        want.append(run(m))
        torch.cuda.synchronize()
    order = np.random.default_rng(0).integers(0, len(masks), 60)
    got = [run(masks[i]) for i in order]
    for i, grads in zip(order, got):
        assert all(torch.equal(a, b) for a, b in zip(grads, want[i]))


def _out_of_memory(call):
    """call() with the allocator limited to what it holds."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + 2**23) / torch.cuda.get_device_properties(0).total_memory)
    try:
        with pytest.raises(torch.cuda.OutOfMemoryError):
            call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


def test_out_of_memory_keeps_its_type():
    from kerneldev_b200 import cocktail_scores, flash_attention
    q = torch.zeros((4, 16, 2048, 64), device=DEV, dtype=torch.bfloat16, requires_grad=True)
    _out_of_memory(lambda: flash_attention(q, q, q))
    o = flash_attention(q, q, q)
    _out_of_memory(lambda: torch.autograd.grad(o, q, torch.zeros_like(o)))
    x = torch.zeros((8, 4096, 512), device=DEV, requires_grad=True)
    tokens = torch.full((8, 4096), 3, dtype=torch.int64, device=DEV)   # a row of spans: the saved means are as large as x
    _out_of_memory(lambda: cocktail_scores(x, tokens))


def test_library_errors_in_the_backward_keep_their_type():
    """A hook that gives O back off a 16-byte boundary: kd_attn_bwd refuses it on the host."""
    from kerneldev_b200 import _capi, flash_attention
    q, k, v = (torch.randn((1, 2, 200, 64), device=DEV).to(torch.bfloat16).requires_grad_() for _ in range(3))
    n = q.numel()

    def unpack(t):
        if t.dtype != torch.bfloat16:
            return t
        return torch.empty(n + 8, dtype=t.dtype, device=DEV)[4:4 + n].view(t.shape).copy_(t)

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach().clone(), unpack):
        o = flash_attention(q, k, v)
    with pytest.raises(_capi.KdError, match="multiples of 16"):
        torch.autograd.grad(o, (q, k, v), torch.ones_like(o))


def test_errors_of_saved_tensor_hooks_come_through():
    from kerneldev_b200 import flash_attention

    class Stop(Exception):
        pass

    def pack(t):
        raise Stop

    q = torch.zeros((1, 1, 128, 64), device=DEV, dtype=torch.bfloat16, requires_grad=True)
    with pytest.raises(Stop), torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        flash_attention(q, q, q)


@pytest.mark.parametrize("arg", [0, 1, 2])
def test_forward_mode_ad_is_refused(arg):
    """There is no formula for tangents; a result without one would read as a derivative of zero."""
    import torch.autograd.forward_ad as fwd
    from kerneldev_b200 import cocktail_scores, flash_attention
    qkv = [torch.zeros((1, 1, 128, 64), device=DEV, dtype=torch.bfloat16) for _ in range(3)]
    x = torch.zeros((1, 64, 16), device=DEV)
    with fwd.dual_level():
        qkv[arg] = fwd.make_dual(qkv[arg], torch.ones_like(qkv[arg]))
        with pytest.raises(NotImplementedError, match="forward mode AD"):
            flash_attention(*qkv)
        with pytest.raises(NotImplementedError, match="forward mode AD"):
            cocktail_scores(fwd.make_dual(x, torch.ones_like(x)), _span_tokens(1, 64))


def test_tracing_is_refused():
    """A trace would hold the allocation of the results without the kernels that fill them."""
    from torch.fx.experimental.proxy_tensor import make_fx
    from kerneldev_b200 import cocktail_scores, flash_attention
    q = torch.zeros((1, 1, 128, 64), device=DEV, dtype=torch.bfloat16)
    x, tokens = torch.zeros((1, 64, 16), device=DEV), _span_tokens(1, 64)
    for trace in (lambda f, a: make_fx(f)(a), torch.jit.trace):
        with pytest.raises(RuntimeError, match="cannot be traced"):
            trace(lambda a: flash_attention(a, a, a), q)
        with pytest.raises(RuntimeError, match="cannot be traced"):
            trace(lambda a: cocktail_scores(a, tokens), x)


def test_allocations_are_seen_by_dispatch_modes():
    """A mode of the caller's sees the tensors that a call allocates; one that hands out tensors without memory makes the call fail."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.utils._python_dispatch import TorchDispatchMode
    from kerneldev_b200 import cocktail_scores, flash_attention, metadata_from_tokens
    seen = []

    class Record(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            out = func(*args, **(kwargs or {}))
            if func.overloadpacket in (torch.ops.aten.empty, torch.ops.aten.empty_like):
                seen.append((tuple(out.shape), out.dtype))
            return out

    q = torch.randn((1, 2, 150, 64), device=DEV).bfloat16()
    x, tokens = torch.randn((1, 64, 16), device=DEV), _span_tokens(1, 64)
    want, want_wide = flash_attention(q, q, q, causal=True), flash_attention(q.float(), q.float(), q.float(), causal=True)
    with Record():
        o, lse = flash_attention(q, q, q, causal=True, return_lse=True)
        wide = flash_attention(q.float(), q.float(), q.float(), causal=True)
        scores = cocktail_scores(x, tokens)
        in_span, _, _ = metadata_from_tokens(tokens)
    assert torch.equal(o, want) and torch.equal(wide, want_wide)
    for t in (o, lse, wide, scores, in_span):
        assert (tuple(t.shape), t.dtype) in seen
    with FakeTensorMode(allow_non_fake_inputs=True), pytest.raises(RuntimeError):
        flash_attention(q, q, q, causal=True)


def test_new_memory_is_filled_where_torch_fills_it():
    """torch.utils.deterministic.fill_uninitialized_memory: what a call allocates and does not write (here dK and dV) reads as NaN."""
    from kerneldev_b200.original_kernel import _backward, _forward
    from kerneldev_b200.plan import AttentionPlan
    q = torch.randn((1, 2, 150, 64), device=DEV).bfloat16()
    plan = AttentionPlan(1, 150, torch.device(DEV))
    o, lse = _forward(q, q, q, plan, 0.125)
    torch.use_deterministic_algorithms(True)
    try:
        dq, dk, dv = _backward(q, q, q, o, lse, q, plan, 0.125, 1, deterministic=True)
    finally:
        torch.use_deterministic_algorithms(False)
    assert torch.isfinite(dq).all() and torch.isnan(dk).all() and torch.isnan(dv).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_undefined_gradients_count_as_zeros(dtype):
    from kerneldev_b200 import cocktail_scores, flash_attention

    class NoGradient(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return x.clone()

        @staticmethod
        def backward(ctx, g):
            return None

    q, k, v = (torch.randn((1, 2, 150, 64), device=DEV).to(dtype).requires_grad_() for _ in range(3))
    x = torch.randn((1, 64, 16), device=DEV).to(dtype).requires_grad_()
    o, s = NoGradient.apply(flash_attention(q, k, v)), NoGradient.apply(cocktail_scores(x, _span_tokens(1, 64)))
    for g, t in zip(torch.autograd.grad(o.sum() + s.sum(), (q, k, v, x)), (q, k, v, x)):
        assert g.shape == t.shape and g.dtype == dtype and not g.any()


@pytest.mark.parametrize("signs", [False, True])
@pytest.mark.parametrize("dtype,other", [(torch.float32, torch.bfloat16), (torch.float32, torch.float16), (torch.float32, torch.float64),
                                         (torch.bfloat16, torch.float32), (torch.float16, torch.bool)])
def test_node_called_by_hand(dtype, other, signs):
    """The engine brings a gradient in the output's type and shape, a caller of the node may not: it is converted or refused, never
    read as what it is not."""
    from kerneldev_b200 import flash_attention, generate_hadamard_signs
    g = torch.Generator(device=DEV).manual_seed(4)
    q, k, v = (torch.randn((1, 2, 150, 64), generator=g, device=DEV).to(dtype).requires_grad_() for _ in range(3))
    do = torch.randint(0, 2, (1, 2, 150, 64), generator=g, device=DEV).to(dtype)   # exact in every type
    o = flash_attention(q, k, v, deterministic=True, hadamard_signs=generate_hadamard_signs(2, 64) if signs else None)
    want = o.grad_fn(do)
    for x, y in zip(o.grad_fn(do.to(other)), want):
        assert x.dtype == dtype and torch.equal(x, y)
    for wrong in (do[:, :, :100], do[:, :1], do.cpu()):
        with pytest.raises(ValueError, match="the gradient of an output"):
            o.grad_fn(wrong)


def test_other_threads_run_while_the_host_waits(monkeypatch):
    """KD_CHECK_STATUS=1 waits for the device in every call: here behind a busy stream."""
    import threading
    import time
    from kerneldev_b200 import flash_attention
    monkeypatch.setenv("KD_CHECK_STATUS", "1")
    q = torch.zeros((1, 2, 128, 64), device=DEV, dtype=torch.bfloat16)
    flash_attention(q, q, q)
    steps, stop = [0], threading.Event()

    def work():
        while not stop.is_set():
            steps[0] += 1
            time.sleep(0.001)

    worker = threading.Thread(target=work)
    worker.start()
    torch.cuda._sleep(500_000_000)   # a quarter of a second or more
    before, t0 = steps[0], time.perf_counter()
    flash_attention(q, q, q)
    waited, done = time.perf_counter() - t0, steps[0] - before
    stop.set()
    worker.join()
    assert waited > 0.1 and done > 20


def test_a_live_plan_keeps_its_status_word():
    """A report that waits in a plan's host word survives any number of further plans, and no two live plans share one."""
    from kerneldev_b200 import _capi
    from kerneldev_b200.plan import AttentionPlan
    plan = AttentionPlan(1, 128, DEV)
    plan._status_host.fill_(_capi.KD_STATUS_TIMEOUT | 0x104)
    for _ in range(1100):
        AttentionPlan(1, 16, DEV)
    with pytest.raises(RuntimeError, match="timed out"):
        plan.poll()
    live = [AttentionPlan(1, 16, DEV) for _ in range(1100)]
    assert len({p._status_host.data_ptr() for p in live + [plan]}) == 1101


@pytest.mark.parametrize("late", [False, True])
def test_a_plan_that_leaves_the_cache_still_reports(late):
    """What the last launch of a step reports, before its plan makes room for the next step's or behind that (the host is ahead of the
    device), is raised once, by a call with new metadata, which then works."""
    from kerneldev_b200 import _capi, clear_plan_cache
    from kerneldev_b200.plan import _CACHE, get_plan
    new = lambda: torch.tensor([100], dtype=torch.int32, device=DEV)
    plan_of = lambda lens: get_plan(1, 128, DEV, lens=lens)
    clear_plan_cache()
    lens = new()
    words = [plan_of(lens)._status_host]
    lens, held = new(), [new()]   # (all at once: no two have the same memory)
    if late:
        plan_of(held[0])   # the first plan goes here
    words[0].fill_(_capi.KD_STATUS_TIMEOUT | 0x104)
    lens = new()
    with pytest.raises(RuntimeError, match="timed out.*0x104"):
        plan_of(lens)
    assert int(words[0]) == 0 and len(_CACHE) == 1 + late
    plan = plan_of(lens)
    held.append(new())
    plan_of(held[-1])
    assert plan_of(lens) is plan and len(_CACHE) == 2 + late
    clear_plan_cache()


def test_one_row_may_have_more_embeddings_than_tokens():
    from kerneldev_b200 import cocktail_scores
    T, more, C = 130, 37, 24
    tokens = _span_tokens(1, T)
    x = torch.randn((1, T + more, C), generator=torch.Generator(device=DEV).manual_seed(2), device=DEV)
    a, b = x.clone().requires_grad_(), x[:, :T].clone().requires_grad_()
    sa, sb = cocktail_scores(a, tokens), cocktail_scores(b, tokens)
    assert sa.shape == (1, 2) and torch.equal(sa, sb)
    (ga,), (gb,) = torch.autograd.grad(sa.sum(), a), torch.autograd.grad(sb.sum(), b)
    assert torch.equal(ga[:, :T], gb) and not ga[:, T:].any()
    with pytest.raises(ValueError):
        cocktail_scores(x[:, :T - 1], tokens)
    with pytest.raises(ValueError):
        cocktail_scores(x.expand(2, -1, -1), tokens.expand(2, -1))


@pytest.mark.parametrize("C", [16, 17])
def test_cocktail_gradient_of_infinities(C):
    """0 times an infinity is not 0: in the tokens of a span whose gradient is zero, and from the padding of a row with
    fewer spans than the widest into its [MASK] row."""
    from kerneldev_b200 import cocktail_scores
    tokens = _span_tokens(2, 64)
    tokens[1, 32:50] = 50    # one span only
    x = torch.randn((2, 64, C), generator=torch.Generator(device=DEV).manual_seed(4), device=DEV)
    x[0, 2, 3] = float("inf")
    x.requires_grad_()
    ds = torch.tensor([[0.0, 0.0], [1.0, float("inf")]], device=DEV)
    (g,) = torch.autograd.grad(cocktail_scores(x, tokens), x, ds)
    nan = torch.zeros((2, 64, C), dtype=torch.bool)
    nan[0, 6:9, 3] = nan[0, 33:49, 3] = True
    nan[1, 2] = True
    assert torch.equal(g.isnan().cpu(), nan)
    assert torch.allclose(g[1, 7], x.detach()[1, 2] / 3, rtol=2.0**-22, atol=0) and not g[1, 33:50].any()


@pytest.mark.parametrize("through_ds", [False, True])
def test_second_derivatives_of_the_cocktail_scores(through_ds):
    """A gradient penalty on the embeddings, against the oracle in 64 bits; with the scores' gradient a constant or itself a
    function of the embeddings. Sums of at most T + C fp32 products in each of the four passes."""
    from kerneldev_b200 import cocktail_scores
    from oracle import attention_oracle as ao
    B, T, C = 2, 70, 20
    tokens = _span_tokens(B, T)
    tokens[1, 5:10] = 50    # the second row has one span
    x0 = torch.randn((B, T, C), generator=torch.Generator().manual_seed(6))
    w0 = torch.randn((B, 2), generator=torch.Generator().manual_seed(7))

    def penalty(scores, x, w):
        (g,) = torch.autograd.grad((scores.tanh() if through_ds else scores).mul(w).sum(), x, create_graph=True)
        return (g * g).sum() + (x * x).sum()

    x = x0.to(DEV).requires_grad_()
    (got,) = torch.autograd.grad(penalty(cocktail_scores(x, tokens), x, w0.to(DEV)), x)
    y = x0.double().requires_grad_()
    (want,) = torch.autograd.grad(penalty(ao.cocktail_scores(y, tokens.cpu())[0], y, w0.double()), y)
    assert (want - 2 * y).abs().max() > 0.1
    assert torch.allclose(got.double().cpu(), want, rtol=4 * (T + C) * 2.0**-24, atol=4 * (T + C) * 2.0**-24 * float(want.abs().max()))


def test_cached_plans_whose_metadata_is_gone_leave_the_cache():
    """A plan is kept as long as somebody could ask for it again: as long as the caller holds its metadata, or a tensor that the metadata is a
    view of, and not when a new batch has taken its place."""
    from kerneldev_b200 import clear_plan_cache
    from kerneldev_b200.plan import _CACHE, get_plan
    B, T = 2, 300
    dev = torch.device(DEV)

    def new(more=0):
        ids = torch.zeros((B, T + more), dtype=torch.int64, device=DEV)
        return ids > 0, ids

    def plan_of(ins, sid):
        return get_plan(B, T, dev, ins, sid, None, None, True, True)._core

    def plan_of_views(ins, sid):
        return plan_of(ins[:, :T], sid[:, :T].to(torch.int32))

    clear_plan_cache()
    held = [(ins, sid.to(torch.int32)) for ins, sid in (new(20) for _ in range(3))]   # (converted for the kernels)
    first = [plan_of_views(*h) for h in held]
    span = torch.ones((B, T), dtype=torch.bool, device=DEV)   # no view, and alone
    alone = get_plan(B, T, dev, span, None, None, None, True, True)._core
    plain = get_plan(B, T, dev, None, None, None, None, True, False)._core
    for _ in range(20):
        plan_of(*new())
    assert len(_CACHE) <= len(first) + 2 + 1
    assert all(plan_of_views(*h) is f for h, f in zip(held, first))
    assert get_plan(B, T, dev, span, None, None, None, True, True)._core is alone
    assert get_plan(B, T, dev, None, None, None, None, True, False)._core is plain
    clear_plan_cache()


@pytest.mark.parametrize("gone", ["metadata", "cache"])
@pytest.mark.parametrize("grad", [False, True])
def test_graphs_keep_the_plans_they_read(monkeypatch, grad, gone):
    """A captured launch has the address of its plan: the memory stays the plan's when its metadata is gone and newer plans come, or when the
    cache is cleared, and is given back when the graph goes."""
    monkeypatch.setenv("KD_CHECK_STATUS", "0")   # a check waits for the device
    import gc
    import time
    from kerneldev_b200 import clear_plan_cache, flash_attention
    from kerneldev_b200.plan import _CACHE
    B, H, T, D = 2, 3, 700, 64
    q, k, v, do = (torch.randn((B, H, T, D), device=DEV, dtype=torch.bfloat16) for _ in range(4))

    def plain_plan(length):
        flash_attention(q, k, v, lens=torch.tensor([length] * B, dtype=torch.int32, device=DEV))

    def call(lens):
        if not grad:
            with torch.no_grad():
                return (flash_attention(q, k, v, lens=lens),)
        o = flash_attention(*(x.detach().requires_grad_() for x in (q, k, v)), lens=lens, deterministic=True)
        return (o.detach(), *o.grad_fn(do))

    clear_plan_cache()
    lens = torch.tensor([T, 430], dtype=torch.int32, device=DEV)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        want = [x.clone() for x in call(lens)]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            outs = call(lens)
    torch.cuda.synchronize()
    (plan,) = _CACHE.values()
    first, nbytes = plan.ptr, plan.layout.total
    del plan
    if gone == "metadata":
        del lens
    else:
        clear_plan_cache()
    with torch.cuda.stream(side):   # whose allocations the plan's memory would go to
        for length in range(1, 9):
            plain_plan(length)
        blocks = [torch.full((nbytes,), 255, dtype=torch.uint8, device=DEV) for _ in range(16)]
    torch.cuda.synchronize()
    # (before the replay: on memory that is not the plan's any more it would read anything)
    for p in [p.ptr for p in _CACHE.values()] + [x.data_ptr() for x in blocks]:
        assert p + nbytes <= first or first + nbytes <= p
    for x in outs:
        x.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(outs, want))
    # the graph's end gives the plan back (its destructors run on a thread of the driver's)
    del blocks, outs, want
    clear_plan_cache()
    plain_plan(9)
    held = torch.cuda.memory_allocated()
    del graph
    gc.collect()
    deadline = time.time() + 10
    while torch.cuda.memory_allocated() > held - nbytes and time.time() < deadline:
        plain_plan(9)
        clear_plan_cache()
        time.sleep(0.05)
    assert torch.cuda.memory_allocated() <= held - nbytes
