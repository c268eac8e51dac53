"""Workloads of the attention framework for performance measurement.

A case is a dict of plain values; ``kind`` selects the program a user would run:

  attn      one flash_attention call, forward only or forward + backward
  step      token ids -> metadata_from_tokens -> a stack of attention layers that share the metadata
            (model.GPTModel derives the metadata once per batch and passes it to every layer); the
            metadata is new on every pass, as it is for every batch of a training run or token of a
            generation
  cocktail  the span-mean scoring head on the last layer's embeddings, forward + backward

Attention cases name the mask: ``hier`` (prefix, causal context, spans, one [MASKQ], padding cut off by
``lens``), ``causal`` or ``full``. The section lengths of a hierarchical mask scale with the sequence
length T as in the benchmark configurations. ``layout`` is ``bhtd`` (contiguous heads) or ``bthd`` (the
model's (batch, time, heads, dim) memory seen through a transpose, outputs in the same memory order).
"""
import numpy as np
import torch

from kerneldev_b200 import cocktail_scores, flash_attention, generate_hadamard_signs, metadata_from_tokens
from kerneldev_b200.metadata import SPECIAL_TOKENS
from kerneldev_b200.synthetic import batch_metadata

_DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32}


def _attn(name, B, H, T, D, dtype, mask, grad, layout="bhtd", hadamard=False, deterministic=False):
    return {"name": name, "kind": "attn", "B": B, "H": H, "T": T, "D": D, "dtype": dtype, "mask": mask, "grad": grad,
            "layout": layout, "hadamard": hadamard, "deterministic": deterministic}


def listed():
    return [
        # one token of a generation: the whole (short) sequence of one request goes through the model's layers again
        # for every new token, with metadata derived from the token ids; latency and launches are what it costs
        {"name": "generate_t173", "kind": "step", "B": 1, "H": 16, "T": 173, "D": 64, "dtype": "bfloat16", "layers": 8, "grad": False},
        # the smallest training call: the correctness configuration (B=2, H=4, L=256), float32 tensors
        _attn("train_small_fp32", 2, 4, 256, 64, "float32", "hier", True),
        # teacher-forcing training at an ordinary length that is no multiple of a tile
        _attn("train_causal_t1000", 8, 16, 1000, 64, "bfloat16", "causal", True, layout="bthd"),
        # odd head dim, odd length, few heads, fp16: a model whose sizes nobody tuned for
        _attn("train_ragged_d80", 3, 6, 1357, 80, "float16", "hier", True, layout="bthd"),
        # a micro-batch of the end-to-end training configuration (L=2048, micro-batch 8, 16 heads of 64): half
        # teacher-forcing rows, half cocktail-party rows, metadata from token ids, four layers on one plan
        {"name": "train_step_t2048", "kind": "step", "B": 8, "H": 16, "T": 2048, "D": 64, "dtype": "bfloat16", "layers": 4, "grad": True},
        # reproducible training runs ask for the deterministic backward
        _attn("train_determ_t2048", 4, 16, 2048, 64, "bfloat16", "hier", True, layout="bthd", deterministic=True),
        # teacher-forcing causal configuration at head dim 128
        _attn("train_causal_d128", 8, 16, 2048, 128, "bfloat16", "causal", True),
        # validation: forward only, hierarchical mask, O and LSE
        _attn("eval_hier_t4096", 8, 16, 4096, 64, "bfloat16", "hier", False, layout="bthd"),
        # the headline configuration: hierarchical mask, forward + backward
        _attn("train_hier_t4096", 16, 16, 4096, 64, "bfloat16", "hier", True),
        # prefill of the longest sequence the operator takes
        _attn("prefill_t16384_d128", 1, 16, 16384, 128, "bfloat16", "causal", False, layout="bthd"),
        # incoherent processing: Hadamard transform of Q and K, fp16, inputs with outliers (the largest case)
        _attn("train_hadamard_t8192", 4, 32, 8192, 128, "float16", "hier", True, hadamard=True),
        # the span-mean scoring head of the model on a full batch
        {"name": "cocktail_head_t4096", "kind": "cocktail", "B": 16, "T": 4096, "C": 1024, "dtype": "bfloat16"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    largest = next(c for c in listed() if c["name"] == "train_hadamard_t8192")
    top = work(largest)
    while True:
        kind = rng.choices(("attn", "step", "cocktail"), (8, 3, 1))[0]
        if kind == "cocktail":
            c = {"kind": kind, "B": rng.randint(1, 16), "T": _log_uniform(rng, 64, 4096), "C": 8 * _log_uniform(rng, 8, 256),
                 "dtype": rng.choice(("bfloat16", "float16", "float32"))}
        else:
            T = _log_uniform(rng, 24, 16384)
            D = rng.choice((64, 64, 64, 128, 128, 16, 32, 48, 80, 96, 112))
            # from a call that is nothing but launches to one that fills the device
            H = rng.choice((2, 4, 6, 8, 12, 16, 16, 24, 32))
            B = max(1, _log_uniform(rng, 1, 32) if T < 4096 else rng.randint(1, 8))
            dtype = rng.choice(("bfloat16", "bfloat16", "float16", "float32"))
            if kind == "step":
                c = {"kind": kind, "B": B, "H": H, "T": T, "D": D, "dtype": rng.choice(("bfloat16", "float16")),
                     "layers": rng.randint(2, 8), "grad": rng.random() < 0.6}
            else:
                mask = rng.choice(("hier", "hier", "hier", "causal", "causal", "full"))
                c = _attn("", B, H, T, D, dtype, mask, rng.random() < 0.7, layout=rng.choice(("bhtd", "bthd")),
                          hadamard=D in (16, 32, 64, 128) and dtype != "float32" and rng.random() < 0.15,
                          deterministic=rng.random() < 0.15)
                del c["name"]
        w = work(c)
        if w["flops"] <= 0.8 * top["flops"] and w["bytes"] <= 0.8 * top["bytes"]:
            return c


# ---- metadata ---------------------------------------------------------------------------------------------------

def _ranges(T):
    """Section-length ranges (inclusive) for sequences of T tokens: those of the 4096-token configuration at T = 4096,
    twice the context and the spans at 8192, half of everything at 2048, and in proportion below."""
    at_least = lambda x: max(1, int(x))
    return {"prefix": (at_least(min(32, T // 128)), at_least(min(256, T // 16))),
            "context": (at_least(T // 4), at_least(T // 2)),
            "n_spans": (at_least(T // 1024), max(2, T // 128)),
            "span_len": (max(2, min(16, T // 256)), max(3, min(128, T // 32)))}


def _sections(case, seed):
    r = _ranges(case["T"])
    if case["kind"] == "cocktail":   # a fixed number of spans to a row: the width of the scores
        r["n_spans"] = (max(1, case["T"] // 256),) * 2
    return batch_metadata(seed, case["B"], case["T"], **r)


def _token_rows(case, seed, mark_context):
    """Token ids with the collate's layout; the second half of a batch of several rows of a step is teacher-forcing
    text ([CLS] and bytes). ``mark_context``: one [MASK] at the end of each context (the cocktail head's query)."""
    B, T = case["B"], case["T"]
    st = SPECIAL_TOKENS
    rng = np.random.default_rng(seed)
    x = rng.integers(6, 262, size=(B, T))
    in_span, span_id, is_prefix, lens = _sections(case, seed)
    for b in range(B):
        if not mark_context and B > 1 and b >= B // 2:
            x[b, 0] = st["[CLS]"]
            continue
        x[b, int(is_prefix[b].sum()) - 1] = st["[CLS]"]
        ids = span_id[b] * in_span[b]
        edge = np.diff(ids, prepend=0)
        starts = np.flatnonzero((edge != 0) & (ids > 0))
        ends = np.flatnonzero((np.diff(ids, append=0) != 0) & (ids > 0))
        x[b, starts] = st["[SPAN]"]
        x[b, ends] = st["[ES]"]
        x[b, lens[b] - 1] = st["[MASKQ]"]
        x[b, lens[b]:] = st["[PAD]"]
        if mark_context:
            first = starts[0] if len(starts) else lens[b] - 1
            x[b, max(first - 1, 0)] = st["[MASK]"]
    return torch.as_tensor(x, dtype=torch.int64, device="cuda")


def _tensors(case, seed, count):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, H, T, D = case["B"], case["H"], case["T"], case["D"]
    bthd = case.get("layout", "bthd") == "bthd"
    out = []
    for i in range(count):
        shape = (B, T, H, D) if bthd else (B, H, T, D)
        x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)
        if case.get("hadamard") and i % 4 < 3:   # 0.1 % outliers in Q, K and V
            hit = torch.rand(shape, generator=g, device="cuda") < 1e-3
            x = torch.where(hit, torch.randn(shape, generator=g, device="cuda") * 20.0, x)
            del hit
        x = x.to(_DTYPES[case["dtype"]])
        out.append(x.transpose(1, 2) if bthd else x)
    return out


def prepare(case, seed):
    if case["kind"] == "cocktail":
        g = torch.Generator(device="cuda").manual_seed(seed)
        dt = _DTYPES[case["dtype"]]
        tokens = _token_rows(case, seed, mark_context=True)
        x = torch.randn((case["B"], case["T"], case["C"]), generator=g, device="cuda").to(dt).requires_grad_()
        n_spans = int((tokens == SPECIAL_TOKENS["[SPAN]"]).sum(1).max())
        # gradient of the scores, as the loss hands it back
        ds = torch.randn((case["B"], n_spans), generator=g, device="cuda").to(dt)
        return {"case": case, "tokens": tokens, "x": x, "ds": ds}
    if case["kind"] == "step":
        per = 4 if case["grad"] else 3
        flat = _tensors(case, seed, per * case["layers"])
        layers = []
        for n in range(case["layers"]):
            q, k, v = flat[per * n:per * n + 3]
            if case["grad"]:
                for t in (q, k, v):
                    t.requires_grad_()
            layers.append((q, k, v, flat[per * n + 3] if case["grad"] else None))
        return {"case": case, "tokens": _token_rows(case, seed, mark_context=False), "layers": layers}
    q, k, v, do = _tensors(case, seed, 4)
    if case["grad"]:
        for t in (q, k, v):
            t.requires_grad_()
    options = {"causal": case["mask"] != "full", "deterministic": case["deterministic"],
               "out_layout": "input" if case["layout"] == "bthd" else "contiguous"}
    if case["mask"] == "hier":
        in_span, span_id, is_prefix, lens = (torch.as_tensor(a, device="cuda") for a in _sections(case, seed))
        options.update(in_span=in_span, span_id=span_id, is_prefix=is_prefix, lens=lens)
    if case["hadamard"]:
        options["hadamard_signs"] = generate_hadamard_signs(case["H"], case["D"], seed=seed % 1000)
    return {"case": case, "q": q, "k": k, "v": v, "do": do, "options": options}


def run(state):
    case = state["case"]
    if case["kind"] == "cocktail":
        scores = cocktail_scores(state["x"], state["tokens"])
        (gx,) = torch.autograd.grad(scores, state["x"], state["ds"])
        return scores.detach(), gx
    if case["kind"] == "step":
        in_span, span_id, is_prefix = metadata_from_tokens(state["tokens"])
        meta = {"in_span": in_span, "span_id": span_id, "is_prefix": is_prefix, "causal": True, "out_layout": "input"}
        if not case["grad"]:
            with torch.no_grad():
                return [flash_attention(q, k, v, **meta) for q, k, v, _ in state["layers"]]
        outs = [flash_attention(q, k, v, **meta) for q, k, v, _ in state["layers"]]
        result = []
        for (q, k, v, do), o in zip(reversed(state["layers"]), reversed(outs)):
            result.append((o.detach(), *torch.autograd.grad(o, (q, k, v), do)))
        return result
    q, k, v = state["q"], state["k"], state["v"]
    if not case["grad"]:
        with torch.no_grad():
            return flash_attention(q, k, v, return_lse=True, **state["options"])
    o = flash_attention(q, k, v, **state["options"])
    return (o.detach(), *torch.autograd.grad(o, (q, k, v), state["do"]))


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def _allowed_pairs(in_span, span_id, is_prefix, lens):
    """(query, key) pairs of one sequence that the rule allows (the sections do not overlap)."""
    p = int(is_prefix[:lens].sum())
    n_ins = int(in_span[:lens].sum())
    c = int(lens) - p - n_ins - int((span_id[:lens] == -1).sum())
    spans = np.bincount(span_id[:lens][in_span[:lens]]).astype(np.int64)
    return p * p + c * (c + 1) // 2 + c * p + n_ins * c + int((spans * spans).sum()) + (p + n_ins) * int((span_id[:lens] == -1).sum())


def _pairs(case):
    """Allowed pairs of the whole batch for one head (hierarchical masks: of the batch drawn from seed 0)."""
    B, T = case["B"], case["T"]
    if case["kind"] == "attn" and case["mask"] != "hier":
        return B * (T * T if case["mask"] == "full" else T * (T + 1) // 2)
    in_span, span_id, is_prefix, lens = _sections(case, 0)
    if case["kind"] == "attn":
        return sum(_allowed_pairs(in_span[b], span_id[b], is_prefix[b], lens[b]) for b in range(B))
    plain = B - B // 2 if B > 1 else 0   # teacher-forcing rows; without lens, padding counts as context
    return (sum(_allowed_pairs(in_span[b], span_id[b], is_prefix[b], T) for b in range(B - plain)) + plain * (T * (T + 1) // 2))


def work(case):
    es = 4 if case["dtype"] == "float32" else 2
    if case["kind"] == "cocktail":
        B, T, C = case["B"], case["T"], case["C"]
        in_span = _sections(case, 0)[0]
        live = int(in_span.sum())   # embeddings the scores depend on; the gradient is written for every token
        return {"bytes": B * T * 8 + (live + B * T) * C * es, "flops": 2 * live * C * 2}
    n = case["B"] * case["H"] * case["T"] * case["D"] * es
    layers = case.get("layers", 1)
    tokens = case["B"] * case["T"] * 8 if case["kind"] == "step" else (case["B"] * case["T"] * 10 if case["mask"] == "hier" else 0)
    lse = 0 if case["kind"] == "step" or case["grad"] else case["B"] * case["H"] * case["T"] * 4
    # forward: Q, K, V in, O out; with the backward also dO in and dQ, dK, dV out
    return {"bytes": layers * n * (8 if case["grad"] else 4) + tokens + lse,
            "flops": layers * (14 if case["grad"] else 4) * case["D"] * case["H"] * _pairs(case)}


def tolerance(case):
    # P, dS, O and the gradients are rounded to the operands' 16-bit type: 2^-9 (bf16) or 2^-12 (fp16) relative for each
    # rounding. float32 tensors take part as fp16 operands (tf32's mantissa). Outliers of 20 sigma make single products
    # large against the sums they enter.
    if case["kind"] == "cocktail" and case["dtype"] == "float32":
        return {"rel": 1e-5}
    if case["dtype"] == "bfloat16":
        return {"rel": 1e-2}
    return {"rel": 4e-3 if case.get("hadamard") else 2e-3}
