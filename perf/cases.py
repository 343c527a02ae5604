"""The work that users of this framework have it do, as cases that can be timed and compared.

Every case goes through a public entry point with the inputs a user's program has in hand before the call: embeddings
in the model's dtype, masks or lengths as the collator built them, an index as it was loaded.  Shapes are those of
this repository's own benchmark and tests, or generic ones of the same use.

The families, and the range ``draw`` covers for each:

  train     in-batch contrastive step, forward + backward (``maxsim``): from a handful of pairs on a small GPU share to
            512 x 512; text passages to page-sized documents and page-sized queries; with and without fused normalisation
  kd        distillation / hard-negative step on candidate lists, forward + backward (4-D ``maxsim``)
  varlen    packed (padding-free) in-batch step, forward + backward (``maxsim_varlen``)
  fp32      exact fp32 scoring, as evaluation scripts and CPU-trained checkpoints use it
  rerank    one or a few queries against a candidate set, inference (``MaxSimScorer.score``, normalisation fused)
  fp8       the same on e4m3 embeddings with per-token scales (``maxsim_inference_fp8``)
  pairs     a ragged (query, document) pair list on packed batches, inference (``score_pairs_packed``)
  retrieve  top-k over a corpus that stays on the GPU (``retrieve``), one query to a large batch
  plaid     top-k over a compressed index (``retrieve_residual_varlen``)
  head      document head trained through the scores: hidden states projected inside the call, forward + backward
            (``maxsim_from_hidden``)
"""

import os

import torch
import torch.nn.functional as F

# what a training script sets once (the hint is for interactive use and reads the queries' norms back to the host)
os.environ.setdefault("LIK_SUPPRESS_NORM_WARN", "1")

import late_interaction_kernels_b200 as lik
from late_interaction_kernels_b200.fp8 import maxsim_inference_fp8, quantize_fp8_per_token
from late_interaction_kernels_b200.fused_head import maxsim_from_hidden
from late_interaction_kernels_b200.plaid import retrieve_residual_varlen
from late_interaction_kernels_b200.score_pairs import score_pairs_packed

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
ITEM = {"bf16": 2, "fp16": 2, "fp32": 4}


def listed():
    return [
        # a small training batch (one GPU's share of a fine-tuning run): the call's own latency and its launches count
        {"name": "train_16x16", "family": "train", "nq": 16, "nd": 16, "lq": 32, "ld": 180, "d": 128, "dtype": "bf16", "normalize": True},
        # the headline in-batch step: 512 pairs of 32-token queries and passages of 64 to 300 tokens
        {"name": "train_512x512", "family": "train", "nq": 512, "nd": 512, "lq": 32, "ld": 300, "d": 128, "dtype": "bf16", "normalize": False},
        # page-to-page training: queries as long as the pages (an odd token count), few pairs
        {"name": "train_pages_32x32", "family": "train", "nq": 32, "nd": 32, "lq": 1030, "ld": 1030, "d": 128, "dtype": "fp16", "normalize": False},
        # distillation: 64 queries, 32 scored candidates each
        {"name": "kd_64x32", "family": "kd", "nq": 64, "nd": 32, "lq": 32, "ld": 300, "d": 128, "dtype": "bf16", "normalize": False},
        # packed visual-document step: short ragged queries, pages of 900 to 1030 tokens
        {"name": "varlen_128x128", "family": "varlen", "nq": 128, "nd": 128, "lq": 32, "ld": 1030, "d": 128, "dtype": "bf16"},
        # fp32 scoring of a small batch with masks on both sides
        {"name": "fp32_32x32", "family": "fp32", "nq": 32, "nd": 32, "lq": 32, "ld": 180, "d": 128, "dtype": "fp32", "normalize": True},
        # serving: one query, its first-stage candidates, normalisation fused (the scorer's default)
        {"name": "rerank_1x1000", "family": "rerank", "nq": 1, "nd": 1000, "lq": 32, "ld": 300, "d": 128, "dtype": "fp16", "normalize": True},
        # serving from an e4m3 store with per-token scales
        {"name": "fp8_4x4096", "family": "fp8", "nq": 4, "nd": 4096, "lq": 32, "ld": 256, "d": 128, "dtype": "bf16"},
        # a ragged pair list from a cascade: odd counts, 96-wide embeddings
        {"name": "pairs_3001", "family": "pairs", "nq": 61, "nd": 1201, "n_pairs": 3001, "lq": 32, "ld": 300, "d": 96, "dtype": "bf16"},
        # first-stage search over a dense corpus, a batch of queries (the largest case)
        {"name": "retrieve_256x100k", "family": "retrieve", "nq": 256, "nd": 100000, "lq": 32, "ld": 300, "d": 128, "dtype": "bf16", "k": 100, "normalize": False},
        # an interactive query against a compressed index
        {"name": "plaid_1x25k", "family": "plaid", "nq": 1, "nd": 25000, "lq": 32, "ld": 300, "d": 128, "dtype": "fp16", "k": 10, "nbits": 2, "n_centroids": 65536},
        # training the projection head from cached hidden states
        {"name": "head_256x1024", "family": "head", "nq": 1, "nd": 256, "lq": 32, "ld": 1024, "d": 128, "dtype": "bf16", "d_model": 768},
    ]


def _spread(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm, odd ones among them."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    """One more case of the ranges above; never more work than the largest listed case."""
    while True:
        c = _draw(rng)
        if _scoring_flops(c) <= 4e12 and _doc_tokens(c) * c["d"] <= 1.5e9:
            return c


def _draw(rng):
    fam = rng.choice(["train", "train", "kd", "varlen", "fp32", "rerank", "fp8", "pairs", "retrieve", "plaid", "head"])
    half = rng.choice(["bf16", "fp16"])
    d = rng.choice([96, 128, 128])
    c = {"family": fam, "d": d, "dtype": half, "lq": rng.choice([24, 32, 32, 48]), "ld": _spread(rng, 64, 512)}
    if fam == "train":
        if rng.random() < 0.25:  # pages on both sides
            c.update(nq=_spread(rng, 4, 48), lq=_spread(rng, 128, 1030), ld=_spread(rng, 256, 2048))
        else:
            c.update(nq=_spread(rng, 8, 512), lq=_spread(rng, 16, 128), ld=_spread(rng, 64, 1030))
        c["nd"] = c["nq"]
        c["normalize"] = rng.random() < 0.5
    elif fam == "kd":
        c.update(nq=_spread(rng, 8, 128), nd=_spread(rng, 2, 32), ld=_spread(rng, 64, 1030), normalize=rng.random() < 0.5)
    elif fam == "varlen":
        c.update(nq=_spread(rng, 8, 256), ld=_spread(rng, 64, 1030))
        c["nd"] = c["nq"]
    elif fam == "fp32":
        c.update(nq=_spread(rng, 1, 64), nd=_spread(rng, 8, 256), dtype="fp32", normalize=rng.random() < 0.5)
    elif fam == "rerank":
        c.update(nq=_spread(rng, 1, 8), nd=_spread(rng, 50, 10000), lq=_spread(rng, 8, 128), ld=_spread(rng, 64, 1030), normalize=rng.random() < 0.7)
    elif fam == "fp8":
        c.update(nq=_spread(rng, 1, 16), nd=_spread(rng, 100, 16384))
    elif fam == "pairs":
        c.update(nq=_spread(rng, 4, 256), nd=_spread(rng, 64, 4096), n_pairs=_spread(rng, 100, 20000))
    elif fam == "retrieve":
        c.update(nq=_spread(rng, 1, 256), nd=_spread(rng, 2000, 100000), k=rng.choice([10, 20, 100]), ld=_spread(rng, 64, 300), normalize=rng.random() < 0.5)
    elif fam == "plaid":
        c.update(nq=_spread(rng, 1, 64), nd=_spread(rng, 1000, 50000), k=rng.choice([10, 100]), ld=_spread(rng, 64, 300), nbits=rng.choice([2, 4]), d=128,
                 n_centroids=rng.choice([8192, 65536]))
    else:
        c.update(nq=_spread(rng, 1, 8), nd=_spread(rng, 32, 512), ld=_spread(rng, 128, 2048), d=128, d_model=768)
    return c


# ---- lengths ------------------------------------------------------------------------------------------------------

def _doc_range(c):
    """Shortest and longest document of a case: passages vary a lot, packed pages are nearly all full."""
    hi = c["ld"]
    return (max(1, hi * 7 // 8), hi) if c["family"] == "varlen" or c["lq"] > 128 else (max(1, min(32, hi // 4) if hi <= 64 else hi // 5), hi)


def _query_range(c):
    """Queries are padded to a fixed length with tokens that count, except where the collator keeps them ragged."""
    return (max(1, c["lq"] // 2), c["lq"]) if c["family"] in ("varlen", "fp32", "pairs") else (c["lq"], c["lq"])


def _mean(r):
    return (r[0] + r[1]) / 2


def _n_docs(c):
    return c["nq"] * c["nd"] if c["family"] == "kd" else c["nd"]


def _doc_tokens(c):
    return _n_docs(c) * _mean(_doc_range(c))


def _n_scores(c):
    return c["n_pairs"] if c["family"] == "pairs" else c["nq"] * c["nd"]


def _scoring_flops(c):
    return 2.0 * c["d"] * _n_scores(c) * _mean(_query_range(c)) * _mean(_doc_range(c))


# ---- inputs -------------------------------------------------------------------------------------------------------

def _unit_rows(shape, dtype, gen):
    """L2-normalised Gaussian token embeddings, made a slice at a time so that no fp32 copy of a corpus exists."""
    x = torch.empty(shape, dtype=dtype, device="cuda")
    flat = x.view(-1, shape[-1])
    for lo in range(0, flat.shape[0], 1 << 22):
        part = flat[lo:lo + (1 << 22)]
        part.copy_(F.normalize(torch.randn(part.shape, generator=gen, device="cuda"), dim=-1))
    return x


def _raw_rows(shape, dtype, gen):
    """Token embeddings as a model's head gives them, before normalisation: norms differ from token to token."""
    x = torch.randn(shape, generator=gen, device="cuda")
    return (x * (0.5 + torch.rand(shape[:-1] + (1,), generator=gen, device="cuda"))).to(dtype)


def _lengths(n, r, gen):
    """n lengths spread evenly over the range, in random order: every seed has the same number of tokens."""
    even = torch.linspace(r[0], r[1], n, dtype=torch.float64, device="cuda").round().to(torch.int64)
    return even[torch.randperm(n, generator=gen, device="cuda")]


def _prefix_mask(lens, width):
    return torch.arange(width, device="cuda") < lens[..., None]


def _offsets(lens):
    return F.pad(lens.cumsum(0), (1, 0)).to(torch.int32)


def prepare(case, seed):
    c, fam = case, case["family"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dt = DTYPES[c["dtype"]]
    s = {"case": c}
    nq, lq, ld, d, nd = c["nq"], c["lq"], c["ld"], c["d"], _n_docs(c)
    rows = _raw_rows if c.get("normalize") and fam != "retrieve" else _unit_rows
    if fam in ("train", "kd", "fp32", "rerank", "retrieve"):
        dl = _lengths(nd, _doc_range(c), gen)
        s["Q"] = rows((nq, lq, d), dt, gen)
        s["D"] = rows((nd, ld, d), dt, gen)
        s["dm"] = _prefix_mask(dl, ld)
        if fam == "kd":
            s["D"], s["dm"] = s["D"].view(nq, c["nd"], ld, d), s["dm"].view(nq, c["nd"], ld)
        if fam == "fp32":
            s["qm"] = _prefix_mask(_lengths(nq, _query_range(c), gen), lq)
        if fam in ("train", "kd"):  # what the loss hands back: of the size of softmax gradients
            s["g"] = torch.randn((nq, c["nd"]), generator=gen, device="cuda") / c["nd"]
            s["Q"].requires_grad_()
            s["D"].requires_grad_()
        if fam == "rerank":
            s["scorer"] = lik.MaxSimScorer(normalize=c["normalize"])
    elif fam in ("varlen", "pairs"):
        ql, dl = _lengths(nq, _query_range(c), gen), _lengths(nd, _doc_range(c), gen)
        s["Q"], s["D"] = _unit_rows((int(ql.sum()), d), dt, gen), _unit_rows((int(dl.sum()), d), dt, gen)
        s["cu_q"], s["cu_d"] = _offsets(ql), _offsets(dl)
        s["max_q"], s["max_d"] = int(ql.max()), int(dl.max())
        if fam == "varlen":
            s["g"] = torch.randn((nq, nd), generator=gen, device="cuda") / nd
            s["Q"].requires_grad_()
            s["D"].requires_grad_()
        else:  # a first stage's output: grouped by query, its candidates in any order
            s["pq"] = torch.randint(0, nq, (c["n_pairs"],), generator=gen, device="cuda").sort().values.to(torch.int32)
            s["pd"] = torch.randint(0, nd, (c["n_pairs"],), generator=gen, device="cuda").to(torch.int32)
    elif fam == "fp8":
        s["Q"], s["sq"] = quantize_fp8_per_token(_unit_rows((nq, lq, d), dt, gen))
        s["D"], s["sd"] = quantize_fp8_per_token(_unit_rows((nd, ld, d), dt, gen))
        s["dm"] = _prefix_mask(_lengths(nd, _doc_range(c), gen), ld)
    elif fam == "plaid":
        dl = _lengths(nd, _doc_range(c), gen)
        total = int(dl.sum())
        s["Q"] = _unit_rows((nq, lq, d), dt, gen)
        s["codes"] = torch.randint(0, c["n_centroids"], (total,), generator=gen, device="cuda", dtype=torch.int32)
        s["residuals"] = torch.randint(0, 256, (total, d * c["nbits"] // 8), generator=gen, device="cuda", dtype=torch.uint8)
        s["centroids"] = _unit_rows((c["n_centroids"], d), torch.float16, gen)
        s["weights"] = torch.linspace(-0.1, 0.1, 2 ** c["nbits"], device="cuda")
        s["cu_d"], s["lens_host"] = _offsets(dl), dl.cpu()
    else:
        s["Q"] = _unit_rows((nq, lq, d), dt, gen).requires_grad_()
        s["H"] = torch.randn((nd, ld, c["d_model"]), generator=gen, device="cuda").to(dt).requires_grad_()
        s["W"] = (torch.randn((d, c["d_model"]), generator=gen, device="cuda") / c["d_model"] ** 0.5).to(dt).requires_grad_()
        s["b"] = (0.1 * torch.randn((d,), generator=gen, device="cuda")).to(dt)
        s["dm"] = _prefix_mask(_lengths(nd, _doc_range(c), gen), ld)
        s["g"] = torch.randn((nq, nd), generator=gen, device="cuda") / nd
    return s


# ---- one pass -----------------------------------------------------------------------------------------------------

def run(s):
    c = s["case"]
    fam = c["family"]
    if fam in ("train", "kd"):
        scores = lik.maxsim(s["Q"], s["D"], d_mask=s["dm"], normalize=c["normalize"])
        gq, gd = torch.autograd.grad(scores, (s["Q"], s["D"]), s["g"])
        return {"scores": scores.detach(), "grad_q": gq, "grad_d": gd}
    if fam == "varlen":
        scores = lik.maxsim_varlen(s["Q"], s["D"], s["cu_q"], s["cu_d"], s["max_q"], s["max_d"])
        gq, gd = torch.autograd.grad(scores, (s["Q"], s["D"]), s["g"])
        return {"scores": scores.detach(), "grad_q": gq, "grad_d": gd}
    if fam == "head":
        scores = maxsim_from_hidden(s["Q"], s["H"], s["W"], s["b"], s["dm"])
        gq, gh, gw = torch.autograd.grad(scores, (s["Q"], s["H"], s["W"]), s["g"])
        return {"scores": scores.detach(), "grad_q": gq, "grad_h": gh, "grad_w": gw}
    with torch.no_grad():
        if fam == "fp32":
            return lik.maxsim(s["Q"], s["D"], s["qm"], s["dm"], normalize=c["normalize"])
        if fam == "rerank":
            return s["scorer"].score(s["Q"], s["D"], d_mask=s["dm"])
        if fam == "fp8":
            return maxsim_inference_fp8(s["Q"], s["D"], scale_Q=s["sq"], scale_D=s["sd"], d_mask=s["dm"])
        if fam == "pairs":
            return score_pairs_packed(s["Q"], s["D"], s["cu_q"], s["cu_d"], s["pq"], s["pd"], max_seqlen_q=s["max_q"], max_seqlen_d=s["max_d"])
        if fam == "retrieve":
            return lik.retrieve(s["Q"], s["D"], c["k"], d_mask=s["dm"], normalize=c["normalize"])
        return retrieve_residual_varlen(s["Q"], s["codes"], s["residuals"], s["cu_d"], s["centroids"], s["weights"], c["nbits"], c["k"],
                                        doc_lengths_host=s["lens_host"])


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def work(case):
    """Valid tokens only (padding is neither read nor multiplied): inputs read once, outputs written once; a backward
    adds its gradients, one multiply-add per feature for either side of every (score, query token)."""
    c, fam = case, case["family"]
    nq, d = c["nq"], c["d"]
    q_tok, d_tok = nq * _mean(_query_range(c)), _doc_tokens(c)
    item = 1 if fam == "fp8" else ITEM[c["dtype"]]
    flops = _scoring_flops(c)
    if fam == "pairs":  # documents that no pair names are not read
        d_tok *= 1.0 - (1.0 - 1.0 / c["nd"]) ** c["n_pairs"]
    bytes_ = (q_tok + d_tok) * d * item
    if fam in ("retrieve", "plaid"):
        bytes_ += nq * c["k"] * 12
    else:
        bytes_ += _n_scores(c) * 4
    if fam == "fp8":
        bytes_ += (q_tok + d_tok) * 4
    if fam == "plaid":
        bytes_ = q_tok * d * item + d_tok * (4 + d * c["nbits"] // 8) + nq * c["k"] * 12
        bytes_ += c["n_centroids"] * d * 2
    winners = _n_scores(c) * _mean(_query_range(c))
    if fam in ("train", "kd", "varlen"):
        # gradients have the inputs' shapes, padding included
        rows = (nq * c["lq"] + _n_docs(c) * c["ld"]) if fam != "varlen" else q_tok + d_tok
        bytes_ += rows * d * item + _n_scores(c) * 4
        flops += 4.0 * d * winners
    if fam == "head":
        dm = c["d_model"]
        bytes_ = (q_tok * d + d_tok * dm + d * dm) * item + _n_scores(c) * 8 + (q_tok * d + c["nd"] * c["ld"] * dm + d * dm) * item
        flops += 2.0 * d_tok * dm * d + 4.0 * d * winners + 4.0 * dm * d * min(winners, d_tok)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """Scores are fp32 sums of exact 8- or 16-bit products; gradients are rounded to the inputs' type, and a pair of
    document tokens whose products tie within fp32 rounding may swap."""
    fam, dt = case["family"], case["dtype"]
    if fam == "head":  # projected tokens are rounded to the operand type before they are scored
        return {"rel": 1e-2}
    if fam in ("train", "kd", "varlen"):
        return {"rel": 1e-2 if dt == "bf16" else 2e-3}
    if fam == "plaid":  # decoded tokens are rounded to the operand type before they are scored
        return {"rel": 1e-3 if dt == "fp16" else 5e-3, "differ": 0.01}
    if fam == "retrieve":
        return {"rel": 1e-5, "differ": 1e-3}
    return {"rel": 1e-5}
