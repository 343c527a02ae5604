"""User-facing differentiable MaxSim: ``maxsim`` and ``maxsim_pairs``.

Same signatures, shape dispatch, error messages and warn-once behaviour as the
reference's ``autograd.py`` (autograd.py:356-501).  What is gone is everything
that only served the Triton autotuner: no power-of-two padding of ``Lq``
(autograd.py:49-98) and no 128-token chunking of long queries
(autograd.py:322-353) — the kernels take any ``Lq`` directly.  The call itself (argument
checks, launches, the autograd node whose backward runs without the interpreter lock)
is native: ``csrc/host/lik_host.cpp``.
"""

from __future__ import annotations

import os
import warnings

import torch

from . import _lib, _ops

_VALID_METHODS = ("auto", "unified", "lowmem")

# The un-normalised-input heuristic needs a device->host sync, so it runs on the first call only
# (same policy as autograd.py:129-166).
_NORM_CHECKED = False


def _maybe_warn_unnormalized(Q: torch.Tensor) -> None:
    """Warn once when ``normalize=False`` meets queries whose median token norm is far from 1.
    Silence with ``LIK_SUPPRESS_NORM_WARN=1``."""
    global _NORM_CHECKED
    if _NORM_CHECKED or os.environ.get("LIK_SUPPRESS_NORM_WARN", "0") == "1":
        return
    _NORM_CHECKED = True
    if torch.cuda.is_current_stream_capturing():
        return
    with torch.no_grad():
        sample = Q.detach().reshape(-1, Q.shape[-1])[:64]
        if sample.numel() == 0:
            return
        med = sample.float().norm(dim=-1).median().item()
    if not (0.9 <= med <= 1.1):
        warnings.warn(
            f"late-interaction-kernels: `maxsim(..., normalize=False)` but Q's median L2 norm is {med:.3f} "
            "(ColBERT-style models expect ≈1.0). Pass `normalize=True` to fuse the L2-norm into the kernel, "
            "or pre-normalize with `F.normalize(Q, dim=-1)`. Silence with `LIK_SUPPRESS_NORM_WARN=1`.",
            UserWarning,
            stacklevel=3,
        )


def _explain(Q, D, q_mask, d_mask) -> None:
    """Raise the error that belongs to arguments the native call refused."""
    if D.dim() == 4:
        if Q.dim() != 3:
            raise ValueError(f"KD layout (D.dim()==4) needs Q to be [Nq, Lq, d]; got Q.shape={tuple(Q.shape)}")
        Nq, Lq, d_q = Q.shape
        Nq_d, K, Ld, d_d = D.shape
        if Nq != Nq_d:
            raise ValueError(f"KD layout needs D.shape[0] == Q.shape[0]; got Q.shape[0]={Nq} vs D.shape[0]={Nq_d}.")
        if d_q != d_d:
            raise ValueError(f"Q and D must share the embedding dim; got {d_q} vs {d_d}.")
        if q_mask is not None and q_mask.shape != (Nq, Lq):
            raise ValueError(f"q_mask must be [Nq={Nq}, Lq={Lq}] for KD layout; got {tuple(q_mask.shape)}.")
        if d_mask is not None and d_mask.shape != (Nq, K, Ld):
            raise ValueError(f"d_mask must be [Nq={Nq}, K={K}, Ld={Ld}] for KD layout; got {tuple(d_mask.shape)}.")
    else:
        if Q.dim() not in (2, 3) or D.dim() not in (2, 3):
            raise ValueError(f"maxsim needs Q [Nq, Lq, d] and D [Nd, Ld, d]; got {tuple(Q.shape)} and {tuple(D.shape)}.")
        if Q.shape[-1] != D.shape[-1]:
            raise ValueError(
                f"Q and D must share the embedding dim; got Q.shape[-1]={Q.shape[-1]} vs D.shape[-1]={D.shape[-1]}."
            )
    if Q.device != D.device:
        raise ValueError(f"Q and D must be on the same device; got Q.device={Q.device} vs D.device={D.device}.")
    if q_mask is not None and q_mask.device != Q.device:
        raise ValueError(f"q_mask must be on the same device as Q; got {q_mask.device} vs {Q.device}.")
    if d_mask is not None and d_mask.device != D.device:
        raise ValueError(f"d_mask must be on the same device as D; got {d_mask.device} vs {D.device}.")
    _lib.require_cuda(Q, D, op="maxsim")
    raise RuntimeError("maxsim: the arguments were refused without a reason")  # the checks above mirror the native ones


def maxsim(Q, D, q_mask=None, d_mask=None, *, normalize=False, backward=None):
    """Differentiable fused MaxSim; drop-in for PyLate's ``colbert_scores`` (autograd.py:356-459).

    Args:
        Q: ``[Nq, Lq, d]`` or ``[Lq, d]``.
        D: ``[Ld, d]`` (one document), ``[Nd, Ld, d]`` (cross product -> ``[Nq, Nd]``) or
            ``[Nq, K, Ld, d]`` (per-query candidate lists -> ``[Nq, K]``).
        q_mask, d_mask: bool tensors shaped like the token axes (``True`` = valid token); any pattern.
        normalize: L2-normalise every token inside the kernel.
        backward: ``None``/"auto", "unified" (fp32 atomics) or "lowmem" (deterministic, dtype-direct).

    Returns fp32 scores; 2-D inputs squeeze the matching axis.  Inputs may be fp16 / bf16 / fp32;
    gradients flow into Q and D in their own dtypes.
    """
    if backward is not None and backward not in _VALID_METHODS:
        raise ValueError(f"backward= must be one of {_VALID_METHODS} or None, got {backward!r}")
    # "unified" keeps the fp32-atomic scatter; "lowmem" and "auto" use the destination-owned reduction, which on this
    # hardware is both the deterministic and the faster one
    scores = _ops.native_call(_lib.host().maxsim, Q, D, q_mask, d_mask, normalize, backward != "unified")
    if scores is None:
        _explain(Q, D, q_mask, d_mask)
    if not normalize and not _NORM_CHECKED and D.dim() != 4:
        _maybe_warn_unnormalized(Q)
    return scores


def maxsim_pairs(Q, D, q_mask=None, d_mask=None, *, normalize=False, backward=None):
    """Same-index pairs ``(Q[i], D[i]) -> [B]``; drop-in for PyLate's ``colbert_scores_pairwise``
    (autograd.py:462-501).  This is the K = 1 case of the candidate-list layout."""
    if Q.dim() != 3 or D.dim() != 3:
        raise ValueError(
            f"maxsim_pairs needs both Q and D to be [B, L, d]; got Q.shape={tuple(Q.shape)}, D.shape={tuple(D.shape)}."
        )
    if Q.shape[0] != D.shape[0]:
        raise ValueError(f"maxsim_pairs needs Q.shape[0] == D.shape[0]; got {Q.shape[0]} vs {D.shape[0]}.")
    dm = d_mask.unsqueeze(1) if d_mask is not None else None
    return maxsim(Q, D.unsqueeze(1), q_mask=q_mask, d_mask=dm, normalize=normalize, backward=backward).squeeze(-1)
