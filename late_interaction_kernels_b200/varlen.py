"""MaxSim on packed (padding-free) inputs: ``maxsim_varlen`` (reference: varlen.py:271-493).

``Q_packed`` / ``D_packed`` are ``[sum L, d]`` token matrices with int32 cumulative offsets.
The kernels take their loop bounds from ``cu_seqlens`` themselves, so ``max_seqlen_*`` only
sizes per-query buffers: a value that is too small for the queries is reported through the
device status word (``check_device_status()``) instead of a device-side assert, and a too-small
``max_seqlen_d`` cannot truncate documents.
"""

from __future__ import annotations

from . import _lib, _ops
from ._utils import common_dtype


def _check_packed(Q_packed, D_packed):
    if Q_packed.dim() != 2:
        raise ValueError(
            f"Q_packed must be 2-D [sum(Lq_i), d]; got shape {tuple(Q_packed.shape)} (ndim={Q_packed.dim()}). "
            "For padded inputs use `maxsim(Q, D, ...)` instead."
        )
    if D_packed.dim() != 2:
        raise ValueError(
            f"D_packed must be 2-D [sum(Ld_j), d]; got shape {tuple(D_packed.shape)} (ndim={D_packed.dim()}). "
            "For padded inputs use `maxsim(Q, D, ...)` instead."
        )
    if D_packed.shape[1] != Q_packed.shape[1]:
        raise ValueError(
            "Q_packed and D_packed must share the embedding dim; got "
            f"Q_packed.shape[1]={Q_packed.shape[1]} vs D_packed.shape[1]={D_packed.shape[1]}."
        )


def _longest(cu):
    return int((cu[1:] - cu[:-1]).max()) if cu.numel() > 1 else 0


def _varlen_forward(Q_packed, D_packed, cu_seqlens_q, cu_seqlens_d, max_seqlen_q, max_seqlen_d, save_argmax):
    """Scores and winners outside autograd: ``(scores [Nq, Nd], argmax [Nq, Nd, max_q] | None, max_q, max_d)``
    (varlen.py:271-364).  A longest length that is not given is read from the offsets, the documents' only for winners."""
    _check_packed(Q_packed, D_packed)
    _lib.require_cuda(Q_packed, D_packed, cu_seqlens_q, cu_seqlens_d, op="maxsim_varlen")
    dt = common_dtype(Q_packed, D_packed)
    if max_seqlen_q is None:
        max_seqlen_q = _longest(cu_seqlens_q)
    if max_seqlen_d is None:
        max_seqlen_d = _longest(cu_seqlens_d) if save_argmax else 0
    q = _ops.packed_spec(Q_packed.to(dt), cu_seqlens_q, max_seqlen_q)
    d = _ops.packed_spec(D_packed.to(dt), cu_seqlens_d, max_seqlen_d)
    scores, argmax = _ops.forward(q, d, pairing=_lib.PAIR_CROSS, save_argmax=save_argmax, argmax_stride=q.max_len)
    if argmax is not None:
        argmax = argmax.view(q.n_seq, d.n_seq, q.max_len)
    return scores.view(q.n_seq, d.n_seq), argmax, q.max_len, d.max_len


def maxsim_varlen(Q_packed, D_packed, cu_seqlens_q, cu_seqlens_d, max_seqlen_q=None, max_seqlen_d=None):
    """MaxSim on packed inputs -> fp32 ``[Nq, Nd]``; autograd-aware (varlen.py:452-493).

    Empty sequences score 0.  ``max_seqlen_q`` sizes the query tiles and the saved argmax, ``max_seqlen_d``
    the backward grid; when omitted they are read from ``cu_seqlens`` with one device->host sync (pass them
    to stay sync-free, e.g. under CUDA-graph capture)."""
    _check_packed(Q_packed, D_packed)
    _lib.require_cuda(Q_packed, D_packed, cu_seqlens_q, cu_seqlens_d, op="maxsim_varlen")
    return _ops.native_call(_lib.host().maxsim_packed, Q_packed, D_packed, cu_seqlens_q, cu_seqlens_d, None, None,
                            None if max_seqlen_q is None else int(max_seqlen_q), None if max_seqlen_d is None else int(max_seqlen_d))
