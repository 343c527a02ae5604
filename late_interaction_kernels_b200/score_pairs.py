"""Arbitrary ``(query, document)`` pair lists on packed batches: ``score_pairs_packed``
(reference: score_pairs.py:281-511).

The forward runs on the tensor-core kernel (one pair per work unit; consecutive pairs of the same query share the
resident query tile).  The backward groups the pairs by query and by document with two stable device sorts and then
uses the same destination-owned kernels as the other layouts, so the gradients are bitwise reproducible (the
reference scatters both with fp32 atomics, score_pairs.py:148-273)."""

from __future__ import annotations

from . import _lib, _ops


def score_pairs_packed(Q_packed, D_packed, cu_seqlens_q, cu_seqlens_d, pair_q_idx, pair_d_idx, *,
                       max_seqlen_q=None, max_seqlen_d=None):
    """``scores[k] = MaxSim(query pair_q_idx[k], document pair_d_idx[k])`` on packed batches -> fp32
    ``[num_pairs]``; autograd-aware (score_pairs.py:423-508).  A pair index outside the batch scores 0
    and sets the device status word instead of faulting."""
    if Q_packed.dim() != 2 or D_packed.dim() != 2:
        raise ValueError(
            f"Q_packed / D_packed must be 2-D [sum(L), d]; got Q={tuple(Q_packed.shape)}, D={tuple(D_packed.shape)}."
        )
    if D_packed.shape[1] != Q_packed.shape[1]:
        raise ValueError(f"Q / D embedding dims mismatch: {Q_packed.shape[1]} vs {D_packed.shape[1]}.")
    if pair_q_idx.shape != pair_d_idx.shape or pair_q_idx.dim() != 1:
        raise ValueError(
            f"pair_q_idx / pair_d_idx must be matching 1-D tensors; got {tuple(pair_q_idx.shape)} vs {tuple(pair_d_idx.shape)}."
        )
    _lib.require_cuda(Q_packed, D_packed, cu_seqlens_q, cu_seqlens_d, pair_q_idx, pair_d_idx, op="score_pairs_packed")
    return _ops.native_call(_lib.host().maxsim_packed, Q_packed, D_packed, cu_seqlens_q, cu_seqlens_d, pair_q_idx, pair_d_idx,
                            None if max_seqlen_q is None else int(max_seqlen_q), None if max_seqlen_d is None else int(max_seqlen_d))


__all__ = ["score_pairs_packed"]
