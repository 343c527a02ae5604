"""The native host path under what a program puts around a call: activation checkpointing, saved-tensor hooks, arguments
on the host."""

import numpy as np
import pytest
import torch
from torch.utils.checkpoint import checkpoint

import cases

pytestmark = pytest.mark.gpu


def dev(x, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    return t.to(dtype) if dtype is not None else t


def scoring_calls():
    """name -> (function of its differentiable inputs, those inputs)"""
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200.fused_head import maxsim_from_hidden
    from late_interaction_kernels_b200.padded import maxsim_padded
    from late_interaction_kernels_b200.score_pairs import score_pairs_packed

    rng = np.random.default_rng(3)
    half = torch.bfloat16
    Q, D = dev(rng.standard_normal((4, 8, 64)), half), dev(rng.standard_normal((5, 24, 64)), half)
    dm = dev(cases.prefix_mask(np.array([24, 3, 17, 1, 9]), 24))
    cu_q, cu_d = dev(np.arange(0, 33, 8, dtype=np.int32)), dev(np.arange(0, 121, 24, dtype=np.int32))
    pq, pd = dev(np.array([0, 0, 3], np.int32)), dev(np.array([4, 1, 2], np.int32))
    W, b = dev(rng.standard_normal((64, 128)) / 12, half), dev(rng.standard_normal(64), half)
    H = dev(rng.standard_normal((5, 24, 128)), half)
    flat = lambda x: x.reshape(-1, x.shape[-1])
    return {
        "maxsim": (lambda q, d: lik.maxsim(q, d, d_mask=dm), (Q, D)),
        "normalised": (lambda q, d: lik.maxsim(q, d, d_mask=dm, normalize=True), (Q, D)),
        "varlen": (lambda q, d: lik.maxsim_varlen(q, d, cu_q, cu_d), (flat(Q), flat(D))),
        "pairs": (lambda q, d: score_pairs_packed(q, d, cu_q, cu_d, pq, pd), (flat(Q), flat(D))),
        "padded": (lambda q, d: maxsim_padded(q, d.unsqueeze(1), torch.full((5,), 8), torch.full((5, 1), 20)), (Q[[0, 1, 2, 3, 0]], D)),
        "head": (lambda q, h, w, c: maxsim_from_hidden(q, h, w, c, dm), (Q, H, W, b)),
        "head fp32": (lambda q, h, w, c: maxsim_from_hidden(q, h, w, c, dm), (Q.float(), H.float(), W.float(), b.float())),
    }


NAMES = ["maxsim", "normalised", "varlen", "pairs", "padded", "head", "head fp32"]


def gradients(fn, inputs):
    leaves = [x.detach().clone().requires_grad_() for x in inputs]
    out = fn(*leaves)
    (out * torch.arange(1, out.numel() + 1, device="cuda").view(out.shape)).sum().backward()
    return [out.detach()] + [x.grad for x in leaves]


@pytest.mark.parametrize("name", NAMES)
def test_checkpointed_call_has_the_gradients_of_the_plain_one(name):
    """Non-reentrant checkpointing computes the forward again inside the hook that unpacks a saved tensor."""
    fn, inputs = scoring_calls()[name]
    plain = gradients(fn, inputs)
    again = gradients(lambda *x: checkpoint(fn, *x, use_reentrant=False), inputs)
    # (work in front of the call: what the checkpoint saves then includes tensors of other operators)
    chained = gradients(lambda *x: checkpoint(lambda *y: fn(*[t * 1 for t in y]), *x, use_reentrant=False), inputs)
    for a, b, c in zip(plain, again, chained):
        assert torch.equal(a, b) and torch.equal(a, c)


@pytest.mark.parametrize("name", NAMES)
def test_saved_tensors_may_travel(name):
    fn, inputs = scoring_calls()[name]
    plain = gradients(fn, inputs)
    with torch.autograd.graph.save_on_cpu():
        kept = gradients(fn, inputs)
    for a, b in zip(plain, kept):
        assert torch.equal(a, b)


@pytest.mark.parametrize("per_token_q,per_token_d", [(False, False), (True, False), (False, True), (True, True)])
def test_fp8_scales_on_the_host(per_token_q, per_token_d):
    from late_interaction_kernels_b200.fp8 import maxsim_inference_fp8

    rng = np.random.default_rng(5)
    e4m3 = torch.float8_e4m3fn
    Q, D = dev(rng.standard_normal((3, 8, 64)), e4m3), dev(rng.standard_normal((6, 20, 64)), e4m3)
    sq = torch.rand((3, 8)) if per_token_q else torch.tensor(0.5)
    sd = torch.rand((6, 20)) if per_token_d else torch.tensor(0.02)
    want = maxsim_inference_fp8(Q, D, scale_Q=sq.cuda(), scale_D=sd.cuda())
    assert torch.equal(maxsim_inference_fp8(Q, D, scale_Q=sq, scale_D=sd), want)


def test_what_was_copied_for_the_kernel_may_be_overwritten():
    """A mask of integers and strided embeddings are brought to the kernels' layout by a copy; a program that reuses their
    memory before the backward (a mask buffer filled for the next batch) gets the gradients of the values it passed."""
    import late_interaction_kernels_b200 as lik

    rng = np.random.default_rng(9)
    Q, D = dev(rng.standard_normal((3, 16, 8)), torch.bfloat16), dev(rng.standard_normal((20, 4, 16)), torch.bfloat16)  # [., d, Lq], [Ld, Nd, d]
    qm, dm = dev(rng.integers(0, 2, (3, 8))), dev(rng.integers(0, 2, (4, 20)))

    def step(touch):
        bq, bd = Q.clone().requires_grad_(), D.clone().requires_grad_()
        q, d, m, n = bq * 1, bd * 1, qm.clone(), dm.clone()
        out = lik.maxsim(q.transpose(1, 2), d.transpose(0, 1), q_mask=m, d_mask=n)
        if touch:
            for t in (q, d, m, n):
                t.detach().zero_() if t.is_floating_point() else t.zero_()
        out.sum().backward()
        return out.detach(), bq.grad, bd.grad

    for a, b in zip(step(False), step(True)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("name", NAMES)
def test_forward_mode_is_refused(name):
    """There is no forward-mode rule; a tangent must not get lost on the way."""
    fn, inputs = scoring_calls()[name]
    with torch.autograd.forward_ad.dual_level():
        for i in range(len(inputs)):
            x = [t.clone() for t in inputs]
            x[i] = torch.autograd.forward_ad.make_dual(x[i].requires_grad_(), torch.ones_like(x[i]))
            with pytest.raises(NotImplementedError):
                fn(*x)


def test_an_empty_pair_list_does_not_wait_for_the_gpu():
    """A cascade stage without survivors: no offsets need to be read back (a captured graph could not)."""
    from late_interaction_kernels_b200.score_pairs import score_pairs_packed

    Q, D = torch.randn((6, 64), device="cuda", dtype=torch.bfloat16), torch.randn((9, 64), device="cuda", dtype=torch.bfloat16)
    cu_q, cu_d, none = dev(np.array([0, 2, 6], np.int32)), dev(np.array([0, 9], np.int32)), torch.empty(0, dtype=torch.int32, device="cuda")
    torch.cuda.set_sync_debug_mode("error")
    try:
        scores = score_pairs_packed(Q, D, cu_q, cu_d, none, none)
        grad = score_pairs_packed(Q.requires_grad_(), D, cu_q, cu_d, none, none)
    finally:
        torch.cuda.set_sync_debug_mode("default")
    assert scores.shape == grad.shape == (0,)
    (gq,) = torch.autograd.grad(grad.sum(), Q)
    assert not gq.any()
