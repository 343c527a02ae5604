"""Kernels and launch rules at the sizes where a split or a tile changes: one parametrised test each.

Integer-valued inputs make sums exact in fp32 (every partial sum is far below 2**24), whatever their order: scores and
winners are compared with ``==``, and a gradient is the exact sum rounded once to the output type."""

import numpy as np
import pytest
import torch

import cases
from oracle import maxsim_oracle as O

pytestmark = pytest.mark.gpu


def dev(x, dtype=None):
    if x is None:
        return None
    t = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    return t.to(dtype) if dtype is not None else t


def f32(t):
    return t.detach().float().cpu().numpy()


def ints(rng, *shape):
    return rng.integers(-2, 3, size=shape).astype(np.float32)


def once_rounded(x, dtype):
    return torch.from_numpy(np.ascontiguousarray(x, dtype=np.float32)).to(dtype)


# entries of a document = queries x query tokens.  One launch for both gradients up to 4096 entries and 1536 document
# tokens (from 1025 entries on only with 96 documents or more; from 2**20 winners in all on only with many per token); sorted by a cluster of CTAs per document from 4096 entries
# with few documents; one CTA per document otherwise.
@pytest.mark.parametrize("Nq,Lq,Nd,Ld,dtype", [
    (1, 1, 1, 1, torch.bfloat16),         # one entry, one row
    (3, 5, 2, 1536, torch.float16),       # the longest document of one launch, several blocks per document
    (3, 5, 2, 1537, torch.bfloat16),      # one token more: sorted and reduced separately
    (16, 32, 7, 180, torch.bfloat16),     # 512 entries: 256 threads
    (3, 171, 7, 33, torch.bfloat16),      # 513 entries, rows of 171 winners (not a multiple of four): 512 threads
    (32, 32, 95, 17, torch.float16),      # 1024 entries: the last with few documents
    (25, 41, 95, 17, torch.bfloat16),     # 1025 entries and 95 documents: separate
    (25, 41, 96, 17, torch.bfloat16),     # ... and 96: one launch
    (32, 128, 97, 40, torch.bfloat16),    # 4096 entries
    (241, 17, 97, 40, torch.bfloat16),    # 4097
    (64, 130, 3, 50, torch.bfloat16),     # cluster of four, rows of 130 winners
    (300, 128, 1, 2000, torch.float16),   # cluster of eight, one document, query rows split over blocks
    (2, 5, 200, 17, torch.bfloat16),      # one launch with grad_q split over document ranges
    (8, 128, 1023, 20, torch.bfloat16),   # ... the last of these before 2**20 winners
    (8, 128, 1024, 20, torch.bfloat16),   # 2**20: two streams
    (128, 32, 256, 20, torch.float16),    # 2**20, many winners per token, grad_q not split: one launch
])
def test_backward_splits(Nq, Lq, Nd, Ld, dtype):
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200.forward import maxsim_forward

    rng = np.random.default_rng(Nq * 131 + Nd)
    Q, D, g = ints(rng, Nq, Lq, 64), ints(rng, Nd, Ld, 64), ints(rng, Nq, Nd)
    dm = cases.prefix_mask(rng.integers(0, Ld + 1, size=Nd), Ld)
    dm[0] = True
    tQ, tD = dev(Q, dtype).requires_grad_(True), dev(D, dtype).requires_grad_(True)
    (lik.maxsim(tQ, tD, None, dev(dm)) * dev(g)).sum().backward()
    _, am = maxsim_forward(tQ.detach(), tD.detach(), None, dev(dm), save_argmax=True)
    wq, wd = O.backward_from_argmax(g, Q, D, am.cpu().numpy().reshape(Nq, Nd, Lq))
    assert torch.equal(tQ.grad.cpu(), once_rounded(wq, dtype))
    assert torch.equal(tD.grad.cpu(), once_rounded(wd, dtype))


@pytest.mark.parametrize("Nq,K,Lq,Ld", [(1, 1, 4, 9), (5, 7, 30, 129), (40, 5, 33, 64)])
def test_backward_of_candidate_lists_and_packed_rows_without_owner(Nq, K, Lq, Ld):
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200.forward import maxsim_forward

    rng = np.random.default_rng(Nq + K)
    Q, D, g = ints(rng, Nq, Lq, 128), ints(rng, Nq, K, Ld, 128), ints(rng, Nq, K)
    tQ, tD = dev(Q, torch.bfloat16).requires_grad_(True), dev(D, torch.bfloat16).requires_grad_(True)
    (lik.maxsim(tQ, tD) * dev(g)).sum().backward()
    wq, wd = np.zeros_like(Q), np.zeros_like(D)
    for i in range(Nq):
        _, am = O.maxsim(Q[i : i + 1], D[i], None, None, return_argmax=True)  # ties to the lower column, as the kernel
        wq[i : i + 1], wd[i] = O.backward_from_argmax(g[i : i + 1], Q[i : i + 1], D[i], am)
    assert torch.equal(tQ.grad.cpu(), once_rounded(wq, torch.bfloat16))
    assert torch.equal(tD.grad.cpu(), once_rounded(wd, torch.bfloat16))
    # packed: rows in front of the first and behind the last document belong to none, their gradient is zero
    dl = rng.integers(0, Ld + 1, size=K)
    dl[-1] = Ld
    cu_d = (3 + np.concatenate([[0], np.cumsum(dl)])).astype(np.int32)
    cu_q = (np.arange(Nq + 1) * Lq).astype(np.int32)
    Dp = ints(rng, int(cu_d[-1]) + 13, 128)
    tQ, tD = dev(Q.reshape(-1, 128), torch.bfloat16).requires_grad_(True), dev(Dp, torch.bfloat16).requires_grad_(True)
    (lik.maxsim_varlen(tQ, tD, dev(cu_q), dev(cu_d), Lq, Ld) * dev(g)).sum().backward()
    wq, wd = O.varlen_grads(g, Q.reshape(-1, 128), Dp, cu_q, cu_d)
    assert torch.equal(tQ.grad.cpu(), once_rounded(wq, torch.bfloat16))
    assert torch.equal(tD.grad.cpu(), once_rounded(wd, torch.bfloat16))


# fp32 tiles: 32 query tokens of one query, or of two (from two blocks per SM on), x 128 document tokens, slabs of 64 features
@pytest.mark.parametrize("Nq,Lq,Nd,Ld,d", [(1, 1, 1, 1, 1), (2, 31, 3, 127, 63), (2, 32, 2, 128, 64), (3, 33, 5, 129, 65), (5, 7, 4, 257, 132),
                                              (34, 31, 19, 127, 64), (35, 33, 19, 129, 65)])
def test_exact_fp32_tiles(Nq, Lq, Nd, Ld, d):
    from late_interaction_kernels_b200.forward import maxsim_forward

    rng = np.random.default_rng(Ld)
    Q, D = ints(rng, Nq, Lq, d), ints(rng, Nd, Ld, d)
    dm = cases.prefix_mask(rng.integers(1, Ld + 1, size=Nd), Ld)
    holes = rng.random((Nd, Ld)) < 0.6
    for m in (None, dm, holes):
        want, am = O.maxsim(Q, D, None, m, return_argmax=True)
        s, got = maxsim_forward(dev(Q), dev(D), None, dev(m), save_argmax=True)
        assert np.array_equal(f32(s), want) and np.array_equal(got.cpu().numpy().reshape(am.shape), am)


# candidate lists of every CTA merged at once (many queries) or in parts (few), lists shorter and longer than k, ties
@pytest.mark.parametrize("Nq,Nd,k", [(1, 1, 1), (1, 149, 149), (1, 20000, 100), (2, 30000, 128), (9, 9000, 127), (40, 3000, 33)])
def test_candidate_lists_are_merged_in_order(Nq, Nd, k):
    from late_interaction_kernels_b200.topk import maxsim_topk

    rng = np.random.default_rng(Nd)
    Q, D = ints(rng, Nq, 8, 32), ints(rng, Nd, 3, 32)
    for largest in (True, False):
        s, i = maxsim_topk(dev(Q, torch.bfloat16), dev(D, torch.bfloat16), k, largest=largest)
        full = torch.from_numpy(O.maxsim(Q, D))
        order = torch.sort(full, dim=-1, descending=largest, stable=True).indices[:, :k]
        assert torch.equal(i.cpu(), order) and torch.equal(s.cpu().double(), torch.gather(full, 1, order).double())


# norm groups of 8, 16 and 32 lanes with 16-byte loads; rows that do not start on 16 bytes element by element.  Rows are
# one-hot times a power of two: the norm is a power of two, the normalised row and so the scores are exact.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("d", [1, 8, 33, 64, 136, 264, 520])
def test_row_norms_by_width(dtype, d):
    import late_interaction_kernels_b200 as lik

    rng = np.random.default_rng(d)
    def rows(n, length):
        x = np.zeros((n, length, d), np.float32)
        at = rng.integers(0, d, size=(n, length))
        np.put_along_axis(x, at[..., None], (2.0 ** rng.integers(-3, 4, size=(n, length)) * rng.choice([-1, 1], size=(n, length)))[..., None].astype(np.float32), -1)
        return x
    Q, D = rows(3, 5), rows(37, 21)
    dm = cases.prefix_mask(rng.integers(1, 22, size=37), 21)
    want = O.maxsim(np.sign(Q), np.sign(D), None, dm)
    big = torch.zeros(D.size + 1, device="cuda", dtype=dtype)
    shifted = big[1:].view(D.shape)  # starts 2 or 4 bytes behind a 16-byte boundary
    shifted.copy_(dev(D))
    for t in (dev(D, dtype), shifted):
        assert np.array_equal(f32(lik.maxsim(dev(Q, dtype), t, None, dev(dm), normalize=True)), want)


# documents of a masked batch are dealt to the CTAs by length up to 1024 of them, in ranges beyond
@pytest.mark.parametrize("Nd,Ld,lens", [(149, 130, "empty"), (300, 70, "ragged"), (297, 140, "same"), (1024, 9, "ragged"), (1025, 9, "ragged")])
def test_document_head_deals_ragged_documents(Nd, Ld, lens):
    from late_interaction_kernels_b200.fused_head import maxsim_from_hidden

    rng = np.random.default_rng(Nd)
    n = {"empty": np.where(np.arange(Nd) % 3, 0, Ld), "ragged": rng.integers(0, Ld + 1, size=Nd), "same": np.full(Nd, Ld - 1)}[lens]
    Q, H, W = ints(rng, 2, 9, 32), ints(rng, Nd, Ld, 64), np.eye(32, 64, dtype=np.float32)  # projected rows are integers too
    dm = cases.prefix_mask(n, Ld)
    got = maxsim_from_hidden(*(dev(x, torch.bfloat16) for x in (Q, H, W)), None, dev(dm), normalize=False)
    assert np.array_equal(f32(got), O.maxsim(Q, H[..., :32], None, dm))


# up to four groups of query tiles: norms taken inside the scoring kernel; more groups: by a pass in front.  The two sum a row in
# the same order, so a query scores the same bits alone and in a large batch.
@pytest.mark.parametrize("Lq,Nd,Ld,d,dtype,mask", [
    (32, 1, 1, 128, torch.bfloat16, "none"),
    (32, 301, 300, 128, torch.float16, "prefix"),
    (8, 150, 257, 96, torch.bfloat16, "holes"),   # two tiles, the second of one row
    (128, 40, 1030, 64, torch.float16, "holes"),  # many tiles per document, one K slab
    (17, 299, 33, 40, torch.bfloat16, "prefix"),  # rows of 80 bytes
    (31, 7, 2049, 16, torch.float16, "none"),
])
def test_norms_in_the_scoring_kernel(Lq, Nd, Ld, d, dtype, mask):
    from late_interaction_kernels_b200.forward import maxsim_forward
    import late_interaction_kernels_b200 as lik

    rng = np.random.default_rng(Nd + d)
    D = dev(rng.standard_normal((Nd, Ld, d)).astype(np.float32) * rng.uniform(0.01, 30, size=(Nd, Ld, 1)).astype(np.float32), dtype)
    Q = dev(rng.standard_normal((1040 // Lq + 9, Lq, d)).astype(np.float32), dtype)  # more rows than eight query tiles hold
    dm = {"none": None, "prefix": cases.prefix_mask(rng.integers(0, Ld + 1, size=Nd), Ld), "holes": rng.random((Nd, Ld)) < 0.6}[mask]
    many, many_am = maxsim_forward(Q, D, None, dev(dm), save_argmax=True, normalize=True)
    for lo, n in ((0, 1), (1, 128 // Lq * 2), (1, 128 // Lq * 3), (0, 128 // Lq * 8)):  # one tile, two, three (the last alone), eight
        q = Q[lo : lo + n]
        s, am = maxsim_forward(q, D, None, dev(dm), save_argmax=True, normalize=True)
        assert torch.equal(s, many[lo : lo + q.shape[0]])
        assert torch.equal(am.view(q.shape[0], Nd, Lq), many_am.view(-1, Nd, Lq)[lo : lo + q.shape[0]])
        assert torch.equal(lik.maxsim(q, D, d_mask=dev(dm), normalize=True), s)
    # candidate lists: documents belong to one query each
    K = min(Nd, 5)
    n = min(Q.shape[0], Nd // K)
    D4, m4 = D[: n * K].view(n, K, Ld, d), None if dm is None else dev(dm)[: n * K].view(n, K, Ld)
    kd = lik.maxsim(Q[:n], D4, d_mask=m4, normalize=True)
    assert torch.equal(kd, torch.stack([many[i, i * K : (i + 1) * K] for i in range(n)]))
    lik.check_device_status()


# documents behind 10 240 tokens, where a cluster's counts would no longer fit in shared memory: a CTA per document, and one
# histogram from 12 800 tokens on
@pytest.mark.parametrize("Nq,Lq,Nd,Ld", [(4, 32, 3, 10_240), (64, 130, 2, 10_241), (40, 128, 2, 25_000)])
@pytest.mark.parametrize("as_list", [False, True])
def test_backward_of_very_long_documents(Nq, Lq, Nd, Ld, as_list):
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200.forward import maxsim_forward
    from late_interaction_kernels_b200.score_pairs import score_pairs_packed

    rng = np.random.default_rng(Ld)
    Q, D, g = ints(rng, Nq, Lq, 64), ints(rng, Nd, Ld, 64), ints(rng, Nq, Nd)
    tQ, tD = dev(Q, torch.bfloat16).requires_grad_(True), dev(D, torch.bfloat16).requires_grad_(True)
    _, am = maxsim_forward(tQ.detach(), tD.detach(), save_argmax=True)
    if as_list:
        at = lambda n, step: dev(np.arange(0, (n + 1) * step, step, dtype=np.int32))
        i, j = np.divmod(np.arange(Nq * Nd, dtype=np.int32), Nd)
        s = score_pairs_packed(tQ.view(-1, 64), tD.view(-1, 64), at(Nq, Lq), at(Nd, Ld), dev(i), dev(j), max_seqlen_q=Lq, max_seqlen_d=Ld)
        s.backward(dev(g).view(-1))
    else:
        lik.maxsim(tQ, tD).backward(dev(g))
    win = am.view(Nq, Nd, Lq).cpu().numpy()
    wq, wd = np.zeros_like(Q), np.zeros_like(D)
    for i in range(Nq):
        for j in range(Nd):
            wq[i] += g[i, j] * D[j, win[i, j]]
            np.add.at(wd[j], win[i, j], g[i, j] * Q[i])
    assert torch.equal(tQ.grad.cpu(), once_rounded(wq, torch.bfloat16))
    assert torch.equal(tD.grad.cpu(), once_rounded(wd, torch.bfloat16))


# the one-launch backward (documents without gaps) against the sort and reduction kernels (a row between the documents)
@pytest.mark.parametrize("Nq,Lq,Nd,Ld,stride,grouped", [
    (1, 32, 3, 40, 32, False),
    (5, 7, 9, 33, 7, False),       # winners read one at a time
    (16, 32, 16, 60, 32, False),   # 512 entries
    (3, 171, 7, 33, 172, False),   # padded winner rows
    (25, 41, 97, 17, 44, False),   # 1100 entries
    (32, 128, 97, 40, 128, False),  # 4096
    (6, 24, 24, 50, 24, True),     # candidate lists
])
def test_gradients_do_not_depend_on_the_route(Nq, Lq, Nd, Ld, stride, grouped):
    from late_interaction_kernels_b200 import _lib, _ops

    gen = torch.Generator(device="cuda").manual_seed(Nd * 64 + Ld)
    rand = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    Q, D, dmask = rand(Nq * Lq, 64).bfloat16(), rand(Nd, Ld + 1, 64).bfloat16(), torch.rand((Nd, Ld + 1), generator=gen, device="cuda") < 0.8
    g = rand(Nd if grouped else Nq * Nd)
    how = dict(pairing=_lib.PAIR_GROUPED if grouped else _lib.PAIR_CROSS, group=Nd // Nq if grouped else 0)
    q = _ops.SeqSpec(Q, Nq, Lq, Lq)
    apart = _ops.SeqSpec(D.view(-1, 64), Nd, Ld, Ld + 1, mask=dmask.view(torch.uint8).view(-1))
    packed = _ops.SeqSpec(D[:, :Ld].reshape(-1, 64), Nd, Ld, Ld, mask=dmask[:, :Ld].contiguous().view(torch.uint8).view(-1))
    _, am = _ops.forward(q, packed, save_argmax=True, argmax_stride=stride, **how)
    for norm in (_lib.NORM_NONE, _lib.NORM_BOTH):
        a, b = (_ops.backward(q, d, g, am, normalize=norm, **how) for d in (apart, packed))
        assert torch.equal(a[0], b[0])
        assert torch.equal(a[1].view(Nd, Ld + 1, 64)[:, :Ld], b[1].view(Nd, Ld, 64))


# the portable forward stages four elements at a time where rows allow it and one by one otherwise: the same scores
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16, torch.float8_e4m3fn])
@pytest.mark.parametrize("d", [4, 60, 64, 68, 196])
def test_staging_of_the_portable_forward(dtype, d):
    from late_interaction_kernels_b200 import _ops

    gen = torch.Generator(device="cuda").manual_seed(d)

    def sides(shift):  # the same rows, `shift` elements behind a boundary and at a pitch that is a multiple of four or not
        out = []
        for i, (n, length) in enumerate([(3, 35), (4, 130)]):
            rows = torch.randn((n * length, d), generator=gen.manual_seed(i), device="cuda").to(dtype)
            buf = torch.zeros((n * length, d + 4 + shift), dtype=torch.float32, device="cuda").to(dtype)
            buf[:, shift:shift + d] = rows
            out.append(_ops.SeqSpec(buf[:, shift:shift + d], n, length, length))
        return out

    want = _ops.forward(*sides(1), engine=1, save_argmax=True)
    for shift in (0, 4):
        got = _ops.forward(*sides(shift), engine=1, save_argmax=True)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("bad", [-1, 9])
def test_portable_forward_reports_lengths_out_of_range_under_a_mask(bad):
    """Masked documents are trimmed before the kernel sees their lengths; what is wrong with them is reported all the same."""
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200 import _ops

    q = _ops.SeqSpec(torch.ones((4, 8), device="cuda"), 2, 2, 2)
    lens = torch.tensor([3, bad, 8], dtype=torch.int32, device="cuda")
    d = _ops.SeqSpec(torch.ones((24, 8), device="cuda"), 3, 8, 8, lens=lens, mask=torch.ones(24, dtype=torch.uint8, device="cuda"))
    lik.check_device_status()
    scores, _ = _ops.forward(q, d)
    with pytest.raises(RuntimeError):
        lik.check_device_status()
    assert scores.tolist() == [16.0, 16.0 if bad > 0 else 0.0, 16.0] * 2


def test_portable_forward_without_room_for_trimmed_lengths():
    """The scores of masked documents whether their padding is trimmed or read."""
    import ctypes as C

    from late_interaction_kernels_b200 import _lib, _ops

    rng = np.random.default_rng(0)
    mask = dev(rng.integers(0, 2, (5, 40)).astype(np.uint8))
    q = _ops.SeqSpec(dev(ints(rng, 21, 20)), 3, 7, 7)
    d = _ops.SeqSpec(dev(ints(rng, 200, 20)), 5, 40, 40, mask=mask.view(-1))
    want, _ = _ops.forward(q, d, engine=1)
    got = torch.full((15,), -7.0, device="cuda")
    a = _lib.FwdArgs(q=q.c_struct(), d=d.c_struct(), dtype=_lib.LIK_F32, dim=20, pairing=_lib.PAIR_CROSS, engine=1, scores=got.data_ptr(),
                     status=_ops.status_word(got.device).data_ptr())
    assert _lib.load().lik_maxsim_fwd_workspace(C.byref(a)) > 0
    _lib.check(_lib.load().lik_maxsim_fwd(C.byref(a), _lib.stream_ptr(got.device)), "lik_maxsim_fwd")
    assert torch.equal(got, want)


@pytest.mark.parametrize("shift", [0, 8, 16])
def test_workspaces_and_winners_off_a_16_byte_boundary(shift):
    """A caller's workspace of the C interface may start on any multiple of eight bytes, its array of winners anywhere:
    fused top-k, a packed backward with clustered sorting, and winners of queries shorter than their rows."""
    import ctypes as C

    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200 import _lib, _ops

    lib, cuda = _lib.load(), torch.device("cuda")
    rng = np.random.default_rng(1)
    status, st = _ops.status_word(torch.device("cuda", 0)), _lib.stream_ptr(torch.device("cuda", 0))
    room = lambda n: torch.empty(n + 64, dtype=torch.uint8, device=cuda)

    # top-k
    Q, D = dev(ints(rng, 3, 8, 64), torch.bfloat16), dev(ints(rng, 300, 9, 64), torch.bfloat16)
    want = lik.retrieve(Q, D, 5, normalize=False)
    q, d = _ops.padded_spec(Q), _ops.padded_spec(D)
    s, i = torch.empty((3, 5), device=cuda), torch.empty((3, 5), dtype=torch.int64, device=cuda)
    a = _lib.FwdArgs(q=q.c_struct(), d=d.c_struct(), dtype=_lib.LIK_BF16, dim=64, pairing=_lib.PAIR_CROSS, argmax_stride=8, status=status.data_ptr())
    t = _lib.TopkSpec(k=5, largest=1, index_offset=0, out_scores=s.data_ptr(), out_index=i.data_ptr(), flags=0, doc_base=0)
    n = lib.lik_maxsim_fwd_topk_workspace(C.byref(a), C.byref(t))
    ws = room(n)
    a.workspace, a.workspace_bytes = ws.data_ptr() + shift, n
    _lib.check(lib.lik_maxsim_fwd_topk(C.byref(a), C.byref(t), st), "lik_maxsim_fwd_topk")
    assert torch.equal(s, want[0]) and torch.equal(i, want[1])

    # packed queries of 90 to 130 tokens, so that the winners' rows are partly behind their query, and their backward
    ql, dl = rng.integers(90, 131, 60), rng.integers(20, 41, 5)
    cu = lambda x: dev(np.concatenate([[0], np.cumsum(x)]).astype(np.int32))
    Qp, Dp = dev(ints(rng, int(ql.sum()), 64), torch.bfloat16), dev(ints(rng, int(dl.sum()), 64), torch.bfloat16)
    q, d = _ops.packed_spec(Qp, cu(ql), 130), _ops.packed_spec(Dp, cu(dl), 40)
    want_s, want_am = _ops.forward(q, d, save_argmax=True, argmax_stride=132)
    am = torch.zeros(300 * 132 + 16, dtype=torch.int32, device=cuda)[shift // 8:][:300 * 132].view(300, 132)
    got_s = torch.empty(300, device=cuda)
    a = _lib.FwdArgs(q=q.c_struct(), d=d.c_struct(), dtype=_lib.LIK_BF16, dim=64, pairing=_lib.PAIR_CROSS, scores=got_s.data_ptr(),
                     argmax=am.data_ptr(), argmax_stride=132, status=status.data_ptr())
    n = lib.lik_maxsim_fwd_workspace(C.byref(a))
    ws = room(n)
    a.workspace, a.workspace_bytes = ws.data_ptr(), n
    _lib.check(lib.lik_maxsim_fwd(C.byref(a), st), "lik_maxsim_fwd")
    assert torch.equal(got_s, want_s) and torch.equal(am, want_am)
    g = dev(ints(rng, 300))
    want_q, want_d = _ops.backward(q, d, g, want_am)
    gq, gd = torch.empty_like(Qp), torch.empty_like(Dp)
    b = _lib.BwdArgs(q=q.c_struct(), d=d.c_struct(), dtype=_lib.LIK_BF16, dim=64, pairing=_lib.PAIR_CROSS, deterministic=1, grad_scores=g.data_ptr(),
                     argmax=am.data_ptr(), argmax_stride=132, grad_dtype=_lib.LIK_BF16, grad_q=gq.data_ptr(), grad_d=gd.data_ptr(),
                     status=status.data_ptr())
    n = lib.lik_maxsim_bwd_workspace(C.byref(b))
    ws = room(n)
    b.workspace, b.workspace_bytes = ws.data_ptr() + shift, n
    _lib.check(lib.lik_maxsim_bwd(C.byref(b), st), "lik_maxsim_bwd")
    assert torch.equal(gq, want_q) and torch.equal(gd, want_d)
    lik.check_device_status()


@pytest.mark.parametrize("Nq,Nd", [(4, 256), (4, 257), (1, 256), (9, 255), (3, 1)])
def test_fp32_documents_in_the_order_of_their_lengths(Nq, Nd):
    """Up to 256 documents with given lengths are dealt longest first (equal lengths in their own order), more as they come.
    Small integers: every sum is exact."""
    import late_interaction_kernels_b200 as lik

    gen = torch.Generator(device="cuda").manual_seed(Nd)
    Lq, Ld, d = 20, 70, 40
    Q, D = (torch.randint(-2, 3, s, generator=gen, device="cuda").float() for s in ((Nq, Lq, d), (Nd, Ld, d)))
    lens = torch.tensor([0, 1, 33, 64, Ld, Ld], device="cuda")[torch.randint(0, 6, (Nd,), generator=gen, device="cuda")]
    mask = torch.arange(Ld, device="cuda")[None] < lens[:, None]
    s = torch.einsum("isd,jtd->ijst", Q, D).masked_fill(~mask[None, :, None, :], float("-inf")).amax(-1)
    want = torch.where(torch.isinf(s), torch.zeros_like(s), s).sum(-1)
    assert torch.equal(lik.maxsim(Q, D, d_mask=mask), want)
