"""The scoring kernel of two streams per CTA, which takes problems of at least twelve units per SM, at the sizes where its pieces
(96 tokens), boxes (32) and query tiles (128 rows, two at a time) change.

Integer-valued inputs make every sum exact in fp32, so scores and winners are compared with ``==`` against plain torch."""

import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 159, 191, 192, 193, 223, 287, 288, 289, 300]


def ints(gen, *shape, scale=1.0):
    return torch.randint(-2, 3, shape, generator=gen, device="cuda").float() * scale


def lengths(n, ld, gen):
    pool = torch.tensor([x for x in LENGTHS if x <= ld] + [ld], device="cuda")
    return pool[torch.randint(0, len(pool), (n,), generator=gen, device="cuda")]


def reference(Q, D, mask):
    """Row maxima [Nq, Nd, Lq] and their first positions (-1: none), a slice of documents at a time."""
    vals, pos = [], []
    for j in range(0, D.shape[0], 64):
        s = torch.einsum("isd,jtd->ijst", Q, D[j:j + 64])
        s = s.masked_fill(~mask[None, j:j + 64, None, :], float("-inf"))
        m = s.amax(-1)
        t = torch.arange(s.shape[-1], device="cuda").expand_as(s)
        p = torch.where(s == m[..., None], t, s.shape[-1]).amin(-1)
        none = torch.isinf(m)
        vals.append(torch.where(none, torch.zeros_like(m), m))
        pos.append(torch.where(none, torch.full_like(p, -1), p))
    return torch.cat(vals, 1), torch.cat(pos, 1)


# units = ceil(query tiles / 2) * documents; tiles: 128 // lq queries each, or 128-row pieces of one query
@pytest.mark.parametrize("Nq,Nd,Lq,Ld,d,dtype", [
    (4, 1800, 32, 300, 128, torch.bfloat16),   # one tile: the streams' accumulators take turns
    (1, 1777, 5, 65, 64, torch.float16),       # one query of five tokens, rows of one slab
    (8, 1800, 32, 129, 128, torch.float16),    # two tiles
    (9, 900, 32, 193, 96, torch.bfloat16),     # three tiles, the last group's second place empty; rows that do not fill two slabs
    (11, 900, 24, 97, 128, torch.bfloat16),    # queries that lie across warps
    (30, 450, 128, 33, 32, torch.float16),     # full tiles, documents of one or two boxes
    (5, 450, 300, 289, 64, torch.bfloat16),    # queries of three pieces, the last short
    (7, 1800, 16, 31, 128, torch.bfloat16),    # documents shorter than a box
])
@pytest.mark.parametrize("holes", [False, True])
def test_scores_and_winners(Nq, Nd, Lq, Ld, d, dtype, holes):
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200.forward import maxsim_forward

    gen = torch.Generator(device="cuda").manual_seed(Nq * 1009 + Ld)
    Q, D = ints(gen, Nq, Lq, d), ints(gen, Nd, Ld, d)
    mask = torch.arange(Ld, device="cuda")[None] < lengths(Nd, Ld, gen)[:, None]
    if holes:
        mask &= torch.rand(Nd, Ld, generator=gen, device="cuda") < 0.7
    val, pos = reference(Q, D, mask)
    tq, td = Q.to(dtype), D.to(dtype)
    scores, am = maxsim_forward(tq, td, None, mask, save_argmax=True)
    assert torch.equal(scores.view(Nq, Nd), val.sum(-1))
    assert torch.equal(am.view(Nq, Nd, Lq).long(), pos)
    assert torch.equal(lik.maxsim(tq, td, d_mask=mask), val.sum(-1))
    if Lq <= 128:
        k = 37
        ts, ti = lik.retrieve(tq, td, k, d_mask=mask, normalize=False)
        order = torch.sort(val.sum(-1), dim=1, descending=True, stable=True)
        assert torch.equal(ts, order.values[:, :k]) and torch.equal(ti, order.indices[:, :k])
    lik.check_device_status(scores.device)


def test_scores_beyond_two_to_the_64():
    from late_interaction_kernels_b200.forward import maxsim_forward

    gen = torch.Generator(device="cuda").manual_seed(5)
    Q, D = ints(gen, 4, 32, 64, scale=2.0**31), ints(gen, 1800, 100, 64, scale=2.0**31)
    mask = torch.ones(1800, 100, dtype=torch.bool, device="cuda")
    val, pos = reference(Q, D, mask)
    scores, am = maxsim_forward(Q.bfloat16(), D.bfloat16(), None, mask, save_argmax=True)
    assert torch.equal(scores.view(4, 1800), val.sum(-1)) and torch.equal(am.view(4, 1800, 32).long(), pos)


# candidate lists and pair lists: the query tile changes with every query
@pytest.mark.parametrize("Nq,K,Lq,Ld", [(64, 30, 32, 300), (300, 7, 30, 97)])
def test_lists(Nq, K, Lq, Ld):
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200.score_pairs import score_pairs_packed

    gen = torch.Generator(device="cuda").manual_seed(K)
    Q, D = ints(gen, Nq, Lq, 128), ints(gen, Nq * K, Ld, 128)
    lens = lengths(Nq * K, Ld, gen)
    mask = torch.arange(Ld, device="cuda")[None] < lens[:, None]
    want = torch.cat([reference(Q[i:i + 1], D[i * K:(i + 1) * K], mask[i * K:(i + 1) * K])[0].sum(-1) for i in range(Nq)])
    got = lik.maxsim(Q.bfloat16(), D.view(Nq, K, Ld, 128).bfloat16(), d_mask=mask.view(Nq, K, Ld))
    assert torch.equal(got, want)
    # the same pairs as a list over packed documents, often enough for 32 units per SM
    rep = -(-32 * 160 // (Nq * K))
    cu_q = torch.arange(Nq + 1, device="cuda", dtype=torch.int32) * Lq
    cu_d = torch.nn.functional.pad(lens.cumsum(0), (1, 0)).int()
    pq = torch.arange(Nq, device="cuda", dtype=torch.int32).repeat_interleave(K).repeat(rep)
    pd = torch.arange(Nq * K, device="cuda", dtype=torch.int32).repeat(rep)
    s = score_pairs_packed(Q.view(-1, 128).bfloat16(), D[mask].bfloat16(), cu_q, cu_d, pq, pd, max_seqlen_q=Lq, max_seqlen_d=Ld)
    assert torch.equal(s.view(rep, Nq, K), want.expand(rep, Nq, K))
    lik.check_device_status(s.device)


# multipliers per document token: inverse norms that ride with the tiles (row counts that are multiples of four) or are staged by
# the epilogue, per-token scales of e4m3; 1e-5 as for all fp32 sums of exact products
@pytest.mark.parametrize("Ld", [96, 97, 128, 300])
@pytest.mark.parametrize("holes", [False, True])
def test_multipliers(Ld, holes):
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200.fp8 import maxsim_inference_fp8, quantize_fp8_per_token

    gen = torch.Generator(device="cuda").manual_seed(Ld)
    Nq, Nd, Lq = 40, 400, 32
    Q, D = torch.randn(Nq, Lq, 128, generator=gen, device="cuda").bfloat16(), torch.randn(Nd, Ld, 128, generator=gen, device="cuda").bfloat16()
    mask = torch.arange(Ld, device="cuda")[None] < lengths(Nd, Ld, gen)[:, None]
    if holes:
        mask &= torch.rand(Nd, Ld, generator=gen, device="cuda") < 0.7
    unit = [x.double() / x.double().norm(dim=-1, keepdim=True) for x in (Q, D)]
    want = reference(*unit, mask)[0].sum(-1)
    got = lik.maxsim(Q, D, d_mask=mask, normalize=True).double()
    assert (got - want).abs().max() <= 1e-5 * want.abs().max()
    (q8, sq), (d8, sd) = quantize_fp8_per_token(Q), quantize_fp8_per_token(D)
    want = reference(q8.double() * sq.double()[..., None], d8.double() * sd.double()[..., None], mask)[0].sum(-1)
    got = maxsim_inference_fp8(q8, d8, scale_Q=sq, scale_D=sd, d_mask=mask).double()
    assert (got - want).abs().max() <= 1e-5 * want.abs().max()


def test_long_queries_need_one_partial_sum_per_tile_and_document():
    """Queries of more than 128 tokens leave one partial sum per 128-row tile and document in either kernel: the static scratch
    (16 MiB) holds those of 128 tiles x 9000 documents with room to spare."""
    import ctypes as C

    from late_interaction_kernels_b200 import _lib, _ops

    lib = _lib.load()
    gen = torch.Generator(device="cuda").manual_seed(9)
    Nq, Lq, Nd, Ld, d = 64, 130, 9000, 4, 16  # 128 tiles x 9000 documents
    Q, D = ints(gen, Nq, Lq, d).bfloat16(), ints(gen, Nd, Ld, d).bfloat16()
    q, dd = _ops.padded_spec(Q), _ops.padded_spec(D)
    out = torch.full((Nq, Nd), float("nan"), device="cuda")
    a = _lib.FwdArgs(
        q=q.c_struct(), d=dd.c_struct(), dtype=_lib.lik_dtype(Q.dtype), dim=d, pairing=_lib.PAIR_CROSS, group=0, pair_q=None, pair_d=None,
        n_pairs=0, normalize=_lib.NORM_NONE, engine=0, scores=out.data_ptr(), argmax=None, argmax_stride=Lq, reserved=0, workspace=None,
        workspace_bytes=0, status=_ops.status_word(Q.device).data_ptr(),
    )
    assert 128 * Nd * 4 <= lib.lik_maxsim_fwd_workspace(C.byref(a)) <= 128 * Nd * 4 + 4096
    _lib.check(lib.lik_maxsim_fwd_static(C.byref(a), torch.cuda.current_stream().cuda_stream), "lik_maxsim_fwd_static")
    want = reference(Q.float(), D.float(), torch.ones(Nd, Ld, dtype=torch.bool, device="cuda"))[0].sum(-1)
    assert torch.equal(out, want)


@pytest.mark.parametrize("Nq,Lq,Ld,d", [(5, 300, 289, 64), (16, 24, 97, 128), (40, 32, 300, 96)])
def test_few_documents_and_many_give_the_same_bits(Nq, Lq, Ld, d):
    """The first documents alone go to the kernel of smaller problems: same products, same order of every sum."""
    import late_interaction_kernels_b200 as lik

    gen = torch.Generator(device="cuda").manual_seed(Lq)
    Q, D = torch.randn(Nq, Lq, d, generator=gen, device="cuda").bfloat16(), torch.randn(1800, Ld, d, generator=gen, device="cuda").bfloat16()
    mask = torch.arange(Ld, device="cuda")[None] < lengths(1800, Ld, gen)[:, None]
    with torch.no_grad():
        assert torch.equal(lik.maxsim(Q, D, d_mask=mask)[:, :20], lik.maxsim(Q, D[:20], d_mask=mask[:20]))


def topk_args(Q, D, mask, k, out_s=None, out_i=None, flags=0, doc_base=0):
    from late_interaction_kernels_b200 import _lib, _ops

    q, d = _ops.padded_spec(Q), _ops.padded_spec(D, mask)
    a = _lib.FwdArgs(
        q=q.c_struct(), d=d.c_struct(), dtype=_lib.lik_dtype(Q.dtype), dim=Q.shape[-1], pairing=_lib.PAIR_CROSS,
        group=0, pair_q=None, pair_d=None, n_pairs=0, normalize=_lib.NORM_NONE, engine=0, scores=None, argmax=None, argmax_stride=Q.shape[1],
        reserved=0, workspace=None, workspace_bytes=0, status=_ops.status_word(Q.device).data_ptr(),
    )
    a.keep = q, d
    return a, _lib.TopkSpec(k=k, largest=1, index_offset=0, out_scores=_lib.ptr(out_s), out_index=_lib.ptr(out_i), flags=flags, doc_base=doc_base)


@pytest.mark.parametrize("Nq", [3, 40])
def test_topk_in_a_workspace_that_holds_the_lists_of_the_smaller_kernel(Nq):
    """A call of its own falls back to the kernel whose lists take half the bytes when the buffer holds no more."""
    import ctypes as C

    from late_interaction_kernels_b200 import _lib

    lib = _lib.load()
    gen = torch.Generator(device="cuda").manual_seed(Nq)
    k, Nd = 17, 32 * torch.cuda.get_device_properties(0).multi_processor_count * (2 if Nq < 5 else 1)
    Q, D = ints(gen, Nq, 32, 64).bfloat16(), ints(gen, Nd, 40, 64).bfloat16()
    mask = torch.arange(40, device="cuda")[None] < lengths(Nd, 40, gen)[:, None]
    s, i = torch.empty(Nq, k, device="cuda"), torch.empty(Nq, k, dtype=torch.long, device="cuda")
    a, t = topk_args(Q, D, mask, k, s, i)
    assert lib.lik_maxsim_fwd_kernel(C.byref(a), C.byref(t)) == 2
    whole = lib.lik_maxsim_fwd_topk_workspace(C.byref(a), C.byref(t))
    t.flags = _lib.TOPK_PARTIAL  # the size that a piece without LIK_TOPK_LARGE needs
    small = lib.lik_maxsim_fwd_topk_workspace(C.byref(a), C.byref(t))
    t.flags |= _lib.TOPK_LARGE
    assert lib.lik_maxsim_fwd_topk_workspace(C.byref(a), C.byref(t)) == whole and small < 0.6 * whole
    t.flags = 0
    want = torch.sort(reference(Q.float(), D.float(), mask)[0].sum(-1), dim=1, descending=True, stable=True)
    for size in (whole, small):
        s.fill_(float("nan"))
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        a.workspace, a.workspace_bytes = ws.data_ptr(), size
        _lib.check(lib.lik_maxsim_fwd_topk(C.byref(a), C.byref(t), _lib.stream_ptr(ws.device)), "lik_maxsim_fwd_topk")
        assert torch.equal(s, want.values[:, :k]) and torch.equal(i, want.indices[:, :k])
    a.workspace_bytes = small - 256
    assert lib.lik_maxsim_fwd_topk(C.byref(a), C.byref(t), _lib.stream_ptr(ws.device)) == -4


def test_topk_lists_of_many_queries_take_no_more_than_before():
    """The second set of lists is for batches whose lists are small."""
    import ctypes as C

    from late_interaction_kernels_b200 import _lib

    lib = _lib.load()
    Q, D = torch.zeros(1, 32, 128, device="cuda").bfloat16(), torch.zeros(4000, 4, 128, device="cuda").bfloat16()
    a, t = topk_args(Q, D, None, 100, torch.empty(1, device="cuda"), torch.empty(1, dtype=torch.long, device="cuda"))
    a.q.n_seq, a.q.n_rows = 100_000, 3_200_000  # (only the size is asked for)
    assert lib.lik_maxsim_fwd_topk_workspace(C.byref(a), C.byref(t)) < 215e6


@pytest.mark.parametrize("large", [False, True])
@pytest.mark.parametrize("Nq", [2, 9, 40])
def test_topk_in_pieces_of_different_sizes(Nq, large):
    """Pieces of one document up to several super-blocks (their window is 48 MB) share one workspace and one kernel."""
    import ctypes as C

    from late_interaction_kernels_b200 import _lib

    lib = _lib.load()
    gen = torch.Generator(device="cuda").manual_seed(Nq)
    k, sizes = 29, [1500, 1, 700, 40]
    Nd, Ld = sum(sizes), 420  # 1500 x 420 x 256 bytes = 161 MB
    Q, D = ints(gen, Nq, 32, 128).bfloat16(), ints(gen, Nd, Ld, 128).bfloat16()
    mask = torch.arange(Ld, device="cuda")[None] < lengths(Nd, Ld, gen)[:, None]
    s, i = torch.empty(Nq, k, device="cuda"), torch.empty(Nq, k, dtype=torch.long, device="cuda")
    ws, base = None, 0
    for n, size in enumerate(sizes):
        flags = (_lib.TOPK_CONTINUE if n else 0) | (_lib.TOPK_PARTIAL if n + 1 < len(sizes) else 0) | (_lib.TOPK_LARGE if large else 0)
        m = mask[base:base + size].contiguous()
        a, t = topk_args(Q, D[base:base + size], m, k, s, i, flags, base)
        if ws is None:
            ws = torch.empty(lib.lik_maxsim_fwd_topk_workspace(C.byref(a), C.byref(t)), dtype=torch.uint8, device="cuda")
        a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
        _lib.check(lib.lik_maxsim_fwd_topk(C.byref(a), C.byref(t), _lib.stream_ptr(ws.device)), "lik_maxsim_fwd_topk")
        base += size
    want = torch.sort(reference(Q.float(), D.float(), mask)[0].sum(-1), dim=1, descending=True, stable=True)
    assert torch.equal(s, want.values[:, :k]) and torch.equal(i, want.indices[:, :k])


def route(Nq, Nd, Lq, Ld, *, masked=True, winners=False, k=0, group=0, n_pairs=0, queries=0, normalize=0, dtype=torch.bfloat16, scaled=False):
    """The kernel that a call goes to by itself (only its sizes are looked at)."""
    import ctypes as C

    from late_interaction_kernels_b200 import _lib

    lib = _lib.load()
    x = torch.zeros(16, device="cuda")

    def side(n, length):
        return _lib.Seqs(data=x.data_ptr(), row_stride=128, n_rows=n * length, n_seq=n, max_len=length, seq_stride=length, cu=None, lens=None, mask=None,
                         scale=x.data_ptr() if scaled else None, scale_scalar=1.0, reserved=0)

    q, d = side(Nq, Lq), side(Nd, Ld)
    if masked:
        d.lens = x.data_ptr()
    a = _lib.FwdArgs(
        q=q, d=d, dtype=_lib.lik_dtype(dtype), dim=128, pairing=_lib.PAIR_GROUPED if group else _lib.PAIR_LIST if n_pairs else _lib.PAIR_CROSS, group=group,
        pair_q=x.data_ptr(), pair_d=x.data_ptr(), n_pairs=n_pairs, normalize=normalize, engine=0, scores=x.data_ptr(),
        argmax=x.data_ptr() if winners else None, argmax_stride=Lq, reserved=0, workspace=None, workspace_bytes=0, status=None,
    )
    t = _lib.TopkSpec(k=k, largest=1, index_offset=0, out_scores=None, out_index=None, flags=0, doc_base=0)
    return lib.lik_maxsim_fwd_kernel(C.byref(a), C.byref(t) if k else None)


def test_which_kernel_takes_a_call():
    """Both sides of every line of the rule: units per SM, units per query tile, document lengths, full documents, merges."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert route(4, 12 * sms, 32, 64) == 2 and route(4, 12 * sms - 1, 32, 64) == 1
    assert route(4, 12 * sms, 32, 300) == 2 and route(4, 12 * sms - 1, 32, 300) == 1
    # more than 100 and up to 256 tokens: twice as much with one query tile
    assert route(1, 12 * sms, 32, 100) == 2 and route(1, 12 * sms, 32, 101) == 1 and route(1, 12 * sms, 32, 256) == 1
    assert route(1, 12 * sms, 32, 257) == 2 and route(1, 24 * sms, 32, 180) == 2 and route(8, 12 * sms, 32, 180) == 2
    # query tiles that change with every few documents
    many = 8 * 12 * sms
    assert route(many, 1, 32, 64) == 1 and route(many // 2, 2, 32, 64) == 2 and route(many // 3 + 8, 3, 32, 64) == 1 and route(many // 4, 4, 32, 64) == 2
    assert route(many, 1, 32, 300) == 1 and route(many // 7 + 8, 7, 32, 300) == 1 and route(many // 8, 8, 32, 300) == 2
    for group, at_64, at_180, at_300 in ((1, 2, 1, 1), (2, 2, 1, 2), (3, 2, 1, 1), (5, 2, 1, 1), (6, 2, 1, 2), (11, 2, 1, 2), (12, 2, 2, 2)):
        n = 24 * sms // group + 1
        assert [route(n, n * group, 32, ld, group=group, winners=True) for ld in (64, 180, 300)] == [at_64, at_180, at_300]
    assert route(64, 1000, 32, 300, n_pairs=32 * sms) == 2 and route(64, 1000, 32, 300, n_pairs=32 * sms - 1) == 1
    assert route(64, 1000, 32, 180, n_pairs=95 * sms) == 1 and route(64, 1000, 32, 180, n_pairs=96 * sms) == 2
    assert route(8 * sms, 1000, 32, 300, n_pairs=32 * sms) == 1  # four pairs per query
    # documents known to fill their last tile of 256
    assert route(64, 3 * sms, 32, 256, masked=False) == 1 and route(64, 3 * sms, 32, 256, masked=False, winners=True) == 2
    assert route(64, 3 * sms, 32, 256) == 2 and route(64, 3 * sms, 32, 300, masked=False) == 2
    # norms from the tiles, multipliers that arrive with the tiles
    assert route(4, 40 * sms, 32, 300, normalize=3) == 1 and route(72, 2 * sms, 32, 300, normalize=3) == 2
    assert route(4, 40 * sms, 32, 64, scaled=True, dtype=torch.float8_e4m3fn) == 1
    assert route(4, 40 * sms + 1, 32, 65, scaled=True, dtype=torch.float8_e4m3fn) == 2  # (the set stages them)
    # fused top-k: as everything else, and more where the lists need one more pass
    assert route(1, 12 * sms, 32, 300, k=10) == 2 and route(1, 12 * sms - 1, 32, 300, k=10) == 1
    assert route(40, 8 * sms, 32, 300, k=10) == 2 and route(40, 8 * sms - 1, 32, 300, k=10) == 1 and route(40, 100 * sms, 32, 1030, k=10) == 1
    assert route(80, 2 * sms, 32, 300, k=10) == 2 and route(100_000, 2 * sms, 32, 300, k=10) == 1


# documents of more than one piece and fewer than three, in the amounts from which they go to this kernel
@pytest.mark.parametrize("Nq,units,Lq,Ld,dtype,norm", [
    (1, 24, 32, 101, torch.bfloat16, False), (3, 24, 40, 192, torch.float16, False), (4, 25, 32, 256, torch.bfloat16, False), (8, 13, 31, 129, torch.float16, False),
])
def test_middling_documents(Nq, units, Lq, Ld, dtype, norm):
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200.forward import maxsim_forward

    Nd = units * torch.cuda.get_device_properties(0).multi_processor_count
    assert route(Nq, Nd, Lq, Ld, winners=True, dtype=dtype) == 2 and route(Nq, Nd, Lq, Ld, k=9, dtype=dtype) == 2
    gen = torch.Generator(device="cuda").manual_seed(Ld)
    Q, D = ints(gen, Nq, Lq, 128), ints(gen, Nd, Ld, 128)
    mask = torch.arange(Ld, device="cuda")[None] < lengths(Nd, Ld, gen)[:, None]
    val, pos = reference(Q, D, mask)
    scores, am = maxsim_forward(Q.to(dtype), D.to(dtype), None, mask, save_argmax=True)
    assert torch.equal(scores.view(Nq, Nd), val.sum(-1)) and torch.equal(am.view(Nq, Nd, Lq).long(), pos)
    ts, ti = lik.retrieve(Q.to(dtype), D.to(dtype), 9, d_mask=mask, normalize=False)
    order = torch.sort(val.sum(-1), dim=1, descending=True, stable=True)
    assert torch.equal(ts, order.values[:, :9]) and torch.equal(ti, order.indices[:, :9])


@pytest.mark.parametrize("holes", [False, True])
def test_multipliers_staged_with_one_query_tile(holes):
    """Per-token scales whose rows do not start on 16 bytes: the epilogue sets stage them, and a stream's two accumulators take
    turns.  1e-5 as for all fp32 sums of exact products."""
    from late_interaction_kernels_b200.fp8 import maxsim_inference_fp8, quantize_fp8_per_token

    Nq, Lq, Ld = 4, 32, 97
    Nd = 12 * torch.cuda.get_device_properties(0).multi_processor_count + 25
    assert route(Nq, Nd, Lq, Ld, scaled=True, dtype=torch.float8_e4m3fn) == 2
    gen = torch.Generator(device="cuda").manual_seed(97)
    Q, D = torch.randn(Nq, Lq, 128, generator=gen, device="cuda"), torch.randn(Nd, Ld, 128, generator=gen, device="cuda")
    mask = torch.arange(Ld, device="cuda")[None] < lengths(Nd, Ld, gen)[:, None]
    if holes:
        mask &= torch.rand(Nd, Ld, generator=gen, device="cuda") < 0.7
    (q8, sq), (d8, sd) = quantize_fp8_per_token(Q), quantize_fp8_per_token(D)
    want = reference(q8.double() * sq.double()[..., None], d8.double() * sd.double()[..., None], mask)[0].sum(-1)
    got = maxsim_inference_fp8(q8, d8, scale_Q=sq, scale_D=sd, d_mask=mask).double()
    assert (got - want).abs().max() <= 1e-5 * want.abs().max()


def test_infinities_and_nan_rows_as_in_the_other_kernel():
    """Rows of infinities and NaN in documents and queries: the first documents alone, which the other kernel takes, agree bit for
    bit (NaN with NaN), winners included."""
    from late_interaction_kernels_b200.forward import maxsim_forward

    gen = torch.Generator(device="cuda").manual_seed(3)
    Nq, Lq, Ld, few = 9, 32, 120, 40
    Nd = 12 * torch.cuda.get_device_properties(0).multi_processor_count
    assert route(Nq, Nd, Lq, Ld, winners=True, masked=False) == 2 and route(Nq, few, Lq, Ld, winners=True, masked=False) == 1
    Q, D = torch.randn(Nq, Lq, 128, generator=gen, device="cuda"), torch.randn(Nd, Ld, 128, generator=gen, device="cuda")
    for x, values in ((Q, (float("inf"), float("nan"))), (D, (float("inf"), float("-inf"), float("nan")))):
        hit = torch.rand(x.shape[:2], generator=gen, device="cuda")
        for n, v in enumerate(values):
            x[(hit > 0.02 * n) & (hit < 0.02 * n + 0.015)] = v
    D[3] = float("nan")
    D[5] = float("-inf")
    Q, D = Q.bfloat16(), D.bfloat16()
    s, am = maxsim_forward(Q, D, save_argmax=True)
    s1, am1 = maxsim_forward(Q, D[:few], save_argmax=True)
    assert torch.equal(s[:, :few].nan_to_num(7.0), s1.nan_to_num(7.0)) and torch.equal(s[:, :few].isnan(), s1.isnan())
    assert torch.equal(am.view(Nq, Nd, Lq)[:, :few], am1.view(Nq, few, Lq))


def test_rows_with_a_stride_wider_than_the_row():
    import ctypes as C

    from late_interaction_kernels_b200 import _lib, _ops

    lib = _lib.load()
    gen = torch.Generator(device="cuda").manual_seed(8)
    Nq, Lq, Ld, d, wide = 8, 32, 50, 128, 136
    Nd = 12 * torch.cuda.get_device_properties(0).multi_processor_count
    Q, big = ints(gen, Nq, Lq, d).bfloat16(), ints(gen, Nd * Ld, wide).bfloat16()
    out = torch.empty(Nq, Nd, device="cuda")
    q = _ops.padded_spec(Q).c_struct()
    dd = _lib.Seqs(data=big.data_ptr(), row_stride=wide, n_rows=Nd * Ld, n_seq=Nd, max_len=Ld, seq_stride=Ld, cu=None, lens=None, mask=None, scale=None,
                   scale_scalar=1.0, reserved=0)
    a = _lib.FwdArgs(
        q=q, d=dd, dtype=_lib.lik_dtype(Q.dtype), dim=d, pairing=_lib.PAIR_CROSS, group=0, pair_q=None, pair_d=None, n_pairs=0, normalize=_lib.NORM_NONE,
        engine=0, scores=out.data_ptr(), argmax=None, argmax_stride=Lq, reserved=0, workspace=None, workspace_bytes=0, status=None,
    )
    assert lib.lik_maxsim_fwd_kernel(C.byref(a), None) == 2
    _lib.check(lib.lik_maxsim_fwd_static(C.byref(a), _lib.stream_ptr(out.device)), "lik_maxsim_fwd_static")
    D = big[:, :d].float().view(Nd, Ld, d)
    want = reference(Q.float(), D, torch.ones(Nd, Ld, dtype=torch.bool, device="cuda"))[0].sum(-1)
    assert torch.equal(out, want)


def test_host_threads_with_different_shared_memory_sizes():
    """The limit of a kernel's shared memory is one per process: launches of other widths in other threads leave it alone."""
    import threading

    from late_interaction_kernels_b200.forward import maxsim_forward

    Nd = 12 * torch.cuda.get_device_properties(0).multi_processor_count
    gen = torch.Generator(device="cuda").manual_seed(1)
    sets, errors = [], []
    for d in (16, 32, 64, 80, 96, 128):  # one slab or two, deeper and shallower rings
        Q, D = ints(gen, 8, 32, d).bfloat16(), ints(gen, Nd, 40, d).bfloat16()
        sets.append((Q, D, maxsim_forward(Q, D)[0], maxsim_forward(Q, D[:20])[0]))

    def work(n):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(60):
                    Q, D, many, few = sets[(n + i) % len(sets)]
                    assert torch.equal(maxsim_forward(Q, D)[0], many) and torch.equal(maxsim_forward(Q, D[:20])[0], few)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(n,)) for n in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
