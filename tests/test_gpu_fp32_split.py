"""fp32 scores on the tensor cores (rows cut into three parts, a bound per product, dot products in fp32 where the bound is too wide) against
the fused multiply-add kernel (``engine=1``) and against 64 bits: at the edges of pieces and tiles, on rows whose features differ much in size, on
rows that the cut does not fit, where products tie, and on integers, where both kernels must be exact.

Bounds used: a product that is taken from the tensor cores is within max(4, d / 4) 2^-24 of itself, one taken in fp32 within 9 roundings of
sum |q_k d_k|; a score sums up to 128 of them.  For Gaussian rows that is below 2^-19 of a score, and what is seen is about 2^-24."""

import pytest
import torch

pytestmark = pytest.mark.gpu
PARTS = 3  # the kernel under test, also at sizes where the other one is faster


def _run(Q, D, engine, normalize=0, qm=None, dm=None, lens=None, cu=None, max_d=None):
    from late_interaction_kernels_b200 import _ops, check_device_status

    q = _ops.padded_spec(Q, mask=qm)
    d = _ops.packed_spec(D, cu, max_d) if cu is not None else _ops.padded_spec(D, mask=dm, lens=lens)
    s = _ops.forward(q, d, normalize=normalize, engine=engine or PARTS)[0].view(Q.shape[0], -1)
    check_device_status()
    return s


def _exact(Q, D, normalize, qm, dm):
    Q, D = Q.double(), D.double()
    if normalize:
        Q, D = torch.nn.functional.normalize(Q, dim=-1), torch.nn.functional.normalize(D, dim=-1)
    x = torch.einsum("isd,jtd->ijst", Q, D).masked_fill(~dm[None, :, None, :], -torch.inf).amax(-1)
    return x.masked_fill(x == -torch.inf, 0.0).masked_fill(~qm[:, None, :], 0.0).sum(-1)


def _masks(nq, lq, nd, ld, g):
    dl = torch.tensor(([0, 1, 15, 16, 17, 63, 64, 65, 127, 128, 129, ld] * nd)[:nd]).clamp(max=ld)
    dm = torch.arange(ld) < dl[:, None]
    holes = torch.rand((nd, ld), generator=g) > 0.2
    dm[nd // 2 :] &= holes[nd // 2 :]
    qm = torch.arange(lq) < torch.randint(0, lq + 1, (nq, 1), generator=g)
    return qm.cuda(), dm.cuda()


@pytest.mark.parametrize("nq,lq,nd,ld,d", [(1, 1, 1, 1, 4), (1, 128, 24, 200, 128), (9, 32, 24, 130, 128), (13, 24, 300, 70, 96), (5, 33, 24, 129, 100),
                                           (40, 5, 24, 65, 20), (3, 100, 24, 200, 12), (130, 1, 24, 64, 128)])
@pytest.mark.parametrize("normalize", [0, 3])
def test_scores_against_64_bits_and_the_chain(nq, lq, nd, ld, d, normalize):
    g = torch.Generator().manual_seed(nq * 7 + d)
    Q, D = torch.randn((nq, lq, d), generator=g).cuda(), (torch.randn((nd, ld, d), generator=g) * torch.rand((nd, ld, 1), generator=g)).cuda()
    qm, dm = _masks(nq, lq, nd, ld, g)
    a, b = _run(Q, D, 0, normalize, qm, dm), _run(Q, D, 1, normalize, qm, dm)
    e = _exact(Q, D, normalize, qm, dm)
    scale = e.abs().max().clamp(min=1e-30)
    err = ((a.double() - e).norm() / e.norm().clamp(min=1e-30)).item()
    assert ((a.double() - e).abs().max() / scale).item() < 2e-6 and ((b.double() - e).abs().max() / scale).item() < 2e-6
    assert err < 1e-6


@pytest.mark.parametrize("nq,lq,nd,ld,d", [(8, 4, 40, 180, 128), (17, 3, 20, 64, 64)])
def test_integers_are_exact(nq, lq, nd, ld, d):
    """Whole numbers of up to 16 bits: any product of parts that went missing shows.  A dot product is below 3 * 30000 * 128 and a
    score of four of them, for rows in random directions a third of that at most, below 2^24."""
    g = torch.Generator().manual_seed(5)
    Q = torch.randint(-3, 4, (nq, lq, d), generator=g).float().cuda()
    D = torch.randint(-30000, 30001, (nd, ld, d), generator=g).float().cuda()
    qm, dm = _masks(nq, lq, nd, ld, g)
    want = _exact(Q, D, 0, qm, dm)
    assert torch.equal(_run(Q, D, 0, 0, qm, dm).double(), want)
    assert torch.equal(_run(D[:nq, :lq].contiguous(), Q[:, :, :], 0).double(),
                       _exact(D[:nq, :lq], Q, 0, torch.ones(nq, min(lq, ld), dtype=torch.bool, device="cuda"), torch.ones(nq, lq, dtype=torch.bool, device="cuda")))


@pytest.mark.parametrize("nq,lq,nd,ld,d", [(5, 32, 40, 200, 128), (7, 20, 40, 130, 64), (2, 128, 40, 300, 32), (130, 1, 20, 65, 16)])
@pytest.mark.parametrize("extra", [0, 3])
def test_winners(nq, lq, nd, ld, d, extra):
    """Small whole numbers tie often: the first token wins, in the order of the two sets' pieces too; scores have the same bits with
    and without winners; places behind a query hold -1."""
    from late_interaction_kernels_b200 import _ops

    g = torch.Generator().manual_seed(11)
    Q, D = torch.randint(-1, 2, (nq, lq, d), generator=g).float().cuda(), torch.randint(-1, 2, (nd, ld, d), generator=g).float().cuda()
    qm, dm = _masks(nq, lq, nd, ld, g)
    got = [_ops.forward(_ops.padded_spec(Q, mask=qm), _ops.padded_spec(D, mask=dm), save_argmax=True, argmax_stride=lq + extra, engine=e) for e in (PARTS, 1)]
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert torch.equal(got[0][0].view(nq, nd), _run(Q, D, 0, 0, qm, dm))
    Q, D = torch.randn((nq, lq, d), generator=g).cuda(), torch.randn((nd, ld, d), generator=g).cuda()
    for n in (0, 3):
        a, _ = _ops.forward(_ops.padded_spec(Q, mask=qm), _ops.padded_spec(D, mask=dm), normalize=n, save_argmax=True, argmax_stride=lq + extra, engine=PARTS)
        assert torch.equal(a.view(nq, nd), _run(Q, D, 0, n, qm, dm))


def test_layouts():
    """Packed documents, lengths, row strides and offsets, and what stays with the other kernel (unaligned rows)."""
    g = torch.Generator().manual_seed(1)
    Q = torch.randn((6, 20, 64), generator=g).cuda()
    lens = torch.tensor([0, 64, 1, 200, 65, 0, 33, 128, 5, 0])
    cu = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)]).to(torch.int32).cuda()
    Dp = torch.randn((int(lens.sum()), 64), generator=g).cuda()
    a, b = _run(Q, Dp, 0, 3, cu=cu, max_d=200), _run(Q, Dp, 1, 3, cu=cu, max_d=200)
    assert torch.allclose(a, b, rtol=1e-5, atol=1e-5) and (a[:, lens == 0] == 0).all()
    D = torch.zeros((10, 200, 64), device="cuda")
    for j, n in enumerate(lens):
        D[j, :n] = Dp[cu[j] : cu[j + 1]]
    assert torch.equal(_run(Q, D, 0, 3, lens=lens.cuda()), a)
    from late_interaction_kernels_b200 import _ops

    wide = torch.randn((10 * 200, 80), device="cuda")
    wide[:, 4:68] = D.view(-1, 64)
    for lo in (4, 3):  # rows sixteen bytes apart from a boundary of sixteen bytes, and not
        wide[:, lo : lo + 64] = D.view(-1, 64).clone()
        spec = _ops.padded_spec(D, lens=lens.cuda())
        spec.data = wide[:, lo : lo + 64]
        s = _ops.forward(_ops.padded_spec(Q), spec, normalize=3, engine=PARTS)[0].view(6, 10)
        assert torch.allclose(s, a, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("where", ["document", "query", "both"])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 1e30, 3e38, 1e-30, 1e-42])
@pytest.mark.parametrize("normalize", [0, 3])
def test_rows_that_do_not_fit(where, value, normalize):
    """A piece or tile with such a row takes the chain: the same numbers as that kernel's, also infinities, NaN and subnormals."""
    g = torch.Generator().manual_seed(2)
    Q, D = torch.randn((5, 32, 128), generator=g).cuda(), torch.randn((12, 150, 128), generator=g).cuda()
    if where != "query":
        D[3, 70] = value if abs(value) < 1e-20 else D[3, 70]
        D[3, 70, 5] = value
        D[7, :] *= value if abs(value) < 1e20 else 1.0
    if where != "document":
        Q[1, 4] = value if abs(value) < 1e-20 else Q[1, 4]
        Q[1, 4, 9] = value
    a, b = _run(Q, D, 0, normalize), _run(Q, D, 1, normalize)
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
    ok = a.isfinite()
    assert torch.allclose(a[ok], b[ok], rtol=2e-6, atol=0 if normalize or abs(value) > 1e20 else 1e-5)
    if where != "document":  # the whole first tile (four queries) is taken by the chain
        assert torch.equal(a[:4].nan_to_num(1.5), b[:4].nan_to_num(1.5)) or torch.allclose(a[:4], b[:4], rtol=1e-6, equal_nan=True)


def test_what_masked_rows_hold_does_not_matter():
    """Padding of either side holds infinities and NaN: the scores are those with zeros there, bit for bit, with and without winners."""
    from late_interaction_kernels_b200 import _ops

    g = torch.Generator().manual_seed(8)
    Q, D = torch.randn((9, 32, 128), generator=g).cuda(), torch.randn((20, 100, 128), generator=g).cuda()
    qm, dm = _masks(9, 32, 20, 100, g)
    want = _run(Q * qm[..., None], D * dm[..., None], 0, 3, qm, dm)
    bad = torch.tensor([float("nan"), float("inf"), -float("inf"), 3e38], device="cuda").repeat(32)
    Qn, Dn = torch.where(qm[..., None], Q, bad), torch.where(dm[..., None], D, bad)
    assert torch.equal(_run(Qn, Dn, 0, 3, qm, dm), want)
    s, am = _ops.forward(_ops.padded_spec(Qn, mask=qm), _ops.padded_spec(Dn, mask=dm), normalize=3, save_argmax=True, argmax_stride=32, engine=PARTS)
    assert torch.equal(s.view(9, 20), want) and int(am.max()) < 100 and int(am.min()) >= -1


# Rows whose features differ much in size: bounds relative to the products' own magnitudes, sum |q_k d_k|.  A dot product of 128 features is at
# most 9 roundings deep, its two norms 10 each (halved by the root), the multipliers 6: 2^-24 * 25 with normalisation, below it without.
UNEVEN = 25 * 2.0**-24


def _uneven(nq, lq, nd, ld, d, ratio, form, g):
    """``form``: which side has features `ratio` times the others', where the other side's counterparts lie."""
    Q, D = torch.randn((nq, lq, d), generator=g), torch.randn((nd, ld, d), generator=g)
    if form == "documents, query 0 there":
        D[..., 3] *= ratio
        Q[..., 3] = 0
    elif form == "eight features of the queries":
        Q[..., 8:16] *= ratio
    elif form == "both, same feature":
        Q[..., 7] *= ratio
        D[..., 7] *= ratio
    elif form == "both, other features":
        Q[..., 7] *= ratio
        D[..., 70 % d] *= ratio
    elif form == "both, other side 0 there":
        Q[..., 7], D[..., 7] = Q[..., 7] * ratio, 0
        D[..., 70 % d], Q[..., 70 % d] = D[..., 70 % d] * ratio, 0
    elif form == "one feature counts":  # a query of one feature against a small one of the document
        Q[:] = 0
        Q[..., 1] = 1.0
        D[..., 0] *= ratio
    return Q.cuda(), D.cuda()


FORMS = ["documents, query 0 there", "eight features of the queries", "both, same feature", "both, other features", "both, other side 0 there", "one feature counts"]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("log_ratio", [2, 4, 7, 10, 13, 16, 20])
@pytest.mark.parametrize("normalize", [0, 3])
def test_uneven_features_keep_every_product(form, log_ratio, normalize):
    g = torch.Generator().manual_seed(log_ratio)
    Q, D = _uneven(150, 1, 160, 1, 128, 2.0**log_ratio, form, g)
    q, d = Q.double()[:, 0], D.double()[:, 0]
    if normalize:
        q, d = torch.nn.functional.normalize(q, dim=-1), torch.nn.functional.normalize(d, dim=-1)
    want, size = q @ d.T, q.abs() @ d.abs().T
    err = [((_run(Q, D, e, normalize).double() - want).abs() / size) for e in (0, 1)]
    assert err[0].max().item() < UNEVEN
    assert err[0].norm().item() <= 2 * err[1].norm().item()


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("log_ratio", [4, 10, 16])
@pytest.mark.parametrize("nq,lq,nd,ld,d", [(5, 32, 24, 300, 128), (3, 100, 24, 130, 96), (9, 24, 24, 64, 128)])
@pytest.mark.parametrize("normalize", [0, 3])
def test_uneven_features_scores_and_winners(form, log_ratio, nq, lq, nd, ld, d, normalize):
    from late_interaction_kernels_b200 import _ops

    g = torch.Generator().manual_seed(log_ratio + nq)
    Q, D = _uneven(nq, lq, nd, ld, d, 2.0**log_ratio, form, g)
    qm, dm = _masks(nq, lq, nd, ld, g)
    s, am = _ops.forward(_ops.padded_spec(Q, mask=qm), _ops.padded_spec(D, mask=dm), normalize=normalize, save_argmax=True, argmax_stride=lq, engine=PARTS)
    s, am = s.view(nq, nd), am.view(nq, nd, lq).long()
    assert torch.equal(s, _run(Q, D, 0, normalize, qm, dm))
    q, x = Q.double(), D.double()
    if normalize:
        q, x = torch.nn.functional.normalize(q, dim=-1), torch.nn.functional.normalize(x, dim=-1)
    p = torch.einsum("isd,jtd->ijst", q, x).masked_fill(~dm[None, :, None, :], -torch.inf)
    size = torch.einsum("isd,jtd->ijst", q.abs(), x.abs()).masked_fill(~dm[None, :, None, :], 0)
    full = dm.any(-1)[None, :, None].expand_as(am)
    assert (am[full] >= 0).all() and (am[~full] == -1).all()
    # the winner's own product is the largest but for what either may be off
    won, won_size = p.gather(3, am.clamp(min=0)[..., None])[..., 0], size.gather(3, am.clamp(min=0)[..., None])[..., 0]
    assert (p <= (won + UNEVEN * won_size)[..., None] + UNEVEN * size)[full].all()
    live = full & qm[:, None, :]
    want, bound = torch.where(live, won, 0).sum(-1), torch.where(live, won_size, 0).sum(-1) * (UNEVEN + 8 * 2.0**-24)  # (a sum of up to 128 on top)
    assert ((s.double() - want).abs() <= bound).all()
    e = [((t.double() - _exact(Q, D, normalize, qm, dm)) / (bound + 1e-300)).norm().item() for t in (s, _run(Q, D, 1, normalize, qm, dm))]
    assert e[0] <= 2 * e[1]


@pytest.mark.parametrize("what", ["repeated tokens", "signs", "zero queries", "zero documents", "scales"])
@pytest.mark.parametrize("normalize", [0, 3])
def test_products_that_tie(what, normalize):
    """More than one token may be the best, in one group of sixteen columns, in both sets' pieces, in the whole document: the products are whole numbers (or
    equal for equal rows), so the first of them wins, as in the other kernel."""
    from late_interaction_kernels_b200 import _ops

    g = torch.Generator().manual_seed(3)
    nq, lq, nd, ld, d = 6, 24, 24, 200, 64
    Q, D = torch.randint(-3, 4, (nq, lq, d), generator=g).float(), torch.randint(-3, 4, (nd, ld, d), generator=g).float()
    scale = None
    if what == "repeated tokens":
        D[:, 100:] = D[:, :100]
        D[:, 40:60] = D[:, 20:40]
        D[:8] = D[:8, :1]
    elif what == "signs":
        Q, D = torch.where(Q >= 0, 1.0, -1.0), torch.where(D >= 0, 1.0, -1.0)
    elif what == "zero queries":
        Q[:, ::3] = 0
    elif what == "zero documents":
        D[::2] = 0
        D[1::2, 5:150] = 0
    else:
        scale = torch.tensor([2.0, -1.0, 0.0, 0.5], dtype=torch.float32).repeat(nd * ld // 4).cuda()
    qm, dm = _masks(nq, lq, nd, ld, g)
    got = [_ops.forward(_ops.padded_spec(Q.cuda(), mask=qm), _ops.padded_spec(D.cuda(), mask=dm, scale=scale), normalize=normalize, save_argmax=True, argmax_stride=lq, engine=e)
           for e in (PARTS, 1)]
    if not normalize:
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    else:
        assert torch.allclose(got[0][0], got[1][0], rtol=1e-6, atol=1e-6)
        if what in ("zero queries", "repeated tokens"):  # equal rows have equal products; the first of them
            first = got[0][1].view(nq, nd, lq)
            assert (first[..., ::3][dm.any(-1)[None, :].expand(nq, nd)] == dm.float().argmax(-1)[None, :, None].expand(nq, nd, lq)[..., ::3][dm.any(-1)[None, :].expand(nq, nd)]).all() if what == "zero queries" else True


def test_a_row_that_does_not_fit_changes_nobody_else():
    """Infinities in one query, in one document: the scores of the others keep their bits."""
    g = torch.Generator().manual_seed(12)
    Q, D = torch.randn((9, 32, 128), generator=g).cuda(), torch.randn((20, 200, 128), generator=g).cuda()
    want = _run(Q, D, 0, 3)
    Q[1, 3, 5], D[7, 70, 9], D[8, 3] = float("inf"), float("nan"), 1e30
    s = _run(Q, D, 0, 3)
    others = torch.ones_like(s, dtype=torch.bool)
    others[1], others[:, 7], others[:, 8] = False, False, False
    assert torch.equal(s[others], want[others])


@pytest.mark.parametrize("nq,lq,nd,ld,d,parts", [(1, 32, 8, 16, 128, False), (1, 32, 1000, 512, 32, False), (16, 32, 100, 64, 32, False),
                                                 (1, 32, 1000, 512, 128, True), (1, 128, 8, 64, 128, True), (32, 32, 32, 180, 128, True)])
def test_the_faster_kernel_takes_a_call(nq, lq, nd, ld, d, parts):
    """The two kernels add in different orders: a call's bits say which one it went to."""
    from late_interaction_kernels_b200 import _ops

    g = torch.Generator().manual_seed(nq + d)
    Q, D = torch.randn((nq, lq, d), generator=g).cuda(), torch.randn((nd, ld, d), generator=g).cuda()
    auto = _ops.forward(_ops.padded_spec(Q), _ops.padded_spec(D), normalize=3)[0].view(nq, nd)
    fma, split = _run(Q, D, 1, 3), _run(Q, D, PARTS, 3)
    assert not torch.equal(fma, split) and torch.equal(auto, split if parts else fma)
