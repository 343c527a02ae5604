"""Scores and top-k of a few queries decoded inside the scoring kernel, at the places where its tiles, tables and lists end:
compared bit for bit with decoding to memory first and scoring the rows (whose own tests compare with the CPU oracle)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _index(lens, d, nbits, cdtype, seed=0, ncent=64):
    g = torch.Generator().manual_seed(seed)
    T = int(sum(lens))
    codes = torch.randint(0, ncent, (T,), generator=g, dtype=torch.int32).cuda()
    res = torch.randint(0, 256, (T, d * nbits // 8), generator=g, dtype=torch.uint8).cuda()
    cent = torch.nn.functional.normalize(torch.randn((ncent, d), generator=g), dim=-1).cuda().to(cdtype)
    bw = torch.linspace(-0.1, 0.1, 2**nbits).cuda()
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32).cuda()
    return codes, res, cu, cent, bw


def _both(monkeypatch, call):
    from late_interaction_kernels_b200 import check_device_status, plaid

    monkeypatch.setattr(plaid, "_decode_in_kernel", lambda *a: True)  # (the rule takes some of these sizes elsewhere)
    got = call()
    check_device_status()
    monkeypatch.setattr(plaid, "_decode_in_kernel", lambda *a: False)
    want = call()
    monkeypatch.undo()
    return got, want


LENS = {
    "tile edges": [127, 128, 129, 1, 7, 8, 9, 255, 256, 257, 120, 121, 900, 3] * 9,
    "single tokens": [1] * 5000,  # sixteen documents per tile
    "empty ones": [0] * 700 + [5] + [0] * 130 + [200, 0, 0, 64] * 40 + [0] * 70,  # more segments than a table holds
    "one document": [333],
    "fewer than CTAs": [40, 0, 300],
}


@pytest.mark.parametrize("name", LENS)
@pytest.mark.parametrize("nq,lq", [(1, 32), (4, 32), (1, 5), (5, 24), (128, 1), (1, 128), (3, 33)])
def test_scores_at_edges_of_tiles_and_tables(name, nq, lq, monkeypatch):
    from late_interaction_kernels_b200 import plaid

    ix = _index(LENS[name], 128, 2, torch.float16)
    Q = torch.randn((nq, lq, 128), generator=torch.Generator().manual_seed(nq)).cuda().to(torch.bfloat16)
    got, want = _both(monkeypatch, lambda: plaid.maxsim_residual_varlen(Q, *ix, 2))
    assert torch.equal(got, want)


@pytest.mark.parametrize("nbits", [2, 4, 8])
@pytest.mark.parametrize("d,cdtype", [(16, torch.float16), (48, torch.float32), (64, torch.bfloat16), (80, torch.float16), (112, torch.float32), (128, torch.bfloat16), (128, torch.float32)])
def test_widths_code_widths_and_centroid_types(nbits, d, cdtype, monkeypatch):
    from late_interaction_kernels_b200 import plaid

    ix = _index([0, 1, 130, 64, 77, 300] * 60, d, nbits, cdtype, seed=d + nbits)
    for nq, qdtype, normalize in ((2, torch.float16, True), (1, torch.bfloat16, False)):
        Q = torch.randn((nq, 32, d), generator=torch.Generator().manual_seed(d)).cuda().to(qdtype)
        got, want = _both(monkeypatch, lambda: plaid.maxsim_residual_varlen(Q, *ix, nbits, normalize=normalize))
        assert torch.equal(got, want)
        # padded layout: lengths instead of offsets
        n, width = 50, 90
        codes, res = ix[0][: n * width].view(n, width), ix[1][: n * width].view(n, width, -1)
        lens = torch.arange(n, device="cuda") * 2 % (width + 1)
        got, want = _both(monkeypatch, lambda: plaid.maxsim_residual(Q, codes, res, lens, ix[3], ix[4], nbits, normalize=normalize))
        assert torch.equal(got, want)


@pytest.mark.parametrize("nq,lq,k", [(1, 32, 10), (4, 32, 128), (5, 24, 100), (1, 32, 1), (100, 1, 7)])
@pytest.mark.parametrize("order", ["rising", "falling", "equal"])
def test_candidate_lists_that_fill_up(nq, lq, k, order, monkeypatch):
    """Scores that rise with the document enter a list every time, so that it is cut back again and again; equal scores
    must keep the lowest documents."""
    from late_interaction_kernels_b200 import plaid

    nd, d = 60000, 128
    lens = [2 if j % 3 else 3 for j in range(nd)]
    T = sum(lens)
    # one centroid per step along the query's direction; residuals add nothing (all weights are zero)
    ncent = 2048
    doc = torch.repeat_interleave(torch.arange(nd), torch.tensor(lens))
    step = doc * (ncent - 1) // nd if order == "rising" else (nd - 1 - doc) * (ncent - 1) // nd if order == "falling" else torch.zeros_like(doc)
    cent = torch.zeros((ncent, d))
    cent[:, 0] = torch.arange(ncent) / 2048.0
    ix = (step.to(torch.int32).cuda(), torch.zeros((T, 32), dtype=torch.uint8).cuda(),
          torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32).cuda(), cent.cuda().to(torch.float16), torch.zeros(4).cuda())
    Q = torch.zeros((nq, lq, d))
    Q[..., 0] = 1.0
    Q = Q.cuda().to(torch.float16)
    for largest in (True, False):
        got, want = _both(monkeypatch, lambda: plaid.retrieve_residual_varlen(Q, *ix, 2, k, normalize=False, largest=largest))
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_codes_out_of_range_are_reported():
    from late_interaction_kernels_b200 import check_device_status, plaid

    codes, res, cu, cent, bw = _index([64] * 20, 128, 2, torch.float16)
    codes[100], codes[700] = -3, 64
    Q = torch.randn((1, 32, 128)).cuda().to(torch.float16)
    s = plaid.maxsim_residual_varlen(Q, codes, res, cu, cent, bw, 2)
    with pytest.raises(RuntimeError, match="centroid"):
        check_device_status()
    codes[100], codes[700] = 0, 0
    assert torch.equal(s, plaid.maxsim_residual_varlen(Q, codes, res, cu, cent, bw, 2))


def test_the_knob_says_which_way_a_call_goes(monkeypatch):
    """Decoding to memory is a launch of its own, so a call's launches tell; both ways give the same bits."""
    from late_interaction_kernels_b200 import _lib, plaid

    lib, ix = _lib.load(), _index([100, 30, 64] * 40, 128, 2, torch.float16)
    Q = torch.randn((2, 32, 128)).cuda().to(torch.float16)
    seen = {}
    for knob in (None, 1 << 30, 0):
        monkeypatch.setattr(plaid, "_FUSED_DECODE_MAX_GROUPS", knob)
        n0 = lib.lik_launch_count()
        s = plaid.maxsim_residual_varlen(Q, *ix, 2)
        t = plaid.retrieve_residual_varlen(Q, *ix, 2, 5)
        seen[knob] = (lib.lik_launch_count() - n0, s, *t)
    assert seen[None][0] == seen[1 << 30][0] < seen[0][0]
    assert all(torch.equal(a, b) for k in (None, 1 << 30) for a, b in zip(seen[k][1:], seen[0][1:]))


@pytest.mark.parametrize("nbits", [2, 4, 8])
@pytest.mark.parametrize("cdtype", [torch.float16, torch.bfloat16, torch.float32])
def test_infinities_and_nan_in_the_index(nbits, cdtype, monkeypatch):
    """Centroids and weights that are no numbers: what they do to a token stays with its document, and both ways agree bit for bit."""
    from late_interaction_kernels_b200 import plaid

    codes, res, cu, cent, bw = _index([30, 1, 0, 129, 64, 7] * 30, 128, nbits, cdtype, seed=nbits)
    Q = torch.randn((3, 32, 128), generator=torch.Generator().manual_seed(1)).cuda().to(torch.float16)
    for normalize in (True, False):
        for what in ("centroids", "weight"):
            c, w = cent.clone(), bw.clone()
            if what == "centroids":
                c[3, 5], c[9], c[20, ::2] = float("inf"), float("nan"), -float("inf")
            else:
                w[1] = float("inf")
            got, want = _both(monkeypatch, lambda: plaid.maxsim_residual_varlen(Q, codes, res, cu, c, w, nbits, normalize=normalize))
            assert torch.equal(got.nan_to_num(1.5, 2.5, 3.5), want.nan_to_num(1.5, 2.5, 3.5))
            got, want = _both(monkeypatch, lambda: plaid.retrieve_residual_varlen(Q, codes, res, cu, c, w, nbits, 20, normalize=normalize))
            assert torch.equal(got[0].nan_to_num(1.5, 2.5, 3.5), want[0].nan_to_num(1.5, 2.5, 3.5)) and torch.equal(got[1], want[1])


def test_two_streams_at_once(monkeypatch):
    """Calls of this kernel, of the one for fp32 rows and of the others beside each other: each allocates tensor memory on the same SMs."""
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200 import plaid

    monkeypatch.setattr(plaid, "_decode_in_kernel", lambda *a: True)
    g = torch.Generator().manual_seed(4)
    ix = _index([60, 200, 300] * 300, 128, 2, torch.float16)
    Q = torch.randn((2, 32, 128), generator=g).cuda().to(torch.float16)
    Qf, Df = torch.randn((32, 32, 128), generator=g).cuda(), torch.randn((40, 180, 128), generator=g).cuda()
    Qh, Dh = Qf.half(), Df.half()
    calls = [lambda: plaid.maxsim_residual_varlen(Q, *ix, 2), lambda: lik.maxsim(Qf, Df), lambda: lik.maxsim(Qh, Dh), lambda: plaid.retrieve_residual_varlen(Q, *ix, 2, 10)[0]]
    want = [f() for f in calls]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(3)]
    out = []
    for r in range(12):
        for n, s in enumerate(streams):
            with torch.cuda.stream(s):
                out.append(((r + n) % 4, calls[(r + n) % 4]()))
    torch.cuda.synchronize()
    assert all(torch.equal(x, want[k]) for k, x in out)
