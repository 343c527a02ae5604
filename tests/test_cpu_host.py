"""CPU-side checks: the C-ABI library loads and exports everything ``include/lik_b200.h`` declares,
host-side validation raises the documented errors, and nothing falls back to the CPU."""

import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    from late_interaction_kernels_b200 import _build, _lib

    _build.build()
    return _lib.load()


def test_header_symbols_are_exported(lib):
    from late_interaction_kernels_b200 import _lib

    text = open(os.path.join(ROOT, "include", "lik_b200.h")).read()
    declared = set(re.findall(r"\b(lik_[a-z0-9_]+)\s*\(", text))
    assert declared, "no declarations found"
    for sym in declared:
        assert hasattr(lib, sym), f"{sym} declared in the header but not exported"
    assert declared == set(_lib.EXPORTED_SYMBOLS)
    assert lib.lik_version() >= 200


def test_struct_sizes_match_the_header_layout():
    import ctypes as C

    from late_interaction_kernels_b200 import _lib

    assert C.sizeof(_lib.Seqs) == 80
    assert C.sizeof(_lib.FwdArgs) == 2 * 80 + 96
    assert C.sizeof(_lib.PlaidIndex) == 56
    assert C.sizeof(_lib.TopkSpec) == 40
    assert C.sizeof(_lib.HiddenFwdArgs) == 2 * 80 + 88


def test_argument_validation_without_a_gpu(lib):
    import ctypes as C

    from late_interaction_kernels_b200 import _lib

    a = _lib.FwdArgs()
    a.dim = 0
    assert lib.lik_maxsim_fwd(C.byref(a), None) == -1
    assert b"dim" in lib.lik_last_error()
    assert lib.lik_maxsim_fwd(None, None) == -1
    assert lib.lik_topk_rows(None, 1, 1, 1, 0, 1, 0, 0, None, None, None) == -1
    ix = _lib.PlaidIndex()
    ix.nbits = 3
    assert lib.lik_plaid_decompress(C.byref(ix), 0, 0, 1, None, 2, None, None) == -1
    assert b"nbits must be 2, 4, or 8" in lib.lik_last_error()
    # document head: NULL arguments and bad sizes are refused before any CUDA call; without a GPU nothing is supported
    assert lib.lik_maxsim_hidden_fwd(None, None) == -1
    h = _lib.HiddenFwdArgs()
    assert lib.lik_maxsim_hidden_fwd(C.byref(h), None) == -1
    assert b"must not be NULL" in lib.lik_last_error()
    assert lib.lik_maxsim_hidden_fwd_supported(C.byref(h)) == 0
    assert lib.lik_maxsim_hidden_fwd_workspace(C.byref(h)) == 0
    assert lib.lik_hidden_winners(None, 1, 1, 0, 1, 1, None, None, None, None, None, None, None) == -1
    assert lib.lik_hidden_winners(None, 1, 0, 4, 8, 4, None, None, None, None, None, None, None) == 0  # no documents: nothing to do
    assert lib.lik_hidden_scatter_rows(None, 24, 1, 8, 4, None, None, None, None) == -1


def test_no_cpu_fallback_anywhere():
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200 import fp8, plaid
    from late_interaction_kernels_b200.backward import maxsim_backward_lowmem, maxsim_backward_unified
    from late_interaction_kernels_b200.score_pairs import score_pairs_packed

    Q, D = torch.randn(2, 3, 16), torch.randn(2, 4, 16)
    cu = torch.tensor([0, 3, 6], dtype=torch.int32)
    for fn in (
        lambda: lik.maxsim(Q, D),
        lambda: lik.maxsim_pairs(Q, D),
        lambda: lik.maxsim_varlen(Q.view(-1, 16), D.view(-1, 16), cu, torch.tensor([0, 4, 8], dtype=torch.int32)),
        lambda: lik.maxsim_padded(Q, D[:, None], torch.tensor([3, 3]), torch.tensor([[4], [4]])),
        lambda: lik.retrieve(Q, D, 1),
        lambda: lik.MaxSimScorer()(Q, D),
        lambda: score_pairs_packed(Q.view(-1, 16), D.view(-1, 16), cu, cu, torch.tensor([0]), torch.tensor([1])),
        lambda: maxsim_backward_unified(torch.zeros(2, 2), Q, D, torch.zeros(4, 3, dtype=torch.int32)),
        lambda: maxsim_backward_lowmem(torch.zeros(2, 2), Q, D, torch.zeros(4, 3, dtype=torch.int32)),
        lambda: plaid.plaid_approx_score(torch.randn(4, 3), torch.zeros(2, 5, dtype=torch.int32), torch.tensor([1, 2])),
    ):
        with pytest.raises(RuntimeError, match="CUDA"):
            fn()
    with pytest.raises(ValueError, match="float8_e4m3fn"):
        fp8.maxsim_inference_fp8(Q, D, scale_Q=torch.ones(()), scale_D=torch.ones(()))


def test_host_validation_messages():
    import late_interaction_kernels_b200 as lik
    from late_interaction_kernels_b200 import plaid
    from late_interaction_kernels_b200.padded import pack_padded

    Q, D = torch.randn(2, 3, 16), torch.randn(2, 4, 16)
    with pytest.raises(ValueError, match="backward= must be one of"):
        lik.maxsim(Q, D, backward="nope")
    with pytest.raises(ValueError, match="backward= must be one of"):
        lik.MaxSimScorer(backward="nope")
    with pytest.raises(ValueError, match="top_k must be positive"):
        lik.retrieve(Q, D, 0)
    with pytest.raises(ValueError, match="mask_pad_token"):
        lik.MaxSimScorer().forward_with_ids(Q, D, None, None)
    with pytest.raises(ValueError, match="2-D"):
        lik.maxsim_varlen(Q, D, None, None)
    with pytest.raises(ValueError, match="nbits must be 2, 4, or 8"):
        plaid.maxsim_residual_varlen(Q, None, None, None, None, None, 3)
    with pytest.raises(ValueError, match=r"queries must be \[B, Lq, d\]"):
        pack_padded(Q[0], D[:, None], torch.tensor([3]), torch.tensor([[4]]))
    with pytest.raises(ValueError, match="doc_lengths must be"):
        pack_padded(Q, D[:, None], torch.tensor([3, 3]), torch.tensor([4, 4]))


def test_loss_head_helpers_validate_on_the_host():
    from late_interaction_kernels_b200.loss_heads import maxsim_pos_neg, maxsim_tiles

    q, d = torch.randn(2, 3, 16), torch.randn(2, 4, 16)
    with pytest.raises(ValueError, match="at least one"):
        maxsim_tiles([], [d])
    with pytest.raises(ValueError, match="same d"):
        maxsim_tiles([q], [torch.randn(2, 4, 8)])
    with pytest.raises(ValueError, match="one mask"):
        maxsim_tiles([q, q], [d], q_masks=[None])
    with pytest.raises(RuntimeError, match="CUDA"):
        maxsim_tiles([q], [d])  # host tensors: no CPU path
    with pytest.raises(ValueError, match="expected Q"):
        maxsim_pos_neg(q, d, d)


def test_pack_padded_on_cpu_matches_reference_golden():
    """pack_padded is pure host/torch logic, so it also runs on CPU tensors."""
    import numpy as np
    from conftest import load_golden

    import cases
    from late_interaction_kernels_b200.padded import pack_padded

    g = load_golden("padded")
    q, docs, ql, dl = cases.padded_case(8)
    pk = pack_padded(torch.tensor(q), torch.tensor(docs), torch.tensor(ql), torch.tensor(dl))
    Qp, cq, Dp, cd, pq, pd, mq, md = pk
    for a, k in ((Qp, "Q_packed"), (cq, "cu_q"), (Dp, "D_packed"), (cd, "cu_d"), (pq, "pair_q"), (pd, "pair_d")):
        assert np.array_equal(a.numpy(), g[k]), k
    assert (mq, md) == (int(g["max_q"]), int(g["max_d"]))
    with pytest.raises(ValueError, match="> 0"):
        pack_padded(torch.tensor(q), torch.tensor(docs), torch.tensor(ql * 0), torch.tensor(dl), validate=True)
    with pytest.raises(ValueError, match="exceeds the padded extent"):
        pack_padded(torch.tensor(q), torch.tensor(docs), torch.tensor(ql + 100), torch.tensor(dl), validate=True)
    e = pack_padded(torch.zeros(0, 8, 16), torch.zeros(0, 4, 13, 16), torch.zeros(0, dtype=torch.long), torch.zeros(0, 4, dtype=torch.long))
    assert e.Q_packed.shape == (0, 16) and e.max_seqlen_q == 0 and e.cu_seqlens_d.tolist() == [0]


def test_fp8_quantisers_on_cpu_match_reference_golden():
    import numpy as np
    from conftest import load_golden

    from late_interaction_kernels_b200 import fp8

    g = load_golden("fp8")
    rng = np.random.default_rng(9)
    X = (rng.standard_normal((5, 7, 32)) * np.array([1e-3, 0.1, 1, 10, 300]).reshape(5, 1, 1)).astype(np.float32)
    X[0, 0] = 0.0
    xq, sc = fp8.quantize_fp8_per_token(torch.tensor(X))
    assert np.array_equal(xq.float().numpy(), g["q_tok"]) and np.array_equal(sc.numpy(), g["s_tok"])
    assert np.array_equal(fp8.dequantize_fp8_per_token(xq, sc).numpy(), g["deq_tok"])
    xq2, sc2 = fp8.quantize_fp8_per_tensor(torch.tensor(X))
    assert np.array_equal(xq2.float().numpy(), g["q_ten"]) and np.array_equal(sc2.numpy(), g["s_ten"])


def test_reference_package_name_resolves_to_this_build():
    import importlib

    import late_interaction_kernels as alias
    import late_interaction_kernels_b200 as impl

    assert alias.maxsim is impl.maxsim and alias.MaxSimScorer is impl.MaxSimScorer and callable(alias.retrieve)
    assert importlib.import_module("late_interaction_kernels.plaid").maxsim_residual is impl.plaid.maxsim_residual
    assert importlib.import_module("late_interaction_kernels.retrieve").retrieve is impl.retrieve
    from late_interaction_kernels.backward.lowmem import maxsim_backward_lowmem  # noqa: F401


@pytest.mark.parametrize("per_token_q,per_token_d,kd", [(False, False, False), (True, False, False), (False, True, True), (True, True, True)])
def test_fp8_scales_reach_the_kernel_on_the_inputs_device(monkeypatch, per_token_q, per_token_d, kd):
    """Scales read from a checkpoint are host tensors; what the native call gets must sit where the embeddings are."""
    from late_interaction_kernels_b200 import _lib, fp8

    got = {}

    class Host:
        @staticmethod
        def maxsim_fp8(Q, D, scale_Q, scale_D, q_mask, d_mask, group):
            got.update(q=scale_Q, d=scale_D)
            return torch.empty((Q.shape[0], group or D.shape[0]), device=Q.device)

    monkeypatch.setattr(_lib, "host", lambda: Host)
    monkeypatch.setattr(_lib, "require_cuda", lambda *a, **k: None)
    e4m3 = torch.float8_e4m3fn
    Q = torch.empty((2, 3, 16), dtype=e4m3, device="meta")  # stands in for a GPU: any device that is not the host
    D = torch.empty((2, 5, 4, 16) if kd else (5, 4, 16), dtype=e4m3, device="meta")
    sq = torch.ones((2, 3), dtype=torch.float64) if per_token_q else torch.tensor(0.5)
    sd = torch.ones(D.shape[:-1], dtype=torch.float64) if per_token_d else torch.tensor(0.25)
    fp8.maxsim_inference_fp8(Q, D, scale_Q=sq, scale_D=sd)
    for t in got.values():
        assert t is None or (t.device == Q.device and t.dtype == torch.float32)
    assert any(t is not None for t in got.values())


def test_native_entries_refuse_tensors_of_another_device(lib):
    """Addresses go to a kernel as they are: a tensor that is not where the queries are is refused on the host, before
    anything touches a GPU."""
    from late_interaction_kernels_b200 import _lib

    host = _lib.host()
    here, there = torch.device("meta"), torch.device("cpu")  # two devices that a machine without a GPU has
    e = lambda *shape, dev=here, dtype=torch.bfloat16: torch.zeros(shape, dtype=dtype, device=dev)
    Q, D, qm, dm = e(2, 3, 16), e(4, 5, 16), e(2, 3, dtype=torch.bool), e(4, 5, dtype=torch.bool)
    Qp, Dp, cu = e(6, 16), e(8, 16), torch.tensor([0, 3, 6], dtype=torch.int32)
    ql, dl = e(2, dtype=torch.int32), e(4, dtype=torch.int32)
    Q8, D8 = e(2, 3, 16, dtype=torch.float8_e4m3fn), e(4, 5, 16, dtype=torch.float8_e4m3fn)
    sq, sd = e(2, 3, dtype=torch.float32), e(4, 5, dtype=torch.float32)
    H, W, b = e(4, 5, 32), e(16, 32), e(16)
    calls = [
        (host.maxsim_padded, [Q, e(2, 2, 5, 16), ql, dl], [1, 2, 3]),
        (host.maxsim_packed, [Qp, Dp, cu, cu, None, None, 3, 3], [1]),
        (host.maxsim_fp8, [Q8, D8, sq, sd, qm, dm, 0], [1, 2, 3, 4, 5]),
        (host.topk, [Q, D, 2, qm, dm, False, True], [1, 3, 4]),
        (host.maxsim_from_hidden, [Q, H, W, b, dm, True], [1, 2, 3, 4]),
    ]
    for fn, args, movable in calls:
        for i in movable:
            bad = list(args)
            bad[i] = torch.zeros(args[i].shape, dtype=args[i].dtype, device=there)
            with pytest.raises(ValueError, match="same device"):
                fn(*bad)


@pytest.mark.parametrize("save_argmax", [False, True])
def test_varlen_forward_finds_the_longest_lengths(monkeypatch, save_argmax):
    from late_interaction_kernels_b200 import _lib, _ops, varlen

    monkeypatch.setattr(_lib, "require_cuda", lambda *a, **k: None)
    monkeypatch.setattr(_ops, "forward", lambda q, d, **k: (torch.zeros(q.n_seq * d.n_seq), None))
    cu_q, cu_d = torch.tensor([0, 2, 6], dtype=torch.int32), torch.tensor([0, 1, 1, 9], dtype=torch.int32)
    s, _, max_q, max_d = varlen._varlen_forward(torch.zeros(6, 8), torch.zeros(9, 8), cu_q, cu_d, None, None, save_argmax)
    assert s.shape == (2, 3) and max_q == 4 and max_d == (8 if save_argmax else 0)


@pytest.mark.parametrize("max_len", [300, 10_239, 10_241, 24_000])
@pytest.mark.parametrize("pairing,n_q,n_d", [("cross", 4, 64), ("cross", 64, 8), ("cross", 600, 2), ("list", 8, 10)])
def test_long_documents_keep_the_sorted_backward(lib, pairing, n_q, n_d, max_len):
    """The winners of a document are sorted in shared memory up to about 25 000 tokens.  Beyond that a pair list scatters with
    atomics, in no fixed order, into fp32 buffers of the gradients' size; the sort's lists grow with the winners alone."""
    import ctypes as C

    from late_interaction_kernels_b200 import _lib

    def workspace(dim):
        a = _lib.BwdArgs()
        for side, n in ((a.q, n_q), (a.d, n_d)):
            side.n_seq, side.row_stride = n, dim
        a.q.max_len = a.q.seq_stride = 32
        a.d.max_len = a.d.seq_stride = max_len
        a.q.n_rows, a.d.n_rows = n_q * 32, n_d * max_len
        a.dtype = a.grad_dtype = _lib.LIK_BF16
        a.dim, a.argmax_stride, a.deterministic = dim, 32, 1
        a.grad_d = 1 << 20  # (an address that is never read: the plan looks at its alignment)
        a.pairing = _lib.PAIR_LIST if pairing == "list" else _lib.PAIR_CROSS
        a.n_pairs = 30 if pairing == "list" else 0
        return lib.lik_maxsim_bwd_workspace(C.byref(a))

    entries = (30 if pairing == "list" else n_q * n_d) * 32
    assert workspace(64) == workspace(128)
    if n_q * 32 > 4096 or max_len > 1536 or pairing == "list":  # (smaller problems sort in the one-launch kernel)
        assert workspace(64) >= entries * 8 + n_d * max_len * 12


@pytest.mark.skipif(torch.cuda.is_available(), reason="looks at what happens before the first launch")
def test_more_pairs_than_a_grid_has_blocks_are_not_refused(lib):
    """The portable forward launches 2**30 blocks at a time.  (On the GPU 65 536 x 65 537 one-token pairs, 17 GB of scores
    in three launches, take half a minute: too long for the suite.)  Without a GPU it is the launch that fails."""
    import ctypes as C

    from late_interaction_kernels_b200 import _lib

    a = _lib.FwdArgs()
    for side, n in ((a.q, 65536), (a.d, 65537)):
        side.data, side.row_stride, side.n_rows, side.n_seq, side.max_len, side.seq_stride = 1 << 20, 4, n, n, 1, 1
    a.dtype, a.dim, a.engine, a.scores = _lib.LIK_F32, 4, 1, 1 << 20
    assert lib.lik_maxsim_fwd(C.byref(a), None) != 0
    assert b"too many" not in lib.lik_last_error(), lib.lik_last_error()


@pytest.mark.skipif(torch.cuda.is_available(), reason="looks at what happens before the first launch")
@pytest.mark.parametrize("entry", ["lik_maxsim_fwd", "lik_maxsim_fwd_static"])
def test_trimmed_lengths_are_not_demanded_of_a_workspace(lib, entry):
    """Five million masked one-token documents need no scratch at all; room for their trimmed lengths (20 MB) is asked for
    but not insisted on.  Without a GPU it is the launch that fails."""
    import ctypes as C

    from late_interaction_kernels_b200 import _lib

    a = _lib.FwdArgs()
    for side, n in ((a.q, 1), (a.d, 5_000_000)):
        side.data, side.row_stride, side.n_rows, side.n_seq, side.max_len, side.seq_stride = 1 << 20, 4, n, n, 1, 1
    a.d.mask = 1 << 20
    a.dtype, a.dim, a.engine, a.scores = _lib.LIK_F32, 4, 1, 1 << 20
    assert lib.lik_maxsim_fwd_workspace(C.byref(a)) >= 20_000_000
    assert getattr(lib, entry)(C.byref(a), None) != 0
    assert b"workspace" not in lib.lik_last_error() and b"scratch" not in lib.lik_last_error(), lib.lik_last_error()


def test_host_path_of_another_torch_is_stale(lib, monkeypatch):
    """The native host path is bound to torch's class layouts: after an upgrade in place it is rebuilt, sources unchanged."""
    from late_interaction_kernels_b200 import _build, _lib

    assert _lib.host().abi == _build._host_abi() and _build._host_fits(_build.HOST_PATH)
    monkeypatch.setattr(_build, "_host_abi", lambda: "host path for torch 99.0, cpython-99")
    assert not _build._host_fits(_build.HOST_PATH)
    ran = []
    monkeypatch.setattr(_build, "_run", lambda cmd, what: ran.append(what) or "")
    monkeypatch.setattr(_build.os, "replace", lambda a, b: None)
    _build.build()
    assert sorted(w.split()[0] for w in ran) == ["compiling"] * len(_build._host_sources()) + ["linking"]
