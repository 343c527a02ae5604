"""CPU checks of the PLAID front stage's host logic: the fast-plaid file reader and the inverted file."""

import json
import os

import numpy as np
import torch

import cases
from oracle import maxsim_oracle as O


def write_fastplaid_files(path, codes, residuals, lens, centroids, buckets, nbits, *, merged, pad_rows=0, chunks=2):
    """Files in the layout the reference's benchmark reads (benchmarks/plaid/bench_fastplaid_e2e.py:76-140)."""
    os.makedirs(path, exist_ok=True)
    with open(os.path.join(path, "metadata.json"), "w") as f:
        json.dump({"nbits": nbits, "num_chunks": chunks}, f)
    np.save(os.path.join(path, "centroids.npy"), centroids)
    np.save(os.path.join(path, "bucket_weights.npy"), buckets)
    bounds = np.linspace(0, len(lens), chunks + 1).astype(int)
    cu = np.concatenate([[0], np.cumsum(lens)])
    for c in range(chunks):
        with open(os.path.join(path, f"doclens.{c}.json"), "w") as f:
            json.dump([int(x) for x in lens[bounds[c]:bounds[c + 1]]], f)
        if not merged:
            a, b = cu[bounds[c]], cu[bounds[c + 1]]
            np.save(os.path.join(path, f"codes.{c}.npy"), codes[a:b].astype(np.int64))
            np.save(os.path.join(path, f"residuals.{c}.npy"), residuals[a:b])
    if merged:
        pad_c = np.concatenate([codes, np.zeros(pad_rows, codes.dtype)]).astype(np.int64)
        pad_r = np.concatenate([residuals, np.zeros((pad_rows, residuals.shape[1]), np.uint8)])
        np.save(os.path.join(path, "merged_codes.npy"), pad_c)
        np.save(os.path.join(path, "merged_residuals.npy"), pad_r.reshape(-1))  # stored flat, as fast-plaid may


def small_index(seed=3, nd=40, d=32, nbits=2, ncent=16, max_len=12):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, max_len + 1, size=nd)
    T = int(lens.sum())
    codes = rng.integers(0, ncent, size=T).astype(np.int32)
    res = rng.integers(0, 256, size=(T, d * nbits // 8)).astype(np.uint8)
    cent = cases.unit(rng.standard_normal((ncent, d))).astype(np.float16)
    bw = np.linspace(-0.1, 0.1, 2**nbits).astype(np.float32)
    return codes, res, lens, cent, bw, nbits


def test_reader_round_trip_merged_and_chunked(tmp_path):
    from late_interaction_kernels_b200.plaid_index import read_fastplaid_index

    codes, res, lens, cent, bw, nbits = small_index()
    for merged in (True, False):
        p = str(tmp_path / f"idx_{int(merged)}")
        write_fastplaid_files(p, codes, res, lens, cent, bw, nbits, merged=merged, pad_rows=5)
        ix = read_fastplaid_index(p, device="cpu")
        assert ix.nbits == nbits and ix.n_docs == len(lens) and ix.dim == 32
        assert ix.codes_flat.dtype == torch.int32 and np.array_equal(ix.codes_flat.numpy(), codes)
        assert ix.residuals_flat.dtype == torch.uint8 and np.array_equal(ix.residuals_flat.numpy(), res)
        assert np.array_equal(ix.doc_lengths.numpy(), lens)
        assert np.array_equal(ix.cu_seqlens_d.numpy(), np.concatenate([[0], np.cumsum(lens)]))
        assert np.array_equal(ix.centroids.numpy(), cent) and np.array_equal(ix.bucket_weights.numpy(), bw)


def test_inverted_file_matches_the_oracle():
    from late_interaction_kernels_b200.plaid_index import PlaidIndexData, build_ivf

    codes, res, lens, cent, bw, nbits = small_index(seed=5, nd=60, ncent=23)
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ix = PlaidIndexData(nbits, torch.from_numpy(cent), torch.from_numpy(bw), torch.from_numpy(codes), torch.from_numpy(res),
                        torch.from_numpy(lens.astype(np.int64)), torch.from_numpy(cu))
    build_ivf(ix)
    docs, off = O.plaid_ivf(codes, cu, 23)
    assert np.array_equal(ix.ivf_docs.numpy(), docs) and np.array_equal(ix.ivf_offsets.numpy(), off)
    # brute force: document j is on the list of centroid c exactly when one of its tokens has code c
    for c in range(23):
        want = [j for j in range(60) if (codes[cu[j]:cu[j + 1]] == c).any()]
        assert docs[off[c]:off[c + 1]].tolist() == want


def test_which_way_a_compressed_index_is_scored():
    """Both sides of the rule's lines, at sizes where the two ways are far apart; the knob overrides it."""
    from late_interaction_kernels_b200 import plaid

    def way(nq, lq, nd, longest, tokens=None, winners=False, nbits=2, **kw):
        return plaid._decode_in_kernel(nq, lq, winners, nd, longest * nd if tokens is None else tokens, longest, nbits, **kw)

    assert way(1, 32, 25000, 300, 4_500_000) and way(4, 32, 25000, 300, 4_500_000) and way(1, 32, 8, 64) and way(1, 128, 1000, 300, 180_000)
    assert way(1, 32, 1184, 4096, 2_900_000) and way(16, 8, 25000, 300, 4_500_000)
    assert not way(1, 32, 8, 4096) and not way(4, 20, 78, 3449, 161_205, nbits=8)  # few long documents
    assert not way(128, 1, 2925, 71, 35_242, nbits=8) and not way(64, 2, 10000, 8, 45_000)  # many queries, short documents
    assert way(1, 32, 8, 4096, host=125.0) and way(128, 1, 2925, 71, 35_242, host=float("inf"))  # where the host is what takes the time
    assert not way(5, 32, 25000, 300) and not way(1, 129, 8, 64) and not way(1, 32, 8, 64, winners=True) and not way(0, 32, 8, 64) and not way(1, 0, 8, 64)
    assert plaid._longest(10, 1000, 0) == 200 and plaid._longest(10, 1000, 150) == 150 and plaid._longest(0, 0, 0) == 0 and plaid._longest(1, 1000, 0) == 1000
    try:
        plaid._FUSED_DECODE_MAX_GROUPS = 0
        assert not way(1, 32, 25000, 300)
        plaid._FUSED_DECODE_MAX_GROUPS = 3
        assert way(1, 32, 8, 4096) and way(24, 32, 8, 64, winners=True) and not way(32, 32, 8, 64)
    finally:
        plaid._FUSED_DECODE_MAX_GROUPS = None
