// What a scoring or gradient kernel needs written before it starts, in one launch (lik_prep.cu): inverse norms of either
// side, effective document lengths under a token mask, and cleared words.
#pragma once

#include "lik_common.cuh"

namespace lik {

struct NormJob {  // out[r] = 1 / max(||x_r||, eps); rows that no valid token sits in get 0 and are not read
  const void* data = nullptr;  // nullptr: no job
  int dtype = 0, dim = 0;
  long long n_rows = 0, stride = 0;
  const unsigned char* mask = nullptr;  // optional, one byte per row
  const int* lens = nullptr;            // optional, padded layout: rows t >= lens[row / seq_stride]
  long long seq_stride = 0;
  float eps = 0.f;
  float* out = nullptr;
};

struct MaskLensJob {  // out[j] = 1 + last valid token, tagged with `flag` when the valid tokens are not a prefix
  const unsigned char* mask = nullptr;  // nullptr: no job
  const int* lens = nullptr;
  int n_seq = 0, max_len = 0;
  long long seq_stride = 0;
  int* out = nullptr;
  int flag = 0;  // or-ed into out[j] when the mask has holes
  int* status = nullptr;  // lengths outside [0, max_len] are reported here (they are clamped either way)
};

struct FillJob {  // whole 32-bit words (sixteen bytes at a time where they lie on such a boundary)
  void* ptr = nullptr;  // nullptr: no job
  size_t bytes = 0;
  int word = 0;
};

struct PrepJobs {
  NormJob norm[2];
  MaskLensJob mask_lens;
  FillJob fill[2];
};

NormJob norm_job(const lik_seqs& s, int dtype, int dim, float eps, float* out, bool all_rows);
int launch_prep(const PrepJobs& jobs, cudaStream_t st);

}  // namespace lik
