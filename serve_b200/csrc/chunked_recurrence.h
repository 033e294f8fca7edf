// The walk of sequence_ops.cu, 32 tokens at a time: see chunked_recurrence.cu.
#pragma once
#include <cuda_runtime.h>

struct SbChunkedWalk {
  // what recurrence_prep_kernel leaves, as float: q and k [T, Hqk, dkp], a decay per row [T, H, dkp] (or null), v [T, H, dvp],
  // and [T, H]: the factor of the update (dt, beta; WKV: the bonus sum) and one decay for the whole state
  const float *qf, *kf, *af, *vf, *sc, *dec;
  int n_tokens, H, Hqk, dk, dv, dkp, dvp;
  int mode;                    // as in sequence_ops.cu
  int head_rate;               // af holds one decay a head: the first of its dkp numbers is read, the others need not be there
  const void* skip;            // SSM: D of every head, float or bfloat16 (skip_dtype, as in common.cuh)
  int skip_dtype;
  float* state;
  long long state_stride;
  const int *slots, *cu_q;
  const int* rows;             // the requests by falling number of tokens, or null: all of them in order
  int n_list, max_q;           // entries of the list to look at; most tokens a request brings
  int min_tokens;              // requests with at most this many tokens are left alone
  float* out;
  int out_stride;
  int* timeouts;               // counts waits on a copy that ran out
  float* work;                 // sb_chunked_walk_floats() floats, 16-byte aligned
};

// Floats of work space for ``chunks`` chunks of 32 tokens (each listed request's rounded up), or -1 if the sizes are not taken.
long long sb_chunked_walk_floats(int mode, int n_tokens, int chunks, int H, int dk, int dvp);
int sb_chunked_walk(const SbChunkedWalk& a, int chunks, cudaStream_t stream);
