// Persistent recurrences (rnn_sequence.cu): all time steps of one layer, both of its directions
// side by side where they fit, in one kernel.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace flb200 {

// A job is one direction of one layer over up to 48 rows of the batch.  All pointers are at the
// job's first batch row; time steps are B_total rows apart.
// G = 4: LSTM, cells = cell states.  G = 3: GRU, cells = q = U_n h + b_hn per step (what its gradient
// needs), c0 unused, b_hn = the candidate gate's recurrent bias.  G = 1: the plain cells (act 0 relu,
// 1 tanh): gates receives h, no cell tensor.
struct SeqJob {
  const float* w_hh;       // [G*H][H]
  float* gates;            // [T][B_total][G*H]: input projections + biases in, activated gates out
  float* cells;            // [T][B_total][H]
  const float* b_hn;
  float* out;              // [T][B_total] rows of out_stride floats, this direction's first column
  const float* h0;         // [B][H], never null
  const float* c0;
  int B, reverse;
};
struct SeqBwdJob {
  const float* w_hh;
  const float* gates;      // what the forward pass left
  const float* cells;
  const float* first;      // [B][H]: LSTM c0, GRU h0
  const float* out;        // GRU: the forward output, this direction's first column
  const float* dy;         // gradient of the output, this direction's first column, or null
  const float* dh0;        // [B][H] gradient of the final state, or null
  const float* dc0;
  float* dgates;           // [T][B_total][G*H] out
  float* dgh;              // GRU: the gate gradients of the recurrent side; else == dgates
  float* dh_out;           // [B][H] out
  float* dc_out;
  int B, reverse;
};
struct SeqShape {
  int T, B, H, G, dirs, act;
  long long out_stride, dy_stride;
};

// Whether (and with how many rows of the batch per job) the persistent kernels take this shape:
// TF32 mode, a hidden size of a multiple of 4 up to 1024, 16-byte aligned weights, and a device that
// holds a job's CTAs at once.  0: no; the caller then runs a kernel per step.
int rnn_sequence_rows(int math_mode, const SeqShape& s, const float* w_hh, bool backward);
// Scratch for all jobs of a layer (the exchange buffers of the running step).
size_t rnn_sequence_scratch_bytes(const SeqShape& s, bool backward);
// Runs the jobs, as many at a time as the device holds.  wait_budget: clocks a CTA waits for another
// one's values before it gives up (0: about two seconds); absent_cta >= 0: that CTA of a job never
// publishes any (used by the bounded-wait test only).
int rnn_sequence_forward(const SeqShape& s, const SeqJob* jobs, int n, void* scratch, cudaStream_t st,
                         long long wait_budget = 0, int absent_cta = -1);
int rnn_sequence_backward(const SeqShape& s, const SeqBwdJob* jobs, int n, void* scratch,
                          cudaStream_t st);

}  // namespace flb200
