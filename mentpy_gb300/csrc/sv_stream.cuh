// Shared by the wide-window sweeps: the streamed passes (sv_stream.cu) and the
// on-chip kernel (sv_chip.cu).
#pragma once

#include "sv_reg.cuh"

namespace mbqc {

struct StreamArgs {
  const DevStep *steps;  // this circuit's steps
  int W, M, n_in, n_out;
  int S;                 // log2 of a run's amplitudes in the workspace: W - 1 (half) or W
  int64_t B;
  const double *angles;
  int64_t astride;
  const float2 *psi_in;
  int64_t istride;
  float2 *state;   // [B][2^S]
  double *norms;   // [3][B]
  int32_t *expo;   // [B] total applied exponent
  int8_t in_bits[32];
  int8_t out_bits[32];
  uint32_t init_cz[32];
};

// a pass step on register bit J (lower half amp = 1 unless GEN)
template <bool GEN, int R, int J>
__device__ __forceinline__ void pass_reg_step(float2 (&v)[R], float2 c, float amp, uint32_t ts, bool dead) {
  if constexpr (GEN)
    reg_step_g<float, R, J>(v, c, amp, ts, dead);
  else
    reg_step<float, R, J>(v, c, ts, dead);
}
// The same on a pair of phi_{k-1} that becomes a pair of phi_k (HALF): both halves
// of the entered qubit, the second with the sign of its CZs and c1 = -c where one
// of them is with the measured qubit.
template <bool GEN, int R, int J>
__device__ __forceinline__ void pass_half_step(float2 (&v)[R], float2 c, float amp, uint32_t flip, uint32_t ts,
                                               bool dead) {
  const float2 c1 = flip_sign(c, flip);
#pragma unroll
  for (int j = 0; j < R; ++j) {
    if (j & (1 << J)) continue;
    const int jh = j | (1 << J);
    const float2 x0 = v[j], x1 = v[jh];
    float2 o;
    if constexpr (GEN) {
      v[j] = make_float2(amp * x0.x + c.x * x1.x - c.y * x1.y, amp * x0.y + c.x * x1.y + c.y * x1.x);
      o = make_float2(amp * x0.x + c1.x * x1.x - c1.y * x1.y, amp * x0.y + c1.x * x1.y + c1.y * x1.x);
    } else {
      v[j] = make_float2(x0.x + c.x * x1.x - c.y * x1.y, x0.y + c.x * x1.y + c.y * x1.x);
      o = make_float2(x0.x + c1.x * x1.x - c1.y * x1.y, x0.y + c1.x * x1.y + c1.y * x1.x);
    }
    v[jh] = sign_bit_flip(o, ts * (1u << (31 - jh)));
  }
  if (dead) {
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (j & (1 << J)) v[j] = make_float2(0.f, 0.f);
  }
}

// Half windows: the stored bit of the qubit at a window bit after `done` steps.  The
// window holds the qubits done .. done + w - 1 of the schedule at bit (index mod w);
// all but the last are stored, qubit s at bit (s - 1) mod (w - 1): the bit of the
// measured qubit is the entering one's.
__host__ __device__ inline int half_bit(int pos, int done, int w) {
  const int s = done + ((pos - done) % w + w) % w;
  return (s - 1) % (w - 1);
}

// The whole sweep in shared memory: one launch, no workspace.  chip_plan: the
// blocks that share a run (0: not for this kernel).
int chip_plan(const DevCircuit &hc, int64_t batch, size_t *smem);
int launch_sv_chip(const StreamArgs &a, const DevCircuit &hc, int cs, size_t smem, uint32_t flags, float2 *out,
                   double *logprob, int32_t *status, cudaStream_t s);

}  // namespace mbqc
