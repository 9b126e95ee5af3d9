// Adjoint gradient of the statevector sweep for windows 9..20, and for plans
// with XZ / YZ steps at any window up to 20: a block per run.
//
// The chain is the one of sv_adj.cuh: per step k the window is scaled by an
// exact power of two alpha_k (its norm then lies in [1, 4)), measured and
// expanded,
//   psi_k = E_k C_k(alpha_k u_{k-1}),  C_k: phi[r] = v[r, 0] + c_k v[r, 1],
// and the output is z = u_M / |u_M|.  Backward, with lambda_M = dL/du_M:
//   mu[r]              = lambda_k[r, 0] + s_k(r) lambda_k[r, 1]
//   dL/dtheta_k        = alpha_k Im(c_k sum_r conj(mu[r]) u_{k-1}[r, 1])
//   lambda_{k-1}[r, 0] = alpha_k mu[r],  lambda_{k-1}[r, 1] = alpha_k conj(c_k) mu[r].
//
// The window does not fit in registers here, so the block keeps it in shared
// memory (w <= 14) or in its workspace slot (w >= 15).  The forward pass writes
// what it needs of the pre-step half-state u_{k-1}[., 1] of every step to the
// slot's history and the backward pass reads it back: one forward, one backward,
// no recompute.  The grid is persistent (a workspace slot per
// block); the slot count is capped so the workspace stays within
// kWideAdjMaxWorkspace.  Block sums (norms, <z|g>, the gradient terms) are a
// butterfly per warp, then the warps' partials in a fixed order, so every
// thread holds the same bits.  The input placement and the output gather are
// computed from the plan's bit tables (no index map, which stops at w = 16).
//
// GEN (plans with XZ / YZ steps): the step is phi = amp v[., 0] + c v[., 1]
// with both coefficients depending on theta (sv_coef_gen: amp = C + S and
// c = C - S (XZ) or -i (C - S) (YZ), C, S = cos, sin of half the reduced
// angle), so d amp / dtheta = (C - S) / 2 and dc / dtheta = -amp / 2 (XZ) or
// i amp / 2 (YZ); an XY step keeps amp = 1 and dc = -i c.  Backward:
//   dL/dtheta_k = alpha_k Re(damp sum conj(mu) u[., 0] + dc sum conj(mu) u[., 1])
//   lambda_{k-1}[r, 0] = alpha_k amp mu[r],  lambda_{k-1}[r, 1] = alpha_k conj(c) mu[r]
// and the history keeps both halves of every pre-step state.
//
// CS > 1 (windows >= 15, batches smaller than the GPU): a cluster of CS blocks
// shares one run, each block taking a 1/CS slice of every pass; the block
// sums are then summed over the cluster (each block's partials read through
// distributed shared memory, in rank order, so every thread still holds the
// same bits) and the cluster barrier that does it also orders the window's
// global writes between the blocks.  Every block of a cluster runs the same
// loops, so every barrier is reached by all of them.
#include <cuda_runtime.h>

#include <type_traits>

#include "cluster_sum.cuh"
#include "dispatch.h"
#include "sv_adj.cuh"

namespace mbqc {

template <int W>
struct WideAdjCfg {
  static constexpr int D = 1 << W;
  static constexpr int TPR = W <= 9 ? 128 : (W == 10 ? 256 : (W == 11 ? 512 : 1024));
  static constexpr int NW = TPR / 32;
  static constexpr bool kWs = W > 14;  // the window itself in the workspace slot
};

__device__ __forceinline__ uint32_t wide_insert_bit(uint32_t r, int p) {
  return ((r >> p) << (p + 1)) | (r & ((1u << p) - 1u));
}

__host__ __device__ inline size_t wide_al(size_t b) { return (b + 15) & ~(size_t)15; }

// shared memory of one block: [window (w <= 14)] [coef M] [mask M] [aidx M] [expo M] [red 2 x NW x 4]
// [general-plane derivative table M (GEN)]
__host__ __device__ inline size_t wide_smem_bytes(int w, int M, bool gen) {
  const int tpr = w <= 9 ? 128 : (w == 10 ? 256 : (w == 11 ? 512 : 1024));
  return (w > 14 ? 0 : wide_al(((size_t)1 << w) * 8)) + wide_al((size_t)M * 8) + 3 * wide_al((size_t)M * 4) +
         wide_al((size_t)2 * (tpr / 32) * 4 * sizeof(float)) + (gen ? wide_al((size_t)M * 16) : 0);
}

// Sum of NV per-thread values over the block; the same bits in every thread.
// red is double-buffered: a fast thread's next call cannot overwrite partials
// a slow thread is still reading (it waits at the next barrier first).
template <int NW, int NV>
__device__ __forceinline__ void block_sum(float (&v)[NV], float *red, int &par) {
#pragma unroll
  for (int j = 0; j < NV; ++j)
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
  float *r = red + par * (NW * 4);
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int j = 0; j < NV; ++j) r[(threadIdx.x >> 5) * 4 + j] = v[j];
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) s += r[w * 4 + j];
    v[j] = s;
  }
  par ^= 1;
}


// Plans with XZ / YZ steps, any window up to 20: one block per run.
template <int W>
__global__ void __launch_bounds__(WideAdjCfg<W>::TPR) sv_adj_wide_gen(SvAdjArgs A, WideAdjGeom G) {
  using Cfg = WideAdjCfg<W>;
  constexpr int D = Cfg::D, TPR = Cfg::TPR, NW = Cfg::NW, H2 = D / 2;
  // a pass gives each thread NIT pairs (q = tid + n TPR), taken U at a
  // time: the U pairs' loads are all issued before the first write-back (the
  // window sits in the workspace above w = 14, and a load after a store to
  // it cannot be hoisted by the compiler), so a thread keeps 2U window loads
  // (4U in the backward pass, with the history) in flight instead of two;
  // each thread still sums its pairs in q order
  constexpr int NIT = H2 >= TPR ? H2 / TPR : 1;
  constexpr int U = NIT < 2 ? NIT : 2;  // 4 or 8 spill: both halves of a pair's history are held
  static_assert((H2 < TPR || H2 % TPR == 0) && NIT % U == 0, "pairs per thread");
  const bool live = H2 >= TPR || threadIdx.x < (unsigned)H2;  // small windows: fewer pairs than threads
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x;
  const int M = A.M, NA = A.n_angles;
  size_t off = Cfg::kWs ? 0 : wide_al((size_t)D * 8);
  float2 *s_coef = reinterpret_cast<float2 *>(smem + off);
  off += wide_al((size_t)M * 8);
  uint32_t *s_mask = reinterpret_cast<uint32_t *>(smem + off);
  off += wide_al((size_t)M * 4);
  int32_t *s_aidx = reinterpret_cast<int32_t *>(smem + off);
  off += wide_al((size_t)M * 4);
  int32_t *s_expo = reinterpret_cast<int32_t *>(smem + off);
  off += wide_al((size_t)M * 4);
  float *red = reinterpret_cast<float *>(smem + off);
  off += wide_al((size_t)2 * NW * 4 * sizeof(float));
  float4 *s_gen = reinterpret_cast<float4 *>(smem + off);  // [M] (amp, damp, dc)

  float2 *slot = reinterpret_cast<float2 *>(A.ckpt) + (size_t)blockIdx.x * G.slot_elems;
  float2 *s = Cfg::kWs ? slot : reinterpret_cast<float2 *>(smem);
  float4 *hist = reinterpret_cast<float4 *>(slot + (Cfg::kWs ? D : 0));

  for (int k = tid; k < M; k += TPR) {
    const DevStep st = A.steps[k];
    s_mask[k] = st.mask;
    s_aidx[k] = st.aidx;
  }
  const bool fid = A.J > 0;
  const int n_in = A.n_in, n_out = A.n_out;
  const int64_t dout = (int64_t)1 << n_out;
  int par = 0;

  for (int64_t run = blockIdx.x; run < A.B; run += gridDim.x) {
    const int64_t vrow = fid ? run / A.J : run;
    const int64_t irow = fid ? run % A.J : (A.istride ? run : 0);
    for (int k = tid; k < M; k += TPR) {
      const DevStep st = A.steps[k];
      const double th = st.aidx >= 0 ? A.angles[vrow * A.astride + st.aidx] : st.fixed;
      float2 c, ph;
      float amp;
      sv_coef_gen(st.plane, th, false, c, amp, ph);
      float damp = 0.f;
      float2 dc = make_float2(c.y, -c.x);  // XY: -i c
      if (st.plane == MBQC_PLANE_XZ) {
        damp = 0.5f * c.x;  // (C - S) / 2
        dc = make_float2(-0.5f * amp, 0.f);
      } else if (st.plane == MBQC_PLANE_YZ) {
        damp = -0.5f * c.y;  // c = -i (C - S)
        dc = make_float2(0.f, 0.5f * amp);
      }
      s_gen[k] = make_float4(amp, damp, dc.x, dc.y);
      s_coef[k] = c;
    }
    // ---- initial window: input on its bits, |+> elsewhere, the CZ layer's signs
    const float2 *in = reinterpret_cast<const float2 *>(A.psi_in) +
                       irow * (fid ? ((int64_t)1 << n_in) : A.istride);
    float nv[1] = {0.f};
    for (int i = tid; i < D; i += TPR) {
      const float2 v = flip_sign(in[gather_bits((uint32_t)i, G.in_bits, n_in)],
                                 init_parity((uint32_t)i, G.init_cz, W) << 31);
      s[i] = v;
      nv[0] += v.x * v.x + v.y * v.y;
    }
    block_sum<NW, 1>(nv, red, par);
    float nrm = nv[0];

    // ---- forward, keeping every step's pre-step half-state
    for (int k = 0; k < M; ++k) {
      const int e = renorm_exponent<float>(nrm);
      if (tid == 0) s_expo[k] = e;
      const float al = RealBits<float>::pow2(-e);
      const float2 c = s_coef[k];
      const float amp = s_gen[k].x;
      const uint32_t mask = s_mask[k];
      const bool dead = (mask & kDead) != 0u;
      const int p = k % W;
      float4 *hk = hist + (size_t)k * D / 2;
      float acc[1] = {0.f};
      if (live) {
        for (int b = 0; b < NIT; b += U) {
          float2 u0[U], u1[U];  // U pairs loaded before any is written back
#pragma unroll
          for (int j = 0; j < U; ++j) {
            const uint32_t i0 = wide_insert_bit((uint32_t)(tid + (b + j) * TPR), p);
            u0[j] = s[i0];
            u1[j] = s[i0 | (1u << p)];
          }
#pragma unroll
          for (int j = 0; j < U; ++j) {
            const int q = tid + (b + j) * TPR;
            const uint32_t i0 = wide_insert_bit((uint32_t)q, p), i1 = i0 | (1u << p);
            hk[q] = make_float4(u0[j].x, u0[j].y, u1[j].x, u1[j].y);
            const float2 phi = make_float2(al * (amp * u0[j].x + c.x * u1[j].x - c.y * u1[j].y),
                                           al * (amp * u0[j].y + c.x * u1[j].y + c.y * u1[j].x));
            s[i0] = phi;
            s[i1] = dead ? make_float2(0.f, 0.f) : flip_sign(phi, (uint32_t)(__popc(i1 & mask) & 1u) << 31);
            acc[0] += phi.x * phi.x + phi.y * phi.y;
          }
        }
      }
      block_sum<NW, 1>(acc, red, par);
      nrm = dead ? acc[0] : 2.f * acc[0];
    }

    // ---- output and the seed lambda_M = dL/du_M
    const bool ok = RealBits<float>::finite_pos(nrm);
    float inv = 0.f;
    if (ok) {
      const float y = rsqrtf(nrm);
      inv = y * (1.5f - 0.5f * nrm * y * y);  // one Newton step
    }
    if (!ok) {
      if (!fid)
        for (int ai = tid; ai < NA; ai += TPR) A.grad[run * NA + ai] = NAN;
      if (tid == 0 && A.status) A.status[run] = isnan(nrm) ? MBQC_RUN_NAN : MBQC_RUN_ZERO_NORM;
      __syncthreads();  // the next run overwrites the coefficients
      continue;
    }
    float loss_term = 0.f;
    if (fid) {
      const float2 *tg = reinterpret_cast<const float2 *>(A.targets) + irow * dout;
      float pv[2] = {0.f, 0.f};  // <t|u_M>
      for (int i = tid; i < D; i += TPR) {
        if ((uint32_t)i & ~G.out_mask) continue;
        const float2 t = tg[gather_bits((uint32_t)i, G.out_bits, n_out)], a = s[i];
        pv[0] += t.x * a.x + t.y * a.y;
        pv[1] += t.x * a.y - t.y * a.x;
      }
      block_sum<NW, 2>(pv, red, par);
      const float ar = pv[0] * inv, ai = pv[1] * inv;
      const float F = ar * ar + ai * ai;
      const float wJ = 1.f / (float)A.J;
      loss_term = (1.f - F) * wJ;
      // lambda = (2/J)(F z - a t) / |u_M|
      const float k2 = 2.f * wJ * inv, fz = F * inv;
      for (int i = tid; i < D; i += TPR) {
        float2 l = make_float2(0.f, 0.f);
        if (!((uint32_t)i & ~G.out_mask)) {
          const float2 t = tg[gather_bits((uint32_t)i, G.out_bits, n_out)], a = s[i];
          l = make_float2(k2 * (fz * a.x - (ar * t.x - ai * t.y)), k2 * (fz * a.y - (ar * t.y + ai * t.x)));
        }
        s[i] = l;
      }
    } else {
      const float2 *go = reinterpret_cast<const float2 *>(A.grad_out) + run * dout;
      float zv[1] = {0.f};  // Re <u_M|g>
      for (int i = tid; i < D; i += TPR) {
        if ((uint32_t)i & ~G.out_mask) continue;
        const float2 g = go[gather_bits((uint32_t)i, G.out_bits, n_out)], a = s[i];
        zv[0] += a.x * g.x + a.y * g.y;
      }
      block_sum<NW, 1>(zv, red, par);
      const float zgi = zv[0] * inv * inv;
      for (int i = tid; i < D; i += TPR) {
        float2 l = make_float2(0.f, 0.f);
        if (!((uint32_t)i & ~G.out_mask)) {
          const float2 g = go[gather_bits((uint32_t)i, G.out_bits, n_out)], a = s[i];
          l = make_float2(inv * (g.x - zgi * a.x), inv * (g.y - zgi * a.y));
        }
        s[i] = l;
      }
    }
    __syncthreads();

    // ---- backward
    for (int k = M - 1; k >= 0; --k) {
      const float al = RealBits<float>::pow2(-s_expo[k]);
      const float2 c = s_coef[k];
      const float amp = s_gen[k].x;
      const uint32_t mask = s_mask[k];
      const bool dead = (mask & kDead) != 0u;
      const int p = k % W;
      const float4 *hk = hist + (size_t)k * D / 2;
      float t[4] = {};  // sum conj(mu) u[., 1] and sum conj(mu) u[., 0]
      if (live) {
        for (int b = 0; b < NIT; b += U) {
          // U pairs and their history entries loaded before any is written back
          float2 l0[U], l1[U];
          float4 hh[U];
#pragma unroll
          for (int j = 0; j < U; ++j) {
            const int q = tid + (b + j) * TPR;
            const uint32_t i0 = wide_insert_bit((uint32_t)q, p);
            l0[j] = s[i0];
            l1[j] = dead ? make_float2(0.f, 0.f) : s[i0 | (1u << p)];
            hh[j] = hk[q];
          }
#pragma unroll
          for (int j = 0; j < U; ++j) {
            const int q = tid + (b + j) * TPR;
            const uint32_t i0 = wide_insert_bit((uint32_t)q, p), i1 = i0 | (1u << p);
            float2 mu = l0[j];
            if (!dead) {
              const float2 m1 = flip_sign(l1[j], (uint32_t)(__popc(i1 & mask) & 1u) << 31);
              mu.x += m1.x;
              mu.y += m1.y;
            }
            const float2 h = make_float2(hh[j].z, hh[j].w);
            t[2] += mu.x * hh[j].x + mu.y * hh[j].y;
            t[3] += mu.x * hh[j].y - mu.y * hh[j].x;
            t[0] += mu.x * h.x + mu.y * h.y;
            t[1] += mu.x * h.y - mu.y * h.x;
            s[i0] = make_float2(al * amp * mu.x, al * amp * mu.y);
            s[i1] = make_float2(al * (c.x * mu.x + c.y * mu.y), al * (c.x * mu.y - c.y * mu.x));  // conj(c) mu
          }
        }
      }
      block_sum<NW, 4>(t, red, par);
      const int ai = s_aidx[k];
      if (tid == 0 && ai >= 0) {
        const float4 gd = s_gen[k];  // alpha Re(damp t0 + dc t1)
        const double g = (double)al * ((double)gd.y * t[2] + (double)gd.z * t[0] - (double)gd.w * t[1]);
        if (fid)
          atomicAdd(&A.grad[vrow * NA + ai], g);
        else
          A.grad[run * NA + ai] = g;
      }
    }
    if (tid == 0) {
      if (fid) atomicAdd(&A.loss[vrow], (double)loss_term);
      if (A.status) A.status[run] = MBQC_RUN_OK;
    }
    __syncthreads();  // the next run overwrites the window, the coefficients and the exponents
  }
}

// XY, X and Y plans, windows 9..20.  After step k the window is phi_k and its
// signed copy on the entering qubit's bit (or zero), so only phi_k's N = 2^(w-1)
// amplitudes are kept: index q = the window index without bit p_k = k mod w.
// Step k reads phi_{k-1}: a (measured bit 0) and b (1) give the two halves
//   phi_k[entered bit 0] = a + c b,   phi_k[entered bit 1] = s (a + s' c b),
// s the sign of the entered qubit's CZs, s' = -1 where one of them is with the
// measured qubit: a pair of slots that differ in bit p - 1 of q, in place.  At
// p = 0 (the removed bit moves from w - 1 to 0) the slots move: that step reads
// the window and writes its scratch copy, the next reads that and writes back.
// The history of a step is b alone (N / 2); lambda is kept the same way
// (lambda[., 1] = conj(c) lambda[., 0]): pairs on bit p, w - 1 the step that moves.
//
// What bounds it at w = 17 (64 runs of the 16 x 10 grid, two blocks a run, 2.41 ms)
// is latency at four warps a scheduler: a forward pass of three steps 13 us, a
// backward step 8.6 us on a low bit, 6.2 us in order, 11 to 13 us where it takes
// two passes or joins slices; the history's DRAM floor is 2.5 us a step.
//   * What fits of the block's slice stays in its shared memory (RES: all of it).
//     Entries are placed so that lanes which leave out low bits miss each other's
//     banks (wide_place), indices are split into a thread's part and a uniform one.
//   * The forward pass takes three steps at a time on pairs inside the slice (p = 1:
//     the slots of an item are neighbours and move as 16 bytes).
//   * The gradient's sums are those of TPR = 2 BT threads, thread v taking the q = v
//     mod TPR in turn.  A backward step on a bit below log2 TPR gives a thread two
//     of those (insert_bit(tid, p) and its partner); on the three bits above, the
//     pairs are 2, 4 and 8 apart in one thread's order and a group of them is held;
//     above that, and on bits that join slices, lambda is updated first and summed
//     over q in order afterwards.  Only the warps' sums are made per step.
// Both halves kept, one or two steps a pass: w = 17, 64 runs 4.98 ms; w = 15, 256
// runs 2.80 -> 1.77; w = 12, 512 runs 0.60 -> 0.52; w = 19, 32 runs of 18 x 6 9.44 ->
// 4.32 ms.  Loading the history a batch ahead was slower (2.64 ms).
// Short circuits in small batches pay for the set-up and the sums at the run's end: w =
// 9, 16 steps, 1 run 21.0 -> 22.8 us on the device, 64 runs 22.3 -> 25.1; w = 10, 18
// steps 25.1 -> 27.2; from 24 steps on no case is slower.
template <int W, int CS> struct WideHalfCfg {
  static constexpr int D = 1 << W, N = D / 2, NS = N / CS;
  static constexpr int LT = W <= 9 ? 7 : (W == 10 ? 8 : (W == 11 ? 9 : 10));
  static constexpr int TPR = 1 << LT, BT = TPR / 2, VW = TPR / 32;
  static constexpr bool kWs = W > 14;
  static constexpr int LOGCS = CS == 4 ? 2 : (CS == 2 ? 1 : 0);
  static constexpr int SB = W - 1 - LOGCS;  // index bits of a block's slice
  static constexpr int FMAX = SB - LT + 1 < 3 ? SB - LT + 1 : 3;
  static constexpr int MINB = W >= 14 ? 1 : 1024 / BT;
  static constexpr int U = W >= 14 ? 4 : 2;  // items whose loads are issued together
  static_assert(W >= 9 && SB >= LT + 1, "entries per thread");
  static_assert(CS == 1 || kWs, "clusters share a run only with the window in the workspace");
};

// Warp sums of NV values of 2 BT virtual threads, in the order of block_sum over
// them: thread tid holds those of insert_bit(tid, p) (v[j][0]) and its partner on
// bit p; put(j, virtual warp, sum).
template <int NV, typename Put>
__device__ __forceinline__ void warp_sums_pair(const float (&v)[NV][2], int p, Put put) {
  const int wq = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (p < 5) {
    const int top = threadIdx.x >> 4;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      float a = v[j][0], b = v[j][1];
      for (int o = 16; o > (1 << p); o >>= 1) {  // bits above p sit one lane bit lower
        a += __shfl_xor_sync(0xffffffffu, a, o >> 1);
        b += __shfl_xor_sync(0xffffffffu, b, o >> 1);
      }
      a += b;
      for (int o = (1 << p) >> 1; o >= 1; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if ((lane & 15) == 0) put(j, top, a);
    }
  } else {
    const int w0 = (int)wide_insert_bit((uint32_t)wq, p - 5);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      float a = v[j][0], b = v[j][1];
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
      }
      if (lane == 0) {
        put(j, w0, a);
        put(j, w0 | (1 << (p - 5)), b);
      }
    }
  }
}

template <int VW, int NV>
__device__ __forceinline__ void block_sum_pair(const float (&v)[NV][2], float (&out)[NV], float *red, int &par) {
  float *r = red + par * (VW * 4);
  warp_sums_pair<NV>(v, 0, [&](int j, int w, float a) { r[w * 4 + j] = a; });
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < VW; ++w) s += r[w * 4 + j];
    out[j] = s;
  }
  par ^= 1;
}

__device__ __forceinline__ uint32_t wide_remove_bit(uint32_t q, int p) {
  return ((q >> (p + 1)) << p) | (q & ((1u << p) - 1u));
}
// Place of an entry in its slice: bits 4..6 folded into 1..3, so that accesses of
// 8 bytes whose lanes leave out a bit below 4, or three bits from 0 or 3 on, find
// 16 different banks.  Linear, and 16-byte pairs stay together.
__device__ __forceinline__ uint32_t wide_place(uint32_t e) {
  return e ^ ((e >> 3) & 12u) ^ (((e >> 4) & 1u) * 14u);
}
__device__ __forceinline__ float sign_f(float v, uint32_t s) { return __uint_as_float(__float_as_uint(v) ^ s); }
__device__ __forceinline__ uint32_t sign_of(uint32_t v, uint32_t mask) { return (uint32_t)__popc(v & mask) << 31; }

template <int W, int CS, bool RES>
__global__ void __launch_bounds__((WideHalfCfg<W, CS>::BT), (WideHalfCfg<W, CS>::MINB))
    sv_adj_wide(SvAdjArgs A, WideAdjGeom G) {
  using Cfg = WideHalfCfg<W, CS>;
  constexpr int N = Cfg::N, NS = Cfg::NS, TPR = Cfg::TPR, BT = Cfg::BT, VW = Cfg::VW, LT = Cfg::LT, SB = Cfg::SB,
                FMAX = Cfg::FMAX;
  __shared__ float cred[8];
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x;
  const int M = A.M, NA = A.n_angles;
  size_t off = Cfg::kWs ? 0 : wide_al((size_t)2 * N * 8);
  float2 *s_coef = reinterpret_cast<float2 *>(smem + off);
  off += wide_al((size_t)M * 8);
  uint32_t *s_mask = reinterpret_cast<uint32_t *>(smem + off);
  off += wide_al((size_t)M * 4);
  int32_t *s_aidx = reinterpret_cast<int32_t *>(smem + off);
  off += wide_al((size_t)M * 4);
  int32_t *s_expo = reinterpret_cast<int32_t *>(smem + off);
  off += wide_al((size_t)M * 4);
  float *red = reinterpret_cast<float *>(smem + off);
  off += wide_al((size_t)2 * VW * 4 * sizeof(float));

  int crank = 0, cid = blockIdx.x, ncl = gridDim.x, cpar = 0;
  if constexpr (CS > 1) {
    crank = (int)cooperative_groups::this_cluster().block_rank();
    cid = blockIdx.x / CS;
    ncl = gridDim.x / CS;
  }
  const uint32_t q_lo = (uint32_t)crank * NS, h_lo = q_lo / 2;  // this block's entries, its pairs
  float2 *slot = reinterpret_cast<float2 *>(A.ckpt) + (size_t)cid * G.slot_elems;
  float2 *hist = slot + (Cfg::kWs ? 2 * N : 0);  // step 0: N entries; step k: N / 2 at (k + 1) N / 2
  float2 *part = hist + (size_t)(M + 1) * (N / 2);  // [step][rank][warp]
  float2 *swin = reinterpret_cast<float2 *>(smem + (Cfg::kWs ? off : 0));
  float2 *scratch = (Cfg::kWs ? slot : swin) + N;
  float2 *gown = slot + q_lo;
  const uint32_t res = (uint32_t)G.res;
  auto home = [&](uint32_t q) -> float2 * {  // an entry of this block's slice
    const uint32_t local = wide_place(q & (NS - 1));
    if constexpr (RES) return swin + local;
    return ((local >> 10) < res ? swin : gown) + local;
  };
  auto home_at = [&](uint32_t local) -> float2 * {  // by its place
    if constexpr (RES) return swin + local;
    return ((local >> 10) < res ? swin : gown) + local;
  };
  auto slice_at = [&](uint32_t qn) -> float2 * {  // the slice holding the piece of 1,024 from qn on
    if constexpr (RES) return swin;
    return (qn >> 10) < res ? swin : gown;
  };
  auto any = [&](uint32_t q) -> float2 * {  // of any block's
    if constexpr (CS == 1) return home(q);
    const uint32_t local = wide_place(q & (NS - 1));
    if (!RES && (local >> 10) >= res) return slot + (q & ~(uint32_t)(NS - 1)) + local;
    return cooperative_groups::this_cluster().map_shared_rank(swin, (int)(q / NS)) + local;
  };
  auto scr = [&](uint32_t q) -> float2 * { return scratch + q; };
  auto hist_of = [&](int k) -> float2 * { return hist + (size_t)(k ? k + 1 : 0) * (N / 2); };
  using One = std::integral_constant<int, 1>;
  using Max = std::integral_constant<int, FMAX>;
  using Yes = std::true_type;
  using No = std::false_type;

  for (int k = tid; k < M; k += BT) {
    const DevStep st = A.steps[k];
    s_mask[k] = st.mask;
    s_aidx[k] = st.aidx;
  }
  const bool fid = A.J > 0;
  const int n_in = A.n_in, n_out = A.n_out;
  const int64_t dout = (int64_t)1 << n_out;
  int par = 0;
  auto phi_of = [](float2 a, float2 b, float2 c) {
    return make_float2(fmaf(-c.y, b.y, fmaf(c.x, b.x, a.x)), fmaf(c.y, b.x, fmaf(c.x, b.y, a.y)));
  };
  auto times = [](float s, float2 v) { return make_float2(s * v.x, s * v.y); };
  auto norm2 = [](float2 v) { return v.x * v.x + v.y * v.y; };
  auto add_norm = [](float &s, float2 v) { s = fmaf(v.x, v.x, fmaf(v.y, v.y, s)); };  // for a scale alone
  auto conj_mul = [](float2 c, float2 m) {
    return make_float2(fmaf(c.y, m.y, __fmul_rn(c.x, m.x)), fmaf(c.x, m.y, -__fmul_rn(c.y, m.x)));
  };
  auto plus = [](float2 a, float2 b, uint32_t s) {
    const float2 m = flip_sign(b, s);
    return make_float2(a.x + m.x, a.y + m.y);
  };
  auto add_t = [](float (&t)[2][2], int z, float2 m, float2 h) {  // conj(mu) u
    t[0][z] += fmaf(m.x, h.x, __fmul_rn(m.y, h.y));
    t[1][z] += fmaf(m.x, h.y, -__fmul_rn(m.y, h.x));
  };
  auto add_ts = [](float (&t)[2][2], int z, float2 m, float2 h, float s) {  // u = s h, s = 1, -1 or 0
    t[0][z] = fmaf(s, fmaf(m.x, h.x, __fmul_rn(m.y, h.y)), t[0][z]);
    t[1][z] = fmaf(s, fmaf(m.x, h.y, -__fmul_rn(m.y, h.x)), t[1][z]);
  };

  for (int64_t run = cid; run < A.B; run += ncl) {
    const int64_t vrow = fid ? run / A.J : run;
    const int64_t irow = fid ? run % A.J : (A.istride ? run : 0);
    for (int k = tid; k < M; k += BT) {
      const DevStep st = A.steps[k];
      const double th = st.aidx >= 0 ? A.angles[vrow * A.astride + st.aidx] : st.fixed;
      float2 c, ph;
      sv_coef(st.plane, th, false, c, ph);
      s_coef[k] = c;
      s_expo[k] = 0;
    }
    const float2 *in = reinterpret_cast<const float2 *>(A.psi_in) +
                       irow * (fid ? ((int64_t)1 << n_in) : A.istride);
    // ---- norm of the first window (input on its bits, |+> elsewhere)
    float nrm;
    {
      float nv[1][2] = {{0.f, 0.f}}, sum[1];
      for (uint32_t x = (uint32_t)(crank * BT + tid); x < (1u << n_in); x += CS * BT) nv[0][0] += norm2(in[x]);
      block_sum_pair<VW, 1>(nv, sum, red, par);
      cluster_sum<CS, 1>(sum, cred, cpar);
      nrm = sum[0] * RealBits<float>::pow2(W - n_in);
    }

    // ---- forward
    bool moved = false;  // the window is in its scratch copy
    {  // step 0: from the input and the CZ layer's signs
      const int e = renorm_exponent<float>(nrm);
      const float al = RealBits<float>::pow2(-e);
      const float2 c = times(al, s_coef[0]);
      if (tid == 0) s_expo[0] = e;
      float acc[1][2] = {{0.f, 0.f}}, sum[1];
      // input index and CZ sign of i = t ^ n (no bit in common): x(t) ^ x(n) and
      // Q(t) ^ Q(n) ^ |n & a(t)| ^ |t & a(n)|, a(v) the couplings of v's bits; the
      // part of the next 32 n is made by the lanes
      auto couplings = [&](uint32_t v) {
        uint32_t a = 0;
        for (int q = 0; q < W; ++q) a ^= (0u - ((v >> q) & 1u)) & G.init_cz[q];
        return a;
      };
      uint32_t xt[2], at[2], qt[2], xn = 0, an = 0;
#pragma unroll
      for (uint32_t z = 0; z < 2; ++z) {
        const uint32_t i = 2 * (q_lo + tid) + z;
        xt[z] = (uint32_t)gather_bits(i, G.in_bits, n_in);
        at[z] = couplings(i);
        qt[z] = init_parity(i, G.init_cz, W);
      }
      for (uint32_t n = 0; n < NS / BT; ++n) {
        const uint32_t q = q_lo + tid + n * BT, in2 = 2 * n * BT;
        if ((n & 31u) == 0) {
          const uint32_t i = 2 * (n + (tid & 31)) * BT;
          xn = (uint32_t)gather_bits(i, G.in_bits, n_in) | (init_parity(i, G.init_cz, W) << 31);
          an = couplings(i);
        }
        const uint32_t xj = __shfl_sync(0xffffffffu, xn, n & 31), aj = __shfl_sync(0xffffffffu, an, n & 31);
        float2 v[2];
#pragma unroll
        for (uint32_t z = 0; z < 2; ++z) {
          const uint32_t odd = qt[z] ^ (xj >> 31) ^ (uint32_t)__popc(in2 & at[z]) ^
                               (uint32_t)__popc((2 * (q_lo + tid) + z) & aj);
          v[z] = flip_sign(in[xt[z] ^ (xj & 0x7fffffffu)], odd << 31);
        }
        hist[q] = v[1];
        const float2 o = phi_of(times(al, v[0]), v[1], c);
        acc[0][0] += norm2(o);
        *home(q) = o;
      }
      block_sum_pair<VW, 1>(acc, sum, red, par);
      cluster_sum<CS, 1>(sum, cred, cpar);
      nrm = (s_mask[0] & kDead) ? sum[0] : 2.f * sum[0];
    }
    // F steps from step k on (p >= 1): the slots' bits p - 1 .. p + F - 2
    // (p1: p = 1, the slots of an item are neighbours; sc: read from the scratch
    // copy; jn: the pair joins two slices)
    auto fwd = [&](auto fc, auto p1, auto sc, auto jn, int k, float al, float (&acc)[1][2]) {
      constexpr int F = decltype(fc)::value, Z = 1 << F, U = F == 1 ? 4 : 2;
      constexpr int CNT = NS / Z / BT, UU = CNT < U ? CNT : U;
      constexpr bool B0 = p1.value && F > 1;
      const int b = B0 ? 0 : k % W - 1;
      const uint32_t low = (1u << b) - 1u;
      float2 c[F], c1[F];
      uint32_t m[F], sg[F], zt[F];
      uint32_t keep[F];
      float2 *hk[F];
      // index maps are bitwise: the thread's part once, the rest uniform
      const uint32_t r0 = (uint32_t)crank * (NS / Z) + tid;
      const uint32_t s0 = ((r0 >> b) << (b + F)) | (r0 & low), l0 = wide_place(s0 & (NS - 1));
#pragma unroll
      for (int f = 0; f < F; ++f) {
        m[f] = s_mask[k + f - 1];
        keep[f] = (m[f] & kDead) ? 0u : ~0u;
        hk[f] = hist_of(k + f) + (((r0 >> b) << (b + F - 1)) | (r0 & low));
        c[f] = s_coef[k + f];
        if (f == 0) c[f] = times(al, c[f]);
        c1[f] = flip_sign(c[f], ((m[f] >> (b + f + 1)) & 1u) << 31);
        const uint32_t ib = ((r0 >> b) << (b + F + 1)) | (r0 & low) | (1u << (b + f));
        sg[f] = (uint32_t)__popc(ib & m[f]) & 1u;
        zt[f] = 0;
#pragma unroll
        for (int z = 0; z < Z; ++z)
          zt[f] |= ((uint32_t)__popc((((uint32_t)((z & ((1 << f) - 1)) | ((z >> (f + 1)) << (f + 2)))) << b) & m[f]) & 1u)
                   << z;
      }
      for (int n = 0; n < CNT; n += UU) {
        float2 x[UU][Z];
#pragma unroll
        for (int j = 0; j < UU; ++j) {
          const uint32_t rn = (uint32_t)(n + j) * BT;
          const uint32_t sn = ((rn >> b) << (b + F)) | (rn & low);
#pragma unroll
          for (int z = 0; z < Z; ++z) {
            const uint32_t zb = sn | ((uint32_t)z << b);
            if constexpr (B0) {
              if (z & 1) continue;
              const float4 v = *reinterpret_cast<const float4 *>(sc.value ? scr(s0 | zb) : home_at(l0 ^ wide_place(zb)));
              x[j][z] = make_float2(v.x, v.y);
              x[j][z | 1] = make_float2(v.z, v.w);
            } else if constexpr (sc.value)
              x[j][z] = *scr(s0 | zb);
            else if constexpr (jn.value)
              x[j][z] = *any(s0 | zb);
            else
              x[j][z] = *home_at(l0 ^ wide_place(zb));
          }
        }
#pragma unroll
        for (int j = 0; j < UU; ++j) {
          const uint32_t rn = (uint32_t)(n + j) * BT;
          const uint32_t sn = ((rn >> b) << (b + F)) | (rn & low);
          const uint32_t hn = ((rn >> b) << (b + F - 1)) | (rn & low);
          const uint32_t ibn = ((rn >> b) << (b + F + 1)) | (rn & low);
#pragma unroll
          for (int f = 0; f < F; ++f) {
            const uint32_t zs = zt[f] ^ (0u - (sg[f] ^ ((uint32_t)__popc(ibn & m[f]) & 1u)));
            float2 hv[Z / 2];
#pragma unroll
            for (int z = 0; z < Z; ++z) {
              if ((z >> f) & 1) continue;
              const int hz = (z & ((1 << f) - 1)) | ((z >> (f + 1)) << f);
              const float2 bb = x[j][z | (1 << f)];
              const float2 aa = f == 0 ? times(al, x[j][z]) : x[j][z];
              if constexpr (B0)
                hv[hz] = bb;
              else
                hk[f][hn | ((uint32_t)hz << b)] = bb;
              x[j][z] = phi_of(aa, bb, c[f]);
              x[j][z | (1 << f)] = keep_flip(phi_of(aa, bb, c1[f]), keep[f], (zs << (31 - z)) & (keep[f] & 0x80000000u));
            }
            if constexpr (B0) {
#pragma unroll
              for (int z = 0; z < Z / 2; z += 2)
                *reinterpret_cast<float4 *>(hk[f] + (hn | (uint32_t)z)) =
                    make_float4(hv[z].x, hv[z].y, hv[z + 1].x, hv[z + 1].y);
            }
          }
#pragma unroll
          for (int z = 0; z < Z; ++z) {
            add_norm(acc[0][0], x[j][z]);
            const uint32_t zb = sn | ((uint32_t)z << b);
            if constexpr (B0) {
              if (z & 1) continue;
              *reinterpret_cast<float4 *>(home_at(l0 ^ wide_place(zb))) =
                  make_float4(x[j][z].x, x[j][z].y, x[j][z | 1].x, x[j][z | 1].y);
            } else if constexpr (jn.value)
              *any(s0 | zb) = x[j][z];
            else
              *home_at(l0 ^ wide_place(zb)) = x[j][z];
          }
        }
      }
    };
    for (int k = 1; k < M;) {
      const int e = renorm_exponent<float>(nrm);
      const float al = RealBits<float>::pow2(-e);
      const int p = k % W;
      if (tid == 0) s_expo[k] = e;
      float acc[1][2] = {{0.f, 0.f}}, sum[1];
      int f = 1;
      if (p == 0) {
        const uint32_t mask = s_mask[k - 1];
        const bool dead = (mask & kDead) != 0u;
        const float2 c = times(al, s_coef[k]), c1 = flip_sign(c, (mask & 1u) << 31);
        float2 *hk = hist_of(k);
        for (uint32_t m = h_lo + tid; m < h_lo + NS / 2; m += BT) {
          const float4 v = *reinterpret_cast<const float4 *>(home(2 * m));
          const float2 aa = times(al, make_float2(v.x, v.y)), bb = make_float2(v.z, v.w);
          hk[m] = bb;
          const float2 o0 = phi_of(aa, bb, c);
          float2 o1 = flip_sign(phi_of(aa, bb, c1), sign_of((2 * m) | (1u << (W - 1)), mask));
          if (dead) o1 = make_float2(0.f, 0.f);
          *scr(m) = o0;
          *scr(m | (N / 2)) = o1;
          acc[0][0] += norm2(o0) + norm2(o1);
        }
        moved = true;
      } else if (CS > 1 && p - 1 >= SB) {
        fwd(One{}, No{}, No{}, Yes{}, k, al, acc);
      } else {
        if (p - 1 + FMAX <= SB && k + FMAX <= M) f = FMAX;
        if (f == FMAX) {
          if (moved)  // p = 1
            fwd(Max{}, Yes{}, Yes{}, No{}, k, al, acc);
          else if (p == 1)
            fwd(Max{}, Yes{}, No{}, No{}, k, al, acc);
          else
            fwd(Max{}, No{}, No{}, No{}, k, al, acc);
        } else {
          if (moved)
            fwd(One{}, Yes{}, Yes{}, No{}, k, al, acc);
          else
            fwd(One{}, No{}, No{}, No{}, k, al, acc);
        }
        moved = false;
      }
      k += f;
      block_sum_pair<VW, 1>(acc, sum, red, par);
      cluster_sum<CS, 1>(sum, cred, cpar);
      nrm = (s_mask[k - 1] & kDead) ? sum[0] : 2.f * sum[0];
    }
    auto now = [&](uint32_t q) -> float2 * {
      if (moved) return scr(q);
      return any(q);
    };

    // ---- output and the seed lambda_M = dL/du_M
    const int pl = (M - 1) % W;
    const uint32_t mask_l = s_mask[M - 1];
    const bool dead_l = (mask_l & kDead) != 0u;
    auto out_of = [&](uint32_t i) {  // u_M
      const float2 v = *now(wide_remove_bit(i, pl));
      if (!((i >> pl) & 1u)) return v;
      return dead_l ? make_float2(0.f, 0.f) : flip_sign(v, sign_of(i, mask_l));
    };
    {  // the last norm is a result: its sums in order
      float acc[1][2] = {{0.f, 0.f}}, sum[1];
      for (uint32_t q = q_lo + 2 * tid; q < q_lo + NS; q += TPR) {
        const float2 v0 = *now(q), v1 = *now(q + 1);
        acc[0][0] += norm2(v0);
        acc[0][1] += norm2(v1);
      }
      block_sum_pair<VW, 1>(acc, sum, red, par);
      cluster_sum<CS, 1>(sum, cred, cpar);
      nrm = dead_l ? sum[0] : 2.f * sum[0];
    }
    const bool ok = RealBits<float>::finite_pos(nrm);
    float inv = 0.f;
    if (ok) {
      const float y = rsqrtf(nrm);
      inv = y * (1.5f - 0.5f * nrm * y * y);  // one Newton step
    }
    if (!ok) {
      if (!fid)
        for (int ai = tid; ai < NA && crank == 0; ai += BT) A.grad[run * NA + ai] = NAN;
      if (tid == 0 && crank == 0 && A.status) A.status[run] = isnan(nrm) ? MBQC_RUN_NAN : MBQC_RUN_ZERO_NORM;
      run_barrier<CS>();  // the next run overwrites the coefficients
      continue;
    }
    const float2 *row = reinterpret_cast<const float2 *>(fid ? A.targets : A.grad_out) + (fid ? irow : run) * dout;
    float loss_term = 0.f, w0, w1, w2, w3;  // the seed's factors
    {
      float pv[2][2] = {}, ps[2];  // <t|u_M>, or Re <u_M|g>
      const uint32_t i0 = 2 * q_lo + 2 * tid;
      const uint32_t ot[2] = {(uint32_t)gather_bits(i0, G.out_bits, n_out), (uint32_t)gather_bits(i0 + 1, G.out_bits, n_out)};
      uint32_t on = 0;
      for (uint32_t n = 0; n < 2 * NS / TPR; ++n) {  // the output index by halves, as the input's
        if ((n & 31u) == 0) on = (uint32_t)gather_bits((n + (tid & 31)) * TPR, G.out_bits, n_out);
        const uint32_t oj = __shfl_sync(0xffffffffu, on, n & 31), i = i0 + n * TPR;
#pragma unroll
        for (uint32_t z = 0; z < 2; ++z) {
          if ((i + z) & ~G.out_mask) continue;
          const float2 t = row[ot[z] ^ oj], a = out_of(i + z);
          if (fid) {
            pv[0][z] += t.x * a.x + t.y * a.y;
            pv[1][z] += t.x * a.y - t.y * a.x;
          } else {
            pv[0][z] += a.x * t.x + a.y * t.y;
          }
        }
      }
      block_sum_pair<VW, 2>(pv, ps, red, par);
      cluster_sum<CS, 2>(ps, cred, cpar);
      if (fid) {
        w0 = ps[0] * inv;
        w1 = ps[1] * inv;
        const float F = w0 * w0 + w1 * w1;
        const float wJ = 1.f / (float)A.J;
        loss_term = (1.f - F) * wJ;
        w2 = 2.f * wJ * inv;
        w3 = F * inv;
      } else {
        w0 = w1 = w2 = 0.f;
        w3 = ps[0] * inv * inv;
      }
    }
    auto seed_of = [&](uint32_t i, uint32_t o, float2 a) {  // i, its output index
      if (i & ~G.out_mask) return make_float2(0.f, 0.f);
      const float2 t = row[o];
      if (fid)  // lambda = (2/J)(F z - a t) / |u_M|
        return make_float2(w2 * (w3 * a.x - (w0 * t.x - w1 * t.y)), w2 * (w3 * a.y - (w0 * t.y + w1 * t.x)));
      return make_float2(inv * (t.x - w3 * a.x), inv * (t.y - w3 * a.y));
    };

    // ---- backward
    // u_{k-1}[., 1] at q: the history's b, or its signed copy
    auto hist_at = [&](int k, uint32_t q) {
      if (k == 0) return hist[q];
      const int p = k % W, pp = p ? p - 1 : W - 2;
      const uint32_t mask = s_mask[k - 1];
      const float2 h = hist_of(k)[wide_remove_bit(q, pp)];
      if (!((q >> pp) & 1u)) return h;
      if (mask & kDead) return make_float2(0.f, 0.f);
      return flip_sign(h, sign_of(wide_insert_bit(q, p) | (1u << p), mask));
    };
    auto prefetch = [&](int k) {  // the block's part of a history
      const char *h = reinterpret_cast<const char *>(hist_of(k) + h_lo);
      for (uint32_t o = tid * 128u; o < (uint32_t)NS * 4u; o += BT * 128u)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(h + o));
    };
    // mu_k and lambda_{k-1} = al mu_k of a pair of lambda_k (a and b, and their
    // copies conj(cn) a, conj(cn) b): al and the signs ride on the factors, exact
    auto pair_back = [&](float2 a, float2 b, float2 cn, float2 acn, float al, bool dead, uint32_t s0, uint32_t s1,
                         float2 &m0, float2 &m1) {
      m0 = times(al, a);
      m1 = conj_mul(acn, a);
      if (!dead) {
        const float2 cb = conj_mul(cn, b);
        const float f0 = sign_f(al, s0), f1 = sign_f(al, s1);
        m0 = make_float2(fmaf(f0, b.x, m0.x), fmaf(f0, b.y, m0.y));
        m1 = make_float2(fmaf(f1, cb.x, m1.x), fmaf(f1, cb.y, m1.y));
      }
    };
    // the warps' sums of a step's gradient terms, added up at the run's end; the
    // barrier orders the window (all: between the cluster's blocks as well)
    auto finish = [&](int k, const float (&t)[2][2], int p, bool all) {
      float *pk = reinterpret_cast<float *>(part + ((size_t)k * CS + crank) * VW);
      warp_sums_pair<2>(t, p, [&](int j, int w, float a) { pk[2 * w + j] = a; });
      if (CS > 1 && all)
        run_barrier<CS>();
      else
        __syncthreads();
    };
    {  // the last step, from the seed
      const int k = M - 1;
      const float al = RealBits<float>::pow2(-s_expo[k]);
      float t[2][2] = {};
      uint32_t ot[2], on = 0;
#pragma unroll
      for (uint32_t z = 0; z < 2; ++z)
        ot[z] = (uint32_t)gather_bits(wide_insert_bit(q_lo + 2 * tid + z, pl), G.out_bits, n_out);
      const uint32_t op = (uint32_t)gather_bits(1u << pl, G.out_bits, n_out);
      for (uint32_t n = 0; n < NS / TPR; ++n) {
        const uint32_t q = q_lo + 2 * tid + n * TPR;
        if ((n & 31u) == 0)
          on = (uint32_t)gather_bits(wide_insert_bit((n + (tid & 31)) * TPR, pl), G.out_bits, n_out);
        const uint32_t oj = __shfl_sync(0xffffffffu, on, n & 31);
        float2 m[2];
#pragma unroll
        for (uint32_t z = 0; z < 2; ++z) {
          const uint32_t i0 = wide_insert_bit(q + z, pl), i1 = i0 | (1u << pl);
          const float2 v = *now(q + z);
          m[z] = seed_of(i0, ot[z] ^ oj, v);
          if (!dead_l) {
            const uint32_t s1 = sign_of(i1, mask_l);
            m[z] = plus(m[z], seed_of(i1, ot[z] ^ oj ^ op, flip_sign(v, s1)), s1);
          }
          m[z] = times(al, m[z]);
          add_t(t, z, m[z], hist_at(k, q + z));
        }
        *home(q) = m[0];
        *home(q + 1) = m[1];
      }
      if (k > 1) prefetch(k - 1);
      finish(k, t, 0, true);
    }
    moved = false;
    // lambda of step k, pairs on bit p (below w - 1), the sums to follow
    auto bwd = [&](auto &&src, auto &&dst, int k, float al, float2 cn, float2 acn, uint32_t mask) {
      constexpr int CNT = NS / 2 / BT, U = CNT < Cfg::U ? CNT : Cfg::U;
      const int p = k % W;
      const uint32_t low = (1u << p) - 1u, r0 = h_lo + tid, qt = wide_insert_bit(r0, p);
      const bool dead = (mask & kDead) != 0u;
      const uint32_t z1 = ((mask >> (p + 1)) & 1u) << 31;
      const uint32_t st = sign_of(((r0 >> p) << (p + 2)) | (r0 & low) | (1u << p), mask);
      for (int n = 0; n < CNT; n += U) {
        float2 x[U], y[U];
#pragma unroll
        for (int j = 0; j < U; ++j) {
          const uint32_t q0 = qt | wide_insert_bit((uint32_t)(n + j) * BT, p);
          x[j] = *src(q0);
          y[j] = *src(q0 | (1u << p));
        }
#pragma unroll
        for (int j = 0; j < U; ++j) {
          const uint32_t rn = (uint32_t)(n + j) * BT, q0 = qt | wide_insert_bit(rn, p);
          const uint32_t s0 = st ^ sign_of(((rn >> p) << (p + 2)) | (rn & low), mask);
          float2 m0, m1;
          pair_back(x[j], y[j], cn, acn, al, dead, s0, s0 ^ z1, m0, m1);
          *dst(q0) = m0;
          *dst(q0 | (1u << p)) = m1;
        }
      }
    };
    for (int k = M - 2; k >= 0; --k) {
      const float al = RealBits<float>::pow2(-s_expo[k]);
      const float2 cn = s_coef[k + 1], acn = times(al, cn);
      const uint32_t mask = s_mask[k];
      const bool dead = (mask & kDead) != 0u;
      const int p = k % W;
      float t[2][2] = {};
      const bool next_joins = p == 0 || p - 1 >= SB;  // step k - 1 reaches into other slices
      if (k > 1) prefetch(k - 1);
      if (p == W - 1) {  // the slots move
        for (uint32_t m = h_lo + tid; m < h_lo + NS / 2; m += BT) {
          const float2 a = *any(m), b = *any(m | (N / 2));
          const float2 h0 = hist_at(k, 2 * m), h1 = hist_at(k, 2 * m + 1);
          const uint32_t s0 = sign_of((2 * m) | (1u << (W - 1)), mask);
          float2 m0, m1;
          pair_back(a, b, cn, acn, al, dead, s0, s0 ^ ((mask & 1u) << 31), m0, m1);
          add_t(t, 0, m0, h0);
          add_t(t, 1, m1, h1);
          *reinterpret_cast<float4 *>(scr(2 * m)) = make_float4(m0.x, m0.y, m1.x, m1.y);
        }
        moved = true;
        finish(k, t, 0, true);
      } else if (p < LT) {
        auto direct = [&](auto first) {
          constexpr int CNT = NS / 2 / BT, U = CNT < Cfg::U ? CNT : Cfg::U;
          const int pp = p ? p - 1 : W - 2;
          const uint32_t low = (1u << p) - 1u, r0 = h_lo + tid, qt = wide_insert_bit(r0, p);
          const uint32_t z1 = ((mask >> (p + 1)) & 1u) << 31;
          const uint32_t it = ((r0 >> p) << (p + 2)) | (r0 & low) | (1u << p);
          const uint32_t st = sign_of(it, mask);
          const float2 *hk = hist_of(k) + (first.value ? qt : wide_remove_bit(qt, pp));
          const uint32_t hp = first.value ? 1u << p : wide_remove_bit(1u << p, pp);
          const uint32_t hm = first.value ? 0u : s_mask[k - 1];
          const uint32_t hz = ((hm >> (p + 1)) & 1u) << 31;
          const uint32_t ht = sign_of(it, hm);
          const float live = (hm & kDead) ? 0.f : 1.f;
          const uint32_t l0 = wide_place(qt & (NS - 1)), lp = wide_place(1u << p);
          for (int n = 0; n < CNT; n += U) {
            float2 x[U], y[U], h0[U], h1[U];
#pragma unroll
            for (int j = 0; j < U; ++j) {
              const uint32_t qn = wide_insert_bit((uint32_t)(n + j) * BT, p);
              const uint32_t hn = first.value ? qn : wide_remove_bit(qn, pp);
              h0[j] = hk[hn];
              h1[j] = hk[hn | hp];
              const uint32_t e = l0 ^ wide_place(qn);
              float2 *hb = slice_at(qn);
              x[j] = hb[e];
              y[j] = hb[e ^ lp];
            }
#pragma unroll
            for (int j = 0; j < U; ++j) {
              const uint32_t rn = (uint32_t)(n + j) * BT, q0 = qt | wide_insert_bit(rn, p);
              const uint32_t in_ = ((rn >> p) << (p + 2)) | (rn & low);
              const uint32_t s0 = st ^ sign_of(in_, mask);
              float2 m0, m1;
              pair_back(x[j], y[j], cn, acn, al, dead, s0, s0 ^ z1, m0, m1);
              float f0 = 1.f, f1 = 1.f;
              if constexpr (!first.value) {
                if ((q0 >> pp) & 1u) {  // the copy on the entered qubit's bit
                  f0 = sign_f(live, ht ^ sign_of(in_, hm));
                  f1 = sign_f(f0, hz);
                }
              }
              add_ts(t, 0, m0, h0[j], f0);
              add_ts(t, 1, m1, h1[j], f1);
              const uint32_t e = l0 ^ wide_place(wide_insert_bit(rn, p));
              float2 *hb = slice_at(wide_insert_bit(rn, p));
              hb[e] = m0;
              hb[e ^ lp] = m1;
            }
          }
        };
        if (k == 0)
          direct(Yes{});
        else
          direct(No{});
        finish(k, t, p, next_joins);
      } else if (p < SB && p < LT + 3) {
        // the two entries of a pair are 2^G apart in one thread's order: groups of
        // 2^(G + 1) of its entries, two threads' worth (v = 2 tid, 2 tid + 1) at once
        auto ordered = [&](auto gc, auto &&src) {
          constexpr int GB = decltype(gc)::value, P = 1 << GB, CNT = NS / TPR / (2 * P);
          constexpr int pb = LT + GB;  // p
          const uint32_t v0 = q_lo + 2 * tid, hm = s_mask[k - 1];
          const uint32_t zz = (mask & 1u) << 31, z1 = ((mask >> (pb + 1)) & 1u) << 31;
          const uint32_t hz = (hm & 1u) << 31, h1 = ((hm >> (pb + 1)) & 1u) << 31;
          const uint32_t it = wide_insert_bit(v0, pb) | (1u << pb), st = sign_of(it, mask), ht = sign_of(it, hm);
          const float live = (hm & kDead) ? 0.f : 1.f;
          const float4 *hk = reinterpret_cast<const float4 *>(hist_of(k)) + (wide_remove_bit(v0, pb - 1) >> 1);
          for (int gi = 0; gi < CNT; ++gi) {
            float4 x[2 * P], h[2 * P];
#pragma unroll
            for (int j = 0; j < 2 * P; ++j) {
              const uint32_t qn = (uint32_t)(gi * 2 * P + j) * TPR;
              h[j] = hk[wide_remove_bit(qn, pb - 1) >> 1];
              x[j] = *reinterpret_cast<const float4 *>(src(v0 | qn));
            }
#pragma unroll
            for (int j = 0; j < P; ++j) {
              const uint32_t qn = (uint32_t)(gi * 2 * P + j) * TPR;
              const uint32_t s0 = st ^ sign_of(wide_insert_bit(qn, pb), mask);
              float2 m0, m1;
              pair_back(make_float2(x[j].x, x[j].y), make_float2(x[j + P].x, x[j + P].y), cn, acn, al, dead, s0, s0 ^ z1, m0,
                        m1);
              float2 n0, n1;
              pair_back(make_float2(x[j].z, x[j].w), make_float2(x[j + P].z, x[j + P].w), cn, acn, al, dead, s0 ^ zz,
                        s0 ^ z1 ^ zz, n0, n1);
              x[j] = make_float4(m0.x, m0.y, n0.x, n0.y);
              x[j + P] = make_float4(m1.x, m1.y, n1.x, n1.y);
              *reinterpret_cast<float4 *>(home(v0 | qn)) = x[j];
              *reinterpret_cast<float4 *>(home(v0 | qn | (1u << pb))) = x[j + P];
            }
#pragma unroll
            for (int j = 0; j < 2 * P; ++j) {
              const uint32_t qn = (uint32_t)(gi * 2 * P + j) * TPR;
              float f0 = 1.f, f1 = 1.f;
              if (((v0 | qn) >> (pb - 1)) & 1u) {
                f0 = sign_f(live, ht ^ sign_of(wide_insert_bit(qn & ~(1u << pb), pb), hm) ^ (j >= P ? h1 : 0u));
                f1 = sign_f(f0, hz);
              }
              add_ts(t, 0, make_float2(x[j].x, x[j].y), make_float2(h[j].x, h[j].y), f0);
              add_ts(t, 1, make_float2(x[j].z, x[j].w), make_float2(h[j].z, h[j].w), f1);
            }
          }
        };
        auto in_order = [&](auto gc) {
          if constexpr (LT + decltype(gc)::value < SB) {
            if (CS == 1 && moved)
              ordered(gc, scr);
            else
              ordered(gc, home);
          }
        };
        if (p == LT)
          in_order(std::integral_constant<int, 0>{});
        else if (p == LT + 1)
          in_order(std::integral_constant<int, 1>{});
        else
          in_order(std::integral_constant<int, 2>{});
        moved = false;
        finish(k, t, 0, next_joins);
      } else {
        bool joined = false;
        if constexpr (CS > 1) {
          if (p >= SB) {  // after the slots moved (p = w - 2), always
            joined = true;
            if (moved)
              bwd(scr, any, k, al, cn, acn, mask);
            else
              bwd(any, any, k, al, cn, acn, mask);
            run_barrier<CS>();
          }
        }
        if (!joined) {
          if (CS == 1 && moved)
            bwd(scr, home, k, al, cn, acn, mask);
          else
            bwd(home, home, k, al, cn, acn, mask);
          __syncthreads();
        }
        moved = false;
        constexpr int CNT = NS / TPR, U = CNT < Cfg::U ? CNT : Cfg::U;
        const int pp = p - 1;  // >= 1
        const uint32_t hm = s_mask[k - 1], r0 = q_lo + 2 * tid;
        const uint32_t hz = (hm & 1u) << 31;
        const float live = (hm & kDead) ? 0.f : 1.f;
        const uint32_t ht = sign_of(wide_insert_bit(r0, p) | (1u << p), hm);
        const float4 *hk = reinterpret_cast<const float4 *>(hist_of(k));
        for (int n = 0; n < CNT; n += U) {
          float4 x[U], h[U];
#pragma unroll
          for (int j = 0; j < U; ++j) {
            const uint32_t q = r0 + (uint32_t)(n + j) * TPR;
            h[j] = hk[wide_remove_bit(q, pp) >> 1];
            x[j] = *reinterpret_cast<const float4 *>(home(q));
          }
#pragma unroll
          for (int j = 0; j < U; ++j) {
            const uint32_t qn = (uint32_t)(n + j) * TPR, q = r0 + qn;
            float f0 = 1.f, f1 = 1.f;
            if ((q >> pp) & 1u) {
              f0 = sign_f(live, ht ^ sign_of(wide_insert_bit(qn, p), hm));
              f1 = sign_f(f0, hz);
            }
            add_ts(t, 0, make_float2(x[j].x, x[j].y), make_float2(h[j].x, h[j].y), f0);
            add_ts(t, 1, make_float2(x[j].z, x[j].w), make_float2(h[j].z, h[j].w), f1);
          }
        }
        finish(k, t, 0, next_joins);
      }
    }
    run_barrier<CS>();
    if (crank == 0) {
      for (int k = tid; k < M; k += BT) {
        const int ai = s_aidx[k];
        if (ai < 0) continue;
        const float2 c = s_coef[k];
        const float2 *pk = part + (size_t)k * CS * VW;
        float2 t01 = make_float2(0.f, 0.f);  // scaled by alpha_k
        for (int rk = 0; rk < CS; ++rk) {
          float2 u = make_float2(0.f, 0.f);
          for (int w = 0; w < VW; ++w) {
            u.x += pk[rk * VW + w].x;
            u.y += pk[rk * VW + w].y;
          }
          t01.x += u.x;
          t01.y += u.y;
        }
        const double g = (double)c.x * t01.y + (double)c.y * t01.x;  // alpha Im(c t)
        if (fid)
          atomicAdd(&A.grad[vrow * NA + ai], g);
        else
          A.grad[run * NA + ai] = g;
      }
    }
    if (tid == 0 && crank == 0) {
      if (fid) atomicAdd(&A.loss[vrow], (double)loss_term);
      if (A.status) A.status[run] = MBQC_RUN_OK;
    }
    run_barrier<CS>();  // the next run overwrites the window, the coefficients and the exponents
  }
}

// 1,024-entry pieces of a block's slice of the window that fit beside its
// tables (windows 15 and up).
int wide_adj_resident(int w, int M, bool gen, int cluster, size_t limit) {
  if (w <= 14 || gen) return 0;
  const size_t base = wide_smem_bytes(w, M, gen) + 64;
  const size_t pieces = ((size_t)1 << (w - 11)) / (size_t)cluster;
  const size_t room = limit > base ? (limit - base) / 8192 : 0;
  return (int)(pieces < room ? pieces : room);
}

template <typename K>
static int wide_launch(K k, const SvAdjArgs &a, const WideAdjGeom &g, const AdjLaunch &l, int threads, int cs,
                       cudaStream_t s) {
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)l.smem) != cudaSuccess)
    return fail(MBQC_E_UNSUPPORTED, "adjoint: %zu bytes of shared memory per block", l.smem);
  if (l.query) {
    int occ = 0;
    int rc = cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, threads, l.smem), "occupancy");
    if (rc) return rc;
    *l.occ = occ;
    return MBQC_OK;
  }
  if (cs == 1) {
    k<<<l.blocks, threads, l.smem, s>>>(a, g);
  } else {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(l.blocks * cs);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = l.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const int rc = cuda_check(cudaLaunchKernelEx(&cfg, k, a, g), "sv_adj_wide cluster launch");
    if (rc) return rc;
  }
  return check_launch("sv_adj_wide");
}

template <int W, int CS>
static int wide_half(const SvAdjArgs &a, const WideAdjGeom &g, const AdjLaunch &l, cudaStream_t s) {
  using Cfg = WideHalfCfg<W, CS>;
  if constexpr (!Cfg::kWs) {
    return wide_launch(sv_adj_wide<W, CS, true>, a, g, l, Cfg::BT, CS, s);
  } else {
    if constexpr (Cfg::NS <= 16384)
      if (g.res == Cfg::NS / 1024) return wide_launch(sv_adj_wide<W, CS, true>, a, g, l, Cfg::BT, CS, s);
    return wide_launch(sv_adj_wide<W, CS, false>, a, g, l, Cfg::BT, CS, s);
  }
}

template <int W>
static int wide_pick(const SvAdjArgs &a, const WideAdjGeom &g, const AdjLaunch &l, cudaStream_t s, bool gen) {
  if (gen) return wide_launch(sv_adj_wide_gen<W>, a, g, l, WideAdjCfg<W>::TPR, 1, s);
  if constexpr (W >= 9) {
    if constexpr (WideAdjCfg<W>::kWs) {
      if (g.cluster == 4) return wide_half<W, 4>(a, g, l, s);
      if (g.cluster == 2) return wide_half<W, 2>(a, g, l, s);
    }
    return wide_half<W, 1>(a, g, l, s);
  }
  return fail(MBQC_E_UNSUPPORTED, "adjoint: window %d takes the register kernel", W);
}

int wide_adj_threads(int w) { return w <= 9 ? 128 : (w == 10 ? 256 : (w == 11 ? 512 : 1024)); }
size_t wide_adj_smem(int w, int M, bool gen) { return wide_smem_bytes(w, M, gen); }

int launch_sv_adj_wide(const SvAdjArgs &a, const WideAdjGeom &g, const AdjLaunch &l, cudaStream_t s, bool gen) {
  switch (a.W) {
    case 1: return wide_pick<1>(a, g, l, s, gen);
    case 2: return wide_pick<2>(a, g, l, s, gen);
    case 3: return wide_pick<3>(a, g, l, s, gen);
    case 4: return wide_pick<4>(a, g, l, s, gen);
    case 5: return wide_pick<5>(a, g, l, s, gen);
    case 6: return wide_pick<6>(a, g, l, s, gen);
    case 7: return wide_pick<7>(a, g, l, s, gen);
    case 8: return wide_pick<8>(a, g, l, s, gen);
    case 9: return wide_pick<9>(a, g, l, s, gen);
    case 10: return wide_pick<10>(a, g, l, s, gen);
    case 11: return wide_pick<11>(a, g, l, s, gen);
    case 12: return wide_pick<12>(a, g, l, s, gen);
    case 13: return wide_pick<13>(a, g, l, s, gen);
    case 14: return wide_pick<14>(a, g, l, s, gen);
    case 15: return wide_pick<15>(a, g, l, s, gen);
    case 16: return wide_pick<16>(a, g, l, s, gen);
    case 17: return wide_pick<17>(a, g, l, s, gen);
    case 18: return wide_pick<18>(a, g, l, s, gen);
    case 19: return wide_pick<19>(a, g, l, s, gen);
    case 20: return wide_pick<20>(a, g, l, s, gen);
    default: return fail(MBQC_E_UNSUPPORTED, "adjoint: window %d", a.W);
  }
}

}  // namespace mbqc
