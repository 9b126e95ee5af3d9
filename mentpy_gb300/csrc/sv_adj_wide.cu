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
// memory (w <= 14) or in its workspace slot (w >= 15).  The forward pass writes the pre-step
// half-state u_{k-1}[., 1] of every step to the slot's history (2^(w-1)
// complex64 per step) and the backward pass reads it back: one forward, one
// backward, no recompute.  The grid is persistent (a workspace slot per
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

// XY, X and Y plans, windows 9..20.  A block's TPR threads of the chain's sums
// are its BT = TPR / 2 threads, each two of them: a thread takes the pairs q and
// q + 1 (q even) of every TPR, so the window and the history move in 16-byte
// accesses and an address, a sign parity and a residency test serve two pairs.
//
// What bounds it at w = 17 (64 runs of the 16 x 10 grid, a cluster of two blocks
// a run) is the traffic between the L2 and the SMs, ~6 TB/s:
//   * two forward steps a pass where both pair entries of the block's slice: the
//     window moves once for both, one barrier.  The second step takes no scale
//     of its own (scales are exact powers of two: the results keep their bits);
//     the last step's norm is a result, so that step is a pass of its own;
//   * what fits of the slice stays in the block's shared memory (at(): 27 of 64
//     pieces of 1,024 entries), the rest in the slot.  Steps on the top bits of
//     a shared run pair entries of two blocks through distributed shared memory;
//   * the gradient's FP64 products are made for all steps at the run's end.
// One pair a thread and step at a time, the window of w >= 15 in the slot, against
// this (10 columns): w = 17, 64 runs 5.91 -> 4.98 ms; w = 15, 60 runs 1.37 -> 0.87;
// w = 12, 512 runs 1.09 -> 0.60; w = 10, 1,024 runs 0.35 -> 0.21 ms.
// The sums keep that kernel's order (its threads' pairs by n, a warp's lanes as
// a butterfly, the warps in turn, the cluster's blocks in turn): the same bits.
template <int W, int CS> struct WideVecCfg {
  static constexpr int D = 1 << W;
  static constexpr int TPR = W <= 9 ? 128 : (W == 10 ? 256 : (W == 11 ? 512 : 1024));
  static constexpr int BT = TPR / 2, VW = TPR / 32;
  static constexpr bool kWs = W > 14;
  static constexpr int QS = D / 2 / CS, DS = D / CS, NIT = QS / TPR;
  static constexpr int U = kWs ? (NIT < 4 ? NIT : 4) : 2;  // items in flight
  static constexpr int LOGCS = CS == 4 ? 2 : (CS == 2 ? 1 : 0);
  static constexpr int MINB = kWs ? 1 : 1024 / BT;
  static_assert(W >= 9 && QS % TPR == 0 && NIT % U == 0 && NIT >= 2, "pairs per thread");
  static_assert(CS == 1 || kWs, "clusters share a run only with the window in the workspace");
};

// Sum of NV values of 2 BT virtual threads (v[j][0], v[j][1]: those of 2 t and
// 2 t + 1), in the order of block_sum over TPR threads.
template <int VW, int NV>
__device__ __forceinline__ void block_sum_vec(const float (&v)[NV][2], float (&out)[NV], float *red, int &par) {
  float *r = red + par * (VW * 4);
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    float a = v[j][0], b = v[j][1];
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 15) == 0) r[(threadIdx.x >> 4) * 4 + j] = a + b;
  }
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

template <int W, int CS>
__global__ void __launch_bounds__((WideVecCfg<W, CS>::BT), (WideVecCfg<W, CS>::MINB))
    sv_adj_wide(SvAdjArgs A, WideAdjGeom G) {
  using Cfg = WideVecCfg<W, CS>;
  constexpr int D = Cfg::D, TPR = Cfg::TPR, BT = Cfg::BT, VW = Cfg::VW, H2 = D / 2, QS = Cfg::QS, DS = Cfg::DS,
                NIT = Cfg::NIT, U = Cfg::U, LOGCS = Cfg::LOGCS;
  __shared__ float cred[8];
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
  off += wide_al((size_t)2 * VW * 4 * sizeof(float));

  int crank = 0, cid = blockIdx.x, ncl = gridDim.x, cpar = 0;
  if constexpr (CS > 1) {
    crank = (int)cooperative_groups::this_cluster().block_rank();
    cid = blockIdx.x / CS;
    ncl = gridDim.x / CS;
  }
  const uint32_t q_lo = (uint32_t)crank * QS, i_lo = (uint32_t)crank * DS;
  float2 *slot = reinterpret_cast<float2 *>(A.ckpt) + (size_t)cid * G.slot_elems;
  float2 *hist = slot + (Cfg::kWs ? D : 0);
  float2 *swin = reinterpret_cast<float2 *>(smem + (Cfg::kWs ? off : 0));
  float2 *gown = slot + i_lo;
  const uint32_t res = (uint32_t)G.res;
  auto at = [&](uint32_t i) -> float4 * {  // entries i, i + 1 (i even) of this block's slice
    const uint32_t local = i & (DS - 1);
    if constexpr (!Cfg::kWs) return reinterpret_cast<float4 *>(swin + local);
    return reinterpret_cast<float4 *>(((local >> 10) < res ? swin : gown) + local);
  };
  auto at_any = [&](uint32_t i) -> float4 * {  // of any block's
    if constexpr (CS == 1) return at(i);
    const uint32_t local = i & (DS - 1);
    if ((local >> 10) >= res) return reinterpret_cast<float4 *>(slot + i);
    return reinterpret_cast<float4 *>(cooperative_groups::this_cluster().map_shared_rank(swin, (int)(i / DS)) + local);
  };
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
  auto phi_of = [](float2 u0, float2 u1, float2 c, float al) {
    return make_float2(al * (u0.x + c.x * u1.x - c.y * u1.y), al * (u0.y + c.x * u1.y + c.y * u1.x));
  };
  auto other = [](float2 v, uint32_t odd, bool dead) {  // the entering qubit's half
    return dead ? make_float2(0.f, 0.f) : flip_sign(v, odd << 31);
  };
  auto parity = [](uint32_t v) { return (uint32_t)__popc(v) & 1u; };
  auto lo2 = [](float4 v) { return make_float2(v.x, v.y); };
  auto hi2 = [](float4 v) { return make_float2(v.z, v.w); };
  auto join = [](float2 a, float2 b) { return make_float4(a.x, a.y, b.x, b.y); };

  for (int64_t run = cid; run < A.B; run += ncl) {
    const int64_t vrow = fid ? run / A.J : run;
    const int64_t irow = fid ? run % A.J : (A.istride ? run : 0);
    for (int k = tid; k < M; k += BT) {
      const DevStep st = A.steps[k];
      const double th = st.aidx >= 0 ? A.angles[vrow * A.astride + st.aidx] : st.fixed;
      float2 c, ph;
      sv_coef(st.plane, th, false, c, ph);
      s_coef[k] = c;
    }
    // ---- initial window: input on its bits, |+> elsewhere, the CZ layer's signs
    const float2 *in = reinterpret_cast<const float2 *>(A.psi_in) +
                       irow * (fid ? ((int64_t)1 << n_in) : A.istride);
    float nrm;
    {
      float nv[1][2] = {{0.f, 0.f}}, sum[1];
      for (uint32_t i = i_lo + 2 * tid; i < i_lo + DS; i += TPR) {
        float2 v[2];
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          v[z] = flip_sign(in[gather_bits(i + z, G.in_bits, n_in)], init_parity(i + z, G.init_cz, W) << 31);
          nv[0][z] += v[z].x * v[z].x + v[z].y * v[z].y;
        }
        *at(i) = join(v[0], v[1]);
      }
      block_sum_vec<VW, 1>(nv, sum, red, par);
      cluster_sum<CS, 1>(sum, cred, cpar);
      nrm = sum[0];
    }

    // ---- forward, keeping every step's pre-step half-state
    for (int k = 0; k < M; ++k) {
      const int e = renorm_exponent<float>(nrm);
      const float al = RealBits<float>::pow2(-e);
      const float2 c = s_coef[k];
      const uint32_t mask = s_mask[k];
      const bool dead = (mask & kDead) != 0u;
      const int p = k % W;
      float4 *hk = reinterpret_cast<float4 *>(hist + (size_t)k * H2);
      float acc[1][2] = {{0.f, 0.f}}, sum[1];
      if (tid == 0) s_expo[k] = e;
      if (p + 1 < W - LOGCS && k + 2 < M) {
        if (tid == 0) s_expo[k + 1] = 0;
        const float2 c2 = s_coef[k + 1];
        const uint32_t mask2 = s_mask[k + 1];
        const bool dead2 = (mask2 & kDead) != 0u;
        float4 *hk2 = hk + H2 / 2;
        constexpr int U2 = NIT / 2 < U ? NIT / 2 : U;
        auto pass = [&](auto p0) {  // p0: bit 0 is measured, quads are 4 consecutive entries
          for (int b = 0; b < NIT / 2; b += U2) {
            float4 x[U2][4];
#pragma unroll
            for (int j = 0; j < U2; ++j) {
              const uint32_t r = q_lo / 2 + 2 * tid + (uint32_t)(b + j) * TPR;
              const uint32_t i = p0.value ? 4 * r : wide_insert_bit(wide_insert_bit(r, p), p + 1);
#pragma unroll
              for (int z = 0; z < 4; ++z) x[j][z] = *at(p0.value ? i + 2 * z : i | ((uint32_t)z << p));
            }
#pragma unroll
            for (int j = 0; j < U2; ++j) {
              const uint32_t r = q_lo / 2 + 2 * tid + (uint32_t)(b + j) * TPR;
              const uint32_t i = p0.value ? 4 * r : wide_insert_bit(wide_insert_bit(r, p), p + 1);
              float2 v[2][4];  // quads r, r + 1: entries (bit p) + 2 (bit p + 1)
#pragma unroll
              for (int z = 0; z < 4; ++z) {
                v[0][z] = p0.value ? ((z & 1) ? hi2(x[j][z >> 1]) : lo2(x[j][z >> 1])) : lo2(x[j][z]);
                v[1][z] = p0.value ? ((z & 1) ? hi2(x[j][2 + (z >> 1)]) : lo2(x[j][2 + (z >> 1)])) : hi2(x[j][z]);
              }
              const uint32_t h = (p0.value ? 2 * r : wide_insert_bit(r, p)) >> 1, hs = (1u << p) >> 1;
              if (p0.value) {
                hk[h] = join(v[0][1], v[0][3]);
                hk[h + 1] = join(v[1][1], v[1][3]);
              } else {
                hk[h] = join(v[0][1], v[1][1]);
                hk[h + hs] = join(v[0][3], v[1][3]);
              }
              // sign parities of the entries, those of quad r + 1 one index bit away
              const uint32_t nb = p0.value ? 4u : 1u;
              const uint32_t s1 = parity((i | (1u << p)) & mask), s3 = parity((i | (3u << p)) & mask);
              const uint32_t t2 = parity((i | (2u << p)) & mask2), t3 = parity((i | (3u << p)) & mask2);
              const uint32_t d1 = parity(nb & mask), d2 = parity(nb & mask2);
#pragma unroll
              for (int z = 0; z < 2; ++z) {
                v[z][0] = phi_of(v[z][0], v[z][1], c, al);
                v[z][2] = phi_of(v[z][2], v[z][3], c, al);
                v[z][1] = other(v[z][0], s1 ^ (z ? d1 : 0u), dead);
                v[z][3] = other(v[z][2], s3 ^ (z ? d1 : 0u), dead);
              }
              if (p0.value) {
                hk2[h] = join(v[0][2], v[0][3]);
                hk2[h + 1] = join(v[1][2], v[1][3]);
              } else {
                hk2[h] = join(v[0][2], v[1][2]);
                hk2[h + hs] = join(v[0][3], v[1][3]);
              }
#pragma unroll
              for (int z = 0; z < 2; ++z) {
                v[z][0] = phi_of(v[z][0], v[z][2], c2, 1.f);
                v[z][1] = phi_of(v[z][1], v[z][3], c2, 1.f);
                v[z][2] = other(v[z][0], t2 ^ (z ? d2 : 0u), dead2);
                v[z][3] = other(v[z][1], t3 ^ (z ? d2 : 0u), dead2);
                acc[0][z] += v[z][0].x * v[z][0].x + v[z][0].y * v[z][0].y;
                acc[0][z] += v[z][1].x * v[z][1].x + v[z][1].y * v[z][1].y;
              }
#pragma unroll
              for (int z = 0; z < 4; ++z)
                *at(p0.value ? i + 2 * z : i | ((uint32_t)z << p)) =
                    p0.value ? join(v[z >> 1][2 * (z & 1)], v[z >> 1][2 * (z & 1) + 1]) : join(v[0][z], v[1][z]);
            }
          }
        };
        if (p == 0)
          pass(Yes{});
        else
          pass(No{});
        block_sum_vec<VW, 1>(acc, sum, red, par);
        cluster_sum<CS, 1>(sum, cred, cpar);
        nrm = dead2 ? sum[0] : 2.f * sum[0];
        ++k;
        continue;
      }
      auto pass = [&](auto p0, auto &&ent) {
        for (int b = 0; b < NIT; b += U) {
          float4 x[U], y[U];  // U items loaded before any is written back
#pragma unroll
          for (int j = 0; j < U; ++j) {
            const uint32_t q = q_lo + 2 * tid + (uint32_t)(b + j) * TPR;
            const uint32_t i0 = wide_insert_bit(q, p);
            x[j] = *ent(i0);
            y[j] = *ent(p0.value ? i0 + 2 : i0 | (1u << p));
          }
#pragma unroll
          for (int j = 0; j < U; ++j) {
            const uint32_t q = q_lo + 2 * tid + (uint32_t)(b + j) * TPR;
            const uint32_t i0 = wide_insert_bit(q, p);
            const float2 ua = lo2(x[j]), va = p0.value ? hi2(x[j]) : lo2(y[j]);
            const float2 ub = p0.value ? lo2(y[j]) : hi2(x[j]), vb = hi2(y[j]);
            hk[q >> 1] = join(va, vb);
            const uint32_t s1 = parity((i0 | (1u << p)) & mask), d1 = parity((p0.value ? 2u : 1u) & mask);
            const float2 pa = phi_of(ua, va, c, al), pb = phi_of(ub, vb, c, al);
            const float2 oa = other(pa, s1, dead), ob = other(pb, s1 ^ d1, dead);
            *ent(i0) = p0.value ? join(pa, oa) : join(pa, pb);
            *ent(p0.value ? i0 + 2 : i0 | (1u << p)) = p0.value ? join(pb, ob) : join(oa, ob);
            acc[0][0] += pa.x * pa.x + pa.y * pa.y;
            acc[0][1] += pb.x * pb.x + pb.y * pb.y;
          }
        }
      };
      if (p == 0)
        pass(Yes{}, at);
      else if (CS > 1 && p >= W - LOGCS)
        pass(No{}, at_any);
      else
        pass(No{}, at);
      block_sum_vec<VW, 1>(acc, sum, red, par);
      cluster_sum<CS, 1>(sum, cred, cpar);
      nrm = dead ? sum[0] : 2.f * sum[0];
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
        for (int ai = tid; ai < NA && crank == 0; ai += BT) A.grad[run * NA + ai] = NAN;
      if (tid == 0 && crank == 0 && A.status) A.status[run] = isnan(nrm) ? MBQC_RUN_NAN : MBQC_RUN_ZERO_NORM;
      run_barrier<CS>();  // the next run overwrites the coefficients
      continue;
    }
    float loss_term = 0.f;
    if (fid) {
      const float2 *tg = reinterpret_cast<const float2 *>(A.targets) + irow * dout;
      float pv[2][2] = {}, ps[2];  // <t|u_M>
      for (uint32_t i = i_lo + 2 * tid; i < i_lo + DS; i += TPR) {
        const float4 w = *at(i);
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          if ((i + z) & ~G.out_mask) continue;
          const float2 t = tg[gather_bits(i + z, G.out_bits, n_out)], a = z ? hi2(w) : lo2(w);
          pv[0][z] += t.x * a.x + t.y * a.y;
          pv[1][z] += t.x * a.y - t.y * a.x;
        }
      }
      block_sum_vec<VW, 2>(pv, ps, red, par);
      cluster_sum<CS, 2>(ps, cred, cpar);
      const float ar = ps[0] * inv, ai = ps[1] * inv;
      const float F = ar * ar + ai * ai;
      const float wJ = 1.f / (float)A.J;
      loss_term = (1.f - F) * wJ;
      // lambda = (2/J)(F z - a t) / |u_M|
      const float k2 = 2.f * wJ * inv, fz = F * inv;
      for (uint32_t i = i_lo + 2 * tid; i < i_lo + DS; i += TPR) {
        const float4 w = *at(i);
        float2 l[2];
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          l[z] = make_float2(0.f, 0.f);
          if (!((i + z) & ~G.out_mask)) {
            const float2 t = tg[gather_bits(i + z, G.out_bits, n_out)], a = z ? hi2(w) : lo2(w);
            l[z] = make_float2(k2 * (fz * a.x - (ar * t.x - ai * t.y)), k2 * (fz * a.y - (ar * t.y + ai * t.x)));
          }
        }
        *at(i) = join(l[0], l[1]);
      }
    } else {
      const float2 *go = reinterpret_cast<const float2 *>(A.grad_out) + run * dout;
      float zv[1][2] = {{0.f, 0.f}}, zs[1];  // Re <u_M|g>
      for (uint32_t i = i_lo + 2 * tid; i < i_lo + DS; i += TPR) {
        const float4 w = *at(i);
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          if ((i + z) & ~G.out_mask) continue;
          const float2 g = go[gather_bits(i + z, G.out_bits, n_out)], a = z ? hi2(w) : lo2(w);
          zv[0][z] += a.x * g.x + a.y * g.y;
        }
      }
      block_sum_vec<VW, 1>(zv, zs, red, par);
      cluster_sum<CS, 1>(zs, cred, cpar);
      const float zgi = zs[0] * inv * inv;
      for (uint32_t i = i_lo + 2 * tid; i < i_lo + DS; i += TPR) {
        const float4 w = *at(i);
        float2 l[2];
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          l[z] = make_float2(0.f, 0.f);
          if (!((i + z) & ~G.out_mask)) {
            const float2 g = go[gather_bits(i + z, G.out_bits, n_out)], a = z ? hi2(w) : lo2(w);
            l[z] = make_float2(inv * (g.x - zgi * a.x), inv * (g.y - zgi * a.y));
          }
        }
        *at(i) = join(l[0], l[1]);
      }
    }
    run_barrier<CS>();

    // ---- backward
    for (int k = M - 1; k >= 0; --k) {
      const float al = RealBits<float>::pow2(-s_expo[k]);
      const float2 c = s_coef[k];
      const uint32_t mask = s_mask[k];
      const bool dead = (mask & kDead) != 0u;
      const int p = k % W;
      float4 *hk = reinterpret_cast<float4 *>(hist + (size_t)k * H2);
      float t[2][2] = {}, ts[2];  // sum conj(mu) u[., 1]
      auto pass = [&](auto p0, auto &&ent) {
        for (int b = 0; b < NIT; b += U) {
          float4 x[U], y[U], hh[U];  // U items and their history loaded before any is written back
#pragma unroll
          for (int j = 0; j < U; ++j) {
            const uint32_t q = q_lo + 2 * tid + (uint32_t)(b + j) * TPR;
            const uint32_t i0 = wide_insert_bit(q, p);
            hh[j] = hk[q >> 1];
            x[j] = *ent(i0);
            y[j] = *ent(p0.value ? i0 + 2 : i0 | (1u << p));
          }
#pragma unroll
          for (int j = 0; j < U; ++j) {
            const uint32_t q = q_lo + 2 * tid + (uint32_t)(b + j) * TPR;
            const uint32_t i0 = wide_insert_bit(q, p);
            const uint32_t s1 = parity((i0 | (1u << p)) & mask), d1 = parity((p0.value ? 2u : 1u) & mask);
            float2 l0[2], l1[2];
            l0[0] = lo2(x[j]);
            l1[0] = p0.value ? hi2(x[j]) : lo2(y[j]);
            l0[1] = p0.value ? lo2(y[j]) : hi2(x[j]);
            l1[1] = hi2(y[j]);
#pragma unroll
            for (int z = 0; z < 2; ++z) {
              float2 mu = l0[z];
              if (!dead) {
                const float2 m1 = flip_sign(l1[z], (s1 ^ (z ? d1 : 0u)) << 31);
                mu.x += m1.x;
                mu.y += m1.y;
              }
              const float2 h = z ? hi2(hh[j]) : lo2(hh[j]);
              t[0][z] += fmaf(mu.x, h.x, __fmul_rn(mu.y, h.y));
              t[1][z] += fmaf(mu.x, h.y, -__fmul_rn(mu.y, h.x));
              l0[z] = make_float2(al * mu.x, al * mu.y);
              l1[z] = make_float2(al * fmaf(c.y, mu.y, __fmul_rn(c.x, mu.x)),  // conj(c) mu
                                  al * fmaf(c.x, mu.y, -__fmul_rn(c.y, mu.x)));
            }
            *ent(i0) = p0.value ? join(l0[0], l1[0]) : join(l0[0], l0[1]);
            *ent(p0.value ? i0 + 2 : i0 | (1u << p)) = p0.value ? join(l0[1], l1[1]) : join(l1[0], l1[1]);
          }
        }
      };
      if (p == 0)
        pass(Yes{}, at);
      else if (CS > 1 && p >= W - LOGCS)
        pass(No{}, at_any);
      else
        pass(No{}, at);
      block_sum_vec<VW, 2>(t, ts, red, par);
      cluster_sum<CS, 2>(ts, cred, cpar);
      // kept in the history this step has finished with
      if (tid == 0 && crank == 0) hist[(size_t)k * H2] = make_float2(ts[0], ts[1]);
    }
    if (crank == 0) {
      __syncthreads();
      for (int k = tid; k < M; k += BT) {
        const int ai = s_aidx[k];
        if (ai < 0) continue;
        const float al = RealBits<float>::pow2(-s_expo[k]);
        const float2 c = s_coef[k], t01 = hist[(size_t)k * H2];
        const double g = (double)al * ((double)c.x * t01.y + (double)c.y * t01.x);  // alpha Im(c t)
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
  const size_t pieces = ((size_t)1 << (w - 10)) / (size_t)cluster;
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

template <int W>
static int wide_pick(const SvAdjArgs &a, const WideAdjGeom &g, const AdjLaunch &l, cudaStream_t s, bool gen) {
  if (gen) return wide_launch(sv_adj_wide_gen<W>, a, g, l, WideAdjCfg<W>::TPR, 1, s);
  if constexpr (W >= 9) {
    if constexpr (WideAdjCfg<W>::kWs) {
      if (g.cluster == 4) return wide_launch(sv_adj_wide<W, 4>, a, g, l, WideVecCfg<W, 4>::BT, 4, s);
      if (g.cluster == 2) return wide_launch(sv_adj_wide<W, 2>, a, g, l, WideVecCfg<W, 2>::BT, 2, s);
    }
    return wide_launch(sv_adj_wide<W, 1>, a, g, l, WideVecCfg<W, 1>::BT, 1, s);
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
