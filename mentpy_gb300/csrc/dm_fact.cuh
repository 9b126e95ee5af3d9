// Density-matrix sweep with the window's density matrix in factored form.
//
// After step k the window bit p = k mod w holds the entering qubit: |+><+|
// with CZs to its partners m_k (or |0><0| when no qubit enters, the window
// shrinking), so the full 2^w x 2^w matrix is
//     rho[x, y] = f[x_p, y_p] s(x) s(y) R[x \ p, y \ p],
//     f = 1/2 [[1, 1], [1, 1]] (|+>) or [[1, 0], [0, 0]] (|0>),
//     s(x) = (-1)^{x_p parity(x & m_k)},
// and only R, the (w-1)-qubit matrix over the other bits, is stored: a
// quarter of the memory and of the shared-memory traffic per step of the
// full matrix (w = 7: 32 KB instead of 128 KB per run), one more window
// (w = 8) within one SM's shared memory.
//
// Step k+1 measures q = (k+1) mod w with the step functional G (outcome
// projector transposed, depolarising noise folded in, as dm.cuh):
//     new[(u,a'), (v,b')] = f[a',b'] (-1)^{a' pi(u) + b' pi(v)} T_{a'b'}(u, v),
//     T_{a'b'}(u, v) = sum_{a,b} G[a,b] (-1)^{(a' a + b' b) m_q} R[(u,a), (v,b)],
// where (u, a) is the index with bit q = a (u: the bits other than p, q),
// (u, a') the index with bit p = a', pi(u) = parity(u & m_k) and m_q = bit q
// of m_k.  new / prob is the next R, stored over the bits other than q: bit
// p takes over the storage position that bit q had, so the pass is in place
// over the 2x2 blocks of that position, like the full-matrix kernel's pass
// (np_simulator_dm.py:307-346 + state_ops.py:77-119 for the measurement and
// trace, np_simulator_dm.py:151-216 for the |+> and CZs).  Step 0 forms R
// from the initial pure window state directly.
#pragma once

#include "cluster_sum.cuh"
#include "dm.cuh"

namespace mbqc {

// Windows up to 8 keep R in shared memory; windows 9..11 (R of 512 KB to
// 8 MB) keep it in a device workspace, a cluster of blocks per run.
constexpr int kDmFactSmemMaxWindow = 8;
constexpr int kDmFactMaxWindow = 11;

template <int W> struct DmFactCfg {
  static_assert(W >= 2 && W <= kDmFactMaxWindow, "factored density matrix: windows 2..11");
  static constexpr int D = 1 << (W - 1);  // side of R
  static constexpr int N = D * D;         // entries of R
  static constexpr int H = D / 2;         // block index range per side
  static constexpr int NB = N / 4;        // 2x2 blocks per step
  static constexpr int DW = 1 << W;       // amplitudes of the initial window
  static constexpr bool kSmemR = W <= kDmFactSmemMaxWindow;
  // threads per run (shared-memory windows): ~8 blocks each, one warp at
  // least, a block at most
  static constexpr int TPR = NB / 8 < 32 ? 32 : (NB / 8 > 256 ? 256 : NB / 8);
};

// Per-step word of the factored pass (staged once per run):
//   aux bits 0-3: storage position of the measured bit in R
//       bit 4: m_q (the previous entering qubit has a CZ to the measured one)
//       bit 5: the previous step's slot is |0> (no qubit entered)
//       bit 6: Z-basis step
//   sgn: the previous entering qubit's CZ partners other than the measured
//        bit, as storage positions of R
constexpr uint32_t kFactMq = 1u << 4, kFactDead = 1u << 5, kFactZ = 1u << 6;

// bytes of one run's shared-memory slice (16-byte aligned): R (when it is
// shared-memory resident), the initial window, the step tables, the
// reduction scratch (one entry per warp of the group) and the position table
template <int W> __host__ __device__ constexpr size_t dm_fact_slice_bytes(int maxm) {
  return ((DmFactCfg<W>::kSmemR ? (size_t)DmFactCfg<W>::N * 8 : 0) + (size_t)DmFactCfg<W>::DW * 8 +
          (size_t)maxm * 24 + 64 * 8 + 16 + 15) &
         ~(size_t)15;
}

// Column swizzle of R's rows (float2 index within a row): columns 16..31 of
// every 32 are stored with bits 1..3 flipped.  In a pass over storage
// position 1, 2 or 3 the eight threads of a 16-byte access phase touch the
// even (or odd) float4 slots of 16 consecutive ones, which without the
// swizzle fall on four banks twice (a two-way conflict on every access);
// flipping the slot's low three bits in the upper half of each 16 makes the
// eight slots distinct modulo 8.  Positions 0, 4, 5 touch 8 consecutive
// slots and stay conflict free.  A column pair (c, c + 1), c even, stays one
// float4.
__device__ __forceinline__ uint32_t rsw(uint32_t col) { return col ^ (((col >> 4) & 1u) * 14u); }

// group_sum2 with a double-buffered scratch: one barrier a call.  ``par``
// alternates between calls; a buffer is written again only two calls later,
// after a barrier that every reader of its previous contents has passed.
template <int TPR>
__device__ __forceinline__ float2 group_sum2_db(float v, float2 *scratch, int tid, int group, int &par) {
  float hi = v, lo = 0.f;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
    const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
    two_sum_acc(hi, lo, oh, ol);
  }
  if constexpr (TPR != 32) {
    constexpr int NW = TPR / 32;
    float2 *buf = scratch + par * 32;
    par ^= 1;
    if ((tid & 31) == 0) buf[tid >> 5] = make_float2(hi, lo);
    group_sync(TPR, group);
    float2 p = buf[0];
    hi = p.x;
    lo = p.y;
#pragma unroll
    for (int i = 1; i < NW; ++i) {
      p = buf[i];
      two_sum_acc(hi, lo, p.x, p.y);
    }
  }
  const float s = hi + lo;  // renormalise
  return make_float2(s, lo - (s - hi));
}

// Step words and final positions, every step on its own: the qubit at
// schedule index s (initial window or entering) is always stored at position
// (s - 1) mod (W - 1), since an entering qubit takes the position of the qubit
// measured W - 1 steps later than its predecessor there.  (As one thread's
// walk over the steps with a running position table this took ~10 us of a
// 66-step window-7 run.)
template <int W>
__device__ __forceinline__ void fact_tables(const DevStep *steps, int M, uint2 *sSt, int8_t *sPos, int tid, int n) {
  for (int k = tid; k < M; k += n) {
    uint32_t aux = steps[k].plane == MBQC_PLANE_Z ? kFactZ : 0u, sgn = 0u;
    if (k > 0) {
      const uint32_t pmask = steps[k - 1].mask;
      const int q = k % W;
      aux |= (uint32_t)((k - 1) % (W - 1));
      if (pmask & kDead) {
        aux |= kFactDead;
      } else {
        if ((pmask >> q) & 1u) aux |= kFactMq;
#pragma unroll
        for (int d = 1; d < W - 1; ++d)  // the qubits d places after the measured one (d = W - 1: the slot)
          if ((pmask >> ((q + d) % W)) & 1u) sgn |= 1u << ((k + d - 1) % (W - 1));
      }
    }
    sSt[k] = make_uint2(aux, sgn);
  }
  if (sPos && tid < W) sPos[tid] = (int8_t)((M + (tid + W - M % W) % W + W - 2) % (W - 1));
}

// Outputs of one 2x2 block from its entries x_ab (a: row half, b: column
// half); hA, hB, hR, hI: the functional with the step's scale folded in.
// LINKED: the slot has a CZ to the measured qubit (pdead, mq not looked at);
// SIGNED: pr, pc may be nonzero.
template <bool LINKED = false, bool SIGNED = true>
__device__ __forceinline__ void fact_combine(float hA, float hB, float hR, float hI, bool pdead, bool mq, float2 x00,
                                             float2 x01, float2 x10, float2 x11, uint32_t pr, uint32_t pc,
                                             float2 &o00, float2 &o01, float2 &o10, float2 &o11) {
  // sA = G00 x00 + G11 x11, dA = G00 x00 - G11 x11 (a == b terms)
  const float px = hA * x00.x, py = hA * x00.y;
  const float2 sA = make_float2(fmaf(hB, x11.x, px), fmaf(hB, x11.y, py));
  // sB = G01 x01 + conj(G01) x10 (a != b terms), dB = conj(G01) x10 - G01 x01
  const float2 u = make_float2(x01.x + x10.x, x01.y + x10.y), v = make_float2(x01.x - x10.x, x01.y - x10.y);
  const float2 sB = make_float2(fmaf(hR, u.x, -hI * v.y), fmaf(hR, u.y, hI * v.x));
  o00 = make_float2(sA.x + sB.x, sA.y + sB.y);
  if (!LINKED && pdead) {
    o01 = o10 = o11 = make_float2(0.f, 0.f);
    return;
  }
  if (LINKED || mq) {
    // signs (-1)^{a' a + b' b} on the terms: T01 = dA + dB, T10 = dA - dB, T11 = sA - sB
    const float2 dA = make_float2(fmaf(-hB, x11.x, px), fmaf(-hB, x11.y, py));
    const float2 dB = make_float2(fmaf(hI, u.y, -hR * v.x), fmaf(-hI, u.x, -hR * v.y));
    o01 = make_float2(dA.x + dB.x, dA.y + dB.y);
    o10 = make_float2(dA.x - dB.x, dA.y - dB.y);
    o11 = make_float2(sA.x - sB.x, sA.y - sB.y);
  } else {
    o01 = o10 = o11 = o00;
  }
  if (SIGNED) {
    o01 = flip_sign(o01, pc);
    o10 = flip_sign(o10, pr);
    o11 = flip_sign(o11, pr ^ pc);
  }
}

// One in-place pass over the 2x2 blocks of position pos.  16-byte
// shared-memory accesses: at pos 0 a block's two columns are adjacent (one
// float4 per row); at pos > 0 a unit is the two blocks of columns c0 and c0 + 1
// (one float4 per row and column half).  A thread keeps one column (pair) for
// the whole pass and walks rows, so its column index, signs and the
// row-independent address parts are computed once; all loads of U units before
// their stores (distinct units never alias).
template <int W, int TPR, bool LINKED, bool SIGNED>
__device__ __forceinline__ void fact_pass(float2 *R, int tid, int pos, float hA, float hB, float hR, float hI,
                                          bool pdead, bool mq, uint32_t sgn) {
  using Cfg = DmFactCfg<W>;
  constexpr int D = Cfg::D, H = Cfg::H;
  auto combine = [&](float2 x00, float2 x01, float2 x10, float2 x11, uint32_t pr, uint32_t pc, float2 &o00,
                     float2 &o01, float2 &o10, float2 &o11) {
    fact_combine<LINKED, SIGNED>(hA, hB, hR, hI, pdead, mq, x00, x01, x10, x11, pr, pc, o00, o01, o10, o11);
  };
  auto sign = [&](uint32_t i) { return SIGNED ? (__popc(i & sgn) & 1u) << 31 : 0u; };
  float4 *R4 = reinterpret_cast<float4 *>(R);
  if (pos == 0) {
    // H columns of blocks; thread tid: column tid % H, rows tid / H + j * (TPR / H)
    constexpr int CPT = H < TPR ? H : TPR;  // threads per row of blocks
    constexpr int RSTEP = TPR / CPT, NJ = (H + RSTEP - 1) / RSTEP;
    constexpr int U = NJ >= 4 ? 4 : NJ;
    constexpr bool ALL = NJ * RSTEP == H;  // every row index is in range
    const uint32_t c = (uint32_t)(tid % CPT), r_first = (uint32_t)(tid / CPT);
    for (int cc = (int)c; cc < H; cc += CPT) {  // one iteration unless H > TPR
      const uint32_t pc = sign(2u * (uint32_t)cc);
      const uint32_t ccs = rsw(2u * (uint32_t)cc) >> 1;  // the column pair's float4 slot in its row
      for (int j0 = 0; j0 < NJ; j0 += U) {
        float4 top[U], bot[U];
        uint32_t at[U], pr[U];
#pragma unroll
        for (int uu = 0; uu < U; ++uu) {
          const uint32_t r = r_first + (uint32_t)(j0 + uu) * RSTEP;
          if (ALL || r < (uint32_t)H) {
            at[uu] = r * D + ccs;  // float4 index of (row 2r, columns 2c, 2c + 1)
            pr[uu] = sign(2u * r);
            top[uu] = R4[at[uu]];
            bot[uu] = R4[at[uu] + D / 2];
          }
        }
#pragma unroll
        for (int uu = 0; uu < U; ++uu) {
          const uint32_t r = r_first + (uint32_t)(j0 + uu) * RSTEP;
          if (ALL || r < (uint32_t)H) {
            float2 o00, o01, o10, o11;
            combine(make_float2(top[uu].x, top[uu].y), make_float2(top[uu].z, top[uu].w),
                    make_float2(bot[uu].x, bot[uu].y), make_float2(bot[uu].z, bot[uu].w), pr[uu], pc, o00, o01,
                    o10, o11);
            R4[at[uu]] = make_float4(o00.x, o00.y, o01.x, o01.y);
            R4[at[uu] + D / 2] = make_float4(o10.x, o10.y, o11.x, o11.y);
          }
        }
      }
    }
  } else if constexpr (W >= 3) {  // window 2 has position 0 only
    // H/2 column pairs; thread tid: pair tid % HU, rows tid / HU + j * (TPR / HU)
    constexpr int HU = H / 2;
    constexpr int CPT = HU < TPR ? HU : TPR;
    constexpr int RSTEP = TPR / CPT, NJ = (H + RSTEP - 1) / RSTEP;
    constexpr int U = NJ >= 2 ? 2 : NJ;
    constexpr bool ALL = NJ * RSTEP == H;
    const uint32_t rs = ((uint32_t)D << pos) >> 1;  // row step in float4
    const uint32_t r_first = (uint32_t)(tid / CPT);
    for (int cp = tid % CPT; cp < HU; cp += CPT) {  // one iteration unless HU > TPR
      const uint32_t c0 = ins_bit(2u * (uint32_t)cp, pos, 0);  // even
      const uint32_t pc0 = sign(c0), pc1 = sign(c0 + 1u);
      // float4 slots of the column pairs (c0, c0 + 1) and (c0 + 2^pos, c0 + 2^pos + 1) in a row
      const uint32_t s0 = rsw(c0) >> 1, s1 = rsw(c0 | (1u << pos)) >> 1;
      for (int j0 = 0; j0 < NJ; j0 += U) {
        float4 q00[U], q01[U], q10[U], q11[U];
        uint32_t at[U], pr[U];
#pragma unroll
        for (int uu = 0; uu < U; ++uu) {
          const uint32_t r = r_first + (uint32_t)(j0 + uu) * RSTEP;
          if (ALL || r < (uint32_t)H) {
            const uint32_t r0 = ins_bit(r, pos, 0);
            at[uu] = (r0 * D) >> 1;  // float4 index of row r0
            pr[uu] = sign(r0);
            q00[uu] = R4[at[uu] + s0];
            q01[uu] = R4[at[uu] + s1];
            q10[uu] = R4[at[uu] + rs + s0];
            q11[uu] = R4[at[uu] + rs + s1];
          }
        }
#pragma unroll
        for (int uu = 0; uu < U; ++uu) {
          const uint32_t r = r_first + (uint32_t)(j0 + uu) * RSTEP;
          if (ALL || r < (uint32_t)H) {
            float2 a00, a01, a10, a11, b00, b01, b10, b11;
            combine(make_float2(q00[uu].x, q00[uu].y), make_float2(q01[uu].x, q01[uu].y),
                    make_float2(q10[uu].x, q10[uu].y), make_float2(q11[uu].x, q11[uu].y), pr[uu], pc0, a00, a01,
                    a10, a11);
            combine(make_float2(q00[uu].z, q00[uu].w), make_float2(q01[uu].z, q01[uu].w),
                    make_float2(q10[uu].z, q10[uu].w), make_float2(q11[uu].z, q11[uu].w), pr[uu], pc1, b00, b01,
                    b10, b11);
            R4[at[uu] + s0] = make_float4(a00.x, a00.y, b00.x, b00.y);
            R4[at[uu] + s1] = make_float4(a01.x, a01.y, b01.x, b01.y);
            R4[at[uu] + rs + s0] = make_float4(a10.x, a10.y, b10.x, b10.y);
            R4[at[uu] + rs + s1] = make_float4(a11.x, a11.y, b11.x, b11.y);
          }
        }
      }
    }
  }
}

// One run of the factored sweep by a group of TPR threads.  ``base`` is the
// group's slice of shared memory; every thread of the group calls this with
// the same slot.
template <int W, int TPR>
__device__ __forceinline__ void dm_fact_run(const DmArgs &A, int64_t slot, int tid, int group,
                                            unsigned char *base) {
  using Cfg = DmFactCfg<W>;
  constexpr int D = Cfg::D, N = Cfg::N, H = Cfg::H, NB = Cfg::NB, DW = Cfg::DW;
  float2 *R = reinterpret_cast<float2 *>(base);
  float2 *psi = R + N;
  float4 *sF = reinterpret_cast<float4 *>(psi + DW);
  uint2 *sSt = reinterpret_cast<uint2 *>(sF + A.maxm);
  float2 *sRed = reinterpret_cast<float2 *>(sSt + A.maxm);  // 2 x 32 entries (one per warp of the group)
  int8_t *sPos = reinterpret_cast<int8_t *>(sRed + 64);     // [W] storage position of each window bit
  int red_par = 0;

  const int ci = A.run_circuit ? A.run_circuit[slot] : 0;
  const int64_t run = A.run_circuit ? (int64_t)ci : slot;
  const DevCircuit &C = A.circ[ci];
  const int M = C.n_steps;
  const DevStep *steps = A.steps + C.step_off;
  if (C.w != W || M > A.maxm || M < 1 || C.map_off < 0 || !(steps[M - 1].mask & kDead)) {
    if (tid == 0 && A.status) A.status[run] = MBQC_RUN_NAN;  // the host routes such plans elsewhere
    return;
  }
  const int2 *map = A.maps + C.map_off;
  const double *ang = A.angles + run * A.astride;
  const float qn = f64_to_f32_rn(A.noise);
  const float a_n = 1.f - (4.f / 3.f) * qn, b_n = (2.f / 3.f) * qn;

  // ---- stage the step functionals (noise folded in) and the position table
  for (int k = tid; k < M; k += TPR) {
    const DevStep st = steps[k];
    const double th = st.aidx >= 0 ? ang[st.aidx] : st.fixed;
    float nx, ny, nz;
    bloch(st.plane, th, nx, ny, nz);
    sF[k] = make_float4(a_n * 0.5f * (1.f + nz) + b_n, a_n * 0.5f * (1.f - nz) + b_n, a_n * 0.5f * nx,
                        a_n * 0.5f * ny);
  }
  fact_tables<W>(steps, M, sSt, sPos, tid, TPR);
  // ---- the initial window |psi_0> (input, |+> padding, initial CZ signs)
  {
    const float2 *in = A.psi_in + (A.istride ? run * A.istride : 0);
    const float pad = exp2f(-0.5f * (float)(W - C.n_in));
    for (int i = tid; i < DW; i += TPR) {
      const int2 mi = __ldg(&map[i]);
      const float2 u = flip_sign(in[mi.x & 0x7fffffff], (uint32_t)mi.x & 0x80000000u);
      psi[i] = make_float2(pad * u.x, pad * u.y);
    }
  }
  group_sync(TPR, group);

  int32_t st_code = MBQC_RUN_OK;
  int n_rec = 0;                           // steps with a recorded probability
  const float tr_noise = a_n + 2.f * b_n;  // functional of I after noise folding
  for (int k = 0; k < M; ++k) {
    const float4 F = sF[k];
    const uint2 ss = sSt[k];
    const bool zstep = (ss.x & kFactZ) != 0u;
    const int pos = (int)(ss.x & 15u);
    const bool mq = (ss.x & kFactMq) != 0u, pdead = (ss.x & kFactDead) != 0u;
    // 1. outcome probability (what = 0): trace of the contraction (diagonal
    //    blocks), step 0 from |psi_0> over bit 0, later from R over position pos
    //    (with a |+> slot entangled to the measured qubit, the coherences of
    //    the measured qubit drop out of the trace).  what = 1: the trace, 2:
    //    prob1 = trace - prob0 term by term.  One warp reads and sums the
    //    diagonal; the barrier that hands the sum on also says that it was read.
    const bool drop_coh = k > 0 && !pdead && mq;
    auto diagonal = [&](int what) -> float2 {
      if (k == 0) {
        float p_re = 0.f, p_off = 0.f, t_re = 0.f;  // sums of G00 x00 + G11 x11, of 2 Re(G01 x01), of the trace
        for (int r = tid; r < DW / 2; r += TPR) {
          const float2 u0 = psi[2 * r], u1 = psi[2 * r + 1];
          const float q00 = u0.x * u0.x + u0.y * u0.y, q11 = u1.x * u1.x + u1.y * u1.y;
          p_re += F.x * q00 + F.y * q11;
          // x01 = psi0 conj(psi1)
          p_off += 2.f * (F.z * (u0.x * u1.x + u0.y * u1.y) - F.w * (u0.y * u1.x - u0.x * u1.y));
          t_re += q00 + q11;
        }
        return group_sum2_db<TPR>(what == 0 ? p_re + p_off : what == 1 ? t_re : tr_noise * t_re - p_re - p_off, sRed,
                                  tid, group, red_par);
      }
      constexpr int L = H < 32 ? H : 32;  // lanes with a term of their own (the others repeat them)
      float hi = 0.f, lo = 0.f;
      if (tid < 32) {
#pragma unroll
        for (int r = tid & (L - 1), n = 0; n < H / L; r += L, ++n) {
          const uint32_t i0 = ins_bit(r, pos, 0), i1 = i0 | (1u << pos);
          const float2 q00 = R[i0 * D + rsw(i0)], q11 = R[i1 * D + rsw(i1)];
          const float p_re = F.x * q00.x + F.y * q11.x, t_re = q00.x + q11.x;
          float v;
          if (what == 1) {
            v = t_re;
          } else if (drop_coh) {
            v = what == 0 ? p_re : tr_noise * t_re - p_re;
          } else {
            const float2 q01 = R[i0 * D + rsw(i1)];
            const float p_off = 2.f * (F.z * q01.x - F.w * q01.y);
            v = what == 0 ? p_re + p_off : tr_noise * t_re - p_re - p_off;
          }
          two_sum_acc(hi, lo, v, 0.f);
        }
#pragma unroll
        for (int o = L / 2; o >= 1; o >>= 1) {
          const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
          const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
          two_sum_acc(hi, lo, oh, ol);
        }
        const float sum = hi + lo;  // renormalise
        lo = lo - (sum - hi);
        hi = sum;
      }
      if constexpr (TPR > 32) {
        float2 *buf = sRed + red_par * 32;
        red_par ^= 1;
        if (tid == 0) *buf = make_float2(hi, lo);
        group_sync(TPR, group);
        return *buf;
      }
      return make_float2(hi, lo);
    };
    float2 prob = diagonal(0);
    float4 G = F;
    int outcome = 0;
    bool take1 = false;
    bool unprojected = false;
    if (zstep) {
      const float2 tot = diagonal(1);
      if (A.flags & MBQC_F_DM_EXPECTATION) {
        if (tid == 0) sF[k] = make_float4(prob.x, prob.y, tot.x, tot.y);
        G = make_float4(1.f, 1.f, 0.f, 0.f);
        prob = make_float2(1.f, 0.f);
        outcome = 2;
        unprojected = true;
      } else {
        take1 = !(draw_uniform(A.seed, run, k) * tot.x < prob.x);
      }
    } else {
      take1 = !pair_ge(prob, 1e-4);  // prob0 < 1e-4 (or NaN): outcome 1 (np_simulator_dm.py:335-338)
    }
    if (take1) {  // outcome 1 with P1 = I - P0
      G = make_float4(tr_noise - F.x, tr_noise - F.y, -F.z, -F.w);
      const float2 prob1 = diagonal(2);
      if (tid == 0) sF[k] = make_float4(prob.x, prob.y, kNoTrace, 0.f);
      prob = prob1;
      outcome = 1;
    } else if (tid == 0 && !unprojected) {
      sF[k] = make_float4(prob.x, prob.y, kNoTrace, 0.f);
    }
    n_rec = k + 1;
    if (tid == 0 && A.outcomes) A.outcomes[run * A.ostride + k] = (int8_t)outcome;
    if (!(prob.x > 0.f) || isnan(prob.x) || isinf(prob.x)) {  // the reference's NaN check
      st_code = MBQC_RUN_NAN;
      break;
    }
    float inv = __frcp_rn(prob.x);        // correctly rounded 1/hi
    inv = fmaf(-inv * inv, prob.y, inv);  // 1/(hi + lo) to first order in lo
    // G01 as the coefficient of x01; x10 takes its conjugate
    const float g00 = G.x, g11 = G.y, gr = G.z, gi = G.w;
    if (k == 0) {
      // R = (1/prob) sum_{a,b} G[a,b] psi(x', a) conj(psi(y', b)) over bits 1..w-1
      for (int e = tid; e < N; e += TPR) {
        const int x = e / D, y = e % D;
        const float2 u0 = psi[2 * x], u1 = psi[2 * x + 1], v0 = psi[2 * y], v1 = psi[2 * y + 1];
        // x_ab = psi(x,a) conj(psi(y,b))
        const float2 x00 = make_float2(u0.x * v0.x + u0.y * v0.y, u0.y * v0.x - u0.x * v0.y);
        const float2 x11 = make_float2(u1.x * v1.x + u1.y * v1.y, u1.y * v1.x - u1.x * v1.y);
        const float2 x01 = make_float2(u0.x * v1.x + u0.y * v1.y, u0.y * v1.x - u0.x * v1.y);
        const float2 x10 = make_float2(u1.x * v0.x + u1.y * v0.y, u1.y * v0.x - u1.x * v0.y);
        const float sr = g00 * x00.x + g11 * x11.x + gr * (x01.x + x10.x) - gi * (x01.y - x10.y);
        const float si = g00 * x00.y + g11 * x11.y + gr * (x01.y + x10.y) + gi * (x01.x - x10.x);
        R[x * D + rsw((uint32_t)y)] = make_float2(sr * inv, si * inv);
      }
      group_sync(TPR, group);
      continue;
    }
    // every thread has read the diagonal before it changes: the barrier of the
    // probability sum above follows each thread's reads (a warp-sized group
    // syncs here)
    if constexpr (TPR == 32) group_sync(TPR, group);
    // 2. the pass, the scale folded into the functional.  Slots of circuits
    //    with a causal flow are linked to the measured qubit, and on wires to no
    //    other: those passes are straight-line code without sign operations
    //    (the general one spent ~460 of its 770 warp instructions a step beside
    //    the arithmetic)
    const uint32_t sgn = ss.y;
    const float half = pdead ? inv : 0.5f * inv;
    const float hA = g00 * half, hB = g11 * half, hR = gr * half, hI = gi * half;
    if (mq && !pdead) {
      if (sgn == 0u)
        fact_pass<W, TPR, true, false>(R, tid, pos, hA, hB, hR, hI, pdead, mq, sgn);
      else
        fact_pass<W, TPR, true, true>(R, tid, pos, hA, hB, hR, hI, pdead, mq, sgn);
    } else {
      fact_pass<W, TPR, false, true>(R, tid, pos, hA, hB, hR, hI, pdead, mq, sgn);
    }
    group_sync(TPR, group);
  }

  // ---- output noise (each output qubit once, on its storage position)
  if (st_code == MBQC_RUN_OK && qn != 0.f) {
    for (int j = 0; j < C.n_out; ++j) {
      const int pos = sPos[C.out_bits[j]];
      for (int e = tid; e < NB; e += TPR) {
        const uint32_t r = (uint32_t)e / H, c = (uint32_t)e % H;
        const uint32_t r0 = ins_bit(r, pos, 0), r1 = ins_bit(r, pos, 1);
        const uint32_t c0 = ins_bit(c, pos, 0), c1 = ins_bit(c, pos, 1);
        const uint32_t c0s = rsw(c0), c1s = rsw(c1);
        const float2 x00 = R[r0 * D + c0s], x01 = R[r0 * D + c1s];
        const float2 x10 = R[r1 * D + c0s], x11 = R[r1 * D + c1s];
        const float2 tr = make_float2(x00.x + x11.x, x00.y + x11.y);
        R[r0 * D + c0s] = make_float2(a_n * x00.x + b_n * tr.x, a_n * x00.y + b_n * tr.y);
        R[r1 * D + c1s] = make_float2(a_n * x11.x + b_n * tr.x, a_n * x11.y + b_n * tr.y);
        R[r0 * D + c1s] = make_float2(a_n * x01.x, a_n * x01.y);
        R[r1 * D + c0s] = make_float2(a_n * x10.x, a_n * x10.y);
      }
      group_sync(TPR, group);
    }
  }
  // ---- gather the outputs in the reference order: output qubit j (the
  // most significant first) sits at storage position sPos[out_bits[j]]; the
  // other stored bits are |0> slots of the shrunk window
  const int n_out = C.n_out, dout = 1 << n_out;
  int *ridx = reinterpret_cast<int *>(psi);  // psi is no longer needed
  for (int y = tid; y < dout; y += TPR) {
    int ri = 0;
    for (int j = 0; j < n_out; ++j) ri |= ((y >> (n_out - 1 - j)) & 1) << sPos[C.out_bits[j]];
    ridx[y] = ri;
  }
  group_sync(TPR, group);
  if (A.probs)
    for (int k = tid; k < n_rec; k += TPR)
      A.probs[run * A.ostride + k] = prob_record(sF[k]);
  float2 *out = A.rho_out + run * A.out_stride;
  for (int e = tid; e < dout * dout; e += TPR) {
    const int yi = e >> n_out, yj = e & (dout - 1);
    out[e] = st_code == MBQC_RUN_OK ? R[ridx[yi] * D + rsw((uint32_t)ridx[yj])] : make_float2(NAN, NAN);
  }
  if (tid == 0 && A.status) A.status[run] = st_code;
  group_sync(TPR, group);  // the slice is reused by the caller's next run
}

// Windows 9 and 10 with R in the shared memory of a cluster: CS blocks of one
// run hold D / CS = 32 rows each (64 KB at window 9, eight blocks; 128 KB at
// window 10, sixteen).  Two row layouts: A deals the rows by their top
// position bits, so positions 0..4 pair rows of one block; B by their lowest
// bits, so positions 5.. do.  Steps meet the positions cyclically, so a run
// stays in a layout for 5 steps, then for n - 5: the last step before a change
// writes its rows straight to their new owners (distributed shared memory) once
// every block's loads have been released to the others.
// A step is then: one warp sums the block's diagonal pairs and sends the
// partial to every block, one cluster barrier, the pass over the block's rows.
// What bounds it is that chain (cycles a step at window 9: ~1,300 to the
// barrier's end, 250 the sum, 970 the pass, 1,400 the layout changes' share);
// the workspace kernel below pays two round trips to the L2 and the slice's
// traffic through it at every step.  Window 9, 40 steps: 228 us for 1 to 8
// runs and 325 us for 24 there, 117 and 186 us here; window 10, 36 steps, 4
// runs: 424 and 189 us.
template <int W> struct DmClCfg {
  static constexpr int N = W - 1, LB = 5, OB = N - LB, CS = 1 << OB;  // positions, local and owner row bits
  static constexpr int D = 1 << N, H = D / 2, RL = 1 << LB;
  static constexpr int BT = D * RL / 16;  // 16 entries a thread
  static constexpr int DW = 1 << W;
};

template <int W> __host__ __device__ constexpr size_t dm_cl_bytes(int maxm) {
  return (size_t)DmClCfg<W>::D * DmClCfg<W>::RL * 8 + (size_t)DmClCfg<W>::DW * 8 + (size_t)maxm * 24 +
         2 * 16 * sizeof(float2) + 32;
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <int W>
__global__ void __launch_bounds__(DmClCfg<W>::BT, 1024 / DmClCfg<W>::BT) dm_fwd_fact_cl(DmArgs A) {
  namespace cg = cooperative_groups;
  using Cfg = DmClCfg<W>;
  constexpr int N = Cfg::N, LB = Cfg::LB, OB = Cfg::OB, CS = Cfg::CS, D = Cfg::D, H = Cfg::H, RL = Cfg::RL,
                BT = Cfg::BT, DW = Cfg::DW, HU = H / 2;
  extern __shared__ __align__(16) unsigned char smem_c[];
  float2 *R = reinterpret_cast<float2 *>(smem_c);
  float4 *R4 = reinterpret_cast<float4 *>(smem_c);
  float2 *psi = R + (size_t)D * RL;
  // step k's functional is sF[k]; its probability is recorded in sF[k - 1],
  // which every thread has read by then (sF[k] is still being read)
  float4 *sF = reinterpret_cast<float4 *>(psi + DW) + 1;
  uint2 *sSt = reinterpret_cast<uint2 *>(sF + A.maxm);
  float2 *sP = reinterpret_cast<float2 *>(sSt + A.maxm);  // two buffers of a partial per block
  int8_t *sPos = reinterpret_cast<int8_t *>(sP + 32);
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, rank = (int)cl.block_rank();
  const float qn = f64_to_f32_rn(A.noise);
  const float a_n = 1.f - (4.f / 3.f) * qn, b_n = (2.f / 3.f) * qn, tr_noise = a_n + 2.f * b_n;
  int par = 0;

  // row of the matrix that local row l is in layout A / B
  auto row_of = [&](bool b, uint32_t l) { return b ? (l << OB) | (uint32_t)rank : ((uint32_t)rank << LB) | l; };
  // the block's partial (warp 0, 16 lanes; float pairs) sent to every block
  auto send = [&](float2 v) {
    float hi = v.x, lo = v.y;
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) {
      const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
      const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
      two_sum_acc(hi, lo, oh, ol);
    }
    if (tid < CS) *cl.map_shared_rank(sP + par * 16 + rank, tid) = make_float2(hi, lo);
  };
  auto collect = [&]() {  // after the cluster barrier: the same bits in every thread
    const float2 w = sP[par * 16 + (tid & (CS - 1))];
    par ^= 1;
    float hi = w.x, lo = w.y;
#pragma unroll
    for (int o = CS / 2; o >= 1; o >>= 1) {
      const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
      const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
      two_sum_acc(hi, lo, oh, ol);
    }
    const float s = hi + lo;  // renormalise
    return make_float2(s, lo - (s - hi));
  };

  cluster_arrive();  // every block of the cluster runs before any writes to another
  cluster_wait();
  // every block of a cluster runs the same loops: each barrier is reached by all
  for (int64_t slot = blockIdx.x / CS; slot < A.B; slot += gridDim.x / CS) {
    const int ci = A.run_circuit ? A.run_circuit[slot] : 0;
    const int64_t run = A.run_circuit ? (int64_t)ci : slot;
    const DevCircuit &C = A.circ[ci];
    const int M = C.n_steps;
    const DevStep *steps = A.steps + C.step_off;
    if (C.w != W || M > A.maxm || M < 1 || C.map_off < 0 || !(steps[M - 1].mask & kDead)) {
      if (tid == 0 && rank == 0 && A.status) A.status[run] = MBQC_RUN_NAN;  // the host routes such plans elsewhere
      continue;
    }
    const int2 *map = A.maps + C.map_off;
    const double *ang = A.angles + run * A.astride;
    for (int k = tid; k < M; k += BT) {
      const DevStep st = steps[k];
      const double th = st.aidx >= 0 ? ang[st.aidx] : st.fixed;
      float nx, ny, nz;
      bloch(st.plane, th, nx, ny, nz);
      sF[k] = make_float4(a_n * 0.5f * (1.f + nz) + b_n, a_n * 0.5f * (1.f - nz) + b_n, a_n * 0.5f * nx,
                          a_n * 0.5f * ny);
    }
    fact_tables<W>(steps, M, sSt, sPos, tid, BT);
    {
      const float2 *in = A.psi_in + (A.istride ? run * A.istride : 0);
      const float pad = exp2f(-0.5f * (float)(W - C.n_in));
      for (int i = tid; i < DW; i += BT) {
        const int2 mi = __ldg(&map[i]);
        const float2 u = flip_sign(in[mi.x & 0x7fffffff], (uint32_t)mi.x & 0x80000000u);
        psi[i] = make_float2(pad * u.x, pad * u.y);
      }
    }
    __syncthreads();

    int32_t st_code = MBQC_RUN_OK;
    int n_rec = 0;    // steps with a recorded probability
    bool lb = false;  // the rows' layout: A, or B
    for (int k = 0; k < M; ++k) {
      // Outcome probability (what = 0), trace (1) or prob1 (2) of the step
      // (dm_fact_run): step 0 from the initial window, later from the block's
      // sixteen diagonal pairs.  Made again where a step needs the trace or
      // prob1: few do, and nothing of it stays live over the barrier (a spilled
      // register is an L2 round trip there, the barrier drops the L1).
      auto partial = [&](int what) {
        const float4 F = sF[k];
        const uint2 ss = sSt[k];
        const int pos = (int)(ss.x & 15u), lp = pos - (lb ? OB : 0);
        const bool drop_coh = k > 0 && (ss.x & kFactDead) == 0u && (ss.x & kFactMq) != 0u;
        float2 sum = make_float2(0.f, 0.f);
        auto add = [&](float v, float off, float tr) {
          float p;
          if (what == 0)
            p = drop_coh ? v : v + off;
          else if (what == 1)
            p = tr;
          else  // prob1 = trace - prob0 term by term
            p = drop_coh ? tr_noise * tr - v : tr_noise * tr - v - off;
          two_sum_acc(sum.x, sum.y, p, 0.f);
        };
        if (k == 0) {
          for (int r = rank * 16 + (tid & 15); r < D; r += CS * 16) {
            const float2 u0 = psi[2 * r], u1 = psi[2 * r + 1];
            const float q00 = u0.x * u0.x + u0.y * u0.y, q11 = u1.x * u1.x + u1.y * u1.y;
            // x01 = psi0 conj(psi1)
            add(F.x * q00 + F.y * q11,
                2.f * (F.z * (u0.x * u1.x + u0.y * u1.y) - F.w * (u0.y * u1.x - u0.x * u1.y)), q00 + q11);
          }
        } else {
          const uint32_t l0 = ins_bit(tid & 15, lp, 0), l1 = l0 | (1u << lp);
          const uint32_t i0 = row_of(lb, l0), i1 = row_of(lb, l1);
          const float2 q00 = R[l0 * D + rsw(i0)], q11 = R[l1 * D + rsw(i1)], q01 = R[l0 * D + rsw(i1)];
          add(F.x * q00.x + F.y * q11.x, 2.f * (F.z * q01.x - F.w * q01.y), q00.x + q11.x);
        }
        return sum;
      };
      // the sum over the cluster.  Warp 0 publishes the partial; the other warps'
      // reads of the buffer that the next exchange but one writes are released by
      // the block barrier that ends the step and warp 0's next arrival, but a
      // step's further exchanges have no such barrier before them.
      auto exchange = [&](int what) {
        if (tid < 32) {
          send(partial(what));
          cluster_arrive();
        } else if (what == 0) {
          cluster_arrive_relaxed();
        } else {
          cluster_arrive();
        }
        cluster_wait();
        return collect();
      };
      float2 prob = exchange(0);
      const float4 F = sF[k];
      const uint2 ss = sSt[k];
      const bool zstep = (ss.x & kFactZ) != 0u;
      const int pos = (int)(ss.x & 15u), lp = pos - (lb ? OB : 0);  // position, local row bit
      const bool mq = (ss.x & kFactMq) != 0u, pdead = (ss.x & kFactDead) != 0u;
      float4 G = F;
      int outcome = 0;
      bool take1 = false, unprojected = false;
      const bool writer = tid == 0 && rank == 0;
      if (zstep) {
        const float2 tot = exchange(1);
        if (A.flags & MBQC_F_DM_EXPECTATION) {
          if (tid == 0) sF[k - 1] = make_float4(prob.x, prob.y, tot.x, tot.y);
          G = make_float4(1.f, 1.f, 0.f, 0.f);
          prob = make_float2(1.f, 0.f);
          outcome = 2;
          unprojected = true;
        } else {
          take1 = !(draw_uniform(A.seed, run, k) * tot.x < prob.x);
        }
      } else {
        take1 = !pair_ge(prob, 1e-4);  // prob0 < 1e-4 (or NaN): outcome 1 (np_simulator_dm.py:335-338)
      }
      if (tid == 0 && !unprojected) sF[k - 1] = make_float4(prob.x, prob.y, kNoTrace, 0.f);
      n_rec = k + 1;
      if (take1) {  // outcome 1 with P1 = I - P0
        G = make_float4(tr_noise - F.x, tr_noise - F.y, -F.z, -F.w);
        prob = exchange(2);
        outcome = 1;
      }
      if (writer && A.outcomes) A.outcomes[run * A.ostride + k] = (int8_t)outcome;
      if (!(prob.x > 0.f) || isnan(prob.x) || isinf(prob.x)) {  // the reference's NaN check
        st_code = MBQC_RUN_NAN;  // the same bits, so the same branch, in every thread of the cluster
        break;
      }
      float inv = __frcp_rn(prob.x);        // correctly rounded 1/hi
      inv = fmaf(-inv * inv, prob.y, inv);  // 1/(hi + lo) to first order in lo
      const float g00 = G.x, g11 = G.y, gr = G.z, gi = G.w;
      if (k == 0) {
        for (int e = tid; e < D * RL; e += BT) {
          const int l = e / D, y = e % D, xr = (int)row_of(false, (uint32_t)l);
          const float2 u0 = psi[2 * xr], u1 = psi[2 * xr + 1], v0 = psi[2 * y], v1 = psi[2 * y + 1];
          // x_ab = psi(x,a) conj(psi(y,b))
          const float2 x00 = make_float2(u0.x * v0.x + u0.y * v0.y, u0.y * v0.x - u0.x * v0.y);
          const float2 x11 = make_float2(u1.x * v1.x + u1.y * v1.y, u1.y * v1.x - u1.x * v1.y);
          const float2 x01 = make_float2(u0.x * v1.x + u0.y * v1.y, u0.y * v1.x - u0.x * v1.y);
          const float2 x10 = make_float2(u1.x * v0.x + u1.y * v0.y, u1.y * v0.x - u1.x * v0.y);
          const float sr = g00 * x00.x + g11 * x11.x + gr * (x01.x + x10.x) - gi * (x01.y - x10.y);
          const float si = g00 * x00.y + g11 * x11.y + gr * (x01.y + x10.y) + gi * (x01.x - x10.x);
          R[l * D + rsw((uint32_t)y)] = make_float2(sr * inv, si * inv);
        }
        __syncthreads();
        continue;
      }
      // 2. the pass.  The last step of a layout stores to the rows' new owners,
      //    once every block has loaded its own
      const uint32_t sgn = ss.y, rs = ((uint32_t)D << lp) >> 1;  // row step in float4
      const float half = pdead ? inv : 0.5f * inv;
      const float hA = g00 * half, hB = g11 * half, hR = gr * half, hI = gi * half;
      if (pos == 0) {
        const uint32_t pc = (__popc((2u * (uint32_t)(tid % H)) & sgn) & 1u) << 31;
        const uint32_t s0 = rsw(2u * (uint32_t)(tid % H)) >> 1;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t l = ins_bit((uint32_t)(tid / H + 4 * u), 0, 0), at = ((l * D) >> 1) + s0;
          const uint32_t pr = (__popc(row_of(lb, l) & sgn) & 1u) << 31;
          const float4 top = R4[at], bot = R4[at + rs];
          float2 o00, o01, o10, o11;
          fact_combine(hA, hB, hR, hI, pdead, mq, make_float2(top.x, top.y), make_float2(top.z, top.w),
                       make_float2(bot.x, bot.y), make_float2(bot.z, bot.w), pr, pc, o00, o01, o10, o11);
          R4[at] = make_float4(o00.x, o00.y, o01.x, o01.y);
          R4[at + rs] = make_float4(o10.x, o10.y, o11.x, o11.y);
        }
        __syncthreads();
        continue;
      }
      const uint32_t c0 = ins_bit(2u * (uint32_t)(tid % HU), pos, 0);  // even
      const uint32_t pc0 = (__popc(c0 & sgn) & 1u) << 31, pc1 = (__popc((c0 + 1u) & sgn) & 1u) << 31;
      const uint32_t s0 = rsw(c0) >> 1, s1 = rsw(c0 | (1u << pos)) >> 1;
      // the unit of rows l, l + 2^lp: its outputs in place of its inputs
      auto unit = [&](uint32_t l, float4 (&x)[4]) {
        const uint32_t at = (l * D) >> 1;
        x[0] = R4[at + s0];
        x[1] = R4[at + s1];
        x[2] = R4[at + rs + s0];
        x[3] = R4[at + rs + s1];
        const uint32_t pr = (__popc(row_of(lb, l) & sgn) & 1u) << 31;
        float2 a00, a01, a10, a11, b00, b01, b10, b11;
        fact_combine(hA, hB, hR, hI, pdead, mq, make_float2(x[0].x, x[0].y), make_float2(x[1].x, x[1].y),
                     make_float2(x[2].x, x[2].y), make_float2(x[3].x, x[3].y), pr, pc0, a00, a01, a10, a11);
        fact_combine(hA, hB, hR, hI, pdead, mq, make_float2(x[0].z, x[0].w), make_float2(x[1].z, x[1].w),
                     make_float2(x[2].z, x[2].w), make_float2(x[3].z, x[3].w), pr, pc1, b00, b01, b10, b11);
        x[0] = make_float4(a00.x, a00.y, b00.x, b00.y);
        x[1] = make_float4(a01.x, a01.y, b01.x, b01.y);
        x[2] = make_float4(a10.x, a10.y, b10.x, b10.y);
        x[3] = make_float4(a11.x, a11.y, b11.x, b11.y);
      };
      const uint32_t l0 = ins_bit((uint32_t)(tid / HU), lp, 0), l1 = ins_bit((uint32_t)(tid / HU + 8), lp, 0);
      if (k + 1 == M || pos != (lb ? N - 1 : LB - 1)) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint32_t l = u ? l1 : l0, at = (l * D) >> 1;
          float4 x[4];
          unit(l, x);
          R4[at + s0] = x[0];
          R4[at + s1] = x[1];
          R4[at + rs + s0] = x[2];
          R4[at + rs + s1] = x[3];
        }
        __syncthreads();
      } else {
        float4 x[4], y[4];
        unit(l0, x);
        unit(l1, y);
        cluster_arrive();  // release: this block's loads come before the others' stores
        cluster_wait();
        auto row_ptr = [&](uint32_t l) {
          const uint32_t i = row_of(lb, l), owner = lb ? i >> LB : i & (CS - 1), q = lb ? i & (RL - 1) : i >> OB;
          return cl.map_shared_rank(R4 + q * (D / 2), (int)owner);
        };
        float4 *p = row_ptr(l0), *q = row_ptr(l0 | (1u << lp));
        p[s0] = x[0];
        p[s1] = x[1];
        q[s0] = x[2];
        q[s1] = x[3];
        p = row_ptr(l1);
        q = row_ptr(l1 | (1u << lp));
        p[s0] = y[0];
        p[s1] = y[1];
        q[s0] = y[2];
        q[s1] = y[3];
        lb = !lb;
        cluster_arrive();
        cluster_wait();
      }
    }

    // ---- output noise: the positions this layout pairs, then the others
    const int n_out = C.n_out, dout = 1 << n_out;
    if (st_code == MBQC_RUN_OK && qn != 0.f) {
      for (int half = 0; half < 2; ++half) {
        for (int j = 0; j < n_out; ++j) {
          const int pos = sPos[C.out_bits[j]], lp = pos - (lb ? OB : 0);
          // positions both layouts pair are taken in the first one
          const bool here = lp >= 0 && lp < LB;
          const int lq = pos - (lb ? 0 : OB);
          const bool other = lq >= 0 && lq < LB;
          if (!here || (half == 1 && other)) continue;
          for (int e = tid; e < RL / 2 * H; e += BT) {
            const uint32_t l0 = ins_bit((uint32_t)e / H, lp, 0) * D, l1 = l0 + ((uint32_t)D << lp);
            const uint32_t c = ins_bit((uint32_t)e % H, pos, 0), c0 = rsw(c), c1 = rsw(c | (1u << pos));
            const float2 x00 = R[l0 + c0], x01 = R[l0 + c1], x10 = R[l1 + c0], x11 = R[l1 + c1];
            const float2 tr = make_float2(x00.x + x11.x, x00.y + x11.y);
            R[l0 + c0] = make_float2(a_n * x00.x + b_n * tr.x, a_n * x00.y + b_n * tr.y);
            R[l1 + c1] = make_float2(a_n * x11.x + b_n * tr.x, a_n * x11.y + b_n * tr.y);
            R[l0 + c1] = make_float2(a_n * x01.x, a_n * x01.y);
            R[l1 + c0] = make_float2(a_n * x10.x, a_n * x10.y);
          }
          __syncthreads();
        }
        if (half == 0) {  // every row to its owner in the other layout
          float4 x[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) x[u] = R4[tid + u * BT];
          cluster_arrive();
          cluster_wait();
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const uint32_t e = (uint32_t)(tid + u * BT), i = row_of(lb, e / (D / 2));
            const uint32_t owner = lb ? i >> LB : i & (CS - 1), l = lb ? i & (RL - 1) : i >> OB;
            cl.map_shared_rank(R4, (int)owner)[l * (D / 2) + e % (D / 2)] = x[u];
          }
          lb = !lb;
          cluster_arrive();
          cluster_wait();
        }
      }
    }
    // ---- outputs in the reference order: each block writes the rows it holds
    int *ridx = reinterpret_cast<int *>(psi), *rinv = ridx + D;  // psi is no longer needed
    __syncthreads();
    for (int i = tid; i < D; i += BT) rinv[i] = -1;
    __syncthreads();
    for (int y = tid; y < dout; y += BT) {
      int ri = 0;
      for (int j = 0; j < n_out; ++j) ri |= ((y >> (n_out - 1 - j)) & 1) << sPos[C.out_bits[j]];
      ridx[y] = ri;
      rinv[ri] = y;
    }
    __syncthreads();
    if (rank == 0 && A.probs)
      for (int k = tid; k < n_rec; k += BT)
        A.probs[run * A.ostride + k] = prob_record(sF[k - 1]);
    float2 *out = A.rho_out + run * A.out_stride;
    for (int e = tid; e < RL << n_out; e += BT) {
      const int l = e >> n_out, yj = e & (dout - 1), yi = rinv[row_of(lb, (uint32_t)l)];
      if (yi < 0) continue;
      out[((int64_t)yi << n_out) + yj] =
          st_code == MBQC_RUN_OK ? R[l * D + rsw((uint32_t)ridx[yj])] : make_float2(NAN, NAN);
    }
    if (tid == 0 && rank == 0 && A.status) A.status[run] = st_code;
    cluster_arrive();  // the rows and the tables are reused by the cluster's next run; no block
    cluster_wait();    // leaves while another may still write to it
  }
}

// Windows 9..11: R (512 KB to 8 MB) in the workspace, one slice per cluster of
// CS blocks; the cluster takes a run at a time.  Every block reads the step's
// diagonal and sums the probability itself (no exchange), the 2x2 blocks of
// the pass are dealt over all CS x 512 threads, and a cluster barrier ends the
// step.  In place: a block arrives at a second barrier once it has read the
// diagonal and waits there only before its first store, so the reduction
// overlaps it.  What bounds it is the L2: a step moves the slice in and out
// once.  One 1024-thread block a run left the rest of the GPU idle and ran at
// what one SM draws from L2: 24 runs of an 8 x 6 grid (window 9) took
// 711 us, 325 us with eight blocks a run.
constexpr int kFactWsThreads = 512;

// Sum of the hi + lo pairs of the block's threads, the same bits in each
// (two-sum at every addition); scratch double-buffered as in group_sum2_db.
__device__ __forceinline__ float2 block_sum2_db(float hi, float lo, float2 *scratch, int &par) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
    const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
    two_sum_acc(hi, lo, oh, ol);
  }
  float2 *buf = scratch + par * 32;
  par ^= 1;
  if ((threadIdx.x & 31) == 0) buf[threadIdx.x >> 5] = make_float2(hi, lo);
  __syncthreads();
  constexpr int NW = kFactWsThreads / 32;
  const float2 w = buf[threadIdx.x & (NW - 1)];
  hi = w.x;
  lo = w.y;
#pragma unroll
  for (int o = NW / 2; o >= 1; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
    const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
    two_sum_acc(hi, lo, oh, ol);
  }
  const float s = hi + lo;  // renormalise
  return make_float2(s, lo - (s - hi));
}

template <int W, int CS>
__global__ void __launch_bounds__(kFactWsThreads, 2) dm_fwd_fact_ws(DmArgs A, float2 *ws) {
  using Cfg = DmFactCfg<W>;
  constexpr int D = Cfg::D, H = Cfg::H, NB = Cfg::NB, DW = Cfg::DW, BT = kFactWsThreads, TT = BT * CS;
  extern __shared__ __align__(16) unsigned char smem_w[];
  float2 *psi = reinterpret_cast<float2 *>(smem_w);
  float4 *sF = reinterpret_cast<float4 *>(psi + DW);
  uint2 *sSt = reinterpret_cast<uint2 *>(sF + A.maxm);
  float2 *sRed = reinterpret_cast<float2 *>(sSt + A.maxm);  // 2 x 32 entries
  int8_t *sPos = reinterpret_cast<int8_t *>(sRed + 64);
  const int tid = threadIdx.x;
  const int crank = (int)cooperative_groups::this_cluster().block_rank();
  const int g = crank * BT + tid;  // thread of the cluster
  float2 *R = ws + (size_t)(blockIdx.x / CS) * Cfg::N;
  float4 *R4 = reinterpret_cast<float4 *>(R);
  const float qn = f64_to_f32_rn(A.noise);
  const float a_n = 1.f - (4.f / 3.f) * qn, b_n = (2.f / 3.f) * qn;
  const float tr_noise = a_n + 2.f * b_n;
  int par = 0;

  // every block of a cluster runs the same loops: each barrier is reached by all
  for (int64_t slot = blockIdx.x / CS; slot < A.B; slot += gridDim.x / CS) {
    const int ci = A.run_circuit ? A.run_circuit[slot] : 0;
    const int64_t run = A.run_circuit ? (int64_t)ci : slot;
    const DevCircuit &C = A.circ[ci];
    const int M = C.n_steps;
    const DevStep *steps = A.steps + C.step_off;
    if (C.w != W || M > A.maxm || M < 1 || C.map_off < 0 || !(steps[M - 1].mask & kDead)) {
      if (g == 0 && A.status) A.status[run] = MBQC_RUN_NAN;  // the host routes such plans elsewhere
      continue;
    }
    const int2 *map = A.maps + C.map_off;
    const double *ang = A.angles + run * A.astride;
    for (int k = tid; k < M; k += BT) {
      const DevStep st = steps[k];
      const double th = st.aidx >= 0 ? ang[st.aidx] : st.fixed;
      float nx, ny, nz;
      bloch(st.plane, th, nx, ny, nz);
      sF[k] = make_float4(a_n * 0.5f * (1.f + nz) + b_n, a_n * 0.5f * (1.f - nz) + b_n, a_n * 0.5f * nx,
                          a_n * 0.5f * ny);
    }
    fact_tables<W>(steps, M, sSt, sPos, tid, BT);
    {
      const float2 *in = A.psi_in + (A.istride ? run * A.istride : 0);
      const float pad = exp2f(-0.5f * (float)(W - C.n_in));
      for (int i = tid; i < DW; i += BT) {
        const int2 mi = __ldg(&map[i]);
        const float2 u = flip_sign(in[mi.x & 0x7fffffff], (uint32_t)mi.x & 0x80000000u);
        psi[i] = make_float2(pad * u.x, pad * u.y);
      }
    }
    __syncthreads();

    int32_t st_code = MBQC_RUN_OK;
    int n_rec = 0;  // steps with a recorded probability
    for (int k = 0; k < M; ++k) {
      const float4 F = sF[k];
      const uint2 ss = sSt[k];
      const bool zstep = (ss.x & kFactZ) != 0u;
      const int pos = (int)(ss.x & 15u);
      const bool mq = (ss.x & kFactMq) != 0u, pdead = (ss.x & kFactDead) != 0u;
      const bool drop_coh = k > 0 && !pdead && mq;
      // 1. outcome probability (dm_fact_run), term by term in float pairs
      float p_hi = 0.f, p_lo = 0.f, t_hi = 0.f, t_lo = 0.f, o_hi = 0.f, o_lo = 0.f;
      const int terms = k == 0 ? D : H;
      for (int r = tid; r < terms; r += BT) {
        float v, off = 0.f, tr;
        if (k == 0) {
          const float2 u0 = psi[2 * r], u1 = psi[2 * r + 1];
          const float q00 = u0.x * u0.x + u0.y * u0.y, q11 = u1.x * u1.x + u1.y * u1.y;
          // x01 = psi0 conj(psi1)
          off = 2.f * (F.z * (u0.x * u1.x + u0.y * u1.y) - F.w * (u0.y * u1.x - u0.x * u1.y));
          v = F.x * q00 + F.y * q11;
          tr = q00 + q11;
        } else {
          const uint32_t i0 = ins_bit(r, pos, 0), i1 = ins_bit(r, pos, 1);
          const float2 q00 = __ldcg(&R[i0 * D + i0]), q11 = __ldcg(&R[i1 * D + i1]);
          v = F.x * q00.x + F.y * q11.x;
          if (!drop_coh) {
            const float2 q01 = __ldcg(&R[i0 * D + i1]);
            off = 2.f * (F.z * q01.x - F.w * q01.y);
          }
          tr = q00.x + q11.x;
        }
        two_sum_acc(p_hi, p_lo, drop_coh ? v : v + off, 0.f);
        two_sum_acc(t_hi, t_lo, tr, 0.f);
        // prob1 = trace - prob0 term by term
        two_sum_acc(o_hi, o_lo, drop_coh ? tr_noise * tr - v : tr_noise * tr - v - off, 0.f);
      }
      if (k > 0) cluster_arrive();  // this block has read its diagonal
      float2 prob = block_sum2_db(p_hi, p_lo, sRed, par);
      float4 G = F;
      int outcome = 0;
      bool take1 = false, unprojected = false;
      if (zstep) {
        const float2 tot = block_sum2_db(t_hi, t_lo, sRed, par);
        if (A.flags & MBQC_F_DM_EXPECTATION) {
          if (tid == 0) sF[k] = make_float4(prob.x, prob.y, tot.x, tot.y);
          G = make_float4(1.f, 1.f, 0.f, 0.f);
          prob = make_float2(1.f, 0.f);
          outcome = 2;
          unprojected = true;
        } else {
          take1 = !(draw_uniform(A.seed, run, k) * tot.x < prob.x);
        }
      } else {
        take1 = !pair_ge(prob, 1e-4);  // prob0 < 1e-4 (or NaN): outcome 1 (np_simulator_dm.py:335-338)
      }
      if (tid == 0 && !unprojected) sF[k] = make_float4(prob.x, prob.y, kNoTrace, 0.f);
      n_rec = k + 1;
      if (take1) {  // outcome 1 with P1 = I - P0
        G = make_float4(tr_noise - F.x, tr_noise - F.y, -F.z, -F.w);
        prob = block_sum2_db(o_hi, o_lo, sRed, par);
        outcome = 1;
      }
      if (g == 0 && A.outcomes) A.outcomes[run * A.ostride + k] = (int8_t)outcome;
      const bool bad = !(prob.x > 0.f) || isnan(prob.x) || isinf(prob.x);  // the reference's NaN check
      if (bad) {  // the same bits, so the same branch, in every thread of the cluster
        st_code = MBQC_RUN_NAN;
        if (k > 0) cluster_wait();
        break;
      }
      float inv = __frcp_rn(prob.x);        // correctly rounded 1/hi
      inv = fmaf(-inv * inv, prob.y, inv);  // 1/(hi + lo) to first order in lo
      const float g00 = G.x, g11 = G.y, gr = G.z, gi = G.w;
      if (k == 0) {
        for (int e = g; e < Cfg::N; e += TT) {
          const int x = e / D, y = e % D;
          const float2 u0 = psi[2 * x], u1 = psi[2 * x + 1], v0 = psi[2 * y], v1 = psi[2 * y + 1];
          // x_ab = psi(x,a) conj(psi(y,b))
          const float2 x00 = make_float2(u0.x * v0.x + u0.y * v0.y, u0.y * v0.x - u0.x * v0.y);
          const float2 x11 = make_float2(u1.x * v1.x + u1.y * v1.y, u1.y * v1.x - u1.x * v1.y);
          const float2 x01 = make_float2(u0.x * v1.x + u0.y * v1.y, u0.y * v1.x - u0.x * v1.y);
          const float2 x10 = make_float2(u1.x * v0.x + u1.y * v0.y, u1.y * v0.x - u1.x * v0.y);
          const float sr = g00 * x00.x + g11 * x11.x + gr * (x01.x + x10.x) - gi * (x01.y - x10.y);
          const float si = g00 * x00.y + g11 * x11.y + gr * (x01.y + x10.y) + gi * (x01.x - x10.x);
          __stcg(&R[e], make_float2(sr * inv, si * inv));
        }
      } else {
        // 2. one in-place pass over the 2x2 blocks of position pos: at pos 0 a
        //    block's two columns are one float4 a row, else a unit is the two
        //    blocks of columns c0, c0 + 1; all loads of U units in flight
        //    before their stores
        const uint32_t sgn = ss.y;
        const float half = pdead ? inv : 0.5f * inv;
        const float hA = g00 * half, hB = g11 * half, hR = gr * half, hI = gi * half;
        bool waited = false;
        if (pos == 0) {
          constexpr int RSTEP = TT / H, NJ = H / RSTEP, U = NJ >= 4 ? 4 : NJ;
          static_assert(TT % H == 0 && H % RSTEP == 0 && NJ % U == 0, "rows over the cluster's threads");
          const uint32_t c = (uint32_t)(g % H), r_first = (uint32_t)(g / H);
          const uint32_t pc = (__popc((2u * c) & sgn) & 1u) << 31;
#pragma unroll 1
          for (int j0 = 0; j0 < NJ; j0 += U) {
            float4 top[U], bot[U];
#pragma unroll
            for (int uu = 0; uu < U; ++uu) {
              const uint32_t at = (r_first + (uint32_t)(j0 + uu) * RSTEP) * D + c;
              top[uu] = __ldcg(&R4[at]);
              bot[uu] = __ldcg(&R4[at + D / 2]);
            }
            if (!waited) cluster_wait();
            waited = true;
#pragma unroll
            for (int uu = 0; uu < U; ++uu) {
              const uint32_t r = r_first + (uint32_t)(j0 + uu) * RSTEP, at = r * D + c;
              const uint32_t pr = (__popc((2u * r) & sgn) & 1u) << 31;
              float2 o00, o01, o10, o11;
              fact_combine(hA, hB, hR, hI, pdead, mq, make_float2(top[uu].x, top[uu].y),
                           make_float2(top[uu].z, top[uu].w), make_float2(bot[uu].x, bot[uu].y),
                           make_float2(bot[uu].z, bot[uu].w), pr, pc, o00, o01, o10, o11);
              __stcg(&R4[at], make_float4(o00.x, o00.y, o01.x, o01.y));
              __stcg(&R4[at + D / 2], make_float4(o10.x, o10.y, o11.x, o11.y));
            }
          }
        } else {
          constexpr int HU = H / 2, RSTEP = TT / HU, NJ = H > RSTEP ? H / RSTEP : 1, U = NJ >= 2 ? 2 : NJ;
          static_assert(TT % HU == 0 && RSTEP <= H && H % RSTEP == 0 && NJ % U == 0, "rows over the cluster's threads");
          const uint32_t rs = ((uint32_t)D << pos) >> 1;  // row step in float4
          const uint32_t r_first = (uint32_t)(g / HU);
          const uint32_t c0 = ins_bit(2u * (uint32_t)(g % HU), pos, 0);  // even
          const uint32_t pc0 = (__popc(c0 & sgn) & 1u) << 31, pc1 = (__popc((c0 + 1u) & sgn) & 1u) << 31;
          const uint32_t s0 = c0 >> 1, s1 = (c0 | (1u << pos)) >> 1;
#pragma unroll 1
          for (int j0 = 0; j0 < NJ; j0 += U) {
            float4 q00[U], q01[U], q10[U], q11[U];
            uint32_t at[U], pr[U];
#pragma unroll
            for (int uu = 0; uu < U; ++uu) {
              const uint32_t r0 = ins_bit(r_first + (uint32_t)(j0 + uu) * RSTEP, pos, 0);
              at[uu] = (r0 * D) >> 1;
              pr[uu] = (__popc(r0 & sgn) & 1u) << 31;
              q00[uu] = __ldcg(&R4[at[uu] + s0]);
              q01[uu] = __ldcg(&R4[at[uu] + s1]);
              q10[uu] = __ldcg(&R4[at[uu] + rs + s0]);
              q11[uu] = __ldcg(&R4[at[uu] + rs + s1]);
            }
            if (!waited) cluster_wait();
            waited = true;
#pragma unroll
            for (int uu = 0; uu < U; ++uu) {
              float2 a00, a01, a10, a11, b00, b01, b10, b11;
              fact_combine(hA, hB, hR, hI, pdead, mq, make_float2(q00[uu].x, q00[uu].y),
                           make_float2(q01[uu].x, q01[uu].y), make_float2(q10[uu].x, q10[uu].y),
                           make_float2(q11[uu].x, q11[uu].y), pr[uu], pc0, a00, a01, a10, a11);
              fact_combine(hA, hB, hR, hI, pdead, mq, make_float2(q00[uu].z, q00[uu].w),
                           make_float2(q01[uu].z, q01[uu].w), make_float2(q10[uu].z, q10[uu].w),
                           make_float2(q11[uu].z, q11[uu].w), pr[uu], pc1, b00, b01, b10, b11);
              __stcg(&R4[at[uu] + s0], make_float4(a00.x, a00.y, b00.x, b00.y));
              __stcg(&R4[at[uu] + s1], make_float4(a01.x, a01.y, b01.x, b01.y));
              __stcg(&R4[at[uu] + rs + s0], make_float4(a10.x, a10.y, b10.x, b10.y));
              __stcg(&R4[at[uu] + rs + s1], make_float4(a11.x, a11.y, b11.x, b11.y));
            }
          }
        }
      }
      cluster_arrive();
      cluster_wait();
    }

    // ---- output noise, one output qubit a pass
    if (st_code == MBQC_RUN_OK && qn != 0.f) {
      for (int j = 0; j < C.n_out; ++j) {
        const int pos = sPos[C.out_bits[j]];
        for (int e = g; e < NB; e += TT) {
          const uint32_t r = (uint32_t)e / H, c = (uint32_t)e % H;
          const uint32_t r0 = ins_bit(r, pos, 0) * D, r1 = ins_bit(r, pos, 1) * D;
          const uint32_t c0 = ins_bit(c, pos, 0), c1 = ins_bit(c, pos, 1);
          const float2 x00 = __ldcg(&R[r0 + c0]), x01 = __ldcg(&R[r0 + c1]);
          const float2 x10 = __ldcg(&R[r1 + c0]), x11 = __ldcg(&R[r1 + c1]);
          const float2 tr = make_float2(x00.x + x11.x, x00.y + x11.y);
          __stcg(&R[r0 + c0], make_float2(a_n * x00.x + b_n * tr.x, a_n * x00.y + b_n * tr.y));
          __stcg(&R[r1 + c1], make_float2(a_n * x11.x + b_n * tr.x, a_n * x11.y + b_n * tr.y));
          __stcg(&R[r0 + c1], make_float2(a_n * x01.x, a_n * x01.y));
          __stcg(&R[r1 + c0], make_float2(a_n * x10.x, a_n * x10.y));
        }
        cluster_arrive();
        cluster_wait();
      }
    }
    // ---- gather the outputs in the reference order
    const int n_out = C.n_out, dout = 1 << n_out;
    int *ridx = reinterpret_cast<int *>(psi);  // psi is no longer needed
    __syncthreads();
    for (int y = tid; y < dout; y += BT) {
      int ri = 0;
      for (int j = 0; j < n_out; ++j) ri |= ((y >> (n_out - 1 - j)) & 1) << sPos[C.out_bits[j]];
      ridx[y] = ri;
    }
    __syncthreads();
    if (crank == 0 && A.probs)
      for (int k = tid; k < n_rec; k += BT)
        A.probs[run * A.ostride + k] = prob_record(sF[k]);
    float2 *out = A.rho_out + run * A.out_stride;
    for (int e = g; e < dout * dout; e += TT) {
      const int yi = e >> n_out, yj = e & (dout - 1);
      out[e] = st_code == MBQC_RUN_OK ? __ldcg(&R[ridx[yi] * D + ridx[yj]]) : make_float2(NAN, NAN);
    }
    if (g == 0 && A.status) A.status[run] = st_code;
    cluster_arrive();  // the slice and the tables are reused by the cluster's next run
    cluster_wait();
  }
}

// One run per group of TPR threads, 256 / TPR runs per block.
template <int W, int TPR>
__global__ void __launch_bounds__(256, 3) dm_fwd_fact(DmArgs A) {
  extern __shared__ __align__(16) unsigned char smem_f[];
  const int group = threadIdx.x / TPR, tid = threadIdx.x % TPR;
  const int64_t slot = (int64_t)blockIdx.x * (256 / TPR) + group;
  if (slot >= A.B) return;  // whole group leaves together
  dm_fact_run<W, TPR>(A, slot, tid, group, smem_f + (size_t)group * dm_fact_slice_bytes<W>(A.maxm));
}

}  // namespace mbqc
