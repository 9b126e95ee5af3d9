// Adjoint of the (noisy) density-matrix sweep on the factored matrix, windows
// 5..7 whose last step shrinks the window (dm_adj.cuh takes the others; the
// derivation of the adjoint chain is there).
//
// Why from window 5 on: below it a run has fewer tiles than the warp has threads (1
// at window 3, 4 at window 4) and the whole matrix is small anyway.  Grids of 12
// columns, noise 0.01, full matrix against this: window 3, 500 runs 33 and 54 us,
// 16,000 runs 197 and 603; window 4, 500 runs 68 and 86, 16,000 runs 516 and 1,007;
// window 5, 500 runs 299 and 120, 16,000 runs 2,850 and 1,526; window 6, 500 runs
// 546 and 239; window 7, 500 runs 3,736 and 788.
//
// After step k every entry of the full 2^w x 2^w matrix is +-sigma_k[r, c], 0 or
// a sign of it: sigma_k is the (w-1)-qubit matrix over the bits other than the
// slot of the qubit that entered (dm_fact.cuh); and the cotangent of step k's
// input is conj(G_xx') m_k[r, c] with the same kind of matrix m_k = mu_k / prob_k.
// So only sigma and m are kept: 32 KB a run at window 7 where the full matrix
// took 128 KB (one run per SM), three runs per SM here.  The arithmetic is the
// full matrix's own, entry by entry (a copied entry is recomputed from the same
// operands, signs commute with every rounding), so the results are its bits.
//
// Layout: n = w - 1 storage positions, schedule index s at position
// (s - 1) mod n; step k measures position a = (k - 1) mod n, and b = k mod n is
// the next one's.  A thread owns the 4 x 4 tile of rows and columns over
// positions a and b (T x T tiles, T = 2^(n-2)):
//   sigma_{k-1}:  a = the measured qubit,    b = the next one to be measured
//   sigma_k, mu_k: a = the slot of step k-1, b = the next one to be measured
//   m_{k+1}:      a = the slot of step k-1,  b = the slot of step k
// so one tile holds all 2x2 blocks that step k's forward pass, its reverse pass
// and its derivative need.  The forward pass saves the pre-step entries the
// derivative needs (the measured qubit's coherences: 16 KB a step at window 7,
// written and read by the same thread; with the populations for XZ / YZ steps),
// where the full matrix saved 128 KB a step.
//
// The derivative's terms are summed in the order of the full-matrix kernel
// (float sums of NI terms a thread, then float pairs): the terms go through
// shared memory to the thread that kernel gives them to.
#pragma once

#include "dm_adj.cuh"
#include "dm_fact.cuh"

namespace mbqc {

constexpr int kDmAdjFactMinWindow = 5, kDmAdjFactMaxWindow = 7;

template <int W> struct AdjFactCfg {
  static_assert(W >= kDmAdjFactMinWindow && W <= kDmAdjFactMaxWindow, "factored adjoint: windows 5..7");
  static constexpr int N = W - 1, D = 1 << N, T = D / 4;
  static constexpr int TPR = DmCfg<W>::TPR;
  static constexpr int GROUPS = TPR == 32 ? 2 : 1;  // runs per block: small blocks spread a batch over the SMs
  static constexpr int NB = D * D, NI = NB / TPR;  // derivative terms, terms a thread
  static constexpr int RS = TPR / D;               // row step between a thread's terms
  static constexpr int HIST = 8 * T * T;           // float4 a step
};

// shared memory of one run
template <int W> __host__ __device__ constexpr size_t adj_fact_slice(int maxm) {
  using Cfg = AdjFactCfg<W>;
  return ((size_t)Cfg::NB * 8 + 2 * (size_t)Cfg::NB * 4 + ((size_t)1 << W) * 12 + (size_t)maxm * 32 + 16 +
          2 * 8 * sizeof(float2) + 2 * sizeof(float2) + 15) &
         ~(size_t)15;
}

constexpr uint32_t kAdjOff = 1u << 7, kAdjPop = 1u << 8;  // step word: the derivative needs coherences / populations

// The step functional on a 2x2 block, sum_ab G_ab x_ab (G = G00, G11, Re G01,
// Im G01; x10 takes conj(G01)), and its real diagonal part: the products and
// sums rounded in the full-matrix kernel's order.
__device__ __forceinline__ float2 functional(float4 G, float2 x00, float2 x01, float2 x10, float2 x11) {
  const float pr = fmaf(G.x, x00.x, __fmul_rn(G.y, x11.x)), pi = fmaf(G.x, x00.y, __fmul_rn(G.y, x11.y));
  return make_float2(fmaf(-G.w, x01.y - x10.y, fmaf(G.z, x01.x + x10.x, pr)),
                     fmaf(G.w, x01.x - x10.x, fmaf(G.z, x01.y + x10.y, pi)));
}
__device__ __forceinline__ float diag_term(float4 G, float q00, float q11, float2 q01) {
  return fmaf(2.f, fmaf(G.z, q01.x, -__fmul_rn(G.w, q01.y)), fmaf(G.x, q00, __fmul_rn(G.y, q11)));
}

template <int W>
__global__ void __launch_bounds__(AdjFactCfg<W>::TPR *AdjFactCfg<W>::GROUPS, 512 / (AdjFactCfg<W>::TPR * AdjFactCfg<W>::GROUPS))
    dm_adj_fact(DmAdjArgs A) {
  using Cfg = AdjFactCfg<W>;
  constexpr int N = Cfg::N, D = Cfg::D, T = Cfg::T, TPR = Cfg::TPR, NB = Cfg::NB, NI = Cfg::NI, RS = Cfg::RS,
                GROUPS = Cfg::GROUPS, NW = TPR / 32;
  extern __shared__ __align__(16) unsigned char smem_a[];
  const int group = threadIdx.x / TPR, tid = threadIdx.x % TPR;
  const int maxm = A.f.maxm;
  unsigned char *gb = smem_a + (size_t)group * adj_fact_slice<W>(maxm);
  float4 *sF = reinterpret_cast<float4 *>(gb);
  float2 *R = reinterpret_cast<float2 *>(sF + maxm);
  float2 *psi = R + NB;
  float *tmp = reinterpret_cast<float *>(psi + (1 << W));  // two buffers of derivative terms
  uint2 *sSt = reinterpret_cast<uint2 *>(tmp + 2 * NB);
  float2 *sGr = reinterpret_cast<float2 *>(sSt + maxm);  // two buffers of a partial per warp
  float2 *sBr = sGr + 2 * 8;                             // two broadcast slots
  float *sInv = reinterpret_cast<float *>(sBr + 2);      // 1 / prob_k
  int32_t *sOut = reinterpret_cast<int32_t *>(sInv + maxm);
  int32_t *sMap = sOut + maxm;  // window index -> output index << 8 | storage position of the final matrix, or -1
  const int64_t slot = (int64_t)blockIdx.x * GROUPS + group;
  const DmArgs &F0 = A.f;
  const float qn = f64_to_f32_rn(F0.noise);
  const float a_n = 1.f - (4.f / 3.f) * qn, b_n = (2.f / 3.f) * qn;
  const float tr_noise = a_n + 2.f * b_n;
  // this thread's tile; threads beyond the tiles help with the sums only
  const bool tiled = tid < T * T;
  const uint32_t tr = (uint32_t)tid / T, tc = (uint32_t)tid % T;
  float4 *hist = reinterpret_cast<float4 *>(A.hist) + slot * (int64_t)maxm * Cfg::HIST + tid;
  int par = 0;

  // columns are stored XOR-swizzled (n = 6): the 16 columns of a half warp's
  // tiles, whatever the two cyclically adjacent positions a and b, fall on 16
  // distinct 8-byte banks (any four cyclically consecutive of the vectors 1, 2,
  // 4, 8, 5, 10 are independent)
  auto sw = [](uint32_t c) -> uint32_t { return N == 6 ? c ^ (((c >> 4) & 1u) * 5u) ^ ((c >> 5) * 10u) : c; };
  auto rotl = [](uint32_t v, int h) -> uint32_t { return ((v << h) | (v >> (N - h))) & (uint32_t)(D - 1); };
  // float-pair sum of warp 0's lanes, in every thread of the run
  auto bcast_sum = [&](float hi, float lo) {
    if (tid < 32) {
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
        const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
        two_sum_acc(hi, lo, oh, ol);
      }
      const float s = hi + lo;  // renormalise
      lo = lo - (s - hi);
      hi = s;
    }
    if constexpr (TPR > 32) {
      if (tid == 0) sBr[par] = make_float2(hi, lo);
      group_sync(TPR, group);
      const float2 v = sBr[par];
      par ^= 1;
      return v;
    } else {
      return make_float2(hi, lo);
    }
  };

  // runs back and forth over the slots: lists come longest first, so a slot
  // that began with a long run gets a short one (or none) next
  const int64_t nslots = (int64_t)gridDim.x * GROUPS;
  for (int64_t wave = 0; wave * nslots < F0.B; ++wave) {
    const int64_t bq = wave * nslots + ((wave & 1) ? nslots - 1 - slot : slot);
    if (bq >= F0.B) continue;
    const int ci = F0.run_circuit ? F0.run_circuit[bq] : 0;
    const int64_t run = F0.run_circuit ? (int64_t)ci : bq;
    const DevCircuit &C = F0.circ[ci];
    const int M = C.n_steps;
    if (C.w != W || M > maxm || C.map_off < 0) {
      if (tid == 0 && F0.status) F0.status[run] = MBQC_RUN_NAN;
      continue;
    }
    const DevStep *steps = F0.steps + C.step_off;
    const int2 *map = F0.maps + C.map_off;
    const double *ang = F0.angles + run * F0.astride;
    double *grad = A.grad + run * A.grad_stride;
    group_sync(TPR, group);  // previous run of this group is done with shared memory
    for (int k = tid; k < M; k += TPR) {
      const DevStep st = steps[k];
      const double th = st.aidx >= 0 ? ang[st.aidx] : st.fixed;
      float nx, ny, nz;
      bloch(st.plane, th, nx, ny, nz);
      sF[k] = make_float4(a_n * 0.5f * (1.f + nz) + b_n, a_n * 0.5f * (1.f - nz) + b_n, a_n * 0.5f * nx,
                          a_n * 0.5f * ny);
    }
    fact_tables<W>(steps, M, sSt, nullptr, tid, TPR);
    for (int k = tid; k < M; k += TPR) {
      const DevStep st = steps[k];
      if (st.aidx >= 0 && (st.plane == MBQC_PLANE_XY || st.plane == MBQC_PLANE_XZ || st.plane == MBQC_PLANE_YZ))
        sSt[k].x |= st.plane == MBQC_PLANE_XY ? kAdjOff : kAdjOff | kAdjPop;
    }
    for (int ai = tid; ai < C.n_angles; ai += TPR) grad[ai] = 0.0;  // angles no step uses keep this
    {
      const float2 *in = F0.psi_in + (F0.istride ? run * F0.istride : 0);
      for (int i = tid; i < 1 << W; i += TPR) {
        const int2 mi = __ldg(&map[i]);
        psi[i] = flip_sign(in[mi.x & 0x7fffffff], (uint32_t)mi.x & 0x80000000u);
      }
    }
    const float pad = exp2f(-0.5f * (float)(C.w - C.n_in));
    auto rho0 = [&](uint32_t i, uint32_t j) {  // the initial matrix
      const float2 u = psi[i], v = psi[j];
      const float p2 = pad * pad;
      return make_float2(__fmul_rn(p2, fmaf(u.x, v.x, __fmul_rn(u.y, v.y))),
                         __fmul_rn(p2, fmaf(u.y, v.x, -__fmul_rn(u.x, v.y))));
    };
    group_sync(TPR, group);

    // ---------------------------------------------------------- forward
    int32_t st_code = MBQC_RUN_OK;
    for (int k = 0; k < M; ++k) {
      const float4 Fk = sF[k];
      const uint2 ss = sSt[k];
      const bool mq = (ss.x & kFactMq) != 0u, pdead = (ss.x & kFactDead) != 0u;
      const int pa = (k + N - 1) % N, pb = k % N;
      auto prob_of = [&](float4 G) {
        float hi = 0.f, lo = 0.f;
        if (tid < 32) {
          if (k == 0) {
            for (uint32_t r = tid; r < (uint32_t)D; r += 32) {
              const float2 q00 = rho0(2 * r, 2 * r), q11 = rho0(2 * r + 1, 2 * r + 1), q01 = rho0(2 * r, 2 * r + 1);
              const float v = diag_term(G, q00.x, q11.x, q01);
              two_sum_acc(hi, lo, v, 0.f);
            }
          } else if (tid < D / 2) {
            const uint32_t l0 = ins_bit((uint32_t)tid, pa, 0), l1 = l0 | (1u << pa);
            const float2 q00 = R[l0 * D + sw(l0)], q11 = R[l1 * D + sw(l1)];
            float2 q01 = R[l0 * D + sw(l1)];
            const float v = diag_term(G, q00.x, q11.x, q01);
            two_sum_acc(hi, lo, v, 0.f);
            if (!pdead) {  // the same entries with the slot bit set
              if (mq) q01 = make_float2(-q01.x, -q01.y);
              const float v1 = diag_term(G, q00.x, q11.x, q01);
              two_sum_acc(hi, lo, v1, 0.f);
            }
          }
        }
        return bcast_sum(hi, lo);
      };
      float2 prob = prob_of(Fk);
      float4 G = Fk;
      int outcome = 0;
      if (!pair_ge(prob, 1e-4)) {
        G = make_float4(tr_noise - Fk.x, tr_noise - Fk.y, -Fk.z, -Fk.w);
        prob = prob_of(G);
        outcome = 1;
      }
      if (tid == 0) {
        sOut[k] = outcome;
        if (F0.outcomes) F0.outcomes[run * F0.ostride + k] = (int8_t)outcome;
      }
      if (!(prob.x > 0.f) || isnan(prob.x) || isinf(prob.x)) {
        st_code = MBQC_RUN_NAN;
        break;
      }
      float inv = 1.f / prob.x;
      inv = fmaf(-inv * inv, prob.y, inv);
      if (tid == 0) sInv[k] = inv;
      const bool dead = k + 1 == M || (sSt[k + 1].x & kFactDead) != 0u;
      const float half = dead ? inv : 0.5f * inv;
      if (k == 0) {
        for (int e = tid; e < NB; e += TPR) {
          const uint32_t r = (uint32_t)e / D, c = (uint32_t)e % D;
          const float2 x00 = rho0(2 * r, 2 * c), x01 = rho0(2 * r, 2 * c + 1);
          const float2 x10 = rho0(2 * r + 1, 2 * c), x11 = rho0(2 * r + 1, 2 * c + 1);
          const float2 f = functional(G, x00, x01, x10, x11);
          R[r * D + sw(c)] = make_float2(f.x * half, f.y * half);
        }
      } else if (tiled) {
        const int plo = pa < pb ? pa : pb, phi = pa < pb ? pb : pa;
        const uint32_t rb = ins_bit(ins_bit(tr, plo, 0), phi, 0), cb = ins_bit(ins_bit(tc, plo, 0), phi, 0);
        float4 *h = hist + (int64_t)k * Cfg::HIST;
        const uint32_t ra = (uint32_t)D << pa, ca = sw(1u << pa), cb2 = sw(1u << pb);
#pragma unroll
        for (int xr = 0; xr < 2; ++xr)
#pragma unroll
          for (int xc = 0; xc < 2; ++xc) {
            const uint32_t r0 = rb | ((uint32_t)xr << pb), c0 = cb | ((uint32_t)xc << pb);
            float2 *p0 = R + r0 * D, *p1 = p0 + ra;
            const uint32_t s0 = sw(cb) ^ (xc ? cb2 : 0u), s1 = s0 ^ ca;
            const float2 y00 = p0[s0], y01 = p0[s1], y10 = p1[s0], y11 = p1[s1];
            if (ss.x & kAdjOff) h[(2 * xr + xc) * (T * T)] = make_float4(y01.x, y01.y, y10.x, y10.y);
            if (ss.x & kAdjPop) h[(4 + 2 * xr + xc) * (T * T)] = make_float4(y00.x, y00.y, y11.x, y11.y);
            // the functional on the block (slot bits 0, 0) and on its copies
            // with the slot's link signs: the same sums with y01, y10, y11 negated
            const float tx = __fmul_rn(G.y, y11.x), ty = __fmul_rn(G.y, y11.y);
            const float ux = y01.x + y10.x, uy = y01.y + y10.y, vx = y01.x - y10.x, vy = y01.y - y10.y;
            const float px = fmaf(G.x, y00.x, tx), py = fmaf(G.x, y00.y, ty);
            float2 o00 = make_float2(fmaf(-G.w, vy, fmaf(G.z, ux, px)), fmaf(G.w, vx, fmaf(G.z, uy, py)));
            o00 = make_float2(o00.x * half, o00.y * half);
            p0[s0] = o00;
            if (pdead) {
              p0[s1] = p1[s0] = p1[s1] = make_float2(0.f, 0.f);
            } else {
              float2 o01 = o00, o10 = o00, o11 = o00;
              if (mq) {
                const float mx = fmaf(G.x, y00.x, -tx), my = fmaf(G.x, y00.y, -ty);
                o11 = make_float2(half * fmaf(G.w, vy, fmaf(-G.z, ux, px)), half * fmaf(-G.w, vx, fmaf(-G.z, uy, py)));
                o01 = make_float2(half * fmaf(G.w, uy, fmaf(-G.z, vx, mx)), half * fmaf(-G.w, ux, fmaf(-G.z, vy, my)));
                o10 = make_float2(half * fmaf(-G.w, uy, fmaf(G.z, vx, mx)), half * fmaf(G.w, ux, fmaf(G.z, vy, my)));
              }
              if (ss.y) {
                const uint32_t pr = (__popc(r0 & ss.y) & 1u) << 31, pc = (__popc(c0 & ss.y) & 1u) << 31;
                o01 = flip_sign(o01, pc);
                o10 = flip_sign(o10, pr);
                o11 = flip_sign(o11, pr ^ pc);
              }
              p0[s1] = o01;
              p1[s0] = o10;
              p1[s1] = o11;
            }
          }
      }
      group_sync(TPR, group);
    }
    if (st_code != MBQC_RUN_OK) {
      if (tid == 0 && F0.status) F0.status[run] = st_code;
      group_sync(TPR, group);
      for (int ai = tid; ai < C.n_angles; ai += TPR) grad[ai] = NAN;
      continue;
    }
    // window index <-> storage position of the final matrix (slot bit 0)
    const int ps = (M - 1) % W, hpos = ((M - 1 - ps) % N + N) % N;
    auto pos_of = [&](uint32_t i) { return rotl(((i >> (ps + 1)) << ps) | (i & ((1u << ps) - 1u)), hpos); };
    auto win_of = [&](uint32_t p) { return ins_bit(rotl(p, (N - hpos) % N), ps, 0); };
    // output noise on each output qubit
    auto depolarise = [&](int b) {
      const uint32_t q = pos_of(1u << b);
      const int pos = 31 - __clz(q);
      for (int e = tid; e < NB / 4; e += TPR) {
        const uint32_t r0 = ins_bit((uint32_t)e / (D / 2), pos, 0) * D, r1 = r0 + ((uint32_t)D << pos);
        const uint32_t c = ins_bit((uint32_t)e % (D / 2), pos, 0), c0 = sw(c), c1 = sw(c | (1u << pos));
        const float2 x00 = R[r0 + c0], x01 = R[r0 + c1], x10 = R[r1 + c0], x11 = R[r1 + c1];
        const float2 tr2 = make_float2(x00.x + x11.x, x00.y + x11.y);
        R[r0 + c0] = make_float2(a_n * x00.x + b_n * tr2.x, a_n * x00.y + b_n * tr2.y);
        R[r1 + c1] = make_float2(a_n * x11.x + b_n * tr2.x, a_n * x11.y + b_n * tr2.y);
        R[r0 + c1] = make_float2(a_n * x01.x, a_n * x01.y);
        R[r1 + c0] = make_float2(a_n * x10.x, a_n * x10.y);
      }
      group_sync(TPR, group);
    };
    if (F0.noise != 0.0)
      for (int j = 0; j < C.n_out; ++j) depolarise(C.out_bits[j]);
    // output, and Re<Gamma|rho_out>
    const int dout = 1 << C.n_out;
    const float2 *gam = A.grad_out + run * A.gout_stride;
    for (int i = tid; i < 1 << W; i += TPR) {
      const int y = __ldg(&map[i]).y;
      sMap[i] = y >= 0 ? (y << 8) | (int)pos_of((uint32_t)i) : -1;
    }
    group_sync(TPR, group);
    float zpart = 0.f;
    for (int e = tid; e < 1 << (2 * W); e += TPR) {
      const int mi = sMap[e >> W], mj = sMap[e & ((1 << W) - 1)];
      if ((mi | mj) >= 0) {
        const int o = (mi >> 8) * dout + (mj >> 8);
        const float2 x = R[(mi & 255) * D + sw(mj & 255)], g = gam[o];
        zpart += fmaf(g.x, x.x, __fmul_rn(g.y, x.y));
        if (F0.rho_out) F0.rho_out[run * F0.out_stride + o] = x;
      }
    }
    const float2 zp = group_sum2<TPR>(zpart, sGr, tid, group);
    const float z = zp.x + zp.y;
    group_sync(TPR, group);
    // seed Lambda = Gamma - z I on the output subspace
    for (int e = tid; e < NB; e += TPR) {
      const uint32_t r = (uint32_t)e / D, c = (uint32_t)e % D;
      const int mi = sMap[win_of(r)], mj = sMap[win_of(c)];
      float2 l = make_float2(0.f, 0.f);
      if ((mi | mj) >= 0) {
        l = gam[(mi >> 8) * dout + (mj >> 8)];
        if (mi == mj) l.x -= z;
      }
      R[r * D + sw(c)] = l;
    }
    group_sync(TPR, group);
    if (F0.noise != 0.0)
      for (int j = C.n_out - 1; j >= 0; --j) depolarise(C.out_bits[j]);

    // ---------------------------------------------------------- backward
    // R holds mu_{M-1} (the last step shrinks the window), then m_{k+1}
    for (int k = M - 1; k >= 0; --k) {
      const uint2 ss = sSt[k];
      const float ck = sInv[k];
      const int pa = (k + N - 1) % N, pb = k % N;
      float *tb = tmp + (k & 1) * NB;
      if (tiled) {
        const int plo = pa < pb ? pa : pb, phi = pa < pb ? pb : pa;
        const uint32_t rb = ins_bit(ins_bit(tr, plo, 0), phi, 0), cb = ins_bit(ins_bit(tc, plo, 0), phi, 0);
        const float4 *hk = hist + (int64_t)k * Cfg::HIST;
        float4 hv[4];  // the measured qubit's coherences, in flight early
        if ((ss.x & kAdjOff) && k > 0) {
#pragma unroll
          for (int g = 0; g < 4; ++g) hv[g] = hk[g * (T * T)];
        }
        // row and column i, i = (position a) + 2 (position b)
        auto row = [&](int i) { return rb | ((uint32_t)(i & 1) << pa) | ((uint32_t)(i >> 1) << pb); };
        auto col = [&](int j) { return cb | ((uint32_t)(j & 1) << pa) | ((uint32_t)(j >> 1) << pb); };
        uint32_t rp[4], cp[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          rp[i] = row(i) * D;
          cp[i] = sw(col(i));
        }
        float2 mu[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) mu[i][j] = R[rp[i] + cp[j]];
        if (k < M - 1) {
          // Lambda_k from m_{k+1} and step k+1's functional, then mu_k = E^dagger Lambda_k
          float4 G = sF[k + 1];
          if (sOut[k + 1]) G = make_float4(tr_noise - G.x, tr_noise - G.y, -G.z, -G.w);
          const uint2 sn = sSt[k + 1];
          const bool mqn = (sn.x & kFactMq) != 0u, dead = (sn.x & kFactDead) != 0u;
          if (sn.y) {  // the slot's links to the qubits other than the next measured one
#pragma unroll
            for (int o = 0; o < 2; ++o) {
              const uint32_t prs = (__popc(row(o) & sn.y) & 1u) << 31, pcs = (__popc(col(o) & sn.y) & 1u) << 31;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                mu[2 + o][j] = flip_sign(mu[2 + o][j], prs);
                mu[j][2 + o] = flip_sign(mu[j][2 + o], pcs);
              }
            }
          }
          // Lambda entry of (x, x') from m: conj(G_xx') m, rounded before the
          // sums as the stored entries were
          auto lam = [&](int x, int xp, float2 m) {
            if (x == 0 && xp == 0) return make_float2(__fmul_rn(G.x, m.x), __fmul_rn(G.x, m.y));
            if (x == 1 && xp == 1) return make_float2(__fmul_rn(G.y, m.x), __fmul_rn(G.y, m.y));
            const float zx = __fmul_rn(G.z, m.x), wx = __fmul_rn(G.w, m.x);
            if (x == 0) return make_float2(fmaf(G.w, m.y, zx), fmaf(G.z, m.y, -wx));  // conj(G01) m
            return make_float2(fmaf(-G.w, m.y, zx), fmaf(G.z, m.y, wx));              // G01 m
          };
#pragma unroll
          for (int orr = 0; orr < 2; ++orr)
#pragma unroll
            for (int oc = 0; oc < 2; ++oc) {
              const float2 m00 = mu[orr][oc], m01 = mu[orr][oc + 2], m10 = mu[orr + 2][oc], m11 = mu[orr + 2][oc + 2];
              if (mqn && !dead && G.x == G.y) {
                // XY, linked slot: the signs (-1)^x on slot row 1 and (-1)^x' on
                // slot column 1 are additions or subtractions; one product for
                // the two populations
                auto add4 = [](float2 a, float2 b, float2 c, float2 d, float sb, float sc, float sd) {
                  return make_float2(0.5f * (a.x + sb * b.x + sc * c.x + sd * d.x),
                                     0.5f * (a.y + sb * b.y + sc * c.y + sd * d.y));
                };
                const float2 q0 = lam(0, 0, m00), q1 = lam(0, 0, m01), q2 = lam(0, 0, m10), q3 = lam(0, 0, m11);
                mu[orr][oc] = add4(q0, q1, q2, q3, 1.f, 1.f, 1.f);
                mu[orr + 2][oc + 2] = add4(q0, q1, q2, q3, -1.f, -1.f, 1.f);
                mu[orr][oc + 2] = add4(lam(0, 1, m00), lam(0, 1, m01), lam(0, 1, m10), lam(0, 1, m11), -1.f, 1.f, -1.f);
                mu[orr + 2][oc] = add4(lam(1, 0, m00), lam(1, 0, m01), lam(1, 0, m10), lam(1, 0, m11), 1.f, -1.f, -1.f);
                continue;
              }
#pragma unroll
              for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int xp = 0; xp < 2; ++xp) {
                  float2 v = lam(x, xp, m00);
                  if (!dead) {
                    const uint32_t sx = x && mqn ? 0x80000000u : 0u, sxp = xp && mqn ? 0x80000000u : 0u;
                    const float2 l01 = flip_sign(lam(x, xp, m01), sxp), l10 = flip_sign(lam(x, xp, m10), sx);
                    const float2 l11 = flip_sign(lam(x, xp, m11), sx ^ sxp);
                    v = make_float2(0.5f * (v.x + l01.x + l10.x + l11.x), 0.5f * (v.y + l01.y + l10.y + l11.y));
                  }
                  mu[orr + 2 * x][oc + 2 * xp] = v;
                }
            }
        }
        // derivative terms Re(conj(mu) dsigma), each to its full-matrix thread
        if (ss.x & kAdjOff) {
          const int h = ((k % W - k) % N + N) % N;  // position -> bit of the full-matrix block index
          const bool mq = (ss.x & kFactMq) != 0u, pdead = (ss.x & kFactDead) != 0u;
          uint32_t tp[4], tq[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t r = rotl(row(i), h), c = rotl(col(i), h);
            tp[i] = (r * D) ^ (N == 6 ? (__popc(r) & 1u) * 21u : 0u);
            tq[i] = N == 6 ? c ^ ((c >> 5) * 10u) : c;
          }
          auto term = [&](int i, int j, float2 d) {
            tb[tp[i] ^ tq[j]] = fmaf(mu[i][j].x, d.x, __fmul_rn(mu[i][j].y, d.y));
          };
          if (!(ss.x & kAdjPop) && k > 0 && mq && !pdead) {
            // XY, linked slot: dG = (0, 0, -Im G01, Re G01), the coherences' quarter
            // turn; the four copies of a block give +-two values
            const float4 F = sF[k];
            const float dz = sOut[k] ? F.w : -F.w, dw = sOut[k] ? -F.z : F.z;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const int xr = g >> 1, xc = g & 1;
              const float4 v = hv[g];  // y01, y10
              const float ux = v.x + v.z, uy = v.y + v.w, vx = v.x - v.z, vy = v.y - v.w;
              float2 d0 = make_float2(fmaf(-dw, vy, __fmul_rn(dz, ux)), fmaf(dw, vx, __fmul_rn(dz, uy)));
              float2 d1 = make_float2(fmaf(dw, uy, __fmul_rn(-dz, vx)), fmaf(-dw, ux, __fmul_rn(-dz, vy)));
              float2 d2 = make_float2(-d1.x, -d1.y), d3 = make_float2(-d0.x, -d0.y);
              if (ss.y) {
                const uint32_t prs = (__popc(row(2 * xr) & ss.y) & 1u) << 31, pcs = (__popc(col(2 * xc) & ss.y) & 1u) << 31;
                d1 = flip_sign(d1, pcs);
                d2 = flip_sign(d2, prs);
                d3 = flip_sign(d3, prs ^ pcs);
              }
              term(2 * xr, 2 * xc, d0);
              term(2 * xr, 2 * xc + 1, d1);
              term(2 * xr + 1, 2 * xc, d2);
              term(2 * xr + 1, 2 * xc + 1, d3);
            }
          } else {
            float4 dG;
            if (ss.x & kAdjPop) {
              const DevStep st = steps[k];
              float dx, dy, dz;
              dbloch(st.plane, ang[st.aidx], dx, dy, dz);
              dG = make_float4(a_n * 0.5f * dz, -a_n * 0.5f * dz, a_n * 0.5f * dx, a_n * 0.5f * dy);
            } else {
              const float4 F = sF[k];
              dG = make_float4(0.f, 0.f, -F.w, F.z);
            }
            if (sOut[k]) dG = make_float4(-dG.x, -dG.y, -dG.z, -dG.w);
#pragma unroll 1
            for (int e = 0; e < 16; ++e) {  // rows and columns over (slot, next measured)
              const int xr = e >> 3, xc = (e >> 2) & 1, ar = (e >> 1) & 1, ac = e & 1;
              const uint32_t r = rb | ((uint32_t)ar << pa) | ((uint32_t)xr << pb);
              const uint32_t c = cb | ((uint32_t)ac << pa) | ((uint32_t)xc << pb);
              float2 x00 = make_float2(0.f, 0.f), x01 = x00, x10 = x00, x11 = x00;
              if (k == 0) {  // the initial matrix has no slot: each (r, c) has its own block
                x00 = rho0(2 * r, 2 * c);
                x01 = rho0(2 * r, 2 * c + 1);
                x10 = rho0(2 * r + 1, 2 * c);
                x11 = rho0(2 * r + 1, 2 * c + 1);
              } else if (!(pdead && (ar || ac))) {
                const float4 v = hk[(2 * xr + xc) * (T * T)];
                float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
                if (ss.x & kAdjPop) w = hk[(4 + 2 * xr + xc) * (T * T)];
                // entries of the block with slot bits (ar, ac)
                const uint32_t prs = (__popc((rb | ((uint32_t)xr << pb)) & ss.y) & 1u) << 31;
                const uint32_t pcs = (__popc((cb | ((uint32_t)xc << pb)) & ss.y) & 1u) << 31;
                const uint32_t s = (ar ? prs : 0u) ^ (ac ? pcs : 0u);
                const uint32_t sr = ar && mq ? 0x80000000u : 0u, sc = ac && mq ? 0x80000000u : 0u;
                x00 = flip_sign(make_float2(w.x, w.y), s);
                x01 = flip_sign(make_float2(v.x, v.y), s ^ sc);
                x10 = flip_sign(make_float2(v.z, v.w), s ^ sr);
                x11 = flip_sign(make_float2(w.z, w.w), s ^ sr ^ sc);
              }
              const float2 d = functional(dG, x00, x01, x10, x11);
              float2 m = mu[0][0];
#pragma unroll
              for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                  if (i == ar + 2 * xr && j == ac + 2 * xc) m = mu[i][j];
              const uint32_t rr = rotl(r, h), cc = rotl(c, h);
              tb[(rr * D) ^ (N == 6 ? (cc ^ ((cc >> 5) * 10u)) ^ ((__popc(rr) & 1u) * 21u) : cc)] =
                  fmaf(m.x, d.x, __fmul_rn(m.y, d.y));
            }
          }
        }
        // m_k = mu_k / prob_k
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) R[rp[i] + cp[j]] = make_float2(ck * mu[i][j].x, ck * mu[i][j].y);
      }
      group_sync(TPR, group);
      // the partial sums of the step before (their warps wrote them before this barrier)
      auto finish = [&](int kk) {
        float2 p = sGr[(kk & 1) * 8];
#pragma unroll
        for (int i = 1; i < NW; ++i) {
          const float2 q = sGr[(kk & 1) * 8 + i];
          two_sum_acc(p.x, p.y, q.x, q.y);
        }
        const float s = p.x + p.y;  // renormalised pair hi + lo, then their sum
        const float gk = s + (p.y - (s - p.x));
        grad[steps[kk].aidx] = (double)(sInv[kk] * gk);
      };
      if (tid == 0 && k + 1 < M && (sSt[k + 1].x & kAdjOff)) finish(k + 1);
      if (ss.x & kAdjOff) {
        float g = 0.f;
        const uint32_t c = (uint32_t)tid % D, r0 = (uint32_t)tid / D;
        const uint32_t at = r0 * D + (N == 6 ? c ^ ((c >> 5) * 10u) ^ ((__popc(r0) & 1u) * 21u) : c);
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          constexpr uint32_t step = (uint32_t)RS * D;
          const uint32_t odd = ((i ^ (i >> 1) ^ (i >> 2) ^ (i >> 3)) & 1) && N == 6 ? 21u : 0u;
          g += tb[(at ^ odd) + i * step];
        }
        float hi = g, lo = 0.f;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
          const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
          const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
          two_sum_acc(hi, lo, oh, ol);
        }
        if ((tid & 31) == 0) sGr[(k & 1) * 8 + (tid >> 5)] = make_float2(hi, lo);
      }
      if (k == 0) {
        group_sync(TPR, group);
        if (tid == 0 && (ss.x & kAdjOff)) finish(0);
      }
    }
    if (tid == 0 && F0.status) F0.status[run] = MBQC_RUN_OK;
  }
}

}  // namespace mbqc
