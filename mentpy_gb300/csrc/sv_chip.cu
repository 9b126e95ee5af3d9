// Wide-window statevector sweep on chip, windows 11..17: the kept half of a run's
// window (phi_k, 2^(w-1) amplitudes: sv_stream.cu) stays in the shared memory of
// one block, or of a cluster of 2, 4 or 8 blocks with NS = 2^SB amplitudes each,
// from the first window to the output: one launch, no workspace traffic.
//
// Qubit s of the schedule sits at bit (s - 1) mod (w - 1) and step k works on bit
// (k - 1) mod (w - 1), so a cycle of w - 1 steps goes once over the bits.  A thread
// holds 32 amplitudes, five bits at a time: bits 0..4, 5..9 and SB - 5..SB - 1 (of
// which the steps from bit 10 on are left), a block barrier after each; the bits
// that number the cluster's blocks are one pass whose items take an amplitude of
// every block through distributed shared memory.  Amplitude e lies at place(e) =
// e with bits 5..13 folded onto 1..3: pairs stay together (16-byte accesses on bits
// 0..4 and between blocks) and a warp finds the banks whichever bits its lanes
// leave out.
//
// An exact power-of-two scale follows from the norm twice a cycle (after bits 0..4
// and before the blocks' bits); a final float-pair sum normalises.  Scale, phase
// and log-probability are those of the streamed sweep, the amplitudes its bits.
//
// What bounds it is the alternation of load, compute and store phases between the
// barriers: w = 17, 64 runs issue in 38 % of the slots at one block (16 warps) an SM,
// shared memory and DRAM far from their rates (two blocks an SM, windows up to 14,
// overlap the phases: a quarter better).  Against the streamed passes: grid 16 x 10 (w = 17),
// 64 runs 577 -> 453 us (two rounds of 38 clusters), 16 runs 264 -> 214; 14 x 10,
// 256 runs 509 -> 274; 12 x 10 (w = 13), 1,000 runs 594 (whole window streamed) ->
// 240; 10 x 10, 512 runs 149 -> 77 us.  w = 18 (eight blocks a run) was slower, 64
// runs 558 -> 703 us: those stream.
#include <cuda_runtime.h>

#include <algorithm>

#include "cluster_sum.cuh"
#include "dispatch.h"
#include "sv_stream.cuh"

namespace mbqc {

constexpr int kChipMaxSB = 14;  // 128 KB of amplitudes a block
constexpr int kChipFlagOwn = 29, kChipFlagCpl = 30;  // of a step's stored mask (bit 31: kDead)

struct ChipDesc {
  int8_t in_e[16];   // slice bits in the order of the input bits they hold
  int n_free;        // output bits inside a slice
  int8_t out_y[16];  // those output bits, ascending
  int8_t out_e[16];  // their slice bits
  int8_t rank_y[4];  // output bit of each rank bit, -1 = none
};

__host__ __device__ constexpr uint32_t chip_place(uint32_t e) {
  return e ^ ((((e >> 5) ^ (e >> 8) ^ (e >> 11)) & 7u) << 1);
}

// shared memory: [amplitudes][coef M][mask M][sign pattern M][thread tables 8 x BT][pass tables 5 x 32]
static size_t chip_smem(int sb, int M) {
  const size_t bt = (size_t)1 << (sb - 5);
  return ((size_t)8 << sb) + (size_t)M * 16 + bt * 32 + 5 * 32 * 4 + 64;
}

template <int SB, int CS>
__global__ void __launch_bounds__(1 << (SB - 5), SB >= 14 ? 1 : 512 >> (SB - 5))
    sv_chip(StreamArgs a, ChipDesc d, uint32_t flags, int lp_const, float2 *out, double *logprob, int32_t *status) {
  constexpr int NS = 1 << SB, BT = NS / 32, NW = BT / 32;
  constexpr int LOGCS = CS == 8 ? 3 : (CS == 4 ? 2 : (CS == 2 ? 1 : 0));
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float s_part[2][NW], s_tot[2];
  __shared__ float2 s_pair[NW], s_red[2], s_ph[NW];
  float2 *s = reinterpret_cast<float2 *>(smem);
  const int M = a.M, W = a.W, H = W - 1;
  float2 *s_coef = s + NS;
  uint32_t *s_mask = reinterpret_cast<uint32_t *>(s_coef + M), *s_ptab = s_mask + M;
  uint32_t *s_thr = s_ptab + M;         // [8][BT]: input x(0), x(1), couplings(0), (1), e | signs; output e, y
  uint32_t *s_it = s_thr + 8 * BT;      // [5][32]: input x | sign, couplings, e; output e, y
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  int crank = 0, cid = blockIdx.x, ncl = gridDim.x;
  if constexpr (CS > 1) {
    crank = (int)cg::this_cluster().block_rank();
    cid = blockIdx.x / CS;
    ncl = gridDim.x / CS;
  }
  const uint32_t e_hi = (uint32_t)crank << SB;

  // ---- tables of the plan: masks on the stored bits, index parts
  for (int k = tid + 1; k < M; k += BT) {
    const uint32_t prev = a.steps[k - 1].mask;
    uint32_t m = prev & kDead;
    for (int q = k + 1; q <= k + W - 2; ++q)
      if ((prev >> (q % W)) & 1u) m |= 1u << ((q - 1) % H);
    if ((prev >> (k % W)) & 1u) m |= 1u << kChipFlagCpl;
    if ((prev >> ((k - 1) % W)) & 1u) m |= 1u << kChipFlagOwn;
    s_mask[k] = m;
    const int b = (k - 1) % H, b0 = b < 5 ? 0 : (b < 10 ? 5 : SB - 5);
    s_ptab[k] = parity_table((m >> b0) & 31u, 5) ^ (((m >> kChipFlagOwn) & 1u) ? ~0u : 0u);
  }
  auto couplings = [&](uint32_t v) {
    uint32_t x = 0;
    for (int q = 0; q < W; ++q) x ^= (0u - ((v >> q) & 1u)) & a.init_cz[q];
    return x;
  };
  auto in_bits_of = [&](uint32_t j) {  // slice index of input-order index j
    uint32_t e = 0;
    for (int t = 0; t < SB; ++t) e |= ((j >> t) & 1u) << d.in_e[t];
    return e;
  };
  auto out_bits_of = [&](uint32_t j, const int8_t *bits) {
    uint32_t e = 0;
    for (int t = 0; t < d.n_free; ++t) e |= ((j >> t) & 1u) << bits[t];
    return e;
  };
  {
    const uint32_t e = in_bits_of((uint32_t)tid), i = (e_hi | e) << 1;
    s_thr[tid] = (uint32_t)gather_bits(i, a.in_bits, a.n_in);
    s_thr[BT + tid] = (uint32_t)gather_bits(i | 1u, a.in_bits, a.n_in);
    s_thr[2 * BT + tid] = couplings(i);
    s_thr[3 * BT + tid] = couplings(i | 1u);
    s_thr[4 * BT + tid] =
        e | (init_parity(i, a.init_cz, W) << 30) | (init_parity(i | 1u, a.init_cz, W) << 31);
    s_thr[5 * BT + tid] = chip_place(out_bits_of((uint32_t)tid, d.out_e));
    s_thr[6 * BT + tid] = out_bits_of((uint32_t)tid, d.out_y);
    if (tid < 32) {
      const uint32_t en = in_bits_of((uint32_t)tid * BT), in2 = en << 1;
      s_it[tid] = (uint32_t)gather_bits(in2, a.in_bits, a.n_in) | (init_parity(in2, a.init_cz, W) << 31);
      s_it[32 + tid] = couplings(in2);
      s_it[64 + tid] = en;
      s_it[96 + tid] = chip_place(out_bits_of((uint32_t)tid * BT, d.out_e));
      s_it[128 + tid] = out_bits_of((uint32_t)tid * BT, d.out_y);
    }
  }
  uint32_t y_rank = 0;
  bool has_out = true;
  for (int r = 0; r < LOGCS; ++r)
    if ((crank >> r) & 1) {
      if (d.rank_y[r] < 0)
        has_out = false;
      else
        y_rank |= 1u << d.rank_y[r];
    }

  // Norms that choose a scale are float sums over a warp (as the streamed passes'),
  // a block and a cluster.  Only their exponent is used and the scale is exact, so
  // their rounding reaches no result; their range has to be that of the warps'
  // parts: a total that a float cannot hold is kept as minus its 2^-8 times.
  constexpr float kDown = 0.00390625f;
  auto renorm_of = [](float t) {  // half the exponent of a norm
    const int up = t < 0.f ? 8 : 0;
    t = up ? -t : t;
    if (!RealBits<float>::finite_pos(t)) return 0;
    const int f = (RealBits<float>::expo(t) + up) >> 1;
    return f > 100 ? 100 : (f < -100 ? -100 : f);
  };
  // norm of the amplitudes a thread holds, and the block's in s_part[x]
  auto add_norm = [&](const float2 (&v)[32], int x) {
    float p[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int z = 0; z < 32; ++z) p[z & 3] = fmaf(v[z].x, v[z].x, fmaf(v[z].y, v[z].y, p[z & 3]));
    float t = (p[0] + p[1]) + (p[2] + p[3]);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) s_part[x][wid] = t;
  };
  auto block_total = [&](int x) {
    float t = 0.f;
    for (int i = 0; i < NW; ++i) t += s_part[x][i];
    if (t > 3.0e38f) {
      t = 0.f;
      for (int i = 0; i < NW; ++i) t -= kDown * s_part[x][i];
    }
    return t;
  };
  auto run_total = [&](int x) {  // the same in every block
    if constexpr (CS == 1) {
      return block_total(x);
    } else {
      float q[CS], t = 0.f, low = 0.f;
#pragma unroll
      for (int r = 0; r < CS; ++r) {
        q[r] = *cg::this_cluster().map_shared_rank(&s_tot[x], r);
        t += q[r];
        low = fminf(low, q[r]);
      }
      if (low < 0.f || t > 3.0e38f) {
        t = 0.f;
#pragma unroll
        for (int r = 0; r < CS; ++r) t += q[r] < 0.f ? q[r] : -kDown * q[r];
      }
      return t;
    }
  };
  auto scale = [&](float2 (&v)[32], int x, int &expo) {
    const int e = renorm_of(run_total(x));
    if (e) {
      const float al = RealBits<float>::pow2(-e);
      expo += e;
#pragma unroll
      for (int z = 0; z < 32; ++z) v[z] = make_float2(al * v[z].x, al * v[z].y);
    }
  };

  for (int64_t run = cid; run < a.B; run += ncl) {
    // ---- coefficients, the phase product, the input's norm
    float2 ph = make_float2(1.f, 0.f);
    for (int k = tid; k < M; k += BT) {
      const DevStep st = a.steps[k];
      const double th = st.aidx >= 0 ? a.angles[run * a.astride + st.aidx] : st.fixed;
      float2 c, p;
      sv_coef(st.plane, th, (flags & MBQC_F_REF_PHASE) != 0u, c, p);
      s_coef[k] = c;
      if (flags & MBQC_F_REF_PHASE) ph = cmul(ph, p);
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1)
      ph = cmul(ph, make_float2(__shfl_xor_sync(0xffffffffu, ph.x, o), __shfl_xor_sync(0xffffffffu, ph.y, o)));
    if (lane == 0) s_ph[wid] = ph;
    __syncthreads();

    auto pair_sum = [&](float2 t) {  // over the block, in s_red[0]'s order for every thread
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1)
        two_sum_acc(t.x, t.y, __shfl_xor_sync(0xffffffffu, t.x, o), __shfl_xor_sync(0xffffffffu, t.y, o));
      __syncthreads();
      if (lane == 0) s_pair[wid] = t;
      __syncthreads();
      t = s_pair[0];
      for (int i = 1; i < NW; ++i) two_sum_acc(t.x, t.y, s_pair[i].x, s_pair[i].y);
      return t;
    };
    const float2 *in = a.psi_in + (a.istride ? run * a.istride : 0);
    float2 nin = make_float2(1.f, 0.f);  // before any output: the outputs may lie on the inputs
    if (logprob && crank == 0) {
      nin.x = 0.f;
      for (int x = tid; x < (1 << a.n_in); x += BT) {
        const float2 v = in[x];
        two_sum_acc(nin.x, nin.y, v.x * v.x + v.y * v.y, 0.f);
      }
      nin = pair_sum(nin);
    }
    // ---- phi_0 from the input: index parts as in stream_init
    {
      const uint32_t x0 = s_thr[tid], x1 = s_thr[BT + tid], a0 = s_thr[2 * BT + tid], a1 = s_thr[3 * BT + tid];
      const uint32_t et = s_thr[4 * BT + tid], q0 = (et >> 30) & 1u, q1 = et >> 31, e = et & (NS - 1);
      const uint32_t i0 = (e_hi | e) << 1;
      const float2 c = s_coef[0];
#pragma unroll 8
      for (int n = 0; n < 32; ++n) {
        const uint32_t xn = s_it[n], an = s_it[32 + n], en = s_it[64 + n], in2 = en << 1;
        const uint32_t o0 = q0 ^ (xn >> 31) ^ (uint32_t)__popc(in2 & a0) ^ (uint32_t)__popc(i0 & an);
        const uint32_t o1 = q1 ^ (xn >> 31) ^ (uint32_t)__popc(in2 & a1) ^ (uint32_t)__popc((i0 | 1u) & an);
        float2 v[2] = {flip_sign(__ldg(in + (x0 ^ (xn & 0x7fffffffu))), o0 << 31),
                       flip_sign(__ldg(in + (x1 ^ (xn & 0x7fffffffu))), o1 << 31)};
        pass_reg_step<false, 2, 0>(v, c, 1.f, 0u, false);
        s[chip_place(e ^ en)] = v[0];
      }
    }
    __syncthreads();

    // ---- cycles of H steps
    int expo = 0;
    bool pend = false;  // s_part[1] holds a norm that has not been applied (one block)
    auto group = [&](auto b0c, int k, int j0, int j1, int scale_x, int norm_x) {
      constexpr int B0 = decltype(b0c)::value;
      const uint32_t e0 = (((uint32_t)tid >> B0) << (B0 + 5)) | ((uint32_t)tid & ((1u << B0) - 1u));
      const uint32_t p0 = chip_place(e0), full = e_hi | e0;
      float2 v[32];
#pragma unroll
      for (int z = 0; z < 32; ++z) {
        if constexpr (B0 == 0) {
          if (z & 1) continue;
          const float4 x = *reinterpret_cast<const float4 *>(s + (p0 ^ (uint32_t)z));
          v[z] = make_float2(x.x, x.y);
          v[z | 1] = make_float2(x.z, x.w);
        } else {
          v[z] = s[p0 ^ chip_place((uint32_t)z << B0)];
        }
      }
      if (scale_x >= 0) scale(v, scale_x, expo);
      auto step = [&](auto jc) {
        constexpr int J = decltype(jc)::value;
        if (J < j0 || J >= j1) return;
        const int kk = k + J - j0;
        const uint32_t m = s_mask[kk];
        const uint32_t ts = s_ptab[kk] ^ (0u - (__popc(full & m & 0xfffffu) & 1u));
        pass_half_step<false, 32, J>(v, s_coef[kk], 1.f, (m >> kChipFlagCpl) << 31, ts, (m & kDead) != 0u);
      };
      step(std::integral_constant<int, 0>{});
      step(std::integral_constant<int, 1>{});
      step(std::integral_constant<int, 2>{});
      step(std::integral_constant<int, 3>{});
      step(std::integral_constant<int, 4>{});
#pragma unroll
      for (int z = 0; z < 32; ++z) {
        if constexpr (B0 == 0) {
          if (z & 1) continue;
          *reinterpret_cast<float4 *>(s + (p0 ^ (uint32_t)z)) = make_float4(v[z].x, v[z].y, v[z | 1].x, v[z | 1].y);
        } else {
          s[p0 ^ chip_place((uint32_t)z << B0)] = v[z];
        }
      }
      if (norm_x >= 0) add_norm(v, norm_x);
    };
    for (int k = 1; k < M;) {
      int n = min(5, M - k);
      group(std::integral_constant<int, 0>{}, k, 0, n, CS == 1 && pend ? 1 : -1, SB == 10 ? -1 : 0);
      pend = false;
      k += n;
      __syncthreads();
      if (k >= M) break;
      n = min(5, M - k);
      if (CS > 1 && tid == 0) s_tot[0] = block_total(0);
      group(std::integral_constant<int, 5>{}, k, 0, n, -1, SB == 10 ? 1 : -1);
      k += n;
      run_barrier<CS>();
      if constexpr (SB == 10) pend = true;
      if (k >= M) break;
      if constexpr (SB > 10) {
        constexpr int j0 = 15 - SB;
        n = min(5 - j0, M - k);
        group(std::integral_constant<int, SB - 5>{}, k, j0, j0 + n, 0, 1);
        k += n;
        __syncthreads();
        pend = true;
      }
      if constexpr (CS > 1) {
        if (k >= M) break;
        if (tid == 0) s_tot[1] = block_total(1);
        cg::this_cluster().sync();
        constexpr int IT = 32 / CS;
        const uint32_t l0 = (uint32_t)(crank * (NS / CS) + 2 * tid);
        auto item = [&](int i) { return l0 + (uint32_t)((i >> 1) * 2 * BT + (i & 1)); };
        float2 v[32];  // item i, block r at i CS + r; items in neighbouring pairs
#pragma unroll
        for (int r = 0; r < CS; ++r) {
          const float2 *sr = cg::this_cluster().map_shared_rank(s, r);
#pragma unroll
          for (int i = 0; i < IT; i += 2) {
            const float4 x = *reinterpret_cast<const float4 *>(sr + chip_place(item(i)));
            v[i * CS + r] = make_float2(x.x, x.y);
            v[(i + 1) * CS + r] = make_float2(x.z, x.w);
          }
        }
        scale(v, 1, expo);
        n = min(LOGCS, M - k);
        auto step = [&](auto fc) {
          constexpr int F = decltype(fc)::value;
          if (F >= n) return;
          const uint32_t m = s_mask[k + F];
          const float2 c = s_coef[k + F], c1 = flip_sign(c, (m >> kChipFlagCpl) << 31);
          const bool dead = (m & kDead) != 0u;
#pragma unroll
          for (int i = 0; i < IT; ++i) {
            const uint32_t base = (uint32_t)__popc(item(i) & m & 0xfffffu) ^ (m >> kChipFlagOwn);
#pragma unroll
            for (int r = 0; r < CS; ++r) {
              if ((r >> F) & 1) continue;
              const float2 x0 = v[i * CS + r], x1 = v[i * CS + (r | (1 << F))];
              v[i * CS + r] = make_float2(x0.x + c.x * x1.x - c.y * x1.y, x0.y + c.x * x1.y + c.y * x1.x);
              const float2 o =
                  make_float2(x0.x + c1.x * x1.x - c1.y * x1.y, x0.y + c1.x * x1.y + c1.y * x1.x);
              const uint32_t odd = base ^ (uint32_t)__popc(((uint32_t)r << SB) & m & 0xfffffu);
              v[i * CS + (r | (1 << F))] = dead ? make_float2(0.f, 0.f) : flip_sign(o, odd << 31);
            }
          }
        };
        step(std::integral_constant<int, 0>{});
        if constexpr (LOGCS > 1) step(std::integral_constant<int, 1>{});
        if constexpr (LOGCS > 2) step(std::integral_constant<int, 2>{});
        k += n;
#pragma unroll
        for (int r = 0; r < CS; ++r) {
          float2 *sr = cg::this_cluster().map_shared_rank(s, r);
#pragma unroll
          for (int i = 0; i < IT; i += 2)
            *reinterpret_cast<float4 *>(sr + chip_place(item(i))) =
                make_float4(v[i * CS + r].x, v[i * CS + r].y, v[(i + 1) * CS + r].x, v[(i + 1) * CS + r].y);
        }
        cg::this_cluster().sync();
      }
    }

    // ---- normalise (float-pair sums), phase, outputs in the reference's order
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll 8
    for (int i = 0; i < 32; ++i) {
      const float2 x = s[tid + i * BT];
      two_sum_acc(acc.x, acc.y, x.x * x.x + x.y * x.y, 0.f);
    }
    float2 n2p = pair_sum(acc);
    if constexpr (CS > 1) {
      if (tid == 0) s_red[0] = n2p;
      cg::this_cluster().sync();
      n2p = *cg::this_cluster().map_shared_rank(&s_red[0], 0);
#pragma unroll
      for (int r = 1; r < CS; ++r) {
        const float2 o = *cg::this_cluster().map_shared_rank(&s_red[0], r);
        two_sum_acc(n2p.x, n2p.y, o.x, o.y);
      }
    }
    const float n2 = n2p.x + n2p.y;
    const bool ok = (n2 > 0.f) && (n2 < 3.0e38f);
    float inv = rsqrtf(n2);
    inv = ok ? inv * (1.5f - 0.5f * n2 * inv * inv) : NAN;  // one Newton step
    ph = s_ph[0];
    for (int i = 1; i < NW; ++i) ph = cmul(ph, s_ph[i]);
    const float2 sc = make_float2(ph.x * inv, ph.y * inv);
    if (has_out) {
      float2 *o = out + (run << a.n_out) + y_rank;
      const uint32_t et = s_thr[5 * BT + tid], yt = s_thr[6 * BT + tid], cnt = 1u << d.n_free;
#pragma unroll 4
      for (int i = 0; i < 32; ++i)
        if ((uint32_t)(tid + i * BT) < cnt) o[yt | s_it[128 + i]] = cmul(s[et ^ s_it[96 + i]], sc);
    }
    if (crank == 0 && tid == 0) {
      if (status) status[run] = ok ? MBQC_RUN_OK : (isnan(n2) ? MBQC_RUN_NAN : MBQC_RUN_ZERO_NORM);
      if (logprob)
        logprob[run] = log((double)n2p.x + (double)n2p.y) - log((double)nin.x + (double)nin.y) +
                       0.6931471805599453 * (2.0 * expo + lp_const);
    }
    run_barrier<CS>();  // the next run overwrites the tables; other blocks have read this one's norm
  }
}

// Blocks per run: as few as hold the half window at 2^14 amplitudes each, 4 at most
// (eight lose to the streamed passes, see above); twice as many (2^13 each) while the
// batch leaves SMs idle (w = 17, 16 runs: 4 blocks 240, 8 blocks 214 us).  At any batch:
// one run of grid 10 x 10 (w = 11) 121 us on streamed whole windows, 117 on half, 56
// here; 13 x 10 168, 170 and 76; 16 x 10 252, 254 and 139; of 3 columns 43, 45 and 25
// (w = 11), 113, 115 and 57 (w = 17); 128 runs of 16 x 10 1,399, 1,066 and 901.
int chip_plan(const DevCircuit &hc, int64_t batch, size_t *smem) {
  const int H = hc.w - 1;
  if (H < 10 || H > 16) return 0;
  int log = H > kChipMaxSB ? H - kChipMaxSB : 0;
  if (log < 3 && H - log - 1 >= 13 && (batch << (log + 1)) <= sm_count()) ++log;
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return 0;
  *smem = chip_smem(H - log, hc.n_steps);
  return *smem + 1024 <= (size_t)optin ? 1 << log : 0;
}

template <int SB, int CS>
static int chip_launch(const StreamArgs &a, const ChipDesc &d, size_t smem, uint32_t flags, int lp_const, float2 *out,
                       double *logprob, int32_t *status, cudaStream_t s) {
  auto k = sv_chip<SB, CS>;
  const int threads = 1 << (SB - 5);
  int rc = cuda_check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "sv_chip smem");
  if (rc) return rc;
  if (CS == 1) {  // persistent: the tables once a block
    int occ = 0;
    rc = cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, threads, smem), "sv_chip occupancy");
    if (rc) return rc;
    const int64_t nb = std::min<int64_t>(a.B, (int64_t)sm_count() * std::max(occ, 1));
    k<<<(int)nb, threads, smem, s>>>(a, d, flags, lp_const, out, logprob, status);
    return check_launch("sv_chip");
  }
  // a cluster per run: how many are resident depends on the clusters the GPU can place
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(std::min<int64_t>(a.B, 1 << 20) * CS));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CS;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  rc = cuda_check(cudaLaunchKernelEx(&cfg, k, a, d, flags, lp_const, out, logprob, status), "sv_chip cluster launch");
  return rc ? rc : check_launch("sv_chip");
}

int launch_sv_chip(const StreamArgs &a, const DevCircuit &hc, int cs, size_t smem, uint32_t flags, float2 *out,
                   double *logprob, int32_t *status, cudaStream_t s) {
  const int H = hc.w - 1, log = cs == 8 ? 3 : (cs == 4 ? 2 : (cs == 2 ? 1 : 0)), SB = H - log;
  ChipDesc d{};
  // slice bits by the input bit they hold (stored bit b is window bit b + 1 at first); others last
  int key[16], order[16];
  for (int b = 0; b < SB; ++b) {
    key[b] = 64 + b;
    order[b] = b;
    for (int i = 0; i < hc.n_in; ++i)
      if (hc.in_bits[i] == b + 1) key[b] = hc.n_in - 1 - i;
  }
  std::sort(order, order + SB, [&](int x, int y) { return key[x] < key[y]; });
  for (int b = 0; b < SB; ++b) d.in_e[b] = (int8_t)order[b];
  for (int r = 0; r < 4; ++r) d.rank_y[r] = -1;
  for (int j = 0; j < hc.n_out; ++j) {  // output j is bit n_out - 1 - j of y
    const int b = half_bit(hc.out_bits[hc.n_out - 1 - j], hc.n_steps, hc.w);
    if (b < SB) {
      d.out_y[d.n_free] = (int8_t)j;
      d.out_e[d.n_free++] = (int8_t)b;
    } else {
      d.rank_y[b - SB] = (int8_t)j;
    }
  }
  auto go = [&](auto sb, auto c) {
    return chip_launch<decltype(sb)::value, decltype(c)::value>(a, d, smem, flags, hc.lp_const, out, logprob, status, s);
  };
#define MBQC_CHIP(S, C) \
  if (SB == S && cs == C) return go(std::integral_constant<int, S>{}, std::integral_constant<int, C>{});
  MBQC_CHIP(10, 1)
  MBQC_CHIP(11, 1)
  MBQC_CHIP(12, 1)
  MBQC_CHIP(13, 1)
  MBQC_CHIP(14, 1)
  MBQC_CHIP(13, 2)
  MBQC_CHIP(14, 2)
  MBQC_CHIP(13, 4)
  MBQC_CHIP(14, 4)
  MBQC_CHIP(13, 8)
#undef MBQC_CHIP
  return fail(MBQC_E_UNSUPPORTED, "sv_chip: %d bits a block, %d blocks a run", SB, cs);
}

}  // namespace mbqc
