// Statevector sweep of windows 9 and 10 on the kept half of the window (phi_k,
// 2^(w-1) amplitudes: sv_stream.cuh), several runs a warp.
//
// A run owns 2^(w-6) lanes of 32 amplitudes (8 lanes at w = 9, 16 at 10).  Qubit s
// of the schedule sits at bit (s - 1) mod (w - 1): a cycle of w - 1 steps is five
// steps with bits 0..4 in registers, one trip through the warp's shared memory, and
// the other steps with the top five bits in registers.  No shuffle in a step, no
// barrier beyond the warp's.  The full window on 16 or 32 lanes (sv_reg.cuh) spends
// most of its issue on the shuffles of its lane bits.
//
// Each step rounds as that kernel's (a term before its sum on its lane bits, see
// term_step) and the norm is summed as it sums it (2^LL lanes with 2^(w-LL)
// amplitudes of the full window each, pairwise inside a lane, float pairs across),
// so amplitudes before the phase and the log-probability keep their bits; a lane
// here takes V of those lanes in turn.
//
// Against sv_reg: grid 8 x 10 (w = 9), 5,000 runs 105 -> 68 us, 2,500 runs 68 -> 54;
// grid 9 x 10, 5,000 runs 201 -> 140, 1,700 runs 85 -> 62; grids and wires of 3 to 6
// columns, 1,217 to 16,384 runs, no slower than its lane variants.  Latency-bound: 35 %
// of the issue slots at eight warps an SM (5,000 runs), the longest stall for
// instructions (the steps' straight-line code).  Smaller batches stay there: a run here has a quarter to a half of the
// lanes, so that one alone takes 48 us against 21 (sv_half_ok).
#include <cuda_runtime.h>

#include <algorithm>

#include "dispatch.h"
#include "sv_stream.cuh"

namespace mbqc {

__host__ __device__ constexpr uint32_t half_place(uint32_t e) { return e ^ (((e >> 5) & 7u) << 1); }

constexpr int kHalfWarps = 4;

// A step as the register kernel does it on its lane bits: the measured 1-entry's
// term is rounded before it is added (pass_half_step fuses the two).
template <int R, int J>
__device__ __forceinline__ void term_step(float2 (&v)[R], float2 c, uint32_t flip, uint32_t ts, bool dead) {
#pragma unroll
  for (int j = 0; j < R; ++j) {
    if (j & (1 << J)) continue;
    const int jh = j | (1 << J);
    const float2 x0 = v[j], m = v[jh];
    const float2 term = make_float2(fmaf(c.x, m.x, -__fmul_rn(c.y, m.y)), fmaf(c.y, m.x, __fmul_rn(c.x, m.y)));
    const float2 t1 = flip_sign(term, flip);
    v[j] = make_float2(__fadd_rn(x0.x, term.x), __fadd_rn(x0.y, term.y));
    v[jh] = sign_bit_flip(make_float2(__fadd_rn(x0.x, t1.x), __fadd_rn(x0.y, t1.y)), ts * (1u << (31 - jh)));
  }
  if (dead) {
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (j & (1 << J)) v[j] = make_float2(0.f, 0.f);
  }
}

template <int SB>
__host__ __device__ constexpr size_t half_smem(int M) {
  const size_t runs = (size_t)kHalfWarps * (32 >> (SB - 5));
  return runs * ((1u << SB) + 8) * 8 + runs * M * 8 + ((size_t)M * 8 + 15) / 16 * 16 + (8u << SB) + (4u << SB) + (2u << SB);
}

template <int SB, int LL>
__global__ void __launch_bounds__(32 * kHalfWarps, 4) sv_half(SvArgs a) {
  constexpr int W = SB + 1, H = SB, NS = 1 << SB, LR = 1 << (SB - 5), RPW = 32 / LR, STR = NS + 8;
  constexpr int L = 1 << LL, RB = W - LL, R = 1 << RB, V = L / LR;
  static_assert(V >= 1, "sums' lanes");
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, sub = lane / LR, li = lane % LR;
  const int M = a.M;
  float2 *s_state = reinterpret_cast<float2 *>(smem);
  float2 *s_cf = s_state + kHalfWarps * RPW * STR;
  uint32_t *s_mask = reinterpret_cast<uint32_t *>(s_cf + kHalfWarps * RPW * M), *s_ptab = s_mask + M;
  uint2 *s_in = reinterpret_cast<uint2 *>(s_mask + ((M * 2 + 3) & ~3));  // [place(e)]: input index | sign << 31 of 2 e, 2 e + 1
  uint16_t *s_e = reinterpret_cast<uint16_t *>(s_in + NS);   // [full window index]: place, 0xffff = zero
  int16_t *s_out = reinterpret_cast<int16_t *>(s_e + 2 * NS);  // [place(e)]: output index or -1
  float2 *s = s_state + (wid * RPW + sub) * STR;
  float2 *coef = s_cf + (wid * RPW + sub) * M;

  // ---- tables of the plan
  for (int k = tid + 1; k < M; k += 32 * kHalfWarps) {
    const uint32_t prev = a.steps[k - 1].mask;
    uint32_t m = prev & kDead;
    for (int q = k + 1; q <= k + W - 2; ++q)
      if ((prev >> (q % W)) & 1u) m |= 1u << ((q - 1) % H);
    if ((prev >> (k % W)) & 1u) m |= 1u << 30;
    if (k % W >= RB) m |= 1u << 29;  // a lane bit of the register kernel
    const int b = (k - 1) % H, b0 = b < 5 ? 0 : SB - 5;
    s_mask[k] = m;
    s_ptab[k] = parity_table((m >> b0) & 31u, 5) ^ (((prev >> ((k - 1) % W)) & 1u) ? ~0u : 0u);
  }
  for (int e = tid; e < NS; e += 32 * kHalfWarps) {
    s_in[half_place(e)] = make_uint2((uint32_t)a.map[2 * e].x, (uint32_t)a.map[2 * e + 1].x);
    s_out[half_place(e)] = -1;
  }
  __syncthreads();
  for (int i = tid; i < 2 * NS; i += 32 * kHalfWarps) {
    uint32_t e = 0;
    bool zero = false;
    for (int pos = 0; pos < W; ++pos) {
      const int q = M + ((pos - M) % W + W) % W;
      if (!((i >> pos) & 1)) continue;
      if (q == M + W - 1)
        zero = true;  // the last step's slot: no qubit entered
      else
        e |= 1u << ((q - 1) % H);
    }
    s_e[i] = zero ? 0xffff : (uint16_t)half_place(e);
    if (!zero) s_out[half_place(e)] = (int16_t)a.map[i].y;
  }
  __syncthreads();

  const bool want_phase = (a.flags & MBQC_F_REF_PHASE) != 0u;
  const int din = 1 << a.n_in, dout = 1 << a.n_out;
  const int64_t n_groups = (a.B + RPW - 1) / RPW;
  for (int64_t g = (int64_t)blockIdx.x * kHalfWarps + wid; g < n_groups; g += (int64_t)gridDim.x * kHalfWarps) {
    const int64_t run = g * RPW + sub, runc = run < a.B ? run : a.B - 1;
    const double *arow = a.angles + runc * a.astride;
    const float2 *in = reinterpret_cast<const float2 *>(a.psi_in) + (a.istride ? runc * a.istride : 0);
    // ---- coefficients (item i on the sums' lane i mod L), input row
    float2 ph[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      ph[v] = make_float2(1.f, 0.f);
      for (int i = li * V + v; i < M; i += L) {
        int k = i, plane, ai;
        double th;
        if (a.items) {
          const DevItem it = a.items[i];
          k = it.step;
          plane = it.plane;
          ai = i < a.A ? i : -1;
          th = it.fixed;
        } else {
          const DevStep st = a.steps[i];
          plane = st.plane;
          ai = st.aidx;
          th = st.fixed;
        }
        if (ai >= 0) th = arow[ai];
        float2 c, p;
        sv_coef(plane, th, want_phase, c, p);
        coef[k] = c;
        if (want_phase) ph[v] = cmul(ph[v], p);
      }
    }
    for (int x = li; x < din; x += LR) s[x] = in[x];
    __syncwarp();
    // the input's norm, as sv_fwd_reg sums it, before any output is written (they
    // may lie on the inputs); kept in the row's padding
    if (a.logprob && li == 0) {
      float nin = 0.f;
      for (int x = 0; x < din; ++x) nin += fmaf(s[x].x, s[x].x, __fmul_rn(s[x].y, s[x].y));
      s[NS].x = nin;
    }

    float2 v[32];
    {  // phi_0, bits 0..4 in registers
      const float2 c = coef[0];
#pragma unroll
      for (int z = 0; z < 32; ++z) {
        const uint2 x = s_in[half_place((uint32_t)li << 5) ^ (uint32_t)z];
        float2 u[2] = {flip_sign(s[x.x & 0x7fffffffu], x.x & 0x80000000u),
                       flip_sign(s[x.y & 0x7fffffffu], x.y & 0x80000000u)};
        pass_reg_step<false, 2, 0>(u, c, 1.f, 0u, false);
        v[z] = u[0];
      }
      __syncwarp();
    }
    int expo = 0;
    auto steps = [&](auto b0c, int k, int j0, int j1) {
      constexpr int B0 = decltype(b0c)::value;
      const uint32_t full = B0 == 0 ? (uint32_t)li << 5 : (uint32_t)li;
      auto step = [&](auto jc) {
        constexpr int J = decltype(jc)::value;
        if (J < j0 || J >= j1) return;
        const int kk = k + J - j0;
        const uint32_t m = s_mask[kk];
        const uint32_t ts = s_ptab[kk] ^ (0u - (__popc(full & m & 0xfffffu) & 1u));
        if (m & (1u << 29))
          term_step<32, J>(v, coef[kk], (m >> 30) << 31, ts, (m & kDead) != 0u);
        else
          pass_half_step<false, 32, J>(v, coef[kk], 1.f, (m >> 30) << 31, ts, (m & kDead) != 0u);
      };
      step(std::integral_constant<int, 0>{});
      step(std::integral_constant<int, 1>{});
      step(std::integral_constant<int, 2>{});
      step(std::integral_constant<int, 3>{});
      step(std::integral_constant<int, 4>{});
    };
    const uint32_t p0 = half_place((uint32_t)li << 5);
    auto store_low = [&] {
#pragma unroll
      for (int z = 0; z < 32; z += 2)
        *reinterpret_cast<float4 *>(s + (p0 ^ (uint32_t)z)) = make_float4(v[z].x, v[z].y, v[z + 1].x, v[z + 1].y);
    };
    auto load_low = [&] {
#pragma unroll
      for (int z = 0; z < 32; z += 2) {
        const float4 x = *reinterpret_cast<const float4 *>(s + (p0 ^ (uint32_t)z));
        v[z] = make_float2(x.x, x.y);
        v[z + 1] = make_float2(x.z, x.w);
      }
    };
    constexpr int BT = SB - 5, j0 = 10 - SB;
    for (int k = 1;;) {  // amplitudes in registers, bits 0..4
      int n = min(5, M - k);
      if (n > 0) {
        steps(std::integral_constant<int, 0>{}, k, 0, n);
        k += n;
      }
      float t = 0.f;
#pragma unroll
      for (int z = 0; z < 32; ++z) t = fmaf(v[z].x, v[z].x, fmaf(v[z].y, v[z].y, t));
      store_low();
      __syncwarp();
      if (k >= M) break;
#pragma unroll
      for (int o = 1; o < LR; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      int f = RealBits<float>::finite_pos(t) ? (RealBits<float>::expo(t) >> 1) : 0;
      f = f > 100 ? 100 : (f < -100 ? -100 : f);
      const float al = RealBits<float>::pow2(-f);
      expo += f;
#pragma unroll
      for (int z = 0; z < 32; ++z) {
        const float2 x = s[half_place((uint32_t)z << BT) ^ (uint32_t)li];
        v[z] = make_float2(al * x.x, al * x.y);
      }
      n = min(5 - j0, M - k);
      steps(std::integral_constant<int, BT>{}, k, j0, j0 + n);
      k += n;
#pragma unroll
      for (int z = 0; z < 32; ++z) s[half_place((uint32_t)z << BT) ^ (uint32_t)li] = v[z];
      __syncwarp();
      if (k >= M) break;
      load_low();
      __syncwarp();
    }

    // ---- norm, in the register kernel's order
    float hi[V], lo[V];
#pragma unroll
    for (int u = 0; u < V; ++u) {
      float p[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const uint32_t e = s_e[((li * V + u) << RB) | j];
        const float2 x = e == 0xffffu ? make_float2(0.f, 0.f) : s[e];
        p[j] = fmaf(x.x, x.x, __fmul_rn(x.y, x.y));
      }
#pragma unroll
      for (int h = R / 2; h >= 1; h >>= 1)
#pragma unroll
        for (int j = 0; j < h; ++j) p[j] += p[j + h];
      hi[u] = p[0];
      lo[u] = 0.f;
    }
#pragma unroll
    for (int o = 1; o < V; o <<= 1)
#pragma unroll
      for (int u = 0; u < V; u += 2 * o) {
        two_sum_acc(hi[u], lo[u], hi[u + o], lo[u + o]);
        if (want_phase) ph[u] = cmul(ph[u], ph[u + o]);
      }
#pragma unroll
    for (int o = 1; o < LR; o <<= 1) {
      two_sum_acc(hi[0], lo[0], __shfl_xor_sync(0xffffffffu, hi[0], o), __shfl_xor_sync(0xffffffffu, lo[0], o));
      const float2 q =
          make_float2(__shfl_xor_sync(0xffffffffu, ph[0].x, o), __shfl_xor_sync(0xffffffffu, ph[0].y, o));
      if (want_phase) ph[0] = cmul(ph[0], q);
    }
    const float n2 = hi[0] + lo[0], n2lo = lo[0] - (n2 - hi[0]);
    const bool ok = (n2 > 0.f) && (n2 < 3.0e38f);
    float y = rsqrtf(n2);
    y = y * (1.5f - 0.5f * n2 * y * y);  // one Newton step
    const float inv = ok ? y : NAN;
    const float2 sc = make_float2(ph[0].x * inv, ph[0].y * inv);

    // ---- outputs through the run's shared memory in output order
    load_low();
    __syncwarp();
#pragma unroll
    for (int z = 0; z < 32; ++z) {
      const int o = s_out[p0 ^ (uint32_t)z];
      if (o >= 0) s[o] = cmul(v[z], sc);
    }
    __syncwarp();
    if (run < a.B) {
      float2 *out = reinterpret_cast<float2 *>(a.psi_out) + run * dout;
      for (int x = li; x < dout; x += LR) out[x] = s[x];
      if (li == 0) {
        if (a.status) a.status[run] = ok ? MBQC_RUN_OK : (isnan(n2) ? MBQC_RUN_NAN : MBQC_RUN_ZERO_NORM);
        if (a.logprob) {  // as sv_fwd_reg
          int e1, e2;
          const float m1 = frexpf(n2, &e1), m2 = frexpf(s[NS].x, &e2);
          const double ln2 = 0.6931471805599453;
          a.logprob[run] = (double)(logf(m1) - logf(m2)) + (double)n2lo / (double)n2 +
                           ln2 * (double)(e1 - e2 + 2 * expo + a.lp_const);
        }
      }
    }
    __syncwarp();
  }
}

// From the batch on where the register kernel has 16 lanes a run (w = 9: 1,700 runs,
// 32 lanes, take it 35 us against 52 here; 2,500 runs, 16 lanes, 68 against 54) or more
// than eight warps an SM (w = 10: 1,200 runs 52 against 60, 1,700 runs 85 against 62).
// Device inputs, XY / X / Y, the default lanes; the last step lets no qubit in.
bool sv_half_ok(const DevCircuit &hc, const DevStep *steps, int64_t batch, uint32_t flags) {
  if (!(hc.w == 9 && batch >= (int64_t)16 * sm_count()) && !(hc.w == 10 && batch > (int64_t)8 * sm_count())) return false;
  if (flags & MBQC_F_HOST_INPUTS) return false;
  if (hc.n_steps < 1 || hc.n_steps > 256 || hc.n_in >= hc.w || hc.map_off < 0) return false;
  return (steps[hc.n_steps - 1].mask & kDead) != 0u;
}

int launch_sv_half(int w, int ll, const SvArgs &a, cudaStream_t s) {
  auto go = [&](auto k, size_t smem, int rpw) {
    if (smem > 48 * 1024) {
      const int rc =
          cuda_check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "sv_half smem");
      if (rc) return rc;
    }
    const int64_t groups = (a.B + rpw - 1) / rpw, need = (groups + kHalfWarps - 1) / kHalfWarps;
    k<<<(int)std::min<int64_t>(need, (int64_t)sm_count() * 4), 32 * kHalfWarps, smem, s>>>(a);
    return check_launch("sv_half");
  };
  if (w == 9 && ll == 4) return go(sv_half<8, 4>, half_smem<8>(a.M), 4);
  if (w == 10 && ll == 5) return go(sv_half<9, 5>, half_smem<9>(a.M), 2);
  return fail(MBQC_E_UNSUPPORTED, "sv_half: window %d, ll=%d", w, ll);
}

}  // namespace mbqc
