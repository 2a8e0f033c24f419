// bf16 attention with 32-bit probabilities at any length: the three branches on mma.sync, for calls that the tcgen05 kernels do
// not take by default (lengths that are no whole tiles, few compressed blocks, slices of longer buffers).
//
// Those calls used to run on the stride-generic FMA kernels, which hold P and dS in fp32 (a bf16 step of 1000 tokens took 27 ms
// there, 207 ms before they were tiled; 3.98 ms here).  Products of bf16 inputs are exact on the tensor cores; P and dS enter
// their second product as three bf16 terms whose sum is the fp32 value, so nothing is held in 16 bits and the bf16 results
// round alike: from 301 to 1920 tokens the outputs' error against 64 bits is that of the FMA kernels to 2e-7 of itself, the
// gradients' to 1e-3 either way.  (Two terms, 16 bits, take 0.1 ms less, their outputs are 8e-7 further off.  tcgen05 would need
// the further P tiles in TMEM, which the backward kernels have no columns for.)  64 x 64 tiles, four
// warps of 16 rows (forward, dQ) or 16 keys (dK/dV: S^T, so that P^T and dS^T are A operands where they lie in registers); two
// CTAs per SM overlap one's loads with the other's products.  Bound by the mma.sync pipe and its ldmatrix traffic.
//
// A key that a row does not see adds nothing to it, whatever it holds: where a result comes out infinite or NaN the tile is
// redone with sums that skip zero weights.
#include <cooperative_groups.h>

#include <algorithm>

#include "attn_tiles.cuh"
#include "common.cuh"
#include "fa_sm100.cuh"

namespace nsa {

namespace cg = cooperative_groups;

namespace {

constexpr int kT = 64;               // rows and keys of a tile
constexpr int kThreads = kTileThreads;
constexpr int kLdK = kT + 8;         // row distance of the key tile [DK][64]: 16 bytes off a bank period, as all rows here
constexpr int kLdP = kT + 4;
using MmaLists = TileLists<kT, 8192, 1024>;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(void* dst, const void* src, bool full) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(full ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the leading bf16 pair of two values, which keep what rounding left
__device__ __forceinline__ uint32_t take2(float& x, float& y) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const float2 f = __bfloat1622float2(h);
  x -= f.x;
  y -= f.y;
  return *reinterpret_cast<const uint32_t*>(&h);
}
// C fragments of two neighbouring 8-column tiles -> A fragments of the 16-wide k step they span: three terms of 8 bits, the
// whole value (fp32 has 24; the differences are exact)
__device__ __forceinline__ void split_frag(const float (&c0)[4], const float (&c1)[4], uint32_t (&t)[3][4]) {
  float x[8] = {c0[0], c0[1], c0[2], c0[3], c1[0], c1[1], c1[2], c1[3]};
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) t[j][i] = take2(x[2 * i], x[2 * i + 1]);
}

// lane offsets (elements) of the four ldmatrix address patterns; see the fragment layouts of mma.m16n8k16
__device__ __forceinline__ int pat_a(int lane, int ld) { return (lane & 15) * ld + (lane >> 4) * 8; }                              // A from [m][k]; B (trans) from [k][n]
__device__ __forceinline__ int pat_at(int lane, int ld) { return ((lane & 7) + (lane >> 4) * 8) * ld + ((lane >> 3) & 1) * 8; }   // A (trans) from [k][m]; B from [n][k]

template <int DK, int DV>
struct MmaSmem {
  static constexpr int kLdQ = DK + 8, kLdV = DV + 8;
  static constexpr int kQ = kT * kLdQ * 2, kdO = kT * kLdV * 2, kK = DK * kLdK * 2, kV = kT * kLdV * 2, kP = kT * kLdP * 4;
  static constexpr int oQ = 0, odO = oQ + kQ, oK = odO + kdO, oV = oK + kK, oP = oV + kV, oSmall = oP + kP;
  static constexpr int kSmall = 5 * kT * 4;                                      // t, lse, delta, ends, member
  static constexpr int kBase = oSmall + kSmall;
  static constexpr int kSlcBytes = kBase + MmaLists::kIdWindow / 8 + MmaLists::kIdxInts * 4;
  __nv_bfloat16 *q, *dO, *k, *v;
  float *p, *lse, *del;
  int* t;
  MmaLists l;
  __device__ explicit MmaSmem(uint8_t* s) {
    q = (__nv_bfloat16*)(s + oQ); dO = (__nv_bfloat16*)(s + odO); k = (__nv_bfloat16*)(s + oK); v = (__nv_bfloat16*)(s + oV);
    p = (float*)(s + oP);
    t = (int*)(s + oSmall);
    lse = (float*)(t + kT); del = lse + kT;
    l.ends = (int*)(del + kT); l.member = l.ends + kT;
    l.bits = (unsigned*)(s + kBase);
    l.idx = (int*)(l.bits + MmaLists::kIdWindow / 32);
  }
};

// keys [key0, key0 + 64) of one (batch, group): K [DK][64], V [64][DV]; what lies behind key `n` of the tile reads as zero
template <int DK, int DV>
__device__ __forceinline__ void load_kv(const MmaSmem<DK, DV>& s, const AttnArgs& a, int b, int g, int key0, int n) {
  const __nv_bfloat16* k = (const __nv_bfloat16*)a.k + b * a.sk[0] + g * a.sk[1] + key0;
  const __nv_bfloat16* v = (const __nv_bfloat16*)a.v + b * a.sv[0] + g * a.sv[1] + (int64_t)key0 * DV;
  for (int i = threadIdx.x; i < DK * 8; i += kThreads) {
    const int r = i >> 3, c = (i & 7) * 8;
    cp16(s.k + r * kLdK + c, c < n ? k + (int64_t)r * a.sk[3] + c : k, c < n);     // (rows are whole 8-key pieces long)
  }
  for (int i = threadIdx.x; i < kT * (DV / 8); i += kThreads) {
    const int r = i / (DV / 8), c = i % (DV / 8) * 8;
    cp16(s.v + r * s.kLdV + c, r < n ? v + (int64_t)r * DV + c : v, r < n);
  }
  cp_wait_all();
  __syncthreads();
  if (n & 7) {       // the piece that holds the last key: the row's padding is anything
    const int w = 8 - (n & 7);
    for (int i = threadIdx.x; i < DK * w; i += kThreads) s.k[i / w * kLdK + n + i % w] = __float2bfloat16_rn(0.f);
    __syncthreads();
  }
}
__device__ __forceinline__ void load_rows(__nv_bfloat16* dst, const __nv_bfloat16* base, int64_t row, int D, int r) {   // one row by one warp
  for (int c = (threadIdx.x & 31) * 8; c < D; c += 256) cp16(dst + r * (D + 8) + c, row < 0 ? base : base + row * D + c, row >= 0);
}
// Row statistics of the backward: log-sum-exp (+inf: no such row, or it saw nothing) and dO.O, by one warp.  dO.O is of the bf16 dO
// that dP is formed from: taken from a caller who has it of dO before that rounding, dS = P (dP - dO.O) no longer adds up to zero
// over a row, and the compression weights' gradients, sums in which that cancels, were off by up to twice as much.  A pass of its
// own forms it where the scratch has room (a key tile's rows are read by up to 16 tiles: 5.46 ms a step of 1000 tokens without).
template <int DK, int DV>
__device__ __forceinline__ void load_stats(const MmaSmem<DK, DV>& s, const AttnArgs& a, int r, int t, int64_t row) {
  const int lane = threadIdx.x & 31;
  float d = 0.f;
  if (t >= 0 && !a.row_sums) {
    const __nv_bfloat16 *o = (const __nv_bfloat16*)a.o_in + row * DV, *g = (const __nv_bfloat16*)a.dout + row * DV;
    for (int c = lane * 2; c < DV; c += 64) {
      const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(o + c)), y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(g + c));
      d = fmaf(x.x, y.x, fmaf(x.y, y.y, d));
    }
    d = warp_sum(d);
  }
  if (lane == 0) {
    float lse = t >= 0 ? a.Mc[row] + a.Lc[row] : CUDART_INF_F;
    s.lse[r] = isfinite(lse) ? lse : CUDART_INF_F;
    s.del[r] = t >= 0 && a.row_sums ? a.row_sums[row] : d;
    s.t[r] = t;
  }
}

// acc (16 rows x 8 N2 columns) += w (16 x 16 KK, C fragments of 2 KK tiles) * mat [16 KK][ld] from row k0 on; `guard`: the slow form
// that skips zero weights, w through this warp's rows of `wsm`
template <int KK, int N2>
__device__ __forceinline__ void second_product(float (&acc)[2 * N2][4], const float (&w)[2 * KK][4], const __nv_bfloat16* mat, int ld, int k0, bool trans,
                                               bool guard, float* wsm, int wrow) {
  const int lane = threadIdx.x & 31;
  if (!guard) {
#pragma unroll
    for (int kk = 0; kk < KK; ++kk) {
      uint32_t t[3][4];
      split_frag(w[2 * kk], w[2 * kk + 1], t);
#pragma unroll
      for (int nn = 0; nn < N2; ++nn) {
        uint32_t bf[4];
        if (trans) ldsm4t(bf, smem_addr(mat + (k0 + kk * 16) * ld + nn * 16 + pat_a(lane, ld)));      // mat [k][n]
        else ldsm4(bf, smem_addr(mat + nn * 16 * ld + k0 + kk * 16 + pat_at(lane, ld)));               // mat [n][k]
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          mma(acc[2 * nn], t[j], bf[0], bf[1]);
          mma(acc[2 * nn + 1], t[j], bf[2], bf[3]);
        }
      }
    }
    return;
  }
  __syncwarp();
  const int g = lane >> 2, c2 = (lane & 3) * 2;
#pragma unroll
  for (int i = 0; i < 2 * KK; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) wsm[(wrow + g + (e >> 1) * 8) * kLdP + i * 8 + c2 + (e & 1)] = w[i][e];
  __syncwarp();
  for (int k = 0; k < 16 * KK; ++k) {
    const float w0 = wsm[(wrow + g) * kLdP + k], w1 = wsm[(wrow + g + 8) * kLdP + k];
#pragma unroll
    for (int i = 0; i < 2 * N2; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float x = __bfloat162float(trans ? mat[(k0 + k) * ld + i * 8 + c2 + e] : mat[(i * 8 + c2 + e) * ld + k0 + k]);
        if (w0 != 0.f) acc[i][e] = fmaf(w0, x, acc[i][e]);
        if (w1 != 0.f) acc[i][2 + e] = fmaf(w1, x, acc[i][2 + e]);
      }
  }
}
template <int N>
__device__ __forceinline__ bool not_finite(const float (&acc)[N][4]) {
  bool bad = false;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) bad |= !isfinite(acc[i][e]);
  return bad;
}
template <int N>
__device__ __forceinline__ void zero(float (&acc)[N][4]) {
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
}

// ------------------------------------------------------------------------------------------------ forward
template <int DK, int DV, int MODE>
__global__ void __launch_bounds__(kThreads, 2) mma_fwd_kernel(const __grid_constant__ AttnArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  using SM = MmaSmem<DK, DV>;
  const SM s(smem);
  const RowTile<kT> rt(a);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c2 = (lane & 3) * 2;
  for (int r = warp; r < kT; r += 4) {
    const int t = rt.query(r, a.Tq);
    load_rows(s.q, (const __nv_bfloat16*)a.q, t < 0 ? -1 : ((int64_t)rt.b * a.H + rt.head(r)) * a.Tq + t, DK, r);
  }
  const int row[2] = {warp * 16 + g, warp * 16 + g + 8};
  const int t[2] = {rt.query(row[0], a.Tq), rt.query(row[1], a.Tq)};
  for (int pass = 0; pass < 2; ++pass) {       // (the second only where a result of the first is not finite)
    float m[2] = {-CUDART_INF_F, -CUDART_INF_F}, l[2] = {0.f, 0.f}, acc[DV / 8][4];
    zero(acc);
    for_each_key_tile<MODE, kT, MmaLists>(a, rt, s.l, [&](int key0, int n) {
      __syncthreads();
      load_kv<DK, DV>(s, a, rt.b, rt.g, key0, n);
      float x[8][4];
      zero(x);
#pragma unroll 4
      for (int k = 0; k < DK; k += 16) {
        uint32_t af[4];
        ldsm4(af, smem_addr(s.q + warp * 16 * SM::kLdQ + k + pat_a(lane, SM::kLdQ)));
#pragma unroll
        for (int nn = 0; nn < 4; ++nn) {
          uint32_t bf[4];
          ldsm4t(bf, smem_addr(s.k + k * kLdK + nn * 16 + pat_a(lane, kLdK)));
          mma(x[2 * nn], af, bf[0], bf[1]);
          mma(x[2 * nn + 1], af, bf[2], bf[3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float mx = -CUDART_INF_F;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int kk = j * 8 + c2 + e;
            float& y = x[j][2 * i + e];
            y = visible<MODE, MmaLists>(a, s.l, row[i], rt.HT, t[i], key0 + kk, kk, n) ? y * a.scale : -CUDART_INF_F;
            mx = fmaxf(mx, y);
          }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float mnew = fmaxf(m[i], mx), alpha = m[i] == mnew ? 1.f : expf(m[i] - mnew);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float& y = x[j][2 * i + e];
            y = y == -CUDART_INF_F ? 0.f : expf(y - mnew);
            sum += y;
          }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        l[i] = l[i] * alpha + sum;
        m[i] = mnew;
#pragma unroll
        for (int j = 0; j < DV / 8; ++j) { acc[j][2 * i] *= alpha; acc[j][2 * i + 1] *= alpha; }
      }
      second_product<4, DV / 16>(acc, x, s.v, SM::kLdV, 0, true, pass == 1, s.p, warp * 16);
    });
    if (__syncthreads_or(pass == 0 && not_finite(acc))) continue;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (t[i] < 0) continue;
      const int64_t ro = ((int64_t)rt.b * a.H + rt.head(row[i])) * a.Tq + t[i];
      const float inv = l[i] != 0.f ? 1.f / l[i] : 0.f;
      __nv_bfloat16* o = (__nv_bfloat16*)a.o + ro * DV + c2;
#pragma unroll
      for (int j = 0; j < DV / 8; ++j) *reinterpret_cast<__nv_bfloat162*>(o + j * 8) = __floats2bfloat162_rn(acc[j][2 * i] * inv, acc[j][2 * i + 1] * inv);
      if ((lane & 3) == 0) {
        a.L[ro] = l[i] != 0.f ? logf(l[i]) : -CUDART_INF_F;
        a.M[ro] = m[i];
      }
    }
    return;
  }
}

// ------------------------------------------------------------------------------------------------ backward dQ
template <int DK, int DV, int MODE>
__global__ void __launch_bounds__(kThreads, 2) mma_dq_kernel(const __grid_constant__ AttnArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  using SM = MmaSmem<DK, DV>;
  const SM s(smem);
  const RowTile<kT> rt(a);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c2 = (lane & 3) * 2;
  for (int r = warp; r < kT; r += 4) {
    const int t = rt.query(r, a.Tq);
    const int64_t ro = t < 0 ? -1 : ((int64_t)rt.b * a.H + rt.head(r)) * a.Tq + t;
    load_rows(s.q, (const __nv_bfloat16*)a.q, ro, DK, r);
    load_rows(s.dO, (const __nv_bfloat16*)a.dout, ro, DV, r);
    load_stats(s, a, r, t, ro);
  }
  __syncthreads();
  const int row[2] = {warp * 16 + g, warp * 16 + g + 8};
  const int t[2] = {s.t[row[0]], s.t[row[1]]};
  const float lse[2] = {s.lse[row[0]], s.lse[row[1]]}, del[2] = {s.del[row[0]], s.del[row[1]]};
  for (int pass = 0; pass < 2; ++pass) {
    float acc[DK / 8][4];
    zero(acc);
    for_each_key_tile<MODE, kT, MmaLists>(a, rt, s.l, [&](int key0, int n) {
      __syncthreads();
      load_kv<DK, DV>(s, a, rt.b, rt.g, key0, n);
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {       // 32 keys at a time: registers
        float x[4][4], dp[4][4];
        zero(x);
        zero(dp);
#pragma unroll 4
        for (int k = 0; k < DK; k += 16) {
          uint32_t af[4];
          ldsm4(af, smem_addr(s.q + warp * 16 * SM::kLdQ + k + pat_a(lane, SM::kLdQ)));
#pragma unroll
          for (int nn = 0; nn < 2; ++nn) {
            uint32_t bf[4];
            ldsm4t(bf, smem_addr(s.k + k * kLdK + half * 32 + nn * 16 + pat_a(lane, kLdK)));
            mma(x[2 * nn], af, bf[0], bf[1]);
            mma(x[2 * nn + 1], af, bf[2], bf[3]);
          }
        }
#pragma unroll 4
        for (int k = 0; k < DV; k += 16) {
          uint32_t af[4];
          ldsm4(af, smem_addr(s.dO + warp * 16 * SM::kLdV + k + pat_a(lane, SM::kLdV)));
#pragma unroll
          for (int nn = 0; nn < 2; ++nn) {
            uint32_t bf[4];
            ldsm4(bf, smem_addr(s.v + (half * 32 + nn * 16) * SM::kLdV + k + pat_at(lane, SM::kLdV)));
            mma(dp[2 * nn], af, bf[0], bf[1]);
            mma(dp[2 * nn + 1], af, bf[2], bf[3]);
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = e >> 1, kk = half * 32 + j * 8 + c2 + (e & 1);
            const bool in = lse[i] != CUDART_INF_F && visible<MODE, MmaLists>(a, s.l, row[i], rt.HT, t[i], key0 + kk, kk, n);
            x[j][e] = in ? expf(x[j][e] * a.scale - lse[i]) * (dp[j][e] - del[i]) : 0.f;
          }
        second_product<2, DK / 16>(acc, x, s.k, kLdK, half * 32, false, pass == 1, s.p, warp * 16);
      }
    });
    if (__syncthreads_or(pass == 0 && not_finite(acc))) continue;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (t[i] < 0) continue;
      __nv_bfloat16* dq = (__nv_bfloat16*)a.dq + (((int64_t)rt.b * a.H + rt.head(row[i])) * a.Tq + t[i]) * DK + c2;
#pragma unroll
      for (int j = 0; j < DK / 8; ++j) *reinterpret_cast<__nv_bfloat162*>(dq + j * 8) = __floats2bfloat162_rn(acc[j][2 * i] * a.scale, acc[j][2 * i + 1] * a.scale);
    }
    return;
  }
}

// ------------------------------------------------------------------------------------------------ backward dK/dV
// A CTA of the cluster takes every csize-th 64-row tile of the (query, head) rows that see its 64 keys; the CTAs' sums are added
// in rank order through distributed shared memory.
template <int DK, int DV, int MODE>
__global__ void __launch_bounds__(kThreads, 2) mma_dkv_kernel(const __grid_constant__ AttnArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  using SM = MmaSmem<DK, DV>;
  const SM s(smem);
  cg::cluster_group cluster = cg::this_cluster();
  const int csize = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), tile = blockIdx.x / csize;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c2 = (lane & 3) * 2;
  const int b = blockIdx.y / a.G, gr = blockIdx.y % a.G, hpg = a.H / a.G;
  const KeyTile kt = key_tile<MODE, kT>(a, tile, b, gr, s.l.ends, s.l.member);
  const int64_t rows = (int64_t)kt.nq * hpg;
  if (kt.nq > 0) load_kv<DK, DV>(s, a, b, gr, kt.key0, kt.n);
  constexpr int kPieces = DK / 8 + DV / 8;
  float4* mine = reinterpret_cast<float4*>(smem);
  static_assert(kPieces * kThreads * 16 <= SM::oP, "the sums of a CTA lie over its tiles");
  const int key[2] = {warp * 16 + g, warp * 16 + g + 8};
  bool bad = false;
  for (int pass = 0; pass < 2; ++pass) {
    float ak[DK / 8][4], av[DV / 8][4];
    zero(ak);
    zero(av);
    for (int64_t r0 = (int64_t)rank * kT; r0 < rows; r0 += (int64_t)csize * kT) {
      __syncthreads();
      for (int r = warp; r < kT; r += 4) {
        const int64_t e = r0 + r;
        int t = -1;
        int64_t ro = -1;
        if (e < rows) {
          const int q = (int)(e / hpg);
          t = MODE == kSlc ? kt.list[q] & 0xFFFFFF : kt.qbeg + q;
          ro = ((int64_t)b * a.H + gr * hpg + (int)(e % hpg)) * a.Tq + t;
        }
        load_rows(s.q, (const __nv_bfloat16*)a.q, ro, DK, r);
        load_rows(s.dO, (const __nv_bfloat16*)a.dout, ro, DV, r);
        load_stats(s, a, r, t, ro);
      }
      cp_wait_all();
      __syncthreads();
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        float x[4][4], dp[4][4];
        zero(x);
        zero(dp);
#pragma unroll 4
        for (int k = 0; k < DK; k += 16) {
          uint32_t af[4];
          ldsm4t(af, smem_addr(s.k + k * kLdK + warp * 16 + pat_at(lane, kLdK)));
#pragma unroll
          for (int nn = 0; nn < 2; ++nn) {
            uint32_t bf[4];
            ldsm4(bf, smem_addr(s.q + (half * 32 + nn * 16) * SM::kLdQ + k + pat_at(lane, SM::kLdQ)));
            mma(x[2 * nn], af, bf[0], bf[1]);
            mma(x[2 * nn + 1], af, bf[2], bf[3]);
          }
        }
#pragma unroll 4
        for (int k = 0; k < DV; k += 16) {
          uint32_t af[4];
          ldsm4(af, smem_addr(s.v + warp * 16 * SM::kLdV + k + pat_a(lane, SM::kLdV)));
#pragma unroll
          for (int nn = 0; nn < 2; ++nn) {
            uint32_t bf[4];
            ldsm4(bf, smem_addr(s.dO + (half * 32 + nn * 16) * SM::kLdV + k + pat_at(lane, SM::kLdV)));
            mma(dp[2 * nn], af, bf[0], bf[1]);
            mma(dp[2 * nn + 1], af, bf[2], bf[3]);
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int r = half * 32 + j * 8 + c2 + (e & 1), kk = key[e >> 1], t = s.t[r], ky = kt.key0 + kk;
            const float lse = s.lse[r];
            bool in = lse != CUDART_INF_F && kk < kt.n;
            if (MODE == kWin) in = in && ky <= t && ky > t - a.window;
            else if (MODE == kCmp) in = in && s.l.ends[kk] <= t;
            else in = in && !(a.causal && ky > t);
            const float p = in ? expf(x[j][e] * a.scale - lse) : 0.f;
            x[j][e] = p;
            dp[j][e] = in ? p * (dp[j][e] - s.del[r]) : 0.f;
          }
        second_product<2, DV / 16>(av, x, s.dO, SM::kLdV, half * 32, true, pass == 1, s.p, warp * 16);
        second_product<2, DK / 16>(ak, dp, s.q, SM::kLdQ, half * 32, true, pass == 1, s.p, warp * 16);
      }
    }
    bad = __syncthreads_or(pass == 0 && (not_finite(ak) || not_finite(av)));
    if (bad) continue;      // (K and V are still in place: the sums go over them only now)
#pragma unroll
    for (int j = 0; j < DK / 8; ++j) mine[j * kThreads + threadIdx.x] = make_float4(ak[j][0] * a.scale, ak[j][1] * a.scale, ak[j][2] * a.scale, ak[j][3] * a.scale);
#pragma unroll
    for (int j = 0; j < DV / 8; ++j) mine[(DK / 8 + j) * kThreads + threadIdx.x] = make_float4(av[j][0], av[j][1], av[j][2], av[j][3]);
    break;
  }
  cluster.sync();
  for (int pc = rank; pc < kPieces; pc += csize) {
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c = 0; c < csize; ++c) {
      const float4 x = cluster.map_shared_rank(mine, c)[pc * kThreads + threadIdx.x];
      sum.x += x.x; sum.y += x.y; sum.z += x.z; sum.w += x.w;
    }
    const bool isk = pc < DK / 8;
    const int W = isk ? DK : DV, c0 = (isk ? pc : pc - DK / 8) * 8 + c2;
    __nv_bfloat16* out = (__nv_bfloat16*)(isk ? a.dk_out : a.dv_out) + (((int64_t)b * a.G + gr) * a.Tk + kt.key0) * W + c0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (key[i] >= kt.n) continue;
      __nv_bfloat162* d = reinterpret_cast<__nv_bfloat162*>(out + (int64_t)key[i] * W);
      const float2 cur = __bfloat1622float2(*d);
      *d = i == 0 ? __floats2bfloat162_rn(cur.x + sum.x, cur.y + sum.y) : __floats2bfloat162_rn(cur.x + sum.z, cur.y + sum.w);
    }
  }
  cluster.sync();      // nobody leaves while its sums are being read
}

// ------------------------------------------------------------------------------------------------ host launchers
template <int DK, int DV, int MODE>
int launch_t(const AttnArgs& a, bool backward, cudaStream_t st) {
  using SM = MmaSmem<DK, DV>;
  const int sm = MODE == kSlc ? SM::kSlcBytes : SM::kBase;
  const dim3 gq = RowTile<kT>::grid(a);
  if (!backward) {
    KernelTimer kt("attn_fwd_mma", st);
    cudaFuncSetAttribute(mma_fwd_kernel<DK, DV, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    mma_fwd_kernel<DK, DV, MODE><<<gq, kThreads, sm, st>>>(a);
    return check_launch("attn_fwd_mma");
  }
  KernelTimer kt("attn_bwd_mma", st);
  cudaFuncSetAttribute(mma_dq_kernel<DK, DV, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  mma_dq_kernel<DK, DV, MODE><<<gq, kThreads, sm, st>>>(a);
  if (int rc = check_launch("attn_bwd_dq_mma")) return rc;
  const int64_t tiles = key_tiles<MODE, kT>(a);
  int csize = 8;       // CTAs that share a key tile's rows, until the 296 resident ones have about two each
  while (csize > 1 && tiles * a.B * a.G * csize > 640) csize /= 2;
  cudaFuncSetAttribute(mma_dkv_kernel<DK, DV, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::kBase);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * csize), a.B * a.G);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = SM::kBase;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = csize;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaError_t e = cudaLaunchKernelEx(&cfg, mma_dkv_kernel<DK, DV, MODE>, a); e != cudaSuccess)
    return fail(NSA_ERR_LAUNCH, "attn_bwd_dkv_mma: %s", cudaGetErrorString(e));
  return check_launch("attn_bwd_dkv_mma");
}
template <int DK, int DV>
int launch_m(const AttnArgs& a, int mode, bool backward, cudaStream_t st) {
  return mode == kWin ? launch_t<DK, DV, kWin>(a, backward, st) : mode == kCmp ? launch_t<DK, DV, kCmp>(a, backward, st) : launch_t<DK, DV, kSlc>(a, backward, st);
}

}  // namespace

bool attn_mma_supported(int dk, int dv, int mode, int lprime) {
  return ((dk == 192 && dv == 128) || (dk == 128 && dv == 128) || (dk == 64 && dv == 64)) && (mode != kSlc || lprime % kT == 0);
}
// a: bf16 tensors in the canonical layouts (rows of keys a multiple of 8 apart, everything on 16-byte boundaries)
int launch_attn_mma(const AttnArgs& a, int mode, bool backward, cudaStream_t st) {
  if (a.B * a.H == 0 || a.Tq == 0 || a.Tk == 0) return NSA_OK;
  if (a.dk == 192) return launch_m<192, 128>(a, mode, backward, st);
  if (a.dk == 128) return launch_m<128, 128>(a, mode, backward, st);
  return launch_m<64, 64>(a, mode, backward, st);
}

}  // namespace nsa
