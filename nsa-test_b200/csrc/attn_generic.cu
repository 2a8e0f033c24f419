// Stride-generic attention kernels (fp32 math on CUDA cores) for the three NSA branches.
//
// These kernels honour arbitrary element strides and any head dim <= 256, in fp32 or bf16 storage.  They serve the raw
// kernel-call contract (callers may pass any strides), fp32 I/O, and shapes the tensor-core kernels do not cover.
//
// What bounds them is the FMA pipe and the shared-memory reads that feed it, so everything runs on 32 x 32 tiles in shared
// memory with 2 x 4 products per thread: 6 shared 16-byte reads per 32 FMAs.  (One warp per query or key row, with every
// operand read from global memory for every product, took 10.1 ms of a 10.2 ms fp32 training step at B=2, H=8, T=512.)
//   * forward, dQ: a tile's 32 rows are the heads of a group for 32 / heads consecutive queries, so a key tile serves them
//     all; the selection branch walks the union of its queries' blocks and masks per query.
//   * dK/dV: a CTA owns 32 keys and walks the (query, head) rows that see them; up to eight CTAs of a cluster share the walk
//     and their sums are added in rank order through distributed shared memory.  Every reduction has one writer and a fixed
//     order: results are deterministic.
//
// Semantics follow the reference kernels: _nsa_sliding_window_* (nsa/kernels.py:1151-1530),
// _nsa_compression_* (nsa/kernels.py:1533-1917), _nsa_sparse_selection_* (nsa/kernels.py:594-1148):
// logits = (q*scale).k, masked rows give O=0, L=M=-inf, L = log(sum exp(s-M)).  A key that a row does not see adds nothing
// to it, whatever it holds: tiles with infinities or NaN take sums that skip zero weights.
#include <cooperative_groups.h>

#include <algorithm>

#include "attn_tiles.cuh"
#include "common.cuh"

namespace nsa {

namespace cg = cooperative_groups;

constexpr int kGenThreads = kTileThreads;
constexpr int kTile = 32;            // rows and keys of a tile
constexpr int kPs = kTile + 4;       // row distance of the 32 x 32 weight tiles
using GenLists = TileLists<kTile, 32768, 4096>;

// Shared memory: row tiles (Q; backward: dO and O) and two key tiles (K, V) of [32][32 * DC + 4] floats (the odd multiple of four
// puts the rows 4 banks apart), two weight tiles, then the small arrays.
template <int DC>
struct GenSmem : GenLists {
  static constexpr int kLd = 32 * DC + 4, kMat = kTile * kLd;
  float *a, *b, *k, *v, *p, *ds, *lse, *o;
  int* t;
  __device__ explicit GenSmem(float* s) {
    a = s; b = a + kMat; k = b + kMat; v = k + kMat; p = v + kMat; ds = p + kTile * kPs; lse = ds + kTile * kPs;
    t = (int*)(lse + kTile); ends = t + kTile; member = ends + kTile;
    bits = (unsigned*)(member + kTile);
    idx = (int*)(bits + kIdWindow / 32);
    o = lse + 4 * kTile;
  }
  // (the selection's dQ has the bitmap and the index rows in front of O)
  __device__ void o_behind_index() { o = (float*)(idx + kIdxInts); }
  static size_t bytes(bool selection, bool with_o) {
    return (size_t)(4 * kMat + 2 * kTile * kPs + 4 * kTile + (with_o ? kMat : 0)) * 4 + (selection ? kIdWindow / 8 + kIdxInts * 4 : 0);
  }
};

// `n` keys from key0 on -> dst[key][channel], zeros elsewhere; consecutive threads follow the smaller stride.  Returns whether
// this thread met a value that is not finite.
template <typename T, int DC>
__device__ __forceinline__ bool load_keys(float* dst, const T* src, int64_t sn, int64_t sd, int key0, int n, int D) {
  constexpr int kLd = GenSmem<DC>::kLd, kCols = 32 * DC;
  bool odd = false;
  if (sn < sd) {
    const int r = threadIdx.x & 31;
#pragma unroll 8
    for (int c = threadIdx.x >> 5; c < kCols; c += kGenThreads / 32) {
      const float x = r < n && c < D ? Elem<T>::ld(src + (int64_t)(key0 + r) * sn + c * sd) : 0.f;
      odd |= !isfinite(x);
      dst[r * kLd + c] = x;
    }
  } else {
#pragma unroll 8
    for (int i = threadIdx.x; i < kTile * kCols; i += kGenThreads) {
      const int r = i / kCols, c = i % kCols;
      const float x = r < n && c < D ? Elem<T>::ld(src + (int64_t)(key0 + r) * sn + c * sd) : 0.f;
      odd |= !isfinite(x);
      dst[r * kLd + c] = x;
    }
  }
  return odd;
}
// one row of D channels by one warp, scaled; row == nullptr gives zeros
template <typename T, int DC>
__device__ __forceinline__ bool load_row(float* dst, const T* row, int64_t sd, int D, float scale) {
  bool odd = false;
#pragma unroll
  for (int j = 0; j < DC; ++j) {
    const int c = (threadIdx.x & 31) + 32 * j;
    const float x = row && c < D ? Elem<T>::ld(row + c * sd) * scale : 0.f;
    odd |= !isfinite(x);
    dst[c] = x;
  }
  return odd;
}
// acc[i][j] = a[ry + 16 i] . b[kx + 8 j] over D channels
template <int DC>
__device__ __forceinline__ void products(float (&acc)[2][4], const float* a, const float* b, int ry, int kx, int D) {
  constexpr int kLd = GenSmem<DC>::kLd;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 4
  for (int d = 0; d < D; d += 4) {
    float4 x[2], y[4];
#pragma unroll
    for (int i = 0; i < 2; ++i) x[i] = *reinterpret_cast<const float4*>(a + (ry + 16 * i) * kLd + d);
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = *reinterpret_cast<const float4*>(b + (kx + 8 * j) * kLd + d);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        acc[i][j] = fmaf(x[i].w, y[j].w, fmaf(x[i].z, y[j].z, fmaf(x[i].y, y[j].y, fmaf(x[i].x, y[j].x, acc[i][j]))));
  }
}
// The same with acc[i][j] of b minus a[ry + 16 i] . o[ry + 16 i]: both sums run over the channels in one order, so that a row whose
// output is the one value it sees gets exactly zero.
template <int DC>
__device__ __forceinline__ void products_minus_delta(float (&acc)[2][4], const float* a, const float* b, const float* o, int ry, int kx, int D) {
  constexpr int kLd = GenSmem<DC>::kLd;
  float del[2] = {0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 4
  for (int d = 0; d < D; d += 4) {
    float4 x[2], y[4], z[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      x[i] = *reinterpret_cast<const float4*>(a + (ry + 16 * i) * kLd + d);
      z[i] = *reinterpret_cast<const float4*>(o + (ry + 16 * i) * kLd + d);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = *reinterpret_cast<const float4*>(b + (kx + 8 * j) * kLd + d);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        acc[i][j] = fmaf(x[i].w, y[j].w, fmaf(x[i].z, y[j].z, fmaf(x[i].y, y[j].y, fmaf(x[i].x, y[j].x, acc[i][j]))));
      del[i] = fmaf(x[i].w, z[i].w, fmaf(x[i].z, z[i].z, fmaf(x[i].y, z[i].y, fmaf(x[i].x, z[i].x, del[i]))));
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] -= del[i];
}
// acc[i][j] += sum over m of w[r + 16 i][m] * mat[m][4 kx + 32 j ..]; SKIP leaves out zero weights
template <int DC, bool SKIP>
__device__ __forceinline__ void accumulate_t(float4 (&acc)[2][DC], const float* w, const float* mat, int r, int kx) {
  constexpr int kLd = GenSmem<DC>::kLd;
#pragma unroll 2
  for (int m = 0; m < kTile; m += 4) {
    const float4 w0 = *reinterpret_cast<const float4*>(w + r * kPs + m), w1 = *reinterpret_cast<const float4*>(w + (r + 16) * kPs + m);
    const float wa[2][4] = {{w0.x, w0.y, w0.z, w0.w}, {w1.x, w1.y, w1.z, w1.w}};
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int j = 0; j < DC; ++j) {
        const float4 x = *reinterpret_cast<const float4*>(mat + (m + e) * kLd + 4 * kx + 32 * j);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (SKIP && wa[i][e] == 0.f) continue;
          acc[i][j].x = fmaf(wa[i][e], x.x, acc[i][j].x); acc[i][j].y = fmaf(wa[i][e], x.y, acc[i][j].y);
          acc[i][j].z = fmaf(wa[i][e], x.z, acc[i][j].z); acc[i][j].w = fmaf(wa[i][e], x.w, acc[i][j].w);
        }
      }
  }
}
template <int DC>
__device__ __forceinline__ void accumulate(float4 (&acc)[2][DC], const float* w, const float* mat, int r, int kx, bool odd) {
  if (odd) accumulate_t<DC, true>(acc, w, mat, r, kx);
  else accumulate_t<DC, false>(acc, w, mat, r, kx);
}
template <int DC>
__device__ __forceinline__ void clear(float4 (&acc)[2][DC]) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < DC; ++j) acc[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
}

template <typename T>
__device__ __forceinline__ const T* at(const void* p, const int64_t* s, int b, int h, int t) {
  return (const T*)p + b * s[0] + h * s[1] + (int64_t)t * s[2];
}

// ------------------------------------------------------------------------------------------------ forward
template <typename T, int MODE, int DC>
__global__ void __launch_bounds__(kGenThreads) attn_fwd_generic(const __grid_constant__ AttnArgs a) {
  extern __shared__ __align__(16) float smem[];
  const GenSmem<DC> s(smem);
  const RowTile<kTile> rt(a);
  const int warp = threadIdx.x >> 5, ry = threadIdx.x >> 3, kx = threadIdx.x & 7;
  for (int r = warp; r < kTile; r += kGenThreads / 32) {
    const int t = rt.query(r, a.Tq);
    load_row<T, DC>(s.a + r * s.kLd, t < 0 ? nullptr : at<T>(a.q, a.sq, rt.b, rt.head(r), t), a.sq[3], a.dk, a.scale);
  }
  const T* kp = (const T*)a.k + rt.b * a.sk[0] + rt.g * a.sk[1];
  const T* vp = (const T*)a.v + rt.b * a.sv[0] + rt.g * a.sv[1];
  int t[2];
  float m[2], l[2];
  float4 acc[2][DC];
  clear(acc);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    t[i] = rt.query(ry + 16 * i, a.Tq);
    m[i] = -CUDART_INF_F;
    l[i] = 0.f;
  }
  for_each_key_tile<MODE, 1, GenLists>(a, rt, s, [&](int key0, int n) {
    __syncthreads();
    load_keys<T, DC>(s.k, kp, a.sk[2], a.sk[3], key0, n, a.dk);
    const bool odd = __syncthreads_or(load_keys<T, DC>(s.v, vp, a.sv[2], a.sv[3], key0, n, a.dv));
    float x[2][4];
    products<DC>(x, s.a, s.k, ry, kx, a.dk);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float mx = -CUDART_INF_F;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kk = kx + 8 * j;
        if (!visible<MODE, GenLists>(a, s, ry + 16 * i, rt.HT, t[i], key0 + kk, kk, n)) x[i][j] = -CUDART_INF_F;
        mx = fmaxf(mx, x[i][j]);
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float mnew = fmaxf(m[i], mx);
      const float alpha = m[i] == mnew ? 1.f : expf(m[i] - mnew);     // m = -inf -> 0
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = x[i][j] == -CUDART_INF_F ? 0.f : expf(x[i][j] - mnew);
        s.p[(ry + 16 * i) * kPs + kx + 8 * j] = p;
        sum += p;
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l[i] = l[i] * alpha + sum;
      m[i] = mnew;
#pragma unroll
      for (int j = 0; j < DC; ++j) { acc[i][j].x *= alpha; acc[i][j].y *= alpha; acc[i][j].z *= alpha; acc[i][j].w *= alpha; }
    }
    __syncwarp();        // a warp reads back the rows it wrote
    accumulate(acc, s.p, s.v, ry, kx, odd);
  });
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (t[i] < 0) continue;
    const int h = rt.head(ry + 16 * i);
    T* op = const_cast<T*>(at<T>(a.o, a.so, rt.b, h, t[i]));
    const float inv = l[i] != 0.f ? 1.f / l[i] : 0.f;
#pragma unroll
    for (int j = 0; j < DC; ++j) {
      const float o[4] = {acc[i][j].x, acc[i][j].y, acc[i][j].z, acc[i][j].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = 4 * kx + 32 * j + e;
        if (c < a.dv) Elem<T>::st(op + c * a.so[3], o[e] * inv);
      }
    }
    if (kx == 0) {
      if (a.L) a.L[rt.b * a.sL[0] + h * a.sL[1] + (int64_t)t[i] * a.sL[2]] = l[i] != 0.f ? logf(l[i]) : -CUDART_INF_F;
      if (a.M) a.M[rt.b * a.sM[0] + h * a.sM[1] + (int64_t)t[i] * a.sM[2]] = m[i];
    }
  }
}

// Q (scaled), dO, O and log-sum-exp of a row by one warp; a row that does not exist or saw nothing gets lse = +inf.
template <typename T, int DC>
__device__ __forceinline__ bool load_bwd_row(const AttnArgs& a, const GenSmem<DC>& s, int r, int b, int h, int t) {
  const bool ok = t >= 0;
  bool odd = load_row<T, DC>(s.a + r * s.kLd, ok ? at<T>(a.q, a.sq, b, h, t) : nullptr, a.sq[3], a.dk, a.scale);
  odd |= load_row<T, DC>(s.b + r * s.kLd, ok ? at<T>(a.dout, a.so, b, h, t) : nullptr, a.so[3], a.dv, 1.f);
  load_row<T, DC>(s.o + r * s.kLd, ok ? at<T>(a.o_in, a.so, b, h, t) : nullptr, a.so[3], a.dv, 1.f);
  if ((threadIdx.x & 31) == 0) {
    float lse = CUDART_INF_F;
    if (ok) {
      lse = a.Mc[b * a.sM[0] + h * a.sM[1] + (int64_t)t * a.sM[2]] + a.Lc[b * a.sL[0] + h * a.sL[1] + (int64_t)t * a.sL[2]];
      if (!isfinite(lse)) lse = CUDART_INF_F;
    }
    s.lse[r] = lse;
    s.t[r] = t;
  }
  return odd;
}

// ------------------------------------------------------------------------------------------------ backward dQ
template <typename T, int MODE, int DC>
__global__ void __launch_bounds__(kGenThreads) attn_bwd_dq_generic(const __grid_constant__ AttnArgs a) {
  extern __shared__ __align__(16) float smem[];
  GenSmem<DC> s(smem);
  if (MODE == kSlc) s.o_behind_index();
  const RowTile<kTile> rt(a);
  const int warp = threadIdx.x >> 5, ry = threadIdx.x >> 3, kx = threadIdx.x & 7;
  for (int r = warp; r < kTile; r += kGenThreads / 32) load_bwd_row<T, DC>(a, s, r, rt.b, rt.head(r), rt.query(r, a.Tq));
  __syncthreads();
  const T* kp = (const T*)a.k + rt.b * a.sk[0] + rt.g * a.sk[1];
  const T* vp = (const T*)a.v + rt.b * a.sv[0] + rt.g * a.sv[1];
  float4 acc[2][DC];
  clear(acc);
  for_each_key_tile<MODE, 1, GenLists>(a, rt, s, [&](int key0, int n) {
    __syncthreads();
    load_keys<T, DC>(s.v, vp, a.sv[2], a.sv[3], key0, n, a.dv);
    const bool odd = __syncthreads_or(load_keys<T, DC>(s.k, kp, a.sk[2], a.sk[3], key0, n, a.dk));
    float x[2][4], dp[2][4];
    products<DC>(x, s.a, s.k, ry, kx, a.dk);
    products_minus_delta<DC>(dp, s.b, s.v, s.o, ry, kx, a.dv);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = ry + 16 * i;
      const float lse = s.lse[r];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kk = kx + 8 * j;
        const bool in = lse != CUDART_INF_F && visible<MODE, GenLists>(a, s, r, rt.HT, s.t[r], key0 + kk, kk, n);
        s.ds[r * kPs + kk] = in ? expf(x[i][j] - lse) * dp[i][j] : 0.f;
      }
    }
    __syncwarp();
    accumulate(acc, s.ds, s.k, ry, kx, odd);
  });
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int t = s.t[ry + 16 * i];
    if (t < 0) continue;
    T* dqp = const_cast<T*>(at<T>(a.dq, a.sdq, rt.b, rt.head(ry + 16 * i), t));
#pragma unroll
    for (int j = 0; j < DC; ++j) {
      const float o[4] = {acc[i][j].x, acc[i][j].y, acc[i][j].z, acc[i][j].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = 4 * kx + 32 * j + e;
        if (c < a.dk) Elem<T>::st(dqp + c * a.sdq[3], o[e] * a.scale);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ backward dK/dV
// blockIdx.x = key tile * cluster size + rank; key tiles do not cross selection blocks.
template <typename T, int MODE, int DC>
__global__ void __launch_bounds__(kGenThreads) attn_bwd_dkv_generic(const __grid_constant__ AttnArgs a) {
  extern __shared__ __align__(16) float smem[];
  const GenSmem<DC> s(smem);
  cg::cluster_group cluster = cg::this_cluster();
  const int csize = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), tile = blockIdx.x / csize;
  const int warp = threadIdx.x >> 5, ry = threadIdx.x >> 3, kx = threadIdx.x & 7;
  const int b = blockIdx.y / a.G, g = blockIdx.y % a.G, hpg = a.H / a.G;
  const KeyTile kt = key_tile<MODE, kTile>(a, tile, b, g, s.ends, s.member);
  const int key0 = kt.key0, n = kt.n;
  load_keys<T, DC>(s.k, (const T*)a.k + b * a.sk[0] + g * a.sk[1], a.sk[2], a.sk[3], key0, n, a.dk);
  load_keys<T, DC>(s.v, (const T*)a.v + b * a.sv[0] + g * a.sv[1], a.sv[2], a.sv[3], key0, n, a.dv);
  float4 acck[2][DC], accv[2][DC];
  clear(acck);
  clear(accv);
  const int64_t rows = (int64_t)kt.nq * hpg;
  for (int64_t r0 = (int64_t)rank * kTile; r0 < rows; r0 += (int64_t)csize * kTile) {
    __syncthreads();
    bool odd = false;
    for (int r = warp; r < kTile; r += kGenThreads / 32) {
      const int64_t e = r0 + r;
      int t = -1, h = 0;
      if (e < rows) {
        const int q = (int)(e / hpg);
        h = g * hpg + (int)(e % hpg);
        t = MODE == kSlc ? kt.list[q] & 0xFFFFFF : kt.qbeg + q;
      }
      odd |= load_bwd_row<T, DC>(a, s, r, b, h, t);
    }
    odd = __syncthreads_or(odd);
    float x[2][4], dp[2][4];
    products<DC>(x, s.a, s.k, ry, kx, a.dk);
    products_minus_delta<DC>(dp, s.b, s.v, s.o, ry, kx, a.dv);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = ry + 16 * i, t = s.t[r];
      const float lse = s.lse[r];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kk = kx + 8 * j, key = key0 + kk;
        bool in = lse != CUDART_INF_F && kk < n;
        if (MODE == kWin) in = in && key <= t && key > t - a.window;
        else if (MODE == kCmp) in = in && s.ends[kk] <= t;
        else in = in && !(a.causal && key > t);
        const float p = in ? expf(x[i][j] - lse) : 0.f;
        s.p[kk * kPs + r] = p;
        s.ds[kk * kPs + r] = in ? p * dp[i][j] : 0.f;
      }
    }
    __syncthreads();
    accumulate(accv, s.p, s.b, ry, kx, odd);
    accumulate(acck, s.ds, s.a, ry, kx, odd);
  }
  if (csize > 1) {       // the CTAs' sums, added in rank order: rank i finishes every csize-th piece
    __syncthreads();
    float4* mine = reinterpret_cast<float4*>(smem);      // (over the row tiles: 4 x DC x 128 float4 fit into Q and dO)
    constexpr int kPieces = 4 * DC;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < DC; ++j) {
        mine[((i * DC + j) * 2) * kGenThreads + threadIdx.x] = acck[i][j];
        mine[((i * DC + j) * 2 + 1) * kGenThreads + threadIdx.x] = accv[i][j];
      }
    cluster.sync();
    for (int pc = rank; pc < kPieces; pc += csize) {
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int c = 0; c < csize; ++c) {
        const float4 x = cluster.map_shared_rank(mine, c)[pc * kGenThreads + threadIdx.x];
        sum.x += x.x; sum.y += x.y; sum.z += x.z; sum.w += x.w;
      }
      const int i = pc / 2 / DC, j = pc / 2 % DC, r = ry + 16 * i, c0 = 4 * kx + 32 * j;
      if (r < n) {
        const bool isv = pc & 1;
        T* dst = isv ? const_cast<T*>(at<T>(a.dv_out, a.sdv, b, g, key0 + r)) : const_cast<T*>(at<T>(a.dk_out, a.sdk, b, g, key0 + r));
        const int64_t sd = isv ? a.sdv[3] : a.sdk[3];
        const int D = isv ? a.dv : a.dk;
        const float o[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (c0 + e < D) Elem<T>::st(dst + (c0 + e) * sd, Elem<T>::ld(dst + (c0 + e) * sd) + o[e]);
      }
    }
    cluster.sync();      // nobody leaves while its sums are being read
    return;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = ry + 16 * i;
    if (r >= n) continue;
    T* dkp = const_cast<T*>(at<T>(a.dk_out, a.sdk, b, g, key0 + r));
    T* dvp = const_cast<T*>(at<T>(a.dv_out, a.sdv, b, g, key0 + r));
#pragma unroll
    for (int j = 0; j < DC; ++j) {
      const float ok[4] = {acck[i][j].x, acck[i][j].y, acck[i][j].z, acck[i][j].w};
      const float ov[4] = {accv[i][j].x, accv[i][j].y, accv[i][j].z, accv[i][j].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = 4 * kx + 32 * j + e;
        if (c < a.dk) Elem<T>::st(dkp + c * a.sdk[3], Elem<T>::ld(dkp + c * a.sdk[3]) + ok[e]);
        if (c < a.dv) Elem<T>::st(dvp + c * a.sdv[3], Elem<T>::ld(dvp + c * a.sdv[3]) + ov[e]);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------
// host launchers
// ------------------------------------------------------------------------------------------------
template <typename T, int MODE, int DC>
static int launch_t(const AttnArgs& a, bool backward, cudaStream_t st) {
  const size_t sm = GenSmem<DC>::bytes(MODE == kSlc, backward), sm_dkv = GenSmem<DC>::bytes(false, true);
  const dim3 gq = RowTile<kTile>::grid(a);
  if (!backward) {
    KernelTimer kt("attn_fwd_generic", st);
    cudaFuncSetAttribute(attn_fwd_generic<T, MODE, DC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    attn_fwd_generic<T, MODE, DC><<<gq, kGenThreads, sm, st>>>(a);
    return check_launch("attn_fwd_generic");
  }
  KernelTimer kt("attn_bwd_generic", st);
  cudaFuncSetAttribute(attn_bwd_dq_generic<T, MODE, DC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  attn_bwd_dq_generic<T, MODE, DC><<<gq, kGenThreads, sm, st>>>(a);
  if (int rc = check_launch("attn_bwd_dq_generic")) return rc;
  if (a.Tk == 0) return NSA_OK;
  const int64_t tiles = key_tiles<MODE, kTile>(a);
  // few key tiles: several CTAs share the walk over the rows, as long as the SMs are not full of CTAs already
  int csize = 8;
  while (csize > 1 && tiles * a.B * a.G * csize > 1024) csize /= 2;
  cudaFuncSetAttribute(attn_bwd_dkv_generic<T, MODE, DC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_dkv);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * csize), a.B * a.G);
  cfg.blockDim = dim3(kGenThreads);
  cfg.dynamicSmemBytes = sm_dkv;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = csize;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaError_t e = cudaLaunchKernelEx(&cfg, attn_bwd_dkv_generic<T, MODE, DC>, a); e != cudaSuccess)
    return fail(NSA_ERR_LAUNCH, "attn_bwd_dkv_generic: %s", cudaGetErrorString(e));
  return check_launch("attn_bwd_dkv_generic");
}
template <typename T, int MODE>
static int launch_d(const AttnArgs& a, bool backward, cudaStream_t st) {
  const int D = std::max(a.dk, a.dv);
  return D <= 64 ? launch_t<T, MODE, 2>(a, backward, st) : D <= 128 ? launch_t<T, MODE, 4>(a, backward, st) : launch_t<T, MODE, 8>(a, backward, st);
}

int launch_attn_generic(const AttnArgs& a, int mode, int dtype, bool backward, cudaStream_t st) {
  if (a.B * a.H == 0 || a.Tq == 0) return NSA_OK;
#define NSA_DISPATCH(T)                                     \
  switch (mode) {                                           \
    case kWin: return launch_d<T, kWin>(a, backward, st);   \
    case kCmp: return launch_d<T, kCmp>(a, backward, st);   \
    case kSlc: return launch_d<T, kSlc>(a, backward, st);   \
  }
  if (dtype == NSA_F32) {
    NSA_DISPATCH(float)
  } else if (dtype == NSA_BF16) {
    NSA_DISPATCH(__nv_bfloat16)
  }
#undef NSA_DISPATCH
  return fail(NSA_ERR_ARG, "unsupported dtype %d / mode %d", dtype, mode);
}

}  // namespace nsa
