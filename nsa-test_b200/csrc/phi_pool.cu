// Pooling half of the block-compression MLP phi (NSAAttention.compress_tokens,
// nsa/kernels.py:2119-2208): with A[t] = W1[:, :dk] k_t precomputed by a GEMM and the per-offset
// table C[j] = W1[:, dk:] pos_embed[j] + b1, block i is hbar[i] = mean_j relu(A[i*d+j] + C[j]);
// values are mean-pooled.  All of it is HBM-bound streaming work.  For the default blocks (l = 32 = 2 d) a thread owns one
// hidden unit and walks the tokens of a run of blocks 16 at a time, both offsets' table entries in registers, so that A is
// read once for the two blocks that hold a token; other block sizes take the per-block kernels, which read it l/d times.
#include <algorithm>

#include "common.cuh"
#include "phi.cuh"

namespace nsa {

template <typename T>
__global__ void phi_pool_fwd_kernel(const float* __restrict__ a, const float* __restrict__ c, const T* __restrict__ v,
                                    int64_t svz, int64_t svg, int64_t svn, int64_t svk, float* __restrict__ hbar,
                                    T* __restrict__ v_cmp, int G, int T_, int U, int dv, int l, int d, int nb,
                                    int nbp) {
  const int i = blockIdx.x, bg = blockIdx.y, b = bg / G, g = bg % G;
  const float* ab = a + ((int64_t)bg * T_ + (int64_t)i * d) * U;
  const float inv = 1.f / (float)l;
  for (int u = threadIdx.x; u < U; u += blockDim.x) {
    float acc = 0.f;
    for (int j = 0; j < l; ++j) acc += fmaxf(ab[(int64_t)j * U + u] + c[j * U + u], 0.f);
    hbar[((int64_t)bg * nb + i) * U + u] = acc * inv;
  }
  const T* vb = v + b * svz + g * svg + (int64_t)i * d * svn;
  for (int x = threadIdx.x; x < dv; x += blockDim.x) {
    float acc = 0.f;
    for (int j = 0; j < l; ++j) acc += Elem<T>::ld(vb + (int64_t)j * svn + x * svk);
    Elem<T>::st(v_cmp + ((int64_t)bg * nbp + i) * dv + x, acc * inv);
  }
}

// l = 32, d = 16: hbar and v_cmp of blocks [i0, i0 + cb), the sums in the same order as above.  Segment s holds tokens
// 16 s .. 16 s + 15: the first half of block s and the second half of block s - 1.
constexpr int kSeg = 16;
__host__ __device__ inline int seg_value_threads(int dv) { return dv >= 128 ? 128 : (dv + 31) / 32 * 32; }
static int seg_threads(int U, int dv) { return std::min(384, (U + 31) / 32 * 32) + seg_value_threads(dv); }
template <typename T>
__global__ void __launch_bounds__(512) phi_pool_fwd_seg_kernel(const float* __restrict__ a, const float* __restrict__ c, const T* __restrict__ v,
                                                               int64_t svz, int64_t svg, int64_t svn, int64_t svk, float* __restrict__ hbar,
                                                               T* __restrict__ v_cmp, int G, int T_, int U, int dv, int nb, int nbp, int cb) {
  const int i0 = blockIdx.x * cb, i1 = min(nb, i0 + cb), bg = blockIdx.y, b = bg / G, g = bg % G;
  const float inv = 1.f / (2 * kSeg);
  const int nv = seg_value_threads(dv), nu = blockDim.x - nv;      // the last threads pool the values
  for (int u = threadIdx.x; u < U && (int)threadIdx.x < nu; u += nu) {
    float c0[kSeg], c1[kSeg], x[kSeg];
#pragma unroll
    for (int j = 0; j < kSeg; ++j) { c0[j] = c[j * U + u]; c1[j] = c[(kSeg + j) * U + u]; }
    const float* ab = a + ((int64_t)bg * T_ + (int64_t)i0 * kSeg) * U + u;
    float prev = 0.f;
    for (int s = i0; s <= i1; ++s, ab += (int64_t)kSeg * U) {
#pragma unroll
      for (int j = 0; j < kSeg; ++j) x[j] = ab[(int64_t)j * U];
      if (s > i0) {
#pragma unroll
        for (int j = 0; j < kSeg; ++j) prev += fmaxf(x[j] + c1[j], 0.f);
        hbar[((int64_t)bg * nb + s - 1) * U + u] = prev * inv;
      }
      prev = 0.f;
#pragma unroll
      for (int j = 0; j < kSeg; ++j) prev += fmaxf(x[j] + c0[j], 0.f);
    }
  }
  for (int e = (int)threadIdx.x - nu; e >= 0 && e < dv; e += nv) {
    const T* vb = v + b * svz + g * svg + (int64_t)i0 * kSeg * svn + e * svk;
    float prev = 0.f, y[kSeg];
    for (int s = i0; s <= i1; ++s, vb += kSeg * svn) {
#pragma unroll
      for (int j = 0; j < kSeg; ++j) y[j] = Elem<T>::ld(vb + j * svn);
      if (s > i0) {
#pragma unroll
        for (int j = 0; j < kSeg; ++j) prev += y[j];
        Elem<T>::st(v_cmp + ((int64_t)bg * nbp + s - 1) * dv + e, prev * inv);
      }
      prev = 0.f;
#pragma unroll
      for (int j = 0; j < kSeg; ++j) prev += y[j];
    }
  }
}

// da[t,u] = sum_{blocks i holding t} [A[t,u] + C[t-i*d,u] > 0] * dhbar[i,u] / l; dv likewise without a mask.
__global__ void phi_pool_bwd_tok_kernel(const float* __restrict__ a, const float* __restrict__ c,
                                        const float* __restrict__ dhbar, const float* __restrict__ dv_cmp,
                                        float* __restrict__ da, float* __restrict__ dv, int T_, int U, int dvd,
                                        int l, int d, int nb, int nbp) {
  const int t = blockIdx.x, bg = blockIdx.y;
  const int ilo = t - l + 1 <= 0 ? 0 : (t - l + d) / d;  // ceil((t-l+1)/d)
  const int ihi = min(nb - 1, t / d);
  const float inv = 1.f / (float)l;
  for (int u = threadIdx.x; u < U; u += blockDim.x) {
    const float av = a[((int64_t)bg * T_ + t) * U + u];
    float acc = 0.f;
    for (int i = ilo; i <= ihi; ++i)
      if (av + c[(t - i * d) * U + u] > 0.f) acc += dhbar[((int64_t)bg * nb + i) * U + u];
    da[((int64_t)bg * T_ + t) * U + u] = acc * inv;
  }
  for (int x = threadIdx.x; x < dvd; x += blockDim.x) {
    float acc = 0.f;
    for (int i = ilo; i <= ihi; ++i) acc += dv_cmp[((int64_t)bg * nbp + i) * dvd + x];
    dv[((int64_t)bg * T_ + t) * dvd + x] = acc * inv;
  }
}

// dc_part[bg,j,u] = sum_i [A[i*d+j,u] + C[j,u] > 0] * dhbar[i,u] / l.  The blocks are dealt round-robin to kTabGroups
// thread groups whose sums are added in group order, so the result does not depend on scheduling.
constexpr int kTabGroups = 8, kTabLanes = 128;
__global__ void __launch_bounds__(kTabGroups * kTabLanes)
phi_pool_bwd_tab_kernel(const float* __restrict__ a, const float* __restrict__ c, const float* __restrict__ dhbar,
                        float* __restrict__ dc_part, int T_, int U, int l, int d, int nb) {
  __shared__ float part[kTabGroups][kTabLanes];
  const int j = blockIdx.x, bg = blockIdx.y;
  const int ul = threadIdx.x % kTabLanes, grp = threadIdx.x / kTabLanes;
  const float inv = 1.f / (float)l;
  for (int u0 = 0; u0 < U; u0 += kTabLanes) {
    const int u = u0 + ul;
    float acc = 0.f;
    if (u < U) {
      const float cv = c[j * U + u];
#pragma unroll 4
      for (int i = grp; i < nb; i += kTabGroups)
        if (a[((int64_t)bg * T_ + (int64_t)i * d + j) * U + u] + cv > 0.f) acc += dhbar[((int64_t)bg * nb + i) * U + u];
    }
    part[grp][ul] = acc;
    __syncthreads();
    if (grp == 0 && u < U) {
      float tot = 0.f;
#pragma unroll
      for (int g2 = 0; g2 < kTabGroups; ++g2) tot += part[g2][ul];
      dc_part[((int64_t)bg * l + j) * U + u] = tot * inv;
    }
    __syncthreads();
  }
}

// l = 32, d = 16: da (in the I/O type), dv_out += dv and the table's partial sums dc_part[chunk,bg,j,u] of a run of segments
// in one pass over A.  Was three kernels and two casts through fp32: A read three times, da written, read and written again.
template <typename T>
__global__ void __launch_bounds__(512) phi_pool_bwd_seg_kernel(const float* __restrict__ a, const float* __restrict__ c,
                                                               const float* __restrict__ dhbar, const float* __restrict__ dv_cmp,
                                                               T* __restrict__ da, float* __restrict__ dc_part, T* __restrict__ dv_out, int T_,
                                                               int arows, int U, int dvd, int nb, int nbp, int cs) {
  const int nseg = (T_ + kSeg - 1) / kSeg, s0 = blockIdx.x * cs, s1 = min(nseg, s0 + cs), bg = blockIdx.y;
  const float inv = 1.f / (2 * kSeg);
  const int nv = seg_value_threads(dvd), nu = blockDim.x - nv;
  for (int u = threadIdx.x; u < U && (int)threadIdx.x < nu; u += nu) {
    float c0[kSeg], c1[kSeg], acc0[kSeg], acc1[kSeg], x[kSeg];
#pragma unroll
    for (int j = 0; j < kSeg; ++j) { c0[j] = c[j * U + u]; c1[j] = c[(kSeg + j) * U + u]; acc0[j] = acc1[j] = 0.f; }
    const float* dh = dhbar + (int64_t)bg * nb * U + u;
    float before = s0 > 0 && s0 - 1 < nb ? dh[(int64_t)(s0 - 1) * U] : 0.f;
    for (int s = s0; s < s1; ++s) {
      const int64_t at = ((int64_t)bg * arows + (int64_t)s * kSeg) * U + u;
      const float here = s < nb ? dh[(int64_t)s * U] : 0.f;
#pragma unroll
      for (int j = 0; j < kSeg; ++j) x[j] = s * kSeg + j < T_ ? a[at + (int64_t)j * U] : 0.f;
#pragma unroll
      for (int j = 0; j < kSeg; ++j) {
        const float p = x[j] + c1[j] > 0.f ? before : 0.f, q = x[j] + c0[j] > 0.f ? here : 0.f;
        acc1[j] += p;
        acc0[j] += q;
        if (s * kSeg + j < T_) Elem<T>::st(da + at + (int64_t)j * U, (p + q) * inv);
      }
      before = here;
    }
    float* part = dc_part + ((int64_t)(blockIdx.x * gridDim.y + bg) * 2 * kSeg) * U + u;
#pragma unroll
    for (int j = 0; j < kSeg; ++j) {
      part[(int64_t)j * U] = acc0[j] * inv;
      part[(int64_t)(kSeg + j) * U] = acc1[j] * inv;
    }
  }
  for (int e = (int)threadIdx.x - nu; e >= 0 && e < dvd; e += nv)
    for (int s = s0; s < s1; ++s) {
      float y = 0.f, cur[kSeg];      // y: the same for every token of the segment
      T* out = dv_out + ((int64_t)bg * T_ + (int64_t)s * kSeg) * dvd + e;
      const int n = min(kSeg, T_ - s * kSeg);
#pragma unroll
      for (int j = 0; j < kSeg; ++j) cur[j] = j < n ? Elem<T>::ld(out + (int64_t)j * dvd) : 0.f;   // (all of them before the first store)
      if (s > 0 && s - 1 < nb) y += dv_cmp[((int64_t)bg * nbp + s - 1) * dvd + e];
      if (s < nb) y += dv_cmp[((int64_t)bg * nbp + s) * dvd + e];
#pragma unroll
      for (int j = 0; j < kSeg; ++j)
        if (j < n) Elem<T>::st(out + (int64_t)j * dvd, cur[j] + y * inv);
    }
}

bool phi_pool_bwd_fused_ok(int l, int d) { return l == 2 * kSeg && d == kSeg; }
// segments per CTA: two waves of the SMs, but no fewer than four (the partial tables are l * U floats each)
static int bwd_seg_chunk(int BG, int T) {
  const int nseg = (T + kSeg - 1) / kSeg;
  return (int)std::max<int64_t>(4, ((int64_t)nseg * BG + 295) / 296);
}
int phi_pool_bwd_parts(int BG, int T) {
  const int nseg = (T + kSeg - 1) / kSeg, cs = bwd_seg_chunk(BG, T);
  return (nseg + cs - 1) / cs;
}
template <typename T>
int phi_pool_bwd_fused(const float* a, const float* c, const float* dhbar, const float* dv_cmp, T* da, float* dc_part, T* dv_out, int BG, int Tn,
                       int arows, int U, int dv, int nb, int nbp, cudaStream_t st) {
  KernelTimer kt("phi_pool_bwd", st);
  phi_pool_bwd_seg_kernel<T><<<dim3(phi_pool_bwd_parts(BG, Tn), BG), seg_threads(U, dv), 0, st>>>(a, c, dhbar, dv_cmp, da, dc_part, dv_out, Tn, arows, U,
                                                                                                  dv, nb, nbp, bwd_seg_chunk(BG, Tn));
  return check_launch("phi_pool_bwd");
}
template int phi_pool_bwd_fused<float>(const float*, const float*, const float*, const float*, float*, float*, float*, int, int, int, int, int, int, int,
                                       cudaStream_t);
template int phi_pool_bwd_fused<__nv_bfloat16>(const float*, const float*, const float*, const float*, __nv_bfloat16*, float*, __nv_bfloat16*, int,
                                               int, int, int, int, int, int, cudaStream_t);

}  // namespace nsa

using namespace nsa;

extern "C" NSA_API int nsa_phi_pool_fwd(const float* a, const float* c, const void* v, const int64_t* vs, float* hbar,
                                void* v_cmp, int B, int G, int T, int U, int dv, int l, int d, int n_blocks, int nbp,
                                int dtype, void* stream) {
  NSA_REQUIRE(a && c && v && vs && hbar && v_cmp, "phi_pool_fwd: null pointer");
  NSA_REQUIRE(l > 0 && d > 0 && n_blocks >= 0 && nbp >= n_blocks && (int64_t)(n_blocks - 1) * d + l <= T,
              "phi_pool_fwd: blocks (n=%d,l=%d,d=%d) exceed T=%d", n_blocks, l, d, T);
  if (n_blocks == 0 || B * G == 0) return NSA_OK;
  dim3 grid(n_blocks, B * G);
  cudaStream_t st = (cudaStream_t)stream;
  KernelTimer kt("phi_pool_fwd", st);
  const bool seg = l == 2 * kSeg && d == kSeg;
  const int cb = (int)std::min<int64_t>(16, std::max<int64_t>(1, (int64_t)n_blocks * B * G / (148 * 4)));   // four waves, one segment of overlap per run
  const dim3 sgrid((n_blocks + cb - 1) / cb, B * G);
#define NSA_POOL(TYPE)                                                                                                                  \
  if (seg)                                                                                                                              \
    phi_pool_fwd_seg_kernel<TYPE><<<sgrid, seg_threads(U, dv), 0, st>>>(a, c, (const TYPE*)v, vs[0], vs[1], vs[2], vs[3], hbar,          \
                                                                        (TYPE*)v_cmp, G, T, U, dv, n_blocks, nbp, cb);                  \
  else                                                                                                                                  \
    phi_pool_fwd_kernel<TYPE><<<grid, 128, 0, st>>>(a, c, (const TYPE*)v, vs[0], vs[1], vs[2], vs[3], hbar, (TYPE*)v_cmp, G, T, U, dv, l, \
                                                    d, n_blocks, nbp)
  if (dtype == NSA_F32) {
    NSA_POOL(float);
  } else if (dtype == NSA_BF16) {
    NSA_POOL(__nv_bfloat16);
  } else {
    return fail(NSA_ERR_ARG, "phi_pool_fwd: unsupported dtype %d", dtype);
  }
#undef NSA_POOL
  return check_launch("phi_pool_fwd");
}

extern "C" NSA_API int nsa_phi_pool_bwd(const float* a, const float* c, const float* dhbar, const float* dv_cmp, float* da,
                                float* dc_part, float* dv, int B, int G, int T, int U, int dv_dim, int l, int d,
                                int n_blocks, int nbp, void* stream) {
  NSA_REQUIRE(a && c && dhbar && dv_cmp && da && dc_part && dv, "phi_pool_bwd: null pointer");
  NSA_REQUIRE(l > 0 && d > 0 && n_blocks >= 0 && (int64_t)(n_blocks - 1) * d + l <= T, "phi_pool_bwd: bad blocks");
  if (B * G == 0 || T == 0) return NSA_OK;
  cudaStream_t st = (cudaStream_t)stream;
  KernelTimer kt("phi_pool_bwd", st);
  phi_pool_bwd_tok_kernel<<<dim3(T, B * G), 128, 0, st>>>(a, c, dhbar, dv_cmp, da, dv, T, U, dv_dim, l, d, n_blocks,
                                                          nbp);
  if (int rc = check_launch("phi_pool_bwd_tok")) return rc;
  phi_pool_bwd_tab_kernel<<<dim3(l, B * G), kTabGroups * kTabLanes, 0, st>>>(a, c, dhbar, dc_part, T, U, l, d, n_blocks);
  return check_launch("phi_pool_bwd_tab");
}
