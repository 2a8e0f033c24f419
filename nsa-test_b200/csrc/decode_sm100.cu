// A handful of newest tokens against a key/value cache (decode): projections, cache update, block compression, Eq. 8-11
// block choice, the three attention branches and the gate mix, for up to 64 (sequence, group, token) rows.
//
// The tile kernels pad such a call to 128 query rows and need an inverse index, padded copies and one launch per piece:
// 45 launches and 760 us per token at B=1, 2K cached; 80 launches and 1400 us at B=8, 32K (137 and 167 us here).
// What the work cannot do without is reading the weights once (131 MB for the 64-head configuration, 20 us) and the visible
// keys and values once, so here the keys of a row are cut into 64-key chunks, one CTA each, that serve all heads of the group,
// and everything between two grid-wide dependencies is one launch:
//   1 project     weights x tokens on mma.sync (8 tokens are one n tile; the weights stream through once), written straight
//                 into the caches; the gate MLP's hidden layer is one more row range
//   2 phi         only when the tokens complete compression blocks: the block compression of every other path
//   3 chunks      compressed and sliding-window chunks + the gate logits
//   4 top-n       Eq. 8-11 from the fp32 logits the chunks left
//   5 chunks      the selected blocks
//   6 combine     merge of the chunk partials, gates, mix
// Launches overlap their ramp-up by programmatic dependent launch.
//
// The block choice is a discrete function of rounded sums: q and the compression's keys that round differently, or sums in
// another order, let near-ties fall the other way (in 2 of 384 rows at 32000 cached tokens).  So all that the choice reads is
// made as on the other paths: q and the new compression keys come from the caller, who forms them with the products that the
// tile kernels' callers use; logits are one fma chain over the head dimension and the Eq. 8-10 sums run in the order of
// score_topn.cu.  The chosen blocks are the same bit for bit.
//
// Keys of the compressed blocks stay fp32 and their products run on the FMA pipe (they rank the blocks); bf16 keys and P V run
// on mma.sync, with P as bf16 hi + lo, so the probabilities keep 16 mantissa bits (the tile kernels: 8).  (tcgen05 tiles have 64
// rows at least; a group has at most 16 heads.)
#include <algorithm>

#include "common.cuh"
#include "fa_sm100.cuh"
#include "phi.cuh"

namespace nsa {
namespace {

constexpr int kDecThreads = 256;
constexpr int kDecRows = 64;     // (sequence, group, token) rows
constexpr int kDecTokens = 8;    // tokens of one projection call: an mma n tile
constexpr int kDecMaxN = 64;
constexpr int kProjThreads = 128;

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
int launch_pdl(const char* what, void (*kern)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  if (e != cudaSuccess) return fail(NSA_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e));
  return NSA_OK;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(void* dst, const void* src, bool full) {   // bytes beyond the source count are zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(full ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ld_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// ------------------------------------------------------------------------------------------------ projections
// Row ranges ("segments") of stacked weight matrices, 16 rows a CTA; the four warps split d_model.  The weights stream from
// HBM once: 16-byte loads, 64 consecutive k of 16 rows per warp and step.  The 32-k groups are multiplied in permuted order
// (both operands alike), so that a thread's 16 bytes are two mma fragments.
enum { kSegK = 0, kSegV, kSegGate, kSegCopy };      // kSegCopy: no product, k_new goes into its cache
struct ProjSeg {
  const __nv_bfloat16 *w, *bias;
  __nv_bfloat16* dst;
  int tile0, D, kind;    // first tile of the segment, head dim (width for the gate), layout
};
struct ProjArgs {
  ProjSeg seg[7];
  int nseg, R, Tn, K, G, pos;
  int64_t cap, sxb, sxt, sk[4];
  const __nv_bfloat16 *x, *k_new;
};
__global__ void __launch_bounds__(kProjThreads) decode_project_kernel(const __grid_constant__ ProjArgs p) {
  __shared__ float red[4][16][9];
  pdl_wait();
  pdl_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, qd = lane & 3;
  int si = 0;
  while (si + 1 < p.nseg && (int)blockIdx.x >= p.seg[si + 1].tile0) ++si;
  const ProjSeg& sg = p.seg[si];
  const int row0 = ((int)blockIdx.x - sg.tile0) * 16;
  const int n = threadIdx.x >> 4, r = threadIdx.x & 15, row = row0 + r, b = n / p.Tn, t = n % p.Tn, hd = row / sg.D, e = row % sg.D;
  if (sg.kind == kSegCopy) {
    if (n < p.R) sg.dst[(((int64_t)b * p.G + hd) * sg.D + e) * p.cap + p.pos + t] = p.k_new[b * p.sk[0] + hd * p.sk[1] + e * p.sk[2] + t * p.sk[3]];
    return;
  }
  const __nv_bfloat16* wa = sg.w + (int64_t)(row0 + g) * p.K + qd * 8;
  const __nv_bfloat16* wb = wa + (int64_t)8 * p.K;
  const bool have = g < p.R;
  const __nv_bfloat16* xr = p.x + (have ? (g / p.Tn) * p.sxb + (g % p.Tn) * p.sxt : 0) + qd * 8;
  float c[4] = {0.f, 0.f, 0.f, 0.f};
  const int steps = p.K / 64;
  constexpr int U = 3;
  for (int s0 = warp; s0 < steps; s0 += 4 * U) {
    uint4 a[U][2], b[U][2], x[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int s = s0 + 4 * u;
      if (s < steps) {
        a[u][0] = ld_stream(wa + s * 64); a[u][1] = ld_stream(wa + s * 64 + 32);
        b[u][0] = ld_stream(wb + s * 64); b[u][1] = ld_stream(wb + s * 64 + 32);
        x[u][0] = have ? *reinterpret_cast<const uint4*>(xr + s * 64) : make_uint4(0, 0, 0, 0);
        x[u][1] = have ? *reinterpret_cast<const uint4*>(xr + s * 64 + 32) : make_uint4(0, 0, 0, 0);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (s0 + 4 * u < steps) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          mma16816(c, a[u][hf].x, b[u][hf].x, a[u][hf].y, b[u][hf].y, x[u][hf].x, x[u][hf].y);
          mma16816(c, a[u][hf].z, b[u][hf].z, a[u][hf].w, b[u][hf].w, x[u][hf].z, x[u][hf].w);
        }
      }
  }
  red[warp][g][qd * 2] = c[0];     red[warp][g][qd * 2 + 1] = c[1];
  red[warp][g + 8][qd * 2] = c[2]; red[warp][g + 8][qd * 2 + 1] = c[3];
  __syncthreads();
  if (n >= p.R) return;
  const float y = (red[0][r][n] + red[1][r][n]) + (red[2][r][n] + red[3][r][n]);
  __nv_bfloat16 o = __float2bfloat16_rn(y);
  if (sg.bias) o = __float2bfloat16_rn(__bfloat162float(o) + __bfloat162float(sg.bias[row]));
  if (sg.kind == kSegK) sg.dst[(((int64_t)b * p.G + hd) * sg.D + e) * p.cap + p.pos + t] = o;
  else if (sg.kind == kSegV) sg.dst[(((int64_t)b * p.G + hd) * p.cap + p.pos + t) * sg.D + e] = o;
  else sg.dst[(int64_t)n * sg.D + row] = __bfloat162float(o) > 0.f ? o : __float2bfloat16_rn(0.f);
}

// ------------------------------------------------------------------------------------------------ attention chunks
struct DecArgs {
  const __nv_bfloat16* q;
  int64_t sqb, sqh, sqt;
  const __nv_bfloat16 *k_slc, *v_slc, *k_win, *v_win, *v_cmp;
  const float* k_cmp;
  int64_t cap, nbp;
  int B, H, G, Tn, hpg, nb, pos, window, l, d, n, n_fixed, s_, a_, gate_mode;
  int nc, nw, P;             // chunks per row: compressed, window; all (with the n slots)
  float scale;
  const __nv_bfloat16 *gh, *gw2, *gb2;   // gate hidden layer [R, D2] and second linear layer: logits computed here
  int D2;
  float* logits;             // [B,Tn,3H]
  float* part_o;             // [rows][P][16][DV], not normalised
  float2* part_st;           // [rows][P][16]: (max, sum)
  float* slog;               // [rows][16][nc*64]: logits of the compressed blocks, -inf where hidden
  int* idx;                  // [rows][n]
  __nv_bfloat16* out;        // [B,Tn,H,DV]
  __nv_bfloat16 *o_cmp, *o_slc, *o_win;   // optional [B,H,Tn,DV]
  float* gates;              // optional [B,H,Tn,3]
};

template <int DK, int DV, bool WITH_CMP>
struct DecSmem {
  static constexpr int kQ = 16 * (DK + 8) * 2;       // bf16 queries (rows 16 bytes off a bank period)
  static constexpr int kK = DK * 72 * 2;             // bf16 key tile [DK][64]
  static constexpr int kC = DK * 16 * 4 + DK * 64 * 4;   // compressed: fp32 queries [DK][16], fp32 key tile [DK][64]
  static constexpr int kKC = WITH_CMP ? kC : kK;
  static constexpr int kV = 64 * (DV + 8) * 2;
  static constexpr int kS = 16 * 66 * 4;
  static constexpr int kP = 2 * 16 * 72 * 2;
  static constexpr int oQ = 0, oK = oQ + kQ, oV = oK + kKC, oS = oV + kV, oP = oS + kS, kBytes = oP + kP;
};

// One chunk of 64 keys [key0, key0 + 64) for the heads of a group: S, its softmax over the chunk, P V.  Keys klo <= key < khi
// count.  CMP: fp32 keys [DK][ld], whose logits are also kept for the block choice: a thread owns a key and four heads and
// walks the head dimension in one chain, the sums of score_logits_kernel.
template <int DK, int DV, bool CMP, bool WITH_CMP>
__device__ __forceinline__ void attend_chunk(const DecArgs& p, uint8_t* sm, int row, int chunk, const void* kbase, const __nv_bfloat16* vbase,
                                             int64_t ld, int key0, int klo, int khi, int b, int h0, int tn) {
  using SM = DecSmem<DK, DV, WITH_CMP>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  __nv_bfloat16* sQ = (__nv_bfloat16*)(sm + SM::oQ);
  __nv_bfloat16* sK = (__nv_bfloat16*)(sm + SM::oK);
  __nv_bfloat16* sV = (__nv_bfloat16*)(sm + SM::oV);
  float* sS = (float*)(sm + SM::oS);
  __nv_bfloat16* sP = (__nv_bfloat16*)(sm + SM::oP);
  const __nv_bfloat16* qb = p.q + b * p.sqb + (int64_t)h0 * p.sqh + tn * p.sqt;
  if (!CMP) {
    for (int i = tid; i < DK * 8; i += kDecThreads) {
      const int r = i >> 3, cc = i & 7;
      cp16(sK + r * 72 + cc * 8, (const __nv_bfloat16*)kbase + (int64_t)r * ld + key0 + cc * 8, true);
    }
    for (int i = tid; i < 16 * (DK / 8); i += kDecThreads) {
      const int r = i / (DK / 8), cc = i % (DK / 8);
      cp16(sQ + r * (DK + 8) + cc * 8, qb + (r < p.hpg ? r * p.sqh : 0) + cc * 8, r < p.hpg);
    }
    cp_commit();
  } else {
    float* sKf = (float*)(sm + SM::oK) + DK * 16;
    for (int i = tid; i < DK * 16; i += kDecThreads) {
      const int r = i >> 4, cc = i & 15;
      cp16(sKf + r * 64 + cc * 4, (const float*)kbase + (int64_t)r * ld + key0 + cc * 4, true);
    }
    cp_commit();
  }
  // (rows outside the visible range arrive as zeros: stale values behind the newest token must not meet P = 0)
  for (int i = tid; i < 64 * (DV / 8); i += kDecThreads) {
    const int r = i / (DV / 8), cc = i % (DV / 8);
    const bool in = key0 + r >= klo && key0 + r < khi;
    cp16(sV + r * (DV + 8) + cc * 8, vbase + (int64_t)(in ? key0 + r : 0) * DV + cc * 8, in);
  }
  cp_commit();
  if (CMP) {
    float* qf = (float*)(sm + SM::oK);          // [DK][16]
    const float* sKf = qf + DK * 16;            // [DK][64]
    for (int i = tid; i < DK * 16; i += kDecThreads) {
      const int r = i / DK, dd = i % DK;
      qf[dd * 16 + r] = r < p.hpg ? __bfloat162float(qb[r * p.sqh + dd]) : 0.f;
    }
    cp_wait<1>();
    __syncthreads();
    const int kk = tid & 63, h4 = (tid >> 6) * 4;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 16
    for (int dd = 0; dd < DK; ++dd) {
      const float kv = sKf[dd * 64 + kk];
      const float4 qv = *reinterpret_cast<const float4*>(qf + dd * 16 + h4);
      acc[0] = fmaf(qv.x, kv, acc[0]); acc[1] = fmaf(qv.y, kv, acc[1]);
      acc[2] = fmaf(qv.z, kv, acc[2]); acc[3] = fmaf(qv.w, kv, acc[3]);
    }
    float* lg = p.slog + (int64_t)row * 16 * (p.nc * 64) + chunk * 64;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int u = h4 + e;
      const float x = key0 + kk < khi && u < p.hpg ? acc[e] * p.scale : -CUDART_INF_F;
      sS[u * 66 + kk] = x;
      if (u < p.hpg) lg[(int64_t)u * (p.nc * 64) + kk] = x;
    }
  } else {
    cp_wait<1>();
    __syncthreads();
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    const uint32_t aq = smem_addr(sQ + (lane & 15) * (DK + 8) + (lane >> 4) * 8);
    const uint32_t ak = smem_addr(sK + lane * 72 + warp * 8);
#pragma unroll
    for (int k0 = 0; k0 < DK; k0 += 32) {
      uint32_t bf[4], a0[4], a1[4];
      ldsm4t(bf, ak + k0 * 144);
      ldsm4(a0, aq + k0 * 2);
      ldsm4(a1, aq + k0 * 2 + 32);
      mma16816(c, a0[0], a0[1], a0[2], a0[3], bf[0], bf[1]);
      mma16816(c, a1[0], a1[1], a1[2], a1[3], bf[2], bf[3]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int u = (lane >> 2) + (e >> 1) * 8, kk = warp * 8 + (lane & 3) * 2 + (e & 1);
      sS[u * 66 + kk] = key0 + kk >= klo && key0 + kk < khi ? c[e] * p.scale : -CUDART_INF_F;
    }
  }
  __syncthreads();
  float2* st = p.part_st + ((int64_t)row * p.P + chunk) * 16;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int u = warp * 2 + e;
    const float x0 = sS[u * 66 + lane], x1 = sS[u * 66 + 32 + lane];
    const float m = warp_max(fmaxf(x0, x1));
    const float p0 = m == -CUDART_INF_F ? 0.f : expf(x0 - m), p1 = m == -CUDART_INF_F ? 0.f : expf(x1 - m);
    const float sum = warp_sum(p0 + p1);
    if (lane == 0) st[u] = make_float2(m, sum);
    const __nv_bfloat16 h0_ = __float2bfloat16_rn(p0), h1_ = __float2bfloat16_rn(p1);
    sP[u * 72 + lane] = h0_;
    sP[u * 72 + 32 + lane] = h1_;
    sP[(16 + u) * 72 + lane] = __float2bfloat16_rn(p0 - __bfloat162float(h0_));
    sP[(16 + u) * 72 + 32 + lane] = __float2bfloat16_rn(p1 - __bfloat162float(h1_));
  }
  cp_wait<0>();
  __syncthreads();
  constexpr int NT = DV / 64;     // 8-column tiles per warp
  float o[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
  const uint32_t ap = smem_addr(sP + (lane & 15) * 72 + (lane >> 4) * 8);
#pragma unroll
  for (int k0 = 0; k0 < 64; k0 += 32) {
    uint32_t h0f[4], h1f[4], l0f[4], l1f[4];
    ldsm4(h0f, ap + k0 * 2);
    ldsm4(h1f, ap + k0 * 2 + 32);
    ldsm4(l0f, ap + 16 * 144 + k0 * 2);
    ldsm4(l1f, ap + 16 * 144 + k0 * 2 + 32);
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      uint32_t bf[4];
      ldsm4t(bf, smem_addr(sV + (k0 + lane) * (DV + 8) + (warp * NT + i) * 8));
      mma16816(o[i], h0f[0], h0f[1], h0f[2], h0f[3], bf[0], bf[1]);
      mma16816(o[i], h1f[0], h1f[1], h1f[2], h1f[3], bf[2], bf[3]);
      mma16816(o[i], l0f[0], l0f[1], l0f[2], l0f[3], bf[0], bf[1]);
      mma16816(o[i], l1f[0], l1f[1], l1f[2], l1f[3], bf[2], bf[3]);
    }
  }
  float* po = p.part_o + ((int64_t)row * p.P + chunk) * 16 * DV;
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    const int u = lane >> 2, cc = (warp * NT + i) * 8 + (lane & 3) * 2;
    if (u < p.hpg) *reinterpret_cast<float2*>(po + u * DV + cc) = make_float2(o[i][0], o[i][1]);
    if (u + 8 < p.hpg) *reinterpret_cast<float2*>(po + (u + 8) * DV + cc) = make_float2(o[i][2], o[i][3]);
  }
}
__device__ __forceinline__ void empty_chunk(const DecArgs& p, int row, int chunk) {
  if (threadIdx.x < 16) p.part_st[((int64_t)row * p.P + chunk) * 16 + threadIdx.x] = make_float2(-CUDART_INF_F, 0.f);
}

template <int DK, int DV>
__global__ void __launch_bounds__(kDecThreads) decode_dense_kernel(const __grid_constant__ DecArgs p) {
  extern __shared__ __align__(16) uint8_t dsm[];
  pdl_wait();
  pdl_launch();
  const int rows = p.B * p.G * p.Tn, per = p.nc + p.nw;
  const int x = blockIdx.x;
  if (x >= rows * per) {   // gate logits: a warp per output, all tokens (the second linear layer, bias added in fp32)
    const int o = (x - rows * per) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, R = p.B * p.Tn, O = 3 * p.H;
    if (o >= O) return;
    float acc[kDecTokens];
#pragma unroll
    for (int r = 0; r < kDecTokens; ++r) acc[r] = 0.f;
    for (int c = lane * 8; c < p.D2; c += 256) {
      const uint4 wv = *reinterpret_cast<const uint4*>(p.gw2 + (int64_t)o * p.D2 + c);
      const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&wv);
#pragma unroll
      for (int r = 0; r < kDecTokens; ++r)
        if (r < R) {
          const uint4 hv = *reinterpret_cast<const uint4*>(p.gh + (int64_t)r * p.D2 + c);
          const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&hv);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 wf = __bfloat1622float2(w2[e]), hf = __bfloat1622float2(h2[e]);
            acc[r] = fmaf(wf.x, hf.x, fmaf(wf.y, hf.y, acc[r]));
          }
        }
    }
#pragma unroll
    for (int r = 0; r < kDecTokens; ++r) {
      const float s = warp_sum(acc[r]);
      if (lane == 0 && r < R) p.logits[(int64_t)r * O + o] = s + (p.gb2 ? __bfloat162float(p.gb2[o]) : 0.f);
    }
    return;
  }
  const int row = x / per, chunk = x % per, bg = row / p.Tn, tn = row % p.Tn, b = bg / p.G, h0 = (bg % p.G) * p.hpg;
  const int t = p.pos + tn;
  if (chunk < p.nc) {
    // block i is visible when it ends at or before t
    const int vis = t >= p.l - 1 ? min(p.nb, (t - p.l + 1) / p.d + 1) : 0;
    attend_chunk<DK, DV, true, true>(p, dsm, row, chunk, p.k_cmp + (int64_t)bg * DK * p.nbp, p.v_cmp + (int64_t)bg * p.nbp * DV, p.nbp,
                               chunk * 64, 0, vis, b, h0, tn);
  } else {
    const int klo = max(0, t - p.window + 1), key0 = (klo / 64 + chunk - p.nc) * 64;
    if (key0 > t) { empty_chunk(p, row, chunk); return; }
    attend_chunk<DK, DV, false, true>(p, dsm, row, chunk, p.k_win + (int64_t)bg * DK * p.cap, p.v_win + (int64_t)bg * p.cap * DV, p.cap, key0,
                                klo, t + 1, b, h0, tn);
  }
}

template <int DK, int DV>
__global__ void __launch_bounds__(kDecThreads) decode_selected_kernel(const __grid_constant__ DecArgs p) {
  extern __shared__ __align__(16) uint8_t dsm[];
  pdl_wait();
  pdl_launch();
  const int row = blockIdx.y, slot = blockIdx.x, bg = row / p.Tn, tn = row % p.Tn, b = bg / p.G, h0 = (bg % p.G) * p.hpg;
  const int t = p.pos + tn, id = p.idx[(int64_t)row * p.n + slot];    // (ids of a row are distinct)
  if (id < 0 || (int64_t)id * 64 > t) { empty_chunk(p, row, p.nc + p.nw + slot); return; }
  attend_chunk<DK, DV, false, false>(p, dsm, row, p.nc + p.nw + slot, p.k_slc + (int64_t)bg * DK * p.cap, p.v_slc + (int64_t)bg * p.cap * DV,
                              p.cap, id * 64, 0, t + 1, b, h0, tn);
}

// ------------------------------------------------------------------------------------------------ block choice
// Largest (score, lower id first) `k` of keys[first], keys[first + step], ... by one warp: the lanes keep their own maximum, two
// warp-wide integer maxima decide a round and only the winner looks through its share again.  Scores are >= 0, so their bits
// order like integers.
__device__ __forceinline__ void warp_top(unsigned long long* keys, int first, int step, int total, int k, unsigned long long* out) {
  const int lane = threadIdx.x & 31;
  auto best = [&](int& at) {
    unsigned long long m = 0;
    at = -1;
    for (int j = first + lane * step; j < total; j += 32 * step)
      if (keys[j] > m) { m = keys[j]; at = j; }
    return m;
  };
  int at;
  unsigned long long mine = best(at);
  for (int r = 0; r < k; ++r) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(mine >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(mine >> 32) == hi ? (unsigned)mine : 0u);
    const unsigned long long w = ((unsigned long long)hi << 32) | lo;
    if (lane == 0) out[r] = w;
    if (w != 0 && mine == w) {      // (ids make the keys distinct)
      keys[at] = 0;
      mine = best(at);
    }
  }
  __syncwarp();
}
constexpr int kTopWarps = 16;
constexpr size_t kTopSmemMax = 200 * 1024;
// One CTA per row: softmax statistics of the heads, Eq. 9 sums per selection block summed over the heads in order, then the top
// n: each warp of its share, one warp of the survivors.  All sums run in the order of score_topn_kernel: a head's denominator as
// that kernel's 256 threads form it (block i belongs to thread i % 256; a warp's sum, then the eight warps'), p = e * (1 / sum)
// rounded, and a block's terms one after the other from zero.
__global__ void __launch_bounds__(kTopWarps * 32) decode_topn_kernel(const __grid_constant__ DecArgs p, int n_sel, int n_eff) {
  extern __shared__ __align__(16) unsigned long long keys[];   // [n_eff], then [kTopWarps * n]
  unsigned long long* cand = keys + n_eff;
  __shared__ float hm[16], hinv[16], red[16][8];
  __shared__ unsigned long long top[kDecMaxN];
  pdl_wait();
  pdl_launch();
  const int row = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = p.pos + row % p.Tn;
  if (warp < p.hpg) {
    const float2* st = p.part_st + (int64_t)row * p.P * 16 + warp;
    float m = -CUDART_INF_F;
    for (int c = lane; c < p.nc; c += 32) m = fmaxf(m, st[c * 16].x);
    m = warp_max(m);
    if (lane == 0) hm[warp] = m;
  }
  __syncthreads();
  const int ncol = p.nc * 64;
  const float* lg = p.slog + (int64_t)row * 16 * ncol;
  for (int i = warp; i < p.hpg * 8; i += kTopWarps) {
    const int h = i >> 3, w8 = i & 7;
    const float m = hm[h];
    float s = 0.f;
    if (m != -CUDART_INF_F)
#pragma unroll 8
      for (int c = w8 * 32 + lane; c < ncol; c += 256) s += expf(lg[(int64_t)h * ncol + c] - m);   // (hidden blocks add zero)
    s = warp_sum(s);
    if (lane == 0) red[h][w8] = s;
  }
  __syncthreads();
  if (threadIdx.x < p.hpg) {
    float s = red[threadIdx.x][0];
#pragma unroll
    for (int w = 1; w < 8; ++w) s += red[threadIdx.x][w];
    hinv[threadIdx.x] = 1.f / s;
  }
  __syncthreads();
  for (int j = threadIdx.x; j < n_eff; j += kTopWarps * 32) {
    float agg = 0.f;
    for (int h = 0; h < p.hpg; ++h) {
      const float m = hm[h], inv = hinv[h];
      const bool none = m == -CUDART_INF_F;    // nothing visible: block 0 alone (nsa/kernels.py:2316-2343)
      const float* lh = lg + (int64_t)h * ncol;
      auto prob = [&](int c) { return none ? (c == 0 ? 1.f : 0.f) : c < ncol ? __fmul_rn(expf(lh[c] - m), inv) : 0.f; };
      float sel = 0.f;
      if (p.a_ == 2) {                         // (a block's term is the next sum's first one)
        float cur = prob(p.s_ * j);
        for (int mm = 0; mm < p.s_; ++mm) {
          const float next = prob(p.s_ * j + mm + 1);
          sel = __fadd_rn(__fadd_rn(sel, cur), next);
          cur = next;
        }
      } else {
        for (int mm = 0; mm < p.s_; ++mm)
          for (int nn = 0; nn < p.a_; ++nn) sel = __fadd_rn(sel, prob(p.s_ * j + mm + nn));
      }
      agg = __fadd_rn(agg, sel);
    }
    if (!(agg >= 0.f)) agg = 0.f;          // (not a number)
    keys[j] = ((unsigned long long)__float_as_uint(agg) << 32) | (unsigned)~j;
  }
  __syncthreads();
  const int k = min(p.n, n_sel);
  warp_top(keys, warp, kTopWarps, n_eff, k, cand + warp * k);
  __syncthreads();
  if (warp == 0) {
    warp_top(cand, 0, 1, kTopWarps * k, k, top);
    if (lane == 0) {
      int* out = p.idx + (int64_t)row * p.n;
      int cnt = 0;
      auto push = [&](int id) {
        if (cnt >= p.n) return;
        for (int i = 0; i < cnt; ++i)
          if (out[i] == id) return;
        out[cnt++] = id;
      };
      if (p.n_fixed > 0) {
        push(0);
        push(t < 64 ? 0 : (t - 64) / 64);
        push(t / 64);
      }
      for (int r = 0; r < k; ++r)
        if (top[r] != 0) push((int)~(unsigned)top[r]);
      for (; cnt < p.n; ++cnt) out[cnt] = -1;
    }
  }
}

// ------------------------------------------------------------------------------------------------ merge + gates + mix
// One CTA per (row, head): DV columns x 4 lanes of chunks, added in a fixed order.
template <int DV>
__global__ void __launch_bounds__(4 * DV) decode_combine_kernel(const __grid_constant__ DecArgs p) {
  extern __shared__ float wsm[];       // [P] weights
  __shared__ float red[4][3][DV];
  __shared__ float bl[3];
  pdl_wait();
  pdl_launch();
  const int row = blockIdx.x, u = blockIdx.y, tid = threadIdx.x;
  const int bg = row / p.Tn, tn = row % p.Tn, b = bg / p.G, h = (bg % p.G) * p.hpg + u;
  const float2* st = p.part_st + (int64_t)row * p.P * 16 + u;
  const int beg[4] = {0, p.nc, p.nc + p.nw, p.P};
  const int br = tid >> 5, lane = tid & 31;
  if (br < 3) {
    float m = -CUDART_INF_F;
    for (int c = beg[br] + lane; c < beg[br + 1]; c += 32) m = fmaxf(m, st[c * 16].x);
    m = warp_max(m);
    float s = 0.f;
    for (int c = beg[br] + lane; c < beg[br + 1]; c += 32) {
      const float2 v = st[c * 16];
      const float w = v.y != 0.f ? expf(v.x - m) : 0.f;
      wsm[c] = w;
      s += w * v.y;
    }
    s = warp_sum(s);
    if (lane == 0) bl[br] = s;
  }
  __syncthreads();
  const int col = tid % DV, part = tid / DV;
  const float* po = p.part_o + ((int64_t)row * p.P * 16 + u) * DV + col;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    float acc = 0.f;
#pragma unroll 4
    for (int c = beg[i] + part; c < beg[i + 1]; c += 4) {
      const float w = wsm[c];
      if (w != 0.f) acc = fmaf(w, po[(int64_t)c * 16 * DV], acc);      // (empty chunks left nothing to read)
    }
    red[part][i][col] = acc;
  }
  __syncthreads();
  if (part != 0) return;
  float o[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float s = (red[0][i][col] + red[1][i][col]) + (red[2][i][col] + red[3][i][col]);
    o[i] = bl[i] != 0.f ? s / bl[i] : 0.f;
  }
  float gt[3];
  gates3(p.logits + ((int64_t)(b * p.Tn + tn) * p.H + h) * 3, p.gate_mode, gt);
  // branch order: compressed, window, selected in the partials; the gates are (compressed, selected, window)
  const float y = (o[0] * gt[0] + o[2] * gt[1]) + o[1] * gt[2];
  p.out[((int64_t)(b * p.Tn + tn) * p.H + h) * DV + col] = __float2bfloat16_rn(y);
  const int64_t hr = (int64_t)(b * p.H + h) * p.Tn + tn;
  if (p.o_cmp) p.o_cmp[hr * DV + col] = __float2bfloat16_rn(o[0]);
  if (p.o_win) p.o_win[hr * DV + col] = __float2bfloat16_rn(o[1]);
  if (p.o_slc) p.o_slc[hr * DV + col] = __float2bfloat16_rn(o[2]);
  if (p.gates && col < 3) p.gates[hr * 3 + col] = gt[col];
}

// ------------------------------------------------------------------------------------------------ host side
size_t al256(size_t x) { return (x + 255) & ~size_t(255); }
bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

struct DecLayout {
  int rows, nc, nw, P, n_sel, n_eff;
  size_t o_gh, o_logits, o_phi, o_part, o_st, o_slog, o_idx, total;
};
DecLayout dec_layout(const nsa_decode_desc& d) {
  DecLayout L;
  L.rows = d.B * d.G * d.Tn;
  L.nc = (d.nb + 63) / 64;
  L.nw = (int)std::min<int64_t>(((int64_t)d.window + 62) / 64 + 1, ((int64_t)d.pos + d.Tn + 63) / 64);
  L.P = L.nc + L.nw + d.n;
  const int s = d.l_prime / d.d;
  L.n_sel = (d.nbp + s - 1) / s;
  L.n_eff = std::min(L.n_sel, (d.nb + s - 1) / s + d.n);     // blocks beyond the compressed ones score zero, lowest ids first
  size_t o = 0;
  auto take = [&](size_t b) { const size_t r = o; o += al256(b); return r; };
  const size_t R = (size_t)d.B * d.Tn;
  L.o_gh = take(R * d.d_gate * 2);
  L.o_logits = take(R * 3 * d.H * 4);
  L.o_phi = take(d.project && d.nb_new > 0 ? compress_blocks_workspace_bytes(d, NSA_BF16) : 0);
  L.o_part = take((size_t)L.rows * L.P * 16 * d.dv * 4);
  L.o_st = take((size_t)L.rows * L.P * 16 * sizeof(float2));
  L.o_slog = take((size_t)L.rows * 16 * L.nc * 64 * 4);
  L.o_idx = take((size_t)L.rows * d.n * 4);
  L.total = o;
  return L;
}
size_t topn_smem(const nsa_decode_desc& d, const DecLayout& L) {
  return ((size_t)L.n_eff + (size_t)kTopWarps * std::min(d.n, L.n_sel)) * sizeof(unsigned long long);
}

template <int DK, int DV>
int launch_attend(const DecArgs& a, const nsa_decode_desc& d, const DecLayout& L, cudaStream_t st) {
  constexpr int kDense = DecSmem<DK, DV, true>::kBytes, kSelected = DecSmem<DK, DV, false>::kBytes;
  // (the attributes are the kernels' own, shared by all threads: bounds that do not depend on the call)
  cudaFuncSetAttribute(decode_dense_kernel<DK, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDense);
  cudaFuncSetAttribute(decode_selected_kernel<DK, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSelected);
  cudaFuncSetAttribute(decode_topn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTopSmemMax);
  {
    KernelTimer kt("decode_dense", st);
    const int gate_ctas = a.gh ? (3 * d.H + 7) / 8 : 0;
    if (int rc = launch_pdl("decode_dense", decode_dense_kernel<DK, DV>, dim3(L.rows * (L.nc + L.nw) + gate_ctas), kDecThreads, kDense, st, a)) return rc;
  }
  {
    KernelTimer kt("decode_topn", st);
    if (int rc = launch_pdl("decode_topn", decode_topn_kernel, dim3(L.rows), kTopWarps * 32, topn_smem(d, L), st, a, L.n_sel, L.n_eff)) return rc;
  }
  {
    KernelTimer kt("decode_selected", st);
    if (int rc = launch_pdl("decode_selected", decode_selected_kernel<DK, DV>, dim3(d.n, L.rows), kDecThreads, kSelected, st, a)) return rc;
  }
  KernelTimer kt("decode_combine", st);
  return launch_pdl("decode_combine", decode_combine_kernel<DV>, dim3(L.rows, a.hpg), 4 * DV, (size_t)L.P * 4, st, a);
}

}  // namespace
}  // namespace nsa

using namespace nsa;

extern "C" NSA_API int nsa_decode_supported(const nsa_decode_desc* dp) {
  if (!dp) return 0;
  const nsa_decode_desc& d = *dp;
  if (d.B <= 0 || d.Tn <= 0 || d.G <= 0 || d.H <= 0 || d.H % d.G != 0 || d.H / d.G > 16) return 0;
  if ((int64_t)d.B * d.G * d.Tn > kDecRows) return 0;
  if (!((d.dk == 192 && d.dv == 128) || (d.dk == 128 && d.dv == 128) || (d.dk == 64 && d.dv == 64))) return 0;
  if (d.l <= 0 || d.d <= 0 || d.l % d.d != 0 || d.l_prime != 64 || 64 % d.d != 0 || d.n <= 0 || d.n > kDecMaxN || d.window <= 0) return 0;
  if (d.nb <= 0 || d.nb > d.nbp || d.nbp % 64 != 0 || d.cap % 64 != 0 || d.pos < 0 || (int64_t)d.pos + d.Tn > d.cap) return 0;
  if (d.project) {
    if (d.B * d.Tn > kDecTokens || d.d_model <= 0 || d.d_model % 64 != 0 || d.d_gate <= 0 || d.d_gate % 16 != 0) return 0;
    if (d.nb_new < 0 || d.nb_new > d.nb || (d.nb_new > 0 && d.U <= 0)) return 0;
  }
  const DecLayout L = dec_layout(d);
  return topn_smem(d, L) <= kTopSmemMax && (size_t)L.P * 4 <= 32 * 1024;
}

extern "C" NSA_API size_t nsa_decode_workspace_bytes(const nsa_decode_desc* d) {
  return nsa_decode_supported(d) ? dec_layout(*d).total : 256;
}

extern "C" NSA_API int nsa_decode_fwd(const nsa_decode_desc* dp, void* workspace, size_t workspace_bytes, void* stream) {
  NSA_REQUIRE(dp, "decode_fwd: null descriptor");
  const nsa_decode_desc& d = *dp;
  if (timeout_flagged())
    return fail(NSA_ERR_LAUNCH, "decode_fwd: a tensor-core kernel gave up on a barrier wait earlier (device time-out); results since "
                "then are invalid.  nsa_device_timeouts(1) reports and clears the condition");
  if (!nsa_decode_supported(dp)) return fail(NSA_ERR_UNSUPPORTED, "decode_fwd: sizes outside this entry point's range (see nsa_decode_supported)");
  NSA_REQUIRE(d.k_slc && d.v_slc && d.k_win && d.v_win && d.k_cmp && d.v_cmp && d.out, "decode_fwd: null pointer");
  NSA_REQUIRE(al16(d.k_slc) && al16(d.v_slc) && al16(d.k_win) && al16(d.v_win) && al16(d.k_cmp) && al16(d.v_cmp) && al16(workspace),
              "decode_fwd: pointers must be 16-byte aligned");
  const DecLayout L = dec_layout(d);
  if (!workspace || workspace_bytes < L.total) return fail(NSA_ERR_WORKSPACE, "decode_fwd needs %zu workspace bytes, got %zu", L.total, workspace_bytes);
  cudaStream_t st = (cudaStream_t)stream;
  char* w = (char*)workspace;
  DecArgs a = {};
  NSA_REQUIRE(d.q && al16(d.q), "decode_fwd: null or misaligned q");
  NSA_REQUIRE(d.sq[0] % 8 == 0 && d.sq[1] % 8 == 0 && d.sq[2] % 8 == 0, "decode_fwd: q rows must start on 16-byte boundaries");
  a.q = (const __nv_bfloat16*)d.q;
  a.sqb = d.sq[0]; a.sqh = d.sq[1]; a.sqt = d.sq[2];
  if (d.project) {
    NSA_REQUIRE(d.x && al16(d.x) && d.gate_w1 && d.gate_w2 && al16(d.gate_w1) && al16(d.gate_w2) && d.k_src && d.v_src && d.k_new,
                "decode_fwd: projection inputs missing or not 16-byte aligned");
    NSA_REQUIRE(d.sx[0] % 8 == 0 && d.sx[1] % 8 == 0, "decode_fwd: x rows must start on 16-byte boundaries");
    NSA_REQUIRE(d.nb_new == 0 || (d.pos_embed && d.phi_w1 && d.phi_w2 && d.k_cmp_lp && d.block_ends), "decode_fwd: phi parameters missing");
    ProjArgs p = {};
    p.R = d.B * d.Tn; p.Tn = d.Tn; p.K = d.d_model; p.G = d.G; p.pos = d.pos; p.cap = d.cap;
    p.x = (const __nv_bfloat16*)d.x;
    p.sxb = d.sx[0]; p.sxt = d.sx[1];
    p.k_new = (const __nv_bfloat16*)d.k_new;
    for (int i = 0; i < 4; ++i) p.sk[i] = d.sk[i];
    int tile = 0;
    auto segment = [&](const void* wt, const void* bias, void* dst, int rows, int D, int kind) {
      p.seg[p.nseg++] = {(const __nv_bfloat16*)wt, (const __nv_bfloat16*)bias, (__nv_bfloat16*)dst, tile, D, kind};
      tile += rows / 16;
    };
    void* dst[5] = {d.k_slc, d.v_slc, d.v_src, d.k_win, d.v_win};
    for (int i = 0; i < 5; ++i) {
      NSA_REQUIRE(d.w[i] && al16(d.w[i]), "decode_fwd: projection weight missing or not 16-byte aligned");
      const bool key = i == 0 || i == 3;
      const int D = key ? d.dk : d.dv;
      segment(d.w[i], d.bias[i], dst[i], d.G * D, D, key ? kSegK : kSegV);
    }
    segment(d.gate_w1, d.gate_b1, w + L.o_gh, d.d_gate, d.d_gate, kSegGate);
    segment(nullptr, nullptr, d.k_src, d.G * d.dk, d.dk, kSegCopy);
    {
      KernelTimer kt("decode_project", st);
      if (int rc = launch_pdl("decode_project", decode_project_kernel, dim3(tile), kProjThreads, 0, st, p)) return rc;
    }
    if (d.nb_new > 0)
      if (int rc = compress_blocks(d, d.k_src, d.v_src, NSA_BF16, NSA_BF16, w + L.o_phi, st)) return rc;
    a.gh = (const __nv_bfloat16*)(w + L.o_gh); a.gw2 = (const __nv_bfloat16*)d.gate_w2; a.gb2 = (const __nv_bfloat16*)d.gate_b2; a.D2 = d.d_gate;
    a.logits = (float*)(w + L.o_logits);
  } else {
    NSA_REQUIRE(d.gate_logits, "decode_fwd: null gate logits");
    a.logits = const_cast<float*>(d.gate_logits);
  }
  a.k_slc = (const __nv_bfloat16*)d.k_slc; a.v_slc = (const __nv_bfloat16*)d.v_slc; a.k_win = (const __nv_bfloat16*)d.k_win;
  a.v_win = (const __nv_bfloat16*)d.v_win; a.v_cmp = (const __nv_bfloat16*)d.v_cmp; a.k_cmp = (const float*)d.k_cmp;
  a.cap = d.cap; a.nbp = d.nbp; a.B = d.B; a.H = d.H; a.G = d.G; a.Tn = d.Tn; a.hpg = d.H / d.G; a.nb = d.nb; a.pos = d.pos;
  a.window = d.window; a.l = d.l; a.d = d.d; a.n = d.n; a.n_fixed = d.n_fixed; a.s_ = d.l_prime / d.d; a.a_ = d.l / d.d;
  a.gate_mode = d.gate_mode; a.nc = L.nc; a.nw = L.nw; a.P = L.P; a.scale = d.scale;
  a.part_o = (float*)(w + L.o_part); a.part_st = (float2*)(w + L.o_st); a.slog = (float*)(w + L.o_slog);
  a.idx = d.indices ? d.indices : (int*)(w + L.o_idx);
  a.out = (__nv_bfloat16*)d.out; a.o_cmp = (__nv_bfloat16*)d.o_cmp; a.o_slc = (__nv_bfloat16*)d.o_slc; a.o_win = (__nv_bfloat16*)d.o_win;
  a.gates = d.gates;
  int rc;
  if (d.dk == 192) rc = launch_attend<192, 128>(a, d, L, st);
  else if (d.dk == 128) rc = launch_attend<128, 128>(a, d, L, st);
  else rc = launch_attend<64, 64>(a, d, L, st);
  return rc ? rc : check_launch("decode_fwd");
}
