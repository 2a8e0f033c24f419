// A handful of newest tokens against a key/value cache (decode): projections, cache update, block compression, Eq. 8-11
// block choice, the three attention branches and the gate mix, for up to 64 (sequence, group, token) rows.
//
// The tile kernels pad such a call to 128 query rows and need an inverse index, padded copies and one launch per piece:
// 45 launches and 760 us per token at B=1, 2K cached; 80 launches and 1400 us at B=8, 32K (91 and 138 us here).  What the work cannot do without
// is reading the weights once (131 MB for the 64-head configuration, 20 us) and the visible keys and values once, so here
// the keys of a row are cut into 64-key chunks, one CTA each, that serve all heads of the group, and everything between
// two grid-wide dependencies is one launch:
//   1 project     weights x tokens on mma.sync (8 tokens are one n tile; the weights stream through once), written straight
//                 into q and the caches; the gate MLP's hidden layer is one more row range
//   2 phi         only when the tokens complete compression blocks: fp32 sums over the bf16 weights
//   3 chunks      compressed and sliding-window chunks + the gate logits
//   4 top-n       Eq. 8-11 from the fp32 logits the chunks left
//   5 chunks      the selected blocks
//   6 combine     merge of the chunk partials, gates, mix
// Launches overlap their ramp-up by programmatic dependent launch.  Keys of the compressed blocks stay fp32 and their
// products run on the FMA pipe (they rank the blocks); bf16 keys and P V run on mma.sync, with P as bf16 hi + lo, so the
// probabilities keep 16 mantissa bits.  (tcgen05 tiles have 64 rows at least; a group has at most 16 heads.)
#include <algorithm>

#include "common.cuh"
#include "fa_sm100.cuh"

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
enum { kSegQ = 0, kSegK, kSegV, kSegGate };
struct ProjSeg {
  const __nv_bfloat16 *w, *bias;
  __nv_bfloat16* dst;
  int tile0, D, kind;    // first tile of the segment, head dim (width for the gate), layout
};
struct ProjArgs {
  ProjSeg seg[8];
  int nseg, R, Tn, K, H, G, pos;
  int64_t cap, sxb, sxt;
  const __nv_bfloat16* x;
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
  const int n = threadIdx.x >> 4, r = threadIdx.x & 15, row = row0 + r;
  if (n >= p.R) return;
  const float y = (red[0][r][n] + red[1][r][n]) + (red[2][r][n] + red[3][r][n]);
  __nv_bfloat16 o = __float2bfloat16_rn(y);
  if (sg.bias) o = __float2bfloat16_rn(__bfloat162float(o) + __bfloat162float(sg.bias[row]));
  const int b = n / p.Tn, t = n % p.Tn, hd = row / sg.D, e = row % sg.D;
  if (sg.kind == kSegQ) sg.dst[(((int64_t)b * p.H + hd) * p.Tn + t) * sg.D + e] = o;
  else if (sg.kind == kSegK) sg.dst[(((int64_t)b * p.G + hd) * sg.D + e) * p.cap + p.pos + t] = o;
  else if (sg.kind == kSegV) sg.dst[(((int64_t)b * p.G + hd) * p.cap + p.pos + t) * sg.D + e] = o;
  else sg.dst[(int64_t)n * sg.D + row] = __bfloat162float(o) > 0.f ? o : __float2bfloat16_rn(0.f);
}

// ------------------------------------------------------------------------------------------------ block compression
// hbar[u] = mean_j relu(b1[u] + W1[u] . [k_{id+j} || pos_j]) of one new block: 64 hidden units a CTA, four threads a unit
// with 8 offsets each; the 32 inputs sit in shared memory as fp32, offsets contiguous.
struct PhiArgs {
  const __nv_bfloat16 *k, *v, *pos, *w1, *b1, *w2, *b2;
  float *hbar, *k_cmp;
  __nv_bfloat16 *k_lp, *v_cmp;
  int32_t* block_ends;
  int64_t cap, nbp;
  int dk, dv, U, l, d, blk0;
};
__global__ void __launch_bounds__(256) decode_phi_hidden_kernel(const __grid_constant__ PhiArgs p) {
  extern __shared__ __align__(16) float z[];     // [dk + l][32]
  pdl_wait();
  pdl_launch();
  const int bg = blockIdx.z, blk = p.blk0 + blockIdx.y, W = p.dk + p.l;
  const __nv_bfloat16* k = p.k + (int64_t)bg * p.dk * p.cap + (int64_t)blk * p.d;
  for (int i = threadIdx.x; i < W * 32; i += 256) {
    const int cidx = i >> 5, j = i & 31;
    z[i] = j >= p.l ? 0.f : __bfloat162float(cidx < p.dk ? k[(int64_t)cidx * p.cap + j] : p.pos[j * p.l + cidx - p.dk]);
  }
  __syncthreads();
  const int u = blockIdx.x * 64 + (threadIdx.x >> 2), jg = threadIdx.x & 3;
  float sum = 0.f;
  if (u < p.U) {
    float acc[8];
    const float b = p.b1 ? __bfloat162float(p.b1[u]) : 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = b;
    const __nv_bfloat16* w = p.w1 + (int64_t)u * W;
    for (int c0 = 0; c0 < W; c0 += 8) {
      const uint4 wv = *reinterpret_cast<const uint4*>(w + c0);
      const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&wv);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float wf = (e & 1) ? __high2float(w2[e >> 1]) : __low2float(w2[e >> 1]);
        const float4 z0 = *reinterpret_cast<const float4*>(z + (c0 + e) * 32 + jg * 8);
        const float4 z1 = *reinterpret_cast<const float4*>(z + (c0 + e) * 32 + jg * 8 + 4);
        acc[0] = fmaf(wf, z0.x, acc[0]); acc[1] = fmaf(wf, z0.y, acc[1]); acc[2] = fmaf(wf, z0.z, acc[2]); acc[3] = fmaf(wf, z0.w, acc[3]);
        acc[4] = fmaf(wf, z1.x, acc[4]); acc[5] = fmaf(wf, z1.y, acc[5]); acc[6] = fmaf(wf, z1.z, acc[6]); acc[7] = fmaf(wf, z1.w, acc[7]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (jg * 8 + i < p.l) sum += fmaxf(acc[i], 0.f);
  }
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);
  sum += __shfl_xor_sync(0xffffffffu, sum, 2);
  if (jg == 0 && u < p.U) p.hbar[((int64_t)bg * gridDim.y + blockIdx.y) * p.U + u] = sum / (float)p.l;
}
__global__ void __launch_bounds__(256) decode_phi_out_kernel(const __grid_constant__ PhiArgs p) {
  pdl_wait();
  pdl_launch();
  const int bg = blockIdx.z, blk = p.blk0 + blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* hb = p.hbar + ((int64_t)bg * gridDim.y + blockIdx.y) * p.U;
  for (int c = blockIdx.x * 8 + warp; c < p.dk; c += gridDim.x * 8) {
    float s = 0.f;
    for (int u = lane; u < p.U; u += 32) s = fmaf(__bfloat162float(p.w2[(int64_t)c * p.U + u]), hb[u], s);
    s = warp_sum(s);
    if (lane == 0) {
      if (p.b2) s += __bfloat162float(p.b2[c]);
      const int64_t o = ((int64_t)bg * p.dk + c) * p.nbp + blk;
      p.k_cmp[o] = s;
      p.k_lp[o] = __float2bfloat16_rn(s);
    }
  }
  if (blockIdx.x == 0) {
    for (int c = threadIdx.x; c < p.dv; c += 256) {
      float s = 0.f;
#pragma unroll 8
      for (int j = 0; j < p.l; ++j) s += __bfloat162float(p.v[((int64_t)bg * p.cap + (int64_t)blk * p.d + j) * p.dv + c]);
      p.v_cmp[((int64_t)bg * p.nbp + blk) * p.dv + c] = __float2bfloat16_rn(s / (float)p.l);
    }
    if (bg == 0 && threadIdx.x == 0) p.block_ends[blk] = blk * p.d + p.l - 1;
  }
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

template <int DK, int DV>
struct DecSmem {
  static constexpr int kQ = 16 * (DK + 8) * 2;       // bf16 queries (rows 16 bytes off a bank period)
  static constexpr int kK = DK * 72 * 2;             // bf16 key tile [DK][64]; compressed: fp32 queries [DK][16] + partial sums
  static constexpr int kC = DK * 16 * 4 + 4 * 16 * 64 * 4;
  static constexpr int kKC = kK > kC ? kK : kC;
  static constexpr int kV = 64 * (DV + 8) * 2;
  static constexpr int kS = 16 * 66 * 4;
  static constexpr int kP = 2 * 16 * 72 * 2;
  static constexpr int oQ = 0, oK = oQ + kQ, oV = oK + kKC, oS = oV + kV, oP = oS + kS, kBytes = oP + kP;
};

// One chunk of 64 keys [key0, key0 + 64) for the heads of a group: S, its softmax over the chunk, P V.  Keys klo <= key < khi
// count.  CMP: fp32 keys [DK][ld], whose logits are also kept for the block choice.
template <int DK, int DV, bool CMP>
__device__ __forceinline__ void attend_chunk(const DecArgs& p, uint8_t* sm, int row, int chunk, const void* kbase, const __nv_bfloat16* vbase,
                                             int64_t ld, int key0, int klo, int khi, int b, int h0, int tn) {
  using SM = DecSmem<DK, DV>;
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
    float* part = qf + DK * 16;                 // [4][16][64]
    for (int i = tid; i < DK * 16; i += kDecThreads) {
      const int r = i / DK, dd = i % DK;
      qf[dd * 16 + r] = r < p.hpg ? __bfloat162float(qb[r * p.sqh + dd]) : 0.f;
    }
    __syncthreads();
    const int key = tid & 63, quarter = tid >> 6;
    const bool in = key0 + key < khi;
    const float* kp = (const float*)kbase + (int64_t)quarter * (DK / 4) * ld + key0 + key;
    float acc[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) acc[u] = 0.f;
#pragma unroll
    for (int d0 = 0; d0 < DK / 4; d0 += 16) {
      float kv[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) kv[e] = in ? kp[(int64_t)(d0 + e) * ld] : 0.f;
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float4* q4 = reinterpret_cast<const float4*>(qf + (quarter * (DK / 4) + d0 + e) * 16);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 qv = q4[u];
          acc[4 * u] = fmaf(qv.x, kv[e], acc[4 * u]);         acc[4 * u + 1] = fmaf(qv.y, kv[e], acc[4 * u + 1]);
          acc[4 * u + 2] = fmaf(qv.z, kv[e], acc[4 * u + 2]); acc[4 * u + 3] = fmaf(qv.w, kv[e], acc[4 * u + 3]);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) part[(quarter * 16 + u) * 64 + key] = acc[u];
    __syncthreads();
    float* lg = p.slog + (int64_t)row * 16 * (p.nc * 64) + chunk * 64;
    for (int i = tid; i < p.hpg * 64; i += kDecThreads) {
      const int u = i >> 6, kk = i & 63;
      const float s = (part[u * 64 + kk] + part[(16 + u) * 64 + kk]) + (part[(32 + u) * 64 + kk] + part[(48 + u) * 64 + kk]);
      const float x = key0 + kk < khi ? s * p.scale : -CUDART_INF_F;
      sS[u * 66 + kk] = x;
      lg[(int64_t)u * (p.nc * 64) + kk] = x;
    }
    for (int i = p.hpg * 64 + tid; i < 16 * 64; i += kDecThreads) sS[(i >> 6) * 66 + (i & 63)] = -CUDART_INF_F;
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
    attend_chunk<DK, DV, true>(p, dsm, row, chunk, p.k_cmp + (int64_t)bg * DK * p.nbp, p.v_cmp + (int64_t)bg * p.nbp * DV, p.nbp,
                               chunk * 64, 0, vis, b, h0, tn);
  } else {
    const int klo = max(0, t - p.window + 1), key0 = (klo / 64 + chunk - p.nc) * 64;
    if (key0 > t) { empty_chunk(p, row, chunk); return; }
    attend_chunk<DK, DV, false>(p, dsm, row, chunk, p.k_win + (int64_t)bg * DK * p.cap, p.v_win + (int64_t)bg * p.cap * DV, p.cap, key0,
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
  attend_chunk<DK, DV, false>(p, dsm, row, p.nc + p.nw + slot, p.k_slc + (int64_t)bg * DK * p.cap, p.v_slc + (int64_t)bg * p.cap * DV,
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
// One CTA per row: softmax statistics of the heads from the chunks', Eq. 9 sums per selection block summed over the heads in
// order, then the top n: each warp of its share, one warp of the survivors.
__global__ void __launch_bounds__(kTopWarps * 32) decode_topn_kernel(const __grid_constant__ DecArgs p, int n_sel, int n_eff) {
  extern __shared__ __align__(16) unsigned long long keys[];   // [n_eff], then [kTopWarps * n]
  unsigned long long* cand = keys + n_eff;
  __shared__ float hm[16], hinv[16];
  __shared__ unsigned long long top[kDecMaxN];
  pdl_wait();
  pdl_launch();
  const int row = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = p.pos + row % p.Tn;
  if (warp < p.hpg) {
    const float2* st = p.part_st + (int64_t)row * p.P * 16 + warp;
    float m = -CUDART_INF_F;
    for (int c = lane; c < p.nc; c += 32) m = fmaxf(m, st[c * 16].x);
    m = warp_max(m);
    float s = 0.f;
    for (int c = lane; c < p.nc; c += 32) {
      const float2 v = st[c * 16];
      if (v.y != 0.f) s += v.y * expf(v.x - m);
    }
    s = warp_sum(s);
    if (lane == 0) { hm[warp] = m; hinv[warp] = s != 0.f ? 1.f / s : 0.f; }
  }
  __syncthreads();
  const int ncol = p.nc * 64;
  const float* lg = p.slog + (int64_t)row * 16 * ncol;
  for (int j = threadIdx.x; j < n_eff; j += kTopWarps * 32) {
    float agg = 0.f;
    for (int h = 0; h < p.hpg; ++h) {
      const float m = hm[h], inv = hinv[h];
      float sel = 0.f;
      if (m == -CUDART_INF_F) {            // nothing visible: block 0 alone (nsa/kernels.py:2316-2343)
        for (int mm = 0; mm < p.s_; ++mm)
          for (int nn = 0; nn < p.a_; ++nn) sel += p.s_ * j + mm + nn == 0 ? 1.f : 0.f;
      } else {
        const float* lh = lg + (int64_t)h * ncol;
        for (int i = 0; i < p.s_ + p.a_ - 1; ++i) {
          const int c = p.s_ * j + i;
          // block c is counted once per (m, n) with m + n = i, m < s, n < a
          const int times = min(min(i + 1, p.s_ + p.a_ - 1 - i), min(p.s_, p.a_));
          if (c < ncol) sel = fmaf((float)times, expf(lh[c] - m) * inv, sel);
        }
      }
      agg += sel;
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
  size_t o_q, o_gh, o_logits, o_hbar, o_part, o_st, o_slog, o_idx, total;
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
  L.o_q = take(R * d.H * d.dk * 2);
  L.o_gh = take(R * d.d_gate * 2);
  L.o_logits = take(R * 3 * d.H * 4);
  L.o_hbar = take((size_t)d.B * d.G * std::max(d.nb_new, 0) * d.U * 4);
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
  constexpr int kBytes = DecSmem<DK, DV>::kBytes;
  cudaFuncSetAttribute(decode_dense_kernel<DK, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  cudaFuncSetAttribute(decode_selected_kernel<DK, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  {
    KernelTimer kt("decode_dense", st);
    const int gate_ctas = a.gh ? (3 * d.H + 7) / 8 : 0;
    if (int rc = launch_pdl("decode_dense", decode_dense_kernel<DK, DV>, dim3(L.rows * (L.nc + L.nw) + gate_ctas), kDecThreads, kBytes, st, a)) return rc;
  }
  {
    KernelTimer kt("decode_topn", st);
    const size_t sm = topn_smem(d, L);
    if (sm > 40 * 1024) cudaFuncSetAttribute(decode_topn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (int rc = launch_pdl("decode_topn", decode_topn_kernel, dim3(L.rows), kTopWarps * 32, sm, st, a, L.n_sel, L.n_eff)) return rc;
  }
  {
    KernelTimer kt("decode_selected", st);
    if (int rc = launch_pdl("decode_selected", decode_selected_kernel<DK, DV>, dim3(d.n, L.rows), kDecThreads, kBytes, st, a)) return rc;
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
    if (d.nb_new < 0 || d.nb_new > d.nb || (d.nb_new > 0 && (d.U <= 0 || d.l > 32 || (d.dk + d.l) % 8 != 0))) return 0;
    if (d.nb_new > 65535) return 0;
  }
  const DecLayout L = dec_layout(d);
  return topn_smem(d, L) <= 200 * 1024 && (size_t)L.P * 4 <= 32 * 1024;
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
  if (d.project) {
    NSA_REQUIRE(d.x && al16(d.x) && d.gate_w1 && d.gate_w2 && al16(d.gate_w1) && al16(d.gate_w2) && d.k_src && d.v_src,
                "decode_fwd: projection inputs missing or not 16-byte aligned");
    NSA_REQUIRE(d.sx[0] % 8 == 0 && d.sx[1] % 8 == 0, "decode_fwd: x rows must start on 16-byte boundaries");
    ProjArgs p = {};
    p.R = d.B * d.Tn; p.Tn = d.Tn; p.K = d.d_model; p.H = d.H; p.G = d.G; p.pos = d.pos; p.cap = d.cap;
    p.x = (const __nv_bfloat16*)d.x;
    p.sxb = d.sx[0]; p.sxt = d.sx[1];
    void* dst[7] = {w + L.o_q, d.k_slc, d.v_slc, d.k_src, d.v_src, d.k_win, d.v_win};
    int tile = 0;
    for (int i = 0; i < 7; ++i) {
      NSA_REQUIRE(d.w[i] && al16(d.w[i]), "decode_fwd: projection weight missing or not 16-byte aligned");
      const bool key = i == 0 || (i & 1);
      ProjSeg& s = p.seg[i];
      s.w = (const __nv_bfloat16*)d.w[i]; s.bias = (const __nv_bfloat16*)d.bias[i]; s.dst = (__nv_bfloat16*)dst[i];
      s.D = key ? d.dk : d.dv; s.kind = i == 0 ? kSegQ : key ? kSegK : kSegV; s.tile0 = tile;
      tile += (i == 0 ? d.H : d.G) * s.D / 16;
    }
    ProjSeg& s = p.seg[7];
    s.w = (const __nv_bfloat16*)d.gate_w1; s.bias = (const __nv_bfloat16*)d.gate_b1; s.dst = (__nv_bfloat16*)(w + L.o_gh);
    s.D = d.d_gate; s.kind = kSegGate; s.tile0 = tile;
    tile += d.d_gate / 16;
    p.nseg = 8;
    {
      KernelTimer kt("decode_project", st);
      if (int rc = launch_pdl("decode_project", decode_project_kernel, dim3(tile), kProjThreads, 0, st, p)) return rc;
    }
    if (d.nb_new > 0) {
      NSA_REQUIRE(d.pos_embed && d.phi_w1 && d.phi_w2 && d.k_cmp_lp && d.block_ends && al16(d.phi_w1), "decode_fwd: phi parameters missing");
      KernelTimer kt("decode_phi", st);
      PhiArgs f = {};
      f.k = (const __nv_bfloat16*)d.k_src; f.v = (const __nv_bfloat16*)d.v_src; f.pos = (const __nv_bfloat16*)d.pos_embed;
      f.w1 = (const __nv_bfloat16*)d.phi_w1; f.b1 = (const __nv_bfloat16*)d.phi_b1; f.w2 = (const __nv_bfloat16*)d.phi_w2; f.b2 = (const __nv_bfloat16*)d.phi_b2;
      f.hbar = (float*)(w + L.o_hbar); f.k_cmp = (float*)d.k_cmp; f.k_lp = (__nv_bfloat16*)d.k_cmp_lp; f.v_cmp = (__nv_bfloat16*)d.v_cmp;
      f.block_ends = d.block_ends; f.cap = d.cap; f.nbp = d.nbp; f.dk = d.dk; f.dv = d.dv; f.U = d.U; f.l = d.l; f.d = d.d; f.blk0 = d.nb - d.nb_new;
      if (int rc = launch_pdl("decode_phi", decode_phi_hidden_kernel, dim3((d.U + 63) / 64, d.nb_new, d.B * d.G), 256, (size_t)(d.dk + d.l) * 32 * 4, st, f)) return rc;
      if (int rc = launch_pdl("decode_phi", decode_phi_out_kernel, dim3(6, d.nb_new, d.B * d.G), 256, 0, st, f)) return rc;
    }
    a.q = (const __nv_bfloat16*)(w + L.o_q);
    a.sqb = (int64_t)d.H * d.Tn * d.dk; a.sqh = (int64_t)d.Tn * d.dk; a.sqt = d.dk;
    a.gh = (const __nv_bfloat16*)(w + L.o_gh); a.gw2 = (const __nv_bfloat16*)d.gate_w2; a.gb2 = (const __nv_bfloat16*)d.gate_b2; a.D2 = d.d_gate;
    a.logits = (float*)(w + L.o_logits);
  } else {
    NSA_REQUIRE(d.q && al16(d.q) && d.gate_logits, "decode_fwd: null or misaligned q / gate logits");
    NSA_REQUIRE(d.sq[0] % 8 == 0 && d.sq[1] % 8 == 0 && d.sq[2] % 8 == 0, "decode_fwd: q rows must start on 16-byte boundaries");
    a.q = (const __nv_bfloat16*)d.q;
    a.sqb = d.sq[0]; a.sqh = d.sq[1]; a.sqt = d.sq[2];
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
