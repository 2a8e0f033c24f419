// Chunks of new tokens against a key/value cache (chunked prefill), behind two C entry points: the append (strided copies into
// the caches as one launch, block compression straight from and into them) and the layer's forward for the new rows with a
// query position offset.  The tensor-core kernels read the caches where they lie and take any row count, so nothing is
// padded, sliced or copied on the way.  (Composed from tensor operations, a chunk of 512 tokens at 7000 cached took 69
// launches and 1.23 ms of host time for 0.60 ms of kernels.)  Handfuls of rows go through decode_sm100.cu instead.
#include <algorithm>

#include "attn_args.cuh"
#include "common.cuh"
#include "fa_sm100.cuh"
#include "phi.cuh"
#include "slc_sm100.cuh"

namespace nsa {
namespace {

size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// ------------------------------------------------------------------------------------------------ append
struct CopyArgs {
  const void* src[6];
  void* dst[6];
  int64_t ss[6][4];     // strides of the source: batch, group, time, channel
  int B, G, Tn, dk, dv, pos;
  int64_t cap;
};
// Keys go to [B,G,dk,cap] (time contiguous), values to [B,G,cap,dv], 32 x 32 tiles through shared memory: reads follow the
// source's smaller stride, writes the destination's.  blockIdx.z = tensor * B*G + (batch, group).
template <typename T>
__global__ void __launch_bounds__(256) append_kernel(const __grid_constant__ CopyArgs a) {
  __shared__ T tile[32][33];
  const int i = blockIdx.z / (a.B * a.G), bg = blockIdx.z % (a.B * a.G), b = bg / a.G, g = bg % a.G;
  const bool key = (i & 1) == 0;
  const int D = key ? a.dk : a.dv, t0 = blockIdx.x * 32, c0 = blockIdx.y * 32, x = threadIdx.x & 31;
  if (c0 >= D) return;
  const T* src = (const T*)a.src[i] + b * a.ss[i][0] + g * a.ss[i][1];
  T* dst = (T*)a.dst[i] + (int64_t)bg * D * a.cap;
  const int64_t st = a.ss[i][2], sc = a.ss[i][3];
  const bool along_t = st < sc;
#pragma unroll
  for (int y = threadIdx.x >> 5; y < 32; y += 8) {
    const int t = along_t ? x : y, c = along_t ? y : x;
    if (t0 + t < a.Tn && c0 + c < D) tile[t][c] = src[(t0 + t) * st + (c0 + c) * sc];
  }
  __syncthreads();
#pragma unroll
  for (int y = threadIdx.x >> 5; y < 32; y += 8) {
    const int t = key ? x : y, c = key ? y : x;
    if (t0 + t < a.Tn && c0 + c < D)
      dst[key ? (int64_t)(c0 + c) * a.cap + a.pos + t0 + t : (int64_t)(a.pos + t0 + t) * D + c0 + c] = tile[t][c];
  }
}
__global__ void append_block_ends_kernel(int32_t* be, int b0, int n, int l, int d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) be[b0 + i] = (b0 + i) * d + l - 1;
}
struct CastArgs {
  const __nv_bfloat16* in[5];
  float* out[5];
  int n[5];
};
__global__ void cast_params_kernel(const __grid_constant__ CastArgs a) {
  for (int k = 0; k < 5; ++k)
    if (a.in[k])
      for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n[k]; i += gridDim.x * blockDim.x) a.out[k][i] = __bfloat162float(a.in[k][i]);
}

struct AppendLayout {
  int T, lo;                // tokens the new blocks cover, the first of them
  size_t o_par[5], o_saved, saved, o_ws, ws, o_kc, total;
};
AppendLayout append_layout(const nsa_decode_desc& d, int dtype) {
  AppendLayout L = {};
  L.lo = (d.nb - d.nb_new) * d.d;
  L.T = d.nb_new > 0 ? (d.nb_new - 1) * d.d + d.l : 0;
  size_t o = 0;
  auto take = [&](size_t n) { const size_t r = o; o += al256(n); return r; };
  if (d.nb_new > 0) {
    const size_t n[5] = {(size_t)d.l * d.l, (size_t)d.U * (d.dk + d.l), (size_t)d.U, (size_t)d.dk * d.U, (size_t)d.dk};
    for (int i = 0; i < 5; ++i) L.o_par[i] = take(n[i] * 4);
    L.saved = nsa_cmp_phi_saved_bytes(d.B, d.G, L.T, d.l, d.d, d.U);
    L.o_saved = take(L.saved);
    L.ws = nsa_cmp_phi_workspace_bytes(d.B, d.G, L.T, d.dk, d.dv, d.l, d.d, d.U, d.nbp, dtype, 0);
    L.o_ws = take(L.ws);
    int nbq = 1;
    while (nbq < d.nb_new) nbq *= 2;
    L.o_kc = take((size_t)d.B * d.G * d.dk * nbq * 4);
  }
  L.total = std::max<size_t>(o, 256);
  return L;
}
int check_cache(const char* who, const nsa_decode_desc& d) {
  NSA_REQUIRE(d.B > 0 && d.G > 0 && d.H > 0 && d.H % d.G == 0 && d.Tn > 0 && d.dk > 0 && d.dv > 0, "%s: bad sizes", who);
  NSA_REQUIRE(d.l > 0 && d.d > 0 && d.l % d.d == 0 && d.l_prime > 0 && d.l_prime % d.d == 0, "%s: bad block sizes", who);
  NSA_REQUIRE(d.pos >= 0 && (int64_t)d.pos + d.Tn <= d.cap && d.nb >= 0 && d.nb <= d.nbp, "%s: positions or blocks outside the cache", who);
  return NSA_OK;
}

// ------------------------------------------------------------------------------------------------ forward
// rows whose slots are all empty attend the block holding the query (nsa/kernels.py:199-205)
__global__ void fallback_kernel(int32_t* idx, int64_t rows, int T, int n, int lprime, int pos) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  int32_t* row = idx + r * n;
  bool any = false;
  for (int s = 0; s < n; ++s) any |= row[s] >= 0;
  if (!any) row[0] = ((int32_t)(r % T) + pos) / lprime;
}
struct ChunkLayout {
  int Tk, ld;
  size_t o_hi, o_lo, o_lse, o_L, o_M, o_cmp, o_slc, o_win, o_gates, o_idx, o_stage, stage, total;
};
// `sums`: with the scratch for the block choice from the forward's own sums; without it the scoring kernel makes the choice
ChunkLayout chunk_layout(const nsa_decode_desc& d, bool sums) {
  ChunkLayout L;
  const size_t BG = (size_t)d.B * d.G, R = (size_t)d.B * d.H * d.Tn;
  L.Tk = d.pos + d.Tn;
  L.ld = (d.nbp + 127) / 128 * 128;
  size_t o = 0;
  auto take = [&](size_t n) { const size_t r = o; o += al256(n); return r; };
  L.o_hi = take(BG * d.dk * L.ld * 2);
  L.o_lo = take(BG * d.dk * L.ld * 2);
  L.o_lse = take(R * 4);
  L.o_L = take(R * 4);
  L.o_M = take(R * 4);
  L.o_cmp = take(R * d.dv * 2);
  L.o_slc = take(R * d.dv * 2);
  L.o_win = take(R * d.dv * 2);
  L.o_gates = take(R * 3 * 4);
  L.o_idx = take(BG * d.Tn * d.n * 4);
  L.stage = std::max(sums ? nsa_cmp_attn_topn_workspace_bytes(d.B, d.H, d.G, d.Tn, d.nbp, d.dk, d.dv, d.l, d.d, d.l_prime, d.n, d.nb, NSA_FLAG_ANY_LENGTH)
                          : nsa_score_topn_workspace_bytes(d.B, d.H, d.G, d.Tn, d.dk, d.nbp, d.l, d.d, d.l_prime, d.n, NSA_BF16, NSA_FLAG_ANY_LENGTH),
                     nsa_slc_fwd_workspace_bytes(d.B, d.H, d.G, d.Tn, L.Tk, d.dk, d.dv, d.n, d.l_prime, NSA_BF16, NSA_FLAG_ANY_LENGTH));
  L.o_stage = take(L.stage);
  L.total = o;
  return L;
}
bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

size_t compress_blocks_workspace_bytes(const nsa_decode_desc& d, int dtype) { return append_layout(d, dtype).total; }

int compress_blocks(const nsa_decode_desc& d, const void* k, const void* v, int dtype, int param_dtype, void* workspace, cudaStream_t st) {
  const AppendLayout L = append_layout(d, dtype);
  char* w = (char*)workspace;
  const void* in[5] = {d.pos_embed, d.phi_w1, d.phi_b1, d.phi_w2, d.phi_b2};
  const float* par[5];
  for (int i = 0; i < 5; ++i) par[i] = (const float*)in[i];
  if (param_dtype == NSA_BF16) {
    CastArgs c = {};
    const int n[5] = {d.l * d.l, d.U * (d.dk + d.l), d.U, d.dk * d.U, d.dk};
    for (int i = 0; i < 5; ++i) {
      c.in[i] = (const __nv_bfloat16*)in[i];
      c.out[i] = (float*)(w + L.o_par[i]);
      c.n[i] = n[i];
      par[i] = in[i] ? c.out[i] : nullptr;
    }
    cast_params_kernel<<<148, 256, 0, st>>>(c);
  }
  const size_t es = dtype == NSA_BF16 ? 2 : 4;
  const int b0 = d.nb - d.nb_new;
  append_block_ends_kernel<<<(d.nb_new + 255) / 256, 256, 0, st>>>(d.block_ends, b0, d.nb_new, d.l, d.d);
  const char *ks = (const char*)k + (size_t)L.lo * es, *vs = (const char*)v + (size_t)L.lo * d.dv * es;
  const int64_t vst[4] = {(int64_t)d.G * d.cap * d.dv, (int64_t)d.cap * d.dv, d.dv, 1};
  return cmp_phi_fwd_strided(ks, d.cap, (int64_t)d.dk * d.cap, vs, vst, par[0], par[1], par[2], par[3], par[4], (float*)d.k_cmp + b0,
                             d.k_cmp_lp ? (char*)d.k_cmp_lp + b0 * es : nullptr, (char*)d.v_cmp + (size_t)b0 * d.dv * es, d.B, d.G, L.T, L.T, d.dk,
                             d.dv, d.l, d.d, d.U, d.nbp, (float*)(w + L.o_kc), dtype, w + L.o_saved, L.saved, w + L.o_ws, L.ws, st);
}

}  // namespace nsa

using namespace nsa;

extern "C" NSA_API size_t nsa_cache_append_workspace_bytes(const nsa_decode_desc* d, int dtype) {
  if (!d || check_cache("cache_append", *d) || d->nb_new < 0 || d->nb_new > d->nb) return 256;
  return append_layout(*d, dtype).total;
}

extern "C" NSA_API int nsa_cache_append(const nsa_decode_desc* dp, const void* const* src, const int64_t* strides, int n_tensors, int dtype,
                                        int param_dtype, void* workspace, size_t workspace_bytes, void* stream) {
  NSA_REQUIRE(dp && src && strides, "cache_append: null pointer");
  const nsa_decode_desc& d = *dp;
  if (int rc = check_cache("cache_append", d)) return rc;
  NSA_REQUIRE(dtype == NSA_F32 || dtype == NSA_BF16, "cache_append: unsupported dtype %d", dtype);
  NSA_REQUIRE(param_dtype == NSA_F32 || param_dtype == NSA_BF16, "cache_append: unsupported parameter dtype %d", param_dtype);
  NSA_REQUIRE(n_tensors == 2 || n_tensors == 6, "cache_append: one or three key/value pairs");
  NSA_REQUIRE(d.nb_new >= 0 && d.nb_new <= d.nb, "cache_append: bad block count");
  NSA_REQUIRE((int64_t)d.B * d.G * n_tensors <= 65535, "cache_append: too many planes");
  const AppendLayout L = append_layout(d, dtype);
  if (d.nb_new > 0) {
    NSA_REQUIRE(d.pos_embed && d.phi_w1 && d.phi_w2 && d.k_cmp && d.v_cmp && d.block_ends && d.U > 0, "cache_append: phi parameters missing");
    NSA_REQUIRE(L.lo + L.T <= d.pos + d.Tn, "cache_append: the new blocks reach past the last token");
    if (!workspace || workspace_bytes < L.total) return fail(NSA_ERR_WORKSPACE, "cache_append needs %zu workspace bytes, got %zu", L.total, workspace_bytes);
  }
  cudaStream_t st = (cudaStream_t)stream;
  CopyArgs a = {};
  void* dst[6] = {d.k_slc, d.v_slc, d.k_src, d.v_src, d.k_win, d.v_win};
  for (int i = 0; i < n_tensors; ++i) {
    NSA_REQUIRE(src[i] && dst[i], "cache_append: null pointer");
    a.src[i] = src[i];
    a.dst[i] = dst[i];
    for (int j = 0; j < 4; ++j) a.ss[i][j] = strides[4 * i + j];
  }
  a.B = d.B; a.G = d.G; a.Tn = d.Tn; a.dk = d.dk; a.dv = d.dv; a.pos = d.pos; a.cap = d.cap;
  {
    KernelTimer kt("cache_append", st);
    const dim3 grid((d.Tn + 31) / 32, (std::max(d.dk, d.dv) + 31) / 32, n_tensors * d.B * d.G);
    if (dtype == NSA_BF16) append_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(a);
    else append_kernel<float><<<grid, 256, 0, st>>>(a);
  }
  if (int rc = check_launch("cache_append")) return rc;
  if (d.nb_new == 0) return NSA_OK;
  return compress_blocks(d, n_tensors == 2 ? d.k_slc : d.k_src, n_tensors == 2 ? d.v_slc : d.v_src, dtype, param_dtype, workspace, st);
}

extern "C" NSA_API int nsa_incremental_supported(const nsa_decode_desc* dp) {
  if (!dp || check_cache("incremental", *dp)) return 0;
  const nsa_decode_desc& d = *dp;
  if (d.nb <= 0 || d.cap % 8 != 0 || d.n <= 0 || d.n_fixed < 0 || d.window <= 0 || (int64_t)d.B * d.H > 65535) return 0;
  if ((int64_t)d.B * d.G * d.Tn <= 64) return 0;      // (the scoring would take its few-rows form: decode_sm100.cu serves these)
  return fa_fwd_sm100_supported(d.H, d.G, d.Tn, d.nbp, d.dk, d.dv) &&
         score_sm100_supported(d.H, d.G, d.Tn, d.dk, d.nbp, d.l, d.d, d.l_prime, d.n) &&
         slc_sm100_supported(d.H, d.G, d.Tn, d.pos + d.Tn, d.dk, d.dv, d.n, d.l_prime);
}

extern "C" NSA_API size_t nsa_incremental_workspace_bytes(const nsa_decode_desc* d) {
  return nsa_incremental_supported(d) ? chunk_layout(*d, true).total : 256;
}

extern "C" NSA_API size_t nsa_incremental_workspace_min_bytes(const nsa_decode_desc* d) {
  return nsa_incremental_supported(d) ? chunk_layout(*d, false).total : 256;
}

extern "C" NSA_API int nsa_incremental_fwd(const nsa_decode_desc* dp, void* workspace, size_t workspace_bytes, void* stream) {
  NSA_REQUIRE(dp, "incremental_fwd: null descriptor");
  const nsa_decode_desc& d = *dp;
  if (!nsa_incremental_supported(dp)) return fail(NSA_ERR_UNSUPPORTED, "incremental_fwd: sizes outside this entry point's range (see nsa_incremental_supported)");
  NSA_REQUIRE(d.q && d.gate_logits && d.k_slc && d.v_slc && d.k_win && d.v_win && d.k_cmp && d.v_cmp && d.block_ends && d.out,
              "incremental_fwd: null pointer");
  NSA_REQUIRE(al16(d.q) && al16(d.k_slc) && al16(d.v_slc) && al16(d.k_win) && al16(d.v_win) && al16(d.v_cmp) && al16(d.out) && al16(workspace),
              "incremental_fwd: pointers must be 16-byte aligned");
  const int64_t H = d.H, G = d.G, T = d.Tn, dk = d.dk, dv = d.dv;
  NSA_REQUIRE(d.sq[0] == H * T * dk && d.sq[1] == T * dk && d.sq[2] == dk, "incremental_fwd: q must be contiguous");
  if (timeout_flagged())
    return fail(NSA_ERR_LAUNCH, "incremental_fwd: a tensor-core kernel gave up on a barrier wait earlier (device time-out); results since "
                "then are invalid.  nsa_device_timeouts(1) reports and clears the condition");
  ChunkLayout L = chunk_layout(d, true);
  if (workspace_bytes < L.total) L = chunk_layout(d, false);
  if (!workspace || workspace_bytes < L.total) return fail(NSA_ERR_WORKSPACE, "incremental_fwd needs %zu workspace bytes, got %zu", L.total, workspace_bytes);
  cudaStream_t st = (cudaStream_t)stream;
  char* w = (char*)workspace;
  void *hi = w + L.o_hi, *lo = w + L.o_lo;
  void *o_cmp = d.o_cmp ? d.o_cmp : w + L.o_cmp, *o_slc = d.o_slc ? d.o_slc : w + L.o_slc, *o_win = d.o_win ? d.o_win : w + L.o_win;
  float *lse2 = (float*)(w + L.o_lse), *Ls = (float*)(w + L.o_L), *Ms = (float*)(w + L.o_M);
  float* gates = d.gates ? d.gates : (float*)(w + L.o_gates);
  int32_t* idx = d.indices ? d.indices : (int32_t*)(w + L.o_idx);
  // strides of one branch call: q, keys with rows ld apart, values with planes `plane` apart, output, statistics, indices
  int64_t s[26];
  auto strides = [&](int64_t ld, int64_t plane) {
    const int64_t v[26] = {H * T * dk, T * dk, dk, 1, G * dk * ld, dk * ld, 1, ld, G * plane, plane, dv, 1, H * T * dv, T * dv, dv, 1,
                           H * T, T, 1, H * T, T, 1, G * T * d.n, T * d.n, d.n, 1};
    std::copy(v, v + 26, s);
  };
  // compressed attention on the fp32 keys as a bf16 pair hi + lo; its log-sum-exp normalises the scoring
  if (int rc = split_keys_padded((const float*)d.k_cmp, hi, lo, G * d.B * dk, d.nbp, L.ld, st)) return rc;
  strides(L.ld, (int64_t)d.nbp * dv);
  if (int rc = nsa_cmp_attn_topn_fwd(d.q, hi, lo, (const float*)d.k_cmp, d.v_cmp, d.block_ends, o_cmp, Ls, Ms, lse2, idx, s, d.B, d.H, d.G, d.Tn, d.nb,
                                     d.nbp, d.dk, d.dv, d.l, d.d, d.l_prime, d.n, d.n_fixed, d.nb, d.scale, d.pos, NSA_FLAG_ANY_LENGTH, w + L.o_stage,
                                     L.stage, stream))
    return rc;
  const int64_t rows = (int64_t)d.B * G * T;
  fallback_kernel<<<(unsigned)((rows + 255) / 256), 256, 0, st>>>(idx, rows, d.Tn, d.n, d.l_prime, d.pos);
  const KvLayout kv = {d.cap, (int64_t)d.cap * dv};
  if (int rc = fa_fwd_sm100(d.q, d.k_win, d.v_win, o_win, Ls, Ms, d.B, d.H, d.G, d.Tn, L.Tk, d.dk, d.dv, kWin, d.window, 0, 0, 0, d.scale,
                            nullptr, nullptr, kv, st, d.pos))
    return rc;
  strides(d.cap, (int64_t)d.cap * dv);
  return nsa_slc_fwd_mix(d.q, d.k_slc, d.v_slc, idx, o_slc, Ls, Ms, s, d.B, d.H, d.G, d.Tn, L.Tk, d.n, d.l_prime, d.dk, d.dv, d.scale,
                         NSA_BF16, d.pos, NSA_FLAG_ANY_LENGTH, d.gate_logits, o_cmp, o_win, d.out, gates, d.gate_mode, 1, w + L.o_stage, L.stage, stream);
}
