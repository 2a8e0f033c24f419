// Inverse index for the selected-block attention backward: for every (batch, group, key block) the
// list of (query position | slot << 24) entries of the queries that selected the block, in ascending
// query order.
//
// The reference accumulates dK/dV of selected blocks with atomics from every query tile
// (nsa/kernels.py:1111-1115, 1140-1144); here each key block instead walks its own query list in a
// fixed order, which needs this "block -> queries" map.  It is a counting sort of the (query, slot)
// pairs by block id: per-chunk histograms, a scan, and an ordered fill.  Integer atomics are used
// only for counts, whose totals do not depend on the order of arrival.
#include "attn_args.cuh"
#include "common.cuh"

namespace nsa {

constexpr int kChunk = 128;      // queries per histogram chunk
// Bounds of the two kernels' dynamic shared memory: the attribute that admits a launch belongs to the kernel and is shared by all
// host threads, so it is set to the bound, never to the size of one call, which another thread's launch may exceed.
constexpr size_t kCountSmemMax = 160 * 1024, kFillSmemMax = 200 * 1024;
constexpr int kFillWarps = 8;    // warps ordering the entries of a chunk (one when the counters of eight do not fit)

struct CsrArgs {
  const int* indices;
  int64_t sidx[4];
  int B, G, Tq, Tkv, nslots, lprime, nblk, nchunks, causal, q0, slots_pad;
  int *hist, *off, *csr_t;       // hist: [BG][nchunks + 1][nblk], the last row holds the totals
};

// Block id of the (query, slot) pair a lane covers: lanes hold `slots_pad` slots of 32 / slots_pad consecutive queries.
// -1 when the slot contributes nothing (the rules of slot_block); a repeated id is found by matching the lanes of one query.
__device__ __forceinline__ int lane_block(const CsrArgs& a, int b, int g, int t, int t1, int lane) {
  const int s = lane & (a.slots_pad - 1);
  int id = -1;
  if (t < t1 && s < a.nslots) id = a.indices[b * a.sidx[0] + g * a.sidx[1] + (int64_t)t * a.sidx[2] + s * a.sidx[3]];
  const bool in = id >= 0 && (int64_t)id * a.lprime < a.Tkv && !(a.causal && (int64_t)id * a.lprime > a.q0 + t);
  const int key = in ? id * 32 + (lane & ~(a.slots_pad - 1)) : -1 - lane;   // id < 2^26: checked by the host
  const unsigned same = __match_any_sync(0xffffffffu, key);
  return in && (same & ((1u << lane) - 1u)) == 0 ? id : -1;
}

__global__ void csr_count(const CsrArgs a) {
  extern __shared__ int sh[];
  const int c = blockIdx.x, bg = blockIdx.y, b = bg / a.G, g = bg % a.G;
  for (int i = threadIdx.x; i < a.nblk; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int t0 = c * kChunk, t1 = min(a.Tq, t0 + kChunk);
  const int lane = threadIdx.x & 31, qpw = 32 / a.slots_pad;
  for (int tb = t0 + (threadIdx.x >> 5) * qpw; tb < t1; tb += (blockDim.x >> 5) * qpw) {
    const int id = lane_block(a, b, g, tb + lane / a.slots_pad, t1, lane);
    if (id >= 0) atomicAdd(&sh[id], 1);
  }
  __syncthreads();
  int* h = a.hist + ((int64_t)bg * (a.nchunks + 1) + c) * a.nblk;
  for (int i = threadIdx.x; i < a.nblk; i += blockDim.x) h[i] = sh[i];
}

// hist[bg][c][blk] becomes the count of entries of blk in chunks < c; row nchunks the block's total.  32 columns per
// thread block, 32 threads per column, each owning a run of chunks.
__global__ void csr_scan(const CsrArgs a) {
  __shared__ int part[32][33];
  const int bg = blockIdx.y, x = threadIdx.x, y = threadIdx.y, blk = blockIdx.x * 32 + x;
  int* h = a.hist + (int64_t)bg * (a.nchunks + 1) * a.nblk + blk;
  const int per = (a.nchunks + 31) / 32, lo = min(a.nchunks, y * per), hi = min(a.nchunks, lo + per);
  int sum = 0;
  if (blk < a.nblk)
#pragma unroll 4
    for (int c = lo; c < hi; ++c) sum += h[(int64_t)c * a.nblk];
  part[y][x] = sum;
  __syncthreads();
  int run = 0;
  for (int i = 0; i < y; ++i) run += part[i][x];
  if (blk >= a.nblk) return;
  if (y == 31) h[(int64_t)a.nchunks * a.nblk] = run + sum;
#pragma unroll 4
  for (int c = lo; c < hi; ++c) {
    const int v = h[(int64_t)c * a.nblk];
    h[(int64_t)c * a.nblk] = run;
    run += v;
  }
}

// Ordered fill of one chunk.  Latency-bound (the chunk's 128 x nslots ids are 8 KB): one warp walking the whole chunk
// needed 64 dependent steps of a few hundred cycles each, 47 us per launch at every size.  Each of W warps now orders its
// own kChunk / W queries with byte counters of its own (an id occurs at most once per query, so a chunk holds at most
// 128 of it), the counters are prefixed over the warps, and a second walk writes the entries.
// Lanes cover (query, slot) pairs so that a lower lane is always an earlier query; equal ids of a step are ranked by lane.
__global__ void csr_fill(const CsrArgs a) {
  extern __shared__ int base[];                                    // [nblk] start of each block's entries of this chunk
  const int W = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* cnt = reinterpret_cast<uint8_t*>(base + a.nblk);        // [W][nblk]
  __shared__ int wsum[32];
  const int c = blockIdx.x, bg = blockIdx.y, b = bg / a.G, g = bg % a.G;
  const int* h = a.hist + ((int64_t)bg * (a.nchunks + 1) + c) * a.nblk;
  const int* tot = a.hist + ((int64_t)bg * (a.nchunks + 1) + a.nchunks) * a.nblk;
  // block starts: exclusive prefix of the totals, every thread owning a run of blocks
  const int per = (a.nblk + blockDim.x - 1) / blockDim.x, lo = min(a.nblk, (int)threadIdx.x * per), hi = min(a.nblk, lo + per);
  int mine = 0;
  for (int i = lo; i < hi; ++i) mine += tot[i];
  int run = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += v;
  }
  if (lane == 31) wsum[warp] = run;
  for (int i = threadIdx.x; i < W * a.nblk; i += blockDim.x) cnt[i] = 0;
  __syncthreads();
  run -= mine;
  for (int w = 0; w < warp; ++w) run += wsum[w];
  int* off = a.off + (int64_t)bg * (a.nblk + 1);
  if (c == 0 && threadIdx.x == 0) off[0] = 0;
  for (int i = lo; i < hi; ++i) {
    base[i] = run + h[i];
    run += tot[i];
    if (c == 0) off[i + 1] = run;
  }
  const int qpw = 32 / a.slots_pad, per_warp = kChunk / W;
  const int t0 = c * kChunk + warp * per_warp, t1 = min(a.Tq, t0 + per_warp);
  uint8_t* my = cnt + warp * a.nblk;
  for (int tb = t0; tb < t1; tb += qpw) {
    const int id = lane_block(a, b, g, tb + lane / a.slots_pad, t1, lane);
    const unsigned peers = __match_any_sync(0xffffffffu, id >= 0 ? id : -1 - lane);
    if (id >= 0 && (peers & ((1u << lane) - 1u)) == 0) my[id] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  for (int i = threadIdx.x; i < a.nblk; i += blockDim.x) {
    int before = 0;
    for (int w = 0; w < W; ++w) {
      const int v = cnt[w * a.nblk + i];
      cnt[w * a.nblk + i] = (uint8_t)before;
      before += v;
    }
  }
  __syncthreads();
  int* out = a.csr_t + (int64_t)bg * a.Tq * a.nslots;
  for (int tb = t0; tb < t1; tb += qpw) {
    const int t = tb + lane / a.slots_pad, s = lane & (a.slots_pad - 1);
    const int id = lane_block(a, b, g, t, t1, lane);
    const unsigned peers = __match_any_sync(0xffffffffu, id >= 0 ? id : -1 - lane);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    if (id >= 0) out[base[id] + my[id] + rank] = t | (s << 24);  // query position and its slot
    __syncwarp();
    if (id >= 0 && rank == 0) my[id] += __popc(peers);
    __syncwarp();
  }
}

static size_t align_up(size_t x) { return (x + 255) & ~size_t(255); }

static void csr_layout(int B, int G, int Tq, int Tkv, int nslots, int lprime, int* nblk, int* nchunks,
                       size_t* o_hist, size_t* o_off, size_t* o_t, size_t* total) {
  *nblk = (Tkv + lprime - 1) / lprime;
  *nchunks = (Tq + kChunk - 1) / kChunk;
  const size_t BG = (size_t)B * G;
  *o_hist = 0;
  *o_off = align_up(*o_hist + BG * (*nchunks + 1) * *nblk * sizeof(int));
  *o_t = align_up(*o_off + BG * (*nblk + 1) * sizeof(int));
  *total = align_up(*o_t + BG * (size_t)Tq * nslots * sizeof(int));
}

size_t slc_csr_workspace_bytes(int B, int G, int Tq, int Tkv, int nslots, int lprime) {
  int nblk, nchunks;
  size_t a, b, c, total;
  csr_layout(B, G, Tq, Tkv, nslots, lprime, &nblk, &nchunks, &a, &b, &c, &total);
  return total;
}

int build_slc_csr(const int* indices, const int64_t* sidx, int B, int G, int Tq, int Tkv, int nslots,
                  int lprime, int causal, int q0, void* workspace, size_t workspace_bytes, const int** csr_off,
                  const int** csr_t, cudaStream_t st) {
  CsrArgs a;
  size_t o_hist, o_off, o_t, total;
  csr_layout(B, G, Tq, Tkv, nslots, lprime, &a.nblk, &a.nchunks, &o_hist, &o_off, &o_t, &total);
  if (!workspace || workspace_bytes < total)
    return fail(NSA_ERR_WORKSPACE, "selection backward needs %zu workspace bytes, got %zu", total, workspace_bytes);
  if (nslots > 32) return fail(NSA_ERR_UNSUPPORTED, "selection supports at most 32 slots per query here");
  if (Tq >= (1 << 24)) return fail(NSA_ERR_UNSUPPORTED, "selection inverse index supports fewer than 2^24 queries");
  if ((size_t)a.nblk * sizeof(int) > kCountSmemMax) return fail(NSA_ERR_UNSUPPORTED, "too many key blocks (%d)", a.nblk);
  a.indices = indices;
  for (int i = 0; i < 4; ++i) a.sidx[i] = sidx[i];
  a.B = B; a.G = G; a.Tq = Tq; a.Tkv = Tkv; a.nslots = nslots; a.lprime = lprime; a.causal = causal; a.q0 = q0;
  char* w = (char*)workspace;
  a.hist = (int*)(w + o_hist);
  a.off = (int*)(w + o_off);
  a.csr_t = (int*)(w + o_t);
  a.slots_pad = 1;
  while (a.slots_pad < nslots) a.slots_pad *= 2;
  const size_t sm = (size_t)a.nblk * sizeof(int);
  const int W = (size_t)a.nblk * (sizeof(int) + kFillWarps) <= kFillSmemMax ? kFillWarps : 1;
  const size_t sm_fill = (size_t)a.nblk * (sizeof(int) + W);
  if (sm > 48 * 1024) cudaFuncSetAttribute(csr_count, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCountSmemMax);
  if (sm_fill > 48 * 1024) cudaFuncSetAttribute(csr_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFillSmemMax);
  KernelTimer kt("slc_inverse_index", st);
  dim3 grid(a.nchunks, B * G);
  csr_count<<<grid, 256, sm, st>>>(a);
  if (int rc = check_launch("csr_count")) return rc;
  csr_scan<<<dim3((a.nblk + 31) / 32, B * G), dim3(32, 32), 0, st>>>(a);
  if (int rc = check_launch("csr_scan")) return rc;
  csr_fill<<<grid, 32 * W, sm_fill, st>>>(a);
  if (int rc = check_launch("csr_fill")) return rc;
  *csr_off = a.off;
  *csr_t = a.csr_t;
  return NSA_OK;
}

}  // namespace nsa
