// How the tile kernels of the strided families (attn_generic.cu, attn_mma.cu) cut a branch into row tiles and key tiles.
#pragma once
#include "attn_args.cuh"

namespace nsa {

constexpr int kTileThreads = 128;

// What describes the current key tile (`ends`, `member`), and scratch for the selection's union of blocks; in shared memory.
template <int TILE, int WINDOW, int IDX>
struct TileLists {
  static constexpr int kTile = TILE, kIdWindow = WINDOW, kIdxInts = IDX;   // block ids per pass of the bitmap, index entries kept
  int *ends, *member;      // [TILE] each
  unsigned* bits;          // [WINDOW / 32]
  int* idx;                // [IDX]
};

// Rows of a query tile: HT heads of a group x QT consecutive queries, row = qi * HT + hh.
template <int TILE>
struct RowTile {
  int b, g, h0, nh, t0, HT, QT;
  __device__ RowTile(const AttnArgs& a) {
    const int hpg = a.H / a.G;
    HT = min(hpg, TILE);
    QT = TILE / HT;
    const int nhc = (hpg + HT - 1) / HT, hc = blockIdx.y % nhc, bg = blockIdx.y / nhc;
    b = bg / a.G;
    g = bg % a.G;
    h0 = g * hpg + hc * HT;
    nh = min(HT, hpg - hc * HT);
    t0 = blockIdx.x * QT;
  }
  __device__ int head(int r) const { return h0 + r % HT; }
  __device__ int query(int r, int Tq) const {       // -1: the row does not exist
    const int t = t0 + r / HT;
    return r < QT * HT && r % HT < nh && t < Tq ? t : -1;
  }
  static dim3 grid(const AttnArgs& a) {
    const int hpg = a.H / a.G, HT = hpg < TILE ? hpg : TILE, QT = TILE / HT, nhc = (hpg + HT - 1) / HT;
    return dim3((a.Tq + QT - 1) / QT, a.B * a.G * nhc);
  }
};

// Calls f(key0, n) with every run of up to TILE candidate keys of the tile's queries (ALIGN: the window's runs start at
// multiples of it); the lists then describe the run for `visible`.
template <int MODE, int ALIGN, typename LISTS, typename F>
__device__ __forceinline__ void for_each_key_tile(const AttnArgs& a, const RowTile<LISTS::kTile>& rt, const LISTS& s, F&& f) {
  constexpr int kTile = LISTS::kTile;
  const int tlast = min(rt.t0 + rt.QT, a.Tq) - 1;
  if (MODE == kWin) {
    const int beg = max(0, rt.t0 - a.window + 1) / ALIGN * ALIGN, end = min(tlast + 1, a.Tk);
    for (int k0 = beg; k0 < end; k0 += kTile) f(k0, min(kTile, end - k0));
  } else if (MODE == kCmp) {
    for (int k0 = 0; k0 < a.Tk; k0 += kTile) {
      const int n = min(kTile, a.Tk - k0);
      bool any = false;
      __syncthreads();
      if (threadIdx.x < kTile) {
        const int e = threadIdx.x < n ? a.block_ends[k0 + threadIdx.x] : 0x7fffffff;
        s.ends[threadIdx.x] = e;
        any = e <= tlast;
      }
      if (__syncthreads_or(any)) f(k0, n);
    }
  } else {
    const int nq = tlast - rt.t0 + 1, total = nq * a.nslots;
    const int* rows = a.indices + rt.b * a.sidx[0] + rt.g * a.sidx[1] + (int64_t)rt.t0 * a.sidx[2];
    const bool kept = total <= LISTS::kIdxInts;
    if (kept)
      for (int i = threadIdx.x; i < total; i += kTileThreads) s.idx[i] = rows[(int64_t)(i / a.nslots) * a.sidx[2] + (i % a.nslots) * a.sidx[3]];
    for (int w0 = 0; w0 < a.nblk; w0 += LISTS::kIdWindow) {
      if (a.causal && (int64_t)w0 * a.lprime > tlast) break;
      __syncthreads();
      for (int i = threadIdx.x; i < LISTS::kIdWindow / 32; i += kTileThreads) s.bits[i] = 0;
      __syncthreads();
      for (int i = threadIdx.x; i < total; i += kTileThreads) {
        const int q = i / a.nslots;
        const int id = kept ? s.idx[i] : rows[(int64_t)q * a.sidx[2] + (i % a.nslots) * a.sidx[3]];
        if (id < w0 || id >= w0 + LISTS::kIdWindow || (int64_t)id * a.lprime >= a.Tk || (a.causal && (int64_t)id * a.lprime > rt.t0 + q)) continue;
        atomicOr(&s.bits[(id - w0) >> 5], 1u << ((id - w0) & 31));
      }
      __syncthreads();
      const int words = min(LISTS::kIdWindow, a.nblk - w0 + 31) / 32;
      for (int w = 0; w < words; ++w) {
        unsigned m = s.bits[w];
        while (m) {
          const int id = w0 + w * 32 + __ffs(m) - 1;
          m &= m - 1;
          __syncthreads();
          if (threadIdx.x < nq) {        // (QT <= TILE <= threads)
            bool in = false;
            for (int i = 0; i < a.nslots; ++i)
              in |= (kept ? s.idx[threadIdx.x * a.nslots + i] : rows[(int64_t)threadIdx.x * a.sidx[2] + i * a.sidx[3]]) == id;
            s.member[threadIdx.x] = in;
          }
          __syncthreads();
          const int beg = id * a.lprime;
          int end = (int)min((int64_t)beg + a.lprime, (int64_t)a.Tk);
          if (a.causal) end = min(end, tlast + 1);
          for (int k0 = beg; k0 < end; k0 += kTile) f(k0, min(kTile, end - k0));
        }
      }
    }
  }
}
// key key0 + kk of the current run, seen by row r's query at position t (-1: no such row)?
template <int MODE, typename LISTS>
__device__ __forceinline__ bool visible(const AttnArgs& a, const LISTS& s, int r, int HT, int t, int key, int kk, int n) {
  if (t < 0 || kk >= n) return false;
  if (MODE == kWin) return key <= t && key > t - a.window;
  if (MODE == kCmp) return s.ends[kk] <= t;
  return s.member[r / HT] != 0 && !(a.causal && key > t);
}

// The keys of a dK/dV tile (TILE keys that do not cross a selection block) and the queries that may see them: nq positions from
// qbeg on, or the entries list[0..nq) of the inverse index.
struct KeyTile {
  int key0, n, qbeg, nq;
  const int* list;
};
template <int MODE, int TILE>
__device__ __forceinline__ KeyTile key_tile(const AttnArgs& a, int tile, int b, int g, int* ends, int* first_sm) {
  KeyTile k;
  k.qbeg = 0;
  k.list = nullptr;
  int kend;
  if (MODE == kSlc) {
    const int per = (a.lprime + TILE - 1) / TILE, blk = tile / per;
    k.key0 = blk * a.lprime + tile % per * TILE;
    kend = min(min(k.key0 + TILE, (blk + 1) * a.lprime), a.Tk);
    const int* off = a.csr_off + (int64_t)(b * a.G + g) * (a.nblk + 1);
    k.list = a.csr_t + (int64_t)(b * a.G + g) * a.Tq * a.nslots + off[blk];
    k.nq = off[blk + 1] - off[blk];
  } else {
    k.key0 = tile * TILE;
    kend = min(k.key0 + TILE, a.Tk);
    if (MODE == kWin) {
      k.qbeg = k.key0;
      k.nq = (int)min((int64_t)a.Tq, (int64_t)kend - 1 + a.window) - k.qbeg;
    } else {
      if (threadIdx.x == 0) *first_sm = 0x7fffffff;
      __syncthreads();
      if (threadIdx.x < TILE) {
        const int e = k.key0 + (int)threadIdx.x < kend ? max(a.block_ends[k.key0 + threadIdx.x], 0) : 0x7fffffff;
        ends[threadIdx.x] = e;
        atomicMin(first_sm, e);
      }
      __syncthreads();
      k.qbeg = *first_sm;
      k.nq = k.qbeg < a.Tq ? a.Tq - k.qbeg : 0;
    }
  }
  k.n = max(kend - k.key0, 0);      // (a tile behind the last key of a clipped block holds none)
  if (k.n == 0 || k.nq < 0) k.nq = 0;
  return k;
}
template <int MODE, int TILE>
inline int64_t key_tiles(const AttnArgs& a) {
  return MODE == kSlc ? (int64_t)a.nblk * ((a.lprime + TILE - 1) / TILE) : (a.Tk + TILE - 1) / TILE;
}

}  // namespace nsa
