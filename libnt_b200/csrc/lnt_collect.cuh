// Fold of runs of equal keys of key-sorted pairs whose count lives on the
// device, with the kept runs chosen and re-keyed by a functor.
//
// Resident CTAs take tiles of 2048 pairs in order, eight warps of 256
// consecutive ones, held in registers lane-striped (eight rows of 32 per warp:
// coalesced loads, and no shared-memory staging).  A row's runs are summed by
// a segmented scan over the lanes; what is open at the end of a row, a warp or
// the tile is carried on.  A run is written by the tile in which it ends.  Only
// there is the part in earlier tiles needed: every tile publishes what is open
// at its end (before it waits for anything), and the tile adds them up back to
// the run's first key, in a fixed order.  Output offsets come from a decoupled
// look-back over the tiles' counts.
//
// Sink: bool keep(key, sum); u64 out_key(key).
#pragma once

#include "lnt_common.cuh"

namespace lnt {
namespace collect {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRows = 8;
constexpr int kTile = kThreads * kRows;
constexpr u32 FULL = 0xffffffffu;
constexpr unsigned long long kFlagAgg = 1ull << 62;
constexpr unsigned long long kFlagPre = 2ull << 62;
constexpr unsigned long long kFlagMask = 3ull << 62;
constexpr unsigned long long kValMask = (1ull << 62) - 1ull;

// What is open at the end of a tile: the sum from its last head on (kHead), or
// of the whole tile when no run starts in it (kWhole).
constexpr u32 kWhole = 1, kHead = 2;

struct Ctrl {
  unsigned long long* status;  // per tile: output count
  double* open;                // per tile: open sum
  u32* oflag;                  // per tile: kWhole or kHead
  u32* counter;
};

struct Layout {
  u32 ntiles;
  size_t off_status, off_oflag, off_counter, zero_bytes, off_open, total;
};

inline Layout layout(size_t n) {
  Layout L;
  L.ntiles = (u32)((n + kTile - 1) / kTile);
  size_t off = 0;
  L.off_status = off;
  off += align_up((size_t)L.ntiles * 8, 256);
  L.off_oflag = off;
  off += align_up((size_t)L.ntiles * 4, 256);
  L.off_counter = off;
  off += 256;
  L.zero_bytes = off;
  L.off_open = off;
  off += align_up((size_t)L.ntiles * 8, 256);
  L.total = off;
  return L;
}

// Sum of what is open before `tile` (one warp): back to the nearest tile in
// which a run starts, 32 tiles per round, each round waited for as a whole so
// that the order of the additions does not depend on timing.
__device__ __forceinline__ double open_before(const Ctrl& c, u32 tile) {
  const int lane = threadIdx.x & 31;
  double sum = -0.0;  // the additive identity that keeps the sign of zero sums
  int base = (int)tile - 1;
  u32 spins = 0;
  while (base >= 0) {
    const int p = base - lane;
    const u32 f = p >= 0 ? *reinterpret_cast<const volatile u32*>(c.oflag + p) : kHead;
    const u32 notready = __ballot_sync(FULL, f == 0);
    const u32 heads = __ballot_sync(FULL, (f & kHead) != 0);
    const int upto = heads ? __ffs(heads) : 32;  // lanes [0, upto) contribute
    if (notready & (upto == 32 ? FULL : (1u << upto) - 1u)) {
      if (++spins > spin_limit()) {
        latch_error(kErrReduceLookback);
        break;
      }
      continue;
    }
    __threadfence();
    double v = lane < upto && p >= 0 ? __ldcg(c.open + p) : -0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    sum = v + sum;
    if (heads) break;
    base -= 32;
  }
  return sum;
}

template <class Sink>
__global__ void __launch_bounds__(kThreads, 3) collect_runs_kernel(const u64* keys, const double* vals,
                                                                   const Sink sink, const u64* d_n, const Ctrl c,
                                                                   u64* __restrict__ out_k,
                                                                   double* __restrict__ out_v,
                                                                   u64* __restrict__ d_nout) {
  __shared__ double s_open[kWarps], s_carry;
  __shared__ u32 s_flag[kWarps], s_cnt[kWarps], s_tile;
  __shared__ unsigned long long s_off;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const u32 le = lane == 31 ? FULL : (2u << lane) - 1u;  // this lane and those before it
  const size_t n = *d_n;
  const u32 ntiles = (u32)((n + kTile - 1) / kTile);
  if (ntiles == 0 && blockIdx.x == 0 && tid == 0) *d_nout = 0;
  for (;;) {
    if (tid == 0) s_tile = atomicAdd(c.counter, 1u);
    __syncthreads();
    const u32 tile = s_tile;
    if (tile >= ntiles) return;
    const size_t wbase = (size_t)tile * kTile + (size_t)warp * (32 * kRows);
    u64 k[kRows];
    double v[kRows];
    u32 heads[kRows], ends[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const size_t i = wbase + r * 32 + lane;
      k[r] = i < n ? keys[i] : 0;
      v[r] = i < n ? vals[i] : -0.0;
    }
    const u64 before = wbase > 0 && wbase < n ? keys[wbase - 1] : 0;
    const size_t wend = wbase + 32 * kRows;
    const u64 after = wend < n ? keys[wend] : 0;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const size_t i = wbase + r * 32 + lane;
      u64 prev = __shfl_up_sync(FULL, k[r], 1);
      const u64 last = r > 0 ? __shfl_sync(FULL, k[r > 0 ? r - 1 : 0], 31) : before;
      if (lane == 0) prev = last;
      heads[r] = __ballot_sync(FULL, i >= n || i == 0 || k[r] != prev);  // (beyond n: heads of nothing)
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const u32 next = r + 1 < kRows ? heads[r + 1 < kRows ? r + 1 : r] & 1u
                                     : (u32)(wend >= n || after != __shfl_sync(FULL, k[r], 31));
      ends[r] = (heads[r] >> 1) | (next << 31);
    }
    // sums from the start of each run (or of the warp) to every entry
    double carry = -0.0;
    u32 any_head = 0;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const u32 mine = heads[r] & le;
      const int start = mine ? 31 - __clz(mine) : 0;
      double s = v[r];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(FULL, s, o);
        if (lane - o >= start) s = y + s;
      }
      if (!mine) s = carry + s;
      v[r] = s;
      carry = __shfl_sync(FULL, s, 31);
      any_head |= heads[r];
    }
    if (lane == 0) {
      s_open[warp] = carry;
      s_flag[warp] = any_head ? kHead : kWhole;
    }
    __syncthreads();
    // warp 0: publish what is open at the tile's end; fetch what is open
    // before the tile if a run that ends here started earlier
    if (warp == 0) {
      if (lane == 0) {
        double o = -0.0;
        u32 f = kWhole;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
          if (s_flag[w] & kHead) {
            o = s_open[w];
            f = kHead;
          } else {
            o = o + s_open[w];
          }
        }
        c.open[tile] = o;
        __threadfence();
        *reinterpret_cast<volatile u32*>(c.oflag + tile) = f;
      }
      // the tile's first entry continues a run, which ends in this tile unless
      // the whole tile, and the entry after it, belong to it
      const size_t tbase = (size_t)tile * kTile;
      const bool continued = tbase > 0 && keys[tbase] == keys[tbase - 1];
      const size_t tend = tbase + kTile;
      if (continued && (tend >= n || keys[tend] != keys[tbase])) {
        const double o = open_before(c, tile);
        if (lane == 0) s_carry = o;
      }
    }
    __syncthreads();
    {  // the part of this warp's first run that lies before the warp
      const u32 first_heads = heads[0];
      if (!(first_heads & 1u)) {
        double o = -0.0;
        bool tile_open = true;
        for (int w = 0; w < warp; ++w) {
          if (s_flag[w] & kHead) {
            o = s_open[w];
            tile_open = false;
          } else {
            o = o + s_open[w];
          }
        }
        if (tile_open && tile > 0) o = s_carry + o;
        u32 seen = 0;
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          if (!seen && !(heads[r] & le)) v[r] = o + v[r];
          seen |= heads[r];
        }
      }
    }
    u32 kept[kRows], total = 0;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const size_t i = wbase + r * 32 + lane;
      const bool end = i < n && ((ends[r] >> lane) & 1u);
      kept[r] = __ballot_sync(FULL, end && sink.keep(k[r], v[r]));
      total += __popc(kept[r]);
    }
    if (lane == 0) s_cnt[warp] = total;
    __syncthreads();
    if (warp == 0) {  // output offset of the tile
      u32 tot = 0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) tot += s_cnt[w];
      if (lane == 0)
        *reinterpret_cast<volatile unsigned long long*>(&c.status[tile]) = (tile == 0 ? kFlagPre : kFlagAgg) | tot;
      unsigned long long off = 0;
      int base = (int)tile - 1;
      u32 spins = 0;
      while (base >= 0) {
        const int p = base - lane;
        const unsigned long long w =
            p >= 0 ? *reinterpret_cast<const volatile unsigned long long*>(c.status + p) : kFlagPre;
        const unsigned long long f = w & kFlagMask;
        const u32 notready = __ballot_sync(FULL, f == 0);
        const u32 pre = __ballot_sync(FULL, f == kFlagPre);
        const int first_nr = notready ? __ffs(notready) - 1 : 32;
        const int first_pre = pre ? __ffs(pre) - 1 : 32;
        const int take = first_pre < first_nr ? first_pre + 1 : first_nr;
        unsigned long long x = lane < take ? (w & kValMask) : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
        off += x;
        if (first_pre < first_nr) break;
        base -= first_nr;
        if (first_nr < 32 && ++spins > spin_limit()) {
          latch_error(kErrReduceLookback);
          break;
        }
      }
      if (lane == 0) {
        if (tile != 0) *reinterpret_cast<volatile unsigned long long*>(&c.status[tile]) = kFlagPre | (off + tot);
        s_off = off;
        if (tile == ntiles - 1) *d_nout = off + tot;
      }
    }
    __syncthreads();
    unsigned long long o = s_off;
    for (int w = 0; w < warp; ++w) o += s_cnt[w];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      if ((kept[r] >> lane) & 1u) {
        const u64 at = o + __popc(kept[r] & (le >> 1));
        __stcs(out_k + at, sink.out_key(k[r]));
        __stcs(out_v + at, v[r]);
      }
      o += __popc(kept[r]);
    }
    __syncthreads();  // the shared words are reused by the next tile
  }
}

// n_max: the most pairs there can be.
template <class Sink>
int run(const u64* keys, const double* vals, const u64* d_n, size_t n_max, const Sink& sink, u64* out_k, double* out_v,
        u64* d_nout, void* ws, cudaStream_t s, const char* prof_name) {
  const Layout L = layout(n_max);
  unsigned char* w = static_cast<unsigned char*>(ws);
  if (cudaMemsetAsync(w, 0, L.zero_bytes, s) != cudaSuccess) return LNT_DEVICE_ERROR;
  Ctrl c;
  c.status = reinterpret_cast<unsigned long long*>(w + L.off_status);
  c.open = reinterpret_cast<double*>(w + L.off_open);
  c.oflag = reinterpret_cast<u32*>(w + L.off_oflag);
  c.counter = reinterpret_cast<u32*>(w + L.off_counter);
  const u32 grid = L.ntiles < 3u * (u32)sm_count() ? L.ntiles : 3u * (u32)sm_count();
  ProfScope prof(prof_name, s);
  collect_runs_kernel<Sink><<<grid ? grid : 1u, kThreads, 0, s>>>(keys, vals, sink, d_n, c, out_k, out_v, d_nout);
  count_launch();
  return launch_status();
}

}  // namespace collect
}  // namespace lnt
