// One-sweep LSD radix sort of (u64 key, f64 value) pairs and the
// lnt_sort_pairs entry point.  Replaces the reference's in-place MSD radix
// sort RadixSortInPlace_PowerOf2Radix_Unsigned (LibMIARadix.h:444-484,
// 119-180): same ordering of keys; equal keys keep input order here (the
// reference's sort is unstable, so no order among equal keys is promised
// there).
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "lnt_msd.cuh"

namespace lnt {
namespace {

constexpr int kThreads = 256;  // histogram kernel CTA size
constexpr int kWarps = kThreads / 32;
constexpr u32 kFlagAgg = 1u << 30;
constexpr u32 kFlagPre = 2u << 30;
constexpr u32 kFlagMask = 3u << 30;
constexpr u32 kValMask = (1u << 30) - 1u;

__device__ __forceinline__ u32 ld_volatile(const u32* p) {
  return *reinterpret_cast<const volatile u32*>(p);
}
__device__ __forceinline__ void st_volatile(u32* p, u32 v) {
  *reinterpret_cast<volatile u32*>(p) = v;
}

template <bool FIRST>
__device__ __forceinline__ u64 load_key(const PairSource& s, size_t i) {
  if (!FIRST) return __ldcs(s.ak + i);
  if (i < s.na) return rekey(__ldcs(s.ak + i), s.ra);
  return rekey(__ldcs(s.bk + (i - s.na)), s.rb);
}

template <bool FIRST>
__device__ __forceinline__ double load_val(const PairSource& s, size_t i) {
  if (!FIRST) return __ldcs(s.av + i);
  if (i < s.na) return __ldcs(s.av + i);
  return s.bscale * __ldcs(s.bv + (i - s.na));
}

// ---------------------------------------------------------------------------
// Histogram of every pass's digits in one read of the keys.
// ---------------------------------------------------------------------------
// Block `block` of `nblocks` (THREADS threads); sh_hist: passes * RADIX words.
template <int BITS, int THREADS>
__device__ __forceinline__ void hist_block(const PairSource& src, u32 n, int passes, int key_bits, u32* ghist,
                                           u32* bstart, u32* done, u32* sh_hist, u32 block, u32 nblocks) {
  constexpr int RADIX = 1 << BITS;
  __shared__ bool s_last;
  for (int i = threadIdx.x; i < passes * RADIX; i += THREADS) sh_hist[i] = 0;
  __syncthreads();
  const u32 stride = nblocks * THREADS;
  constexpr int U = 8;  // independent loads in flight per thread
  u32 i = block * THREADS + threadIdx.x;
  for (; i + (U - 1) * stride < n; i += U * stride) {
    u64 k[U];
#pragma unroll
    for (int u = 0; u < U; ++u) k[u] = load_key<true>(src, i + u * stride);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      for (int p = 0; p < passes; ++p) {
        const int shift = p * BITS;
        const int w = min(BITS, key_bits - shift);
        atomicAdd(&sh_hist[p * RADIX + ((u32)(k[u] >> shift) & ((1u << w) - 1u))], 1u);
      }
    }
  }
  for (; i < n; i += stride) {
    u64 k = load_key<true>(src, i);
    for (int p = 0; p < passes; ++p) {
      const int shift = p * BITS;
      const int w = min(BITS, key_bits - shift);
      atomicAdd(&sh_hist[p * RADIX + ((u32)(k >> shift) & ((1u << w) - 1u))], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * RADIX; i += THREADS) {
    u32 c = sh_hist[i];
    if (c) atomicAdd(&ghist[i], c);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = (atomicAdd(done, 1u) == nblocks - 1);
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // Last block: exclusive scan of each pass's histogram into bin starts.
  __shared__ u32 s_warp[THREADS / 32];
  constexpr int DPT = (RADIX + THREADS - 1) / THREADS;
  for (int p = 0; p < passes; ++p) {
    u32 c[DPT];
    u32 local = 0;
#pragma unroll
    for (int j = 0; j < DPT; ++j) {
      int d = threadIdx.x * DPT + j;
      c[j] = d < RADIX ? __ldcg(&ghist[p * RADIX + d]) : 0u;
      local += c[j];
    }
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u32 inc = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      u32 t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    u32 wpre = 0;
    for (int w = 0; w < warp; ++w) wpre += s_warp[w];
    u32 run = wpre + inc - local;
#pragma unroll
    for (int j = 0; j < DPT; ++j) {
      int d = threadIdx.x * DPT + j;
      if (d < RADIX) bstart[p * RADIX + d] = run;
      run += c[j];
    }
    __syncthreads();
  }
}

template <int BITS>
__global__ void __launch_bounds__(kThreads) hist_kernel(const PairSource src, u32 n, int passes, int key_bits,
                                                        u32* ghist, u32* bstart, u32* done) {
  extern __shared__ u32 sh_hist[];
  hist_block<BITS, kThreads>(src, n, passes, key_bits, ghist, bstart, done, sh_hist, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------
// One digit pass.
// ---------------------------------------------------------------------------
template <int BITS, int THREADS, int ITEMS>
struct OnesweepShape {
  static constexpr int RADIX = 1 << BITS;
  static constexpr int WARPS = THREADS / 32;
  static constexpr int TILE = THREADS * ITEMS;
  static constexpr int DPT = (RADIX + THREADS - 1) / THREADS;  // digits per thread
  static constexpr size_t smem = (size_t)TILE * 16 + (size_t)WARPS * RADIX * 4 + (size_t)RADIX * 8 + 64;
  // CTAs per SM that shared memory allows (228 KB per SM, 1 KB reserved per CTA), at most 4
  static constexpr int kFit = (int)((228u * 1024u) / (smem + 1024u));
  static constexpr int MINB = kFit < 1 ? 1 : (kFit > 4 ? 4 : kFit);
};

__device__ __forceinline__ void cp_async8(void* smem_dst, const void* gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

template <bool FIRST>
__device__ __forceinline__ const double* val_ptr(const PairSource& s, size_t i) {
  if (!FIRST || i < s.na) return s.av + i;
  return s.bv + (i - s.na);
}

// Lanes of the warp holding the same BITS-bit digit (one ballot per bit).
template <int BITS>
__device__ __forceinline__ u32 match_digit(u32 d) {
  u32 peers = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < BITS; ++b) {
    const u32 bit = (d >> b) & 1u;
    const u32 m = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? m : ~m;
  }
  return peers;
}

// One tile of a digit pass.  Tiles are handed out in order, so every
// predecessor a look-back waits on belongs to a running CTA.  QUEUE: part of
// lsd_queue_kernel.
struct QueueState {
  u32 task;
  u32 step;   // the step this CTA is in
  u32 count;  // its finished tasks of that step, not yet reported
  u32 taken;  // `task` is the next one already
  u32 expired;  // a wait ran out
};

template <int BITS, int THREADS, int ITEMS, int W, bool FIRST, bool QUEUE = false>
__device__ __forceinline__ void onesweep_tile(const PairSource& src, u64* out_k, double* out_v, u32 n, u32 shift,
                                              u32 mask, const u32* bstart, u32* status, u32 tile,
                                              unsigned char* smem, QueueState* q = nullptr,
                                              u32* gate = nullptr) {
  using S = OnesweepShape<BITS, THREADS, ITEMS>;
  constexpr int RADIX = S::RADIX;
  constexpr int WARPS = S::WARPS;
  constexpr int TILE = S::TILE;
  constexpr int DPT = S::DPT;
  u64* s_x = reinterpret_cast<u64*>(smem);               // TILE: tile in digit order
  double* s_v = reinterpret_cast<double*>(s_x + TILE);   // TILE: values in input order
  u32* s_whist = reinterpret_cast<u32*>(s_v + TILE);     // WARPS * RADIX
  u32* s_tstart = s_whist + WARPS * RADIX;               // RADIX
  u32* s_glob = s_tstart + RADIX;                        // RADIX
  u32* s_misc = s_glob + RADIX;                          // 16

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < WARPS * RADIX; i += THREADS) s_whist[i] = 0;
  __syncthreads();
  const size_t tile_base = (size_t)tile * TILE;
  const u32 tile_n = (u32)min((size_t)TILE, (size_t)n - tile_base);
  const u32 warp_base = warp * ITEMS * 32;

  // ---- load keys (warp-striped: coalesced 256 B per warp per item) -------
  u64 key[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const u32 off = warp_base + i * 32 + lane;
    key[i] = off < tile_n ? load_key<FIRST>(src, tile_base + off) : 0ull;
  }
  // values go straight to shared memory; the copy overlaps everything up to
  // the value scatter and holds no registers
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const u32 off = warp_base + i * 32 + lane;
    if (off < tile_n) cp_async8(&s_v[off], val_ptr<FIRST>(src, tile_base + off));
  }
  cp_async_commit();

  // ---- per-warp digit counts (no return values: fire-and-forget) ---------
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const u32 off = warp_base + i * 32 + lane;
    if (off < tile_n) atomicAdd(&s_whist[warp * RADIX + ((u32)(key[i] >> shift) & mask)], 1u);
  }
  __syncthreads();

  // ---- tile counts: publish at once so successors can look back ----------
  u32 cnt[DPT];
  u32 local = 0;
#pragma unroll
  for (int j = 0; j < DPT; ++j) {
    const int d = tid * DPT + j;
    u32 c = 0;
    if (d < RADIX) {
#pragma unroll
      for (int w = 0; w < WARPS; ++w) c += s_whist[w * RADIX + d];
      const u32 word = tile == 0 ? (kFlagPre | (__ldcg(bstart + d) + c)) : (kFlagAgg | c);
      st_volatile(&status[(size_t)tile * RADIX + d], word);
    }
    cnt[j] = c;
    local += c;
  }
  // ---- block exclusive scan of digit counts; per-(warp, digit) bases ------
  u32 tstart[DPT];
  {
    u32 inc = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) s_misc[4 + warp] = inc;
    __syncthreads();
    u32 run = inc - local;
    for (int w = 0; w < warp; ++w) run += s_misc[4 + w];
#pragma unroll
    for (int j = 0; j < DPT; ++j) {
      const int d = tid * DPT + j;
      tstart[j] = run;
      if (d < RADIX) {
        u32 b = run;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
          const u32 c = s_whist[w * RADIX + d];
          s_whist[w * RADIX + d] = b;
          b += c;
        }
      }
      run += cnt[j];
    }
  }

  __syncthreads();  // the per-(warp, digit) bases are complete
  // ---- stable rank: ballot match + per-(warp, digit) running base ---------
  u32 pos[ITEMS];
  const u32 lt_mask = (1u << lane) - 1u;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const u32 off = warp_base + i * 32 + lane;
    const bool valid = off < tile_n;
    const u32 vmask = __ballot_sync(0xffffffffu, valid);
    const u32 d = valid ? ((u32)(key[i] >> shift) & mask) : 0u;
    const u32 peers = match_digit<BITS>(d) & vmask;
    u32 base = 0;
    if (valid) base = s_whist[warp * RADIX + d];
    __syncwarp();
    if (valid && lane == __ffs(peers) - 1) s_whist[warp * RADIX + d] = base + __popc(peers);
    __syncwarp();
    pos[i] = base + __popc(peers & lt_mask);
  }
  // ---- stage keys in digit order ------------------------------------------
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const u32 off = warp_base + i * 32 + lane;
    if (off < tile_n) s_x[pos[i]] = key[i];
  }
  __syncthreads();

  // ---- decoupled look-back, W predecessors per round trip per digit -------
  // (after the local ranking: predecessors have had that long to publish
  // their inclusive prefixes, so the walk back is shorter)
  {
    u32 excl[DPT];
    int p[DPT];
    bool done[DPT];
#pragma unroll
    for (int j = 0; j < DPT; ++j) {
      const int d = tid * DPT + j;
      excl[j] = (tile == 0 && d < RADIX) ? __ldcg(bstart + d) : 0u;
      p[j] = (int)tile - 1;
      done[j] = (d >= RADIX) || tile == 0;
    }
    u32 spins = 0;
    while (true) {
      bool all_done = true;
#pragma unroll
      for (int j = 0; j < DPT; ++j) all_done = all_done && done[j];
      if (all_done) break;
      u32 w[DPT][W];
#pragma unroll
      for (int j = 0; j < DPT; ++j) {
        const int d = tid * DPT + j;
#pragma unroll
        for (int q = 0; q < W; ++q) {
          const int pp = p[j] - q;
          w[j][q] = (!done[j] && pp >= 0) ? ld_volatile(&status[(size_t)pp * RADIX + d]) : kFlagPre;
        }
      }
      bool stalled = false;
#pragma unroll
      for (int j = 0; j < DPT; ++j) {
        if (done[j]) continue;
        int q = 0;
#pragma unroll
        for (; q < W; ++q) {
          const u32 f = w[j][q] & kFlagMask;
          if (f == 0) break;
          excl[j] += w[j][q] & kValMask;
          if (f == kFlagPre) {
            done[j] = true;
            break;
          }
        }
        if (!done[j]) {
          p[j] -= q;
          if (q < W) stalled = true;
        }
      }
      if (stalled && ++spins > spin_limit()) {
        latch_error(kErrSortLookback);
        break;
      }
    }
#pragma unroll
    for (int j = 0; j < DPT; ++j) {
      const int d = tid * DPT + j;
      if (d >= RADIX) break;
      if (tile != 0) st_volatile(&status[(size_t)tile * RADIX + d], kFlagPre | (excl[j] + cnt[j]));
      s_glob[d] = excl[j] - tstart[j];
    }
  }
  if (QUEUE && tid == 0) {
    q->task = atomicAdd(&gate[1], 1u);  // (arrives while the tile is written)
    q->taken = 1u;
  }
  __syncthreads();

  // ---- scatter keys (digit runs -> contiguous destination ranges) ---------
  // The clamp changes nothing in a correct run (every position is < n).  It
  // keeps writes inside the output after a look-back gave up: a pass that
  // reads a previous pass's partial output sees digit counts that no longer
  // match the histogram, so its offsets could otherwise pass n.
  u32 dst[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const u32 idx = j * THREADS + tid;
    if (idx < tile_n) {
      const u64 k = s_x[idx];
      dst[j] = min(s_glob[(u32)(k >> shift) & mask] + idx, n - 1u);
      __stcs(out_k + dst[j], k);
    }
  }
  cp_async_wait_all();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const u32 off = warp_base + i * 32 + lane;
    if (off < tile_n) {
      double v = s_v[off];
      if (FIRST && tile_base + off >= src.na) v *= src.bscale;
      reinterpret_cast<double*>(s_x)[pos[i]] = v;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const u32 idx = j * THREADS + tid;
    if (idx < tile_n) __stcs(out_v + dst[j], reinterpret_cast<const double*>(s_x)[idx]);
  }
}

template <int BITS, int THREADS, int ITEMS, int W, bool FIRST>
__global__ void __launch_bounds__(THREADS, (OnesweepShape<BITS, THREADS, ITEMS>::MINB))
    onesweep_kernel(const PairSource src, u64* __restrict__ out_k, double* __restrict__ out_v, u32 n, u32 shift,
                    u32 mask, const u32* __restrict__ bstart, u32* __restrict__ status,
                    u32* __restrict__ tile_counter) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ u32 s_tile;
  if (threadIdx.x == 0) s_tile = atomicAdd(tile_counter, 1u);
  __syncthreads();
  onesweep_tile<BITS, THREADS, ITEMS, W, FIRST>(src, out_k, out_v, n, shift, mask, bstart, status, s_tile, smem);
}

// The whole sort in one launch, for the path behind a gate: it is nearly
// always skipped, and a skipped launch costs 1.6 us in the stream (seven to
// ten of them when every step was a kernel of its own).  CTAs take the tasks
// (zero the counts, histogram, the tiles of every pass) in order from a queue; at
// its first task of a step a CTA waits until the step before is complete, whose
// tasks all belong to running CTAs.  gate[1]: queue, gate[2 + step]: tasks done;
// zeroed by whoever writes the gate.  A CTA reports its tasks when it leaves a
// step, all at once (a report per tile, whose fence waits for the tile's scattered
// stores: 2^25 pairs of 36 bits 2.05 ms in all, 1.97 like this), and a pass's
// look-back words are zeroed by the step before instead of all of them first.  A
// CTA whose wait ran out waits no more (there may be hundreds of tasks left) and
// goes on: the error is latched, and every write stays inside the output whatever
// the histogram holds (see the clamp in onesweep_tile).
// Sorts behind a closed gate (95% of the keys in 1/4096 of the range), all told,
// against the digit passes alone: 2^17 pairs of 36 bits 92 and 70 us, 2^21 212 and
// 177, 2^25 1.96 and 1.82 ms.  The difference is the bucket histogram, the three
// skipped launches and the waits between the steps; evenly spread keys gain 41, 87
// us and 0.83 ms against the same figures.

// True when the wait ran out.
__device__ __forceinline__ bool queue_wait(const u32* done, u32 want) {
  bool expired = false;
  if (threadIdx.x == 0) {
    u32 spins = 0;
    while (!expired && ld_volatile(done) < want) {
      __nanosleep(100);
      expired = ++spins > spin_limit();
    }
    if (expired) latch_error(kErrSortLookback);
    __threadfence();
  }
  return __syncthreads_or(expired) != 0;
}

template <int BITS, int THREADS, int ITEMS, int W>
__global__ void __launch_bounds__(THREADS, (OnesweepShape<BITS, THREADS, ITEMS>::MINB))
    lsd_queue_kernel(const PairSource src, const SortPlan plan, u64* buf0_k, double* buf0_v, u64* buf1_k,
                     double* buf1_v, unsigned char* ctrl, u32* gate) {
  if (gated_off(src.gate, src.gate_run)) return;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ QueueState s_q;
  constexpr int RADIX = 1 << BITS;
  const u32 nh = min((plan.n + THREADS * 16 - 1) / (THREADS * 16), gridDim.x);
  u32* ghist = reinterpret_cast<u32*>(ctrl + plan.off_ghist);
  u32* bstart = reinterpret_cast<u32*>(ctrl + plan.off_bstart);
  u32* status = reinterpret_cast<u32*>(ctrl + plan.off_status);
  u32* counters = reinterpret_cast<u32*>(ctrl + plan.off_counters);
  if (threadIdx.x == 0) s_q = {0u, 0u, 0u, 0u, 0u};
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0 && !s_q.taken) s_q.task = atomicAdd(&gate[1], 1u);
    __syncthreads();
    // steps: 0 zero the counts (one task), 1 histogram, 2 + p pass p, the last:
    // nothing left.  The look-back words of a pass are zeroed in the step before.
    u32 t = s_q.task, step = 0;
    if (t >= 1) {
      t -= 1;
      step = 1;
      if (t >= nh) {
        t -= nh;
        step = 2 + min(t / plan.ntiles, (u32)plan.passes);
        t -= (step - 2) * plan.ntiles;
      }
    }
    if (step != s_q.step) {
      if (threadIdx.x == 0 && s_q.count) {  // (behind the barriers above: for the whole CTA)
        __threadfence();
        atomicAdd(&gate[2 + s_q.step], s_q.count);
      }
      if (step == 2 + (u32)plan.passes) return;
      bool expired = s_q.expired != 0u;
      if (!expired) expired = queue_wait(&gate[1 + step], step == 1 ? 1 : step == 2 ? nh : plan.ntiles);
      __syncthreads();
      if (threadIdx.x == 0) {
        s_q.step = step;
        s_q.count = 0u;
        s_q.expired = expired;
      }
    }
    if (step == 0) {
      u32* z = reinterpret_cast<u32*>(ctrl);
      for (size_t i = threadIdx.x; i < plan.off_status / 4; i += THREADS) z[i] = 0u;
      for (size_t i = plan.off_counters / 4 + threadIdx.x; i < plan.ctrl_bytes / 4; i += THREADS) z[i] = 0u;
    } else if (step == 1) {
      uint4* z = reinterpret_cast<uint4*>(status);
      for (size_t i = (size_t)t * THREADS + threadIdx.x; i < (size_t)plan.ntiles * (RADIX / 4); i += (size_t)nh * THREADS)
        z[i] = make_uint4(0u, 0u, 0u, 0u);
      hist_block<BITS, THREADS>(src, plan.n, plan.passes, plan.key_bits, ghist, bstart, counters + plan.passes,
                                reinterpret_cast<u32*>(smem), t, nh);
    } else {
      const int p = (int)step - 2, which = (plan.passes - 1 - p) & 1, shift = p * BITS;
      const u32 mask = (1u << min(BITS, plan.key_bits - shift)) - 1u;
      u64* ok = which ? buf1_k : buf0_k;
      double* ov = which ? buf1_v : buf0_v;
      u32* st = status + (size_t)(p & 1) * plan.ntiles * RADIX;
      if (p + 1 < plan.passes) {
        u32* after = status + ((size_t)(~p & 1) * plan.ntiles + t) * RADIX;
        for (int d = threadIdx.x; d < RADIX; d += THREADS) after[d] = 0u;
      }
      if (p == 0) {
        onesweep_tile<BITS, THREADS, ITEMS, W, true, true>(src, ok, ov, plan.n, (u32)shift, mask, bstart, st, t, smem,
                                                           &s_q, gate);
      } else {
        PairSource in = src;
        in.ak = which ? buf0_k : buf1_k;
        in.av = which ? buf0_v : buf1_v;
        onesweep_tile<BITS, THREADS, ITEMS, W, false, true>(in, ok, ov, plan.n, (u32)shift, mask, bstart + p * RADIX,
                                                            st, t, smem, &s_q, gate);
      }
    }
    if (threadIdx.x == 0) ++s_q.count;
  }
}

// Copies the (possibly re-keyed / concatenated) source into buf0 unchanged;
// used when there is nothing to sort (all keys equal).
__global__ void copy_source_kernel(const PairSource src, u64* __restrict__ ok, double* __restrict__ ov, u32 n) {
  if (gated_off(src.gate, src.gate_run)) return;
  const u32 stride = gridDim.x * blockDim.x;
  for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    ok[i] = load_key<true>(src, i);
    ov[i] = load_val<true>(src, i);
  }
}

#define LNT_SV_ENTRY(B, T, I, W) {B, T, I, W},
const SortVariant kVariants[] = {LNT_SORT_VARIANTS(LNT_SV_ENTRY)};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);

template <int BITS, int THREADS, int ITEMS, int W>
int run_sort_queue(const SortPlan& plan, const PairSource& src, u64* buf0_k, double* buf0_v, u64* buf1_k,
                   double* buf1_v, void* ctrl, cudaStream_t s) {
  using Sh = OnesweepShape<BITS, THREADS, ITEMS>;
  static_assert(Sh::smem >= ((63 + BITS) / BITS) * (size_t)Sh::RADIX * 4, "the histogram of every pass fits");
  auto kern = lsd_queue_kernel<BITS, THREADS, ITEMS, W>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::smem) != cudaSuccess)
    return LNT_DEVICE_ERROR;
  const u32 grid = std::min(plan.ntiles, (u32)(Sh::MINB * sm_count()));
  ProfScope prof("sort_fallback", s);
  kern<<<grid, THREADS, Sh::smem, s>>>(src, plan, buf0_k, buf0_v, buf1_k, buf1_v, static_cast<unsigned char*>(ctrl),
                                       const_cast<u32*>(src.gate));
  count_launch();
  return launch_status();
}

template <int BITS, int THREADS, int ITEMS, int W>
int run_sort_variant(const SortPlan& plan, const PairSource& src, u64* buf0_k, double* buf0_v, u64* buf1_k,
                     double* buf1_v, void* ctrl, cudaStream_t s) {
  using Sh = OnesweepShape<BITS, THREADS, ITEMS>;
  constexpr int RADIX = Sh::RADIX;
  if (plan.tile != (u32)Sh::TILE || plan.bits != BITS) return LNT_BAD_ARG;
  unsigned char* c = static_cast<unsigned char*>(ctrl);
  u32* ghist = reinterpret_cast<u32*>(c + plan.off_ghist);
  u32* bstart = reinterpret_cast<u32*>(c + plan.off_bstart);
  u32* status = reinterpret_cast<u32*>(c + plan.off_status);
  u32* counters = reinterpret_cast<u32*>(c + plan.off_counters);
  if (cudaMemsetAsync(ctrl, 0, plan.ctrl_bytes, s) != cudaSuccess) return LNT_DEVICE_ERROR;

  // histogram of all passes
  {
    const size_t sh = (size_t)plan.passes * RADIX * 4;
    auto kern = hist_kernel<BITS>;
    if (sh > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
    const int blocks =
        std::max(1, std::min((int)((plan.n + kThreads * 16 - 1) / (kThreads * 16)), sm_count() * 4));
    ProfScope prof("sort_hist", s);
    kern<<<blocks, kThreads, sh, s>>>(src, plan.n, plan.passes, plan.key_bits, ghist, bstart,
                                      counters + plan.passes);
    count_launch();
  }
  constexpr size_t sh = Sh::smem;
  // (function attributes are per device: set them on every call)
  cudaFuncSetAttribute(onesweep_kernel<BITS, THREADS, ITEMS, W, true>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  cudaFuncSetAttribute(onesweep_kernel<BITS, THREADS, ITEMS, W, false>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
  const u32 grid = plan.ntiles;
  const u64* in_k = nullptr;
  const double* in_v = nullptr;
  for (int p = 0; p < plan.passes; ++p) {
    const int which = (plan.passes - 1 - p) & 1;
    u64* ok = which ? buf1_k : buf0_k;
    double* ov = which ? buf1_v : buf0_v;
    const int shift = p * BITS;
    const int w = std::min(BITS, plan.key_bits - shift);
    const u32 mask = (1u << w) - 1u;
    u32* st = status + (size_t)p * plan.ntiles * RADIX;
    ProfScope prof("sort_onesweep", s);
    if (p == 0)
      onesweep_kernel<BITS, THREADS, ITEMS, W, true><<<grid, THREADS, sh, s>>>(
          src, ok, ov, plan.n, (u32)shift, mask, bstart + p * RADIX, st, counters + p);
    else
      onesweep_kernel<BITS, THREADS, ITEMS, W, false><<<grid, THREADS, sh, s>>>(
          plain_source(in_k, in_v, plan.n), ok, ov, plan.n, (u32)shift, mask, bstart + p * RADIX, st, counters + p);
    count_launch();
    in_k = ok;
    in_v = ov;
  }
  return launch_status();
}

}  // namespace

}  // namespace lnt

#include "lnt_tuned.h"

namespace lnt {

int sort_variant_count() { return kNumVariants; }
const SortVariant& sort_variant(int i) { return kVariants[i]; }

int choose_sort_variant(size_t n, int key_bits) {
  if (const char* e = getenv("LNT_SORT_VARIANT")) {
    const int v = atoi(e);
    if (v >= 0 && v < kNumVariants) return v;
  }
  // tuned table: first entry whose key-width and size ranges contain the request
  for (const TunedSortEntry& t : kTunedSort) {
    if (key_bits <= t.key_bits_max && n <= t.n_max && t.variant >= 0 && t.variant < kNumVariants)
      return t.variant;
  }
  // untuned default: fewest passes, then the narrower digit
  int best = 0, best_passes = 1 << 20;
  for (int i = 0; i < kNumVariants; ++i) {
    const int p = key_bits <= 0 ? 0 : (key_bits + kVariants[i].bits - 1) / kVariants[i].bits;
    if (p < best_passes) {
      best = i;
      best_passes = p;
    }
  }
  return best;
}

// The shape behind a gate, of three compiled as a queue.  Below 2^22 pairs CTAs of
// 512 threads, with nine-bit digits where those save a pass; above, 256 threads of
// twelve keys (clustered keys, 512 and 256 threads: 2^19 pairs of 36 bits 101 and
// 117 us, 2^21 211 and 227, 2^23 622 and 599, 2^25 2.17 and 1.96 ms).
#define LNT_QUEUE_VARIANTS(X) \
  X(8, 512, 8, 16)            \
  X(9, 512, 8, 16)            \
  X(8, 256, 12, 16)
const SortVariant kQueueVariants[] = {LNT_QUEUE_VARIANTS(LNT_SV_ENTRY)};

int choose_queue_variant(size_t n, int key_bits) {
  if (n >= (1u << 22)) return 2;
  return (key_bits + 8) / 9 < (key_bits + 7) / 8 ? 1 : 0;
}

SortPlan make_sort_plan(size_t n, u64 max_key, bool gated) {
  SortPlan p;
  p.key_bits = key_bits_for(max_key);
  p.variant = gated ? choose_queue_variant(n, p.key_bits) : choose_sort_variant(n, p.key_bits);
  p.gated = gated;
  const SortVariant v = gated ? kQueueVariants[p.variant] : kVariants[p.variant];
  p.bits = v.bits;
  p.passes = p.key_bits == 0 ? 0 : (p.key_bits + v.bits - 1) / v.bits;
  p.n = (u32)n;
  p.tile = (u32)(v.threads * v.items);
  p.ntiles = (u32)((n + p.tile - 1) / p.tile);
  const size_t radix = (size_t)1 << v.bits;
  size_t off = 0;
  p.off_ghist = off;
  off += align_up((size_t)std::max(p.passes, 1) * radix * 4, 256);
  p.off_bstart = off;
  off += align_up((size_t)std::max(p.passes, 1) * radix * 4, 256);
  p.off_status = off;
  // (behind a gate the passes take turns in two sets of look-back words)
  off += align_up((size_t)(gated ? std::min(p.passes, 2) : p.passes) * p.ntiles * radix * 4, 256);
  p.off_counters = off;
  off += 256;
  p.ctrl_bytes = off;
  return p;
}

int run_sort(const SortPlan& plan, const PairSource& src, u64* buf0_k, double* buf0_v, u64* buf1_k,
             double* buf1_v, void* ctrl, cudaStream_t s) {
  if (plan.n == 0) return LNT_OK;
  if (plan.passes == 0) {
    const int blocks = std::max(1, std::min((int)((plan.n + 255) / 256), sm_count() * 8));
    ProfScope prof("sort_copy", s);
    copy_source_kernel<<<blocks, 256, 0, s>>>(src, buf0_k, buf0_v, plan.n);
    count_launch();
    return launch_status();
  }
  int i = 0;
  if (plan.gated) {
#define LNT_QV_CASE(B, T, I, W)                                                          \
  if (plan.variant == i) return run_sort_queue<B, T, I, W>(plan, src, buf0_k, buf0_v,   \
                                                           buf1_k, buf1_v, ctrl, s);     \
  ++i;
    LNT_QUEUE_VARIANTS(LNT_QV_CASE)
#undef LNT_QV_CASE
    return LNT_UNSUPPORTED;
  }
#define LNT_SV_CASE(B, T, I, W)                                                                           \
  if (plan.variant == i) return run_sort_variant<B, T, I, W>(plan, src, buf0_k, buf0_v, \
                                                             buf1_k, buf1_v, ctrl, s);   \
  ++i;
  LNT_SORT_VARIANTS(LNT_SV_CASE)
#undef LNT_SV_CASE
  return LNT_UNSUPPORTED;
}

}  // namespace lnt

using namespace lnt;

namespace {
// Workspace of lnt_sort_pairs: [ctrl | scratch pairs a | scratch pairs b].
struct SortPairsLayout {
  PairSort sort;
  size_t off_a, off_b, total;
};

SortPairsLayout sort_pairs_layout(size_t n, u64 max_key, bool buckets = true) {
  SortPairsLayout L;
  L.sort = make_pair_sort(n, max_key, buckets);
  size_t off = align_up(L.sort.ctrl_bytes, 256);
  L.off_a = off;
  off += L.sort.a_bytes;
  L.off_b = off;
  off += L.sort.a_bytes;  // (an in-place LSD sort of an odd number of passes needs both)
  L.total = off;
  return L;
}
}  // namespace

extern "C" {

int lnt_sort_variant_count(void) { return sort_variant_count(); }

int lnt_sort_variant(int index, int* bits, int* threads, int* items, int* window) {
  if (index < 0 || index >= sort_variant_count() || !bits || !threads || !items || !window) return LNT_BAD_ARG;
  const SortVariant& v = sort_variant(index);
  *bits = v.bits;
  *threads = v.threads;
  *items = v.items;
  *window = v.window;
  return LNT_OK;
}

int lnt_sort_pairs_workspace(size_t n, uint64_t max_key, size_t* bytes) {
  if (!bytes) return LNT_BAD_ARG;
  if (n >= (1u << 30)) return LNT_UNSUPPORTED;
  *bytes = sort_pairs_layout(n, max_key).total;
  return LNT_OK;
}

int lnt_sort_pairs(const uint64_t* keys_in, const double* vals_in, uint64_t* keys_out, double* vals_out,
                   size_t n, uint64_t max_key, void* workspace, size_t workspace_bytes, void* stream) {
  if (n == 0) return LNT_OK;
  if (!keys_in || !vals_in || !keys_out || !vals_out) return LNT_BAD_ARG;
  if (n >= (1u << 30)) return LNT_UNSUPPORTED;
  SortPairsLayout L = sort_pairs_layout(n, max_key);
  if (workspace_bytes < L.total) L = sort_pairs_layout(n, max_key, false);  // the digit passes may need less
  if (!workspace || workspace_bytes < L.total) return LNT_WORKSPACE;
  if ((uintptr_t)workspace % 256) return LNT_BAD_ARG;
  cudaStream_t s = as_stream(stream);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  PairSource src = plain_source((const u64*)keys_in, vals_in, n);
  const bool inplace =
      (const void*)keys_in == (const void*)keys_out || (const void*)vals_in == (const void*)vals_out;
  if (!inplace)
    return run_pair_sort(L.sort, src, (u64*)keys_out, vals_out, ws + L.off_a, ws + L.off_b, ws, s);
  // In place.  The bucketed path reads all input before it writes output, and
  // leaves the output alone when its gate closes.
  const SortPlan& lsd = L.sort.lsd;
  u32* gate = nullptr;
  if (L.sort.msd.ok) {
    gate = reinterpret_cast<u32*>(ws + L.sort.ctrl_bytes - 256);
    const int st = run_msd_sort(L.sort.msd, src, ws + L.off_b, ws + L.off_a, ws, nullptr, (u64*)keys_out, vals_out,
                                gate, s);
    if (st != LNT_OK || L.sort.msd.single) return st;
    src = gated_source(src, gate, 1);
  }
  if (lsd.passes == 0) return LNT_OK;  // all keys equal: input order is the stable order
  u64* tk = reinterpret_cast<u64*>(ws + L.off_a);
  double* tv = reinterpret_cast<double*>(ws + L.off_a + L.sort.a_bytes / 2);
  if (lsd.passes % 2 == 0)  // the first pass writes the scratch pairs
    return run_sort(lsd, src, (u64*)keys_out, vals_out, tk, tv, ws, s);
  // odd pass count: sort into the second scratch pairs and copy back
  u64* t2k = reinterpret_cast<u64*>(ws + L.off_b);
  double* t2v = reinterpret_cast<double*>(ws + L.off_b + L.sort.a_bytes / 2);
  const int st = run_sort(lsd, src, t2k, t2v, tk, tv, ws, s);
  if (st != LNT_OK) return st;
  const int blocks = std::max(1, std::min((int)((n + 255) / 256), sm_count() * 8));
  copy_source_kernel<<<blocks, 256, 0, s>>>(gated_source(plain_source(t2k, t2v, n), gate, 1), (u64*)keys_out, vals_out,
                                            (u32)n);
  count_launch();
  return launch_status();
}

}  // extern "C"
