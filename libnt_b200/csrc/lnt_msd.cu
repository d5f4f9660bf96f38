// Bucketed sort of (u64 key, f64 value) pairs, optionally folding equal keys:
//
//   1. msd_hist_kernel: one read of all (re-keyed, concatenated) keys counts
//      the 2^T buckets named by the top T key bits (T <= 15); the last CTA
//      derives the bucket starts, the partition passes' cursors and the gate.
//   2. one (T <= 8) or two partition passes group the pairs by bucket, most
//      significant digit first: a CTA takes a tile, ranks its pairs within
//      their digits by shared-memory atomics, reserves room for each digit
//      with one global atomic and writes the tile's digit runs.  The rank is
//      not stable, so the passes need no ballots, no per-warp counters and no
//      look-back; the order is restored at the end because every pair carries
//      its input index below its key (word = key << ib | index; the bits that
//      a pass has used up may fall off the top).  The second pass partitions
//      each first-pass segment for itself.
//   3. bucket_sort_kernel: one CTA per bucket sorts its words (low key bits,
//      then index: the stable order) in shared memory: the words are counted
//      into sub-buckets, placed, and ranked within their sub-bucket (or sorted
//      by digits when a sub-bucket is crowded).  FOLD adds up runs of equal
//      keys, in input order unless they are long, and writes at offsets from a
//      look-back over the buckets; a plain sort knows its offsets already.
//
// DRAM traffic: 8 B (histogram) + 32 B per pass + 16 B + 16 B per pair.
// Measured on 2^27 pairs with 36-bit keys (B200): histogram 0.36 ms, partition
// passes 0.80 and 0.86 ms (80% of the measured copy rate), bucket kernel 1.9 ms
// (bound by the latency of its block-wide phases and of the look-back); 3.98 ms
// against 5.90 ms for the stable 7- and 8-bit onesweep passes (1.59 + 1.30 ms:
// eight ballots, a per-warp counter and a look-back per pass) and a bucket
// kernel whose threads each ranked ten words by looping over their sub-buckets
// (2.43 ms).
#include <algorithm>
#include <cstdlib>

#include "lnt_msd.cuh"

namespace lnt {
namespace {

constexpr int kHistThreads = 1024;
constexpr int kMaxT = 15;
// Smallest sort taken, where one cluster does not do it all (more than 49 key
// bits).  Down to 2048 pairs the bucketed path with the skipped fallback behind it
// takes 18-21 us against 33-57 us for the digit passes; below, the histogram and
// one CTA are all there is to gain.
constexpr size_t kMinPairs = 2048;
constexpr double kMaxPerKey = 24.0;
constexpr int kMaxDigits = 256;
// Partition tile: 256 threads x 8 records, four CTAs per SM at 64 registers.
// What matters is that nothing spills: 12 records per thread ran the same
// (0.84 + 0.85 ms for the two passes over 2^27 pairs against 0.81 + 0.86), 16
// per thread spilled and took 1.16 + 1.17 ms.
constexpr int kPartThreads = 256, kPartItems = 8, kPartBlocks = 4;
constexpr int kPartTile = kPartThreads * kPartItems;
constexpr unsigned long long kFlagAgg = 1ull << 62;
constexpr unsigned long long kFlagPre = 2ull << 62;
constexpr unsigned long long kFlagMask = 3ull << 62;
constexpr unsigned long long kValMask = (1ull << 62) - 1ull;

// A bucket's records are counted into 2^SUBB sub-buckets (8-bit counts, four
// to a word), about four per record, so that most records are alone in theirs.
template <int BT, int ITEMS, int SUBB>
struct BucketGeom {
  static constexpr int kBT = BT;
  static constexpr int kWarps = BT / 32;
  static constexpr int kItems = ITEMS;
  static constexpr int kCap = BT * ITEMS;
  static constexpr int kSubBits = SUBB;
  static constexpr int kSubWords = 1 << (SUBB - 2);
  static constexpr int kSubPer = kSubWords / BT;  // count words per thread
  static constexpr int kGroups = kCap / 32;       // 32-position groups
  static constexpr int kMinBlocks = BT >= 512 ? 2 : 4;
  static constexpr size_t smem = (size_t)kCap * 16 + (size_t)kSubWords * 6 + (size_t)kGroups * 8 + 64 * 4;
  static_assert(kSubPer == 8, "one uint4 of 16-bit starts per thread");
};
using GeomLarge = BucketGeom<512, 10, 14>;
using GeomSmall = BucketGeom<256, 10, 13>;
// largest expected bucket (uniform keys): four fifths of the capacity
constexpr double kAvgLarge = 4096.0, kAvgSmall = 2048.0;
constexpr int kSubMax = 48;  // largest sub-bucket ranked by comparing its words
constexpr int kSubThread = 8;  // largest one sorted (and folded) by a single thread

struct MsdCtrl {
  u32* counts;    // 2^T
  u32* start;     // 2^T + 1
  u32* cur1;      // first pass cursors (up to 256)
  u32* cur2;      // second pass cursors (2^T)
  u32* segtile;   // second pass: first tile of every segment (up to 257)
  u32* misc;      // [0] histogram CTAs done, [1] bucket counter, [2] the gate closes, whatever the counts say
  unsigned long long* status;  // 2^T look-back words (FOLD)
  u32* gate;      // 0: every bucket fits a CTA (and no key loses bits), 1: take the LSD path
};

// Loads I keys at positions base + j * stride + tid (those below `end`; 0
// beyond) of the concatenated source and re-keys them.
template <int I>
__device__ __forceinline__ void source_keys(const PairSource& s, u32 base, u32 stride, u32 end, u64 (&k)[I]) {
  const u32 first = base + threadIdx.x;
  const bool all_a = end <= s.na, all_b = base >= s.na;
  u32 in_a = 0;
#pragma unroll
  for (int j = 0; j < I; ++j) {
    const u32 i = first + j * stride;
    k[j] = 0;
    if (all_a || (!all_b && i < s.na)) {
      in_a |= 1u << j;
      if (i < end) k[j] = __ldcs(s.ak + i);
    } else if (i < end) {
      k[j] = __ldcs(s.bk + (i - s.na));
    }
  }
  if (!all_b) rekey_items(k, s.ra, in_a);
  if (!all_a) rekey_items(k, s.rb, ~in_a);
}

// 32-bit counts, one CTA of 1024 threads per SM with eight keys per thread in
// flight: 2^27 keys in 0.36 ms (0.48 with 16-bit counts, whose every increment
// had to be checked, and two CTAs of half the registers).
__global__ void __launch_bounds__(kHistThreads, 1) msd_hist_kernel(const PairSource src, u32 n, int T, int db,
                                                                   int shift, int key_bits, u32 cap, MsdCtrl c) {
  extern __shared__ u32 sh[];  // 2^T counts
  __shared__ bool s_last;
  __shared__ u32 s_w[kHistThreads / 32], s_mx[kHistThreads / 32];
  const int nb = 1 << T;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < nb; i += kHistThreads) sh[i] = 0;
  __syncthreads();
  const u32 bmask = (u32)(nb - 1);
  u64 any = 0;
  constexpr int U = 8;
  // Clustered keys: once a CTA has counted more of one bucket than fits, the rest
  // need not be read.  Looked for after 2, 8, 32 .. rounds, while at least as many
  // are left (2 to 3 us each).
  u32 round = 0, next_look = 2;
  bool closed = false;
  const u32 rounds = (u32)(n / ((u64)gridDim.x * (kHistThreads * U)));
  for (u64 base = (u64)blockIdx.x * (kHistThreads * U); base < n; base += (u64)gridDim.x * (kHistThreads * U)) {
    const u32 end = (u32)min((u64)n, base + kHistThreads * U);
    u64 k[U];
    source_keys<U>(src, (u32)base, kHistThreads, end, k);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if ((u32)base + u * kHistThreads + tid < end) {
        atomicAdd(&sh[(u32)(k[u] >> shift) & bmask], 1u);
        any |= k[u];
      }
    if (++round == next_look && 2 * round <= rounds) {
      next_look *= 4;
      __syncthreads();
      u32 most = 0;
      for (int i = tid; i < nb; i += kHistThreads) most = max(most, sh[i]);
      closed = __syncthreads_or(most > cap) != 0;
      if (closed) break;
    }
  }
  if (closed && tid == 0) atomicOr(&c.misc[2], 1u);
  // bits above the sorted ones (a key >= max_key): the records would lose them
  if (key_bits < 64 && (any >> key_bits) != 0) atomicOr(&c.misc[2], 1u);
  __syncthreads();
  for (int b = tid; b < nb && !closed; b += kHistThreads) {
    const u32 v = sh[b];
    if (v) atomicAdd(&c.counts[b], v);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&c.misc[0], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // ---- last CTA: bucket starts and cursors, the largest bucket ----
  const int per = (nb + kHistThreads - 1) / kHistThreads;
  u32 local = 0, mx = 0;
  for (int j = 0; j < per; ++j) {
    const int b = tid * per + j;
    const u32 v = b < nb ? __ldcg(&c.counts[b]) : 0u;
    local += v;
    mx = max(mx, v);
  }
  u32 inc = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 31) s_w[warp] = inc;
  if (lane == 0) s_mx[warp] = mx;
  __syncthreads();
  u32 run = inc - local;
  for (int w = 0; w < warp; ++w) run += s_w[w];
  const u32 dmask = (1u << db) - 1u;
  for (int j = 0; j < per; ++j) {
    const int b = tid * per + j;
    if (b < nb) {
      c.start[b] = run;
      c.cur2[b] = run;
      if (((u32)b & dmask) == 0u) c.cur1[b >> db] = run;  // a first-pass segment begins here
      run += __ldcg(&c.counts[b]);
    }
  }
  if (tid >= 1 && tid < kGateWords) c.gate[tid] = 0;
  if (tid == 0) {
    u32 m = 0;
    for (int w = 0; w < kHistThreads / 32; ++w) m = max(m, s_mx[w]);
    c.gate[0] = m > cap || __ldcg(&c.misc[2]) != 0u ? 1u : 0u;
    c.start[nb] = n;
  }
  __threadfence_block();
  __syncthreads();
  // ---- tiles of the second pass per segment (at most 256 segments) ----
  const int nseg = nb >> db;
  u32 tiles = 0;
  if (tid < nseg) {
    const u32 s0 = c.start[tid << db], s1 = c.start[(tid + 1) << db];
    tiles = (s1 - s0 + kPartTile - 1) / kPartTile;
  }
  u32 tinc = tiles;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 t = __shfl_up_sync(0xffffffffu, tinc, o);
    if (lane >= o) tinc += t;
  }
  __syncthreads();
  if (lane == 31) s_w[warp] = tinc;
  __syncthreads();
  u32 tb = tinc - tiles;
  for (int w = 0; w < warp; ++w) tb += s_w[w];
  if (tid < nseg) c.segtile[tid] = tb;
  if (tid == nseg) c.segtile[nseg] = tb;
}

template <int THREADS, int ITEMS, int MINB>
struct PartShape {
  static constexpr int kThreads = THREADS, kItems = ITEMS, kMinBlocks = MINB;
  static constexpr int kTile = THREADS * ITEMS;
  static constexpr int kPer = kMaxDigits / THREADS;  // digits per thread
  static constexpr size_t smem = (size_t)kTile * 16 + kMaxDigits * 8 + 128;
};

// One partition pass over records (word, value).  FIRST reads the source and
// builds the words; otherwise the records of every segment (first-pass digit)
// are partitioned among the buckets of that segment.  DIGITS: the digit of
// every staged record is kept beside it (FIRST, when the word has lost it).
template <class P, bool FIRST, bool DIGITS>
__global__ void __launch_bounds__(P::kThreads, P::kMinBlocks)
    partition_kernel(const PairSource src, const ulonglong2* __restrict__ in, ulonglong2* __restrict__ out, u32 n,
                     int ib, int dshift, u32 dmask, int nseg, int db, const MsdCtrl c) {
  if (gated_off(c.gate, 0)) return;  // a bucket is too large: the LSD path runs instead
  constexpr int T = P::kThreads, I = P::kItems, PER = P::kPer;
  extern __shared__ __align__(16) unsigned char smem[];
  ulonglong2* s_r = reinterpret_cast<ulonglong2*>(smem);         // tile records in digit order
  u32* s_cnt = reinterpret_cast<u32*>(s_r + P::kTile);           // per digit: count, then destination - tile start
  u32* s_ts = s_cnt + kMaxDigits;                                // per digit: first slot in the tile
  u32* s_misc = s_ts + kMaxDigits;                               // 32
  unsigned char* s_d = reinterpret_cast<unsigned char*>(s_misc + 32);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int q = 0; q < PER; ++q) s_cnt[q * T + tid] = 0;
  u32 base, tile_n;
  u32* cursor;
  if (FIRST) {
    base = blockIdx.x * (u32)P::kTile;
    tile_n = min((u32)P::kTile, n - base);
    cursor = c.cur1;
  } else {
    if (blockIdx.x >= c.segtile[nseg]) return;
    for (int q = tid; q < nseg; q += T) {  // the segment this tile belongs to
      const u32 t0 = c.segtile[q], t1 = c.segtile[q + 1];
      if (t0 <= blockIdx.x && blockIdx.x < t1) {
        const u32 s0 = c.start[(u32)q << db], s1 = c.start[(u32)(q + 1) << db];
        const u32 b = s0 + (blockIdx.x - t0) * (u32)P::kTile;
        s_misc[16] = (u32)q;
        s_misc[17] = b;
        s_misc[18] = min((u32)P::kTile, s1 - b);
      }
    }
  }
  __syncthreads();
  if (!FIRST) {
    cursor = c.cur2 + (s_misc[16] << db);
    base = s_misc[17];
    tile_n = s_misc[18];
  }
  u64 w[I];
  double v[I];
  u32 slot[I];
  if (FIRST) {
    source_keys<I>(src, base, (u32)T, base + tile_n, w);
    const bool all_a = base + tile_n <= src.na, all_b = base >= src.na;
#pragma unroll
    for (int j = 0; j < I; ++j) {
      const u32 p = j * T + tid, i = base + p;
      v[j] = 0.0;
      if (all_a || (!all_b && i < src.na)) {
        if (p < tile_n) v[j] = __ldcs(src.av + i);
      } else if (p < tile_n) {
        v[j] = __ldcs(src.bv + (i - src.na));
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < I; ++j) {
      const u32 p = j * T + tid;
      ulonglong2 r = make_ulonglong2(0, 0);
      if (p < tile_n) r = __ldcs(in + base + p);
      w[j] = r.x;
      v[j] = __longlong_as_double((long long)r.y);
    }
  }
  // rank within the digit by one shared atomic per pair; one per warp and
  // item where the warp's 32 pairs share their digit, as in key-ordered input
  // (32 atomics on one address would take turns)
  const u32 d0 = (u32)(w[0] >> dshift) & dmask;
  if (__all_sync(0xffffffffu, d0 == __shfl_sync(0xffffffffu, d0, 0))) {
#pragma unroll
    for (int j = 0; j < I; ++j) {
      const u32 p = j * T + tid;
      const u32 d = (u32)(w[j] >> dshift) & dmask;
      const u32 df = __shfl_sync(0xffffffffu, d, 0);
      if (__all_sync(0xffffffffu, d == df && p < tile_n)) {
        u32 b = 0;
        if (lane == 0) b = atomicAdd(&s_cnt[df], 32u);
        slot[j] = __shfl_sync(0xffffffffu, b, 0) + lane;
      } else {
        slot[j] = p < tile_n ? atomicAdd(&s_cnt[d], 1u) : 0u;
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < I; ++j) {
      const u32 p = j * T + tid;
      slot[j] = p < tile_n ? atomicAdd(&s_cnt[(u32)(w[j] >> dshift) & dmask], 1u) : 0u;
    }
  }
  __syncthreads();
  {  // reserve room in each digit's range; exclusive scan of the counts
    u32 cnt[PER], g[PER], sum = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      cnt[q] = s_cnt[tid * PER + q];
      g[q] = cnt[q] ? atomicAdd(cursor + tid * PER + q, cnt[q]) : 0u;  // (digits beyond dmask have no pairs)
      sum += cnt[q];
    }
    u32 inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) s_misc[warp] = inc;
    __syncthreads();
    u32 ts = inc - sum;
#pragma unroll
    for (int q = 0; q < T / 32; ++q) ts += q < warp ? s_misc[q] : 0u;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      s_ts[tid * PER + q] = ts;
      s_cnt[tid * PER + q] = g[q] - ts;
      ts += cnt[q];
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < I; ++j) {
    const u32 p = j * T + tid;
    if (p < tile_n) {
      const u32 d = (u32)(w[j] >> dshift) & dmask;
      const u32 q = s_ts[d] + slot[j];
      u64 x = w[j];
      double y = v[j];
      if (FIRST) {
        x = (x << ib) | (u64)(base + p);
        if (base + p >= src.na) y *= src.bscale;
        if (DIGITS) s_d[q] = (unsigned char)d;
      }
      s_r[q] = make_ulonglong2(x, (u64)__double_as_longlong(y));
    }
  }
  __syncthreads();
  const int wshift = FIRST ? dshift + ib : dshift;
#pragma unroll
  for (int j = 0; j < I; ++j) {
    const u32 p = j * T + tid;
    if (p < tile_n) {
      const ulonglong2 r = s_r[p];
      const u32 d = DIGITS ? (u32)s_d[p] : (u32)(r.x >> wshift) & dmask;
      out[s_cnt[d] + p] = r;
    }
  }
}

__device__ __forceinline__ u64 word_of(const ulonglong2& r) { return r.x; }
__device__ __forceinline__ u64 word_of(u64 w) { return w; }

// Sorts the cnt records s_r by word, by digits of eight bits from the lowest up,
// without those in which no two words differ.  Stably: a warp takes consecutive
// records, matches their digits and counts per warp and digit.  s_cnt: a word per
// warp and digit; s_tmp: 36 words.  (2^21 pairs, 95% of them of 2^12 keys: 152 us
// in all, 209 with a merge sort, whose rounds search in shared memory.)
template <int BT, int I, class R>
__device__ __forceinline__ void sort_by_digits(R* s_r, u32* s_cnt, u32* s_tmp, u32 cnt) {
  constexpr int W = BT / 32;
  constexpr u32 FULL = 0xffffffffu;
  const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const u32 items = (cnt + BT - 1) / BT, from = warp * items * 32;
  u32* mine = s_cnt + warp * 256;
  unsigned long long* s_diff = reinterpret_cast<unsigned long long*>(s_tmp + 32);
  __syncthreads();
  if (tid == 0) *s_diff = 0ull;
  __syncthreads();
  const u64 w0 = word_of(s_r[0]);
  u64 diff = 0;
  for (u32 p = tid; p < cnt; p += BT) diff |= word_of(s_r[p]) ^ w0;
  const u32 lo = __reduce_or_sync(FULL, (u32)diff), hi = __reduce_or_sync(FULL, (u32)(diff >> 32));
  if (lane == 0) atomicOr(s_diff, (unsigned long long)hi << 32 | lo);
  __syncthreads();
  diff = *s_diff;
  for (int shift = 0; shift < 64; shift += 8) {
    if (((diff >> shift) & 0xFFull) == 0ull) continue;
    R x[I];
    u32 pos[(I + 1) / 2];  // 16 bits per item
    for (u32 d = lane; d < 256; d += 32) mine[d] = 0u;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < I; ++j) {
      if (j >= (int)items) break;
      const u32 p = from + j * 32 + lane;
      const bool valid = p < cnt;
      if (valid) x[j] = s_r[p];
      const u32 d = valid ? (u32)(word_of(x[j]) >> shift) & 0xFFu : 0u;
      u32 peers = __ballot_sync(FULL, valid);  // the lanes with the same digit
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const u32 m = __ballot_sync(FULL, (d >> b) & 1u);
        peers &= (d >> b) & 1u ? m : ~m;
      }
      u32 at = 0;
      if (valid) at = mine[d];
      __syncwarp();
      if (valid && lane == (u32)__ffs(peers) - 1u) mine[d] = at + __popc(peers);
      __syncwarp();
      at += __popc(peers & ((1u << lane) - 1u));
      pos[j / 2] = j & 1 ? pos[j / 2] | (at << 16) : at;
    }
    __syncthreads();
    u32 run = 0, inc = 0;
    if (tid < 256) {
      for (int q = 0; q < W; ++q) {  // records of this digit in the warps before
        const u32 c = s_cnt[q * 256 + tid];
        s_cnt[q * 256 + tid] = run;
        run += c;
      }
      inc = run;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u32 t = __shfl_up_sync(FULL, inc, o);
        if (lane >= (u32)o) inc += t;
      }
      if (lane == 31) s_tmp[warp] = inc;
    }
    __syncthreads();
    if (tid < 256) {  // and those of the digits before
      u32 start = inc - run;
      for (u32 q = 0; q < warp; ++q) start += s_tmp[q];
      for (int q = 0; q < W; ++q) s_cnt[q * 256 + tid] += start;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < I; ++j) {
      if (j >= (int)items) break;
      if (from + j * 32 + lane < cnt)
        s_r[mine[(u32)(word_of(x[j]) >> shift) & 0xFFu] + ((pos[j / 2] >> (16 * (j & 1))) & 0xFFFFu)] = x[j];
    }
    __syncthreads();
  }
}

// Sorts the sub-buckets where some have more than kSubThread records, which a
// single thread would sort for long (20 equal keys per sub-bucket: 2000 pairs 69
// us, 27 like this): every record counts the smaller words of its sub-bucket and
// goes to its rank.  sub_of(word): the word's sub-bucket.
template <int BT, int I, class R, class SubOf>
__device__ __forceinline__ void rank_sub_buckets(R* s_r, const u32* s_cnt, const unsigned short* s_base, u32 cnt,
                                              const SubOf sub_of) {
  const int tid = threadIdx.x;
  R x[I];
  u32 to[(I + 1) / 2];  // 16 bits per item
#pragma unroll
  for (int j = 0; j < I; ++j) {
    const u32 p = j * BT + tid;
    u32 at = p;
    if (p < cnt) {
      x[j] = s_r[p];
      const u64 w = word_of(x[j]);
      const u32 sub = sub_of(w), sh = 8u * (sub & 3u), c4 = s_cnt[sub >> 2], k = (c4 >> sh) & 0xFFu;
      if (k > 1u) {
        const u32 lo = s_base[sub >> 2] + __dp4a(c4 & ((1u << sh) - 1u), 0x01010101u, 0u);
        u32 rank = 0;
        for (u32 q = 0; q < k; ++q) rank += word_of(s_r[lo + q]) < w ? 1u : 0u;
        at = lo + rank;
      }
    }
    to[j / 2] = j & 1 ? to[j / 2] | (at << 16) : at;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < I; ++j) {
    const u32 p = j * BT + tid, at = (to[j / 2] >> (16 * (j & 1))) & 0xFFFFu;
    if (p < cnt && at != p) s_r[at] = x[j];
  }
  __syncthreads();
}

// The run of equal keys that starts at each head of row g (32 sorted positions,
// one warp): adds the rest of the run to the head's sum, and sets anynz when
// something in it is not zero.  heads: the rows' head masks (valid positions
// only), rows of them, cnt positions.  A run that ends in its own row or the
// next is added up in input order by the head's lane; a longer one, which only
// the row's last head can have, by the whole warp, lane by lane over the rows
// and then over the lanes (one key 20,000 times: 1470 us by one lane).
template <class Val>
__device__ __forceinline__ void fold_row(const u32* heads, u32 rows, u32 g, u32 cnt, bool head, double& sum,
                                         bool& anynz, const Val& val) {
  constexpr u32 FULL = 0xffffffffu;
  const u32 lane = threadIdx.x & 31, p = g * 32 + lane;
  bool far = false;
  if (head) {
    const u32 later = lane == 31 ? 0u : heads[g] >> (lane + 1);
    u32 end = cnt;
    if (later) {
      end = p + __ffs(later);
    } else if (g + 1 < rows) {
      const u32 next = heads[g + 1];
      far = next == 0u;
      if (next) end = (g + 1) * 32 + __ffs(next) - 1;
    }
    if (!far) {
      for (u32 q = p + 1; q < end; ++q) {
        const double y = val(q);
        sum += y;
        anynz |= y != 0.0;
      }
    }
  }
  const u32 who = __ballot_sync(FULL, far);
  if (who == 0u) return;
  const u32 from = __ffs(who) - 1;
  double part = -0.0;  // the additive identity that keeps the sign of a zero
  bool nz = false;
  auto add = [&](u32 q) {
    const double y = val(q);
    part += y;
    nz |= y != 0.0;
  };
  if (lane > from && p < cnt) add(p);
  for (u32 r0 = g + 1; r0 < rows; r0 += 32) {
    const u32 mine = r0 + lane < rows ? heads[r0 + lane] : 0u;
    const u32 some = __ballot_sync(FULL, mine != 0u);
    const u32 whole = min(some ? __ffs(some) - 1u : 32u, rows - r0);  // rows without a head
    u32 r = r0;
    for (; r + 4 <= r0 + whole && (r + 4) * 32 <= cnt; r += 4) {
      double y[4];
#pragma unroll
      for (u32 u = 0; u < 4; ++u) y[u] = val((r + u) * 32 + lane);
#pragma unroll
      for (u32 u = 0; u < 4; ++u) {
        part += y[u];
        nz |= y[u] != 0.0;
      }
    }
    for (; r < r0 + whole; ++r)
      if (r * 32 + lane < cnt) add(r * 32 + lane);
    if (some) {
      const u32 last = __shfl_sync(FULL, mine, whole);  // the run ends before this row's first head
      if (lane < __ffs(last) - 1u) add((r0 + whole) * 32 + lane);
      break;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(FULL, part, o);
  nz = __any_sync(FULL, nz);
  if (lane == from) {
    sum += part;
    anynz |= nz;
  }
}

// Folds the cnt sorted records of a whole bucket: every head's value becomes the
// sum of its run, and s_kept the mask of the heads that are written.  s_head:
// room for a mask per 32 positions; first: the bucket begins the sorted array.
template <int BT>
__device__ __forceinline__ void fold_bucket(ulonglong2* s_r, u32* s_head, u32* s_kept, u32 cnt, int ib,
                                         int skip_zero_heads, bool first) {
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rows = (cnt + 31) / 32;
  for (u32 g = warp; g < rows; g += BT / 32) {
    const u32 p = g * 32 + lane;
    const u32 m =
        __ballot_sync(0xffffffffu, p < cnt && (p == 0 || ((s_r[p > 0 ? p - 1 : 0].x ^ s_r[p].x) >> ib) != 0));
    if (lane == 0) s_head[g] = m;
  }
  __syncthreads();
  for (u32 g = warp; g < rows; g += BT / 32) {
    const u32 p = g * 32 + lane;
    const bool head = (s_head[g] >> lane & 1u) != 0u;
    double sum = head ? __longlong_as_double((long long)s_r[p].y) : 0.0;
    bool anynz = sum != 0.0;
    fold_row(s_head, rows, g, cnt, head, sum, anynz,
             [&](u32 q) { return __longlong_as_double((long long)s_r[q].y); });
    if (head) s_r[p].y = (u64)__double_as_longlong(sum);  // (nobody else reads a head's value)
    const u32 kept = __ballot_sync(0xffffffffu, head && (!skip_zero_heads || anynz || (first && p == 0)));
    if (lane == 0) s_kept[g] = kept;
  }
}

// Sorts and folds a bucket that has a sub-bucket too long for a thread, or that is
// crowded.  (A function of its own: such buckets are rare, and their registers
// would be taken from the others.)
template <class G, bool FOLD>
__device__ __noinline__ void long_bucket(ulonglong2* s_r, u32* s_cnt, unsigned short* s_base, u32* s_head, u32* s_kept,
                                         u32 cnt, int sshift, bool crowded, int ib, int skip_zero_heads, bool first) {
  static_assert(G::kWarps * 256 <= G::kSubWords, "the counts of the sub-buckets hold one per warp and digit");
  if (crowded) sort_by_digits<G::kBT, G::kItems>(s_r, s_cnt, reinterpret_cast<u32*>(s_base), cnt);
  else rank_sub_buckets<G::kBT, G::kItems>(s_r, s_cnt, s_base, cnt, [=](u64 w) { return (u32)(w >> sshift); });
  if (FOLD) fold_bucket<G::kBT>(s_r, s_head, s_kept, cnt, ib, skip_zero_heads, first);
}

// Sorts the k records of one sub-bucket by word (one thread); FOLD adds up its
// runs of equal keys in that (input) order into their first record and clears
// the kept bits of the others and of the dropped ones.  `at`: the position of
// r[0] in the bucket; first: it is the first of the whole sorted array.
template <bool FOLD>
__device__ __forceinline__ void fold_sub_bucket(ulonglong2* r, int k, int ib, int skip_zero_heads, bool first, u32 at,
                                                u32* kept) {
  for (int i = 1; i < k; ++i) {  // insertion sort
    const ulonglong2 x = r[i];
    int q = i;
    for (; q > 0; --q) {
      const ulonglong2 y = r[q - 1];
      if (y.x < x.x) break;
      r[q] = y;
    }
    if (q != i) r[q] = x;
  }
  if (!FOLD) return;
  for (int i = 0; i < k;) {
    const u64 low = r[i].x >> ib;
    double sum = __longlong_as_double((long long)r[i].y);
    bool anynz = sum != 0.0;
    int q = i + 1;
    for (; q < k && (r[q].x >> ib) == low; ++q) {
      const double y = __longlong_as_double((long long)r[q].y);
      sum += y;
      anynz |= y != 0.0;
      atomicAnd(&kept[(at + q) >> 5], ~(1u << ((at + q) & 31)));
    }
    if (q > i + 1) r[i].y = (u64)__double_as_longlong(sum);
    if (skip_zero_heads && !anynz && !(first && i == 0)) atomicAnd(&kept[(at + i) >> 5], ~(1u << ((at + i) & 31)));
    i = q;
  }
}

template <class G, bool FOLD>
__global__ void __launch_bounds__(G::kBT, G::kMinBlocks)
    bucket_sort_kernel(const ulonglong2* __restrict__ rec, const MsdCtrl c, int T, int shift, int ib,
                       int skip_zero_heads, u64* __restrict__ out_k, double* __restrict__ out_v,
                       u64* __restrict__ d_nout) {
  if (gated_off(c.gate, 0)) return;
  constexpr int BT = G::kBT, I = G::kItems, W = G::kWarps, P2 = (I + 1) / 2;
  extern __shared__ __align__(16) unsigned char smem[];
  ulonglong2* s_r = reinterpret_cast<ulonglong2*>(smem);       // kCap records in sub-bucket order
  u32* s_cnt = reinterpret_cast<u32*>(s_r + G::kCap);              // sub-bucket counts, four to a word
  unsigned short* s_base = reinterpret_cast<unsigned short*>(s_cnt + G::kSubWords);  // records before each word's
  u32* s_kept = reinterpret_cast<u32*>(s_base + G::kSubWords);     // per 32 positions: kept mask
  u32* s_pre = s_kept + G::kGroups;                                // per 32 positions: kept before them
  u32* s_misc = s_pre + G::kGroups;                                // 64
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int sb = min(shift, G::kSubBits);
  const int sshift = ib + shift - sb;
  const u64 wmask = ib + shift >= 64 ? ~0ull : (1ull << (ib + shift)) - 1ull;
  if (FOLD && tid == 0) s_misc[0] = atomicAdd(&c.misc[1], 1u);
#pragma unroll
  for (int j = 0; j < G::kSubPer; ++j) s_cnt[j * BT + tid] = 0;
  if (tid == 0) s_misc[1] = 0;
  __syncthreads();
  const u32 b = FOLD ? s_misc[0] : blockIdx.x;  // FOLD: in order of arrival, for the look-back
  const u32 start = c.start[b];
  const u32 cnt = min(c.start[b + 1] - start, (u32)G::kCap);  // (the gate is open: no bucket exceeds kCap)
  rec += start;
  if (FOLD)  // every position is kept until its record turns out not to be the first of its run
    for (int x = tid; x < G::kGroups; x += BT)
      s_kept[x] = x * 32 + 32 <= cnt ? ~0u : x * 32 < cnt ? (1u << (cnt - x * 32)) - 1u : 0u;
  ulonglong2 r[I];
  u32 pos[P2];  // 16 bits per item
#pragma unroll
  for (int j = 0; j < I; ++j) {
    const u32 p = j * BT + tid;
    r[j] = make_ulonglong2(~0ull, 0);
    if (p < cnt) {
      r[j] = __ldcs(rec + p);
      r[j].x &= wmask;
    }
  }
  {  // count the sub-buckets; slot of every record in its own
#pragma unroll
    for (int j = 0; j < I; ++j) {
      const u32 p = j * BT + tid;
      const u32 sub = (u32)(r[j].x >> sshift), sh = 8u * (sub & 3u);
      const u32 slot = p < cnt ? (atomicAdd(&s_cnt[sub >> 2], 1u << sh) >> sh) & 0xFFu : 0u;
      pos[j / 2] = j & 1 ? pos[j / 2] | (slot << 16) : slot;
    }
    u32 most = 0;
#pragma unroll
    for (int j = 0; j < P2; ++j) most = __vmaxu2(most, pos[j]);
    most = max(most & 0xFFFFu, most >> 16);
    // bit 0: some sub-bucket is too long for a thread; bit 1, crowded (some slot
    // at the limit): the counts may have run over, and are not used
    if (most >= (u32)kSubThread) atomicOr(&s_misc[1], most >= (u32)kSubMax ? 3u : 1u);
  }
  __syncthreads();
  {  // records before every count word
    u32 sum = 0;
    u32 c8[8];
#pragma unroll
    for (int j = 0; j < 8; j += 4) {
      const uint4 q = *reinterpret_cast<const uint4*>(&s_cnt[tid * 8 + j]);
      c8[j] = __dp4a(q.x, 0x01010101u, 0u);
      c8[j + 1] = __dp4a(q.y, 0x01010101u, 0u);
      c8[j + 2] = __dp4a(q.z, 0x01010101u, 0u);
      c8[j + 3] = __dp4a(q.w, 0x01010101u, 0u);
      sum += c8[j] + c8[j + 1] + c8[j + 2] + c8[j + 3];
    }
    u32 inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) s_misc[8 + warp] = inc;
    __syncthreads();
    u32 run = inc - sum;
#pragma unroll
    for (int q = 0; q < W; ++q) run += q < warp ? s_misc[8 + q] : 0u;
    u32 pk[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const u32 lo = run;
      run += c8[2 * j];
      pk[j] = (lo & 0xFFFFu) | (run << 16);
      run += c8[2 * j + 1];
    }
    *reinterpret_cast<uint4*>(&s_base[tid * 8]) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
  }
  __syncthreads();
  const u32 how = s_misc[1];
  const bool ranked = how < 2u;
#pragma unroll
  for (int j = 0; j < I; ++j) {  // place every record in its sub-bucket (crowded: as they are, to be sorted)
    const u32 p = j * BT + tid;
    u32 q = p;
    if (ranked && p < cnt) {
      const u32 sub = (u32)(r[j].x >> sshift), sh = 8u * (sub & 3u), c4 = s_cnt[sub >> 2];
      q = s_base[sub >> 2] + __dp4a(c4 & ((1u << sh) - 1u), 0x01010101u, 0u) +
          ((pos[j / 2] >> (16 * (j & 1))) & 0xFFFFu);
      // alone in its sub-bucket and zero: dropped (unless it is the first of all)
      if (FOLD && skip_zero_heads && ((c4 >> sh) & 0xFFu) == 1u && __longlong_as_double((long long)r[j].y) == 0.0 &&
          start + q != 0)
        atomicAnd(&s_kept[q >> 5], ~(1u << (q & 31)));
    }
    s_r[q] = r[j];
  }
  __syncthreads();
  if (how == 0u) {
    // sort (and fold) the sub-buckets of more than one record, each by one
    // thread: about one per thread, of two records.  Count words go to the
    // threads in turn, so that each gets its share also when the key has
    // fewer bits than there are sub-buckets.
    u32 todo = 0;  // bit 4 j + i: count i of word j * BT + tid is above 1
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const u32 gt = __vcmpgtu4(s_cnt[j * BT + tid], 0x01010101u) & 0x08040201u;
      todo |= ((gt | (gt >> 8) | (gt >> 16) | (gt >> 24)) & 0xFu) << (4 * j);
    }
    while (todo) {
      const int i = __ffs(todo) - 1, sh = 8 * (i & 3);
      todo &= todo - 1u;
      const u32 c4 = s_cnt[(i >> 2) * BT + tid];
      const u32 lo = s_base[(i >> 2) * BT + tid] + __dp4a(c4 & ((1u << sh) - 1u), 0x01010101u, 0u);
      const u32 k = (c4 >> sh) & 0xFFu;
      const ulonglong2 e0 = s_r[lo], e1 = s_r[lo + 1];
      if (k == 2) {  // nearly always
        const bool swap = e1.x < e0.x;
        const ulonglong2 f = swap ? e1 : e0, g = swap ? e0 : e1;
        if (FOLD) {
          const double x = __longlong_as_double((long long)f.y), y = __longlong_as_double((long long)g.y);
          const bool equal = ((f.x ^ g.x) >> ib) == 0;
          u32 drop = equal ? 2u : 0u;  // bit q: position lo + q is not written
          if (skip_zero_heads) {
            if (x == 0.0 && !(equal && y != 0.0) && start + lo != 0) drop |= 1u;
            if (!equal && y == 0.0) drop |= 2u;
          }
          if (drop & 1u) atomicAnd(&s_kept[lo >> 5], ~(1u << (lo & 31)));
          if (drop & 2u) atomicAnd(&s_kept[(lo + 1) >> 5], ~(1u << ((lo + 1) & 31)));
          if (equal) {
            s_r[lo] = make_ulonglong2(f.x, (u64)__double_as_longlong(x + y));
          } else if (swap) {
            s_r[lo] = f;
            s_r[lo + 1] = g;
          }
        } else if (swap) {
          s_r[lo] = f;
          s_r[lo + 1] = g;
        }
      } else {
        fold_sub_bucket<FOLD>(s_r + lo, (int)k, ib, skip_zero_heads, start + lo == 0, lo, s_kept);
      }
    }
  } else {
    long_bucket<G, FOLD>(s_r, s_cnt, s_base, s_pre, s_kept, cnt, sshift, !ranked, ib, skip_zero_heads, start == 0);
  }
  __syncthreads();
  const u64 prefix = (u64)b << shift;
  if (!FOLD) {
#pragma unroll
    for (int j = 0; j < I; ++j) {
      const u32 p = j * BT + tid;
      if (p < cnt) {
        const ulonglong2 e = s_r[p];
        __stcs(out_k + start + p, prefix | (e.x >> ib));
        __stcs(out_v + start + p, __longlong_as_double((long long)e.y));
      }
    }
    return;
  }
  // ---- warp 0: kept positions before every group of 32; output offset by
  // decoupled look-back over buckets
  if (warp == 0) {
    constexpr int R = (G::kGroups + 31) / 32;
    u32 total = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int x = r * 32 + lane;
      const u32 k = x < G::kGroups ? __popc(s_kept[x]) : 0u;
      u32 inc = k;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      if (x < G::kGroups) s_pre[x] = total + inc - k;
      total += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0)
      *reinterpret_cast<volatile unsigned long long*>(&c.status[b]) = (b == 0 ? kFlagPre : kFlagAgg) | total;
    unsigned long long off = 0;
    if (b != 0) {
      int base = (int)b - 1;
      u32 spins = 0;
      while (base >= 0) {
        const int p = base - lane;
        const unsigned long long wv =
            p >= 0 ? *reinterpret_cast<const volatile unsigned long long*>(&c.status[p]) : kFlagPre;
        const unsigned long long f = wv & kFlagMask;
        const u32 notready = __ballot_sync(0xffffffffu, f == 0);
        const u32 pre = __ballot_sync(0xffffffffu, f == kFlagPre);
        const int first_nr = notready ? __ffs(notready) - 1 : 32;
        const int first_pre = pre ? __ffs(pre) - 1 : 32;
        const int take = first_pre < first_nr ? first_pre + 1 : first_nr;
        unsigned long long x = lane < take ? (wv & kValMask) : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        off += x;
        if (first_pre < first_nr) break;
        base -= first_nr;
        if (first_nr < 32 && ++spins > spin_limit()) {
          latch_error(kErrReduceLookback);
          break;
        }
      }
      if (lane == 0) *reinterpret_cast<volatile unsigned long long*>(&c.status[b]) = kFlagPre | (off + total);
    }
    if (lane == 0) {
      *reinterpret_cast<unsigned long long*>(&s_misc[2]) = off;
      if (b == (1u << T) - 1u) *d_nout = off + total;
    }
  }
  __syncthreads();
  const unsigned long long off = *reinterpret_cast<const unsigned long long*>(&s_misc[2]);
#pragma unroll
  for (int j = 0; j < I; ++j) {
    const u32 m = s_kept[j * W + warp];
    if (m & (1u << lane)) {
      const ulonglong2 e = s_r[j * BT + tid];
      const u64 o = off + s_pre[j * W + warp] + __popc(m & ((1u << lane) - 1u));
      __stcs(out_k + o, prefix | (e.x >> ib));
      __stcs(out_v + o, __longlong_as_double((long long)e.y));
    }
  }
}

// ---- small sorts: one cluster, one launch --------------------------------------
// Up to 20480 pairs.  Every CTA of a cluster of C reads all keys and keeps those
// of its own range (the c-th part of [0, max_key)), so that it knows without
// asking how many lie before; a single CTA could hold all pairs, whatever their
// distribution.  It sorts its words (key << 15 | index) in shared memory as the
// bucket kernel does, fetches their values, and writes once the whole cluster has
// read its input (the output may be the input).  FOLD exchanges the CTAs' output counts through distributed
// shared memory.  Bound by latency (B200, replayed in a graph,
// 20 to 41 key bits, evenly spread): 2048 pairs 8-10 us, 10,000 14.5, 20,000 18.6,
// against 20.6 to 22.7 us for histogram, partition, buckets and the skipped path
// behind them; one CTA alone takes 12.5, 20.6 and 33 us.  (Enqueued one by one,
// sort_reduce of 20,000 pairs: distinct keys 26 us, 100 keys 51, one key 56.)
constexpr int kOneThreads = 1024, kOneItems = 20, kOneCap = kOneThreads * kOneItems;
constexpr int kOneIb = 15;       // index bits (kOneCap < 2^15)
constexpr int kOneSubBits = 15;  // 2^15 sub-buckets: 8 count words per thread
constexpr int kOneSubWords = 1 << (kOneSubBits - 2);
constexpr int kOneGroups = kOneCap / 32;
constexpr size_t kOneSmem = (size_t)kOneCap * 8 + (size_t)kOneSubWords * 6 + (size_t)kOneGroups * 12 + 64 * 4;
static_assert(kOneSubWords == 8 * kOneThreads, "eight count words per thread");

__device__ __forceinline__ u32 cluster_rank() {
  u32 r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
  cluster_arrive();
  cluster_wait();
}
// *(p in the shared memory of CTA `rank`) = v
__device__ __forceinline__ void st_cluster(u32* p, u32 rank, u32 v) {
  u32 at;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(at)
               : "r"((u32)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}

// Exclusive sum over the CTA (kOneThreads threads); s: 32 words.
__device__ __forceinline__ u32 one_sum(u32 v, u32* s, u32* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  u32 inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) s[warp] = inc;
  __syncthreads();
  u32 w = s[lane];  // every warp scans the warps' sums
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 t = __shfl_up_sync(0xffffffffu, w, o);
    if (lane >= o) w += t;
  }
  *total = __shfl_sync(0xffffffffu, w, 31);
  const u32 before = __shfl_sync(0xffffffffu, w, warp == 0 ? 0 : warp - 1);
  return (warp == 0 ? 0u : before) + inc - v;
}

// As long_bucket, without the fold; a crowded CTA with one key throughout, and all of its pairs, has
// them in input order.
__device__ __noinline__ void small_sort_long(u64* s_w, u32* s_cnt, unsigned short* s_base, u32 n, u32 cnt,
                                             u64 first_key, int sshift, bool crowded) {
  constexpr int BT = kOneThreads;
  static_assert(BT / 32 * 256 <= kOneSubWords, "the counts of the sub-buckets hold one per warp and digit");
  if (!crowded) {
    rank_sub_buckets<BT, kOneItems>(s_w, s_cnt, s_base, cnt, [=](u64 x) {
      return min((u32)(((x >> kOneIb) - first_key) >> sshift), (u32)(4 * kOneSubWords - 1));
    });
    return;
  }
  const u64 key = s_w[0] >> kOneIb;
  bool other = false;
  for (u32 p = threadIdx.x; p < cnt; p += BT) other = other || s_w[p] >> kOneIb != key;
  if (__syncthreads_or(other) == 0 && cnt == n) {
    for (u32 p = threadIdx.x; p < cnt; p += BT) s_w[p] = key << kOneIb | p;
    __syncthreads();
  } else {
    sort_by_digits<BT, kOneItems>(s_w, s_cnt, reinterpret_cast<u32*>(s_base), cnt);
  }
}

template <bool FOLD>
__global__ void __launch_bounds__(kOneThreads, 1)
    small_sort_kernel(const PairSource src, u32 n, int key_bits, u64 width, int sshift, u32 C, int skip_zero_heads,
                      u64* out_k, double* out_v, u64* d_nout) {
  constexpr int BT = kOneThreads, I = kOneItems, ib = kOneIb;
  extern __shared__ __align__(16) unsigned char smem[];
  u64* s_w = reinterpret_cast<u64*>(smem);
  u32* s_cnt = reinterpret_cast<u32*>(s_w + kOneCap);            // sub-bucket counts, four to a word
  unsigned short* s_base = reinterpret_cast<unsigned short*>(s_cnt + kOneSubWords);
  u32* s_head = reinterpret_cast<u32*>(s_base + kOneSubWords);   // per 32 positions: first of their runs
  u32* s_kept = s_head + kOneGroups;
  u32* s_pre = s_kept + kOneGroups;
  u32* s_misc = s_pre + kOneGroups;  // [0, 32) sums, [40] crowded, [41] kept here, [42] before, [43] long
                                     // sub-buckets, [48, 56) CTA totals
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const u32 le = lane == 31 ? ~0u : (2u << lane) - 1u;
  const u32 rank = C > 1 ? cluster_rank() : 0u;
  if (FOLD && C > 1) cluster_arrive();  // (this CTA runs: its shared memory may be written to)
  const u64 kmask = (1ull << key_bits) - 1ull;
  const u64 first_key = width * rank, end_key = rank + 1 == C ? ~0ull : first_key + width;
#pragma unroll
  for (int j = 0; j < 8; ++j) s_cnt[j * BT + tid] = 0;
  if (tid >= 40 && tid < 44) s_misc[tid] = 0;
  __syncthreads();
  // ---- this CTA's words, in any order; how many keys lie before them ----------
  u64 high = 0;
  u32 before = 0;
#pragma unroll 1
  for (u32 base = 0; base < n; base += 5 * BT) {
    u64 k[5];
    source_keys<5>(src, base, (u32)BT, n, k);
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const u32 p = base + j * BT + tid;
      high |= k[j] & ~kmask;
      const u64 key = k[j] & kmask;
      const bool mine = p < n && key >= first_key && key < end_key;
      before += p < n && key < first_key ? 1u : 0u;
      const u32 m = __ballot_sync(0xffffffffu, mine);
      if (m == 0u) continue;
      u32 at = 0;
      if (lane == 0) at = atomicAdd(&s_misc[41], __popc(m));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (mine) s_w[at + __popc(m & (le >> 1))] = (key << ib) | p;
    }
  }
  before = __reduce_add_sync(0xffffffffu, before);
  if (lane == 0 && before) atomicAdd(&s_misc[42], before);
  // keys with bits above the sorted ones keep them: they are read again below
  const bool wide = __syncthreads_or(high != 0) != 0;
  const u32 cnt = s_misc[41], start = s_misc[42];
  const int items = (int)((cnt + BT - 1) / BT);  // (uniform; a handful, all only when every key is here)
  u64 w[I];
  u32 pos[I / 2], most = 0;
#pragma unroll
  for (int j = 0; j < I; ++j) {
    if (j >= items) break;
    const u32 p = j * BT + tid;
    w[j] = p < cnt ? s_w[p] : ~0ull;
    u32 slot = 0;
    const u32 sub =
        p < cnt ? min((u32)(((w[j] >> ib) - first_key) >> sshift), (u32)(4 * kOneSubWords - 1)) : ~0u;
    const u32 sh = 8u * (sub & 3u);
    // (keys that gather in one CTA may gather in one sub-bucket: one atomic per warp)
    const u32 sub0 = __shfl_sync(0xffffffffu, sub, 0);
    if (__all_sync(0xffffffffu, items > 5 && sub != ~0u && sub == sub0)) {
      if (lane == 0) slot = (atomicAdd(&s_cnt[sub >> 2], 32u << sh) >> sh) & 0xFFu;
      slot = __shfl_sync(0xffffffffu, slot, 0) + lane;
    } else if (p < cnt) {
      slot = (atomicAdd(&s_cnt[sub >> 2], 1u << sh) >> sh) & 0xFFu;
    }
    pos[j / 2] = j & 1 ? pos[j / 2] | (slot << 16) : slot;
    most = max(most, slot);
  }
  if (most >= (u32)kSubThread) s_misc[43] = 1;
  if (most >= (u32)kSubMax) s_misc[40] = 1;  // crowded: the counts may have run over, and are not used
  __syncthreads();
  {  // records before every count word
    u32 c8[8], sum = 0, total;
#pragma unroll
    for (int j = 0; j < 8; j += 4) {
      const uint4 q = *reinterpret_cast<const uint4*>(&s_cnt[tid * 8 + j]);
      c8[j] = __dp4a(q.x, 0x01010101u, 0u);
      c8[j + 1] = __dp4a(q.y, 0x01010101u, 0u);
      c8[j + 2] = __dp4a(q.z, 0x01010101u, 0u);
      c8[j + 3] = __dp4a(q.w, 0x01010101u, 0u);
      sum += c8[j] + c8[j + 1] + c8[j + 2] + c8[j + 3];
    }
    u32 run = one_sum(sum, s_misc, &total);
    u32 pk[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const u32 lo = run;
      run += c8[2 * j];
      pk[j] = (lo & 0xFFFFu) | (run << 16);
      run += c8[2 * j + 1];
    }
    *reinterpret_cast<uint4*>(&s_base[tid * 8]) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
  }
  __syncthreads();
  const bool ranked = s_misc[40] == 0;
  if (ranked) {
#pragma unroll
    for (int j = 0; j < I; ++j) {
      if (j >= items) break;
      if (j * BT + tid < cnt) {
        const u32 sub = min((u32)(((w[j] >> ib) - first_key) >> sshift), (u32)(4 * kOneSubWords - 1));
        const u32 sh = 8u * (sub & 3u), c4 = s_cnt[sub >> 2];
        s_w[s_base[sub >> 2] + __dp4a(c4 & ((1u << sh) - 1u), 0x01010101u, 0u) +
            ((pos[j / 2] >> (16 * (j & 1))) & 0xFFFFu)] = w[j];
      }
    }
    __syncthreads();
  }
  if (s_misc[43]) {
    small_sort_long(s_w, s_cnt, s_base, n, cnt, first_key, sshift, !ranked);
  } else {
    u32 todo = 0;  // bit 4 j + i: count i of word j * BT + tid is above 1
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const u32 gt = __vcmpgtu4(s_cnt[j * BT + tid], 0x01010101u) & 0x08040201u;
      todo |= ((gt | (gt >> 8) | (gt >> 16) | (gt >> 24)) & 0xFu) << (4 * j);
    }
    while (todo) {  // insertion sort of a sub-bucket (mostly two words)
      const int i = __ffs(todo) - 1, sh = 8 * (i & 3);
      todo &= todo - 1u;
      const u32 c4 = s_cnt[(i >> 2) * BT + tid];
      u64* r = s_w + s_base[(i >> 2) * BT + tid] + __dp4a(c4 & ((1u << sh) - 1u), 0x01010101u, 0u);
      const int k = (int)((c4 >> sh) & 0xFFu);
      for (int x = 1; x < k; ++x) {
        const u64 a = r[x];
        int q = x;
        for (; q > 0; --q) {
          const u64 y = r[q - 1];
          if (y < a) break;
          r[q] = y;
        }
        if (q != x) r[q] = a;
      }
    }
  }
  __syncthreads();
  // ---- the words by position, and their values ----------------------------------
  double v[I];
#pragma unroll
  for (int j = 0; j < I; ++j) {
    if (j >= items) break;
    const u32 p = j * BT + tid;
    w[j] = p < cnt ? s_w[p] : 0ull;
  }
#pragma unroll
  for (int j = 0; j < I; ++j) {
    if (j >= items) break;
    const u32 i = (u32)w[j] & ((1u << ib) - 1u);
    v[j] = 0.0;
    if (j * BT + tid < cnt) v[j] = i < src.na ? __ldcs(src.av + i) : src.bscale * __ldcs(src.bv + (i - src.na));
  }
  if (wide) {  // (rare) the whole keys in the words' place
    __syncthreads();
#pragma unroll
    for (int j = 0; j < I; ++j) {
      if (j >= items) break;
      const u32 i = (u32)w[j] & ((1u << ib) - 1u);
      if (j * BT + tid < cnt) {
        w[j] = i < src.na ? rekey(src.ak[i], src.ra) : rekey(src.bk[i - src.na], src.rb);
        s_w[j * BT + tid] = w[j];
      }
    }
    __syncthreads();
  }
  const int kshift = wide ? 0 : ib;
  if (!FOLD) {
    if (C > 1) cluster_sync();  // everyone has read the input, which the output may be
    else __syncthreads();
#pragma unroll
    for (int j = 0; j < I; ++j) {
      if (j >= items) break;
      const u32 p = j * BT + tid;
      if (p < cnt) {
        out_k[start + p] = w[j] >> kshift;
        out_v[start + p] = v[j];
      }
    }
    return;
  }
  // ---- fold runs of equal keys in input order: into the value of the first -------
#pragma unroll
  for (int j = 0; j < I; ++j) {
    if (j >= items) break;
    const u32 p = j * BT + tid;
    const u32 m = __ballot_sync(0xffffffffu, p < cnt && (p == 0 || (s_w[p - 1] >> kshift) != (w[j] >> kshift)));
    if (lane == 0) s_head[j * (BT / 32) + warp] = m;
  }
  __syncthreads();
  double* s_v = reinterpret_cast<double*>(s_w);  // the values in the words' place
#pragma unroll
  for (int j = 0; j < I; ++j) {
    if (j >= items) break;
    if (j * BT + tid < cnt) s_v[j * BT + tid] = v[j];
  }
  __syncthreads();
  const u32 groups = (u32)items * (BT / 32);
#pragma unroll 1
  for (int j = 0; j < items; ++j) {  // (a head's value becomes its run's sum: nobody else reads it)
    const u32 p = j * BT + tid, g = j * (BT / 32) + warp;
    const bool head = p < cnt && (s_head[g] >> lane & 1u);
    double sum = head ? s_v[p] : 0.0;
    bool anynz = sum != 0.0;
    fold_row(s_head, groups, g, cnt, head, sum, anynz, [&](u32 q) { return s_v[q]; });
    if (head) s_v[p] = sum;
    const u32 m = __ballot_sync(0xffffffffu, head && (!skip_zero_heads || anynz || start + p == 0));
    if (lane == 0) s_kept[g] = m;
  }
  __syncthreads();
  u32 total;
  const u32 at = one_sum((u32)tid < groups ? __popc(s_kept[tid]) : 0u, s_misc, &total);
  if ((u32)tid < groups) s_pre[tid] = at;
  u32 off = 0;
  if (C > 1) {
    cluster_wait();
    if ((u32)tid < C) st_cluster(&s_misc[48 + rank], (u32)tid, total);
    cluster_sync();
    u32 all = 0;
    for (u32 q = 0; q < C; ++q) {
      off += q < rank ? s_misc[48 + q] : 0u;
      all += s_misc[48 + q];
    }
    if (rank == 0 && tid == 0) *d_nout = all;
  } else {
    if (tid == 0) *d_nout = total;
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < I; ++j) {
    if (j >= items) break;
    const u32 g = j * (BT / 32) + warp, m = s_kept[g];
    if (m >> lane & 1u) {
      const u32 o = off + s_pre[g] + __popc(m & (le >> 1));
      out_k[o] = w[j] >> kshift;
      out_v[o] = s_v[j * BT + tid];
    }
  }
}

template <bool FOLD>
int launch_small_sort(const MsdPlan& p, const PairSource& src, const MsdFold* fold, u64* out_k, double* out_v,
                      cudaStream_t s) {
  // CTAs of about 2560 pairs
  u32 C = 1;
  while (C < 8 && p.n > C * 2560) C *= 2;
  const u64 width = (p.max_key + C - 1) / C;
  const int sshift = std::max(0, key_bits_for(width) - kOneSubBits);
  auto kern = small_sort_kernel<FOLD>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOneSmem) != cudaSuccess)
    return LNT_DEVICE_ERROR;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(kOneThreads);
  cfg.dynamicSmemBytes = kOneSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = C > 1 ? 1 : 0;
  ProfScope prof(FOLD ? "small_sort_collect" : "small_sort", s);
  if (cudaLaunchKernelEx(&cfg, kern, src, p.n, p.key_bits, width, sshift, C, FOLD ? fold->skip_zero_heads : 0, out_k,
                         out_v, FOLD ? fold->d_nout : (u64*)nullptr) != cudaSuccess)
    return LNT_DEVICE_ERROR;
  count_launch();
  return launch_status();
}

template <bool FIRST>
int launch_partition(const MsdPlan& p, const PairSource& src, const ulonglong2* in, ulonglong2* out, u32 tiles,
                     int dshift, int dbits, int nseg, const MsdCtrl& c, cudaStream_t s) {
  using P = PartShape<kPartThreads, kPartItems, kPartBlocks>;
  const bool digits = FIRST && p.key_bits + p.ib > 64;
  auto kern = digits ? partition_kernel<P, FIRST, FIRST> : partition_kernel<P, FIRST, false>;
  const size_t sh = P::smem + (digits ? P::kTile : 0);
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh) != cudaSuccess)
    return LNT_DEVICE_ERROR;
  ProfScope prof("sort_partition", s);
  kern<<<tiles, P::kThreads, sh, s>>>(src, in, out, p.n, p.ib, dshift, (1u << dbits) - 1u, nseg, p.db, c);
  count_launch();
  return launch_status();
}

template <class G>
int launch_bucket_sort(const MsdPlan& p, const ulonglong2* rec, const MsdCtrl& c, const MsdFold* fold,
                       u64* out_k, double* out_v, cudaStream_t s) {
  auto kern = fold ? bucket_sort_kernel<G, true> : bucket_sort_kernel<G, false>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::smem) != cudaSuccess)
    return LNT_DEVICE_ERROR;
  ProfScope prof(fold ? "bucket_sort_collect" : "bucket_sort", s);
  kern<<<1u << p.T, G::kBT, G::smem, s>>>(rec, c, p.T, p.shift, p.ib, fold ? fold->skip_zero_heads : 0, out_k,
                                          out_v, fold ? fold->d_nout : nullptr);
  count_launch();
  return launch_status();
}

// Keeps the bit-field moves that reach bits >= shift (pow2 re-keys).
void top_fields(RekeyParams* r, int shift) {
  if (r->order <= 1 || !r->pow2) return;
  int m = 0;
  for (int i = 0; i < r->order; ++i) {
    const u32 f = r->field[i];
    if ((int)((f >> 8) & 63u) + (int)((f >> 16) & 63u) > shift) r->field[m++] = f;
  }
  while (m < 2) r->field[m++] = 0;  // (moves nothing; order 1 would mean no re-key)
  r->order = m;
}

}  // namespace

MsdPlan make_msd_plan(size_t n, u64 max_key) {
  MsdPlan p;
  p.n = (u32)n;
  p.max_key = max_key;
  p.key_bits = key_bits_for(max_key);
  if (n == 0 || n >= (1u << 30) || getenv("LNT_NO_BUCKETS") || getenv("LNT_SORT_VARIANT")) return p;
  if (n <= (size_t)kOneCap && p.key_bits > 0 && p.key_bits + kOneIb <= 64) {
    p.ok = p.single = true;
    return p;
  }
  if (n < kMinPairs) return p;
  // More pairs per key than a thread's or a warp's share of a sub-bucket: the
  // digit passes and their collect are ahead from 32 pairs per key on (2^20 pairs
  // of 2^15 keys: fold 133 us by buckets, 80 by digits; 2^26 of 2^21: 4.2 and 2.9
  // ms), the buckets up to 16 (79 and 81 us; 2.7 and 2.9 ms).
  if ((double)n > kMaxPerKey * (double)max_key) return p;
  const char* force = getenv("LNT_BUCKET_SMALL");
  int bestT = 99;
  for (int large = 0; large < 2; ++large) {
    if (force && (atoi(force) != 0) == (large != 0)) continue;
    // the widest buckets whose expected size (uniform keys) stays below the limit
    const double per_key = (double)n / (double)max_key, lim = large ? kAvgLarge : kAvgSmall;
    if (per_key > lim) continue;
    int shift = 0;
    while (shift < p.key_bits - 1 && per_key * (double)(2ull << shift) <= lim) ++shift;
    const int T = p.key_bits - shift;
    if (T > kMaxT) continue;
    if (bestT == 99 || (bestT > 8 && T <= 8)) {
      bestT = T;
      p.large = large != 0;
      p.shift = shift;
    }
  }
  if (bestT == 99) return p;
  p.T = bestT;
  p.passes = p.T <= 8 ? 1 : 2;
  p.db = p.passes == 1 ? p.T : (p.T + 1) / 2;
  while ((1ull << p.ib) < n) ++p.ib;
  // the word must hold what is left of the key after the first pass; a wider
  // first digit (at most 8 bits) leaves less
  if (p.passes == 2 && p.key_bits + p.ib - (p.T - p.db) > 64) p.db = p.T - 8;
  if (p.key_bits + p.ib - (p.passes == 1 ? p.T : p.T - p.db) > 64) return p;
  const size_t nb = (size_t)1 << p.T;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += align_up(bytes, 256);
    return o;
  };
  p.off_counts = take(nb * 4);
  p.off_misc = take(256);
  p.off_status = take(nb * 8);
  p.zero_bytes = off;
  p.off_start = take((nb + 1) * 4);
  p.off_cur1 = take(kMaxDigits * 4);
  p.off_cur2 = take(nb * 4 + kMaxDigits * 4);
  p.off_segtile = take((kMaxDigits + 1) * 4);
  p.ctrl_bytes = off;
  p.ok = true;
  return p;
}

int run_msd_sort(const MsdPlan& p, const PairSource& src, void* x, void* y, void* ctrl, const MsdFold* fold, u64* out_k, double* out_v, u32* gate, cudaStream_t s) {
  if (p.single) {
    return fold ? launch_small_sort<true>(p, src, fold, out_k, out_v, s)
                : launch_small_sort<false>(p, src, fold, out_k, out_v, s);
  }
  unsigned char* w = static_cast<unsigned char*>(ctrl);
  MsdCtrl c;
  c.counts = reinterpret_cast<u32*>(w + p.off_counts);
  c.start = reinterpret_cast<u32*>(w + p.off_start);
  c.cur1 = reinterpret_cast<u32*>(w + p.off_cur1);
  c.cur2 = reinterpret_cast<u32*>(w + p.off_cur2);
  c.segtile = reinterpret_cast<u32*>(w + p.off_segtile);
  c.misc = reinterpret_cast<u32*>(w + p.off_misc);
  c.status = reinterpret_cast<unsigned long long*>(w + p.off_status);
  c.gate = gate;
  if (cudaMemsetAsync(ctrl, 0, p.zero_bytes, s) != cudaSuccess) return LNT_DEVICE_ERROR;
  const u32 cap = p.large ? (u32)GeomLarge::kCap : (u32)GeomSmall::kCap;
  {
    const size_t sh = ((size_t)1 << p.T) * 4;
    if (cudaFuncSetAttribute(msd_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh) != cudaSuccess)
      return LNT_DEVICE_ERROR;
    const u32 want = (p.n + kHistThreads * 4 - 1) / (kHistThreads * 4);
    ProfScope prof("sort_hist", s);
    // the buckets need only the top key bits: with power-of-two extents, only
    // the modes that reach them are moved
    PairSource top = src;
    top_fields(&top.ra, p.shift);
    top_fields(&top.rb, p.shift);
    // (with one pass the cursors are the bucket starts: every bucket is its own segment)
    msd_hist_kernel<<<std::min(want, (u32)sm_count()), kHistThreads, sh, s>>>(
        top, p.n, p.T, p.passes == 1 ? 0 : p.db, p.shift, p.key_bits, cap, c);
    count_launch();
  }
  ulonglong2* rx = static_cast<ulonglong2*>(x);
  ulonglong2* ry = static_cast<ulonglong2*>(y);
  {
    const int dbits = p.passes == 1 ? p.T : p.T - p.db;  // this pass's digit: the top bits
    const int st = launch_partition<true>(p, src, nullptr, p.passes == 1 ? ry : rx, (p.n + kPartTile - 1) / kPartTile,
                                          p.key_bits - dbits, dbits, 0, c, s);
    if (st != LNT_OK) return st;
  }
  if (p.passes == 2) {
    const int nseg = 1 << (p.T - p.db);
    const int st = launch_partition<false>(p, src, rx, ry, (p.n + kPartTile - 1) / kPartTile + nseg, p.ib + p.shift,
                                           p.db, nseg, c, s);
    if (st != LNT_OK) return st;
  }
  return p.large ? launch_bucket_sort<GeomLarge>(p, ry, c, fold, out_k, out_v, s)
                 : launch_bucket_sort<GeomSmall>(p, ry, c, fold, out_k, out_v, s);
}

PairSort make_pair_sort(size_t n, u64 max_key, bool buckets) {
  PairSort p;
  if (buckets) p.msd = make_msd_plan(n, max_key);
  p.lsd = make_sort_plan(n, max_key, p.msd.ok);
  p.ctrl_bytes = align_up(std::max(p.lsd.ctrl_bytes, p.msd.ctrl_bytes), 256) + (p.msd.ok ? 256 : 0);
  if (p.msd.single) {  // needs no scratch
    p.ctrl_bytes = 256;
    return p;
  }
  p.a_bytes = 2 * align_up(n * 8, 256);
  p.b_bytes = p.msd.ok && p.msd.passes == 2 ? p.a_bytes : 0;
  return p;
}

int run_pair_sort(const PairSort& p, const PairSource& src, u64* out_k, double* out_v, void* a, void* b, void* ctrl,
                  cudaStream_t s) {
  u32* gate = nullptr;
  if (p.msd.ok) {
    gate = reinterpret_cast<u32*>(static_cast<unsigned char*>(ctrl) + p.ctrl_bytes - 256);
    const int st = run_msd_sort(p.msd, src, b, a, ctrl, nullptr, out_k, out_v, gate, s);
    if (st != LNT_OK || p.msd.single) return st;
  }
  u64* ak = static_cast<u64*>(a);
  double* av = reinterpret_cast<double*>(static_cast<unsigned char*>(a) + p.a_bytes / 2);
  return run_sort(p.lsd, gated_source(src, gate, 1), out_k, out_v, ak, av, ctrl, s);
}

}  // namespace lnt
