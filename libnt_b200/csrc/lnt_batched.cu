// Batched sparse lattice products: thousands of independent, unevenly sized
// C_p = A_p * B_p (each as in lnt_lattice_mult) in a fixed number of launches,
// all stream-ordered and capturable in one CUDA graph.  The reference has no
// batching: its equivalent is a loop of csc_no_accum calls
// (SparseLatticeBase.h:1854-1990), one per contraction.
//
// Layout: operands are concatenated (A of problem p at a_off[p] .. a_off[p+1],
// likewise B); a descriptor per problem holds its dims, magic dividers and
// offsets into the scratch tables.  Output C is concatenated too; problem p's
// part starts at c_off[p].
//
// Pipeline (per call):
//   colptr (A and B): dense column pointers of every problem (u32 offsets);
//   spa<symbolic>: persistent warps pull chunks of output columns ("units") of
//     all problems from an atomic queue and count each column's output rows;
//   scan: global exclusive sum over units -> output position of every column;
//   spa<numeric>: persistent warps pull chunks again and write each column's
//     rows (dense accumulator in shared memory, ascending emission);
//   coff: per-problem output offsets.
// The queue chunk size (units per grab) is the segment-split knob the
// autotuner sets: small chunks balance uneven columns, large ones cut queue
// traffic.  Problems with more than 512 rows are accumulated in blocks of
// 512 rows (each A column's entries for the block found by binary search).
//
// lnt_batched_contract takes the operands as the tensors are stored (unsorted,
// keys in each tensor's own mode order) and does the per-problem work of
// toLatticeSort (SparseMIABase.h:1457-1586) inside the call.  The products need
// no sorted operands, only A's entries grouped by column and B's by output
// column, and most entries meet no partner at all (a matched column or row is
// rare when a problem has far more contracted indices than entries).  So, for
// problems of at most 512 rows:
//   mark:   one read of the keys (re-keyed on the fly) sets a bit per contracted
//           index that occurs in A, and one per index that occurs in B;
//   rank:   the indices in both are numbered;
//   filter: a second read keeps the entries with a partner (their values are
//           read only now), counts A's per contracted index and B's per output
//           column;
//   base, place: room for every group, and the entries into their groups, in the
//           order in which their atomics come: the products then add up in an
//           order that differs from run to run (the sorted operands of
//           lnt_batched_lattice_mult add up in a fixed one).  Sorting the groups
//           to fix the order was measured at 0.7 ms on the batch below, a quarter
//           of the call;
//   then spa<symbolic>, scan, spa<numeric> and coff as above on the groups.
// The work is cut into tasks of one operand of one problem (at most 64 K
// entries, less when the batch is small), largest first.
// 4096 problems of 100 to 10^5 entries (1.18e8 pairs, 4.4e7 products), B200:
// mark 0.33, rank 0.03, filter 0.57, base 0.02, place 0.51, symbolic 0.45,
// numeric 0.61, the call 2.57 ms (11.7 ms when the batch was sorted: compose 0.61,
// histogram 0.50, five digit passes 5.9, column pointers 1.3, symbolic 1.3,
// numeric 2.05).  2.7e7 entries and 6.7e6 of 3.7e7 indices have a partner.
// Batches with taller problems sort instead: one kernel re-keys every pair into
// its problem's lattice order and prefixes the key with (problem, operand), one
// stable radix sort of all pairs orders every problem's A and B at once (their
// segments end up interleaved: A_0 B_0 A_1 B_1 ..), and the product kernels read
// the sorted pairs with the prefix masked off.
#include <algorithm>
#include <cstdlib>
#include <vector>

#include "lnt_tuned.h"
#include "lnt_scan.cuh"
#include "lnt_sort.cuh"

namespace lnt {
namespace {

constexpr int kMaxRows = 512;  // accumulator rows per warp (4 KB of FP64 sums: eight 4-warp CTAs per SM)
constexpr int kWarps = 4;

struct ProbDesc {
  u64 a_off, a_n, b_off, b_n;
  u64 aptr_off, bptr_off;  // into the u32 pointer tables
  u64 unit_off, units;     // global unit range (units = wB * d)
  u64 word_off;            // first bitmap word (grouped path: one bit per contracted index and tab)
  u64 h, w, wB, d;
  Divider div_h, div_w, div_wB;
};

struct BatchArgs {
  const u64* ak;
  const double* av;
  const u64* bk;
  const double* bv;
  const ProbDesc* prob;
  int count;
  u64 total_units;
  u32* aptr;
  u32* bptr;
  u64 kmask;  // lattice key bits of the stored keys (the rest is the sort prefix)
  const u32* uprob;  // the problem of every unit (output column), built at prepare time
};

// Column pointers of every problem's A (which == 0) or B (which == 1).
// Position q enumerates, problem by problem, the n_p + 1 boundaries; position
// i of problem p fills the pointer entries of the (possibly many empty)
// columns between entry i-1's column and entry i's.  A warp takes 256
// consecutive positions, lane-striped (w0 + 32 k + lane: coalesced key loads,
// adjacent lanes' short ranges adjacent), each lane one binary search for its
// problem, and each thread fills short ranges itself; a range longer than kLongRun columns (a run of empty columns,
// common in problems with far more columns than entries) is filled by the
// whole warp together in coalesced stores, so no thread writes a long run
// alone.
__global__ void batch_colptr_kernel(BatchArgs args, int which, const u64* __restrict__ pos_off, u64 total_pos) {
  constexpr u64 kPer = 8;
  constexpr long long kLongRun = 32;
  const int lane = threadIdx.x & 31;
  const u64 warps = ((u64)gridDim.x * blockDim.x) >> 5;
  const u64 warp_id = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  for (u64 w0 = warp_id * 32 * kPer; w0 < total_pos; w0 += warps * 32 * kPer) {
    const u64 q0 = w0 + (u64)lane;  // lane-striped: positions w0 + 32 k + lane
    int p = 0;
    if (q0 < total_pos) {
      int lo = 0, hi = args.count - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pos_off[mid] <= q0) lo = mid; else hi = mid - 1;
      }
      p = lo;
    }
    for (u64 k = 0; k < kPer; ++k) {
      const u64 q = q0 + 32 * k;
      long long prev = 0, cur = -1;
      u32 idx = 0;
      u32* ptr = nullptr;
      if (q < total_pos) {
        while (p + 1 < args.count && pos_off[p + 1] <= q) ++p;
        const ProbDesc& P = args.prob[p];
        const u64 i = q - pos_off[p];
        const u64 n = which == 0 ? P.a_n : P.b_n;
        const u64* keys = which == 0 ? args.ak + P.a_off : args.bk + P.b_off;
        const Divider& dv = which == 0 ? P.div_h : P.div_w;
        const u64 ncol = which == 0 ? P.w * P.d : P.units;
        ptr = which == 0 ? args.aptr + P.aptr_off : args.bptr + P.bptr_off;
        prev = i == 0 ? -1ll : (long long)min(divide(keys[i - 1] & args.kmask, dv), ncol);
        cur = i == n ? (long long)ncol : (long long)min(divide(keys[i] & args.kmask, dv), ncol);
        idx = (u32)i;
        if (cur - prev <= kLongRun)
          for (long long c = prev + 1; c <= cur; ++c) ptr[c] = idx;
      }
      u32 longm = __ballot_sync(0xffffffffu, cur - prev > kLongRun);
      while (longm) {
        const int j = __ffs(longm) - 1;
        longm &= longm - 1u;
        const long long pj = __shfl_sync(0xffffffffu, prev, j);
        const long long cj = __shfl_sync(0xffffffffu, cur, j);
        const u32 ij = __shfl_sync(0xffffffffu, idx, j);
        u32* pp = reinterpret_cast<u32*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(ptr), j));
        for (long long c = pj + 1 + lane; c <= cj; c += 32) pp[c] = ij;
      }
    }
  }
}

// First entry at or after position lo of A column acol (entries lo..hi-1,
// ascending rows) whose row is >= r0.
__device__ __forceinline__ u32 lower_row(const u64* __restrict__ ak, u64 kmask, u32 lo, u32 hi, u64 base, u64 r0) {
  while (lo < hi) {
    const u32 mid = (lo + hi) >> 1;
    if ((ak[mid] & kmask) - base < r0) lo = mid + 1; else hi = mid;
  }
  return lo;
}

template <bool NUMERIC>
__global__ void __launch_bounds__(kWarps * 32, 8) batch_spa_kernel(BatchArgs args, u32 chunk, u32* __restrict__ queue,
                                                                 u64* __restrict__ ucount,
                                                                 const u64* __restrict__ uoff,
                                                                 u64* __restrict__ ck, double* __restrict__ cv) {
  __shared__ u32 s_bits[kWarps][kMaxRows / 32];
  __shared__ double s_acc[NUMERIC ? kWarps : 1][NUMERIC ? kMaxRows : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  u32* bits = s_bits[warp];
  double* acc = s_acc[NUMERIC ? warp : 0];
  const u64 kmask = args.kmask;
  while (true) {
    u64 first = 0;
    if (lane == 0) first = (u64)atomicAdd(queue, chunk);
    first = __shfl_sync(0xffffffffu, first, 0);
    if (first >= args.total_units) break;
    const u64 last = min(first + chunk, args.total_units);
    for (u64 u = first; u < last; ++u) {
      const ProbDesc& P = args.prob[args.uprob[u]];  // chunks may span problems
      const u64 lu = u - P.unit_off;  // column id within the problem: col + wB*tab
      const u32* bptr = args.bptr + P.bptr_off;
      const u64 e0 = bptr[lu], e1 = bptr[lu + 1];
      if (e0 == e1) {
        if (!NUMERIC && lane == 0) ucount[u] = 0;
        continue;
      }
      const u64 h = P.h, w = P.w;
      const u64 t = divide(lu, P.div_wB);
      const u64* ak = args.ak + P.a_off;
      const double* av = args.av + P.a_off;
      const u64* bk = args.bk + P.b_off;
      const double* bv = args.bv + P.b_off;
      const u32* aptr = args.aptr + P.aptr_off;
      const bool blocked = h > (u64)kMaxRows;
      u64 out = NUMERIC ? uoff[u] : 0;
      u32 count = 0;
      const u64 colkey = h * lu;
      // rows in blocks of kMaxRows (one block unless h > kMaxRows), ascending
      for (u64 r0 = 0; r0 < h; r0 += kMaxRows) {
        const u64 hb = min((u64)kMaxRows, h - r0);
        const int hw = (int)((hb + 31) / 32);
        for (int i = lane; i < hw; i += 32) bits[i] = 0u;
        if (NUMERIC)
          for (int i = lane; i < (int)hb; i += 32) acc[i] = 0.0;
        __syncwarp();
        for (u64 e = e0 + lane; e < e1; e += 32) {
          const u64 acol = ((bk[e] & kmask) - w * lu) + w * t;
          const u64 abase = acol * h;
          u32 lo = aptr[acol];
          const u32 hi = aptr[acol + 1];
          if (blocked) lo = lower_row(ak, kmask, lo, hi, abase, r0);
          const double beta = NUMERIC ? bv[e] : 0.0;
          // four A entries loaded before their accumulations, so that their
          // loads overlap instead of each waiting behind the previous atomics
          bool stop = false;
          u32 x = lo;
          for (; x + 4 <= hi && !stop; x += 4) {
            u64 kk[4];
            double vv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              kk[j] = ak[x + j];
              vv[j] = NUMERIC ? av[x + j] : 0.0;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const u64 rr = (kk[j] & kmask) - abase;
              if (blocked && rr >= r0 + hb) {
                stop = true;
                break;
              }
              const u32 r = (u32)(rr - r0);
              atomicOr(&bits[r >> 5], 1u << (r & 31));
              if (NUMERIC) atomicAdd(&acc[r], vv[j] * beta);
            }
          }
          for (; x < hi && !stop; ++x) {
            const u64 rr = (ak[x] & kmask) - abase;
            if (blocked && rr >= r0 + hb) break;
            const u32 r = (u32)(rr - r0);
            atomicOr(&bits[r >> 5], 1u << (r & 31));
            if (NUMERIC) atomicAdd(&acc[r], av[x] * beta);
          }
        }
        __syncwarp();
        if (!NUMERIC) {
          u32 c = 0;
          for (int i = lane; i < hw; i += 32) c += __popc(bits[i]);
          count += c;
        } else {
          for (int g = 0; g < hw; ++g) {
            const u32 word = bits[g];
            if (word & (1u << lane)) {
              const u32 r = (u32)g * 32 + lane;
              const u64 o = out + __popc(word & ((1u << lane) - 1u));
              ck[o] = colkey + r0 + r;
              cv[o] = acc[r];
            }
            out += __popc(word);
          }
        }
        __syncwarp();
      }
      if (!NUMERIC) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
        if (lane == 0) ucount[u] = count;
      }
    }
  }
}

__global__ void batch_coff_kernel(const ProbDesc* __restrict__ prob, int count, const u64* __restrict__ uoff,
                                  u64 total_units, u64* __restrict__ c_off) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < count) c_off[p] = uoff[prob[p].unit_off];
  if (p == count) c_off[count] = uoff[total_units];
}

struct BatchLayout {
  u64 total_units, aptr_len, bptr_len, a_pos, b_pos, c_bound, words, max_words, max_h;
  size_t off_prob, off_apos, off_bpos, off_aptr, off_bptr, off_ucount, off_uoff, off_queue, off_scan, off_uprob,
      total;
};

// The contract path groups its entries instead of sorting them: 32-bit
// contracted indices and output columns, and rows that fit the accumulators.
bool grouped_applies(const BatchLayout& L) {
  return L.max_h <= (u64)kMaxRows && L.max_words < (1ull << 27) && L.total_units < (1ull << 32);
}

// interleaved: the operands are read from one array holding A_0 B_0 A_1 B_1 ..
// (the output of the contract path's sort) instead of two concatenations.
int batch_layout(int count, const int64_t* dims, const uint64_t* a_off, const uint64_t* b_off, BatchLayout* L,
                 std::vector<ProbDesc>* descs, std::vector<u64>* apos, std::vector<u64>* bpos,
                 bool interleaved = false) {
  if (count <= 0 || !dims || !a_off || !b_off) return LNT_BAD_ARG;
  L->total_units = L->aptr_len = L->bptr_len = L->a_pos = L->b_pos = L->c_bound = 0;
  L->words = L->max_words = L->max_h = 0;
  if (descs) descs->resize(count);
  if (apos) apos->resize(count);
  if (bpos) bpos->resize(count);
  for (int p = 0; p < count; ++p) {
    const int64_t h = dims[4 * p], w = dims[4 * p + 1], wB = dims[4 * p + 2], d = dims[4 * p + 3];
    if (h <= 0 || w <= 0 || wB <= 0 || d <= 0) return LNT_BAD_DIMS;
    if (a_off[p + 1] < a_off[p] || b_off[p + 1] < b_off[p]) return LNT_BAD_ARG;
    const u64 na = a_off[p + 1] - a_off[p], nb = b_off[p + 1] - b_off[p];
    if (na >= (1ull << 32) || nb >= (1ull << 32)) return LNT_UNSUPPORTED;
    unsigned __int128 ka = (unsigned __int128)h * w * d, kb = (unsigned __int128)w * wB * d;
    if ((ka >> 63) || (kb >> 63)) return LNT_OVERFLOW_KEYBITS;
    if (descs) {
      ProbDesc& P = (*descs)[p];
      P.a_off = interleaved ? a_off[p] + b_off[p] : a_off[p];
      P.a_n = na;
      P.b_off = interleaved ? P.a_off + na : b_off[p];
      P.b_n = nb;
      P.aptr_off = L->aptr_len;
      P.bptr_off = L->bptr_len;
      P.unit_off = L->total_units;
      P.units = (u64)wB * d;
      P.word_off = L->words;
      P.h = h;
      P.w = w;
      P.wB = wB;
      P.d = d;
      P.div_h = make_divider(h);
      P.div_w = make_divider(w);
      P.div_wB = make_divider(wB);
    }
    if (apos) (*apos)[p] = L->a_pos;
    if (bpos) (*bpos)[p] = L->b_pos;
    const u64 words = ((u64)w * d + 31) / 32;
    L->words += words;
    L->max_words = std::max(L->max_words, words);
    L->max_h = std::max(L->max_h, (u64)h);
    L->aptr_len += (u64)w * d + 1;
    L->bptr_len += (u64)wB * d + 1;
    L->total_units += (u64)wB * d;
    L->a_pos += na + 1;
    L->b_pos += nb + 1;
    L->c_bound += (u64)std::min<unsigned __int128>((unsigned __int128)h * wB * d, (unsigned __int128)nb * h);
  }
  size_t off = 0;
  L->off_prob = off;
  off += align_up((size_t)count * sizeof(ProbDesc), 256);
  L->off_apos = off;
  off += align_up((size_t)count * 8, 256);
  L->off_bpos = off;
  off += align_up((size_t)count * 8, 256);
  const bool tables = !interleaved || !grouped_applies(*L);  // the grouped path needs no column pointers
  L->off_aptr = off;
  off += tables ? align_up(L->aptr_len * 4, 256) : 0;
  L->off_bptr = off;
  off += tables ? align_up(L->bptr_len * 4, 256) : 0;
  L->off_ucount = off;
  off += align_up((L->total_units + 1) * 8, 256);
  L->off_uoff = off;
  off += align_up((L->total_units + 1) * 8, 256);
  L->off_queue = off;
  off += 256;
  L->off_scan = off;
  off += align_up(scan::workspace_bytes(L->total_units), 256);
  L->off_uprob = off;
  off += align_up(std::max<u64>(L->total_units, 1) * 4, 256);
  L->total = off;
  return LNT_OK;
}

// The problem of every unit, from the descriptors (units are numbered problem
// by problem): the product kernels read it instead of searching the
// descriptors for each column they take.
std::vector<u32> unit_problems(const std::vector<ProbDesc>& descs, u64 total_units) {
  std::vector<u32> up(total_units);
  for (size_t p = 0; p < descs.size(); ++p)
    std::fill(up.begin() + descs[p].unit_off, up.begin() + descs[p].unit_off + descs[p].units, (u32)p);
  return up;
}

struct U64Of {
  const u64* v;
  __device__ __forceinline__ u64 operator()(size_t i) const { return v[i]; }
};

// Composite sort keys of the contract path: position q of the concatenated
// operand (A or B) belongs to the problem p with off[p] <= q < off[p+1]; its
// key is re-keyed into p's lattice order and prefixed with (p, which).  A warp
// takes 256 consecutive positions, lane-striped (position base + 32 j + lane),
// so loads and stores are coalesced; each lane finds its first position's
// problem by binary search and walks forward from there.  (A thread taking 8
// consecutive positions issued 8-byte stores 64 bytes apart: 0.86 ms for the
// 4096-problem batch.)
__global__ void batch_compose_kernel(const u64* __restrict__ keys, u64 n, const uint64_t* __restrict__ off,
                                     int count, const RekeyParams* __restrict__ rk, u64 which_bit, int S,
                                     u64* __restrict__ out) {
  constexpr u64 kSpan = 256;
  const int lane = threadIdx.x & 31;
  const u64 nwarps = ((u64)gridDim.x * blockDim.x) >> 5;
  for (u64 base = (((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kSpan; base < n; base += nwarps * kSpan) {
    const u64 q0 = base + lane;
    if (q0 >= n) continue;
    int lo = 0, hi = count - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (off[mid] <= q0) lo = mid; else hi = mid - 1;
    }
    int p = lo;
    const u64 q1 = min(base + kSpan, n);
    for (u64 q = q0; q < q1; q += 32) {
      while (q >= off[p + 1]) ++p;
      out[q] = ((u64)p << (S + 1)) | which_bit | rekey(keys[q], rk[p]);
    }
  }
}

// ---- grouped path --------------------------------------------------------------
struct GroupTask {
  u64 begin;  // first entry of the operand's concatenation
  u32 n;
  u32 prob;   // problem | which << 31 (0: A, 1: B)
};

struct GroupArgs {
  const u64* ak;
  const double* av;
  const u64* bk;
  const double* bv;
  u64 NA;
  const ProbDesc* prob;
  const RekeyParams* rk;  // A's, then B's
  int count;
  const GroupTask* tasks;
  const uint2* places;  // the tasks' entries in problem order: (task, first)
  u32* bits_a;   // contracted indices that occur in A, in B
  u32* bits_b;
  u64 words;
  uint2* rank;   // per word: (indices in both, number of the first)
  uint2* acol;   // per numbered index: (cursor, entries of A)
  uint2* bcol;   // per output column: (cursor, entries of B)
  u64 units;
  uint4* kept;   // kept entries, at their task's place: (group, row or index, value)
  u32* kept_n;   // per task
  ulonglong2* arec;  // (row, value) grouped by index
  ulonglong2* brec;  // (index, later its (end, count) in arec; value) grouped by output column
  u32* counters;     // [0] numbered indices, [1], [2] next free arec, brec
};

constexpr u32 kGrab = 8;      // output columns per queue grab, past the first eighth of them
constexpr u32 kPlace = 2048;  // entries per piece of a task (group_place_kernel)
constexpr int kGroupThreads = 256;
constexpr int kGroupItems = 8;
constexpr u64 kGroupSmemWords = 16384;  // largest bitmap built in shared memory

// What an operand's entries are to the product: A: g = contracted index, r =
// row; B: g = contracted index, r = output column.  g = ~0: no entry, or a key
// outside its lattice.
template <int I>
__device__ __forceinline__ void group_items(const u64* keys, const RekeyParams& rk, const ProbDesc& P, bool is_b,
                                            u32 first, u32 n, u32 (&g)[I], u32 (&r)[I]) {
  u64 k[I];
  u32 use = 0;
#pragma unroll
  for (int j = 0; j < I; ++j) {
    const u32 i = first + j * kGroupThreads + threadIdx.x;
    k[j] = 0;
    if (i < n) {
      k[j] = __ldg(keys + i);
      use |= 1u << j;
    }
  }
  rekey_items(k, rk, use);
  const u64 wd = P.w * P.d;
  u64 high = 0;
#pragma unroll
  for (int j = 0; j < I; ++j) high |= k[j];
  if ((high >> 32) == 0 && ((wd * max(P.h, P.wB)) >> 31) == 0) {  // 32-bit arithmetic
#pragma unroll
    for (int j = 0; j < I; ++j) {
      const u32 key = (u32)k[j];
      u32 x, y;
      if (!is_b) {
        x = divide32(key, P.div_h);
        y = key - x * (u32)P.h;
      } else {
        y = divide32(key, P.div_w);
        x = key - y * (u32)P.w + (u32)P.w * divide32(y, P.div_wB);
      }
      g[j] = (use >> j & 1u) && x < (u32)wd && (!is_b || y < (u32)P.units) ? x : ~0u;
      r[j] = y;
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < I; ++j) {
    u64 x, y;
    if (!is_b) {  // row + h * index
      x = divide(k[j], P.div_h);
      y = k[j] - x * P.h;
    } else {  // (index without its tab) + w * (column + wB * tab)
      y = divide(k[j], P.div_w);
      const u64 t = divide(y, P.div_wB);
      x = k[j] - y * P.w + P.w * t;
    }
    g[j] = (use >> j & 1u) && x < wd && (!is_b || y < P.units) ? (u32)x : ~0u;
    r[j] = (u32)y;
  }
}

// The task's operand, problem and re-key parameters (the latter to shared memory).
struct GroupCtx {
  RekeyParams rk;
  ProbDesc P;
};
__device__ __forceinline__ void load_ctx(const GroupArgs& a, const GroupTask& t, GroupCtx* c) {
  const u32 p = t.prob & 0x7FFFFFFFu;
  const u32* s0 = reinterpret_cast<const u32*>(a.rk + (t.prob >> 31 ? (size_t)a.count + p : (size_t)p));
  const u32* s1 = reinterpret_cast<const u32*>(a.prob + p);
  u32* d0 = reinterpret_cast<u32*>(&c->rk);
  u32* d1 = reinterpret_cast<u32*>(&c->P);
  for (u32 i = threadIdx.x; i < sizeof(RekeyParams) / 4; i += kGroupThreads) d0[i] = s0[i];
  for (u32 i = threadIdx.x; i < sizeof(ProbDesc) / 4; i += kGroupThreads) d1[i] = s1[i];
}

__global__ void __launch_bounds__(kGroupThreads) group_mark_kernel(const GroupArgs a, u32 smem_words) {
  extern __shared__ u32 s_bits[];
  __shared__ GroupCtx c;
  const GroupTask t = a.tasks[blockIdx.x];
  const bool is_b = (t.prob >> 31) != 0;
  load_ctx(a, t, &c);
  __syncthreads();
  const u32 words = (u32)((c.P.w * c.P.d + 31) / 32);
  u32* out = (is_b ? a.bits_b : a.bits_a) + c.P.word_off;
  // a bitmap in shared memory, or-ed in word by word, once the entries outnumber the words
  const bool local = words <= smem_words && t.n >= words / 2;
  if (local)
    for (u32 i = threadIdx.x; i < words; i += kGroupThreads) s_bits[i] = 0;
  __syncthreads();
  const u64* keys = (is_b ? a.bk : a.ak) + t.begin;
  for (u32 base = 0; base < t.n; base += kGroupThreads * kGroupItems) {
    u32 g[kGroupItems], r[kGroupItems];
    group_items(keys, c.rk, c.P, is_b, base, t.n, g, r);
#pragma unroll
    for (int j = 0; j < kGroupItems; ++j) {
      if (g[j] == ~0u) continue;
      if (local) atomicOr(&s_bits[g[j] >> 5], 1u << (g[j] & 31));
      else atomicOr(&out[g[j] >> 5], 1u << (g[j] & 31));
    }
  }
  if (!local) return;
  __syncthreads();
  for (u32 i = threadIdx.x; i < words; i += kGroupThreads)
    if (s_bits[i]) atomicOr(&out[i], s_bits[i]);
}

// Block-wide exclusive sum of `v`; the block's total in *total.
__device__ __forceinline__ u32 block_sum(u32 v, u32* s_w, u32* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  u32 inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 x = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += x;
  }
  __syncthreads();
  if (lane == 31) s_w[warp] = inc;
  __syncthreads();
  u32 before = 0, tot = 0;
#pragma unroll
  for (int q = 0; q < kGroupThreads / 32; ++q) {
    before += q < warp ? s_w[q] : 0u;
    tot += s_w[q];
  }
  *total = tot;
  return before + inc - v;
}

// Numbers the indices that occur in both operands.  Which numbers a block's
// indices get does not matter, so a block reserves its range with one atomic;
// it also zeroes the range's entry counts.
__global__ void __launch_bounds__(kGroupThreads) group_rank_kernel(const GroupArgs a) {
  __shared__ u32 s_w[kGroupThreads / 32], s_base;
  constexpr int I = 8;
  const u64 base = (u64)blockIdx.x * (kGroupThreads * I);
  u32 m[I], sum = 0;
#pragma unroll
  for (int j = 0; j < I; ++j) {  // (lane-striped: any order will do)
    const u64 i = base + j * kGroupThreads + threadIdx.x;
    m[j] = i < a.words ? a.bits_a[i] & a.bits_b[i] : 0u;
    sum += __popc(m[j]);
  }
  u32 total;
  u32 at = block_sum(sum, s_w, &total);
  if (threadIdx.x == 0) s_base = total ? atomicAdd(&a.counters[0], total) : 0u;
  __syncthreads();
  at += s_base;
#pragma unroll
  for (int j = 0; j < I; ++j) {
    const u64 i = base + j * kGroupThreads + threadIdx.x;
    if (i < a.words) a.rank[i] = make_uint2(m[j], at);
    at += __popc(m[j]);
  }
  for (u32 i = threadIdx.x; i < total; i += kGroupThreads) a.acol[s_base + i] = make_uint2(0u, 0u);
}

__global__ void __launch_bounds__(kGroupThreads) group_filter_kernel(const GroupArgs a) {
  __shared__ GroupCtx c;
  __shared__ u32 s_n;
  const GroupTask t = a.tasks[blockIdx.x];
  const bool is_b = (t.prob >> 31) != 0;
  load_ctx(a, t, &c);
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  const u64* keys = (is_b ? a.bk : a.ak) + t.begin;
  const double* vals = (is_b ? a.bv : a.av) + t.begin;
  uint4* kept = a.kept + (is_b ? a.NA : 0) + t.begin;
  const uint2* rank = a.rank + c.P.word_off;
  const int lane = threadIdx.x & 31;
  for (u32 base = 0; base < t.n; base += kGroupThreads * kGroupItems) {
    u32 g[kGroupItems], r[kGroupItems];
    group_items(keys, c.rk, c.P, is_b, base, t.n, g, r);
    u32 live = 0;
#pragma unroll
    for (int j = 0; j < kGroupItems; ++j) {
      const uint2 q = g[j] != ~0u ? rank[g[j] >> 5] : make_uint2(0u, 0u);
      const u32 bit = 1u << (g[j] & 31);
      if (q.x & bit) {
        live |= 1u << j;
        g[j] = q.y + __popc(q.x & (bit - 1u));
      }
    }
    double v[kGroupItems];
#pragma unroll
    for (int j = 0; j < kGroupItems; ++j)
      v[j] = live >> j & 1u ? __ldcs(vals + base + j * kGroupThreads + threadIdx.x) : 0.0;
    u32 mine = __popc(live), inc = mine;  // room for the warp's kept entries: one atomic
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 x = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += x;
    }
    u32 room = 0;
    if (lane == 31 && inc) room = atomicAdd(&s_n, inc);
    u32 pos = __shfl_sync(0xffffffffu, room, 31) + inc - mine;
#pragma unroll
    for (int j = 0; j < kGroupItems; ++j) {
      if (!(live >> j & 1u)) continue;
      const long long bits = __double_as_longlong(v[j]);
      const u32 unit = (u32)c.P.unit_off + r[j];
      // A: (index, row); B: (output column, index)
      kept[pos++] = is_b ? make_uint4(unit, g[j], (u32)bits, (u32)(bits >> 32))
                         : make_uint4(g[j], r[j], (u32)bits, (u32)(bits >> 32));
      atomicAdd(is_b ? &a.bcol[unit].y : &a.acol[g[j]].y, 1u);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) a.kept_n[blockIdx.x] = s_n;
}

// Room for every group (again in any order): cursor = first record.
__global__ void __launch_bounds__(kGroupThreads) group_base_kernel(const GroupArgs a) {
  __shared__ u32 s_w[kGroupThreads / 32], s_base;
  constexpr int I = 8;
  constexpr u64 kTile = kGroupThreads * I;
  const u64 na = __ldcg(&a.counters[0]);
  const u64 ta = (na + kTile - 1) / kTile, tb = (a.units + kTile - 1) / kTile;
  for (u64 tile = blockIdx.x; tile < ta + tb; tile += gridDim.x) {
    uint2* col = tile < ta ? a.acol : a.bcol;
    const u64 n = tile < ta ? na : a.units, base = (tile < ta ? tile : tile - ta) * kTile;
    u32 cnt[I], sum = 0;
#pragma unroll
    for (int j = 0; j < I; ++j) {
      const u64 i = base + j * kGroupThreads + threadIdx.x;
      cnt[j] = i < n ? col[i].y : 0u;
      sum += cnt[j];
    }
    u32 total;
    u32 at = block_sum(sum, s_w, &total);
    if (threadIdx.x == 0) s_base = total ? atomicAdd(&a.counters[tile < ta ? 1 : 2], total) : 0u;
    __syncthreads();
    at += s_base;
#pragma unroll
    for (int j = 0; j < I; ++j) {
      const u64 i = base + j * kGroupThreads + threadIdx.x;
      if (i < n) col[i].x = at;
      at += cnt[j];
    }
  }
}

// One atomic and one scattered store per record.  The tasks are cut into pieces
// of kPlace entries and taken problem by problem, so that what is being written
// stays in the L2 until its sectors are complete: whole tasks, the largest of
// the batch first, spread the stores over about 1 GB at a time (0.94 ms for
// 2.7e7 records; pieces of 16384, 8192, 4096, 2048: 0.75, 0.63, 0.54, 0.52 ms).
__global__ void __launch_bounds__(kGroupThreads) group_place_kernel(const GroupArgs a) {
  const uint2 place = a.places[blockIdx.x];
  const GroupTask t = a.tasks[place.x];
  const bool is_b = (t.prob >> 31) != 0;
  const u32 kept_n = a.kept_n[place.x];
  if (place.y >= kept_n) return;
  const uint4* kept = a.kept + (is_b ? a.NA : 0) + t.begin + place.y;
  const u32 n = min(kPlace, kept_n - place.y);
  constexpr int I = 4;
  uint2* col = is_b ? a.bcol : a.acol;
  ulonglong2* rec = is_b ? a.brec : a.arec;
  for (u32 base = threadIdx.x; base < n; base += kGroupThreads * I) {
    uint4 e[I];
    u32 at[I];
#pragma unroll
    for (int j = 0; j < I; ++j)
      if (base + j * kGroupThreads < n) e[j] = __ldcs(kept + base + j * kGroupThreads);
#pragma unroll
    for (int j = 0; j < I; ++j)
      if (base + j * kGroupThreads < n) at[j] = atomicAdd(&col[e[j].x].x, 1u);
#pragma unroll
    for (int j = 0; j < I; ++j)
      if (base + j * kGroupThreads < n)
        rec[at[j]] = make_ulonglong2(e[j].y, (u64)e[j].z | ((u64)e[j].w << 32));
  }
}

// Gustavson's product on the groups (at most kMaxRows rows): a warp per output
// column, taken from a queue in `order`: the problems with the most products per
// column first and one column at a time, so that no long column is left for the
// end or behind another (in the batch's order a grab of 4 columns took 1.16 ms
// in the numeric pass and one of 16 3.5 ms); after `singles` columns kGrab at a
// time, which saves most of the latency of the queue and the tables.  Lanes take entries of B; an index with many
// entries of A is walked by the whole warp.  The symbolic pass leaves an index's
// (end, count) in the entry of B, which saves the numeric pass one of its three
// dependent loads (0.66 -> 0.61 ms; the symbolic pass 0.43 -> 0.45).  Reading the
// next column's entries ahead of the accumulation gained nothing: the loads of A
// are 16 scattered bytes per product, 3 TB/s from the L2.
template <bool NUMERIC>
__global__ void __launch_bounds__(kWarps * 32, 8) group_spa_kernel(const GroupArgs a, const uint2* __restrict__ order,
                                                                 u64 singles, u32* __restrict__ queue,
                                                                 u64* __restrict__ ucount,
                                                                 const u64* __restrict__ uoff, u64* __restrict__ ck,
                                                                 double* __restrict__ cv) {
  __shared__ u32 s_bits[kWarps][kMaxRows / 32];
  __shared__ double s_acc[NUMERIC ? kWarps : 1][NUMERIC ? kMaxRows : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  u32* bits = s_bits[warp];
  double* acc = s_acc[NUMERIC ? warp : 0];
  constexpr u32 kLong = 24;  // entries of A from which on the warp walks them together
  while (true) {
    u64 first = 0;
    if (lane == 0) first = (u64)atomicAdd(queue, 1u);
    first = __shfl_sync(0xffffffffu, first, 0);
    const u32 grab = first < singles ? 1u : kGrab;
    if (first >= singles) first = singles + (first - singles) * kGrab;
    if (first >= a.units) break;
    const u32 nu = (u32)min((u64)grab, a.units - first);
    // the grab's columns, one per lane
    uint2 mine = make_uint2(0u, 0u), mine_u = make_uint2(0u, 0u);
    u64 mine_off = 0;
    if ((u32)lane < nu) {
      mine_u = order[first + lane];  // (output column, problem)
      mine = a.bcol[mine_u.x];       // (end, count)
      if (NUMERIC) mine_off = uoff[mine_u.x];
    }
    for (u32 i = 0; i < nu; ++i) {
      const u64 u = __shfl_sync(0xffffffffu, mine_u.x, i);
      const uint2 bc = make_uint2(__shfl_sync(0xffffffffu, mine.x, i), __shfl_sync(0xffffffffu, mine.y, i));
      if (bc.y == 0) {
        if (!NUMERIC && lane == 0) ucount[u] = 0;
        continue;
      }
      const ProbDesc& P = a.prob[__shfl_sync(0xffffffffu, mine_u.y, i)];
      const u32 h = (u32)P.h;
      const int hw = (int)((h + 31) / 32);
      if (lane < hw) bits[lane] = 0u;
      if (NUMERIC)
        for (u32 i = lane; i < h; i += 32) acc[i] = 0.0;
      __syncwarp();
      ulonglong2* b = a.brec + (bc.x - bc.y);
      for (u32 e0 = 0; e0 < bc.y; e0 += 32) {
        uint2 ac = make_uint2(0u, 0u);
        double beta = 0.0;
        if (e0 + lane < bc.y) {
          if (NUMERIC) {
            const ulonglong2 rb = b[e0 + lane];
            ac = make_uint2((u32)rb.x, (u32)(rb.x >> 32));
            beta = __longlong_as_double((long long)rb.y);
          } else {
            ac = a.acol[(u32)b[e0 + lane].x];  // (end, count)
            b[e0 + lane].x = (u64)ac.x | ((u64)ac.y << 32);
          }
        }
        u32 many = __ballot_sync(0xffffffffu, ac.y >= kLong);
        while (many) {
          const int j = __ffs(many) - 1;
          many &= many - 1u;
          const u32 end = __shfl_sync(0xffffffffu, ac.x, j), n = __shfl_sync(0xffffffffu, ac.y, j);
          const double bj = __shfl_sync(0xffffffffu, beta, j);
          for (u32 x = end - n + lane; x < end; x += 32) {
            const ulonglong2 ra = a.arec[x];
            const u32 r = (u32)ra.x;
            atomicOr(&bits[r >> 5], 1u << (r & 31));
            if (NUMERIC) atomicAdd(&acc[r], __longlong_as_double((long long)ra.y) * bj);
          }
        }
        if (ac.y < kLong) {
          u32 x = ac.x - ac.y;
          for (; x + 4 <= ac.x; x += 4) {  // four loads before their accumulations
            ulonglong2 ra[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) ra[j] = a.arec[x + j];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const u32 r = (u32)ra[j].x;
              atomicOr(&bits[r >> 5], 1u << (r & 31));
              if (NUMERIC) atomicAdd(&acc[r], __longlong_as_double((long long)ra[j].y) * beta);
            }
          }
          for (; x < ac.x; ++x) {
            const ulonglong2 ra = a.arec[x];
            const u32 r = (u32)ra.x;
            atomicOr(&bits[r >> 5], 1u << (r & 31));
            if (NUMERIC) atomicAdd(&acc[r], __longlong_as_double((long long)ra.y) * beta);
          }
        }
      }
      __syncwarp();
      if (!NUMERIC) {
        const u32 n = __reduce_add_sync(0xffffffffu, lane < hw ? (u32)__popc(bits[lane]) : 0u);
        if (lane == 0) ucount[u] = n;
      } else {
        u64 out = __shfl_sync(0xffffffffu, mine_off, i);
        const u64 colkey = P.h * (u - P.unit_off);
        for (int q = 0; q < hw; ++q) {
          const u32 word = bits[q];
          if (word & (1u << lane)) {
            const u32 r = (u32)q * 32 + lane;
            const u64 o = out + __popc(word & ((1u << lane) - 1u));
            ck[o] = colkey + r;
            cv[o] = acc[r];
          }
          out += __popc(word);
        }
      }
      __syncwarp();
    }
  }
}

// order[.] = (output column, problem) from the problems' order (prepare time).
__global__ void group_order_kernel(const ProbDesc* __restrict__ prob, const uint2* __restrict__ porder,
                                   uint2* __restrict__ order) {
  const uint2 x = porder[blockIdx.x];
  const u64 units = prob[x.x].units, unit0 = prob[x.x].unit_off;
  for (u64 u = threadIdx.x; u < units; u += blockDim.x) order[x.y + u] = make_uint2((u32)(unit0 + u), x.x);
}

// Entries per task: 64 K, less when that would leave SMs without work.
u64 group_chunk(u64 N) {
  const u64 c = std::min<u64>(65536, std::max<u64>(4096, N / ((u64)sm_count() * 8)));
  return align_up(c, kPlace);
}

struct ContractLayout {
  BatchLayout B;
  u64 NA, NB;
  int S;  // lattice key bits of the widest operand
  bool grouped;
  u64 ntasks, nplaces;
  SortPlan plan;
  size_t off_rk, off_aoff, off_boff, off_ck, off_k0, off_v0, off_k1, off_v1, off_ctrl;
  // grouped path ([off_zero, off_zero + zero_bytes) is zeroed by every call)
  size_t off_tasks, off_places, off_porder, off_order, off_kept_n, off_zero, zero_bytes, off_bits_a, off_bits_b, off_bcol, off_counters, off_rank,
      off_acol, off_kept, off_arec, off_brec;
  size_t total;
};

int contract_layout(int count, const int64_t* dims, const uint64_t* a_off, const uint64_t* b_off,
                    ContractLayout* C) {
  int st = batch_layout(count, dims, a_off, b_off, &C->B, nullptr, nullptr, nullptr, true);
  if (st != LNT_OK) return st;
  if (a_off[0] != 0 || b_off[0] != 0) return LNT_BAD_ARG;
  C->NA = a_off[count];
  C->NB = b_off[count];
  const u64 N = C->NA + C->NB;
  if (N >= (1ull << 30)) return LNT_UNSUPPORTED;  // one radix sort of all pairs
  int S = 1;
  for (int p = 0; p < count; ++p) {
    const u64 h = dims[4 * p], w = dims[4 * p + 1], wB = dims[4 * p + 2], d = dims[4 * p + 3];
    S = std::max(S, std::max(key_bits_for(h * w * d), key_bits_for(w * wB * d)));
  }
  if (S + 1 + key_bits_for((u64)count) > 63) return LNT_OVERFLOW_KEYBITS;
  C->S = S;
  size_t off = align_up(C->B.total, 256);
  C->off_rk = off;
  off += align_up((size_t)2 * count * sizeof(RekeyParams), 256);
  C->grouped = grouped_applies(C->B);
  if (C->grouped) {
    auto take = [&](size_t bytes) {
      const size_t o = off;
      off += align_up(std::max<size_t>(bytes, 8), 256);
      return o;
    };
    const u64 chunk = group_chunk(N);
    C->ntasks = C->nplaces = 0;
    for (int p = 0; p < count; ++p)
      for (const uint64_t* o : {a_off, b_off}) {  // (a chunk is a multiple of kPlace)
        const u64 n = o[p + 1] - o[p];
        C->ntasks += (n + chunk - 1) / chunk;
        C->nplaces += (n + kPlace - 1) / kPlace;
      }
    C->off_tasks = take(C->ntasks * sizeof(GroupTask));
    C->off_places = take(C->nplaces * sizeof(uint2));
    C->off_porder = take((size_t)count * sizeof(uint2));
    C->off_order = take(C->B.total_units * sizeof(uint2));
    C->off_kept_n = take(C->ntasks * 4);
    C->off_zero = off;
    C->off_bits_a = take(C->B.words * 4);
    C->off_bits_b = take(C->B.words * 4);
    C->off_bcol = take(C->B.total_units * 8);
    C->off_counters = take(256);
    C->zero_bytes = off - C->off_zero;
    C->off_rank = take(C->B.words * 8);
    C->off_acol = take(std::min(C->NA, std::min(C->NB, C->B.words * 32)) * 8);
    C->off_kept = take(N * 16);
    C->off_arec = take(C->NA * 16);
    C->off_brec = take(C->NB * 16);
    C->total = off;
    return LNT_OK;
  }
  C->plan = make_sort_plan(N, (u64)count << (S + 1));
  C->off_aoff = off;
  off += align_up((size_t)(count + 1) * 8, 256);
  C->off_boff = off;
  off += align_up((size_t)(count + 1) * 8, 256);
  C->off_ck = off;
  off += align_up(N * 8, 256);
  C->off_k0 = off;
  off += align_up(N * 8, 256);
  C->off_v0 = off;
  off += align_up(N * 8, 256);
  C->off_k1 = off;
  off += align_up(N * 8, 256);
  C->off_v1 = off;
  off += align_up(N * 8, 256);
  C->off_ctrl = off;
  off += align_up(C->plan.ctrl_bytes, 256);
  C->total = off;
  return LNT_OK;
}

u32 batch_chunk() {
  if (const char* e = getenv("LNT_BATCH_CHUNK")) {
    const int c = atoi(e);
    if (c >= 1 && c <= 4096) return (u32)c;
  }
  return kTunedBatchChunk;
}

int run_grouped(const ContractLayout& C, const u64* a_keys, const double* a_vals, const u64* b_keys,
                const double* b_vals, unsigned char* w, int count, uint64_t* c_keys, double* c_vals,
                uint64_t* d_c_off, cudaStream_t s) {
  const BatchLayout& L = C.B;
  GroupArgs a;
  a.ak = a_keys;
  a.av = a_vals;
  a.bk = b_keys;
  a.bv = b_vals;
  a.NA = C.NA;
  a.prob = reinterpret_cast<const ProbDesc*>(w + L.off_prob);
  a.rk = reinterpret_cast<const RekeyParams*>(w + C.off_rk);
  a.count = count;
  a.tasks = reinterpret_cast<const GroupTask*>(w + C.off_tasks);
  a.places = reinterpret_cast<const uint2*>(w + C.off_places);
  a.bits_a = reinterpret_cast<u32*>(w + C.off_bits_a);
  a.bits_b = reinterpret_cast<u32*>(w + C.off_bits_b);
  a.words = L.words;
  a.rank = reinterpret_cast<uint2*>(w + C.off_rank);
  a.acol = reinterpret_cast<uint2*>(w + C.off_acol);
  a.bcol = reinterpret_cast<uint2*>(w + C.off_bcol);
  a.units = L.total_units;
  a.kept = reinterpret_cast<uint4*>(w + C.off_kept);
  a.kept_n = reinterpret_cast<u32*>(w + C.off_kept_n);
  a.arec = reinterpret_cast<ulonglong2*>(w + C.off_arec);
  a.brec = reinterpret_cast<ulonglong2*>(w + C.off_brec);
  a.counters = reinterpret_cast<u32*>(w + C.off_counters);
  u64* ucount = reinterpret_cast<u64*>(w + L.off_ucount);
  u64* uoff = reinterpret_cast<u64*>(w + L.off_uoff);
  u32* queue = reinterpret_cast<u32*>(w + L.off_queue);
  const uint2* order = reinterpret_cast<const uint2*>(w + C.off_order);
  const int sms = sm_count();
  if (cudaMemsetAsync(w + C.off_zero, 0, C.zero_bytes, s) != cudaSuccess) return LNT_DEVICE_ERROR;
  if (cudaMemsetAsync(queue, 0, 256, s) != cudaSuccess) return LNT_DEVICE_ERROR;
  if (C.ntasks) {
    const unsigned nt = (unsigned)C.ntasks;
    {
      const u32 sw = (u32)std::min(L.max_words, kGroupSmemWords);
      if (cudaFuncSetAttribute(group_mark_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(kGroupSmemWords * 4)) != cudaSuccess)
        return LNT_DEVICE_ERROR;
      ProfScope prof("batch_mark", s);
      group_mark_kernel<<<nt, kGroupThreads, sw * 4, s>>>(a, sw);
    }
    {
      ProfScope prof("batch_rank", s);
      group_rank_kernel<<<(unsigned)((L.words + kGroupThreads * 8 - 1) / (kGroupThreads * 8)), kGroupThreads, 0, s>>>(a);
    }
    {
      ProfScope prof("batch_filter", s);
      group_filter_kernel<<<nt, kGroupThreads, 0, s>>>(a);
    }
    {
      ProfScope prof("batch_base", s);
      group_base_kernel<<<sms * 8, kGroupThreads, 0, s>>>(a);
    }
    {
      ProfScope prof("batch_place", s);
      group_place_kernel<<<(unsigned)C.nplaces, kGroupThreads, 0, s>>>(a);
    }
    count_launch(5);
  }
  const u64 singles = L.total_units / 8;
  {
    ProfScope prof("batch_spa_symbolic", s);
    group_spa_kernel<false><<<sms * 8, kWarps * 32, 0, s>>>(a, order, singles, queue, ucount, nullptr, nullptr, nullptr);
    count_launch();
  }
  int st = scan::run(U64Of{ucount}, L.total_units, (unsigned long long*)uoff, nullptr, w + L.off_scan, s, "batch_scan");
  if (st != LNT_OK) return st;
  {
    ProfScope prof("batch_spa_numeric", s);
    group_spa_kernel<true><<<sms * 8, kWarps * 32, 0, s>>>(a, order, singles, queue + 1, nullptr, uoff, (u64*)c_keys,
                                                           c_vals);
    count_launch();
  }
  {
    ProfScope prof("batch_coff", s);
    batch_coff_kernel<<<(count + 1 + 255) / 256, 256, 0, s>>>(a.prob, count, uoff, L.total_units, (u64*)d_c_off);
    count_launch();
  }
  return launch_status();
}

int run_batch_product(const BatchArgs& args, const BatchLayout& L, unsigned char* w, int count, uint64_t* c_keys,
                      double* c_vals, uint64_t* d_c_off, cudaStream_t s) {
  int st = LNT_OK;
  u64* ucount = reinterpret_cast<u64*>(w + L.off_ucount);
  u64* uoff = reinterpret_cast<u64*>(w + L.off_uoff);
  u32* queue = reinterpret_cast<u32*>(w + L.off_queue);
  const int sms = sm_count();
  if (cudaMemsetAsync(queue, 0, 256, s) != cudaSuccess) return LNT_DEVICE_ERROR;
  {
    ProfScope prof("batch_colptr", s);
    const int ga = (int)std::max<u64>(1, std::min<u64>((L.a_pos / 8 + 255) / 256, (u64)sms * 16));
    batch_colptr_kernel<<<ga, 256, 0, s>>>(args, 0, reinterpret_cast<const u64*>(w + L.off_apos), L.a_pos);
    const int gb = (int)std::max<u64>(1, std::min<u64>((L.b_pos / 8 + 255) / 256, (u64)sms * 16));
    batch_colptr_kernel<<<gb, 256, 0, s>>>(args, 1, reinterpret_cast<const u64*>(w + L.off_bpos), L.b_pos);
    count_launch(2);
  }
  const u32 chunk = batch_chunk();
  {
    ProfScope prof("batch_spa_symbolic", s);
    int per_sm = 0;  // persistent: as many CTAs as fit
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_spa_kernel<false>, kWarps * 32, 0) != cudaSuccess)
      return LNT_DEVICE_ERROR;
    batch_spa_kernel<false><<<sms * std::max(per_sm, 1), kWarps * 32, 0, s>>>(args, chunk, queue, ucount, nullptr,
                                                                              nullptr, nullptr);
    count_launch();
  }
  st = scan::run(U64Of{ucount}, L.total_units, (unsigned long long*)uoff, nullptr, w + L.off_scan, s, "batch_scan");
  if (st != LNT_OK) return st;
  {
    ProfScope prof("batch_spa_numeric", s);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_spa_kernel<true>, kWarps * 32, 0) != cudaSuccess)
      return LNT_DEVICE_ERROR;
    batch_spa_kernel<true><<<sms * std::max(per_sm, 1), kWarps * 32, 0, s>>>(args, chunk, queue + 1, nullptr, uoff,
                                                                             (u64*)c_keys, c_vals);
    count_launch();
  }
  {
    ProfScope prof("batch_coff", s);
    batch_coff_kernel<<<(count + 1 + 255) / 256, 256, 0, s>>>(args.prob, count, uoff, L.total_units,
                                                               (u64*)d_c_off);
    count_launch();
  }
  return launch_status();
}

}  // namespace
}  // namespace lnt

using namespace lnt;

extern "C" {

int lnt_batched_workspace(int count, const int64_t* dims_host, const uint64_t* a_off_host,
                          const uint64_t* b_off_host, size_t* bytes, uint64_t* c_capacity) {
  if (!bytes) return LNT_BAD_ARG;
  BatchLayout L;
  int st = batch_layout(count, dims_host, a_off_host, b_off_host, &L, nullptr, nullptr, nullptr);
  if (st != LNT_OK) return st;
  *bytes = L.total;
  if (c_capacity) *c_capacity = L.c_bound;
  return LNT_OK;
}

int lnt_batched_prepare(int count, const int64_t* dims_host, const uint64_t* a_off_host,
                        const uint64_t* b_off_host, void* workspace, size_t workspace_bytes, void* stream) {
  BatchLayout L;
  std::vector<ProbDesc> descs;
  std::vector<u64> apos, bpos;
  int st = batch_layout(count, dims_host, a_off_host, b_off_host, &L, &descs, &apos, &bpos);
  if (st != LNT_OK) return st;
  if (!workspace || workspace_bytes < L.total || (uintptr_t)workspace % 256) return LNT_WORKSPACE;
  unsigned char* w = static_cast<unsigned char*>(workspace);
  cudaStream_t s = as_stream(stream);
  // synchronous copies: the host vectors die with this call
  if (cudaStreamSynchronize(s) != cudaSuccess) return LNT_DEVICE_ERROR;
  if (cudaMemcpy(w + L.off_prob, descs.data(), descs.size() * sizeof(ProbDesc), cudaMemcpyHostToDevice) != cudaSuccess)
    return LNT_DEVICE_ERROR;
  if (cudaMemcpy(w + L.off_apos, apos.data(), apos.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess)
    return LNT_DEVICE_ERROR;
  if (cudaMemcpy(w + L.off_bpos, bpos.data(), bpos.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess)
    return LNT_DEVICE_ERROR;
  const std::vector<u32> up = unit_problems(descs, L.total_units);
  if (!up.empty() && cudaMemcpy(w + L.off_uprob, up.data(), up.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess)
    return LNT_DEVICE_ERROR;
  return LNT_OK;
}

int lnt_batched_lattice_mult(int count, const int64_t* dims_host, const uint64_t* a_off_host,
                             const uint64_t* b_off_host, const uint64_t* a_keys, const double* a_vals,
                             const uint64_t* b_keys, const double* b_vals, void* workspace, size_t workspace_bytes,
                             uint64_t* c_keys, double* c_vals, uint64_t* d_c_off, void* stream) {
  BatchLayout L;
  int st = batch_layout(count, dims_host, a_off_host, b_off_host, &L, nullptr, nullptr, nullptr);
  if (st != LNT_OK) return st;
  if (!workspace || workspace_bytes < L.total || (uintptr_t)workspace % 256) return LNT_WORKSPACE;
  if (!d_c_off) return LNT_BAD_ARG;
  if ((L.a_pos > (u64)count && (!a_keys || !a_vals)) || (L.b_pos > (u64)count && (!b_keys || !b_vals)))
    return LNT_BAD_ARG;
  unsigned char* w = static_cast<unsigned char*>(workspace);
  cudaStream_t s = as_stream(stream);
  BatchArgs args;
  args.ak = (const u64*)a_keys;
  args.av = a_vals;
  args.bk = (const u64*)b_keys;
  args.bv = b_vals;
  args.prob = reinterpret_cast<const ProbDesc*>(w + L.off_prob);
  args.count = count;
  args.total_units = L.total_units;
  args.aptr = reinterpret_cast<u32*>(w + L.off_aptr);
  args.bptr = reinterpret_cast<u32*>(w + L.off_bptr);
  args.kmask = ~0ull;
  args.uprob = reinterpret_cast<const u32*>(w + L.off_uprob);
  return run_batch_product(args, L, w, count, c_keys, c_vals, d_c_off, s);
}

}  // extern "C"

extern "C" {

int lnt_batched_contract_workspace(int count, const int64_t* dims_host, const uint64_t* a_off_host,
                                   const uint64_t* b_off_host, size_t* bytes, uint64_t* c_capacity) {
  if (!bytes) return LNT_BAD_ARG;
  ContractLayout C;
  int st = contract_layout(count, dims_host, a_off_host, b_off_host, &C);
  if (st != LNT_OK) return st;
  *bytes = C.total;
  if (c_capacity) *c_capacity = C.B.c_bound;
  return LNT_OK;
}

int lnt_batched_contract_prepare(int count, const int64_t* dims_host, const uint64_t* a_off_host,
                                 const uint64_t* b_off_host, const lnt_rekey_spec* a_rekey_host,
                                 const lnt_rekey_spec* b_rekey_host, void* workspace, size_t workspace_bytes,
                                 void* stream) {
  ContractLayout C;
  int st = contract_layout(count, dims_host, a_off_host, b_off_host, &C);
  if (st != LNT_OK) return st;
  if (!workspace || workspace_bytes < C.total || (uintptr_t)workspace % 256) return LNT_WORKSPACE;
  BatchLayout L;
  std::vector<ProbDesc> descs;
  std::vector<u64> apos, bpos;
  st = batch_layout(count, dims_host, a_off_host, b_off_host, &L, &descs, &apos, &bpos, true);
  if (st != LNT_OK) return st;
  std::vector<RekeyParams> rk(2 * (size_t)count);
  for (int p = 0; p < count; ++p) {
    st = make_rekey_params(a_rekey_host ? &a_rekey_host[p] : nullptr, &rk[p]);
    if (st != LNT_OK) return st;
    st = make_rekey_params(b_rekey_host ? &b_rekey_host[p] : nullptr, &rk[count + p]);
    if (st != LNT_OK) return st;
  }
  std::vector<u32> uprob;
  std::vector<GroupTask> tasks;
  std::vector<uint2> order, places;
  if (!C.grouped) {
    uprob = unit_problems(descs, L.total_units);
  } else {
    // output columns by the expected products per column of their problem
    std::vector<std::pair<double, u32>> weight(count);
    for (int p = 0; p < count; ++p) {
      const ProbDesc& P = descs[p];
      weight[p] = {-(double)P.a_n * (double)P.b_n / ((double)P.w * P.d * P.units), (u32)p};
    }
    std::sort(weight.begin(), weight.end());
    u64 first = 0;
    for (const auto& x : weight) {  // (problem, its first place in the order)
      order.push_back(make_uint2(x.second, (u32)first));
      first += descs[x.second].units;
    }
    const u64 chunk = group_chunk(C.NA + C.NB);
    tasks.reserve(C.ntasks);
    for (int p = 0; p < count; ++p)
      for (u32 which = 0; which < 2; ++which) {
        const uint64_t* o = which ? b_off_host : a_off_host;
        for (u64 x = o[p]; x < o[p + 1]; x += chunk)
          tasks.push_back({x, (u32)std::min<u64>(chunk, o[p + 1] - x), (u32)p | which << 31});
      }
    // the largest first; their pieces in problem order
    std::vector<u32> by_size(tasks.size()), slot(tasks.size());
    for (size_t i = 0; i < tasks.size(); ++i) by_size[i] = (u32)i;
    std::stable_sort(by_size.begin(), by_size.end(), [&](u32 x, u32 y) { return tasks[x].n > tasks[y].n; });
    std::vector<GroupTask> sorted(tasks.size());
    for (size_t i = 0; i < tasks.size(); ++i) {
      sorted[i] = tasks[by_size[i]];
      slot[by_size[i]] = (u32)i;
    }
    places.reserve(C.nplaces);
    for (size_t i = 0; i < tasks.size(); ++i)
      for (u32 x = 0; x < tasks[i].n; x += kPlace) places.push_back(make_uint2(slot[i], x));
    tasks.swap(sorted);
  }
  unsigned char* w = static_cast<unsigned char*>(workspace);
  cudaStream_t s = as_stream(stream);
  // synchronous copies: the host vectors die with this call
  if (cudaStreamSynchronize(s) != cudaSuccess) return LNT_DEVICE_ERROR;
  const struct {
    size_t off;
    const void* src;
    size_t bytes;
  } copies[] = {{L.off_prob, descs.data(), descs.size() * sizeof(ProbDesc)},
                {L.off_apos, apos.data(), apos.size() * 8},
                {L.off_bpos, bpos.data(), bpos.size() * 8},
                {L.off_uprob, uprob.data(), uprob.size() * 4},
                {C.off_rk, rk.data(), rk.size() * sizeof(RekeyParams)},
                {C.grouped ? C.off_tasks : C.off_aoff, C.grouped ? (const void*)tasks.data() : a_off_host,
                 C.grouped ? tasks.size() * sizeof(GroupTask) : (size_t)(count + 1) * 8},
                {C.grouped ? C.off_porder : C.off_boff, C.grouped ? (const void*)order.data() : b_off_host,
                 C.grouped ? order.size() * sizeof(uint2) : (size_t)(count + 1) * 8},
                {C.off_places, places.data(), places.size() * sizeof(uint2)}};
  for (const auto& c : copies)
    if (c.bytes && cudaMemcpy(w + c.off, c.src, c.bytes, cudaMemcpyHostToDevice) != cudaSuccess)
      return LNT_DEVICE_ERROR;
  if (C.grouped) {
    // on the stream of the copies, behind them
    group_order_kernel<<<(unsigned)count, 128, 0, cudaStreamLegacy>>>(
        reinterpret_cast<const ProbDesc*>(w + L.off_prob), reinterpret_cast<const uint2*>(w + C.off_porder),
        reinterpret_cast<uint2*>(w + C.off_order));
    count_launch();
    if (launch_status() != LNT_OK) return LNT_DEVICE_ERROR;
  }
  // the tables are complete when the call returns, for whichever stream runs the batch
  return cudaStreamSynchronize(cudaStreamLegacy) == cudaSuccess ? LNT_OK : LNT_DEVICE_ERROR;
}

int lnt_batched_contract(int count, const int64_t* dims_host, const uint64_t* a_off_host, const uint64_t* b_off_host,
                         const uint64_t* a_keys, const double* a_vals, const uint64_t* b_keys, const double* b_vals,
                         void* workspace, size_t workspace_bytes, uint64_t* c_keys, double* c_vals,
                         uint64_t* d_c_off, void* stream) {
  ContractLayout C;
  int st = contract_layout(count, dims_host, a_off_host, b_off_host, &C);
  if (st != LNT_OK) return st;
  if (!workspace || workspace_bytes < C.total || (uintptr_t)workspace % 256) return LNT_WORKSPACE;
  if (!d_c_off) return LNT_BAD_ARG;
  if ((C.NA && (!a_keys || !a_vals)) || (C.NB && (!b_keys || !b_vals))) return LNT_BAD_ARG;
  unsigned char* w = static_cast<unsigned char*>(workspace);
  cudaStream_t s = as_stream(stream);
  const u64 N = C.NA + C.NB;
  if (C.grouped)
    return run_grouped(C, (const u64*)a_keys, a_vals, (const u64*)b_keys, b_vals, w, count, c_keys, c_vals, d_c_off, s);
  u64* ck = reinterpret_cast<u64*>(w + C.off_ck);
  u64* k0 = reinterpret_cast<u64*>(w + C.off_k0);
  double* v0 = reinterpret_cast<double*>(w + C.off_v0);
  const RekeyParams* rk = reinterpret_cast<const RekeyParams*>(w + C.off_rk);
  const int sms = sm_count();
  {
    ProfScope prof("batch_compose", s);
    // one warp per 256 positions, at most 16 CTAs of 8 warps per SM
    const u64 ga = std::max<u64>(1, std::min<u64>((C.NA + 2047) / 2048, (u64)sms * 16));
    const u64 gb = std::max<u64>(1, std::min<u64>((C.NB + 2047) / 2048, (u64)sms * 16));
    if (C.NA)
      batch_compose_kernel<<<(unsigned)ga, 256, 0, s>>>((const u64*)a_keys, C.NA,
                                                        reinterpret_cast<const uint64_t*>(w + C.off_aoff), count, rk,
                                                        0ull, C.S, ck);
    if (C.NB)
      batch_compose_kernel<<<(unsigned)gb, 256, 0, s>>>((const u64*)b_keys, C.NB,
                                                        reinterpret_cast<const uint64_t*>(w + C.off_boff), count,
                                                        rk + count, 1ull << C.S, C.S, ck + C.NA);
    count_launch(2);
  }
  if (N) {
    PairSource src = plain_source(ck, a_vals, C.NA);
    src.bk = ck + C.NA;
    src.bv = b_vals;
    src.nb = C.NB;
    st = run_sort(C.plan, src, k0, v0, reinterpret_cast<u64*>(w + C.off_k1), reinterpret_cast<double*>(w + C.off_v1),
                  w + C.off_ctrl, s);
    if (st != LNT_OK) return st;
  }
  BatchArgs args;
  args.ak = k0;
  args.av = v0;
  args.bk = k0;
  args.bv = v0;
  args.prob = reinterpret_cast<const ProbDesc*>(w + C.B.off_prob);
  args.count = count;
  args.total_units = C.B.total_units;
  args.aptr = reinterpret_cast<u32*>(w + C.B.off_aptr);
  args.bptr = reinterpret_cast<u32*>(w + C.B.off_bptr);
  args.kmask = (1ull << C.S) - 1ull;
  args.uprob = reinterpret_cast<const u32*>(w + C.B.off_uprob);
  return run_batch_product(args, C.B, w, count, c_keys, c_vals, d_c_off, s);
}

}  // extern "C"
