// Merge of two key-sorted operands (the scan-merge path) and the fused
// re-key + sort entry point.
//
// lnt_merge_sorted reproduces outside_merge_sparse_storage_containers
// (FunctionUtil.h:373-419): walking both arrays, A-only keys are copied,
// B-only keys become op(0, b), and equal keys consume one A and one B into
// op(a, b).  Within a run of equal keys this pairs the j-th A with the j-th B;
// surplus A's are copied and surplus B's become op(0, b).
//
// GPU formulation: the stable merge of A and B (A first on ties) is split by
// merge-path diagonals into tiles of 1536 merged elements.  In that order the
// j-th A of a key run sits before every B of the run, so each element decides
// locally (from its merged position and at most two neighbour reads) whether
// it is emitted and with which partner:
//   A_i with key k: lbB = (merged position) - i is the first B with key k;
//     j = occurrence of k in A up to i; partner B[lbB + j] if it has key k.
//   B_i with key k: ubA = (merged position) - i is one past the last A with
//     key k; j = occurrence of k in B up to i; B_i is consumed iff
//     A[ubA - 1 - j] has key k.
// A partition kernel finds every tile's split first (one merge-path search per
// tile boundary, all in parallel); each tile then stages its A and B slices
// (keys and values) in shared memory with coalesced loads, and run indices and
// partners are read from there - global memory only when a run of equal keys
// crosses the slice boundary.  Emitted elements keep merged order; their output
// offsets come from a block scan plus a decoupled look-back over tiles.
// A tile in which no key repeats inside an operand (checked on the staged keys)
// needs none of the run bookkeeping: an A meets at most the B at hand, a B only
// the A taken last.
// CTAs are persistent and the look-back is off their path: a ninth warp runs it
// while the other eight go on with the CTA's next tile, and a tile's elements
// wait for their offset in shared memory, in one of two buffers.  (When every
// warp waited for the offset, 40% of the stalls were at that barrier.)  Tile ids
// are taken as late as possible: the longer a CTA sits on an id, the longer the
// others look back.
// Traffic: 16 B read per input pair + 16 B written per output pair; bound by the
// latency of a tile's steps.  20M + 12M pairs 0.41 ms (0.47 before the ninth
// warp), 2 x 2^26 pairs 1.75 ms (2.04), 2 x 2^24 with many repeats 0.57 (0.60).
// Also measured for the first two: tiles of 2048 with three CTAs per SM 0.41 and
// 1.85, of 1024 with four 0.44 and 1.82; the next id taken before the merge (at
// 2048) 0.43 and 1.89; the next tile's loads held in registers across the write
// 0.50 and 2.2.
#include <algorithm>

#include "lnt_msd.cuh"

namespace lnt {
namespace {

constexpr int kThreads = 256;
constexpr int kItems = 6;
constexpr int kCtas = 4;  // per SM: 54 KB of shared memory and 56 registers a thread
constexpr int kTile = kThreads * kItems;
constexpr unsigned long long kFlagAgg = 1ull << 62;
constexpr unsigned long long kFlagPre = 2ull << 62;
constexpr unsigned long long kFlagMask = 3ull << 62;
constexpr unsigned long long kValMask = (1ull << 62) - 1ull;

// Number of A elements among the first d of the stable merge (A first on ties).
__device__ __forceinline__ size_t merge_path(const u64* __restrict__ a, size_t na, const u64* __restrict__ b,
                                             size_t nb, size_t d) {
  size_t lo = d > nb ? d - nb : 0;
  size_t hi = d < na ? d : na;
  while (lo < hi) {
    const size_t mid = (lo + hi) >> 1;
    if (a[mid] <= b[d - 1 - mid])
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// Shared-memory place of slice element i: a thread's elements are 32 or 64
// bytes from its neighbour's, so a spare word pair per 16 elements spreads a
// warp's accesses over the banks (0.46 -> 0.41 ms on 20M + 12M pairs).
__device__ __forceinline__ int pad(int i) { return i + (i >> 4); }
constexpr int kPadded = kTile + kTile / 16;

// Same search over the padded slices (A, then B from la on).
__device__ __forceinline__ int merge_path_smem(const u64* k, int la, int lb, int d) {
  int lo = d > lb ? d - lb : 0;
  int hi = d < la ? d : la;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (k[pad(mid)] <= k[pad(la + d - 1 - mid)])
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// Occurrence index of x[i] within its run of equal keys.
__device__ __forceinline__ size_t run_index(const u64* __restrict__ x, size_t i, u64 k) {
  size_t j = 0;
  while (i > j && x[i - 1 - j] == k) ++j;
  return j;
}

__device__ __forceinline__ double apply_op(int op, double a, double b) { return op == 0 ? a + b : a - b; }

// splits[t] = A elements among the first min(t * kTile, na + nb) of the merge.
// (Split: 32 bits for fewer than 2^32 pairs, which keeps the scratch at 12 bytes
// per tile.)
template <class Split>
__global__ void merge_partition_kernel(const u64* __restrict__ a, size_t na, const u64* __restrict__ b, size_t nb,
                                       u32 ntiles, Split* __restrict__ splits) {
  const u32 t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t > ntiles) return;
  splits[t] = (Split)merge_path(a, na, b, nb, min(na + nb, (size_t)t * kTile));
}

// Barriers of part of a CTA (ids 1..; 0 is __syncthreads).
__device__ __forceinline__ void bar_sync(int id, int threads) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ bool bar_or(int id, int threads, bool p) {
  int r;
  __syncwarp();
  asm volatile("{.reg .pred p, q; setp.ne.s32 p, %3, 0; bar.red.or.pred q, %1, %2, p; selp.s32 %0, 1, 0, q;}"
               : "=r"(r)
               : "r"(id), "r"(threads), "r"((int)p)
               : "memory");
  return r != 0;
}
constexpr int kMainBar = 1, kReqBar = 2, kOffBar = 4;  // the last two for both buffers
constexpr int kMergeSmem = 2 * kPadded * 16;

template <class Split>
__global__ void __launch_bounds__(kThreads + 32, kCtas)
    merge_kernel(const u64* __restrict__ ak, const double* __restrict__ av, size_t na, const u64* __restrict__ bk,
                 const double* __restrict__ bv, size_t nb, int op, u32 ntiles, const Split* __restrict__ splits,
                 unsigned long long* __restrict__ status, u32* __restrict__ tile_counter, u64* __restrict__ ck,
                 double* __restrict__ cv, u64* __restrict__ d_nout) {
  extern __shared__ u64 smem[];
  __shared__ u32 s_warp[kThreads / 32];
  __shared__ u32 s_tile, s_rt[2], s_tot[2];
  __shared__ unsigned long long s_off[2];
  __shared__ u64 s_edge[3];
  __shared__ double s_edge_v;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (warp == kThreads / 32) {
    // ---- look-back for the tiles' output offsets ----------------------------
    for (int buf = 0;; buf ^= 1) {
      bar_sync(kReqBar + buf, 64);
      const u32 tile = *(volatile u32*)&s_rt[buf], tot = *(volatile u32*)&s_tot[buf];
      if (tile >= ntiles) return;
      unsigned long long off = 0;
      if (tile != 0) {
        int base = (int)tile - 1;
        u32 spins = 0;
        while (base >= 0) {
          const int p = base - lane;
          const unsigned long long w =
              p >= 0 ? *reinterpret_cast<const volatile unsigned long long*>(status + p) : kFlagPre;
          const unsigned long long f = w & kFlagMask;
          const u32 notready = __ballot_sync(0xffffffffu, f == 0);
          const u32 pre = __ballot_sync(0xffffffffu, f == kFlagPre);
          const int first_nr = notready ? __ffs(notready) - 1 : 32;
          const int first_pre = pre ? __ffs(pre) - 1 : 32;
          const int take = first_pre < first_nr ? first_pre + 1 : first_nr;
          unsigned long long v = lane < take ? (w & kValMask) : 0ull;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          off += v;
          if (first_pre < first_nr) break;
          base -= first_nr;
          if (first_nr < 32 && ++spins > spin_limit()) {
            latch_error(kErrMergeLookback);
            break;
          }
        }
        if (lane == 0) *reinterpret_cast<volatile unsigned long long*>(&status[tile]) = kFlagPre | (off + tot);
      }
      if (lane == 0) {
        s_off[buf] = off;
        if (tile == ntiles - 1) *d_nout = off + tot;
      }
      __syncwarp();
      bar_arrive(kOffBar + buf, kThreads + 32);
    }
  }
  const size_t total = na + nb;
  u32 held = 0;  // elements of the previous tile, still to be written
  auto write_held = [&](int b) {
    const u64* h_k = smem + b * 2 * kPadded;
    const double* h_v = reinterpret_cast<const double*>(h_k + kPadded);
    bar_sync(kOffBar + b, kThreads + 32);
    const unsigned long long off = *(volatile unsigned long long*)&s_off[b];
    for (u32 i = tid; i < held; i += kThreads) {
      __stcs(ck + off + i, h_k[pad(i)]);
      __stcs(cv + off + i, h_v[pad(i)]);
    }
  };
  for (int n = 0;; ++n) {
    const int buf = n & 1;
    u64* s_k = smem + buf * 2 * kPadded;
    double* s_v = reinterpret_cast<double*>(s_k + kPadded);
    if (tid == 0) s_tile = atomicAdd(tile_counter, 1u);
    bar_sync(kMainBar, kThreads);  // also: the buffer's last tile is written
    const u32 tile = s_tile;
    if (tile >= ntiles) {
      if (warp == 0) {  // ends the look-back warp
        if (lane == 0) s_rt[buf] = tile;
        bar_arrive(kReqBar + buf, 64);
      }
      if (n > 0) write_held(buf ^ 1);
      return;
    }
    const size_t d0 = (size_t)tile * kTile;
    const size_t d1 = min(total, d0 + kTile);
    const size_t a0 = splits[tile], a1 = splits[tile + 1];
    const size_t b0 = d0 - a0, b1 = d1 - a1;
    const int la = (int)(a1 - a0), lb = (int)(b1 - b0);
    if (warp == kThreads / 32 - 1) {  // what lies just outside the slices
      if (lane == 0 && a0 > 0) s_edge[0] = ak[a0 - 1];
      if (lane == 1 && b1 < nb) s_edge[1] = bk[b1];
      if (lane == 2 && b1 < nb) s_edge_v = bv[b1];
      if (lane == 3 && b0 > 0) s_edge[2] = bk[b0 - 1];
    }
    // stage the tile's A slice then its B slice, keys and values, in shared memory
    for (int i = tid; i < la + lb; i += kThreads) {
      if (i < la) {
        s_k[pad(i)] = __ldcs(ak + a0 + i);
        s_v[pad(i)] = __ldcs(av + a0 + i);
      } else {
        s_k[pad(i)] = __ldcs(bk + b0 + (i - la));
        s_v[pad(i)] = __ldcs(bv + b0 + (i - la));
      }
    }
    bar_sync(kMainBar, kThreads);
    // a key repeated inside an operand (also across the slice's start)?
    bool repeat = false;
    for (int i = tid; i < la + lb; i += kThreads) {
      const bool first = i == 0 || i == la;
      repeat = repeat || (first ? (i < la ? a0 > 0 && s_k[pad(i)] == s_edge[0] : b0 > 0 && s_k[pad(i)] == s_edge[2])
                                : s_k[pad(i)] == s_k[pad(i - 1)]);
    }
    // each thread merges kItems consecutive merged positions
    const int dt = min(tid * kItems, la + lb);
    int ia = merge_path_smem(s_k, la, lb, dt);
    int ib = dt - ia;
    u32 emit = 0;  // bit q: item q is written
    u64 ek[kItems];
    double evv[kItems];
    if (!bar_or(kMainBar, kThreads, repeat)) {
      // no: an A meets at most the B at hand, a B only the last A
      u64 ka = ia < la ? s_k[pad(ia)] : ~0ull, kb = ib < lb ? s_k[pad(la + ib)] : s_edge[1];
      u64 last = ia > 0 ? s_k[pad(ia - 1)] : s_edge[0];
      bool any_last = a0 + ia > 0;
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        ek[q] = 0;
        evv[q] = 0.0;
        if (dt + q >= la + lb) continue;
        if (ib >= lb || (ia < la && ka <= kb)) {
          double v = s_v[pad(ia)];
          if (kb == ka && (ib < lb || b1 < nb)) v = apply_op(op, v, ib < lb ? s_v[pad(la + ib)] : s_edge_v);
          emit |= 1u << q;
          ek[q] = ka;
          evv[q] = v;
          last = ka;
          any_last = true;
          ++ia;
          ka = ia < la ? s_k[pad(ia)] : ~0ull;
        } else {
          if (!any_last || last != kb) {
            emit |= 1u << q;
            ek[q] = kb;
            evv[q] = apply_op(op, 0.0, s_v[pad(la + ib)]);
          }
          ++ib;
          kb = ib < lb ? s_k[pad(la + ib)] : s_edge[1];
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        ek[q] = 0;
        evv[q] = 0.0;
        const int m = dt + q;
        if (m >= la + lb) continue;
        const bool take_a = ib >= lb || (ia < la && s_k[pad(ia)] <= s_k[pad(la + ib)]);
        const size_t mg = d0 + (size_t)m;  // global merged position
        if (take_a) {
          const size_t i = a0 + ia;
          const u64 k = s_k[pad(ia)];
          const size_t lbB = mg - i;  // B elements before A_i: those with key < k
          size_t j = 0;               // occurrence of k in A before A_i
          while ((int)j < ia && s_k[pad(ia - 1 - j)] == k) ++j;
          if ((int)j == ia) j += run_index(ak, a0, k);
          double v = s_v[pad(ia)];
          const size_t pb = lbB + j;  // the partner B, if it has key k
          if (pb >= b0 && pb < b1) {
            if (s_k[pad(la + (int)(pb - b0))] == k) v = apply_op(op, v, s_v[pad(la + (int)(pb - b0))]);
          } else if (pb < nb && bk[pb] == k) {
            v = apply_op(op, v, bv[pb]);
          }
          emit |= 1u << q;
          ek[q] = k;
          evv[q] = v;
          ++ia;
        } else {
          const size_t i = b0 + ib;
          const u64 k = s_k[pad(la + ib)];
          const size_t ubA = mg - i;  // A elements before B_i: those with key <= k
          size_t j = 0;               // occurrence of k in B before B_i
          while ((int)j < ib && s_k[pad(la + ib - 1 - j)] == k) ++j;
          if ((int)j == ib) j += run_index(bk, b0, k);
          bool consumed = false;
          if (ubA >= j + 1) {
            const size_t pa = ubA - 1 - j;  // the A it would pair with
            consumed = (pa >= a0 && pa < a1) ? s_k[pad((int)(pa - a0))] == k : ak[pa] == k;
          }
          if (!consumed) {
            emit |= 1u << q;
            ek[q] = k;
            evv[q] = apply_op(op, 0.0, s_v[pad(la + ib)]);
          }
          ++ib;
        }
      }
    }
    const u32 nemit = __popc(emit);
    // ---- block scan of emitted counts -------------------------------------
    u32 inc = nemit;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    bar_sync(kMainBar, kThreads);
    u32 excl = inc - nemit, tot = 0;
    for (int w = 0; w < kThreads / 32; ++w) {
      if (w < warp) excl += s_warp[w];
      tot += s_warp[w];
    }
    if (tid == 0)
      *reinterpret_cast<volatile unsigned long long*>(&status[tile]) = (tile == 0 ? kFlagPre : kFlagAgg) | tot;
    // the emitted elements to the front (every thread is past its reads)
    u32 r = excl;
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
      if (emit & (1u << q)) {
        s_k[pad(r)] = ek[q];
        s_v[pad(r)] = evv[q];
        ++r;
      }
    }
    if (warp == 0) {  // hand the tile to the look-back warp
      if (lane == 0) {
        s_rt[buf] = tile;
        s_tot[buf] = tot;
      }
      bar_arrive(kReqBar + buf, 64);
    }
    if (n > 0) write_held(buf ^ 1);
    held = tot;
  }
}

}  // namespace

struct MergeLayout {
  u32 ntiles;
  size_t off_status, off_counter, off_splits, total;
};

static MergeLayout merge_layout(size_t n) {
  MergeLayout L;
  L.ntiles = (u32)((n + kTile - 1) / kTile);
  L.off_status = 0;
  L.off_counter = (size_t)std::max<u32>(L.ntiles, 1) * 8;
  L.off_splits = L.off_counter + 8;
  L.total = align_up(L.off_splits + ((size_t)L.ntiles + 1) * (n >> 32 ? 8 : 4), 256);
  return L;
}

template <class Split>
static int run_merge(const MergeLayout& L, const u64* ak, const double* av, size_t na, const u64* bk, const double* bv,
                     size_t nb, int op, u64* ck, double* cv, u64* d_nout, unsigned char* w, cudaStream_t s) {
  Split* splits = reinterpret_cast<Split*>(w + L.off_splits);
  if (cudaMemsetAsync(w, 0, L.off_splits, s) != cudaSuccess) return LNT_DEVICE_ERROR;
  if (cudaFuncSetAttribute(merge_kernel<Split>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMergeSmem) != cudaSuccess)
    return LNT_DEVICE_ERROR;
  ProfScope prof("merge", s);
  merge_partition_kernel<Split><<<(L.ntiles + 1 + 255) / 256, 256, 0, s>>>(ak, na, bk, nb, L.ntiles, splits);
  const u32 grid = std::min<u32>(L.ntiles, (u32)kCtas * (u32)sm_count());
  merge_kernel<Split><<<grid, kThreads + 32, kMergeSmem, s>>>(
      ak, av, na, bk, bv, nb, op, L.ntiles, splits, reinterpret_cast<unsigned long long*>(w + L.off_status),
      reinterpret_cast<u32*>(w + L.off_counter), ck, cv, d_nout);
  count_launch(2);
  return launch_status();
}

}  // namespace lnt

using namespace lnt;

namespace {
struct PermuteSortLayout {
  PairSort sort;
  size_t off_ctrl, off_a, off_b, total;
};
PermuteSortLayout permute_sort_layout(size_t n, u64 max_key, bool buckets = true) {
  PermuteSortLayout L;
  L.sort = make_pair_sort(n, max_key, buckets);
  size_t off = 0;
  L.off_ctrl = off;
  off += align_up(L.sort.ctrl_bytes, 256);
  L.off_a = off;
  off += L.sort.a_bytes;
  L.off_b = off;
  off += L.sort.b_bytes;
  L.total = off;
  return L;
}
}  // namespace

extern "C" {

int lnt_merge_sorted_workspace(size_t na, size_t nb, size_t* bytes) {
  if (!bytes) return LNT_BAD_ARG;
  *bytes = merge_layout(na + nb).total;
  return LNT_OK;
}

int lnt_merge_sorted(const uint64_t* a_keys, const double* a_vals, size_t na, const uint64_t* b_keys,
                     const double* b_vals, size_t nb, int op, uint64_t* c_keys, double* c_vals, uint64_t* d_nout,
                     void* workspace, size_t workspace_bytes, void* stream) {
  if (!d_nout || (op != 0 && op != 1)) return LNT_BAD_ARG;
  if ((na && (!a_keys || !a_vals)) || (nb && (!b_keys || !b_vals))) return LNT_BAD_ARG;
  const size_t n = na + nb;
  cudaStream_t s = as_stream(stream);
  if (n == 0) return cudaMemsetAsync(d_nout, 0, 8, s) == cudaSuccess ? LNT_OK : LNT_DEVICE_ERROR;
  if (!c_keys || !c_vals) return LNT_BAD_ARG;
  MergeLayout L = merge_layout(n);
  if (!workspace || workspace_bytes < L.total) return LNT_WORKSPACE;
  auto run = n >> 32 ? run_merge<u64> : run_merge<u32>;
  return run(L, (const u64*)a_keys, a_vals, na, (const u64*)b_keys, b_vals, nb, op, (u64*)c_keys, c_vals, (u64*)d_nout,
             static_cast<unsigned char*>(workspace), s);
}

int lnt_permute_sort_workspace(size_t n, uint64_t max_key, size_t* bytes) {
  if (!bytes) return LNT_BAD_ARG;
  if (n >= (1u << 30)) return LNT_UNSUPPORTED;
  *bytes = permute_sort_layout(n, max_key).total;
  return LNT_OK;
}

int lnt_permute_sort(const uint64_t* keys_in, const double* vals_in, size_t n, const lnt_rekey_spec* rekey,
                     uint64_t* keys_out, double* vals_out, uint64_t max_key, void* workspace,
                     size_t workspace_bytes, void* stream) {
  if (n == 0) return LNT_OK;
  if (!keys_in || !vals_in || !keys_out || !vals_out) return LNT_BAD_ARG;
  if ((const void*)keys_in == (const void*)keys_out || (const void*)vals_in == (const void*)vals_out)
    return LNT_BAD_ARG;  // out of place only
  if (n >= (1u << 30)) return LNT_UNSUPPORTED;
  PermuteSortLayout L = permute_sort_layout(n, max_key);
  if (workspace_bytes < L.total) L = permute_sort_layout(n, max_key, false);  // the digit passes may need less
  if (!workspace || workspace_bytes < L.total) return LNT_WORKSPACE;
  if ((uintptr_t)workspace % 256) return LNT_BAD_ARG;
  PairSource src = plain_source((const u64*)keys_in, vals_in, n);
  int st = make_rekey_params(rekey, &src.ra);
  if (st != LNT_OK) return st;
  unsigned char* w = static_cast<unsigned char*>(workspace);
  return run_pair_sort(L.sort, src, (u64*)keys_out, vals_out, w + L.off_a, w + L.off_b, w + L.off_ctrl,
                       as_stream(stream));
}

}  // extern "C"
