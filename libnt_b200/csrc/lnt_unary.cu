// Unary contraction / attraction of a sparse tensor: the reference's
// SparseMIABase::contract_attract (SparseMIABase.h:1913-2053), reached from
// index labels that repeat inside one operand (perform_unary, MIA_Expr.h:
// 690-735), e.g. b(k) = a(i,j,i,j,k) (a double trace) or b(k,!i) =
// a(!i,j,!i,k,j).
//
// Input: keys sorted under [contraction modes, attraction modes, other modes]
// with those modes' extents sdims.
//   1. unary_fold_kernel: one read of the keys, and of the values whose
//      contraction sets agree (the others are not summed).  Every warp folds a
//      chunk of consecutive entries into one partial sum per group key g = key
//      / |contraction modes| (equal attraction + other indices), the
//      reference's inner summation loop.  No warp waits for another: the
//      partial sums go to the chunk's own slots, and their number to a table.
//   2. scan_kernel + unary_gather_kernel: the chunks' partial sums made
//      contiguous (at most one per group and one per chunk).
//   3. collect_runs_kernel (lnt_collect.cuh) adds up the partial sums of each
//      group and keeps a group when its attraction sets agree and its sum is
//      not zero (the reference's "if (sum)"); key other + |other| * attraction
//      index, in the groups' order (the reference's emission order).
//   4. unary_sorted_kernel flags whether those keys never decrease (the
//      result's sorted flag, as push_back maintains it).
// HBM bound: 8 B per entry and 8 B per agreeing entry read.  Measured on 6.7e7
// entries in 65,536 groups, a tenth of them agreeing (B200): fold 0.25 ms,
// everything 0.29 ms, against 1.58 ms when the entries were mapped, folded,
// scanned and written by kernels that each passed over them.  Folding in one
// pass with a look-back per tile of 2048 took 0.58 ms (0.37 ms of it without
// the look-back); two CTAs per SM 0.28 ms, four (64 registers, spilling) 0.27.
#include <algorithm>

#include "lnt_collect.cuh"
#include "lnt_scan.cuh"

namespace lnt {

namespace {

struct UnaryParams {
  int order;      // modes in the sorted sequence
  int ncon_sets;  // contraction sets, over the first ncon modes
  int natt_sets;  // attraction sets, over the next natt modes
  int ncon, natt;
  int con_part[LNT_MAX_ORDER];
  int att_part[LNT_MAX_ORDER];
  Divider sd[LNT_MAX_ORDER];  // extents in sorted order
  Divider cdim;               // product of the contraction extents
  Divider afull;              // product of the attraction extents
  u64 other_dim;              // product of the other extents
};

// Clears ok[j] where one of the sets of consecutive digits of c[j] disagrees
// (the loops over the modes are outside the one over the entries).
template <int I>
__device__ __forceinline__ void sets_agree(u64 (&c)[I], bool (&ok)[I], const Divider* sd, const int* part, int nsets) {
  int q = 0;
#pragma unroll 1
  for (int p = 0; p < nsets; ++p) {
    const Divider dv = sd[q];  // the extents of a set are equal
    u64 d0[I];
#pragma unroll
    for (int j = 0; j < I; ++j) {
      const u64 nk = divide(c[j], dv);
      d0[j] = c[j] - nk * dv.d;
      c[j] = nk;
    }
#pragma unroll 1
    for (int t = 1; t < part[p]; ++t) {
#pragma unroll
      for (int j = 0; j < I; ++j) {
        const u64 nk = p == nsets - 1 && t == part[p] - 1 ? 0 : divide(c[j], dv);  // (the last digit is what is left)
        ok[j] = ok[j] && c[j] - nk * dv.d == d0[j];
        c[j] = nk;
      }
    }
    q += part[p];
  }
}

constexpr int kFoldThreads = 256, kFoldRows = 8, kFoldBatch = 32 * kFoldRows;

// One warp per chunk of `chunk` (a multiple of 256) entries, in batches of
// eight rows of 32.  A row inside the open run only adds to the lanes' partial
// sums; a row with heads closes the open run by a reduction over the warp, and
// the runs inside it by a segmented scan.
__global__ void __launch_bounds__(kFoldThreads, 3) unary_fold_kernel(const u64* __restrict__ keys,
                                                                     const double* __restrict__ vals, size_t n,
                                                                     u32 chunk, u32 nchunks, const UnaryParams P,
                                                                     u64* __restrict__ gk, double* __restrict__ gv,
                                                                     u32* __restrict__ counts) {
  constexpr int R = kFoldRows;
  constexpr u32 FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const u32 le = lane == 31 ? FULL : (2u << lane) - 1u;  // this lane and those before it
  const u32 ci = (u32)((blockIdx.x * (size_t)kFoldThreads + threadIdx.x) >> 5);
  if (ci >= nchunks) return;
  const size_t begin = (size_t)ci * chunk, end = min(n, begin + chunk);
  gk += begin;
  gv += begin;
  u64 last = divide(__ldg(keys + begin), P.cdim);  // the open run's group
  double acc = 0.0;                                // this lane's part of it
  u32 cnt = 0;
  for (size_t base = begin; base < end; base += kFoldBatch) {
    u64 g[R], con[R];
    double v[R];
    bool ok[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const size_t i = base + r * 32 + lane;
      con[r] = i < end ? __ldcs(keys + i) : 0;
      ok[r] = i < end;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      g[r] = divide(con[r], P.cdim);
      con[r] -= g[r] * P.cdim.d;
    }
    sets_agree(con, ok, P.sd, P.con_part, P.ncon_sets);
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ok[r] ? __ldcs(vals + base + r * 32 + lane) : 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool valid = base + r * 32 + lane < end;
      if (__all_sync(FULL, !valid || g[r] == last)) {
        acc += v[r];
        continue;
      }
      u64 prev = __shfl_up_sync(FULL, g[r], 1);
      if (lane == 0) prev = last;
      const u32 heads = __ballot_sync(FULL, valid && g[r] != prev);
      const int first = __ffs(heads) - 1, newest = 31 - __clz(heads);
      double open = acc + (lane < first ? v[r] : 0.0);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) open += __shfl_xor_sync(FULL, open, o);
      if (lane == 0) {
        gk[cnt] = last;
        gv[cnt] = open;
      }
      if (first != newest) {  // runs that begin and end in this row
        const u32 mine = heads & le;
        const int start = mine ? 31 - __clz(mine) : 0;
        double x = v[r];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double y = __shfl_up_sync(FULL, x, o);
          if (lane - o >= start) x = y + x;
        }
        if (mine && ((heads >> 1) >> lane & 1u)) {  // the last entry of its run
          gk[cnt + __popc(mine)] = g[r];
          gv[cnt + __popc(mine)] = x;
        }
      }
      cnt += __popc(heads);
      last = __shfl_sync(FULL, g[r], newest);
      acc = lane >= newest ? v[r] : 0.0;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
  if (lane == 0) {
    gk[cnt] = last;
    gv[cnt] = acc;
    counts[ci] = cnt + 1;
  }
}

struct CountOf {
  const u32* counts;
  __device__ __forceinline__ u64 operator()(size_t i) const { return counts[i]; }
};

// Chunk i's partial sums (at i * chunk) to pos[i] (one warp per chunk).
// (counts, not pos[i + 1] - pos[i]: after an expired look-back of the scan that
// difference could be negative.)
__global__ void __launch_bounds__(256) unary_gather_kernel(const u64* __restrict__ gk, const double* __restrict__ gv,
                                                           const u32* __restrict__ counts, u32 chunk, u32 nchunks,
                                                           const unsigned long long* __restrict__ pos,
                                                           u64* __restrict__ ck, double* __restrict__ cv) {
  const int lane = threadIdx.x & 31;
  const u32 ci = (u32)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
  if (ci >= nchunks) return;
  const u64 to = pos[ci];
  const u32 cnt = counts[ci];
  const size_t from = (size_t)ci * chunk;
#pragma unroll 4
  for (u32 j = lane; j < cnt; j += 32) {
    ck[to + j] = gk[from + j];
    cv[to + j] = gv[from + j];
  }
}

struct UnaryGroups {
  UnaryParams P;
  __device__ __forceinline__ bool keep(u64 g, double sum) const {
    if (sum == 0.0) return false;
    u64 c[1] = {g - divide(g, P.afull) * P.afull.d};
    bool ok[1] = {true};
    sets_agree(c, ok, P.sd + P.ncon, P.att_part, P.natt_sets);
    return ok[0];
  }
  __device__ __forceinline__ u64 out_key(u64 g) const {
    const u64 other = divide(g, P.afull);
    u64 c = g - other * P.afull.d, att = 0, stride = 1;
    int q = P.ncon;
    for (int p = 0; p < P.natt_sets; ++p) {  // sub2ind over the attraction ranges
      for (int t = 0; t < P.att_part[p]; ++t, ++q) {
        const u64 nk = divide(c, P.sd[q]);
        if (t == 0) {
          att += (c - nk * P.sd[q].d) * stride;
          stride *= P.sd[q].d;
        }
        c = nk;
      }
    }
    return other + P.other_dim * att;
  }
};

__global__ void unary_sorted_kernel(const u64* __restrict__ out_k, const u64* __restrict__ d_nout,
                                    u32* __restrict__ d_sorted) {
  const u64 m = *d_nout;
  const u64 stride = (u64)gridDim.x * blockDim.x;
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x + 1; i < m; i += stride)
    if (out_k[i] < out_k[i - 1]) *d_sorted = 0u;
}

// Entries per warp: 256, growing with n to 2048 (fewer partial sums) while
// every SM still has 32 warps.
u32 fold_chunk(size_t n) {
  u32 c = kFoldBatch;
  while (c < 2048 && n / (2 * c) >= (size_t)sm_count() * 32) c *= 2;
  return c;
}

struct UnaryLayout {
  u32 chunk, nchunks;
  size_t counts, pos, scan, gk, gv, ck, cv, coll, total;
};

UnaryLayout unary_layout(size_t n) {
  UnaryLayout L;
  L.chunk = fold_chunk(n);
  L.nchunks = (u32)((n + L.chunk - 1) / L.chunk);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += align_up(std::max<size_t>(bytes, 8), 256);
    return o;
  };
  L.counts = take((size_t)L.nchunks * 4);
  L.pos = take(((size_t)L.nchunks + 1) * 8);
  L.scan = take(scan::workspace_bytes(L.nchunks));
  L.gk = take(n * 8);
  L.gv = take(n * 8);
  L.ck = take(n * 8);
  L.cv = take(n * 8);
  L.coll = take(collect::layout(n).total);
  L.total = off;
  return L;
}

int grid_n(u64 work) {
  const u64 want = (work + 255) / 256;
  const u64 cap = (u64)sm_count() * 8;
  return (int)std::max<u64>(1, std::min(want, cap));
}

}  // namespace
}  // namespace lnt

using namespace lnt;

extern "C" {

int lnt_contract_attract_workspace(size_t n, size_t* bytes) {
  if (!bytes) return LNT_BAD_ARG;
  *bytes = unary_layout(n).total;
  return LNT_OK;
}

int lnt_contract_attract(const uint64_t* keys, const double* vals, size_t n, int order, const int64_t* sdims,
                         int ncon_sets, const int* con_part, int natt_sets, const int* att_part, uint64_t* out_keys,
                         double* out_vals, uint64_t* d_nout, uint32_t* d_sorted, void* workspace,
                         size_t workspace_bytes, void* stream) {
  if (order < 1 || order > LNT_MAX_ORDER || !sdims || ncon_sets < 0 || natt_sets < 0 || !d_nout) return LNT_BAD_ARG;
  if ((ncon_sets && !con_part) || (natt_sets && !att_part)) return LNT_BAD_ARG;
  if (n && (!keys || !vals || !out_keys || !out_vals)) return LNT_BAD_ARG;
  UnaryParams P{};
  P.order = order;
  P.ncon_sets = ncon_sets;
  P.natt_sets = natt_sets;
  unsigned __int128 total = 1;
  for (int q = 0; q < order; ++q) {
    if (sdims[q] <= 0) return LNT_BAD_DIMS;
    P.sd[q] = make_divider((u64)sdims[q]);
    total *= (u64)sdims[q];
  }
  if (total >> 63) return LNT_OVERFLOW_KEYBITS;
  int m = 0;
  u64 cd = 1, ad = 1, od = 1;
  for (int p = 0; p < ncon_sets; ++p) {
    if (con_part[p] < 2 || m + con_part[p] > order) return LNT_BAD_ARG;
    for (int q = m; q < m + con_part[p]; ++q) {
      if (sdims[q] != sdims[m]) return LNT_BAD_DIMS;  // a contraction set runs over equal extents
      cd *= (u64)sdims[q];
    }
    P.con_part[p] = con_part[p];
    m += con_part[p];
  }
  P.ncon = m;
  for (int p = 0; p < natt_sets; ++p) {
    if (att_part[p] < 2 || m + att_part[p] > order) return LNT_BAD_ARG;
    for (int q = m; q < m + att_part[p]; ++q) {
      if (sdims[q] != sdims[m]) return LNT_BAD_DIMS;
      ad *= (u64)sdims[q];
    }
    P.att_part[p] = att_part[p];
    m += att_part[p];
  }
  P.natt = m - P.ncon;
  for (int q = m; q < order; ++q) od *= (u64)sdims[q];
  P.cdim = make_divider(cd);
  P.afull = make_divider(ad);
  P.other_dim = od;
  const UnaryLayout L = unary_layout(n);
  if (!workspace || workspace_bytes < L.total || (uintptr_t)workspace % 256) return LNT_WORKSPACE;
  cudaStream_t s = as_stream(stream);
  if (d_sorted && cudaMemsetAsync(d_sorted, 0xff, 4, s) != cudaSuccess) return LNT_DEVICE_ERROR;
  if (n == 0) return cudaMemsetAsync(d_nout, 0, 8, s) == cudaSuccess ? LNT_OK : LNT_DEVICE_ERROR;
  unsigned char* W = static_cast<unsigned char*>(workspace);
  u32* counts = reinterpret_cast<u32*>(W + L.counts);
  unsigned long long* pos = reinterpret_cast<unsigned long long*>(W + L.pos);
  u64* gk = reinterpret_cast<u64*>(W + L.gk);
  double* gv = reinterpret_cast<double*>(W + L.gv);
  u64* ck = reinterpret_cast<u64*>(W + L.ck);
  double* cv = reinterpret_cast<double*>(W + L.cv);
  const u32 blocks = (L.nchunks + kFoldThreads / 32 - 1) / (kFoldThreads / 32);
  {
    ProfScope prof("unary_fold", s);
    unary_fold_kernel<<<blocks, kFoldThreads, 0, s>>>((const u64*)keys, vals, n, L.chunk, L.nchunks, P, gk, gv, counts);
    count_launch();
  }
  int st = scan::run(CountOf{counts}, L.nchunks, pos, nullptr, W + L.scan, s, "unary_scan");
  if (st != LNT_OK) return st;
  {
    ProfScope prof("unary_gather", s);
    unary_gather_kernel<<<blocks, 256, 0, s>>>(gk, gv, counts, L.chunk, L.nchunks, pos, ck, cv);
    count_launch();
  }
  st = collect::run(ck, cv, (const u64*)(pos + L.nchunks), n, UnaryGroups{P}, (u64*)out_keys, out_vals, (u64*)d_nout,
                    W + L.coll, s, "unary_groups");
  if (st != LNT_OK) return st;
  if (d_sorted) {
    ProfScope prof("unary_sorted", s);
    unary_sorted_kernel<<<grid_n(n), 256, 0, s>>>((const u64*)out_keys, (const u64*)d_nout, d_sorted);
    count_launch();
  }
  return launch_status();
}

}  // extern "C"
