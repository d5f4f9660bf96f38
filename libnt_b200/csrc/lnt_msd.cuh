// Bucketed (most significant digit first) sort of (u64 key, f64 value) pairs,
// with or without folding equal keys; see lnt_msd.cu.
#pragma once

#include "lnt_sort.cuh"

namespace lnt {

// How a sort of n pairs with keys < max_key is bucketed: the top T key bits
// name the bucket, `shift` bits remain below them.
struct MsdPlan {
  bool ok = false;   // the bucketed path applies
  bool single = false;  // one cluster does it all (small_sort_kernel): no scratch, no gate, no path behind it
  bool large = false;  // bucket geometry: 512-thread CTAs of up to 5120 pairs, else 256 threads, 2560 pairs
  u32 n = 0;
  u64 max_key = 0;
  int key_bits = 0;
  int shift = 0;     // key bits below the bucket bits
  int T = 0;         // bucket bits
  int db = 0;        // digit bits of the last partition pass (T when there is only one)
  int passes = 0;    // 1 or 2
  int ib = 0;        // bits of the input index carried below the key
  // byte offsets inside the control block
  size_t off_counts = 0, off_start = 0, off_cur1 = 0, off_cur2 = 0, off_segtile = 0, off_misc = 0, off_status = 0;
  size_t zero_bytes = 0, ctrl_bytes = 0;  // zero_bytes: the prefix cleared before every run
};

MsdPlan make_msd_plan(size_t n, u64 max_key);

// Enqueues the bucketed sort of `src`.  The histogram kernel writes *gate: 0
// when every bucket fits a CTA (the remaining kernels run), 1 when one does
// not (they return at once; the caller's LSD path, gated on 1, runs instead).
// x, y: scratch of plan.n 16-byte records each, 16-byte aligned (x is used when
// plan.passes == 2 only).  gate: a gate block (kGateWords words).  Nothing
// waits on the host.
struct MsdFold {
  int skip_zero_heads;  // as in lnt_collect_duplicates
  u64* d_nout;
};
// fold == nullptr: plain stable sort.
int run_msd_sort(const MsdPlan& plan, const PairSource& src, void* x, void* y, void* ctrl, const MsdFold* fold,
                 u64* out_k, double* out_v, u32* gate, cudaStream_t s);

// A stable sort of n pairs by the bucketed path where it applies, with the LSD
// path behind it.
struct PairSort {
  SortPlan lsd;
  MsdPlan msd;
  size_t ctrl_bytes = 0;  // control block: either path's, then the gate word
  size_t a_bytes = 0, b_bytes = 0;  // scratch (b: 0 when not needed)
};
PairSort make_pair_sort(size_t n, u64 max_key, bool buckets = true);
// out must not overlap the source; a, b, ctrl: 256-byte aligned.
int run_pair_sort(const PairSort& p, const PairSource& src, u64* out_k, double* out_v, void* a, void* b, void* ctrl,
                  cudaStream_t s);

}  // namespace lnt
