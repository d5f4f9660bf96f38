// Sparse lattice product C_t = A_t * B_t for every tab t (the reference's
// SparseLatticeBase::operator* -> csc_no_accum<true>, SparseLatticeBase.h:
// 1572-1576, 1854-1990).  Lattices are column-major LCO: A key =
// row + h*(col + w*tab), B key = row + w*(col + wB*tab), both ascending; C key
// = row + h*(col + wB*tab), ascending, duplicates summed, exact zeros kept.
//
// Plan phase (both engines): A column pointers (dense over w*d columns when
// that fits, else binary search on A's keys), product count per B entry and
// its prefix sum (total = products P).
//
// SPA engine (h <= 1024, and A's w*d and B's w_B*d columns fit dense pointer
// arrays): one warp per output column (tab, col).  Lanes take B
// entries of the column, walk the matching A columns and add a*b into a
// dense h-row accumulator in shared memory while setting a row bitmap; the
// column's rows are then emitted in ascending order.  A symbolic pass counts
// rows per column first, so output offsets come from a prefix sum and the
// numeric pass writes C directly, already sorted.  This is Gustavson's
// column-by-column product; the reference does the same per column with a
// scatter + radix sort + duplicate fold.
//
// ESC engine (any shape): expand all P products (key, a*b) load-balanced by
// product index, radix-sort them by key, fold duplicates (no zero skipping).
//
// Tile engine (lnt_tile.cu): products whose output is dense or nearly so.
//
// Engine choice (lnt_lattice_mult_workspace and lnt_lattice_mult, from the
// shape and the product count P): SPA when h <= 1024; else the tile engine
// when its bitmaps fit and P >= 2^30 or P >= (nnz(A) + h*d) * ceil(wB/64)
// (the tile engine's work per 64-column tile is one pass over A's entries);
// else ESC.  LNT_SPGEMM_ENGINE=tile|esc in the environment forces an engine
// (tile only where its bitmaps fit).
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "lnt_scan.cuh"
#include "lnt_msd.cuh"

namespace lnt {

size_t collect_workspace_bytes(size_t n);
bool tile_shape_ok(u64 h, u64 w, u64 wB, u64 d, u64 na, u64 nb);
size_t tile_workspace_bytes(u64 h, u64 w, u64 wB, u64 d, u64 na, u64 nb, bool buckets);
int run_tile_mult(const u64* akeys, const double* avals, u64 na, const u64* bkeys, const double* bvals, u64 nb,
                  u64 h, u64 w, u64 wB, u64 d, void* ws, size_t ws_bytes, u64* ck, double* cv, u64* d_nc,
                  cudaStream_t s);

namespace {

constexpr u64 kMaxDenseAColumns = 1ull << 27;
constexpr u64 kMaxDenseBColumns = 1ull << 24;
constexpr int kSpaMaxRows = 1024;
constexpr int kSpaWarps = 4;  // 4 x (8 KB accumulator + 128 B bitmap) of static shared memory

struct Lat {
  const u64* keys;
  const double* vals;
  u64 nnz;
  u64 rows, cols, tabs;
};

// ptr[c] = first index whose column id (key / div) is >= c, for c in [0, ncol],
// of one operand, or of both (the blocks from `blocks_a` on: B).
struct ColPtr {
  const u64* keys;
  u64 n;
  Divider div;
  u64 ncol;
  u64* ptr;
};

__global__ void colptr_kernel(const ColPtr a, const ColPtr b, u32 blocks_a) {
  const bool is_b = blockIdx.x >= blocks_a;
  const ColPtr& c = is_b ? b : a;
  const u64 block = is_b ? blockIdx.x - blocks_a : blockIdx.x, blocks = is_b ? gridDim.x - blocks_a : blocks_a;
  const u64 stride = blocks * blockDim.x;
  for (u64 i = block * blockDim.x + threadIdx.x; i <= c.n; i += stride) {
    const long long prev = i == 0 ? -1ll : (long long)min(divide(c.keys[i - 1], c.div), c.ncol);
    const u64 cur = i == c.n ? c.ncol : min(divide(c.keys[i], c.div), c.ncol);
    for (long long x = prev + 1; x <= (long long)cur; ++x) c.ptr[x] = i;
  }
}

// [lo, hi) of A entries in A column `acol` (acol = col + w*tab).
struct AColumns {
  const u64* ptr;  // dense pointers, or null
  const u64* keys;
  u64 n, h;
  __device__ __forceinline__ void range(u64 acol, u64& lo, u64& hi) const {
    if (ptr) {
      lo = ptr[acol];
      hi = ptr[acol + 1];
      return;
    }
    const u64 k0 = acol * h, k1 = k0 + h;
    u64 a = 0, b = n;
    while (a < b) {
      const u64 m = (a + b) >> 1;
      if (keys[m] < k0) a = m + 1; else b = m;
    }
    lo = a;
    b = n;
    while (a < b) {
      const u64 m = (a + b) >> 1;
      if (keys[m] < k1) a = m + 1; else b = m;
    }
    hi = a;
  }
};

// Products contributed by B entry e: size of the A column its row selects.
struct ProductCount {
  AColumns ac;
  const u64* bkeys;
  Divider div_w, div_wB;
  u64 w;
  __device__ __forceinline__ u64 operator()(size_t e) const {
    const u64 k = bkeys[e];
    const u64 bcol = divide(k, div_w);  // col + wB*tab
    const u64 t = divide(bcol, div_wB);
    const u64 brow = k - bcol * w;
    u64 lo, hi;
    ac.range(brow + w * t, lo, hi);
    return hi - lo;
  }
};

struct Identity64 {
  const u64* v;
  __device__ __forceinline__ u64 operator()(size_t i) const { return v[i]; }
};

// ---- ESC engine ----------------------------------------------------------
// One CTA per 2048 consecutive products.  The B entries they belong to (found
// by two searches for the tile, not one per product) are decoded once each
// into shared memory; their first products are marked and a maximum scan gives
// every product its entry.  Then a product costs its A entry's load and its
// store.  17.4M products of 1M x 1.1M entries: 0.49 -> 0.12 ms.  The bounds on a
// mark and on an A position change nothing in a correct run; they keep the
// accesses inside when the prefix is not ascending because a look-back of its
// scan gave up.
constexpr int kExpandThreads = 256;
constexpr int kExpandTile = 2048;
constexpr int kExpandEntries = 1024;  // decoded B entries a tile has room for

// Last e in [a, b] with boff[e] <= p.
__device__ __forceinline__ u64 entry_of(const u64* __restrict__ boff, u64 a, u64 b, u64 p) {
  while (a < b) {
    const u64 m = (a + b + 1) >> 1;
    if (boff[m] <= p) a = m; else b = m - 1;
  }
  return a;
}

struct ExpandEntry {
  u64 x0;      // A position of product p: x0 + p (modulo 2^64)
  u64 kshift;  // C key = A key + kshift
  double beta;
};

__device__ __forceinline__ ExpandEntry expand_entry(const Lat& A, const Lat& B, const AColumns& ac, u64 boff_e, u64 e,
                                                    const Divider& div_w, const Divider& div_wB) {
  const u64 k = B.keys[e];
  const u64 bcol = divide(k, div_w);  // col + wB*tab
  const u64 t = divide(bcol, div_wB);
  const u64 acol = k - bcol * A.cols + A.cols * t;
  u64 lo, hi;
  ac.range(acol, lo, hi);
  // A key = row + h*acol -> C key = row + h*(col + wB*tab)
  return {lo - boff_e, A.rows * bcol - A.rows * acol, B.vals[e]};
}

__global__ void __launch_bounds__(kExpandThreads) expand_kernel(Lat A, Lat B, AColumns ac,
                                                                const u64* __restrict__ boff, u64 P, Divider div_w,
                                                                Divider div_wB, u64* __restrict__ pk,
                                                                double* __restrict__ pv) {
  constexpr int I = kExpandTile / kExpandThreads;
  __shared__ ExpandEntry s_e[kExpandEntries];
  __shared__ __align__(16) unsigned short s_ent[kExpandTile];
  __shared__ u32 s_warp[kExpandThreads / 32];
  __shared__ u64 s_range[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const u64 p0 = (u64)blockIdx.x * kExpandTile, p1 = min(P, p0 + kExpandTile);
  if (tid == 0) s_range[0] = entry_of(boff, 0, B.nnz - 1, p0);
  if (tid == 32) s_range[1] = entry_of(boff, 0, B.nnz - 1, p1 - 1);
  reinterpret_cast<uint4*>(s_ent)[tid] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const u64 e0 = s_range[0], ne = s_range[1] - e0 + 1;
  if (ne > (u64)kExpandEntries) {  // many B entries without products: each product searches the tile's range
    for (u64 p = p0 + tid; p < p1; p += kExpandThreads) {
      const u64 e = entry_of(boff, e0, e0 + ne - 1, p);
      const ExpandEntry q = expand_entry(A, B, ac, boff[e], e, div_w, div_wB);
      const u64 x = min(q.x0 + p, A.nnz - 1);
      pk[p] = A.keys[x] + q.kshift;
      pv[p] = A.vals[x] * q.beta;
    }
    return;
  }
  for (u32 i = tid; i < (u32)ne; i += kExpandThreads) {
    const u64 b = boff[e0 + i];
    // (of the entries that start at one product only the last has products)
    if (boff[e0 + i + 1] > b) {
      s_e[i] = expand_entry(A, B, ac, b, e0 + i, div_w, div_wB);
      if (b > p0 && b < p1) s_ent[b - p0] = (unsigned short)i;  // (entry 0 covers the tile's start)
    }
  }
  __syncthreads();
  {  // maximum scan over the tile: the entry of every product
    uint4 q = reinterpret_cast<uint4*>(s_ent)[tid];  // eight consecutive products
    u32 w[4] = {q.x, q.y, q.z, q.w};
    u32 run = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const u32 a0 = max(run, w[j] & 0xFFFFu), a1 = max(a0, w[j] >> 16);
      w[j] = a0 | (a1 << 16);
      run = a1;
    }
    u32 inc = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc = max(inc, t);
    }
    if (lane == 31) s_warp[warp] = inc;
    u32 before = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) before = 0;
    __syncthreads();
    for (int x = 0; x < warp; ++x) before = max(before, s_warp[x]);
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = max(w[j] & 0xFFFFu, before) | (max(w[j] >> 16, before) << 16);
    reinterpret_cast<uint4*>(s_ent)[tid] = make_uint4(w[0], w[1], w[2], w[3]);
  }
  __syncthreads();
  static_assert(I == 8, "eight products per thread");
#pragma unroll
  for (int j = 0; j < I; ++j) {
    const u32 o = j * kExpandThreads + tid;
    if (p0 + o < p1) {
      const ExpandEntry q = s_e[s_ent[o]];
      const u64 x = min(q.x0 + p0 + o, A.nnz - 1);
      pk[p0 + o] = A.keys[x] + q.kshift;
      pv[p0 + o] = A.vals[x] * q.beta;
    }
  }
}

// ---- SPA engine ----------------------------------------------------------
// One warp per output column; with few columns (BLOCK) one CTA per column: a
// column of 100 entries then takes one round of dependent loads of its four
// warps instead of four of one (100 columns: 10.4 -> 5.2 us numeric, 7.4 -> 4.6 us
// symbolic).  Every warp has accumulators of its own, added up in the warps'
// order at the end, so that a result does not depend on which warp was faster
// (one set for all four took the same time).  The symbolic pass also counts the
// products.
template <bool NUMERIC, bool BLOCK>
__global__ void __launch_bounds__(kSpaWarps * 32) spa_kernel(Lat A, Lat B, AColumns ac, const u64* __restrict__ bptr,
                                                              u64 units, u64* __restrict__ ucount,
                                                              unsigned long long* __restrict__ d_products,
                                                              const u64* __restrict__ uoff, u64* __restrict__ ck,
                                                              double* __restrict__ cv, u64* __restrict__ d_nc) {
  constexpr int N = BLOCK ? 1 : kSpaWarps;
  constexpr int T = BLOCK ? kSpaWarps * 32 : 32;  // threads per column
  __shared__ u32 s_bits[N][kSpaMaxRows / 32];
  __shared__ double s_acc[NUMERIC ? kSpaWarps : 1][NUMERIC ? kSpaMaxRows : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ct = BLOCK ? threadIdx.x : lane;
  const u64 h = A.rows, w = A.cols, wB = B.cols;
  const int hw = (int)((h + 31) / 32);  // at most 32
  u32* bits = s_bits[BLOCK ? 0 : warp];
  double* acc = s_acc[NUMERIC ? warp : 0];
  auto sync = [] {
    if (BLOCK) __syncthreads();
    else __syncwarp();
  };
  const u64 nteams = BLOCK ? gridDim.x : (u64)gridDim.x * kSpaWarps;
  unsigned long long products = 0;
  if (NUMERIC && blockIdx.x == 0 && threadIdx.x == 0) *d_nc = uoff[units];
  for (u64 u = BLOCK ? blockIdx.x : (u64)blockIdx.x * kSpaWarps + warp; u < units; u += nteams) {
    const u64 e0 = bptr[u], e1 = bptr[u + 1];
    if (e0 == e1) {  // empty B column: no output rows
      if (!NUMERIC && ct == 0) ucount[u] = 0;
      continue;
    }
    for (int i = ct; i < hw; i += T) bits[i] = 0u;
    if (NUMERIC)
      for (int i = lane; i < (int)h; i += 32) acc[i] = 0.0;
    sync();
    const u64 t = u / wB;
    for (u64 e = e0 + ct; e < e1; e += T) {
      const u64 brow = B.keys[e] - w * u;  // B col id of this unit is u
      const u64 acol = brow + w * t;
      u64 lo, hi;
      ac.range(acol, lo, hi);
      const double beta = NUMERIC ? B.vals[e] : 0.0;
      if (!NUMERIC) products += hi - lo;
      for (u64 x = lo; x < hi; ++x) {
        const u32 r = (u32)(A.keys[x] - acol * h);
        atomicOr(&bits[r >> 5], 1u << (r & 31));
        if (NUMERIC) atomicAdd(&acc[r], A.vals[x] * beta);
      }
    }
    sync();
    // rows before every word of 32 (each warp for itself)
    const u32 mine = lane < hw ? __popc(bits[lane]) : 0u;
    if (!NUMERIC) {
      const u32 c = __reduce_add_sync(0xffffffffu, mine);
      if (ct == 0) ucount[u] = c;
    } else {
      u32 inc = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      const u64 out = uoff[u];
      const u64 colkey = h * u;  // h*(col + wB*tab)
      for (int g = BLOCK ? warp : 0; g < hw; g += BLOCK ? kSpaWarps : 1) {
        const u32 word = bits[g], before = __shfl_sync(0xffffffffu, inc - mine, g);
        if (word & (1u << lane)) {
          const u32 r = (u32)g * 32 + lane;
          const u64 o = out + before + __popc(word & ((1u << lane) - 1u));
          double v = acc[r];
          if (BLOCK) {
            v = s_acc[0][r];
#pragma unroll
            for (int q = 1; q < (NUMERIC ? kSpaWarps : 1); ++q) v += s_acc[q][r];
          }
          ck[o] = colkey + r;
          cv[o] = v;
        }
      }
    }
    sync();
  }
  if (!NUMERIC) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) products += __shfl_xor_sync(0xffffffffu, products, o);
    if (lane == 0 && products) atomicAdd(d_products, products);
  }
}

// ---- host side ------------------------------------------------------------
struct Shape {
  Lat A, B;
  u64 h, w, wB, d;
  bool dense_a, dense_b;
};

int check_shape(const lnt_lattice* a, const lnt_lattice* b, Shape* s) {
  if (!a || !b) return LNT_BAD_ARG;
  if (a->rows <= 0 || a->cols <= 0 || a->tabs <= 0 || b->rows <= 0 || b->cols <= 0 || b->tabs <= 0)
    return LNT_BAD_DIMS;
  if (a->cols != b->rows || a->tabs != b->tabs) return LNT_BAD_DIMS;  // check_mult_dims
  if ((a->nnz && (!a->keys || !a->vals)) || (b->nnz && (!b->keys || !b->vals))) return LNT_BAD_ARG;
  unsigned __int128 ka = (unsigned __int128)a->rows * a->cols * a->tabs;
  unsigned __int128 kb = (unsigned __int128)b->rows * b->cols * b->tabs;
  unsigned __int128 kc = (unsigned __int128)a->rows * b->cols * a->tabs;
  if ((ka >> 63) || (kb >> 63) || (kc >> 63)) return LNT_OVERFLOW_KEYBITS;
  s->A = {(const u64*)a->keys, a->vals, a->nnz, (u64)a->rows, (u64)a->cols, (u64)a->tabs};
  s->B = {(const u64*)b->keys, b->vals, b->nnz, (u64)b->rows, (u64)b->cols, (u64)b->tabs};
  s->h = (u64)a->rows;
  s->w = (u64)a->cols;
  s->wB = (u64)b->cols;
  s->d = (u64)a->tabs;
  s->dense_a = s->w * s->d <= kMaxDenseAColumns;
  s->dense_b = s->wB * s->d <= kMaxDenseBColumns;
  return LNT_OK;
}

// Plan workspace layout.
struct PlanLayout {
  size_t off_aptr, off_bptr, off_boff, off_ucount, off_uoff, off_scan, total;
  u64 units;
};

PlanLayout plan_layout(const Shape& s) {
  PlanLayout L;
  size_t off = 0;
  L.units = s.dense_b ? s.wB * s.d : 0;
  L.off_aptr = off;
  off += align_up(s.dense_a ? (s.w * s.d + 1) * 8 : 8, 256);
  L.off_bptr = off;
  off += align_up(s.dense_b ? (L.units + 1) * 8 : 8, 256);
  L.off_boff = off;
  off += align_up((s.B.nnz + 1) * 8, 256);
  L.off_ucount = off;
  off += align_up((L.units + 1) * 8, 256);
  L.off_uoff = off;
  off += align_up((L.units + 1) * 8, 256);
  L.off_scan = off;
  off += align_up(std::max(scan::workspace_bytes(s.B.nnz), scan::workspace_bytes(L.units)), 256);
  L.total = off;
  return L;
}

bool spa_eligible(const Shape& s) { return s.h <= (u64)kSpaMaxRows && s.dense_a && s.dense_b; }

// A CTA per output column up to this many columns (two waves of resident CTAs).
u64 spa_block_units() { return (u64)sm_count() * 16; }

// Products per B entry, summed up: boff[e] before entry e, the total to *d_total.
int product_prefix(const Shape& s, const AColumns& ac, u64* boff, unsigned long long* d_total, void* ws,
                   cudaStream_t cs) {
  const ProductCount pc{ac, s.B.keys, make_divider(s.w), make_divider(s.wB), s.w};
  return scan::run(pc, s.B.nnz, (unsigned long long*)boff, d_total, ws, cs, "spgemm_count");
}

enum class Engine { Spa, Esc, Tile };

Engine choose_engine(const Shape& s, u64 products) {
  const bool tile_ok = tile_shape_ok(s.h, s.w, s.wB, s.d, s.A.nnz, s.B.nnz);
  if (const char* e = std::getenv("LNT_SPGEMM_ENGINE")) {
    if (!std::strcmp(e, "tile") && tile_ok) return Engine::Tile;
    if (!std::strcmp(e, "esc")) return Engine::Esc;
  }
  if (spa_eligible(s)) return Engine::Spa;
  const u64 nt = (s.wB + 63) / 64;
  if (tile_ok && (products >= (1ull << 30) || products >= (s.A.nnz + s.h * s.d) * nt)) return Engine::Tile;
  return Engine::Esc;
}

// Workspace of the ESC engine: the products and the sort's other pairs (A, B).
struct EscLayout {
  PairSort sort;
  size_t pair_bytes;  // of A and of B: keys, then values
  size_t off_ctrl, off_a, off_b, off_coll, total;
};

EscLayout esc_layout(u64 products, u64 max_key, bool buckets = true) {
  EscLayout L;
  L.sort = make_pair_sort(products, max_key, buckets);
  L.pair_bytes = 2 * align_up(products * 8, 256);
  size_t off = 0;
  L.off_ctrl = off;
  off += align_up(L.sort.ctrl_bytes, 256);
  L.off_a = off;
  off += L.pair_bytes;
  L.off_b = off;
  off += L.pair_bytes;
  L.off_coll = off;
  off += align_up(collect_workspace_bytes(products), 256);
  L.total = off;
  return L;
}

// The SPA engine's plan holds no product prefix; the ESC engine forced on such
// a shape makes its own, behind its workspace.
size_t esc_prefix_bytes(const Shape& s) {
  return spa_eligible(s) ? align_up((s.B.nnz + 1) * 8, 256) + align_up(scan::workspace_bytes(s.B.nnz), 256) : 0;
}

// counts[1] = min(counts[0], dense): the output holds at most one entry per
// (row, col, tab) and at most one per product.
__global__ void capacity_kernel(u64* counts, u64 dense) { counts[1] = min(counts[0], dense); }

int grid_for(u64 work, int threads, int per_sm = 8) {
  const u64 want = (work + threads - 1) / threads;
  const u64 cap = (u64)sm_count() * per_sm;
  return (int)std::max<u64>(1, std::min(want, cap));
}

}  // namespace
}  // namespace lnt

using namespace lnt;

extern "C" {

int lnt_lattice_mult_plan_workspace(const lnt_lattice* a, const lnt_lattice* b, size_t* bytes) {
  Shape s;
  int st = check_shape(a, b, &s);
  if (st != LNT_OK) return st;
  if (!bytes) return LNT_BAD_ARG;
  *bytes = plan_layout(s).total;
  return LNT_OK;
}

int lnt_lattice_mult_plan(const lnt_lattice* a, const lnt_lattice* b, void* plan, size_t plan_bytes,
                          uint64_t* d_counts, void* stream) {
  Shape s;
  int st = check_shape(a, b, &s);
  if (st != LNT_OK) return st;
  if (!d_counts) return LNT_BAD_ARG;
  PlanLayout L = plan_layout(s);
  if (!plan || plan_bytes < L.total || (uintptr_t)plan % 256) return LNT_WORKSPACE;
  cudaStream_t cs = as_stream(stream);
  unsigned char* p = static_cast<unsigned char*>(plan);
  u64* aptr = reinterpret_cast<u64*>(p + L.off_aptr);
  u64* bptr = reinterpret_cast<u64*>(p + L.off_bptr);
  u64* boff = reinterpret_cast<u64*>(p + L.off_boff);
  u64* ucount = reinterpret_cast<u64*>(p + L.off_ucount);
  u64* uoff = reinterpret_cast<u64*>(p + L.off_uoff);
  const bool spa = spa_eligible(s);
  if (s.dense_a) {
    const ColPtr ca{s.A.keys, s.A.nnz, make_divider(s.h), s.w * s.d, aptr};
    const ColPtr cb{s.B.keys, s.B.nnz, make_divider(s.w), L.units, bptr};
    const u32 ga = (u32)grid_for(s.A.nnz + 1, 256), gb = spa ? (u32)grid_for(s.B.nnz + 1, 256) : 0u;
    ProfScope prof("spgemm_colptr", cs);
    colptr_kernel<<<ga + gb, 256, 0, cs>>>(ca, cb, ga);
    count_launch();
  }
  AColumns ac{s.dense_a ? aptr : nullptr, s.A.keys, s.A.nnz, s.h};
  if (spa) {
    if (cudaMemsetAsync(d_counts, 0, 8, cs) != cudaSuccess) return LNT_DEVICE_ERROR;
    {
      ProfScope prof("spgemm_spa_symbolic", cs);
      if (L.units <= spa_block_units())
        spa_kernel<false, true><<<(unsigned)L.units, kSpaWarps * 32, 0, cs>>>(
            s.A, s.B, ac, bptr, L.units, ucount, (unsigned long long*)d_counts, nullptr, nullptr, nullptr, nullptr);
      else
        spa_kernel<false, false><<<grid_for(L.units * 32, kSpaWarps * 32), kSpaWarps * 32, 0, cs>>>(
            s.A, s.B, ac, bptr, L.units, ucount, (unsigned long long*)d_counts, nullptr, nullptr, nullptr, nullptr);
      count_launch();
    }
    // output rows per column -> prefix -> exact output count into d_counts[1]
    st = scan::run(Identity64{ucount}, L.units, (unsigned long long*)uoff, (unsigned long long*)(d_counts + 1),
                   p + L.off_scan, cs, "spgemm_scan");
    if (st != LNT_OK) return st;
  } else {
    // products per B entry -> prefix -> total products into d_counts[0]
    st = product_prefix(s, ac, boff, (unsigned long long*)d_counts, p + L.off_scan, cs);
    if (st != LNT_OK) return st;
    capacity_kernel<<<1, 1, 0, cs>>>((u64*)d_counts, s.h * s.wB * s.d);
    count_launch();
  }
  return launch_status();
}

int lnt_lattice_mult_workspace(const lnt_lattice* a, const lnt_lattice* b, uint64_t products, size_t* bytes) {
  Shape s;
  int st = check_shape(a, b, &s);
  if (st != LNT_OK) return st;
  if (!bytes) return LNT_BAD_ARG;
  const Engine eng = choose_engine(s, products);
  if (eng == Engine::Spa) {
    *bytes = 256;
    return LNT_OK;
  }
  if (eng == Engine::Tile) {
    *bytes = tile_workspace_bytes(s.h, s.w, s.wB, s.d, s.A.nnz, s.B.nnz, true);
    return LNT_OK;
  }
  if (products >= (1ull << 30)) return LNT_UNSUPPORTED;
  *bytes = esc_layout(products, s.h * s.wB * s.d).total + esc_prefix_bytes(s);
  return LNT_OK;
}

int lnt_lattice_mult(const lnt_lattice* a, const lnt_lattice* b, const void* plan, uint64_t products,
                     void* workspace, size_t workspace_bytes, uint64_t* c_keys, double* c_vals, uint64_t* d_nc,
                     void* stream) {
  Shape s;
  int st = check_shape(a, b, &s);
  if (st != LNT_OK) return st;
  if (!plan || !d_nc) return LNT_BAD_ARG;
  PlanLayout L = plan_layout(s);
  cudaStream_t cs = as_stream(stream);
  const unsigned char* p = static_cast<const unsigned char*>(plan);
  const u64* aptr = reinterpret_cast<const u64*>(p + L.off_aptr);
  const u64* bptr = reinterpret_cast<const u64*>(p + L.off_bptr);
  const u64* boff = reinterpret_cast<const u64*>(p + L.off_boff);
  const u64* uoff = reinterpret_cast<const u64*>(p + L.off_uoff);
  AColumns ac{s.dense_a ? aptr : nullptr, s.A.keys, s.A.nnz, s.h};
  size_t need = 0;
  st = lnt_lattice_mult_workspace(a, b, products, &need);
  if (st != LNT_OK) return st;
  const Engine eng = choose_engine(s, products);
  const bool buckets = workspace_bytes >= need;  // else sort by digit passes, which may need less
  if (!buckets && eng == Engine::Esc) need = esc_layout(products, s.h * s.wB * s.d, false).total + esc_prefix_bytes(s);
  if (!buckets && eng == Engine::Tile)
    need = tile_workspace_bytes(s.h, s.w, s.wB, s.d, s.A.nnz, s.B.nnz, false);
  if (workspace_bytes < need || (need > 256 && !workspace)) return LNT_WORKSPACE;
  if (products && (!c_keys || !c_vals)) return LNT_BAD_ARG;
  if (eng == Engine::Tile)
    return run_tile_mult(s.A.keys, s.A.vals, s.A.nnz, s.B.keys, s.B.vals, s.B.nnz, s.h, s.w, s.wB, s.d, workspace,
                         workspace_bytes, (u64*)c_keys, c_vals, (u64*)d_nc, cs);
  if (eng == Engine::Spa) {
    {
      ProfScope prof("spgemm_spa_numeric", cs);
      if (L.units <= spa_block_units())
        spa_kernel<true, true><<<(unsigned)L.units, kSpaWarps * 32, 0, cs>>>(
            s.A, s.B, ac, bptr, L.units, nullptr, nullptr, uoff, (u64*)c_keys, c_vals, (u64*)d_nc);
      else
        spa_kernel<true, false><<<grid_for(L.units * 32, kSpaWarps * 32), kSpaWarps * 32, 0, cs>>>(
            s.A, s.B, ac, bptr, L.units, nullptr, nullptr, uoff, (u64*)c_keys, c_vals, (u64*)d_nc);
      count_launch();
    }
    return launch_status();
  }
  // ESC
  if (products == 0) return cudaMemsetAsync(d_nc, 0, 8, cs) == cudaSuccess ? LNT_OK : LNT_DEVICE_ERROR;
  const EscLayout E = esc_layout(products, s.h * s.wB * s.d, buckets);
  unsigned char* w = static_cast<unsigned char*>(workspace);
  void* ctrl = w + E.off_ctrl;
  if (spa_eligible(s)) {
    u64* own = reinterpret_cast<u64*>(w + E.total);
    st = product_prefix(s, ac, own, nullptr, w + E.total + align_up((s.B.nnz + 1) * 8, 256), cs);
    if (st != LNT_OK) return st;
    boff = own;
  }
  // Pass p of the LSD sort writes buffer (passes-1-p)&1 (0 = A, the final
  // one); expand into the buffer its pass 0 does not write.
  const bool even = E.sort.lsd.passes % 2 == 0;
  unsigned char* pe = w + (even ? E.off_a : E.off_b);
  unsigned char* po = w + (even ? E.off_b : E.off_a);
  u64* ek = reinterpret_cast<u64*>(pe);
  double* ev = reinterpret_cast<double*>(pe + E.pair_bytes / 2);
  {
    ProfScope prof("spgemm_expand", cs);
    expand_kernel<<<(unsigned)((products + kExpandTile - 1) / kExpandTile), kExpandThreads, 0, cs>>>(
        s.A, s.B, ac, boff, products, make_divider(s.w), make_divider(s.wB), ek, ev);
    count_launch();
  }
  const PairSource src = plain_source(ek, ev, products);
  u32* gate = nullptr;
  if (E.sort.msd.ok) {  // sort by output key and add up, in one go
    gate = reinterpret_cast<u32*>(w + E.off_ctrl + E.sort.ctrl_bytes - 256);
    const MsdFold fold{0, (u64*)d_nc};
    // (two passes: the second may write over the products, which the first has read)
    void* x = E.sort.msd.passes == 2 ? po : nullptr;
    void* y = E.sort.msd.passes == 2 ? pe : po;
    st = run_msd_sort(E.sort.msd, src, x, y, ctrl, &fold, (u64*)c_keys, c_vals, gate, cs);
    if (st != LNT_OK || E.sort.msd.single) return st;
  }
  u64* k0 = reinterpret_cast<u64*>(w + E.off_a);
  double* v0 = reinterpret_cast<double*>(w + E.off_a + E.pair_bytes / 2);
  u64* k1 = reinterpret_cast<u64*>(w + E.off_b);
  double* v1 = reinterpret_cast<double*>(w + E.off_b + E.pair_bytes / 2);
  st = run_sort(E.sort.lsd, gated_source(src, gate, 1), k0, v0, k1, v1, ctrl, cs);
  if (st != LNT_OK) return st;
  return run_collect_gated(k0, v0, products, 0, (u64*)c_keys, c_vals, (u64*)d_nc, w + E.off_coll, cs, gate, 1);
}

}  // extern "C"

// ---- noLatticeMult ----------------------------------------------------------
// Products with no contracted index (SparseMIABase::perform_noLatticeMult,
// SparseMIABase.h:1716-1826): A as a lattice (h = its outer size) x 1 x d and B
// as 1 x wB x d (d = the inter size), both key-sorted.  Expanding every B
// entry's products against the A entries of its tab (a warp per B entry, at
// the entry's prefix-summed offset) yields them in the reference's emission
// order - B entries major, A entries minor, tab by tab - which is ascending
// key order, so C needs neither a sort nor a fold (equal keys from operands
// with duplicate keys stay separate, as in the reference).
namespace lnt {
namespace {
// One warp per B entry e (grid-stride): its products are the A entries of its
// tab, written contiguously at boff[e] with coalesced reads of A and writes.
__global__ void nolattice_expand_kernel(Lat A, Lat B, AColumns ac, const u64* __restrict__ boff, Divider div_wB,
                                        u64* __restrict__ ck, double* __restrict__ cv) {
  const int lane = threadIdx.x & 31;
  const u64 nw = ((u64)gridDim.x * blockDim.x) >> 5;
  const u64 h = A.rows;
  for (u64 e = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < B.nnz; e += nw) {
    const u64 bk = B.keys[e];          // col + wB * tab (B has one row)
    const u64 t = divide(bk, div_wB);
    u64 lo, hi;
    ac.range(t, lo, hi);
    const double bv = B.vals[e];
    const u64 o = boff[e];
    const u64 shift = h * bk - t * h;  // output key = A key - t*h + h*bk
    for (u64 x0 = lo + lane; x0 < hi; x0 += 128) {  // four products per lane: loads first, then stores
      u64 k[4];
      double v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const u64 x = x0 + 32 * q;
        k[q] = x < hi ? A.keys[x] : 0;
        v[q] = x < hi ? A.vals[x] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const u64 x = x0 + 32 * q;
        if (x < hi) {
          ck[o + (x - lo)] = k[q] + shift;
          cv[o + (x - lo)] = v[q] * bv;
        }
      }
    }
  }
}

struct NoLatLayout {
  size_t off_aptr, off_boff, off_scan, total;
};
NoLatLayout nolat_layout(const Shape& s) {
  NoLatLayout L;
  size_t off = 0;
  L.off_aptr = off;
  off += align_up(s.dense_a ? (s.w * s.d + 1) * 8 : 8, 256);
  L.off_boff = off;
  off += align_up((s.B.nnz + 1) * 8, 256);
  L.off_scan = off;
  off += align_up(scan::workspace_bytes(s.B.nnz), 256);
  L.total = off;
  return L;
}
int nolat_shape(const lnt_lattice* a, const lnt_lattice* b, Shape* s) {
  int st = check_shape(a, b, s);
  if (st != LNT_OK) return st;
  if (s->w != 1) return LNT_BAD_DIMS;  // A: h x 1 x d, B: 1 x wB x d
  return LNT_OK;
}
}  // namespace
}  // namespace lnt

extern "C" {

int lnt_nolattice_mult_workspace(const lnt_lattice* a, const lnt_lattice* b, size_t* bytes) {
  Shape s;
  int st = nolat_shape(a, b, &s);
  if (st != LNT_OK) return st;
  if (!bytes) return LNT_BAD_ARG;
  *bytes = nolat_layout(s).total;
  return LNT_OK;
}

int lnt_nolattice_mult_count(const lnt_lattice* a, const lnt_lattice* b, void* workspace, size_t workspace_bytes,
                             uint64_t* d_products, void* stream) {
  Shape s;
  int st = nolat_shape(a, b, &s);
  if (st != LNT_OK) return st;
  if (!d_products) return LNT_BAD_ARG;
  const NoLatLayout L = nolat_layout(s);
  if (!workspace || workspace_bytes < L.total || (uintptr_t)workspace % 256) return LNT_WORKSPACE;
  cudaStream_t cs = as_stream(stream);
  unsigned char* p = static_cast<unsigned char*>(workspace);
  u64* aptr = reinterpret_cast<u64*>(p + L.off_aptr);
  if (s.dense_a) {
    ProfScope prof("spgemm_colptr", cs);
    const ColPtr ca{s.A.keys, s.A.nnz, make_divider(s.h), s.w * s.d, aptr};
    const unsigned ga = (unsigned)grid_for(s.A.nnz + 1, 256);
    colptr_kernel<<<ga, 256, 0, cs>>>(ca, ca, ga);
    count_launch();
  }
  AColumns ac{s.dense_a ? aptr : nullptr, s.A.keys, s.A.nnz, s.h};
  ProductCount pc{ac, s.B.keys, make_divider(s.w), make_divider(s.wB), s.w};
  st = scan::run(pc, s.B.nnz, (unsigned long long*)(p + L.off_boff), (unsigned long long*)d_products,
                 p + L.off_scan, cs, "spgemm_count");
  if (st != LNT_OK) return st;
  return launch_status();
}

int lnt_nolattice_mult(const lnt_lattice* a, const lnt_lattice* b, uint64_t products, void* workspace,
                       size_t workspace_bytes, uint64_t* c_keys, double* c_vals, void* stream) {
  Shape s;
  int st = nolat_shape(a, b, &s);
  if (st != LNT_OK) return st;
  const NoLatLayout L = nolat_layout(s);
  if (!workspace || workspace_bytes < L.total || (uintptr_t)workspace % 256) return LNT_WORKSPACE;
  if (products == 0) return LNT_OK;
  if (!c_keys || !c_vals) return LNT_BAD_ARG;
  cudaStream_t cs = as_stream(stream);
  unsigned char* p = static_cast<unsigned char*>(workspace);
  AColumns ac{s.dense_a ? reinterpret_cast<const u64*>(p + L.off_aptr) : nullptr, s.A.keys, s.A.nnz, s.h};
  {
    ProfScope prof("nolattice_expand", cs);
    nolattice_expand_kernel<<<grid_for(s.B.nnz * 32, 256), 256, 0, cs>>>(
        s.A, s.B, ac, reinterpret_cast<const u64*>(p + L.off_boff), make_divider(s.wB), (u64*)c_keys, c_vals);
    count_launch();
  }
  return launch_status();
}

}  // extern "C"
