// CSR x CSR SpGEMM (Gustavson) for sm_100a.
//
// Rows of A are binned by their product upper bound U_i = sum over the row's entries of the
// length of the matching B row:
//   bin 0  U <= 128     one warp per row, products sorted by (column, ordinal) in registers
//   bin 1  U <= 512     one 64-thread CTA per row, the same network across its warps
//   bin 2  U <= 2048    one 128-thread CTA per row
//   bin 3  U <= 8192    one CTA per row, 512 threads (1024 where there are no more such rows than SMs), its columns in
//                       segments of a warp each
//   bin 4  U  > 8192    the row's columns are cut into buckets of some 700 products, the products
//                       scattered to their buckets in global memory and every bucket sorted by a CTA
// (spgemm_rows.cuh: the sorting kernels of bins 0-3.)  Columns come out ascending like the
// reference's per-row sort; the structure is the symbolic union: an entry whose value cancels to 0
// is kept.  Two ways to run it:
//   two phases (sb_spgemm_symbolic / _numeric, like the reference): count, then the same kernels
//     again with values;
//   one pass (sb_spgemm_begin / _rows / _finish): every row's entries are written at the row's
//     product offset (an upper bound of its entry offset) and moved together afterwards - one
//     expansion and sort less for one copy of the result more.
// Row pointers come from an exclusive scan in int64, stored as int32 with an overflow check.
//
// Values are reproducible bit for bit from run to run.  Bins 0-3 sum the products of an entry in the
// order of their ordinals.  A bucket's products arrive in no order; where several land on one
// entry, every product is computed exactly in double, scaled by a power of two chosen per output row
// so that no partial sum can overflow (2^61 / (sum |a| of the row * max |b|)), rounded to a 64-bit
// integer and added as an integer, whose result does not depend on the order.  The rounding step is
// 2^-61 of the row's bound, far below fp32 (and fp64) resolution of the sum itself.  Rows whose bound
// is not finite add floats.  Integer dtypes wrap like the reference's and need none of this.
#include <limits.h>
#include <string.h>

#include <algorithm>
#include <exception>
#include <vector>

#include <cooperative_groups.h>

#include "spgemm_rows.cuh"

namespace sb {

constexpr int kBins = 5;

// Long rows (bin 4) are handled in batches of at most `products` products (the area's capacity); a
// single row with more than that takes the dense kernel, whose bitmap and accumulator of n columns
// lie in the same area.
constexpr int64_t kBigProductsMax = (int64_t)1 << 26;
constexpr int64_t kBucketProducts = 1024;      // buckets per row: U / this, rounded up to a power of two
constexpr int kBucketSort = 2048;              // products a bucket's sorting kernel takes
constexpr int kBigTasks = 1 << 17;
constexpr int kTurnProducts = 8192;            // products of 256 entries of A that a task takes; the rest is dealt out
// Columns up to which long rows are summed in shared memory (spgemm_smem_kernel) and need no area.
constexpr int kSmemColumns = 24576;

static int64_t big_products(int64_t m, int64_t n) {
  return std::min<int64_t>(kBigProductsMax, std::max<int64_t>((int64_t)1 << 20, 64 * (m + n)));
}
static int64_t big_buckets(int64_t products) { return products / (kBucketProducts / 2) + 64; }

struct WsLayout {
  long long* hdr;       // 16 int64: [0..4] rows per bin, [8] total of the last scan
  int* bin_cursor;      // kBins ints (+ padding)
  int* upper;           // m + 1 ints: product upper bound per row (saturating)
  int* bin_rows;        // kBins * m ints
  int* row_cnt;         // m ints
  unsigned long long* max_b;  // bit pattern of max |b| over the right operand
  long long* block_sum; // scan temporaries
  char* area;           // long rows (empty up to kSmemColumns columns)
  int64_t products;     // its capacity
  size_t area_bytes;
  size_t total;
};

static size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

struct alignas(16) BigRecord {
  unsigned col, pad;
  Slot prod;
};

// Arrays of a batch of long rows inside the area.
struct BigArea {
  int* row;             // [rows] row id
  int* p0;              // [rows + 1] first bucket
  int* shift;           // [rows] bucket of a column = first bucket + (column >> shift)
  int4* tasks;          // row index, first and last + 1 entry of A, part << 16 | parts (0: see big_expand)
  int* nrest;           // number of ...
  int4* rest;           // ... products left over: row index, first and last + 1 entry of A, first product
  double* scale;        // [rows] fixed-point scale
  int *cnt, *off, *cursor, *bucket_row, *ucnt, *uoff;   // per bucket
  long long* block_sum;
  unsigned* key;        // products, symbolic phase: the column
  BigRecord *rec, *rec2; // numeric phase (the same memory), and a second copy for rewritten buckets
  size_t bytes;
};
static BigArea big_area(char* p, int64_t products) {
  BigArea b;
  const size_t nb = (size_t)big_buckets(products) + 1;
  size_t off = 0;
  auto take = [&](size_t bytes) { char* q = p + off; off += align_up(bytes); return q; };
  b.row = (int*)take(nb * 4); b.p0 = (int*)take(nb * 4); b.shift = (int*)take(nb * 4);
  b.tasks = (int4*)take((size_t)kBigTasks * sizeof(int4));
  b.nrest = (int*)take(4);
  b.rest = (int4*)take((size_t)(products / kTurnProducts + 1) * sizeof(int4));
  b.scale = (double*)take(nb * 8);
  b.cnt = (int*)take(nb * 4); b.off = (int*)take(nb * 4); b.cursor = (int*)take(nb * 4);
  b.bucket_row = (int*)take(nb * 4); b.ucnt = (int*)take(nb * 4); b.uoff = (int*)take(nb * 4);
  b.block_sum = (long long*)take((nb / 4096 + 4) * 8);
  b.rec = (BigRecord*)take((size_t)products * sizeof(BigRecord));
  b.rec2 = (BigRecord*)take((size_t)products * sizeof(BigRecord));
  b.key = (unsigned*)b.rec;
  b.bytes = off;
  return b;
}

// Dense fallback: one bitmap + accumulator of n columns.
static size_t dense_words(int64_t n) { return (size_t)((n + 31) / 32); }
static size_t dense_bytes(int64_t n) { return align_up(4096) + align_up(dense_words(n) * 4) + align_up((size_t)n * 8); }

static WsLayout ws_layout(void* base, int64_t m, int64_t n) {
  WsLayout w;
  char* p = static_cast<char*>(base);
  size_t off = 0;
  auto take = [&](size_t bytes) { char* q = p + off; off += align_up(bytes); return q; };
  w.hdr = (long long*)take(16 * 8);
  w.bin_cursor = (int*)take(16 * 4);
  w.upper = (int*)take((size_t)(m + 1) * 4);
  w.bin_rows = (int*)take((size_t)m * 4 * kBins);
  w.row_cnt = (int*)take((size_t)(m + 1) * 4);
  w.max_b = (unsigned long long*)take(8);
  w.block_sum = (long long*)take((size_t)(ceil_div(m > 0 ? m : 1, 4096) + 1) * 8);
  w.products = big_products(m, n);
  w.area_bytes = n <= kSmemColumns ? 0 : std::max(big_area(nullptr, w.products).bytes, dense_bytes(n));
  w.area = take(w.area_bytes);
  w.total = off;
  return w;
}

// ---- binning ---------------------------------------------------------------------------------
// U_i of every row of A and the row's bin.  A CTA takes up to 1024 rows (fewer where that leaves SMs
// idle): 8 lanes per row, rows of more
// than 64 entries by a warp, of more than 2048 by the CTA (8 lanes alone needed 2 ms for the hub rows
// of a 2 M-row matrix); it appends them to the bins' lists with one atomic per bin (one per warp and
// bin is 0.4 ms there: five addresses for everybody).  Rows with U = 0 get row_cnt = 0 and join no bin.
constexpr int kBinThreads = 1024, kBinRows = 1024, kBinLaneRow = 64, kBinWarpRow = 2048;

// (Numbers of entries of A are stepped through unsigned: they may end at 2^31 - 1, and the step behind wraps an int.)
// Products of the entries b + x, b + x + step, ... before e.
__device__ __forceinline__ long long count_products(const int* __restrict__ Acrd, const int* __restrict__ Bpos,
                                                    int b, int e, int x, int step) {
  long long u = 0;
#pragma unroll 4
  for (unsigned p = (unsigned)b + x; p < (unsigned)e; p += step) {
    const int j = ld_stream(Acrd + p);
    u += __ldg(Bpos + j + 1) - __ldg(Bpos + j);
  }
  return u;
}

__global__ void __launch_bounds__(kBinThreads)
spgemm_bin_kernel(int m, int rows_per_cta, const int* __restrict__ Apos, const int* __restrict__ Acrd,
                  const int* __restrict__ Bpos, int* __restrict__ upper, int* __restrict__ bin_rows,
                  int* __restrict__ bin_cursor, int* __restrict__ row_cnt) {
  __shared__ int s_u[kBinRows], s_pos[kBinRows + 1];
  __shared__ int s_warp_rows[kBinRows], s_cta_rows[kBinRows];
  __shared__ int s_nwarp, s_ncta, s_next;
  __shared__ long long s_part[32];
  __shared__ int s_cnt[kBins], s_base[kBins];
  const int tid = threadIdx.x, l = tid & 7, warp = tid >> 5, lane = tid & 31;
  const long long row0 = (long long)blockIdx.x * rows_per_cta;
  const int rows = (int)min((long long)rows_per_cta, m - row0);
  if (tid < kBins) s_cnt[tid] = 0;
  if (tid == 0) s_nwarp = s_ncta = s_next = 0;
  for (int x = tid; x <= rows; x += kBinThreads) s_pos[x] = __ldg(Apos + row0 + x);
  __syncthreads();
#pragma unroll 2
  for (int x0 = 0; x0 < rows; x0 += kBinThreads / 8) {
    const int x = x0 + (tid >> 3);
    long long u = 0;
    bool put = false;
    if (x < rows) {
      const int b = s_pos[x], e = s_pos[x + 1];
      if (e - b <= kBinLaneRow) {
        u = count_products(Acrd, Bpos, b, e, l, 8);
        put = l == 0;
      } else if (l == 0) {
        if (e - b <= kBinWarpRow) s_warp_rows[atomicAdd(&s_nwarp, 1)] = x;
        else s_cta_rows[atomicAdd(&s_ncta, 1)] = x;
      }
    }
    u += __shfl_xor_sync(FULL, u, 4);
    u += __shfl_xor_sync(FULL, u, 2);
    u += __shfl_xor_sync(FULL, u, 1);
    if (put) s_u[x] = (int)min(u, (long long)INT_MAX);
  }
  __syncthreads();
  const int nwarp = s_nwarp, ncta = s_ncta;
  for (int i = 0; i < ncta; i++) {
    const int x = s_cta_rows[i];
    long long u = count_products(Acrd, Bpos, s_pos[x], s_pos[x + 1], tid, kBinThreads);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) u += __shfl_xor_sync(FULL, u, o);
    if (lane == 0) s_part[warp] = u;
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < 32; w++) u += s_part[w];
      s_u[x] = (int)min(u, (long long)INT_MAX);
    }
    __syncthreads();
  }
  while (true) {
    int i = 0;
    if (lane == 0) i = atomicAdd(&s_next, 1);
    i = __shfl_sync(FULL, i, 0);
    if (i >= nwarp) break;
    const int x = s_warp_rows[i];
    long long u = count_products(Acrd, Bpos, s_pos[x], s_pos[x + 1], lane, 32);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) u += __shfl_xor_sync(FULL, u, o);
    if (lane == 0) s_u[x] = (int)min(u, (long long)INT_MAX);
  }
  __syncthreads();
  int bin = -1, slot = 0;
  if (tid < rows) {
    const int u = s_u[tid];
    upper[row0 + tid] = u;
    if (u == 0) row_cnt[row0 + tid] = 0;
    else bin = (u > 128) + (u > 512) + (u > 2048) + (u > 8192);
  }
  if (bin >= 0) slot = atomicAdd(&s_cnt[bin], 1);
  __syncthreads();
  if (tid < kBins && s_cnt[tid]) s_base[tid] = atomicAdd(&bin_cursor[tid], s_cnt[tid]);
  __syncthreads();
  if (bin >= 0) bin_rows[(long long)bin * m + s_base[bin] + slot] = (int)(row0 + tid);
}

// ---- long rows: fixed-point accumulation ------------------------------------------------------
// scale = 2^(61 - exponent of bound); NaN marks "not fixed point"
__device__ __forceinline__ double scale_for_bound(double bound) {
  if (!(bound < 1.0e300)) return __longlong_as_double(0x7ff8000000000000LL);  // Inf / NaN
  if (bound <= 0.0) return 1.0;
  int e;
  frexp(bound, &e);                 // bound = f * 2^e, f in [0.5, 1)
  return ldexp(1.0, 61 - e);        // bound * scale < 2^61
}


template <typename T>
__device__ __forceinline__ Slot to_fixed(Slot bits, double scale) {
  return (Slot)__double2ll_rn(__longlong_as_double((long long)bits) * scale);
}
template <typename T>
__device__ __forceinline__ T from_fixed(Slot sum, double scale) {
  return (T)((double)(long long)sum * (1.0 / scale));
}
template <typename T>
__device__ __forceinline__ T one_product(Slot bits) {
  if constexpr (kIsFloat<T>) return (T)__longlong_as_double((long long)bits);
  else return (T)bits;
}

// Sum of products that arrive in no particular order (`fixed` false: the row's bound is not finite).
template <typename T>
__device__ __forceinline__ void acc_add(Slot* slot, Slot bits, double scale, bool fixed) {
  if constexpr (kIsFloat<T>) {
    if (fixed) atomicAdd(slot, to_fixed<T>(bits, scale));
    else atomicAdd(reinterpret_cast<double*>(slot), __longlong_as_double((long long)bits));
  } else {
    atomicAdd(slot, bits);
  }
}
// The same for a slot in shared memory, where a 64-bit atomic addition is a compare-and-swap loop: two
// 32-bit additions, the carry of the lower one into the upper one.
template <typename T>
__device__ __forceinline__ void acc_add_smem(Slot* slot, Slot bits, double scale, bool fixed) {
  if constexpr (kIsFloat<T>) {
    if (!fixed) {
      atomicAdd(reinterpret_cast<double*>(slot), __longlong_as_double((long long)bits));
      return;
    }
    bits = to_fixed<T>(bits, scale);
  }
  unsigned* half = reinterpret_cast<unsigned*>(slot);
  const unsigned lo = (unsigned)bits, old = atomicAdd(half, lo);
  if constexpr (sizeof(T) == 8 || kIsFloat<T>) atomicAdd(half + 1, (unsigned)(bits >> 32) + (old + lo < old));
}

template <typename T>
__device__ __forceinline__ T acc_value(Slot v, double scale, bool fixed) {
  if constexpr (kIsFloat<T>) return fixed ? from_fixed<T>(v, scale) : (T)__longlong_as_double((long long)v);
  else return (T)v;
}

template <typename T>
__global__ void spgemm_max_abs_kernel(const int* __restrict__ nnz_ptr, const T* __restrict__ val,
                                      unsigned long long* out) {
  const long long nnz = *nnz_ptr;
  double mx = 0.0;
  bool bad = false;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < nnz;
       p += (long long)gridDim.x * blockDim.x) {
    const double v = fabs((double)val[p]);
    if (!(v < 1.0e300)) bad = true; else mx = fmax(mx, v);
  }
  if (bad) mx = __longlong_as_double(0x7ff0000000000000LL);  // +inf: sorts above every finite bit pattern
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(FULL, mx, o));
  // non-negative doubles order like their bit patterns
  if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(mx));
}


constexpr int kHistBuckets = 2048;    // buckets counted in shared memory

// Buckets of every row of the batch: their row; counts zeroed.
__global__ void big_setup_kernel(BigArea b, int rows) {
  const int r = blockIdx.x;
  const int p1 = b.p0[r + 1];
  for (int p = b.p0[r] + threadIdx.x; p < p1; p += blockDim.x) {
    b.bucket_row[p] = r;
    b.cnt[p] = 0;
  }
}

// Fixed-point scale of every row of the batch, from sum |a| over the row and max |b|.
template <typename T>
__global__ void __launch_bounds__(256)
big_scale_kernel(BigArea b, const int* __restrict__ Apos, const T* __restrict__ Aval,
                 const unsigned long long* __restrict__ max_b) {
  __shared__ double s_part[8];
  const int row = b.row[blockIdx.x];
  const unsigned e = __ldg(Apos + row + 1);
  double s = 0.0;
  for (unsigned p = __ldg(Apos + row) + threadIdx.x; p < e; p += 256) s += fabs((double)Aval[p]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) s += s_part[w];
    b.scale[blockIdx.x] = scale_for_bound(s * __longlong_as_double((long long)*max_b));
  }
}

// One task = some entries of one long row of A, or, of a row of up to 512 entries, a part of the products.  SCATTER
// false: products per bucket; true: every product's column (and value) to the next free place of its bucket.  A task of
// the first kind takes up to kTurnProducts products per 256 entries; what is beyond that - an entry of A can bring
// 400,000 - is noted by the counting kernel in equal parts, which REST launches of both take: the CTA that had such an
// entry kept the GPU waiting.
// (One 16-byte record per product: a column and a value array cost a third scattered access.)
// Bound: the latency of a batch (B's entries in short pieces, places, stores).  A CTA counts kScatter products a
// thread per bucket, takes their places together, one atomic per bucket, and writes them in the buckets' order.
// Rows of more buckets than are counted in shared memory take a place per product.  67 M products of 2,350 rows:
// counted in 0.27 ms (0.56 with a task per 512 entries), scattered in 1.0 (1.47).
constexpr int kScatter = 8, kScatterCta = 256 * kScatter;
template <typename T, bool NUMERIC, bool SCATTER>
struct BigExpandSmem {
  int hist[kHistBuckets], to[SCATTER ? kHistBuckets : 1], warp[8];
  unsigned col[SCATTER ? kScatterCta : 1];
  Slot val[SCATTER && NUMERIC ? kScatterCta : 1];
  ExpandSmem<T, 256> expand;
};
template <typename T, bool NUMERIC, bool SCATTER, bool REST>
__device__ __forceinline__ void big_expand(const BigArea& b, const CsrIn& in, BigExpandSmem<T, NUMERIC, SCATTER>& sm,
                                           int r, int ab, int ae, int begin, int step, int end) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int p0 = b.p0[r], buckets = b.p0[r + 1] - p0, shift = b.shift[r], per = (buckets + 255) / 256;
  const bool in_smem = buckets <= kHistBuckets;
  if (in_smem) {
    for (int p = tid; p < buckets; p += 256) sm.hist[p] = 0;
    __syncthreads();
  }
  const T* Bval = static_cast<const T*>(in.Bval);
  auto put = [&](int slot, unsigned c, Slot v) {
    if (NUMERIC) b.rec[slot] = BigRecord{c, 0u, v};
    else b.key[slot] = c;
  };
  unsigned turn0 = ab;
  expand_turns<T, NUMERIC, 256>(in, ab, ae, sm.expand, tid, [&](int, int total, auto&& find) {
    if (!REST && !SCATTER && total > end) {
      __shared__ int s_rest;
      const int n = (total - 1) / kTurnProducts;
      if (tid == 0) s_rest = atomicAdd(b.nrest, n);
      __syncthreads();
      for (int x = tid; x < n; x += 256)
        b.rest[s_rest + x] = make_int4(r, (int)turn0, (int)min(turn0 + 256, (unsigned)ae), (x + 1) * kTurnProducts);
      __syncthreads();
    }
    turn0 += 256;
    total = min(total, end);
    for (int q0 = begin; q0 < total; q0 += step) {
      unsigned c[kScatter];
      Slot v[kScatter];
      int rank[kScatter];
#pragma unroll
      for (int k = 0; k < kScatter; k++) {
        const int q = q0 + k * 256 + tid;
        if (q >= total) continue;
        const int e = find(q), pb = sm.expand.off[e] + q;
        c[k] = (unsigned)__ldg(in.Bcrd + pb);
        if (SCATTER) v[k] = NUMERIC ? product_bits<T>(sm.expand.a[e], __ldg(Bval + pb)) : 0;
      }
      if (!in_smem) {
#pragma unroll
        for (int k = 0; k < kScatter; k++) {
          if (q0 + k * 256 + tid >= total) continue;
          const int p = p0 + (int)(c[k] >> shift);
          if (SCATTER) put(atomicAdd(&b.cursor[p], 1), c[k], v[k]);
          else atomicAdd(&b.cnt[p], 1);
        }
        continue;
      }
#pragma unroll
      for (int k = 0; k < kScatter; k++)
        if (q0 + k * 256 + tid < total) rank[k] = atomicAdd(&sm.hist[c[k] >> shift], 1);
      if constexpr (SCATTER) {
        __syncthreads();
        // counts to places of the buckets in the batch (hist) and, less these, in the area (to)
        int sum = 0;
        for (int p = tid * per; p < min(buckets, tid * per + per); p++) sum += sm.hist[p];
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(FULL, incl, o);
          if (lane >= o) incl += y;
        }
        if (lane == 31) sm.warp[warp] = incl;
        __syncthreads();
        int at = incl - sum;
#pragma unroll
        for (int w = 0; w < 8; w++) at += w < warp ? sm.warp[w] : 0;
        for (int p = tid * per; p < min(buckets, tid * per + per); p++) {
          const int n = sm.hist[p];
          if (n) sm.to[p] = atomicAdd(&b.cursor[p0 + p], n) - at;
          sm.hist[p] = at;
          at += n;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kScatter; k++) {
          if (q0 + k * 256 + tid < total) {
            const int x = sm.hist[c[k] >> shift] + rank[k];
            sm.col[x] = c[k];
            if (NUMERIC) sm.val[x] = v[k];
          }
        }
        __syncthreads();
        for (int x = tid; x < min(total - q0, kScatterCta); x += 256)
          put(sm.to[sm.col[x] >> shift] + x, sm.col[x], NUMERIC ? sm.val[x] : 0);
        for (int p = tid; p < buckets; p += 256) sm.hist[p] = 0;
        __syncthreads();
      }
    }
  });
  if (!SCATTER && in_smem) {
    __syncthreads();
    for (int p = tid; p < buckets; p += 256) {
      const int c = sm.hist[p];
      if (c) atomicAdd(&b.cnt[p0 + p], c);
    }
    __syncthreads();
  }
}

template <typename T, bool NUMERIC, bool SCATTER, bool REST>
__global__ void __launch_bounds__(256)
big_expand_kernel(BigArea b, CsrIn in) {
  __shared__ BigExpandSmem<T, NUMERIC, SCATTER> sm;
  if (REST) {
    const int n = *b.nrest;
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
      const int4 x = b.rest[i];
      big_expand<T, NUMERIC, SCATTER, true>(b, in, sm, x.x, x.y, x.z, x.w, kScatterCta, x.w + kTurnProducts);
      __syncthreads();
    }
  } else {
    const int4 x = b.tasks[blockIdx.x];
    const int part = x.w >> 16, parts = x.w & 0xffff;
    big_expand<T, NUMERIC, SCATTER, false>(b, in, sm, x.x, x.y, x.z, part * kScatterCta, max(parts, 1) * kScatterCta,
                                           parts ? INT_MAX : kTurnProducts);
  }
}

// Buckets of at most kBucketSort products: sorted by column, the sums of equal columns left, in
// place, at the bucket's start.  ucnt: distinct columns.
template <typename T, bool NUMERIC, typename KEY>
__global__ void __launch_bounds__(128)
big_sort_kernel(BigArea b) {
  constexpr int NT = 128;
  __shared__ __align__(16) KEY s_keys[kBucketSort];
  __shared__ Slot s_prods[NUMERIC ? kBucketSort : 1];
  __shared__ int s_part[NT / 32];
  const int p = blockIdx.x, tid = threadIdx.x;
  const int o = b.off[p], count = b.off[p + 1] - o;
  if (count > kBucketSort) return;
  if (count == 0) {
    if (tid == 0) b.ucnt[p] = 0;
    return;
  }
  const int r = b.bucket_row[p], shift = b.shift[r], lo = (int)((unsigned)(p - b.p0[r]) << shift);
  constexpr int kOrd = 11;   // 2048 ordinals
  for (int x = tid; x < count; x += NT) {
    unsigned c;
    if (NUMERIC) {
      const BigRecord q = b.rec[o + x];
      c = q.col;
      s_prods[x] = q.prod;
    } else {
      c = b.key[o + x];
    }
    s_keys[x] = ((KEY)(c - (unsigned)lo) << kOrd) | (KEY)x;
  }
  __syncthreads();
  if (count <= 4 * NT) sort_keys<KEY, 4, NT>(s_keys, count, tid);
  else if (count <= 8 * NT) sort_keys<KEY, 8, NT>(s_keys, count, tid);
  else sort_keys<KEY, 16, NT>(s_keys, count, tid);
  double scale = 1.0;
  if (NUMERIC && kIsFloat<T>) scale = b.scale[r];
  const bool fixed = scale == scale;
  const int u = emit_runs<KEY, NT, NUMERIC>(s_keys, count, kOrd, tid, s_part, lo, o,
                                            [&](long long at, int col, int x, int last) {
    const KEY mask = ((KEY)1 << kOrd) - 1;
    T v;
    if (last == x + 1) {
      v = one_product<T>(s_prods[(int)(s_keys[x] & mask)]);
    } else {
      // (the ordinals are the order of arrival: sums that do not depend on it)
      Slot s = 0;
      double f = 0.0;
      for (; x < last; x++) {
        const Slot q = s_prods[(int)(s_keys[x] & mask)];
        if (!kIsFloat<T>) s += q;
        else if (fixed) s += to_fixed<T>(q, scale);
        else f += __longlong_as_double((long long)q);
      }
      v = kIsFloat<T> && !fixed ? (T)f : acc_value<T>(s, scale, true);
    }
    b.rec[at].col = (unsigned)col;
    *reinterpret_cast<T*>(&b.rec[at].prod) = v;
  });
  if (tid == 0) b.ucnt[p] = u;
}

// Larger buckets (columns that many products share): windows of kWindow columns, the bucket's
// products run through once per window and added to accumulators in shared memory.  The result goes
// to the second copy of the bucket, since the products are read again for the next window.
constexpr int kWindow = 8192;
template <typename T, bool NUMERIC>
__global__ void __launch_bounds__(512)
big_window_kernel(BigArea b, int buckets, long long n) {
  constexpr int NT = 512;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned* bits = reinterpret_cast<unsigned*>(smem_raw);           // kWindow / 32 words
  Slot* acc = reinterpret_cast<Slot*>(smem_raw + kWindow / 8);
  __shared__ int s_part[NT / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int q0 = blockIdx.x * NT; q0 < buckets; q0 += gridDim.x * NT) {
    const bool mine = q0 + tid < buckets && b.off[q0 + tid + 1] - b.off[q0 + tid] > kBucketSort;
    if (!__syncthreads_or(mine)) continue;
    for (int p = q0; p < min(buckets, q0 + NT); p++) {
      const int o = b.off[p], count = b.off[p + 1] - o;
      if (count <= kBucketSort) continue;
      const int r = b.bucket_row[p], shift = b.shift[r];
      const long long lo = (long long)(p - b.p0[r]) << shift, hi = min(n, lo + (1ll << shift));
      double scale = 1.0;
      if (NUMERIC && kIsFloat<T>) scale = b.scale[r];
      const bool fixed = scale == scale;
      int done = 0;
      for (long long w0 = lo; w0 < hi; w0 += kWindow) {
        __syncthreads();
        for (int x = tid; x < kWindow / 32; x += NT) bits[x] = 0;
        if (NUMERIC)
          for (int x = tid; x < kWindow; x += NT) acc[x] = 0;
        __syncthreads();
        for (int x = tid; x < count; x += NT) {
          const long long d = (long long)(NUMERIC ? b.rec[o + x].col : b.key[o + x]) - w0;
          if (d < 0 || d >= kWindow) continue;
          atomicOr(&bits[d >> 5], 1u << (d & 31));
          if (NUMERIC) acc_add_smem<T>(&acc[d], b.rec[o + x].prod, scale, fixed);
        }
        __syncthreads();
        // 256 words: threads 0..255 take one each, in column order
        unsigned m = tid < kWindow / 32 ? bits[tid] : 0;
        const int c = __popc(m);
        int incl = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int y = __shfl_up_sync(FULL, incl, d);
          if (lane >= d) incl += y;
        }
        if (lane == 31) s_part[warp] = incl;
        __syncthreads();
        int before = 0, total = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; w++) {
          const int v = s_part[w];
          if (w < warp) before += v;
          total += v;
        }
        if (NUMERIC) {
          int at = o + done + before + incl - c;
          while (m) {
            const int d = tid * 32 + __ffs(m) - 1;
            m &= m - 1;
            b.rec2[at].col = (unsigned)(w0 + d);
            *reinterpret_cast<T*>(&b.rec2[at].prod) = acc_value<T>(acc[d], scale, fixed);
            at++;
          }
        }
        done += total;
      }
      if (tid == 0) b.ucnt[p] = done;
      __syncthreads();
    }
  }
}

// Distinct columns per row of the batch.
__global__ void big_count_rows_kernel(BigArea b, int rows, int* __restrict__ row_cnt) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < rows) row_cnt[b.row[r]] = b.uoff[b.p0[r + 1]] - b.uoff[b.p0[r]];
}

// The buckets' results to their rows: a warp per bucket.
template <typename T>
__global__ void __launch_bounds__(256)
big_store_kernel(BigArea b, int buckets, RowsOut out) {
  const int p = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (p >= buckets) return;
  const int o = b.off[p], u = b.ucnt[p], r = b.bucket_row[p];
  const bool second = b.off[p + 1] - o > kBucketSort;
  const BigRecord* rec = (second ? b.rec2 : b.rec) + o;
  const long long dst = (long long)out.off[b.row[r]] + (b.uoff[p] - b.uoff[b.p0[r]]);
#pragma unroll 4
  for (int x = lane; x < u; x += 32) {
    const BigRecord q = rec[x];
    out.crd[dst + x] = (int)q.col;
    static_cast<T*>(out.val)[dst + x] = *reinterpret_cast<const T*>(&q.prod);
  }
}

// ---- rows of more products than the area holds -------------------------------------------------
// Dense bitmap (+ accumulator) of n columns in the area.  Rows are handled in batches of up to `slots` rows, one
// slot each; a row's A entries are cut into chunks of kDenseChunk entries and the (row, chunk)
// tasks of a batch are handed out through an atomic queue, so a hub row with hundreds of
// thousands of entries is spread over the whole GPU.  The CTA that finishes a row's last chunk
// (a counter per row, no spinning) walks the row's bitmap in ascending column order, emits the
// row and leaves bitmap and accumulator all-zero for the next batch.
constexpr int kDenseChunk = 2048;     // A entries per task

struct DenseCtl {
  int* task_pref;  // [slots + 1]
  int* done;       // [slots]
  int* queue;      // [1]
};

__global__ void dense_batch_setup_kernel(const int* __restrict__ rows, int r0, int nb,
                                         const int* __restrict__ Apos, DenseCtl ctl) {
  if (threadIdx.x == 0) {
    int run = 0;
    for (int k = 0; k < nb; k++) {
      ctl.task_pref[k] = run;
      const int i = rows[r0 + k];
      const int len = Apos[i + 1] - Apos[i];
      run += len > 0 ? (len - 1) / kDenseChunk + 1 : 1;
      ctl.done[k] = 0;
    }
    ctl.task_pref[nb] = run;
    *ctl.queue = 0;
  }
}

template <typename T, bool NUMERIC>
__global__ void __launch_bounds__(256)
spgemm_dense_kernel(const int* __restrict__ rows, int r0, int nb, CsrIn in, long long words,
                    unsigned* __restrict__ bitmap_all, Slot* __restrict__ acc_all, long long n,
                    DenseCtl ctl, const double* __restrict__ row_scale, int* __restrict__ row_cnt,
                    const int* __restrict__ Cpos,
                    int* __restrict__ Ccrd, T* __restrict__ Cval) {
  __shared__ int s_warp[8];
  __shared__ int s_base;
  __shared__ int s_task;
  __shared__ int s_last;
  __shared__ ExpandSmem<T, 256> s_expand;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int total = __ldg(ctl.task_pref + nb);
  while (true) {
    if (tid == 0) s_task = atomicAdd(ctl.queue, 1);
    __syncthreads();
    const int task = s_task;
    if (task >= total) return;
    // slot k with task_pref[k] <= task < task_pref[k+1]
    int lo = 0, hi = nb;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(ctl.task_pref + mid) <= task) lo = mid; else hi = mid;
    }
    const int k = lo;
    const int chunk = task - __ldg(ctl.task_pref + k);
    const int nchunks = __ldg(ctl.task_pref + k + 1) - __ldg(ctl.task_pref + k);
    const int i = __ldg(rows + r0 + k);
    unsigned* bitmap = bitmap_all + (long long)k * words;
    Slot* acc = NUMERIC ? acc_all + (long long)k * n : nullptr;
    double scale = 1.0;
    if (NUMERIC && kIsFloat<T>) scale = row_scale[k];
    const bool fixed = scale == scale;
    const int ab = __ldg(in.Apos + i) + chunk * kDenseChunk;
    const int ae = ab + min(__ldg(in.Apos + i + 1) - ab, kDenseChunk);
    auto add = [&](T av, int pb) {
      const int c = __ldg(in.Bcrd + pb);
      if (NUMERIC) acc_add<T>(acc + c, product_bits<T>(av, static_cast<const T*>(in.Bval)[pb]), scale, fixed);
      atomicOr(&bitmap[c >> 5], 1u << (c & 31));
    };
    expand_cta<T, NUMERIC, 256>(in, ab, ae, s_expand, tid, [&](int, T a, int pb) { add(a, pb); });
    // publish this chunk, then find out whether it was the row's last one
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = (atomicAdd(ctl.done + k, 1) == nchunks - 1);
    __syncthreads();
    if (!s_last) continue;
    __threadfence();
    // walk the bitmap in ascending order, 256 words per step
    if (tid == 0) s_base = 0;
    __syncthreads();
    const int out0 = NUMERIC ? __ldg(Cpos + i) : 0;
    for (long long w0 = 0; w0 < words; w0 += 256) {
      const long long w = w0 + tid;
      unsigned bits = 0;
      if (w < words) {
        bits = __ldcg(bitmap + w);  // the bits were set by L2 atomics: do not trust L1
        if (bits) bitmap[w] = 0;
      }
      const int cnt = __popc(bits);
      // block-wide exclusive scan of cnt
      int incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) s_warp[warp] = incl;
      __syncthreads();
      int warp_off = 0, step_total = 0;
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const int v = s_warp[q];
        if (q < warp) warp_off += v;
        step_total += v;
      }
      const int base = s_base;
      if (NUMERIC && bits) {
        int o = out0 + base + warp_off + incl - cnt;
        while (bits) {
          const int bit = __ffs(bits) - 1;
          bits &= bits - 1;
          const long long c = w * 32 + bit;
          Ccrd[o] = (int)c;
          Cval[o] = acc_value<T>(__ldcg(acc + c), scale, fixed);
          acc[c] = 0;
          o++;
        }
      }
      __syncthreads();
      if (tid == 0) s_base = base + step_total;
      __syncthreads();
    }
    if (row_cnt && tid == 0) row_cnt[i] = s_base;
    __syncthreads();
  }
}

// ---- exclusive scan of row counts (int64 accumulate, int32 store) ------------------------------
constexpr int kScanTile = 4096;

__global__ void __launch_bounds__(1024)
scan_reduce_kernel(int m, const int* __restrict__ cnt, long long* __restrict__ block_sum) {
  __shared__ long long s[32];
  const long long base = (long long)blockIdx.x * kScanTile;
  long long v = 0;
  for (int q = 0; q < 4; q++) {
    const long long i = base + q * 1024 + threadIdx.x;
    if (i < m) v += cnt[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = s[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    if (threadIdx.x == 0) block_sum[blockIdx.x] = v;
  }
}

// Exclusive scan of the tiles' sums by one CTA, 1024 at a time.
__global__ void __launch_bounds__(1024)
scan_blocks_kernel(int nb, long long* block_sum, long long* hdr_total) {
  __shared__ long long s[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long run = 0;
  for (int b0 = 0; b0 < nb; b0 += 1024) {
    const int b = b0 + threadIdx.x;
    const long long v = b < nb ? block_sum[b] : 0;
    long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      long long w = s[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(FULL, w, o);
        if (lane >= o) w += y;
      }
      s[lane] = w;
    }
    __syncthreads();
    if (b < nb) block_sum[b] = run + (warp ? s[warp - 1] : 0) + incl - v;
    run += s[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) *hdr_total = run;
}

__global__ void __launch_bounds__(1024)
scan_write_kernel(int m, const int* __restrict__ cnt, const long long* __restrict__ block_sum,
                  int* __restrict__ Cpos) {
  __shared__ long long s[32];
  const long long base = (long long)blockIdx.x * kScanTile;
  // each thread owns 4 consecutive rows
  const long long i0 = base + (long long)threadIdx.x * 4;
  int c[4];
  long long mine = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    c[q] = (i0 + q < m) ? cnt[i0 + q] : 0;
    mine += c[q];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    long long v = s[lane];
    long long iv = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(FULL, iv, o);
      if (lane >= o) iv += y;
    }
    s[lane] = iv - v;  // exclusive over warps
  }
  __syncthreads();
  long long run = block_sum[blockIdx.x] + s[warp] + incl - mine;
  if (blockIdx.x == 0 && threadIdx.x == 0) Cpos[0] = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    run += c[q];
    if (i0 + q < m) Cpos[i0 + q + 1] = (int)run;
  }
}

// Short arrays in one launch: a CTA scans 1024 counts and adds up all that lie before them, so that no CTA
// waits for another.  (By one CTA: 7.3 us for 20,000 counts, 4.0 this way.)
constexpr int kScanSmall = 32768;
__global__ void __launch_bounds__(1024)
scan_small_kernel(int m, const int* __restrict__ cnt, int* __restrict__ out, long long* __restrict__ total) {
  __shared__ long long s_before[32], s_sum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, b0 = blockIdx.x * 1024;
  long long before = 0;
#pragma unroll 8
  for (int x = tid; x < b0; x += 1024) before += __ldg(cnt + x);
  const int i = b0 + tid, c = i < m ? __ldg(cnt + i) : 0;
  long long incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(FULL, before, o);
  if (lane == 0) s_before[warp] = before;
  if (lane == 31) s_sum[warp] = incl;
  __syncthreads();
  long long at = s_before[lane] + (lane < warp ? s_sum[lane] : 0);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) at += __shfl_xor_sync(FULL, at, o);
  at += incl;
  if (i < m) out[i + 1] = (int)at;
  if (i == 0) out[0] = 0;
  if (i == m - 1) *total = at;
}

// Exclusive scan of n int counts into out[0..n] (int32), running total in int64 at *total_dev.
// `block_sum` needs ceil(n / 4096) + 1 int64 slots.
int exclusive_scan_i32(int n, const int* cnt, int* out, long long* block_sum, long long* total_dev,
                       cudaStream_t st) {
  if (n <= 0) {
    SB_CUDA(cudaMemsetAsync(out, 0, 4, st));
    SB_CUDA(cudaMemsetAsync(total_dev, 0, 8, st));
    return SB_OK;
  }
  if (n <= kScanSmall) {
    scan_small_kernel<<<(unsigned)ceil_div(n, 1024), 1024, 0, st>>>(n, cnt, out, total_dev);
    SB_LAUNCH_CHECK("scan_small_kernel");
    return SB_OK;
  }
  const int nb = (int)ceil_div(n, kScanTile);
  scan_reduce_kernel<<<nb, 1024, 0, st>>>(n, cnt, block_sum);
  SB_LAUNCH_CHECK("scan_reduce_kernel");
  scan_blocks_kernel<<<1, 1024, 0, st>>>(nb, block_sum, total_dev);
  SB_LAUNCH_CHECK("scan_blocks_kernel");
  scan_write_kernel<<<nb, 1024, 0, st>>>(n, cnt, block_sum, out);
  SB_LAUNCH_CHECK("scan_write_kernel");
  return SB_OK;
}

// ---- long rows of a matrix of few columns ---------------------------------------------------------
// Bitmap and accumulators of all n columns in shared memory (n up to kSmemColumns): no plan, no read-back,
// one launch instead of the bucket path's ten.  Few such rows leave most of the GPU to the others, so up to
// eight CTAs - a cluster - share a row: each takes its part of the products into a bitmap and accumulators
// of its own, then emits a slice of the columns, adding the others' sums out of their shared memory
// (CLUSTERED).  20,011 columns, ten rows of 8,200 to 80,000 products: 190 us by buckets, 92 by one CTA per
// row (beside the other bins' kernels), 49 by clusters of eight.
constexpr int kSmemThreads = 1024, kSmemParts = 8;
template <typename T, bool NUMERIC, bool CLUSTERED>
__global__ void __launch_bounds__(kSmemThreads)
spgemm_smem_kernel(const int* __restrict__ rows, CsrIn in, int n, const unsigned long long* __restrict__ max_b,
                   RowsOut out) {
  constexpr int NT = kSmemThreads, NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned* bits = reinterpret_cast<unsigned*>(smem_raw);            // kSmemColumns / 32 words
  Slot* acc = reinterpret_cast<Slot*>(smem_raw + kSmemColumns / 8);
  __shared__ ExpandSmem<T, NT> s_expand;
  __shared__ double s_abs[NW];
  __shared__ int s_part[NW], s_at[kSmemColumns / 32];
  __shared__ unsigned s_words[CLUSTERED ? kSmemColumns / 32 : 1];   // the parts' words of this CTA's columns
  __shared__ int s_total;
  let_next_begin();
  namespace cg = cooperative_groups;
  const int parts = CLUSTERED ? (int)cg::this_cluster().num_blocks() : 1;
  const int part = CLUSTERED ? (int)cg::this_cluster().block_rank() : 0;
  const int i = __ldg(rows + blockIdx.x / parts), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ab = __ldg(in.Apos + i), ae = __ldg(in.Apos + i + 1);
  for (int x = tid; x < kSmemColumns / 32; x += NT) bits[x] = 0;
  if (NUMERIC)
    for (int x = tid; x < (n + 1) / 2; x += NT) reinterpret_cast<ulonglong2*>(acc)[x] = ulonglong2{0, 0};
  double scale = 1.0;
  if constexpr (NUMERIC && kIsFloat<T>) {
    double s = 0.0;
    const T* Aval = static_cast<const T*>(in.Aval);
    for (unsigned p = (unsigned)ab + tid; p < (unsigned)ae; p += NT) s += fabs((double)Aval[p]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
    if (lane == 0) s_abs[warp] = s;
    __syncthreads();
    s = 0.0;
    for (int w = 0; w < NW; w++) s += s_abs[w];
    scale = scale_for_bound(s * __longlong_as_double((long long)*max_b));
  }
  const bool fixed = scale == scale;
  __syncthreads();
  const T* Bval = static_cast<const T*>(in.Bval);
  // a row of many entries is cut by entries (every part looking all of them up took 51,000 cycles for 10,014 of
  // them, 23,000 to 43,000 this way), one of few by products: a single entry can bring most of them
  const bool by_entries = parts > 1 && ae - ab >= 2 * NT;
  const int share = by_entries ? (ae - ab - 1) / parts + 1 : ae - ab;
  const int eb = by_entries ? ab + part * share : ab, ee = by_entries ? eb + min(ae - eb, share) : ae;
  expand_cta<T, NUMERIC, NT>(in, eb, ee, s_expand, tid, [&](int, T a, int pb) {
    const int c = __ldg(in.Bcrd + pb);
    const unsigned bit = 1u << (c & 31);
    if (!(bits[c >> 5] & bit)) atomicOr(&bits[c >> 5], bit);
    if (NUMERIC) acc_add_smem<T>(&acc[c], product_bits<T>(a, __ldg(Bval + pb)), scale, fixed);
  }, by_entries ? 0 : part, by_entries ? 1 : parts);
  // this CTA's words of the bitmap (kSmemColumns / 32 = 768 in all), one per thread, in column order
  const int words = kSmemColumns / 32 / parts, w0 = part * words;
  unsigned m = 0;
  if constexpr (CLUSTERED) {
    cg::this_cluster().sync();
    if (tid < words) {
#pragma unroll
      for (int p = 0; p < kSmemParts; p++) {
        if (p >= parts) break;
        const unsigned x = cg::this_cluster().map_shared_rank(bits, p)[w0 + tid];
        s_words[p * words + tid] = x;
        m |= x;
      }
      bits[w0 + tid] = m;      // (a part's words are read by that part alone)
    }
  } else {
    __syncthreads();
    if (tid < words) m = bits[tid];
  }
  const int c = __popc(m);
  int incl = c;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, d);
    if (lane >= d) incl += y;
  }
  if (lane == 31) s_part[warp] = incl;
  __syncthreads();
  int before = 0, total = 0;
#pragma unroll
  for (int w = 0; w < NW; w++) {
    const int v = s_part[w];
    if (w < warp) before += v;
    total += v;
  }
  int before_parts = 0;
  if constexpr (CLUSTERED) {
    if (tid == 0) s_total = total;
    cg::this_cluster().sync();
    total = 0;
#pragma unroll
    for (int p = 0; p < kSmemParts; p++) {
      const int v = p < parts ? *cg::this_cluster().map_shared_rank(&s_total, p) : 0;
      if (p < part) before_parts += v;
      total += v;
    }
  }
  if (out.row_cnt && tid == 0 && part == 0) out.row_cnt[i] = total;
  if (NUMERIC) {
    // a warp per word, a lane per column
    if (tid < words) s_at[tid] = before + incl - c;
    __syncthreads();
    const long long base = __ldg(out.off + i) + before_parts;
    const double inv = 1.0 / scale;
    for (int w = warp; w < words; w += NW) {
      const unsigned word = bits[w0 + w];
      if (!(word >> lane & 1)) continue;
      const long long at = base + s_at[w] + __popc(word & ((1u << lane) - 1u));
      const int col = (w0 + w) * 32 + lane;
      Slot v = acc[col];
      if constexpr (CLUSTERED) {
        Slot x[kSmemParts];
#pragma unroll
        for (int p = 0; p < kSmemParts; p++) {   // (only what a part has: 140 KB a CTA otherwise)
          const bool has = p < parts && s_words[p * words + w] >> lane & 1;
          x[p] = has ? *cg::this_cluster().map_shared_rank(acc + col, p) : 0;
        }
        v = x[0];
#pragma unroll
        for (int p = 1; p < kSmemParts; p++) {
          if (kIsFloat<T> && !fixed)
            v = (Slot)__double_as_longlong(__longlong_as_double((long long)v) + __longlong_as_double((long long)x[p]));
          else
            v += x[p];
        }
      }
      out.crd[at] = col;
      T value;
      if constexpr (kIsFloat<T>)
        value = fixed ? (T)((double)(long long)v * inv) : (T)__longlong_as_double((long long)v);
      else
        value = (T)v;
      static_cast<T*>(out.val)[at] = value;
    }
  }
  if constexpr (CLUSTERED) cg::this_cluster().sync();   // (the others read this CTA's sums)
  end_after_previous();
}

// ---- one-pass form: the rows' entries from their product offsets to their place ------------------
// A CTA moves `tile` consecutive entries of the result, whatever the rows' lengths (a warp per row
// left the hub rows to a warp each: 4.7 ms for 272 M entries); a thread finds the row of its entry
// among the tile's row pointers in shared memory.  Tiles of kMoveTile entries, smaller where that leaves SMs idle
// (1.1 M entries: 15.3 us in 136 tiles of 8192, 9.4 in 542 of 2048).
// The places of kMoveAhead entries are found before the first is loaded: 284 M entries 1.06 ms one by one, 0.76 so =
// 6.0 TB/s.
constexpr int kMoveTile = 8192, kMoveRows = 1024, kMoveAhead = 4;
template <typename T>
__global__ void __launch_bounds__(256)
spgemm_move_kernel(int m, int nnz, int tile, const int* __restrict__ off, const int* __restrict__ Cpos,
                   const int* __restrict__ tcrd, const T* __restrict__ tval, int* __restrict__ Ccrd,
                   T* __restrict__ Cval) {
  __shared__ int s_pos[kMoveRows + 1], s_shift[kMoveRows];
  __shared__ int s_first[kMoveRows / 32], s_count[8];
  const int tid = threadIdx.x, lane = tid & 31;
  const int e1 = min((long long)nnz, ((long long)blockIdx.x + 1) * tile);
  for (int e = blockIdx.x * tile; e < e1;) {
    const int r0 = cta_row_of<256>(Cpos, m, e, s_count);
    for (int x = tid; x < kMoveRows + 1; x += 256) {
      const int r = min(m, r0 + x), p = __ldg(Cpos + r);
      s_pos[x] = p;
      if (x % 32 == 0 && x < kMoveRows) s_first[x / 32] = p;
      if (x < kMoveRows && r < m) s_shift[x] = __ldg(off + r) - p;
    }
    __syncthreads();
    const int stop = min(e1, s_pos[kMoveRows]), count = stop - e;
    // (counted from the first entry: entry numbers themselves may end at 2^31 - 1, a step beyond it wraps)
    for (int t0 = tid & ~31; t0 < count; t0 += 256 * kMoveAhead) {
      int src[kMoveAhead];
#pragma unroll
      for (int q = 0; q < kMoveAhead; q++) {
        // the row of the warp's first entry by two rounds of 32 looks, this lane's a few rows behind it
        const int t = t0 + q * 256, first = e + min(t, count - 1), o = e + min(t + lane, count - 1);
        const int c = __popc(__ballot_sync(FULL, s_first[lane] <= first)) - 1;
        int r = 32 * c + __popc(__ballot_sync(FULL, s_pos[32 * c + lane] <= first)) - 1;
#pragma unroll 1
        for (int step = 0; step < 6 && s_pos[r + 1] <= o; step++) r++;
        if (s_pos[r + 1] <= o) {           // many short or empty rows
          int hi = kMoveRows;
          while (hi - r > 1) {
            const int mid = (r + hi) >> 1;
            if (s_pos[mid] <= o) r = mid; else hi = mid;
          }
        }
        src[q] = o + s_shift[r];
      }
      int crd[kMoveAhead];
      T val[kMoveAhead];
#pragma unroll
      for (int q = 0; q < kMoveAhead; q++) {
        if (t0 + q * 256 + lane >= count) continue;
        crd[q] = __ldg(tcrd + src[q]);
        val[q] = __ldg(tval + src[q]);
      }
#pragma unroll
      for (int q = 0; q < kMoveAhead; q++) {
        const int t = t0 + q * 256 + lane;
        if (t >= count) continue;
        Ccrd[e + t] = crd[q];
        Cval[e + t] = val[q];
      }
    }
    e = stop;
    __syncthreads();
  }
}

// ---- host side ---------------------------------------------------------------------------------
__global__ void big_info_kernel(const int* __restrict__ rows, int count, const int* __restrict__ upper,
                                const int* __restrict__ Apos, int4* __restrict__ info) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= count) return;
  const int i = rows[x];
  info[x] = make_int4(i, upper[i], Apos[i], Apos[i + 1]);
}

static int ceil_log2(int64_t x) {
  int b = 0;
  while (((int64_t)1 << b) < x) b++;
  return b;
}

// Rows with more products than the area holds, one after the other.
template <typename T, bool NUMERIC>
static int dense_row(const WsLayout& w, int row, int64_t n, const CsrIn& in, const RowsOut& out, cudaStream_t st) {
  char* p = w.area;
  int* ctl = reinterpret_cast<int*>(p);                         // [0..1] tasks, [2] done, [3] queue, [4] row
  double* scale = reinterpret_cast<double*>(p + 64);
  unsigned* bitmap = reinterpret_cast<unsigned*>(p + align_up(4096));
  Slot* acc = reinterpret_cast<Slot*>(p + align_up(4096) + align_up(dense_words(n) * 4));
  SB_CUDA(cudaMemsetAsync(bitmap, 0, dense_words(n) * 4, st));
  SB_CUDA(cudaMemcpyAsync(ctl + 4, &row, 4, cudaMemcpyHostToDevice, st));
  if (NUMERIC) {
    SB_CUDA(cudaMemsetAsync(acc, 0, (size_t)n * 8, st));
    if constexpr (kIsFloat<T>) {
      BigArea b{};
      b.row = ctl + 4;
      b.scale = scale;
      big_scale_kernel<T><<<1, 256, 0, st>>>(b, in.Apos, static_cast<const T*>(in.Aval), w.max_b);
      SB_LAUNCH_CHECK("big_scale_kernel");
    }
  }
  DenseCtl c{ctl, ctl + 2, ctl + 3};
  dense_batch_setup_kernel<<<1, 32, 0, st>>>(ctl + 4, 0, 1, in.Apos, c);
  SB_LAUNCH_CHECK("dense_batch_setup_kernel");
  spgemm_dense_kernel<T, NUMERIC><<<4 * sm_count(), 256, 0, st>>>(
      ctl + 4, 0, 1, in, (long long)dense_words(n), bitmap, acc, (long long)n, c, scale, out.row_cnt, out.off, out.crd,
      static_cast<T*>(out.val));
  SB_LAUNCH_CHECK("spgemm_dense_kernel");
  return SB_OK;
}

// One batch of long rows whose plan (rows, first buckets, shifts, tasks) is in host memory.
template <typename T, bool NUMERIC>
static int big_batch(const WsLayout& w, const std::vector<int>& row, const std::vector<int>& p0,
                     const std::vector<int>& shift, const std::vector<int4>& tasks, int64_t n, const CsrIn& in,
                     const RowsOut& out, cudaStream_t st) {
  const BigArea b = big_area(w.area, w.products);
  const int rows = (int)row.size(), buckets = p0.back();
  SB_CUDA(cudaMemcpyAsync(b.row, row.data(), row.size() * 4, cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(b.p0, p0.data(), p0.size() * 4, cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(b.shift, shift.data(), shift.size() * 4, cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaMemcpyAsync(b.tasks, tasks.data(), tasks.size() * sizeof(int4), cudaMemcpyHostToDevice, st));
  // products may be left over where a row is cut by entries
  bool left = false;
  for (const int4& x : tasks) left = left || !x.w;
  if (left) SB_CUDA(cudaMemsetAsync(b.nrest, 0, 4, st));
  const unsigned ntasks = (unsigned)tasks.size(), nrest = 4u * sm_count();
  big_setup_kernel<<<rows, 128, 0, st>>>(b, rows);
  SB_LAUNCH_CHECK("big_setup_kernel");
  if constexpr (NUMERIC && kIsFloat<T>) {
    big_scale_kernel<T><<<rows, 256, 0, st>>>(b, in.Apos, static_cast<const T*>(in.Aval), w.max_b);
    SB_LAUNCH_CHECK("big_scale_kernel");
  }
  big_expand_kernel<T, false, false, false><<<ntasks, 256, 0, st>>>(b, in);
  SB_LAUNCH_CHECK("big_expand_kernel");
  if (left) {
    big_expand_kernel<T, false, false, true><<<nrest, 256, 0, st>>>(b, in);
    SB_LAUNCH_CHECK("big_expand_kernel");
  }
  int rc = exclusive_scan_i32(buckets, b.cnt, b.off, b.block_sum, w.hdr + 8, st);
  if (rc != SB_OK) return rc;
  SB_CUDA(cudaMemcpyAsync(b.cursor, b.off, (size_t)buckets * 4, cudaMemcpyDeviceToDevice, st));
  big_expand_kernel<T, NUMERIC, true, false><<<ntasks, 256, 0, st>>>(b, in);
  SB_LAUNCH_CHECK("big_expand_kernel");
  if (left) {
    big_expand_kernel<T, NUMERIC, true, true><<<nrest, 256, 0, st>>>(b, in);
    SB_LAUNCH_CHECK("big_expand_kernel");
  }
  const int widest = *std::max_element(shift.begin(), shift.end());
  if (widest + 11 <= 32) big_sort_kernel<T, NUMERIC, unsigned><<<buckets, 128, 0, st>>>(b);
  else big_sort_kernel<T, NUMERIC, unsigned long long><<<buckets, 128, 0, st>>>(b);
  SB_LAUNCH_CHECK("big_sort_kernel");
  auto window = big_window_kernel<T, NUMERIC>;
  const int smem = kWindow / 8 + (NUMERIC ? kWindow * 8 : 0);
  SB_CUDA(cudaFuncSetAttribute(window, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  window<<<(unsigned)std::min<int64_t>(ceil_div(buckets, 512), 2 * sm_count()), 512, smem, st>>>(b, buckets, n);
  SB_LAUNCH_CHECK("big_window_kernel");
  rc = exclusive_scan_i32(buckets, b.ucnt, b.uoff, b.block_sum, w.hdr + 8, st);
  if (rc != SB_OK) return rc;
  if (out.row_cnt) {
    big_count_rows_kernel<<<(unsigned)ceil_div(rows, 128), 128, 0, st>>>(b, rows, out.row_cnt);
    SB_LAUNCH_CHECK("big_count_rows_kernel");
  }
  if (NUMERIC) {
    big_store_kernel<T><<<(unsigned)ceil_div(buckets, 8), 256, 0, st>>>(b, buckets, out);
    SB_LAUNCH_CHECK("big_store_kernel");
  }
  return SB_OK;
}

// max |b|, for the fixed-point scales of the long rows.
template <typename T>
static int max_abs(const WsLayout& w, const CsrIn& in, int64_t kb, cudaStream_t st) {
  SB_CUDA(cudaMemsetAsync(w.max_b, 0, 8, st));
  spgemm_max_abs_kernel<T><<<8 * sm_count(), 256, 0, st>>>(in.Bpos + kb, static_cast<const T*>(in.Bval), w.max_b);
  SB_LAUNCH_CHECK("spgemm_max_abs_kernel");
  return SB_OK;
}

template <typename T, bool NUMERIC>
static int launch_smem_bin(const int* rows, int64_t count, const WsLayout& w, int64_t n, const CsrIn& in,
                           const RowsOut& out, bool early, cudaStream_t st) {
  const int smem = kSmemColumns / 8 + (NUMERIC ? (int)(n + 1) / 2 * 16 : 0);
  // CTAs per row: as many as keep all of them (one per SM) on the GPU at a time
  unsigned parts = kSmemParts;
  while (parts > 1 && (int64_t)parts * count > sm_count()) parts /= 2;
  if (parts == 1) {
    auto k = spgemm_smem_kernel<T, NUMERIC, false>;
    SB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    SB_CUDA(launch_kernel(early, k, dim3((unsigned)count), kSmemThreads, smem, st, rows, in, (int)n, w.max_b, out));
    return SB_OK;
  }
  auto k = spgemm_smem_kernel<T, NUMERIC, true>;
  SB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = parts;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)count * parts);
  cfg.blockDim = dim3(kSmemThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 2 : 1;
  SB_CUDA(cudaLaunchKernelEx(&cfg, k, rows, in, (int)n, (const unsigned long long*)w.max_b, out));
  return SB_OK;
}

// The long rows' numbers, products and entries, to the host.
static int big_list(const WsLayout& w, int64_t count, int64_t m, const CsrIn& in, std::vector<int4>& info,
                    cudaStream_t st) {
  info.resize((size_t)count);
  const int64_t room = (int64_t)(w.area_bytes / sizeof(int4));
  for (int64_t x0 = 0; x0 < count; x0 += room) {
    const int part = (int)std::min<int64_t>(room, count - x0);
    big_info_kernel<<<(unsigned)ceil_div(part, 256), 256, 0, st>>>(w.bin_rows + (kBins - 1) * m + x0, part, w.upper,
                                                                   in.Apos, reinterpret_cast<int4*>(w.area));
    SB_LAUNCH_CHECK("big_info_kernel");
    SB_CUDA(cudaMemcpyAsync(info.data() + x0, w.area, (size_t)part * sizeof(int4), cudaMemcpyDeviceToHost, st));
    SB_CUDA(cudaStreamSynchronize(st));
  }
  return SB_OK;
}

template <typename T, bool NUMERIC>
static int big_rows(const WsLayout& w, const std::vector<int4>& info, int64_t n, const CsrIn& in, const RowsOut& out,
                    cudaStream_t st) {
  const int nbits = ceil_log2(std::max<int64_t>(n, 1));
  std::vector<int> row, p0{0}, shift;
  std::vector<int4> tasks;
  // batches of about equal size, as few as the area allows
  int64_t products = 0, total = 0;
  for (const int4& x : info) total += x.y > w.products ? 0 : x.y;
  const int64_t target = total / std::max<int64_t>(1, ceil_div(total, w.products));
  // products per task: small enough to give every SM a few tasks
  const int64_t share = total / (4 * sm_count()) / kScatterCta * kScatterCta;
  const int64_t task_products = std::min<int64_t>(kTurnProducts, std::max<int64_t>(kScatterCta, share));
  auto flush = [&]() -> int {
    if (row.empty()) return SB_OK;
    const int rc = big_batch<T, NUMERIC>(w, row, p0, shift, tasks, n, in, out, st);
    row.clear(); shift.clear(); tasks.clear();
    p0.assign(1, 0);
    products = 0;
    return rc;
  };
  for (const int4& x : info) {
    if (x.y > w.products) {
      int rc = flush();
      if (rc == SB_OK) rc = dense_row<T, NUMERIC>(w, x.x, n, in, out, st);
      if (rc != SB_OK) return rc;
      continue;
    }
    const int s = std::max(0, nbits - ceil_log2(ceil_div(x.y, kBucketProducts)));
    const int buckets = (int)((n - 1) >> s) + 1;
    const int len = x.w - x.z;
    int chunk = 512;                     // A entries per task; the products of up to that many are cut evenly
    while (ceil_div(len, chunk) > kBigTasks / 4) chunk *= 2;
    const int parts = len <= chunk ? (int)std::min<int64_t>(kBigTasks / 4, ceil_div(x.y, task_products)) : 0;
    const int64_t more = std::max<int64_t>(parts, ceil_div(len, chunk));
    if (products >= target || products + x.y > w.products || p0.back() + buckets > big_buckets(w.products) ||
        (int64_t)tasks.size() + more > kBigTasks) {
      const int rc = flush();
      if (rc != SB_OK) return rc;
    }
    for (int part = 0; part < parts; part++) tasks.push_back(make_int4((int)row.size(), x.z, x.w, part << 16 | parts));
    if (!parts)
      for (int64_t b = x.z; b < x.w; b += chunk)
        tasks.push_back(make_int4((int)row.size(), (int)b, (int)std::min<int64_t>(b + chunk, x.w), 0));
    row.push_back(x.x);
    shift.push_back(s);
    p0.push_back(p0.back() + buckets);
    products += x.y;
  }
  return flush();
}

template <typename T, bool NUMERIC, typename KEY>
static int launch_warp_bin(const int* rows, int64_t count, const WsLayout& w, const CsrIn& in, int shift,
                           const RowsOut& out, bool early, cudaStream_t st) {
  constexpr int WARPS = 4;
  SB_CUDA(launch_kernel(early, spgemm_warp_kernel<T, NUMERIC, KEY, WARPS>, dim3((unsigned)ceil_div(count, WARPS)),
                        32 * WARPS, 0, st, rows, (int)count, w.upper, in, shift, out));
  return SB_OK;
}

template <typename T, bool NUMERIC, typename KEY, int NT, int RMAX>
static int launch_cta_bin(const int* rows, int64_t count, const WsLayout& w, const CsrIn& in, int shift,
                          const RowsOut& out, bool early, cudaStream_t st) {
  auto k = spgemm_cta_kernel<T, NUMERIC, KEY, NT, RMAX>;
  const int smem = RMAX * NT * (int)(sizeof(KEY) + (NUMERIC ? sizeof(Slot) : 0));
  SB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  SB_CUDA(launch_kernel(early, k, dim3((unsigned)count), NT, smem, st, rows, w.upper, in, shift, out));
  return SB_OK;
}

template <typename T, bool NUMERIC, int NT>
static int launch_split_rows(const int* rows, int64_t count, const WsLayout& w, const CsrIn& in, int64_t n,
                             const RowsOut& out, cudaStream_t st) {
  auto k = spgemm_split_kernel<T, NUMERIC, NT>;
  const int smem = kSplitCap * (int)(sizeof(unsigned) + (NUMERIC ? sizeof(Slot) : 0));
  SB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const unsigned width = (unsigned)std::max<int64_t>(1, ceil_div(n, kSplitSegments<NT>));
  k<<<(unsigned)count, NT, smem, st>>>(rows, w.upper, in, (int)width,
                                       (unsigned)(((1ull << 32) + width - 1) / width), out);
  SB_LAUNCH_CHECK("spgemm_split_kernel");
  return SB_OK;
}
// (a CTA per SM while all rows fit so, with twice the threads; beyond that two per SM)
template <typename T, bool NUMERIC>
static int launch_split_bin(const int* rows, int64_t count, const WsLayout& w, const CsrIn& in, int64_t n,
                            const RowsOut& out, cudaStream_t st) {
  return count <= sm_count() ? launch_split_rows<T, NUMERIC, 1024>(rows, count, w, in, n, out, st)
                             : launch_split_rows<T, NUMERIC, 512>(rows, count, w, in, n, out, st);
}

// All rows.  Bins 3 to 0 in this order, so that the short rows fill in behind the longer ones: a bin's
// kernel lets the next one start as soon as its own CTAs have (they do not depend on one another) and ends
// after the one before it.  The first of them is an ordinary launch: it begins behind the completed work of
// the stream (max |b|, the operands), and so do all that begin after it, which read these without a wait
// of their own.  The long rows of bin 4 come last.  In shared memory, theirs is one more such kernel.  By
// buckets, they are a chain of ordinary launches, which the stream holds until all the bins are done: their
// tasks are planned by the host, and planned behind the bins' launches that work keeps no GPU waiting.
// A key holds the column above the product's ordinal: 32 bits where both fit.
template <typename T, bool NUMERIC>
static int launch_bins(const WsLayout& w, const long long* counts, int64_t m, int64_t kb, int64_t n,
                       const CsrIn& in, const RowsOut& out, cudaStream_t st) {
  const int nbits = ceil_log2(std::max<int64_t>(n, 1));
  int rc = SB_OK;
  const bool in_smem = n <= kSmemColumns;
  if constexpr (NUMERIC && kIsFloat<T>) {
    if (counts[4] > 0) rc = max_abs<T>(w, in, kb, st);
    if (rc != SB_OK) return rc;
  }
  // (The long rows' list is read back ahead of the other bins, which run while the host plans the long rows' tasks.
  // A plan of more than 64 KB, which comes from pageable memory, is copied once the stream has come to it: from there
  // on the host waits for the bins, and for the batch before with every further one.)
  std::vector<int4> info;
  if (counts[4] > 0 && !in_smem) rc = big_list(w, counts[4], m, in, info, st);
  if (rc != SB_OK) return rc;
  typedef unsigned K32;
  typedef unsigned long long K64;
  const int* rows = w.bin_rows;
  bool early = false;
  if (counts[3] > 0) {
    // (a segment's part of the column and 13 bits of ordinal fit one key up to 2^24 columns)
    rc = nbits <= 24 ? launch_split_bin<T, NUMERIC>(rows + 3 * m, counts[3], w, in, n, out, st)
                     : launch_cta_bin<T, NUMERIC, K64, 512, 16>(rows + 3 * m, counts[3], w, in, 13, out, early, st);
    if (rc != SB_OK) return rc;
    early = true;
  }
  if (counts[2] > 0) {
    rc = nbits <= 21 ? launch_cta_bin<T, NUMERIC, K32, 128, 16>(rows + 2 * m, counts[2], w, in, 11, out, early, st)
                     : launch_cta_bin<T, NUMERIC, K64, 128, 16>(rows + 2 * m, counts[2], w, in, 11, out, early, st);
    if (rc != SB_OK) return rc;
    early = true;
  }
  if (counts[1] > 0) {
    rc = nbits <= 23 ? launch_cta_bin<T, NUMERIC, K32, 64, 8>(rows + m, counts[1], w, in, 9, out, early, st)
                     : launch_cta_bin<T, NUMERIC, K64, 64, 8>(rows + m, counts[1], w, in, 9, out, early, st);
    if (rc != SB_OK) return rc;
    early = true;
  }
  if (counts[0] > 0) {
    rc = nbits <= 25 ? launch_warp_bin<T, NUMERIC, K32>(rows, counts[0], w, in, 7, out, early, st)
                     : launch_warp_bin<T, NUMERIC, K64>(rows, counts[0], w, in, 7, out, early, st);
    if (rc != SB_OK) return rc;
    early = true;
  }
  if (counts[4] > 0)
    rc = in_smem ? launch_smem_bin<T, NUMERIC>(rows + 4 * m, counts[4], w, n, in, out, early, st)
                 : big_rows<T, NUMERIC>(w, info, n, in, out, st);
  return rc;
}

template <bool NUMERIC>
static int launch_bins_typed(int dtype, const WsLayout& w, const long long* counts, int64_t m, int64_t kb, int64_t n,
                             const CsrIn& in, const RowsOut& out, cudaStream_t st) {
  switch (dtype) {
    case SB_F32: return launch_bins<float, NUMERIC>(w, counts, m, kb, n, in, out, st);
    case SB_F64: return launch_bins<double, NUMERIC>(w, counts, m, kb, n, in, out, st);
    case SB_I32: return launch_bins<unsigned int, NUMERIC>(w, counts, m, kb, n, in, out, st);
    default: return launch_bins<unsigned long long, NUMERIC>(w, counts, m, kb, n, in, out, st);
  }
}

static int check_spgemm(int64_t m, int64_t kb, int64_t n, const void* Apos, const void* Bpos,
                        void* ws, size_t ws_bytes) {
  SB_CHECK_ARG(m >= 0 && kb >= 0 && n >= 0, "spgemm: negative size");
  SB_CHECK_ARG(m < INT32_MAX / 8 && kb < INT32_MAX && n < INT32_MAX - 1,
               "spgemm: dimension exceeds the supported int32 range");
  SB_CHECK_ARG(Apos && Bpos, "spgemm: null row pointers");
  SB_CHECK_ARG(ws && aligned16(ws), "spgemm: workspace is null or misaligned");
  const size_t need = sb_spgemm_workspace_bytes(m, n, SB_F32);  // the same for every dtype
  if (ws_bytes < need)
    return fail(SB_ERR_WORKSPACE, "spgemm: workspace has %zu bytes, needs %zu", ws_bytes, need);
  return SB_OK;
}

// Product bounds and bins of the rows.
static int bin_rows(const WsLayout& w, int64_t m, const int32_t* Apos, const int32_t* Acrd, const int32_t* Bpos,
                    cudaStream_t st) {
  SB_CUDA(cudaMemsetAsync(w.hdr, 0, 256 + 16 * 4, st));   // header and cursors are neighbours
  const int rows = (int)std::min<int64_t>(kBinRows, std::max<int64_t>(32, ceil_div(m, 2 * sm_count() * 32) * 32));
  spgemm_bin_kernel<<<(unsigned)ceil_div(m, rows), kBinThreads, 0, st>>>((int)m, rows, Apos, Acrd, Bpos, w.upper,
                                                                         w.bin_rows, w.bin_cursor, w.row_cnt);
  SB_LAUNCH_CHECK("spgemm_bin_kernel");
  return SB_OK;
}

// Row pointers from the rows' counts; the total, checked against int32.
static int row_pointers(const WsLayout& w, int64_t m, int32_t* Cpos, int64_t* total_host, cudaStream_t st) {
  int rc = exclusive_scan_i32((int)m, w.row_cnt, Cpos, w.block_sum, w.hdr + 8, st);
  if (rc != SB_OK) return rc;
  long long total = 0;
  SB_CUDA(cudaMemcpyAsync(&total, w.hdr + 8, 8, cudaMemcpyDeviceToHost, st));
  SB_CUDA(cudaStreamSynchronize(st));
  *total_host = total;
  if (total > INT32_MAX)
    return fail(SB_ERR_OVERFLOW, "spgemm: the product has %lld stored entries, which does not fit "
                "the int32 row pointers", total);
  return SB_OK;
}

// No C++ exception leaves a C entry point: the long rows' plans are vectors in host memory.
template <typename F>
static int caught(const char* name, F&& f) {
  try {
    return f();
  } catch (const std::exception& e) {
    return fail(SB_ERR_CUDA, "%s: out of host memory (%s)", name, e.what());
  }
}

}  // namespace sb

using namespace sb;

extern "C" {

size_t sb_spgemm_workspace_bytes(int64_t m, int64_t n, int dtype) {
  (void)dtype;   // one size for all: the symbolic phase does not know the numeric dtype
  return ws_layout(nullptr, m < 0 ? 0 : m, n < 0 ? 0 : n).total;
}

int sb_spgemm_symbolic(int64_t m, int64_t kb, int64_t n, const int32_t* Apos, const int32_t* Acrd,
                       const int32_t* Bpos, const int32_t* Bcrd, int32_t* Cpos,
                       int64_t* total_nnz_host, void* ws, size_t ws_bytes, void* stream) {
  int rc = check_spgemm(m, kb, n, Apos, Bpos, ws, ws_bytes);
  if (rc != SB_OK) return rc;
  SB_CHECK_ARG(Cpos && total_nnz_host, "spgemm_symbolic: null output");
  cudaStream_t st = (cudaStream_t)stream;
  const WsLayout w = ws_layout(ws, m, n);
  *total_nnz_host = 0;
  if (m == 0) {
    SB_CUDA(cudaMemsetAsync(w.hdr, 0, 16 * 8, st));
    SB_CUDA(cudaMemsetAsync(Cpos, 0, 4, st));
    SB_CUDA(cudaStreamSynchronize(st));
    return SB_OK;
  }
  rc = bin_rows(w, m, Apos, Acrd, Bpos, st);
  if (rc != SB_OK) return rc;
  int cursors[kBins];
  SB_CUDA(cudaMemcpyAsync(cursors, w.bin_cursor, sizeof(cursors), cudaMemcpyDeviceToHost, st));
  SB_CUDA(cudaStreamSynchronize(st));
  long long counts[kBins];
  for (int b = 0; b < kBins; b++) counts[b] = cursors[b];
  const CsrIn in{Apos, Acrd, nullptr, Bpos, Bcrd, nullptr};
  rc = caught("spgemm_symbolic", [&] {
    return launch_bins<float, false>(w, counts, m, kb, n, in, RowsOut{w.row_cnt, nullptr, nullptr, nullptr}, st);
  });
  if (rc != SB_OK) return rc;
  // keep the bin sizes in the workspace header for the numeric phase
  SB_CUDA(cudaMemcpyAsync(w.hdr, counts, sizeof(counts), cudaMemcpyHostToDevice, st));
  return row_pointers(w, m, Cpos, total_nnz_host, st);
}

int sb_spgemm_numeric(int dtype, int64_t m, int64_t kb, int64_t n, const int32_t* Apos,
                      const int32_t* Acrd, const void* Aval, const int32_t* Bpos,
                      const int32_t* Bcrd, const void* Bval, const int32_t* Cpos, int32_t* Ccrd,
                      void* Cval, void* ws, size_t ws_bytes, void* stream) {
  SB_CHECK_ARG(dtype >= SB_F32 && dtype <= SB_I64, "spgemm_numeric: unknown dtype");
  int rc = check_spgemm(m, kb, n, Apos, Bpos, ws, ws_bytes);
  if (rc != SB_OK) return rc;
  SB_CHECK_ARG(Cpos, "spgemm_numeric: Cpos is null");
  if (m == 0) return SB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const WsLayout w = ws_layout(ws, m, n);
  long long counts[kBins];
  SB_CUDA(cudaMemcpyAsync(counts, w.hdr, sizeof(counts), cudaMemcpyDeviceToHost, st));
  SB_CUDA(cudaStreamSynchronize(st));
  long long binned = 0;
  for (int b = 0; b < kBins; b++) {
    SB_CHECK_ARG(counts[b] >= 0 && counts[b] <= m, "spgemm_numeric: workspace does not hold the "
                 "bins of a symbolic call");
    binned += counts[b];
  }
  SB_CHECK_ARG(binned <= m, "spgemm_numeric: workspace does not hold the bins of a symbolic call");
  if (binned == 0) return SB_OK;
  SB_CHECK_ARG(Ccrd && Cval && Aval && Bval, "spgemm_numeric: null pointer");
  const CsrIn in{Apos, Acrd, Aval, Bpos, Bcrd, Bval};
  return caught("spgemm_numeric", [&] {
    return launch_bins_typed<true>(dtype, w, counts, m, kb, n, in, RowsOut{nullptr, Cpos, Ccrd, Cval}, st);
  });
}

int sb_spgemm_begin(int64_t m, int64_t kb, int64_t n, const int32_t* Apos, const int32_t* Acrd,
                    const int32_t* Bpos, int32_t* off, int64_t* counts_host, int64_t* products_host, void* ws,
                    size_t ws_bytes, void* stream) {
  int rc = check_spgemm(m, kb, n, Apos, Bpos, ws, ws_bytes);
  if (rc != SB_OK) return rc;
  SB_CHECK_ARG(off && counts_host && products_host, "spgemm_begin: null output");
  cudaStream_t st = (cudaStream_t)stream;
  const WsLayout w = ws_layout(ws, m, n);
  for (int b = 0; b < kBins; b++) counts_host[b] = 0;
  *products_host = 0;
  if (m == 0) return SB_OK;
  rc = bin_rows(w, m, Apos, Acrd, Bpos, st);
  if (rc != SB_OK) return rc;
  rc = exclusive_scan_i32((int)m, w.upper, off, w.block_sum, w.hdr + 8, st);
  if (rc != SB_OK) return rc;
  struct { long long hdr[32]; int cursors[16]; } h;   // header and cursors are neighbours
  static_assert(sizeof(long long) * 32 == 256, "the header takes one 256-byte unit of the workspace");
  SB_CUDA(cudaMemcpyAsync(&h, w.hdr, sizeof(h), cudaMemcpyDeviceToHost, st));
  SB_CUDA(cudaStreamSynchronize(st));
  for (int b = 0; b < kBins; b++) counts_host[b] = h.cursors[b];
  *products_host = h.hdr[8];
  return SB_OK;
}

int sb_spgemm_rows(int dtype, int64_t m, int64_t kb, int64_t n, const int32_t* Apos, const int32_t* Acrd,
                   const void* Aval, const int32_t* Bpos, const int32_t* Bcrd, const void* Bval, const int32_t* off,
                   const int64_t* counts_host, int32_t* tcrd, void* tval, int32_t* Cpos, int64_t* total_nnz_host,
                   void* ws, size_t ws_bytes, void* stream) {
  SB_CHECK_ARG(dtype >= SB_F32 && dtype <= SB_I64, "spgemm_rows: unknown dtype");
  int rc = check_spgemm(m, kb, n, Apos, Bpos, ws, ws_bytes);
  if (rc != SB_OK) return rc;
  SB_CHECK_ARG(off && counts_host && Cpos && total_nnz_host, "spgemm_rows: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const WsLayout w = ws_layout(ws, m, n);
  *total_nnz_host = 0;
  if (m == 0) {
    SB_CUDA(cudaMemsetAsync(Cpos, 0, 4, st));
    return SB_OK;
  }
  long long counts[kBins], binned = 0;
  for (int b = 0; b < kBins; b++) {
    counts[b] = counts_host[b];
    SB_CHECK_ARG(counts[b] >= 0 && counts[b] <= m, "spgemm_rows: counts are not those of sb_spgemm_begin");
    binned += counts[b];
  }
  SB_CHECK_ARG(binned <= m, "spgemm_rows: counts are not those of sb_spgemm_begin");
  SB_CHECK_ARG(binned == 0 || (tcrd && tval && Aval && Bval), "spgemm_rows: null pointer");
  const CsrIn in{Apos, Acrd, Aval, Bpos, Bcrd, Bval};
  rc = caught("spgemm_rows", [&] {
    return launch_bins_typed<true>(dtype, w, counts, m, kb, n, in, RowsOut{w.row_cnt, off, tcrd, tval}, st);
  });
  if (rc != SB_OK) return rc;
  return row_pointers(w, m, Cpos, total_nnz_host, st);
}

int sb_spgemm_finish(int dtype, int64_t m, int64_t nnz, const int32_t* off, const int32_t* tcrd, const void* tval,
                     const int32_t* Cpos, int32_t* Ccrd, void* Cval, void* stream) {
  SB_CHECK_ARG(dtype >= SB_F32 && dtype <= SB_I64, "spgemm_finish: unknown dtype");
  SB_CHECK_ARG(m >= 0 && m < INT32_MAX / 32 && nnz >= 0 && nnz <= INT32_MAX, "spgemm_finish: bad size");
  if (m == 0 || nnz == 0) return SB_OK;
  SB_CHECK_ARG(off && tcrd && tval && Cpos && Ccrd && Cval, "spgemm_finish: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t share = ceil_div(ceil_div(nnz, 4 * sm_count()), 256) * 256;
  const int tile = (int)std::min<int64_t>(kMoveTile, std::max<int64_t>(256 * kMoveAhead, share));
  const unsigned grid = (unsigned)ceil_div(nnz, tile);
  if (dtype == SB_F32 || dtype == SB_I32)
    spgemm_move_kernel<unsigned><<<grid, 256, 0, st>>>((int)m, (int)nnz, tile, off, Cpos, tcrd, (const unsigned*)tval,
                                                       Ccrd, (unsigned*)Cval);
  else
    spgemm_move_kernel<unsigned long long><<<grid, 256, 0, st>>>(
        (int)m, (int)nnz, tile, off, Cpos, tcrd, (const unsigned long long*)tval, Ccrd, (unsigned long long*)Cval);
  SB_LAUNCH_CHECK("spgemm_move_kernel");
  return SB_OK;
}

}  // extern "C"
