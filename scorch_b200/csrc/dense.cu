// Dense transform of the GCN layers: C = A W in fp32 accuracy on the 5th-generation tensor cores.
// A is tall (one row per node), W small.
//
// Every operand value is split into three bf16 parts (x = h + m + l exactly but for the last bit) and
// six products are summed: h h in one accumulator, h m + m h + m m + h l + l h (2^-8 of it) in another,
// the two added in fp32 at the end.  Against float64 the result is as close as cuBLAS's fp32 FMA
// kernel's.  The tensor core's additions truncate, so what counts is how often the main sum is added
// to: two TF32 parts (K 8 instead of 16, all products in one accumulator: 96 additions for K = 256)
// were 6 times further off than cuBLAS, this form adds 16 times (2.3e-7 of the result's norm, cuBLAS
// 2.9e-7; beyond K = 256 the order turns round, the caller keeps to that).
// Bound: the tensor cores for wide outputs (2 M x 256 x 256: 1.57 PFLOP of bf16), DRAM on A and C for
// narrow ones.  2 M x 256 x 256: 4.57 ms with cuBLAS, 1.88 ms here; 2 M x 256 x 64: 1.28 and 0.74 ms.
//
// One persistent CTA per SM takes tiles of 128 rows x NMAX columns (the column panels of a row tile run
// beside one another, so A comes from DRAM once):
//   * a small kernel splits W once per call, into the layout of the shared-memory stages;
//   * eight producer warps copy 32-column chunks of A to shared memory by cp.async, kRaw chunks ahead
//     (each thread the values it will split itself, so nothing is synchronised), split them and store
//     the parts to a ring of STAGES stages in the tensor core's K-major layout without swizzle; one
//     thread has the chunk's parts of W brought in by one cp.async.bulk;
//   * one thread issues the 12 tcgen05.mma (M 128, N up to 128, K 16) of a chunk into one of two pairs
//     of accumulators in tensor memory;
//   * four warps write the other pair to C, so that the stores overlap the next tile's products.
// Every wait is bounded; one that runs out sets a status word and ends the CTA's pipeline.
// The CTA's tiles that the pipeline left - behind a wait that ran out, or with a value too large for the
// split (2^127 and above, Inf, NaN) in the rows of A, or all of them with one in W - it does with fp32
// FMAs at its end, so C is complete whatever happened; and so the tiles with a result that is not finite
// (the parts' products overflow to opposite infinities) or below 2^-100 and not 0 (the parts are denormal
// and short of bits: 3e-5 off at 1e-36).
#include <algorithm>

#include "tensor_core.cuh"

namespace sb {

constexpr int kGemmRows = 128, kGemmK = 32;
constexpr int kGemmProducers = 256, kGemmThreads = kGemmProducers + 128 + 32;
constexpr int kRaw = 4;                       // chunks of A on their way
constexpr int kRedoWords = 512;               // tiles of a CTA that are noted one by one (14,170 at most on 148 SMs)
constexpr unsigned kSplitMax = 0x7f000000u;   // bits of 2^127: values from here on, Inf and NaN are not split
constexpr unsigned kResultMin = 0x0d800000u;  // bits of 2^-100: results from here to the largest float are kept

__device__ int g_gemm_status = 0;  // 0 ok; 1 a wait ran out

struct GemmArgs {
  long long m;
  int n, k;
  const float* A;
  long long lda;
  const float* W;
  long long ldw;
  const int* w_flag;   // a value of W cannot be split
  const uint4* parts;  // W split: [panel][chunk][part][NMAX * 4] rows of core matrices
  float* C;
  long long ldc;
  int tiles, chunks;   // row tiles x column panels; 32-column chunks of K
  int panels;
  int stop;            // self-test: the issuing thread gives up at this chunk of every CTA (-1: never)
};

// Two values as three packed pairs of bf16 parts.
__device__ __forceinline__ void split3(float x, float y, unsigned (&part)[3]) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(part[i]) : "f"(y), "f"(x));
    x -= __uint_as_float(part[i] << 16);
    y -= __uint_as_float(part[i] & 0xffff0000u);
  }
}

// Eight values along K as row `at` of the three parts' core matrices; `top`: largest magnitude bits so far.
template <typename P>
__device__ __forceinline__ void put_parts(P& parts, int at, const float (&x)[8], unsigned& top) {
  uint4 q[3];
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    unsigned part[3];
    split3(x[j], x[j + 1], part);
#pragma unroll
    for (int i = 0; i < 3; i++) (j == 0 ? q[i].x : j == 2 ? q[i].y : j == 4 ? q[i].z : q[i].w) = part[i];
  }
#pragma unroll
  for (int j = 0; j < 8; j++) top = max(top, __float_as_uint(x[j]) & 0x7fffffffu);
#pragma unroll
  for (int i = 0; i < 3; i++) parts[i][at] = q[i];
}

// W split: one thread per (column, 8 rows); flag = 1 where a value cannot be split (all tiles are then
// done with fp32 FMAs).
template <int NMAX>
__global__ void __launch_bounds__(256)
gemm_split_w_kernel(int n, int k, int chunks, int panels, const float* __restrict__ W, long long ldw,
                    uint4* __restrict__ parts, int* __restrict__ flag) {
  const int t = blockIdx.x * 256 + threadIdx.x;
  const int c = t % NMAX, core = (t / NMAX) % 4, chunk = t / (4 * NMAX) % chunks, panel = t / (4 * NMAX) / chunks;
  if (panel >= panels) return;
  const int col = panel * NMAX + c, k0 = chunk * kGemmK + core * 8;
  float x[8];
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = (col < n && k0 + j < k) ? __ldg(W + (long long)(k0 + j) * ldw + col) : 0.f;
  struct Out {
    uint4* p;
    __device__ __forceinline__ uint4* operator[](int i) { return p + i * (NMAX * kGemmK / 8); }
  } out{parts + ((long long)panel * chunks + chunk) * (3 * NMAX * kGemmK / 8)};
  unsigned top = 0;
  put_parts(out, (c >> 3) * 32 + core * 8 + (c & 7), x, top);
  if (top >= kSplitMax) atomicOr(flag, 1);
}

__device__ __forceinline__ void umma_ss_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// Instruction descriptor of kind::f16 with bf16 operands (formats 1 in bits 7-9 and 10-12), fp32
// accumulation (bits 4-5 = 1), both operands K-major.
__device__ __forceinline__ uint32_t umma_idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

template <int NMAX, int STAGES>
struct GemmSmem {
  uint4 a[STAGES][3][kGemmRows * kGemmK / 8];   // 16-byte rows of core matrices: 8 bf16 along K
  uint4 w[STAGES][3][NMAX * kGemmK / 8];
  float4 raw[kRaw][8][kGemmProducers / 2];
  unsigned long long full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
  uint32_t tmem;
  // the tile (its number mod 8) holds a value the split cannot take; the producers are at most
  // 2 + STAGES tiles ahead of the epilogue, so a place is free again before it is used again
  int odd[8];
  int done;                   // tiles the epilogue has finished ...
  unsigned redo[kRedoWords];  // ... and those among them that are to be done again, a bit each
};

// One tile by fp32 FMAs, in the order of K: 256 threads, 4 rows x NMAX / 16 columns each at a time,
// operands through L1 (2 M x 256 x 256: 18.3 ms against cuBLAS's 4.6; one thread per row, which the epilogue
// used to fall back on, took 474).
template <int NMAX>
__device__ __forceinline__ void gemm_redo_tile(const GemmArgs& g, long long row0, int n0) {
  constexpr int RT = 4, CT = NMAX / 16;
  if (threadIdx.x >= 256) return;
  const int cols = min(NMAX, g.n - n0), cl = threadIdx.x & 15, rl = threadIdx.x >> 4;
#pragma unroll 1
  for (int r0 = rl; r0 < kGemmRows; r0 += 16 * RT) {
    const float* a[RT];
#pragma unroll
    for (int i = 0; i < RT; i++) a[i] = g.A + min(row0 + r0 + 16 * i, g.m - 1) * g.lda;
    float acc[RT][CT];
#pragma unroll
    for (int i = 0; i < RT; i++) {
#pragma unroll
      for (int j = 0; j < CT; j++) acc[i][j] = 0.f;
    }
#pragma unroll 1
    for (int k = 0; k < g.k; k += 4) {
      float4 x[RT];
#pragma unroll
      for (int i = 0; i < RT; i++) x[i] = ldg4(a[i] + k);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float* w = g.W + (k + q) * g.ldw + n0 + cl;
#pragma unroll
        for (int j = 0; j < CT; j++) {
          const float y = cl + 16 * j < cols ? __ldg(w + 16 * j) : 0.f;
#pragma unroll
          for (int i = 0; i < RT; i++)
            acc[i][j] = fmaf(q == 0 ? x[i].x : q == 1 ? x[i].y : q == 2 ? x[i].z : x[i].w, y, acc[i][j]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < RT; i++) {
      const long long row = row0 + r0 + 16 * i;
#pragma unroll
      for (int j = 0; j < CT; j++)
        if (row < g.m && cl + 16 * j < cols) g.C[row * g.ldc + n0 + cl + 16 * j] = acc[i][j];
    }
  }
}

template <int NMAX, int STAGES>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_f32_kernel(const __grid_constant__ GemmArgs g) {
  using Smem = GemmSmem<NMAX, STAGES>;
  constexpr uint32_t TMEM_COLS = 4 * NMAX;       // two pairs of accumulators
  constexpr uint32_t GROUP = 8 * kGemmK * 2;     // bytes of an 8-row group: 4 core matrices of 128 bytes
  extern __shared__ __align__(128) unsigned char gemm_smem[];
  Smem& sm = *reinterpret_cast<Smem*>(gemm_smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(smem_u32(&sm.full[s]), kGemmProducers / 2);
      mbar_init(smem_u32(&sm.empty[s]), 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(smem_u32(&sm.acc_full[i]), 1);
      mbar_init(smem_u32(&sm.acc_empty[i]), 128);
    }
    for (int i = 0; i < 8; i++) sm.odd[i] = 0;
    sm.done = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = threadIdx.x; i < kRedoWords; i += kGemmThreads) sm.redo[i] = 0;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&sm.tmem)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  asm volatile("griddepcontrol.wait;" ::: "memory");   // the parts of W
  const uint32_t tmem = sm.tmem;
  const int my_tiles = ((int)blockIdx.x < g.tiles) ? (g.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  // (a value of W that cannot be split: no tile takes the tensor cores)
  const int run_tiles = *g.w_flag ? 0 : my_tiles, steps = run_tiles * g.chunks;
  auto tile_of = [&](int i) { return (int)blockIdx.x + i * (int)gridDim.x; };
  auto give_up = [&]() { atomicExch(&g_gemm_status, 1); };

  if (warp < 8) {
    // ---- producers: two groups of four warps, every other chunk each ----
    // (the chain wait - read - split - store - fence of a chunk is latency: two chains side by side)
    const int grp = warp >> 2, tid = threadIdx.x & 127, r8 = lane & 7, core = lane >> 3;
    struct Place {          // a chunk: its number, its tile (among this CTA's) and columns
      int step, chunk, tile, panel;
      long long row0;
    };
    auto set_tile = [&](Place& p) {
      const int work = tile_of(p.tile), rt = work / g.panels;
      p.panel = work - rt * g.panels;
      p.row0 = (long long)rt * kGemmRows + (warp & 3) * 8 + r8;
    };
    auto advance = [&](Place& p, int by) {
      p.step += by;
      p.chunk += by;
      if (p.chunk < g.chunks) return;
      while (p.chunk >= g.chunks) { p.chunk -= g.chunks; p.tile++; }
      set_tile(p);
    };
    Place at{0, 0, 0, 0, 0};
    set_tile(at);
    advance(at, grp);
    Place ahead = at;
    // the next chunk of A: this thread's 8 consecutive columns of four rows
    auto fetch = [&]() {
      if (ahead.step < steps) {
        const int k0 = ahead.chunk * kGemmK + core * 8;
        float4* dst = &sm.raw[ahead.step % kRaw][0][tid];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const long long row = ahead.row0 + i * 32;
          const float* src = g.A + row * g.lda + k0;
#pragma unroll
          for (int j = 0; j < 2; j++) {
            const bool in = row < g.m && k0 + j * 4 < g.k;
            // (0 source bytes: the 16 bytes are filled with zeros)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                         ::"r"(smem_u32(dst + (i * 2 + j) * 128)), "l"(in ? src + j * 4 : g.A), "r"(in ? 16 : 0)
                         : "memory");
          }
        }
        advance(ahead, 2);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch();
    fetch();
    int stage = grp % STAGES, use = grp / STAGES;
    while (at.step < steps) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      if (use > 0 && !mbar_wait(smem_u32(&sm.empty[stage]), (uint32_t)((use - 1) & 1))) { give_up(); break; }
      const uint32_t full = smem_u32(&sm.full[stage]);
      if (tid == 0) {
        const uint32_t bytes = sizeof(sm.w[0]);
        const uint4* src = g.parts + ((long long)at.panel * g.chunks + at.chunk) * (long long)(sizeof(sm.w[0]) / sizeof(uint4));
        asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(full), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(smem_u32(sm.w[stage])), "l"(src), "r"(bytes), "r"(full) : "memory");
      }
      unsigned top = 0;
      const float4* raw = &sm.raw[at.step % kRaw][0][tid];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const float4 x = raw[(i * 2) * 128], y = raw[(i * 2 + 1) * 128];
        const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        put_parts(sm.a[stage], (i * 4 + (warp & 3)) * 32 + core * 8 + r8, v, top);
      }
      if (top >= kSplitMax) *(volatile int*)&sm.odd[at.tile & 7] = 1;
      async_proxy_fence();
      mbar_arrive(full);
      fetch();                                   // (into the place just read, by the same thread)
      advance(at, 2);
      stage += 2;
      if (stage >= STAGES) { stage -= STAGES; use++; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == 12) {
    // ---- tensor-core issue: one thread ----
    if (lane == 0) {
      int i = 0, c = 0, stage = 0, use = 0;
      uint32_t acc = 0, idesc = 0;
      for (int step = 0; step < steps; step++) {
        if (step == g.stop) { give_up(); break; }
        if (c == 0) {
          acc = tmem + (uint32_t)((i & 1) * 2 * NMAX);
          const int cols = min(NMAX, g.n - (tile_of(i) % g.panels) * NMAX);
          idesc = umma_idesc_bf16(kGemmRows, (cols + 15) / 16 * 16);
          if (i >= 2 && !mbar_wait(smem_u32(&sm.acc_empty[i & 1]), (uint32_t)(((i >> 1) - 1) & 1))) { give_up(); break; }
        }
        if (!mbar_wait(smem_u32(&sm.full[stage]), (uint32_t)(use & 1))) { give_up(); break; }
        tc_fence_after();
        uint64_t da[3], dw[3];
#pragma unroll
        for (int p = 0; p < 3; p++) {
          da[p] = umma_desc(smem_u32(sm.a[stage][p]), 128, GROUP);
          dw[p] = umma_desc(smem_u32(sm.w[stage][p]), 128, GROUP);
        }
#pragma unroll
        for (int ks = 0; ks < kGemmK / 16; ks++) {
          const uint32_t later = (c | ks) != 0 ? 1u : 0u;
          umma_ss_bf16(acc + NMAX, da[2] + ks * 16, dw[0] + ks * 16, idesc, later);
          umma_ss_bf16(acc, da[0] + ks * 16, dw[0] + ks * 16, idesc, later);
          umma_ss_bf16(acc + NMAX, da[0] + ks * 16, dw[2] + ks * 16, idesc, 1u);
          umma_ss_bf16(acc + NMAX, da[1] + ks * 16, dw[1] + ks * 16, idesc, 1u);
          umma_ss_bf16(acc + NMAX, da[1] + ks * 16, dw[0] + ks * 16, idesc, 1u);
          umma_ss_bf16(acc + NMAX, da[0] + ks * 16, dw[1] + ks * 16, idesc, 1u);
        }
        umma_commit(smem_u32(&sm.empty[stage]));
        if (++c == g.chunks) {
          umma_commit(smem_u32(&sm.acc_full[i & 1]));
          c = 0;
          i++;
        }
        if (++stage == STAGES) { stage = 0; use++; }
      }
    }
  } else {
    // ---- epilogue: warps 8..11, a row per thread ----
    const int r = (warp & 3) * 32 + lane;
    const uint32_t t_row = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    for (int i = 0; i < run_tiles; i++) {
      const int work = tile_of(i), n0 = (work % g.panels) * NMAX, cols = min(NMAX, g.n - n0);
      const long long row = (long long)(work / g.panels) * kGemmRows + r;
      // (the four warps agree on the outcome: they meet at a barrier below)
      uint32_t ok = mbar_wait(smem_u32(&sm.acc_full[i & 1]), (uint32_t)((i >> 1) & 1));
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %0, 0;\n\t"
                   "barrier.cta.red.and.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "+r"(ok)::"memory");
      if (!ok) { give_up(); break; }
      tc_fence_after();
      const bool odd = *(volatile int*)&sm.odd[i & 7] != 0;
      float* crow = g.C + row * g.ldc + n0;
      float finite = 0.f;          // (NaN once a result is not)
      unsigned least = ~0u;        // 2 x (bits of the smallest magnitude but 0) - 2
      for (int c0 = 0; c0 < cols; c0 += 32) {
        float v[32], small[32];
        tmem_ld32(t_row + (uint32_t)((i & 1) * 2 * NMAX + c0), v);
        tmem_ld32(t_row + (uint32_t)((i & 1) * 2 * NMAX + NMAX + c0), small);
        // (columns from `cols` on hold what an earlier kernel left there)
        auto look = [&](float x) {
          finite = fmaf(x, 0.f, finite);
          least = min(least, 2u * __float_as_uint(x) - 2u);
        };
#pragma unroll
        for (int j = 0; j < 32; j++) v[j] += small[j];
        if (c0 + 32 <= cols) {
#pragma unroll
          for (int j = 0; j < 32; j++) look(v[j]);
          if (row < g.m && !odd) {
#pragma unroll
            for (int j = 0; j < 32; j += 8)
              asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(crow + c0 + j), "f"(v[j]),
                           "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3]), "f"(v[j + 4]), "f"(v[j + 5]), "f"(v[j + 6]),
                           "f"(v[j + 7])
                           : "memory");
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; j++) {
            if (c0 + j >= cols) continue;
            look(v[j]);
            if (row < g.m && !odd) crow[c0 + j] = v[j];
          }
        }
      }
      tc_fence_before();
      asm volatile("barrier.cta.sync 1, 128;" ::: "memory");   // all four warps have read `odd`
      if (odd || finite != 0.f || least < 2u * kResultMin - 2u)
        atomicOr(&sm.redo[min(i >> 5, kRedoWords - 1)], 1u << (i & 31));
      if (r == 0) {
        if (odd) *(volatile int*)&sm.odd[i & 7] = 0;
        sm.done = i + 1;
      }
      mbar_arrive(smem_u32(&sm.acc_empty[i & 1]));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  // What the pipeline left.  (Behind a wait that ran out nothing of it is in flight any more: the last
  // copies and products were issued before that wait, a second ago.)  Tiles from the last word on share
  // its bits: some are then done a second time.
  for (int i = 0; i < my_tiles; i++) {
    if (i < sm.done && !(sm.redo[min(i >> 5, kRedoWords - 1)] >> (i & 31) & 1)) continue;
    const int work = tile_of(i);
    gemm_redo_tile<NMAX>(g, (long long)(work / g.panels) * kGemmRows, (work % g.panels) * NMAX);
  }
}

template <int NMAX, int STAGES>
static int launch_gemm(GemmArgs g, void* ws, cudaStream_t st) {
  auto kernel = gemm_f32_kernel<NMAX, STAGES>;
  const size_t smem = sizeof(GemmSmem<NMAX, STAGES>);
  SB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  g.panels = (int)ceil_div(g.n, NMAX);
  g.tiles *= g.panels;
  int* flag = static_cast<int*>(ws);
  uint4* parts = reinterpret_cast<uint4*>(static_cast<char*>(ws) + 256);
  g.w_flag = flag;
  g.parts = parts;
  SB_CUDA(cudaMemsetAsync(flag, 0, 4, st));
  const int64_t threads = (int64_t)g.panels * g.chunks * 4 * NMAX;
  gemm_split_w_kernel<NMAX><<<(unsigned)ceil_div(threads, 256), 256, 0, st>>>(g.n, g.k, g.chunks, g.panels, g.W, g.ldw,
                                                                             parts, flag);
  SB_LAUNCH_CHECK("gemm_split_w_kernel");
  SB_CUDA(launch_early(kernel, dim3((unsigned)std::min(g.tiles, sm_count())), kGemmThreads, smem, st, g));
  return SB_OK;
}

}  // namespace sb

using namespace sb;

extern "C" {

// the flag, then 3 bf16 parts of W with columns padded to the panel width and rows to the chunk
size_t sb_dense_matmul_workspace_bytes(int64_t n, int64_t k) {
  if (n <= 0 || k <= 0) return 256;
  const int64_t panel = n <= 64 ? 64 : 128;
  return 256 + (size_t)(ceil_div(n, panel) * panel) * (size_t)(ceil_div(k, kGemmK) * kGemmK) * 6;
}

static int dense_matmul(int64_t m, int64_t n, int64_t k, const float* A, int64_t lda, const float* W, int64_t ldw,
                        float* C, int64_t ldc, void* ws, size_t ws_bytes, int stop, void* stream) {
  SB_CHECK_ARG(m >= 0 && n >= 0 && k >= 0 && n < INT32_MAX / 2 && k < INT32_MAX / 2 && m < INT32_MAX &&
               ceil_div(m, 128) * ceil_div(n, 64) < INT32_MAX / 1024, "dense_matmul: bad size");
  SB_CHECK_ARG(lda >= k && ldw >= n && ldc >= n, "dense_matmul: leading dimension smaller than the row");
  cudaStream_t st = (cudaStream_t)stream;
  if (m == 0 || n == 0) return SB_OK;
  SB_CHECK_ARG(C && (k == 0 || (A && W)), "dense_matmul: null pointer");
  if (k == 0 || k > 32768 || k % 4 || lda % 4 || !aligned16(A) || ldc % 8 || (reinterpret_cast<uintptr_t>(C) & 31))
    return fail(SB_ERR_UNSUPPORTED, "dense_matmul: A needs 16-byte aligned rows, C 32-byte aligned rows");
  SB_CHECK_ARG(ws && aligned16(ws), "dense_matmul: workspace is null or misaligned");
  if (ws_bytes < sb_dense_matmul_workspace_bytes(n, k))
    return fail(SB_ERR_WORKSPACE, "dense_matmul: workspace has %zu bytes, needs %zu", ws_bytes,
                sb_dense_matmul_workspace_bytes(n, k));
  GemmArgs g;
  g.m = m; g.n = (int)n; g.k = (int)k; g.A = A; g.lda = lda; g.W = W; g.ldw = ldw; g.C = C; g.ldc = ldc;
  g.tiles = (int)ceil_div(m, kGemmRows);
  g.stop = stop;
  g.chunks = (int)ceil_div(k, kGemmK);
  if (n <= 64) return launch_gemm<64, 4>(g, ws, st);
  return launch_gemm<128, 3>(g, ws, st);
}

int sb_dense_matmul_f32(int64_t m, int64_t n, int64_t k, const float* A, int64_t lda, const float* W, int64_t ldw,
                        float* C, int64_t ldc, void* ws, size_t ws_bytes, void* stream) {
  return dense_matmul(m, n, k, A, lda, W, ldw, C, ldc, ws, ws_bytes, -1, stream);
}

int sb_dense_matmul_probe(int64_t m, int64_t n, int64_t k, const float* A, int64_t lda, const float* W, int64_t ldw,
                          float* C, int64_t ldc, void* ws, size_t ws_bytes, int stop, int* status_host, void* stream) {
  SB_CHECK_ARG(status_host && stop >= 0, "dense_matmul_probe: null status or negative chunk");
  const int before = sb_dense_matmul_status();
  const int rc = dense_matmul(m, n, k, A, lda, W, ldw, C, ldc, ws, ws_bytes, stop, stream);
  if (rc != SB_OK) return rc;
  SB_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
  *status_host = sb_dense_matmul_status();
  // (what the probe has set on purpose is no finding of a later reader)
  SB_CUDA(cudaMemcpyToSymbol(g_gemm_status, &before, sizeof(int)));
  return SB_OK;
}

int sb_dense_matmul_status(void) {
  int v = -1;
  if (cudaMemcpyFromSymbol(&v, g_gemm_status, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

}  // extern "C"
