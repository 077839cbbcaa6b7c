// CSR SpMM, C = A * B straight from the CSR arrays.
#include "lf_spmm_group.cuh"

namespace lf {
namespace {

// ---------------------------------------------------------------------------------------------
// CSR SpMM (the kernel behind bench_naive, format_algos.py:1660-1755), balanced over entries
// instead of rows: every thread group takes `spg` consecutive stored entries, whatever rows they
// belong to, so a 100 000-entry row is shared by hundreds of groups and short rows are packed
// together.  A row that lies inside one group's range is written with a plain store; a row cut
// by a range boundary is accumulated with vector atomics after csr_prepare_kernel cleared it.
// ---------------------------------------------------------------------------------------------
// A row has to be cleared when it has no entry, or when a multiple of spg = 1 << spg_log lies inside
// it (two groups then add to it).  Both follow from its two row pointers, so a thread looks at one
// row, and the warp clears what its 32 rows need with coalesced (128-bit when VEC == 4) stores.
// A warp per row or group, its lane 0 looking for the row of each range start by bisection, took
// 152 us for 2^19 rows of 14 entries at 32 features; this takes 8.
template <int VEC>
__global__ void __launch_bounds__(256)
csr_prepare_kernel(const int64_t* __restrict__ indptr, int64_t row_begin, int64_t row_end, int spg_log,
                   float* __restrict__ C, int64_t ldc, int N) {
  let_dependents_launch();
  const int lane = threadIdx.x & 31;
  const int64_t rows = row_end - row_begin;
  const int64_t base = indptr[row_begin];
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i - lane < rows; i += step) {
    bool clear = false;
    if (i < rows) {
      const int64_t s = indptr[row_begin + i] - base, e = indptr[row_begin + i + 1] - base;
      clear = s == e || (s >> spg_log) != ((e - 1) >> spg_log);
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, clear); todo; todo &= todo - 1) {
      float* dst = C + (i - lane + __ffs(todo) - 1) * ldc;
      if (VEC == 4) {
        for (int f = lane * 4; f < N; f += 128) *reinterpret_cast<float4*>(dst + f) = make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
        for (int f = lane; f < N; f += 32) dst[f] = 0.f;
      }
    }
  }
}

template <int G, int V, int VEC>
__global__ void __launch_bounds__(kThreads, 3)
spmm_csr_kernel(const int64_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                const float* __restrict__ data, int64_t row_begin, int64_t row_end,
                const float* __restrict__ B, int ldb, float* __restrict__ C, int64_t ldc, int N, int spg) {
  constexpr int GPC = kThreads / G;
  constexpr int U = V == 1 ? 8 : (V == 2 ? 4 : 2);
  __shared__ int2 s_cv[kThreads];
  __shared__ int64_t s_bd[kThreads];
  const int g = threadIdx.x / G, lane = threadIdx.x % G;
  const int shift = (threadIdx.x & 31) / G * G;
  const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << shift);
  const int64_t base = indptr[row_begin];
  const int64_t total = indptr[row_end] - base;
  const int64_t s0 = ((int64_t)blockIdx.x * GPC + g) * (int64_t)spg;
  if (s0 >= total) return;
  const int64_t s1 = min(s0 + spg, total);
  int2* cv = s_cv + g * G;
  int64_t* bd = s_bd + g * G;

  // (G+1)-ary search, one probe per lane: the row that holds entry s0
  int64_t lo = row_begin, hi = row_end;   // indptr[lo] - base <= s0, answer in [lo, hi)
  while (hi - lo > 1) {
    const int64_t span = hi - lo;
    int64_t q = lo + ((int64_t)(lane + 1) * span) / (G + 1);
    if (q <= lo) q = lo + 1;
    const bool le = indptr[q] - base <= s0;
    const int cnt = __popc((__ballot_sync(gmask, le) & gmask) >> shift);   // probes are monotone
    const int64_t qlo = __shfl_sync(gmask, q, cnt > 0 ? cnt - 1 : 0, G);
    const int64_t qhi = __shfl_sync(gmask, q, cnt < G ? cnt : G - 1, G);
    if (cnt > 0) lo = qlo;
    if (cnt < G) hi = qhi;
  }
  int64_t cur = lo;
  const int64_t first_row = cur;
  const bool head_open = indptr[cur] - base < s0;

  // boundaries of the next G rows, refilled when used up
  int kb = 0;
  auto refill = [&]() {
    __syncwarp(gmask);
    const int64_t r = cur + 1 + lane;
    bd[lane] = indptr[r < row_end ? r : row_end] - base;
    __syncwarp(gmask);
    kb = 0;
  };
  refill();
  int64_t nb = bd[0];   // first entry of the next row

  const int f0 = blockIdx.y * (G * V * VEC) + lane * VEC;
  bool active[V];
  Chunk<VEC> acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) { active[v] = f0 + v * G * VEC < N; acc[v].zero(); }

  auto flush = [&](int64_t row, bool open) {
    float* dst = C + (row - row_begin) * ldc + f0;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (active[v]) {
        if (open) acc[v].red(dst + v * G * VEC); else acc[v].store_stream(dst + v * G * VEC);
      }
      acc[v].zero();
    }
  };

  const float* __restrict__ Bf = B + f0;
  wait_for_prior_grid();   // csr_prepare_kernel has cleared the rows that receive atomics
  for (int64_t s = s0; s < s1; s += G) {
    const int64_t idx = s + lane;
    const bool in = idx < s1;
    const int my_col = in ? __ldcs(indices + base + idx) : 0;
    const float my_val = in ? (data ? __ldcs(data + base + idx) : 1.f) : 0.f;
    __syncwarp(gmask);
    cv[lane] = make_int2(my_col, __float_as_int(my_val));
    __syncwarp(gmask);
    const int nstrip = (int)min((int64_t)G, s1 - s);
    for (int t = 0; t < nstrip; t += U) {
      float val[U];
      Chunk<VEC> b[U][V];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int2 p = cv[t + u];
        val[u] = __int_as_float(p.y);
        const float* src = Bf + (int64_t)p.x * ldb;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          if (val[u] != 0.f && active[v]) b[u][v].load(src + v * G * VEC); else b[u][v].zero();
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t pos = s + t + u;
        if (pos < s1) {
          while (pos == nb) {   // the current row ended here (and empty rows may follow)
            flush(cur, cur == first_row && head_open);
            ++cur;
            if (++kb == G) refill();
            nb = bd[kb];
          }
#pragma unroll
          for (int v = 0; v < V; ++v) acc[v].fma(val[u], b[u][v]);
        }
      }
    }
  }
  flush(cur, (cur == first_row && head_open) || s1 < nb);
}

// The CSR product with the gathers staged through the group ring (lf_spmm_group.cuh): a group takes
// spg consecutive entries and flushes by the rules of the register kernel above.  2^18 power-law rows, 3.7 M
// entries, register kernel / ring: 16 features 164 / 50 us, 64 features 225 / 93 us, 128 features 235 / 137 us.
//
// Two levels (2): chains as long as the register kernel's ranges, which add up into the row's sum, so that a
// range can hold several of them; a row inside one chain has the register kernel's sum, bit for bit.  The second
// sum costs registers: at 64 a thread and four blocks per SM 2^19 power-law rows at 32 features take 139 us, at
// 74 and three blocks 124, with one level 130 (and 114 with ranges of one chain of 128, 1.3 times the error);
// 2^17 rows at 384 features one level 227, two 204.  One level where a range's start is cheap beside its rows: up to
// 16 features (2^18 rows 48 / 53) and shifted rows (47 features 146 / 150).
template <int G, bool SH> constexpr int kCsrSums = SH || G == 4 ? 1 : 2;

template <int G, int CH, bool SH>
__global__ void __launch_bounds__(kThreads, CH == 1 && kCsrSums<G, SH> == 1 ? 4 : 3)
spmm_csr_ring_kernel(const int64_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                     const float* __restrict__ data, int64_t row_begin, int64_t row_end,
                     const float* __restrict__ B, int ldb, float* __restrict__ C, int64_t ldc, int N, int spg,
                     int chain) {
  extern __shared__ __align__(16) unsigned char group_bytes[];
  constexpr int R = 32 / G, kFeatures = kGroupFeatures<G, CH, 4, SH>;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane / G, gl = lane % G;
  const int64_t base = indptr[row_begin];
  const int64_t total = indptr[row_end] - base;
  const int64_t first = ((int64_t)blockIdx.x * (kThreads / 32) + w) * R;   // the warp's first group
  if (first * spg >= total) return;
  const int64_t s0 = min((first + g) * spg, total), s1 = min(s0 + spg, total);
  CsrRowIds<G> ids;
  ids.init(indptr + row_begin, (int)(row_end - row_begin), base, s0, s1, g, gl);
  const int f0 = blockIdx.y * kFeatures;
  walk_group_ring<G, CH, 4, SH, 1, kCsrSums<G, SH>, 0>(ids, false, indices + base + s0, data ? data + base + s0 : nullptr,
                                                    B + f0, ldb, C + f0, ldc, min(N - f0, kFeatures), g, gl,
                                                    group_bytes + w * GroupSmem<G, CH, SH>::kBytes, chain);
}

}  // namespace
}  // namespace lf

using namespace lf;

extern "C" {

int lf_spmm_csr_f32(const int64_t* indptr, const int32_t* indices, const float* data, int64_t row_begin,
                    int64_t row_end, int64_t nnz, const float* B, int64_t ldb, float* C, int64_t ldc, int32_t N,
                    void* stream) {
  LF_REQUIRE(N >= 1 && ldb >= N && ldc >= N && ldb < (1ll << 31), "bad arguments");
  LF_REQUIRE(0 <= row_begin && row_begin <= row_end, "bad row range");
  if (row_begin == row_end) return LF_OK;
  LF_REQUIRE(indptr && B && C, "null pointer argument");
  cudaStream_t st = (cudaStream_t)stream;
  if (nnz < 0) {   // the launch shape depends on the number of entries: read it back
    int64_t ends[2] = {0, 0};
    LF_CUDA_CHECK(cudaMemcpyAsync(&ends[0], indptr + row_begin, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    LF_CUDA_CHECK(cudaMemcpyAsync(&ends[1], indptr + row_end, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    LF_CUDA_CHECK(cudaStreamSynchronize(st));
    nnz = ends[1] - ends[0];
  }
  LF_REQUIRE(nnz == 0 || indices, "indices missing");
  const FeatCfg cfg = pick_cfg(B, ldb, C, ldc, N);
  // the ring form multiplies row numbers by 32-bit pitches in bytes and keeps row numbers in 32 bits
  const bool ring = gather_ring() > 0 && ldb < (1ll << 30) && ldc < (1ll << 30) && row_end - row_begin < (1ll << 31) - 64;
  GroupCfg group = cfg.VEC == 4 ? pick_group(N, 4) : pick_group_shifted(N);
  // one walk of full warps for up to 256 features (2^18 power-law rows at 200: 244 us, two walks of 128
  // features 278); beyond that pieces of 128 (uniform rows, 300 features: two walks of 256 1543 us, three of
  // 128 1239; 2^17 power-law rows at 384 217 / 200)
  if (cfg.VEC == 4 && N > 128 && N <= 256) group = {32, 2, 1};
  const int gpc = kThreads / (ring ? group.G : cfg.G);
  // Entries per group.  Every range boundary cuts a row (cleared before, added to twice) and costs a
  // search, so long ranges win as soon as the grid fills the chip about twice; measured on
  // 3.7 M entries, 16 features: 32 / 64 / 128 / 256 entries 74.8 / 68.1 / 65.4 / 63.6 us, on 1 M entries, 128
  // features 51.3 / 45.1 / 45.3 / 51.4 us.  Below that, more blocks win until a range is one strip.
  // But a row's error grows with the chain of additions it is summed in: a chain is no longer than the range
  // that fills the chip eight times at cfg.G lanes per row.  Where the sum has two levels (kCsrSums), a range is
  // several chains.
  int chain = 256;
  while (chain > 32 && ceil_div64(nnz, (int64_t)chain * (kThreads / cfg.G)) < (int64_t)sm_count() * 3 * 8) chain >>= 1;
  int spg = chain;
  if (ring) {
    const int longest = cfg.VEC == 4 && group.G > 4 ? 256 : chain;
    for (spg = 256; spg > 32; spg >>= 1)
      if (spg <= longest && ceil_div64(nnz, (int64_t)spg * gpc) >= (int64_t)sm_count() * 3 * 2) break;
    if (chain > spg) chain = spg;
  }
  const int64_t rows = row_end - row_begin;
  {
    const int spg_log = 31 - __builtin_clz((unsigned)spg);
    const int64_t want = ceil_div64(rows, 256);
    const unsigned pgrid = (unsigned)(want > (int64_t)sm_count() * 32 ? sm_count() * 32 : want);
    if (cfg.VEC == 4) csr_prepare_kernel<4><<<pgrid, 256, 0, st>>>(indptr, row_begin, row_end, spg_log, C, ldc, N);
    else csr_prepare_kernel<1><<<pgrid, 256, 0, st>>>(indptr, row_begin, row_end, spg_log, C, ldc, N);
    LF_CUDA_CHECK(cudaGetLastError());
  }
  if (nnz == 0) return LF_OK;
  const int64_t blocks = ceil_div64(nnz, (int64_t)spg * gpc);
  LF_REQUIRE(blocks < (1ll << 31), "too many thread blocks");
  if (ring) {
    const dim3 rgrid((unsigned)blocks, (unsigned)group.passes);
#define LF_RING(G_, CH_, SH_)                                                                                   \
  do {                                                                                                          \
    constexpr auto kern = spmm_csr_ring_kernel<G_, CH_, SH_>;                                                   \
    constexpr int smem = kThreads / 32 * GroupSmem<G_, CH_, SH_>::kBytes;                                       \
    LF_CUDA_CHECK(allow_smem<kern>(smem));                                                                      \
    LF_CUDA_CHECK(launch_dep_smem(kern, rgrid, kThreads, smem, st, true, indptr, indices, data, row_begin, row_end, \
                                  B, (int)ldb, C, ldc, N, spg, chain));                                         \
    return LF_OK;                                                                                               \
  } while (0)
    if (cfg.VEC == 4) {
      if (group.G == 4) LF_RING(4, 1, false);
      else if (group.G == 8 && group.CH == 1) LF_RING(8, 1, false);
      else if (group.G == 8) LF_RING(8, 2, false);
      else if (group.G == 16) LF_RING(16, 2, false);
      else LF_RING(32, 2, false);
    } else {
      if (group.G == 4) LF_RING(4, 1, true);
      else if (group.G == 8) LF_RING(8, 1, true);
      else if (group.G == 16) LF_RING(16, 1, true);
      else LF_RING(32, 1, true);
    }
#undef LF_RING
  }
  dim3 grid((unsigned)blocks, (unsigned)((N + cfg.pass - 1) / cfg.pass));
#define LF_LAUNCH(G_, V_, VEC_)                                                                              \
  LF_CUDA_CHECK(launch_dep(spmm_csr_kernel<G_, V_, VEC_>, grid, kThreads, st, true, indptr, indices, data, row_begin, \
                           row_end, B, (int)ldb, C, ldc, N, spg))
  if (cfg.VEC == 4) {
    if (cfg.G == 8) LF_LAUNCH(8, 1, 4);
    else if (cfg.G == 16) LF_LAUNCH(16, 1, 4);
    else if (cfg.V == 1) LF_LAUNCH(32, 1, 4);
    else if (cfg.V == 2) LF_LAUNCH(32, 2, 4);
    else LF_LAUNCH(32, 4, 4);
  } else {
    if (cfg.V == 1) LF_LAUNCH(32, 1, 1);
    else if (cfg.V == 2) LF_LAUNCH(32, 2, 1);
    else LF_LAUNCH(32, 4, 1);
  }
#undef LF_LAUNCH
  return LF_OK;
}

}  // extern "C"
