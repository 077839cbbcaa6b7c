// Device helpers and launch plumbing shared by the composed-format product (lf_spmm_hyb.cu) and
// the CSR product (lf_spmm_csr.cu): register images of gathered rows of B, asynchronous copies into
// shared memory, programmatic dependent launches and the choice of lanes per row.
#pragma once

#include <stdlib.h>

#include <type_traits>

#include "lf_common.cuh"

namespace lf {

constexpr int kThreads = 256;

// Destinations of a broadcasting launch: full-size C matrices (row 0 first), one per GPU of the
// group, addressed through peer mappings; the shard's rows are written into every one of them.
struct DestList {
  float* p[LF_MAX_DESTS];
  int32_t n;
  int32_t pad_;
};

__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// Programmatic dependent launch: the product kernel is launched while the launch that clears
// rows is still running; everything up to this point (bucket look-up, first loads) overlaps with
// it, and nothing is written to C before the clearing launch has completed and flushed.  Without
// a programmatic dependency the instruction returns at once.
__device__ __forceinline__ void wait_for_prior_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <int VEC> struct Chunk;
template <> struct Chunk<4> {
  float4 v;
  __device__ __forceinline__ void zero() { v = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void load(const float* p) { v = __ldg(reinterpret_cast<const float4*>(p)); }
  __device__ __forceinline__ void store_stream(float* p) const { __stcs(reinterpret_cast<float4*>(p), v); }
  __device__ __forceinline__ void fma(float a, const Chunk& x) {
    v.x = fmaf(a, x.v.x, v.x); v.y = fmaf(a, x.v.y, v.y); v.z = fmaf(a, x.v.z, v.z); v.w = fmaf(a, x.v.w, v.w);
  }
  __device__ __forceinline__ void store(float* p) const { *reinterpret_cast<float4*>(p) = v; }
  __device__ __forceinline__ void red(float* p) const { red_add_v4(p, v.x, v.y, v.z, v.w); }
};
template <> struct Chunk<1> {
  float v;
  __device__ __forceinline__ void zero() { v = 0.f; }
  __device__ __forceinline__ void load(const float* p) { v = __ldg(p); }
  __device__ __forceinline__ void store_stream(float* p) const { __stcs(p, v); }
  __device__ __forceinline__ void fma(float a, const Chunk& x) { v = fmaf(a, x.v, v); }
  __device__ __forceinline__ void store(float* p) const { *p = v; }
  __device__ __forceinline__ void red(float* p) const { atomicAdd(p, v); }
};

// VEC = 8 stands for "B holds bf16": a lane gathers 8 consecutive 16-bit features with one
// 128-bit load and accumulates them in 8 floats (fp32 accumulation, fp32 C).
template <> struct Chunk<8> {
  float a[8];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = 0.f;
  }
  __device__ __forceinline__ void store(float* p) const {
    *reinterpret_cast<float4*>(p) = make_float4(a[0], a[1], a[2], a[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(a[4], a[5], a[6], a[7]);
  }
  __device__ __forceinline__ void store_stream(float* p) const {
    __stcs(reinterpret_cast<float4*>(p), make_float4(a[0], a[1], a[2], a[3]));
    __stcs(reinterpret_cast<float4*>(p + 4), make_float4(a[4], a[5], a[6], a[7]));
  }
  __device__ __forceinline__ void red(float* p) const {
    red_add_v4(p, a[0], a[1], a[2], a[3]);
    red_add_v4(p + 4, a[4], a[5], a[6], a[7]);
  }
};
struct RawBf16x8 {
  uint4 v;
  __device__ __forceinline__ void zero() { v = make_uint4(0u, 0u, 0u, 0u); }
  __device__ __forceinline__ void load(const uint16_t* p) { v = __ldg(reinterpret_cast<const uint4*>(p)); }
};
// element type of B and the register image of one gathered chunk, per VEC
template <int VEC> struct BTraits { using elem = float; using raw = Chunk<VEC>; };
template <> struct BTraits<8> { using elem = uint16_t; using raw = RawBf16x8; };

__device__ __forceinline__ void chunk_fma(Chunk<4>& acc, float a, const Chunk<4>& x) { acc.fma(a, x); }
__device__ __forceinline__ void chunk_fma(Chunk<1>& acc, float a, const Chunk<1>& x) { acc.fma(a, x); }
__device__ __forceinline__ void chunk_fma(Chunk<8>& acc, float a, const RawBf16x8& x) {
  const uint32_t w[4] = {x.v.x, x.v.y, x.v.z, x.v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {   // a bf16 is the upper half of the float with the same value
    acc.a[2 * i] = fmaf(a, __uint_as_float(w[i] << 16), acc.a[2 * i]);
    acc.a[2 * i + 1] = fmaf(a, __uint_as_float(w[i] & 0xffff0000u), acc.a[2 * i + 1]);
  }
}

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// address of row `col` of a matrix whose rows are `pitch_bytes` apart: one 32 x 32 + 64 bit multiply-add
__device__ __forceinline__ const void* row_of_b(const void* base, uint32_t col, uint32_t pitch_bytes) {
  uint64_t a;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(a) : "r"(col), "r"(pitch_bytes), "l"(reinterpret_cast<uint64_t>(base)));
  return reinterpret_cast<const void*>(a);
}

constexpr int kRingFeatures = 128;   // features one warp of the ring kernel covers

constexpr uint32_t kNoGather = 0xffffffffu;   // column of a slot that gathers nothing (padding, stored zero)

struct FeatCfg { int G, V, VEC, pass; };

// Kernel launch with, optionally, a programmatic dependency on the previous kernel of the stream
// (the row-clearing launch): the product kernel may start before that kernel has finished and
// orders itself with griddepcontrol.wait.
template <typename... Params, typename... Args>
cudaError_t launch_dep_smem(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t st,
                            bool dependent, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
template <typename... Params, typename... Args>
cudaError_t launch_dep(void (*kernel)(Params...), dim3 grid, int threads, cudaStream_t st, bool dependent, Args... args) {
  return launch_dep_smem(kernel, grid, threads, 0, st, dependent, args...);
}

inline FeatCfg pick_cfg(const void* B, int64_t ldb, const void* C, int64_t ldc, int N) {
  const bool vec = (N % 4 == 0) && (ldb % 4 == 0) && (ldc % 4 == 0) && ((uintptr_t)B % 16 == 0) &&
                   ((uintptr_t)C % 16 == 0);
  FeatCfg c;
  if (vec) {
    c.VEC = 4;
    if (N <= 32) { c.G = 8; c.V = 1; }
    else if (N <= 64) { c.G = 16; c.V = 1; }
    else if (N <= 128) { c.G = 32; c.V = 1; }
    else if (N <= 256) { c.G = 32; c.V = 2; }
    else { c.G = 32; c.V = 4; }
  } else {
    c.VEC = 1;
    c.G = 32;
    c.V = N <= 32 ? 1 : (N <= 64 ? 2 : 4);
  }
  c.pass = c.G * c.V * c.VEC;
  return c;
}


int sm_count();       // SMs of the current device
int gather_ring();    // LF_OPT_SPMM_GATHER_RING: rows in flight per warp in shared memory, 0 = in registers

// The ring kernels exist for 128-bit gathers over full warps; they multiply the column by a 32-bit
// row pitch in bytes.
inline bool ring_applies(const FeatCfg& cfg, int64_t ldb) { return cfg.VEC == 4 && cfg.G == 32 && ldb < (1ll << 30); }

}  // namespace lf
