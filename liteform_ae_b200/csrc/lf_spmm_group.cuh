// The gather ring for thread groups of 8, 16 or 32 lanes.
//
// A warp is R = 32 / G groups of G lanes; a row of B is one 16-byte chunk per lane of a group, and
// every group walks a run of consecutive slots (entries) of its own.  Per step the warp therefore
// multiplies R rows of B, one per group: a 128-byte row (32 float32 features) costs a quarter of the
// instructions it would cost a whole warp.  Groups are independent -- own slots, own row
// changes, own sum -- so a flush needs no sum over the warp and a bucket of any width (or a CSR row
// of any length) may end at any step.  The gathers land in a ring of 16 steps in shared memory,
// filled by cp.async; columns, values and row changes of G steps (a strip) are staged by the
// group's lanes, one slot each, so that what is the same for all lanes is computed once.
//
// What bounds it: the L2 hands a streaming multiprocessor about 30 bytes per clock of scattered
// 128-byte rows (42 of 512-byte rows), and the ring keeps enough of them in flight to be there.
//
// ODD is the form for operands without 16-byte alignment (feature counts, leading dimensions or
// bases that are no multiple of four floats).  A row of B then starts at any word: the group copies
// the aligned 16-byte chunks that cover it -- every chunk holds at least one word of the row, so it
// never leaves the 16-byte granule, hence the page, of valid memory -- and reads its features back
// word by word behind the row's shift of 0..3 words.  A lane owns features gl + G * v; which v it
// takes first is rotated by the group so that the groups of a warp read different banks.
#pragma once

#include "lf_spmm_gather.cuh"

namespace lf {

constexpr int kGroupSteps = 16;                                                      // steps in flight
template <int G> constexpr int kGroupStrips = (kGroupSteps + G - 1) / G + 1;         // strips held: those ahead and the one in use
template <int G> constexpr int kGroupOddFeatures = 4 * G - 4;                        // features per group behind any shift

// Lanes per group for N features and the number of times the slots are walked for it (blocks along y).
// Operands with 16-byte alignment: the smallest group that holds a row of B, 32 lanes from 128 features
// on.  Others: a group of G lanes takes 4 G - 4 features; the walk itself costs about a fifth of the
// multiplication by a full warp (staging, addresses), the rest goes down with the rows per step.
struct GroupCfg { int G, passes; };
inline GroupCfg pick_group(bool aligned, int N) {
  if (aligned) {
    const int G = N <= 32 ? 8 : (N <= 64 ? 16 : 32);
    return {G, (N + 4 * G - 1) / (4 * G)};
  }
  GroupCfg best{32, 0};
  float cheapest = 0.f;
  for (int G = 32; G >= 8; G >>= 1) {
    const int passes = (N + 4 * G - 5) / (4 * G - 4);
    const float cost = passes * (0.2f + G / 32.f);
    if (!best.passes || cost < cheapest) {
      best = {G, passes};
      cheapest = cost;
    }
  }
  return best;
}

// Shared memory of one warp: the ring (a few words longer, because a shifted read of features past the
// row's end is not masked), then columns, values and row ids of the strips, then the shifts.
template <int G, bool ODD>
struct GroupSmem {
  static constexpr int kStrip = kGroupStrips<G> * 32;
  static constexpr int kBytes = kGroupSteps * 512 + (ODD ? 16 : 0) + kStrip * 12 + (ODD ? kStrip : 0);
  static_assert(kBytes % 16 == 0, "the next warp's ring starts on a 16-byte boundary");
};

// Row ids of the slots of one bucket: slot i belongs to ELL row i >> wlog.
template <int G>
struct EllRowIds {
  const int32_t* __restrict__ rows;   // of the group's first ELL row
  int wlog, n;                        // log2(width), slots of the group
  int first, last;
  bool head_open, tail_open, all_open;
  int pr, carry;

  __device__ __forceinline__ void init(const int32_t* bucket_rows, int wlog_, int64_t e0, int64_t e1, int64_t ell_rows,
                                       bool all) {
    rows = bucket_rows + e0;
    wlog = wlog_;
    n = e1 > e0 ? (int)((e1 - e0) << wlog_) : 0;
    all_open = all;
    first = last = 0;
    head_open = tail_open = false;
    if (n > 0) {
      first = bucket_rows[e0];
      last = bucket_rows[e1 - 1];
      head_open = e0 > 0 && bucket_rows[e0 - 1] == first;
      tail_open = e1 < ell_rows && bucket_rows[e1] == last;
    }
    carry = first;
    pr = 0;
  }
  __device__ __forceinline__ void prefetch(int k, int gl) {
    if (n > 0) pr = rows[min(k * G + gl, n - 1) >> wlog];
  }
  // writes the row ids of strip k; bit (lane) of the result: that slot carries another row than the one before
  __device__ __forceinline__ uint32_t stage(int, int32_t* rd, int gl) {
    rd[gl] = pr;
    int before = __shfl_up_sync(0xffffffffu, pr, 1, G);
    if (gl == 0) before = carry;
    carry = __shfl_sync(0xffffffffu, pr, G - 1, G);
    return __ballot_sync(0xffffffffu, pr != before);
  }
  __device__ __forceinline__ int first_row() const { return first; }
  // may another group hold a part of this row?
  __device__ __forceinline__ bool open(int row, bool /*at_end*/) const {
    return all_open || (row == first && head_open) || (row == last && tail_open);
  }
  __device__ __forceinline__ void finish() {}
};

// Rows of consecutive CSR entries.  Lane gl watches the start of row r + 1 + gl, r being the row the
// walk has reached; starts that fall into a strip become bits, the rows they start their ids.
template <int G>
struct CsrRowIds {
  const int64_t* __restrict__ indptr;   // of the first row of the range
  int64_t origin;                       // entry the group starts with
  int64_t num_rows;
  int n;
  int64_t r;
  int first, nb;
  bool head_open, tail_open;

  __device__ __forceinline__ int start_of(int64_t row) const {   // relative to the group's first entry, saturated
    const int64_t d = indptr[row < num_rows ? row : num_rows] - origin;
    return d > 0x3fffffff ? 0x3fffffff : (int)d;
  }
  // entries [s0, s1) of the range whose first entry is `base`; every lane of the warp takes part
  __device__ __forceinline__ void init(const int64_t* range_indptr, int64_t rows, int64_t base, int64_t s0, int64_t s1, int lane) {
    constexpr unsigned kAll = 0xffffffffu;
    const int gl = lane % G, shift = lane / G * G;
    indptr = range_indptr;
    num_rows = rows;
    n = s1 > s0 ? (int)(s1 - s0) : 0;
    origin = base + s0;
    int64_t lo = 0, hi = n > 0 ? rows : 1;   // indptr[lo] <= origin, answer in [lo, hi): one probe per lane and round
    while (__any_sync(kAll, hi - lo > 1)) {
      const int64_t span = hi - lo;
      int64_t q = lo + ((int64_t)(gl + 1) * span) / (G + 1);
      if (q <= lo) q = lo + 1;
      const bool le = span > 1 && indptr[q] <= origin;
      const uint32_t m = __ballot_sync(kAll, le) >> shift;
      const int cnt = __popc(G == 32 ? m : m & ((1u << (G % 32)) - 1u));   // probes are monotone
      const int64_t qlo = __shfl_sync(kAll, q, cnt > 0 ? cnt - 1 : 0, G);
      const int64_t qhi = __shfl_sync(kAll, q, cnt < G ? cnt : G - 1, G);
      if (span > 1) {
        if (cnt > 0) lo = qlo;
        if (cnt < G) hi = qhi;
      }
    }
    r = lo;
    first = (int)lo;
    head_open = n > 0 && indptr[lo] < origin;
    tail_open = false;
    nb = 0x3fffffff;
  }
  __device__ __forceinline__ void prefetch(int, int gl) {
    if (n > 0) nb = start_of(r + 1 + gl);
  }
  __device__ __forceinline__ uint32_t stage(int k, int32_t* rd, int gl) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lo = k * G, hi = min(lo + G, n);
    const int shift = (threadIdx.x & 31) / G * G;
    uint32_t starts = 0;
    for (;;) {
      const bool in = nb < hi;
      const int after = __shfl_down_sync(kAll, nb, 1, G);
      if (in && (gl == G - 1 || after != nb)) rd[nb - lo] = (int)(r + 1 + gl);   // of empty rows in between the last one counts
      starts |= __reduce_or_sync(kAll, in ? 1u << (shift + nb - lo) : 0u);
      const uint32_t m = __ballot_sync(kAll, in) >> shift;
      const int cnt = __popc(G == 32 ? m : m & ((1u << (G % 32)) - 1u));
      r += cnt;
      if (!__any_sync(kAll, cnt == G)) break;   // all G watched starts passed: there may be more (many short rows)
      __syncwarp();
      prefetch(k, gl);
    }
    return starts;
  }
  __device__ __forceinline__ int first_row() const { return first; }
  __device__ __forceinline__ bool open(int row, bool at_end) const {
    return (row == first && head_open) || (at_end && tail_open);
  }
  __device__ __forceinline__ void finish() {
    if (n > 0) tail_open = start_of(r + 1) > n;
  }
};

// Sums and write-out of one group's row: VEC features per lane, or four single words per lane (ODD).
template <int G, int VEC, bool ODD>
struct GroupSum {
  Chunk<VEC> acc;
  __device__ __forceinline__ void zero() { acc.zero(); }
  __device__ __forceinline__ void write(float* row, int gl, int, int nf, bool open) const {
    if (gl * VEC < nf) {
      if (open) acc.red(row + gl * VEC); else acc.store_stream(row + gl * VEC);
    }
  }
};
template <int G, int VEC>
struct GroupSum<G, VEC, true> {
  float a[4];
  __device__ __forceinline__ void zero() { a[0] = a[1] = a[2] = a[3] = 0.f; }
  static __device__ __forceinline__ int feature(int v, int gl, int g) { return gl + G * ((v + g) & 3); }
  __device__ __forceinline__ void write(float* row, int gl, int g, int nf, bool open) const {
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int f = feature(v, gl, g);
      if (f < nf) {
        if (open) atomicAdd(row + f, a[v]); else __stcs(row + f, a[v]);
      }
    }
  }
};

// One warp; cols / vals point at the calling group's first slot (vals == nullptr: all ones), `ids`
// knows the rows of its ids.n slots (0: the group has nothing to do).  WC: row changes happen only at
// multiples of WC slots.  C: row 0 of the output the row ids count from, at feature f0.
template <int G, int VEC, bool ODD, int WC, class Rows>
__device__ __forceinline__ void walk_group_ring(Rows& ids, const int32_t* __restrict__ cols, const float* __restrict__ vals,
                                                const typename BTraits<VEC>::elem* __restrict__ B, int ldb,
                                                float* __restrict__ C, int64_t ldc, int nf, int lane, unsigned char* smem) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int U = 8, D = kGroupSteps, NB = kGroupStrips<G>, kStrip = GroupSmem<G, ODD>::kStrip;
  static_assert(D == 2 * U && G % U == 0 && U % WC == 0, "two commit groups of eight steps in flight");
  static_assert(!ODD || VEC == 4, "the shifted form is for float32 rows");
  const int gl = lane % G, g = lane / G;
  uint32_t* so = reinterpret_cast<uint32_t*>(smem + D * 512 + (ODD ? 16 : 0));
  float* sv = reinterpret_cast<float*>(so + kStrip);
  int32_t* rd = reinterpret_cast<int32_t*>(sv + kStrip);
  uint8_t* ss = reinterpret_cast<uint8_t*>(rd + kStrip);
  const int n = ids.n;
  const int nmax = __reduce_max_sync(kAll, n);
  const int nstrips = (nmax + G - 1) / G;
  const bool active = ODD || gl * VEC < nf;
  GroupSum<G, VEC, ODD> sum;
  sum.zero();
  int cur = ids.first_row();
  auto flush = [&](int row, bool at_end) {
    sum.write(C + (int64_t)row * ldc, gl, g, nf, ids.open(row, at_end));
    sum.zero();
  };

  int pc = 0;
  float pv = 0.f;
  auto load_strip = [&](int k) {
    const int i = k * G + gl;
    const bool in = i < n;
    pc = in ? __ldcs(cols + i) : 0;
    pv = in ? (vals ? __ldcs(vals + i) : 1.f) : 0.f;
    ids.prefetch(k, gl);
  };
  uint32_t chg[NB];   // per strip held: bit (lane) = that slot starts another row
#pragma unroll
  for (int b = 0; b < NB; ++b) chg[b] = 0;
  const uint32_t base_shift = (uint32_t)(reinterpret_cast<uintptr_t>(B) >> 2);
  auto store_strip = [&](int k, int at) {
    const int cell = at * 32 + lane;
    so[cell] = pv != 0.f ? (uint32_t)pc : kNoGather;
    sv[cell] = pv;
    if constexpr (ODD) ss[cell] = (uint8_t)((base_shift + (uint32_t)pc * (uint32_t)ldb) & 3u);
    const uint32_t m = ids.stage(k, rd + at * 32 + g * G, gl);
#pragma unroll
    for (int b = 0; b < NB; ++b)
      if (b == at) chg[b] = m;
  };
  int in_at = 0;   // place of the newest strip
  load_strip(0);
  store_strip(0, 0);
  __syncwarp();
  if (nstrips > 1) load_strip(1);

  const float4* ring_lane = reinterpret_cast<const float4*>(smem) + lane;
  const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring_lane);
  const uint32_t pitch = (uint32_t)ldb * (uint32_t)sizeof(typename BTraits<VEC>::elem);   // checked by the launch
  const typename BTraits<VEC>::elem* __restrict__ Bl = ODD ? B : B + gl * VEC;
  const uint4* so4 = reinterpret_cast<const uint4*>(so);
  const float4* sv4 = reinterpret_cast<const float4*>(sv);
  auto issue_batch = [&](int j0, auto slot_tag) {
    constexpr int SLOT = decltype(slot_tag)::value;
    if (j0 < nstrips * G) {
      const int q0 = j0 % G;
      if (q0 == 0 && j0 > 0) {   // first steps of a strip: it moves from registers to shared memory
        const int k = j0 / G;    // (its place held a strip that has been added up)
        in_at = in_at + 1 == NB ? 0 : in_at + 1;
        __syncwarp();
        store_strip(k, in_at);
        __syncwarp();
        if (k + 1 < nstrips) load_strip(k + 1);
      }
      const int at = in_at * 32 + g * G + q0;
      const uint4 oa = so4[at >> 2], ob = so4[(at >> 2) + 1];
      const uint32_t o[U] = {oa.x, oa.y, oa.z, oa.w, ob.x, ob.y, ob.z, ob.w};
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if constexpr (ODD) {
          if (o[u] != kNoGather) {
            const uint64_t a = reinterpret_cast<uint64_t>(row_of_b(Bl, o[u], pitch));
            if (gl * 4 < (int)((a >> 2) & 3) + nf)
              cp_async_16(ring_s + (uint32_t)(SLOT + u) * 512u, reinterpret_cast<const void*>((a & ~15ull) + gl * 16));
          }
        } else {
          if (o[u] != kNoGather && active) cp_async_16(ring_s + (uint32_t)(SLOT + u) * 512u, row_of_b(Bl, o[u], pitch));
        }
      }
    }
    cp_async_commit();
  };
  issue_batch(0, std::integral_constant<int, 0>{});
  issue_batch(U, std::integral_constant<int, U>{});
  wait_for_prior_grid();   // no store or atomic to C before the row-clearing launch is complete

  int out_at = 0;          // place of the strip being added up
  auto add_batch = [&](int jc, auto slot_tag) {
    constexpr int SLOT = decltype(slot_tag)::value;
    const int q0 = jc % G;
    if (q0 == 0 && jc > 0) out_at = out_at + 1 == NB ? 0 : out_at + 1;
    const int at = out_at * 32 + g * G + q0;
    const float4 va = sv4[at >> 2], vb = sv4[(at >> 2) + 1];
    const float val[U] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
    uint32_t m = chg[0];
#pragma unroll
    for (int b = 1; b < NB; ++b)
      if (b == out_at) m = chg[b];
    const uint32_t starts = m >> (g * G + q0);
    uint2 shifts = make_uint2(0u, 0u);
    if constexpr (ODD) shifts = *reinterpret_cast<const uint2*>(ss + at);
    cp_async_wait<1>();            // all but the newest group of copies have landed
    if constexpr (ODD) __syncwarp();   // lanes read words that other lanes copied
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u % WC == 0 && ((starts >> u) & 1u)) {
        flush(cur, false);
        cur = rd[at + u];
      }
      if (val[u] != 0.f && active) {
        if constexpr (ODD) {
          const uint32_t sh = ((u < 4 ? shifts.x : shifts.y) >> (8 * (u & 3))) & 3u;
          const float* x = reinterpret_cast<const float*>(smem) + (SLOT + u) * 128 + g * G * 4 + sh;
#pragma unroll
          for (int v = 0; v < 4; ++v) sum.a[v] = fmaf(val[u], x[sum.feature(v, gl, g)], sum.a[v]);
        } else {
          typename BTraits<VEC>::raw x;
          const float4 raw = ring_lane[(SLOT + u) * 32];
          if constexpr (VEC == 8) x.v = make_uint4(__float_as_uint(raw.x), __float_as_uint(raw.y), __float_as_uint(raw.z), __float_as_uint(raw.w));
          else x.v = raw;
          chunk_fma(sum.acc, val[u], x);
        }
      }
    }
    if constexpr (ODD) __syncwarp();   // every lane has read before the slots are refilled
    issue_batch(jc + D, slot_tag);     // refills exactly the ring slots read above
  };
  for (int jc0 = 0; jc0 < nmax; jc0 += D) {
    add_batch(jc0, std::integral_constant<int, 0>{});
    if (jc0 + U >= nmax) break;
    add_batch(jc0 + U, std::integral_constant<int, U>{});
  }
  ids.finish();
  if (n > 0) flush(cur, true);
}

}  // namespace lf
