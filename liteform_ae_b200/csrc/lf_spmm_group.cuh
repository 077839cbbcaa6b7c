// The gather ring for groups of lanes.
//
// A warp is R = 32 / G groups of G lanes.  A row of B is CH chunks of 16 bytes per lane of a group, and
// every group walks a run of consecutive slots (entries) of its own, so per step the warp multiplies R
// rows of B, one per group.  Groups are independent -- own slots, own row changes, own sum -- so a
// flush needs no sum over the warp and a row may end at any step.  The rows of B land in a ring of
// eight steps in shared memory, filled by cp.async; columns, values and row changes of G steps (a
// strip) are staged by the group's lanes, one slot each.
//
// What bounds it: instructions.  On 6.8 M entries a walk of one row (128 features) per warp and step
// takes 275 us, of two rows of 64 features 182 us, of four rows of 32 features 128 us: the time goes
// down with the bytes at 17 TB/s and with the steps not at all, because the work per row that does not
// depend on its length (its address, its row change, its share of staging and of the flush) stays.
// Everything below is written for that share:
//   * two chunks per lane (CH = 2), so that half the lanes carry a row and the other half another one;
//   * columns, row changes and values are read four steps at a time; a row change is the row id
//     itself in the slot where the row starts, -1 elsewhere, so that it needs neither masks nor a second
//     look-up; values are staged as pairs for the two-wide FMA;
//   * only copies and the write-out look at whether a lane has features; sums of lanes that have none
//     run on whatever the ring holds and are dropped;
//   * whether a row may also be held by another group is decided once for the first and once for the
//     last row of a walk.
//
// SH is the form for operands without 16-byte alignment (feature counts, leading dimensions or bases
// that are no multiple of four floats).  A row of B then starts at any word: the group copies the
// aligned 16-byte chunks that cover it -- each of them holds at least one word of the row, so it never
// leaves the 16-byte granule, hence the page, of valid memory -- and reads its features back word by
// word behind the row's shift of 0..3 words.  A lane owns features gl + G * v; which v it takes first
// is rotated by the group so that the groups of a warp read different banks.
#pragma once

#include "lf_spmm_gather.cuh"

namespace lf {

constexpr int kGroupSteps = 8;   // steps in flight: two commit groups of four
constexpr unsigned kAllLanes = 0xffffffffu;

template <int G> constexpr int kGroupStrips = G == 4 ? 4 : 2;   // strips held: those being copied and the one in use

// Lanes per group, chunks per lane and the number of walks (blocks along y) for N features.
struct GroupCfg { int G, CH, passes; };
// 16-byte aligned rows of `vec` features per chunk: groups as narrow as the row, two chunks per
// lane for rows of more than 128 bytes, pieces of 512 bytes for wider ones.
inline GroupCfg pick_group(int N, int vec) {
  if (N <= 4 * vec) return {4, 1, 1};
  if (N <= 8 * vec) return {8, 1, 1};
  if (N <= 16 * vec) return {8, 2, 1};
  return {16, 2, (N + 32 * vec - 1) / (32 * vec)};
}
// Shifted rows: a group of G lanes takes 4 G - 4 features behind any shift; a third of a full warp's
// time per walk is work that fewer lanes do not save.
inline GroupCfg pick_group_shifted(int N) {
  GroupCfg best{32, 1, 0};
  float cheapest = 0.f;
  for (int G = 32; G >= 4; G >>= 1) {
    const int passes = (N + 4 * G - 5) / (4 * G - 4);
    const float cost = passes * (0.35f + 0.65f * G / 32.f);
    if (!best.passes || cost < cheapest) {
      best = {G, 1, passes};
      cheapest = cost;
    }
  }
  return best;
}
template <int G, int CH, int VEC, bool SH> constexpr int kGroupFeatures = SH ? 4 * G - 4 : G * CH * VEC;

// Shared memory of one warp: the ring, then value pairs, columns and row starts of the strips, then (SH) the
// shifts in bytes.  A shifted read past the row's end takes words of the next row, at the end of the ring of
// the value pairs behind it; the sums that get them have no feature and are dropped.
template <int G, int CH, bool SH>
struct GroupSmem {
  static constexpr int kCells = kGroupStrips<G> * 32;
  static constexpr int kRing = kGroupSteps * CH * 512;
  static constexpr int kBytes = kRing + kCells * 16 + (SH ? kCells * 4 : 0);
  static_assert(kBytes % 16 == 0, "the next warp's ring starts on a 16-byte boundary");
};

// place of step q (0 .. G-1) of group g inside a strip: four steps of a group are adjacent
template <int G>
__device__ __forceinline__ int group_cell(int q, int g) { return (q >> 2) * (4 * (32 / G)) + g * 4 + (q & 3); }

// Row ids of the slots of one bucket: slot i belongs to ELL row i >> wlog.
template <int G>
struct EllRowIds {
  const int32_t* __restrict__ rows;   // of the group's first ELL row
  int wlog, n;                        // log2(width), slots of the group
  int first, pr, carry;
  bool head_open, tail_open;

  __device__ __forceinline__ void init(const int32_t* bucket_rows, int wlog_, int64_t e0, int64_t e1, int64_t ell_rows) {
    rows = bucket_rows + e0;
    wlog = wlog_;
    n = e1 > e0 ? (int)((e1 - e0) << wlog_) : 0;
    first = pr = 0;
    head_open = tail_open = false;
    if (n > 0) {
      first = bucket_rows[e0];
      head_open = e0 > 0 && bucket_rows[e0 - 1] == first;
      tail_open = e1 < ell_rows && bucket_rows[e1] == bucket_rows[e1 - 1];
    }
    carry = first;
  }
  __device__ __forceinline__ void prefetch(int k, int gl) {
    if (n > 0) pr = rows[min(k * G + gl, n - 1) >> wlog];
  }
  __device__ __forceinline__ void stage(int, int32_t* rd, int g, int gl) {
    int before = __shfl_up_sync(kAllLanes, pr, 1, G);
    if (gl == 0) before = carry;
    rd[group_cell<G>(gl, g)] = pr != before ? pr : -1;
    carry = __shfl_sync(kAllLanes, pr, G - 1, G);
  }
  __device__ __forceinline__ bool last_open() const { return tail_open; }
};

// Rows of consecutive CSR entries.  Lane gl watches the start of row r + 1 + gl, r being the row the
// walk has reached; a start that falls into a strip puts the row's number into its slot.
template <int G>
struct CsrRowIds {
  const int64_t* __restrict__ indptr;   // of the first row of the range
  int64_t origin;                       // entry the group starts with
  int num_rows, n, r, first, nb;
  bool head_open;

  __device__ __forceinline__ int start_of(int row) const {   // relative to the group's first entry, saturated
    const int64_t d = indptr[min(row, num_rows)] - origin;
    return d > 0x3fffffff ? 0x3fffffff : (int)d;
  }
  static __device__ __forceinline__ int count(bool mine, int g) {   // lanes of the group with `mine`
    const uint32_t m = __ballot_sync(kAllLanes, mine);
    return __popc(G == 32 ? m : (m >> (g * G)) & ((1u << (G % 32)) - 1u));
  }
  // entries [s0, s1) of the range whose first entry is `base`; every lane of the warp takes part
  __device__ __forceinline__ void init(const int64_t* range_indptr, int rows, int64_t base, int64_t s0, int64_t s1, int g, int gl) {
    indptr = range_indptr;
    num_rows = rows;
    n = s1 > s0 ? (int)(s1 - s0) : 0;
    origin = base + s0;
    int lo = 0, hi = n > 0 ? rows : 1;   // indptr[lo] <= origin, answer in [lo, hi): one probe per lane and round
    while (__any_sync(kAllLanes, hi - lo > 1)) {
      const int span = hi - lo;
      int q = lo + (int)(((int64_t)(gl + 1) * span) / (G + 1));
      if (q <= lo) q = lo + 1;
      const int cnt = count(span > 1 && indptr[q] <= origin, g);   // probes are monotone
      const int qlo = __shfl_sync(kAllLanes, q, cnt > 0 ? cnt - 1 : 0, G);
      const int qhi = __shfl_sync(kAllLanes, q, cnt < G ? cnt : G - 1, G);
      if (span > 1) {
        if (cnt > 0) lo = qlo;
        if (cnt < G) hi = qhi;
      }
    }
    first = r = lo;
    head_open = n > 0 && indptr[lo] < origin;
    nb = 0x3fffffff;
  }
  __device__ __forceinline__ void prefetch(int, int gl) {
    if (n > 0) nb = start_of(r + 1 + gl);
  }
  __device__ __forceinline__ void stage(int k, int32_t* rd, int g, int gl) {
    const int lo = k * G, hi = min(lo + G, n);
    rd[group_cell<G>(gl, g)] = -1;
    for (;;) {
      __syncwarp();
      const bool in = nb < hi;
      const int after = __shfl_down_sync(kAllLanes, nb, 1, G);
      if (in && (gl == G - 1 || after != nb)) rd[group_cell<G>(nb - lo, g)] = r + 1 + gl;   // of empty rows in between the last one counts
      const int cnt = count(in, g);
      r += cnt;
      if (!__any_sync(kAllLanes, cnt == G)) break;   // all G watched starts passed: there may be more (many short rows)
      prefetch(k, gl);
    }
  }
  __device__ __forceinline__ bool last_open() const { return start_of(r + 1) > n; }
};

__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add_pair(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float2 as_floats(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ uint64_t as_pair(uint32_t lo, uint32_t hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  return v;
}

// The sum of one row, and its way to C.  SUMS: how its terms are grouped, hence how its error grows.
//   1  one chain, the order of the register kernels: n terms of one size leave a variance of n^2 / 2 roundings;
//   2  the terms between two ends of a batch in a chain of their own, the batches in another: with four of them a
//      batch, n^2 / 8;
//   3  batches to two chains in turn: n^2 / 16 + 4 n, at every n no more than four interleaved chains leave.
// A chain per step of a batch would do as much but has to be added up at every row change, by one group of a
// warp while the others wait: 2^18 power-law rows at 32 features 67 us against 47 for one chain.
template <int G, int CH, int VEC, bool SH, int SUMS>
struct GroupSum {
  static constexpr int kPairs = CH * VEC / 2;
  uint64_t s[SUMS][kPairs];   // s[0]: the total in the end; s[SUMS - 1]: the batch (SUMS > 1); s[1]: the other chain (3)
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int p = 0; p < SUMS; ++p)
#pragma unroll
      for (int i = 0; i < kPairs; ++i) s[p][i] = 0;
  }
  __device__ __forceinline__ void end_batch(int turn) {   // turn: the chain that takes the batch
    if constexpr (SUMS > 1) {
#pragma unroll
      for (int i = 0; i < kPairs; ++i) {
        s[turn][i] = add_pair(s[turn][i], s[SUMS - 1][i]);
        s[SUMS - 1][i] = 0;
      }
    }
  }
  // everything into s[0]; inside: terms of a batch that has not ended may be there
  __device__ __forceinline__ void total(bool inside) {
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
      if (SUMS == 3) s[0][i] = add_pair(s[0][i], s[1][i]);
      if (SUMS > 1 && inside) s[0][i] = add_pair(s[0][i], s[SUMS - 1][i]);
    }
  }
  // after total(): nothing but the total is left
  __device__ __forceinline__ void settle() {
#pragma unroll
    for (int p = 1; p < SUMS; ++p)
#pragma unroll
      for (int i = 0; i < kPairs; ++i) s[p][i] = 0;
  }
  // adds the total that the lane `from` further up holds, if `take`
  __device__ __forceinline__ void join(int from, bool take, int) {
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
      const uint64_t y = __shfl_down_sync(kAllLanes, (unsigned long long)s[0][i], from);
      if (take) s[0][i] = add_pair(s[0][i], y);
    }
  }
  // x: this lane's first chunk of the row in the ring (CH chunks, 512 bytes apart)
  __device__ __forceinline__ void add(uint64_t val, const unsigned char* x) {
    uint64_t* a = s[SUMS - 1];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if constexpr (VEC == 4) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(x + c * 512);
        a[2 * c] = fma_pair(val, v.x, a[2 * c]);
        a[2 * c + 1] = fma_pair(val, v.y, a[2 * c + 1]);
      } else {
        const uint4 v = *reinterpret_cast<const uint4*>(x + c * 512);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)   // a bf16 is the upper half of the float with the same value
          a[4 * c + i] = fma_pair(val, as_pair(w[i] << 16, w[i] & 0xffff0000u), a[4 * c + i]);
      }
    }
  }
  // row: this lane's first feature in C; nf: features from there to the end of the row
  __device__ __forceinline__ void write(float* row, int nf, bool open) const {
    const uint64_t* a = s[0];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (c * G * VEC < nf) {
#pragma unroll
        for (int h = 0; h < VEC / 4; ++h) {
          float* p = row + c * G * VEC + 4 * h;
          const uint64_t lo = a[c * VEC / 2 + 2 * h], hi = a[c * VEC / 2 + 2 * h + 1];
          if (open) {
            const float2 x = as_floats(lo), y = as_floats(hi);
            red_add_v4(p, x.x, x.y, y.x, y.y);
          } else {
            __stcs(reinterpret_cast<ulonglong2*>(p), make_ulonglong2(lo, hi));
          }
        }
      }
    }
  }
};
template <int G, int VEC>
struct GroupSum<G, 1, VEC, true, 1> {
  float a[4];
  __device__ __forceinline__ void zero() { a[0] = a[1] = a[2] = a[3] = 0.f; }
  __device__ __forceinline__ void end_batch(int) {}
  __device__ __forceinline__ void total(bool) {}
  __device__ __forceinline__ void settle() {}
  // h: the group that gives.  Its lanes hold the features of the group before it, one place on where the two
  // groups start with different features.
  __device__ __forceinline__ void join(int from, bool take, int h) {
    const bool turned = G != 4 || (h & 1) == 0;
    float y[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) y[v] = __shfl_down_sync(kAllLanes, turned ? a[(v + 3) & 3] : a[v], from);
#pragma unroll
    for (int v = 0; v < 4; ++v)
      if (take) a[v] += y[v];
  }
  // feature v of lane gl: the groups that share banks (G = 4: every other one) start with different v
  static __device__ __forceinline__ int feature(int v, int g, int gl) { return gl + G * ((v + (G == 4 ? g >> 1 : g)) & 3); }
};

// One warp; cols / vals point at the calling group's first slot (vals == nullptr: all ones), `ids`
// knows the rows of its ids.n slots (0: the group has nothing to do).  WC: row changes happen only at
// multiples of WC slots.  all_open: every row may be held by other groups too.  C: row 0 of the output
// the row ids count from, at the first feature of this walk; nf: features from there on.  The groups of
// a warp hold neighbouring ranges.  BATCH: steps to a batch of the sums, 0: as many as `chain` (a power of two)
// says.
template <int G, int CH, int VEC, bool SH, int WC, int SUMS, int BATCH, class Rows>
__device__ __forceinline__ void walk_group_ring(Rows& ids, bool all_open, const int32_t* __restrict__ cols,
                                                const float* __restrict__ vals,
                                                const typename BTraits<VEC>::elem* __restrict__ B, int ldb,
                                                float* __restrict__ C, int64_t ldc, int nf, int g, int gl,
                                                unsigned char* smem, int chain = 0) {
  using Elem = typename BTraits<VEC>::elem;
  using Smem = GroupSmem<G, CH, SH>;
  constexpr int U = 4, R = 32 / G, kCells = Smem::kCells, kHalf = U * CH * 512;
  static_assert(kGroupSteps == 2 * U && G % U == 0, "two commit groups of four steps in flight");
  static_assert(BATCH == 0 || BATCH == U, "the steps of a loop turn, or a number of turns");
  static_assert(!SH || (VEC == 4 && CH == 1), "the shifted form is for float32 rows, one chunk per lane");
  uint64_t* sv = reinterpret_cast<uint64_t*>(smem + Smem::kRing);   // {value, value}
  uint32_t* so = reinterpret_cast<uint32_t*>(sv + kCells);          // column or kNoGather
  int32_t* rd = reinterpret_cast<int32_t*>(so + kCells);            // row that starts here, or -1
  uint32_t* ss = reinterpret_cast<uint32_t*>(rd + kCells);          // SH: bytes between chunk and row start
  const int lane = g * G + gl;
  const int n = ids.n;
  const int nmax = __reduce_max_sync(kAllLanes, n);
  const int nstrips = (nmax + G - 1) / G;

  // where this lane's chunks lie in a row, and whether they hold features (lanes past the last feature
  // copying its last chunk again took 237 us, masking them 181 us, on 3.7 M entries, 100 features)
  const char* Bl = reinterpret_cast<const char*>(B) + (SH ? 0 : gl * 16);
  const bool in1 = SH || gl * VEC < nf, in2 = CH == 2 && (gl + G) * VEC < nf;
  const uint32_t pitch = (uint32_t)ldb * (uint32_t)sizeof(Elem), pitch_c = (uint32_t)ldc * 4u;   // checked by the launch
  const int over = SH ? gl * 16 - nf * 4 : 0;   // SH: chunk gl is needed while the shift is larger than this

  GroupSum<G, CH, VEC, SH, SUMS> sum;
  sum.zero();
  int cur = ids.first;
  bool open = all_open || ids.head_open;
  float* Cl = C + (SH ? 0 : gl * VEC);
  auto flush = [&](bool open_now, bool inside) {
    float* row = reinterpret_cast<float*>(const_cast<void*>(row_of_b(Cl, (uint32_t)cur, pitch_c)));
    sum.total(inside);
    if constexpr (SH) {
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int f = sum.feature(v, g, gl);
        if (f < nf) {
          if (open_now) atomicAdd(row + f, sum.a[v]); else __stcs(row + f, sum.a[v]);
        }
      }
    } else {
      sum.write(row, nf - gl * VEC, open_now);
    }
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
  const int my_cell = group_cell<G>(gl, g);
  auto store_strip = [&](int k, int base) {
    const int cell = base + my_cell;
    so[cell] = pv != 0.f ? (uint32_t)pc : kNoGather;
    sv[cell] = as_pair(__float_as_uint(pv), __float_as_uint(pv));
    if constexpr (SH) ss[cell] = ((uint32_t)reinterpret_cast<uintptr_t>(B) + (uint32_t)pc * pitch) & 12u;
    ids.stage(k, rd + base, g, gl);
  };
  load_strip(0);
  store_strip(0, 0);
  __syncwarp();
  if (nstrips > 1) load_strip(1);

  const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(smem) + lane * 16;
  int k_next = 1, in_cell = 0, in_half = 0;   // producer: next strip to store, place in the strips, half of the ring
  // start the copies of four steps and close them as one group; past the end the group is empty, which
  // keeps the number of groups per batch constant
  auto issue_batch = [&](int j) {
    if (j < nstrips * G) {
      if ((in_cell & 31) == 0 && j > 0) {   // first steps of a strip: it moves from registers to shared memory
        __syncwarp();                       // (its place held a strip that has been added up)
        store_strip(k_next, in_cell);
        __syncwarp();
        if (++k_next < nstrips) load_strip(k_next);
      }
      const uint4 o4 = *reinterpret_cast<const uint4*>(so + in_cell + g * 4);
      const uint32_t o[U] = {o4.x, o4.y, o4.z, o4.w};
      const uint32_t dst = ring_s + in_half;
      if constexpr (SH) {
        const int4 h4 = *reinterpret_cast<const int4*>(ss + in_cell + g * 4);
        const int h[U] = {h4.x, h4.y, h4.z, h4.w};
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (o[u] != kNoGather && h[u] > over)
            cp_async_16(dst + u * 512, reinterpret_cast<const void*>((reinterpret_cast<uint64_t>(row_of_b(Bl, o[u], pitch)) & ~15ull) + gl * 16));
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const char* src = reinterpret_cast<const char*>(row_of_b(Bl, o[u], pitch));
          if (o[u] != kNoGather && in1) cp_async_16(dst + u * (CH * 512), src);
          if (CH == 2 && o[u] != kNoGather && in2) cp_async_16(dst + u * (CH * 512) + 512, src + G * 16);
        }
      }
      in_cell = (in_cell + U * R) & (kCells - 1);
      in_half ^= kHalf;
    }
    cp_async_commit();
  };
  issue_batch(0);
  issue_batch(U);
  wait_for_prior_grid();   // no store or atomic to C before the row-clearing launch is complete

  int cell = g * 4, half = 0;   // consumer
  auto batch = [&](int j, int turn) {   // the four steps from j on
    const int4 r4 = *reinterpret_cast<const int4*>(rd + cell);
    const ulonglong2 va = *reinterpret_cast<const ulonglong2*>(sv + cell), vb = *reinterpret_cast<const ulonglong2*>(sv + cell + 2);
    const int start[U] = {r4.x, r4.y, r4.z, r4.w};
    const uint64_t val[U] = {va.x, va.y, vb.x, vb.y};
    int4 h4 = make_int4(0, 0, 0, 0);
    if constexpr (SH) h4 = *reinterpret_cast<const int4*>(ss + cell);
    const int h[U] = {h4.x, h4.y, h4.z, h4.w};
    cp_async_wait<1>();                // all but the newest group of copies have landed
    if constexpr (SH) __syncwarp();    // lanes read words that other lanes copied
    const unsigned char* x = smem + half + (SH ? g * G * 16 : lane * 16);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u % WC == 0 && start[u] >= 0) {
        flush(open, u > 0 || BATCH == 0);
        cur = start[u];
        open = all_open;
      }
      if constexpr (SH) {
        const float v0 = as_floats(val[u]).x;
        if (v0 != 0.f) {
          const unsigned char* w = x + u * 512 + h[u];
#pragma unroll
          for (int v = 0; v < 4; ++v) sum.a[v] = fmaf(v0, *reinterpret_cast<const float*>(w + sum.feature(v, g, gl) * 4), sum.a[v]);
        }
      } else {
        if (as_floats(val[u]).x != 0.f) sum.add(val[u], x + u * (CH * 512));
      }
    }
    if (BATCH == U || ((j + U) & (chain - 1)) == 0) sum.end_batch(turn);
    if constexpr (SH) __syncwarp();    // every lane has read before the slots are refilled
    cell = (cell + U * R) & (kCells - 1);
    half ^= kHalf;
    issue_batch(j + 2 * U);            // refills exactly the ring slots read above
  };
  if constexpr (SUMS == 3) {
    for (int j = 0; j < nmax; j += 2 * U) {
      batch(j, 0);
      if (j + U < nmax) batch(j + U, 1);
    }
  } else {
    for (int j = 0; j < nmax; j += U) batch(j, 0);
  }
  // A row that goes on over whole ranges: a group that saw nothing else hands its sum to the group before it,
  // the last one first, so that such a row costs one atomic add per warp and not one per range, and the chain
  // of those adds is that much shorter.
  bool give = false;
  if constexpr (R > 1) {
    const int before = __shfl_up_sync(kAllLanes, n > 0 ? cur : -1, G);
    give = g > 0 && n > 0 && cur == ids.first && before == cur;
    if (__any_sync(kAllLanes, give)) {
      sum.total(BATCH == 0);
      sum.settle();
      for (int h = R - 1; h > 0; --h) {
        if (__shfl_sync(kAllLanes, give, h * G)) sum.join(G, g == h - 1, h);
      }
    }
  }
  if (n > 0 && !give) flush(open || ids.last_open(), BATCH == 0);
}

}  // namespace lf
