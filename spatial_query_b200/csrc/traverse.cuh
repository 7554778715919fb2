// Persistent, warp-pulled BVH traversal kernels for sm_100a.
//
// Replaces the WGSL `main` of crates/spatial-query/src/gpu/mod.rs:159-226 (one
// invocation per ray, 48-byte nodes, no ordering) with:
//  * a child-pair node record: an interior node holds both children's boxes
//    and codes in 16-byte vectors (64 B at D = 3), so one record fetch tests
//    two boxes;
//  * a persistent grid (a multiple of the SM count) whose warps pull batches
//    of 32 queries from an atomic counter, so uneven per-query work balances;
//  * a per-thread traversal stack in shared memory ([depth][thread], so
//    consecutive lanes hit consecutive banks), each entry carrying the child's
//    slab entry so it can be re-checked exactly against the shrunk limit when
//    popped;
//  * near-first child ordering for nearest queries, or the reference's own
//    order (push child_a, then child_b, pop child_b first; accel/bvh.rs:119-120)
//    when REF is set, which replays the CPU decisions one for one.
//
// Node code: an interior record index, or kLeafBit | the first position of the
// leaf's primitives in the leaf-ordered primitive array. The last primitive of
// a leaf carries kLeafBit in its id word.
#pragma once

#include "sq_math.cuh"

namespace sq {

enum Narrow : int { kNarrowAabb = 0, kNarrowSphere = 1, kNarrowSphereNear = 2, kNarrowTri = 3, kNarrowCustom = 4 };

// A consumer narrow phase (kNarrowCustom) is compiled at run time with NVRTC
// into the same kernels: its source defines
//   __device__ bool sq_narrow(const float* prim, uint32_t leaf, const float* ro, const float* rd,
//                             float max_toi, float* toi, float* normal);
// and SQ_CUSTOM_STRIDE is the number of floats per leaf. Its primitive
// record holds those floats, then the leaf's AABB (the box the tree was built
// from, used to certify near-first answers), then the id word.
#ifndef SQ_CUSTOM_STRIDE
#define SQ_CUSTOM_STRIDE 1
#endif
#ifdef SQ_RTC_CUSTOM
__device__ bool sq_narrow(const float* prim, uint32_t leaf, const float* ro, const float* rd, float max_toi, float* toi,
                          float* normal);
#endif
// Optionally the source also defines every crossing of a leaf
// (QueryGeometry::test_ray_crossings, consumed by Bvh::raycast_crossings,
// accel/bvh.rs:286-328); SQ_RTC_CROSSINGS is then defined and
// raycast_crossings lists each emit(toi, normal) call:
//   template <class Emit>
//   __device__ void sq_narrow_crossings(const float* prim, uint32_t leaf, const float* ro, const float* rd,
//                                       float max_toi, Emit& emit);
#ifdef SQ_RTC_CROSSINGS
template <class Emit>
__device__ void sq_narrow_crossings(const float* prim, uint32_t leaf, const float* ro, const float* rd, float max_toi,
                                    Emit& emit);
#endif
enum QKind : int { kRayNearest = 0, kRayAll = 1, kCastNearest = 2, kCastAll = 3, kOverlap = 4 };

// Leaves per region the overlap count pass keeps (QueryParams::keep).
constexpr uint32_t kOverlapKeep = 4;

constexpr int kThreads = 128;

// Two walk variants, measured on the 1,048,576-triangle terrain and off by
// default (each slower there; both together are also built as the WALK = 1
// instantiation, SQ_LAYOUT_BINARY_REGTOP, which the autotuner can pick):
//  * SQ_POSTPONE_LEAVES: a lane that reaches a leaf holds it and keeps
//    descending until the whole warp holds leaves (Aila and Laine's
//    speculative traversal): the nodes it visits before the leaf's hit
//    tightens the limit cost more than the leaf tests gain from running
//    together.
//  * SQ_REG_TOP (with postponed leaves): the stack's top entry in registers,
//    older entries in the shared-memory stack: 0.672-0.682 ms per 1,048,576
//    rays against 0.436 ms for the warp-stepped walk; the saved shared-memory
//    round trip is short next to a node fetch from L2, and these walks have no
//    helping lanes.
#ifndef SQ_POSTPONE_LEAVES
#define SQ_POSTPONE_LEAVES 0
#endif
#ifndef SQ_REG_TOP
#define SQ_REG_TOP 0
#endif
// Child order by warp vote (1) in the certified near-first walk: the lanes
// that open the same record with both children hit take the order most of
// them prefer (a __match_any_sync group and a ballot), so lanes that agree
// on a node stay on the same path; 0 (the default): each lane's own nearer
// child first (WALK = 2 builds it as SQ_LAYOUT_BINARY_VOTE). Measured on the
// terrain's 1,048,576 rays (answers identical):
// 0.490 ms against 0.436 ms for each lane's own order; the vote costs every
// node step, and a lane outvoted takes its farther child first.
#ifndef SQ_WARP_ORDER
#define SQ_WARP_ORDER 0
#endif
// query_kernel's warp scheduling. Measured on the terrain (1,048,576
// triangles and rays, each pair by the other values alike): answers written
// and queries loaded once 1 / 4 / 8 / 16 / 24 lanes are free 705 / 641 / 625
// / 615 / 617 us; a leaf pass once 1/2, 2/3, 1/3 or 1/4 of the walking lanes
// wait at one 615 / 627 / 625 / 633 us (before the free lanes helped).
constexpr int kRefill = 16;     // free lanes (of 32) before the warp refills them
constexpr int kLeafWeight = 2;  // a leaf pass when waiting lanes x this reach the walking lanes
constexpr int kMaxStack = 96;  // deepest tree accepted (96 KB of stack per block, 144 KB for f64 scenes)

// 16-byte vectors of a record of `words` words: records longer than one
// vector are padded to whole 32-byte sectors, so that each is read with
// 32-byte loads (load_vec).
__host__ __device__ constexpr int record_vec(int words) { return words <= 4 ? 1 : (words + 7) / 8 * 2; }

// S: the scene's scalar; `words` counts 32-bit words.
template <int D, class S = float> struct NodeLayout {
  static constexpr int words = 4 * D * int(sizeof(S) / 4) + 2;  // a.lo a.hi b.lo b.hi code_a code_b
  static constexpr int vec = record_vec(words);
  static constexpr int scalars = vec * 16 / int(sizeof(S));  // S values that hold a record
};

// Four-wide records (the binary tree with every other level folded into its
// parent): up to four children's boxes, then their codes (kNoHit: an empty
// slot). Same boxes as the binary records, so the walk prunes exactly the
// subtrees the binary walk would, in half the dependent fetches.
template <int D> struct WideLayout {
  static constexpr int words = 8 * D + 4;  // c0.lo c0.hi ... c3.lo c3.hi code0 .. code3
  static constexpr int vec = record_vec(words);
};

// Quantised four-wide records: the same four-wide tree (same numbering and
// codes), each child's box stored as 8-bit steps from the record's origin
// (the lower corner of the union of its children) in a power-of-two step per
// axis, rounded outward: a stored box always contains the exact one, so its
// slab entry is never later and the walk never prunes a subtree the exact
// boxes would keep (it may visit a few more; answers are certified as for
// every near-first walk). Words: origin[D] (f32), the D step exponents
// (biased by 127, one byte each), the 8 x D step counts (child k, axis i: lo
// at byte 2Dk + i, hi at byte 2Dk + D + i), then the four codes.
template <int D> struct QuantLayout {
  static constexpr int exp_words = (D + 3) / 4;
  static constexpr int o_exp = D;
  static constexpr int o_q = D + exp_words;
  static constexpr int o_code = D + exp_words + 2 * D;
  static constexpr int words = o_code + 4;
  static constexpr int vec = record_vec(words);
};

// origin + q x 2^e, in the arithmetic both the quantiser and the walk use.
__host__ __device__ __forceinline__ float q_decode(float origin, uint32_t q, float step) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(origin, __fmul_rn(float(q), step));
#else
  volatile float m = float(q) * step;  // exact: q < 256 and step a power of two
  return origin + m;
#endif
}

__host__ __device__ __forceinline__ float q_step(uint32_t biased) {
  union { uint32_t u; float f; } v;
  v.u = biased << 23;
  return v.f;
}

__host__ __device__ __forceinline__ uint32_t q_byte(const uint32_t* words, int index) {
  return (words[index >> 2] >> (8 * (index & 3))) & 0xFFu;
}

// Quantises one four-wide record: lo/hi of child k at box + 2Dk, codes[k]
// (kNoHit: an empty slot). Writes QuantLayout<D>::words words. Non-finite
// bounds give a record of zeros (the walk reads the exact records of a scene
// with non-finite bounds).
template <int D>
__host__ __device__ void quantize_record(const float* box, const uint32_t* codes, uint32_t* out) {
  using QL = QuantLayout<D>;
  for (int w = 0; w < QL::words; ++w) out[w] = 0u;
  for (int k = 0; k < 4; ++k) out[QL::o_code + k] = codes[k];
  float plo[D], phi[D];
  bool finite = true, any = false;
  for (int i = 0; i < D; ++i) {
    plo[i] = 3.4028235e38f;
    phi[i] = -3.4028235e38f;
  }
  for (int k = 0; k < 4; ++k) {
    if (codes[k] == kNoHit) continue;
    any = true;
    for (int i = 0; i < D; ++i) {
      const float lo = box[2 * D * k + i], hi = box[2 * D * k + D + i];
      finite = finite && (lo - lo == 0.f) && (hi - hi == 0.f);  // false for inf and NaN
      plo[i] = lo < plo[i] ? lo : plo[i];
      phi[i] = hi > phi[i] ? hi : phi[i];
    }
  }
  if (!finite || !any) return;
  union { float f; uint32_t u; } cv;
  for (int i = 0; i < D; ++i) {
    cv.f = plo[i];
    out[i] = cv.u;
    // the smallest step whose 255th multiple reaches the upper corner
    uint32_t e = 1;  // biased exponent 1..254
    const float ext = phi[i] - plo[i];
    if (ext > 0.f) {
      cv.f = ext;
      const int ex = int((cv.u >> 23) & 0xFFu) - 127;  // ext in [2^ex, 2^(ex+1)) for normal ext
      int b = ex - 7 + 127;  // 255 x 2^(ex-7) < 2^(ex+1): start just below
      b = b < 1 ? 1 : (b > 254 ? 254 : b);
      e = uint32_t(b);
      while (e < 254 && q_decode(plo[i], 255u, q_step(e)) < phi[i]) ++e;
      while (e > 1 && q_decode(plo[i], 255u, q_step(e - 1)) >= phi[i]) --e;
    }
    out[QL::o_exp + (i >> 2)] |= e << (8 * (i & 3));
    const float step = q_step(e);
    for (int k = 0; k < 4; ++k) {
      if (codes[k] == kNoHit) continue;
      const float lo = box[2 * D * k + i], hi = box[2 * D * k + D + i];
      // lo: the largest q whose decoded value is <= lo (q = 0 decodes to the origin <= lo)
      float fq = (lo - plo[i]) / step;
      uint32_t ql = fq <= 0.f ? 0u : (fq >= 255.f ? 255u : uint32_t(fq));
      while (ql > 0 && q_decode(plo[i], ql, step) > lo) --ql;
      while (ql < 255 && q_decode(plo[i], ql + 1, step) <= lo) ++ql;
      // hi: the smallest q whose decoded value is >= hi (q = 255 reaches the upper corner)
      fq = (hi - plo[i]) / step;
      uint32_t qh = fq <= 0.f ? 0u : (fq >= 255.f ? 255u : uint32_t(fq));
      while (qh < 255 && q_decode(plo[i], qh, step) < hi) ++qh;
      while (qh > ql && q_decode(plo[i], qh - 1, step) >= hi) --qh;
      const int bl = 2 * D * k + i, bh = 2 * D * k + D + i;
      out[QL::o_q + (bl >> 2)] |= ql << (8 * (bl & 3));
      out[QL::o_q + (bh >> 2)] |= qh << (8 * (bh & 3));
    }
  }
}

template <int D, int N, class S = float> struct PrimLayout {
  static constexpr int payload = (N == kNarrowAabb)     ? 2 * D
                                 : (N == kNarrowTri)    ? 9
                                 : (N == kNarrowCustom) ? SQ_CUSTOM_STRIDE + 2 * D
                                                        : D + 1;
  static constexpr int id_word = payload;  // the scalar whose (low) 32 bits are the id word
  static constexpr int vec = record_vec((payload + 1) * int(sizeof(S) / 4));
  static constexpr int scalars = vec * 16 / int(sizeof(S));
};

template <int K> struct QueryLayout {
  // floats per query record: rays o,d; casts o,d,probe.min,probe.max; regions lo,hi
};

// S: the scalar of the scene and its queries (double: the crate's f64 feature,
// which has no seeds and no four-wide records).
template <class S> struct QueryParamsT {
  static constexpr int kEntryBytes = 4 + int(sizeof(S));  // a stack entry: code and slab entry
  const float4* __restrict__ nodes;
  const float4* __restrict__ wnodes;  // four-wide records (WIDE kernels)
  const float4* __restrict__ qnodes;  // quantised four-wide records (QUANT kernels; same numbering)
  uint32_t wroot;                     // the root's four-wide code
  const float4* __restrict__ prims;
  const uint64_t* __restrict__ layers;
  const uint32_t* __restrict__ sub;
  const S* __restrict__ queries;
  const S* __restrict__ max_toi_arr;
  uint32_t* counter;
  uint32_t* out_leaf;
  S* out_toi;
  uint32_t* out_sub;
  S* out_normal;
  S* out_point;
  uint32_t* out_count;
  const unsigned long long* csr_offsets;
  uint32_t* csr_leaves;
  unsigned long long* stats;
  uint32_t* query_stats;  // optional per-query counters [n][4] (u32)
  uint32_t* replay_count;  // near-first: number of uncertified queries appended to replay_list
  uint32_t* replay_list;   // near-first: their indices
  const uint32_t* q_list;  // optional: work item i is query q_list[i] ...
  const uint32_t* q_count; // ... for i < *q_count (the reference-order replay of replay_list)
  float window;            // relative window past the limit within which near-first still visits nodes
  unsigned long long mask;
  long long exclude;
  const S* root_box;  // min[D], max[D] of the root (device memory: refit updates it)
  const int32_t* seed_bucket;  // learned guide: predicted bucket per query (seeded launches)
  const uint2* buckets;        // per bucket: node code, parent record << 1 | slot (kNoHit: the root)
  const uint32_t* bucket_sibs; // per bucket, sib_stride slots (record << 1 | slot) of its ancestors' other children
  uint32_t n_buckets;
  uint32_t sib_stride;
  const int* nonfinite;   // non-zero when some node bound is not finite (device memory)
  S max_toi;
  int stack;              // traversal-stack entries per thread (dynamic shared memory)
  uint32_t root_code;
  uint32_t n;
  uint32_t k;
  int crossings;
  int fill;  // overlap: 0 count, 1 fill in ascending order, 2 fill in walk order
  int far_first;  // seeded walks: after the bucket, the crate's child order (push a, push b) instead of near-first
  // Overlap regions that visit more than visit_budget records in the count
  // pass are left to overlap_heavy_kernel (a block per region): listed in
  // heavy_list, flagged in heavy_flag (1; the fill pass skips them). With
  // keep set, the regions counted with more than kOverlapKeep results are
  // listed too (flag 2) and filled by that kernel alone.
  uint32_t* heavy_list;
  uint32_t* heavy_count;
  uint8_t* heavy_flag;
  uint32_t visit_budget;
  // Overlap: the count pass writes each region's first kOverlapKeep accepted
  // leaves here ([n][kOverlapKeep]); the fill pass copies, sorted, the
  // segment of every region with no more results instead of walking it again.
  uint32_t* keep;
  // Overlap: overlap_heavy_kernel's staged leaves (see that kernel).
  uint32_t* heavy_store;
  uint32_t* heavy_start;   // per heavy_list entry
  uint32_t* heavy_cursor;
  uint32_t heavy_cap;      // entries of heavy_store
};
using QueryParams = QueryParamsT<float>;

template <class S> __device__ __forceinline__ bool accepts(const QueryParamsT<S>& p, uint32_t id) {
  if (!p.layers) return true;
  if (p.exclude >= 0 && (unsigned long long)p.exclude == id) return false;
  return (__ldg(p.layers + id) & p.mask) != 0ull;
}

// A record of NV 16-byte vectors through the read-only path. Lanes of a warp
// read records of their own, so every load instruction costs the L1 a lookup
// per lane: 32-byte loads (sm_100) halve the lookups of 16-byte ones (terrain
// 621 -> 601 us per 1,048,576 rays). Compilers before 12.9 do not know them;
// the NVRTC that compiles a consumer's narrow phase can be older.
#if __CUDACC_VER_MAJOR__ * 100 + __CUDACC_VER_MINOR__ >= 1209
constexpr bool kWideLoads = true;
#else
constexpr bool kWideLoads = false;
#endif
template <int NV> __device__ __forceinline__ void load_vec(const float4* __restrict__ src, float* dst) {
  if constexpr (kWideLoads && NV % 2 == 0) {
#pragma unroll
    for (int j = 0; j < NV / 2; ++j) {
      float* d = dst + 8 * j;
      asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
          : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]), "=f"(d[4]), "=f"(d[5]), "=f"(d[6]), "=f"(d[7])
          : "l"(src + 2 * j));
    }
  } else {
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      float4 v = __ldg(src + j);
      dst[4 * j + 0] = v.x;
      dst[4 * j + 1] = v.y;
      dst[4 * j + 2] = v.z;
      dst[4 * j + 3] = v.w;
    }
  }
}

template <int NV> __device__ __forceinline__ void load_vec(const float4* __restrict__ src, double* dst) {
  if constexpr (kWideLoads && NV % 2 == 0) {
#pragma unroll
    for (int j = 0; j < NV / 2; ++j) {
      double* d = dst + 4 * j;
      asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
          : "=d"(d[0]), "=d"(d[1]), "=d"(d[2]), "=d"(d[3])
          : "l"(src + 2 * j));
    }
  } else {
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const double2 v = __ldg(reinterpret_cast<const double2*>(src) + j);
      dst[2 * j + 0] = v.x;
      dst[2 * j + 1] = v.y;
    }
  }
}

// A record's 32-bit words: the id word of a primitive, the child codes of a
// node (in f64 records, both in the scalar after the boxes).
__device__ __forceinline__ uint32_t word_of(float x) { return __float_as_uint(x); }
__device__ __forceinline__ uint32_t word_of(double x) { return uint32_t(__double_as_longlong(x)); }
template <int D> __device__ __forceinline__ void node_codes(const float* rec, uint32_t& a, uint32_t& b) {
  a = __float_as_uint(rec[4 * D]);
  b = __float_as_uint(rec[4 * D + 1]);
}
template <int D> __device__ __forceinline__ void node_codes(const double* rec, uint32_t& a, uint32_t& b) {
  const unsigned long long w = (unsigned long long)__double_as_longlong(rec[4 * D]);
  a = uint32_t(w);
  b = uint32_t(w >> 32);
}

// Near-first traversal visits nodes in another order than the reference, so
// its answer is certified before it counts. The reference's limit never
// drops below the global minimum hit h, and every box enclosing h's
// primitive has a slab entry no later than the entry of the primitive's own
// AABB; so when h.toi is not before that entry, the reference's walk reaches
// h whatever its order and answers h. Near-first prunes a node only when its
// entry lies past the best hit by more than a small relative window (2^-16 by
// default), which finds h whenever no hit is computed that far before the
// entry of a box enclosing its primitive. A query whose answer comes before
// its own primitive's AABB entry e still has it if no other hit lies before e:
// the reference's limit is then e or later until it reaches h (the query's
// limit has to be, and e has to lie within the window, so that every hit
// before it was seen). Otherwise the query is not certified: it is appended to
// a list that a second launch answers again in the reference order, one lane
// per query (1,048,576 rays against 100,000 balls: 489 queries without the
// second rule, 87 with it).
__device__ __forceinline__ float near_limit(float limit, float window) {
  return __fadd_rn(limit, __fadd_rn(__fmul_rn(fabsf(limit), window), 0x1p-20f));
}
__device__ __forceinline__ double near_limit(double limit, float window) {
  return __dadd_rn(limit, __dadd_rn(__dmul_rn(fabs(limit), double(window)), 0x1p-20));
}

// The slab entry of a primitive's own AABB for a ray or sweep (computed only
// when the primitive is hit): a hit before it is a hit before every box that
// encloses the primitive.
template <int D, int N, bool CAST, class S>
__device__ __forceinline__ S prim_entry(const S* rec, const RayPre<D, S>& r, const S* pmin, const S* pmax, bool fast) {
  S lo[D], hi[D], te;
  int ax;
  const S inf = Lim<S>::inf();
  if constexpr (N == kNarrowTri) {
    tri_aabb(rec, rec + 3, rec + 6, lo, hi);
  } else if constexpr (N == kNarrowCustom) {
#pragma unroll
    for (int i = 0; i < D; ++i) {
      lo[i] = rec[SQ_CUSTOM_STRIDE + i];
      hi[i] = rec[SQ_CUSTOM_STRIDE + D + i];
    }
  } else if constexpr (N == kNarrowSphere || N == kNarrowSphereNear) {
#pragma unroll
    for (int i = 0; i < D; ++i) {
      lo[i] = fsub(rec[i], rec[D]);
      hi[i] = fadd(rec[i], rec[D]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < D; ++i) {
      lo[i] = rec[i];
      hi[i] = rec[D + i];
    }
  }
  if constexpr (CAST) {
    if (fast) slab_grown_fast<D>(r, lo, hi, pmin, pmax, inf, te);
    else slab_grown<D>(r, lo, hi, pmin, pmax, inf, te, ax);
  } else {
    if (fast) slab_fast<D>(r, lo, hi, inf, te);
    else slab<D>(r, lo, hi, inf, te, ax);
  }
  return te;
}

// One primitive's ray test (QueryGeometry::test_ray for the built-in providers).
template <int D, int N, class S>
__device__ __forceinline__ bool narrow_ray(const S* rec, const RayPre<D, S>& r, S max_toi, S& t, S* n) {
  if constexpr (N == kNarrowAabb) {
    int axis;
    if (!slab<D>(r, rec, rec + D, max_toi, t, axis)) return false;
    entry_normal<D>(r.d, axis, n);
    return true;
  } else if constexpr (N == kNarrowSphere || N == kNarrowSphereNear) {
    return ray_ball<D, N == kNarrowSphere>(r.o, r.d, rec, rec[D], max_toi, t, n);
  } else if constexpr (N == kNarrowCustom) {
#ifdef SQ_RTC_CUSTOM
    const uint32_t leaf = word_of(rec[PrimLayout<D, N>::id_word]) & ~kLeafBit;
    if (!sq_narrow(rec, leaf, r.o, r.d, max_toi, &t, n)) return false;
    return !(t > max_toi);
#else
    return false;
#endif
  } else {
    if (!ray_triangle(r.o, r.d, rec, rec + 3, rec + 6, t)) return false;
    if (t > max_toi) return false;
    tri_normal(rec, rec + 3, rec + 6, n);
    return true;
  }
}

// One primitive's swept-probe test (QueryGeometry::test_shape_cast).
template <int D, int N, class S>
__device__ __forceinline__ bool narrow_cast(const S* rec, const RayPre<D, S>& r, const S* pmin, const S* pmax,
                                            S max_toi, S& t, S* n) {
  if constexpr (N == kNarrowAabb) {
    int axis;
    if (!slab_grown<D>(r, rec, rec + D, pmin, pmax, max_toi, t, axis)) return false;
    entry_normal<D>(r.d, axis, n);
    return true;
  } else if constexpr (N == kNarrowSphere || N == kNarrowSphereNear) {
    return ray_ball<D, N == kNarrowSphere>(r.o, r.d, rec, fadd(rec[D], pmax[0]), max_toi, t, n);
  } else {
    S lo[3], hi[3];
    tri_aabb(rec, rec + 3, rec + 6, lo, hi);
    int axis;
    if (!slab_grown<3>(r, lo, hi, pmin, pmax, max_toi, t, axis)) return false;
    entry_normal<3>(r.d, axis, n);
    return true;
  }
}

// One primitive's overlap test (QueryGeometry::test_overlap): the box itself,
// point_to_aabb <= radius for balls (tests/shape_overlap.rs:59-72,113-115),
// the triangle's AABB for triangles.
template <int D, int N, class S>
__device__ __forceinline__ bool narrow_overlap(const S* rec, const S* qlo, const S* qhi) {
  if constexpr (N == kNarrowAabb) {
    return box_overlap<D>(rec, rec + D, qlo, qhi);
  } else if constexpr (N == kNarrowSphere || N == kNarrowSphereNear) {
    S d2 = S(0);
#pragma unroll
    for (int i = 0; i < D; ++i) {
      S c = rec[i];
      S v = (c < qlo[i]) ? fsub(qlo[i], c) : ((c > qhi[i]) ? fsub(c, qhi[i]) : S(0));
      d2 = fadd(d2, fmul(v, v));
    }
    return fsqrt(d2) <= rec[D];
  } else {
    S lo[3], hi[3];
    tri_aabb(rec, rec + 3, rec + 6, lo, hi);
    return box_overlap<3>(lo, hi, qlo, qhi);
  }
}

// Sorted insertion into query q's bounded hit list (hit_ordering, stable:
// an equal key goes after the entries already present). `count` is the full
// number of hits so far; the first min(count, k) entries are kept.
template <int D, class S>
__device__ __forceinline__ void list_put(uint32_t k, uint32_t* o_leaf, S* o_toi, uint32_t* o_sub, S* o_nrm,
                                         uint32_t q, uint32_t& count, S t, uint32_t leaf, uint32_t subv,
                                         const S* n) {
  uint32_t m = count < k ? count : k;
  ++count;
  if (k == 0) return;
  const size_t base = size_t(q) * k;
  if (m == k) {
    if (!hit_before(t, leaf, o_toi[base + k - 1], o_leaf[base + k - 1])) return;
    m = k - 1;
  }
  uint32_t j = m;
  while (j > 0 && hit_before(t, leaf, o_toi[base + j - 1], o_leaf[base + j - 1])) {
    o_toi[base + j] = o_toi[base + j - 1];
    o_leaf[base + j] = o_leaf[base + j - 1];
    if (o_sub) o_sub[base + j] = o_sub[base + j - 1];
    if (o_nrm)
#pragma unroll
      for (int i = 0; i < D; ++i) o_nrm[(base + j) * D + i] = o_nrm[(base + j - 1) * D + i];
    --j;
  }
  o_toi[base + j] = t;
  o_leaf[base + j] = leaf;
  if (o_sub) o_sub[base + j] = subv;
  if (o_nrm)
#pragma unroll
    for (int i = 0; i < D; ++i) o_nrm[(base + j) * D + i] = n[i];
}

template <int D, class S>
__device__ __forceinline__ void list_insert(const QueryParamsT<S>& p, uint32_t q, uint32_t& count, S t, uint32_t leaf,
                                            const S* n) {
  list_put<D>(p.k, p.out_leaf, p.out_toi, p.out_sub, p.out_normal, q, count, t, leaf,
              p.sub ? __ldg(p.sub + leaf) : kNoHit, n);
}

// Per-lane traversal state of one query.
template <int D, int K, class S> struct Lane {
  RayPre<D, S> r;
  S pmin[D], pmax[D];
  S limit;       // nodes whose entry lies past this are pruned (near-first: the best hit plus the window)
  uint32_t best_pos; // primitive position of the best hit (its certification and normal)
  uint32_t q;
  uint32_t code;
  S code_t;      // entry of the node in code (postponed-leaf walks re-check it after a leaf)
  uint32_t top_code; // postponed-leaf walks: the stack's top entry, held in registers
  S top_t;
  bool has_top;
  int sp;
  bool fast;
  uint32_t best_leaf;
  S best_t;
  S second_t;    // near-first: the nearest of the query's other hits
  S best_n[D];   // consumer narrow phases only
  uint32_t count;
  unsigned long long csr_base;
  uint32_t v_nodes, v_nar, v_hit;
};

// Resident blocks per SM that query_kernel's registers are held to: what the
// walk itself needs (the code that runs once per query or once per launch may
// spill). At D = 3 and 1,048,576 terrain rays, 7 / 8 / 9 / 10 blocks measured
// 512 / 464 / 441 / 483 us (nine: 56 registers, no spills; ten: 48 registers,
// 32 bytes spilled). Longer rays and records (D = 4 and 6, casts, four-wide
// records) need more registers each. Doubles are left to the compiler (200,000
// boxes, 100,001 host rays: 708 us at the natural 88 registers, 691 / 699 / 709
// at 4 / 5 / 6 blocks).
__host__ __device__ constexpr int resident_blocks(int D, int kind, bool stats, bool wide, bool f64) {
  if (stats || f64) return 1;
  if (wide) return D <= 3 ? 8 : (D == 4 ? 6 : 5);
  if (D <= 3 || kind == kOverlap) return 9;
  if (kind == kCastNearest || kind == kCastAll) return D == 4 ? 7 : 5;
  if (D == 6 && kind == kRayAll) return 5;  // 9,081 boxes, 78,852 rays: 55.8 / 53.5 / 52.9 / 49.6 us at 8 / 7 / 6 / 5 blocks
  return D == 4 ? 8 : 7;
}

// The persistent query kernel. Each warp keeps up to 32 queries in flight and
// its lanes step together: a pass tests one record for every lane at an
// interior node, or the primitives of one leaf for every lane at a leaf,
// whichever more lanes wait for (a lane that reaches its leaf early waits for
// company), and the lanes whose queries have ended are refilled together from
// the shared counter (one atomic per refill). A lane visits what it would
// visit alone, in the same order. On the terrain 16.3 of 32 threads are active
// per warp instruction (7.5 when each lane descended to its own leaf before
// the warp tested leaves); the kernel now issues 2.57 instructions per cycle
// and SM, with the L1's data pipe 69% busy.
//
// A launch ends on its longest queries, dependent chains of hundreds of
// fetches at some 0.3 us each. HELP walks split them over the lanes that have
// no query left (see the tail of the kernel), and a batch smaller than the
// grid's lanes is dealt out thinly over every warp, so that each query has
// free lanes beside it from the start. Both together with the passes above:
// terrain 632 -> 441 us per 1,048,576 rays, 100,003 filtered ball casts 268
// -> 150 us, 256 rays against 10,000 boxes 135 -> 26 us.
//
// SEED (nearest rays only): the learned guide's predicted bucket, a subtree
// at a fixed depth, is searched first; its nearest hit becomes the limit for
// the rest of the tree, which is exactly the other children of the bucket's
// ancestors: they wait on the stack from the start and are walked after the
// bucket (no ancestor's record is read twice, so a right seed never costs
// more box tests than the plain walk). The answer is certified exactly as in
// near-first, so it is the reference's whatever the seed.
// WIDE (near-first nearest rays, no counters, no seed): the walk reads the
// four-wide records; a step tests up to four children, goes to the nearest
// and stacks the others farthest first.
// WALK (near-first nearest rays over child-pair records, no counters): 1 =
// postponed leaves with the stack's top entry held in registers; 2 = child
// order by warp vote.
template <int D, int N, int K, bool REF, bool STATS, bool SEED = false, bool WIDE = false, bool QUANT = false,
          int WALK = 0, class S = float>
__global__ void __launch_bounds__(kThreads, resident_blocks(D, K, STATS, WIDE, sizeof(S) == 8)) query_kernel(const QueryParamsT<S> p) {
  static_assert(!WIDE || (K == kRayNearest && !REF && !STATS && !SEED), "four-wide walks serve near-first rays only");
  static_assert(!QUANT || WIDE, "quantised records are a four-wide layout");
  constexpr bool kNearest = (K == kRayNearest || K == kCastNearest);
  constexpr bool kCast = (K == kCastNearest || K == kCastAll);
  constexpr bool kList = (K == kRayAll || K == kCastAll);
  constexpr int QW = kCast ? 4 * D : 2 * D;
  using PL = PrimLayout<D, N, S>;
  using NL = NodeLayout<D, S>;
  using WL = WideLayout<D>;
  constexpr uint32_t FULL = 0xffffffffu;

  extern __shared__ __align__(16) uint32_t smem[];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  S* s_t = reinterpret_cast<S*>(smem);
  uint32_t* s_code = reinterpret_cast<uint32_t*>(s_t + p.stack * kThreads);
  const uint32_t lt_mask = (1u << lane) - 1u;
  const bool scene_finite = p.nonfinite ? (*p.nonfinite == 0) : true;

  unsigned long long c_vis = 0, c_nar = 0, c_hit = 0;
  Lane<D, K, S> L;
  const uint32_t n_queries = p.q_count ? *p.q_count : p.n;

  constexpr bool DETECT = kNearest && !REF;
  // Postponed leaves for the certified near-first walks (their answers do
  // not depend on the order of the visits); the counting and reference-order
  // walks keep the crate's sequence.
  constexpr bool SPEC = (SQ_POSTPONE_LEAVES || WALK == 1) && DETECT && !STATS && !WIDE;
  constexpr bool kRegTop = SQ_REG_TOP || WALK == 1;
  // Idle lanes help where the answer does not depend on the order of the
  // visits and no counter reports them.
  constexpr bool HELP = DETECT && !STATS && !SPEC;
  const S kInf = Lim<S>::inf();

  // Box test of one child (or the root) against the lane's query: the slab
  // without the limit, then the entry against the limit (the same verdict as
  // the reference's slab clipped to the limit, aabb.rs:118-148).
  auto test_box = [&](const S* lo, const S* hi, S& te) -> bool {
    if constexpr (K == kOverlap) {
      te = S(0);
      return box_overlap<D>(lo, hi, L.r.o, L.r.d);  // region lo / hi sit in o / d
    } else {
      bool geo;
      int ax;
      if constexpr (kCast) {
        geo = L.fast ? slab_grown_fast<D>(L.r, lo, hi, L.pmin, L.pmax, kInf, te)
                     : slab_grown<D>(L.r, lo, hi, L.pmin, L.pmax, kInf, te, ax);
      } else {
        geo = L.fast ? slab_fast<D>(L.r, lo, hi, kInf, te) : slab<D>(L.r, lo, hi, kInf, te, ax);
      }
      return geo && te <= L.limit;
    }
  };

  // Pops the next waiting child whose entry still lies within the limit
  // (exactly the reference's slab verdict at pop time). False: stack empty.
  auto pop = [&](int lo) -> bool {
    if constexpr (SPEC && kRegTop) {
      if (L.has_top) {
        L.has_top = false;
        L.code = L.top_code;
        L.code_t = L.top_t;
        if (L.top_t <= L.limit) return true;
      }
    }
    while (L.sp > lo) {
      --L.sp;
      L.code = s_code[L.sp * kThreads + tid];
      const S t = s_t[L.sp * kThreads + tid];
      L.code_t = t;
      if (!kNearest || t <= L.limit) return true;
    }
    return false;
  };

  auto finish = [&]() {
    const uint32_t q = L.q;
    S nrm[D];
    if constexpr (kNearest) {
#pragma unroll
      for (int i = 0; i < D; ++i) nrm[i] = N == kNarrowCustom ? L.best_n[i] : S(0);
      if (L.best_leaf != kNoHit && ((DETECT && N != kNarrowAabb) || (N != kNarrowCustom && p.out_normal))) {
        S rec[PL::scalars];
        load_vec<PL::vec>(p.prims + size_t(L.best_pos) * PL::vec, rec);
        // Certify the answer: not before its own primitive's AABB entry.
        if constexpr (DETECT && N != kNarrowAabb) {
          const S te = prim_entry<D, N, kCast>(rec, L.r, L.pmin, L.pmax, L.fast);
          const S mt = p.max_toi_arr ? p.max_toi_arr[q] : p.max_toi;
          if (L.best_t < te && !(te <= mt && te <= near_limit(L.best_t, p.window) && te <= L.second_t))
            p.replay_list[atomicAdd(p.replay_count, 1u)] = q;
        }
        // The best hit's normal, once per query: the same test of the same
        // primitive bounded by the hit itself.
        if constexpr (N != kNarrowCustom) {
          if (p.out_normal) {
            S t;
            if constexpr (kCast) narrow_cast<D, N>(rec, L.r, L.pmin, L.pmax, L.best_t, t, nrm);
            else if constexpr (N == kNarrowTri) tri_normal(rec, rec + 3, rec + 6, nrm);
            else narrow_ray<D, N>(rec, L.r, L.best_t, t, nrm);
          }
        }
      }
    }
    if constexpr (kNearest) {
      p.out_leaf[q] = L.best_leaf;
      if (p.out_toi) p.out_toi[q] = L.best_t;
      if (p.out_sub) p.out_sub[q] = (L.best_leaf != kNoHit && p.sub) ? __ldg(p.sub + L.best_leaf) : kNoHit;
      if (p.out_normal) {
#pragma unroll
        for (int i = 0; i < D; ++i) p.out_normal[size_t(q) * D + i] = nrm[i];
      }
      if (p.out_point) {
        S pt[D];
        if (L.best_leaf != kNoHit) {
          ray_at<D>(L.r.o, L.r.d, L.best_t, pt);
        } else {
#pragma unroll
          for (int i = 0; i < D; ++i) pt[i] = S(0);
        }
#pragma unroll
        for (int i = 0; i < D; ++i) p.out_point[size_t(q) * D + i] = pt[i];
      }
    } else if constexpr (kList) {
      p.out_count[q] = L.count;  // entries past min(count, k) are left as they were
    } else {
      if (!p.fill) {
        p.out_count[q] = L.count;
        // A counted region with more results than the kept leaves (and not
        // given up on) is filled by the block-per-region kernel too, so the
        // fill pass walks no region again on one lane (flag 2: counted).
        if (p.heavy_list && p.keep && L.count > kOverlapKeep && L.v_nar <= p.visit_budget) {
          p.heavy_flag[q] = 2;
          p.heavy_list[atomicAdd(p.heavy_count, 1u)] = q;
        }
      }
    }
    if (STATS) {
      c_vis += L.v_nodes;
      c_nar += L.v_nar;
      c_hit += L.v_hit;
      if (p.query_stats) {
        p.query_stats[size_t(q) * 4 + 0] = L.v_nodes;
        p.query_stats[size_t(q) * 4 + 1] = L.v_nodes;
        p.query_stats[size_t(q) * 4 + 2] = L.v_nar;
        p.query_stats[size_t(q) * 4 + 3] = L.v_hit;
      }
    }
  };

  // Loads query q and tests the root. False when the query is already done.
  auto start = [&](uint32_t q) -> bool {
    L.q = q;
    const S* src = p.queries + size_t(q) * QW;
#pragma unroll
    for (int i = 0; i < D; ++i) {
      L.r.o[i] = src[i];
      L.r.d[i] = src[D + i];
      if constexpr (kCast) {
        L.pmin[i] = src[2 * D + i];
        L.pmax[i] = src[3 * D + i];
      }
    }
    L.limit = p.max_toi_arr ? p.max_toi_arr[q] : p.max_toi;
    if constexpr (K != kOverlap) {
      ray_prep<D>(L.r);
      bool f = scene_finite && L.r.par == 0u && !isnan(L.limit);
#pragma unroll
      for (int i = 0; i < D; ++i) {
        f = f && isfinite(L.r.o[i]) && isfinite(L.r.d[i]);
        if constexpr (kCast) f = f && isfinite(L.pmin[i]) && isfinite(L.pmax[i]);
      }
      L.fast = f;
    } else {
      L.fast = false;
    }
    L.best_leaf = kNoHit;
    L.best_t = S(0);
    L.second_t = kInf;
    if constexpr (N == kNarrowCustom) {
#pragma unroll
      for (int i = 0; i < D; ++i) L.best_n[i] = S(0);
    }
    L.count = 0;
    L.csr_base = 0;
    if constexpr (K == kOverlap) {
      if (p.fill) L.csr_base = p.csr_offsets[q];
      if (p.fill && p.heavy_flag && p.heavy_flag[q]) return false;  // filled by the block-per-region kernel
      if (p.fill && p.keep) {
        // Every result of a region with at most kOverlapKeep of them was kept
        // by the count pass (the same walk finds the same leaves): written
        // ascending, with no second walk. Most regions have none.
        const uint32_t c = uint32_t(p.csr_offsets[q + 1] - L.csr_base);
        if (c <= kOverlapKeep) {
          if (c) {
            const uint4 k4 = __ldcs(reinterpret_cast<const uint4*>(p.keep) + q);
            uint32_t v0 = k4.x, v1 = c > 1 ? k4.y : kNoHit, v2 = c > 2 ? k4.z : kNoHit, v3 = c > 3 ? k4.w : kNoHit;
            const auto cas = [](uint32_t& a, uint32_t& b) {
              const uint32_t lo = min(a, b);
              b = max(a, b);
              a = lo;
            };
            cas(v0, v1);  // sorting network on four: (0,1) (2,3) (0,2) (1,3) (1,2)
            cas(v2, v3);
            cas(v0, v2);
            cas(v1, v3);
            cas(v1, v2);
            uint32_t* out = p.csr_leaves + L.csr_base;
            out[0] = v0;
            if (c > 1) out[1] = v1;
            if (c > 2) out[2] = v2;
            if (c > 3) out[3] = v3;
          }
          return false;
        }
      }
    }
    L.v_nodes = STATS ? 1u : 0u;
    L.v_nar = 0;
    L.v_hit = 0;
    L.sp = 0;
    L.has_top = false;
    L.code = WIDE ? p.wroot : p.root_code;
    S lo[D], hi[D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
      lo[i] = p.root_box[i];
      hi[i] = p.root_box[D + i];
    }
    S te;
    const bool hit_root = test_box(lo, hi, te);
    L.code_t = te;
    if constexpr (SEED) {
      const int32_t bk = p.seed_bucket[q];
      if (hit_root && bk >= 0 && uint32_t(bk) < p.n_buckets) {
        const uint2 e = __ldg(p.buckets + bk);
        if (e.x != p.root_code) {
          const S* box = (e.y == kNoHit) ? p.root_box
                                             : reinterpret_cast<const float*>(p.nodes + size_t(e.y >> 1) * NL::vec) +
                                                   (e.y & 1u) * 2 * D;
          S blo[D], bhi[D], tb;
#pragma unroll
          for (int i = 0; i < D; ++i) {
            blo[i] = box[i];
            bhi[i] = box[D + i];
          }
          if (STATS) L.v_nodes += 1;
          if (test_box(blo, bhi, tb)) {
            // The bucket goes first. The siblings of its ancestors wait on
            // the stack, the root's child deepest, so the bucket's nearest
            // neighbours in the tree come up first; each is tested against
            // the ray now and against the (shrunk) limit when popped. Their
            // records are independent loads, not a dependent descent.
            const uint32_t* sibs = p.bucket_sibs + size_t(bk) * p.sib_stride;
            for (uint32_t i = 0; i < p.sib_stride; ++i) {
              const uint32_t sl = __ldg(sibs + i);
              if (sl == kNoHit) break;
              S rec[NL::scalars];
              load_vec<NL::vec>(p.nodes + size_t(sl >> 1) * NL::vec, rec);
              const bool second = (sl & 1u) != 0u;
              S slo[D], shi[D];
#pragma unroll
              for (int k = 0; k < D; ++k) {
                slo[k] = second ? rec[2 * D + k] : rec[k];
                shi[k] = second ? rec[3 * D + k] : rec[D + k];
              }
              const uint32_t sc = __float_as_uint(second ? rec[4 * D + 1] : rec[4 * D]);
              S ts;
              if (STATS) L.v_nodes += 1;
              if (test_box(slo, shi, ts)) {
                s_code[L.sp * kThreads + tid] = sc;
                s_t[L.sp * kThreads + tid] = ts;
                ++L.sp;
              }
            }
            L.code = e.x;
            L.code_t = tb;
          }
        }
      }
    }
    return hit_root;
  };

  // A hit of the lane's query: kept when it is before the best one.
  auto take_hit = [&](S t, uint32_t id, uint32_t pos) -> bool {
    const bool first = L.best_leaf == kNoHit || hit_before(t, id, L.best_t, L.best_leaf);
    if constexpr (DETECT && N != kNarrowAabb) {
      // The nearest of the other hits; a NaN marks the query uncertified.
      const S other = first ? (L.best_leaf == kNoHit ? kInf : L.best_t) : t;
      if (!(other >= L.second_t)) L.second_t = other == other ? other : -kInf;
    }
    if (first) {
      L.best_leaf = id;
      L.best_t = t;
      L.best_pos = pos;
      L.limit = DETECT ? near_limit(t, p.window) : t;
    }
    return first;
  };

  // Tests the primitive record at position pos. True: the last of its leaf.
  auto prim = [&](const S* rec, uint32_t pos) -> bool {
    {
      const uint32_t idw = word_of(rec[PL::id_word]);
      const uint32_t id = idw & ~kLeafBit;
      if (accepts(p, id)) {
        if constexpr (K == kOverlap) {
          if (narrow_overlap<D, N>(rec, L.r.o, L.r.d)) {
            if (!p.fill && p.keep && L.count < kOverlapKeep) p.keep[size_t(L.q) * kOverlapKeep + L.count] = id;
            if (p.fill == 2) {
              // appended in walk order; a segmented sort orders each segment afterwards
              p.csr_leaves[L.csr_base + L.count] = id;
            } else if (p.fill) {
              // ascending leaf order within the query's CSR segment, kept by
              // insertion (the allocation-free path, which has no sort scratch)
              uint32_t j = L.count;
              while (j > 0 && p.csr_leaves[L.csr_base + j - 1] > id) {
                p.csr_leaves[L.csr_base + j] = p.csr_leaves[L.csr_base + j - 1];
                --j;
              }
              p.csr_leaves[L.csr_base + j] = id;
            }
            ++L.count;
          }
        } else {
          if (STATS) L.v_nar += 1;
          S t, nrm[D];
          if constexpr (K == kRayNearest || K == kCastNearest) {
            bool h;
            if constexpr (K == kRayNearest) h = narrow_ray<D, N>(rec, L.r, L.limit, t, nrm);
            else h = narrow_cast<D, N>(rec, L.r, L.pmin, L.pmax, L.limit, t, nrm);
            if (h) {
              if (STATS) L.v_hit += 1;
              if (take_hit(t, id, pos)) {
                if constexpr (N == kNarrowCustom) {  // a consumer's normal is the one its own test gave
#pragma unroll
                  for (int i = 0; i < D; ++i) L.best_n[i] = nrm[i];
                }
              }
            }
          } else if constexpr (K == kRayAll) {
            if constexpr (N == kNarrowSphere) {
              if (p.crossings) {
                // Both roots of the unbounded ray (tests/crossings.rs:505-521).
                S oc[D];
#pragma unroll
                for (int i = 0; i < D; ++i) oc[i] = fsub(L.r.o[i], rec[i]);
                const S b = pdot<D>(oc, L.r.d);
                const S disc = fsub(fmul(b, b), fsub(pdot<D>(oc, oc), fmul(rec[D], rec[D])));
                if (!(disc < S(0))) {
                  const S sq = fsqrt(disc);
                  const S roots[2] = {fsub(-b, sq), fadd(-b, sq)};
#pragma unroll
                  for (int j = 0; j < 2; ++j) {
                    const S tt = roots[j];
                    if (tt >= S(0) && tt <= L.limit) {
                      S pt[D];
                      ray_at<D>(L.r.o, L.r.d, tt, pt);
#pragma unroll
                      for (int i = 0; i < D; ++i) nrm[i] = fsub(pt[i], rec[i]);
                      normalize_or_zero<D>(nrm);
                      if (STATS) L.v_hit += 1;
                      list_insert<D>(p, L.q, L.count, tt, id, nrm);
                    }
                  }
                }
              } else if (narrow_ray<D, N>(rec, L.r, L.limit, t, nrm)) {
                if (STATS) L.v_hit += 1;
                list_insert<D>(p, L.q, L.count, t, id, nrm);
              }
            } else {
              bool listed = false;
#ifdef SQ_RTC_CROSSINGS
              if constexpr (N == kNarrowCustom) {
                if (p.crossings) {
                  // Every crossing the consumer emits is listed, as bvh.rs:309-315 pushes them.
                  auto emit = [&](S tt, const S* nn) {
                    if (STATS) L.v_hit += 1;
                    list_insert<D>(p, L.q, L.count, tt, id, nn);
                  };
                  sq_narrow_crossings(rec, id, L.r.o, L.r.d, L.limit, emit);
                  listed = true;
                }
              }
#endif
              if (!listed && narrow_ray<D, N>(rec, L.r, L.limit, t, nrm)) {
                if (STATS) L.v_hit += 1;
                list_insert<D>(p, L.q, L.count, t, id, nrm);
              }
            }
          } else {  // kCastAll
            if (narrow_cast<D, N>(rec, L.r, L.pmin, L.pmax, L.limit, t, nrm)) list_insert<D>(p, L.q, L.count, t, id, nrm);
          }
        }
      }
      return (idw & kLeafBit) != 0u;
    }
  };
  // Tests the primitives of a leaf.
  auto leaf = [&](uint32_t code) {
    for (uint32_t pos = code & ~kLeafBit;; ++pos) {
      S rec[PL::scalars];
      load_vec<PL::vec>(p.prims + size_t(pos) * PL::vec, rec);
      if (prim(rec, pos)) break;
    }
  };

  // One record of the node in L.code: its overlapping children. True: the
  // query has nothing left to visit (its stack is empty down to lo).
  auto node_step = [&](int lo) -> bool {
    if constexpr (WIDE) {
      float t4[4];
      uint32_t c4[4];
      bool exact = true;
      if constexpr (QUANT) {
        if (scene_finite) {
          // Decode each child's box (rounded outward) and test it.
          using QL = QuantLayout<D>;
          float qf[QL::vec * 4];
          load_vec<QL::vec>(p.qnodes + size_t(L.code) * QL::vec, qf);
          uint32_t qw[QL::vec * 4];
#pragma unroll
          for (int w = 0; w < QL::vec * 4; ++w) qw[w] = __float_as_uint(qf[w]);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            c4[k] = qw[QL::o_code + k];
            S lo[D], hi[D];
#pragma unroll
            for (int i = 0; i < D; ++i) {
              const float step = q_step(q_byte(qw + QL::o_exp, i));
              lo[i] = q_decode(qf[i], q_byte(qw + QL::o_q, 2 * D * k + i), step);
              hi[i] = q_decode(qf[i], q_byte(qw + QL::o_q, 2 * D * k + D + i), step);
            }
            S te = kInf;
            if (c4[k] == kNoHit || !test_box(lo, hi, te)) {
              c4[k] = kNoHit;
              te = kInf;
            }
            t4[k] = te;
          }
          exact = false;
        }
      }
      if (exact) {
        S rec[WL::vec * 4];
        load_vec<WL::vec>(p.wnodes + size_t(L.code) * WL::vec, rec);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          c4[i] = __float_as_uint(rec[8 * D + i]);
          S te = kInf;
          if (c4[i] == kNoHit || !test_box(rec + 2 * D * i, rec + 2 * D * i + D, te)) {
            c4[i] = kNoHit;
            te = kInf;
          }
          t4[i] = te;
        }
      }
      // Ascending entry order (a five-comparator network); misses sort last.
      auto cswap = [&](int a, int b) {
        if (t4[b] < t4[a]) {
          const float t = t4[a];
          t4[a] = t4[b];
          t4[b] = t;
          const uint32_t c = c4[a];
          c4[a] = c4[b];
          c4[b] = c;
        }
      };
      cswap(0, 1);
      cswap(2, 3);
      cswap(0, 2);
      cswap(1, 3);
      cswap(1, 2);
#pragma unroll
      for (int i = 3; i >= 1; --i) {
        if (c4[i] != kNoHit) {
          s_code[L.sp * kThreads + tid] = c4[i];
          s_t[L.sp * kThreads + tid] = t4[i];
          ++L.sp;
        }
      }
      if (c4[0] != kNoHit) {
        L.code = c4[0];
      } else {
        return !pop(lo);
      }
      return false;
    }
    S rec[NL::scalars];
    load_vec<NL::vec>(p.nodes + size_t(L.code) * NL::vec, rec);
    uint32_t ca, cb;
    node_codes<D>(rec, ca, cb);
    S ta, tb;
    const bool pa = test_box(rec, rec + D, ta);
    const bool pb = test_box(rec + 2 * D, rec + 3 * D, tb);
    if (STATS) L.v_nodes += 2;
    if constexpr (K == kOverlap) {
      // A region heavier than the budget goes to the block-per-region
      // kernel instead of holding the launch's tail on one thread.
      if (p.heavy_list && !p.fill && ++L.v_nar > p.visit_budget) {
        p.heavy_flag[L.q] = 1;
        p.heavy_list[atomicAdd(p.heavy_count, 1u)] = L.q;
        return true;
      }
    }
    if (pa && pb) {
      // Reference order: child_a waits, child_b goes first. Near-first:
      // the smaller entry goes first.
      bool a_first = (REF || !kNearest || (SEED && p.far_first)) ? false : (ta <= tb);
      if constexpr ((SQ_WARP_ORDER || WALK == 2) && DETECT && !WIDE) {
        const bool voter = !(SEED && p.far_first);
        const uint32_t voters = __ballot_sync(__activemask(), voter);
        if (voter) {
          const uint32_t same = __match_any_sync(voters, L.code);
          const uint32_t yes = __ballot_sync(voters, a_first) & same;
          a_first = 2 * __popc(yes) >= __popc(same);
        }
      }
      s_code[L.sp * kThreads + tid] = a_first ? cb : ca;
      s_t[L.sp * kThreads + tid] = a_first ? tb : ta;
      ++L.sp;
      L.code = a_first ? ca : cb;
    } else if (pa) {
      L.code = ca;
    } else if (pb) {
      L.code = cb;
    } else {
      return !pop(lo);
    }
    return false;
  };

  // The warp steps together: each pass either tests one record for every lane
  // at an interior node or one leaf for every lane at a leaf, whichever more
  // lanes wait for, so a lane that reaches its leaf early waits for company
  // instead of running its primitives in a nearly empty warp. A lane whose
  // query ends keeps its answer until kRefill lanes are free; then the answers
  // are written and the next queries loaded together.
  const uint32_t warps = gridDim.x * (kThreads / 32);
  const int width = int(min(32u, max(1u, (n_queries + warps - 1) / warps)));
  const uint32_t width_mask = width >= 32 ? FULL : (1u << width) - 1u;
  const int refill = max(1, width * kRefill / 32);
  bool live = false;       // the lane walks a query
  bool held = false;       // the lane's query has ended, its answer is not written yet
  bool exhausted = false;  // no query is left to take (the same for the whole warp)
  // One pass over the walking lanes; a lane whose query has nothing left above
  // stack entry lo stops walking.
  auto step = [&](uint32_t live_mask, int lo) {
    const bool at_leaf = live && (L.code & kLeafBit);
    bool more = true;
    const uint32_t leaf_mask = __ballot_sync(FULL, at_leaf);
    if (__popc(leaf_mask) * kLeafWeight >= __popc(live_mask)) {
      if (at_leaf) {
        leaf(L.code);
        more = pop(lo);
      }
    } else if (live && !at_leaf) {
      more = !node_step(lo);
    }
    if (!more) {
      live = false;
      held = true;
    }
  };
  for (;;) {
    uint32_t live_mask = __ballot_sync(FULL, live);
    const uint32_t idle_mask = width_mask & ~live_mask;
    const int idle = __popc(idle_mask);
    if (live_mask == 0u || (!exhausted && idle >= refill)) {
      if (held) {
        finish();
        held = false;
      }
      if (exhausted) break;  // no lane walks and none holds an answer
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(p.counter, uint32_t(idle));
      base = __shfl_sync(FULL, base, 0);
      if ((idle_mask >> lane) & 1u) {
        const uint32_t q = base + uint32_t(__popc(idle_mask & lt_mask));
        if (q < n_queries) {
          live = start(p.q_list ? p.q_list[q] : q);
          held = !live;
        }
      }
      // A batch smaller than the grid's lanes is dealt out in one round.
      exhausted = width < 32 || base + uint32_t(idle) >= n_queries;
      if (HELP && exhausted) break;
      live_mask = __ballot_sync(FULL, live);
      if (live_mask == 0u) continue;
    }
    if constexpr (SPEC) {
      if (live) {
        // Postponed leaves (Aila and Laine's speculative traversal): a lane
        // that reaches a leaf holds it and keeps descending from the next
        // waiting node until every live lane of the warp holds a leaf or
        // has nothing left, so the leaf tests below run with the warp
        // together. The extra nodes are visited with the limit as it stood,
        // which only adds work: near-first answers are certified whatever
        // the order of the visits.
        uint32_t pend = kNoHit;
        bool empty = false;  // nothing left to walk after pend
        for (;;) {
          if (!empty) {
            if (L.code & kLeafBit) {
              if (pend == kNoHit) {
                pend = L.code;
                if (!pop(0)) empty = true;
              }
            } else {
              S rec[NL::scalars];
              load_vec<NL::vec>(p.nodes + size_t(L.code) * NL::vec, rec);
              const uint32_t ca = __float_as_uint(rec[4 * D]);
              const uint32_t cb = __float_as_uint(rec[4 * D + 1]);
              S ta, tb;
              const bool pa = test_box(rec, rec + D, ta);
              const bool pb = test_box(rec + 2 * D, rec + 3 * D, tb);
              if (pa && pb) {
                const bool a_first = (SEED && p.far_first) ? false : (ta <= tb);
                const uint32_t far_code = a_first ? cb : ca;
                const S far_t = a_first ? tb : ta;
                if constexpr (kRegTop) {
                  if (L.has_top) {  // the register entry spills below the new one
                    s_code[L.sp * kThreads + tid] = L.top_code;
                    s_t[L.sp * kThreads + tid] = L.top_t;
                    ++L.sp;
                  }
                  L.top_code = far_code;
                  L.top_t = far_t;
                  L.has_top = true;
                } else {
                  s_code[L.sp * kThreads + tid] = far_code;
                  s_t[L.sp * kThreads + tid] = far_t;
                  ++L.sp;
                }
                L.code = a_first ? ca : cb;
                L.code_t = a_first ? ta : tb;
              } else if (pa) {
                L.code = ca;
                L.code_t = ta;
              } else if (pb) {
                L.code = cb;
                L.code_t = tb;
              } else if (!pop(0)) {
                empty = true;
              }
            }
          }
          if (__all_sync(live_mask, pend != kNoHit || empty)) break;
        }
        if (pend != kNoHit) leaf(pend);
        // The node after the leaf was taken with the limit as it stood:
        // drop it (and what follows, as pop does) if the leaf's hit prunes it.
        if (!empty && L.code_t > L.limit && !pop(0)) empty = true;
        if (empty) {
          live = false;
          held = true;
        }
      }
    } else {
      step(live_mask, 0);
    }
  }

  if constexpr (HELP) {
    // No query is left to take: the lanes without one now help the others of
    // their warp. Every second pass while few lanes walk, else every fourth
    // (256 rays against 10,000 boxes: 25.6 us at 2, 30.5 at 4; 100,003 casts:
    // 157 and 149), a free lane copies a walking lane's query and takes over
    // the bottom entry of its stack (the largest waiting subtree); what it
    // finds goes back to the query's own lane, whose limit its helpers follow.
    // The subtrees are disjoint and near-first answers are certified whatever
    // the order of the visits, so the answers are the same.
    __shared__ uint8_t s_donor[kThreads];
    int owner = lane;  // the lane whose query this one walks
    int lo = 0;        // stack entries below this one have been taken over
    for (uint32_t pass = 0;; ++pass) {
      uint32_t live_mask = __ballot_sync(FULL, live);
      if (live_mask == 0u || ((pass & (__popc(live_mask) <= 8 ? 1u : 3u)) == 0u && live_mask != FULL)) {
        // Hits of the helpers go to their owners, one at a time (they are few).
        uint32_t found = __ballot_sync(FULL, owner != lane && L.best_leaf != kNoHit);
        while (found) {
          const int h = __ffs(found) - 1;
          found &= found - 1u;
          const int to = __shfl_sync(FULL, owner, h);
          const S t = __shfl_sync(FULL, L.best_t, h);
          const S t2 = __shfl_sync(FULL, L.second_t, h);
          const uint32_t id = __shfl_sync(FULL, L.best_leaf, h);
          const uint32_t pos = __shfl_sync(FULL, L.best_pos, h);
          S n[D];
          if constexpr (N == kNarrowCustom) {
#pragma unroll
            for (int i = 0; i < D; ++i) n[i] = __shfl_sync(FULL, L.best_n[i], h);
          }
          if (lane == to) {
            if (take_hit(t, id, pos)) {
              if constexpr (N == kNarrowCustom) {
#pragma unroll
                for (int i = 0; i < D; ++i) L.best_n[i] = n[i];
              }
            }
            if (t2 < L.second_t) L.second_t = t2;
          } else if (lane == h) {
            L.best_leaf = kNoHit;
            L.second_t = kInf;
          }
        }
        L.limit = smin(L.limit, __shfl_sync(FULL, L.limit, owner));
        // A query that no lane walks any more is answered.
        if (!live && owner != lane) owner = lane;  // a helper that has finished is free
        uint32_t walked = 0u;                       // owners of the walking lanes
        if (live) walked = 1u << owner;
        walked = __reduce_or_sync(FULL, walked);
        if (held && !((walked >> lane) & 1u)) {
          finish();
          held = false;
        }
        if (live_mask == 0u) break;
        const bool free = !live && !held;
        const uint32_t free_mask = __ballot_sync(FULL, free);
        const uint32_t donors = __ballot_sync(FULL, live && L.sp > lo);
        if (free_mask != 0u && donors != 0u) {
          const int nd = __popc(donors), nf = __popc(free_mask);
          const int rank = __popc((((donors >> lane) & 1u) ? donors : free_mask) & lt_mask);
          if ((donors >> lane) & 1u) s_donor[(tid & ~31) + rank] = uint8_t(lane);
          __syncwarp();
          const int e = rank / nd;
          const int from = free ? s_donor[(tid & ~31) + rank % nd] : lane;
          const int d_lo = __shfl_sync(FULL, lo, from);
          const int d_sp = __shfl_sync(FULL, L.sp, from);
          const bool taken = free && d_lo + e < d_sp;
#pragma unroll
          for (int i = 0; i < D; ++i) {
            L.r.o[i] = __shfl_sync(FULL, L.r.o[i], from);
            L.r.d[i] = __shfl_sync(FULL, L.r.d[i], from);
            L.r.inv[i] = __shfl_sync(FULL, L.r.inv[i], from);
            if constexpr (kCast) {
              L.pmin[i] = __shfl_sync(FULL, L.pmin[i], from);
              L.pmax[i] = __shfl_sync(FULL, L.pmax[i], from);
            }
          }
          L.r.par = __shfl_sync(FULL, L.r.par, from);
          L.fast = __shfl_sync(FULL, int(L.fast), from) != 0;
          L.limit = __shfl_sync(FULL, L.limit, from);
          const int d_owner = __shfl_sync(FULL, owner, from);
          if (taken) {
            const int at = (d_lo + e) * kThreads + (tid & ~31) + from;
            L.code = s_code[at];
            L.code_t = s_t[at];
            L.best_leaf = kNoHit;
            L.second_t = kInf;
            L.sp = 0;
            lo = 0;
            owner = d_owner;
            live = L.code_t <= L.limit;
            if (!live) owner = lane;
          }
          __syncwarp();
          if ((donors >> lane) & 1u) lo += min(L.sp - lo, (nf - rank + nd - 1) / nd);
          live_mask = __ballot_sync(FULL, live);
        }
      }
      step(live_mask, lo);
      if (owner != lane) held = false;  // a helper has no answer of its own
    }
  }
  if (STATS) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      c_vis += __shfl_down_sync(FULL, c_vis, o);
      c_nar += __shfl_down_sync(FULL, c_nar, o);
      c_hit += __shfl_down_sync(FULL, c_hit, o);
    }
    if (lane == 0 && p.stats) {
      atomicAdd(p.stats + 0, c_vis);
      atomicAdd(p.stats + 1, c_vis);
      atomicAdd(p.stats + 2, c_nar);
      atomicAdd(p.stats + 3, c_hit);
    }
  }
}

// ---------------------------------------------------------------------------
// Heavy overlap regions: one block (128 threads) per region, for the regions
// the count pass gave up on (counted and filled here) and, in the fill pass,
// for those it counted with more results than it kept. The block keeps
// the region's pending nodes in one shared-memory stack and each step takes
// up to 128 of them from the top, one per thread: an interior record's
// overlapping children are pushed (block prefix sum for the slots), a leaf's
// accepted overlapping primitives are counted (count pass) or written to the
// region's CSR segment in any order (fill pass; the segmented sort that
// follows orders them). Any order of visits finds the same set of leaves as
// the crate's walk. (A warp per region left the heaviest region's walk on 32
// lanes: 339 us for the D = 6 mixture's count pass with 5% of warp slots
// busy.) Stack: each step replaces the <= 128 entries it takes with <= 256
// children one level deeper, so at most 128 entries per level stay below the
// top: it never holds more than 128 x (depth + 2) entries; it is sized
// 256 x (depth + 1) (dynamic shared memory), and a push past it is refused
// and reported through heavy_count's high bit instead of written.
// With heavy_store set, the count pass also stages a region's leaves in
// shared memory (up to kHeavyStage) and copies them to heavy_store at a
// slot taken from heavy_cursor (heavy_start[i]: the slot, kNoHit when the
// stage or the store was too small); the fill pass then copies that region's
// segment from there instead of walking it again.
// ---------------------------------------------------------------------------
constexpr int kHeavyWarps = 4;
constexpr uint32_t kHeavyStage = 2048;

template <int D, int N>
__global__ void __launch_bounds__(32 * kHeavyWarps) overlap_heavy_kernel(const QueryParams p) {
  using PL = PrimLayout<D, N>;
  using NL = NodeLayout<D>;
  constexpr uint32_t FULL = 0xffffffffu;
  constexpr int T = 32 * kHeavyWarps;
  extern __shared__ uint32_t stk[];
  __shared__ unsigned long long s_fill;
  __shared__ int s_sp;
  __shared__ int s_wsum[kHeavyWarps];
  __shared__ uint32_t s_n;      // the region's accepted leaves so far
  __shared__ uint32_t s_start;  // its slot in heavy_store (kNoHit: none)
  __shared__ uint32_t s_stage[kHeavyStage];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int cap = p.stack;  // entries
  __shared__ uint32_t s_next;
  const uint32_t nh = *p.heavy_count & 0x7FFFFFFFu;
  for (;;) {
    // The next listed region, taken as blocks become free: their walks differ
    // by orders of magnitude.
    if (tid == 0) s_next = atomicAdd(p.counter, 1u);
    __syncthreads();
    const uint32_t i = s_next;
    __syncthreads();
    if (i >= nh) break;
    const uint32_t q = p.heavy_list[i];
    if (!p.fill && p.heavy_flag[q] == 2) continue;  // counted by the count pass (uniform per block)
    if (p.fill && p.heavy_start) {
      const uint32_t st = p.heavy_start[i];  // uniform per block
      if (st != kNoHit) {
        // staged by the count pass: a copy, no second walk
        const unsigned long long base = p.csr_offsets[q];
        const uint32_t c = uint32_t(p.csr_offsets[q + 1] - base);
        for (uint32_t k = tid; k < c; k += T) p.csr_leaves[base + k] = p.heavy_store[st + k];
        continue;
      }
    }
    float lo[D], hi[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
      lo[k] = p.queries[size_t(q) * 2 * D + k];
      hi[k] = p.queries[size_t(q) * 2 * D + D + k];
    }
    if (tid == 0) {
      s_fill = p.fill ? p.csr_offsets[q] : 0ull;
      s_n = 0;
      const bool in_root = box_overlap<D>(p.root_box, p.root_box + D, lo, hi);
      if (in_root) stk[0] = p.root_code;
      s_sp = in_root ? 1 : 0;
    }
    __syncthreads();
    for (;;) {
      const int sp = s_sp;
      if (sp == 0) break;  // uniform: every thread read the same value
      const int take = sp < T ? sp : T;
      const uint32_t code = tid < take ? stk[sp - take + tid] : kNoHit;
      __syncthreads();  // every entry taken is read before pushes overwrite it
      uint32_t push[2] = {kNoHit, kNoHit};
      if (code != kNoHit) {
        if (code & kLeafBit) {
          uint32_t pos = code & ~kLeafBit;
          for (;;) {
            float rec[PL::vec * 4];
            load_vec<PL::vec>(p.prims + size_t(pos) * PL::vec, rec);
            const uint32_t idw = __float_as_uint(rec[PL::id_word]);
            const uint32_t id = idw & ~kLeafBit;
            if (accepts(p, id) && narrow_overlap<D, N>(rec, lo, hi)) {
              if (p.fill) {
                p.csr_leaves[atomicAdd(&s_fill, 1ull)] = id;
              } else {
                const uint32_t k = atomicAdd(&s_n, 1u);
                if (k < kHeavyStage) s_stage[k] = id;
              }
            }
            if (idw & kLeafBit) break;
            ++pos;
          }
        } else {
          float rec[NL::vec * 4];
          load_vec<NL::vec>(p.nodes + size_t(code) * NL::vec, rec);
          if (box_overlap<D>(rec, rec + D, lo, hi)) push[0] = __float_as_uint(rec[4 * D]);
          if (box_overlap<D>(rec + 2 * D, rec + 3 * D, lo, hi)) push[1] = __float_as_uint(rec[4 * D + 1]);
        }
      }
      // Block prefix sum of the children to push: within each warp, then
      // across the warps' totals.
      const int mine = (push[0] != kNoHit) + (push[1] != kNoHit);
      int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane == 31) s_wsum[w] = incl;
      __syncthreads();
      int before = 0, total = 0;
#pragma unroll
      for (int k = 0; k < kHeavyWarps; ++k) {
        const int ws = s_wsum[k];
        if (k < w) before += ws;
        total += ws;
      }
      const int base = sp - take;
      int at = base + before + incl - mine;
      for (int k = 0; k < 2; ++k) {
        if (push[k] == kNoHit) continue;
        if (at < cap) stk[at] = push[k];
        else atomicOr(p.heavy_count, 0x80000000u);  // refused: reported to the host
        ++at;
      }
      __syncthreads();  // pushes written and s_wsum read before the next step
      if (tid == 0) s_sp = min(base + total, cap);
      __syncthreads();
    }
    if (!p.fill) {
      // The walk's last step ended at a barrier: s_n is final.
      const uint32_t c = s_n;
      if (tid == 0) {
        p.out_count[q] = c;
        uint32_t st = kNoHit;
        if (p.heavy_start && c <= kHeavyStage) {
          const uint32_t at = atomicAdd(p.heavy_cursor, c);
          if (at <= p.heavy_cap && c <= p.heavy_cap - at) st = at;
        }
        s_start = st;
        if (p.heavy_start) p.heavy_start[i] = st;
      }
      __syncthreads();
      const uint32_t st = s_start;
      if (st != kNoHit)
        for (uint32_t k = tid; k < c; k += T) p.heavy_store[st + k] = s_stage[k];
    }
    __syncthreads();  // the region's shared state is done before the next region's
  }
}

// ---------------------------------------------------------------------------
// Device refit: tree::refit (accel/tree.rs:54-75) over the fixed topology.
//
// One thread per leaf rewrites its primitives' records from the new leaf
// parameters and unions their boxes into the leaf box, which it stores in the
// parent's child slot. It then climbs: at each interior node an arrival
// counter lets the second of the two children through, which unions the two
// slots of that node's record into its own slot in its parent, and so on to
// the root. Unions are min/max, exact in any order.
// ---------------------------------------------------------------------------

struct RefitLeaf {
  uint32_t first;   // first position in the leaf-ordered primitive array
  uint32_t count;
  uint32_t parent;  // parent interior record << 1 | slot, or kNoHit for the root
  uint32_t pad;
};

struct RefitParams {
  int* nonfinite;  // set when a refit box is not finite
  float4* nodes;
  float4* prims;
  float* root_box;
  const float* prim_data;  // new leaf parameters, indexed by leaf id
  const uint32_t* prim_ids;
  const RefitLeaf* leaves;
  const uint32_t* parents;  // per interior record: parent << 1 | slot, or kNoHit
  uint32_t* arrivals;       // per interior record, zeroed before the launch
  uint32_t n_leaves;
  uint32_t stride;          // floats per leaf parameter block
};

template <int D, int N>
__device__ __forceinline__ void prim_box(const float* v, float* lo, float* hi) {
  if constexpr (N == kNarrowAabb) {
#pragma unroll
    for (int i = 0; i < D; ++i) { lo[i] = v[i]; hi[i] = v[D + i]; }
  } else if constexpr (N == kNarrowSphere || N == kNarrowSphereNear) {
#pragma unroll
    for (int i = 0; i < D; ++i) { lo[i] = fsub(v[i], v[D]); hi[i] = fadd(v[i], v[D]); }
  } else {
    tri_aabb(v, v + 3, v + 6, lo, hi);
  }
}

// Writes a child's box into its slot of the parent's record (or the root
// box): 2D floats at an 8-byte aligned offset, as D two-float stores.
template <int D>
__device__ __forceinline__ void store_slot(const RefitParams& p, uint32_t parent, const float* lo, const float* hi) {
  float* dst;
  if (parent == kNoHit) {
    dst = p.root_box;
  } else {
    dst = reinterpret_cast<float*>(p.nodes + size_t(parent >> 1) * NodeLayout<D>::vec) + (parent & 1u) * 2 * D;
  }
  float v[2 * D];
#pragma unroll
  for (int i = 0; i < D; ++i) {
    v[i] = lo[i];
    v[D + i] = hi[i];
  }
  float2* d2 = reinterpret_cast<float2*>(dst);
#pragma unroll
  for (int i = 0; i < D; ++i) d2[i] = make_float2(v[2 * i], v[2 * i + 1]);
}

// The union of a record's two child boxes (its own box in its parent),
// read past L1 (the sibling thread wrote them) as D 16-byte loads.
template <int D>
__device__ __forceinline__ void record_union(const float4* rec, float* lo, float* hi) {
  float b[4 * D];
#pragma unroll
  for (int w = 0; w < D; ++w) {
    const float4 x = __ldcg(rec + w);
    b[4 * w] = x.x;
    b[4 * w + 1] = x.y;
    b[4 * w + 2] = x.z;
    b[4 * w + 3] = x.w;
  }
#pragma unroll
  for (int i = 0; i < D; ++i) {
    lo[i] = fminf(b[i], b[2 * D + i]);
    hi[i] = fmaxf(b[D + i], b[3 * D + i]);
  }
}

template <int D, int N> __global__ void __launch_bounds__(256) refit_kernel(const RefitParams p) {
  const uint32_t li = blockIdx.x * blockDim.x + threadIdx.x;
  if (li >= p.n_leaves) return;
  const RefitLeaf L = p.leaves[li];
  using PL = PrimLayout<D, N>;
  float lo[D], hi[D];
#pragma unroll
  for (int i = 0; i < D; ++i) { lo[i] = __int_as_float(0x7f800000); hi[i] = __int_as_float(0xff800000); }
  for (uint32_t j = 0; j < L.count; ++j) {
    const uint32_t pos = L.first + j;
    const uint32_t id = p.prim_ids[pos];
    const float* v = p.prim_data + size_t(id) * p.stride;
    float rec[PL::vec * 4];
#pragma unroll
    for (int w = 0; w < PL::vec * 4; ++w) rec[w] = 0.f;
#pragma unroll
    for (int w = 0; w < PL::payload; ++w) rec[w] = v[w];
    rec[PL::id_word] = __uint_as_float(id | (j + 1 == L.count ? kLeafBit : 0u));
    float4* dst = p.prims + size_t(pos) * PL::vec;
#pragma unroll
    for (int w = 0; w < PL::vec; ++w) dst[w] = make_float4(rec[4 * w], rec[4 * w + 1], rec[4 * w + 2], rec[4 * w + 3]);
    float plo[D], phi[D];
    prim_box<D, N>(rec, plo, phi);
#pragma unroll
    for (int i = 0; i < D; ++i) { lo[i] = fminf(lo[i], plo[i]); hi[i] = fmaxf(hi[i], phi[i]); }
  }
  bool fin = true;
#pragma unroll
  for (int i = 0; i < D; ++i) fin = fin && isfinite(lo[i]) && isfinite(hi[i]);
  if (!fin) atomicOr(p.nonfinite, 1);
  uint32_t parent = L.parent;
  store_slot<D>(p, parent, lo, hi);
  while (parent != kNoHit) {
    __threadfence();
    const uint32_t node = parent >> 1;
    if (atomicAdd(p.arrivals + node, 1u) == 0u) return;  // the sibling finishes this node
    __threadfence();
    record_union<D>(p.nodes + size_t(node) * NodeLayout<D>::vec, lo, hi);
    parent = p.parents[node];
    store_slot<D>(p, parent, lo, hi);
  }
}

// After a refit (and wide_sync_kernel): every quantised record is quantised
// again from its exact four-wide record.
template <int D>
__global__ void quant_sync_kernel(float4* qnodes, const float4* __restrict__ wnodes, uint32_t n_records) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n_records) return;
  float rec[WideLayout<D>::vec * 4];
  load_vec<WideLayout<D>::vec>(wnodes + size_t(r) * WideLayout<D>::vec, rec);
  uint32_t codes[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) codes[k] = __float_as_uint(rec[8 * D + k]);
  uint32_t out[QuantLayout<D>::vec * 4];
#pragma unroll
  for (int w = 0; w < QuantLayout<D>::vec * 4; ++w) out[w] = 0u;
  quantize_record<D>(rec, codes, out);
  uint4* dst = reinterpret_cast<uint4*>(qnodes + size_t(r) * QuantLayout<D>::vec);
#pragma unroll
  for (int w = 0; w < QuantLayout<D>::vec; ++w) dst[w] = make_uint4(out[4 * w], out[4 * w + 1], out[4 * w + 2], out[4 * w + 3]);
}

// Function-pointer table entry for one (D, narrow) pair.
// After a refit: every four-wide slot copies its box from the binary record
// slot that holds the same node's box (src = record << 1 | slot).
template <int D>
__global__ void wide_sync_kernel(float4* wnodes, const float4* __restrict__ nodes, const uint32_t* __restrict__ src,
                                 uint32_t n_slots) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_slots || src[i] == kNoHit) return;
  const float* from = reinterpret_cast<const float*>(nodes + size_t(src[i] >> 1) * NodeLayout<D>::vec) +
                      (src[i] & 1u) * 2 * D;
  float* to = reinterpret_cast<float*>(wnodes + size_t(i / 4) * WideLayout<D>::vec) + (i % 4) * 2 * D;
  for (int k = 0; k < 2 * D; ++k) to[k] = from[k];
}

struct KernelSet {
  const void* ray_nearest[2][2];  // [ref][stats]
  const void* ray_nearest_wide;   // near-first over the four-wide records
  const void* ray_nearest_quant;  // near-first over the quantised four-wide records
  const void* ray_nearest_regtop; // near-first, postponed leaves, stack top in registers (WALK = 1)
  const void* ray_nearest_vote;   // near-first, child order by warp vote (WALK = 2)
  const void* wide_sync;          // refreshes four-wide boxes from the binary records
  const void* quant_sync;         // quantises the four-wide records again
  const void* ray_all[2];         // [stats]
  const void* cast_nearest[2];    // [ref]
  const void* cast_all;
  const void* overlap;
  const void* overlap_heavy;  // block-per-region overlap of the regions over the visit budget
  const void* refit_leaves;
  const void* ray_nearest_seeded[2];  // [stats]; D = 3 only
};

#ifndef __CUDACC_RTC__  // host code: not part of a run-time compiled unit
// The kernels of an f64 scene (the others stay null).
template <int D, int N> KernelSet make_kernel_set64() {
  KernelSet s{};
  s.ray_nearest[0][0] = (const void*)query_kernel<D, N, kRayNearest, false, false, false, false, false, 0, double>;
  s.ray_nearest[1][0] = (const void*)query_kernel<D, N, kRayNearest, true, false, false, false, false, 0, double>;
  s.ray_nearest[1][1] = (const void*)query_kernel<D, N, kRayNearest, true, true, false, false, false, 0, double>;
  s.ray_all[0] = (const void*)query_kernel<D, N, kRayAll, true, false, false, false, false, 0, double>;
  s.cast_nearest[0] = (const void*)query_kernel<D, N, kCastNearest, false, false, false, false, false, 0, double>;
  s.cast_nearest[1] = (const void*)query_kernel<D, N, kCastNearest, true, false, false, false, false, 0, double>;
  s.cast_all = (const void*)query_kernel<D, N, kCastAll, true, false, false, false, false, 0, double>;
  s.overlap = (const void*)query_kernel<D, N, kOverlap, true, false, false, false, false, 0, double>;
  return s;
}

template <int D, int N> KernelSet make_kernel_set() {
  KernelSet s;
  s.ray_nearest[0][0] = (const void*)query_kernel<D, N, kRayNearest, false, false>;
  s.ray_nearest[0][1] = (const void*)query_kernel<D, N, kRayNearest, false, true>;
  s.ray_nearest[1][0] = (const void*)query_kernel<D, N, kRayNearest, true, false>;
  s.ray_nearest[1][1] = (const void*)query_kernel<D, N, kRayNearest, true, true>;
  s.ray_nearest_wide = (const void*)query_kernel<D, N, kRayNearest, false, false, false, true>;
  s.ray_nearest_quant = (const void*)query_kernel<D, N, kRayNearest, false, false, false, true, true>;
  s.ray_nearest_regtop = (const void*)query_kernel<D, N, kRayNearest, false, false, false, false, false, 1>;
  s.ray_nearest_vote = (const void*)query_kernel<D, N, kRayNearest, false, false, false, false, false, 2>;
  s.wide_sync = (const void*)wide_sync_kernel<D>;
  s.quant_sync = (const void*)quant_sync_kernel<D>;
  s.ray_all[0] = (const void*)query_kernel<D, N, kRayAll, true, false>;
  s.ray_all[1] = (const void*)query_kernel<D, N, kRayAll, true, true>;
  s.cast_nearest[0] = (const void*)query_kernel<D, N, kCastNearest, false, false>;
  s.cast_nearest[1] = (const void*)query_kernel<D, N, kCastNearest, true, false>;
  s.cast_all = (const void*)query_kernel<D, N, kCastAll, true, false>;
  s.overlap = (const void*)query_kernel<D, N, kOverlap, true, false>;
  s.overlap_heavy = (const void*)overlap_heavy_kernel<D, N>;
  s.refit_leaves = (const void*)refit_kernel<D, N>;
  s.ray_nearest_seeded[0] = nullptr;
  s.ray_nearest_seeded[1] = nullptr;
  if constexpr (D == 3) {
    s.ray_nearest_seeded[0] = (const void*)query_kernel<D, N, kRayNearest, false, false, true>;
    s.ray_nearest_seeded[1] = (const void*)query_kernel<D, N, kRayNearest, false, true, true>;
  }
  return s;
}
#endif

}  // namespace sq
