// The crate's f64 feature on the device (Scalar = f64, maths/point.rs:14-18):
// queries against an f64 scene, for consumers whose coordinates need double
// precision (large worlds) or who compare against an f64 CPU build.
//
// The kernels are query_kernel's with S = double (traverse.cuh): child-pair
// records of doubles, nearest queries near-first with the certificate (or in
// the crate's own order, which the counters ask for: Bvh::raycast_nearest_impl,
// accel/bvh.rs:73-124), lists, casts and overlap in the crate's order
// (bvh.rs:196-456). All arithmetic is the f64 form of the f32 kernels'
// (sq_math.cuh), so answers and QueryStats counters equal the f64 CPU path's
// bit for bit.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "sq_internal.cuh"

using namespace sq;
using sqi::cuda_fail;
using sqi::fail;

namespace {

using namespace sqi;
using Params64 = QueryParamsT<double>;

bool kernel_set64(int dim, int narrow, KernelSet* out) {
  switch (dim) {
    case 2: return kernel_set64_d2(narrow, out);
    case 3: return kernel_set64_d3(narrow, out);
    case 4: return kernel_set64_d4(narrow, out);
    case 6: return kernel_set64_d6(narrow, out);
    default: return false;
  }
}

Params64 base64(const sq_bvh* b, const sq_filter* filter) {
  Params64 p{};
  p.nodes = b->d_nodes;
  p.prims = b->d_prims;
  p.layers = b->d_layers;
  p.root_box = b->d_root64;
  p.nonfinite = b->d_nonfinite;
  p.root_code = b->root_code;
  p.mask = filter ? filter->layer_mask : ~0ull;
  p.exclude = filter ? filter->exclude : -1;
  return p;
}

// Nearest rays (counted: stats) or casts: near-first with the certificate, or
// the crate's own order when the context asks for it and for counters, which
// are the crate's.
int32_t nearest64(sq_ctx* ctx, const sq_bvh* b, bool cast, Params64& p, bool stats) {
  const void* ref_fn = cast ? b->ks64.cast_nearest[1] : b->ks64.ray_nearest[1][stats ? 1 : 0];
  if (stats || ctx->order == SQ_ORDER_REFERENCE) return launch_persistent(ctx, ref_fn, p, b->depth, p.n);
  return near_first_launch(ctx, b, cast ? b->ks64.cast_nearest[0] : b->ks64.ray_nearest[0][0], ref_fn, p, b->depth);
}

uint32_t stride64(int dim, int narrow) {
  if (narrow == SQ_NARROW_AABB) return 2 * dim;
  if (narrow == SQ_NARROW_TRIANGLE) return 9;
  return dim + 1;
}

int32_t check64(sq_ctx* ctx, const sq_bvh* b) {
  if (!ctx) return SQ_ERR_INVALID;
  if (!b) return fail(ctx, SQ_ERR_INVALID, "null scene");
  if (b->device != ctx->device) return fail(ctx, SQ_ERR_INVALID, "scene and context are on different devices");
  if (b->prec != 64) return fail(ctx, SQ_ERR_UNSUPPORTED, "an f32 scene is queried through the f32 entry points");
  const cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return cuda_fail(ctx, "cudaSetDevice", e);
  return SQ_OK;
}

}  // namespace

extern "C" int32_t sq_bvh_upload_f64(sq_ctx* ctx, int32_t dim, int32_t narrow, uint32_t n_nodes,
                                     const double* node_bounds, const uint32_t* child_a, const uint32_t* child_b,
                                     const uint32_t* prim_count, uint32_t n_prims, const uint32_t* prim_indices,
                                     const double* prim_data, uint32_t prim_stride, const uint64_t* layers,
                                     sq_bvh** out) {
  if (!ctx || !out) return SQ_ERR_INVALID;
  *out = nullptr;
  KernelSet ks;
  if (!kernel_set64(dim, narrow, &ks))
    return fail(ctx, SQ_ERR_UNSUPPORTED, "no f64 kernels for dim " + std::to_string(dim) + " narrow " +
                                             std::to_string(narrow));
  if (prim_stride != stride64(dim, narrow)) return fail(ctx, SQ_ERR_INVALID, "prim_stride does not match the narrow phase");
  if (n_prims >= kLeafBit || n_nodes >= kLeafBit) return fail(ctx, SQ_ERR_INVALID, "too many nodes or leaves");
  if ((n_nodes == 0) != (n_prims == 0)) return fail(ctx, SQ_ERR_INVALID, "empty tree with leaves, or leaves without a tree");
  if (n_nodes && (!node_bounds || !child_a || !child_b || !prim_count || !prim_indices || !prim_data))
    return fail(ctx, SQ_ERR_INVALID, "null tree array");
  CK(cudaSetDevice(ctx->device));
  auto b = std::make_unique<sq_bvh>();
  b->device = ctx->device;
  b->dim = dim;
  b->narrow = narrow;
  b->prec = 64;
  b->n_nodes = n_nodes;
  b->n_prims = n_prims;
  b->stride = prim_stride;
  b->ks64 = ks;
  if (n_nodes == 0) {
    *out = b.release();
    return SQ_OK;
  }
  // The same topology rules as the f32 upload: children after their parent,
  // leaves inside and partitioning a permutation; the depth bounds the stack.
  std::vector<uint32_t> depth(n_nodes, 1);
  for (uint32_t i = n_nodes; i-- > 0;) {
    if (prim_count[i] == 0) {
      if (child_a[i] <= i || child_b[i] <= i || child_a[i] >= n_nodes || child_b[i] >= n_nodes)
        return fail(ctx, SQ_ERR_INVALID, "interior node " + std::to_string(i) + " has a child out of order");
      depth[i] = 1 + std::max(depth[child_a[i]], depth[child_b[i]]);
    } else if (uint64_t(child_a[i]) + prim_count[i] > n_prims || prim_count[i] >= kLeafBit) {
      return fail(ctx, SQ_ERR_INVALID, "leaf node " + std::to_string(i) + " indexes past the primitives");
    }
  }
  b->depth = depth[0];
  if (b->depth + 1 > uint32_t(kMaxStack))
    return fail(ctx, SQ_ERR_DEPTH, "tree depth " + std::to_string(b->depth) + " exceeds the traversal stack");
  {
    std::vector<uint8_t> seen(n_prims, 0), covered(n_prims, 0);
    for (uint32_t k = 0; k < n_prims; ++k) {
      if (prim_indices[k] >= n_prims || seen[prim_indices[k]])
        return fail(ctx, SQ_ERR_INVALID, "prim_indices is not a permutation");
      seen[prim_indices[k]] = 1;
    }
    for (uint32_t i = 0; i < n_nodes; ++i) {
      if (prim_count[i] == 0) continue;
      for (uint32_t k = child_a[i]; k < child_a[i] + prim_count[i]; ++k) {
        if (covered[k]) return fail(ctx, SQ_ERR_INVALID, "leaf ranges overlap");
        covered[k] = 1;
      }
    }
    for (uint32_t k = 0; k < n_prims; ++k)
      if (!covered[k]) return fail(ctx, SQ_ERR_INVALID, "leaf ranges leave a primitive uncovered");
  }
  // Child-pair node records and leaf-ordered primitive records, as the f32
  // upload lays them out: the boxes in doubles, then both codes in one 8-byte
  // word; the parameters in doubles, then the id word in the low half of one.
  const int D = dim;
  std::vector<uint32_t> iidx(n_nodes, kNoHit);
  for (uint32_t i = 0; i < n_nodes; ++i)
    if (prim_count[i] == 0) iidx[i] = b->n_interior++;
  auto code = [&](uint32_t i) { return prim_count[i] == 0 ? iidx[i] : (kLeafBit | child_a[i]); };
  b->root_code = code(0);
  const size_t NS = size_t(record_vec(8 * D + 2)) * 2, PS = size_t(record_vec(2 * (int(prim_stride) + 1))) * 2;
  b->prim_vec = uint32_t(PS / 2);
  std::vector<double> nodes(std::max<size_t>(b->n_interior, 1) * NS, 0.0), prims(size_t(n_prims) * PS, 0.0);
  for (uint32_t i = 0; i < n_nodes; ++i) {
    if (prim_count[i] == 0) {
      double* r = nodes.data() + size_t(iidx[i]) * NS;
      const uint32_t ch[2] = {child_a[i], child_b[i]}, codes[2] = {code(child_a[i]), code(child_b[i])};
      for (int s = 0; s < 2; ++s) std::copy_n(node_bounds + size_t(ch[s]) * 2 * D, 2 * D, r + s * 2 * D);
      std::memcpy(r + 4 * D, codes, sizeof(codes));
      continue;
    }
    for (uint32_t j = 0; j < prim_count[i]; ++j) {
      const uint32_t pos = child_a[i] + j, id = prim_indices[pos];
      double* r = prims.data() + size_t(pos) * PS;
      std::copy_n(prim_data + size_t(id) * prim_stride, prim_stride, r);
      const uint64_t w = id | (j + 1 == prim_count[i] ? kLeafBit : 0u);
      std::memcpy(r + prim_stride, &w, sizeof(w));
    }
  }
  int nonfinite = 0;
  for (size_t k = 0; k < size_t(n_nodes) * 2 * D; ++k)
    if (!std::isfinite(node_bounds[k])) nonfinite = 1;
  auto up = [&](void** dst, const void* src, size_t bytes) -> int32_t {
    CK(cudaMalloc(dst, std::max<size_t>(bytes, 16)));
    if (src && bytes) CK(cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice));
    b->bytes += bytes;
    return SQ_OK;
  };
  int32_t rc;
  auto cleanup = [&](int32_t code) {
    sq_bvh_destroy(b.release());
    return code;
  };
  if ((rc = up((void**)&b->d_nodes, nodes.data(), nodes.size() * 8))) return cleanup(rc);
  if ((rc = up((void**)&b->d_prims, prims.data(), prims.size() * 8))) return cleanup(rc);
  if ((rc = up((void**)&b->d_root64, node_bounds, size_t(2) * D * 8))) return cleanup(rc);
  if ((rc = up((void**)&b->d_nonfinite, &nonfinite, sizeof(int)))) return cleanup(rc);
  if (layers && (rc = up((void**)&b->d_layers, layers, size_t(n_prims) * 8))) return cleanup(rc);
  *out = b.release();
  return SQ_OK;
}

extern "C" int32_t sq_raycast_nearest_f64_d(sq_ctx* ctx, const sq_bvh* b, const double* d_rays, uint32_t n,
                                            double max_toi, const double* d_max_toi_per_query,
                                            const sq_filter* filter, uint32_t* d_leaf, double* d_toi,
                                            double* d_normal, sq_query_stats* stats) {
  int32_t rc = check64(ctx, b);
  if (rc) return rc;
  if (n == 0) return SQ_OK;
  if (!d_rays || !d_leaf) return fail(ctx, SQ_ERR_INVALID, "null rays or leaf output");
  const bool st = stats != nullptr;
  if (st) CK(cudaMemsetAsync(ctx->d_stats, 0, 4 * sizeof(unsigned long long), ctx->stream));
  if (b->n_nodes == 0) {
    CK(cudaMemsetAsync(d_leaf, 0xFF, size_t(n) * 4, ctx->stream));
    if (d_toi) CK(cudaMemsetAsync(d_toi, 0, size_t(n) * 8, ctx->stream));
    if (d_normal) CK(cudaMemsetAsync(d_normal, 0, size_t(n) * b->dim * 8, ctx->stream));
  } else {
    Params64 p = base64(b, filter);
    p.queries = d_rays;
    p.n = n;
    p.max_toi = max_toi;
    p.max_toi_arr = d_max_toi_per_query;
    p.out_leaf = d_leaf;
    p.out_toi = d_toi;
    p.out_normal = d_normal;
    p.stats = st ? ctx->d_stats : nullptr;
    if ((rc = nearest64(ctx, b, false, p, st))) return rc;
  }
  CK(cudaGetLastError());
  if (st) {
    unsigned long long h[4];
    CK(cudaMemcpyAsync(h, ctx->d_stats, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    stats->nodes_visited = h[0];
    stats->aabb_tests = h[1];
    stats->narrow_tests = h[2];
    stats->hits = h[3];
  }
  return SQ_OK;
}

extern "C" int32_t sq_raycast_nearest_f64(sq_ctx* ctx, const sq_bvh* b, const double* rays, uint32_t n,
                                          double max_toi, const double* max_toi_per_query, const sq_filter* filter,
                                          uint32_t* leaf, double* toi, double* normal, sq_query_stats* stats) {
  int32_t rc = check64(ctx, b);
  if (rc) return rc;
  if (n == 0) return SQ_OK;
  if (!rays || !leaf) return fail(ctx, SQ_ERR_INVALID, "null rays or leaf output");
  const int D = b->dim;
  // One scratch allocation for the batch: rays, per-query limits, outputs.
  const size_t b_rays = size_t(n) * 2 * D * 8, b_mt = max_toi_per_query ? size_t(n) * 8 : 0, b_leaf = size_t(n) * 4,
               b_toi = toi ? size_t(n) * 8 : 0, b_nrm = normal ? size_t(n) * D * 8 : 0;
  sqi::Carve cv;
  const size_t o_rays = cv.take(b_rays), o_mt = cv.take(b_mt), o_leaf = cv.take(b_leaf), o_toi = cv.take(b_toi),
               o_nrm = cv.take(b_nrm);
  if ((rc = sqi::arena_reserve(ctx, cv.off))) return rc;
  char* base = static_cast<char*>(ctx->arena.p);
  CK(cudaMemcpyAsync(base + o_rays, rays, b_rays, cudaMemcpyHostToDevice, ctx->stream));
  if (b_mt) CK(cudaMemcpyAsync(base + o_mt, max_toi_per_query, b_mt, cudaMemcpyHostToDevice, ctx->stream));
  if ((rc = sq_raycast_nearest_f64_d(ctx, b, reinterpret_cast<const double*>(base + o_rays), n, max_toi,
                                     b_mt ? reinterpret_cast<const double*>(base + o_mt) : nullptr, filter,
                                     reinterpret_cast<uint32_t*>(base + o_leaf),
                                     b_toi ? reinterpret_cast<double*>(base + o_toi) : nullptr,
                                     b_nrm ? reinterpret_cast<double*>(base + o_nrm) : nullptr, stats)))
    return rc;
  CK(cudaMemcpyAsync(leaf, base + o_leaf, b_leaf, cudaMemcpyDeviceToHost, ctx->stream));
  if (b_toi) CK(cudaMemcpyAsync(toi, base + o_toi, b_toi, cudaMemcpyDeviceToHost, ctx->stream));
  if (b_nrm) CK(cudaMemcpyAsync(normal, base + o_nrm, b_nrm, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  return SQ_OK;
}

// ---------------------------------------------------------------------------
// Lists, casts and overlap on f64 scenes.
// ---------------------------------------------------------------------------

namespace {

int32_t list_args(sq_ctx* ctx, uint32_t n, const double* q, const sq_hit_lists_f64* o) {
  if (!o || (n && (!q || !o->count || (o->k && (!o->leaf || !o->toi)))))
    return fail(ctx, SQ_ERR_INVALID, "null queries or list output");
  return SQ_OK;
}

int32_t lists64(sq_ctx* ctx, const sq_bvh* b, int kind, const double* d_q, uint32_t n, double max_toi,
                const double* d_mt, const sq_filter* filter, int32_t crossings, const sq_hit_lists_f64* o) {
  int32_t rc = check64(ctx, b);
  if (rc || (rc = list_args(ctx, n, d_q, o))) return rc;
  if (n == 0) return SQ_OK;
  if (b->n_nodes == 0) {
    CK(cudaMemsetAsync(o->count, 0, size_t(n) * 4, ctx->stream));
    return SQ_OK;
  }
  Params64 p = base64(b, filter);
  p.queries = d_q;
  p.n = n;
  p.max_toi = max_toi;
  p.max_toi_arr = d_mt;
  p.k = o->k;
  p.crossings = crossings;
  p.out_count = o->count;
  p.out_leaf = o->leaf;
  p.out_toi = o->toi;
  p.out_normal = o->normal;
  return launch_persistent(ctx, kind == kCastAll ? b->ks64.cast_all : b->ks64.ray_all[0], p, b->depth, p.n);
}

// Host-buffer lists: queries (and per-query limits) in, lists out, through
// the context's arena.
int32_t lists64_host(sq_ctx* ctx, const sq_bvh* b, int kind, uint32_t width, const double* q, uint32_t n,
                     double max_toi, const double* mt, const sq_filter* filter, int32_t crossings,
                     const sq_hit_lists_f64* o) {
  int32_t rc = check64(ctx, b);
  if (rc || (rc = list_args(ctx, n, q, o))) return rc;
  if (n == 0) return SQ_OK;
  const int D = b->dim;
  const size_t k = o->k;
  sqi::Carve cv;
  const size_t o_q = cv.take(size_t(n) * width * D * 8), o_mt = cv.take(mt ? size_t(n) * 8 : 0),
               o_cnt = cv.take(size_t(n) * 4), o_leaf = cv.take(size_t(n) * k * 4), o_toi = cv.take(size_t(n) * k * 8),
               o_nrm = cv.take(o->normal ? size_t(n) * k * D * 8 : 0);
  if ((rc = sqi::arena_reserve(ctx, cv.off))) return rc;
  char* base = static_cast<char*>(ctx->arena.p);
  CK(cudaMemcpyAsync(base + o_q, q, size_t(n) * width * D * 8, cudaMemcpyHostToDevice, ctx->stream));
  if (mt) CK(cudaMemcpyAsync(base + o_mt, mt, size_t(n) * 8, cudaMemcpyHostToDevice, ctx->stream));
  sq_hit_lists_f64 d{};
  d.k = o->k;
  d.count = reinterpret_cast<uint32_t*>(base + o_cnt);
  d.leaf = reinterpret_cast<uint32_t*>(base + o_leaf);
  d.toi = reinterpret_cast<double*>(base + o_toi);
  d.normal = o->normal ? reinterpret_cast<double*>(base + o_nrm) : nullptr;
  if ((rc = lists64(ctx, b, kind, reinterpret_cast<const double*>(base + o_q), n, max_toi,
                    mt ? reinterpret_cast<const double*>(base + o_mt) : nullptr, filter, crossings, &d)))
    return rc;
  // Only the stored entries come back: the first min(count, k) of each query.
  std::vector<uint32_t> cnt(n);
  CK(cudaMemcpyAsync(cnt.data(), d.count, size_t(n) * 4, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  std::memcpy(o->count, cnt.data(), size_t(n) * 4);
  if (k) {
    CK(cudaMemcpyAsync(o->leaf, d.leaf, size_t(n) * k * 4, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaMemcpyAsync(o->toi, d.toi, size_t(n) * k * 8, cudaMemcpyDeviceToHost, ctx->stream));
    if (o->normal) CK(cudaMemcpyAsync(o->normal, d.normal, size_t(n) * k * D * 8, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
  }
  return SQ_OK;
}

}  // namespace

extern "C" int32_t sq_raycast_all_f64_d(sq_ctx* ctx, const sq_bvh* b, const double* d_rays, uint32_t n,
                                        double max_toi, const double* d_max_toi_per_query, const sq_filter* filter,
                                        int32_t crossings, const sq_hit_lists_f64* d_out) {
  return lists64(ctx, b, kRayAll, d_rays, n, max_toi, d_max_toi_per_query, filter, crossings, d_out);
}

extern "C" int32_t sq_raycast_all_f64(sq_ctx* ctx, const sq_bvh* b, const double* rays, uint32_t n, double max_toi,
                                      const double* max_toi_per_query, const sq_filter* filter, int32_t crossings,
                                      const sq_hit_lists_f64* out) {
  return lists64_host(ctx, b, kRayAll, 2, rays, n, max_toi, max_toi_per_query, filter, crossings, out);
}

extern "C" int32_t sq_shapecast_all_f64_d(sq_ctx* ctx, const sq_bvh* b, const double* d_casts, uint32_t n,
                                          double max_toi, const double* d_max_toi_per_query, const sq_filter* filter,
                                          const sq_hit_lists_f64* d_out) {
  return lists64(ctx, b, kCastAll, d_casts, n, max_toi, d_max_toi_per_query, filter, 0, d_out);
}

extern "C" int32_t sq_shapecast_all_f64(sq_ctx* ctx, const sq_bvh* b, const double* casts, uint32_t n,
                                        double max_toi, const double* max_toi_per_query, const sq_filter* filter,
                                        const sq_hit_lists_f64* out) {
  return lists64_host(ctx, b, kCastAll, 4, casts, n, max_toi, max_toi_per_query, filter, 0, out);
}

extern "C" int32_t sq_shapecast_nearest_f64_d(sq_ctx* ctx, const sq_bvh* b, const double* d_casts, uint32_t n,
                                              double max_toi, const double* d_max_toi_per_query,
                                              const sq_filter* filter, uint32_t* d_leaf, double* d_toi,
                                              double* d_normal) {
  int32_t rc = check64(ctx, b);
  if (rc) return rc;
  if (n && (!d_casts || !d_leaf)) return fail(ctx, SQ_ERR_INVALID, "null casts or leaf output");
  if (n == 0) return SQ_OK;
  if (b->n_nodes == 0) {
    CK(cudaMemsetAsync(d_leaf, 0xFF, size_t(n) * 4, ctx->stream));
    if (d_toi) CK(cudaMemsetAsync(d_toi, 0, size_t(n) * 8, ctx->stream));
    if (d_normal) CK(cudaMemsetAsync(d_normal, 0, size_t(n) * b->dim * 8, ctx->stream));
    return SQ_OK;
  }
  Params64 p = base64(b, filter);
  p.queries = d_casts;
  p.n = n;
  p.max_toi = max_toi;
  p.max_toi_arr = d_max_toi_per_query;
  p.out_leaf = d_leaf;
  p.out_toi = d_toi;
  p.out_normal = d_normal;
  return nearest64(ctx, b, true, p, false);
}

extern "C" int32_t sq_shapecast_nearest_f64(sq_ctx* ctx, const sq_bvh* b, const double* casts, uint32_t n,
                                            double max_toi, const double* max_toi_per_query, const sq_filter* filter,
                                            uint32_t* leaf, double* toi, double* normal) {
  int32_t rc = check64(ctx, b);
  if (rc) return rc;
  if (n == 0) return SQ_OK;
  if (!casts || !leaf) return fail(ctx, SQ_ERR_INVALID, "null casts or leaf output");
  const int D = b->dim;
  sqi::Carve cv;
  const size_t o_q = cv.take(size_t(n) * 4 * D * 8), o_mt = cv.take(max_toi_per_query ? size_t(n) * 8 : 0),
               o_leaf = cv.take(size_t(n) * 4), o_toi = cv.take(toi ? size_t(n) * 8 : 0),
               o_nrm = cv.take(normal ? size_t(n) * D * 8 : 0);
  if ((rc = sqi::arena_reserve(ctx, cv.off))) return rc;
  char* base = static_cast<char*>(ctx->arena.p);
  CK(cudaMemcpyAsync(base + o_q, casts, size_t(n) * 4 * D * 8, cudaMemcpyHostToDevice, ctx->stream));
  if (max_toi_per_query)
    CK(cudaMemcpyAsync(base + o_mt, max_toi_per_query, size_t(n) * 8, cudaMemcpyHostToDevice, ctx->stream));
  if ((rc = sq_shapecast_nearest_f64_d(ctx, b, reinterpret_cast<const double*>(base + o_q), n, max_toi,
                                       max_toi_per_query ? reinterpret_cast<const double*>(base + o_mt) : nullptr,
                                       filter, reinterpret_cast<uint32_t*>(base + o_leaf),
                                       toi ? reinterpret_cast<double*>(base + o_toi) : nullptr,
                                       normal ? reinterpret_cast<double*>(base + o_nrm) : nullptr)))
    return rc;
  CK(cudaMemcpyAsync(leaf, base + o_leaf, size_t(n) * 4, cudaMemcpyDeviceToHost, ctx->stream));
  if (toi) CK(cudaMemcpyAsync(toi, base + o_toi, size_t(n) * 8, cudaMemcpyDeviceToHost, ctx->stream));
  if (normal) CK(cudaMemcpyAsync(normal, base + o_nrm, size_t(n) * D * 8, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  return SQ_OK;
}

extern "C" int32_t sq_overlap_f64_d(sq_ctx* ctx, const sq_bvh* b, const double* d_regions, uint32_t n,
                                    const sq_filter* filter, uint64_t* d_offsets, uint32_t* d_leaves,
                                    uint64_t leaf_capacity, uint64_t* total) {
  int32_t rc = check64(ctx, b);
  if (rc) return rc;
  if (!d_offsets || !total || (n && !d_regions)) return fail(ctx, SQ_ERR_INVALID, "null argument");
  // Counts and the scan's scratch from the context's arena.
  size_t scan_bytes = 0;
  CK(cub::DeviceScan::ExclusiveScan(nullptr, scan_bytes, static_cast<const uint32_t*>(nullptr),
                                    static_cast<unsigned long long*>(nullptr), cuda::std::plus<>{}, 0ull, int(n) + 1,
                                    ctx->stream));
  sqi::Carve cv;
  const size_t o_cnt = cv.take((size_t(n) + 1) * 4), o_tmp = cv.take(scan_bytes);
  if ((rc = sqi::arena_reserve(ctx, cv.off))) return rc;
  char* base = static_cast<char*>(ctx->arena.p);
  uint32_t* d_counts = reinterpret_cast<uint32_t*>(base + o_cnt);
  CK(cudaMemsetAsync(d_counts, 0, (size_t(n) + 1) * 4, ctx->stream));
  Params64 p = base64(b, filter);
  p.queries = d_regions;
  p.n = n;
  p.out_count = d_counts;
  const void* fn = b->ks64.overlap;
  if (b->n_nodes != 0 && n != 0 && (rc = launch_persistent(ctx, fn, p, b->depth, p.n))) return rc;
  CK(cub::DeviceScan::ExclusiveScan(base + o_tmp, scan_bytes, d_counts, reinterpret_cast<unsigned long long*>(d_offsets),
                                    cuda::std::plus<>{}, 0ull, int(n) + 1, ctx->stream));
  ctx->launches++;
  unsigned long long tot = 0;
  CK(cudaMemcpyAsync(&tot, d_offsets + n, 8, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  *total = tot;
  if (tot > leaf_capacity) return fail(ctx, SQ_ERR_CAPACITY, "overlap results exceed leaf_capacity");
  if (tot && b->n_nodes != 0) {
    if (!d_leaves) return fail(ctx, SQ_ERR_INVALID, "null leaf output");
    p.csr_offsets = reinterpret_cast<const unsigned long long*>(d_offsets);
    p.csr_leaves = d_leaves;
    p.fill = 2;
    if ((rc = launch_persistent(ctx, fn, p, b->depth, p.n))) return rc;
    if ((rc = sqi::sort_csr_segments(ctx, d_leaves, tot, d_offsets, n))) return rc;
  }
  CK(cudaStreamSynchronize(ctx->stream));
  return SQ_OK;
}

extern "C" int32_t sq_overlap_f64(sq_ctx* ctx, const sq_bvh* b, const double* regions, uint32_t n,
                                  const sq_filter* filter, uint64_t* offsets, uint32_t* leaves, uint64_t leaf_capacity,
                                  uint64_t* total) {
  int32_t rc = check64(ctx, b);
  if (rc) return rc;
  if (!offsets || !total || (n && !regions)) return fail(ctx, SQ_ERR_INVALID, "null argument");
  const int D = b->dim;
  // Regions and offsets in a scratch block of their own: the device call
  // takes the arena for its counts.
  char* dq = nullptr;
  const size_t qb = (size_t(n) * 2 * D * 8 + 255) & ~size_t(255);
  CK(sqi::scratch_alloc(ctx, reinterpret_cast<void**>(&dq), qb + (size_t(n) + 1) * 8 + size_t(leaf_capacity) * 4 + 16));
  uint64_t* d_off = reinterpret_cast<uint64_t*>(dq + qb);
  uint32_t* d_lv = reinterpret_cast<uint32_t*>(dq + qb + (size_t(n) + 1) * 8);
  cudaError_t e = n ? cudaMemcpyAsync(dq, regions, size_t(n) * 2 * D * 8, cudaMemcpyHostToDevice, ctx->stream)
                    : cudaSuccess;
  if (e == cudaSuccess) {
    rc = sq_overlap_f64_d(ctx, b, reinterpret_cast<const double*>(dq), n, filter, d_off, d_lv, leaf_capacity, total);
    if (rc == SQ_OK || rc == SQ_ERR_CAPACITY)
      e = cudaMemcpyAsync(offsets, d_off, (size_t(n) + 1) * 8, cudaMemcpyDeviceToHost, ctx->stream);
    if (rc == SQ_OK && e == cudaSuccess && *total && leaves)
      e = cudaMemcpyAsync(leaves, d_lv, size_t(*total) * 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  }
  cudaFreeAsync(dq, ctx->stream);
  if (e != cudaSuccess) return cuda_fail(ctx, "overlap f64 copies", e);
  return rc;
}
