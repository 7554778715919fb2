// The output layer of the learned guide's training step, with the softmax
// cross-entropy inside: two tcgen05 kernels that never write a logit.
//
//   Z = H W^T + b            [B x n_out], H [B x 128], W [n_out x 128] (bf16)
//   loss = sum over labelled rows of logsumexp(Z) - Z[label]
//   dZ = (softmax(Z) - onehot) / n_labelled          (rounded to bf16)
//   dH = dZ W, dW = dZ^T H, db = column sums of dZ
//
// Written out, the logits of a batch of 8,192 are 134 MB (written once, read
// three times) and dZ and its transpose 67 MB each: 280 us of a training step
// for arithmetic that takes the tensor cores 20. Here ce_stats_kernel makes
// the logits of a 128-row tile in TMEM chunk by chunk and keeps each row's
// running maximum and sum of exponentials; ce_grad_kernel makes them again,
// turns each 128 x 128 tile into dZ in shared memory and multiplies it from
// there twice: by W for dH, and, read as its transpose (the same tile as an
// MN-major operand), by H for dW. Both B operands are MN-major too, so W and
// H are each loaded in the one layout that the first product uses.
//
// Tiles in shared memory: 128 rows x 128 bf16 as two 128-byte-swizzled panels
// of 64 columns (umma.cuh), 32 KB.
#pragma once

#include "umma.cuh"

namespace sq {
namespace guide {

constexpr int kCeThreads = 320;  // warps 0..7 epilogue, warp 8 loads, warp 9 issues MMAs
constexpr uint32_t kTile = 32768;

struct CeParams {
  const float* bias;      // [n_out]
  const int32_t* labels;  // [B], outside [0, n_buckets): ignored
  const uint32_t* count;  // labelled rows of the batch
  float2* part;           // [B][2 * splits]: (max, sum of exp(z - max)) over a share of the columns
  float* zy;              // [B]: the label's logit
  float* loss;            // += the rows' losses
  float* dH;              // [B x 128], zeroed: += dZ W
  float* dW;              // [n_out x 128], zeroed: += dZ^T H
  float* db;              // [n_out], zeroed: += column sums of dZ
  uint32_t B, n_chunks, n_buckets, splits;
  int* err;
};

// Rounded share k of n over `parts`: [k * n / parts, (k + 1) * n / parts).
__device__ __forceinline__ uint32_t share(uint32_t k, uint32_t n, uint32_t parts) {
  return uint32_t(uint64_t(k) * n / parts);
}

// Operand descriptors of a tile: K-major (K = the 128 columns, 16 per step),
// or MN-major (K = the 128 rows, 16 per step; the 64-column panels 16 KB apart
// along M or N, the 8-row groups 1 KB apart along K).
__device__ __forceinline__ uint64_t tile_k_major(uint32_t saddr, uint32_t step) {
  return umma::desc_sw128(saddr + (step >> 2) * 16384) + 2 * (step & 3);
}
__device__ __forceinline__ uint64_t tile_mn_major(uint32_t saddr, uint32_t step) {
  uint64_t d = umma::desc_sw128(saddr + step * 2048);
  d &= ~(uint64_t(0x3FFF) << 16);
  return d | uint64_t(16384 >> 4) << 16;
}
constexpr uint32_t kIdescMnA = 1u << 15, kIdescMnB = 1u << 16;  // transpose bits of the instruction descriptor

// Waits that record where they gave up, and every role's way out.
struct CeWait {
  volatile int* err;
  __device__ bool operator()(uint64_t* bar, uint32_t parity, int code) const {
    if (*err == 0 && umma::mbar_wait(bar, parity)) return true;
    atomicCAS(const_cast<int*>(err), 0, code);
    return false;
  }
};

// TMA loads of both panels of rows [row, row + 128) into a tile.
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int row) {
  umma::mbar_arrive_expect_tx(bar, kTile);
  umma::tma_load_2d(dst, map, bar, 0, row);
  umma::tma_load_2d(dst + 16384, map, bar, 64, row);
}

// ---------------------------------------------------------------------------
// Row statistics. One CTA per 128-row tile and share of the column chunks
// (grid: row tiles x splits, about one CTA per SM): the H tile stays, W chunks
// stream through four slots, two TMEM accumulators alternate. Two epilogue
// warps share a quarter of the rows, 64 columns each. Bound by the exponentials
// (128 x 128 per chunk and SM).
// ---------------------------------------------------------------------------
constexpr int kStatSlots = 4;
struct CeStatsSmem {
  static constexpr uint32_t h = 0;
  static constexpr uint32_t ring = kTile;
  static constexpr uint32_t bias = ring + kStatSlots * kTile;
  static constexpr uint32_t bars = bias + 4096 * 4;
  static constexpr uint32_t bytes = bars + 256 + 1024;
};

__global__ void __launch_bounds__(kCeThreads, 1)
    ce_stats_kernel(const __grid_constant__ CUtensorMap th, const __grid_constant__ CUtensorMap tw, const CeParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = smem_raw + ((1024u - (umma::smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + CeStatsSmem::bars);
  uint64_t *h_full = bars, *w_full = bars + 1, *w_empty = w_full + kStatSlots, *z_full = w_empty + kStatSlots,
           *z_empty = z_full + 2;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(z_empty + 2);
  int* s_err = reinterpret_cast<int*>(tslot + 1);
  float* s_bias = reinterpret_cast<float*>(base + CeStatsSmem::bias);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t c0 = share(blockIdx.y, p.n_chunks, p.splits), c1 = share(blockIdx.y + 1, p.n_chunks, p.splits);
  if (threadIdx.x == 0) {
    umma::mbar_init(h_full, 1);
    for (int s = 0; s < kStatSlots; ++s) {
      umma::mbar_init(&w_full[s], 1);
      umma::mbar_init(&w_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      umma::mbar_init(&z_full[s], 1);
      umma::mbar_init(&z_empty[s], 8);
    }
    *s_err = 0;
    umma::fence_barrier_init();
  }
  for (uint32_t i = threadIdx.x; i < (c1 - c0) * 128; i += kCeThreads) s_bias[i] = p.bias[c0 * 128 + i];
  __syncwarp();
  if (warp == 9) umma::tmem_alloc(tslot, 256);
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tbase = *tslot;
  const CeWait wait{s_err};

  if (warp == 8) {
    if (lane == 0) {
      load_tile(base + CeStatsSmem::h, &th, h_full, int(blockIdx.x) * 128);
      uint32_t i = 0;
      for (; i < c1 - c0; ++i) {
        const uint32_t s = i % kStatSlots;
        if (i >= kStatSlots && !wait(&w_empty[s], ((i / kStatSlots) + 1) & 1, 1)) break;
        load_tile(base + CeStatsSmem::ring + s * kTile, &tw, &w_full[s], int(c0 + i) * 128);
      }
      // Every copy lands before the CTA's shared memory goes away.
      umma::mbar_wait(h_full, 0, 100000000ull);
      for (uint32_t k = i > kStatSlots ? i - kStatSlots : 0; k < i; ++k)
        umma::mbar_wait(&w_full[k % kStatSlots], (k / kStatSlots) & 1, 100000000ull);
    }
  } else if (warp == 9) {
    if (lane == 0) {
      bool ok = wait(h_full, 0, 2);
      for (uint32_t i = 0; ok && i < c1 - c0; ++i) {
        const uint32_t s = i % kStatSlots, z = i & 1;
        ok = wait(&w_full[s], (i / kStatSlots) & 1, 3) && (i < 2 || wait(&z_empty[z], ((i / 2) + 1) & 1, 4));
        if (!ok) break;
        umma::tc_fence_after();
        const uint32_t ha = umma::smem_u32(base + CeStatsSmem::h);
        const uint32_t wa = umma::smem_u32(base + CeStatsSmem::ring + s * kTile);
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)
          umma::mma_bf16(tbase + z * 128, tile_k_major(ha, k), tile_k_major(wa, k), umma::idesc_bf16(128, 128), k != 0);
        umma::mma_commit(&z_full[z]);
        umma::mma_commit(&w_empty[s]);
      }
    }
  } else {
    const uint32_t q = warp & 3, half = warp >> 2;
    const uint32_t row = blockIdx.x * 128 + q * 32 + lane;
    const int32_t y = p.labels[row];
    float m = -INFINITY, s = 0.f;
    for (uint32_t i = 0; i < c1 - c0; ++i) {
      const uint32_t z = i & 1;
      if (!__all_sync(0xffffffffu, wait(&z_full[z], (i / 2) & 1, 5))) break;
      umma::tc_fence_after();
      const uint32_t t = tbase + ((q * 32u) << 16) + z * 128 + half * 64;
      float v[64];
      umma::tmem_ld32(t, v);
      umma::tmem_ld32(t + 32, v + 32);
      umma::tc_fence_before();
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(&z_empty[z]);
      const uint32_t col = (c0 + i) * 128 + half * 64;  // of v[0]
      const float* b = s_bias + i * 128 + half * 64;
      float top = -INFINITY;
#pragma unroll
      for (uint32_t j = 0; j < 64; ++j) {
        v[j] = col + j < p.n_buckets ? v[j] + b[j] : -INFINITY;
        top = fmaxf(top, v[j]);
      }
      if (y >= int32_t(col) && y < int32_t(col + 64)) {
#pragma unroll
        for (uint32_t j = 0; j < 64; ++j)
          if (col + j == uint32_t(y)) p.zy[row] = v[j];
      }
      if (top > m) {
        s *= expf(m - top);  // 0 when m was -inf
        m = top;
      }
      if (m > -INFINITY) {
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
        for (uint32_t j = 0; j < 64; j += 4) {
          s0 += expf(v[j] - m);
          s1 += expf(v[j + 1] - m);
          s2 += expf(v[j + 2] - m);
          s3 += expf(v[j + 3] - m);
        }
        s += (s0 + s1) + (s2 + s3);
      }
    }
    p.part[size_t(row) * 2 * p.splits + blockIdx.y * 2 + half] = make_float2(m, s);
  }
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  __syncwarp();
  if (warp == 9) umma::tmem_dealloc(tbase, 256);
  if (threadIdx.x == 0 && *s_err) atomicCAS(p.err, 0, 100 + *s_err);
}

// ---------------------------------------------------------------------------
// Gradients. One CTA per pair of column chunks and share of the row tiles
// (grid: ceil(n_chunks / 2) x row shares, about one CTA per SM): its two W
// chunks stay in shared memory and their two dW accumulators in TMEM while H
// tiles stream through two slots. Per (row tile, chunk):
//   Z = H W^T                 into one TMEM accumulator,
//   dZ                        by the eight epilogue warps, into the chunk's dZ tile,
//   dH += dZ W, dW += dZ^T H  from that tile,
// with the next Z issued before the products of the last dZ, so that the
// tensor core works while the epilogue warps exponentiate. dH of a row tile is
// added to global memory after the next tile's first dZ (by then it is ready),
// dW and db once at the end. TMEM: Z 128 + dH 128 + dW 2 x 128 columns, all of it.
// ---------------------------------------------------------------------------
struct CeGradSmem {
  static constexpr uint32_t w = 0;             // 2 chunks
  static constexpr uint32_t h = 2 * kTile;     // 2 slots
  static constexpr uint32_t dz = 4 * kTile;    // one tile per chunk
  static constexpr uint32_t bias = 6 * kTile;  // 256 floats
  static constexpr uint32_t bars = bias + 1024;
  static constexpr uint32_t bytes = bars + 256 + 1024;
};

__global__ void __launch_bounds__(kCeThreads, 1)
    ce_grad_kernel(const __grid_constant__ CUtensorMap th, const __grid_constant__ CUtensorMap tw, const CeParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = smem_raw + ((1024u - (umma::smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + CeGradSmem::bars);
  uint64_t *w_full = bars, *h_full = bars + 1, *h_empty = bars + 3, *z_full = bars + 5, *z_empty = bars + 6,
           *dz_full = bars + 7, *dz_empty = bars + 9, *dh_full = bars + 11, *dh_empty = bars + 12, *dw_full = bars + 13;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 14);
  int* s_err = reinterpret_cast<int*>(tslot + 1);
  float* s_bias = reinterpret_cast<float*>(base + CeGradSmem::bias);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t chunk0 = blockIdx.x * 2, nc = min(2u, p.n_chunks - chunk0);
  const uint32_t tiles = p.B / 128;
  const uint32_t t0 = share(blockIdx.y, tiles, gridDim.y), nt = share(blockIdx.y + 1, tiles, gridDim.y) - t0;
  const uint32_t n = nt * nc;  // (row tile, chunk) steps
  if (threadIdx.x == 0) {
    umma::mbar_init(w_full, 1);
    for (int s = 0; s < 2; ++s) {
      umma::mbar_init(&h_full[s], 1);
      umma::mbar_init(&h_empty[s], 1);
      umma::mbar_init(&dz_full[s], 8);
      umma::mbar_init(&dz_empty[s], 1);
    }
    umma::mbar_init(z_full, 1);
    umma::mbar_init(z_empty, 8);
    umma::mbar_init(dh_full, 1);
    umma::mbar_init(dh_empty, 8);
    umma::mbar_init(dw_full, 1);
    *s_err = 0;
    umma::fence_barrier_init();
  }
  if (threadIdx.x < nc * 128) s_bias[threadIdx.x] = p.bias[chunk0 * 128 + threadIdx.x];
  __syncwarp();
  if (warp == 9) umma::tmem_alloc(tslot, 512);
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tz = *tslot, tdh = tz + 128, tdw = tz + 256;
  const CeWait wait{s_err};

  if (warp == 8) {
    if (lane == 0) {
      umma::mbar_arrive_expect_tx(w_full, nc * kTile);
      for (uint32_t c = 0; c < nc; ++c) {
        umma::tma_load_2d(base + CeGradSmem::w + c * kTile, &tw, w_full, 0, int(chunk0 + c) * 128);
        umma::tma_load_2d(base + CeGradSmem::w + c * kTile + 16384, &tw, w_full, 64, int(chunk0 + c) * 128);
      }
      uint32_t t = 0;
      for (; t < nt; ++t) {
        if (t >= 2 && !wait(&h_empty[t & 1], ((t / 2) + 1) & 1, 1)) break;
        load_tile(base + CeGradSmem::h + (t & 1) * kTile, &th, &h_full[t & 1], int(t0 + t) * 128);
      }
      umma::mbar_wait(w_full, 0, 100000000ull);
      for (uint32_t k = t > 2 ? t - 2 : 0; k < t; ++k) umma::mbar_wait(&h_full[k & 1], (k / 2) & 1, 100000000ull);
    }
  } else if (warp == 9) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma::idesc_bf16(128, 128);
      bool ok = wait(w_full, 0, 2);
      // Step i issues Z of step i, then the two products of step i - 1.
      for (uint32_t i = 0; ok && i <= n; ++i) {
        if (i < n) {
          const uint32_t t = i / nc, c = i % nc;
          ok = (c != 0 || wait(&h_full[t & 1], (t / 2) & 1, 3)) && (i == 0 || wait(z_empty, (i - 1) & 1, 4));
          if (!ok) break;
          umma::tc_fence_after();
          const uint32_t ha = umma::smem_u32(base + CeGradSmem::h + (t & 1) * kTile);
          const uint32_t wa = umma::smem_u32(base + CeGradSmem::w + c * kTile);
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k)
            umma::mma_bf16(tz, tile_k_major(ha, k), tile_k_major(wa, k), idesc, k != 0);
          umma::mma_commit(z_full);
        }
        if (i > 0) {
          const uint32_t j = i - 1, t = j / nc, c = j % nc;
          ok = wait(&dz_full[c], t & 1, 5) && (c != 0 || t == 0 || wait(dh_empty, (t - 1) & 1, 6));
          if (!ok) break;
          umma::tc_fence_after();
          const uint32_t ha = umma::smem_u32(base + CeGradSmem::h + (t & 1) * kTile);
          const uint32_t wa = umma::smem_u32(base + CeGradSmem::w + c * kTile);
          const uint32_t za = umma::smem_u32(base + CeGradSmem::dz + c * kTile);
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k)  // dH [rows x 128] += dZ [rows x cols] W [cols x 128]
            umma::mma_bf16(tdh, tile_k_major(za, k), tile_mn_major(wa, k), idesc | kIdescMnB, (c | k) != 0);
          if (c == nc - 1) umma::mma_commit(dh_full);
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k)  // dW [cols x 128] += dZ^T [cols x rows] H [rows x 128]
            umma::mma_bf16(tdw + c * 128, tile_mn_major(za, k), tile_mn_major(ha, k), idesc | kIdescMnA | kIdescMnB,
                           (t | k) != 0);
          umma::mma_commit(&dz_empty[c]);
          if (c == nc - 1) umma::mma_commit(&h_empty[t & 1]);
        }
      }
      umma::mma_commit(dw_full);
    }
  } else {
    const uint32_t q = warp & 3, half = warp >> 2;
    const uint32_t r = q * 32 + lane;  // row of the tile; dW: column of the chunk
    const uint32_t lanes = (q * 32u) << 16;
    const float inv_n = 1.0f / float(max(*p.count, 1u));
    // Column sums: this thread adds columns 2 cp and 2 cp + 1 of rows [32 rg, +32) of each dZ tile.
    const uint32_t cp = threadIdx.x & 63, rg = threadIdx.x >> 6;
    float cs[4] = {0.f, 0.f, 0.f, 0.f};
    float m = 0.f, inv_s = 0.f;
    int32_t y = -1;
    // dH of tile t: this thread's row, 64 of its 128 columns, added in the L2.
    auto flush_dh = [&](uint32_t t) -> bool {
      if (!__all_sync(0xffffffffu, wait(dh_full, t & 1, 7))) return false;
      umma::tc_fence_after();
      float v[64];
      umma::tmem_ld32(tdh + lanes + half * 64, v);
      umma::tmem_ld32(tdh + lanes + half * 64 + 32, v + 32);
      umma::tc_fence_before();
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(dh_empty);
      float* dst = p.dH + (size_t(t0 + t) * 128 + r) * 128 + half * 64;
#pragma unroll
      for (int j = 0; j < 64; j += 4) red_add4(dst + j, v[j], v[j + 1], v[j + 2], v[j + 3]);
      return true;
    };
    // After a wait that gave up (ok false) the warps still meet at every
    // barrier of the loop, so that none of them is left behind there.
    bool ok = true;
    for (uint32_t i = 0; i < n; ++i) {
      const uint32_t t = i / nc, c = i % nc;
      if (c == 0) {
        // This row's maximum and sum over all columns, from the shares.
        const uint32_t row = (t0 + t) * 128 + r;
        y = p.labels[row];
        if (uint32_t(y) >= p.n_buckets) y = -1;
        const float2* part = p.part + size_t(row) * 2 * p.splits;
        m = -INFINITY;
        for (uint32_t k = 0; k < 2 * p.splits; ++k) m = fmaxf(m, part[k].x);
        float s = 0.f;
        for (uint32_t k = 0; k < 2 * p.splits; ++k)
          if (part[k].x > -INFINITY) s += part[k].y * expf(part[k].x - m);
        inv_s = 1.0f / s;
        if (blockIdx.x == 0 && half == 0) {
          float l = y >= 0 ? logf(s) + m - p.zy[row] : 0.f;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
          if (lane == 0) atomicAdd(p.loss, l);
        }
      }
      ok = ok && __all_sync(0xffffffffu, wait(z_full, i & 1, 8));
      if (ok) {
        umma::tc_fence_after();
        float v[64];
        umma::tmem_ld32(tz + lanes + half * 64, v);
        umma::tmem_ld32(tz + lanes + half * 64 + 32, v + 32);
        umma::tc_fence_before();
        __syncwarp();
        if (lane == 0) umma::mbar_arrive(z_empty);
        // The tile of this chunk's last dZ is free once its products are done.
        ok = t == 0 || __all_sync(0xffffffffu, wait(&dz_empty[c], (t - 1) & 1, 9));
        const uint32_t col = (chunk0 + c) * 128 + half * 64;
        const float* b = s_bias + c * 128 + half * 64;
        uint8_t* panel = base + CeGradSmem::dz + c * kTile + half * 16384;
        if (ok) {
#pragma unroll
          for (uint32_t j = 0; j < 64; j += 8) {
            __align__(16) __nv_bfloat162 o[4];
#pragma unroll
            for (uint32_t k = 0; k < 8; k += 2) {
              float g[2];
#pragma unroll
              for (uint32_t e = 0; e < 2; ++e) {
                const uint32_t x = col + j + k + e;
                g[e] = expf(v[j + k + e] + b[j + k + e] - m) * inv_s - (x == uint32_t(y) ? 1.f : 0.f);
                g[e] = (y >= 0 && x < p.n_buckets) ? g[e] * inv_n : 0.f;
              }
              o[k / 2] = __floats2bfloat162_rn(g[0], g[1]);
            }
            *reinterpret_cast<uint4*>(panel + umma::sw128_offset(r, j)) = *reinterpret_cast<const uint4*>(o);
          }
          umma::fence_proxy_async();
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");  // the eight epilogue warps: the tile is complete
      if (ok) {
        if (lane == 0) umma::mbar_arrive(&dz_full[c]);
        const uint8_t* src = base + CeGradSmem::dz + c * kTile + (cp >> 5) * 16384;
        float a0 = 0.f, a1 = 0.f;
#pragma unroll 8
        for (uint32_t k = 0; k < 32; ++k) {
          const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(
              src + umma::sw128_offset(rg * 32 + k, (2 * cp) & 63));
          a0 += __low2float(x);
          a1 += __high2float(x);
        }
        if (c == 0) {
          cs[0] += a0;
          cs[1] += a1;
        } else {
          cs[2] += a0;
          cs[3] += a1;
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");  // every sum is read before a tile is written again
      if (ok && c == 0 && t > 0) ok = flush_dh(t - 1);
    }
    if (ok && n) ok = flush_dh(nt - 1);
    if (ok && n && __all_sync(0xffffffffu, wait(dw_full, 0, 10))) {
      umma::tc_fence_after();
      for (uint32_t c = 0; c < nc; ++c) {
        float* dst = p.dW + (size_t(chunk0 + c) * 128 + r) * 128 + half * 64;
        float v[64];
        umma::tmem_ld32(tdw + lanes + c * 128 + half * 64, v);
        umma::tmem_ld32(tdw + lanes + c * 128 + half * 64 + 32, v + 32);
#pragma unroll
        for (int j = 0; j < 64; j += 4) red_add4(dst + j, v[j], v[j + 1], v[j + 2], v[j + 3]);
        atomicAdd(p.db + (chunk0 + c) * 128 + 2 * cp, c == 0 ? cs[0] : cs[2]);
        atomicAdd(p.db + (chunk0 + c) * 128 + 2 * cp + 1, c == 0 ? cs[1] : cs[3]);
      }
    }
  }
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  __syncwarp();
  if (warp == 9) umma::tmem_dealloc(tz, 512);
  if (threadIdx.x == 0 && *s_err) atomicCAS(p.err, 0, 200 + *s_err);
}

}  // namespace guide
}  // namespace sq
