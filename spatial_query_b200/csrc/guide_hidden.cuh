// The hidden layers of the learned guide's training step as two kernels, one
// CTA per 128 rays each:
//
//   hidden_forward_kernel    the batch's rays (through a permutation) -> X, H1,
//                            H2, H3 = relu(H W^T + b) in bf16, labels gathered
//                            and counted;
//   hidden_backward_kernel   dH3 -> dZ_l = bf16(dH_l where H_l > 0), dW_l, db_l and
//                            dH_{l-1} = dZ_l W_l for l = 3, 2, 1.
//
// A layer of 8,192 x 128 x 128 is 0.3 GFLOP: as a product, an activation and
// (backward) two products and a transpose per layer, seventeen launches of 4 to
// 8 us took 130 us of a step. Here a tile's activations stay in shared memory
// from layer to layer, the weights are loaded once per CTA, and dZ serves both
// of its products from one tile (its transpose is the same tile read as an
// MN-major operand, guide_ce.cuh). Bound by the chain of three layers per tile
// (a product, then an epilogue) on 64 of the SMs at a batch of 8,192.
#pragma once

#include "guide_ce.cuh"

namespace sq {
namespace guide {

// ---------------------------------------------------------------------------
// Feature map, shared by training and inference: origin to [-1, 1] over the
// scene box, direction as is. Explicit roundings keep both paths bitwise equal.
// ---------------------------------------------------------------------------
struct Features {
  float lo[3], inv[3];
};

__device__ __forceinline__ void ray_features(const float* ray, const Features& f, float* x) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    x[i] = __fsub_rn(__fmul_rn(__fmul_rn(__fsub_rn(ray[i], f.lo[i]), f.inv[i]), 2.0f), 1.0f);
    x[3 + i] = ray[3 + i];
  }
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(umma::smem_u32(src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

struct HiddenForward {
  const float* rays;        // [.. x 6]
  const int32_t* labels;
  const uint32_t* perm;     // row i of the batch is ray perm[i] (null: i)
  Features f;
  const float* b[3];
  __nv_bfloat16* X;         // [B x 64], zero past the six features
  int32_t* batch_labels;    // gathered labels (null: not wanted)
  uint32_t* count;          // += labels inside [0, n_buckets)
  uint32_t n_buckets;
  int* err;
};

constexpr int kFwdThreads = 160;  // warps 0..3 rows, warp 4 loads and issues MMAs
struct FwdSmem {
  static constexpr uint32_t w1 = 0;  // 128 x 64
  static constexpr uint32_t w2 = 16384, w3 = w2 + kTile, act = w3 + kTile;
  static constexpr uint32_t bias = act + kTile;
  static constexpr uint32_t bars = bias + 3 * 512;
  static constexpr uint32_t bytes = bars + 128 + 1024;
};

__global__ void __launch_bounds__(kFwdThreads, 1)
    hidden_forward_kernel(const __grid_constant__ CUtensorMap tw1, const __grid_constant__ CUtensorMap tw2,
                          const __grid_constant__ CUtensorMap tw3, const __grid_constant__ CUtensorMap th1,
                          const __grid_constant__ CUtensorMap th2, const __grid_constant__ CUtensorMap th3,
                          const HiddenForward p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = smem_raw + ((1024u - (umma::smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + FwdSmem::bars);
  uint64_t *w_full = bars, *act_ready = bars + 1, *acc_full = bars + 2;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 3);
  int* s_err = reinterpret_cast<int*>(tslot + 1);
  float* s_bias = reinterpret_cast<float*>(base + FwdSmem::bias);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    umma::mbar_init(w_full, 1);
    umma::mbar_init(act_ready, 4);
    umma::mbar_init(acc_full, 1);
    *s_err = 0;
    umma::fence_barrier_init();
  }
  for (uint32_t i = threadIdx.x; i < 384; i += kFwdThreads) s_bias[i] = p.b[i / 128][i % 128];
  __syncwarp();
  if (warp == 4) umma::tmem_alloc(tslot, 128);
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tbase = *tslot;
  const CeWait wait{s_err};

  if (warp == 4) {
    if (lane == 0) {
      umma::mbar_arrive_expect_tx(w_full, 16384 + 2 * kTile);
      umma::tma_load_2d(base + FwdSmem::w1, &tw1, w_full, 0, 0);
      umma::tma_load_2d(base + FwdSmem::w2, &tw2, w_full, 0, 0);
      umma::tma_load_2d(base + FwdSmem::w2 + 16384, &tw2, w_full, 64, 0);
      umma::tma_load_2d(base + FwdSmem::w3, &tw3, w_full, 0, 0);
      umma::tma_load_2d(base + FwdSmem::w3 + 16384, &tw3, w_full, 64, 0);
      bool ok = wait(w_full, 0, 1);
      constexpr uint32_t idesc = umma::idesc_bf16(128, 128);
      const uint32_t act = umma::smem_u32(base + FwdSmem::act);
      for (uint32_t l = 0; ok && l < 3; ++l) {
        ok = wait(act_ready, l & 1, 2);
        if (!ok) break;
        umma::tc_fence_after();
        if (l == 0) {  // six features: one step of 16
          umma::mma_bf16(tbase, tile_k_major(act, 0), tile_k_major(umma::smem_u32(base + FwdSmem::w1), 0), idesc, 0);
        } else {
          const uint32_t w = umma::smem_u32(base + (l == 1 ? FwdSmem::w2 : FwdSmem::w3));
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k)
            umma::mma_bf16(tbase, tile_k_major(act, k), tile_k_major(w, k), idesc, k != 0);
        }
        umma::mma_commit(acc_full);
      }
      umma::mbar_wait(w_full, 0, 100000000ull);  // the copies land before the shared memory goes away
    }
  } else {
    const uint32_t r = warp * 32 + lane, row = blockIdx.x * 128 + r;
    uint8_t* act = base + FwdSmem::act;
    {
      const uint32_t src = p.perm ? p.perm[row] : row;
      float x[6];
      ray_features(p.rays + size_t(src) * 6, p.f, x);
      __align__(16) __nv_bfloat16 v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = __float2bfloat16_rn(k < 6 ? x[k] : 0.f);
      const uint4 a = reinterpret_cast<const uint4*>(v)[0], b = reinterpret_cast<const uint4*>(v)[1];
      *reinterpret_cast<uint4*>(act + umma::sw128_offset(r, 0)) = a;
      *reinterpret_cast<uint4*>(act + umma::sw128_offset(r, 8)) = b;
      uint4* out = reinterpret_cast<uint4*>(p.X + size_t(row) * 64);
      out[0] = a;
#pragma unroll
      for (int k = 1; k < 8; ++k) out[k] = make_uint4(0u, 0u, 0u, 0u);
      const int32_t y = p.labels[src];
      if (p.batch_labels) p.batch_labels[row] = y;
      const uint32_t some = __ballot_sync(0xffffffffu, y >= 0 && uint32_t(y) < p.n_buckets);
      if (lane == 0 && some) atomicAdd(p.count, uint32_t(__popc(some)));
    }
    umma::fence_proxy_async();
    __syncwarp();
    if (lane == 0) umma::mbar_arrive(act_ready);
    bool ok = true;
    for (uint32_t l = 0; l < 3; ++l) {
      ok = ok && __all_sync(0xffffffffu, wait(acc_full, l & 1, 3));
      // The last layer's tile has been stored before this one replaces it.
      if (threadIdx.x == 0) bulk_wait_read();
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (ok) {
        umma::tc_fence_after();
        float v[128];
        umma::tmem_ld128(tbase + (uint32_t(warp * 32) << 16), v);
        const float* b = s_bias + l * 128;
#pragma unroll
        for (uint32_t c = 0; c < 128; c += 8) {
          __align__(16) __nv_bfloat162 o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            o[i] = __floats2bfloat162_rn(fmaxf(v[c + 2 * i] + b[c + 2 * i], 0.f),
                                         fmaxf(v[c + 2 * i + 1] + b[c + 2 * i + 1], 0.f));
          *reinterpret_cast<uint4*>(act + (c >> 6) * 16384 + umma::sw128_offset(r, c & 63)) =
              *reinterpret_cast<const uint4*>(o);
        }
        umma::tc_fence_before();
        umma::fence_proxy_async();
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (ok && l < 2 && lane == 0) umma::mbar_arrive(act_ready);
      if (ok && threadIdx.x == 0) {
        const CUtensorMap* out = l == 0 ? &th1 : (l == 1 ? &th2 : &th3);
        tma_store_2d(out, act, 0, int(blockIdx.x) * 128);
        tma_store_2d(out, act + 16384, 64, int(blockIdx.x) * 128);
        bulk_commit();
      }
    }
    if (threadIdx.x == 0) bulk_wait();
  }
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  __syncwarp();
  if (warp == 4) umma::tmem_dealloc(tbase, 128);
  if (threadIdx.x == 0 && *s_err) atomicCAS(p.err, 0, 300 + *s_err);
}

struct HiddenBackward {
  const float* dH3;          // [B x 128]
  const __nv_bfloat16* H3;   // [B x 128]
  float* dW[3];              // W1 [128 x 64], W2, W3 [128 x 128]; zeroed
  float* db[3];              // zeroed
  int* err;
};

struct BwdSmem {
  static constexpr uint32_t h2 = 0, h1 = kTile, w3 = 2 * kTile, w2 = 3 * kTile, dz = 4 * kTile, x = 5 * kTile;
  static constexpr uint32_t stage = x + 16384;  // one per epilogue warp
  static constexpr uint32_t bars = stage + 8 * kStageBytes;
  static constexpr uint32_t bytes = bars + 128 + 1024;
};

__global__ void __launch_bounds__(kCeThreads, 1)
    hidden_backward_kernel(const __grid_constant__ CUtensorMap th2, const __grid_constant__ CUtensorMap th1,
                           const __grid_constant__ CUtensorMap tx, const __grid_constant__ CUtensorMap tw3,
                           const __grid_constant__ CUtensorMap tw2, const HiddenBackward p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = smem_raw + ((1024u - (umma::smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + BwdSmem::bars);
  uint64_t *in_full = bars, *dz_ready = bars + 1, *acc_full = bars + 2;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 3);
  int* s_err = reinterpret_cast<int*>(tslot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int y0 = int(blockIdx.x) * 128;
  if (threadIdx.x == 0) {
    umma::mbar_init(in_full, 1);
    umma::mbar_init(dz_ready, 8);
    umma::mbar_init(acc_full, 1);
    *s_err = 0;
    umma::fence_barrier_init();
  }
  __syncwarp();
  if (warp == 9) umma::tmem_alloc(tslot, 512);
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tdh = *tslot, tdw = tdh + 128;  // dW3, dW2, dW1 at tdw + 0, 128, 256
  const CeWait wait{s_err};

  if (warp == 8) {
    if (lane == 0) {
      umma::mbar_arrive_expect_tx(in_full, 4 * kTile + 16384);
      const CUtensorMap* maps[4] = {&th2, &th1, &tw3, &tw2};
      const uint32_t at[4] = {BwdSmem::h2, BwdSmem::h1, BwdSmem::w3, BwdSmem::w2};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        umma::tma_load_2d(base + at[k], maps[k], in_full, 0, k < 2 ? y0 : 0);
        umma::tma_load_2d(base + at[k] + 16384, maps[k], in_full, 64, k < 2 ? y0 : 0);
      }
      umma::tma_load_2d(base + BwdSmem::x, &tx, in_full, 0, y0);
      umma::mbar_wait(in_full, 0, 100000000ull);
    }
  } else if (warp == 9) {
    if (lane == 0) {
      constexpr uint32_t mn = kIdescMnA | kIdescMnB;
      constexpr uint32_t idesc = umma::idesc_bf16(128, 128);
      const uint32_t za = umma::smem_u32(base + BwdSmem::dz);
      bool ok = wait(in_full, 0, 1);
      for (uint32_t l = 0; ok && l < 3; ++l) {  // layers 3, 2, 1
        ok = wait(dz_ready, l & 1, 2);
        if (!ok) break;
        umma::tc_fence_after();
        if (l < 2) {
          const uint32_t ha = umma::smem_u32(base + (l == 0 ? BwdSmem::h2 : BwdSmem::h1));
          const uint32_t wa = umma::smem_u32(base + (l == 0 ? BwdSmem::w3 : BwdSmem::w2));
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k)  // dH [rows x in] = dZ [rows x out] W [out x in]
            umma::mma_bf16(tdh, tile_k_major(za, k), tile_mn_major(wa, k), idesc | kIdescMnB, k != 0);
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k)  // dW [out x in] = dZ^T [out x rows] H [rows x in]
            umma::mma_bf16(tdw + l * 128, tile_mn_major(za, k), tile_mn_major(ha, k), idesc | mn, k != 0);
        } else {
          const uint32_t xa = umma::smem_u32(base + BwdSmem::x);
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k)  // the six features' 16 columns
            umma::mma_bf16(tdw + 256, tile_mn_major(za, k), tile_mn_major(xa, k), umma::idesc_bf16(128, 16) | mn, k != 0);
        }
        umma::mma_commit(acc_full);
      }
    }
  } else {
    const uint32_t q = warp & 3, half = warp >> 2, r = q * 32 + lane;
    const uint32_t lanes = (q * 32u) << 16;
    const uint32_t cp = threadIdx.x & 63, rg = threadIdx.x >> 6;  // column sums, as in ce_grad_kernel
    float* stage = reinterpret_cast<float*>(base + BwdSmem::stage + warp * kStageBytes);
    uint8_t* panel = base + BwdSmem::dz + half * 16384;
    float v[64];  // dH of this row, 64 of its 128 columns
    {
      const float4* src = reinterpret_cast<const float4*>(p.dH3 + (size_t(y0) + r) * 128 + half * 64);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float4 a = src[j];
        v[4 * j] = a.x;
        v[4 * j + 1] = a.y;
        v[4 * j + 2] = a.z;
        v[4 * j + 3] = a.w;
      }
    }
    // After a wait that gave up the warps still meet at every barrier.
    bool ok = __all_sync(0xffffffffu, wait(in_full, 0, 3));
    for (uint32_t l = 0; l < 3; ++l) {
      if (l > 0) {
        ok = ok && __all_sync(0xffffffffu, wait(acc_full, (l - 1) & 1, 4));
        if (ok) {
          umma::tc_fence_after();
          umma::tmem_ld32(tdh + lanes + half * 64, v);
          umma::tmem_ld32(tdh + lanes + half * 64 + 32, v + 32);
          umma::tc_fence_before();
        }
      }
      if (ok) {
        // dZ = dH where the layer's activation is positive.
        const uint8_t* h = base + (l == 1 ? BwdSmem::h2 : BwdSmem::h1) + half * 16384;
        const uint4* h3 = reinterpret_cast<const uint4*>(p.H3 + (size_t(y0) + r) * 128 + half * 64);
#pragma unroll
        for (uint32_t j = 0; j < 64; j += 8) {
          __align__(16) __nv_bfloat162 a[4], o[4];
          *reinterpret_cast<uint4*>(a) =
              l == 0 ? h3[j / 8] : *reinterpret_cast<const uint4*>(h + umma::sw128_offset(r, j));
#pragma unroll
          for (int k = 0; k < 4; ++k)
            o[k] = __floats2bfloat162_rn(__low2float(a[k]) > 0.f ? v[j + 2 * k] : 0.f,
                                         __high2float(a[k]) > 0.f ? v[j + 2 * k + 1] : 0.f);
          *reinterpret_cast<uint4*>(panel + umma::sw128_offset(r, j)) = *reinterpret_cast<const uint4*>(o);
        }
        umma::fence_proxy_async();
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");  // the tile is complete
      if (ok) {
        if (lane == 0) umma::mbar_arrive(dz_ready);
        const uint8_t* src = base + BwdSmem::dz + (cp >> 5) * 16384;
        float a0 = 0.f, a1 = 0.f;
#pragma unroll 8
        for (uint32_t k = 0; k < 32; ++k) {
          const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(
              src + umma::sw128_offset(rg * 32 + k, (2 * cp) & 63));
          a0 += __low2float(x);
          a1 += __high2float(x);
        }
        atomicAdd(p.db[2 - l] + 2 * cp, a0);
        atomicAdd(p.db[2 - l] + 2 * cp + 1, a1);
        if (l > 0) {  // the last layer's dW is complete: out row r, 64 of its 128 columns
          float w[64];
          umma::tmem_ld32(tdw + (l - 1) * 128 + lanes + half * 64, w);
          umma::tmem_ld32(tdw + (l - 1) * 128 + lanes + half * 64 + 32, w + 32);
          add_rows(stage, w, p.dW[3 - l] + size_t(q * 32) * 128 + half * 64, lane);
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");  // every sum is read before the tile is written again
    }
    ok = ok && __all_sync(0xffffffffu, wait(acc_full, 0, 5));
    if (ok && half == 0) {
      umma::tc_fence_after();
      float w[32];
      umma::tmem_ld32(tdw + 256 + lanes, w);
      red_add4(p.dW[0] + size_t(r) * 64, w[0], w[1], w[2], w[3]);
      red_add4(p.dW[0] + size_t(r) * 64 + 4, w[4], w[5], 0.f, 0.f);
    }
  }
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  __syncwarp();
  if (warp == 9) umma::tmem_dealloc(tdh, 512);
  if (threadIdx.x == 0 && *s_err) atomicCAS(p.err, 0, 400 + *s_err);
}

}  // namespace guide
}  // namespace sq
