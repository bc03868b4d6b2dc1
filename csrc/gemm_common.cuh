// What the bf16 / NVFP4 GEMM kernels share: the launch parameters, tensor maps, and what an epilogue does with 32 finished
// fp32 accumulator columns of one row.
#pragma once

#include "common.cuh"

#include <math.h>

namespace js {

constexpr int kSms = 148;       // of the device this is written for
constexpr int BM = 128;
constexpr int BK = 64;          // 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;

enum GemmEpi : int { EPI_STORE = 0, EPI_SWIGLU = 1, EPI_ARGMAX = 2, EPI_TOPK = 3, EPI_STORE_F32 = 4, EPI_ALLREDUCE = 5, EPI_EP_COMBINE = 6,
                    EPI_INPROJ = 7, EPI_RELU2 = 8, EPI_RESID32 = 9 };
enum GemmAct : int { ACT_GELU_GLU = 0, ACT_RELU2 = 1, ACT_NONE = 2, ACT_GELU_ERF = 3, ACT_XIELU = 4 };

struct GemmParams {
  int M, N, K;
  int ldc;                      // elements
  void* C;                      // bf16 (or fp32 for EPI_STORE_F32) output
  const __nv_bfloat16* residual;  // optional, same shape/ld as C (may alias C)
  float* part_val;              // ARGMAX: [M, n_tiles] ; TOPK: [M, n_tiles, 8] values
  int* part_idx;                // ARGMAX: [M, n_tiles] ; TOPK: [M, n_tiles, 8] indices
  float* part_lse;              // TOPK: [M, n_tiles, 2] (running max, sum of exp)
  int* status;
  unsigned long long* trace;    // optional: 8 phase timestamps (ns) written by CTA (0,0,0)
  // EPI_ALLREDUCE (tensor-parallel row-parallel GEMM): every rank's receive buffer and flag array
  __nv_bfloat16* const* peer_recv;  // [world] -> (world, m_cap, N) bf16 on that rank
  int* const* peer_flags;           // [world] -> one counter per CTA of this grid on that rank
  int rank, world, m_cap;
  // grouped mode (MoE experts): blockIdx.z is the expert; its rows are group_off[e] .. group_off[e+1]
  // of A and C, its weights are rows e*N .. (e+1)*N of W.  No K split in this mode.
  const int* group_off;
  // EPI_EP_COMBINE (expert-parallel down projection): row r of the sorted rows belongs to
  // (token, choice) pair row_pair[r] with routing weight row_weight[r]; the weighted output row is
  // stored into every rank's pair buffer (n_pairs, N) and a per-rank counter is bumped per CTA.
  const int* row_pair;
  const float* row_weight;
  __nv_bfloat16* const* peer_pairs;
  int* const* peer_cnt;
  // EPI_EP_COMBINE with token-sharded dispatch: row r of this rank's receive slab came from rank row_meta[r].x
  // as that rank's (token, choice) pair row_meta[r].y; the weighted output row returns to that rank only, as
  // flagged 8-byte cells {two bf16 values, 1} that the owner's finishing kernel polls (no counters)
  const int2* row_meta;
  // NVFP4 mode: block scales of A and W in 512-byte tiles, per-row scale of A, per-tensor scale of W
  const uint8_t* sfa;
  const uint8_t* sfw;
  const float* row_scale;
  float w_scale;
  // EPI_ALLREDUCE: only push the partial tile and bump the flags; a finishing kernel reduces (no wait in this kernel)
  int ar_push_only;
  // Tile order: 0 = column tiles fastest (consecutive CTAs share the activation tile), 1 = row tiles fastest
  // (consecutive CTAs share the WEIGHT tile: for a vocabulary matrix larger than L2 and many row tiles, each
  // weight tile then comes from HBM once instead of once per row tile)
  int m_fast;
  // A row tile with at most this many rows left loads its activations through the second tensor map, whose box holds
  // only that many rows (0 = always the 128-row box); the accumulator rows beyond the box read stale shared memory
  // and are never stored.  Grouped mode: with ~8 rows per expert (MoE decode) a 128-row box would make the
  // activations half of every stage's bytes although almost none of its rows are used.  Otherwise it is M % 128, so
  // that the last row tile's box ends with the matrix: a box that lies mostly past the end is slow, because every CTA
  // waits for its zero fill (4096 x 24576 weights at 1 row, 128-row box against 1-row box: 69.1 against 40.2 us per
  // launch, 4096 x 6144 at 8 rows 24.2 against 15.5, 4096 x 151936 at 1 row 276 against 203; equal from 16 rows on).
  int a_small_rows;
  // EPI_INPROJ (fused input projections of a parallel block): columns below n_raw (a multiple of 128) are stored as
  // fp32 to C; the rest pass through `act` and go to C2 as bf16.  ACT_GELU_GLU: every 128 weight rows hold 64 gate rows
  // and the 64 up rows of the same outputs; ACT_RELU2: relu(.)^2 of each column; ACT_GELU_ERF: exact gelu of each
  // column; ACT_XIELU: act_a z^2 + z / 2 for z > 0, act_b (e^z - 1 - z) + z / 2 below; ACT_NONE: as it is.
  __nv_bfloat16* C2;
  int ldc2;
  int n_raw;
  int act;
  float act_a, act_b;
  // EPI_RESID32: C (fp32) = res32 + A W^T (+ emb); with norm_w, C2 = bf16(tanh(norm_alpha C) norm_w + norm_b), the
  // next layer's Dynamic Tanh.  res32 may be C.
  const float* res32;
  const __nv_bfloat16* emb;
  int ld_emb;
  const float* norm_w;
  const float* norm_b;
  float norm_alpha;
  // Batched mode: blockIdx.z is the batch element; its K columns of A start at z * a_batch_k, its weights are rows
  // z*N .. (z+1)*N of W, its output starts at C + z * c_batch_stride.  A box that reaches past the element's own K
  // columns meets zero-filled weights.  No K split in this mode.
  int batch;
  int a_batch_k;
  long long c_batch_stride;
};

// ---------------------------------------------------------------------------- 32 accumulator columns of row `grow`
JS_DEVICE void epi_store_bf16(__nv_bfloat16* out, const float* v) {
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    uint4 ov;
    __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
    for (int t = 0; t < 4; ++t) o2[t] = __floats2bfloat162_rn(v[j + 2 * t], v[j + 2 * t + 1]);
    *reinterpret_cast<uint4*>(out + j) = ov;
  }
}

// EPI_STORE (+ residual), EPI_STORE_F32, EPI_RELU2; `offset` elements are added to C
template <int EPI>
JS_DEVICE void epi_store_chunk(const GemmParams& p, int grow, int gc, float* v, long long offset) {
  if constexpr (EPI == EPI_STORE_F32) {
    float* out = reinterpret_cast<float*>(p.C) + static_cast<size_t>(grow) * p.ldc + gc;
#pragma unroll
    for (int j = 0; j < 32; j += 4)
      if (gc + j < p.N) *reinterpret_cast<float4*>(out + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
  } else {
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.C) + static_cast<size_t>(grow) * p.ldc + gc + offset;
    const __nv_bfloat16* res = p.residual ? p.residual + static_cast<size_t>(grow) * p.ldc + gc : nullptr;
    if constexpr (EPI == EPI_RELU2) {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        v[j] = fmaxf(v[j], 0.f);
        v[j] *= v[j];
      }
    }
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      if (gc + j >= p.N) break;
      if (res) {
        uint4 rv = *reinterpret_cast<const uint4*>(res + j);
        const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rv);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          float2 f = __bfloat1622float2(r2[t]);
          v[j + 2 * t] += f.x;
          v[j + 2 * t + 1] += f.y;
        }
      }
      uint4 ov;
      __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
      for (int t = 0; t < 4; ++t) o2[t] = __floats2bfloat162_rn(v[j + 2 * t], v[j + 2 * t + 1]);
      *reinterpret_cast<uint4*>(out + j) = ov;
    }
  }
}

// EPI_SWIGLU: 32 gate and 32 up columns of the outputs gc ..
JS_DEVICE void epi_swiglu_chunk(const GemmParams& p, int grow, int gc, float* g, const float* u) {
#pragma unroll
  for (int j = 0; j < 32; ++j) g[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
  epi_store_bf16(reinterpret_cast<__nv_bfloat16*>(p.C) + static_cast<size_t>(grow) * p.ldc + gc, g);
}

// EPI_INPROJ: columns cb .. of the first and of the second 64 columns of the 128-column block at nb
JS_DEVICE void epi_inproj_halves(const GemmParams& p, int grow, int nb, int cb, float* g, float* u) {
  if (nb < p.n_raw) {
    float* out = reinterpret_cast<float*>(p.C) + static_cast<size_t>(grow) * p.ldc + nb + cb;
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      *reinterpret_cast<float4*>(out + j) = make_float4(g[j], g[j + 1], g[j + 2], g[j + 3]);
      *reinterpret_cast<float4*>(out + 64 + j) = make_float4(u[j], u[j + 1], u[j + 2], u[j + 3]);
    }
    return;
  }
  __nv_bfloat16* out2 = p.C2 + static_cast<size_t>(grow) * p.ldc2;
  if (p.act == ACT_GELU_GLU) {
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const float a = g[j];
      g[j] = 0.5f * a * (1.f + tanhf(0.7978845608028654f * (a + 0.044715f * a * a * a))) * u[j];   // sqrt(2 / pi)
    }
    epi_store_bf16(out2 + (nb - p.n_raw) / 2 + cb, g);
    return;
  }
  if (p.act == ACT_RELU2) {
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      g[j] = fmaxf(g[j], 0.f);
      g[j] *= g[j];
      u[j] = fmaxf(u[j], 0.f);
      u[j] *= u[j];
    }
  } else if (p.act == ACT_GELU_ERF) {
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      g[j] = 0.5f * g[j] * (1.f + erff(g[j] * 0.7071067811865476f));      // 1 / sqrt(2)
      u[j] = 0.5f * u[j] * (1.f + erff(u[j] * 0.7071067811865476f));
    }
  } else if (p.act == ACT_XIELU) {
    auto xielu = [&](float z) { return 0.5f * z + (z > 0.f ? p.act_a * z * z : p.act_b * (__expf(z) - 1.f - z)); };
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      g[j] = xielu(g[j]);
      u[j] = xielu(u[j]);
    }
  }
  epi_store_bf16(out2 + nb - p.n_raw + cb, g);
  epi_store_bf16(out2 + nb - p.n_raw + 64 + cb, u);
}

// EPI_RESID32
JS_DEVICE void epi_resid32_chunk(const GemmParams& p, int grow, int gc, float* v) {
  float* out = reinterpret_cast<float*>(p.C) + static_cast<size_t>(grow) * p.ldc + gc;
  const float* res = p.res32 + static_cast<size_t>(grow) * p.ldc + gc;
  const __nv_bfloat16* emb = p.emb ? p.emb + static_cast<size_t>(grow) * p.ld_emb + gc : nullptr;
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    if (gc + j >= p.N) break;
#pragma unroll
    for (int t = 0; t < 8; t += 4) {
      const float4 rv = *reinterpret_cast<const float4*>(res + j + t);
      v[j + t] += rv.x;
      v[j + t + 1] += rv.y;
      v[j + t + 2] += rv.z;
      v[j + t + 3] += rv.w;
    }
    if (emb != nullptr) {
      const uint4 ev = *reinterpret_cast<const uint4*>(emb + j);
      const __nv_bfloat162* e2 = reinterpret_cast<const __nv_bfloat162*>(&ev);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 f = __bfloat1622float2(e2[t]);
        v[j + 2 * t] += f.x;
        v[j + 2 * t + 1] += f.y;
      }
    }
    *reinterpret_cast<float4*>(out + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    *reinterpret_cast<float4*>(out + j + 4) = make_float4(v[j + 4], v[j + 5], v[j + 6], v[j + 7]);
    if (p.norm_w != nullptr) {
      uint4 ov;
      __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 w2 = __ldg(reinterpret_cast<const float2*>(p.norm_w + gc + j + 2 * t));
        const float2 b2 = __ldg(reinterpret_cast<const float2*>(p.norm_b + gc + j + 2 * t));
        o2[t] = __floats2bfloat162_rn(tanhf(p.norm_alpha * v[j + 2 * t]) * w2.x + b2.x,
                                      tanhf(p.norm_alpha * v[j + 2 * t + 1]) * w2.y + b2.y);
      }
      *reinterpret_cast<uint4*>(p.C2 + static_cast<size_t>(grow) * p.ldc2 + gc + j) = ov;
    }
  }
}

// ---------------------------------------------------------------------------- host side: tensor maps
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// 2-D bf16 row-major tensor [rows, cols] with leading dimension ld (elements), box = [box_rows, 64]
inline int make_map(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return -1;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {BK, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

// 2-D packed-e2m1 matrix seen as bytes: [rows, row_bytes] with leading dimension ld_bytes, box = [box_rows, 128 bytes]
inline int make_map_u8(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t row_bytes, uint64_t ld_bytes, uint32_t box_rows) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return -1;
  cuuint64_t dims[2] = {row_bytes, rows};
  cuuint64_t strides[1] = {ld_bytes};
  cuuint32_t box[2] = {128, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

// Activation maps of a launch over M rows: full 128-row boxes, and the box of the last row tile (GemmParams::a_small_rows)
struct ActMaps { CUtensorMap full, last; };
inline int make_act_maps(ActMaps* m, GemmParams* p, const void* A, uint64_t cols, uint64_t ld, bool u8) {
  auto make = u8 ? make_map_u8 : make_map;
  p->a_small_rows = p->M % BM;
  if (make(&m->full, A, p->M, cols, ld, BM)) return -1;
  return p->a_small_rows > 0 ? make(&m->last, A, p->M, cols, ld, p->a_small_rows) : 0;
}

}  // namespace js
