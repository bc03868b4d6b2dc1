// Many-row bf16 GEMM for sm_100a:  C[M,N] = A[M,K] * W[N,K]^T on CTA pairs (prompt portions, batched verify).
// Reference twins: the library GEMMs of the fused verify stack, jetspec/inference_engine/compiled_verify_stack.py:170-272.
//
// Bound: the tensor cores, fed through the L2-to-SM path.  A pair of CTAs on neighbouring SMs owns one output tile of 256
// rows x TN columns (tcgen05.mma.cta_group::2): each CTA stages half of the rows of A and half of the rows of W and holds its
// 128 rows x TN columns of the accumulator.  At TN = 256 that is 32 KB for 512 tensor cycles of the SM (0.285 us a 64-wide
// k-block measured); TN = 128 is bound by the L2-to-SM path (24 KB, 0.19 us) and taken where half as wide tiles save a
// round.  Two accumulators take turns, so a tile's epilogue runs under the next tile's main loop, and the pairs are
// persistent (one CTA per SM): a 128 x 256 tile per CTA asked 1.5 times the bytes per FLOP, and a 256 x 256 tile per single
// CTA left nothing running during its epilogue.  Tiles go row tiles first, so that the pairs at work share weight
// tiles and the activations stay in L2.
// Measured at 2048 rows (us, before -> now): 6144 x 4096 91.6 -> 78.8, 24576 x 4096 with SwiGLU 388 -> 269 (1530 TFLOP/s),
// 151936 x 4096 with argmax 2037 -> 1542; 4096 x 4096 and 4096 x 12288 as before (49, 140).
//
// Roles per CTA (192 threads): warp 0 = TMA producer of this CTA's halves, warp 1 = tensor-memory owner and, in the pair's
// first CTA, the issuer of all MMAs, warps 2..5 = epilogue of this CTA's 128 rows.  Both CTAs' loads count on the
// first CTA's barriers; a commit frees the stage (and publishes the accumulator) in both.
#include "gemm_common.cuh"

namespace js {

constexpr int kPairThreads = 192;
constexpr int kPairRows = 256;                       // rows of a pair's tile
constexpr int kPairHalfA = BM * BK * 2;              // one CTA's rows of A in a stage
template <int TN>                                    // columns of a pair's tile: 128 or 256
struct PairSmem {
  static constexpr int kHalfW = TN / 2 * BK * 2;     // one CTA's rows of W
  static constexpr int kStage = kPairHalfA + kHalfW;
  static constexpr int kStages = 192 * 1024 / kStage;
  static constexpr int kBytes = kStages * kStage + 1024 + 256;
};

// ---- cta_group::2 forms
JS_DEVICE void tmem_alloc_pair(uint32_t* smem_result, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(cols) : "memory");
}
JS_DEVICE void tmem_relinquish_pair() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
JS_DEVICE void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// Tiled load into this CTA's shared memory whose bytes count on a barrier of the pair (a shared::cluster address).
JS_DEVICE void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
JS_DEVICE void umma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at this offset in both CTAs once every MMA issued so far by this thread has completed.
JS_DEVICE void umma_commit_pair(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b16 both;\n\tmov.b16 both, 3;\n\t"
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], both;\n\t}"
      ::"r"(smem_u32(bar)) : "memory");
}
JS_DEVICE void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// mbar_wait_warp for arrivals of the other CTA too.
JS_DEVICE bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, int* status, int code, uint32_t* gave_up) {
  for (uint32_t i = 0;; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if (i >= kSpinLimit && warp_gives_up(bar, parity, status, code, gave_up)) return false;
  }
}

// HALF (SwiGLU): every 2 HALF weight rows hold HALF gate rows and the HALF up rows of the same outputs
template <int EPI, int TN, int HALF>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW,
                 const __grid_constant__ CUtensorMap tmA2, GemmParams p) {
  constexpr int kPairStages = PairSmem<TN>::kStages, kPairStage = PairSmem<TN>::kStage, kPairHalfW = PairSmem<TN>::kHalfW;
  static_assert(EPI != EPI_SWIGLU || TN % (2 * HALF) == 0, "a tile holds whole gate | up blocks");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kPairStages * kPairStage);    // the first CTA's are used
  uint64_t* empty_bar = full_bar + kPairStages;
  uint64_t* accum_full = empty_bar + kPairStages;      // 2
  uint64_t* accum_free = accum_full + 2;               // 2, the first CTA's: 4 epilogue warps of each CTA arrive
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum_free + 2);
  uint32_t* gave_up = tmem_slot + 2;                   // of the producing and of the issuing warp

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int m_tiles = (p.M + kPairRows - 1) / kPairRows;
  const int tiles = m_tiles * ((p.N + TN - 1) / TN);
  const int nkb = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmW);
    if (p.a_small_rows > 0) tma_prefetch_desc(&tmA2);
    for (int s = 0; s < kPairStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accum_full[b], 1);
      mbar_init(&accum_free[b], 8);
    }
    gave_up[0] = gave_up[1] = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 2 * TN);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();          // the other CTA's barriers exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();

  // Warp-uniform loops, one elected lane issues (see gemm_bf16_kernel): with the loops under `if (lane == 0)` a k-block of
  // a 256 x 128 tile took 0.306 us instead of 0.19.
  if (warp == 0) {
    auto box_rows = [&](int m) {       // rows of the activation box of the 128 rows at m
      if (m >= p.M) return 0;
      return p.a_small_rows > 0 && p.M - m <= p.a_small_rows ? p.a_small_rows : BM;
    };
    const uint32_t full0 = map_to_cta(smem_u32(full_bar), 0);
    pdl_wait();
    int s = 0;
    uint32_t phase = 1;                // of the empty barriers: the first round finds every stage free
    bool ok = true;
    for (int t = pair; t < tiles && ok; t += pairs) {
      const int m0 = (t % m_tiles) * kPairRows, n0 = (t / m_tiles) * TN;
      const int m = m0 + static_cast<int>(rank) * BM, n = n0 + static_cast<int>(rank) * (TN / 2);
      const int rows = box_rows(m);
      const uint32_t bytes = static_cast<uint32_t>(2 * kPairHalfW + (box_rows(m0) + box_rows(m0 + BM)) * BK * 2);
      for (int kb = 0; kb < nkb; ++kb) {
        ok = mbar_wait_warp(&empty_bar[s], phase, p.status, kTimeoutEmpty, &gave_up[0]);
        if (!ok) break;
        if (elect_one()) {
          // The other CTA's bytes may land before this arrival: it passed its own copy of the empty barrier, so they
          // belong to the same phase, which cannot complete without the arrival.
          if (rank == 0) mbar_expect_tx(&full_bar[s], bytes);
          uint8_t* stage = smem + s * kPairStage;
          if (rows == BM) tma_load_2d_pair(stage, &tmA, full0 + 8 * s, kb * BK, m);
          else if (rows > 0) tma_load_2d_pair(stage, &tmA2, full0 + 8 * s, kb * BK, m);
          tma_load_2d_pair(stage + kPairHalfA, &tmW, full0 + 8 * s, kb * BK, n);
        }
        __syncwarp();
        if (++s == kPairStages) { s = 0; phase ^= 1; }
      }
    }
    // Every commit that frees a stage arrives here as well as in the other CTA: a CTA stays until the last of them has
    // landed, and with them its loads (a stage that was never filled counts as free).
    for (int i = 0; i < kPairStages && ok; ++i) {
      ok = mbar_wait_warp(&empty_bar[s], phase, p.status, kTimeoutEmpty, &gave_up[0]);
      if (++s == kPairStages) { s = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(kPairRows, TN);
      const uint64_t desc0 = umma_desc_sw128(smem_u32(smem));
      int s = 0, buf = 0;
      uint32_t phase = 0, free_phase = 1;
      bool ok = true;
      for (int t = pair; t < tiles && ok; t += pairs) {
        ok = mbar_wait_cluster(&accum_free[buf], free_phase, p.status, kTimeoutAccum, &gave_up[1]);
        tc_fence_after();
        const uint32_t acc = tmem_base + buf * TN;
        uint32_t more = 0;
        for (int kb = 0; kb < nkb && ok; ++kb) {
          ok = mbar_wait_cluster(&full_bar[s], phase, p.status, kTimeoutFull, &gave_up[1]);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            const uint64_t a_desc = desc0 + static_cast<uint64_t>(s * (kPairStage >> 4));
            const uint64_t b_desc = a_desc + (kPairHalfA >> 4);
            umma_f16_pair(acc, a_desc, b_desc, idesc, more);
#pragma unroll
            for (int k = 1; k < BK / UMMA_K; ++k) umma_f16_pair(acc, a_desc + 2 * k, b_desc + 2 * k, idesc, 1u);
            umma_commit_pair(&empty_bar[s]);
          }
          __syncwarp();
          more = 1;
          if (++s == kPairStages) { s = 0; phase ^= 1; }
        }
        if (elect_one()) umma_commit_pair(&accum_full[buf]);     // also releases the epilogues on an error path
        __syncwarp();
        if (buf) free_phase ^= 1;
        buf ^= 1;
      }
    }
  } else {
    const int quad = warp & 3, row = quad * 32 + lane;
    pdl_wait();                                  // residual / C may belong to the previous kernel
    bool ok = true;
    int j = 0;
    for (int t = pair; t < tiles && ok; t += pairs, ++j) {
      const int buf = j & 1;
      ok = warp_ok(mbar_wait(&accum_full[buf], (j >> 1) & 1, p.status, kTimeoutAccum));
      if (!ok) break;
      tc_fence_after();
      const int n0 = (t / m_tiles) * TN;
      const int grow = (t % m_tiles) * kPairRows + static_cast<int>(rank) * BM + row;
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(buf * TN);
      const bool valid = grow < p.M;
      auto load_chunk = [&](int c0, float* v) {
        uint32_t r[32];
        tmem_ld_32x32(t_row + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
      };
      if constexpr (EPI == EPI_SWIGLU) {
#pragma unroll 1
        for (int c0 = 0; c0 < TN / 2; c0 += 32) {
          const int at = c0 / HALF * (2 * HALF) + c0 % HALF, gc = n0 / 2 + c0;
          float g[32], u[32];
          load_chunk(at, g);
          load_chunk(at + HALF, u);
          if (valid && gc < p.N / 2) epi_swiglu_chunk(p, grow, gc, g, u);
        }
      } else if constexpr (EPI == EPI_INPROJ) {
#pragma unroll 1
        for (int c0 = 0; c0 < TN / 2; c0 += 32) {
          const int nb = n0 + (c0 >> 6) * 128, cb = c0 & 63;
          float g[32], u[32];
          load_chunk((c0 >> 6) * 128 + cb, g);
          load_chunk((c0 >> 6) * 128 + 64 + cb, u);
          if (valid && nb < p.N) epi_inproj_halves(p, grow, nb, cb, g, u);
        }
      } else if constexpr (EPI == EPI_ARGMAX) {
        // one partial per 128 columns, as the single-CTA kernel leaves them
        const int n_part = (p.N + 127) / 128;
#pragma unroll 1
        for (int h = 0; h < TN / 128; ++h) {
          float best = -INFINITY;
          int best_i = 0x7fffffff;
#pragma unroll 1
          for (int c0 = 0; c0 < 128; c0 += 32) {
            float v[32];
            load_chunk(h * 128 + c0, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const int gc = n0 + h * 128 + c0 + i;
              if (gc < p.N && v[i] > best) { best = v[i]; best_i = gc; }
            }
          }
          const int part = n0 / 128 + h;
          if (valid && part < n_part) {
            p.part_val[static_cast<size_t>(grow) * n_part + part] = best;
            p.part_idx[static_cast<size_t>(grow) * n_part + part] = best_i;
          }
        }
      } else {
#pragma unroll 1
        for (int c0 = 0; c0 < TN; c0 += 32) {
          float v[32];
          load_chunk(c0, v);
          const int gc = n0 + c0;
          if (valid && gc < p.N) {
            if constexpr (EPI == EPI_RESID32) epi_resid32_chunk(p, grow, gc, v);
            else epi_store_chunk<EPI>(p, grow, gc, v, 0);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&accum_free[buf]), 0));
    }
  }

  // Nobody leaves while the pair's MMAs may still read its shared memory or an arrival may still land there: the commits
  // were waited for above, the other CTA's arrivals on accum_free come before it joins this barrier.
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * TN);
  }
}

template <int EPI, int TN, int HALF = 64>
static int launch_pair(const void* A, const void* W, GemmParams p, int lda, int ldw, bool pdl, cudaStream_t stream) {
  static int configured[kMaxDevicesCached] = {};
  static int room[kMaxDevicesCached] = {};      // pairs that are resident at once, 0 = not asked yet
  auto kern = gemm_pair_kernel<EPI, TN, HALF>;
  ActMaps ta;
  CUtensorMap tw;
  if (make_act_maps(&ta, &p, A, p.K, lda, false) || make_map(&tw, W, p.N, p.K, ldw, TN / 2)) return -16;
  if (ensure_dyn_smem(kern, PairSmem<TN>::kBytes, configured) != 0) return -3;
  const int tiles = ((p.M + kPairRows - 1) / kPairRows) * ((p.N + TN - 1) / TN);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * tiles);
  cfg.blockDim = dim3(kPairThreads);
  cfg.dynamicSmemBytes = PairSmem<TN>::kBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -3;
  int n = dev >= 0 && dev < kMaxDevicesCached ? __atomic_load_n(&room[dev], __ATOMIC_RELAXED) : 0;
  if (n == 0) {
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = 64;
    }
    if (dev >= 0 && dev < kMaxDevicesCached) __atomic_store_n(&room[dev], n, __ATOMIC_RELAXED);
  }
  cfg.gridDim = dim3(2 * (tiles < n ? tiles : n));
  cfg.numAttrs = pdl ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, ta.full, tw, p.a_small_rows > 0 ? ta.last : ta.full, p) == cudaSuccess ? 0 : -4;
}

static int pair_args(const void* A, const void* W, int K, int lda, int ldw) {
  if ((K % 8) || (lda % 8) || (ldw % 8)) return -10;           // TMA: 16-byte aligned rows
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) return -11;
  return 0;
}

}  // namespace js

// js_gemm_bf16 on CTA pairs.  epi: 0 store (+ residual), 1 swiglu (`half` 64 or 128: gate rows, then as many up rows), 2 argmax
// partials of 128 columns each.  tn: columns of a tile, 128 or 256.
extern "C" int js_gemm_pair(const void* A, const void* W, void* C, const void* residual, int M, int N, int K, int lda, int ldw,
                            int ldc, int epi, int tn, int half, float* part_val, int* part_idx, int* status, int pdl,
                            cudaStream_t stream) {
  using namespace js;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (const int rc = pair_args(A, W, K, lda, ldw)) return rc;
  if ((epi == EPI_STORE || epi == EPI_SWIGLU) && ((ldc % 8) || (N % 8))) return -15;
  if (epi == EPI_ARGMAX && (part_val == nullptr || part_idx == nullptr)) return -22;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.C = C; p.status = status; p.world = 1;
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  p.part_val = part_val; p.part_idx = part_idx;
#define JS_PAIR(TN_)                                                                                               \
  if (tn == TN_) {                                                                                                 \
    if (epi == EPI_STORE) return launch_pair<EPI_STORE, TN_>(A, W, p, lda, ldw, pdl != 0, stream);                 \
    if (epi == EPI_ARGMAX) return launch_pair<EPI_ARGMAX, TN_>(A, W, p, lda, ldw, pdl != 0, stream);               \
    if (epi == EPI_SWIGLU && N % 128 == 0 && half == 64) return launch_pair<EPI_SWIGLU, TN_, 64>(A, W, p, lda, ldw, pdl != 0, stream); \
  }
  JS_PAIR(128) JS_PAIR(256)
#undef JS_PAIR
  if (tn == 256 && epi == EPI_SWIGLU && N % 256 == 0 && half == 128)
    return launch_pair<EPI_SWIGLU, 256, 128>(A, W, p, lda, ldw, pdl != 0, stream);
  return -17;
}

// js_gemm_inproj on CTA pairs (same arguments; `tn` is the tile's width).
extern "C" int js_gemm_inproj_pair(const void* A, const void* W, float* C, void* C2, int M, int N, int K, int lda, int ldw, int ldc,
                                   int ldc2, int n_raw, int act, float act_a, float act_b, int tn, int* status, int pdl,
                                   cudaStream_t stream) {
  using namespace js;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (const int rc = pair_args(A, W, K, lda, ldw)) return rc;
  if ((N % 128) || (n_raw % 128) || n_raw < 0 || n_raw > N || (ldc % 4) || (ldc2 % 8) || act < 0 || act > 4) return -15;
  if ((n_raw > 0 && (C == nullptr || ldc < n_raw)) || (n_raw < N && C2 == nullptr)) return -22;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.C = C; p.status = status; p.world = 1;
  p.C2 = reinterpret_cast<__nv_bfloat16*>(C2); p.ldc2 = ldc2; p.n_raw = n_raw; p.act = act; p.act_a = act_a; p.act_b = act_b;
  return tn == 128   ? launch_pair<EPI_INPROJ, 128>(A, W, p, lda, ldw, pdl != 0, stream)
         : tn == 256 ? launch_pair<EPI_INPROJ, 256>(A, W, p, lda, ldw, pdl != 0, stream) : -17;
}

// js_gemm_resid32 on CTA pairs (same arguments; `tn` is the tile's width).
extern "C" int js_gemm_resid32_pair(const void* A, const void* W, float* x_out, const float* x_in, int M, int N, int K, int lda,
                                    int ldw, int ldx, const void* emb, int ld_emb, void* h, int ldh, const float* norm_w,
                                    const float* norm_b, float norm_alpha, int tn, int* status, int pdl, cudaStream_t stream) {
  using namespace js;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (const int rc = pair_args(A, W, K, lda, ldw)) return rc;
  if ((N % 8) || (ldx % 4) || (ld_emb % 8) || (ldh % 8)) return -10;
  if (norm_w != nullptr && (norm_b == nullptr || h == nullptr)) return -22;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.ldc = ldx; p.C = x_out; p.status = status; p.world = 1;
  p.res32 = x_in; p.emb = reinterpret_cast<const __nv_bfloat16*>(emb); p.ld_emb = ld_emb;
  p.C2 = reinterpret_cast<__nv_bfloat16*>(h); p.ldc2 = ldh; p.norm_w = norm_w; p.norm_b = norm_b; p.norm_alpha = norm_alpha;
  return tn == 128   ? launch_pair<EPI_RESID32, 128>(A, W, p, lda, ldw, pdl != 0, stream)
         : tn == 256 ? launch_pair<EPI_RESID32, 256>(A, W, p, lda, ldw, pdl != 0, stream) : -17;
}
