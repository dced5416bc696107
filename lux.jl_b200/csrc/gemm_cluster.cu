// Tensor-core GEMM for problems with too few output tiles to fill the GPU (small layers, inference on a handful of columns):
//   D[Mm x Nn] = A[Mm x Kc] * B[Nn x Kc]^T, 128 x 64 tiles, the contraction of a tile split over the CTAs of one cluster.
//
// The CTAs of a cluster (up to 8) each take a range of k-blocks of the same tile, leave their fp32 partial in their own shared
// memory and, after a cluster barrier, each adds every partial of its share of the columns through distributed shared memory
// in rank order (deterministic), applies bias and activation and stores. One launch, no workspace.
//
// bf16: operands through TMA as in gemm_tc.cu. Float32: sixteen worker warps read the operands with plain loads (any leading
// dimension, any alignment), split them into tf32 hi / lo on the way and write both as K-major swizzled tiles, so the
// separate split passes and their copies are not needed; the same warps take the partial products out of TMEM (two k-steps of
// hi*hi per accumulator, the small products in one accumulator) and add them in fp32 registers. Error against 64 bits 0.9e-7 to
// 1.6e-7 (gemm_tc_f32acc_kernel, which took these products before: 0.9e-7 to 3.2e-7); an infinite operand gives NaN, as there.
//
// Measured against the kernels of gemm_tc.cu (which the larger shapes keep), forward with bias and activation: bf16 4096 x 8 x
// 4096 14.5 us (28.8; 33.5 MB of weights at 2.3 TB/s), 256 x 8 x 8192 12.5 us (49); Float32 4096 x 8 x 4096 47 us (169),
// 1001 x 300 x 515 17 us (55), 256 x 128 x 784 14 us (60). Float32 1024 x 2048 x 1024 (256 tiles) was 103 us against 73: the
// line between the two lies at one wave of tiles.
// What bounds it: one pass over the operands from HBM / L2 and the latency of a short chain (load, MMA, cluster barrier).
#include "gemm.cuh"
#include "tc_ptx.cuh"

namespace lb2 {

namespace {

constexpr int kClBM = 128, kClBN = 64;
constexpr int kClWorkers = 16;           // warps that load (Float32), accumulate and store; then one for MMA and TMEM, one for TMA (bf16).
                                         // Eight left the Float32 loop waiting on its own instructions (2 warps per scheduler).
constexpr int kClThreads = (kClWorkers + 2) * 32;
constexpr int kClMaxSplits = 8;          // portable cluster size

template <bool F32> struct ClCfg {
  static constexpr int A_BYTES = kClBM * 128, B_BYTES = kClBN * 128;
  static constexpr int STAGE_BYTES = (A_BYTES + B_BYTES) * (F32 ? 2 : 1);     // Float32: [A_hi | A_lo | B_hi | B_lo]
  static constexpr int STAGES = F32 ? 4 : 8;
  static constexpr int SLOTS = F32 ? 7 : 0;                                   // TMEM ring of 64-column accumulators + one for the small products
  static constexpr int TMEM_COLS = F32 ? 512 : 64;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 512;
};

struct ClParams {
  GemmTmaPlan a, b;                      // bf16
  const float *A, *B;                    // Float32
  int64_t lda, ldb;
  int32_t a_vec, b_vec;                  // 16-byte loads along K allowed
  int32_t Mm, Nn, Kc;
  int32_t tiles_m, num_kb, splits, kb_per_split;
  uint32_t idesc;
  void* D;
  int64_t ldd;
  const void* bias;
  void* preact;
  int32_t act, accumulate;
  unsigned int* status;
};

// hi = v rounded to 11 significant bits, ties away from zero (two integer operations: the conversion instruction takes seven
// cycles for eight warps, and this loop is issue-bound); lo = v - hi
__device__ __forceinline__ void cl_split(float v, float& hi, float& lo) {
  hi = __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xFFFFE000u);
  lo = v - hi;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// Loads that stay where they are written (two k-blocks ahead of their use): the compiler would sink plain ones to it.
__device__ __forceinline__ float cl_ld(const float* p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void cl_ld4(float (&v)[4], const float* p) {
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p));
}

// How a thread walks one Float32 operand: U units of four consecutive contracted elements of one row per k-block, U * 64 rows
// x 32 elements for the sixteen warps. MN (rows contiguous): lanes along the rows, a warp per half of the rows and group of
// four k, one pointer per k. K-major: eight lanes along k, four rows per warp, one pointer per unit.
template <int U, bool MN> struct ClWalk {
  static constexpr int P = MN ? 4 : U;
  const float* ptr[P];
  int64_t step;              // elements from one k-block to the next
  uint32_t live;             // bit u: the unit's row exists
  int k_in;                  // first contracted index of the thread inside a k-block
  bool vec;
  uint32_t off[U];           // where the unit lands in the K-major, 128-byte swizzled tile

  __device__ __forceinline__ ClWalk(const float* p, int64_t ld, bool v, int row0, int rows, int k0, int warp, int lane) {
    static_assert(kClWorkers == 16, "two halves of the rows x eight groups of k");
    const int kg = MN ? (warp & 7) : (lane & 7);
    const int r_in = MN ? (warp >> 3) * (U * 32) + lane : warp * 4 + (lane >> 3);
    constexpr int R_STEP = MN ? 32 : 64;
    k_in = kg * 4;
    vec = v;
    live = 0;
    step = MN ? 32 * ld : 32;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int row = u * R_STEP + r_in;
      if (row0 + row < rows) live |= 1u << u;
      off[u] = (uint32_t)(row * 128 + ((kg ^ (row & 7)) << 4));
    }
#pragma unroll
    for (int j = 0; j < P; ++j)
      ptr[j] = MN ? p + row0 + r_in + (int64_t)(k0 + k_in + j) * ld : p + k0 + k_in + (int64_t)(row0 + j * R_STEP + r_in) * ld;
  }
  // the k-block at the pointers, of which `k_left` contracted elements exist; advances them
  __device__ __forceinline__ void load(float (&v)[U][4], int k_left) {
    if (live == (1u << U) - 1u && k_left >= 32) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if constexpr (MN) {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[u][j] = cl_ld(ptr[j] + u * 32);
        } else if (vec) {
          cl_ld4(v[u], ptr[u]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[u][j] = cl_ld(ptr[u] + j);
        }
      }
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          v[u][j] = ((live >> u) & 1u) != 0 && k_in + j < k_left ? cl_ld(MN ? ptr[MN ? j : 0] + u * 32 : ptr[MN ? 0 : u] + j) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < P; ++j) ptr[j] += step;
  }
  __device__ __forceinline__ void store(const float (&v)[U][4], uint32_t s_hi, uint32_t lo_off) const {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float h[4], l[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) cl_split(v[u][j], h[j], l[j]);
      sts128(s_hi + off[u], h[0], h[1], h[2], h[3]);
      sts128(s_hi + lo_off + off[u], l[0], l[1], l[2], l[3]);
    }
  }
};

template <bool F32, int ACT, bool A_MN, bool B_MN>   // A_MN, B_MN: Float32 only
__global__ void __launch_bounds__(kClThreads, 1)
gemm_cluster_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ ClParams p) {
  using Cfg = ClCfg<F32>;
  using T = typename std::conditional<F32, float, __nv_bfloat16>::type;
  constexpr int STAGES = Cfg::STAGES, SLOTS = Cfg::SLOTS, BN = kClBN, COLS = BN * 4 / kClWorkers;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_gen + STAGES * Cfg::STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* acc_full = bars + 2 * STAGES;        // [SLOTS] ring, [SLOTS] = small products (Float32) / the accumulator (bf16)
  uint64_t* acc_empty = acc_full + SLOTS + 1;    // [SLOTS]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + SLOTS);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / p.splits, rank = blockIdx.x - tile * p.splits;
  const int m0 = (tile % p.tiles_m) * kClBM, n0 = (tile / p.tiles_m) * BN;
  const int kb_lo = rank * p.kb_per_split, kb_hi = min(p.num_kb, kb_lo + p.kb_per_split);
  const int n_kb = kb_hi > kb_lo ? kb_hi - kb_lo : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], F32 ? kClWorkers : 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a <= SLOTS; ++a) mbar_init(&acc_full[a], 1);
    for (int a = 0; a < SLOTS; ++a) mbar_init(&acc_empty[a], kClWorkers);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kClWorkers) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  float sum[COLS];
#pragma unroll
  for (int j = 0; j < COLS; ++j) sum[j] = 0.f;

  if (warp == kClWorkers + 1) {
    if constexpr (!F32) {
      uint32_t stage = 0, phase = 0;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait_uniform(&empty[stage], phase ^ 1u, p.status, 0x1u)) break;
        if (elect_one()) {
          mbar_expect_tx(&full[stage], Cfg::STAGE_BYTES);
          const uint32_t sA = smem_base + stage * Cfg::STAGE_BYTES, sB = sA + Cfg::A_BYTES;
          const int k0 = kb * 64;
          for (int bx = 0; bx < p.a.boxes; ++bx)
            tma_load_2d(sA + bx * p.a.box_bytes, &tmA, p.a.mn_major ? m0 + bx * p.a.mn_step : k0, p.a.mn_major ? k0 : m0, &full[stage]);
          for (int bx = 0; bx < p.b.boxes; ++bx)
            tma_load_2d(sB + bx * p.b.box_bytes, &tmB, p.b.mn_major ? n0 + bx * p.b.mn_step : k0, p.b.mn_major ? k0 : n0, &full[stage]);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == kClWorkers) {
    uint32_t stage = 0, phase = 0, slot = 0, slot_phase = 0;
    bool ok = true;
    for (int i = 0; i < n_kb && ok; ++i) {
      if (!mbar_wait_uniform(&full[stage], phase, p.status, 0x4u)) { ok = false; break; }
      tc_fence_after();
      const uint32_t sA = smem_base + stage * Cfg::STAGE_BYTES, sB = sA + Cfg::A_BYTES * (F32 ? 2 : 1);
      if constexpr (F32) {
        // The workers' plain stores become visible to the tensor core here, behind their arrivals.
        fence_proxy_async_smem();
        constexpr uint32_t DESC = (uint32_t)((1024u >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
        constexpr uint32_t A_LO = Cfg::A_BYTES >> 4, B_LO = Cfg::B_BYTES >> 4;
        const uint64_t top = (uint64_t)DESC << 32;
        const uint32_t a32 = ((sA >> 4) & 0x3FFFu) | (1u << 16), b32 = ((sB >> 4) & 0x3FFFu) | (1u << 16);
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          if (!mbar_wait_uniform(&acc_empty[slot], slot_phase ^ 1u, p.status, 0x2u)) { ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int ks = 2 * part; ks < 2 * part + 2; ++ks)
              umma<true>(tmem_base + slot * BN, top | (uint64_t)(a32 + 2 * ks), top | (uint64_t)(b32 + 2 * ks), p.idesc, ks != 2 * part ? 1u : 0u);
            umma_commit(&acc_full[slot]);
#pragma unroll
            for (int ks = 2 * part; ks < 2 * part + 2; ++ks) {
              umma<true>(tmem_base + SLOTS * BN, top | (uint64_t)(a32 + 2 * ks), top | (uint64_t)(b32 + B_LO + 2 * ks), p.idesc, (i | ks) != 0 ? 1u : 0u);
              umma<true>(tmem_base + SLOTS * BN, top | (uint64_t)(a32 + A_LO + 2 * ks), top | (uint64_t)(b32 + 2 * ks), p.idesc, 1u);
            }
            if (part == 1) umma_commit(&empty[stage]);
          }
          __syncwarp();
          if (++slot == SLOTS) { slot = 0; slot_phase ^= 1u; }
        }
        if (!ok) break;
      } else {
        const uint32_t a32 = ((sA >> 4) & 0x3FFFu) | p.a.desc_lbo, b32 = ((sB >> 4) & 0x3FFFu) | p.b.desc_lbo;
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma<false>(tmem_base, ((uint64_t)p.a.desc_hi << 32) | (uint64_t)(a32 + ks * p.a.k_advance),
                        ((uint64_t)p.b.desc_hi << 32) | (uint64_t)(b32 + ks * p.b.k_advance), p.idesc, (i | ks) != 0 ? 1u : 0u);
          umma_commit(&empty[stage]);
        }
        __syncwarp();
      }
      if (++stage == STAGES) { stage = 0; phase ^= 1u; }
    }
    if (ok && n_kb > 0 && elect_one()) umma_commit(&acc_full[SLOTS]);
    __syncwarp();
  } else {
    const uint32_t tmem_lane = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * COLS;
    bool ok = true;
    if constexpr (F32) {
      uint32_t stage = 0, phase = 0, slot = 0, slot_phase = 0;
      // a k-block's two hi*hi accumulators, added to each other and then to the sum
      auto drain = [&]() {
        const uint32_t s0 = slot, p0 = slot_phase;
        if (++slot == SLOTS) { slot = 0; slot_phase ^= 1u; }
        const uint32_t s1 = slot, p1 = slot_phase;
        if (++slot == SLOTS) { slot = 0; slot_phase ^= 1u; }
        if (!mbar_wait_warp(&acc_full[s0], p0, p.status, 0x8u) || !mbar_wait_warp(&acc_full[s1], p1, p.status, 0x8u)) return false;
        tc_fence_after();
        uint32_t r0[COLS], r1[COLS];
        tmem_ld16(tmem_lane + s0 * BN, r0);
        tmem_ld16(tmem_lane + s1 * BN, r1);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { mbar_arrive(&acc_empty[s0]); mbar_arrive(&acc_empty[s1]); }
#pragma unroll
        for (int j = 0; j < COLS; ++j) sum[j] += __uint_as_float(r0[j]) + __uint_as_float(r1[j]);
        return true;
      };
      float a0[2][4], b0[1][4], a1[2][4], b1[1][4];   // the next two k-blocks, on their way from memory
      ClWalk<2, A_MN> wa(p.A, p.lda, p.a_vec != 0, m0, p.Mm, kb_lo * 32, warp, lane);
      ClWalk<1, B_MN> wb(p.B, p.ldb, p.b_vec != 0, n0, p.Nn, kb_lo * 32, warp, lane);
      int k_left = p.Kc - kb_lo * 32, loaded = 0;
      auto load = [&](float (&a)[2][4], float (&b)[1][4]) {
        if (loaded >= n_kb) return;
        wa.load(a, k_left);
        wb.load(b, k_left);
        k_left -= 32;
        ++loaded;
      };
      auto step = [&](float (&a)[2][4], float (&b)[1][4], int i) {
        if (!mbar_wait_warp(&empty[stage], phase ^ 1u, p.status, 0x10u)) return false;
        const uint32_t sA = smem_base + stage * Cfg::STAGE_BYTES;
        wa.store(a, sA, Cfg::A_BYTES);
        wb.store(b, sA + 2 * Cfg::A_BYTES, Cfg::B_BYTES);
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        load(a, b);
        return i == 0 || drain();
      };
      load(a0, b0);
      load(a1, b1);
      for (int i = 0; i < n_kb; i += 2) {
        if (!step(a0, b0, i)) { ok = false; break; }
        if (i + 1 < n_kb && !step(a1, b1, i + 1)) { ok = false; break; }
      }
      if (ok && n_kb > 0) ok = drain();
    }
    if (ok && n_kb > 0) {
      if (mbar_wait_warp(&acc_full[SLOTS], 0u, p.status, 0x20u)) {
        tc_fence_after();
        uint32_t r[COLS];
        tmem_ld16(tmem_lane + SLOTS * BN, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < COLS; ++j) sum[j] += __uint_as_float(r[j]);
      }
    }
  }

  // ---------------- epilogue ----------------
  __syncwarp();
  T* D = static_cast<T*>(p.D);
  T* P = static_cast<T*>(p.preact);
  const T* bias = static_cast<const T*>(p.bias);
  auto put = [&](float v, int m, int n, float bv) {
    const int64_t off = (int64_t)n * p.ldd + m;
    v += bv;
    if (P != nullptr) P[off] = from_f32<T>(v);
    v = act_apply_any<ACT, !F32>(p.act, v);
    if (p.accumulate) v += to_f32(D[off]);
    D[off] = from_f32<T>(v);
  };
  if (p.splits == 1) {
    if (warp < kClWorkers) {
      const int m = m0 + (warp & 3) * 32 + lane, c0 = n0 + (warp >> 2) * COLS;
      if (m < p.Mm) {
        const float bv = bias != nullptr ? to_f32(bias[m]) : 0.f;
#pragma unroll
        for (int j = 0; j < COLS; ++j)
          if (c0 + j < p.Nn) put(sum[j], m, c0 + j, bv);
      }
    }
  } else {
    // every MMA of this CTA has finished, so its ring is free: the partial goes there as [column][128 rows]
    float* park = reinterpret_cast<float*>(smem_gen);
    if (warp < kClWorkers) {
#pragma unroll
      for (int j = 0; j < COLS; ++j) park[((warp >> 2) * COLS + j) * kClBM + (warp & 3) * 32 + lane] = sum[j];
    }
    cluster_sync_all();
    if (warp < kClWorkers) {
      const int row = (warp & 3) * 32 + lane, m = m0 + row;
      const int cols = min(BN, p.Nn - n0);
      if (m < p.Mm) {
        const float bv = bias != nullptr ? to_f32(bias[m]) : 0.f;
        for (int c = rank + (warp >> 2) * p.splits; c < cols; c += (kClWorkers / 4) * p.splits) {
          const uint32_t local = smem_base + (uint32_t)(c * kClBM + row) * 4u;
          float v = 0.f;
          for (int z = 0; z < p.splits; ++z) v += ld_cluster_f32(map_to_cta(local, (uint32_t)z));
          put(v, m, n0 + c, bv);
        }
      }
    }
  }
  __syncwarp();                           // rows past the last took no part above; the barrier wants whole warps
  tc_fence_before();
  if (p.splits > 1) cluster_sync_all();   // nobody leaves while its partial may still be read
  else __syncthreads();
  if (warp == kClWorkers) {
    if (*reinterpret_cast<volatile unsigned int*>(p.status) != 0) drain_after_abort();
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// Splits of the contraction of `tiles` tiles with `kb` k-blocks each: the count whose waves of k-blocks (plus about six
// k-blocks' time for a tile's start and end, two more for the cluster's exchange) are shortest.
int cl_splits(int64_t tiles, int kb) {
  const int sms = sm_count();
  int best = 1, best_cost = 0;
  for (int s = 1; s <= kClMaxSplits && s <= kb; ++s) {
    const int waves = (int)((tiles * s + sms - 1) / sms);
    const int cost = waves * ((kb + s - 1) / s + (s > 1 ? 8 : 6));
    if (s == 1 || cost < best_cost) { best = s; best_cost = cost; }
  }
  return best;
}

}  // namespace

// Where this kernel is the better one: bf16, when 128 x 64 tiles leave at least half of the SMs idle; Float32, as long as one
// wave of 128 x 64 tiles covers the result (1024 x 1024 x 1024: 47 against 68 us; beyond, the split passes of gemm_tc.cu are
// small beside the product).
bool gemm_cluster_wanted(int64_t Mm, int64_t Nn, int64_t Kc, int32_t dtype) {
  if (Mm > 0x7FFFFFFF - 128 || Nn > 0x7FFFFFFF - 128 || Kc > 0x7FFFFFFF - 128) return false;
  const int64_t tiles = ((Mm + kClBM - 1) / kClBM) * ((Nn + kClBN - 1) / kClBN);
  return dtype == LB2_F32 ? tiles <= sm_count() : 2 * tiles <= sm_count();
}

int32_t gemm_cluster_launch(void* D, int64_t ldd, GemmOperand A, GemmOperand B, int64_t Mm, int64_t Nn, int64_t Kc, int32_t dtype,
                            const GemmEpilogue& epi, cudaStream_t st) {
  ClParams p{};
  CUtensorMap mA{}, mB{};
  const bool f32 = dtype == LB2_F32;
  if (f32) {
    p.A = static_cast<const float*>(A.ptr); p.B = static_cast<const float*>(B.ptr);
    p.lda = A.ld; p.ldb = B.ld;
    p.a_vec = aligned_to(A.ptr, 16) && A.ld % 4 == 0; p.b_vec = aligned_to(B.ptr, 16) && B.ld % 4 == 0;
  } else if (!gemm_tma_map(&mA, A, Mm, Kc, 2, kClBM, 64, &p.a, false) || !gemm_tma_map(&mB, B, Nn, Kc, 2, kClBN, 64, &p.b, false)) {
    return fail(LB2_LAUNCH_FAIL, "gemm_cluster: cuTensorMapEncodeTiled failed");
  }
  p.Mm = (int)Mm; p.Nn = (int)Nn; p.Kc = (int)Kc;
  p.tiles_m = (int)((Mm + kClBM - 1) / kClBM);
  const int64_t tiles = (int64_t)p.tiles_m * ((Nn + kClBN - 1) / kClBN);
  const int bk = f32 ? 32 : 64;
  p.num_kb = (int)((Kc + bk - 1) / bk);
  const int s = cl_splits(tiles, p.num_kb);
  p.kb_per_split = (p.num_kb + s - 1) / s;
  p.splits = (p.num_kb + p.kb_per_split - 1) / p.kb_per_split;
  const uint32_t fmt = f32 ? 2u : 1u;
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((!f32 && A.mn_major ? 1u : 0u) << 15) | ((!f32 && B.mn_major ? 1u : 0u) << 16) |
            ((uint32_t)(kClBN >> 3) << 17) | ((uint32_t)(kClBM >> 4) << 24);
  p.D = D; p.ldd = ldd; p.bias = epi.bias; p.preact = epi.preact; p.act = epi.act; p.accumulate = epi.accumulate;
  p.status = device_status_word();
  LB2_REQUIRE(p.status != nullptr, LB2_LAUNCH_FAIL, "gemm_cluster: device status word unavailable");
  auto launch = [&](auto kernel, int smem) -> int32_t {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail(LB2_LAUNCH_FAIL, "gemm_cluster: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * p.splits), 1, 1);
    cfg.blockDim = dim3(kClThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kernel, mA, mB, p);
    if (e != cudaSuccess) return fail(LB2_LAUNCH_FAIL, "gemm_cluster: %s", cudaGetErrorString(e));
    return LB2_OK;
  };
  record_gemm_plan(3, kClBM, kClBN, (int)tiles, (int)(tiles * p.splits), (int)tiles, (int)(tiles * p.splits));
  const bool plain = p.act == LB2_ACT_IDENTITY;
  if (f32) {
    auto pick = [&](auto mn_a, auto mn_b) -> int32_t {
      constexpr bool MA = decltype(mn_a)::value, MB = decltype(mn_b)::value;
      return plain ? launch(gemm_cluster_kernel<true, LB2_ACT_IDENTITY, MA, MB>, ClCfg<true>::SMEM_BYTES)
                   : launch(gemm_cluster_kernel<true, -1, MA, MB>, ClCfg<true>::SMEM_BYTES);
    };
    if (A.mn_major) return B.mn_major ? pick(std::true_type{}, std::true_type{}) : pick(std::true_type{}, std::false_type{});
    return B.mn_major ? pick(std::false_type{}, std::true_type{}) : pick(std::false_type{}, std::false_type{});
  }
  return plain ? launch(gemm_cluster_kernel<false, LB2_ACT_IDENTITY, false, false>, ClCfg<false>::SMEM_BYTES)
               : launch(gemm_cluster_kernel<false, -1, false, false>, ClCfg<false>::SMEM_BYTES);
}

}  // namespace lb2
