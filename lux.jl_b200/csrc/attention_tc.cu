// Scaled dot-product attention and its pullback on the tensor cores: the six products of
// lib/LuxLib/src/impl/attention.jl:76-118 (logits, x; dw, dq, dk, dv) as ONE launch each over all heads and samples, with
// the softmax passes between them.
//
// Every product is D[m][n] = sum over k of A[m][k] * B[n][k] per (head, sample) with n contiguous in D:
//   logits[l][s] = q . k      dw[l][s] = dx . v        M = queries, N = keys
//   x[l][e] = w . v           dq[l][d] = dl . k        M = queries, contraction over the keys
//   dk[s][d] = dl' . q        dv[s][e] = w' . dx       M = keys, contraction over the queries of all heads that share the key
// The arrays are read through TMA maps (feature, head, token, sample; Float32: part), bf16 in place; either index of an
// operand may be the contiguous one (K-major / MN-major shared-memory descriptors), so nothing is transposed. A causal mask
// skips the tiles and the k-blocks that are zero.
// bf16: one accumulator per tile, two in flight. Float32: operands in three bf16 parts (parts.cuh), six products per k-block,
// k-blocks added in fp32 registers.
//
// Measured, forward + pullback through the operator, 8 heads x 8 samples, 512 x 512, 64 features, causal, bf16: 122 us (one
// tensor-core GEMM launch per head, sample and product before: 4.1 ms); Float32 4 x 4, 771 x 771: 285 us (3.07 ms;
// 270 us with two tf32 parts, whose results were further from 64 bits than fp32 sums).
// What bounds it: a contraction over a head's 64 features is one k-block, so the products move the S x L weights and little
// else; the passes over the weights (in L2 for the usual sizes) are the cost.
#include "common.cuh"
#include "parts.cuh"

namespace lb2 {

namespace {

constexpr int kAtThreads = 384;    // warps 0-2: TMA / MMA / TMEM, warps 4-11: epilogue
constexpr int kAtBM = 128;

struct AtOperand {
  int32_t boxes, box_bytes, mn_step, mn_major, head_first, head_div;   // Float32: a box holds all parts
  uint32_t desc_hi, lbo, k_adv, part;
};
enum { kCausalNone = 0, kCausalTiles = 1, kCausalKeys = 2, kCausalQueries = 3 };
struct AtParams {
  AtOperand a, b;
  int32_t bk, tiles_m, tiles_n, heads, rep, batch, num_kb;
  int32_t M, N;                      // N rounded up to the vector the rows of D are padded to
  int32_t causal;                    // which of the enum's rules applies to this product
  int32_t wide;                      // rows of D start on 32-byte boundaries: whole sectors per store
  uint32_t idesc;
  void* D;
  int64_t ldd, head_stride, batch_stride;
  unsigned int* status;
};

template <int BN, bool F32> struct AtCfg {
  static constexpr int ROW = F32 ? 64 : 128;                                // bytes of a k-block's row: 32 / 64 elements
  static constexpr int A_BYTES = kAtBM * ROW, B_BYTES = BN * ROW;           // one part
  static constexpr int PARTS = F32 ? 3 : 1;
  static constexpr int STAGE_BYTES = (A_BYTES + B_BYTES) * PARTS;           // F32: [A1 | A2 | A3 | B1 | B2 | B3]; MN-major: boxes of all parts
  static constexpr int STAGES = (200 * 1024) / STAGE_BYTES < 6 ? (200 * 1024) / STAGE_BYTES : 6;
  static constexpr int ACC_COLS = F32 ? 2 * BN : BN;                        // F32: [A1*B1 | the small products] of one k-block
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
};

template <bool F32>
__device__ __forceinline__ void at_load(uint32_t dst, const CUtensorMap* map, const AtOperand& o, int mn, int k, int head, int img, uint64_t* bar) {
  const int inner = o.mn_major ? mn : k, outer = o.mn_major ? k : mn;
  const int c1 = o.head_first ? head : outer, c2 = o.head_first ? outer : head;
  if constexpr (F32) tma_load_5d(dst, map, inner, c1, c2, img, 0, bar);
  else tma_load_4d(dst, map, inner, c1, c2, img, bar);
}

__device__ __forceinline__ void at_store32(void* p, const uint32_t (&w)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]),
               "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

template <int BN, bool F32>
__global__ void __launch_bounds__(kAtThreads, 1)
attn_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ AtParams p) {
  using Cfg = AtCfg<BN, F32>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_gen + STAGES * Cfg::STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* acc_full = bars + 2 * STAGES;    // [2] bf16: a tile; F32: one k-block of products
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t num_items = (int64_t)p.tiles_m * p.tiles_n * p.heads * p.batch;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 8); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 2 * Cfg::ACC_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // item -> (n tile fastest, m tile, head, sample) and its range of k-blocks; false: a tile the causal mask leaves empty
  // and nobody reads
  struct Item { int m0, n0, head, img, kb_lo, kb_hi; };
  auto decode = [&](int64_t item, Item* t) {
    const int tn = (int)(item % p.tiles_n); item /= p.tiles_n;
    const int tm = (int)(item % p.tiles_m); item /= p.tiles_m;
    t->m0 = tm * kAtBM; t->n0 = tn * BN;
    t->head = (int)(item % p.heads); t->img = (int)(item / p.heads);
    t->kb_lo = 0; t->kb_hi = p.num_kb;
    if (p.causal == kCausalTiles) return t->n0 <= t->m0 + kAtBM - 1;
    if (p.causal == kCausalKeys) t->kb_hi = min(p.num_kb, (t->m0 + kAtBM + p.bk - 1) / p.bk);
    if (p.causal == kCausalQueries) t->kb_lo = min(p.num_kb, t->m0 / p.bk);
    return true;
  };

  if (warp == 0) {
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int64_t item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      Item t;
      if (!decode(item, &t)) continue;
      for (int j = 0; j < p.rep && ok; ++j) {
        const int hh = t.head * p.rep + j, ha = hh / p.a.head_div, hb = hh / p.b.head_div;
        for (int kb = t.kb_lo; kb < t.kb_hi; ++kb) {
          if (!mbar_wait_uniform(&empty[stage], phase ^ 1u, p.status, 0x1u)) { ok = false; break; }
          if (elect_one()) {
            mbar_expect_tx(&full[stage], Cfg::STAGE_BYTES);
            const uint32_t sA = smem_base + stage * Cfg::STAGE_BYTES, sB = sA + Cfg::A_BYTES * Cfg::PARTS;
            const int k0 = kb * p.bk;
            for (int bx = 0; bx < p.a.boxes; ++bx)
              at_load<F32>(sA + bx * p.a.box_bytes, &tmA, p.a, t.m0 + bx * p.a.mn_step, k0, ha, t.img, &full[stage]);
            for (int bx = 0; bx < p.b.boxes; ++bx)
              at_load<F32>(sB + bx * p.b.box_bytes, &tmB, p.b, t.n0 + bx * p.b.mn_step, k0, hb, t.img, &full[stage]);
          }
          __syncwarp();
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
    bool ok = true;
    for (int64_t item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      Item t;
      if (!decode(item, &t)) continue;
      const int n_kb = (t.kb_hi - t.kb_lo) * p.rep;
      for (int kb = 0; kb < n_kb; ++kb) {
        if (F32 || kb == 0) {
          if (!mbar_wait_uniform(&acc_empty[acc], acc_phase ^ 1u, p.status, 0x2u)) { ok = false; break; }
        }
        if (!mbar_wait_uniform(&full[stage], phase, p.status, 0x4u)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * Cfg::ACC_COLS;
        const uint32_t sA = smem_base + stage * Cfg::STAGE_BYTES, sB = sA + Cfg::A_BYTES * Cfg::PARTS;
        const uint64_t ad = ((uint64_t)p.a.desc_hi << 32) | (uint64_t)(((sA >> 4) & 0x3FFFu) | p.a.lbo);
        const uint64_t bd = ((uint64_t)p.b.desc_hi << 32) | (uint64_t)(((sB >> 4) & 0x3FFFu) | p.b.lbo);
        if (elect_one()) {
          if constexpr (F32) {
            parts_issue(d_tmem, d_tmem + BN, ad, bd, p.a.part, p.b.part, p.a.k_adv, p.b.k_adv, p.idesc, true, nullptr);
          } else {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) umma<false>(d_tmem, ad + ks * p.a.k_adv, bd + ks * p.b.k_adv, p.idesc, (kb | ks) != 0 ? 1u : 0u);
          }
          umma_commit(&empty[stage]);
          if (F32 || kb == n_kb - 1) umma_commit(&acc_full[acc]);
        }
        __syncwarp();
        if (F32 || kb == n_kb - 1) {
          if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp >= 4) {
    // two warps share each TMEM lane quarter and split the tile's columns; a thread owns one row m and writes its columns
    // as 16-byte vectors
    using T = typename std::conditional<F32, float, __nv_bfloat16>::type;
    constexpr int VEC = 16 / sizeof(T);
    const int q = warp & 3, half = (warp - 4) >> 2;
    constexpr int COLS = BN / 2;
    uint32_t acc = 0, acc_phase = 0;
    bool ok = true;
    for (int64_t item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      __syncwarp();                        // rows past the last left the stores below early; the TMEM loads want whole warps
      Item t;
      if (!decode(item, &t)) continue;
      const int n_kb = (t.kb_hi - t.kb_lo) * p.rep;
      const int rounds = F32 ? n_kb : (n_kb > 0 ? 1 : 0);
      const int m = t.m0 + q * 32 + lane, n0 = t.n0 + half * COLS;
      T* d = static_cast<T*>(p.D) + (int64_t)t.img * p.batch_stride + (int64_t)t.head * p.head_stride + (int64_t)m * p.ldd + n0;
      float sum[COLS];
#pragma unroll
      for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
      for (int r = 0; r < rounds; ++r) {
        if (!mbar_wait_warp(&acc_full[acc], acc_phase, p.status, 0x8u)) { ok = false; break; }
        tc_fence_after();
        const uint32_t t0 = tmem_base + ((uint32_t)(q * 32) << 16) + acc * Cfg::ACC_COLS + half * COLS;
#pragma unroll
        for (int c = 0; c < COLS / 32; ++c) {
          uint32_t v[32], vs[32];
          tmem_ld32(t0 + c * 32, v);
          if constexpr (F32) tmem_ld32(t0 + BN + c * 32, vs);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if constexpr (F32) sum[c * 32 + j] += parts_unbias(__uint_as_float(v[j]), __uint_as_float(vs[j]));
            else sum[c * 32 + j] = __uint_as_float(v[j]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
      if (!ok) break;
      if (m < p.M) {
        if (p.wide && n0 + COLS <= p.N) {
#pragma unroll
          for (int j = 0; j < COLS; j += 2 * VEC) {
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              if constexpr (F32) {
                w[i] = __float_as_uint(sum[j + i]);
              } else {
                const __nv_bfloat162 h = __floats2bfloat162_rn(sum[j + 2 * i], sum[j + 2 * i + 1]);
                w[i] = *reinterpret_cast<const uint32_t*>(&h);
              }
            }
            at_store32(d + j, w);
          }
          continue;
        }
#pragma unroll
        for (int j = 0; j < COLS; j += VEC) {
          if (n0 + j < p.N) {
            if constexpr (F32) {
              *reinterpret_cast<float4*>(d + j) = make_float4(sum[j], sum[j + 1], sum[j + 2], sum[j + 3]);
            } else {
              uint32_t w[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(sum[j + 2 * i], sum[j + 2 * i + 1]);
                w[i] = *reinterpret_cast<const uint32_t*>(&h);
              }
              *reinterpret_cast<uint4*>(d + j) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    if (*reinterpret_cast<volatile unsigned int*>(p.status) != 0) drain_after_abort();
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * Cfg::ACC_COLS);
  }
}

// ----------------------------------------------------------------------------------------------
// softmax passes: a warp per query row, four elements per lane and step
// ----------------------------------------------------------------------------------------------
template <typename T> struct At4;
template <> struct At4<float> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[4]) {
    const float4 u = *reinterpret_cast<const float4*>(p);
    v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
};
template <> struct At4<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(u.x << 16); v[1] = __uint_as_float(u.x & 0xFFFF0000u);
    v[2] = __uint_as_float(u.y << 16); v[3] = __uint_as_float(u.y & 0xFFFF0000u);
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&v)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  }
};
// row of S elements at p (element-aligned): vector access where `vec` says rows are aligned, else one by one up to S
template <typename T> __device__ __forceinline__ void at_load_row(const T* row, int s, int S, bool vec, float (&v)[4]) {
  if (vec) { At4<T>::load(row + s, v); return; }
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = s + i < S ? to_f32(row[s + i]) : 0.f;
}
template <typename T> __device__ __forceinline__ void at_store_row(T* row, int s, int S, bool vec, const float (&v)[4]) {
  if (vec) { At4<T>::store(row + s, v); return; }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (s + i < S) row[s + i] = from_f32<T>(v[i]);
}
// operand copies of a row for the products that follow: rows padded to Sp; Float32 in parts
template <typename T> __device__ __forceinline__ void at_store_operand(uint16_t* op, int64_t part_stride, int64_t off, const float (&v)[4]) {
  if constexpr (sizeof(T) == 4) store_parts4(op + off, part_stride, v);
  else At4<T>::store(reinterpret_cast<T*>(op) + off, v);
}

// NV > 0: rows of at most NV * 128 keys are kept in registers; NV = 0: longer rows are read again for each pass.
template <typename T, int NV>
__global__ void __launch_bounds__(256) attn_rows_fwd_kernel(T* __restrict__ w, uint16_t* __restrict__ op, int64_t part_stride, const T* __restrict__ logits,
                                                            const T* __restrict__ bias, int64_t bias_bs, const uint8_t* __restrict__ mask,
                                                            int64_t mask_bs, int causal, float scale, int S, int Sp, int L, int64_t rows) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int l = (int)(row % L);
  const int64_t hb = row / L;
  const T* z = logits + row * Sp;
  const T* bz = bias != nullptr ? bias + hb * bias_bs + (int64_t)l * S : nullptr;
  const uint8_t* mz = mask != nullptr ? mask + hb * mask_bs + (int64_t)l * S : nullptr;
  const int lim = causal ? min(S, l + 1) : S;                 // keys past it are masked
  const bool vec = S % 4 == 0;
  auto value4 = [&](int s, float (&v)[4]) {
    At4<T>::load(z + s, v);                                    // rows of logits are padded
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool keep = s + i < lim && (mz == nullptr || mz[s + i] != 0);
      float u = v[i] * scale;
      if (bz != nullptr && keep) u += to_f32(bz[s + i]);
      v[i] = keep ? u : -INFINITY;
    }
  };
  float r[NV > 0 ? NV : 1][4];
  float m = -INFINITY, se = 0.f;
  auto max4 = [&](const float (&v)[4]) { m = fmaxf(fmaxf(m, fmaxf(v[0], v[1])), fmaxf(v[2], v[3])); };
  if constexpr (NV > 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int s = (i * 32 + lane) * 4;
      if (s < lim) value4(s, r[i]);
      else r[i][0] = r[i][1] = r[i][2] = r[i][3] = -INFINITY;
      max4(r[i]);
    }
  } else {
    for (int s = lane * 4; s < lim; s += 128) { float v[4]; value4(s, v); max4(v); }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  // a row with every key masked: m = -inf and every difference below is NaN, as in the reference
  const float off = expf(-INFINITY - m);                       // weight of a key past lim, before the division: 0 (or NaN)
  if constexpr (NV > 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if ((i * 32 + lane) * 4 < lim) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if ((i * 32 + lane) * 4 + k < S) { r[i][k] = expf(r[i][k] - m); se += r[i][k]; }
      } else {
        r[i][0] = r[i][1] = r[i][2] = r[i][3] = off;
      }
    }
  } else {
    for (int s = lane * 4; s < lim; s += 128) {
      float v[4];
      value4(s, v);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (s + k < S) se += expf(v[k] - m);
    }
  }
  se = warp_sum(se);
  const float inv = 1.f / se;
  const int op_lim = causal ? min(Sp, (l / kAtBM + 1) * kAtBM) : Sp;   // what the products read of this row
  auto put = [&](int s, float (&v)[4]) {
    at_store_row(w + row * S, s, S, vec, v);
    if (op != nullptr && s < op_lim) at_store_operand<T>(op, part_stride, row * Sp + s, v);
  };
  if constexpr (NV > 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int s = (i * 32 + lane) * 4;
      if (s < S) {
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = s + k < S ? r[i][k] * inv : 0.f;
        put(s, v);
      }
    }
  } else {
    for (int s = lane * 4; s < S; s += 128) {
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (s < lim) value4(s, v);
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = s < lim && s + k < S ? expf(v[k] - m) * inv : (s + k < S ? off * inv : 0.f);
      put(s, v);
    }
  }
}

// dl = scale * w .* (dw - sum_s w dw) as an operand (bf16: written over dw); dbias = dl / scale; op = operand copy of w
template <typename T, int NV>
__global__ void __launch_bounds__(256) attn_rows_bwd_kernel(uint16_t* dl, const T* dw, T* __restrict__ dbias, uint16_t* __restrict__ op,
                                                            int64_t part_stride, const T* __restrict__ w, int causal, float scale, int S,
                                                            int Sp, int L, int64_t rows) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int l = (int)(row % L);
  const int lim = causal ? min(S, l + 1) : S;
  const int op_lim = causal ? min(Sp, (l / kAtBM + 1) * kAtBM) : Sp;
  const bool vec = S % 4 == 0;
  const T* wr = w + row * S;
  const T* g = dw + row * Sp;
  float rw[NV > 0 ? NV : 1][4], rg[NV > 0 ? NV : 1][4];
  auto get = [&](int s, float (&a)[4], float (&b)[4]) {
    if (s < lim) {
      at_load_row(wr, s, S, vec, a);
      At4<T>::load(g + s, b);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (s + k >= lim) { a[k] = 0.f; b[k] = 0.f; }          // dw is not formed where the mask leaves nothing
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) { a[k] = 0.f; b[k] = 0.f; }
    }
  };
  float dot = 0.f;
  if constexpr (NV > 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      get((i * 32 + lane) * 4, rw[i], rg[i]);
#pragma unroll
      for (int k = 0; k < 4; ++k) dot = fmaf(rw[i][k], rg[i][k], dot);
    }
  } else {
    for (int s = lane * 4; s < lim; s += 128) {
      float a[4], b[4];
      get(s, a, b);
#pragma unroll
      for (int k = 0; k < 4; ++k) dot = fmaf(a[k], b[k], dot);
    }
  }
  dot = warp_sum(dot);
  auto put = [&](int s, const float (&a)[4], const float (&b)[4]) {
    float d[4], e[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) { d[k] = a[k] * (b[k] - dot); e[k] = d[k] * scale; }
    if (dbias != nullptr) at_store_row(dbias + row * S, s, S, vec, d);
    if (s < op_lim) {
      at_store_operand<T>(dl, part_stride, row * Sp + s, e);
      if (op != nullptr) at_store_operand<T>(op, part_stride, row * Sp + s, a);
    }
  };
  if constexpr (NV > 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int s = (i * 32 + lane) * 4;
      if (s < S) put(s, rw[i], rg[i]);
    }
  } else {
    for (int s = lane * 4; s < S; s += 128) {
      float a[4], b[4];
      get(s, a, b);
      put(s, a, b);
    }
  }
}

// rows of `features` (a multiple of 4) floats -> three parts, rows padded to `ld`
__global__ void __launch_bounds__(256) attn_split_kernel(uint16_t* __restrict__ out, int64_t part_stride, const float* __restrict__ x, int64_t n4,
                                                         int quads, int ld) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / quads;
    float v[4];
    At4<float>::load(x + i * 4, v);
    store_parts4(out + row * ld + (i - row * quads) * 4, part_stride, v);
  }
}

// ----------------------------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------------------------
// An operand: (feature, head, token, sample) arrays [head_first] or (key, query, head, sample) arrays of weights; 2-byte elements
// (bf16, or a part of a Float32 value; the parts `part_stride` elements apart).
struct AtArray {
  const void* ptr;
  int64_t part_stride;
  int64_t inner, outer, ld, heads, head_stride, batch_stride;
  bool head_first;
};

bool at_encode(CUtensorMap* map, const AtArray& t, int64_t batch, bool f32, int box_outer) {
  TensorMapEncodeFn enc = tensor_map_encoder();
  if (!enc) return false;
  const int o = t.head_first ? 2 : 1, h = t.head_first ? 1 : 2;
  cuuint64_t dims[5], strides[4];                     // Float32: the parts are a fifth dimension
  cuuint32_t box[5] = {f32 ? 32u : 64u, 1, 1, 1, 3}, estr[5] = {1, 1, 1, 1, 1};
  dims[0] = (cuuint64_t)t.inner; dims[o] = (cuuint64_t)t.outer; dims[h] = (cuuint64_t)t.heads; dims[3] = (cuuint64_t)batch; dims[4] = 3;
  strides[o - 1] = (cuuint64_t)(t.ld * 2); strides[h - 1] = (cuuint64_t)(t.head_stride * 2); strides[2] = (cuuint64_t)(t.batch_stride * 2);
  strides[3] = (cuuint64_t)(t.part_stride * 2);
  box[o] = (cuuint32_t)box_outer;
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, f32 ? 5 : 4, const_cast<void*>(t.ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             f32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool at_operand(CUtensorMap* map, const AtArray& t, bool mn_major, int head_div, int64_t batch, bool f32, int tile_mn, AtOperand* o) {
  const int row = f32 ? 32 : 64, row_bytes = row * 2, parts = f32 ? 3 : 1;   // a k-block's row: its depth, or the elements of the other index in a box
  o->mn_major = mn_major; o->head_first = t.head_first; o->head_div = head_div;
  if (mn_major) {
    o->boxes = tile_mn / row; o->box_bytes = row * row_bytes * parts; o->mn_step = row;
    o->lbo = ((uint32_t)(o->box_bytes >> 4) & 0x3FFFu) << 16;
    o->k_adv = (uint32_t)((16 * row_bytes) >> 4);
  } else {
    o->boxes = 1; o->box_bytes = tile_mn * row_bytes * parts; o->mn_step = 0;
    o->lbo = 1u << 16;
    o->k_adv = 2u;
  }
  o->part = (uint32_t)((o->box_bytes / parts) >> 4);
  // eight-row swizzle atoms of 128-byte (2) or 64-byte (4) rows
  o->desc_hi = ((uint32_t)((8 * row_bytes) >> 4) & 0x3FFFu) | (1u << 14) | ((f32 ? 4u : 2u) << 29);
  return at_encode(map, t, batch, f32, mn_major ? row : tile_mn);
}

struct AtProduct {
  AtArray A, B;
  bool a_mn, b_mn;
  int a_div, b_div;
  int64_t M, N, K, heads, rep;
  int causal;
  void* D;
  int64_t n_store, ldd, head_stride, batch_stride;
};
int32_t at_gemm(const AtProduct& g, int64_t batch, int32_t dtype, cudaStream_t st) {
  const int es = (int)dtype_size(dtype);
  const bool f32 = dtype == LB2_F32;
  const int bn = g.N <= 64 ? 64 : 128;
  AtParams p{};
  CUtensorMap mA, mB;
  if (!at_operand(&mA, g.A, g.a_mn, g.a_div, batch, f32, kAtBM, &p.a) || !at_operand(&mB, g.B, g.b_mn, g.b_div, batch, f32, bn, &p.b))
    return fail(LB2_LAUNCH_FAIL, "attention: cuTensorMapEncodeTiled failed");
  p.bk = f32 ? 32 : 64;
  p.M = (int)g.M; p.N = (int)g.n_store;
  p.tiles_m = (int)((g.M + kAtBM - 1) / kAtBM); p.tiles_n = (int)((g.N + bn - 1) / bn);
  p.heads = (int)g.heads; p.rep = (int)g.rep; p.batch = (int)batch;
  p.num_kb = (int)((g.K + p.bk - 1) / p.bk);
  p.causal = g.causal;
  p.idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((g.a_mn ? 1u : 0u) << 15) | ((g.b_mn ? 1u : 0u) << 16) | ((uint32_t)(bn >> 3) << 17) |
            ((uint32_t)(kAtBM >> 4) << 24);
  p.wide = aligned_to(g.D, 32) && (g.ldd * es) % 32 == 0 && (g.head_stride * es) % 32 == 0 && (g.batch_stride * es) % 32 == 0;
  p.D = g.D; p.ldd = g.ldd; p.head_stride = g.head_stride; p.batch_stride = g.batch_stride;
  p.status = device_status_word();
  LB2_REQUIRE(p.status != nullptr, LB2_LAUNCH_FAIL, "attention: device status word unavailable");
  const int64_t items = (int64_t)p.tiles_m * p.tiles_n * p.heads * p.batch;
  const int grid = (int)(items < sm_count() ? items : sm_count());
  auto launch = [&](auto kernel, int smem) -> int32_t {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail(LB2_LAUNCH_FAIL, "attention: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
    kernel<<<grid, kAtThreads, smem, st>>>(mA, mB, p);
    LB2_CHECK_LAUNCH("attention product");
    return LB2_OK;
  };
  if (f32) return bn == 64 ? launch(attn_gemm_kernel<64, true>, AtCfg<64, true>::SMEM_BYTES) : launch(attn_gemm_kernel<128, true>, AtCfg<128, true>::SMEM_BYTES);
  return bn == 64 ? launch(attn_gemm_kernel<64, false>, AtCfg<64, false>::SMEM_BYTES) : launch(attn_gemm_kernel<128, false>, AtCfg<128, false>::SMEM_BYTES);
}

int64_t at_pad(int64_t S) { return (S + 7) / 8 * 8; }
size_t at_bytes(int64_t elems, int es) { return align_up((size_t)elems * es, 1024); }
// weights need an operand copy of their own: parts for Float32, padded rows where S breaks the 16-byte stride rule
bool at_needs_copy(const lb2_attention_dims& d, int es) { return es == 4 || d.keys % 8 != 0; }
// an operand copy of n elements: bf16, or the three parts of Float32
size_t at_operand_bytes(int64_t n, int es) { return at_bytes(n, 2) * (es == 4 ? 3 : 1); }
int64_t at_part_stride(int64_t n) { return (int64_t)(at_bytes(n, 2) / 2); }
// Float32 token arrays are copied into parts, rows padded to the 16-byte rule
int64_t at_token_ld(int64_t features, int es) { return es == 4 ? at_pad(features) : features; }
size_t at_token_bytes(int64_t features, int64_t rows, int es) { return es == 4 ? at_operand_bytes(at_pad(features) * rows, es) : 0; }

int32_t at_check(const lb2_attention_dims* d, int32_t dtype) {
  LB2_REQUIRE(valid_dtype(dtype), LB2_UNSUPPORTED_DTYPE, "dtype %d not supported", (int)dtype);
  LB2_REQUIRE(d != nullptr, LB2_BAD_ARG, "attention dims are null");
  LB2_REQUIRE(lb2_attention_is_fused(d, dtype) == 1, LB2_BAD_SHAPE, "attention dims not served by the tensor-core path");
  return LB2_OK;
}

// weights (keys padded to ld, queries, heads, samples)
AtArray at_weights(const void* ptr, int64_t part_stride, int64_t keys, int64_t ld, int64_t queries, int64_t heads) {
  return AtArray{ptr, part_stride, keys, queries, ld, heads, ld * queries, ld * queries * heads, false};
}
// feature-major array (features, heads, tokens, samples): bf16 in place, Float32 as a copy in the workspace
int32_t at_tokens(AtArray* out, const void* x, int64_t features, int64_t heads, int64_t tokens, int64_t batch, int es, uint8_t** ws, cudaStream_t st) {
  const int64_t ld = at_token_ld(features, es), rows = heads * tokens * batch;
  *out = AtArray{x, 0, features, tokens, ld * heads, heads, ld, ld * heads * tokens, true};
  if (es == 2) return LB2_OK;
  out->ptr = *ws; out->part_stride = at_part_stride(ld * rows);
  const int64_t n4 = features / 4 * rows, blocks = (n4 + 255) / 256, cap = (int64_t)sm_count() * 8;
  attn_split_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, st>>>(reinterpret_cast<uint16_t*>(*ws), out->part_stride, (const float*)x, n4,
                                                                            (int)(features / 4), (int)ld);
  LB2_CHECK_LAUNCH("attention split");
  *ws += at_token_bytes(features, rows, es);
  return LB2_OK;
}

#define LB2_AT_ROWS(KERNEL, T, S, ...)                                                        \
  do {                                                                                        \
    const unsigned grid_ = (unsigned)((rows + 7) / 8);                                        \
    if ((S) <= 128) KERNEL<T, 1><<<grid_, 256, 0, st>>>(__VA_ARGS__);                         \
    else if ((S) <= 512) KERNEL<T, 4><<<grid_, 256, 0, st>>>(__VA_ARGS__);                    \
    else if ((S) <= 1024) KERNEL<T, 8><<<grid_, 256, 0, st>>>(__VA_ARGS__);                   \
    else KERNEL<T, 0><<<grid_, 256, 0, st>>>(__VA_ARGS__);                                    \
  } while (0)

}  // namespace

}  // namespace lb2

using namespace lb2;

extern "C" {

int32_t lb2_attention_is_fused(const lb2_attention_dims* d, int32_t dtype) {
  if (d == nullptr || !valid_dtype(dtype)) return 0;
  if (d->head_dim <= 0 || d->value_dim <= 0 || d->heads <= 0 || d->kv_heads <= 0 || d->queries <= 0 || d->keys <= 0 || d->batch <= 0) return 0;
  if (d->heads % d->kv_heads != 0) return 0;
  const int64_t es = (int64_t)dtype_size(dtype), big = 1 << 24;
  if ((d->head_dim * es) % 16 != 0 || (d->value_dim * es) % 16 != 0) return 0;     // TMA strides
  if (d->head_dim > big || d->value_dim > big || d->heads > big || d->queries > big || d->keys > big || d->batch > big) return 0;
  const int64_t rows = d->queries * d->heads * d->batch;
  if (rows / 8 >= 0x7FFFFFFF || (d->keys + 8) * d->queries * d->heads * es >= ((int64_t)1 << 40)) return 0;
  if (d->head_dim * d->heads * d->queries * es >= ((int64_t)1 << 40) || d->value_dim * d->heads * d->queries * es >= ((int64_t)1 << 40)) return 0;
  if (d->head_dim * d->kv_heads * d->keys * es >= ((int64_t)1 << 40) || d->value_dim * d->kv_heads * d->keys * es >= ((int64_t)1 << 40)) return 0;
  return tensor_map_encoder() != nullptr ? 1 : 0;
}

size_t lb2_attention_fwd_workspace_bytes(const lb2_attention_dims* d, int32_t dtype) {
  if (lb2_attention_is_fused(d, dtype) != 1) return 0;
  const int es = (int)dtype_size(dtype);
  const int64_t w = at_pad(d->keys) * d->queries * d->heads * d->batch;
  const int64_t qr = d->heads * d->queries * d->batch, kr = d->kv_heads * d->keys * d->batch;
  return at_bytes(w, es) + (at_needs_copy(*d, es) ? at_operand_bytes(w, es) : 0) + at_token_bytes(d->head_dim, qr, es) +
         at_token_bytes(d->head_dim, kr, es) + at_token_bytes(d->value_dim, kr, es);
}

int32_t lb2_attention_fwd(void* x, void* w, const void* q, const void* k, const void* v, const void* bias, int64_t bias_batch_stride,
                          const uint8_t* mask, int64_t mask_batch_stride, int32_t causal, double scale, const lb2_attention_dims* d,
                          int32_t dtype, void* workspace, size_t workspace_bytes, void* stream) {
  int32_t rc = at_check(d, dtype);
  if (rc != LB2_OK) return rc;
  const int64_t S = d->keys, L = d->queries, Sp = at_pad(S), H = d->heads, B = d->batch, rows = L * H * B;
  LB2_REQUIRE(bias_batch_stride == 0 || bias_batch_stride == S * L, LB2_BAD_SHAPE, "bias batch stride must be 0 or S*L");
  LB2_REQUIRE(mask_batch_stride == 0 || mask_batch_stride == S * L, LB2_BAD_SHAPE, "mask batch stride must be 0 or S*L");
  LB2_REQUIRE(x && w && q && k && v, LB2_BAD_ARG, "null tensor pointer");
  LB2_REQUIRE(aligned_to(x, 16) && aligned_to(w, 16) && aligned_to(q, 16) && aligned_to(k, 16) && aligned_to(v, 16) &&
                  aligned_to(bias, dtype_size(dtype)),
              LB2_BAD_ALIGN, "arrays must be 16-byte aligned");
  LB2_REQUIRE(workspace != nullptr && workspace_bytes >= lb2_attention_fwd_workspace_bytes(d, dtype), LB2_WORKSPACE_TOO_SMALL,
              "workspace of %zu bytes needed", lb2_attention_fwd_workspace_bytes(d, dtype));
  LB2_REQUIRE(aligned_to(workspace, 256), LB2_BAD_ALIGN, "workspace must be 256-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int es = (int)dtype_size(dtype);
  const int gs = (int)(H / d->kv_heads);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  const int64_t wn = Sp * L * H * B, wps = at_part_stride(wn);
  void* logits = ws; ws += at_bytes(wn, es);
  uint16_t* op = nullptr;
  if (at_needs_copy(*d, es)) { op = reinterpret_cast<uint16_t*>(ws); ws += at_operand_bytes(wn, es); }
  AtArray Q, K, V;
  if ((rc = at_tokens(&Q, q, d->head_dim, H, L, B, es, &ws, st)) != LB2_OK) return rc;
  if ((rc = at_tokens(&K, k, d->head_dim, d->kv_heads, S, B, es, &ws, st)) != LB2_OK) return rc;
  if ((rc = at_tokens(&V, v, d->value_dim, d->kv_heads, S, B, es, &ws, st)) != LB2_OK) return rc;
  rc = at_gemm(AtProduct{Q, K, false, false, 1, gs, L, S, d->head_dim, H, 1, causal ? kCausalTiles : kCausalNone, logits, Sp, Sp, Sp * L, Sp * L * H},
               B, dtype, st);
  if (rc != LB2_OK) return rc;
  LB2_DISPATCH_DTYPE(dtype, {
    LB2_AT_ROWS(attn_rows_fwd_kernel, T, S, (T*)w, op, wps, (const T*)logits, (const T*)bias, bias_batch_stride, mask, mask_batch_stride,
                causal, (float)scale, (int)S, (int)Sp, (int)L, rows);
  });
  LB2_CHECK_LAUNCH("attention softmax");
  const AtArray W = op != nullptr ? at_weights(op, wps, S, Sp, L, H) : at_weights(w, 0, S, S, L, H);
  return at_gemm(AtProduct{W, V, false, true, 1, gs, L, d->value_dim, S, H, 1, causal ? kCausalKeys : kCausalNone, x, d->value_dim,
                           d->value_dim * H, d->value_dim, d->value_dim * H * L},
                 B, dtype, st);
}

size_t lb2_attention_bwd_workspace_bytes(const lb2_attention_dims* d, int32_t dtype) {
  if (lb2_attention_is_fused(d, dtype) != 1) return 0;
  const int es = (int)dtype_size(dtype);
  const int64_t w = at_pad(d->keys) * d->queries * d->heads * d->batch;
  const int64_t qr = d->heads * d->queries * d->batch, kr = d->kv_heads * d->keys * d->batch;
  return at_bytes(w, es) + (es == 4 ? at_operand_bytes(w, es) : 0) + (at_needs_copy(*d, es) ? at_operand_bytes(w, es) : 0) +
         at_token_bytes(d->head_dim, qr, es) + at_token_bytes(d->value_dim, qr, es) + at_token_bytes(d->head_dim, kr, es) +
         at_token_bytes(d->value_dim, kr, es);
}

int32_t lb2_attention_bwd(void* dq, void* dk, void* dv, void* dbias, const void* dx, const void* w, const void* q, const void* k, const void* v,
                          int32_t causal, double scale, const lb2_attention_dims* d, int32_t dtype, void* workspace, size_t workspace_bytes,
                          void* stream) {
  int32_t rc = at_check(d, dtype);
  if (rc != LB2_OK) return rc;
  LB2_REQUIRE(dq && dk && dv && dx && w && q && k && v, LB2_BAD_ARG, "null tensor pointer");
  LB2_REQUIRE(aligned_to(dq, 16) && aligned_to(dk, 16) && aligned_to(dv, 16) && aligned_to(dx, 16) && aligned_to(w, 16) && aligned_to(q, 16) &&
                  aligned_to(k, 16) && aligned_to(v, 16) && aligned_to(dbias, 16),
              LB2_BAD_ALIGN, "arrays must be 16-byte aligned");
  LB2_REQUIRE(workspace != nullptr && workspace_bytes >= lb2_attention_bwd_workspace_bytes(d, dtype), LB2_WORKSPACE_TOO_SMALL,
              "workspace of %zu bytes needed", lb2_attention_bwd_workspace_bytes(d, dtype));
  LB2_REQUIRE(aligned_to(workspace, 256), LB2_BAD_ALIGN, "workspace must be 256-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t S = d->keys, L = d->queries, Sp = at_pad(S), H = d->heads, Hkv = d->kv_heads, B = d->batch, rows = L * H * B;
  const int64_t D = d->head_dim, E = d->value_dim;
  const int es = (int)dtype_size(dtype);
  const int gs = (int)(H / Hkv);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  const int64_t wn = Sp * L * H * B, wps = at_part_stride(wn);
  void* dw = ws; ws += at_bytes(wn, es);
  uint16_t *dl = static_cast<uint16_t*>(dw), *op = nullptr;       // bf16: dlogits over dw
  if (es == 4) { dl = reinterpret_cast<uint16_t*>(ws); ws += at_operand_bytes(wn, es); }
  if (at_needs_copy(*d, es)) { op = reinterpret_cast<uint16_t*>(ws); ws += at_operand_bytes(wn, es); }
  AtArray Q, G, K, V;
  if ((rc = at_tokens(&Q, q, D, H, L, B, es, &ws, st)) != LB2_OK) return rc;
  if ((rc = at_tokens(&G, dx, E, H, L, B, es, &ws, st)) != LB2_OK) return rc;
  if ((rc = at_tokens(&K, k, D, Hkv, S, B, es, &ws, st)) != LB2_OK) return rc;
  if ((rc = at_tokens(&V, v, E, Hkv, S, B, es, &ws, st)) != LB2_OK) return rc;
  rc = at_gemm(AtProduct{G, V, false, false, 1, gs, L, S, E, H, 1, causal ? kCausalTiles : kCausalNone, dw, Sp, Sp, Sp * L, Sp * L * H}, B, dtype, st);
  if (rc != LB2_OK) return rc;
  LB2_DISPATCH_DTYPE(dtype, {
    LB2_AT_ROWS(attn_rows_bwd_kernel, T, S, dl, (const T*)dw, (T*)dbias, op, wps, (const T*)w, causal, (float)scale, (int)S, (int)Sp, (int)L, rows);
  });
  LB2_CHECK_LAUNCH("attention softmax backward");
  const AtArray W = op != nullptr ? at_weights(op, wps, S, Sp, L, H) : at_weights(w, 0, S, S, L, H), DL = at_weights(dl, wps, S, Sp, L, H);
  rc = at_gemm(AtProduct{DL, K, false, true, 1, gs, L, D, S, H, 1, causal ? kCausalKeys : kCausalNone, dq, D, D * H, D, D * H * L}, B, dtype, st);
  if (rc != LB2_OK) return rc;
  const int cq = causal ? kCausalQueries : kCausalNone;
  rc = at_gemm(AtProduct{DL, Q, true, true, 1, 1, S, D, L, Hkv, gs, cq, dk, D, D * Hkv, D, D * Hkv * S}, B, dtype, st);
  if (rc != LB2_OK) return rc;
  return at_gemm(AtProduct{W, G, true, true, 1, 1, S, E, L, Hkv, gs, cq, dv, E, E * Hkv, E, E * Hkv * S}, B, dtype, st);
}

}  // extern "C"
