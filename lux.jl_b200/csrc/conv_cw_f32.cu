// General tensor-core convolution for Float32 storage on sm_100a: the channel-innermost implicit GEMM of conv_cw.cu on three
// bf16 parts per operand, for any 2-D padding / dilation / kernel size / channel counts with groups == 1 and strides up to 4
// whose position boxes fit a TMA box (conv_cwf_supported).
//
// Accuracy: products and partial sums as in parts.cuh, x1*w1 taken out of TMEM after every k-block of 32. The filter gradient, a
// sum over all positions, goes to memory in segments of kSegment k-blocks, so that no register adds up more than that many, and
// its splits are added with a compensated sum.
//
// Zero-filled positions outside the arrays, which are no terms of the sum, make NaN of an infinity or NaN on the other side:
// elements that come out as NaN are formed again, term by term, by the warp that stored them (cwf_redo_*). Ordinary data never
// gets there.
//
//   layout       x (and dy) are rewritten channel-innermost, three parts (one pass: read 4 bytes, write 6 per element); a tap
//                shift, the padding and the stride are then start coordinates / box parameters of a TMA map
//   forward      M = 128 output positions (a w x h x image box), N = 64 / 128 output channels, both operands K-major
//   data grad.   the same kernel on the copy of dy with the filter transposed; stride s: s*s classes of input positions
//   filter grad. rows = four (tap, 32-channel chunk) boxes of x, columns = 64 / 128 output channels of dy, contraction over
//                32-position boxes; both operands MN-major, split over CTAs, fixed-order reduction
// A problem with too few tiles for the SMs is split along the contraction as well: fp32 partials in the layout of the
// output and one elementwise pass that adds them in order (deterministic) and applies bias and activation.
//
// Measured (forward / both gradients, fp32 TFLOP/s of the convolution): 3x3 256 -> 256 on 14x14, batch 32: 81 / 158 us (92 /
// 94 TFLOP/s); 3x3 512 -> 512 on 7x7: 91 / 172 us. Two tf32 parts took 90 / 154 and 99 / 168 us, the gradients with the forward
// call's copy of x, and were less accurate than fp32 sums in the filter gradient. The CUDA-core kernels of conv_direct.cu, which
// took these geometries before, made a ResNet-18 training step at batch 32 last 333 ms; it now takes 6.3 ms. Error against 64
// bits (2-norm, normal data): 5e-8 to 1.6e-7, the CUDA-core kernels' 6e-8 to 1.1e-6.
// What bounds it: a 128 x 128 x 32 k-block is 768 tensor-pipe cycles (12 MMAs) against about 1150 cycles of shared-memory
// traffic (48 KB written by TMA, 96 KB read by the MMAs at 128 B/cycle).
#include "conv.cuh"
#include "parts.cuh"

namespace lb2 {

namespace {

constexpr int kFThreads = 384;   // warps 0-2: TMA / MMA / TMEM, warps 4-11: accumulate + epilogue
constexpr int kFBM = 128;
constexpr int kFMaxTaps = 128;
constexpr int kFMaxSplits = 16;

// ----------------------------------------------------------------------------------------------
// layout passes
// ----------------------------------------------------------------------------------------------
// parts[n][s][c] (c contiguous, Cp channels, zero beyond C)  <-  in[n][c][s]: 32 channels x 64 positions per tile through
// shared memory. V4: 16-byte loads (planes of S % 4 == 0 floats on a 16-byte base); stores are 16 bytes along c.
template <bool V4>
__global__ void __launch_bounds__(256) cwf_transpose_kernel(uint16_t* __restrict__ out, int64_t part_stride, const float* __restrict__ in,
                                                            int S, int C, int Cp, int N) {
  __shared__ float tile[32 * 65];
  const int st = (S + 63) / 64, ct = (Cp + 31) / 32;
  const int64_t blocks = (int64_t)N * st * ct;
  for (int64_t b = blockIdx.x; b < blocks; b += gridDim.x) {
    int64_t r = b;
    const int ci = (int)(r % ct); r /= ct;
    const int si = (int)(r % st);
    const int n = (int)(r / st);
    const int s0 = si * 64, c0 = ci * 32;
    __syncthreads();
    if constexpr (V4) {
#pragma unroll
      for (int v = threadIdx.x; v < 32 * 16; v += 256) {
        const int j = v / 16, q = (v % 16) * 4;
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c0 + j < C && s0 + q < S) u = __ldg(reinterpret_cast<const float4*>(in + ((int64_t)n * C + c0 + j) * S + s0 + q));
        float* t = tile + j * 65 + q;
        t[0] = u.x; t[1] = u.y; t[2] = u.z; t[3] = u.w;
      }
    } else {
#pragma unroll
      for (int v = threadIdx.x; v < 32 * 64; v += 256) {
        const int j = v / 64, q = v % 64;
        tile[j * 65 + q] = (c0 + j < C && s0 + q < S) ? __ldg(in + ((int64_t)n * C + c0 + j) * S + s0 + q) : 0.f;
      }
    }
    __syncthreads();
    const int j = threadIdx.x / 4, q = (threadIdx.x % 4) * 8;   // one position, eight channels
    if (s0 + j < S && c0 + q < Cp) {
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = tile[(q + k) * 65 + j];
      store_parts8(out + ((int64_t)n * S + s0 + j) * Cp + c0 + q, part_stride, v);
    }
  }
}

// Small channel counts, the kW taps folded into the channel index: parts[n][h][ow][tw*C + c] = in[n][c][h][ow*s + tw*dil - pad]
// (0 outside), padded to Cp. One thread per eight channels of the copy.
__global__ void __launch_bounds__(256) cwf_fold_kernel(uint16_t* __restrict__ out, int64_t part_stride, const float* __restrict__ in,
                                                       int W, int H, int C, int Cp, int N, int OW, int kW, int s, int dil, int pad) {
  const int groups = Cp / 8;
  const int64_t total = (int64_t)N * H * OW * groups;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = i;
    const int qg = (int)(r % groups); r /= groups;
    const int ow = (int)(r % OW); r /= OW;
    const int h = (int)(r % H);
    const int n = (int)(r / H);
    const float* plane0 = in + (int64_t)n * C * H * W;
    int tw = (qg * 8) / C, c = (qg * 8) % C;
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int w = ow * s + tw * dil - pad;
      v[k] = tw < kW && w >= 0 && w < W ? __ldg(plane0 + ((int64_t)c * H + h) * W + w) : 0.f;
      if (++c == C) { c = 0; ++tw; }
    }
    store_parts8(out + i * 8, part_stride, v);
  }
}

// Packed filter Wp[row][tap][chunk][32], three parts. Forward: row = co, contracted channel = ci. Data gradient (transpose):
// row = ci, contracted = co. tap = th*kW + tw in tap positions (filter index = flip ? t : K-1-t per dim); fold: tap = th and
// the contracted index of a tap is (tw, ci).
struct CwfPack {
  int kW, kH, cin, cout, flip, transpose, fold, chunks, n_rows, k_total;
};
__global__ void __launch_bounds__(256) cwf_pack_flat_kernel(uint16_t* __restrict__ out, int64_t part_stride, const float* __restrict__ w,
                                                            const CwfPack g) {
  const int64_t total = (int64_t)g.n_rows * g.k_total;
  const int kc = g.transpose ? g.cout : g.cin, nc = g.transpose ? g.cin : g.cout;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int row = (int)(i / g.k_total), col = (int)(i % g.k_total);
    const int kb = col / 32, j = col % 32;
    int tw, th, c;
    bool live = row < nc;
    if (g.fold) {
      th = kb; tw = j / g.cin; c = j % g.cin;
      live = live && tw < g.kW;
    } else {
      const int tap = kb / g.chunks;
      tw = tap % g.kW; th = tap / g.kW;
      c = (kb % g.chunks) * 32 + j;
      live = live && c < kc;
    }
    float v = 0.f;
    if (live) {
      const int kw = g.flip ? tw : g.kW - 1 - tw, kh = g.flip ? th : g.kH - 1 - th;
      const int ci = g.transpose ? row : c, co = g.transpose ? c : row;
      v = w[((int64_t)(co * g.cin + ci) * g.kH + kh) * g.kW + kw];
    }
    const Parts q = split_parts(v);
    out[i] = q.a; out[i + part_stride] = q.b; out[i + 2 * part_stride] = q.c;
  }
}
// The same for unfolded filters: a block turns 8 packed rows x 32 contracted channels x all taps through shared memory, so
// that the filter is read in runs of its own order and the packed rows are written in runs of 64 bytes.
__global__ void __launch_bounds__(256) cwf_pack_tile_kernel(uint16_t* __restrict__ out, int64_t part_stride, const float* __restrict__ w,
                                                            const CwfPack g) {
  extern __shared__ float cwf_tile[];                 // [8 rows][32 channels][taps] in the order it is read
  const int taps = g.kW * g.kH;
  const int kc = g.transpose ? g.cout : g.cin, nc = g.transpose ? g.cin : g.cout;
  const int chunk = blockIdx.x % g.chunks, row0 = (blockIdx.x / g.chunks) * 8;
  for (int e = threadIdx.x; e < 256 * taps; e += 256) {
    // forward: (row, c, t) with t fastest = runs of 32*taps; transposed: (c, row, t) = runs of 8*taps
    const int t = e % taps, q = e / taps;
    const int r = g.transpose ? q & 7 : q >> 5, c = g.transpose ? q >> 3 : q & 31;
    float v = 0.f;
    if (row0 + r < nc && chunk * 32 + c < kc) {
      const int ci = g.transpose ? row0 + r : chunk * 32 + c, co = g.transpose ? chunk * 32 + c : row0 + r;
      v = w[(int64_t)(co * g.cin + ci) * taps + t];
    }
    cwf_tile[(r * 32 + c) * taps + t] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 128 * taps; e += 256) {   // two channels: 4-byte stores
    const int c = (e & 15) * 2, r = (e >> 4) & 7, tap = e >> 7;
    const int tw = tap % g.kW, th = tap / g.kW;
    const int kw = g.flip ? tw : g.kW - 1 - tw, kh = g.flip ? th : g.kH - 1 - th;
    const int64_t o = (int64_t)(row0 + r) * g.k_total + (tap * g.chunks + chunk) * 32 + c;
    const float* v = cwf_tile + (r * 32 + c) * taps + kh * g.kW + kw;
    const Parts l = split_parts(v[0]), h = split_parts(v[taps]);
    *reinterpret_cast<uint32_t*>(out + o) = l.a | ((uint32_t)h.a << 16);
    *reinterpret_cast<uint32_t*>(out + o + part_stride) = l.b | ((uint32_t)h.b << 16);
    *reinterpret_cast<uint32_t*>(out + o + 2 * part_stride) = l.c | ((uint32_t)h.c << 16);
  }
}

// ----------------------------------------------------------------------------------------------
// kernels
// ----------------------------------------------------------------------------------------------
// K-major operands: 64-byte swizzle, 8-row atoms of 512 bytes, 32 bytes of K per MMA step
constexpr uint32_t kDescHi = (uint32_t)((512u >> 4) & 0x3FFFu) | (1u << 14) | (4u << 29);
constexpr uint32_t kLboK = 1u << 16, kAdvK = 2u;
// MN-major operands: the same swizzle, atoms of 32 elements x 8 rows; a box is the three parts of 32 elements, 2048 bytes each, 16
// rows of 64 bytes per MMA step
constexpr uint32_t kPartMN = 2048u >> 4, kLboMN = ((3u * 2048u) >> 4) << 16, kAdvMN = (16u * 64u) >> 4;

template <int BN> struct CwfCfg {
  static constexpr int A_BYTES = kFBM * 64;                     // 128 rows x 32 bf16, one part
  static constexpr int B_BYTES = BN * 64;
  static constexpr int STAGE_BYTES = 3 * (A_BYTES + B_BYTES);   // [A1 | A2 | A3 | B1 | B2 | B3]; MN-major: boxes of all parts
  static constexpr int SLOTS = 512 / BN - 1;                    // TMEM: a ring of BN-column accumulators and one for the small products
  static constexpr int STAGES = (200 * 1024) / STAGE_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
};

// TMEM between the MMA thread and the accumulating warps: x1*w1 has an accumulator for each k-block (a ring of BN-column slots),
// the small products, 2^-9 of the result, gather in one accumulator for a segment of kSegment k-blocks.
constexpr int kSegment = 16;
template <int SLOTS> struct CwfRing {
  uint64_t *full, *empty;             // [SLOTS] of the ring, [SLOTS] = the small products'
  uint32_t slot, phase, small_phase;
  __device__ __forceinline__ void next() {
    if (++slot == SLOTS) { slot = 0; phase ^= 1u; }
  }
};
// k-block i of `n` of an item
template <int BN, bool MN>
__device__ __forceinline__ bool cwf_issue_kblock(CwfRing<CwfCfg<BN>::SLOTS>& ring, uint32_t tmem_base, uint32_t sA, uint32_t sB, uint32_t idesc,
                                                 int i, int n, uint64_t* stage_empty, unsigned int* status, unsigned int code) {
  constexpr int SLOTS = CwfCfg<BN>::SLOTS;
  const bool first = i % kSegment == 0, last = i % kSegment == kSegment - 1 || i == n - 1;   // of its segment
  constexpr uint32_t LBO = MN ? kLboMN : kLboK, K_ADV = MN ? kAdvMN : kAdvK;
  constexpr uint32_t A_PART = MN ? kPartMN : CwfCfg<BN>::A_BYTES >> 4, B_PART = MN ? kPartMN : CwfCfg<BN>::B_BYTES >> 4;
  const uint32_t a32 = ((sA >> 4) & 0x3FFFu) | LBO, b32 = ((sB >> 4) & 0x3FFFu) | LBO;
  constexpr uint64_t top = (uint64_t)kDescHi << 32;
  if (!mbar_wait_uniform(&ring.empty[ring.slot], ring.phase ^ 1u, status, code)) return false;
  if (first) {
    if (!mbar_wait_uniform(&ring.empty[SLOTS], ring.small_phase ^ 1u, status, code)) return false;
  }
  tc_fence_after();
  if (elect_one()) {
    parts_issue(tmem_base + ring.slot * BN, tmem_base + SLOTS * BN, top | (uint64_t)a32, top | (uint64_t)b32, A_PART, B_PART, K_ADV, K_ADV, idesc,
                first, &ring.full[ring.slot]);
    umma_commit(stage_empty);
    if (last) umma_commit(&ring.full[SLOTS]);
  }
  __syncwarp();
  ring.next();
  if (last) ring.small_phase ^= 1u;
  return true;
}
// accumulating side: the next `kblocks` (at most a segment) of an item, columns [col, col + BN / 2) of the warp's lane quarter,
// added to `sum`; `last`: the final ones of the sum
template <int BN>
__device__ __forceinline__ bool cwf_accumulate(CwfRing<CwfCfg<BN>::SLOTS>& ring, uint32_t tmem_lane, int col, int kblocks, bool last,
                                               float (&sum)[BN / 2], unsigned int* status, unsigned int code) {
  constexpr int COLS = BN / 2, SLOTS = CwfCfg<BN>::SLOTS;
  const bool lead = (threadIdx.x & 31) == 0;
  for (int i = 0; i < kblocks; ++i) {
    if (!mbar_wait_warp(&ring.full[ring.slot], ring.phase, status, code)) return false;
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < COLS / 32; ++c) {
      uint32_t r[32];
      tmem_ld32(tmem_lane + ring.slot * BN + col + c * 32, r);
      tmem_ld_wait();
      if (c == COLS / 32 - 1) {
        tc_fence_before();
        __syncwarp();
        if (lead) mbar_arrive(&ring.empty[ring.slot]);
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) sum[c * 32 + j] += __uint_as_float(r[j]);
    }
    ring.next();
  }
  if (kblocks > 0) {
    if (!mbar_wait_warp(&ring.full[SLOTS], ring.small_phase, status, code)) return false;
    ring.small_phase ^= 1u;
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < COLS / 32; ++c) {
      uint32_t r[32];
      tmem_ld32(tmem_lane + SLOTS * BN + col + c * 32, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float v = __uint_as_float(r[j]);
        sum[c * 32 + j] = last ? parts_unbias(sum[c * 32 + j], v) : sum[c * 32 + j] + v;
      }
    }
    tc_fence_before();
    __syncwarp();
    if (lead) mbar_arrive(&ring.empty[SLOTS]);
  }
  return true;
}

// A channel-innermost array of parts and what of it exists; the taps a folded copy (fold = cin) holds beside one another
struct CwfSource {
  const uint16_t* ptr;
  int64_t part_stride;
  int32_t Cp, W, H;
  int32_t fold, fold_step, fold_dil, fold_pad, fold_W;
  // channel c of position (w, h, img) belongs to the arrays
  __device__ __forceinline__ bool has(int c, int w, int h) const {
    if (c >= Cp || w < 0 || w >= W || h < 0 || h >= H) return false;
    if (fold == 0) return true;
    const int iw = w * fold_step + (c / fold) * fold_dil - fold_pad;
    return iw >= 0 && iw < fold_W;
  }
  __device__ __forceinline__ float at(int c, int w, int h, int img) const {
    return join_parts(ptr + (((int64_t)img * H + h) * W + w) * Cp + c, part_stride);
  }
};

struct CwfFwdParams {
  int32_t OW, OH, NI;          // grid of output positions; a tile is a BW x BH x BI box of them
  int32_t BW, BH, BI;
  int32_t tiles_w, tiles_h, tiles_i, tiles_n;
  int32_t splits, kb_per_split, num_kb, chunks;   // k-block = (tap, 32-channel chunk), chunk fastest
  int32_t sw, sh;              // input coordinate step per output position (the TMA traversal stride)
  int32_t n_out;
  int32_t FW, FH, ow_step, ow_off, oh_step, oh_off;   // where a grid position lands in the output array
  uint32_t idesc;
  float* y;
  float* preact;
  const float* bias;
  float* partial;              // splits > 1: [splits][output numel], added up by cwf_finish_kernel
  int64_t split_stride;
  int32_t act;
  unsigned int* status;
  CwfSource src;
  const uint16_t* wp;          // packed filter
  int64_t wp_part_stride;
  int32_t wp_cols;
  int16_t tap_dw[kFMaxTaps], tap_dh[kFMaxTaps], tap_index[kFMaxTaps];

  // item -> (channel tile fastest, w tile, h tile, image tile, split)
  __device__ __forceinline__ void item_coords(int item, int* tn, int* tw, int* th, int* ti, int* z) const {
    *tn = item % tiles_n; item /= tiles_n;
    *tw = item % tiles_w; item /= tiles_w;
    *th = item % tiles_h; item /= tiles_h;
    *ti = item % tiles_i;
    *z = item / tiles_i;
  }
  __device__ __forceinline__ int64_t out_index(int a, int b, int img, int col) const {
    return (int64_t)(a * ow_step + ow_off) + (int64_t)FW * (b * oh_step + oh_off) + (int64_t)FW * FH * ((int64_t)n_out * img + col);
  }
};

// A warp's elements that came out as NaN once more, as the sum of their terms (positions outside the arrays are none). The lanes
// share an element's channels. A NaN among the terms stays NaN and ends the sum early; a NaN among a position's inputs settles
// all its channels, and where everything is NaN the first term of each element settles it, a lane per element. (3x3 256 -> 256 on
// 14x14, batch 32, one NaN in x: 0.28 ms; all of x: 0.47 ms; the CUDA-core kernel takes 4.5 ms whatever the values.)
template <int BN>
__device__ __noinline__ void cwf_redo_fwd(const CwfFwdParams& p, int q, int half) {
  constexpr int COLS = BN / 2;
  const int lane = threadIdx.x & 31, pos = q * 32 + lane;
  const int iw = pos % p.BW, ih = (pos / p.BW) % p.BH, ii = pos / (p.BW * p.BH);
  const int num_items = p.tiles_w * p.tiles_h * p.tiles_i * p.tiles_n * p.splits;
  for (int item = blockIdx.x; item < num_items; item += gridDim.x) {
    int tn, tw, th, ti, z;
    p.item_coords(item, &tn, &tw, &th, &ti, &z);
    const int kb_lo = z * p.kb_per_split, kb_hi = min(p.num_kb, kb_lo + p.kb_per_split);
    const int a = tw * p.BW + iw, b = th * p.BH + ih, img = ti * p.BI + ii;
    const bool live = ii < p.BI && a < p.OW && b < p.OH && img < p.NI;
    uint32_t seen = 0, nan_rows = 0;                     // lanes whose position's inputs were looked through / hold a NaN
    for (int j = 0; j < COLS; ++j) {
      const int col = tn * BN + half * COLS + j;
      if (col >= p.n_out) break;
      const int64_t out = p.out_index(a, b, img, col);
      float* const dst = p.splits > 1 ? p.partial + z * p.split_stride + out : p.y + out;
      const uint16_t* const wrow = p.wp + (int64_t)col * p.wp_cols;
      const float old = live ? *dst : 0.f;
      const uint32_t todo = __ballot_sync(0xffffffffu, old != old);
      if (todo == 0) continue;
      bool settled = false;
      if (old != old) {
        for (int kb = kb_lo; kb < kb_hi; ++kb) {
          const int tap = kb / p.chunks, c = (kb - tap * p.chunks) * 32, w = a * p.sw + p.tap_dw[tap], h = b * p.sh + p.tap_dh[tap];
          if (!p.src.has(c, w, h)) continue;
          const float v = p.src.at(c, w, h, img) * join_parts(wrow + p.tap_index[tap] * p.chunks * 32 + c, p.wp_part_stride);
          settled = v != v;
          break;
        }
      }
      float result = old;
      for (uint32_t rest = todo & ~__ballot_sync(0xffffffffu, settled); rest != 0; rest &= rest - 1) {
        const int who = __ffs(rest) - 1;
        const int wa = __shfl_sync(0xffffffffu, a, who) * p.sw, wb = __shfl_sync(0xffffffffu, b, who) * p.sh, wi = __shfl_sync(0xffffffffu, img, who);
        auto walk = [&](auto term) {                     // term(x, filter offset) until it says stop
          for (int kb = kb_lo; kb < kb_hi; ++kb) {
            const int tap = kb / p.chunks, c = (kb - tap * p.chunks) * 32 + lane, w = wa + p.tap_dw[tap], h = wb + p.tap_dh[tap];
            bool stop = false;
            if (p.src.has(c, w, h)) stop = term(p.src.at(c, w, h, wi), p.tap_index[tap] * p.chunks * 32 + c);
            if (__any_sync(0xffffffffu, stop)) return true;
          }
          return false;
        };
        if ((seen >> who & 1u) == 0) {
          seen |= 1u << who;
          if (walk([](float x, int) { return x != x; })) nan_rows |= 1u << who;
        }
        if ((nan_rows >> who & 1u) != 0) continue;
        float sum = 0.f;
        walk([&](float x, int at) {
          sum = fmaf(x, join_parts(wrow + at, p.wp_part_stride), sum);
          return sum != sum;
        });
        sum = warp_sum(sum);
        if (lane == who) result = sum;
      }
      if (old != old) {
        if (p.splits == 1) {
          if (p.bias != nullptr) result += __ldg(p.bias + col);
          if (p.preact != nullptr) p.preact[out] = result;
          result = act_apply_any<-1, false>(p.act, result);
        }
        *dst = result;
      }
    }
  }
}

template <int BN, int ACT>
__global__ void __launch_bounds__(kFThreads, 1)
conv_cwf_fwd_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CwfFwdParams p) {
  using Cfg = CwfCfg<BN>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_gen + STAGES * Cfg::STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  CwfRing<Cfg::SLOTS> ring{bars + 2 * STAGES, bars + 2 * STAGES + Cfg::SLOTS + 1, 0, 0, 0};   // MMA -> accumulating warps and back
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ring.empty + Cfg::SLOTS + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_items = p.tiles_w * p.tiles_h * p.tiles_i * p.tiles_n * p.splits;
  // Rows of an A stage past the box's positions are never written; they only feed accumulator rows that are never stored.
  const uint32_t tx = (uint32_t)(3 * (p.BW * p.BH * p.BI * 64 + Cfg::B_BYTES));

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a <= Cfg::SLOTS; ++a) { mbar_init(&ring.full[a], 1); mbar_init(&ring.empty[a], 8); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    tma_prefetch_desc(&tmX); tma_prefetch_desc(&tmW);
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      int tn, tw, th, ti, z;
      p.item_coords(item, &tn, &tw, &th, &ti, &z);
      const int w0 = tw * p.BW * p.sw, h0 = th * p.BH * p.sh, i0 = ti * p.BI, n0 = tn * BN;
      const int kb_lo = z * p.kb_per_split, kb_hi = min(p.num_kb, kb_lo + p.kb_per_split);
      int tap = kb_lo / p.chunks, ch = kb_lo - tap * p.chunks;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait_uniform(&empty[stage], phase ^ 1u, p.status, 0x1000u)) { ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&full[stage], tx);
          const uint32_t sA = smem_base + stage * Cfg::STAGE_BYTES, sB = sA + 3 * Cfg::A_BYTES;
          const int w = w0 + p.tap_dw[tap], h = h0 + p.tap_dh[tap], k0 = (p.tap_index[tap] * p.chunks + ch) * 32;
          tma_load_3d(sB, &tmW, k0, n0, 0, &full[stage]);
#pragma unroll
          for (int part = 0; part < 3; ++part) tma_load_5d(sA + part * Cfg::A_BYTES, &tmX, ch * 32, w, h, i0, part, &full[stage]);
        }
        __syncwarp();
        if (++ch == p.chunks) { ch = 0; ++tap; }
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      int tn, tw, th, ti, z;
      p.item_coords(item, &tn, &tw, &th, &ti, &z);
      const int kb_lo = z * p.kb_per_split, kb_hi = min(p.num_kb, kb_lo + p.kb_per_split);
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait_uniform(&full[stage], phase, p.status, 0x4000u)) { ok = false; break; }
        const uint32_t sA = smem_base + stage * Cfg::STAGE_BYTES, sB = sA + 3 * Cfg::A_BYTES;
        if (!cwf_issue_kblock<BN, false>(ring, tmem_base, sA, sB, p.idesc, kb - kb_lo, kb_hi - kb_lo, &empty[stage], p.status, 0x2000u)) { ok = false; break; }
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp >= 4) {
    // Two warps share each TMEM lane quarter and split the tile's channels; a thread owns one output position.
    const int q = warp & 3, half = (warp - 4) >> 2;
    constexpr int COLS = BN / 2;
    const int64_t plane = (int64_t)p.FW * p.FH;
    const int pos = q * 32 + lane;
    const int iw = pos % p.BW, ih = (pos / p.BW) % p.BH, ii = pos / (p.BW * p.BH);
    bool nan = false, ok = true;
    for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      int tn, tw, th, ti, z;
      p.item_coords(item, &tn, &tw, &th, &ti, &z);
      const int kb_lo = z * p.kb_per_split, kb_hi = min(p.num_kb, kb_lo + p.kb_per_split);
      float sum[COLS];
#pragma unroll
      for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
      for (int kb = kb_lo; kb < kb_hi && ok; kb += kSegment)
        ok = cwf_accumulate<BN>(ring, tmem_base + ((uint32_t)(q * 32) << 16), half * COLS, min(kSegment, kb_hi - kb), kb + kSegment >= kb_hi, sum,
                                p.status, 0x8000u);
      if (!ok) break;
      const int a = tw * p.BW + iw, b = th * p.BH + ih, img = ti * p.BI + ii;
      if (ii < p.BI && a < p.OW && b < p.OH && img < p.NI) {
        const int col0 = tn * BN + half * COLS;
        const int64_t base = p.out_index(a, b, img, col0);
        if (p.splits > 1) {
          float* d = p.partial + z * p.split_stride + base;
#pragma unroll
          for (int j = 0; j < COLS; ++j)
            if (col0 + j < p.n_out) { d[j * plane] = sum[j]; nan |= sum[j] != sum[j]; }
        } else {
          float* yp = p.y + base;
          float* pp = p.preact != nullptr ? p.preact + base : nullptr;
#pragma unroll
          for (int j = 0; j < COLS; ++j) {
            if (col0 + j < p.n_out) {
              const float v = sum[j] + (p.bias != nullptr ? __ldg(p.bias + col0 + j) : 0.f);
              if (pp != nullptr) pp[j * plane] = v;
              yp[j * plane] = v == v ? act_apply_any<ACT, false>(p.act, v) : v;   // cwf_redo_fwd finds it by its value
              nan |= v != v;
            }
          }
        }
      }
      __syncwarp();
    }
    if (ok && __any_sync(0xffffffffu, nan)) cwf_redo_fwd<BN>(p, q, half);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    if (*reinterpret_cast<volatile unsigned int*>(p.status) != 0) drain_after_abort();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// y = act(sum over splits (ascending) of partial + bias), in the layout of y
__global__ void __launch_bounds__(256) cwf_finish_kernel(float* __restrict__ y, float* __restrict__ preact, const float* __restrict__ partial,
                                                         const float* __restrict__ bias, int64_t n, int splits, int64_t split_stride,
                                                         int64_t plane, int channels, int act) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float v = 0.f;
#pragma unroll 4
    for (int z = 0; z < splits; ++z) v += __ldcs(partial + z * split_stride + i);
    if (bias != nullptr) v += __ldg(bias + (i / plane) % channels);
    if (preact != nullptr) preact[i] = v;
    y[i] = act_apply_any<-1, false>(act, v);
  }
}

struct CwfWgParams {
  int32_t KW_, KH_, KI_;              // a k-block is a box of 32 output positions
  int32_t kbw, kbh;                   // k-blocks along w and h
  int32_t sw, sh;
  int32_t m_tiles, tiles_n, splits, kb_total, kb_per_split;
  int32_t n_pairs, chunks, n_pad, cout;
  uint32_t idesc;
  float* partial;                     // [splits][m_tiles * 128][n_pad]
  unsigned int* status;
  CwfSource x, g;
  int32_t NI;
  int16_t tap_dw[kFMaxTaps], tap_dh[kFMaxTaps];
};

// As cwf_redo_fwd: the 32 rows of a warp are the channels of one tap and chunk, a lane forms its own elements.
template <int BN>
__device__ __noinline__ void cwf_redo_wgrad(const CwfWgParams& p, int q, int half) {
  constexpr int COLS = BN / 2;
  const int lane = threadIdx.x & 31, per_split = p.m_tiles * p.tiles_n;
  for (int item = blockIdx.x; item < per_split * p.splits; item += gridDim.x) {
    const int mt = item % p.m_tiles, nt = (item / p.m_tiles) % p.tiles_n, z = item / per_split;
    const int kb_lo = z * p.kb_per_split, kb_hi = min(p.kb_total, kb_lo + p.kb_per_split);
    const int pr = mt * 4 + q;
    if (pr >= p.n_pairs) continue;
    const int tap = pr / p.chunks, c = (pr - tap * p.chunks) * 32 + lane;
    float* const row = p.partial + ((int64_t)z * p.m_tiles * 128 + mt * 128 + q * 32 + lane) * p.n_pad;
    // body(x, position of dy) for every position of the item that is a term of the lane's elements, until done()
    auto walk = [&](auto body, auto done) {
      for (int kb = kb_lo; kb < kb_hi && !done(); ++kb) {
        const int a0 = (kb % p.kbw) * p.KW_, b0 = (kb / p.kbw) % p.kbh * p.KH_, i0 = kb / (p.kbw * p.kbh) * p.KI_;
        for (int t = 0; t < 32; ++t) {
          const int a = a0 + t % p.KW_, b = b0 + t / p.KW_ % p.KH_, img = i0 + t / (p.KW_ * p.KH_);
          const int w = a * p.sw + p.tap_dw[tap], h = b * p.sh + p.tap_dh[tap];
          if (a < p.g.W && b < p.g.H && img < p.NI && p.x.has(c, w, h)) body(p.x.at(c, w, h, img), a, b, img);
        }
      }
    };
    bool seen = false, x_nan = false;                    // a NaN among the channel's inputs settles all its filter elements
    for (int j = 0; j < COLS; ++j) {
      const int col = nt * BN + half * COLS + j;
      if (col >= p.cout) break;
      const bool nan = row[col] != row[col];
      if (!__any_sync(0xffffffffu, nan)) continue;
      if (!seen) {
        seen = true;
        walk([&](float x, int, int, int) { x_nan |= x != x; }, [&]() { return __all_sync(0xffffffffu, x_nan) != 0; });
      }
      const bool todo = nan && !x_nan;
      float sum = 0.f;
      walk([&](float x, int a, int b, int img) { sum = fmaf(x, p.g.at(col, a, b, img), sum); },
           [&]() { return !__any_sync(0xffffffffu, todo && sum == sum); });
      if (todo) row[col] = sum;
    }
  }
}
template <int BN>
__global__ void __launch_bounds__(kFThreads, 1)
conv_cwf_wgrad_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmG, const __grid_constant__ CwfWgParams p) {
  using Cfg = CwfCfg<BN>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_gen + STAGES * Cfg::STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  CwfRing<Cfg::SLOTS> ring{bars + 2 * STAGES, bars + 2 * STAGES + Cfg::SLOTS + 1, 0, 0, 0};
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ring.empty + Cfg::SLOTS + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_split = p.m_tiles * p.tiles_n;
  const int num_items = per_split * p.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a <= Cfg::SLOTS; ++a) { mbar_init(&ring.full[a], 1); mbar_init(&ring.empty[a], 8); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // item -> (m tile fastest, n tile, split)
  if (warp == 0) {
    tma_prefetch_desc(&tmX); tma_prefetch_desc(&tmG);
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      const int mt = item % p.m_tiles, nt = (item / p.m_tiles) % p.tiles_n, z = item / per_split;
      const int kb_lo = z * p.kb_per_split, kb_hi = min(p.kb_total, kb_lo + p.kb_per_split);
      int dw[4], dh[4], c0[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        int pr = mt * 4 + j;
        if (pr >= p.n_pairs) pr = mt * 4;              // filler rows (never read by the reduction)
        const int tap = pr / p.chunks;
        dw[j] = p.tap_dw[tap]; dh[j] = p.tap_dh[tap]; c0[j] = (pr - tap * p.chunks) * 32;
      }
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait_uniform(&empty[stage], phase ^ 1u, p.status, 0x20000u)) { ok = false; break; }
        if (elect_one()) {
          const int bw = kb % p.kbw, bh = (kb / p.kbw) % p.kbh, bi = kb / (p.kbw * p.kbh);
          const int a0 = bw * p.KW_, b0 = bh * p.KH_, i0 = bi * p.KI_;
          const uint32_t sA = smem_base + stage * Cfg::STAGE_BYTES, sB = sA + 3 * Cfg::A_BYTES;
          mbar_expect_tx(&full[stage], (uint32_t)Cfg::STAGE_BYTES);
#pragma unroll
          for (int j = 0; j < 4; ++j) tma_load_5d(sA + j * 6144, &tmX, c0[j], a0 * p.sw + dw[j], b0 * p.sh + dh[j], i0, 0, &full[stage]);
#pragma unroll
          for (int j = 0; j < BN / 32; ++j)              // channels past the last and positions past the ends are zero-filled
            tma_load_5d(sB + j * 6144, &tmG, nt * BN + j * 32, a0, b0, i0, 0, &full[stage]);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      const int z = item / per_split;
      const int kb_lo = z * p.kb_per_split, kb_hi = min(p.kb_total, kb_lo + p.kb_per_split);
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait_uniform(&full[stage], phase, p.status, 0x80000u)) { ok = false; break; }
        const uint32_t sA = smem_base + stage * Cfg::STAGE_BYTES, sB = sA + 3 * Cfg::A_BYTES;
        if (!cwf_issue_kblock<BN, true>(ring, tmem_base, sA, sB, p.idesc, kb - kb_lo, kb_hi - kb_lo, &empty[stage], p.status, 0x40000u)) { ok = false; break; }
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp >= 4) {
    const int q = warp & 3, half = (warp - 4) >> 2;
    constexpr int COLS = BN / 2;
    bool nan = false, ok = true;
    for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      const int mt = item % p.m_tiles, nt = (item / p.m_tiles) % p.tiles_n, z = item / per_split;
      const int kb_lo = z * p.kb_per_split, kb_hi = min(p.kb_total, kb_lo + p.kb_per_split);
      float4* dst = reinterpret_cast<float4*>(p.partial + ((int64_t)z * p.m_tiles * 128 + mt * 128 + q * 32 + lane) * p.n_pad + nt * BN + half * COLS);
      int kb = kb_lo;
      do {                                               // an empty split stores zeros
        float sum[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
        ok = cwf_accumulate<BN>(ring, tmem_base + ((uint32_t)(q * 32) << 16), half * COLS, max(0, min(kSegment, kb_hi - kb)), true, sum, p.status,
                                0x100000u);
        if (!ok) break;
#pragma unroll
        for (int j = 0; j < COLS / 4; ++j) {
          float4 v = make_float4(sum[4 * j], sum[4 * j + 1], sum[4 * j + 2], sum[4 * j + 3]);
          if (kb > kb_lo) { const float4 o = dst[j]; v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
          dst[j] = v;
          nan |= v.x != v.x || v.y != v.y || v.z != v.z || v.w != v.w;
        }
        kb += kSegment;
      } while (kb < kb_hi);
    }
    if (ok && __any_sync(0xffffffffu, nan)) cwf_redo_wgrad<BN>(p, q, half);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    if (*reinterpret_cast<volatile unsigned int*>(p.status) != 0) drain_after_abort();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// partial[0] = sum over splits (ascending, compensated: there are hundreds where the filter is small) of partial[z]
__device__ __forceinline__ void cwf_add(float& s, float& c, float v) {   // Kahan; a sum that is not finite is left as it is
  const float y = v - c, t = s + y;
  c = fabsf(t) < INFINITY ? (t - s) - y : 0.f;
  s = t;
}
__global__ void __launch_bounds__(256) cwf_sum_splits_kernel(float4* __restrict__ partial, int64_t n4, int splits) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
    float4 s = partial[i], c = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int z = 1; z < splits; ++z) {
      const float4 v = __ldcs(partial + z * n4 + i);
      cwf_add(s.x, c.x, v.x); cwf_add(s.y, c.y, v.y); cwf_add(s.z, c.z, v.z); cwf_add(s.w, c.w, v.w);
    }
    partial[i] = s;
  }
}
// dw[kw, kh, ci, co] = partial[(tap * chunks + ci / 32) * 32 + ci % 32][co]. A block takes 4 input channels x 32 output
// channels x all taps: lanes read 32 consecutive co, the block turns them in shared memory and writes runs of 4 * taps elements
// of dw. (Summing the splits here as well left all but 2 to 64 blocks of the GPU idle for small filters: 136 us for a stem's
// 74 splits, 52 us for 512 x 512 x 3 x 3.)
struct CwfReduce {
  int kW, kH, cin, cout, flip, fold, chunks, n_pad;
};
__global__ void __launch_bounds__(256) cwf_wgrad_store_kernel(float* __restrict__ dw, const float* __restrict__ partial, const CwfReduce g) {
  extern __shared__ float cwf_part[];                  // [4 channels][taps][33]
  const int taps = g.kW * g.kH;
  const int cgroups = (g.cin + 3) / 4;
  const int ci0 = (blockIdx.x % cgroups) * 4, co0 = (blockIdx.x / cgroups) * 32;
  const int lane = threadIdx.x & 31;
#pragma unroll 4
  for (int rt = threadIdx.x >> 5; rt < 4 * taps; rt += 8) {
    const int c = rt / taps, t = rt - c * taps, ci = min(ci0 + c, g.cin - 1);   // t in dw's (kh, kw) order
    const int kw = t % g.kW, kh = t / g.kW;
    const int tw = g.flip ? kw : g.kW - 1 - kw, th = g.flip ? kh : g.kH - 1 - kh;
    const int row = g.fold ? th * 32 + tw * g.cin + ci : ((th * g.kW + tw) * g.chunks + ci / 32) * 32 + (ci & 31);
    cwf_part[rt * 33 + lane] = partial[(int64_t)row * g.n_pad + co0 + lane];    // n_pad is a multiple of 64
  }
  __syncthreads();
  const int run = min(4, g.cin - ci0) * taps;
  for (int e = threadIdx.x; e < 32 * run; e += 256) {
    const int co = e / run, k = e - co * run;
    if (co0 + co < g.cout) dw[((int64_t)(co0 + co) * g.cin + ci0) * taps + k] = cwf_part[k * 33 + co];
  }
}

// ----------------------------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------------------------
// 5-D map over a channel-innermost array (Cp, W, H, N, part): box = 32 channels x bw x bh x bi positions of one part or all three
bool cwf_map(CUtensorMap* map, const CwfSource& s, int N, int bw, int bh, int bi, int sw, int sh, int parts) {
  TensorMapEncodeFn enc = tensor_map_encoder();
  if (!enc) return false;
  cuuint64_t dims[5] = {(cuuint64_t)s.Cp, (cuuint64_t)s.W, (cuuint64_t)s.H, (cuuint64_t)N, 3};
  cuuint64_t strides[4] = {(cuuint64_t)s.Cp * 2, (cuuint64_t)s.Cp * s.W * 2, (cuuint64_t)s.Cp * s.W * s.H * 2, (cuuint64_t)s.part_stride * 2};
  cuuint32_t box[5] = {32, (cuuint32_t)(bw * sw), (cuuint32_t)(bh * sh), (cuuint32_t)bi, (cuuint32_t)parts};
  cuuint32_t estr[5] = {1, (cuuint32_t)sw, (cuuint32_t)sh, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<uint16_t*>(s.ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool cwf_map_filter(CUtensorMap* map, const void* ptr, int64_t cols, int64_t rows, size_t packed_one, int box_rows) {
  TensorMapEncodeFn enc = tensor_map_encoder();
  if (!enc) return false;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, 3};
  cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)packed_one};
  cuuint32_t box[3] = {32, (cuuint32_t)box_rows, 3};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

unsigned cwf_flat_grid(int64_t total) {
  const int64_t gsz = (total + 255) / 256, cap = (int64_t)sm_count() * 16;
  return (unsigned)(gsz < 1 ? 1 : (gsz > cap ? cap : gsz));
}
int cwf_bn(int n_out) { return n_out <= 64 ? 64 : 128; }
int cwf_chunks(int c) { return (c + 31) / 32; }
// the kW taps of a small-channel input share one 32-channel chunk
int cwf_fold(const ConvGeom& g) { return g.k[0] > 1 && g.k[0] * g.cin <= 32 ? 1 : 0; }
int cwf_taps(const ConvGeom& g) { return cwf_fold(g) ? g.k[1] : g.k[0] * g.k[1]; }

struct CwfCopy {
  int Cp, W, H;
  size_t one;          // bytes of one part
  size_t bytes() const { return 3 * one; }
  int64_t part_stride() const { return (int64_t)(one / 2); }
};
CwfCopy cwf_copy(int C, int W, int H, int N) {
  CwfCopy c{};
  c.Cp = (C + 7) / 8 * 8; c.W = W; c.H = H;   // TMA strides are multiples of 16 bytes
  c.one = align_up((size_t)c.Cp * W * H * N * 2, 1024);
  return c;
}
CwfCopy cwf_copy_x(const ConvGeom& g) {
  return cwf_fold(g) ? cwf_copy(g.k[0] * g.cin, g.out[0], g.in[1], g.batch) : cwf_copy(g.cin, g.in[0], g.in[1], g.batch);
}
CwfCopy cwf_copy_y(const ConvGeom& g) { return cwf_copy(g.cout, g.out[0], g.out[1], g.batch); }

CwfSource cwf_source(const void* ptr, const CwfCopy& c, const ConvGeom& g, int fold) {
  return CwfSource{static_cast<const uint16_t*>(ptr), c.part_stride(), c.Cp, c.W, c.H, fold ? g.cin : 0, g.stride[0], g.dil[0], g.pad_lo[0], g.in[0]};
}

size_t cwf_packed_one(int rows, int taps, int chunks) {
  return align_up((size_t)((rows + cwf_bn(rows) - 1) / cwf_bn(rows) * cwf_bn(rows)) * taps * chunks * 32 * 2, 1024);
}

// Split along the contraction: cost in k-blocks (about 0.6 us each) of `items` tiles on the SMs in `s` splits, 6 for a
// tile's start and end, and for s > 1 the partials' round trip (8 bytes per element at about 4 TB/s = 2.4 MB per k-block)
// and one more launch.
int cwf_splits(int64_t items, int kb, int64_t numel, int most) {
  const int sms = sm_count();
  double best = 0;
  int pick = 1;
  for (int s = 1; s <= most && s <= kb; s += 1 + s / 16) {
    const double waves = (double)((items * s + sms - 1) / sms);
    const double cost = waves * ((kb + s - 1) / s + 6) + (s > 1 ? 6.0 + (double)s * numel * 8.0 / 2.4e6 : 0.0);
    if (s == 1 || cost < best * 0.97) { best = cost; pick = s; }
  }
  return pick;
}

struct CwfGrid {       // tiling of one launch of the forward kernel
  int BW, BH, BI, tw, th, ti, tn;
  int64_t tiles() const { return (int64_t)tw * th * ti * tn; }
};
CwfGrid cwf_grid(int OW, int OH, int NI, int n_out) {
  CwfGrid t{};
  conv_position_box(OW, OH, NI, kFBM, 1, 1, &t.BW, &t.BH, &t.BI);
  t.tw = (OW + t.BW - 1) / t.BW; t.th = (OH + t.BH - 1) / t.BH; t.ti = (NI + t.BI - 1) / t.BI;
  t.tn = (n_out + cwf_bn(n_out) - 1) / cwf_bn(n_out);
  return t;
}

int cwf_fwd_splits(const ConvGeom& g) {
  const int64_t numel = (int64_t)g.out[0] * g.out[1] * g.cout * g.batch;
  return cwf_splits(cwf_grid(g.out[0], g.out[1], g.batch, g.cout).tiles(), cwf_taps(g) * (cwf_fold(g) ? 1 : cwf_chunks(g.cin)), numel, kFMaxSplits);
}
int64_t x_numel(const ConvGeom& g) { return (int64_t)g.in[0] * g.in[1] * g.cin * g.batch; }
// one split count for all residue classes of the data gradient, from the class with the most taps
int cwf_dgrad_splits(const ConvGeom& g) {
  const int sw = g.stride[0], sh = g.stride[1];
  const int tw = (g.k[0] + sw - 1) / sw, th = (g.k[1] + sh - 1) / sh;
  const CwfGrid t = cwf_grid((g.in[0] + sw - 1) / sw, (g.in[1] + sh - 1) / sh, g.batch, g.cin);
  return cwf_splits(t.tiles(), tw * th * cwf_chunks(g.cout), x_numel(g), kFMaxSplits);
}

int32_t cwf_transpose(void* out, const CwfCopy& c, const float* in, int S, int C, int N, cudaStream_t st) {
  const int64_t blocks = (int64_t)N * ((S + 63) / 64) * ((c.Cp + 31) / 32);
  const int64_t cap = (int64_t)sm_count() * 8;
  const unsigned grid = (unsigned)(blocks < cap ? blocks : cap);
  if (S % 4 == 0 && aligned_to(in, 16)) cwf_transpose_kernel<true><<<grid, 256, 0, st>>>((uint16_t*)out, c.part_stride(), in, S, C, c.Cp, N);
  else cwf_transpose_kernel<false><<<grid, 256, 0, st>>>((uint16_t*)out, c.part_stride(), in, S, C, c.Cp, N);
  LB2_CHECK_LAUNCH("conv_cw_f32 transpose");
  return LB2_OK;
}
int32_t cwf_make_copy_x(void* out, const float* x, const ConvGeom& g, const CwfCopy& c, cudaStream_t st) {
  if (!cwf_fold(g)) return cwf_transpose(out, c, x, g.in[0] * g.in[1], g.cin, g.batch, st);
  cwf_fold_kernel<<<cwf_flat_grid((int64_t)(c.Cp / 8) * c.W * c.H * g.batch), 256, 0, st>>>(
      (uint16_t*)out, c.part_stride(), x, g.in[0], g.in[1], g.cin, c.Cp, g.batch, g.out[0], g.k[0], g.stride[0], g.dil[0], g.pad_lo[0]);
  LB2_CHECK_LAUNCH("conv_cw_f32 folded copy");
  return LB2_OK;
}
int32_t cwf_pack(uint16_t* out, size_t packed_one, const float* w, const CwfPack& pk, cudaStream_t st) {
  const size_t tile = (size_t)pk.kW * pk.kH * 256 * sizeof(float);
  if (!pk.fold && tile <= 48 * 1024)
    cwf_pack_tile_kernel<<<(unsigned)(pk.n_rows / 8 * pk.chunks), 256, tile, st>>>(out, (int64_t)(packed_one / 2), w, pk);
  else
    cwf_pack_flat_kernel<<<cwf_flat_grid((int64_t)pk.n_rows * pk.k_total), 256, 0, st>>>(out, (int64_t)(packed_one / 2), w, pk);
  LB2_CHECK_LAUNCH("conv_cw_f32 filter packing");
  return LB2_OK;
}

uint32_t cwf_idesc(int n, bool mn_major) {
  const uint32_t mj = mn_major ? 1u : 0u;
  return (1u << 4) | (1u << 7) | (1u << 10) | (mj << 15) | (mj << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kFBM >> 4) << 24);
}

struct CwfTap { int dw, dh, index; };
struct CwfOut {         // destination of a forward / data-gradient GEMM
  float *y, *preact;
  const float* bias;
  int32_t act;
  int FW, FH, ow_step, ow_off, oh_step, oh_off;
  float* partial;
  int splits;
  int64_t split_stride;
};
int32_t cwf_run(const CwfOut& o, const CwfSource& src, int NI, int chunks, const uint16_t* wp, size_t packed_one, int wp_rows, int wp_cols,
                const CwfTap* taps, int n_taps, int OW, int OH, int sw, int sh, int n_out, cudaStream_t st) {
  const int bn = cwf_bn(n_out);
  const CwfGrid t = cwf_grid(OW, OH, NI, n_out);
  CwfFwdParams p{};
  p.OW = OW; p.OH = OH; p.NI = NI; p.BW = t.BW; p.BH = t.BH; p.BI = t.BI;
  p.tiles_w = t.tw; p.tiles_h = t.th; p.tiles_i = t.ti; p.tiles_n = t.tn;
  p.chunks = chunks; p.num_kb = n_taps * chunks;
  p.splits = o.splits; p.kb_per_split = (p.num_kb + o.splits - 1) / o.splits;
  p.sw = sw; p.sh = sh; p.n_out = n_out;
  p.FW = o.FW; p.FH = o.FH; p.ow_step = o.ow_step; p.ow_off = o.ow_off; p.oh_step = o.oh_step; p.oh_off = o.oh_off;
  p.idesc = cwf_idesc(bn, false);
  p.y = o.y; p.preact = o.preact; p.bias = o.bias; p.act = o.act; p.partial = o.partial; p.split_stride = o.split_stride;
  p.status = device_status_word();
  LB2_REQUIRE(p.status != nullptr, LB2_LAUNCH_FAIL, "conv_cw_f32: device status word unavailable");
  for (int i = 0; i < n_taps; ++i) {
    p.tap_dw[i] = (int16_t)taps[i].dw; p.tap_dh[i] = (int16_t)taps[i].dh; p.tap_index[i] = (int16_t)taps[i].index;
  }
  p.src = src; p.wp = wp; p.wp_part_stride = (int64_t)(packed_one / 2); p.wp_cols = wp_cols;
  CUtensorMap mX, mW;
  // the parts of a position box that is no multiple of 8 positions would start inside a swizzle atom: one load each
  if (!cwf_map(&mX, src, NI, t.BW, t.BH, t.BI, sw, sh, 1) || !cwf_map_filter(&mW, wp, wp_cols, wp_rows, packed_one, bn))
    return fail(LB2_LAUNCH_FAIL, "conv_cw_f32: cuTensorMapEncodeTiled failed");
  const int64_t items = t.tiles() * o.splits;
  LB2_REQUIRE(items <= 0x7FFFFFFF, LB2_BAD_SHAPE, "conv_cw_f32: too many tiles");
  const int grid = (int)(items < sm_count() ? items : sm_count());
  auto launch = [&](auto kernel, int smem) -> int32_t {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail(LB2_LAUNCH_FAIL, "conv_cw_f32: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
    kernel<<<grid, kFThreads, smem, st>>>(mX, mW, p);
    LB2_CHECK_LAUNCH("conv_cw_f32");
    return LB2_OK;
  };
  const bool plain = o.act == LB2_ACT_IDENTITY || o.splits > 1;
  if (bn == 64) return plain ? launch(conv_cwf_fwd_kernel<64, LB2_ACT_IDENTITY>, CwfCfg<64>::SMEM_BYTES)
                             : launch(conv_cwf_fwd_kernel<64, -1>, CwfCfg<64>::SMEM_BYTES);
  return plain ? launch(conv_cwf_fwd_kernel<128, LB2_ACT_IDENTITY>, CwfCfg<128>::SMEM_BYTES)
               : launch(conv_cwf_fwd_kernel<128, -1>, CwfCfg<128>::SMEM_BYTES);
}
int32_t cwf_finish(const CwfOut& o, int64_t numel, int channels, cudaStream_t st) {
  if (o.splits <= 1) return LB2_OK;
  cwf_finish_kernel<<<cwf_flat_grid(numel), 256, 0, st>>>(o.y, o.preact, o.partial, o.bias, numel, o.splits, o.split_stride,
                                                          (int64_t)o.FW * o.FH, channels, o.act);
  LB2_CHECK_LAUNCH("conv_cw_f32 split sum");
  return LB2_OK;
}

// 32 positions per k-block in power-of-two boxes; of those the one that covers the output in the fewest blocks, among equals
// the widest
void cwf_wg_box(const ConvGeom& g, int* KW, int* KH, int* KI) {
  int64_t best = 0;
  for (int kw = 1; kw <= 32; kw *= 2)
    for (int kh = 1; kh * kw <= 32; kh *= 2) {
      const int ki = 32 / (kw * kh);
      const int64_t n = (int64_t)((g.out[0] + kw - 1) / kw) * ((g.out[1] + kh - 1) / kh) * ((g.batch + ki - 1) / ki);
      if (best == 0 || n <= best) { best = n; *KW = kw; *KH = kh; *KI = ki; }
    }
}
struct CwfWgPlan {
  int chunks, n_pairs, m_tiles, tiles_n, n_pad, KW_, KH_, KI_, kbw, kbh, kb_total, splits, kb_per_split;
  size_t partial_bytes;
};
CwfWgPlan cwf_wg_plan(const ConvGeom& g) {
  CwfWgPlan w{};
  w.chunks = cwf_fold(g) ? 1 : cwf_chunks(g.cin);
  w.n_pairs = cwf_taps(g) * w.chunks;
  w.m_tiles = (w.n_pairs + 3) / 4;
  const int bn = cwf_bn(g.cout);
  w.tiles_n = (g.cout + bn - 1) / bn;
  w.n_pad = w.tiles_n * bn;
  cwf_wg_box(g, &w.KW_, &w.KH_, &w.KI_);
  w.kbw = (g.out[0] + w.KW_ - 1) / w.KW_; w.kbh = (g.out[1] + w.KH_ - 1) / w.KH_;
  w.kb_total = w.kbw * w.kbh * ((g.batch + w.KI_ - 1) / w.KI_);
  const int64_t items = (int64_t)w.m_tiles * w.tiles_n;
  const int splits = cwf_splits(items, w.kb_total, items * 128 * bn, 2 * sm_count());
  w.kb_per_split = (w.kb_total + splits - 1) / splits;
  w.splits = (w.kb_total + w.kb_per_split - 1) / w.kb_per_split;
  w.partial_bytes = align_up((size_t)w.splits * w.m_tiles * 128 * w.n_pad * sizeof(float), 1024);
  return w;
}

}  // namespace

bool conv_cwf_supported(const ConvGeom& g) {
  if (g.ndim != 2 || g.groups != 1) return false;
  if (g.out[0] <= 0 || g.out[1] <= 0 || g.in[0] <= 0 || g.in[1] <= 0 || g.batch <= 0 || g.cin <= 0 || g.cout <= 0) return false;
  if (g.stride[0] > 4 || g.stride[1] > 4) return false;               // box extent = positions x stride must stay <= 256
  if (g.k[0] * g.k[1] > kFMaxTaps) return false;
  if (g.k[0] * g.dil[0] > 120 || g.k[1] * g.dil[1] > 120) return false;
  if (g.pad_lo[0] > 30000 || g.pad_lo[1] > 30000) return false;        // tap offsets are 16 bits wide
  if ((int64_t)g.in[0] * g.in[1] >= (1 << 30) || (int64_t)g.out[0] * g.out[1] >= (1 << 30)) return false;   // positions of a plane: int
  if (x_numel(g) >= ((int64_t)1 << 40)) return false;
  const CwfGrid t = cwf_grid(g.out[0], g.out[1], g.batch, g.cout);
  if (t.BW * g.stride[0] > 256 || t.BH * g.stride[1] > 256) return false;
  return tensor_map_encoder() != nullptr;
}

size_t conv_cwf_fwd_workspace_bytes(const ConvGeom& g) {
  const int s = cwf_fwd_splits(g);
  return cwf_copy_x(g).bytes() + 3 * cwf_packed_one(g.cout, cwf_taps(g), cwf_fold(g) ? 1 : cwf_chunks(g.cin)) +
         (s > 1 ? align_up((size_t)s * g.out[0] * g.out[1] * g.cout * g.batch * 4, 1024) : 0);
}

int32_t conv_cwf_fwd(void* y, void* preact, const void* x, const void* w, const void* bias, const ConvGeom& g, int32_t act, void* ws_,
                     cudaStream_t st) {
  uint8_t* ws = static_cast<uint8_t*>(ws_);
  const int fold = cwf_fold(g), n_taps = cwf_taps(g);
  const CwfCopy xc = cwf_copy_x(g);
  int32_t rc = cwf_make_copy_x(ws, (const float*)x, g, xc, st);
  if (rc != LB2_OK) return rc;
  CwfPack pk{g.k[0], g.k[1], g.cin, g.cout, g.flip, 0, fold, fold ? 1 : cwf_chunks(g.cin), 0, 0};
  pk.n_rows = (g.cout + cwf_bn(g.cout) - 1) / cwf_bn(g.cout) * cwf_bn(g.cout);
  pk.k_total = n_taps * pk.chunks * 32;
  const size_t packed = cwf_packed_one(g.cout, n_taps, pk.chunks);
  uint16_t* wp = reinterpret_cast<uint16_t*>(ws + xc.bytes());
  rc = cwf_pack(wp, packed, (const float*)w, pk, st);
  if (rc != LB2_OK) return rc;
  CwfTap taps[kFMaxTaps];
  for (int t = 0; t < n_taps; ++t)
    taps[t] = fold ? CwfTap{0, t * g.dil[1] - g.pad_lo[1], t}
                   : CwfTap{(t % g.k[0]) * g.dil[0] - g.pad_lo[0], (t / g.k[0]) * g.dil[1] - g.pad_lo[1], t};
  const int64_t numel = (int64_t)g.out[0] * g.out[1] * g.cout * g.batch;
  const CwfOut o{(float*)y, (float*)preact, (const float*)bias, act, g.out[0], g.out[1], 1, 0, 1, 0,
                 reinterpret_cast<float*>(ws + xc.bytes() + 3 * packed), cwf_fwd_splits(g), numel};
  rc = cwf_run(o, cwf_source(ws, xc, g, fold), g.batch, pk.chunks, wp, packed, pk.n_rows, pk.k_total, taps, n_taps, g.out[0], g.out[1],
               fold ? 1 : g.stride[0], g.stride[1], g.cout, st);
  return rc != LB2_OK ? rc : cwf_finish(o, numel, g.cout, st);
}

size_t conv_cwf_bwd_workspace_bytes(const ConvGeom& g) {
  const int s = cwf_dgrad_splits(g);
  const size_t dgrad = 3 * cwf_packed_one(g.cin, g.k[0] * g.k[1], cwf_chunks(g.cout)) + (s > 1 ? align_up((size_t)s * x_numel(g) * 4, 1024) : 0);
  const size_t wgrad = cwf_copy_x(g).bytes() + cwf_wg_plan(g).partial_bytes;
  return cwf_copy_y(g).bytes() + (dgrad > wgrad ? dgrad : wgrad);
}

// both gradients (either output may be null) from one copy of gy
int32_t conv_cwf_bwd(void* dw, void* dx, const void* x, const void* gy, const void* w, const ConvGeom& g, void* ws_, cudaStream_t st) {
  uint8_t* ws = static_cast<uint8_t*>(ws_);
  const CwfCopy yc = cwf_copy_y(g);
  const CwfSource gcopy = cwf_source(ws, yc, g, 0);
  int32_t rc = cwf_transpose(ws, yc, (const float*)gy, g.out[0] * g.out[1], g.cout, g.batch, st);
  if (rc != LB2_OK) return rc;
  uint8_t* rest = ws + yc.bytes();

  if (dw != nullptr) {
    const int fold = cwf_fold(g), n_taps = cwf_taps(g);
    const CwfCopy xc = cwf_copy_x(g);
    const CwfSource xcopy = cwf_source(rest, xc, g, fold);
    rc = cwf_make_copy_x(rest, (const float*)x, g, xc, st);
    if (rc != LB2_OK) return rc;
    const CwfWgPlan pl = cwf_wg_plan(g);
    const int bn = cwf_bn(g.cout);
    CwfWgParams q{};
    q.KW_ = pl.KW_; q.KH_ = pl.KH_; q.KI_ = pl.KI_; q.kbw = pl.kbw; q.kbh = pl.kbh;
    q.sw = fold ? 1 : g.stride[0]; q.sh = g.stride[1];
    q.m_tiles = pl.m_tiles; q.tiles_n = pl.tiles_n; q.splits = pl.splits; q.kb_total = pl.kb_total; q.kb_per_split = pl.kb_per_split;
    q.n_pairs = pl.n_pairs; q.chunks = pl.chunks; q.n_pad = pl.n_pad; q.cout = g.cout;
    q.x = xcopy; q.g = gcopy; q.NI = g.batch;
    q.idesc = cwf_idesc(bn, true);
    q.partial = reinterpret_cast<float*>(rest + xc.bytes());
    q.status = device_status_word();
    LB2_REQUIRE(q.status != nullptr, LB2_LAUNCH_FAIL, "conv_cw_f32: device status word unavailable");
    for (int t = 0; t < n_taps; ++t) {
      q.tap_dw[t] = (int16_t)(fold ? 0 : (t % g.k[0]) * g.dil[0] - g.pad_lo[0]);
      q.tap_dh[t] = (int16_t)((fold ? t : t / g.k[0]) * g.dil[1] - g.pad_lo[1]);
    }
    CUtensorMap mX, mG;
    if (!cwf_map(&mX, xcopy, g.batch, pl.KW_, pl.KH_, pl.KI_, q.sw, q.sh, 3) || !cwf_map(&mG, gcopy, g.batch, pl.KW_, pl.KH_, pl.KI_, 1, 1, 3))
      return fail(LB2_LAUNCH_FAIL, "conv_cw_f32: cuTensorMapEncodeTiled failed");
    const int64_t items = (int64_t)pl.m_tiles * pl.tiles_n * pl.splits;
    LB2_REQUIRE(items <= 0x7FFFFFFF, LB2_BAD_SHAPE, "conv_cw_f32: too many tiles");
    const int grid = (int)(items < sm_count() ? items : sm_count());
    auto launch = [&](auto kernel, int smem) -> int32_t {
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e != cudaSuccess) return fail(LB2_LAUNCH_FAIL, "conv_cw_f32: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
      kernel<<<grid, kFThreads, smem, st>>>(mX, mG, q);
      LB2_CHECK_LAUNCH("conv_cw_f32 filter gradient");
      return LB2_OK;
    };
    rc = bn == 64 ? launch(conv_cwf_wgrad_kernel<64>, CwfCfg<64>::SMEM_BYTES) : launch(conv_cwf_wgrad_kernel<128>, CwfCfg<128>::SMEM_BYTES);
    if (rc != LB2_OK) return rc;
    if (pl.splits > 1) {
      const int64_t n4 = (int64_t)pl.m_tiles * 128 * pl.n_pad / 4;
      cwf_sum_splits_kernel<<<cwf_flat_grid(n4), 256, 0, st>>>(reinterpret_cast<float4*>(q.partial), n4, pl.splits);
      LB2_CHECK_LAUNCH("conv_cw_f32 filter-gradient split sum");
    }
    const CwfReduce rd{g.k[0], g.k[1], g.cin, g.cout, g.flip, fold, pl.chunks, pl.n_pad};
    const int smem = 4 * g.k[0] * g.k[1] * 33 * 4, most = 4 * kFMaxTaps * 33 * 4;   // the limit is the kernel's: the same for every thread
    cudaError_t e = cudaFuncSetAttribute(cwf_wgrad_store_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return fail(LB2_LAUNCH_FAIL, "conv_cw_f32: cannot reserve %d bytes of shared memory: %s", most, cudaGetErrorString(e));
    cwf_wgrad_store_kernel<<<(unsigned)(((g.cin + 3) / 4) * ((g.cout + 31) / 32)), 256, smem, st>>>((float*)dw, q.partial, rd);
    LB2_CHECK_LAUNCH("conv_cw_f32 filter-gradient reduction");
  }

  if (dx != nullptr) {
    // per residue class of the input position (mod stride) a stride-1 problem over gy's copy, written to that class's
    // subset of dx
    CwfPack pk{g.k[0], g.k[1], g.cin, g.cout, g.flip, 1, 0, cwf_chunks(g.cout), 0, 0};
    pk.n_rows = (g.cin + cwf_bn(g.cin) - 1) / cwf_bn(g.cin) * cwf_bn(g.cin);
    pk.k_total = g.k[0] * g.k[1] * pk.chunks * 32;
    const size_t packed = cwf_packed_one(g.cin, g.k[0] * g.k[1], pk.chunks);
    uint16_t* wp = reinterpret_cast<uint16_t*>(rest);
    rc = cwf_pack(wp, packed, (const float*)w, pk, st);
    if (rc != LB2_OK) return rc;
    const int sw = g.stride[0], sh = g.stride[1];
    const int64_t numel = x_numel(g);
    CwfOut o{(float*)dx, nullptr, nullptr, LB2_ACT_IDENTITY, g.in[0], g.in[1], sw, 0, sh, 0, reinterpret_cast<float*>(rest + 3 * packed),
             cwf_dgrad_splits(g), numel};
    auto class_taps = [&](int pw, int ph, CwfTap* taps) {
      int n = 0;
      for (int th = 0; th < g.k[1]; ++th) {
        const int nh = ph + g.pad_lo[1] - th * g.dil[1];
        if (((nh % sh) + sh) % sh != 0) continue;
        for (int tw = 0; tw < g.k[0]; ++tw) {
          const int nw = pw + g.pad_lo[0] - tw * g.dil[0];
          if (((nw % sw) + sw) % sw != 0) continue;
          taps[n++] = CwfTap{nw / sw, nh / sh, th * g.k[0] + tw};   // exact: nw, nh are multiples of the stride
        }
      }
      return n;
    };
    CwfTap taps[kFMaxTaps];
    bool any_empty = false;
    for (int ph = 0; ph < sh && ph < g.in[1]; ++ph)
      for (int pw = 0; pw < sw && pw < g.in[0]; ++pw)
        if (class_taps(pw, ph, taps) == 0) any_empty = true;
    if (any_empty) {   // classes no tap reaches stay zero (in every split)
      cudaError_t e = o.splits > 1 ? cudaMemsetAsync(o.partial, 0, (size_t)o.splits * numel * 4, st) : cudaMemsetAsync(dx, 0, (size_t)numel * 4, st);
      if (e != cudaSuccess) return fail(LB2_LAUNCH_FAIL, "conv_cw_f32: clearing dx failed: %s", cudaGetErrorString(e));
    }
    for (int ph = 0; ph < sh && ph < g.in[1]; ++ph)
      for (int pw = 0; pw < sw && pw < g.in[0]; ++pw) {
        const int n = class_taps(pw, ph, taps);
        if (n == 0) continue;
        o.ow_off = pw; o.oh_off = ph;
        rc = cwf_run(o, gcopy, g.batch, pk.chunks, wp, packed, pk.n_rows, pk.k_total, taps, n, (g.in[0] - pw + sw - 1) / sw,
                     (g.in[1] - ph + sh - 1) / sh, 1, 1, g.cin, st);
        if (rc != LB2_OK) return rc;
      }
    return cwf_finish(o, numel, g.cin, st);
  }
  return LB2_OK;
}

}  // namespace lb2
