// Internal convolution interface.
#pragma once
#include "common.cuh"

namespace lb2 {

// lb2_conv_desc normalised to three spatial dims (missing dims have extent 1).
struct ConvGeom {
  int in[3], k[3], stride[3], pad_lo[3], pad_hi[3], dil[3], out[3];
  int groups, flip, cin, cout, batch, ndim;
};

int32_t conv_fwd_direct(void* y, void* preact, const void* x, const void* w, const void* bias, const ConvGeom& g,
                        int32_t dtype, int32_t act, cudaStream_t st);
int32_t conv_dgrad_direct(void* dx, const void* dy, const void* w, const ConvGeom& g, int32_t dtype, cudaStream_t st);
int32_t conv_wgrad_direct(void* dw, const void* x, const void* dy, const ConvGeom& g, int32_t dtype, cudaStream_t st);

// Tensor-core implicit-GEMM path on the WHCN bytes themselves (2-D, stride 1, dilation 1, groups 1, output width ==
// input width, filter small enough to stay resident in shared memory); bf16 in conv_tc.cu, Float32 (split tf32 with
// register accumulation) in conv_tc_f32.cu.
bool conv_tc_supported(const ConvGeom& g, int32_t dtype);
size_t conv_tc_fwd_workspace_bytes(const ConvGeom& g, int32_t dtype);
size_t conv_tc_bwd_workspace_bytes(const ConvGeom& g, int32_t dtype);
int32_t conv_tc_fwd(void* y, void* preact, const void* x, const void* w, const void* bias, const ConvGeom& g,
                    int32_t dtype, int32_t act, void* ws, cudaStream_t st);
int32_t conv_tc_dgrad(void* dx, const void* gy, const void* w, const ConvGeom& g, int32_t dtype, void* ws, cudaStream_t st);
// `db` (optional): also the bias gradient sum_{positions, images} gy, where conv_tc_wgrad_makes_db says the kernel can
int32_t conv_tc_wgrad(void* dw, const void* x, const void* gy, const ConvGeom& g, int32_t dtype, void* ws, cudaStream_t st,
                      void* db = nullptr);
bool conv_tc_wgrad_makes_db(const ConvGeom& g, int32_t dtype);

// General bf16 tensor-core path on channel-innermost copies (conv_cw.cu): any 2-D stride / padding / dilation /
// kernel size / channel counts with groups == 1.
bool conv_cw_supported(const ConvGeom& g, int32_t dtype);
int conv_cw_fwd_kblocks(const ConvGeom& g);
size_t conv_cw_fwd_workspace_bytes(const ConvGeom& g);
size_t conv_cw_bwd_workspace_bytes(const ConvGeom& g);
int32_t conv_cw_fwd(void* y, void* preact, const void* x, const void* w, const void* bias, const ConvGeom& g, int32_t act,
                    void* ws, cudaStream_t st, float* sums = nullptr);
// both gradients (either of dw, dx may be null) from one channel-innermost copy of gy
int32_t conv_cw_bwd(void* dw, void* dx, const void* x, const void* gy, const void* w, const ConvGeom& g, void* ws,
                    cudaStream_t st, bool x_is_copy = false);

// General Float32 tensor-core path on channel-innermost copies in three bf16 parts (conv_cw_f32.cu), same geometries.
bool conv_cwf_supported(const ConvGeom& g);
size_t conv_cwf_fwd_workspace_bytes(const ConvGeom& g);
size_t conv_cwf_bwd_workspace_bytes(const ConvGeom& g);
int32_t conv_cwf_fwd(void* y, void* preact, const void* x, const void* w, const void* bias, const ConvGeom& g, int32_t act,
                     void* ws, cudaStream_t st);
int32_t conv_cwf_bwd(void* dw, void* dx, const void* x, const void* gy, const void* w, const ConvGeom& g, void* ws,
                     cudaStream_t st);

// Box of at most `most` positions (BW columns x BH rows x BI images) for an OW x OH x NI grid, rows cut into equal pieces of at
// least 8 columns: the one whose boxes, `per_box` tiles each, take the fewest waves of `wave` tiles (wave = 1: the fewest
// boxes); among equals the widest and tallest, whose stores are the longest runs. 14 x 14 maps in whole rows fill 98 of 128
// positions, in 14 x 1 x 9 boxes 126 (3x3 256 -> 256, batch 256, bf16: forward 91 -> 79 us); on 7 x 7 both take two waves and
// the whole planes are 4 % faster.
inline void conv_position_box(int OW, int OH, int NI, int most, int64_t per_box, int64_t wave, int* BW, int* BH, int* BI) {
  int64_t best = 0;
  for (int bw = OW < most ? OW : most; bw >= 1; --bw) {   // widths, not counts of pieces: at most `most` of them for rows of any length
    const int pieces = (OW + bw - 1) / bw;
    if ((OW + pieces - 1) / pieces != bw) continue;       // no width of equal pieces
    if (best != 0 && bw < 8) break;
    const int rows = most / bw;
    for (int bh = rows < OH ? rows : OH; bh >= 1; --bh) {
      const int bi = rows / bh < NI ? rows / bh : NI;
      const int64_t n = (int64_t)pieces * ((OH + bh - 1) / bh) * ((NI + bi - 1) / bi);
      const int64_t waves = (n * per_box + wave - 1) / wave;
      if (best == 0 || waves < best) { best = waves; *BW = bw; *BH = bh; *BI = bi; }
    }
  }
}

bool conv_tc_f32_supported(const ConvGeom& g);
size_t conv_tc_f32_fwd_workspace_bytes(const ConvGeom& g);
size_t conv_tc_f32_bwd_workspace_bytes(const ConvGeom& g);
int32_t conv_tc_f32_fwd(void* y, void* preact, const void* x, const void* w, const void* bias, const ConvGeom& g,
                        int32_t act, void* ws, cudaStream_t st);
// both gradients (either of dw, dx may be null) from one set of shifted copies of gy
int32_t conv_tc_f32_bwd(void* dw, void* dx, const void* x, const void* gy, const void* w, const ConvGeom& g, void* ws,
                        cudaStream_t st);

}  // namespace lb2
