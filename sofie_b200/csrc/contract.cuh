// Internal launcher interface between api.cu (validation, dispatch) and the kernel files.
#pragma once
#include "common.cuh"

namespace sofie {

struct ConvGeom {
   int N, C, H, W, Cout, kH, kW, pad_h, pad_w, sh, sw, dh, dw, group;
   int oH, oW;    // convolution output extent
   int pH, pW;    // stored output extent (halved when pool == 2)
   int x_nhwc, y_nhwc, w_packed, relu, pool;
};

int launch_gemm_f32_simt(cudaStream_t, const sofie_gemm_f32_desc &, const float *, const float *, const float *, float *);
// at most 8 rows or columns, any layout (gemm_skinny.cu)
bool gemm_f32_skinny_ok(const sofie_gemm_f32_desc &);
int launch_gemm_f32_skinny(cudaStream_t, const sofie_gemm_f32_desc &, const float *, const float *, const float *, float *);
// few FMAs, any layout
bool gemm_f32_tiny_ok(const sofie_gemm_f32_desc &);
int launch_gemm_f32_tiny(cudaStream_t, const sofie_gemm_f32_desc &, const float *, const float *, const float *, float *);
int launch_gemm_f32_umma(cudaStream_t, const sofie_gemm_f32_desc &, const float *, const float *, const float *, float *);
// any layout, alignment and K; long K split over a cluster (umma_gemm_any.cu). tma: operands the TMA kernel takes too; others are refused
// where the CUDA-core kernel is the faster one
int launch_gemm_f32_any(cudaStream_t, const sofie_gemm_f32_desc &, bool tma, const float *, const float *, const float *, float *);
// the time in ns that such a product is estimated to take there or on the CUDA cores, whichever is faster
long long gemm_f32_whole_ns(const sofie_gemm_f32_desc &, bool tma);
// the same out of operands split into a workspace first (umma_gemm_parts.cu): UNSUPPORTED without one of gemm_f32_parts_bytes (0: not its shape)
size_t gemm_f32_parts_bytes(const sofie_gemm_f32_desc &);
int launch_gemm_f32_parts(cudaStream_t, const sofie_gemm_f32_desc &, const float *, const float *, const float *, float *, void *workspace, size_t bytes);
int launch_qgemm_simt(cudaStream_t, const sofie_qgemm_desc &, const uint8_t *, const int8_t *, const float *,
                      const int32_t *, uint8_t *, float *Yf32, float dq_scale);
int launch_qgemm_umma(cudaStream_t, const sofie_qgemm_desc &, const uint8_t *, const int8_t *, const float *,
                      const int32_t *, uint8_t *, float *Yf32, float dq_scale);
int launch_gemm_e4m3_simt(cudaStream_t, const sofie_fp8_gemm_desc &, const uint8_t *, const uint8_t *, const float *,
                          uint16_t *, uint8_t *, float *Yf32, const float *a_scale_dev = nullptr);
int launch_gemm_e4m3_umma(cudaStream_t, const sofie_fp8_gemm_desc &, const uint8_t *, const uint8_t *, const float *,
                          uint16_t *, uint8_t *, float *Yf32, const float *a_scale_dev = nullptr);
int launch_conv2d_f32_simt(cudaStream_t, const ConvGeom &, const float *, const float *, const float *, float *);
int launch_conv2d_f32_umma(cudaStream_t, const ConvGeom &, const float *, const float *, const float *, float *);
// half-precision parts, 16 or 32 input channels (umma_conv_half.cu): -1 when the shape is not its own
int launch_conv2d_f32_half(cudaStream_t, const ConvGeom &, const float *, const float *, const float *, float *);
int launch_qconv2d_simt(cudaStream_t, const ConvGeom &, const uint8_t *, const int8_t *, const float *, const int32_t *,
                        int x_zp, int y_zp, uint8_t *);
int launch_qconv2d_umma(cudaStream_t, const ConvGeom &, const uint8_t *, const int8_t *, const float *, const int32_t *,
                        int x_zp, int y_zp, uint8_t *);
// pooled-window kernel (umma_conv_pool.cu): -1 when the shape is not its own
int launch_qconv2d_umma_pooled(cudaStream_t, const ConvGeom &, const uint8_t *, const int8_t *, const float *, const int32_t *,
                               int x_zp, int y_zp, uint8_t *);
// fused chain of small Gemm layers on the tensor cores (umma_mlp.cu): -1 when the widths are not its own
int launch_mlp_f32_umma(cudaStream_t, const sofie_mlp_desc *, const float *, const float *const *, const float *const *, float *);
// first-layer kernels (conv_first.cu): -1 when the shape is not theirs
int launch_conv2d_f32_first(cudaStream_t, const ConvGeom &, const float *, const float *, const float *, float *);
// 3x3 of any layout and size on the CUDA cores (conv3x3_direct.cu): -1 when the shape is not its own
int launch_conv2d_f32_direct3x3(cudaStream_t, const ConvGeom &, const float *, const float *, const float *, float *);
int launch_qconv2d_first(cudaStream_t, const ConvGeom &, const uint8_t *, const int8_t *, const float *, const int32_t *,
                         int x_zp, int y_zp, uint8_t *);
// split-K skinny GEMM (splitk_gemm.cu)
bool splitk_shape_ok(const sofie_gemm_f32_desc &);
bool rowblock_shape_ok(const sofie_gemm_f32_desc &, const float *A, const float *B);
int launch_gemm_f32_rowblock(cudaStream_t, const sofie_gemm_f32_desc &, const float *, const float *, const float *, float *);
int launch_gemm_f32_splitk(cudaStream_t, const sofie_gemm_f32_desc &, const float *, const float *, const float *, float *,
                           float *scratch, size_t scratch_floats);
int launch_gemm_f32_splitk_auto(cudaStream_t, const sofie_gemm_f32_desc &, const float *, const float *, const float *,
                                float *);
// gives the split-K scratch buffer of a stream back to the per-device pool (context teardown)
void splitk_scratch_release(int device, cudaStream_t stream);
template <typename T>
int launch_pack_ohwi(cudaStream_t, const T *, T *, int Cout, int C, int kH, int kW);

} // namespace sofie
