// The 32-bit products of gemm_f32.cu as the dispatchers of gemm_simt.cu call them.
#pragma once
#include <cuda_runtime.h>

struct FbGemmF32 {
  const float* x;
  const float* w;
  float* out;
  int M, N, K;
  long long ldx, ldw, ldo;
  int count;  // products of the same sizes, their operands bx / bw / bo elements apart
  long long bx, bw, bo;
};

// Rows up to which the weights are streamed instead of tiled (32 rows, 2048 -> 16384: 80 us, tiles
// 134; 2048 -> 3072: 24 against 36; from there on the stream is read three times and more).
constexpr int FB_GEMM_F32_ROWS = 32;

bool fb_gemm_f32_fits(const FbGemmF32& p);
// gemm_f32_tcgen05.cu; FB_GEMM_F32_NOT_HERE: the kernel does not fit this build's registers or this
// device, and nothing was launched.
constexpr int FB_GEMM_F32_NOT_HERE = -1;
int fb_gemm_f32_tc_launch(const FbGemmF32& p, cudaStream_t stream);
int fb_gemm_f32_launch(const FbGemmF32& p, cudaStream_t stream);
