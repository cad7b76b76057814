// The 32-bit attention kernels of attention_f32.cu as the dispatcher of attention_simt.cu calls
// them.
#pragma once
#include <cuda_runtime.h>

struct FbAttentionF32 {
  const float* q;
  long long q_stride;
  float* out;
  long long out_stride;
  const int* positions;
  const int* seq_of_token;
  const int* page_table;
  int max_pages, n_seqs;
  const float* k;
  const float* v;
  long long page_stride, head_stride;
  int ring_pages, window;
  int T, A, Kh, D;
  float scale;
};

bool fb_attention_f32_fits(const FbAttentionF32& p);
int fb_attention_f32_launch(const FbAttentionF32& p, cudaStream_t stream);
