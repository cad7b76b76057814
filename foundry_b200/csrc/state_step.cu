// One token a sequence of the recurrences with a decay from its own projection, everything between
// the decays' product and the output's as one kernel: the decays, a step of the recurrence on the
// state, the norm of a head's output and the output gate.
//
// delta:  S <- diag(g) S;  u = sigmoid(beta) (v - S^T k);  S <- S + k u^T;  o = S^T q
// wkv:    o = (S + diag(b) k v^T)^T r;  S <- diag(g) S + k v^T
//         out = o / sqrt(mean(o^2) + eps) * w * act(gate)
// g: exp(-exp(A) softplus(x + bias)), exp(-exp(x + bias)) or x itself, a key channel or a head.
//
// A step is a pass over the state, read, changed and written once, but what bounds it is the chain
// of launches and of loads: the four kernels it takes the place of (decay_gate, scan, head_norm_gate
// in sequence_mix.cu) took 13 us for 8 sequences of 32 heads of 64 x 64 (8 MB); eight tokens through
// four such layers 4,565 -> 4,356 us. A block a
// (sequence, head); a thread owns four neighbouring columns of every R-th key row, and asks for them
// before it waits for the kernel in front. That is right because what wrote it (the last step's scan or
// step, or the zeros of a new sequence) let nobody start before its writes, and a kernel behind it that
// let its successor start had waited for it: every kernel that writes states either never calls
// fb_pdl_launch or calls it behind its writes. The same goes for the slots. Sums over the key rows meet in shared memory, in row order. All arithmetic is 32-bit.
#include "common.cuh"

namespace {

struct Step {
  const float* q; long long q_ld;   // [n, *]: query (delta) or receptance (wkv); head h at (h / rep) * dim
  const float* k; long long k_ld;   // keys, same head mapping
  const float* v; long long v_ld;   // values: head h at h * vdim
  const float* g; long long g_ld;   // decays: head h at h * dim, or at h (one a head)
  const float* A; const float* bias;  // of the decays: [H]; [H * dim] or [H]
  const float* beta; long long beta_ld;  // delta: raw step size a head
  const float* bonus;               // wkv: [H, dim]
  const float* gate; long long gate_ld;  // head h at h * vdim
  const float* norm; int norm_stride;    // of a head: at h * norm_stride
  float* state; long long state_stride, s_offset;
  void* out; long long out_ld;
  const int* cu_tokens; const int* slots;
  int H, rep, dim, vdim;
  int form;    // of the decays: 0 as they are, 1 with A, 2 without
  int a_head;  // one decay a head
  int act;     // of the gate: 0 sigmoid, 1 SiLU
  float eps;
};

__device__ __forceinline__ float sigmoid_of(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float softplus_of(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// NR: key rows a thread holds at most.
template <typename TO, bool DELTA, int THREADS, int NR>
__global__ void __launch_bounds__(THREADS) state_step_kernel(const Step a) {
  extern __shared__ __align__(16) float sm[];
  const int dim = a.dim, vdim = a.vdim, dim4 = (dim + 3) / 4 * 4;
  float* sq = sm;            // [dim] each: query, key, decay, bonus
  float* sk = sq + dim4;
  float* sg = sk + dim4;
  float* sb = sg + dim4;
  float* so = sb + dim4;     // [vdim]: v - S^T k, then the output
  float* part = so + vdim;   // [R][vdim]
  __shared__ float scratch[32];
  const int seq = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int groups = vdim / 4, R = THREADS / groups;
  const int c4 = tid % groups, r0 = tid / groups;
  float* S = a.state + (long long)a.slots[seq] * a.state_stride + a.s_offset + (long long)h * dim * vdim;
  float4 s[NR];
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int row = r0 + i * R;
    s[i] = row < dim ? __ldcg(reinterpret_cast<const float4*>(S + (size_t)row * vdim) + c4)
                     : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const float A = a.form == 1 ? expf(a.A[h]) : 0.f;
  fb_pdl_wait();
  const int t = a.cu_tokens[seq];
  const bool here = a.cu_tokens[seq + 1] > t;  // (a sequence without a token keeps its state)
  if (!here) return;
  const size_t at_k = (size_t)(h / a.rep) * dim;
  for (int i = tid; i < dim; i += THREADS) {
    sq[i] = __ldcg(a.q + (size_t)t * a.q_ld + at_k + i);
    sk[i] = __ldcg(a.k + (size_t)t * a.k_ld + at_k + i);
    const int c = a.a_head ? h : h * dim + i;
    float g = __ldcg(a.g + (size_t)t * a.g_ld + c);
    if (a.form == 1) g = expf(-A * softplus_of(g + a.bias[c]));
    if (a.form == 2) g = expf(-expf(g + a.bias[c]));
    sg[i] = g;
    if (!DELTA) sb[i] = a.bonus[(size_t)h * dim + i];
  }
  float mine = 0.f, gated = 0.f, weight = 0.f;  // of the thread's output column
  if (tid < vdim) {
    mine = __ldcg(a.v + (size_t)t * a.v_ld + (size_t)h * vdim + tid);
    gated = __ldcg(a.gate + (size_t)t * a.gate_ld + (size_t)h * vdim + tid);
    weight = a.norm[(size_t)h * a.norm_stride + tid];
    so[tid] = mine;
  }
  const float beta = DELTA ? sigmoid_of(__ldcg(a.beta + (size_t)t * a.beta_ld + h)) : 0.f;
  __syncthreads();

  // the rows' shares of a sum for the thread's columns, then column `tid`'s sum of them
  auto meet = [&](float4 share) {
    *reinterpret_cast<float4*>(part + (size_t)r0 * vdim + 4 * c4) = share;
    __syncthreads();
    float sum = 0.f;
    if (tid < vdim)
      for (int r = 0; r < R; ++r) sum += part[(size_t)r * vdim + tid];
    return sum;
  };
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  if (DELTA) {
    float4 kv = o;
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int row = r0 + i * R;
      if (row >= dim) break;
      const float g = sg[row], k = sk[row];
      s[i] = make_float4(g * s[i].x, g * s[i].y, g * s[i].z, g * s[i].w);
      kv = make_float4(fmaf(s[i].x, k, kv.x), fmaf(s[i].y, k, kv.y), fmaf(s[i].z, k, kv.z),
                       fmaf(s[i].w, k, kv.w));
    }
    const float sum = meet(kv);
    if (tid < vdim) so[tid] = beta * (mine - sum);
    __syncthreads();
    const float4 u = *reinterpret_cast<const float4*>(so + 4 * c4);
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int row = r0 + i * R;
      if (row >= dim) break;
      const float k = sk[row], q = sq[row];
      s[i] = make_float4(fmaf(k, u.x, s[i].x), fmaf(k, u.y, s[i].y), fmaf(k, u.z, s[i].z),
                         fmaf(k, u.w, s[i].w));
      o = make_float4(fmaf(s[i].x, q, o.x), fmaf(s[i].y, q, o.y), fmaf(s[i].z, q, o.z),
                      fmaf(s[i].w, q, o.w));
    }
  } else {
    const float4 v = *reinterpret_cast<const float4*>(so + 4 * c4);
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int row = r0 + i * R;
      if (row >= dim) break;
      const float g = sg[row], k = sk[row], q = sq[row], b = sb[row];
      const float4 kv = make_float4(k * v.x, k * v.y, k * v.z, k * v.w);
      o = make_float4(fmaf(q, fmaf(b, kv.x, s[i].x), o.x), fmaf(q, fmaf(b, kv.y, s[i].y), o.y),
                      fmaf(q, fmaf(b, kv.z, s[i].z), o.z), fmaf(q, fmaf(b, kv.w, s[i].w), o.w));
      s[i] = make_float4(fmaf(g, s[i].x, kv.x), fmaf(g, s[i].y, kv.y), fmaf(g, s[i].z, kv.z),
                         fmaf(g, s[i].w, kv.w));
    }
  }
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int row = r0 + i * R;
    if (row < dim) *(reinterpret_cast<float4*>(S + (size_t)row * vdim) + c4) = s[i];
  }
  const float out = meet(o);
  const float r = 1.0f / sqrtf(fb_block_sum(tid < vdim ? out * out : 0.f, scratch) / (float)vdim + a.eps);
  if (tid < vdim) {
    const float gate = a.act == 0 ? sigmoid_of(gated) : gated * sigmoid_of(gated);
    reinterpret_cast<TO*>(a.out)[(size_t)t * a.out_ld + (size_t)h * vdim + tid] =
        fb_from_float<TO>(out * r * weight * gate);
  }
}

template <typename TO, bool DELTA, int THREADS, int NR>
int launch_step(const Step& a, int n_seqs, cudaStream_t stream) {
  const int R = THREADS / (a.vdim / 4);
  const size_t smem = (size_t)(4 * ((a.dim + 3) / 4 * 4) + a.vdim + R * a.vdim) * 4;  // < 48 KB
  fb_launch(state_step_kernel<TO, DELTA, THREADS, NR>, dim3(n_seqs, a.H), dim3(THREADS), smem, stream, a);
  return fb_check_launch("state_step");
}
}  // namespace

// Whether the step takes heads of these sizes: four columns a thread, the columns a power of two of
// pieces that all are one block's, at most 8 rows a thread.
FB_API int fb_state_step_fits(int dim, int vdim) {
  const int groups = vdim / 4;
  return dim > 0 && dim <= 512 && vdim >= 8 && vdim <= 256 && (vdim & (vdim - 1)) == 0 &&
         (long long)dim * groups <= 512 * 8;
}

FB_API int fb_state_step(int delta, const float* q, long long q_ld, const float* k, long long k_ld,
                         const float* v, long long v_ld, const float* g, long long g_ld, const float* A,
                         const float* bias, int form, int a_head, const float* beta, long long beta_ld,
                         const float* bonus, const float* gate, long long gate_ld, int act,
                         const float* norm, int norm_stride, float* state, long long state_stride,
                         long long s_offset, void* out, long long out_ld, int out_dtype,
                         const int* cu_tokens, const int* slots, int n_seqs, int H, int rep, int dim,
                         int vdim, float eps, cudaStream_t stream) {
  FB_REQUIRE(n_seqs >= 0 && H > 0 && H <= 65535 && rep > 0, "state_step: bad sizes");
  FB_REQUIRE(fb_state_step_fits(dim, vdim), "state_step: heads of %d x %d do not fit", dim, vdim);
  FB_REQUIRE(((uintptr_t)state % 16) == 0 && state_stride % 4 == 0 && s_offset % 4 == 0,
             "state_step: the state is not on 16-byte boundaries");
  FB_REQUIRE(form >= 0 && form <= 2 && (form == 0 || bias) && (form != 1 || A),
             "state_step: the decays lack a parameter");
  FB_REQUIRE(delta ? beta != nullptr : bonus != nullptr, "state_step: an input is missing");
  if (n_seqs == 0) return 0;
  const Step a = {q, q_ld, k, k_ld, v, v_ld, g, g_ld, A, bias, beta, beta_ld, bonus, gate, gate_ld,
                  norm, norm_stride, state, state_stride, s_offset, out, out_ld, cu_tokens, slots,
                  H, rep, dim, vdim, form, a_head, act, eps};
  // (the block's width decides the order of sums: by the head's sizes alone)
  const int pieces = dim * (vdim / 4);
#define FB_STEP(TO, DELTA)                                                          \
  return pieces <= 256 * 4   ? launch_step<TO, DELTA, 256, 4>(a, n_seqs, stream)    \
         : pieces <= 512 * 4 ? launch_step<TO, DELTA, 512, 4>(a, n_seqs, stream)    \
                             : launch_step<TO, DELTA, 512, 8>(a, n_seqs, stream)
  if (delta) FB_DISPATCH_DTYPE(out_dtype, TO, FB_STEP(TO, true));
  FB_DISPATCH_DTYPE(out_dtype, TO, FB_STEP(TO, false));
#undef FB_STEP
}
