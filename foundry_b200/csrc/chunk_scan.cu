// The gated delta rule of sequence_mix.cu over prompts, 32 tokens at a time as small products:
//
//   S <- diag(g) S;  u = b (v - S^T k);  S <- S + k u^T;  o = S^T q
//
// With S0 the state in front of a chunk of C tokens and P(t, i) = prod_{j = i+1 .. t} g_j, which
// never exceeds one (all decays are products of decays, nothing is divided):
//
//   L[t, i] = sum_c k_t k_i P(t, i)   (i < t)       A[t, i] = sum_c q_t k_i P(t, i)   (i <= t)
//   u_t = b_t (v_t - (k_t P(t, -1)) . S0 - sum_{i<t} L[t, i] u_i)   =  U0_t - W_t . S0
//   o_t = (q_t P(t, -1)) . S0 + sum_{i<=t} A[t, i] u_i
//   S  <- diag(P(C-1, -1)) S0 + sum_i (k_i P(C-1, i)) u_i^T
//
// `prepare_kernel` makes W, U0, A and the decayed copies of q and k for every chunk of the prompt
// side by side; they do not depend on the state. `walk_kernel` goes through the chunks in order,
// 16 or 24 columns of a head's state a block, with the two products that the next chunk waits for,
// and leaves u and every chunk's S0; `output_kernel` makes all outputs from them side by side. The
// token-by-token scan has 32 dependent steps of two dot products each where a walk has one chunk:
// 0.35 us a step with heads of 64 x 64, 0.59 with 128 x 128 (latency: a few warps a scheduler in
// one chain). A step's heads that fill the SMs that way need no chunks (`ops.chunk_scan_unit`).
// All of it is 32-bit arithmetic on the FMA pipe, reordered.
//
// Measured: 2,048 tokens, 32 heads of 64 x 64: 199 us (89, 82 and 35), token by token 709. 1,500
// tokens, 24 heads of 128 x 128: 301 us (91, 155 and 55) against 892. Outputs made in the walk
// itself, from the same registers (blocks of 16 columns): 217 for 199 and 378 for 355 us. Error against 64 bits with a decay a channel:
// outputs 1.29e-7 and 1.37e-7, token by token 1.39e-7 and 1.40e-7; states 1.09e-7 and 1.00e-7 for
// 1.02e-7 and 0.99e-7 (a chunk's own sum, added to the decayed state last, left that as it was).
#include "common.cuh"

namespace {

constexpr int C = 32, SUB = 16;  // tokens a chunk; tokens whose decays are multiplied out pairwise
constexpr int MAX_VDIM = 128;

struct ChunkArgs {
  const float* q; long long q_ld;  // [T, *]: head h at (h / rep) * dim
  const float* k; long long k_ld;
  const float* v; long long v_ld;  // head h at h * vdim
  const float* g; long long g_ld;  // head h at h * dim, or one per head at h (g_scalar)
  const float* beta; long long beta_ld;  // raw step size a head (sigmoid applied here)
  float* state; long long state_stride; long long s_offset;
  float* out;  // [T, H * vdim]
  const int* cu_tokens; const int* slots;
  int n_seqs, H, rep, vdim, g_scalar;
  float* ws;
  int first_chunk, chunks;  // the part of the step's chunks that `ws` holds
};

// What one chunk of one head leaves in the workspace, in floats.
template <int D>
struct Unit {
  static constexpr int W = 0, Q = C * D, K = 2 * C * D, A = 3 * C * D, G = A + C * C, U = G + D;
  __host__ __device__ static long long state(int vdim) { return U + (long long)C * vdim; }  // S0
  __host__ __device__ static long long size(int vdim) { return state(vdim) + (long long)D * vdim; }
};

__device__ __forceinline__ float4 ldcg4(const float* p) {
  return __ldcg(reinterpret_cast<const float4*>(p));
}
__device__ __forceinline__ void copy16(float* dst, const float* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ float sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }

// The sequence of the step's chunk number `chunk`, and how many chunks lie in front of the
// sequence; every lane of a warp calls it and gets both (-1: there is no such chunk).
__device__ __forceinline__ int find_chunk(const int* cu, int n_seqs, int chunk, int& before) {
  const int lane = threadIdx.x & 31;
  int base = 0;
  for (int s0 = 0; s0 < n_seqs; s0 += 32) {
    const int s = s0 + lane;
    const int own = s < n_seqs ? (cu[s + 1] - cu[s] + C - 1) / C : 0;
    int sum = own;  // inclusive
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const int x = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += x;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, chunk < base + sum);
    if (hit) {
      const int l = __ffs(hit) - 1;
      before = base + __shfl_sync(0xffffffffu, sum - own, l);
      return s0 + l;
    }
    base += __shfl_sync(0xffffffffu, sum, 31);
  }
  return -1;
}

// ------------------------------------------------------------------ what needs no state
// Bound by instruction issue: per chunk and head 16 rounds of the pairwise decays (a multiply and
// two FMAs a channel and pair), one 16 x 16 block of plain dot products, and the substitution, a
// column of [W | U0] a thread.
constexpr int PREP_THREADS = 256;

template <int D>
struct Prep {
  static constexpr int P = D + 4;
  static constexpr int FLOATS = 3 * C * P + 3 * SUB * P + 2 * C * (C + 4) + C;
};

template <int D>
__global__ void __launch_bounds__(PREP_THREADS, 2) prepare_kernel(ChunkArgs a) {
  constexpr int P = Prep<D>::P, PL = C + 4;
  extern __shared__ __align__(16) float smem[];
  float(*K)[P] = reinterpret_cast<float(*)[P]>(smem);
  float(*Q)[P] = K + C;
  float(*G)[P] = Q + C;
  float(*QG)[P] = G + C;     // q of the second half, decayed since the half's start
  float(*KG)[P] = QG + SUB;  // k of the second half, likewise
  float(*KD)[P] = KG + SUB;  // k of the first half, decayed to the half's end
  float(*L)[PL] = reinterpret_cast<float(*)[PL]>(smem + 3 * C * P + 3 * SUB * P);
  float(*A)[PL] = L + C;
  float* step = smem + 3 * C * P + 3 * SUB * P + 2 * C * PL;
  fb_pdl_wait();
  const int tid = threadIdx.x, h = blockIdx.y;
  int before = 0;
  const int seq = find_chunk(a.cu_tokens, a.n_seqs, a.first_chunk + blockIdx.x, before);
  if (seq < 0) return;
  const int first = a.cu_tokens[seq], local = a.first_chunk + blockIdx.x - before;
  const int start = first + local * C, n = min(C, a.cu_tokens[seq + 1] - start);
  float* ws = a.ws + ((long long)blockIdx.x * a.H + h) * Unit<D>::size(a.vdim);

  // rows beyond the sequence's end: no key, no query, no decay
  for (int i = tid; i < C * (D / 4); i += PREP_THREADS) {
    const int t = i / (D / 4), c = i % (D / 4) * 4;
    const long long row = start + t, at = (long long)(h / a.rep) * D + c;
    const bool in = t < n;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(&K[t][c]) = in ? ldcg4(a.k + row * a.k_ld + at) : zero;
    *reinterpret_cast<float4*>(&Q[t][c]) = in ? ldcg4(a.q + row * a.q_ld + at) : zero;
    float4 g = make_float4(1.f, 1.f, 1.f, 1.f);
    if (in && a.g_scalar) {
      g.x = __ldcg(a.g + row * a.g_ld + h);
      g.y = g.z = g.w = g.x;
    } else if (in) {
      g = ldcg4(a.g + row * a.g_ld + (long long)h * D + c);
    }
    *reinterpret_cast<float4*>(&G[t][c]) = g;
  }
  if (tid < C) {
    step[tid] = tid < n ? sigmoid(__ldcg(a.beta + (long long)(start + tid) * a.beta_ld + h)) : 0.f;
  }
  for (int i = tid; i < 2 * C * PL; i += PREP_THREADS) (&L[0][0])[i] = 0.f;  // L and A
  __syncthreads();

  // decays along the tokens, a channel a thread: forward for q (and k), backward for k
  for (int i = tid; i < 2 * D; i += PREP_THREADS) {
    const int c = i % D;
    if (i < D) {
      float all = 1.f, half = 1.f;
#pragma unroll
      for (int t = 0; t < C; ++t) {
        if (t == SUB) half = 1.f;
        all *= G[t][c];
        half *= G[t][c];
        ws[Unit<D>::Q + t * D + c] = Q[t][c] * all;
        if (t >= SUB) {
          QG[t - SUB][c] = Q[t][c] * half;
          KG[t - SUB][c] = K[t][c] * half;
        }
      }
      ws[Unit<D>::G + c] = all;
    } else {
      float all = 1.f, half = 1.f;
#pragma unroll
      for (int t = C - 1; t >= 0; --t) {
        if (t == SUB - 1) half = 1.f;
        ws[Unit<D>::K + t * D + c] = K[t][c] * all;
        if (t < SUB) KD[t][c] = K[t][c] * half;
        all *= G[t][c];
        half *= G[t][c];
      }
    }
  }
  // pairs within a half: eight threads a key, which decays as the tokens pass
  {
    const int group = tid / 8, part = tid % 8, s0 = group / SUB * SUB, i = group % SUB;
    float x[D / 8];
#pragma unroll
    for (int e = 0; e < D / 8; ++e) x[e] = 0.f;
#pragma unroll 2
    for (int t = 0; t < SUB; ++t) {
      float sa[4] = {}, sl[4] = {};
#pragma unroll
      for (int e = 0; e < D / 8; e += 4) {
        const int c = part * 4 + e * 8;
        const float4 q = *reinterpret_cast<const float4*>(&Q[s0 + t][c]);
        const float4 k = *reinterpret_cast<const float4*>(&K[s0 + t][c]);
        const float4 g = *reinterpret_cast<const float4*>(&G[s0 + t][c]);
        const float qq[4] = {q.x, q.y, q.z, q.w}, kk[4] = {k.x, k.y, k.z, k.w},
                    gg[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
        for (int b = 0; b < 4; ++b) {  // (x is zero in front of its own token)
          x[e + b] = t == i ? kk[b] : x[e + b] * gg[b];
          sa[b] = fmaf(qq[b], x[e + b], sa[b]);
          sl[b] = fmaf(kk[b], x[e + b], sl[b]);
        }
      }
      float pa = (sa[0] + sa[1]) + (sa[2] + sa[3]), pl = (sl[0] + sl[1]) + (sl[2] + sl[3]);
#pragma unroll
      for (int o = 1; o < 8; o *= 2) {
        pa += __shfl_xor_sync(0xffffffffu, pa, o);
        pl += __shfl_xor_sync(0xffffffffu, pl, o);
      }
      if (part == 0 && t >= i) {
        A[s0 + t][s0 + i] = pa;
        if (t > i) L[s0 + t][s0 + i] = pl;
      }
    }
  }
  __syncthreads();
  // the second half's tokens with the first half's keys
  {
    const int i = tid % SUB, t = tid / SUB;
    float4 sa = make_float4(0.f, 0.f, 0.f, 0.f), sl = sa;
#pragma unroll 8
    for (int c = 0; c < D; c += 4) {
      const float4 q = *reinterpret_cast<const float4*>(&QG[t][c]);
      const float4 k = *reinterpret_cast<const float4*>(&KD[i][c]);
      sa.x = fmaf(q.x, k.x, sa.x); sa.y = fmaf(q.y, k.y, sa.y);
      sa.z = fmaf(q.z, k.z, sa.z); sa.w = fmaf(q.w, k.w, sa.w);
      const float4 y = *reinterpret_cast<const float4*>(&KG[t][c]);
      sl.x = fmaf(y.x, k.x, sl.x); sl.y = fmaf(y.y, k.y, sl.y);
      sl.z = fmaf(y.z, k.z, sl.z); sl.w = fmaf(y.w, k.w, sl.w);
    }
    A[SUB + t][i] = (sa.x + sa.y) + (sa.z + sa.w);
    L[SUB + t][i] = (sl.x + sl.y) + (sl.z + sl.w);
  }
  __syncthreads();
  for (int i = tid; i < C * C; i += PREP_THREADS) ws[Unit<D>::A + i] = A[i / C][i % C];
  for (int col = tid; col < D + a.vdim; col += PREP_THREADS) {
    float x[C];
    if (col < D) {
      float all = 1.f;
#pragma unroll
      for (int t = 0; t < C; ++t) {
        all *= G[t][col];
        x[t] = K[t][col] * all;
      }
    } else {
      const float* v = a.v + (long long)start * a.v_ld + (long long)h * a.vdim + (col - D);
#pragma unroll
      for (int t = 0; t < C; ++t) x[t] = t < n ? __ldcg(v + t * a.v_ld) : 0.f;
    }
#pragma unroll
    for (int t = 0; t < C; ++t) {
      float sum[4] = {};
#pragma unroll
      for (int i = 0; i < t; i += 4) {
        const float4 l = *reinterpret_cast<const float4*>(&L[t][i]);
        sum[0] = fmaf(l.x, x[i], sum[0]);
        if (i + 1 < t) sum[1] = fmaf(l.y, x[i + 1], sum[1]);
        if (i + 2 < t) sum[2] = fmaf(l.z, x[i + 2], sum[2]);
        if (i + 3 < t) sum[3] = fmaf(l.w, x[i + 3], sum[3]);
      }
      x[t] = step[t] * (x[t] - ((sum[0] + sum[1]) + (sum[2] + sum[3])));
    }
    if (col < D) {
#pragma unroll
      for (int t = 0; t < C; ++t) ws[Unit<D>::W + t * D + col] = x[t];
    } else {
#pragma unroll
      for (int t = 0; t < C; ++t) ws[Unit<D>::U + t * a.vdim + col - D] = x[t];
    }
  }
}

// ------------------------------------------------------------------------ chunk after chunk
// Bound by shared-memory reads and their latency, a chunk at a time (two warps a scheduler), so
// the block does only what the next chunk waits for: u = U0 - W . S0, a thread two tokens by two
// columns and half the channels; then the state, a thread one channel by 4 or 8 columns in
// registers. Two neighbouring terms of a sum share an instruction (fma.rn.f32x2). The next
// chunk's matrices arrive by asynchronous copies while this one is multiplied.
// COLS: columns of the state a block owns, 16 threads each; the last block of a head may have fewer.
// The walk takes as long as its slowest SM: 24 heads of 128 x 128 are 192 blocks of 16 columns, two of
// them on 44 SMs, or 144 of 24, one an SM: 1,500 tokens 155 us, 207 with 16. (1,000 tokens, 40 heads
// of 64 x 64, all three kernels: 151 us, 170 with 16.)

typedef unsigned long long f32x2;
__device__ __forceinline__ void fma2(f32x2& d, f32x2 x, f32x2 y) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(x), "l"(y));
}
__device__ __forceinline__ f32x2 mul2(f32x2 x, f32x2 y) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
  return d;
}
__device__ __forceinline__ f32x2 pack2(float x, float y) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ float sum2(f32x2 v) {
  const float2 f = unpack2(v);
  return f.x + f.y;
}
__device__ __forceinline__ ulonglong2 lds2(const float* p) {
  return *reinterpret_cast<const ulonglong2*>(p);
}

template <int D, int COLS>
struct Walk {
  static constexpr int P = D + 4, PU = COLS + 4;
  static constexpr int W = 0, K = W + C * P, U = K + C * D, G = U + C * PU, BUFFER = G + D;
  static constexpr int S = 2 * BUFFER, US = S + COLS * P, FLOATS = US + C * PU;  // S by columns
};

template <int D, int COLS>
__global__ void __launch_bounds__(16 * COLS, COLS > 16 ? 1 : 2) walk_kernel(ChunkArgs a) {
  constexpr int WALK_THREADS = 16 * COLS;
  using B = Walk<D, COLS>;
  constexpr int P = B::P, PU = B::PU;
  extern __shared__ __align__(16) float smem[];
  float(*S)[P] = reinterpret_cast<float(*)[P]>(smem + B::S);
  float(*Us)[PU] = reinterpret_cast<float(*)[PU]>(smem + B::US);
  fb_pdl_wait();
  const int tid = threadIdx.x, seq = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * COLS;
  const int tokens = a.cu_tokens[seq + 1] - a.cu_tokens[seq];
  if (tokens <= 0) return;
  // the chunks in front of this sequence's
  int before = 0;
  for (int s0 = 0; s0 < seq; s0 += 32) {
    const int s = s0 + (tid & 31);
    int x = s < seq ? (a.cu_tokens[s + 1] - a.cu_tokens[s] + C - 1) / C : 0;
#pragma unroll
    for (int o = 16; o > 0; o /= 2) x += __shfl_xor_sync(0xffffffffu, x, o);
    before += x;
  }
  const int from = max(a.first_chunk - before, 0);
  const int to = min(a.first_chunk + a.chunks - before, (tokens + C - 1) / C);
  if (from >= to) return;
  const long long unit = (long long)a.H * Unit<D>::size(a.vdim);
  float* ws = a.ws + (long long)(before + from - a.first_chunk) * unit +
              (long long)h * Unit<D>::size(a.vdim);

  auto fetch = [&](int b, const float* u) {
    float* dst = smem + b * B::BUFFER;
#pragma unroll
    for (int i = tid; i < C * (D / 4); i += WALK_THREADS) {
      const int t = i / (D / 4), c = i % (D / 4) * 4;
      copy16(dst + B::W + t * P + c, u + Unit<D>::W + t * D + c);
      copy16(dst + B::K + i * 4, u + Unit<D>::K + i * 4);
    }
    if (tid < C * COLS / 4) {
      const int t = tid / (COLS / 4), c = tid % (COLS / 4) * 4;
      if (col0 + c < a.vdim)
        copy16(dst + B::U + t * PU + c, u + Unit<D>::U + (long long)t * a.vdim + col0 + c);
    } else if (tid - C * COLS / 4 < D / 4) {
      const int c = (tid - C * COLS / 4) * 4;
      copy16(dst + B::G + c, u + Unit<D>::G + c);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  static_assert(C * COLS / 4 + D / 4 <= WALK_THREADS, "one piece each");

  constexpr int OWN = D * COLS / WALK_THREADS;  // columns of a channel that a thread holds
  const int ch = tid % D, own0 = tid / D * OWN;
  const long long mine = (long long)ch * a.vdim + col0 + own0;  // its place in a head's state
  const bool inside = col0 + own0 < a.vdim;  // (whole runs of columns: a.vdim is a multiple of 16)
  float* state = a.state + (long long)a.slots[seq] * a.state_stride + a.s_offset +
                 (long long)h * D * a.vdim + mine;
  f32x2 s[OWN / 2];
  fetch(0, ws);
#pragma unroll
  for (int j = 0; j < OWN; j += 4) {
    const float4 x = inside ? ldcg4(state + j) : make_float4(0.f, 0.f, 0.f, 0.f);
    s[j / 2] = pack2(x.x, x.y);
    s[j / 2 + 1] = pack2(x.z, x.w);
    S[own0 + j][ch] = x.x; S[own0 + j + 1][ch] = x.y;
    S[own0 + j + 2][ch] = x.z; S[own0 + j + 3][ch] = x.w;
  }
  auto put_state = [&](float* to_) {
    if (!inside) return;
#pragma unroll
    for (int j = 0; j < OWN; j += 4) {
      const float2 x = unpack2(s[j / 2]), y = unpack2(s[j / 2 + 1]);
      *reinterpret_cast<float4*>(to_ + j) = make_float4(x.x, x.y, y.x, y.y);
    }
  };
  // in the first product: tokens t0 and t0 + 4, columns j0 and j0 + 4, half the channels. (The
  // second half starts 16 channels on, so that the halves' reads lie in other banks.)
  const int lane = tid & 31, warp = tid >> 5, half = lane / 16;
  constexpr int CW = COLS / 8;  // warps side by side over the columns, four over the tokens
  const int t0 = warp / CW * 8 + lane / 4 % 4, j0 = warp % CW * 8 + lane % 4;
  for (int c0 = from; c0 < to; ++c0, ws += unit) {
    const int b = (c0 - from) & 1;
    const float* buf = smem + b * B::BUFFER;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the copies are in, the state is whole, the other buffer is free
    if (c0 + 1 < to) fetch(b ^ 1, ws + unit);
    put_state(ws + Unit<D>::state(a.vdim) + mine);
    f32x2 w[2][2][2] = {};  // [token][column][pairs of channels apart]
#pragma unroll 8
    for (int cc = 0; cc < D / 2; cc += 4) {
      const int c = half ? D / 2 + (cc + 16) % (D / 2) : cc;
      const ulonglong2 x0 = lds2(&S[j0][c]), x1 = lds2(&S[j0 + 4][c]);
      const ulonglong2 y0 = lds2(buf + B::W + t0 * P + c), y1 = lds2(buf + B::W + (t0 + 4) * P + c);
      fma2(w[0][0][0], y0.x, x0.x); fma2(w[0][0][1], y0.y, x0.y);
      fma2(w[0][1][0], y0.x, x1.x); fma2(w[0][1][1], y0.y, x1.y);
      fma2(w[1][0][0], y1.x, x0.x); fma2(w[1][0][1], y1.y, x0.y);
      fma2(w[1][1][0], y1.x, x1.x); fma2(w[1][1][1], y1.y, x1.y);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float v[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        v[r] = sum2(w[r][j][0]) + sum2(w[r][j][1]);
        v[r] += __shfl_xor_sync(0xffffffffu, v[r], 16);
      }
      const int t = t0 + 4 * half, col = j0 + 4 * j;  // either half finishes one token
      Us[t][col] = buf[B::U + t * PU + col] - (half ? v[1] : v[0]);
    }
    __syncthreads();  // u is whole; the state and W have been read
    {
      const int t = tid / (COLS / 2), col = tid % (COLS / 2) * 2;
      if (col0 + col < a.vdim)
        *reinterpret_cast<float2*>(ws + Unit<D>::U + (long long)t * a.vdim + col0 + col) =
            *reinterpret_cast<const float2*>(&Us[t][col]);
    }
    const f32x2 decay = pack2(buf[B::G + ch], buf[B::G + ch]);
#pragma unroll
    for (int j = 0; j < OWN / 2; ++j) s[j] = mul2(s[j], decay);
#pragma unroll
    for (int i = 0; i < C; ++i) {
      const float k = buf[B::K + i * D + ch];
      const f32x2 kk = pack2(k, k);
#pragma unroll
      for (int j = 0; j < OWN; j += 4) {
        const ulonglong2 u = lds2(&Us[i][own0 + j]);
        fma2(s[j / 2], kk, u.x);
        fma2(s[j / 2 + 1], kk, u.y);
      }
    }
#pragma unroll
    for (int j = 0; j < OWN; j += 2) {
      const float2 x = unpack2(s[j / 2]);
      S[own0 + j][ch] = x.x;
      S[own0 + j + 1][ch] = x.y;
    }
  }
  put_state(state);
}

// ----------------------------------------------------------------------------- the outputs
// [q decayed | A] times [S0 over u], a chunk of a head a block, a thread 4 tokens by 4 columns.
constexpr int OUT_GROUPS = 8;  // threads with the same columns

template <int D>
__global__ void __launch_bounds__(OUT_GROUPS * 32, 2) output_kernel(ChunkArgs a) {
  constexpr int P = D + 4, PA = C + 4;
  extern __shared__ __align__(16) float smem[];
  fb_pdl_wait();
  const int tid = threadIdx.x, h = blockIdx.y, E = a.vdim, PE = E + 4, threads = blockDim.x;
  float* Q = smem;
  float* A = Q + C * P;
  float* S = A + C * PA;
  float* U = S + D * PE;
  int before = 0;
  const int seq = find_chunk(a.cu_tokens, a.n_seqs, a.first_chunk + blockIdx.x, before);
  if (seq < 0) return;
  const int start = a.cu_tokens[seq] + (a.first_chunk + blockIdx.x - before) * C;
  const int n = min(C, a.cu_tokens[seq + 1] - start);
  const float* ws = a.ws + ((long long)blockIdx.x * a.H + h) * Unit<D>::size(E);
  const float* s0 = ws + Unit<D>::state(E);
  for (int i = tid; i < C * (D / 4); i += threads)
    copy16(Q + i / (D / 4) * P + i % (D / 4) * 4, ws + Unit<D>::Q + i * 4);
  for (int i = tid; i < C * C / 4; i += threads)
    copy16(A + i / (C / 4) * PA + i % (C / 4) * 4, ws + Unit<D>::A + i * 4);
  for (int i = tid; i < D * (E / 4); i += threads) {
    const int c = i / (E / 4), j = i - c * (E / 4);
    copy16(S + c * PE + j * 4, s0 + i * 4);
  }
  for (int i = tid; i < C * (E / 4); i += threads) {
    const int t = i / (E / 4), j = i - t * (E / 4);
    copy16(U + t * PE + j * 4, ws + Unit<D>::U + i * 4);
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int col = tid % (E / 4) * 4, t0 = tid / (E / 4);  // tokens t0, t0 + 8, ...
  f32x2 o[4][4][2] = {};  // [token][terms four apart][pair of columns]: short sums
  auto add = [&](f32x2 (&to_)[2], float x, const ulonglong2& y) {
    const f32x2 xx = pack2(x, x);
    fma2(to_[0], xx, y.x);
    fma2(to_[1], xx, y.y);
  };
#pragma unroll 4
  for (int c = 0; c < D; c += 4) {
    ulonglong2 y[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) y[e] = lds2(S + (c + e) * PE + col);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float4 x = *reinterpret_cast<const float4*>(Q + (t0 + OUT_GROUPS * r) * P + c);
      add(o[r][0], x.x, y[0]);
      add(o[r][1], x.y, y[1]);
      add(o[r][2], x.z, y[2]);
      add(o[r][3], x.w, y[3]);
    }
  }
#pragma unroll
  for (int i = 0; i < C; i += 4) {
    ulonglong2 u[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) u[e] = lds2(U + (i + e) * PE + col);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int t = t0 + OUT_GROUPS * r;
      if (i > t) continue;  // (a later token's u must not count even times zero)
      const float4 x = *reinterpret_cast<const float4*>(A + t * PA + i);
      add(o[r][0], x.x, u[0]);
      if (i + 1 <= t) add(o[r][1], x.y, u[1]);
      if (i + 2 <= t) add(o[r][2], x.z, u[2]);
      if (i + 3 <= t) add(o[r][3], x.w, u[3]);
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int t = t0 + OUT_GROUPS * r;
    if (t >= n) continue;
    float y[4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float2 p0 = unpack2(o[r][0][j]), p1 = unpack2(o[r][1][j]);
      const float2 p2 = unpack2(o[r][2][j]), p3 = unpack2(o[r][3][j]);
      y[2 * j] = (p0.x + p1.x) + (p2.x + p3.x);
      y[2 * j + 1] = (p0.y + p1.y) + (p2.y + p3.y);
    }
    *reinterpret_cast<float4*>(a.out + (long long)(start + t) * a.H * E + (long long)h * E + col) =
        make_float4(y[0], y[1], y[2], y[3]);
  }
}

template <int D>
int run(ChunkArgs a, int total, cudaStream_t stream) {
  constexpr int prep = Prep<D>::FLOATS * 4;
  constexpr int most = (C * (D + 4) + C * (C + 4) + (D + C) * (MAX_VDIM + 4)) * 4;
  const int outs = (C * (D + 4) + C * (C + 4) + (D + C) * (a.vdim + 4)) * 4;
  static bool seen[64] = {};
  const auto room_for = [](const void* kernel, int bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) ==
           cudaSuccess;
  };
  if (fb_first_use_on_device(seen) &&
      !(room_for((const void*)prepare_kernel<D>, prep) &&
        room_for((const void*)walk_kernel<D, 16>, Walk<D, 16>::FLOATS * 4) &&
        room_for((const void*)walk_kernel<D, 24>, Walk<D, 24>::FLOATS * 4) &&
        room_for((const void*)output_kernel<D>, most)))
    return fb_fail(2, "chunk_scan: cannot set %d bytes of shared memory", most);
  const int room = a.chunks;
  const long long heads = (long long)a.n_seqs * a.H;
  // 24 columns only where 16 would put two blocks on some SMs and 24 puts at most one on each: with
  // more blocks than that, two a SM hide each other's waits (2 sequences of 750: 315 us both ways)
  const bool wide = heads * (a.vdim / 16) > sm_count() && heads * ((a.vdim + 23) / 24) <= sm_count();
  for (a.first_chunk = 0; a.first_chunk < total; a.first_chunk += room) {
    a.chunks = total - a.first_chunk < room ? total - a.first_chunk : room;
    fb_launch(prepare_kernel<D>, dim3(a.chunks, a.H), dim3(PREP_THREADS), (size_t)prep, stream, a);
    if (wide)
      fb_launch(walk_kernel<D, 24>, dim3(a.n_seqs, a.H, (a.vdim + 23) / 24), dim3(16 * 24),
                (size_t)Walk<D, 24>::FLOATS * 4, stream, a);
    else
      fb_launch(walk_kernel<D, 16>, dim3(a.n_seqs, a.H, a.vdim / 16), dim3(16 * 16),
                (size_t)Walk<D, 16>::FLOATS * 4, stream, a);
    fb_launch(output_kernel<D>, dim3(a.chunks, a.H), dim3(OUT_GROUPS * a.vdim / 4), (size_t)outs,
              stream, a);
  }
  return fb_check_launch("chunk_scan");
}
}  // namespace

// Floats of workspace that one chunk of 32 tokens takes over all heads (0: sizes that the chunked
// kernels are not built for).
FB_API int fb_chunk_scan_unit(int H, int dim, int vdim) {
  if (vdim <= 0 || vdim % 16 != 0 || vdim > MAX_VDIM || H > 4096) return 0;
  if (dim == 64) return (int)(H * Unit<64>::size(vdim));
  if (dim == 128) return (int)(H * Unit<128>::size(vdim));
  return 0;
}

// The delta rule's arguments of fb_state_scan; `total`: no fewer chunks than the step's sequences
// have together; `room`: chunks that `ws` holds (the step is worked in as many parts as that takes).
FB_API int fb_chunk_scan(const float* q, long long q_ld, const float* k, long long k_ld,
                         const float* v, long long v_ld, const float* g, long long g_ld,
                         const float* beta, long long beta_ld, float* state,
                         long long state_stride, long long s_offset, float* out,
                         const int* cu_tokens, const int* slots, int n_seqs, int H, int rep,
                         int dim, int vdim, int g_scalar, float* ws, int total, int room,
                         cudaStream_t stream) {
  FB_REQUIRE(H > 0 && rep > 0 && H % rep == 0 && n_seqs >= 0 && room > 0 && beta != nullptr,
             "chunk_scan: bad arguments");
  FB_REQUIRE(fb_chunk_scan_unit(H, dim, vdim) > 0, "chunk_scan: heads of %d x %d", dim, vdim);
  const auto whole = [](const float* p, long long ld) {
    return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 4 == 0;
  };
  FB_REQUIRE(whole(q, q_ld) && whole(k, k_ld) && (g_scalar || whole(g, g_ld)) &&
                 whole(state + s_offset, state_stride) && whole(ws, 0) && whole(out, 0),
             "chunk_scan: rows that are no whole 16-byte pieces");
  if (n_seqs == 0 || total <= 0) return 0;
  const ChunkArgs a = {q, q_ld, k, k_ld, v, v_ld, g, g_ld, beta, beta_ld, state, state_stride,
                       s_offset, out, cu_tokens, slots, n_seqs, H, rep, vdim, g_scalar, ws, 0,
                       room < total ? room : total};
  return dim == 64 ? run<64>(a, total, stream) : run<128>(a, total, stream);
}
