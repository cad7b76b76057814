// out[M,N] = x[M,K] * w[N,K]^T in 32 bits on the CUDA cores (IEEE FFMA), for operands that 16-byte
// loads can address; large products of more than 32 rows are gemm_f32_tcgen05.cu's.
//
// few rows (single-token steps): the weights stream once, and that stream is the bound.
//   `rows_kernel`: 8 rows of 2048 -> 16384 in 31 us (134 MB, 4.3 TB/s), one row in 22 us
//   (6.1 TB/s); the 64 x 64 tiles of gemm_simt.cu took 208 us, a block walking all of K alone.
// many rows (prompts): register tiles, bound by the FMA pipe and the shared-memory reads beside
//   it (46 of 74 TFLOP/s). `tile_kernel`. Two FMAs to an instruction (fma.rn.f32x2) measured
//   10 % slower here: the pipe gives 128 a clock either way and the pairs cost moves.
//
// Where K is shared among warps or blocks the parts are summed in a fixed order; the error against
// 64 bits falls with the length of a part (K = 2048: 8.1e-7 in one run, 2.9e-7 in eight, 1.2e-7
// over a warp's lanes).
//
// Sizes and views that 16-byte loads do not fit (K or a stride that is no multiple of 4 elements,
// a base that is not 16-byte aligned), and bfloat16, stay on gemm_simt.cu.
#include "common.cuh"
#include "gemm_f32.h"

namespace {

__device__ __forceinline__ void cp_async16(unsigned dst, const void* src, int bytes) {
  // copies `bytes` (0 or 16) and fills the rest of the 16 with zeros; goes through L2 only
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ float4 ld_stream(const float* p) {
  // weights: constant, read once
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p));
  return v;
}

// ------------------------------------------------------------------------ few rows
// A warp owns 4 weight rows and a 128-wide slice of every K block; a lane takes 4 neighbouring
// k of each row, so a warp's load of a row is 512 contiguous bytes. x is staged in shared memory
// a chunk of K at a time for all warps of the block (a lane's 16 bytes of a token serve its 4
// weight rows). WK warps share the K of the same rows, the others own other rows; a result is
// the sum over lanes by halving exchanges, then over the WK warps in order, whatever M is.
constexpr int ROWS_WARPS = 8, ROWS_R = 4;
// K that is staged at a time (one warp a row group: no more than there is, see launch_rows_by_shape)
template <int WK>
constexpr int ROWS_CHUNK = WK == 1 ? 128 : 512;

template <int MR, int WK>
__global__ void __launch_bounds__(ROWS_WARPS * 32, 2)
rows_kernel(const float* x /* written by the kernel before: no read-only promise */,
            const float* __restrict__ w, float* out, int M, int N, int K, long long ldx,
            long long ldw, long long ldo) {
  constexpr int WR = ROWS_WARPS / WK, KB = 128 * WK, CH = ROWS_CHUNK<WK>, IT = CH / KB;
  constexpr int V = MR * ROWS_R;
  extern __shared__ __align__(16) float smem[];  // [2][MR][CH]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wk = warp % WK, wr = warp / WK;
  const int n0 = (blockIdx.x * WR + wr) * ROWS_R;
  const int m0 = blockIdx.y * MR;
  const float* wrow[ROWS_R];
#pragma unroll
  for (int r = 0; r < ROWS_R; ++r) wrow[r] = w + (long long)min(n0 + r, N - 1) * ldw;
  const int chunks = (K + CH - 1) / CH, T = chunks * IT;
  const int k_first = wk * 128 + lane * 4;

  auto fetch = [&](float4 (&to)[ROWS_R], int t) {
    const int k = k_first + t * KB;
#pragma unroll
    for (int r = 0; r < ROWS_R; ++r)
      to[r] = k < K ? ld_stream(wrow[r] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  auto stage = [&](int c) {
    const unsigned base =
        (unsigned)__cvta_generic_to_shared(smem) + (unsigned)((c & 1) * MR * CH * 4);
#pragma unroll
    for (int i = tid; i < MR * CH / 4; i += ROWS_WARPS * 32) {
      const int m = i / (CH / 4), kk = (i % (CH / 4)) * 4, k = c * CH + kk;
      const bool have = m0 + m < M && k < K;
      cp_async16(base + (unsigned)(m * CH + kk) * 4u,
                 x + (have ? (long long)(m0 + m) * ldx + k : 0), have ? 16 : 0);
    }
    cp_commit();
  };

  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.f;
  float4 wa[ROWS_R], wb[ROWS_R];
  fetch(wa, 0);
  fetch(wb, 1);
  fb_pdl_wait();
  stage(0);

  auto multiply = [&](const float4 (&ww)[ROWS_R], int t) {
    if (t % IT == 0) {  // a new chunk: its copies are in, and the other buffer is free
      const int c = t / IT;
      cp_wait<0>();
      __syncthreads();
      if (c + 1 < chunks) stage(c + 1);
    }
    const float* xs = smem + ((t / IT) & 1) * MR * CH + (t % IT) * KB + k_first;
#pragma unroll
    for (int m = 0; m < MR; ++m) {
      const float4 a = *reinterpret_cast<const float4*>(xs + m * CH);
#pragma unroll
      for (int r = 0; r < ROWS_R; ++r) {
        float s = acc[m * ROWS_R + r];
        s = fmaf(a.x, ww[r].x, s);
        s = fmaf(a.y, ww[r].y, s);
        s = fmaf(a.z, ww[r].z, s);
        acc[m * ROWS_R + r] = fmaf(a.w, ww[r].w, s);
      }
    }
  };
  for (int t = 0; t < T; t += 2) {
    multiply(wa, t);
    fetch(wa, t + 2);  // beyond K: zeros without a load
    if (t + 1 < T) {
      multiply(wb, t + 1);
      fetch(wb, t + 3);
    }
  }
  fb_pdl_launch();

  // lanes trade halves of their V sums until each holds V / 32 whole ones (or lanes hold copies)
  int index = 0;
  {
    int held = V;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      if (held > 1) {
        const int half = held / 2;
        const bool upper = lane & o;
#pragma unroll
        for (int i = 0; i < V / 2; ++i)
          if (i < half) {
            const float give = upper ? acc[i] : acc[i + half];
            const float keep = upper ? acc[i + half] : acc[i];
            acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
          }
        index += upper ? half : 0;
        held = half;
      } else {
        acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
      }
    }
  }
  constexpr int HELD = V >= 32 ? V / 32 : 1;
  __syncthreads();  // the staged x is no longer read
  float* red = smem + warp * V;
#pragma unroll
  for (int i = 0; i < HELD; ++i) red[index + i] = acc[i];  // copies write the same number
  __syncthreads();
  for (int i = tid; i < WR * V; i += ROWS_WARPS * 32) {
    const int g = i / V, v = i % V, m = m0 + v / ROWS_R;
    const int n = (blockIdx.x * WR + g) * ROWS_R + v % ROWS_R;
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < WK; ++q) s += smem[(g * WK + q) * V + v];
    if (m < M && n < N) out[(long long)m * ldo + n] = s;
  }
}

// ----------------------------------------------------------------------- many rows
// A block owns BM x BN results, a thread 8 x TN of them (in runs of 4 in either direction, a warp
// 4 x 8 threads, so that its 16-byte shared-memory reads meet no conflicts). K goes through two
// shared-memory buffers BK at a time, kept [k][row]; the global loads of the next block are in
// registers while this one is multiplied. Where the tiles alone leave SMs idle or a thin last
// round, the S blocks of a cluster share a tile's K: each leaves its partial tile in its own
// shared memory, and every block sums its share of the rows out of all of them, in rank order.
constexpr int BK = 16;

__device__ __forceinline__ void cluster_sync() {
  __syncwarp();  // the aligned form wants whole warps
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_peer(unsigned addr, unsigned rank) {
  unsigned there;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(there)
               : "memory");
  return v;
}

template <int BM, int BN, int TN>
struct Tile {
  static constexpr int THREADS = BM * BN / (8 * TN), PA = BM + 4, PB = BN + 4;
  static constexpr int STAGING = 2 * BK * (PA + PB) * 4, PARTIAL = BM * BN * 4;
};

template <int BM, int BN, int TN, int S, int OCC>
__global__ void __launch_bounds__(BM * BN / (8 * TN), OCC)
tile_kernel(const float* x /* written by the kernel before: no read-only promise */,
            const float* __restrict__ w, float* out, int M, int N, int K, long long ldx,
            long long ldw, long long ldo, long long bx, long long bw, long long bo) {
  using G = Tile<BM, BN, TN>;
  constexpr int THREADS = G::THREADS, TX = BN / TN, WX = TX / 8, NB = TN / 4;
  constexpr int LA = BM * BK / 4 / THREADS, LB = BN * BK / 4 / THREADS;  // 16-byte loads a thread
  static_assert(LA * THREADS * 4 == BM * BK && LB * THREADS * 4 == BN * BK, "uneven loads");
  extern __shared__ __align__(16) float smem[];
  float(*as)[G::PA] = reinterpret_cast<float(*)[G::PA]>(smem);  // [2 * BK][BM]
  float(*bs)[G::PB] = reinterpret_cast<float(*)[G::PB]>(smem + 2 * BK * G::PA);
  const int product = blockIdx.z / S, rank = blockIdx.z % S;
  x += (long long)product * bx;
  w += (long long)product * bw;
  out += (long long)product * bo;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = (warp % WX) * 8 + lane % 8, ty = (warp / WX) * 4 + lane / 8;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // this block's K blocks: whole ones of BK, shared as evenly as they go
  const int all = (K + BK - 1) / BK, first = all * rank / S, blocks = all * (rank + 1) / S - first;
  float4 ra[LA], rb[LB];
  auto load_b = [&](int c) {
#pragma unroll
    for (int i = 0; i < LB; ++i) {
      const int e = tid + i * THREADS, row = e / (BK / 4), k = (first + c) * BK + (e % (BK / 4)) * 4;
      rb[i] = (n0 + row < N && k < K)
                  ? __ldg(reinterpret_cast<const float4*>(w + (long long)(n0 + row) * ldw + k))
                  : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto load_a = [&](int c) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int e = tid + i * THREADS, row = e / (BK / 4), k = (first + c) * BK + (e % (BK / 4)) * 4;
      ra[i] = (m0 + row < M && k < K)
                  ? __ldcg(reinterpret_cast<const float4*>(x + (long long)(m0 + row) * ldx + k))
                  : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int e = tid + i * THREADS, row = e / (BK / 4), k = buf * BK + (e % (BK / 4)) * 4;
      as[k][row] = ra[i].x;
      as[k + 1][row] = ra[i].y;
      as[k + 2][row] = ra[i].z;
      as[k + 3][row] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < LB; ++i) {
      const int e = tid + i * THREADS, row = e / (BK / 4), k = buf * BK + (e % (BK / 4)) * 4;
      bs[k][row] = rb[i].x;
      bs[k + 1][row] = rb[i].y;
      bs[k + 2][row] = rb[i].z;
      bs[k + 3][row] = rb[i].w;
    }
  };
  float acc[8][TN];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  load_b(0);
  fb_pdl_wait();
  load_a(0);
  put(0);
  __syncthreads();
  for (int c = 0; c < blocks; ++c) {
    const int buf = c & 1;
    if (c + 1 < blocks) {
      load_a(c + 1);
      load_b(c + 1);
    }
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      const int k = buf * BK + kk;
      float a[8], b[TN];
      *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&as[k][ty * 4]);
      *reinterpret_cast<float4*>(a + 4) =
          *reinterpret_cast<const float4*>(&as[k][BM / 2 + ty * 4]);
#pragma unroll
      for (int q = 0; q < NB; ++q)
        *reinterpret_cast<float4*>(b + 4 * q) =
            *reinterpret_cast<const float4*>(&bs[k][q * (BN / NB) + tx * 4]);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    if (c + 1 < blocks) put(buf ^ 1);
    __syncthreads();
  }
  fb_pdl_launch();
  if (S == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = m0 + (i / 4) * (BM / 2) + ty * 4 + i % 4;
      if (m >= M) continue;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int n = n0 + (j / 4) * (BN / NB) + tx * 4 + j % 4;
        if (n < N) out[(long long)m * ldo + n] = acc[i][j];
      }
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int q = 0; q < NB; ++q)
      *reinterpret_cast<float4*>(smem + ((i / 4) * (BM / 2) + ty * 4 + i % 4) * BN + q * (BN / NB) +
                                 tx * 4) =
          make_float4(acc[i][4 * q], acc[i][4 * q + 1], acc[i][4 * q + 2], acc[i][4 * q + 3]);
  cluster_sync();
  const unsigned base = (unsigned)__cvta_generic_to_shared(smem);
  constexpr int SHARE = BM / S;  // rows that this block finishes
#pragma unroll 2
  for (int e = tid; e < SHARE * BN / 4; e += THREADS) {
    const int row = rank * SHARE + e / (BN / 4), col = (e % (BN / 4)) * 4;
    float4 part[S];
#pragma unroll
    for (int r = 0; r < S; ++r) part[r] = ld_peer(base + (unsigned)(row * BN + col) * 4u, r);
    float4 s = part[0];
#pragma unroll
    for (int r = 1; r < S; ++r) {
      s.x += part[r].x;
      s.y += part[r].y;
      s.z += part[r].z;
      s.w += part[r].w;
    }
    const int m = m0 + row, n = n0 + col;
    if (m < M) {
      float* o = out + (long long)m * ldo + n;
      if (n < N) o[0] = s.x;
      if (n + 1 < N) o[1] = s.y;
      if (n + 2 < N) o[2] = s.z;
      if (n + 3 < N) o[3] = s.w;
    }
  }
  cluster_sync();  // a peer may still read this block's partial tile
}

template <int MR, int WK>
int launch_rows(const FbGemmF32& p, cudaStream_t stream) {
  constexpr int CH = ROWS_CHUNK<WK>, WR = ROWS_WARPS / WK;
  constexpr int bytes = 2 * MR * CH * 4;
  static_assert(bytes >= ROWS_WARPS * MR * ROWS_R * 4, "room for the sums");
  static bool seen[64] = {};
  if (bytes > 48 * 1024 && fb_first_use_on_device(seen) &&
      cudaFuncSetAttribute(rows_kernel<MR, WK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           bytes) != cudaSuccess)
    return fb_fail(2, "gemm_f32: cannot set %d bytes of shared memory", bytes);
  const dim3 grid((p.N + WR * ROWS_R - 1) / (WR * ROWS_R), (p.M + MR - 1) / MR);
  fb_launch(rows_kernel<MR, WK>, grid, dim3(ROWS_WARPS * 32), (size_t)bytes, stream, p.x, p.w,
            p.out, p.M, p.N, p.K, p.ldx, p.ldw, p.ldo);
  return fb_check_launch("gemm_f32_rows");
}

template <int MR>
int launch_rows_by_shape(const FbGemmF32& p, cudaStream_t stream) {
  // WK from N and K alone, so that a result's order of summation does not depend on M. Up to 128 of
  // K is one warp's: the others of four had nothing to do, and blocks of 8 rows of w each staged a
  // whole chunk (32 rows, 64 -> 2048: 2.6 us for 7.2; 16 rows, 64 -> 16384: 6.1 for 14.0; the general
  // kernel 5.3 and 7.6).
  if (p.K <= 128) return launch_rows<MR, 1>(p, stream);
  if constexpr (MR <= 8) {  // (16 rows a pass go with N > 8192)
    if (p.N <= 8192) return launch_rows<MR, 4>(p, stream);
  }
  return launch_rows<MR, 2>(p, stream);
}

template <int BM, int BN, int TN, int S, int OCC>
int launch_tile(const FbGemmF32& p, cudaStream_t stream) {
  using G = Tile<BM, BN, TN>;
  constexpr int bytes = S > 1 && G::PARTIAL > G::STAGING ? G::PARTIAL : G::STAGING;
  const dim3 grid((p.N + BN - 1) / BN, (p.M + BM - 1) / BM, p.count * S);
  if (grid.y > 65535 || grid.z > 65535)
    return fb_fail(1, "gemm_f32: M=%d x %d exceeds the grid limit", p.M, p.count);
  auto kernel = tile_kernel<BM, BN, TN, S, OCC>;
  static bool seen[64] = {};
  if (bytes > 48 * 1024 && fb_first_use_on_device(seen) &&
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
          cudaSuccess)
    return fb_fail(2, "gemm_f32: cannot set %d bytes of shared memory", bytes);
  if (S == 1)
    fb_launch(kernel, grid, dim3(G::THREADS), (size_t)bytes, stream, p.x, p.w, p.out, p.M, p.N, p.K,
              p.ldx, p.ldw, p.ldo, p.bx, p.bw, p.bo);
  else
    fb_launch_cluster(kernel, grid, dim3(G::THREADS), (size_t)bytes, stream, S, p.x, p.w, p.out,
                      p.M, p.N, p.K, p.ldx, p.ldw, p.ldo, p.bx, p.bw, p.bo);
  return fb_check_launch("gemm_f32_tile");
}
}  // namespace

bool fb_gemm_f32_fits(const FbGemmF32& p) {
  const auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (p.count > 1 && p.M <= 16) return false;  // little to share: the general kernel's tiles
  // what the grids of both kernels carry (the general kernel's limits are wider)
  if ((p.M + 63) / 64 > 65535 || (long long)p.count * 8 > 65535) return false;
  return p.K % 4 == 0 && p.ldx % 4 == 0 && p.ldw % 4 == 0 && p.bx % 4 == 0 && p.bw % 4 == 0 &&
         aligned(p.x) && aligned(p.w);
}

int fb_gemm_f32_launch(const FbGemmF32& p, cudaStream_t stream) {
  // (17 to 32 rows of many short columns are a tile's: 32 rows, 64 -> 16384 7.0 us against 10.1, 96
  // 9.4 against 10.2, 128 11.9 against 10.4, 256 20.7 against 27.0)
  const bool thin = p.M > 16 && p.N > 8192 && (p.K <= 96 || (p.K > 128 && p.K <= 256));
  if (p.count == 1 && p.M <= FB_GEMM_F32_ROWS && !thin) {
    if (p.M == 1) return launch_rows_by_shape<1>(p, stream);
    if (p.M == 2) return launch_rows_by_shape<2>(p, stream);
    if (p.M <= 4) return launch_rows_by_shape<4>(p, stream);
    // 16 tokens a pass halve the weights' traffic of 9 to 32 rows and the blocks in flight: worth
    // it where the rows of w alone fill the SMs (16 rows, 2048 -> 16384: 42 against 56 us with 8;
    // 32 rows, 8192 -> 2048: 51 against 48 us)
    if (p.M <= 8 || p.N <= 8192) return launch_rows_by_shape<8>(p, stream);
    return launch_rows_by_shape<16>(p, stream);
  }
  // The tensor cores (gemm_f32_tcgen05.cu) from 33 rows on, where there is enough to do: their kernel
  // starts 4 us later (tensor memory, a pair of SMs, the first split). 64 rows of 2048 -> 128 20.5 us
  // against 24.6 with tiles, -> 2048 22.6 against 32.8; 1000 rows of 256 -> 2048 20.5 against 45; but
  // 512 rows of 512 -> 512 22.5 against 18.4, 1000 rows of 64 -> 1024 16.4 against 12.3, 300 rows of
  // 2048 -> 64 both 24.6. Rows count in whole 128s: a step that is padded to a bucket sums as the
  // plain one does.
  const long long rows = (p.M + 127) / 128 * 128;
  if (p.count == 1 && p.M > FB_GEMM_F32_ROWS && p.N >= 128 &&
      (p.K >= 1024 || rows * p.N * p.K >= 1LL << 28)) {
    const int code = fb_gemm_f32_tc_launch(p, stream);
    if (code != FB_GEMM_F32_NOT_HERE) return code;
  }
  // What is left: batched products, fewer than 128 results a row, little to do. 128 x 128 tiles move
  // the least through shared memory and need three full rounds of two blocks an SM to hide their last
  // one; below that 64 x 64 tiles, K shared eightfold from 1,024 on. (The lines were drawn where large
  // single products were these tiles', too: 2048 rows, 2048 -> 16384 46 TFLOP/s, 37 with 64 x 64; 777
  // rows, 2048 -> 3072 305 us with 64 x 64, 412 with 128 x 128; 128 rows, 2048 -> 64: 14 and 230.)
  // Rows count in whole 128s here, too.
  const long long big = (long long)((p.M + 127) / 128) * ((p.N + 127) / 128) * p.count;
  if (big >= 3 * 2 * sm_count()) return launch_tile<128, 128, 8, 1, 2>(p, stream);
  if (p.K >= 1024) return launch_tile<64, 64, 4, 8, 4>(p, stream);
  if (p.K >= 512) return launch_tile<64, 64, 4, 4, 4>(p, stream);
  if (p.K >= 256) return launch_tile<64, 64, 4, 2, 4>(p, stream);
  return launch_tile<64, 64, 4, 1, 4>(p, stream);
}
