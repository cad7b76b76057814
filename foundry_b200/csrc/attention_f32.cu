// The attention of attention_simt.cu (same formulas, same 32-bit arithmetic) for float32 caches
// and head sizes of 32, 64 and 128, in two forms:
//
// `split_kernel`, few tokens a sequence (single-token steps): a (token, key head) is walked by
//   the CTAs of a cluster, a range of its keys each, all query heads of the key head on one walk.
//   Bound by the cache's bytes and by how many of them are under way; a lane keeps the rows of
//   four keys in flight. attention_simt.cu's warp a (token, head) reads one value row after
//   another. 4 tokens over 600 keys, 32 heads over 8 of 64: 11 us against 511.
// `tile_kernel`, many tokens a sequence (prompts): 64 neighbouring tokens of one sequence and one
//   query head a block, keys in tiles through shared memory, register tiles for both products.
//   Bound by latency with three warps a scheduler (the issue slots are 38 % busy; registers and
//   shared memory hold no more). 777 tokens, 32 heads over 8 of 64: 169 us, 204 before a tile's
//   product lost a branch a channel and two blocks shared the keys, 1405 in attention_simt.cu.
//
// Queries, keys and values are read with coherent (L2) loads: the kernel that wrote this step's
// rows may have overlapped this kernel's start.
#include <type_traits>

#include "attention_f32.h"
#include "common.cuh"

namespace {

__device__ __forceinline__ float4 ldcg4(const float* p) {
  return __ldcg(reinterpret_cast<const float4*>(p));
}
__device__ __forceinline__ long long row_of(const int* pages, int j, int ring_pages,
                                            long long page_stride, int D) {
  int lp = j / FB_PAGE;
  if (ring_pages > 0) lp %= ring_pages;
  return (long long)pages[lp] * page_stride + (long long)(j % FB_PAGE) * D;
}
// All threads of the cluster's blocks meet. (The aligned form wants whole warps: some lanes may still
// be in the branch or the loop in front.)
__device__ __forceinline__ void meet_cluster() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}
// exp(a - b) for a running maximum b that is -inf while nothing has been seen (a NaN stays one)
__device__ __forceinline__ float exp_below(float a, float b) {
  return a == -INFINITY ? 0.f : expf(a - b);
}

// ------------------------------------------------------------------- few tokens a sequence
// Eight lanes share a key (a lane holds D / 8 elements of every query head and of its sums, in
// runs of 4), W warps share a pair, each takes four keys side by side and U of each lane group's
// keys at a time (two where four would not fit the registers);
// lane groups, warps and CTAs keep a maximum and a sum of their own and are merged in a fixed
// order at the end.
template <int D, int GH, int S, int W>
__global__ void __launch_bounds__(W * 32)
split_kernel(FbAttentionF32 p, int head_chunks) {
  constexpr int V4 = D / 32, SPLIT_WARPS = W, SPLIT_GROUPS = W * 4;
  constexpr bool FEW = W < 4;  // mostly few keys
  constexpr int U = FEW && D >= 128 ? 2 : 4;
  __shared__ float stat_m[SPLIT_GROUPS][GH], stat_l[SPLIT_GROUPS][GH];
  __shared__ __align__(16) float sums[SPLIT_GROUPS][GH][D];
  __shared__ float cta_m[GH], cta_l[GH];
  fb_pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = lane % 8, group = warp * 4 + lane / 8;
  const int t = blockIdx.x, kvh = blockIdx.y / head_chunks, rank = S > 1 ? blockIdx.z : 0;
  const int G = p.A / p.Kh, h0 = (blockIdx.y % head_chunks) * GH, heads = min(GH, G - h0);
  const int a0 = kvh * G + h0;
  const int seq = p.seq_of_token[t];
  float* o = p.out + (size_t)t * p.out_stride + (size_t)a0 * D;
  if (seq < 0) {  // padding token: defined output, no cache access (the whole cluster agrees)
    if (rank == 0)
      for (int i = threadIdx.x; i < heads * D; i += SPLIT_WARPS * 32) o[i] = 0.f;
    return;
  }
  const int pos = p.positions[t];
  const int lo = p.window > 0 && pos - p.window + 1 > 0 ? pos - p.window + 1 : 0;
  const int each = ((pos + 1 - lo + S - 1) / S + SPLIT_GROUPS - 1) / SPLIT_GROUPS * SPLIT_GROUPS;
  const int begin = lo + rank * each, end = min(pos + 1, begin + each);
  const int* pages = p.page_table + (size_t)seq * p.max_pages;
  const float* kbase = p.k + (long long)kvh * p.head_stride + part * 4;
  const float* vbase = p.v + (long long)kvh * p.head_stride + part * 4;

  float4 q[GH][V4];
  const float* qrow = p.q + (size_t)t * p.q_stride + (size_t)a0 * D + part * 4;
#pragma unroll
  for (int h = 0; h < GH; ++h)
#pragma unroll
    for (int i = 0; i < V4; ++i)
      q[h][i] = h < heads ? ldcg4(qrow + h * D + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
  float m[GH], l[GH];
  float4 acc[GH][V4];
#pragma unroll
  for (int h = 0; h < GH; ++h) {
    m[h] = -INFINITY;
    l[h] = 0.f;
#pragma unroll
    for (int i = 0; i < V4; ++i) acc[h][i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // every lane of a warp makes the same number of rounds: the exchanges need them all
  for (int j0 = begin; j0 < end; j0 += SPLIT_GROUPS * U) {
    float4 kk[U][V4], vv[U][V4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (FEW && u > 0 && j0 + u * SPLIT_GROUPS >= end) {  // no group has a key there
#pragma unroll
        for (int i = 0; i < V4; ++i) kk[u][i] = vv[u][i] = make_float4(0.f, 0.f, 0.f, 0.f);
        continue;
      }
      const int j = min(j0 + u * SPLIT_GROUPS + group, end - 1);  // beyond the end: masked below
      const long long row = row_of(pages, j, p.ring_pages, p.page_stride, D);
#pragma unroll
      for (int i = 0; i < V4; ++i) kk[u][i] = ldcg4(kbase + row + 32 * i);
#pragma unroll
      for (int i = 0; i < V4; ++i) vv[u][i] = ldcg4(vbase + row + 32 * i);
    }
    float s[GH][U];
#pragma unroll
    for (int h = 0; h < GH; ++h)
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < V4; ++i) {
          dot = fmaf(q[h][i].x, kk[u][i].x, dot);
          dot = fmaf(q[h][i].y, kk[u][i].y, dot);
          dot = fmaf(q[h][i].z, kk[u][i].z, dot);
          dot = fmaf(q[h][i].w, kk[u][i].w, dot);
        }
        s[h][u] = dot;
      }
#pragma unroll
    for (int x = 1; x < 8; x *= 2)
#pragma unroll
      for (int h = 0; h < GH; ++h)
#pragma unroll
        for (int u = 0; u < U; ++u) s[h][u] += __shfl_xor_sync(0xffffffffu, s[h][u], x);
#pragma unroll
    for (int h = 0; h < GH; ++h) {
      float top = m[h];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        s[h][u] = j0 + u * SPLIT_GROUPS + group < end ? s[h][u] * p.scale : -INFINITY;
        top = fmaxf(top, s[h][u]);
      }
      const float corr = exp_below(m[h], top);
      m[h] = top;
      l[h] *= corr;
#pragma unroll
      for (int i = 0; i < V4; ++i) {
        acc[h][i].x *= corr;
        acc[h][i].y *= corr;
        acc[h][i].z *= corr;
        acc[h][i].w *= corr;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (j0 + u * SPLIT_GROUPS + group >= end) continue;
        const float e = exp_below(s[h][u], top);
        l[h] += e;
#pragma unroll
        for (int i = 0; i < V4; ++i) {
          acc[h][i].x = fmaf(e, vv[u][i].x, acc[h][i].x);
          acc[h][i].y = fmaf(e, vv[u][i].y, acc[h][i].y);
          acc[h][i].z = fmaf(e, vv[u][i].z, acc[h][i].z);
          acc[h][i].w = fmaf(e, vv[u][i].w, acc[h][i].w);
        }
      }
    }
  }
#pragma unroll
  for (int h = 0; h < GH; ++h) {
    if (part == 0) {
      stat_m[group][h] = m[h];
      stat_l[group][h] = l[h];
    }
#pragma unroll
    for (int i = 0; i < V4; ++i)
      *reinterpret_cast<float4*>(&sums[group][h][part * 4 + 32 * i]) = acc[h][i];
  }
  __syncthreads();
  // the block's groups into group 0's place (each element by one thread); groups that saw no key
  // hold nothing
  const int seen = FEW ? max(1, min(SPLIT_GROUPS, end - begin)) : SPLIT_GROUPS;
  for (int i = threadIdx.x; i < GH * D; i += SPLIT_WARPS * 32) {
    const int h = i / D, d = i % D;
    float top = -INFINITY, sum = 0.f, total = 0.f;
#pragma unroll
    for (int g = 0; g < SPLIT_GROUPS; ++g)
      if (g < seen) top = fmaxf(top, stat_m[g][h]);
#pragma unroll
    for (int g = 0; g < SPLIT_GROUPS; ++g) {
      if (g >= seen) break;
      const float f = exp_below(stat_m[g][h], top);
      sum = fmaf(f, sums[g][h][d], sum);
      total = fmaf(f, stat_l[g][h], total);
    }
    if (S == 1) {
      if (h < heads) o[i] = sum / total;
    } else {
      sums[0][h][d] = sum;
      if (d == 0) {
        cta_m[h] = top;
        cta_l[h] = total;
      }
    }
  }
  if (S == 1) return;
  meet_cluster();
  auto peer = [](const float* mine, int r) {
    unsigned there;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(there)
                 : "r"((unsigned)__cvta_generic_to_shared(mine)), "r"(r));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(there) : "memory");
    return v;
  };
  for (int i = rank * (SPLIT_WARPS * 32) + threadIdx.x; i < heads * D; i += S * SPLIT_WARPS * 32) {
    const int h = i / D, d = i % D;
    float pm[S], pl[S], ps[S], top = -INFINITY, sum = 0.f, total = 0.f;
#pragma unroll
    for (int r = 0; r < S; ++r) {
      pm[r] = peer(&cta_m[h], r);
      pl[r] = peer(&cta_l[h], r);
      ps[r] = peer(&sums[0][h][d], r);
    }
#pragma unroll
    for (int r = 0; r < S; ++r) top = fmaxf(top, pm[r]);
#pragma unroll
    for (int r = 0; r < S; ++r) {
      const float f = exp_below(pm[r], top);
      sum = fmaf(f, ps[r], sum);
      total = fmaf(f, pl[r], total);
    }
    o[i] = sum / total;
  }
  meet_cluster();
}

// ------------------------------------------------------------------ many tokens a sequence
// A block takes the 64 tokens from 64 * its number on, those that belong to one sequence at a
// time (`runs`: z of the grid shares a block's runs among neighbours, so that many short
// sequences side by side are not walked one after another). A thread owns 4 rows; the 8 threads
// of a row lie in one warp, so the weights between the two products pass through shared memory
// that only the warp reads. A causal prompt's blocks have one tile of keys to many: the S blocks of a
// cluster (neighbours in z) take every S-th tile of the same rows and merge what they hold, in rank
// order, each a share of the rows.
constexpr int BQ = 64, TILE_THREADS = 128;

template <int D, int BKEY>
struct AttnTile {
  static constexpr int PQ = BQ + 4, PK = BKEY + 4, PV = D + 4, PP = BQ + 4;
  static constexpr int BYTES = (D * PQ + D * PK + BKEY * PV + BKEY * PP) * 4;
};

__device__ __forceinline__ unsigned shared_of(const float* mine, int rank) {
  unsigned there;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(there)
               : "r"((unsigned)__cvta_generic_to_shared(mine)), "r"(rank));
  return there;
}
__device__ __forceinline__ float ld_peer(unsigned there) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(there) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_peer4(unsigned there) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(there)
               : "memory");
  return v;
}

template <int D, int BKEY, int S>
__global__ void __launch_bounds__(TILE_THREADS, D >= 128 ? 2 : 3) tile_kernel(FbAttentionF32 p) {
  using G = AttnTile<D, BKEY>;
  constexpr int NK = BKEY / 32, NV = D / 32;
  extern __shared__ __align__(16) float smem[];
  float(*qt)[G::PQ] = reinterpret_cast<float(*)[G::PQ]>(smem);  // [D][token]
  float(*kt)[G::PK] = reinterpret_cast<float(*)[G::PK]>(smem + D * G::PQ);  // [D][key]
  float(*vt)[G::PV] = reinterpret_cast<float(*)[G::PV]>(smem + D * G::PQ + D * G::PK);
  float(*pt)[G::PP] =
      reinterpret_cast<float(*)[G::PP]>(smem + D * G::PQ + D * G::PK + BKEY * G::PV);
  __shared__ int seq_of[BQ], pos_of[BQ];
  fb_pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = lane % 8, ty = warp * 4 + lane / 8;
  const int t0 = (gridDim.x - 1 - blockIdx.x) * BQ;  // later tokens see more keys: first
  const int a = blockIdx.y, kvh = a / (p.A / p.Kh);
  const int rows = min(BQ, p.T - t0), rank = S > 1 ? blockIdx.z % S : 0;
  // (a cluster's own results, over the tiles of keys and values: rows of D, maxima, sums)
  float* held = smem + D * G::PQ;
  float* held_m = held + BQ * D;
  float* held_l = held_m + BQ;
  static_assert(BQ * D + 2 * BQ <= D * G::PK + BKEY * G::PV, "room for a cluster's results");
  if (tid < BQ) {
    seq_of[tid] = tid < rows ? p.seq_of_token[t0 + tid] : -1;
    pos_of[tid] = tid < rows ? p.positions[t0 + tid] : 0;
  }
  __syncthreads();
  const int breaks = __syncthreads_count(tid > 0 && tid < rows && seq_of[tid] != seq_of[tid - 1]);
  if ((int)blockIdx.z / S > breaks) return;  // no run for this block, nor for its cluster
  for (int i = tid; i < BQ * (D / 4); i += TILE_THREADS) {
    const int r = i % BQ, d = (i / BQ) * 4;
    const float4 v = seq_of[r] >= 0 ? ldcg4(p.q + (size_t)(t0 + r) * p.q_stride + (size_t)a * D + d)
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
    qt[d][r] = v.x;
    qt[d + 1][r] = v.y;
    qt[d + 2][r] = v.z;
    qt[d + 3][r] = v.w;
  }
  const int warp_row = warp * 16;  // a warp's 16 rows
  for (int first = 0, run = 0; first < rows; ++run) {
    const int seq = seq_of[first];
    int last = first;  // the run's last row
    while (last + 1 < rows && seq_of[last + 1] == seq) ++last;
    const int begin_row = first;
    first = last + 1;
    if (run % (gridDim.z / S) != blockIdx.z / S) continue;
    if (seq < 0 && rank > 0) continue;
    if (seq < 0) {  // padding tokens: defined output, no cache access
      for (int i = tid; i < (last - begin_row + 1) * D; i += TILE_THREADS)
        p.out[(size_t)(t0 + begin_row + i / D) * p.out_stride + (size_t)a * D + i % D] = 0.f;
      continue;
    }
    int low[4], high[4];  // the keys that each of this thread's rows sees
    int from = 0x7fffffff, to = -1;             // what any row of the run sees
    int inner_from = 0, inner_to = 0x7fffffff;  // what every row of it sees
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty * 4 + i;
      const bool mine = r >= begin_row && r <= last;
      high[i] = mine ? pos_of[r] : -1;
      low[i] = p.window > 0 ? max(0, high[i] - p.window + 1) : 0;
    }
    for (int r = begin_row; r <= last; ++r) {
      const int lo = p.window > 0 ? max(0, pos_of[r] - p.window + 1) : 0;
      to = max(to, pos_of[r]);
      from = min(from, lo);
      inner_to = min(inner_to, pos_of[r]);
      inner_from = max(inner_from, lo);
    }
    // a warp without a row of the run only helps to load
    const bool mine_here = warp_row <= last && warp_row + 15 >= begin_row;
    const int* pages = p.page_table + (size_t)seq * p.max_pages;
    const float* kbase = p.k + (long long)kvh * p.head_stride;
    const float* vbase = p.v + (long long)kvh * p.head_stride;
    float m[4], l[4];
    float4 acc[4][NV];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      m[i] = -INFINITY;
      l[i] = 0.f;
#pragma unroll
      for (int q = 0; q < NV; ++q) acc[i][q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int j0 = (from / BKEY + rank) * BKEY; j0 <= to; j0 += S * BKEY) {
      __syncthreads();  // the tile before is no longer read (and the queries are in)
#pragma unroll 4
      for (int i = tid; i < BKEY * (D / 4); i += TILE_THREADS) {
        // four neighbouring 16-byte pieces of eight keys a warp
        const int key = (i / 32) % (BKEY / 8) * 8 + i % 32 / 4;
        const int d = (i / 32 / (BKEY / 8) * 4 + i % 4) * 4;
        const int j = j0 + key;
        const bool have = j >= from && j <= to;
        const float4 v = have ? ldcg4(kbase + row_of(pages, j, p.ring_pages, p.page_stride, D) + d)
                              : make_float4(0.f, 0.f, 0.f, 0.f);
        kt[d][key] = v.x;
        kt[d + 1][key] = v.y;
        kt[d + 2][key] = v.z;
        kt[d + 3][key] = v.w;
      }
#pragma unroll 4
      for (int i = tid; i < BKEY * (D / 4); i += TILE_THREADS) {
        const int key = i / (D / 4), d = i % (D / 4) * 4, j = j0 + key;
        const bool have = j >= from && j <= to;
        *reinterpret_cast<float4*>(&vt[key][d]) =
            have ? ldcg4(vbase + row_of(pages, j, p.ring_pages, p.page_stride, D) + d)
                 : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      __syncthreads();
      if (!mine_here) continue;
      const int keys = min(BKEY, to - j0 + 1);  // (the rest of the tile counts as nothing)
      float s[4][4 * NK];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 4 * NK; ++c) s[i][c] = 0.f;
      // (a short tile's second half is multiplied, too: it is zeros)
#pragma unroll 8
      for (int d = 0; d < D; ++d) {
        float x[4], y[4 * NK];
        *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(&qt[d][ty * 4]);
#pragma unroll
        for (int q = 0; q < NK; ++q) {
          *reinterpret_cast<float4*>(y + 4 * q) =
              *reinterpret_cast<const float4*>(&kt[d][q * 32 + tx * 4]);
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 4 * q; c < 4 * q + 4; ++c) s[i][c] = fmaf(x[i], y[c], s[i][c]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float top = m[i];
#pragma unroll
        for (int c = 0; c < 4 * NK; ++c) {
          const int j = j0 + (c / 4) * 32 + tx * 4 + c % 4;
          s[i][c] = j >= low[i] && j <= high[i] ? s[i][c] * p.scale : -INFINITY;
          top = fmaxf(top, s[i][c]);
        }
#pragma unroll
        for (int x = 1; x < 8; x *= 2) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
        const float corr = exp_below(m[i], top);
        m[i] = top;
        float sum = 0.f;
#pragma unroll
        for (int c = 0; c < 4 * NK; ++c) {
          s[i][c] = exp_below(s[i][c], top);
          sum += s[i][c];
        }
#pragma unroll
        for (int x = 1; x < 8; x *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, x);
        l[i] = l[i] * corr + sum;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          acc[i][q].x *= corr;
          acc[i][q].y *= corr;
          acc[i][q].z *= corr;
          acc[i][q].w *= corr;
        }
      }
#pragma unroll
      for (int c = 0; c < 4 * NK; ++c)
        *reinterpret_cast<float4*>(&pt[(c / 4) * 32 + tx * 4 + c % 4][ty * 4]) =
            make_float4(s[0][c], s[1][c], s[2][c], s[3][c]);
      __syncwarp();
      // A key that a row does not see has weight 0, and its value must not count even where it is
      // no number (a later token's): tiles on the edge of what the run sees leave such values out.
      auto add_values = [&](auto edge) {
#pragma unroll 4
        for (int key = 0; key < (decltype(edge)::value ? keys : BKEY); ++key) {
          float x[4];
          *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(&pt[key][ty * 4]);
#pragma unroll
          for (int q = 0; q < NV; ++q) {
            const float4 y = *reinterpret_cast<const float4*>(&vt[key][q * 32 + tx * 4]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (decltype(edge)::value && (j0 + key < low[i] || j0 + key > high[i])) continue;
              acc[i][q].x = fmaf(x[i], y.x, acc[i][q].x);
              acc[i][q].y = fmaf(x[i], y.y, acc[i][q].y);
              acc[i][q].z = fmaf(x[i], y.z, acc[i][q].z);
              acc[i][q].w = fmaf(x[i], y.w, acc[i][q].w);
            }
          }
        }
      };
      if (j0 >= inner_from && j0 + BKEY - 1 <= inner_to)
        add_values(std::false_type{});
      else
        add_values(std::true_type{});
      __syncwarp();  // the weights are read before the next tile's replace them
    }
    if constexpr (S > 1) {
      __syncthreads();  // the last tile is no longer read
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i;
        if (tx == 0) {
          held_m[r] = m[i];
          held_l[r] = l[i];
        }
#pragma unroll
        for (int q = 0; q < NV; ++q)
          *reinterpret_cast<float4*>(held + r * D + q * 32 + tx * 4) = acc[i][q];
      }
      meet_cluster();
      unsigned sums[S], tops[S], totals[S];
#pragma unroll
      for (int k = 0; k < S; ++k) {
        sums[k] = shared_of(held, k);
        tops[k] = shared_of(held_m, k);
        totals[k] = shared_of(held_l, k);
      }
      for (int e = tid; e < BQ / S * (D / 4); e += TILE_THREADS) {
        const int r = rank * (BQ / S) + e / (D / 4), d = e % (D / 4) * 4;
        if (r < begin_row || r > last) continue;
        float pm[S], pl[S], top = -INFINITY, total = 0.f;
        float4 ps[S], sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < S; ++k) {
          pm[k] = ld_peer(tops[k] + r * 4);
          pl[k] = ld_peer(totals[k] + r * 4);
          ps[k] = ld_peer4(sums[k] + (r * D + d) * 4);
        }
#pragma unroll
        for (int k = 0; k < S; ++k) top = fmaxf(top, pm[k]);
#pragma unroll
        for (int k = 0; k < S; ++k) {
          const float f = exp_below(pm[k], top);
          total = fmaf(f, pl[k], total);
          sum.x = fmaf(f, ps[k].x, sum.x);
          sum.y = fmaf(f, ps[k].y, sum.y);
          sum.z = fmaf(f, ps[k].z, sum.z);
          sum.w = fmaf(f, ps[k].w, sum.w);
        }
        const float inv = 1.0f / total;
        float* o = p.out + (size_t)(t0 + r) * p.out_stride + (size_t)a * D + d;
        o[0] = sum.x * inv;
        o[1] = sum.y * inv;
        o[2] = sum.z * inv;
        o[3] = sum.w * inv;
      }
      meet_cluster();  // a peer may still read this block's results
      continue;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty * 4 + i;
      if (r < begin_row || r > last) continue;
      const float inv = 1.0f / l[i];
      float* o = p.out + (size_t)(t0 + r) * p.out_stride + (size_t)a * D + tx * 4;
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        o[q * 32] = acc[i][q].x * inv;
        o[q * 32 + 1] = acc[i][q].y * inv;
        o[q * 32 + 2] = acc[i][q].z * inv;
        o[q * 32 + 3] = acc[i][q].w * inv;
      }
    }
  }
}

template <int D, int GH, int S, int W = 4>
int launch_split(const FbAttentionF32& p, cudaStream_t stream) {
  const int chunks = (p.A / p.Kh + GH - 1) / GH;
  const dim3 grid(p.T, p.Kh * chunks, S);
  if (S == 1)
    fb_launch(split_kernel<D, GH, S, W>, grid, dim3(W * 32), 0, stream, p, chunks);
  else
    fb_launch_cluster(split_kernel<D, GH, S, W>, grid, dim3(W * 32), 0, stream, S, p, chunks);
  return fb_check_launch("attention_f32_split");
}

template <int D, int S>
int launch_tiles(const FbAttentionF32& p, cudaStream_t stream) {
  constexpr int BKEY = D >= 128 ? 32 : 64, bytes = AttnTile<D, BKEY>::BYTES;
  static bool seen[64] = {};
  if (fb_first_use_on_device(seen) &&
      cudaFuncSetAttribute(tile_kernel<D, BKEY, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           bytes) != cudaSuccess)
    return fb_fail(2, "attention: cannot set %d bytes of shared memory", bytes);
  const dim3 grid((p.T + BQ - 1) / BQ, p.A, (p.n_seqs < 4 ? p.n_seqs : 4) * S);
  if (S == 1) fb_launch(tile_kernel<D, BKEY, S>, grid, dim3(TILE_THREADS), (size_t)bytes, stream, p);
  else fb_launch_cluster(tile_kernel<D, BKEY, S>, grid, dim3(TILE_THREADS), (size_t)bytes, stream, S, p);
  return fb_check_launch("attention_f32_tile");
}

int power_of_two(int n, int from) {
  while (from < n) from *= 2;
  return from;
}

template <int D>
int launch_d(const FbAttentionF32& p, cudaStream_t stream) {
  // A replayed step is padded to a bucket (16, 32, 64, 128 tokens, then whole 128s; sequences and
  // the page table's width to powers of two) and has to give the plain step's bits: the choice
  // and the ranges go by the padded sizes in both.
  const int tokens = p.T <= 128 ? power_of_two(p.T, 16) : (p.T + 127) / 128 * 128;
  const int seqs = power_of_two(p.n_seqs, 1), width = power_of_two(p.max_pages, 8);
  // At most 16 tokens a sequence on average: a tile of 64 rows would be mostly empty, and a
  // walk over a long cache by one block is what the split form avoids.
  if (tokens <= 16 * seqs) {
    const int G = p.A / p.Kh;
    const long long pairs = (long long)tokens * p.Kh * (G == 1 ? 1 : (G + 3) / 4);
    // ranges until two blocks an SM are there, each of two pages and more; several tokens a
    // sequence with no more than eight pages mostly have few keys each (no more than 16 tokens may
    // also be single ones, padded)
    const bool several = tokens > 16 && tokens > seqs;
    int S = 1;
    while (S < 8 && pairs * S < 2 * sm_count() && S * 2 * 2 <= width && !(several && width <= 8)) S *= 2;
    // With few keys, 16 lane groups of four warps have more to merge than to add, and the pairs
    // fill the SMs without them. 100 x 8 tokens, 32 heads over 8 of 64: 25 us with one warp a pair,
    // 60 with four (attention_simt.cu 35); 4 x 8 tokens: 6.1 with two, 11.3 with four in two ranges
    // (8.2). Single tokens keep four warps: 128 of them over 600 keys 94 us, 117 with two.
    if (several && S == 1) {
      if (pairs >= 1024)
        return G == 1 ? launch_split<D, 1, 1, 1>(p, stream) : launch_split<D, 4, 1, 1>(p, stream);
      return G == 1 ? launch_split<D, 1, 1, 2>(p, stream) : launch_split<D, 4, 1, 2>(p, stream);
    }
    if (G == 1)
      return S == 8   ? launch_split<D, 1, 8>(p, stream)
             : S == 4 ? launch_split<D, 1, 4>(p, stream)
             : S == 2 ? launch_split<D, 1, 2>(p, stream)
                      : launch_split<D, 1, 1>(p, stream);
    return S == 8   ? launch_split<D, 4, 8>(p, stream)
           : S == 4 ? launch_split<D, 4, 4>(p, stream)
           : S == 2 ? launch_split<D, 4, 2>(p, stream)
                    : launch_split<D, 4, 1>(p, stream);
  }
  // One sequence: two blocks share a row block's keys (777 tokens, 32 heads over 8 of 64: 169 us for
  // 191; 400: 54 for 85; 33: 15 for 14), four where the cache holds eight times the step's tokens and
  // more (64 tokens behind 3,000: 127 for 471, with two 242). The blocks of several sequences fill the
  // SMs as they are (2 x 400: 99 us, 107 with two, 4 x 200: 57 and 84).
  if (seqs == 1 && width >= 16 && width * FB_PAGE >= 8 * tokens) return launch_tiles<D, 4>(p, stream);
  if (seqs == 1 && tokens > BQ) return launch_tiles<D, 2>(p, stream);
  return launch_tiles<D, 1>(p, stream);
}
}  // namespace

bool fb_attention_f32_fits(const FbAttentionF32& p) {
  const auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  return (p.D == 32 || p.D == 64 || p.D == 128) && p.q_stride % 4 == 0 && p.page_stride % 4 == 0 &&
         p.head_stride % 4 == 0 && aligned(p.q) && aligned(p.k) && aligned(p.v) && p.n_seqs > 0 &&
         p.A <= 65535;
}

int fb_attention_f32_launch(const FbAttentionF32& p, cudaStream_t stream) {
  if (p.D == 128) return launch_d<128>(p, stream);
  if (p.D == 64) return launch_d<64>(p, stream);
  return launch_d<32>(p, stream);
}
