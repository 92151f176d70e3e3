// Generic grouped GEMM (any dtype, any shape): out[s:t] = a[s:t] . w[e]^T with fp32 FMA
// accumulation, optionally two projections fused with SwiGLU.
// Follows mini_qwen/kernels/moe_grouped_gemm.py:17-37 and mini_qwen/model/layers/moe.py:24-25.
//
// This is the shape-agnostic kernel: fp32 layers, 16-bit layers whose sizes the tcgen05 kernel
// does not cover.  Tiles of 64x64 outputs; the (expert, row-tile) of a CTA is found on the device
// from the offsets, so no host synchronisation is needed.
#include "common.cuh"

namespace mq {
namespace {

constexpr int G_TM = 64, G_TN = 64, G_KC = 16, G_THREADS = 256, G_PITCH = 68;

template <typename T>
__device__ __forceinline__ void load4_vec(const T* p, float (&v)[4]) {
  if (sizeof(T) == 4) {
    const float4 f = *reinterpret_cast<const float4*>(p);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const T* h = reinterpret_cast<const T*>(&r);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = to_float<T>(h[j]);
  }
}
template <typename T>
__device__ __forceinline__ void load4(const T* p, size_t base, int64_t k, int64_t Kd, bool vec_ok, float (&v)[4]) {
  if (vec_ok && k + 4 <= Kd) {
    load4_vec<T>(p + base + k, v);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = (k + j < Kd) ? to_float<T>(p[base + k + j]) : 0.0f;
  }
}

// Finds the expert and row-tile of linear tile index `tile`; false when past the last tile.
__device__ bool locate_tile(const int32_t* offsets, int E, int tile, int tm, int* s_out /* shared [3] */) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int base = 0;
    int found_e = -1, found_mt = 0;
    for (int e0 = 0; e0 < E && found_e < 0; e0 += 32) {
      int e = e0 + lane;
      int n = (e < E) ? offsets[e + 1] - offsets[e] : 0;
      int tiles = (n + tm - 1) / tm;
      int incl = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      int lo = base + incl - tiles, hi = base + incl;
      unsigned hit = __ballot_sync(0xffffffffu, tile >= lo && tile < hi);
      if (hit) {
        int src = __ffs(hit) - 1;
        found_e = __shfl_sync(0xffffffffu, e, src);
        found_mt = tile - __shfl_sync(0xffffffffu, lo, src);
      }
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) { s_out[0] = found_e; s_out[1] = found_mt; }
  }
  __syncthreads();
  return s_out[0] >= 0;
}

template <typename T, bool SWIGLU>
__global__ void __launch_bounds__(G_THREADS)
grouped_gemm_generic(const T* __restrict__ a, const T* __restrict__ w, const int32_t* __restrict__ offsets,
                     int E, int period, int64_t N, int64_t Kd, int vec_ok, T* __restrict__ out) {
  // w is [E, N, Kd]; with SWIGLU it is [E, 2N, Kd] (gate rows, then up rows) and out is [S, N].
  __shared__ __align__(16) float As[G_KC][G_PITCH];
  __shared__ __align__(16) float Bs[SWIGLU ? 2 : 1][G_KC][G_PITCH];
  __shared__ int loc[3];
  if (!locate_tile(offsets, E, blockIdx.x, G_TM, loc)) return;
  const int e = loc[0];
  const int64_t row_lo = offsets[e] + (int64_t)loc[1] * G_TM;
  const int64_t row_hi = offsets[e + 1];
  const int64_t n0 = (int64_t)blockIdx.y * G_TN;

  const int tid = threadIdx.x;
  const int ty = tid >> 4, tx = tid & 15;
  const int lr = tid >> 2, lk = (tid & 3) * 4;   // loader: row/col lr of the tile, 4 k values

  const bool a_in = row_lo + lr < row_hi;
  const bool b_in = n0 + lr < N;
  const size_t a_base = (size_t)(row_lo + lr) * Kd;
  const int64_t w_rows = SWIGLU ? 2 * N : N;
  const size_t b_base = ((size_t)(e % period) * w_rows + n0 + lr) * Kd;
  const size_t b2_base = b_base + (size_t)N * Kd;

  float acc[SWIGLU ? 2 : 1][4][4];
#pragma unroll
  for (int p = 0; p < (SWIGLU ? 2 : 1); ++p)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[p][i][j] = 0.0f;

  for (int64_t k0 = 0; k0 < Kd; k0 += G_KC) {
    float va[4] = {0, 0, 0, 0}, vb[4] = {0, 0, 0, 0}, vb2[4] = {0, 0, 0, 0};
    if (a_in) load4<T>(a, a_base, k0 + lk, Kd, vec_ok, va);
    if (b_in) {
      load4<T>(w, b_base, k0 + lk, Kd, vec_ok, vb);
      if (SWIGLU) load4<T>(w, b2_base, k0 + lk, Kd, vec_ok, vb2);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      As[lk + j][lr] = va[j];
      Bs[0][lk + j][lr] = vb[j];
      if (SWIGLU) Bs[1][lk + j][lr] = vb2[j];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < G_KC; ++k) {
      float4 av = *reinterpret_cast<const float4*>(&As[k][4 * ty]);
      const float aa[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int p = 0; p < (SWIGLU ? 2 : 1); ++p) {
        float4 bv = *reinterpret_cast<const float4*>(&Bs[p][k][4 * tx]);
        const float bb[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[p][i][j] = fmaf(aa[i], bb[j], acc[p][i][j]);
      }
    }
    __syncthreads();
  }

#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t r = row_lo + 4 * ty + i;
    if (r >= row_hi) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t n = n0 + 4 * tx + j;
      if (n >= N) continue;
      float v = SWIGLU ? swiglu_rounded<T>(acc[0][i][j], acc[SWIGLU ? 1 : 0][i][j]) : acc[0][i][j];
      out[r * N + n] = from_float<T>(v);
    }
  }
}

// Groups of few rows (generic_small_groups): tiles of 16 rows x 32 columns, so that a small layer spreads over the
// whole GPU, and 128 k at a time through registers into shared memory, the next 128 already on their way.  A layer of
// these sizes is bound by the latency of its K loop: with the 64 x 64 tiles above and 16 k per round trip the two
// projections of an fp32 layer of 64 tokens (8 experts, 256 x 512) took 23.5 and 33.6 us.
// 256 threads = 4 quarters of a chunk's K x (8 row pairs x 8 column quads); the quarters meet in shared memory at the
// end, added in order.
constexpr int GS_TM = 16, GS_TN = 32, GS_KC = 128, GS_PITCH = GS_KC + 4, GS_THREADS = 256, GS_KQ = GS_THREADS / 64;

// VEC: rows of 4-element pieces (Kd a multiple of 4, 16-byte aligned tensors).
template <typename T, bool SWIGLU, bool VEC>
__global__ void __launch_bounds__(GS_THREADS, 2)
grouped_gemm_small(const T* __restrict__ a, const int32_t* __restrict__ perm, int top_k, const T* __restrict__ w,
                   const int32_t* __restrict__ offsets, int E, int period, int64_t N, int64_t Kd,
                   T* __restrict__ out) {
  constexpr int NP = SWIGLU ? 2 : 1;
  constexpr int WROWS = NP * GS_TN, ROWS = GS_TM + WROWS;       // rows of a chunk: tokens, then weight rows
  constexpr int PER = ROWS * (GS_KC / 4) / GS_THREADS;          // 4-element pieces per thread and chunk
  __shared__ __align__(16) float sm[ROWS][GS_PITCH];
  __shared__ int loc[3];
  if (!locate_tile(offsets, E, blockIdx.x, GS_TM, loc)) return;
  const int e = loc[0];
  const int64_t row_lo = offsets[e] + (int64_t)loc[1] * GS_TM;
  const int rows = (int)min((int64_t)GS_TM, offsets[e + 1] - row_lo);
  const int64_t n0 = (int64_t)blockIdx.y * GS_TN;
  const int tid = threadIdx.x, kq = tid >> 6, rp = (tid >> 3) & 7, cq = tid & 7;
  const int64_t w_rows = (int64_t)NP * N;

  // piece p of a chunk = row p / 32, k 4 (p % 32): this thread's pieces lie in rows tid / 32 + 8 i
  const int pk = 4 * (tid & 31), pr = tid >> 5;
  // Rows past the tile's last repeat a valid one: computed, not stored.  All loads of a chunk are then unconditional
  // and in flight together (as ten conditional loads they took ten round trips to L2).
  const T* src[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int r = pr + 8 * i;
    if (r < GS_TM) {
      const int64_t row = row_lo + min(r, rows - 1);
      src[i] = a + (size_t)(perm != nullptr ? perm[row] / top_k : row) * Kd;
    } else {
      const int wr = r - GS_TM, p = wr / GS_TN;
      const int64_t n = min(n0 + wr % GS_TN, N - 1);
      src[i] = w + ((size_t)(e % period) * w_rows + (size_t)p * N + n) * Kd;
    }
  }
  float next[PER][4];
  auto fetch = [&](int64_t k0) {
    const int64_t k = k0 + pk;
    if (VEC) {
      const int64_t kc = k < Kd ? k : 0;
#pragma unroll
      for (int i = 0; i < PER; ++i) load4_vec<T>(src[i] + kc, next[i]);
      if (k >= Kd) {
#pragma unroll
        for (int i = 0; i < PER; ++i) next[i][0] = next[i][1] = next[i][2] = next[i][3] = 0.0f;
      }
    } else {
#pragma unroll
      for (int i = 0; i < PER; ++i) load4<T>(src[i], 0, k, Kd, false, next[i]);
    }
  };
  float acc[NP][2][4];
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[p][i][j] = 0.0f;

  fetch(0);
  for (int64_t k0 = 0; k0 < Kd; k0 += GS_KC) {
#pragma unroll
    for (int i = 0; i < PER; ++i)
      *reinterpret_cast<float4*>(&sm[pr + 8 * i][pk]) = make_float4(next[i][0], next[i][1], next[i][2], next[i][3]);
    __syncthreads();
    if (k0 + GS_KC < Kd) fetch(k0 + GS_KC);
#pragma unroll 4
    for (int k4 = 0; k4 < GS_KC / 4 / GS_KQ; ++k4) {
      const int k = kq * (GS_KC / GS_KQ) + 4 * k4;
      float4 av[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) av[i] = *reinterpret_cast<const float4*>(&sm[rp + 8 * i][k]);
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 bv = *reinterpret_cast<const float4*>(&sm[GS_TM + p * GS_TN + cq + 8 * j][k]);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            float v = acc[p][i][j];
            v = fmaf(av[i].x, bv.x, v);
            v = fmaf(av[i].y, bv.y, v);
            v = fmaf(av[i].z, bv.z, v);
            acc[p][i][j] = fmaf(av[i].w, bv.w, v);
          }
        }
    }
    __syncthreads();
  }
  // the other quarters hand their sums over
  float* red = &sm[0][0];                                        // [quarter - 1][value][64 threads]
  if (kq > 0) {
#pragma unroll
    for (int v = 0; v < NP * 8; ++v)
      red[((kq - 1) * NP * 8 + v) * 64 + (tid & 63)] = acc[v >> 3][(v >> 2) & 1][v & 3];
  }
  __syncthreads();
  if (kq > 0) return;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (rp + 8 * i >= rows) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t n = n0 + cq + 8 * j;
      if (n >= N) continue;
      float v[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        v[p] = acc[p][i][j];
#pragma unroll
        for (int q = 0; q < GS_KQ - 1; ++q) v[p] += red[((q * NP + p) * 8 + i * 4 + j) * 64 + tid];
      }
      out[(row_lo + rp + 8 * i) * N + n] = from_float<T>(SWIGLU ? swiglu_rounded<T>(v[0], v[NP - 1]) : v[0]);
    }
  }
}

template <typename T>
int launch_small(const void* a, const int32_t* perm, int64_t top_k, const void* w, const int32_t* offsets, int64_t S,
                 int64_t E, int64_t period, int64_t N, int64_t Kd, bool swiglu, void* out, cudaStream_t st) {
  const dim3 grid((unsigned)((S + GS_TM - 1) / GS_TM + (E < S ? E : S)), (unsigned)((N + GS_TN - 1) / GS_TN));
  const bool vec = (Kd % 4 == 0) && aligned16(a) && aligned16(w);
  auto go = [&](auto kernel) {
    kernel<<<grid, GS_THREADS, 0, st>>>(reinterpret_cast<const T*>(a), perm, (int)top_k, reinterpret_cast<const T*>(w),
                                        offsets, (int)E, (int)period, N, Kd, reinterpret_cast<T*>(out));
  };
  if (swiglu) vec ? go(grouped_gemm_small<T, true, true>) : go(grouped_gemm_small<T, true, false>);
  else vec ? go(grouped_gemm_small<T, false, true>) : go(grouped_gemm_small<T, false, false>);
  return check_launch();
}

template <typename T>
int launch_generic(const void* a, const void* w, const int32_t* offsets, int64_t S, int64_t E, int64_t period,
                   int64_t N, int64_t Kd, bool swiglu, void* out, cudaStream_t st) {
  const int64_t tiles = (S + G_TM - 1) / G_TM + E;
  dim3 grid((unsigned)tiles, (unsigned)((N + G_TN - 1) / G_TN));
  const int vec_ok = (Kd % 4 == 0) && aligned16(a) && aligned16(w);
  if (swiglu)
    grouped_gemm_generic<T, true><<<grid, G_THREADS, 0, st>>>(reinterpret_cast<const T*>(a),
        reinterpret_cast<const T*>(w), offsets, (int)E, (int)period, N, Kd, vec_ok, reinterpret_cast<T*>(out));
  else
    grouped_gemm_generic<T, false><<<grid, G_THREADS, 0, st>>>(reinterpret_cast<const T*>(a),
        reinterpret_cast<const T*>(w), offsets, (int)E, (int)period, N, Kd, vec_ok, reinterpret_cast<T*>(out));
  return check_launch();
}

}  // namespace

// Whether the small-group kernel takes these sizes: at most 32 rows per group on average (more rows fill the 64-row
// tiles well enough to need a quarter of the weight reads), and fewer where there are groups enough for the 64-row tiles
// to fill the GPU.  us, 64-row | 16-row tiles, fp32, K 256, N 512.  Plain: 32 groups of 32 rows 35.6 | 27.6; 64 of 24
// 48.5 | 40.3, of 28 42.0 | 43.9; 128 of 24 86 | 84, of 32 86 | 101; 256 of 16 142 | 138, of 20 143 | 161.  Fused: 32 of 32
// 52.4 | 45.3; 64 of 28 98 | 73; 96 of 28 104 | 110; 128 of 32 150 | 163; 256 of 20 254 | 247, of 24 255 | 280.
bool generic_small_groups(int64_t S, int64_t E, int64_t N, bool swiglu) {
  const bool few = S <= 1024 || (swiglu ? S <= 28 * E && S <= 5120 : S <= 24 * E && S <= 4096);
  return S <= 32 * E && few && (N + GS_TN - 1) / GS_TN <= 65535;
}

// perm (small groups only): row p is a[perm[p] / top_k].
int grouped_gemm_generic_dispatch(const void* a, const void* w, const int32_t* offsets, int64_t S, int64_t E,
                                  int64_t period, int64_t N, int64_t Kd, int dtype, bool swiglu, void* out,
                                  cudaStream_t st, const int32_t* perm, int64_t top_k) {
  if (generic_small_groups(S, E, N, swiglu)) {
    if (dtype == MQ_F32) return launch_small<float>(a, perm, top_k, w, offsets, S, E, period, N, Kd, swiglu, out, st);
    if (dtype == MQ_BF16)
      return launch_small<__nv_bfloat16>(a, perm, top_k, w, offsets, S, E, period, N, Kd, swiglu, out, st);
    return launch_small<__half>(a, perm, top_k, w, offsets, S, E, period, N, Kd, swiglu, out, st);
  }
  if (perm != nullptr) return MQ_ERR_UNSUPPORTED_SHAPE;
  if (dtype == MQ_F32) return launch_generic<float>(a, w, offsets, S, E, period, N, Kd, swiglu, out, st);
  if (dtype == MQ_BF16) return launch_generic<__nv_bfloat16>(a, w, offsets, S, E, period, N, Kd, swiglu, out, st);
  return launch_generic<__half>(a, w, offsets, S, E, period, N, Kd, swiglu, out, st);
}

}  // namespace mq
