// W4A16 grouped GEMM for prefill-size groups on the 5th-generation tensor cores:
//   out[r, n] = bf16( sum_k x[r,k] * (q[e][k,n] - z[e][k/128, n]) * s[e][k/128, n] ),  rows r of group e,
// optionally two projections with SwiGLU.  Format and arithmetic follow mini_qwen/kernels/w4a16_gemm.py:8-15 of the
// reference (fp32 sums, one rounding of the result); the rows of an expert as in mini_qwen/model/layers/moe.py:59-65.
//
// What bounds it: a tile of 128 tokens costs the tensor core 512 cycles per 128 columns x 128 k, in which 16 K
// weights have to be unpacked by the CUDA cores and, because a scale belongs to (128 k, column), 16 K sums have to
// be folded into fp32 master sums.  Everything is laid out so that both fit under the MMAs:
//   * output columns are the TMEM lanes (M = 128), tokens are N: a thread owns one column, its scale is a scalar;
//   * a UNIT is 128 columns x 128 k.  Its 16 x 128 packed words come by TMA straight from the checkpoint layout with
//     the unit's scales and zero points.  Two sets of four warps unpack alternate units (a byte permute
//     and a packed FMA per pair of weights and three logic ops per word give q - z exactly, in natural k order) and write them to TENSOR MEMORY,
//     from where the MMA takes its A operand;
//   * the unit's sum lands in one of two TMEM accumulators; eight fold warps add scale * sum to 2 x 64 (tokens)
//     master sums per thread with packed fp32 FMAs while the other accumulator is being computed.  The dequantised
//     weight is never rounded;
//   * the token rows come by TMA, or, gathered through the permutation, by two warps' 16-byte asynchronous copies.
// Unpacking, MMAs and folding are separate warps because each is a chain of latencies (barrier, shared or tensor
// memory, arithmetic, barrier) of several hundred cycles: in one set of warps they ran one after the other and a
// unit took 2000 cycles.
// Modes: SWIGLU folds gate and up of the same 128 columns; WIDE two neighbouring 128-column tiles (a token tile is
// then fetched once for 256 columns); NARROW one tile (more CTAs where columns x tokens leave SMs idle).
// Register shares of the five warpgroups: 3 x 40 + 2 x 176 (the masters), within the launch's 5 x 96.
#include <cmath>

#include "tc5.cuh"

namespace mq {
namespace {

using namespace tc5;

constexpr int TL_M = 128;                        // output columns of a unit = TMEM lanes
constexpr int TL_K = 128;                        // k of a unit = one quantisation group
constexpr int TL_TN = 128;                       // most tokens per tile
constexpr int TL_WORDS = (TL_K / 8) * TL_M * 4;  // 8 KB of packed words
constexpr int TL_SC_OFF = TL_WORDS;              // then 256 bytes of scales, 64 bytes of zero points
constexpr int TL_QZ_OFF = TL_SC_OFF + 2 * TL_M;
constexpr int TL_WSLOT = TL_WORDS + 512;
constexpr int TL_NW = 10;                        // units in the weight ring
constexpr int TL_XATOM = TL_TN * 128;            // token rows of 64 k
constexpr int TL_XSLOT = 2 * TL_XATOM;           // a group's 128 k: 32 KB
constexpr int TL_NX = 4;
constexpr int TL_XBOX = 32;                      // token rows per TMA box
constexpr int TL_MAX_E = 1024;
constexpr int TL_TABLE = 2 * (TL_MAX_E + 1) * 4;
constexpr int TL_BARS = 512;
constexpr int TL_ROWS = 2 * TL_TN * 4;          // where a tile's token rows lie, two tiles
constexpr int TL_SMEM = TL_NX * TL_XSLOT + TL_NW * TL_WSLOT + TL_BARS + TL_ROWS + ((TL_TABLE + 15) & ~15) + 1024;
constexpr int TL_THREADS = 640;
constexpr int TL_A_COL = 256;                    // TMEM: two accumulators of 128 columns, then four A buffers of 64

// SWIGLU_EXACT: SWIGLU with expf and a true quotient, for the calls that had them on the cp.async kernel (the stream
// kernel's SwiGLU has the approximations).
enum TileMode { TILE_SWIGLU, TILE_SWIGLU_EXACT, TILE_WIDE, TILE_NARROW };
__host__ __device__ constexpr bool tile_swiglu(int mode) { return mode == TILE_SWIGLU || mode == TILE_SWIGLU_EXACT; }

struct TileProj {
  const __nv_bfloat16* sc;                       // [period, G, N]
  const int32_t* qz;                             // [period, G, N/8]
};
struct TileParams {
  const __nv_bfloat16* x;                        // token rows [*, Kd]
  const int32_t* perm;                           // optional: sorted row p is x[perm[p] / top_k]
  int top_k;
  const int32_t* offsets;                        // [E + 1], or null: one group of all S rows
  int S;
  int E, period, N, Kd, tn;                      // tn: most tokens per tile (a multiple of 16)
  TileProj p0, p1;
  __nv_bfloat16* out;                            // [*, N]
  int32_t* d_status;
};

// A tile of work: 128 (256: WIDE) columns from n0, the token rows [tok0, tok0 + ntok) of one group.
struct TileWork {
  int expert, n0, tok0, ntok, n_mma;
};

struct TileTable {
  const int* off;                                // [E + 1]
  const int* first;                              // [E + 1]: first tile of the group
  int E, nwt, cols, tn;
  __device__ TileWork locate(int t) const {
    int lo = 0, hi = E;                          // first[lo] <= t < first[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (first[mid] <= t) lo = mid; else hi = mid;
    }
    const int n = off[lo + 1] - off[lo], local = t - first[lo];
    const int ntt = (n + tn - 1) / tn;
    const int width = (((n + ntt - 1) / ntt) + 15) & ~15;      // balanced token tiles
    const int tt = local / nwt;
    TileWork w;
    w.expert = lo;
    w.n0 = (local - tt * nwt) * cols;
    w.tok0 = off[lo] + tt * width;
    w.ntok = min(width, n - tt * width);
    w.n_mma = (w.ntok + 15) & ~15;
    return w;
  }
};

template <int MODE, bool GATHER>
__global__ void __launch_bounds__(TL_THREADS, 1)
w4a16_tile_kernel(const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                  const __grid_constant__ CUtensorMap map_x, const TileParams P) {
  constexpr int NSUB = MODE == TILE_NARROW ? 1 : 2;             // units per quantisation group
  extern __shared__ uint8_t tl_smem_raw[];
  const uint32_t raw = smem_addr(tl_smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;                 // the swizzle pattern repeats every 1024 bytes
  uint8_t* ptr = tl_smem_raw + (base - raw);
  const uint32_t wring = base + TL_NX * TL_XSLOT;
  const uint8_t* wptr = ptr + TL_NX * TL_XSLOT;
  const uint32_t bars = wring + TL_NW * TL_WSLOT;
  uint8_t* bar_mem = ptr + TL_NX * TL_XSLOT + TL_NW * TL_WSLOT;
  uint32_t* s_rows = reinterpret_cast<uint32_t*>(bar_mem + TL_BARS);
  int* s_off = reinterpret_cast<int*>(bar_mem + TL_BARS + TL_ROWS);
  int* s_first = s_off + P.E + 1;
  auto wfull = [&](int s) { return bars + 8u * s; };
  auto wempty = [&](int s) { return bars + 8u * (TL_NW + s); };
  auto xfull = [&](int s) { return bars + 8u * (2 * TL_NW + s); };
  auto xempty = [&](int s) { return bars + 8u * (2 * TL_NW + TL_NX + s); };
  constexpr int B0 = 2 * TL_NW + 2 * TL_NX;
  auto afull = [&](int b) { return bars + 8u * (B0 + b); };     // 4 A buffers
  auto done = [&](int b) { return bars + 8u * (B0 + 4 + b); };  // 2 accumulators
  auto dempty = [&](int b) { return bars + 8u * (B0 + 6 + b); };
  auto aempty = [&](int b) { return bars + 8u * (B0 + 8 + b); };
  static_assert(8 * (B0 + 12) + 16 <= TL_BARS, "barriers fit their space");
  volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(bar_mem + 8 * (B0 + 12));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_mem + 8 * (B0 + 12) + 8);

  const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int E = P.E, N = P.N, Kd = P.Kd, G = Kd / TL_K;
  constexpr int COLS = MODE == TILE_WIDE ? 2 * TL_M : TL_M;
  const int nwt = (N + COLS - 1) / COLS;

  if (threadIdx.x == 0) {
    for (int s = 0; s < TL_NW; ++s) { mbar_init(wfull(s), 1); mbar_init(wempty(s), 8); }
    for (int s = 0; s < TL_NX; ++s) { mbar_init(xfull(s), GATHER ? 64 : 1); mbar_init(xempty(s), 1); }
    for (int b = 0; b < 4; ++b) { mbar_init(afull(b), 4); mbar_init(aempty(b), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(done(b), 1); mbar_init(dempty(b), 8); }
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(smem_addr((const void*)tmem_ptr), 512u);
  for (int e = threadIdx.x; e <= E; e += TL_THREADS) s_off[e] = P.offsets != nullptr ? P.offsets[e] : e * P.S;
  __syncthreads();
  if (warp == 0) {                                              // first[]: exclusive sums of the groups' tile counts
    int carry = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const int c = e < E ? (s_off[e + 1] - s_off[e] + P.tn - 1) / P.tn * nwt : 0;
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (e < E) s_first[e] = carry + incl - c;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_first[E] = carry;
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = uniform(*tmem_ptr);
  const TileTable table{s_off, s_first, E, nwt, COLS, P.tn};
  const int total = s_first[E];
  const int grid = (int)gridDim.x;
  const int n_tiles = total > (int)blockIdx.x ? (total - (int)blockIdx.x + grid - 1) / grid : 0;
  const int U = G * NSUB;                                       // units per tile

  if (warp < 4) {
    regs_give<40>();
    if (warp == 0 && lane == 0) {
      // ---------------------------------------------------------------- weights: words, scales, zero points
      int slot = 0, filled = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = 0; i < n_tiles && ok; ++i) {
        const TileWork w = table.locate(blockIdx.x + i * grid);
        const int we = w.expert % P.period;
        for (int u = 0; u < U; ++u) {
          const int g = NSUB == 2 ? u >> 1 : u, sub = NSUB == 2 ? u & 1 : 0;
          const int n0 = w.n0 + (MODE == TILE_WIDE ? sub * TL_M : 0);
          const TileProj& p = (tile_swiglu(MODE) && sub) ? P.p1 : P.p0;
          ok = mbar_wait(wempty(slot), phase ^ 1u, abort_flag, P.d_status);
          if (!ok) break;
          const uint32_t dst = wring + slot * TL_WSLOT;
          const int cols = max(0, min(TL_M, N - n0));           // a multiple of 32
          mbar_expect_tx(wfull(slot), (uint32_t)(TL_WORDS + 2 * cols + cols / 2));
          tma_load_2d(dst, (tile_swiglu(MODE) && sub) ? &map_w1 : &map_w0, wfull(slot), n0, (we * G + g) * (TL_K / 8));
          if (cols > 0) {
            const size_t row = (size_t)we * G + g;
            bulk_load(dst + TL_SC_OFF, p.sc + row * N + n0, 2 * cols, wfull(slot));
            bulk_load(dst + TL_QZ_OFF, p.qz + row * (N / 8) + n0 / 8, cols / 2, wfull(slot));
          }
          ++filled;
          if (++slot == TL_NW) { slot = 0; phase ^= 1u; }
        }
      }
      if (!ok) {                                                // gave up: let the copies in flight land first
        for (int f = max(0, filled - TL_NW); f < filled; ++f)
          mbar_wait_limited(wfull(f % TL_NW), (uint32_t)(f / TL_NW) & 1u, 1u << 16);
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer
      // The whole warp walks the loop and one elected lane issues: addresses and descriptors then stay in uniform
      // registers (with a single lane in the loop every MMA cost the issuing thread about 100 cycles).
      const bool leader = elect_one();
      const int total_units = n_tiles * U;
      int xs = 0, u = 0;                                        // ring slot of the unit's token rows; unit inside the tile
      uint32_t xphase = 0;
      uint32_t idesc = 0;
      bool ok = true;
      int tile = 0;
      for (int uc = 0; uc < total_units; ++uc) {
        if (u == 0) idesc = uniform(idesc_bf16(TL_M, table.locate(blockIdx.x + tile * grid).n_mma));
        const int b = uc & 1;
        if (NSUB == 1 || (u & 1) == 0) ok = mbar_wait_warp(xfull(xs), xphase, abort_flag, P.d_status);
        ok = ok && mbar_wait_warp(afull(uc & 3), (uint32_t)(uc >> 2) & 1u, abort_flag, P.d_status) &&
             mbar_wait_warp(dempty(b), ((uint32_t)(uc >> 1) & 1u) ^ 1u, abort_flag, P.d_status);
        if (!ok) break;
        fence_after_sync();
        const uint32_t d = tmem + b * TL_TN, a = tmem + TL_A_COL + (uc & 3) * 64;
        const uint64_t xd = smem_desc(base + xs * TL_XSLOT);
        const bool group_ends = NSUB == 1 || (u & 1) != 0;
        if (leader) {
#pragma unroll
          for (int k = 0; k < TL_K / 16; ++k)
            mma_ts(d, a + 8 * k, xd + (uint64_t)((k >> 2) * (TL_XATOM >> 4) + 2 * (k & 3)), idesc, k != 0 ? 1u : 0u);
          mma_commit(done(b));
          mma_commit(aempty(uc & 3));
          if (group_ends) mma_commit(xempty(xs));
        }
        __syncwarp();
        if (group_ends && ++xs == TL_NX) { xs = 0; xphase ^= 1u; }
        if (++u == U) { u = 0; ++tile; }
      }
    } else if (!GATHER && warp == 2) {
      // ---------------------------------------------------------------- token rows, contiguous: by TMA
      if (lane == 0) {
        int xs = 0;
        uint32_t xphase = 0;
        bool ok = true;
        for (int i = 0; i < n_tiles && ok; ++i) {
          const TileWork w = table.locate(blockIdx.x + i * grid);
          const int nbox = (w.n_mma + TL_XBOX - 1) / TL_XBOX;   // rows past the tile's last: computed, not stored
          for (int g = 0; g < G; ++g) {
            ok = mbar_wait(xempty(xs), xphase ^ 1u, abort_flag, P.d_status);
            if (!ok) break;
            const uint32_t dst = base + xs * TL_XSLOT;
            mbar_expect_tx(xfull(xs), (uint32_t)(nbox * 2 * TL_XBOX * 128));
            for (int r = 0; r < nbox; ++r) {
              tma_load_2d(dst + r * TL_XBOX * 128, &map_x, xfull(xs), g * TL_K, w.tok0 + r * TL_XBOX);
              tma_load_2d(dst + TL_XATOM + r * TL_XBOX * 128, &map_x, xfull(xs), g * TL_K + 64, w.tok0 + r * TL_XBOX);
            }
            if (++xs == TL_NX) { xs = 0; xphase ^= 1u; }
          }
        }
        if (!ok) {                                              // gave up: let the copies in flight land first
          for (int f = 0; f < TL_NX; ++f) mbar_wait_limited(xfull(f), 0u, 1u << 12), mbar_wait_limited(xfull(f), 1u, 1u << 12);
        }
      }
    } else if (GATHER && warp >= 2) {
      // ---------------------------------------------------------------- token rows
      // Thread = one 16-byte piece (8 k) of rows r0, r0 + 4, ...; 16 neighbouring threads copy 256 contiguous bytes.
      // s_rows holds where the tile's rows lie (in 16-byte pieces of x), transposed so that a thread reads four of
      // its rows at once; a warp looks up the rows that it copies itself (r0 = 0, 1 or 2, 3), so that neither warp
      // ever waits for the other, which may have given up.  Two tables in turn: a lane may still read the last tile's.
      const int th = threadIdx.x - 64, piece = th & 15, r0 = th >> 4;
      const uint4* xv = reinterpret_cast<const uint4*>(P.x) + piece;
      int xs = 0, pending = 0, pslot = 0;                       // groups copied but not yet announced, the oldest's slot
      uint32_t xphase = 0;
      bool ok = true;
      TileWork w = {}, wn = {};
      const int own = 2 * (warp - 2) + (lane & 1);              // this lane looks up rows own + 4 (lane / 2), + 64
      int at[2];                                                // of the next tile
      auto fetch_rows = [&](const TileWork& t) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = own + 4 * (lane >> 1) + 64 * h;
          at[h] = P.perm[t.tok0 + min(r, t.ntok - 1)];          // rows past the last repeat it: computed, not stored
        }
      };
      if (n_tiles > 0) {
        wn = table.locate(blockIdx.x);
        fetch_rows(wn);
      }
      for (int i = 0; i < n_tiles && ok; ++i) {
        w = wn;
        uint32_t* rows = s_rows + (i & 1) * TL_TN;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          rows[own * (TL_TN / 4) + (lane >> 1) + 16 * h] = (uint32_t)(at[h] / P.top_k) * (uint32_t)(Kd / 8);
        __syncwarp();
        if (i + 1 < n_tiles) {
          wn = table.locate(blockIdx.x + (i + 1) * grid);
          fetch_rows(wn);                                       // its latency passes under this tile's copies
        }
        for (int g = 0; g < G; ++g) {
          ok = mbar_wait_warp(xempty(xs), xphase ^ 1u, abort_flag, P.d_status);
          if (!ok) break;
          // row r0 + 4 j lands at 128 (r0 + 4 j), its piece exchanged with (row & 7): two patterns, by j's parity
          const uint32_t dst = base + xs * TL_XSLOT + (piece >> 3) * TL_XATOM + r0 * 128;
          const uint32_t dst0 = dst + (((piece & 7) ^ r0) << 4), dst1 = dst + (((piece & 7) ^ (r0 + 4)) << 4) + 512;
          const uint4* xg = xv + g * (TL_K / 8);
#pragma unroll
          for (int j4 = 0; j4 < TL_TN / 16; ++j4) {
            if (16 * j4 < w.n_mma) {
              const uint4 src = *reinterpret_cast<const uint4*>(rows + r0 * (TL_TN / 4) + 4 * j4);
              cp_async16(dst0 + 2048 * j4, xg + src.x);
              cp_async16(dst1 + 2048 * j4, xg + src.y);
              cp_async16(dst0 + 2048 * j4 + 1024, xg + src.z);
              cp_async16(dst1 + 2048 * j4 + 1024, xg + src.w);
            }
          }
          cp_async_commit();
          if (++pending == TL_NX - 1) {                         // the oldest group in flight has landed
            cp_async_wait<TL_NX - 2>();
            fence_proxy_async();
            mbar_arrive(xfull(pslot));
            if (++pslot == TL_NX) pslot = 0;
            --pending;
          }
          if (++xs == TL_NX) { xs = 0; xphase ^= 1u; }
        }
      }
      cp_async_wait<0>();
      fence_proxy_async();
      for (; ok && pending > 0; --pending) {
        mbar_arrive(xfull(pslot));
        if (++pslot == TL_NX) pslot = 0;
      }
    }
  } else if (warp < 12) {
    regs_give<40>();
    // ------------------------------------------------------------------ unpack (warps 4..7: even units, 8..11: odd)
    const int quad = warp & 3, set = (warp - 4) >> 2;
    const int col = quad * 32 + lane;                           // this thread's column inside a unit
    const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
    const int total_units = n_tiles * U;
    int slot = set;
    uint32_t phase = 0;
    for (int q = set; q < total_units; q += 2) {
      if (!mbar_wait_warp(wfull(slot), phase, abort_flag, P.d_status) ||
          !mbar_wait_warp(aempty(q & 3), ((uint32_t)(q >> 2) & 1u) ^ 1u, abort_flag, P.d_status))
        break;
      fence_after_sync();
      const uint8_t* s = wptr + slot * TL_WSLOT;
      const uint32_t* words = reinterpret_cast<const uint32_t*>(s) + col;
      const uint32_t a = lanes + TL_A_COL + (q & 3) * 64;
      uint32_t w[4], wn[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = words[j * TL_M];
      // -z / 64 in both halves
      const uint32_t z = (reinterpret_cast<const uint32_t*>(s + TL_QZ_OFF)[col >> 3] >> (4 * (col & 7))) & 15u;
      const __nv_bfloat162 nz2 = __float2bfloat162_rn((float)z * -0.015625f);
      const uint32_t nz = *reinterpret_cast<const uint32_t*>(&nz2);
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        if (h < 3) {
#pragma unroll
          for (int j = 0; j < 4; ++j) wn[j] = words[(4 * h + 4 + j) * TL_M];
        }
        uint32_t r[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t even = w[j] & 0x0F0F0F0Fu, odd = (w[j] >> 4) & 0x0F0F0F0Fu;
          // Byte p of both side by side, the other bytes zero (the permute's sign mode: a nibble's byte has sign 0):
          // read as bf16 these are the subnormals q * 2^-133, which the FMA turns into (q - z) / 64 exactly.
          asm("prmt.b32 %0, %1, %2, 0xC480;" : "=r"(r[4 * j + 0]) : "r"(even), "r"(odd));
          asm("prmt.b32 %0, %1, %2, 0xD591;" : "=r"(r[4 * j + 1]) : "r"(even), "r"(odd));
          asm("prmt.b32 %0, %1, %2, 0xE6A2;" : "=r"(r[4 * j + 2]) : "r"(even), "r"(odd));
          asm("prmt.b32 %0, %1, %2, 0xF7B3;" : "=r"(r[4 * j + 3]) : "r"(even), "r"(odd));
        }
#pragma unroll
        for (int i = 0; i < 16; ++i)
          asm("fma.rn.bf16x2 %0, %0, %1, %2;" : "+r"(r[i]) : "r"(0x7F007F00u), "r"(nz));
        tmem_st16(a + 16 * h, r);
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = wn[j];
      }
      tmem_st_wait();
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(afull(q & 3));
      slot += 2;
      if (slot >= TL_NW) { slot -= TL_NW; phase ^= 1u; }
    }
  } else {
    regs_take<176>();
    // ------------------------------------------------------------------ fold and store (warps 12..19)
    const int quad = warp & 3, half = (warp - 12) >> 2;
    const int col = quad * 32 + lane;
    const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
    f32x2 master[NSUB][4][8];                                   // [unit of the group][32-token block][pair of tokens]
    const uint8_t* scales = wptr + TL_SC_OFF + 2 * col;
    bool ok = true;
    int uc = 0, slot = 0;
    for (int i = 0; i < n_tiles && ok; ++i) {
      const TileWork w = table.locate(blockIdx.x + i * grid);
#pragma unroll
      for (int s = 0; s < NSUB; ++s)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int j = 0; j < 8; ++j) master[s][c][j] = 0ull;
      for (int g = 0; g < G && ok; ++g) {
#pragma unroll
        for (int sub = 0; sub < NSUB; ++sub) {
          const int b = NSUB == 2 ? sub : uc & 1;               // with two units a group, the accumulator is the sub-tile's
          ok = ok && mbar_wait_warp(done(b), (uint32_t)(uc >> 1) & 1u, abort_flag, P.d_status);
          if (!ok) break;
          fence_after_sync();
          const uint32_t acc = lanes + b * TL_TN + 16 * half;
          f32x2 s = 0;
#pragma unroll
          for (int c2 = 0; c2 < 4; c2 += 2) {                   // two 16-token blocks in flight
            if (32 * c2 + 16 * half < w.n_mma) {
              uint32_t d0[16], d1[16];
              const bool second = 32 * (c2 + 1) + 16 * half < w.n_mma;
              tmem_ld16(acc + 32 * c2, d0);
              if (second) tmem_ld16(acc + 32 * (c2 + 1), d1);
              if (c2 == 0) {                                    // the unit's scale; the weights were multiplied as (q - z) / 64
                const float sc = 64.0f * __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(scales + slot * TL_WSLOT));
                s = pack2(sc, sc);
              }
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 8; ++j) fma2(master[sub][c2][j], pack2(d0[2 * j], d0[2 * j + 1]), s);
              if (second) {
#pragma unroll
                for (int j = 0; j < 8; ++j) fma2(master[sub][c2 + 1][j], pack2(d1[2 * j], d1[2 * j + 1]), s);
              }
            }
          }
          fence_before_sync();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(dempty(b));
            mbar_arrive(wempty(slot));
          }
          ++uc;
          if (++slot == TL_NW) slot = 0;
        }
      }
      if (!ok) break;
      // Neighbouring lanes (columns) swap one of every two tokens, so that a lane stores two columns of one token: a
      // warp's store covers 64 contiguous bytes of two rows.
      const int odd = lane & 1, n = w.n0 + (col & ~1);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int left = w.ntok - (32 * c + 16 * half) - odd;   // rows of this block from the lane's first one
        if (left + odd <= 0) continue;
        __nv_bfloat16* o = P.out + (size_t)(w.tok0 + 32 * c + 16 * half + odd) * N + n;
#pragma unroll
        for (int s = 0; s < (MODE == TILE_WIDE ? 2 : 1); ++s) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float2 v = unpack2(master[s][c][j]);
            if (tile_swiglu(MODE)) {
              const float2 u = unpack2(master[NSUB - 1][c][j]);
              if (MODE == TILE_SWIGLU_EXACT)
                v = make_float2(swiglu_rounded<__nv_bfloat16>(v.x, u.x), swiglu_rounded<__nv_bfloat16>(v.y, u.y));
              else
                v = make_float2(swiglu_fast(v.x, u.x), swiglu_fast(v.y, u.y));
            }
            const float other = __shfl_xor_sync(0xffffffffu, odd ? v.x : v.y, 1);
            const __nv_bfloat162 r = odd ? __floats2bfloat162_rn(other, v.y) : __floats2bfloat162_rn(v.x, other);
            if (2 * j < left && n + s * TL_M < N)
              *reinterpret_cast<__nv_bfloat162*>(o + (size_t)(2 * j) * N + s * TL_M) = r;
          }
        }
      }
    }
  }

  fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    fence_after_sync();
    tmem_dealloc(tmem, 512u);
  }
}

// qweight [period, Kd/8, N] as [period * Kd/8, N]: boxes of 16 word rows x 128 columns (columns past N read as zero)
bool tile_map(CUtensorMap* map, const void* qweight, int64_t rows, int64_t N) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)N * 4};
  cuuint32_t box[2] = {(cuuint32_t)TL_M, (cuuint32_t)(TL_K / 8)};
  cuuint32_t estr[2] = {1u, 1u};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<void*>(qweight), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// token rows [rows, Kd] bf16: boxes of 64 k x TL_XBOX rows, 128-byte swizzle (rows past the last read as zero)
bool tile_map_x(CUtensorMap* map, const void* x, int64_t rows, int64_t Kd) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)Kd, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)Kd * 2};
  cuuint32_t box[2] = {64u, (cuuint32_t)TL_XBOX};
  cuuint32_t estr[2] = {1u, 1u};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

bool w4a16_stream_covers(int64_t S, int64_t E, int64_t period, int64_t N, int64_t Kd, int64_t group);
int w4a16_stream_panels(int64_t S, int64_t E, int64_t N, bool swiglu);

namespace {

// How a call is cut into tiles.  Plain projection: 256 columns per tile as long as that leaves a tile for every SM;
// otherwise 128, and narrower token tiles while there is less than a tile per SM (a tile's time hardly depends on its
// tokens below 64).
struct TileShape {
  bool wide;
  int tn;                                        // most tokens per tile
  int64_t col_tiles;
};
// Most token tiles there can be in S rows, with tiles of tn tokens.
int64_t most_token_tiles(int64_t S, int64_t E, int64_t tn) { return (S + tn - 1) / tn + (E > 1 ? (E < S ? E : S) : 0); }
TileShape tile_shape(int64_t rows, int64_t E, int64_t N, bool swiglu, int sms) {
  auto token_tiles = [&](int64_t tn) { return most_token_tiles(rows, E, tn); };
  TileShape t;
  t.wide = !swiglu && token_tiles(TL_TN) * ((N + 255) / 256) >= sms;
  t.col_tiles = t.wide ? (N + 255) / 256 : (N + 127) / 128;
  t.tn = TL_TN;
  while (t.tn > 32 && token_tiles(t.tn) * t.col_tiles < sms && token_tiles(t.tn / 2) * t.col_tiles <= sms) t.tn /= 2;
  return t;
}

}  // namespace

// Whether this kernel is the faster one for `rows` rows in E groups (by the sizes alone; w4a16_tile_covers says whether
// it takes them).  It unpacks a weight once for up to 128 rows where the others do for every eight, but its units of 128
// columns x 128 k run one after the other: a tile takes half a microsecond a unit however few its rows.  So the two are
// compared by their times in us.  The figures are fits to 960 calls of 1 to 128 groups of over 8 to 100 rows (K and N 128
// to 4096, even and skewed).  Fused, as a block calls it: the slower kernel is chosen by more than 4 % for 6 of 261, by
// 15 % at most; by the eight rows alone for 32, up to 1.75 times as long (16 groups of 14 rows, K 2048, N 128: 12.2 us on
// the stream kernel, 21.4 on this; one group of 32 rows, N 768: 7.5 | 20.1).  Plain: for 20 of 697, most of them of K 128,
// where skewed groups, which a rule on sizes does not see, make the cp.async kernel up to 3.6 times slower.
// alternative: the fused projection's other kernel: 0 stream or (under 32 rows) cp.async, as the dispatch has it; 1 stream
// on activations that are prepared already; 2 stream after a launch that prepares them.
bool w4a16_tile_faster(int64_t rows, int64_t E, int64_t N, int64_t Kd, bool swiglu, int alternative) {
  if (rows <= 8 * E) return false;               // one block of eight rows a group: a weight is unpacked once anyway
  const int sms = device_sm_count();
  const TileShape t = tile_shape(rows, E, N, swiglu, sms);
  const double units = (double)(Kd / TL_K) * (swiglu || t.wide ? 2 : 1), k = (double)Kd;
  const int64_t group_tiles = E * ((rows + TL_TN * E - 1) / (TL_TN * E)) * t.col_tiles;      // groups of equal size
  const double rounds = (double)((group_tiles + sms - 1) / sms), per_group = (double)rows / (8.0 * E);
  const double blocks = ceil(E == 1 ? per_group : per_group + 0.55);       // of eight rows, in the larger groups
  if (swiglu) {
    const double tile = 3.0 + rounds * (0.55 * units + 2.0);
    if (rows < 32 && alternative == 0)           // the cp.async kernel, and an exact SwiGLU, which takes 1.5 us longer
      return tile + 1.5 < 2.3 + blocks * (1.7 + 0.0019 * k);
    // the stream kernel: items of eight rows x `panels` of 32 columns, dealt out to all SMs
    const int panels = w4a16_stream_panels(rows, E, N, true);
    const double items = (E == 1 ? ceil(per_group) : (per_group + 0.6) * E) * (double)((N / 32 + panels - 1) / panels);
    double waves = items / sms;
    waves = waves < 3.0 ? ceil(waves) : waves + 0.5;
    return tile < 3.0 + (alternative == 2 ? 2.0 : 0.0) + waves * (2.0 + 0.0013 * k * panels);
  }
  const double tile = 2.7 + rounds * (0.5 * units + 2.0), words = (double)N * k * E;
  if (rows <= 32)                                // the cp.async kernel with K split over four warps
    return tile < 2.3 + blocks * (1.1 + 0.0017 * k) + (E == 1 ? words / 7e6 : 0.0);
  // and without: a warp takes a group's blocks of eight rows one after the other
  const double even = 5.7 + 0.0025 * k + (per_group + 0.4) * words / 4.5e6, chain = 4.0 + (per_group + 0.5) * 0.006 * k;
  return tile < (even > chain ? even : chain);
}

bool w4a16_tile_covers(int64_t S, int64_t E, int64_t period, int64_t N, int64_t Kd, int64_t group) {
  return group == 128 && Kd % 128 == 0 && N % 32 == 0 && E <= TL_MAX_E && S < ((int64_t)1 << 30) &&
         period * (Kd / 8) < ((int64_t)1 << 31) && (S / 16 + E) * (N / 32) < ((int64_t)1 << 30);
}

// x: rows in natural k order, [S, Kd] or (perm) [x_rows, Kd] gathered by row = perm[p] / top_k.  `rows` of the S rows are
// expected to lie in the groups.
int w4a16_tile(const void* x, int64_t x_rows, const int32_t* perm, int64_t top_k, const int32_t* qw0, const void* sc0,
               const int32_t* qz0, const int32_t* qw1, const void* sc1, const int32_t* qz1, bool swiglu,
               const int32_t* offsets, int64_t S, int64_t rows, int64_t E, int64_t period, int64_t N, int64_t Kd,
               void* out, int32_t* d_status, cudaStream_t st) {
  if (x_rows * (Kd / 8) >= ((int64_t)1 << 32)) return MQ_ERR_UNSUPPORTED_SHAPE;
  if ((reinterpret_cast<uintptr_t>(qz0) & 15u) != 0 || (swiglu && (reinterpret_cast<uintptr_t>(qz1) & 15u) != 0))
    return MQ_ERR_INVALID_ARGUMENT;
  CUtensorMap map0, map1, mapx;
  const int64_t wrows = period * (Kd / 8);
  if (!tile_map(&map0, qw0, wrows, N) || !tile_map(&map1, swiglu ? qw1 : qw0, wrows, N) ||
      !tile_map_x(&mapx, x, x_rows, Kd))
    return MQ_ERR_DRIVER_ENTRY;
  TileParams P;
  P.x = reinterpret_cast<const __nv_bfloat16*>(x);
  P.perm = perm;
  P.top_k = (int)top_k;
  P.offsets = offsets;
  P.S = (int)S;
  P.E = (int)E;
  P.period = (int)period;
  P.N = (int)N;
  P.Kd = (int)Kd;
  P.p0 = TileProj{reinterpret_cast<const __nv_bfloat16*>(sc0), qz0};
  P.p1 = TileProj{reinterpret_cast<const __nv_bfloat16*>(swiglu ? sc1 : sc0), swiglu ? qz1 : qz0};
  P.out = reinterpret_cast<__nv_bfloat16*>(out);
  P.d_status = d_status;
  const int sms = device_sm_count();
  const TileShape shape = tile_shape(rows, E, N, swiglu, sms);
  P.tn = shape.tn;
  const int64_t tiles = most_token_tiles(S, E, shape.tn) * shape.col_tiles;
  const int grid = (int)(tiles < sms ? tiles : sms);
#define MQ_TILE_LAUNCH(MODE, GATHER)                                                                                \
  do {                                                                                                              \
    cudaFuncSetAttribute(w4a16_tile_kernel<MODE, GATHER>, cudaFuncAttributeMaxDynamicSharedMemorySize, TL_SMEM);    \
    w4a16_tile_kernel<MODE, GATHER><<<grid, TL_THREADS, TL_SMEM, st>>>(map0, map1, mapx, P);                        \
  } while (0)
  // no coarser a SwiGLU than without this kernel: the stream kernel takes 32 rows or more of up to 384 groups
  const bool exact = swiglu && (S < 32 || !w4a16_stream_covers(S, E, period, N, Kd, 128));
  if (perm != nullptr && !swiglu) return MQ_ERR_UNSUPPORTED_SHAPE;
  if (exact && perm != nullptr) MQ_TILE_LAUNCH(TILE_SWIGLU_EXACT, true);
  else if (exact) MQ_TILE_LAUNCH(TILE_SWIGLU_EXACT, false);
  else if (swiglu && perm != nullptr) MQ_TILE_LAUNCH(TILE_SWIGLU, true);
  else if (swiglu) MQ_TILE_LAUNCH(TILE_SWIGLU, false);
  else if (shape.wide) MQ_TILE_LAUNCH(TILE_WIDE, false);
  else MQ_TILE_LAUNCH(TILE_NARROW, false);
#undef MQ_TILE_LAUNCH
  return check_launch();
}

}  // namespace mq
