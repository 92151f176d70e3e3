// bf16 grouped expert GEMM on CTA pairs (tcgen05.mma.cta_group::2), optionally with the row gather in front and the
// gate/up SwiGLU behind.  Same result as grouped_gemm_tc5.cu (mini_qwen/kernels/moe_grouped_gemm.py:17-37,
// mini_qwen/model/layers/moe.py:24-25 of the reference): fp32 sums in k order, one rounding of each projection.
//
// What bounds it: at 256 rows per expert the weights of a layer take as long to read as the tensor cores take to
// multiply them, so both have to run at full rate.  The single-CTA kernel could do neither: an MMA of 128 weight rows
// by 256 tokens reads 96 bytes of shared memory per clock and its operands arrive at 64, together more than the 128 a
// shared memory delivers, and an expert with a few rows more than 256 cost two tiles, which fetched and read its
// weights twice.  Here two SMs work on one tile:
//   * weight rows are M = 256 (128 lanes in either CTA), tokens are N.  Each CTA stages its own 128 weight rows and
//     HALF of the tokens; the MMA, issued by the even CTA, reads both halves: 64 bytes per clock and SM;
//   * a sub-tile is 128 weight rows per CTA.  SwiGLU: 64 gate rows and the up rows of the same columns, 16 of either in
//     turn, so that an epilogue warp holds both factors of its outputs;
//   * three tile shapes by the rows n of the expert share one ring (four stages of 48 KB) and two accumulators:
//       WEIGHTS2  128 < n <= 256: two sub-tiles against one token tile;
//       TOKENS2   n > 256: one sub-tile against two token tiles (up to 512 rows in all);
//       DEEP      n <= 128: one sub-tile, 128 k per stage; consecutive tiles alternate between the accumulators, so
//                 the epilogue runs under the next tile's MMAs.
// Warps: 0 TMA, 1 MMA (even CTA), 2-9 epilogue, 10-13 (gathering variant) row copies.  Barriers on which the MMA waits
// lie in the even CTA and are signalled by both; the MMA's commits signal both.
// Every wait is bounded: when one runs out, MQ_DEV_WAIT_EXPIRED is set, all roles leave their loops, copies in flight
// are waited for and TMEM is freed.
#include "tc5.cuh"

namespace mq {
namespace {

using namespace tc5;

constexpr int PM = 128;                          // weight rows per sub-tile and CTA = TMEM lanes
constexpr int PK = 64;                           // k per operand block: one 128-byte swizzle span
constexpr int PN = 256;                          // most tokens per MMA (N)
constexpr int P_BLOCK = PM * PK * 2;             // 16 KB: an operand block (128 rows x 64 k)
constexpr int P_STAGE = 3 * P_BLOCK;             // A0 | A1 or B1 | B0 (DEEP: A k0 | A k1 | B k0, B k1)
constexpr int P_NST = 4;
constexpr int P_BOX = 32;                        // token rows per TMA box
constexpr int P_BOX_BYTES = P_BOX * PK * 2;
constexpr int P_EPI = 8, P_GATHER = 4;           // warps
constexpr int P_STG = 32 * 64;                   // staged output rows of an epilogue warp
constexpr int P_MAX_E = 1024;
constexpr int P_SORT_E = 256;                    // most groups that are put in order of size
constexpr int P_TABLE = (2 * (P_MAX_E + 1) + P_SORT_E) * 4;
constexpr int P_SMEM = 1024 + P_NST * P_STAGE + P_EPI * P_STG + 256 + ((P_TABLE + 15) & ~15);
static_assert(P_SMEM <= 232448, "shared memory of a CTA");

enum PairShape { WEIGHTS2, TOKENS2, DEEP };

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the even CTA's copy of a shared-memory location
__device__ __forceinline__ uint32_t in_leader(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait of a warp on a barrier that the other CTA signals too.
__device__ __forceinline__ bool wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag, int32_t* d_status) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .u32 n;\n\t"
      "mov.u32 n, %3;\n\t"
      "LOOK_%=:\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "@p bra SEEN_%=;\n\t"
      "sub.u32 n, n, 1;\n\t"
      "setp.ne.u32 q, n, 0;\n\t"
      "@q bra LOOK_%=;\n\t"
      "SEEN_%=:\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity), "r"(SPIN_LIMIT) : "memory");
  if (__all_sync(0xffffffffu, ok != 0)) return true;
  if (!*abort_flag && d_status != nullptr) atomicOr(d_status, (int)MQ_DEV_WAIT_EXPIRED);
  *abort_flag = 1;
  return false;
}
// The copies land in this CTA; their bytes count on a barrier of the even CTA.
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap* map, uint32_t leader_bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(leader_bar), "r"(x), "r"(y) : "memory");
}
// from the gate/up weights' five dimensions: k, row of a group of 16, gate or up, group, expert
__device__ __forceinline__ void tma_load_5d_pair(uint32_t dst, const CUtensorMap* map, uint32_t leader_bar, int x, int group,
                                                 int expert) {
  asm volatile(
      "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(leader_bar), "r"(x), "r"(0), "r"(group), "r"(expert) : "memory");
}
// four rows of 64 columns from x, 128 bytes apart in shared memory
__device__ __forceinline__ void tma_gather4_pair(uint32_t dst, const CUtensorMap* map, uint32_t leader_bar, int x,
                                                 const int (&row)[4]) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(dst), "l"(map), "r"(leader_bar), "r"(x), "r"(row[0]), "r"(row[1]), "r"(row[2]), "r"(row[3]) : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
}
// signals the barrier at this offset in both CTAs once the MMAs issued so far are complete
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(bar), "h"((uint16_t)3) : "memory");
}

// 16 TMEM lanes x 32 columns in the fragment layout of m16n8 accumulators (four 8-column blocks); not waited for.
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t saddr, uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};"
               ::"r"(saddr), "r"(m0), "r"(m1), "r"(m2), "r"(m3) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(uint32_t lo_bits, uint32_t hi_bits) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(__uint_as_float(lo_bits), __uint_as_float(hi_bits));
  return *reinterpret_cast<const uint32_t*>(&p);
}
// silu(g) * u of two pairs that are already rounded to bf16, rounded after silu and after the product.
__device__ __forceinline__ uint32_t swiglu_bf16x2(uint32_t g, uint32_t u) {
  const float2 gf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g));
  const float2 uf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u));
  const float s0 = __fdividef(gf.x, 1.0f + __expf(-gf.x));
  const float s1 = __fdividef(gf.y, 1.0f + __expf(-gf.y));
  const float2 sf = __bfloat1622float2(__floats2bfloat162_rn(s0, s1));
  const __nv_bfloat162 o = __floats2bfloat162_rn(sf.x * uf.x, sf.y * uf.y);
  return *reinterpret_cast<const uint32_t*>(&o);
}

// A tile of work.  Chunk c (0, 1) is the token tile of accumulator c; with WEIGHTS2 both are the same rows.
struct PairTile {
  int expert, unit, shape;                       // unit: first sub-tile (256 weight rows over the pair)
  bool two;                                      // both accumulators are used
  int tok0, ntok;                                // first token row and token rows of the tile
  int n0, n1;                                    // MMA N of the token chunks (multiples of 32; n1 = 0: one chunk)
};

// Tiles are dealt out in the groups' order, the pairs in turn.  With skewed groups and more than one round of tiles:
// largest groups first, the pairs back and forth.  A tile of 512 rows takes four times one of 128, and in the groups' own
// order one pair got two of the largest while others had none (gate/up, us, own order | by size, on the single-CTA kernel:
// 16 groups, 1024 Zipf-distributed rows, K 768, N 768: 23.4 | 19.7, 17.5; 32 groups, 10296 rows, K 1280, N 640: 59.3 | 46.4,
// 47.0; 128 groups, 131072 rows, K 2048, N 768: 661 | 639, 678).
struct PairTable {
  const int* off;                                // [E + 1]
  const int* group;                              // [E]: the groups by size, or null: in their own order
  const int* first;                              // [E + 1]: first tile of the group in that order
  int E, units;
  __device__ static int shape_of(int n) { return n <= 128 ? DEEP : n <= PN ? WEIGHTS2 : TOKENS2; }
  __device__ static int tiles_of(int n, int units) {
    return n <= 0 ? 0 : n <= 128 ? units : n <= PN ? (units + 1) / 2 : (n + 2 * PN - 1) / (2 * PN) * units;
  }
  __device__ PairTile locate(int t) const {
    int lo = 0, hi = E;                          // first[lo] <= t < first[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (first[mid] <= t) lo = mid; else hi = mid;
    }
    const int local = t - first[lo], e = group != nullptr ? group[lo] : lo, n = off[e + 1] - off[e];
    PairTile w;
    w.expert = e;
    w.shape = shape_of(n);
    if (w.shape != TOKENS2) {
      w.unit = w.shape == WEIGHTS2 ? 2 * local : local;
      w.two = w.shape == WEIGHTS2 && w.unit + 1 < units;
      w.tok0 = off[e];
      w.ntok = n;
      w.n0 = (n + 31) & ~31;
      w.n1 = 0;
    } else {
      const int ntt = (n + 2 * PN - 1) / (2 * PN), tt = local / units;
      const int width = (((n + ntt - 1) / ntt) + 31) & ~31;      // balanced token tiles, at most 512 rows
      w.unit = local - tt * units;
      w.tok0 = off[e] + tt * width;
      w.ntok = min(width, n - tt * width);
      w.n0 = (((w.ntok + 1) >> 1) + 31) & ~31;
      w.n1 = w.ntok > w.n0 ? (w.ntok - w.n0 + 31) & ~31 : 0;
      w.two = w.n1 > 0;
    }
    return w;
  }
};

struct PairParams {
  const int32_t* offsets;                        // [E + 1]
  int E, period, N, Kd;
  const int32_t* perm;
  int top_k;
  __nv_bfloat16* out;
  int32_t* d_status;
};

template <bool SWIGLU, bool GATHER>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__((2 + P_EPI + (GATHER ? P_GATHER : 0)) * 32, 1)
grouped_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                         const PairParams P) {
  constexpr int CW = SWIGLU ? 64 : 128;          // output columns per sub-tile and CTA
  extern __shared__ uint8_t pair_smem_raw[];
  const uint32_t raw = smem_addr(pair_smem_raw);
  const uint32_t ring = (raw + 1023u) & ~1023u;  // the swizzle pattern repeats every 1024 bytes
  uint8_t* ptr = pair_smem_raw + (ring - raw);
  uint8_t* stg_mem = ptr + P_NST * P_STAGE;
  uint8_t* bar_mem = stg_mem + P_EPI * P_STG;
  const uint32_t bars = ring + P_NST * P_STAGE + P_EPI * P_STG;
  auto full = [&](int s) { return bars + 8u * s; };              // waited on by the even CTA's MMA warp only
  auto empty = [&](int s) { return bars + 8u * (P_NST + s); };
  auto tfull = [&](int b) { return bars + 8u * (2 * P_NST + b); };
  auto tempty = [&](int b) { return bars + 8u * (2 * P_NST + 2 + b); };   // even CTA only
  volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(bar_mem + 8 * (2 * P_NST + 4));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_mem + 8 * (2 * P_NST + 4) + 8);
  int* s_off = reinterpret_cast<int*>(bar_mem + 256);
  int* s_first = s_off + P.E + 1;
  int* s_group = s_first + P.E + 1;
  volatile int* skew_flag = reinterpret_cast<volatile int*>(bar_mem + 8 * (2 * P_NST + 4) + 12);

  const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int rank = (int)uniform(cluster_rank());
  const int E = P.E, N = P.N, KB = P.Kd / PK;
  const int units = N / (2 * CW);

  if (threadIdx.x == 0) {
    for (int s = 0; s < P_NST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull(b), 1);
      mbar_init(tempty(b), 2 * P_EPI);
    }
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_addr((const void*)tmem_ptr)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  for (int e = threadIdx.x; e <= E; e += blockDim.x) s_off[e] = P.offsets[e];
  __syncthreads();
  const int pairs = (int)(gridDim.x >> 1), pair = (int)(blockIdx.x >> 1);
  // first[]: exclusive sums of the groups' tile counts; the largest group's rows
  auto count_tiles = [&](const int* order) {
    int carry = 0, most = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int at = e0 + lane, e = order != nullptr && at < E ? order[at] : at;
      const int n = at < E ? s_off[e + 1] - s_off[e] : 0, c = PairTable::tiles_of(n, units);
      most = max(most, n);
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (at < E) s_first[at] = carry + incl - c;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_first[E] = carry;
    return __reduce_max_sync(0xffffffffu, most);
  };
  if (warp == 0) {
    const int most = count_tiles(nullptr);
    // skewed: the largest group is over twice the average
    if (lane == 0) *skew_flag = E <= P_SORT_E && s_first[E] > pairs && most > PN && most / 2 > (s_off[E] - s_off[0]) / E;
  }
  fence_before_sync();
  __syncthreads();
  const bool skewed = *skew_flag != 0;
  if (skewed) {                                  // a group's place is the number of larger ones, equals in their order
    int n[P_SORT_E / 32];
#pragma unroll
    for (int j = 0; j < P_SORT_E / 32; ++j) {
      const int e = 32 * j + lane;
      n[j] = e < E ? s_off[e + 1] - s_off[e] : -1;
    }
    for (int e = warp; e < E; e += (int)(blockDim.x >> 5)) {
      const int mine = s_off[e + 1] - s_off[e];
      int before = 0;
#pragma unroll
      for (int j = 0; j < P_SORT_E / 32; ++j) before += n[j] > mine || (n[j] == mine && 32 * j + lane < e) ? 1 : 0;
      before = __reduce_add_sync(0xffffffffu, before);
      if (lane == 0) s_group[before] = e;
    }
    __syncthreads();
    if (warp == 0) count_tiles(s_group);
  }
  cluster_sync();                                // barriers, TMEM and table of both CTAs are ready
  fence_after_sync();
  const uint32_t tmem = uniform(*tmem_ptr);
  const PairTable table{s_off, skewed ? s_group : nullptr, s_first, E, units};
  const int total = s_first[E];
  auto deal = [&](int i) { return i * pairs + (skewed && (i & 1) != 0 ? pairs - 1 - pair : pair); };   // its i-th tile

  if (warp == 0) {
    // ------------------------------------------------------------------ operand copies by TMA
    // Like the MMA issuer: the whole warp walks the loop and one elected lane issues, so that addresses and coordinates
    // are in uniform registers (a single lane's loop spent 150 clocks on every copy: 1000 a stage, the MMAs' whole time).
    const bool leader = elect_one();
    const uint32_t full0 = uniform(in_leader(full(0)));
    int stage = 0, filled = 0;
    uint32_t phase = 0;
    bool ok = true;
    // this CTA's 128 weight rows of sub-tile `unit`, 64 k from k
    auto load_a = [&](uint32_t dst, uint32_t bar, int k, int wexpert, int unit) {
      const int c = unit * 2 * CW + rank * CW;
      if (SWIGLU) tma_load_5d_pair(dst, &map_w, bar, k, c / 16, wexpert);
      else tma_load_pair(dst, &map_w, bar, k, wexpert * N + c);
    };
    auto load_b = [&](uint32_t dst, uint32_t bar, int k, int row, int boxes) {
      for (int b = 0; b < boxes; ++b) tma_load_pair(dst + b * P_BOX_BYTES, &map_x, bar, k, row + b * P_BOX);
    };
    for (int nth = 0; deal(nth) < total && ok; ++nth) {
      const PairTile w = table.locate(deal(nth));
      const int we = (int)uniform(w.expert % P.period), unit = (int)uniform(w.unit), shape = (int)uniform(w.shape);
      const bool two = uniform(w.two) != 0;
      const int h0 = (int)uniform(w.n0 >> 1), h1 = (int)uniform(w.n1 >> 1);     // this CTA's halves of the token chunks
      const int box0 = (h0 + P_BOX - 1) / P_BOX, box1 = (h1 + P_BOX - 1) / P_BOX;   // rows past the half: not read
      const int tok0 = (int)uniform(w.tok0), row0 = tok0 + rank * h0, row1 = tok0 + 2 * h0 + rank * h1;
      const int step = shape == DEEP ? 2 : 1;
      uint32_t bytes = P_BLOCK * ((shape == WEIGHTS2 && two) ? 2 : 1) + (GATHER ? (h0 + h1) * PK * 2 : (box0 + box1) * P_BOX_BYTES);
      if (shape == DEEP) bytes *= 2;
      for (int kb = 0; kb < KB; kb += step) {
        ok = mbar_wait_warp(empty(stage), phase ^ 1u, abort_flag, P.d_status);
        if (!ok) break;
        const uint32_t a = ring + stage * P_STAGE, a1 = a + P_BLOCK, b = a + 2 * P_BLOCK;
        const uint32_t bar = full0 + 8u * stage;
        if (leader) {
          if (rank == 0) mbar_expect_tx(full(stage), 2 * bytes);           // both CTAs' copies
          load_a(a, bar, kb * PK, we, unit);
          if (shape == WEIGHTS2 && two) load_a(a1, bar, kb * PK, we, unit + 1);
          if (shape == DEEP) load_a(a1, bar, (kb + 1) * PK, we, unit);
          if (!GATHER) {
            load_b(b, bar, kb * PK, row0, box0);
            if (shape == DEEP) load_b(b + P_BLOCK / 2, bar, (kb + 1) * PK, row0, box0);
            else load_b(a1, bar, kb * PK, row1, box1);
          }
        }
        __syncwarp();
        ++filled;
        if (++stage == P_NST) { stage = 0; phase ^= 1u; }
      }
    }
    // every stage that was filled has been read before the CTA exits; after giving up: the copies have landed
    for (int s = 0; s < P_NST && ok; ++s) {
      ok = mbar_wait_warp(empty(stage), phase ^ 1u, abort_flag, P.d_status);
      if (++stage == P_NST) { stage = 0; phase ^= 1u; }
    }
    if (!ok && rank == 0) {
      for (int f = max(0, filled - P_NST); f < filled; ++f)
        mbar_wait_limited(full(f % P_NST), (uint32_t)(f / P_NST) & 1u, 1u << 16);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (even CTA)
    if (rank == 0) {
      const bool leader = elect_one();
      int stage = 0, cur = 0;                    // cur: accumulator of the next single-accumulator tile
      uint32_t phase = 0, used = 0;              // used: parity of the tiles each accumulator has held, a bit each
      bool ok = true;
      for (int nth = 0; deal(nth) < total && ok; ++nth) {
        PairTile w = table.locate(deal(nth));
        w.shape = (int)uniform(w.shape);
        w.two = uniform(w.two) != 0;
        const int b0 = w.two ? 0 : cur;
        ok = wait_cluster(tempty(b0), ((used >> b0) & 1u) ^ 1u, abort_flag, P.d_status);
        if (!ok) break;
        fence_after_sync();
        // A stage is four MMAs on (A0, B0) and, unless the tile has one accumulator and 64 k per stage, four more on the
        // operands its shape pairs up.  Everything they are issued with is uniform over the warp: taken from a lane's
        // registers each MMA waits for it to be moved.
        const bool second = w.two || w.shape == DEEP;
        const uint32_t acc0 = uniform(tmem + b0 * PN), acc1 = w.shape == DEEP ? acc0 : uniform(tmem + PN);
        const uint32_t id0 = uniform(idesc_bf16(2 * PM, w.n0));
        const uint32_t id1 = w.shape == TOKENS2 ? uniform(idesc_bf16(2 * PM, w.n1)) : id0;
        const uint32_t a1 = w.shape == TOKENS2 ? 0 : P_BLOCK;                       // offsets inside a stage
        const uint32_t b1 = w.shape == TOKENS2 ? P_BLOCK : 2 * P_BLOCK + (w.shape == DEEP ? P_BLOCK / 2 : 0);
        const int steps = w.shape == DEEP ? KB / 2 : KB;
        // With two accumulators a tile starts on the first one while the epilogue still drains the second: the first
        // `ahead` stages' MMAs on it go out before the second is waited for.
        const int ahead = w.two ? min(P_NST, steps) : 0;
        auto four = [&](uint32_t acc, uint32_t a, uint32_t b, uint32_t id, uint32_t add) {
          const uint64_t da = smem_desc(a), db = smem_desc(b);
          // 16 k = 32 bytes along the swizzled row: + 2 in the descriptor's address field
          mma_pair(acc, da, db, id, add);
#pragma unroll
          for (int k = 1; k < PK / 16; ++k) mma_pair(acc, da + 2u * k, db + 2u * k, id, 1u);
        };
        for (int i = 0; i < ahead && ok; ++i) {
          int st = stage + i;
          const uint32_t ph = st >= P_NST ? phase ^ 1u : phase;
          if (st >= P_NST) st -= P_NST;
          ok = wait_cluster(full(st), ph, abort_flag, P.d_status);
          if (!ok) break;
          fence_after_sync();
          const uint32_t s = ring + st * P_STAGE;
          if (leader) {
            four(acc0, s, s + 2 * P_BLOCK, id0, i != 0 ? 1u : 0u);
            if (i == steps - 1) commit_pair(tfull(b0));
          }
          __syncwarp();
        }
        if (ok && w.two) ok = wait_cluster(tempty(1), (used >> 1) ^ 1u, abort_flag, P.d_status);
        for (int i = 0; i < steps && ok; ++i) {
          if (i >= ahead) ok = wait_cluster(full(stage), phase, abort_flag, P.d_status);
          if (!ok) break;
          fence_after_sync();
          const uint32_t s = ring + stage * P_STAGE;
          if (leader) {
            if (i >= ahead) four(acc0, s, s + 2 * P_BLOCK, id0, i != 0 ? 1u : 0u);
            if (i >= ahead && w.two && i == steps - 1) commit_pair(tfull(b0));
            if (second) four(acc1, s + a1, s + b1, id1, w.shape == DEEP || i != 0 ? 1u : 0u);
            commit_pair(empty(stage));
            if (i == steps - 1) commit_pair(tfull(w.two ? 1 : b0));
          }
          __syncwarp();
          if (++stage == P_NST) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        used ^= w.two ? 3u : 1u << b0;
        cur = w.two ? 0 : cur ^ 1;
      }
    }
  } else if (GATHER && warp >= 2 + P_EPI) {
    // ------------------------------------------------------------------ row copies of the gathering variant
    // A copy moves four rows x 64 k of x, gathered by TMA into four rows of a swizzled operand.  A stage's copies (this
    // CTA's halves of its token chunks; with DEEP one chunk, twice 64 k) are dealt out to the warps; lane i keeps what
    // its warp's copy i needs and hands it over by shuffle, so that the copies are issued from uniform registers.
    // Rows past the expert's last repeat it: computed, not stored.
    const bool leader = elect_one();
    const uint32_t full0 = uniform(in_leader(full(0)));
    const int gw = warp - (2 + P_EPI);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int next[4] = {0, 0, 0, 0}, count_next = 0, step_next = 1;
    uint32_t at_next = 0;                        // where in a stage the copy lands; bit 0: the second 64 k of the stage
    auto fetch = [&](int t) {
      const PairTile tl = table.locate(t);
      const int h0 = tl.n0 >> 1, h1 = tl.n1 >> 1, c0 = h0 >> 2, copy = gw + P_GATHER * lane;
      const bool deep = tl.shape == DEEP, later = copy >= c0;               // in the second half of the list
      const int i = later ? copy - c0 : copy, copies = c0 + (deep ? c0 : h1 >> 2);
      at_next = (!later ? 2 * P_BLOCK : deep ? 2 * P_BLOCK + P_BLOCK / 2 + 1 : P_BLOCK) + 512u * i;
      step_next = deep ? 2 : 1;
      count_next = (copies - gw + P_GATHER - 1) / P_GATHER;                 // this warp's (at most 16)
      if (copy < copies) {
        const int first = tl.tok0 + (later && !deep ? tl.n0 + rank * h1 : rank * h0) + 4 * i, last = tl.tok0 + tl.ntok - 1;
#pragma unroll
        for (int j = 0; j < 4; ++j) next[j] = P.perm[min(first + j, last)];
      }
    };
    if (pair < total) fetch(pair);
    for (int nth = 0; deal(nth) < total && ok; ++nth) {
      int row[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) row[i] = next[i] / P.top_k;
      const uint32_t at = at_next;
      const int count = (int)uniform(count_next), step = (int)uniform(step_next);
      if (deal(nth + 1) < total) fetch(deal(nth + 1));   // the next tile's positions travel under this tile's copies
      for (int kb = 0; kb < KB; kb += step) {
        ok = mbar_wait_warp(empty(stage), phase ^ 1u, abort_flag, P.d_status);
        if (!ok) break;
        const uint32_t s = ring + stage * P_STAGE, bar = full0 + 8u * stage;
#pragma unroll 4
        for (int i = 0; i < count; ++i) {
          int r[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) r[j] = __shfl_sync(0xffffffffu, row[j], i);
          const uint32_t d = __shfl_sync(0xffffffffu, at, i);
          if (leader) tma_gather4_pair(s + (d & ~1u), &map_x, bar, (kb + (int)(d & 1u)) * PK, r);
        }
        __syncwarp();
        if (++stage == P_NST) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp < 2 + P_EPI) {
    // ------------------------------------------------------------------ epilogue
    // Two groups of four warps drain the even and the odd 32-token blocks of an accumulator.  A warp holds 32 of the
    // CTA's 128 lanes (weight rows) and works by itself: stmatrix.trans turns its block into token-major rows in its own
    // staging space (16-byte pieces placed so that both ways are free of bank conflicts), 64 bytes of 32 output columns,
    // or 32 bytes of 16 columns with SwiGLU (lanes 0..15 are gate rows, 16..31 the up rows of the same columns).
    const int quad = warp & 3, group = (warp - 2) >> 2;
    constexpr int PIECES = SWIGLU ? 2 : 4, ROWB = 16 * PIECES;             // of a staged token row
    uint8_t* stg = stg_mem + (warp - 2) * P_STG;
    const uint32_t stg_s = smem_addr(stg);
    const int mi = lane >> 3, ri = lane & 7;
    auto place = [&](int tok, int piece) { return (uint32_t)(tok * ROWB + ((piece ^ ((tok * PIECES >> 3) & (PIECES - 1))) << 4)); };
    uint32_t used = 0;
    int cur = 0;
    bool ok = true;
    for (int nth = 0; deal(nth) < total && ok; ++nth) {
      const PairTile w = table.locate(deal(nth));
      const int b0 = w.two ? 0 : cur;
      for (int c = 0; c < (w.two ? 2 : 1); ++c) {
        const int b = c == 0 ? b0 : 1;
        ok = mbar_wait_warp(tfull(b), (used >> b) & 1u, abort_flag, P.d_status);
        if (!ok) break;
        used ^= 1u << b;
        fence_after_sync();
        const bool second_rows = c == 1 && w.shape == TOKENS2;
        const int row0 = w.tok0 + (second_rows ? w.n0 : 0);                // first token row of the accumulator
        const int nrow = second_rows ? w.ntok - w.n0 : min(w.ntok, w.n0);
        const int col0 = (w.unit + (c == 1 && w.shape == WEIGHTS2 ? 1 : 0)) * 2 * CW + rank * CW + quad * (CW / 4);
        // Blocks leave tensor memory (packed: 16 registers each) ahead of their stores, so that the accumulator is free
        // early and the stores run under the next tile's MMAs: all four, or two at a time where the warps of the
        // gathering variant leave 128 registers a thread (four spilled there).
        const int rounds = max(0, (nrow - 32 * group + 63) >> 6);
        constexpr int BATCH = GATHER ? 2 : 4;
#pragma unroll
        for (int i0 = 0; i0 < 4; i0 += BATCH) {
          uint32_t v[BATCH][16];
#pragma unroll
          for (int i = 0; i < BATCH; ++i) {
            if (i0 + i < rounds) {
              uint32_t f[2][16];
              const uint32_t ta = tmem + b * PN + ((uint32_t)(quad * 32) << 16) + 32 * group + 64 * (i0 + i);
              tmem_ld_frag(ta, f[0]);
              tmem_ld_frag(ta + (16u << 16), f[1]);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                v[i][j] = pack_bf16(f[0][2 * j], f[0][2 * j + 1]);
                v[i][8 + j] = pack_bf16(f[1][2 * j], f[1][2 * j + 1]);
              }
            }
          }
          if (i0 + BATCH == 4) {
            fence_before_sync();
            __syncwarp();
            if (lane == 0) arrive_cluster(in_leader(tempty(b)));
          }
#pragma unroll
          for (int i = 0; i < BATCH; ++i) {
            if (i0 + i < rounds) {
              const int r = 32 * group + 64 * (i0 + i);
              __syncwarp();                                                // the previous block's rows have been read
#pragma unroll
              for (int j2 = 0; j2 < 2; ++j2) {                             // token octets (0, 1) and (2, 3)
                const int tok = 8 * (2 * j2 + (mi >> 1)) + ri;
#pragma unroll
                for (int hl = 0; hl < (SWIGLU ? 1 : 2); ++hl) {
                  uint32_t m[4];
#pragma unroll
                  for (int q = 0; q < 4; ++q)
                    m[q] = SWIGLU ? swiglu_bf16x2(v[i][4 * j2 + q], v[i][8 + 4 * j2 + q]) : v[i][8 * hl + 4 * j2 + q];
                  stmatrix_x4_trans(stg_s + place(tok, 2 * hl + (mi & 1)), m[0], m[1], m[2], m[3]);
                }
              }
              __syncwarp();
#pragma unroll
              for (int q = 0; q < PIECES; ++q) {
                const int row = (32 / PIECES) * q + lane / PIECES, p = lane % PIECES;
                if (row < nrow - r)
                  *reinterpret_cast<uint4*>(P.out + (size_t)(row0 + r + row) * N + col0 + p * 8) =
                      *reinterpret_cast<const uint4*>(stg + place(row, p));
              }
            }
          }
        }
      }
      cur = w.two ? 0 : cur ^ 1;
    }
  }

  fence_before_sync();
  __syncthreads();
  cluster_sync();                                // nothing of the pair is in flight towards either CTA any more
  if (warp == 1) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// 2-D bf16 row-major [rows, cols] tensor, boxes of 64 columns x box_rows rows, 128-byte swizzle.
bool pair_map(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int box_rows) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  cuuint32_t box[2] = {(cuuint32_t)PK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1u, 1u};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Gate and up rows [experts, 2, N, Kd] as [experts, N / 16 groups, 2, 16, Kd]: a box is four groups, 16 gate rows and the
// 16 up rows of the same columns in turn: the 128 lanes of a sub-tile.
bool pair_map_gate_up(CUtensorMap* map, const void* base, int64_t experts, int64_t N, int64_t Kd) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return false;
  const cuuint64_t row = (cuuint64_t)Kd * 2;
  cuuint64_t dims[5] = {(cuuint64_t)Kd, 16, 2, (cuuint64_t)(N / 16), (cuuint64_t)experts};
  cuuint64_t strides[4] = {row, row * N, row * 16, row * 2 * N};
  cuuint32_t box[5] = {(cuuint32_t)PK, 16, 2, 4, 1};
  cuuint32_t estr[5] = {1u, 1u, 1u, 1u, 1u};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// Whole sub-tiles of 256 weight rows, whole 128-k stages; coordinates and tile counts are 32-bit.  A plain projection
// of a short K with every expert hit stays with the single-CTA kernel: a tile is then 12 stages, too few to hide the
// two epilogues of a pair behind (K = 768, N = 2048, 128 experts, us, single against pair: 95 | 101 at 144 rows per
// expert, 111 | 118 at 256, 131 | 136 at 272; but 48 | 44 with 50 of the experts hit by one row, where the finer tiles
// spread better).  From K = 1024 on it goes by pairs up to 100 rows a group (K 2048, N 768, 128 experts: 85 | 81 at 92 rows;
// with fewer 8 to 28 % faster on average over 140 shapes), and with more where there are few groups and a long K (16 and 32
// groups: 0.86 to 1.39 times as fast); 64 and more groups are slower (89 | 98 at 122 rows, 100 | 110 at 191), as is K 1024 (16
// groups, N 1536: 20.0 | 22.9 at 215 rows).  SwiGLU over K = 2048, gathered: 94 | 73 with 50 rows, 176 | 148 at 48 per expert, 222 | 208 at 256,
// 281 | 230 at 272, 355 | 327 at 512.  Two ranges of it stay there as well.  Fewer than 16 groups of over 256 rows: a pair's
// tile is four times a CTA's, and a round that is not full costs as much more (8 experts: 31 | 50 at 2217 rows, K 2048,
// N 256; 28 | 42 at 622, K 1792, N 768; by 5 % the slower on average over 36 shapes).  A K of 512 or less with up to 32 groups of 128 rows or
// more: again too few stages (K 512, N 768, 16 experts: 16.0 | 16.8 at 144 rows, 25.3 | 29.7 at 512; 32 experts: 27.8 | 29.3
// at 200; but 69 | 61 with 128 experts, 144 rows, and 14.4 | 10.1 with N 128, 16 experts).  Of 871 measured calls (8 to 128 experts, K 512 to 2048, even
// and skewed) the pair kernel is then the slower one by over 3 % in 27, the faster one by 22 % on average.
bool grouped_gemm_pair_covers(int64_t S, int64_t E, int64_t period, int64_t N, int64_t Kd, bool swiglu) {
  if (!swiglu && ((Kd < 1024 && S > E) || (S > 100 * E && (E >= 64 || Kd < 1280)))) return false;
  if (swiglu && ((E < 16 && S > 256 * E) || (Kd <= 512 && E <= 32 && N > 128 && S >= 128 * E))) return false;
  return Kd % 128 == 0 && N % (swiglu ? 128 : 256) == 0 && E <= P_MAX_E && S < ((int64_t)1 << 30) &&
         period * N * 2 < ((int64_t)1 << 31) && (S / 256 + 2 * E) * (N / 128) < ((int64_t)1 << 30);
}

// perm == nullptr: `a` holds the S expert-sorted rows; otherwise sorted row p is a[perm[p] / top_k].
int grouped_gemm_pair(const void* a, const void* w, const int32_t* offsets, int64_t S, int64_t E, int64_t period,
                      int64_t N, int64_t Kd, bool swiglu, void* out, int32_t* d_status, cudaStream_t st,
                      const int32_t* perm, int64_t top_k) {
  CUtensorMap map_x, map_w;
  const bool gather = perm != nullptr;
  // a gathered copy takes its rows one by one: boxes of one row
  if (!pair_map(&map_x, a, gather ? S / top_k : S, Kd, gather ? 1 : P_BOX) ||
      !(swiglu ? pair_map_gate_up(&map_w, w, period, N, Kd) : pair_map(&map_w, w, period * N, Kd, PM)))
    return MQ_ERR_DRIVER_ENTRY;
  PairParams P;
  P.offsets = offsets;
  P.E = (int)E;
  P.period = (int)period;
  P.N = (int)N;
  P.Kd = (int)Kd;
  P.perm = perm;
  P.top_k = (int)top_k;
  P.out = reinterpret_cast<__nv_bfloat16*>(out);
  P.d_status = d_status;
  // gathering: the number of rows is offsets[E], known only on the device, so the grid is not trimmed
  const int64_t most = (S / (2 * PN) + (E < S ? E : S)) * (N / (swiglu ? 128 : 256)), pairs = device_sm_count() / 2;
  const int grid = 2 * (int)(!gather && most < pairs ? most : pairs);
#define MQ_PAIR_LAUNCH(SW, GA)                                                                                       \
  do {                                                                                                              \
    cudaFuncSetAttribute(grouped_gemm_pair_kernel<SW, GA>, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM);    \
    grouped_gemm_pair_kernel<SW, GA><<<grid, (2 + P_EPI + (GA ? P_GATHER : 0)) * 32, P_SMEM, st>>>(map_x, map_w, P); \
  } while (0)
  if (swiglu && gather) MQ_PAIR_LAUNCH(true, true);
  else if (swiglu) MQ_PAIR_LAUNCH(true, false);
  else if (gather) return MQ_ERR_UNSUPPORTED_SHAPE;
  else MQ_PAIR_LAUNCH(false, false);
#undef MQ_PAIR_LAUNCH
  return check_launch();
}

}  // namespace mq
