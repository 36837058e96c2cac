// sdg_dense_tc.cu -- the dense screen fused on the 5th-generation tensor cores.
//
// The BF16 screen of the dense path without a slab in HBM.  The work of a
// query block is the grid of (query group, reference tile) items: a query
// group is 128 query columns (one UMMA A tile, M = 128), a reference tile 256
// reference columns (UMMA N = 256).  The items, query-group-major, are split
// into equal contiguous spans, one per CTA (a persistent grid of at most one
// CTA per SM), so every SM gets the same work whatever the block size; a span
// usually covers the tail of one query group and the head of the next, and
// each (query group, CTA) piece of a span is a "segment".
//
// Per segment the query group's 128 x d BF16 columns are loaded into shared
// memory once (TMA, SWIZZLE_128B, K-major, 64-row chunks); reference tiles of
// 256 columns x 64 rows stream through a four-stage TMA ring.  One lane of the
// issuing warp issues tcgen05.mma.cta_group::1.kind::f16 (M = 128 queries, N =
// 256 references, K = 16, BF16 in, FP32 accumulate) into TMEM: two accumulator
// buffers of 256 columns fill all 512, so the MMAs of tile j + 1 run while
// the epilogue reads tile j back with tcgen05.ld.
//
// Epilogue: eight warps; warp w reads TMEM lanes 32 (w % 4) .. + 31 (its 32
// queries) and one half of the tile's 256 columns ((w - 2) / 4).  A thread
// owns one (query, column half) and appends every reference whose optimistic
// key reaches its cut to a per-(query, segment, half) list.  The cut is never
// above the query's final one, so the union of the lists holds every reference
// that the slab screen keeps; k_tc_merge applies the final cut, then a second,
// tighter one from per-pair bounds (the columns' BF16 rounding-error norms) on
// the candidates alone.  Where the cut comes from is the MODE of the kernel:
// a threshold from a sample of the references (a first launch), or, where
// there are too few references to sample, the k-th best pessimistic key of the
// thread's own share so far, kept as a sorted list in registers.
//
// Hot test.  An epilogue thread tests x = a s - w[r] against one threshold
// e_thr per query (a = 1, w = 0 for cosine; a = 2, w = (1 - c) Nr for
// euclidean, c = rel + 2^-20; w = +inf for degenerate and padding references),
// and only references passing it get their exact key bounds.  For euclidean
// 2 rel sqrt(Nq Nr) <= rel (Nq + Nr), so hi <= 2 s - (1 - c)(Nq + Nr) + 1e-30
// and hi >= cut implies x >= cut + (1 - c) Nq; for cosine hi = s + rel.
// e_thr subtracts 2^-12 (|cut| + Nq) (euclidean) or 2^-12 (|cut| + 1)
// (cosine) more, far above the FP32 rounding of x.  Two 32-column chunks are
// tested together: their maxima (trees of three-input maxima), one vote, and
// only in a chunk that holds a passing reference the mask and the picks.  The
// weights of a tile half are fetched a tile ahead, one load per warp, and read
// from shared memory: read from global memory where they are used they cost
// the euclidean launch 5,165 us instead of 3,690 (4,096 x 2,000,000, d = 256).
//
// What bounds it: 4,096 x 2,000,000, cosine, k = 20, both launches: d = 256
// 2.28 ms (3.18 before the sample, the issue loop of one elected lane and
// pairs), d = 128 1.65 (2.65), d = 64 1.44 (2.50); euclidean d = 256 2.89
// (5.17).  At d = 256 the tensor pipe: 1.23 us for 128 x 256 x 256 products, 1.1
// times the rate of a measured cuBLAS burst; up to d = 128 the epilogue, which
// tests 32,768 keys a tile in 0.8 us.
//
// Warp roles (320 threads): warp 0 TMA producer, warp 1 TMEM allocator + MMA
// issuer, warps 2..9 epilogue.  Every mbarrier wait is bounded (1 s of
// %globaltimer, sdg_tc_ptx.cuh) and sleeps instead of spinning; a wait that
// runs out sets *status, raises the CTA's abort flag, and the CTA drains its
// own copies and MMAs, frees TMEM and returns.
//
// CTA pairs (PAIR = true).  A cluster of two CTAs shares each
// UMMA: the even CTA issues tcgen05.mma.cta_group::2 with M = 256 (its 128
// queries in rows 0-127, the odd CTA's in 128-255) and N = 256, each CTA
// holding its own query tile and one 128-column half of every reference chunk
// (16 KB, an 8-stage ring).  Both CTAs' TMA loads (cta_group::2) count their
// bytes on the even CTA's barriers, whose commits multicast to both CTAs; the
// odd CTA's epilogue releases the even CTA's accumulator barrier remotely;
// TMEM is allocated and freed by a warp of each CTA, and a cluster barrier
// keeps either CTA from leaving while the other may still touch its memory.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "../../include/sdgpu.h"
#include "sdg_dense.h"
#include "sdg_kth.cuh"
#include "sdg_tc_ptx.cuh"

namespace sdg {
namespace {

using namespace tc;

constexpr int BM = 128;                 // queries per group (UMMA M, TMEM lanes)
constexpr int BN = 256;                 // references per tile (UMMA N)
constexpr int BK = 64;                  // rows of a K chunk: 64 BF16 = one 128-byte swizzle row
constexpr int NB = 8;                   // buffered passing references per epilogue thread
constexpr int EPI_THREADS = 256;
constexpr int KT = 64;                  // largest k of the fused screen
constexpr int THREADS = 320;
constexpr uint32_t A_BYTES = BM * BK * 2;      // 16 KB: a 128 x 64 BF16 query chunk
constexpr uint32_t RING_BYTES = 128 * 1024;    // the reference chunk ring
constexpr uint32_t TMEM_COLS = 2 * BN;         // two accumulator buffers
constexpr int MAX_DCH = 4;              // dpad <= 256
constexpr int MAX_STAGES = 8;
// 1 KB alignment slack, A chunks, B ring, candidate slots, barriers
constexpr uint32_t W_BYTES = BN / 2 * 4;     // an epilogue warp's weights of one tile half
constexpr size_t SMEM_BYTES = 1024 + (size_t)MAX_DCH * A_BYTES + RING_BYTES + (size_t)NB * EPI_THREADS * 8 +
                              EPI_THREADS / 32 * W_BYTES + 256;

// One CTA (PAIR = false): a query group is 128 queries, the CTA loads whole
// 256-column reference chunks (32 KB, a 4-stage ring) and issues
// cta_group::1 MMAs (M = 128).  A CTA pair (PAIR = true, a cluster of two): a
// query group is 256 queries, 128 per CTA; each CTA loads its 128-column half
// of every reference chunk (16 KB, an 8-stage ring in the same bytes, so the
// ring covers twice the MMA time) and the even CTA issues cta_group::2 MMAs
// (M = 256, N = 256) over both CTAs' operands.
template <bool PAIR>
struct Cfg {
  static constexpr int GM = PAIR ? 2 * BM : BM;            // queries per group
  static constexpr int BNL = PAIR ? BN / 2 : BN;           // reference columns a CTA loads per chunk
  static constexpr uint32_t B_BYTES = BNL * BK * 2;
  static constexpr int STAGES = (int)(RING_BYTES / B_BYTES);
  static constexpr uint32_t IDESC = idesc_f16(GM, BN, true);
};
static_assert(Cfg<true>::STAGES <= MAX_STAGES && Cfg<false>::STAGES <= MAX_STAGES, "barrier space");

// The sample of every s-th reference.  The matrix is SAMPLE_RUNS runs of `span`
// references, a place of a run is s references, and sample tile t takes one
// reference (the (t mod s)-th) of each of SAMPLE_PLACES neighbouring places in
// every run.  A tile half is then spread over half of the matrix, so references
// stored class by class are sampled as evenly as shuffled ones: a tile of 256
// neighbouring places sees one class, the k-th best of the maxima lies outside a
// query's class, its lists overflow and the block repeats.  Screen us of
// references stored in cluster order with 2 / 16 / 64 / 256 runs: 400,000 x 128 in 100
// clusters 2,924 / 837 / 785 / 792, 1,000,000 x 256 in 1,000 3,921 / 3,110 / 2,087 /
// 1,997, 1,000,000 x 64 in 20,000 669 / 647 / 593 / 506; of others, 2,000,000 x 256:
// 2,249 / 2,268 / 2,274 / 2,462.
constexpr int SAMPLE_RUNS = 64, SAMPLE_PLACES = BN / SAMPLE_RUNS;
struct SampleMap {
  int s;
  int64_t span, tiles;
  // the reference of column c
  __host__ __device__ __forceinline__ int64_t at(int64_t c) const {
    const int64_t t = c / BN, col = c % BN;
    return col / SAMPLE_PLACES * span + (t * SAMPLE_PLACES + col % SAMPLE_PLACES) * s + t % s;
  }
  // the column of reference r, or -1
  __host__ __device__ __forceinline__ int64_t column(int64_t r) const {
    const int64_t run = r / span, p = r % span / s, t = p / SAMPLE_PLACES;
    if (run >= SAMPLE_RUNS || t >= tiles || r % span % s != t % s) return -1;
    return t * BN + run * SAMPLE_PLACES + p % SAMPLE_PLACES;
  }
};

struct TcArgs {
  int method, k, dch, ecap;
  int self;                   // queries are columns of the reference (skip r == q)
  int32_t d;
  int64_t n, q0, nq;          // references; the block's first query (index in Q) and size
  int64_t ntiles, tiles_per_cta, nslots;   // reference tiles; items per CTA; list slots per query
  float a;                    // x = a * s - w[r] (1 cosine, 2 euclidean)
  float one_minus_c;          // euclidean hot-test coefficient
  const float* w;             // [ntiles * BN]: +inf for degenerate / padding references
  const float* norm2;         // reference sums of squares
  const float* qnorm2;        // query sums of squares (index in Q)
  const uint8_t* qempty;      // degenerate queries (no list)
  unsigned* tshared;          // [nq]: the best running k-th pessimistic key of any list (ordered bits)
  float* lists;               // [nq][nslots][k] (one pass)
  float* maxima;              // MODE 1: [nq][2 * ntiles * gran]
  int gran;                   // MODE 1: maxima per tile half (1 or 4)
  SampleMap sample;           // MODE 1
  const int* gate;            // nothing to do unless *gate is set (null: always run)
  int use_w;                  // MODE 1, cosine: some reference is degenerate
  int32_t* ecount;            // [nq][nslots]
  int32_t* eidx;              // [nq][nslots][ecap]
  float* es;                  // [nq][nslots][ecap]: the appended references' GEMM values
  int* status;
  int stall;                  // failure-detection test: the MMA issuer's first wait never completes
};

// The order-preserving map of a float onto uint32: atomicMax on the keys is a
// max on the floats.
using kth::fkey;
using kth::fkey_value;
constexpr int SHARE_TILES = 8;          // tiles between exchanges of the shared running key

__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
// two FMAs in one instruction, each rounded as fmaf
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// a NaN loses to a number, as in fmaxf
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// the first and the last work unit (a CTA, or a CTA pair) whose span holds an
// item of query group g
__host__ __device__ __forceinline__ int64_t first_cta(int64_t g, int64_t ntiles, int64_t per) {
  return (g * ntiles) / per;
}
__host__ __device__ __forceinline__ int64_t last_cta(int64_t g, int64_t ntiles, int64_t per) {
  return ((g + 1) * ntiles - 1) / per;
}
// The reference tile of item f of group g.  A group's tiles are taken in cyclic
// order from (g ntiles) mod per, so that every work unit, which starts at a
// multiple of per, is at a tile congruent to its step number modulo per: at
// any time the units together read about ntiles / per places of the reference
// matrix instead of one place each.
__host__ __device__ __forceinline__ int32_t tile_of(int64_t f, int64_t g, int64_t ntiles, int64_t per) {
  return (int32_t)((f - g * ntiles + (g * ntiles) % per) % ntiles);
}

// MODE 0: running lists, one pass over the references; for few references.
// MODE 1 keeps no list: every thread stores the largest x' = a s - w[r] of each
// tile half (or of each of its four 32-column chunks) of a sample of the
// references, with w[r] chosen so that x' less a constant of the query is at
// most the reference's pessimistic key; the k-th largest of a query's maxima
// (k_tc_threshold) is then reached by k references, so it is at most the k-th
// best key, and with many times k maxima hardly below the sample's.
// MODE 2 (cosine) and 3 (euclidean) append the references that pass the hot
// test at that threshold.  A running list starts from nothing in every CTA and
// column half: for 777 queries x 150,001 references each of a query's 44 lists
// saw 3,500 references and took the slow path for a hundred of them, 80 % of
// the launch's instructions; 4,096 x 2,000,000 still appended 2,147 references
// a query where a sample of every 16th leaves 488.
template <int KL, bool PAIR, int MODE>
__global__ void __launch_bounds__(THREADS, 1) k_dense_tc(const __grid_constant__ CUtensorMap qmap,
                                                       const __grid_constant__ CUtensorMap rmap, TcArgs P) {
  using C = Cfg<PAIR>;
  constexpr int STAGES = C::STAGES;
  constexpr uint32_t B_BYTES = C::B_BYTES;
  extern __shared__ uint8_t smem_raw[];
  if (MODE == 0 && P.gate && !*P.gate) return;          // every thread of the grid alike
  uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = base;                                     // MAX_DCH query chunks
  uint8_t* sB = base + (size_t)MAX_DCH * A_BYTES;          // STAGES reference chunks
  // per epilogue thread NB (reference, GEMM value) slots, slot-major so that a
  // warp's accesses to one slot are conflict-free
  int32_t* buf_r = (int32_t*)(sB + (size_t)RING_BYTES);
  float* buf_s = (float*)(buf_r + NB * EPI_THREADS);
  float* wts = buf_s + NB * EPI_THREADS;                   // per epilogue warp: -w of its tile half
  uint64_t* bars = (uint64_t*)(wts + EPI_THREADS / 32 * (W_BYTES / 4));
  uint64_t* full = bars;
  uint64_t* emptyb = bars + MAX_STAGES;
  uint64_t* acc_full = bars + 2 * MAX_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* a_full = acc_empty + 2;
  uint64_t* a_empty = a_full + 1;
  uint64_t* mma_done = a_empty + 1;
  uint32_t* tmem_slot = (uint32_t*)(mma_done + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // this CTA's rank in its pair (0: the MMA issuer) and its work unit
  const uint32_t crank = PAIR ? cluster_rank() : 0u;
  const bool leader = crank == 0;
  const int64_t unit = PAIR ? (int64_t)(blockIdx.x >> 1) : (int64_t)blockIdx.x;
  const int64_t per = P.tiles_per_cta, ntiles = P.ntiles;
  const int64_t f0 = unit * per;
  const int64_t f1 = min(f0 + per, ((P.nq + C::GM - 1) / C::GM) * ntiles);
  const int dch = P.dch;
  // the bounded waits (CTA-scope acquire: the pair's barriers are completed
  // by TMA transactions, tcgen05 commits and the other CTA's arrivals, each
  // ordered by the barrier itself)
  auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return mbar_wait(bar, parity, abort_flag, P.status); };
  auto drain = [&](uint64_t* bar, uint32_t parity) { mbar_drain(bar, parity); };

  if (threadIdx.x == 0) {
    // a pair's MMA waits on the even CTA's barriers: both CTAs' loads count
    // their bytes there, and both CTAs' epilogues release its buffers
    for (int s = 0; s < STAGES; ++s) { mbar_init(full + s, 1); mbar_init(emptyb + s, 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, PAIR ? 16 : 8); }
    mbar_init(a_full, 1);
    mbar_init(a_empty, 1);
    mbar_init(mma_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if constexpr (PAIR) tmem_alloc_pair(tmem_slot, TMEM_COLS);
    else tmem_alloc(tmem_slot, TMEM_COLS);
  }
  fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync();            // both CTAs' barriers exist before any remote arrival
  fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ---- TMA producer ----
    if (lane == 0 && f1 > f0) {
      prefetch_map(&qmap);
      prefetch_map(&rmap);
      int it = 0, seg = 0;
      bool ok = true;
      for (int64_t f = f0; f < f1 && ok; ++seg) {
        const int64_t g = f / ntiles;
        const int64_t fe = min(f1, (g + 1) * ntiles);
        // the previous segment's MMAs have finished reading the query chunks
        if (!wait(a_empty, ((uint32_t)seg & 1u) ^ 1u)) break;
        const int qy = (int)(P.q0 + g * C::GM + crank * BM);
        if constexpr (PAIR) {
          // both CTAs' query chunks are counted on the even CTA's barrier
          if (leader) mbar_expect_tx(a_full, 2u * (uint32_t)dch * A_BYTES);
          const uint32_t bar = cluster_addr(a_full, 0);
          for (int c = 0; c < dch; ++c) tma_load_2d_pair(sA + (size_t)c * A_BYTES, &qmap, bar, c * BK, qy);
        } else {
          mbar_expect_tx(a_full, (uint32_t)dch * A_BYTES);
          for (int c = 0; c < dch; ++c) tma_load_2d(sA + (size_t)c * A_BYTES, &qmap, a_full, c * BK, qy);
        }
        int32_t tile = tile_of(f, g, ntiles, per);
        for (; f < fe && ok; ++f, tile = tile + 1 < (int32_t)ntiles ? tile + 1 : 0) {
          const int rcol = tile * BN + (int)crank * C::BNL;
          for (int c = 0; c < dch; ++c, ++it) {
            const int s = it % STAGES;
            const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
            if (!wait(emptyb + s, ph ^ 1u)) { ok = false; break; }
            if constexpr (PAIR) {
              if (leader) mbar_expect_tx(full + s, 2u * B_BYTES);
              const uint32_t bar = cluster_addr(full + s, 0);
              if constexpr (MODE == 1)
                tma_load_4d_pair(sB + (size_t)s * B_BYTES, &rmap, bar, c * BK, tile % P.sample.s, tile * SAMPLE_PLACES,
                                 (int)crank * (SAMPLE_RUNS / 2));
              else
                tma_load_2d_pair(sB + (size_t)s * B_BYTES, &rmap, bar, c * BK, rcol);
            } else {
              mbar_expect_tx(full + s, B_BYTES);
              if constexpr (MODE == 1)
                tma_load_4d(sB + (size_t)s * B_BYTES, &rmap, full + s, c * BK, tile % P.sample.s, tile * SAMPLE_PLACES,
                            0);
              else
                tma_load_2d(sB + (size_t)s * B_BYTES, &rmap, full + s, c * BK, rcol);
            }
          }
        }
      }
      // every issued copy lands before the CTA can exit; a pair's copies are
      // counted on the even CTA's barriers, so the even CTA waits for both
      // CTAs' (the odd CTA leaves only after it, at the final cluster barrier)
      if (!PAIR || leader) {
        for (int x = max(0, it - STAGES); x < it; ++x) drain(full + x % STAGES, (uint32_t)(x / STAGES) & 1u);
        if (seg > 0) drain(a_full, (uint32_t)(seg - 1) & 1u);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (!PAIR || leader) {
      // ---- MMA issuer: the whole warp walks the loop, one lane issues ----
      if (f1 > f0) {
        const bool one = elect_one();
        auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool {
          return __all_sync(0xffffffffu, wait(bar, parity));
        };
        const uint32_t a_lo = sw128_desc_lo(smem_u32(sA)), b_lo = sw128_desc_lo(smem_u32(sB));
        int it = 0, seg = 0;
        int64_t j = 0;
        bool ok = true;
        for (int64_t f = f0; f < f1 && ok; ++seg) {
          const int64_t g = f / ntiles;
          const int64_t fe = min(f1, (g + 1) * ntiles);
          if (!wait_all(a_full, (uint32_t)seg & 1u)) break;
          fence_after();
          for (; f < fe && ok; ++f, ++j) {
            const int buf = (int)(j & 1);
            // the epilogue has drained this buffer's previous tile
            // (with P.stall the first wait asks for the phase the epilogue has not
            // begun, so it runs out: the failure-detection test's path)
            const uint32_t flip = (P.stall && j == 0) ? 0u : 1u;
            if (!wait_all(acc_empty + buf, ((uint32_t)(j >> 1) & 1u) ^ flip)) {
              ok = false;
              break;
            }
            fence_after();
            const uint32_t d_addr = tmem + (uint32_t)(buf * BN);
            for (int c = 0; c < dch; ++c, ++it) {
              const int s = it % STAGES;
              const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
              if (!wait_all(full + s, ph)) { ok = false; break; }
              fence_after();
              const uint32_t al = a_lo + (uint32_t)c * (A_BYTES >> 4), bl = b_lo + (uint32_t)s * (B_BYTES >> 4);
              if (one) {
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk) {
                  if constexpr (PAIR) umma_f16_pair(d_addr, al + kk * 2, bl + kk * 2, C::IDESC, (c | kk) != 0);
                  else umma_f16(d_addr, al + kk * 2, bl + kk * 2, C::IDESC, (c | kk) != 0);
                }
                // the stage is free (in both CTAs of a pair) once these MMAs have read it
                if constexpr (PAIR) umma_commit_pair(emptyb + s, 3); else umma_commit(emptyb + s);
                // after the last chunk: the tile's accumulators are complete
                if (c == dch - 1) {
                  if constexpr (PAIR) umma_commit_pair(acc_full + buf, 3); else umma_commit(acc_full + buf);
                }
              }
              __syncwarp();
            }
            if (!ok) break;
          }
          // the query chunks are free once the segment's MMAs are done
          if (one) {
            if constexpr (PAIR) umma_commit_pair(a_empty, 3); else umma_commit(a_empty);
          }
          __syncwarp();
        }
        // all issued MMAs complete before TMEM is freed
        if (one) {
          if constexpr (PAIR) umma_commit_pair(mma_done, 3); else umma_commit(mma_done);
        }
        __syncwarp();
        drain(mma_done, 0);
      }
    } else if constexpr (PAIR) {
      // the odd CTA: the even CTA's last commit also arrives on this CTA's
      // barriers; it lands before they go away
      if (lane == 0 && f1 > f0) drain(mma_done, 0);
    }
    __syncwarp();
  } else {
    // ---- epilogue: one thread per (query, column half) ----
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;
    const int K = P.k;
    const int32_t d = P.d;
    const float rel = 0.0040f + (float)d * 2.384185791015625e-7f;
    // known at compile time where references are appended (see MODE)
    const bool cosine = MODE == 2 || (MODE != 3 && P.method == COSINE);
    constexpr bool APPEND = MODE >= 2;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int et = threadIdx.x - 64;                  // epilogue thread 0 .. 255

    // per-segment state
    bool active = false;
    int64_t q = 0;
    float Nq = 0.f;
    // this thread's top k pessimistic keys, sorted descending, in registers:
    // KL - k leading +inf sentinels, so that lst[KL - 1] is the k-th best
    float lst[KL];
    float T = -INFINITY;                       // k-th best pessimistic key of this list so far
    // the best running k-th key of any of the query's lists (segments and
    // halves running on other warps and CTAs), exchanged every SHARE_TILES
    // tiles: each is the k-th best of a subset, so their maximum never
    // exceeds the query's final k-th best and may stand in for T in every test
    float Ts = -INFINITY;
    // hot-loop threshold on x; finite, so that x = -inf (degenerate or padding
    // references) never passes
    float e_thr = -FLT_MAX;
    int cnt = 0, nbuf = 0;
    int32_t* my_idx = P.eidx;
    float* my_s = P.es;

    // hi >= cut implies x >= e_thr (the hot-test bound in the file header),
    // with 2^-12 slack for the FP32 roundings of x and e_thr
    auto set_thr = [&]() {
      const float cut = dense_cut(fmaxf(T, Ts));
      e_thr = cosine ? cut - rel - (2.44140625e-4f * (fabsf(cut) + 1.f) + 1e-30f)
                     : cut + P.one_minus_c * Nq - (2.44140625e-4f * (fabsf(cut) + Nq) + 1e-30f);
      e_thr = fmaxf(-FLT_MAX, e_thr);
    };
    // The exact key bounds of one reference r with GEMM value s (the slow
    // path): append it if its optimistic key reaches the running cut, insert
    // its pessimistic key into the running top k and tighten the hot test.
    // Degenerate and padding references carry w = +inf and are skipped (their
    // GEMM value is exactly 0, so w is read only then).
    auto process = [&](int64_t r, float s) {
      if (P.self && r == q) return;
      if (s == 0.f && P.w[r] == INFINITY) return;
      const float Nr = cosine ? 0.f : P.norm2[r];
      float key, err;
      dense_key(P.method, 0, d, s, Nq, Nr, key, err);
      const float lo = key - err, hi = key + err;
      const float Te = fmaxf(T, Ts);
      if (hi >= dense_cut(Te)) {
        if (cnt < P.ecap) { my_idx[cnt] = (int32_t)r; my_s[cnt] = s; }
        ++cnt;
      }
      if (lo > Te) {
        // sorted insert: the new lst[i] is the median of lst[i - 1], lo, lst[i]
#pragma unroll
        for (int i = KL - 1; i > 0; --i) lst[i] = fmaxf(lst[i], fminf(lst[i - 1], lo));
        lst[0] = fmaxf(lst[0], lo);
        T = lst[KL - 1];
        set_thr();
      }
    };
    // Passing references wait in this thread's NB slots and are processed by
    // the whole warp at once when some lane's slots run out (and at the end of
    // a segment); a deferred reference is judged against the cut current when
    // it is processed, which is never above the final one.
    auto flush = [&]() {
      const int nmax = __reduce_max_sync(0xffffffffu, nbuf);
      for (int i = 0; i < nmax; ++i)
        if (i < nbuf) process(buf_r[i * EPI_THREADS + et], buf_s[i * EPI_THREADS + et]);
      nbuf = 0;
      __syncwarp();
    };
    // The hot test's x of one 32-reference chunk at column c0 of the tile half
    float* sw = wts + (warp - 2) * (W_BYTES / 4);
    const uint64_t aa = pack2(P.a, P.a);
    auto values = [&](const uint32_t (&v)[32], int c0, bool weigh, float (&x)[32]) {
      if (weigh) {
        const ulonglong2* w2 = reinterpret_cast<const ulonglong2*>(sw + c0);
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const ulonglong2 ww = w2[t];
          unpack2(fma2(aa, pack2(__uint_as_float(v[4 * t]), __uint_as_float(v[4 * t + 1])), ww.x), x[4 * t],
                  x[4 * t + 1]);
          unpack2(fma2(aa, pack2(__uint_as_float(v[4 * t + 2]), __uint_as_float(v[4 * t + 3])), ww.y), x[4 * t + 2],
                  x[4 * t + 3]);
        }
      } else {
#pragma unroll
        for (int t = 0; t < 32; ++t) x[t] = __uint_as_float(v[t]);
      }
    };
    auto maximum = [](const float (&x)[32]) -> float {
      float m[11];
#pragma unroll
      for (int t = 0; t < 10; ++t) m[t] = max3(x[3 * t], x[3 * t + 1], x[3 * t + 2]);
      m[10] = fmaxf(x[30], x[31]);
#pragma unroll
      for (int t = 0; t < 3; ++t) m[t] = max3(m[3 * t], m[3 * t + 1], m[3 * t + 2]);
      m[3] = fmaxf(m[9], m[10]);
      return fmaxf(max3(m[0], m[1], m[2]), m[3]);
    };
    // the bits t of x[t] >= e_thr
    auto mask_of = [&](const float (&x)[32]) -> uint32_t {
      uint32_t b[16];
#pragma unroll
      for (int t = 0; t < 16; ++t)
        b[t] = (x[2 * t] >= e_thr ? 1u << (2 * t) : 0u) | (x[2 * t + 1] >= e_thr ? 2u << (2 * t) : 0u);
#pragma unroll
      for (int wdt = 8; wdt > 0; wdt >>= 1)
#pragma unroll
        for (int t = 0; t < wdt; ++t) b[t] |= b[t + wdt];
      return b[0];
    };
    // The mask of the references of one chunk with x >= e_thr (0 for an
    // inactive lane); the warp leaves together when no lane's maximum passes
    auto hot_mask = [&](const uint32_t (&v)[32], int c0) -> uint32_t {
      float x[32];
      values(v, c0, !cosine, x);
      const bool hit = active && maximum(x) >= e_thr;
      if (!__any_sync(0xffffffffu, hit)) return 0u;
      return hit ? mask_of(x) : 0u;
    };
    // v[jj] as a five-level tree of selects on the bits of jj
    auto pick = [](const uint32_t (&v)[32], int jj) -> float {
      uint32_t a[16];
#pragma unroll
      for (int t = 0; t < 16; ++t) a[t] = (jj & 1) ? v[2 * t + 1] : v[2 * t];
#pragma unroll
      for (int lvl = 1, wdt = 8; wdt > 0; ++lvl, wdt >>= 1)
#pragma unroll
        for (int t = 0; t < wdt; ++t) a[t] = ((jj >> lvl) & 1) ? a[2 * t + 1] : a[2 * t];
      return __uint_as_float(a[0]);
    };
    // The passing references of one chunk into this lane's slots (lanes
    // converged): the warp flushes first if some lane's slots would overflow;
    // a lane with more than NB of them (only while its list is filling) takes
    // the slow path at once.
    auto take = [&](const uint32_t (&v)[32], uint32_t mask, int64_t r0) {
      const int nnew = __popc(mask);
      if (__any_sync(0xffffffffu, nbuf + nnew > NB)) flush();
      if (nnew > NB) {
        while (mask) {
          const int jj = __ffs(mask) - 1;
          mask &= mask - 1;
          process(r0 + jj, pick(v, jj));
        }
      } else {
        while (mask) {
          const int jj = __ffs(mask) - 1;
          mask &= mask - 1;
          buf_r[nbuf * EPI_THREADS + et] = (int32_t)(r0 + jj);
          buf_s[nbuf * EPI_THREADS + et] = pick(v, jj);
          ++nbuf;
        }
      }
      __syncwarp();
    };

    // MODE 2: a chunk's passing references straight to the list; mx: this
    // lane's maximum (-inf for an inactive lane).  x is formed again where a
    // lane passes: held since the test, a pair's would be 64 more registers.
    auto append = [&](const uint32_t (&v)[32], float mx, int c0, int64_t r0) {
      if (!__any_sync(0xffffffffu, mx >= e_thr)) return;
      float x[32];
      values(v, c0, !cosine, x);
      uint32_t mask = mx >= e_thr ? mask_of(x) : 0u;
      while (mask) {
        const int jj = __ffs(mask) - 1;
        mask &= mask - 1;
        const float sv = pick(v, jj);
        const int64_t r = r0 + jj;
        if ((P.self && r == q) || (sv == 0.f && P.w[r] == INFINITY)) continue;
        if (cnt < P.ecap) { my_idx[cnt] = (int32_t)r; my_s[cnt] = sv; }
        ++cnt;
      }
      __syncwarp();
    };
    int64_t own = -1;                                 // MODE 1: the query's own column of the sample
    // MODE 1: the largest x' of one chunk; weigh: subtract w[r] (+inf for
    // degenerate and padding references)
    auto chunk_max = [&](const uint32_t (&v)[32], int64_t r0, int c0, bool weigh) -> float {
      float x[32];
      values(v, c0, weigh, x);
      if (P.self && __any_sync(0xffffffffu, own >= r0 && own < r0 + 32)) {
#pragma unroll
        for (int t = 0; t < 32; ++t)
          if (r0 + t == own) x[t] = -INFINITY;
      }
      return maximum(x);
    };
    // this lane's four weights of the tile half that comes next
    const bool weighted = !cosine || MODE == 1;
    float4 wn = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch_w = [&](int32_t tile) {
      if (weighted) wn = __ldg(reinterpret_cast<const float4*>(P.w + (int64_t)tile * BN + half * (BN / 2)) + lane);
    };

    int64_t j = 0;                                    // tile counter (the MMA's order)
    bool ok = true;
    for (int64_t f = f0; f < f1 && ok;) {
      const int64_t g = f / ntiles;
      const int64_t fe = min(f1, (g + 1) * ntiles);
      const int64_t ql = g * C::GM + crank * BM + row;
      q = P.q0 + ql;
      active = ql < P.nq;
      if (active) active = !P.qempty[q];           // a degenerate query has no list
      Nq = active ? P.qnorm2[q] : 0.f;
      if (MODE == 1) own = P.sample.column(q);
#pragma unroll
      for (int i = 0; i < KL; ++i) lst[i] = (i < KL - K) ? INFINITY : -INFINITY;
      T = -INFINITY;
      Ts = (MODE != 1 && active) ? fkey_value(*(volatile unsigned*)(P.tshared + ql)) : -INFINITY;
      e_thr = -FLT_MAX;
      if (Ts > -INFINITY) set_thr();
      cnt = 0;
      nbuf = 0;
      const int64_t slot =
          active ? (ql * P.nslots + (unit - first_cta(g, ntiles, per)) * 2 + half) : 0;
      my_idx = P.eidx + slot * P.ecap;
      my_s = P.es + slot * P.ecap;
      int32_t tile = tile_of(f, g, ntiles, per);
      fetch_w(tile);
      for (int32_t next = 0; f < fe; ++f, ++j, tile = next) {
        next = tile + 1 < (int32_t)ntiles ? tile + 1 : 0;
        if (weighted) {
          __syncwarp();
          reinterpret_cast<float4*>(sw)[lane] = make_float4(-wn.x, -wn.y, -wn.z, -wn.w);
          __syncwarp();
          fetch_w(next);
        }
        const int buf = (int)(j & 1);
        const bool got = wait(acc_full + buf, (uint32_t)(j >> 1) & 1u);
        if (!__all_sync(0xffffffffu, got)) { ok = false; break; }   // the warp leaves together
        fence_after();
        const int64_t r_half = (int64_t)tile * BN + half * (BN / 2);
        const uint32_t tb = tmem + lane_base + (uint32_t)(buf * BN + half * (BN / 2));
        // the buffer goes back to the MMAs as soon as its last TMEM reads are
        // done (the values being processed are in registers by then): the
        // hand-off to the next-but-one tile does not wait for the processing
        auto release = [&]() {
          fence_before();
          __syncwarp();
          if (lane == 0) {
            if constexpr (PAIR) mbar_arrive_remote(acc_empty + buf, 0);   // the even CTA's MMA waits on it
            else mbar_arrive(acc_empty + buf);
          }
        };
        if constexpr (MODE == 1) {
          // the chunks' largest x'
          float cm[4];
          const bool weigh = !cosine || P.use_w || r_half + BN / 2 > P.n;
#pragma unroll
          for (int hh = 0; hh < BN / 64; hh += 2) {
            uint32_t va[32], vb[32];
            tmem_ld32_issue(tb + hh * 32, va);
            tmem_ld32_issue(tb + hh * 32 + 32, vb);
            tmem_ld_wait(va);
            tmem_ld_wait(vb);
            if (hh == BN / 64 - 2) release();
            cm[hh] = chunk_max(va, r_half + hh * 32, hh * 32, weigh);
            cm[hh + 1] = chunk_max(vb, r_half + hh * 32 + 32, hh * 32 + 32, weigh);
          }
          if (active) {
            float* out = P.maxima + ql * (2 * ntiles * P.gran) + ((int64_t)tile * 2 + half) * P.gran;
            if (P.gran == 4) *reinterpret_cast<float4*>(out) = make_float4(cm[0], cm[1], cm[2], cm[3]);
            else *out = fmaxf(fmaxf(cm[0], cm[1]), fmaxf(cm[2], cm[3]));
          }
        } else if constexpr (KL <= 32) {
          // chunks in pairs (the TMEM loads take a few tens of cycles; the
          // pair's hot tests overlap)
#pragma unroll 1
          for (int hh = 0; hh < BN / 64; hh += 2) {
            uint32_t va[32], vb[32];
            tmem_ld32_issue(tb + hh * 32, va);
            tmem_ld32_issue(tb + hh * 32 + 32, vb);
            tmem_ld_wait(va);
            tmem_ld_wait(vb);
            if (hh == BN / 64 - 2) release();
            if constexpr (APPEND) {
              float x[32], y[32];
              values(va, hh * 32, !cosine, x);
              values(vb, hh * 32 + 32, !cosine, y);
              const float mx = active ? maximum(x) : -INFINITY, my = active ? maximum(y) : -INFINITY;
              if (__any_sync(0xffffffffu, fmaxf(mx, my) >= e_thr)) {
                append(va, mx, hh * 32, r_half + hh * 32);
                append(vb, my, hh * 32 + 32, r_half + hh * 32 + 32);
              }
            } else {
              const uint32_t ma = hot_mask(va, hh * 32), mb = hot_mask(vb, hh * 32 + 32);
              if (__any_sync(0xffffffffu, (ma | mb) != 0u)) {
                take(va, ma, r_half + hh * 32);
                take(vb, mb, r_half + hh * 32 + 32);
              }
            }
          }
        } else {
          // longer lists leave registers for one chunk at a time
#pragma unroll 1
          for (int hh = 0; hh < BN / 64; ++hh) {
            uint32_t va[32];
            tmem_ld32(tb + hh * 32, va);
            if (hh == BN / 64 - 1) release();
            const uint32_t ma = hot_mask(va, hh * 32);
            if (__any_sync(0xffffffffu, ma != 0u)) take(va, ma, r_half + hh * 32);
          }
        }
        if (MODE == 0 && (j & (SHARE_TILES - 1)) == SHARE_TILES - 1 && active) {
          // publish this list's running key and take the best one published
          const unsigned prev = atomicMax(P.tshared + ql, fkey(T));
          const float best = fmaxf(fkey_value(prev), T);
          if (best > Ts) { Ts = best; set_thr(); }
        }
      }
      if constexpr (MODE == 0) {
        flush();
        if (active) atomicMax(P.tshared + ql, fkey(T));
        if (active) {
          float* out = P.lists + slot * K;
#pragma unroll
          for (int i = 0; i < KL; ++i)
            if (i >= KL - K) out[i - (KL - K)] = lst[i];
        }
      }
      if (MODE != 1 && active) P.ecount[slot] = cnt;
    }
  }
  fence_before();
  __syncthreads();
  // a pair's MMAs read both CTAs' shared memory and write both TMEMs: neither
  // CTA frees TMEM or exits before the other is done
  if constexpr (PAIR) cluster_sync();
  fence_after();
  if (warp == 1) {
    if constexpr (PAIR) tmem_dealloc_pair(tmem, TMEM_COLS);
    else tmem_dealloc(tmem, TMEM_COLS);
  }
}

// ---- merge: the final cut of each query over its lists ---------------------
// Warps per query: 32 for a handful of queries, 8 while a warp per query would
// leave an SM fewer than 16 warps, else 1.  One query over 302 lists: 113 us
// with 8 warps; 777 over 44: 47 us with 8 against 150 with 1; 3,000: 98 and
// 99; 4,096: 124 and 114; 16,384: 302 and 137.
constexpr int64_t MERGE_WIDEST_MAX = 152 * 2, MERGE_WIDE_MAX = 152 * 16;

struct MergeArgs {
  int64_t q0, nq;
  int gm;                      // queries per group
  int64_t ntiles, per, nslots;
  int K, ecap, method;
  int32_t d;
  const uint8_t* qempty;
  const unsigned* tshared;
  const float* lists;
  const int32_t* ecount;
  const int32_t* eidx;
  const float* es;
  const float* norm2;          // reference sums of squares
  const float* qnorm2;         // query sums of squares (index in Q)
  const float *re, *rn;        // reference copies: rounding-error norm, norm (the method's copy)
  const float *qe, *qn;        // query copies (index in Q)
  int cap;
  int32_t* cand;
  float* cand_s;               // [nq][cap] the candidates' GEMM values
  int32_t* count;
  int32_t* over;
  size_t smem_query;           // shared-memory bytes of one query's prefix and keys
  int* any_over;               // set when a query's list overflows (or null)
  const int* gate;             // nothing to do unless *gate is set (null: always run)
};

// The per-pair bound of one candidate from the columns' BF16 copies: with v
// the exact (unit) columns and b their BF16 copies, |sum v_q v_r - sum b_q b_r|
// <= e_q ||v_r|| + ||b_q|| e_r (Cauchy-Schwarz; e = ||v - b||, computed in
// FP64 and rounded up at upload), the BF16 products are exact in FP32 and the
// tensor cores' FP32 accumulation of d products is allowed (d + 64) 2^-21
// ||b_q|| ||b_r||; ||v_r|| is 1 (unit columns) or sqrt(Nr).  The key is the
// screen's (s for cosine, 2 s - Nq - Nr for euclidean) with the FP32 roundings
// of Nq, Nr and the key allowed 2^-20 of the terms.
__device__ __forceinline__ void tight_bounds(const MergeArgs& A, float s, int64_t r, float Nq, float qe, float qn,
                                             float& lo, float& hi) {
  const float acc = (float)(A.d + 64) * 4.76837158203125e-7f;     // 2^-21
  if (A.method == COSINE) {
    const float E = (1.000001f * qe * 1.000001f + qn * A.re[r] + acc * qn * A.rn[r]) * 1.01f + 1e-12f +
                    2.384185791015625e-7f * fabsf(s);               // 2^-22 |s|
    lo = s - E;
    hi = s + E;
  } else {
    const float Nr = A.norm2[r];
    const float Es = (qe * sqrtf(Nr) * 1.000001f + qn * A.re[r] + acc * qn * A.rn[r]) * 1.01f + 1e-30f;
    const float key = 2.f * s - (Nq + Nr);
    const float E = 2.f * Es + 9.5367431640625e-7f * (Nq + Nr + 2.f * fabsf(s)) + 1e-30f;
    lo = key - E;
    hi = key + E;
  }
}

// Per query: T = the k-th largest pessimistic key over the lists of every
// (segment, half) that covered it (the exact k-th over all references: the top
// k of a union is the top k of the parts' top k), cut = dense_cut(T); the
// candidates are the appended references with hi >= cut, hi the uniform bound
// of the screen.  A second, tighter cut follows on the candidates alone: T2 =
// the k-th largest per-pair lower bound (tight_bounds) among them is again at
// most the exact k-th best key (k candidates reach it), so every member of the
// exact top k (ties included) has its per-pair upper bound at or above
// dense_cut(max(T, T2)) and is kept.  Where more pass the first cut than the table
// holds, T2 is taken over all appended references instead (400,000 references in 50
// clusters, 1,000 queries, k = 5: 913 queries had 576 and more; the block repeated
// with running lists and 26 queries still went through exact rows, 223 ms; 9 ms now
// and 1 such query).
//
// A list keeps only keys above the shared key it saw, so when some list's
// view of the shared key reached the final k-th best, fewer than k keys at or
// above it may be listed; the shared key (the k-th best of a subset, never
// above the final) then is the final k-th best.  So only keys above the
// shared key are collected (in shared memory), and T is their k-th largest
// (kth::largest) or, with fewer than k of them, the shared key.
//
// WPQ warps work on a query, its appended references as one flat range over
// the lists (a shared-memory prefix of their counts, a binary search per
// reference), so their loads do not wait on one another.  What bounds it is
// latency: one warp taking a query's lists in turn, with k-long sorted
// insertions, took 606 us for one query over 302 lists, 209 us for 777 queries
// over 44, 170 us for 3,000 (k = 30) over 14 and 143 us for 4,096 over 12.
__host__ __device__ __forceinline__ size_t merge_prefix_bytes(int64_t nslots) { return (size_t)((nslots + 4) / 4 * 4) * 4; }

template <int WPQ>
__global__ void __launch_bounds__(WPQ == 1 ? 256 : WPQ * 32) k_tc_merge(MergeArgs A) {
  extern __shared__ __align__(16) unsigned char msm[];
  constexpr int QPB = WPQ == 1 ? 8 : 1;
  __shared__ uint32_t red[WPQ];
  __shared__ int s_count[QPB], s_kept[QPB];
  const int lane = threadIdx.x & 31;
  const int slot_q = WPQ == 1 ? (int)(threadIdx.x >> 5) : 0;
  if (A.gate && !*A.gate) return;                        // every thread of the grid alike
  const int64_t ql = (int64_t)blockIdx.x * QPB + slot_q;
  if (ql >= A.nq) return;
  const kth::Group<WPQ> G{red};
  const int rank = G.rank(), nt = G.size();
  const int K = A.K;
  int32_t* pre = reinterpret_cast<int32_t*>(msm + (size_t)slot_q * A.smem_query);    // inclusive list counts
  uint32_t* keys = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(pre) + merge_prefix_bytes(A.nslots));
  if (A.qempty[A.q0 + ql]) {
    if (rank == 0) { A.count[ql] = 0; A.over[ql] = 0; }
    return;
  }
  const int64_t g = ql / A.gm;
  const int used = (int)(2 * (last_cta(g, A.ntiles, A.per) - first_cta(g, A.ntiles, A.per) + 1));
  const float ts = fkey_value(A.tshared[ql]);
  if (rank == 0) s_count[slot_q] = s_kept[slot_q] = 0;
  // the lists' counts, scanned by the group's first warp
  bool big = false;
  if (rank < 32) {
    int run = 0;
    for (int r0 = 0; r0 < used; r0 += 32) {
      const int c = r0 + lane < used ? A.ecount[ql * A.nslots + r0 + lane] : 0;
      if (c > A.ecap) big = true;
      int x = min(c, A.ecap);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (r0 + lane < used) pre[r0 + lane] = run + x;
      run += __shfl_sync(0xffffffffu, x, 31);
    }
  }
  bool ovf = G.sum(big ? 1u : 0u) != 0;
  G.sync();
  if (ovf) {
    if (rank == 0) {
      A.count[ql] = 0;
      A.over[ql] = 1;
      if (A.any_over) *A.any_over = 1;
    }
    return;
  }
  // T from the keys above the shared one
  const float* in = A.lists ? A.lists + ql * A.nslots * (int64_t)K : nullptr;   // two passes: T is the shared key
  const int tot = in ? used * K : 0;
  for (int p = rank; p < tot; p += nt) {
    const float v = in[p];
    if (v > ts) keys[atomicAdd(&s_count[slot_q], 1)] = fkey(v);
  }
  G.sync();
  int n = s_count[slot_q];
  const float T = n >= K ? fkey_value(kth::largest<WPQ>(G, keys, n, K)) : ts;
  const float cut = dense_cut(T);
  const int64_t q = A.q0 + ql;
  const float Nq = A.qnorm2[q];
  int32_t* out = A.cand + ql * (int64_t)A.cap;
  float* out_s = A.cand_s + ql * (int64_t)A.cap;
  const int all = pre[used - 1];
  auto place = [&](int p) -> int64_t {                // of the p-th appended reference
    int lo = 0, hi = used - 1;                       // the first list whose inclusive count exceeds p
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (pre[mid] > p) hi = mid;
      else lo = mid + 1;
    }
    return (ql * A.nslots + lo) * (int64_t)A.ecap + (p - (lo ? pre[lo - 1] : 0));
  };
  for (int p = rank; p < all; p += nt) {
    const int64_t at = place(p);
    const int32_t ref = A.eidx[at];
    const float sv = A.es[at];
    float key, err;
    dense_key(A.method, 0, A.d, sv, Nq, A.method == COSINE ? 0.f : A.norm2[ref], key, err);
    if (key + err >= cut) {
      const int w = atomicAdd(&s_kept[slot_q], 1);
      if (w < A.cap) { out[w] = ref; out_s[w] = sv; }
    }
  }
  G.sync();                                          // the kept pairs are visible to the group
  int total = s_kept[slot_q];
  const float qe = A.qe[q], qn = A.qn[q];
  if (total > A.cap) {
    // More than the table holds (a query in a dense cluster, whose references lie
    // within the uniform bound of one another): the second cut is taken over all
    // appended references, T2 by a histogram of eight bits of the key at a time.
    uint32_t prefix = 0, want = (uint32_t)K;
    for (int shift = 24; shift >= 0; shift -= 8) {
      for (int i = rank; i < 256; i += nt) keys[i] = 0u;
      G.sync();
      for (int p = rank; p < all; p += nt) {
        const int64_t at = place(p);
        float lo, hi;
        tight_bounds(A, A.es[at], A.eidx[at], Nq, qe, qn, lo, hi);
        const uint32_t key = fkey(fmaxf(lo, -INFINITY));
        if (shift == 24 || (key >> (shift + 8)) == prefix) atomicAdd(&keys[(key >> shift) & 255u], 1u);
      }
      G.sync();
      // lane l: bins 255 - 8 l downwards (every warp of the group alike)
      uint32_t own = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) own += keys[255 - 8 * lane - j];
      uint32_t x = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      const int src = __ffs(__ballot_sync(0xffffffffu, x >= want)) - 1;   // all >= want: some lane reaches it
      uint32_t above = x - own;
      int bin = 255 - 8 * lane;
#pragma unroll
      for (int j = 0; j < 7; ++j)
        if (bin == 255 - 8 * lane - j && above + keys[bin] < want) above += keys[bin--];
      prefix = (prefix << 8) | (uint32_t)__shfl_sync(0xffffffffu, bin, src);
      want -= __shfl_sync(0xffffffffu, above, src);
      G.sync();
    }
    const float cut2 = dense_cut(fmaxf(T, fkey_value(prefix)));
    if (rank == 0) s_kept[slot_q] = 0;
    G.sync();
    for (int p = rank; p < all; p += nt) {
      const int64_t at = place(p);
      const int32_t ref = A.eidx[at];
      const float sv = A.es[at];
      float lo, hi;
      tight_bounds(A, sv, ref, Nq, qe, qn, lo, hi);
      if (hi >= cut2) {
        const int w = atomicAdd(&s_kept[slot_q], 1);
        if (w < A.cap) { out[w] = ref; out_s[w] = sv; }
      }
    }
    G.sync();
    total = s_kept[slot_q];
    ovf = total > A.cap;
  } else if (total > K) {
    for (int p = rank; p < total; p += nt) {
      float lo, hi;
      tight_bounds(A, out_s[p], out[p], Nq, qe, qn, lo, hi);
      keys[p] = fkey(fmaxf(lo, -INFINITY));          // NaN: no lower bound
    }
    G.sync();
    const float T2 = fkey_value(kth::largest<WPQ>(G, keys, total, K));
    const float cut2 = dense_cut(fmaxf(T, T2));
    if (rank == 0) s_kept[slot_q] = 0;
    G.sync();
    for (int p0 = 0; p0 < total; p0 += nt) {
      const int p = p0 + rank;
      bool keep = false;
      int32_t ref = 0;
      float sv = 0.f;
      if (p < total) {
        ref = out[p];
        sv = out_s[p];
        float lo, hi;
        tight_bounds(A, sv, ref, Nq, qe, qn, lo, hi);
        keep = hi >= cut2;
      }
      G.sync();                                      // every slot of this round is read before one is written
      if (keep) {
        const int w = atomicAdd(&s_kept[slot_q], 1);
        out[w] = ref;
        out_s[w] = sv;
      }
    }
    G.sync();
    total = s_kept[slot_q];
  }
  if (rank == 0) {
    A.count[ql] = ovf ? 0 : total;
    A.over[ql] = ovf ? 1 : 0;
  }
}

__global__ void k_tc_key_init(int64_t nq, unsigned* keys) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < nq) keys[i] = fkey(-INFINITY);
}

// w[r]: +inf for degenerate references and the padding; 0 (cosine) or
// (1 - c) Nr (euclidean) otherwise; wp: the same with one_plus_c for the x' of
// a first pass over n1 sampled references (at most nw; 0 without one)
__global__ void k_tc_weights(int method, int64_t n, int64_t nw, float one_minus_c,
                             const float* norm2, const uint8_t* empty, float* w, SampleMap sample,
                             int64_t n1, float one_plus_c, float* wp) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  auto weight = [&](int64_t r, float c) {
    if (r >= n || empty[r]) return INFINITY;
    return (method == COSINE) ? 0.f : c * norm2[r];
  };
  if (i < nw) w[i] = weight(i, one_minus_c);
  if (i < n1) wp[i] = weight(sample.at(i), one_plus_c);
}

// Two passes: each query's threshold, the k-th largest of its maxima less what
// separates x' from the pessimistic key.  Cosine: x' = s, lo = s - rel.
// Euclidean: x' = 2 s - (1 + c') Nr with c' = rel + 2^-19; 2 rel sqrt(Nq Nr) <=
// rel (Nq + Nr), so lo = 2 s - (Nq + Nr) - 2 rel sqrt(Nq Nr) - 2^-20 (Nq + Nr) -
// 1e-30 >= x' - (1 + c') Nq + 2^-20 (Nq + Nr) - 1e-30: the last but one term
// covers the FP32 roundings of (1 + c') N, 2^-21 |x'| that of x' and of the
// differences.  A warp per query; the m maxima are first folded into 256 (the
// k-th largest of the folded ones is reached by k references too, and for k <=
// 64 it is hardly lower), which sit in registers for the bit search of kth::largest.
__global__ void __launch_bounds__(256) k_tc_threshold(int method, int64_t q0, int64_t nq, int m, int K, float rel,
                                                      float one_plus_c, const float* qnorm2, const uint8_t* qempty,
                                                      const float* maxima, unsigned* tshared) {
  const int64_t ql = blockIdx.x * (int64_t)8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (ql >= nq) return;
  if (qempty[q0 + ql]) {
    if (lane == 0) tshared[ql] = fkey(-INFINITY);
    return;
  }
  const float* in = maxima + ql * m;
  float v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) v[c] = -INFINITY;
  for (int i = lane; i < m; i += 256)
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (i + 32 * c < m) v[c] = fmaxf(v[c], in[i + 32 * c]);
  uint32_t key[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) key[c] = fkey(v[c]);
  uint32_t ans = 0;
  for (int b = 31; b >= 0; --b) {
    const uint32_t t = ans | (1u << b);
    uint32_t n = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) n += key[c] >= t;
    if (__reduce_add_sync(0xffffffffu, n) >= (uint32_t)K) ans = t;
  }
  const float x = fkey_value(ans);
  if (lane == 0) {
    float T = -INFINITY;
    if (x > -INFINITY) {
      const float base = (method == COSINE) ? rel : one_plus_c * qnorm2[q0 + ql];
      T = x - base - (4.76837158203125e-7f * (fabsf(x) + base) + 1e-30f);
    }
    tshared[ql] = fkey(T);
  }
}

constexpr int64_t granularity(int64_t refs, int k) { return refs >= (int64_t)(BN / 2) * 8 * k ? 1 : 4; }
int64_t maxima_per_query(int64_t refs, int k) { return 2 * ((refs + BN - 1) / BN) * granularity(refs, k); }

// The stride of the sample whose maxima give each query's threshold; 0 (one pass
// with running lists) where even all references give fewer than 4 k maxima.  A
// stride of s leaves about s k references of a query above the threshold, and
// the 768 slots of the query's shortest set of lists (two) have to hold them
// with room to spare, hence s k <= 192 (what overflows them all the same is
// repeated with running lists, see tc_screen); the first pass costs 1 / s of the second
// and the candidates are re-bounded by the merge, so there is nothing to gain
// beyond 8; below 16 k maxima the threshold drops (3,000 x 60,000, d = 64, k =
// 30: 110 us with s = 6 and 4 k maxima against 108, the merge 13 us longer).
// One pass / s = 8, us: 4,096 x 2,000,000, d = 256: 3,184 / 2,926; 4,096 x
// 150,000: 487 / 300; 128 x 2,000,000: 233 / 194; 1 x 2,000,000: 170 / 184, but
// merge and re-rank of fewer candidates make it 430 / 406 a call; 8 x 200,000,
// euclidean: 127 / 37.  s = 1 / rule: 777 x 150,001, d = 100: 96 / 90.
SampleMap sample_of(int64_t n, int k) {
  auto with = [&](int s) {
    const int64_t span = n / SAMPLE_RUNS / s * s;
    return SampleMap{s, span, span / s / SAMPLE_PLACES};
  };
  auto maxima = [&](int s) { return maxima_per_query(with(s).tiles * BN, k); };
  if (maxima(1) < 4 * (int64_t)k || maxima(1) > INT32_MAX) return SampleMap{0, 1, 0};
  int s = std::max(1, std::min(8, 192 / k));
  while (s > 1 && maxima(s) < 16 * (int64_t)k) --s;
  return with(s);
}

// How a block of nq queries is cut into work, and the workspace it takes.
constexpr int ECAP = 768;                    // slots of a list of appended references
struct TcPlan {
  SampleMap sample;
  bool pair = false;
  int64_t units = 1;                         // CTAs, or CTA pairs, at one time
  int64_t groups = 0, ntiles = 0, per = 1, grid = 1, nslots = 0, maxima = 0;
  int gm() const { return pair ? Cfg<true>::GM : Cfg<false>::GM; }
};
TcPlan tc_plan(const sdg_dense* D, int method, int k, int64_t nq, bool allow_pairs) {
  TcPlan z;
  z.sample = sample_of(D->n, k);
  // CTA pairs (clusters of two; the work unit is then a pair) where they pay or
  // are asked for and the device can hold such clusters.  A pair's SM receives
  // half the bytes of a reference chunk.  One CTA / pairs, us: 4,096 x 2,000,000,
  // d = 256: 2,557 / 2,280; 1,024 x 800,000, d = 200: 286 / 274; 4,096 x
  // 2,000,000, d = 128: 1,651 / 1,677; d = 64: 1,440 / 1,488; an odd number of
  // 128-query groups pads one (257 x 1,000,000, d = 256: 161 / 182).  Blocks of too
  // few references for a sample run single CTAs.
  if (z.sample.s > 0 && nq > BM && (allow_pairs || (D->dpad > 2 * BK && (nq + BM - 1) / BM % 2 == 0))) {
    auto kp = method == COSINE ? k_dense_tc<1, true, 2> : k_dense_tc<1, true, 3>;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(2, 1, 1); cfg.blockDim = dim3(THREADS, 1, 1); cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&clusters, kp, &cfg) == cudaSuccess && clusters > 0) {
      z.pair = true;
      z.units = clusters;
    }
    cudaGetLastError();
  }
  if (!z.pair) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, D->device);
    z.units = std::max(sms, 1);
  }
  // (query group, reference tile) items in equal contiguous spans, one per unit
  z.groups = (nq + z.gm() - 1) / z.gm();
  z.ntiles = (D->n + BN - 1) / BN;
  const int64_t items = z.groups * z.ntiles;
  z.grid = std::min<int64_t>(z.units, items);
  z.per = (items + z.grid - 1) / z.grid;
  z.grid = (items + z.per - 1) / z.per;
  // list slots per query: two halves per unit whose span meets its group
  int64_t most = 1;
  for (int64_t g = 0; g < z.groups; ++g)
    most = std::max<int64_t>(most, last_cta(g, z.ntiles, z.per) - first_cta(g, z.ntiles, z.per) + 1);
  z.nslots = 2 * most;
  z.maxima = z.sample.s > 0 ? maxima_per_query(z.sample.tiles * BN, k) : 0;
  return z;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

int fail(int code, const char* msg) { set_error(msg); return code; }

}  // namespace

bool tc_screen_supported(const sdg_dense* R, int method, int k) {
  return (method == COSINE || method == EUCLIDEAN) && k >= 1 && k <= KT && R->dpad <= MAX_DCH * BK &&
         R->n < (int64_t)1 << 30 && encode_fn() != nullptr;
}

int64_t tc_screen_chunk(const sdg_dense* D, int k, int64_t nq) {
  const SampleMap z = sample_of(D->n, k);
  const int64_t per_query = 4 * std::max<int64_t>(1, z.s > 0 ? maxima_per_query(z.tiles * BN, k) : 0);
  const int64_t most = std::max<int64_t>(1, ((int64_t)4 << 30) / per_query / (2 * BM)) * (2 * BM);
  return std::min<int64_t>(nq, std::min<int64_t>(65536, most));
}

int64_t tc_screen_bytes(const sdg_dense* D, int method, int k, int64_t nq, int cap) {
  const TcPlan z = tc_plan(D, method, k, nq, false);
  const int64_t weights = 4 * BN * (z.ntiles + z.sample.tiles);
  return weights + nq * (4 * (z.maxima + z.nslots * (k + 1 + 2 * ECAP) + cap) + 4);
}

int tc_screen(sdg_ctx* ctx, const sdg_dense* Q, const sdg_dense* D, bool self, int method, int k, int64_t q0,
              int64_t nq, int32_t* cand, int32_t* count, int32_t* over, int cap, cudaStream_t s, bool allow_pairs,
              int* status) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return fail(SDG_E_CUDA, "cuTensorMapEncodeTiled is unavailable");
  if (Q->dpad != D->dpad || Q->n >= (int64_t)1 << 30) return fail(SDG_E_ARG, "query and reference shapes differ");
  const int64_t n = D->n;
  const int dch = D->dpad / BK;
  // one map per operand: 64-row x 128-column (query) / 256-column (reference)
  // boxes of the K-major BF16 copy (rows padded to dpad with zeros; columns
  // beyond the matrix read as zero)
  auto base_of = [&](const sdg_dense* M) { return (void*)((method == COSINE) ? M->ubp : M->xbp); };
  auto encode = [&](const sdg_dense* M, int box_cols, CUtensorMap* map) {
    const cuuint64_t gdim[2] = {(cuuint64_t)M->dpad, (cuuint64_t)M->n};
    const cuuint64_t gstride[1] = {(cuuint64_t)M->dpad * 2};
    const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_cols};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base_of(M), gdim, gstride, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  // a box: one of the s references of SAMPLE_PLACES places of `runs` runs
  auto encode_sample = [&](const SampleMap& z, int runs, CUtensorMap* map) {
    const cuuint64_t ld = (cuuint64_t)D->dpad * 2;
    const cuuint64_t gdim[4] = {(cuuint64_t)D->dpad, (cuuint64_t)z.s, (cuuint64_t)(z.span / z.s),
                                (cuuint64_t)SAMPLE_RUNS};
    const cuuint64_t gstride[3] = {ld, ld * z.s, ld * z.span};
    const cuuint32_t box[4] = {(cuuint32_t)BK, 1, (cuuint32_t)SAMPLE_PLACES, (cuuint32_t)runs};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, base_of(D), gdim, gstride, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  // the list length: the smallest of 16 / 24 / 32 / 48 / 64 that holds k
  auto pick_kernel = [&](bool pair) {
    if (pair)
      return (k <= 16) ? k_dense_tc<16, true, 0> : (k <= 24) ? k_dense_tc<24, true, 0>
           : (k <= 32) ? k_dense_tc<32, true, 0> : (k <= 48) ? k_dense_tc<48, true, 0> : k_dense_tc<64, true, 0>;
    return (k <= 16) ? k_dense_tc<16, false, 0> : (k <= 24) ? k_dense_tc<24, false, 0>
         : (k <= 32) ? k_dense_tc<32, false, 0> : (k <= 48) ? k_dense_tc<48, false, 0> : k_dense_tc<64, false, 0>;
  };
  const TcPlan plan = tc_plan(D, method, k, nq, allow_pairs);
  const SampleMap sample = plan.sample;
  // thresholds from a sample (MODE 1), then the references that pass (MODE 2,
  // 3); or one pass with running lists (MODE 0)
  const bool first = sample.s > 0;
  const bool pair = plan.pair;
  const int GM = plan.gm();
  CUtensorMap qmap, rmap;
  if (!encode(Q, BM, &qmap) || !encode(D, pair ? Cfg<true>::BNL : Cfg<false>::BNL, &rmap))
    return fail(SDG_E_CUDA, "cuTensorMapEncodeTiled failed");

  const int64_t G = plan.groups, ntiles = plan.ntiles, per = plan.per, grid = plan.grid, nslots = plan.nslots;
  const int64_t units = plan.units;
  const int ecap = ECAP;
  const float rel = 0.0040f + (float)D->d * 2.384185791015625e-7f;
  const float omc = 1.f - (rel + 9.5367431640625e-7f);

  int* any = status + 1;                               // a list overflowed: the block repeats
  const int64_t ntiles1 = sample.tiles, n1 = ntiles1 * BN;
  const int gran = (int)granularity(n1, k);
  const int64_t m = plan.maxima;
  const float opc = 1.f + rel + 1.9073486328125e-6f;     // 2^-19

  float *w = nullptr, *wp = nullptr, *maxima = nullptr, *lists = nullptr, *es = nullptr, *cand_s = nullptr;
  int32_t *ecount = nullptr, *eidx = nullptr;
  unsigned* tshared = nullptr;
  cudaError_t e = cudaSuccess;
  auto chk = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
  const int64_t nw = ntiles * BN;
  chk(cudaMallocAsync(&w, sizeof(float) * (size_t)nw, s));
  if (first) {
    chk(cudaMallocAsync(&wp, sizeof(float) * (size_t)n1, s));
    chk(cudaMallocAsync(&maxima, sizeof(float) * (size_t)(nq * m), s));
    if (e == cudaSuccess) chk(cudaMemsetAsync(any, 0, sizeof(int), s));
  }
  chk(cudaMallocAsync(&lists, sizeof(float) * (size_t)(nq * nslots * k), s));
  chk(cudaMallocAsync(&ecount, sizeof(int32_t) * (size_t)(nq * nslots), s));
  chk(cudaMallocAsync(&eidx, sizeof(int32_t) * (size_t)(nq * nslots * ecap), s));
  chk(cudaMallocAsync(&es, sizeof(float) * (size_t)(nq * nslots * ecap), s));
  chk(cudaMallocAsync(&cand_s, sizeof(float) * (size_t)(nq * cap), s));
  chk(cudaMallocAsync(&tshared, sizeof(unsigned) * (size_t)nq, s));
  if (e == cudaSuccess) {
    // every query's shared key starts at fkey(-inf) or at its threshold
    if (!first) k_tc_key_init<<<(unsigned)((nq + 255) / 256), 256, 0, s>>>(nq, tshared);
    chk(cudaMemsetAsync(ecount, 0, sizeof(int32_t) * (size_t)(nq * nslots), s));
    k_tc_weights<<<(unsigned)((nw + 255) / 256), 256, 0, s>>>(method, n, nw, omc, D->norm2, D->empty, w, sample, n1, opc,
                                                             wp);
    TcArgs P;
    P.method = method; P.k = k; P.dch = dch; P.ecap = ecap;
    P.self = self ? 1 : 0;
    P.d = D->d; P.n = n; P.q0 = q0; P.nq = nq;
    P.ntiles = ntiles; P.tiles_per_cta = per; P.nslots = nslots;
    P.a = (method == COSINE) ? 1.f : 2.f; P.one_minus_c = omc;
    P.w = w; P.norm2 = D->norm2; P.qnorm2 = Q->norm2; P.qempty = Q->empty;
    P.tshared = tshared;
    P.lists = lists; P.ecount = ecount; P.eidx = eidx; P.es = es;
    P.gate = nullptr; P.maxima = maxima; P.gran = gran; P.sample = sample; P.use_w = D->n_empty > 0 ? 1 : 0;
    P.status = status;
    P.stall = tc_take_stall() ? 1 : 0;
    auto launch = [&](auto kern, int64_t blocks, const CUtensorMap& refs, const TcArgs& A) {
      chk(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES));
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = pair ? 2 : 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3((unsigned)(pair ? 2 * blocks : blocks), 1, 1); cfg.blockDim = dim3(THREADS, 1, 1);
      cfg.dynamicSmemBytes = SMEM_BYTES; cfg.stream = s;
      cfg.attrs = attr; cfg.numAttrs = pair ? 1 : 0;
      if (e == cudaSuccess) chk(cudaLaunchKernelEx(&cfg, kern, qmap, refs, A));
    };
    sdg_time_begin(ctx);
    if (first) {
      CUtensorMap map1;
      if (!encode_sample(sample, pair ? SAMPLE_RUNS / 2 : SAMPLE_RUNS, &map1)) chk(cudaErrorInvalidValue);
      const int64_t items1 = G * ntiles1;
      TcArgs P1 = P;
      P1.w = wp; P1.n = n1; P1.ntiles = ntiles1;
      P1.tiles_per_cta = (items1 + std::min(units, items1) - 1) / std::min(units, items1);
      launch(pair ? k_dense_tc<1, true, 1> : k_dense_tc<1, false, 1>,
             (items1 + P1.tiles_per_cta - 1) / P1.tiles_per_cta, map1, P1);
      P.stall = 0;                                     // one launch is stalled at a time
      if (e == cudaSuccess)
        k_tc_threshold<<<(unsigned)((nq + 7) / 8), 256, 0, s>>>(method, q0, nq, (int)m, k, rel, opc, Q->norm2,
                                                                Q->empty, maxima, tshared);
    }
    launch(!first            ? pick_kernel(pair)
           : method == COSINE ? (pair ? k_dense_tc<1, true, 2> : k_dense_tc<1, false, 2>)
                              : (pair ? k_dense_tc<1, true, 3> : k_dense_tc<1, false, 3>),
           grid, rmap, P);
    sdg_time_end(ctx);
    chk(cudaGetLastError());
    ctx_stats_add(ctx, 3, first ? 7 : 4);   // weights, maxima and threshold (or key init), screen, merge, their repeat
    MergeArgs M;
    M.q0 = q0; M.nq = nq; M.gm = GM; M.ntiles = ntiles; M.per = per; M.nslots = nslots;
    M.K = k; M.ecap = ecap; M.method = method; M.d = D->d;
    M.qempty = Q->empty; M.tshared = tshared; M.lists = first ? nullptr : lists; M.ecount = ecount; M.eidx = eidx; M.es = es;
    M.norm2 = D->norm2; M.qnorm2 = Q->norm2;
    M.re = (method == COSINE) ? D->ue : D->xe; M.rn = (method == COSINE) ? D->un : D->xn;
    M.qe = (method == COSINE) ? Q->ue : Q->xe; M.qn = (method == COSINE) ? Q->un : Q->xn;
    M.cap = cap; M.cand = cand; M.cand_s = cand_s; M.count = count; M.over = over;
    M.smem_query = merge_prefix_bytes(nslots) + (size_t)std::max<int64_t>(nslots * k, cap) * 4;
    M.smem_query = (M.smem_query + 15) / 16 * 16;
    const bool narrow = nq >= MERGE_WIDE_MAX && M.smem_query * 8 <= 220 * 1024;
    const bool widest = nq <= MERGE_WIDEST_MAX;
    auto mk = narrow ? k_tc_merge<1> : widest ? k_tc_merge<32> : k_tc_merge<8>;
    const size_t msm = M.smem_query * (narrow ? 8 : 1);
    if (msm > 48 * 1024) chk(cudaFuncSetAttribute(mk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)msm));
    auto merge = [&](const MergeArgs& A) {
      if (e == cudaSuccess) mk<<<(unsigned)(narrow ? (nq + 7) / 8 : nq), widest ? 1024 : 256, msm, s>>>(A);
      chk(cudaGetLastError());
    };
    M.any_over = any; M.gate = nullptr;
    merge(M);
    // Where a list overflows all the same (thousands of references of one span
    // within the bound of a query's threshold), the block runs once more with
    // running lists, which tighten as they go, from the same thresholds; otherwise
    // both launches return at once.
    if (first) {
      P.gate = any;
      launch(pick_kernel(pair), grid, rmap, P);
      M.lists = lists; M.any_over = nullptr; M.gate = any;
      merge(M);
    }
  }
  // stream-ordered frees: the caller reads *status with its own results
  for (void* p : {(void*)w, (void*)wp, (void*)maxima, (void*)lists, (void*)ecount, (void*)eidx, (void*)es, (void*)cand_s, (void*)tshared})
    if (p) cudaFreeAsync(p, s);
  if (e != cudaSuccess) {
    set_error(cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? SDG_E_NOMEM : SDG_E_CUDA;
  }
  return SDG_OK;
}

}  // namespace sdg
