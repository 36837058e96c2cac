// sdg_screen.cu -- the screened candidate engine (see sdg_screen.h).
//
// GB300 executes FP64 at roughly 1/70 of its FP32 rate, so evaluating every
// column pair exactly in FP64 (as the reference does on the CPU) is bound by
// the FP64 pipe.  This engine evaluates every pair in FP32 instead, with a
// rigorous per-pair error bound E, and re-ranks in exact FP64 only the pairs
// whose optimistic bound can still reach the k-th best pessimistic bound:
//
//   keep (q, c)  iff  key(q, c) + E(q, c) >= T_q - margin,
//   T_q = k-th largest of key(q, c') - E(q, c') over eligible c'.
//
// Every member of the exact top-k (ties included) satisfies the test, so the
// exact re-rank over the kept pairs returns exactly the reference's result.
// A query whose kept set exceeds the candidate capacity is finished by the
// exact slab engine instead.
//
// Screen kernel (k_screen_rows): the reference's screen values in row order.
// A warp owns one (query column, part of the reference columns) item and
// accumulates the part's screen values in shared memory, one float per
// column: for every row the query stores it reads that row's entries of the
// part, coalesced (a row never holds a column twice, so the lanes' columns
// differ), and adds each entry's term to its column.  The work is the matched
// (query entry, reference entry) pairs themselves, whatever the density.
#include <cub/device/device_scan.cuh>
#include <cuda_fp16.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>
#include <vector>

#include "sdg_kernels.h"
#include "sdg_kth.cuh"
#include "sdg_screen.h"
#include "sdg_tc_bounds.cuh"

namespace sdg {
namespace {

constexpr int SELECT_WARPS = 8;
constexpr int kScreenMaxK = 1024;    // largest k of the screens
// shared memory of the screen kernel's accumulators per SM (of 227 KB)
constexpr size_t kScreenAccBytes = 208 * 1024;
constexpr int kScreenMaxWarps = 32;
// entries of the parts that run at one time: 64 MB of the 129 MB L2 (manhattan,
// 20,000 log-count columns, 248 MB of entries, 1,000 queries: 6.2 ms; all at
// once 7.0; 100,000 columns, 2,000 queries: 60 and 91)
constexpr int64_t kScreenGroupBytes = (int64_t)64 << 20;
constexpr int32_t kScreenMaxRows = 53756;   // more rows: the exact engine
constexpr float U32 = 5.9604644775390625e-8f;   // 2^-24

inline unsigned blocks_for(int64_t n, int threads) {
  return (unsigned)((n + threads - 1) / threads);
}

// the failing call of the last screen error on this thread (for the message)
thread_local const char* g_screen_site = "";
#define SK_STR2(l) #l
#define SK_STR(l) SK_STR2(l)
#define SK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) { g_screen_site = #x " at line " SK_STR(__LINE__); return (int)e_; } } while (0)
// a call of a function that records its own failing site
#define SKN(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return (int)e_; } while (0)

// ---------------------------------------------------------------------------
// validation used at upload
// ---------------------------------------------------------------------------
// A warp per column, coalesced: each entry against the one before it.  Bound by
// the launch for small matrices, by the 4 bytes an entry for large ones (a
// thread per column took 811 us for 110 columns of 2,180 entries, 104 us for
// 1,500 + 12,001 of 120).
__global__ void k_check_rows(DevCsc M, int* err) {
  const int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (j >= M.ncol) return;
  const int64_t a0 = M.p[j], a1 = M.p[j + 1];
  bool bad = false;
  for (int64_t a = a0 + lane; a < a1; a += 32) {
    const int32_t r = __ldg(M.i + a);
    const int32_t prev = a > a0 ? __ldg(M.i + a - 1) : -1;
    bad = bad || r <= prev || r < 0 || r >= M.nrow;
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(err, 1);
}

// ---------------------------------------------------------------------------
// per-matrix screening data
// ---------------------------------------------------------------------------
// fval: the value the screen multiplies (unit value for cosine, raw value for
// euclidean / manhattan, 1 for binary); cnorm: sum of squares (euclidean) or
// of magnitudes (manhattan), accumulated in FP64 then rounded; nnz per column.
// One warp per column: the FP32 screen values (coalesced) and the column's
// norm term (a warp sum in FP64, rounded to FP32: the screen bounds allow for
// its rounding whatever the summation order).
// js: fval = the value, fxl = its x log x (from the FP64 values the exact path
// uses), cnorm = the column's sum of |x log x| + x rounded up, and *range_err
// set when a nonzero value lies outside [2^-100, 2^100]; pearson /
// covariance: fval = the value, *range_err when a nonzero |value| lies outside
// [2^-50, 2^50].
__global__ void k_screen_prep(DevCsc M, int method, const double* uval, const double* xl, float* fval,
                              float* fxl, float* cnorm, int32_t* nnz, int* range_err) {
  const int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (j >= M.ncol) return;
  double acc = 0.0;
  bool bad = false;
  const int64_t a0 = M.p[j], a1 = M.p[j + 1];
  for (int64_t a = a0 + lane; a < a1; a += 32) {
    const double v = M.x[a];
    float f;
    if (method == COSINE) f = (float)uval[a];
    else if (method == BINARY) f = 1.0f;
    else f = (float)v;
    fval[a] = f;
    if (method == EUCLIDEAN) acc += v * v;
    else if (method == MANHATTAN) acc += fabs(v);
    else if (method == JS) {
      fxl[a] = (float)xl[a];
      acc += fabs(xl[a]) + v;
      bad = bad || (v != 0.0 && !(v >= 0x1p-100 && v <= 0x1p100));
    } else if (method == PEARSON || method == COVARIANCE) {
      // FP32 products of values within 2^+-50 stay normal and their sums finite
      bad = bad || (v != 0.0 && !(fabs(v) >= 0x1p-50 && fabs(v) <= 0x1p50));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(range_err, 1);
  if (lane == 0) {
    cnorm[j] = (method == JS) ? __double2float_ru(acc * (1.0 + 1e-12)) : (float)acc;
    nnz[j] = (int32_t)(a1 - a0);
  }
}

// ---------------------------------------------------------------------------
// the reference's entries in row order
// ---------------------------------------------------------------------------
// Cell (r, s) holds row r's entries of sub-range s of the columns (2^lg
// columns each); cells are stored row-major, so a row's entries of several
// consecutive sub-ranges are one contiguous run.
__global__ void k_rows_count(DevCsc M, int lg, int32_t nsub, uint32_t* cnt) {
  const int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (j >= M.ncol) return;
  const int64_t sub = j >> lg;
  for (int64_t a = M.p[j] + lane; a < M.p[j + 1]; a += 32) atomicAdd(cnt + (int64_t)M.i[a] * nsub + sub, 1u);
}

// pos: the cells' first free slots, advanced to the cells' ends.  The order of
// a cell's entries is free: they belong to different columns.
__global__ void k_rows_fill(DevCsc M, int lg, int32_t nsub, const float* fval, const float* fxl, uint32_t* pos,
                            int2* ent, float* exl) {
  const int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (j >= M.ncol) return;
  const int64_t sub = j >> lg;
  for (int64_t a = M.p[j] + lane; a < M.p[j + 1]; a += 32) {
    const uint32_t at = atomicAdd(pos + (int64_t)M.i[a] * nsub + sub, 1u);
    ent[at] = make_int2((int)j, __float_as_int(fval[a]));
    if (fxl) exl[at] = fxl[a];
  }
}

// Reorders the entries of every cell so that 32 consecutive ones fall on
// different shared-memory banks (bank = column mod 32) as far as the cell
// allows: by (how many earlier columns of the cell share the bank, bank).  The
// screen's accumulator loads and stores then take 1 to 2 wavefronts instead
// of the 3 to 4 of 32 random columns.  One warp per cell, lane = bank; the
// cell's values go through a shared-memory row of `cols` floats, its columns
// through a bitmap of one word per 32 columns.
constexpr int ROWS_WARPS = 4;
// mean entries of a cell from which it pays: at 26 the screen goes from 10.7 to
// 9.4 ms; at 10 it stays at 0.09 ms and the ordering itself takes 0.11
constexpr double ROWS_BANKS_MIN = 16.0;

__global__ void __launch_bounds__(ROWS_WARPS * 32) k_rows_banks(int64_t cells, int lg, int32_t nsub,
                                                                const uint32_t* rows, int2* ent, float* exl) {
  extern __shared__ __align__(16) uint32_t bsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cols = 1 << lg, words = cols >> 5;
  uint32_t* bits = bsm + (size_t)warp * (words + (exl ? 2 : 1) * cols);
  float* val = reinterpret_cast<float*>(bits + words);
  float* xlv = val + cols;                           // with exl only
  for (int w = lane; w < words; w += 32) bits[w] = 0u;
  __syncwarp();
  for (int64_t cell = (int64_t)blockIdx.x * ROWS_WARPS + warp; cell < cells; cell += (int64_t)gridDim.x * ROWS_WARPS) {
    const uint32_t a = rows[cell], b = rows[cell + 1];
    if (b - a < 2) continue;
    const int32_t base = (int32_t)(cell % nsub) << lg;
    for (uint32_t p = a + lane; p < b; p += 32) {
      const int2 e = ent[p];
      const int c = e.x - base;
      atomicOr(&bits[c >> 5], 1u << (c & 31));
      val[c] = __int_as_float(e.y);
      if (exl) xlv[c] = exl[p];
    }
    __syncwarp();
    // a pass per occurrence: the lanes still holding a column emit their next one
    uint32_t at = a;
    int w = 0;
    for (;;) {
      while (w < words && !((bits[w] >> lane) & 1u)) ++w;
      const unsigned m = __ballot_sync(0xffffffffu, w < words);
      if (!m) break;
      if (w < words) {
        const uint32_t p = at + __popc(m & ((1u << lane) - 1u));
        const int c = (w << 5) + lane;
        ent[p] = make_int2(base + c, __float_as_int(val[c]));
        if (exl) exl[p] = xlv[c];
        ++w;
      }
      at += __popc(m);
    }
    for (int i = lane; i < words; i += 32) bits[i] = 0u;
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// the screen kernel
// ---------------------------------------------------------------------------
struct ScreenArgs {
  // reference, in row order (see k_rows_fill)
  const uint32_t* rows;       // [nrow * nsub + 1] cell offsets
  const int2* ent;            // (column, value bits)
  const float* exl;           // js: x log x of each entry
  int32_t nsub, part_subs;    // sub-ranges; sub-ranges per part
  int lg;                     // log2 columns per sub-range
  int64_t nr;
  // queries (columns of the query matrix)
  const int64_t* qp; const int32_t* qi; const float* qv;
  const float* qxl;           // js: x log x of each query value
  int64_t q_begin, nq;        // local query 0 = query column q_begin
  const int2* order;          // (local query, stretch), longest first
  const int32_t* units;       // their number
  int nparts, group;          // parts; parts of a group
  int64_t ldS;
  float* S;                   // S[qlocal * ldS + column]
  unsigned long long* work;   // work counter
};

// The screen's units of work: a query column, or a stretch of SCREEN_SEG of its
// stored entries where it has more (a lane-parallel walk of one long column
// would outlast the rest of the launch).  order: (local query, stretch) pairs
// by descending length (in 1,024 steps of a full stretch), *total: their
// number.  One block.
constexpr int SCREEN_SEG = 1024;   // whole queries: 6.6 ms where stretches take 6.2, and 4.5 ms where they take 1.8 (5,000 columns)

__global__ void __launch_bounds__(1024) k_screen_order(const int32_t* qnnz, int64_t q_begin, int64_t nq, int2* order,
                                                       int32_t* total) {
  __shared__ int32_t bin[1025], wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bin[tid] = 0;
  __syncthreads();
  // a query's stretches: nfull whole ones (bin 0) and one of the rest, or an empty query's only one
  auto split = [&](int64_t i, int& nfull, int& rest_bin) {
    const int32_t len = qnnz[q_begin + i];
    nfull = len / SCREEN_SEG;
    const int rest = len - nfull * SCREEN_SEG;
    rest_bin = (rest > 0 || nfull == 0) ? 1023 - rest * 1023 / SCREEN_SEG : -1;
  };
  for (int64_t i = tid; i < nq; i += 1024) {
    int nfull, rb;
    split(i, nfull, rb);
    if (nfull) atomicAdd(&bin[0], nfull);
    if (rb >= 0) atomicAdd(&bin[rb], 1);
  }
  __syncthreads();
  const int32_t own = bin[tid];
  int32_t x = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int32_t w = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  bin[tid] = x - own + (warp ? wsum[warp - 1] : 0);
  if (tid == 0) *total = wsum[31];
  __syncthreads();
  for (int64_t i = tid; i < nq; i += 1024) {
    int nfull, rb;
    split(i, nfull, rb);
    if (nfull) {
      const int at = atomicAdd(&bin[0], nfull);
      for (int t = 0; t < nfull; ++t) order[at + t] = make_int2((int)i, t);
    }
    if (rb >= 0) order[atomicAdd(&bin[rb], 1)] = make_int2((int)i, nfull);
  }
}

// The slab rows that several stretches add to start at zero.
__global__ void k_screen_zero(const int32_t* qnnz, int64_t q_begin, int64_t nr, int64_t ldS, float* S) {
  if (qnnz[q_begin + blockIdx.x] <= SCREEN_SEG) return;
  float* row = S + (int64_t)blockIdx.x * ldS;
  for (int64_t c = threadIdx.x; c < nr; c += blockDim.x) row[c] = 0.f;
}

// One matched row's term added to the running value.  js: the shared row's g =
// S log S - P log P - Q log Q (S = P + Q) in FP32, every operation rounded on
// its own (no contraction), summed in order; the logarithm is the __logf
// intrinsic, taken to err by at most 2^-20.41 absolute on [0.5, 2] and 6 ulp
// elsewhere (twice its documented accuracy; tests/test_gpu_logf_bound.py
// checks every FP32 input in [2^-100, 2^102)).  The error analysis of
// js_key_and_bound below follows these steps.
template <int KIND>   // 0: product, 1: manhattan, 2: js
__device__ __forceinline__ float screen_term(float acc, float v, float vx, float q, float qx) {
  if (KIND == 0) return fmaf(v, q, acc);
  if (KIND == 1) return acc + ((fabsf(v) + fabsf(q)) - fabsf(v - q));
  const float S = __fadd_rn(v, q);
  return __fadd_rn(acc, __fsub_rn(__fsub_rn(__fmul_rn(S, __logf(S)), vx), qx));
}

// Items (stretch of a query, part) are handed to the warps by an atomic
// counter, group of parts by group (a group's entries stay in the L2), within
// it the longest stretch first.  A warp takes the query's rows 32 at a time
// (lane l holds row l's run of the part) and the runs four at a time, the next
// four runs' first 32 entries loaded before the current four are added;
// consecutive runs may hit the same column from different lanes, hence the
// __syncwarp between them.  A query of one stretch stores its screen values,
// the stretches of a longer one add theirs (the bounds hold for any order of
// the sum).
//
// What bounds it: shared memory (a load and a store of 32 columns per step, 2
// wavefronts each in bank order) with all warps busy, the runs' latency with
// few.  The kernel it replaced walked reference columns, one per lane, against
// a row-indexed table of 16 queries, with 16 predicated steps per stored entry
// whatever the match probability.  Before and after, ms a launch: manhattan, log
// counts, 1,000 queries x 20,000: 10.2 and 6.2, 2,000 x 100,000: 165 and 60, 256
// x 20,000: 4.7 and 2.1; js, 1,000 x 20,000: 51 and 10.6; manhattan, 1 % uniform
// over 12,000 rows, 1,500 x 12,001: 0.80 and 0.09.
template <int KIND>
__global__ void __launch_bounds__(kScreenMaxWarps * 32, 1) k_screen_rows(ScreenArgs A) {
  extern __shared__ __align__(16) float sacc[];
  const int lane = threadIdx.x & 31;
  const int64_t part_cols = (int64_t)A.part_subs << A.lg;
  float* acc = sacc + (int64_t)(threadIdx.x >> 5) * part_cols;
  const unsigned long long units = (unsigned long long)*A.units;
  const unsigned long long items = units * (unsigned long long)A.nparts;
  const unsigned long long span = units * (unsigned long long)A.group;
  for (;;) {
    unsigned long long item = 0;
    if (lane == 0) item = atomicAdd(A.work, 1ull);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= items) break;
    const int64_t first = (int64_t)(item / span) * A.group, in_group = (int64_t)(item % span);
    const int64_t gp = min((int64_t)A.group, A.nparts - first);
    const int64_t part = first + in_group % gp;
    const int2 unit = A.order[in_group / gp];
    const int64_t ql = unit.x;
    const int32_t s0 = (int32_t)part * A.part_subs, s1 = min(s0 + A.part_subs, A.nsub);
    const int32_t c0 = (int32_t)(part * part_cols);
    const int32_t nc = (int32_t)min(part_cols, A.nr - c0);
    for (int32_t i = lane; i < nc; i += 32) acc[i] = 0.f;
    __syncwarp();
    const int64_t q0 = A.qp[A.q_begin + ql], q1 = A.qp[A.q_begin + ql + 1];
    const int64_t e0 = q0 + (int64_t)unit.y * SCREEN_SEG, e1 = min(e0 + SCREEN_SEG, q1);
    // lane l: the run [a, b) of query entry l of the chunk, its value
    uint32_t a = 0, b = 0;
    float v = 0.f, vx = 0.f;
    auto chunk = [&](int64_t e) {
      a = b = 0;
      if (e + lane < e1) {
        const int64_t cell = (int64_t)__ldg(A.qi + e + lane) * A.nsub;
        v = __ldg(A.qv + e + lane);
        if (KIND == 2) vx = __ldg(A.qxl + e + lane);
        a = __ldg(A.rows + cell + s0);
        b = __ldg(A.rows + cell + s1);
      }
    };
    chunk(e0);
    for (int64_t e = e0; e < e1; e += 32) {
      const uint32_t ca = a, cb = b;
      const float cv = v, cvx = vx;
      chunk(e + 32);                                 // the next 32 runs' bounds
      const int n = (int)(e1 - e < 32 ? e1 - e : 32);
      int2 nx[4];
      float nl[4];
      auto fetch = [&](int j0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t p = __shfl_sync(0xffffffffu, ca, (j0 + u) & 31) + lane;
          const uint32_t pe = __shfl_sync(0xffffffffu, cb, (j0 + u) & 31);
          nx[u] = make_int2(-1, 0);
          nl[u] = 0.f;
          if (j0 + u < n && p < pe) {
            nx[u] = __ldg(A.ent + p);
            if (KIND == 2) nl[u] = __ldg(A.exl + p);
          }
        }
      };
      fetch(0);
      for (int j0 = 0; j0 < n; j0 += 4) {
        int2 cur[4];
        float cl[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) { cur[u] = nx[u]; cl[u] = nl[u]; }
        fetch(j0 + 4);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = (j0 + u) & 31;               // past n: an empty run (a == b)
          const float q = __shfl_sync(0xffffffffu, cv, j);
          const float qx = KIND == 2 ? __shfl_sync(0xffffffffu, cvx, j) : 0.f;
          const uint32_t pa = __shfl_sync(0xffffffffu, ca, j), pe = __shfl_sync(0xffffffffu, cb, j);
          if (cur[u].x >= 0) {
            float* x = acc + (cur[u].x - c0);
            *x = screen_term<KIND>(*x, __int_as_float(cur[u].y), cl[u], q, qx);
          }
          if (j0 + u < n) {
            for (uint32_t p = pa + 32 + lane; p < pe; p += 128) {
              int2 t[4];
              float tl[4];
#pragma unroll
              for (int w = 0; w < 4; ++w) {
                t[w] = make_int2(-1, 0);
                tl[w] = 0.f;
                if (p + 32 * w < pe) {
                  t[w] = __ldg(A.ent + p + 32 * w);
                  if (KIND == 2) tl[w] = __ldg(A.exl + p + 32 * w);
                }
              }
#pragma unroll
              for (int w = 0; w < 4; ++w) {
                if (t[w].x >= 0) {
                  float* x = acc + (t[w].x - c0);
                  *x = screen_term<KIND>(*x, __int_as_float(t[w].y), tl[w], q, qx);
                }
              }
            }
          }
          __syncwarp();
        }
      }
    }
    float* out = A.S + ql * A.ldS + c0;
    if (q1 - q0 > SCREEN_SEG) {
      for (int32_t i = lane; i < nc; i += 32) atomicAdd(out + i, acc[i]);
    } else {
      for (int32_t i = lane; i < nc; i += 32) out[i] = acc[i];
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// screen select: per query, the k-th pessimistic bound and the kept pairs
// ---------------------------------------------------------------------------
struct SelectScreenArgs {
  int method, k;
  const float* S;                            // [qlocal * ldS + column], ldS a multiple of 4
  int64_t nr, ldS;
  const int32_t* rnnz; const float* rnorm;
  const int32_t* qnnz; const float* qnorm;   // indexed by query column
  const double* rsum;                        // js: reference column sums
  const double* qsum;                        // js: query column sums (indexed by query column)
  // pearson / covariance: the columns' FP64 sums and sums of squares, nrow
  const double *rs, *rss, *qs, *qss;
  int32_t nrow;
  const uint8_t* ref_mask;                   // eligible reference columns
  const uint8_t* qry_blank;                  // query rows written all-NA
  const uint8_t* qry_force_exact;            // queries the screen cannot bound
  int64_t q_begin, nq;                       // local queries of this chunk
  int selfmode, include_self;                // self search: query q == reference q
  int cap;
  int slices;                                // stretches of a row in the first pass
  int32_t* cand;                             // [qlocal * cap + t] reference column
  float* hi;                                 // the same places: the candidates' upper bounds (js, pearson, covariance)
  int32_t* count;                            // kept pairs per query (capped)
  int32_t* overflow;                         // 1 = finish with the exact engine
};

// Larger key = better.  E bounds |key_fp32 - key_exact| (see the file header
// and DESIGN notes of each method).
__device__ __forceinline__ void key_and_bound(int method, float s, int32_t nq_, float Nq, int32_t nc_,
                                              float Nc, float& key, float& err) {
  const float n = (float)min(nq_, nc_);
  if (method == COSINE) {
    key = s;
    err = (n + 40.f) * U32 * 1.01f + 1e-12f;
  } else if (method == EUCLIDEAN) {
    const float T = Nq + Nc;
    key = 2.f * s - T;
    err = ((n + 46.f) * U32 * 1.01f + 1e-12f) * T + 1e-30f;
  } else if (method == MANHATTAN) {
    const float T = Nq + Nc;
    key = s - T;
    err = ((n + 46.f) * U32 * 1.01f + 1e-12f) * T + 1e-30f;
  } else {                                   // BINARY: s is the exact count
    const float denom = (float)(nq_ + nc_) - s;
    key = (denom > 0.f) ? s / denom : 1.f;
    err = key * (4.f * U32) + 1e-30f;
  }
}

// js (fastJS2, src/sparseDist.cpp:1099-1108): the value is sqrt(0.5 t) with
// t = (S_P + S_Q) log 2 - G, G = sum over shared rows of g = S log S - P log P
// - Q log Q (every other row adds its value times log 2), so with the query
// fixed the order is that of key = G - S_P log 2 (larger = better).  Error of
// the FP32 G (values in [2^-100, 2^100], u = 2^-24): p, q, S rounded once
// (S~ = S (1 + t), |t| <= 2.0001 u); |__logf(S~) - ln S~| <= 12.06 u + 12 u
// |ln S~| (2^-20.41 absolute on [0.5, 2], 6 ulp <= 12 u relative elsewhere),
// so |L - ln S| <= 14.07 u + 12 u |ln S|; the product and the two differences
// each rounded once, x log x stored to FP32: |g~ - g| <= u (17.0001 |S log S|
// + 14.07 S + 3.0001 |P log P| + 2.0001 |Q log Q|) <= 31.1 u (|P log P| + |Q
// log Q| + S), using |S log S| <= |P log P| + |Q log Q| + S; summed over the
// shared rows <= 31.1 u (A_P + A_Q), A = a column's sum of |x log x| + x.
// The recursive FP32 sum of n <= min(nnz) terms adds <= n u / (1 - n u) times
// sum |g~| <= log 2 (C_P + C_Q) + 31.1 u (A_P + A_Q) (0 <= g <= S log 2, C =
// a column's sum).  With n u <= 1/16 (n is at most kScreenMaxRows)
// the two give E_G = u (33.5 (A_P + A_Q) + 0.75 n (C_P + C_Q)) 1.01; the key's
// own rounding (u |key|, the FP64 S_P log 2 rounded once) is added.
__device__ __forceinline__ void js_key_and_bound(float G, double SP, double SQ, float AP, float AQ,
                                                 int32_t n_, float& key, float& err) {
  const float n = (float)n_;
  key = (float)((double)G - SP * 0.69314718055994530942);
  const float C = (float)(SP + SQ);
  err = U32 * (33.5f * (AP + AQ) + 0.75f * n * C) * 1.01f + 2.f * U32 * fabsf(key) + 1e-30f;
}

// pearson / covariance (fastCorr2 / fastCov2 in the single-pass form of the
// exact path, pearson_finish / covariance_finish): the screen's s~ is the FP32
// FMA chain over the matched rows' FP32 values; with u = 2^-24 and n <= min(nnz)
// terms, |s~ - s| <= (n + 3) u (1 + n u 1.1) sum |ab| <= (n + 4) u 1.01 sqrt(SS_P
// SS_Q) (Cauchy-Schwarz over the full columns' sums of squares; the exact
// path's own FP64 sum is within n 2^-53 of s, inside the factor).  The key is
// the exact path's formula evaluated in FP64 on s~ with the same rounded
// operations, so the decisions that depend only on the moments (a zero or
// non-finite denominator, which makes the exact value 0) are the exact path's:
// cov = (s - S_P S_Q / N) / (N - 1), errs by E_s / (N - 1) plus 2^-50 of its
// terms; pearson c = cov / (sqrt(v_P) sqrt(v_Q)) by E_cov / den plus 2^-50 |c|,
// and both bounds are clamped to [-1, 1] as the exact value is.  A pearson
// denominator below 1e-200 could let cov / den overflow (exact value 0 then):
// the bounds are [-1, 1].  Larger key = better for both methods.
// a column's standard deviation, sqrt(v), with the exact path's rounded operations
__device__ __forceinline__ double moment_root(int32_t nrow, double S, double SS) {
  const double N = (double)nrow;
  const double norm = (nrow > 1) ? __dsub_rn(N, 1.0) : 1.0;
  return sqrt(__dsub_rn(SS, __dmul_rn(S, S) / N) / norm);
}
// root_q: the query's moment_root (pearson)
__device__ __forceinline__ void moment_key_and_bound(bool pearson, float s, int32_t n_, int32_t nrow, double SP,
                                                     double SSP, double SQ, double SSQ, double root_q, float& key,
                                                     float& err) {
  const double N = (double)nrow;
  const double norm = (nrow > 1) ? __dsub_rn(N, 1.0) : 1.0;
  const double sd = (double)s;
  const double Es = (((double)n_ + 4.0) * 5.9604644775390625e-8 * 1.01) * sqrt(SSP * SSQ) + 1e-300;
  const double m = __dmul_rn(SP, SQ) / N;
  const double cov = __dsub_rn(sd, m) / norm;
  const double Ecov = (Es + 0x1p-50 * (fabs(sd) + fabs(m))) / norm;
  double lo, hi;
  if (!pearson) {
    lo = cov - Ecov * 1.0001;
    hi = cov + Ecov * 1.0001;
  } else {
    const double den = __dmul_rn(moment_root(nrow, SP, SSP), root_q);
    if (!(den > 0.0) || !isfinite(den)) { key = 0.f; err = 0.f; return; }   // the exact value is 0
    if (den < 1e-200) { key = 0.f; err = 1.0001f; return; }
    const double c = cov / den;
    const double e = (Ecov / den + 0x1p-50 * fabs(c)) * 1.0001;
    lo = fmin(1.0, fmax(-1.0, c - e));
    hi = fmin(1.0, fmax(-1.0, c + e));
  }
  key = (float)(0.5 * (lo + hi));
  err = (float)(0.5 * (hi - lo)) + 2.f * U32 * (fabsf(key) + 1.f) + 1e-30f;
}

// The key intervals [lo, hi] of four consecutive references from their screen
// values; ok bit u: reference c + u is a candidate.  KIND 0: cosine, 1: euclidean /
// manhattan, 2: binary, 3: js, 4: pearson / covariance.  For KIND 0 and 1 the
// term count of the bound is the query's stored entries (min(nnz_q, nnz_c) is at
// most that), so it is one number per query; KIND 2 divides with __fdividef (2
// ulp: 4 u of the key, doubled here).  A key that is not finite has no lower
// bound and stays a candidate (its exact value decides).
template <int KIND>
struct ScreenBounds {
  const SelectScreenArgs& A;
  const int64_t q;
  const int32_t nq_;
  const float Nq, e, a;
  const double SQ, SSQ, root_q;              // KIND 4: the query's moments
  __device__ __forceinline__ ScreenBounds(const SelectScreenArgs& A_, int64_t q_)
      : A(A_), q(q_), nq_(A_.qnnz[q_]), Nq(A_.qnorm ? A_.qnorm[q_] : 0.f),
        e(((float)nq_ + (KIND == 0 ? 40.f : 46.f)) * U32 * 1.01f + 1e-12f), a(A_.method == EUCLIDEAN ? 2.f : 1.f),
        SQ(KIND == 4 ? A_.qs[q_] : 0.0), SSQ(KIND == 4 ? A_.qss[q_] : 0.0),
        root_q(KIND == 4 && A_.method == PEARSON ? moment_root(A_.nrow, SQ, SSQ) : 0.0) {}
  __device__ __forceinline__ unsigned operator()(int64_t c, int64_t end, const float4& sv, float (&lo)[4],
                                                 float (&hi)[4]) const {
    const float s[4] = {sv.x, sv.y, sv.z, sv.w};
    float4 nc4 = make_float4(0.f, 0.f, 0.f, 0.f);
    int4 nn4 = make_int4(0, 0, 0, 0);
    if (KIND == 1 || KIND == 3) nc4 = __ldg(reinterpret_cast<const float4*>(A.rnorm + c));
    if (KIND >= 2) nn4 = __ldg(reinterpret_cast<const int4*>(A.rnnz + c));
    const float Nc[4] = {nc4.x, nc4.y, nc4.z, nc4.w};
    const int32_t nn[4] = {nn4.x, nn4.y, nn4.z, nn4.w};
    unsigned ok = c + 3 < end ? 15u : (1u << (int)(end - c)) - 1u;
    if (A.ref_mask) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (((ok >> u) & 1u) && A.ref_mask[c + u]) ok &= ~(1u << u);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (KIND == 0) {
        lo[u] = s[u] - e;
        hi[u] = s[u] + e;
        if (!(fabsf(s[u]) <= FLT_MAX)) { lo[u] = -INFINITY; hi[u] = INFINITY; }
      } else {
        float key = 0.f, err = 0.f;
        if (KIND == 1) {
          const float T = Nq + Nc[u];
          key = fmaf(a, s[u], -T);
          err = e * T + 1e-30f;
        } else if (KIND == 2) {
          const float denom = (float)(nq_ + nn[u]) - s[u];
          key = (denom > 0.f) ? __fdividef(s[u], denom) : 1.f;
          err = key * (8.f * U32) + 1e-30f;
        } else if ((ok >> u) & 1u) {
          if (KIND == 3)
            js_key_and_bound(s[u], A.rsum[c + u], A.qsum[q], Nc[u], Nq, min(nq_, nn[u]), key, err);
          else
            moment_key_and_bound(A.method == PEARSON, s[u], min(nq_, nn[u]), A.nrow, A.rs[c + u], A.rss[c + u],
                                 SQ, SSQ, root_q, key, err);
        }
        lo[u] = key - err;
        hi[u] = key + err;
        if (!(fabsf(key) <= FLT_MAX) || !(err <= FLT_MAX)) { lo[u] = -INFINITY; hi[u] = INFINITY; }
      }
    }
    if (A.selfmode && q >= c && q < c + 4 && !(A.include_self && A.method == COVARIANCE)) {
      // A restored self value (R/sparseKNN.R:270-279) is the best value there is:
      // no upper bound.  Its lower bound stays the pair's own: an exact copy of
      // the query ties with it and comes first where its index is lower, so the
      // copy's interval has to reach the k-th best lower bound (with the lower
      // bound at +inf and k = 1 the query alone was kept).  A covariance self
      // pair keeps its computed value and is an ordinary pair.
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c + u == q) {
          hi[u] = INFINITY;
          if (!A.include_self) ok &= ~(1u << u);
        }
    }
    return ok;
  }
};

// One block per query, two passes over its screen values, four columns a load.
// First: every thread's largest pessimistic key in each of `slices` stretches of
// the row, at least four times k of them where the row is that long; their k-th
// largest T0 (found by one warp) is reached by k columns, so it is at most T.
// Second: the columns whose optimistic key reaches T0 - margin are the candidates
// (few more than those that reach T), and T, the k-th largest pessimistic key
// among them, makes the cut.  Should they exceed the table, the k-th of those
// listed is a better T0 and the pass runs again.
//
// Bound by the slab's read (the second pass finds its row in the L2) and, for
// short rows, by the two bit searches; pearson and covariance by the FP64 bounds,
// so their cut at T (and js's) reads the upper bounds that the second pass stored
// (formed again by one warp, four columns a lane, it cost more than a pass: 10,000
// queries x 1,000 references, k = 100, pearson 7,207 us and 4,960 now, covariance
// 3,249 and 2,160; the cheap bounds are formed again: binary, 10,000 x 10,000, 298
// us, stored 319).  us: 10,000 queries x 10,000 references
// (binary) 655 with scalar loads, per-pair term counts and IEEE divisions, 296
// now; 12,001 x 1,500 163 and 126; 1,500 x 12,001 121 and 52.  A warp per query
// with k-long sorted insertions, reading the norms through a column permutation,
// took 668 us for the last and 1,174 us for 1,000 x 20,000.
template <int KIND, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) k_screen_select(SelectScreenArgs A) {
  constexpr int NT = WARPS * 32;
  extern __shared__ uint32_t keys[];                 // max(slices * NT, cap)
  __shared__ float s_t;
  __shared__ int s_n;
  const int tid = threadIdx.x, lane = tid & 31;
  const int64_t ql = blockIdx.x;
  const int64_t q = A.q_begin + ql;
  const int K = A.k;
  const bool blank = A.qry_blank && A.qry_blank[q];
  if (blank || (A.qry_force_exact && A.qry_force_exact[q])) {
    if (tid == 0) { A.count[ql] = 0; A.overflow[ql] = blank ? 0 : 1; }
    return;
  }
  const ScreenBounds<KIND> bounds(A, q);
  const float* Srow = A.S + ql * A.ldS;
  const float4* S4 = reinterpret_cast<const float4*>(Srow);
  const kth::Group<1> G{nullptr};
  const int64_t n4 = (A.nr + 3) / 4, stretch = (n4 + A.slices - 1) / A.slices;
  // The thread's place in a stretch.  KIND 4: the warps take turns at the first
  // places, so that the stretches' short last rounds (always warp 0 otherwise, the
  // same quarter of every SM) spread over the FP64 pipes: covariance, 6,063 queries x
  // 5,669 references, k = 300, 8,156 us without and 7,352 with
  auto turn = [&](int sl) { return KIND == 4 ? (tid + 32 * (int)((blockIdx.x + sl) % WARPS)) % NT : tid; };
  for (int sl = 0; sl < A.slices; ++sl) {
    const int64_t g1 = min((sl + 1) * stretch, n4);
    float best = -INFINITY;
#pragma unroll 2
    for (int64_t g = sl * stretch + turn(sl); g < g1; g += NT) {
      float lo[4], hi[4];
      const unsigned ok = bounds(4 * g, A.nr, S4[g], lo, hi);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if ((ok >> u) & 1u) best = fmaxf(best, lo[u]);
    }
    keys[sl * NT + tid] = kth::fkey(best);
  }
  __syncthreads();
  if (tid < 32) {
    const float t = kth::fkey_value(kth::largest<1>(G, keys, A.slices * NT, K));
    if (lane == 0) s_t = t;
  }
  __syncthreads();
  auto cut_of = [](float T) {
    return T - ((T == -INFINITY || T == INFINITY) ? 0.f : fabsf(T) * (8.f * U32) + 1e-30f);
  };
  int32_t* out = A.cand + ql * (int64_t)A.cap;
  float* his = A.hi + ql * (int64_t)A.cap;
  int n = 0;
  for (int round = 0; round < 4; ++round) {
    const float cut = cut_of(s_t);
    if (tid == 0) s_n = 0;
    __syncthreads();
#pragma unroll 2
    for (int64_t g = turn(0); g < n4; g += NT) {
      float lo[4], hi[4];
      const unsigned ok = bounds(4 * g, A.nr, S4[g], lo, hi);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (((ok >> u) & 1u) && hi[u] >= cut) {
          const int at = atomicAdd(&s_n, 1);
          if (at < A.cap) {
            out[at] = (int32_t)(4 * g + u);
            keys[at] = kth::fkey(lo[u]);
            if constexpr (KIND >= 3) his[at] = hi[u];
          }
        }
      }
    }
    __syncthreads();
    n = s_n;
    if (n <= A.cap) break;
    if (tid < 32) {
      const float t = kth::fkey_value(kth::largest<1>(G, keys, A.cap, K));
      if (lane == 0) s_t = t;
    }
    __syncthreads();
    if (cut_of(s_t) <= cut) break;                   // ties: no better cut
  }
  if (n > A.cap) {
    if (tid == 0) { A.count[ql] = 0; A.overflow[ql] = 1; }
    return;
  }
  // the cut at T, in place, by one warp
  if (tid < 32) {
    int kept = n;
    if (n > K) {
      const float cut = cut_of(kth::fkey_value(kth::largest<1>(G, keys, n, K)));
      kept = 0;
      for (int t0 = 0; t0 < n; t0 += 32) {
        const int t = t0 + lane;
        const int32_t c = t < n ? out[t] : 0;
        bool keep = false;
        if constexpr (KIND >= 3) {
          keep = t < n && his[t] >= cut;
        } else if (t < n) {
          float lo[4], hi[4];
          bounds(c & ~3, A.nr, S4[c >> 2], lo, hi);
          const float h = (c & 2) ? ((c & 1) ? hi[3] : hi[2]) : ((c & 1) ? hi[1] : hi[0]);
          keep = h >= cut;
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);   // every lane has read slot t first
        if (keep) out[kept + __popc(m & ((1u << lane) - 1u))] = c;
        kept += __popc(m);
        __syncwarp();
      }
    }
    if (lane == 0) { A.count[ql] = kept; A.overflow[ql] = 0; }
  }
}

// ---------------------------------------------------------------------------
// the tensor-core screen
//
// For cosine and euclidean the screen value of a pair is an inner product
// over the rows (binary: of the 0 / 1 patterns, the matched-row count), so a
// dense FP16 copy of the screen values of both matrices (TensorCache) turns a
// block of screens into one GEMM on the tensor cores: the fused tcgen05
// kernel of sdg_sparse_tc.cu (FP16 in, FP32 accumulate; FP16 runs at BF16's
// tensor rate and rounds 4x finer, 2^-11) with the selection in its
// epilogue.  The bound (tcb::tc_bounds, sdg_tc_bounds.cuh) is built from each
// column's exact rounding error ||v - h|| (FP64, v the exact values, h the
// FP16 copy), so it covers every way the copy differs: values below FP16's
// smallest normal are written as 0, never as FP16 subnormals, and a value
// above FP16's range makes the copy unusable (TensorCache::usable: the FP32
// screen runs).  The FP16 products are exact in FP32; the FP32 accumulation
// of at most n = min(nnz_q, nnz_c) nonzero products (zero products add no
// error) is allowed (n + 64) 2^-21 of sum |h_q h_c|.
// ---------------------------------------------------------------------------
constexpr float HALF_MAX = 65504.f;
constexpr float HALF_MIN_NORMAL = 6.103515625e-05f;   // 2^-14

// One warp per column: scatter the FP16 values into the dense column and
// compute ||v - b|| and ||b|| in FP64 (v: src, the exact values; b: the FP16
// values the GEMM multiplies), rounded up to FP32.
__global__ void k_tensor_fill(DevCsc M, const float* fval, const double* src, __half* dense, int64_t ld,
                              float* err_out, float* bn_out, int* bad) {
  const int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (j >= M.ncol) return;
  __half* col = dense + j * ld;
  double se = 0.0, sb = 0.0;
  for (int64_t a = M.p[j] + lane; a < M.p[j + 1]; a += 32) {
    const float f = fval[a];
    const float af = fabsf(f);
    if (!(af <= HALF_MAX)) atomicOr(bad, 1);          // beyond FP16, or not finite
    const __half hv = __float2half_rn(af < HALF_MIN_NORMAL ? 0.f : f);
    col[M.i[a]] = hv;
    const double b = (double)__half2float(hv);
    const double v = src ? src[a] : (double)f;
    se += (v - b) * (v - b);
    sb += b * b;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    se += __shfl_xor_sync(0xffffffffu, se, o);
    sb += __shfl_xor_sync(0xffffffffu, sb, o);
  }
  if (lane == 0) {
    // FP64 sums and sqrt are within a few units of 2^-52; the factor and the
    // upward FP32 rounding cover them
    err_out[j] = __double2float_ru(sqrt(se) * (1.0 + 1e-12));
    bn_out[j] = __double2float_ru(sqrt(sb) * (1.0 + 1e-12));
  }
}

// Warp-cooperative insertion of the lanes flagged in m (value v on each lane)
// into lst[0..n), kept sorted descending and at most K long.
__device__ __forceinline__ void warp_insert_desc(float* lst, int K, int& n, unsigned m, float v, int lane) {
  while (m) {
    const int src = __ffs(m) - 1;
    m &= m - 1;
    const float x = __shfl_sync(0xffffffffu, v, src);
    if (n == K && !(x > lst[K - 1])) continue;
    int a = 0, b = n;
    while (a < b) { const int mid = (a + b) >> 1; if (lst[mid] >= x) a = mid + 1; else b = mid; }
    const int last = (n < K) ? n : K - 1;
    if (last > a) {
      for (int cch = (last - 1) >> 5; cch >= (a >> 5); --cch) {
        const int e = cch * 32 + lane;
        const bool mv = (e >= a && e < last);
        float t = 0.f;
        if (mv) t = lst[e];
        __syncwarp();
        if (mv) lst[e + 1] = t;
        __syncwarp();
      }
    }
    if (lane == 0) lst[a] = x;
    __syncwarp();
    if (n < K) ++n;
  }
}

// ---------------------------------------------------------------------------
// second screen of the tensor candidates: FP32 sparse dot products
//
// The FP16 bound keeps a few hundred candidates per query; the FP32 screen's
// bound (key_and_bound) is ~100x tighter.  One CTA per query holds the query
// column as a shared-memory bitmap (with each word's first entry, as in the
// exact re-rank) and its FP32 screen values; a warp per candidate streams the
// candidate column (coalesced, four rounds in flight), multiplies the matched
// FP32 values and reduces across the warp.  The FP32 bound holds for any
// summation order, so the reduction is a tree.  Then, per query, T2 = the
// k-th largest pessimistic key and the list keeps the candidates whose
// optimistic key reaches T2 - margin: the exact re-rank sees only those.
// ---------------------------------------------------------------------------
constexpr int RS_THREADS = 256;
constexpr int RS_MAX_QV = 4096;
constexpr int32_t RS_MAX_NROW = 1 << 18;

struct RescreenArgs {
  int method, k;
  DevCsc ref, qry;
  const float* rf;           // ScreenCache values (unit values / values)
  const float* qf;
  const int32_t* rnnz; const float* rnorm;
  const int32_t* qnnz; const float* qnorm;
  int64_t q_begin, nq;
  int selfmode;
  int cap;
  int32_t* cand;
  int32_t* count;
  float* lo;                 // [ql * cap + t]
  float* hi;
};

__global__ void k_rescreen(RescreenArgs A) {
  extern __shared__ __align__(16) uint32_t rs_smem[];
  const int W = (A.qry.nrow + 31) >> 5;
  float* qvs = reinterpret_cast<float*>(rs_smem);             // RS_MAX_QV
  uint32_t* bits = rs_smem + RS_MAX_QV;
  int32_t* first = reinterpret_cast<int32_t*>(bits + W);
  const int64_t ql = blockIdx.x;
  const int64_t q = A.q_begin + ql;
  const int n = A.count[ql];
  if (n == 0) return;
  for (int w = threadIdx.x; w < W; w += blockDim.x) bits[w] = 0u;
  __syncthreads();
  const int64_t q0 = A.qry.p[q], q1 = A.qry.p[q + 1];
  const bool qv_shared = (q1 - q0) <= RS_MAX_QV;
  for (int64_t e = q0 + threadIdx.x; e < q1; e += blockDim.x) {
    const int32_t r = A.qry.i[e];
    atomicOr(&bits[r >> 5], 1u << (r & 31));
    if (e == q0 || (A.qry.i[e - 1] >> 5) != (r >> 5)) first[r >> 5] = (int32_t)(e - q0);
    if (qv_shared) qvs[e - q0] = A.qf[e];
  }
  __syncthreads();
  const float* qv = qv_shared ? qvs : A.qf + q0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int32_t nq_ = A.qnnz[q];
  const float Nq = A.qnorm ? A.qnorm[q] : 0.f;
  for (int t = warp; t < n; t += nw) {
    const int32_t c = A.cand[ql * (int64_t)A.cap + t];
    float lo, hi;
    float acc = 0.f;
    const int64_t c0 = A.ref.p[c], c1 = A.ref.p[c + 1];
    for (int64_t a0 = c0; a0 < c1; a0 += 128) {
      int32_t r[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t e = a0 + 32 * u + lane;
        r[u] = (e < c1) ? __ldg(A.ref.i + e) : -1;
      }
      int qe[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        qe[u] = -1;
        if (r[u] >= 0) {
          const uint32_t wd = bits[r[u] >> 5];
          const uint32_t bit = 1u << (r[u] & 31);
          if (wd & bit) qe[u] = first[r[u] >> 5] + __popc(wd & (bit - 1u));
        }
      }
      float f[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) f[u] = (qe[u] >= 0) ? __ldg(A.rf + a0 + 32 * u + lane) : 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (qe[u] >= 0) acc = fmaf(f[u], qv[qe[u]], acc);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    float key, err;
    key_and_bound(A.method, acc, nq_, Nq, A.rnnz[c], A.rnorm ? A.rnorm[c] : 0.f, key, err);
    lo = key - err;
    hi = key + err;
    if (!(fabsf(key) <= FLT_MAX) || !(err <= FLT_MAX)) { lo = -INFINITY; hi = INFINITY; }
    if (A.selfmode && c == q) hi = INFINITY;  // the restored self pair (see ScreenBounds)
    if (lane == 0) {
      A.lo[ql * (int64_t)A.cap + t] = lo;
      A.hi[ql * (int64_t)A.cap + t] = hi;
    }
  }
}

// per query: T2 = k-th largest pessimistic key; compact the list in place to
// the candidates whose optimistic key reaches T2 - margin
__global__ void k_rescreen_select(RescreenArgs A) {
  extern __shared__ float lists[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t ql = (int64_t)blockIdx.x * SELECT_WARPS + warp;
  if (ql >= A.nq) return;
  const int n = A.count[ql];
  if (n == 0) return;
  const int K = A.k;
  float* lst = lists + warp * K;
  const float* lo = A.lo + ql * (int64_t)A.cap;
  const float* hi = A.hi + ql * (int64_t)A.cap;
  int m = 0;
  for (int p0 = 0; p0 < n; p0 += 32) {
    const float v = p0 + lane < n ? lo[p0 + lane] : -INFINITY;
    const unsigned b = __ballot_sync(0xffffffffu, v > -INFINITY && (m < K || v > lst[K - 1]));
    if (b) warp_insert_desc(lst, K, m, b, v, lane);
  }
  const float T = (m == K) ? lst[K - 1] : -INFINITY;
  const float cut = T - ((T == -INFINITY || T == INFINITY) ? 0.f : fabsf(T) * (8.f * U32) + 1e-30f);
  int32_t* cl = A.cand + ql * (int64_t)A.cap;
  int w = 0;
  for (int p0 = 0; p0 < n; p0 += 32) {
    const int p = p0 + lane;
    const bool keep = p < n && hi[p] >= cut;
    const int32_t cv = p < n ? cl[p] : 0;
    const unsigned b = __ballot_sync(0xffffffffu, keep);
    __syncwarp();
    if (keep) cl[w + __popc(b & ((1u << lane) - 1u))] = cv;
    w += __popc(b);
    __syncwarp();
  }
  if (lane == 0) A.count[ql] = w;
}

}  // namespace

bool tensor_supported(int method) { return method == BINARY || method == COSINE || method == EUCLIDEAN; }

static int64_t tensor_ld(int32_t nrow) { return ((int64_t)nrow + 63) / 64 * 64; }

size_t tensor_cache_bytes(int32_t nrow, int64_t ncol) {
  return (size_t)tensor_ld(nrow) * (size_t)ncol * 2;
}

void tensor_cache_free(TensorCache* c, cudaStream_t s) {
  if (c && c->dense) cudaFreeAsync(c->dense, s);
  if (c && c->err) cudaFreeAsync(c->err, s);
  if (c && c->bn) cudaFreeAsync(c->bn, s);
  if (c) *c = TensorCache();
}

// Builds (or reuses) the dense FP16 copy of M's screen values for `method`
// from its ScreenCache; an allocation failure leaves it unusable (the FP32
// screen then runs) rather than failing the call.
static int ensure_tensor(TensorCache* t, int method, const DevCsc& M, const ColAux& aux, const ScreenCache* sc,
                         std::mutex* mu, cudaStream_t s) {
  std::lock_guard<std::mutex> lock(*mu);
  if (t->method == method) return 0;
  tensor_cache_free(t, s);
  t->method = method;
  t->ld = tensor_ld(M.nrow);
  const size_t bytes = tensor_cache_bytes(M.nrow, M.ncol) + 256;
  cudaError_t e = cudaMallocAsync(&t->dense, bytes, s);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    t->dense = nullptr;
    t->usable = 0;
    return 0;
  }
  SK(e);
  const size_t nbytes = sizeof(float) * ((size_t)M.ncol + 4);
  SK(cudaMallocAsync(&t->err, nbytes, s));
  SK(cudaMallocAsync(&t->bn, nbytes, s));
  int* bad = nullptr;
  SK(cudaMallocAsync(&bad, sizeof(int), s));
  SK(cudaMemsetAsync(bad, 0, sizeof(int), s));
  SK(cudaMemsetAsync(t->dense, 0, bytes, s));
  if (M.ncol > 0)
    k_tensor_fill<<<blocks_for(M.ncol * 32, 256), 256, 0, s>>>(
        M, sc->fval, (method == COSINE) ? aux.uval : (method == EUCLIDEAN) ? M.x : nullptr,
        static_cast<__half*>(t->dense), t->ld, t->err, t->bn, bad);
  int hbad = 0;
  SK(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
  SK(cudaStreamSynchronize(s));
  SK(cudaFreeAsync(bad, s));
  t->usable = hbad ? 0 : 1;
  if (!t->usable) {
    SK(cudaFreeAsync(t->dense, s));
    t->dense = nullptr;
  }
  return 0;
}

void launch_check_rows(const DevCsc& M, int* err, cudaStream_t s) {
  if (M.ncol > 0) k_check_rows<<<blocks_for((int64_t)M.ncol * 32, 256), 256, 0, s>>>(M, err);
}

bool screen_supported(int method, int k) {
  return (method == BINARY || method == COSINE || method == EUCLIDEAN || method == MANHATTAN || method == JS ||
          method == PEARSON || method == COVARIANCE) &&
         k >= 1 && k <= kScreenMaxK;
}

// js's bound takes at most 2^-24 n <= 1/16 of its FP32 sums' terms (n the
// stored rows), and binary counts are exact in FP32 below 2^24 rows
bool screen_fits(int32_t nrow) { return nrow <= kScreenMaxRows; }

void screen_cache_free(ScreenCache* c, cudaStream_t s) {
  if (c && c->blob) cudaFreeAsync(c->blob, s);
  if (c && c->rows) cudaFreeAsync(c->rows, s);
  if (c && c->ent) cudaFreeAsync(c->ent, s);
  if (c && c->exl) cudaFreeAsync(c->exl, s);
  if (c && c->ready) cudaEventDestroy(c->ready);
  if (c) *c = ScreenCache();
}

// The per-matrix data of a method's screens is built by the first search that
// needs it, under the matrix's lock: searches of several threads may share a
// matrix, each on its stream.  The FP32 values are built without a
// synchronisation; a later search waits for their event on its own stream (on the
// host, knn-size calls from fresh matrices were 20 us slower).  The FP16 copy and
// the row-ordered entries are complete before the lock is released.
static int ensure_cache(ScreenCache* c, int method, const DevCsc& M, int64_t nnz, const ColAux& aux, std::mutex* mu,
                        cudaStream_t s) {
  const int family = method;
  std::lock_guard<std::mutex> lock(*mu);
  if (c->method == family) {
    SK(cudaStreamWaitEvent(s, c->ready, 0));
    return 0;
  }
  if (method == JS && !aux.xl) {                 // the js values' x log x come first
    g_screen_site = "js x log x values missing";
    return (int)cudaErrorInvalidValue;
  }
  screen_cache_free(c, s);
  // each array starts on a 256-byte boundary (16-byte vector loads of cnorm / nnz)
  auto seg = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
  const size_t b_fval = seg(sizeof(float) * ((size_t)nnz + 4));
  const size_t b_col = seg(sizeof(float) * ((size_t)M.ncol + 4));
  const bool js = method == JS;
  const size_t bytes = (js ? 2 : 1) * b_fval + 2 * b_col + 256;
  SK(cudaMallocAsync(&c->blob, bytes, s));
  char* b = static_cast<char*>(c->blob);
  c->fval = reinterpret_cast<float*>(b);
  b += b_fval;
  if (js) {
    c->fxl = reinterpret_cast<float*>(b);
    b += b_fval;
  }
  int* range_err = reinterpret_cast<int*>(static_cast<char*>(c->blob) + bytes - 256);
  c->cnorm = reinterpret_cast<float*>(b);
  b += b_col;
  c->nnz = reinterpret_cast<int32_t*>(b);
  c->nnz_total = nnz;
  if (M.ncol > 0) {
    SK(cudaMemsetAsync(range_err, 0, sizeof(int), s));
    k_screen_prep<<<blocks_for(M.ncol * 32, 256), 256, 0, s>>>(M, method, aux.uval, aux.xl, c->fval, c->fxl,
                                                                c->cnorm, c->nnz, range_err);
  }
  SK(cudaGetLastError());
  c->values_ok = true;
  if ((js || method == PEARSON || method == COVARIANCE) && M.ncol > 0) {
    int h_err = 0;
    SK(cudaMemcpyAsync(&h_err, range_err, sizeof(int), cudaMemcpyDeviceToHost, s));
    SK(cudaStreamSynchronize(s));
    c->values_ok = h_err == 0;
  }
  if (!c->ready) SK(cudaEventCreateWithFlags(&c->ready, cudaEventDisableTiming));
  SK(cudaEventRecord(c->ready, s));
  c->method = family;
  return 0;
}

// The entries of M in row order (see k_rows_fill).  rows stays null when the
// device has no room for it.
static int ensure_rows(ScreenCache* c, const DevCsc& M, std::mutex* mu, cudaStream_t s) {
  std::lock_guard<std::mutex> lock(*mu);
  if (c->rows || M.ncol == 0 || M.nrow == 0) return 0;
  // sub-ranges of 512 to 4,096 columns, about eight entries a cell
  const double density = (double)c->nnz_total / ((double)M.nrow * (double)M.ncol);
  int lg = 9;
  while (lg < 12 && density * (double)(1 << lg) < 8.0) ++lg;
  const int64_t nsub = (M.ncol + ((int64_t)1 << lg) - 1) >> lg;
  const int64_t cells = nsub * M.nrow;
  uint32_t *rows = nullptr, *cnt = nullptr;
  void *tmp = nullptr, *ent = nullptr, *exl = nullptr;
  size_t tb = 0;
  auto run = [&]() -> cudaError_t {
    cudaError_t e;
    if ((e = cudaMallocAsync(&rows, sizeof(uint32_t) * (size_t)(cells + 1), s))) return e;
    if ((e = cudaMallocAsync(&cnt, sizeof(uint32_t) * (size_t)(cells + 1), s))) return e;
    if ((e = cudaMallocAsync(&ent, sizeof(int2) * (size_t)std::max<int64_t>(c->nnz_total, 1), s))) return e;
    if (c->fxl && (e = cudaMallocAsync(&exl, sizeof(float) * (size_t)std::max<int64_t>(c->nnz_total, 1), s))) return e;
    if ((e = cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, rows, cells + 1, s))) return e;
    if ((e = cudaMallocAsync(&tmp, tb + 16, s))) return e;
    if ((e = cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * (size_t)(cells + 1), s))) return e;
    k_rows_count<<<blocks_for((int64_t)M.ncol * 32, 256), 256, 0, s>>>(M, lg, (int32_t)nsub, cnt);
    if ((e = cub::DeviceScan::ExclusiveSum(tmp, tb, cnt, rows, cells + 1, s))) return e;
    if ((e = cudaMemcpyAsync(cnt, rows, sizeof(uint32_t) * (size_t)(cells + 1), cudaMemcpyDeviceToDevice, s))) return e;
    k_rows_fill<<<blocks_for((int64_t)M.ncol * 32, 256), 256, 0, s>>>(M, lg, (int32_t)nsub, c->fval, c->fxl, cnt,
                                                                     static_cast<int2*>(ent), static_cast<float*>(exl));
    if (density * (double)(1 << lg) < ROWS_BANKS_MIN) return cudaStreamSynchronize(s);
    const size_t bsm = (size_t)ROWS_WARPS * 4 * (((size_t)1 << lg) / 32 + ((size_t)(exl ? 2 : 1) << lg));
    if (bsm > 48 * 1024 &&
        (e = cudaFuncSetAttribute(k_rows_banks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsm))) return e;
    k_rows_banks<<<(unsigned)std::min<int64_t>((cells + ROWS_WARPS - 1) / ROWS_WARPS, 152 * 32), ROWS_WARPS * 32, bsm,
                   s>>>(cells, lg, (int32_t)nsub, rows, static_cast<int2*>(ent), static_cast<float*>(exl));
    if ((e = cudaGetLastError())) return e;
    return cudaStreamSynchronize(s);
  };
  const cudaError_t e = run();
  if (cnt) cudaFreeAsync(cnt, s);
  if (tmp) cudaFreeAsync(tmp, s);
  if (e != cudaSuccess) {
    for (void* p : {(void*)rows, ent, exl}) if (p) cudaFreeAsync(p, s);
    if (e != cudaErrorMemoryAllocation) { g_screen_site = "ensure_rows"; return (int)e; }
    cudaGetLastError();
    return 0;
  }
  c->ent = ent;
  c->exl = static_cast<float*>(exl);
  c->nsub = (int32_t)nsub;
  c->sub_lg = lg;
  c->rows = rows;
  return 0;
}

// The columns of a part (a multiple of the sub-range) and the warps of a CTA for
// `units` stretches of queries: a run (one row's entries of a part) should give
// the lanes about 32 entries, the accumulators of a CTA's warps share
// kScreenAccBytes, and there should be an item for every warp of the chip.  At 5 %
// density 1,024 columns take 6.2 ms where 512 take 7.5 and 1,536 take 6.6 (24 or 28
// warps were slower than 32).  With fewer items than warps the CTAs get fewer
// warps, so that the items spread over the SMs.
static void screen_shape(const ScreenCache* rc, int64_t nr, int32_t nrow, int64_t units, int nsm, int* part_subs,
                         int* warps) {
  const int64_t sub = (int64_t)1 << rc->sub_lg;
  const double density = (double)rc->nnz_total / ((double)nrow * (double)nr);
  auto warps_of = [&](int64_t cols) {
    return (int)std::max<int64_t>(1, std::min<int64_t>(kScreenMaxWarps, (int64_t)kScreenAccBytes / (cols * 4)));
  };
  int64_t cols = (int64_t)std::min(13312.0, std::max(1024.0, 32.0 / std::max(density, 1e-9)));
  cols = std::min(cols, std::max<int64_t>(nr, 1));
  int64_t m = std::max<int64_t>(1, cols / sub);
  auto items = [&] { return units * ((nr + m * sub - 1) / (m * sub)); };
  while (m > 1 && items() < (int64_t)nsm * warps_of(m * sub)) m /= 2;
  *part_subs = (int)m;
  *warps = (int)std::min<int64_t>(warps_of(m * sub), std::max<int64_t>(1, (items() + nsm - 1) / nsm));
}

// Device buffers of one call, freed in stream order when it ends, also by an error
// return or an exception of a hook.
struct CallBuffers {
  cudaStream_t s;
  std::vector<void*> held;
  explicit CallBuffers(cudaStream_t stream) : s(stream) {}
  CallBuffers(const CallBuffers&) = delete;
  ~CallBuffers() { release(); }
  template <typename T>
  cudaError_t get(T** p, size_t bytes) {
    const cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(p), bytes, s);
    if (e == cudaSuccess) held.push_back(*p);
    return e;
  }
  void release() {
    for (void* p : held) cudaFreeAsync(p, s);
    held.clear();
  }
};

int screen_knn(cudaStream_t s, const ScreenRun& r, const DevCsc& ref, const ColAux& ra,
               ScreenCache* rc, TensorCache* rt, const DevCsc& qry, const ColAux& qa, ScreenCache* qc,
               TensorCache* qt, int32_t* d_idx, double* d_val, int64_t* stats, const ScreenHooks& hooks) {
  SKN((cudaError_t)ensure_cache(rc, r.method, ref, r.ref_nnz, ra, r.ref_mu, s));
  if (qc != rc) SKN((cudaError_t)ensure_cache(qc, r.method, qry, r.qry_nnz, qa, r.qry_mu, s));
  if ((r.method == JS || r.method == PEARSON || r.method == COVARIANCE) && !(rc->values_ok && qc->values_ok)) {
    // values outside the range the method's FP32 bound covers: every query exactly
    const int64_t lo = r.q_lo, hi = (r.q_hi < 0) ? qry.ncol : r.q_hi;
    if (hi > lo) hooks.exact_range(lo, hi - lo);
    return 0;
  }
  bool use_t = r.tensor && rt && qt && tensor_supported(r.method) && stc_supported(r.k);
  if (use_t) {
    SKN((cudaError_t)ensure_tensor(rt, r.method, ref, ra, rc, r.ref_mu, s));
    if (qt != rt) SKN((cudaError_t)ensure_tensor(qt, r.method, qry, qa, qc, r.qry_mu, s));
    use_t = rt->usable && qt->usable && rt->ld == qt->ld;
  }
  const int64_t nr = ref.ncol, nq = qry.ncol;
  const int32_t nrow = ref.nrow;
  if (!use_t) {
    SKN((cudaError_t)ensure_rows(rc, ref, r.ref_mu, s));
    if (!rc->rows) {                               // no room for the row-ordered entries: every query exactly
      const int64_t lo = r.q_lo, hi = (r.q_hi < 0) ? nq : r.q_hi;
      if (hi > lo) hooks.exact_range(lo, hi - lo);
      return 0;
    }
  }
  const int64_t q_lo = r.q_lo, q_hi = (r.q_hi < 0) ? nq : r.q_hi;
  const int64_t out_ld = (r.out_ld < 0) ? nq : r.out_ld;

  // queries per screen pass: the FP32 sparse screen's slab S is chunk x nr
  // floats; the fused tensor screen writes no slab and takes 4,096 queries
  // (16 query groups of 256, about one CTA per SM at ~10 reference ranges)
  const int64_t sbudget = (int64_t)4 << 30;
  const int64_t ldS = (nr + 3) / 4 * 4;           // float4 rows for the select
  const int64_t chunk = use_t ? std::min<int64_t>(std::max<int64_t>(q_hi - q_lo, 1), 4096)
                              : std::max<int64_t>(16, std::min<int64_t>(std::max<int64_t>(q_hi - q_lo, 1),
                                                                         sbudget / (4 * std::max<int64_t>(ldS, 1))));
  // the FP16 bound is wider than the FP32 one: room for more candidates
  const int cap = use_t ? std::max(512, std::min(16384, 64 * r.k + 256))
                        : std::max(256, std::min(8192, 16 * r.k + 64));
  CallBuffers buf(s);
  float *rlo = nullptr, *rhi = nullptr;
  if (use_t) {
    SK(buf.get(&rlo, sizeof(float) * (size_t)(chunk * cap + 4)));
    SK(buf.get(&rhi, sizeof(float) * (size_t)(chunk * cap + 4)));
  }

  float* S = nullptr;
  int32_t *cand = nullptr, *count = nullptr, *over = nullptr;
  unsigned long long* work = nullptr;
  int2* order = nullptr;
  int32_t* units = nullptr;
  const int64_t max_units = chunk + qc->nnz_total / SCREEN_SEG + 1;
  double* rvals = nullptr;
  uint8_t* force = nullptr;
  const int64_t cslots = chunk * (int64_t)cap;
  if (!use_t) SK(buf.get(&S, sizeof(float) * (size_t)(chunk * ldS + 4)));
  SK(buf.get(&cand, sizeof(int32_t) * (size_t)cslots));
  SK(buf.get(&count, sizeof(int32_t) * (size_t)chunk));
  SK(buf.get(&over, sizeof(int32_t) * (size_t)chunk));
  SK(buf.get(&rvals, sizeof(double) * (size_t)cslots));
  SK(buf.get(&work, sizeof(*work)));
  if (!use_t) {
    SK(buf.get(&order, sizeof(int2) * (size_t)max_units));
    SK(buf.get(&units, sizeof(int32_t)));
  }
  // cosine cannot bound an all-zero query (its convention value is not a dot
  // product): such queries go to the exact engine.
  if (r.method == COSINE && r.qry_empty) force = const_cast<uint8_t*>(r.qry_empty);

  int nsm = 152;
  {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  }

  std::vector<int> overflow_queries;
  for (int64_t q0 = q_lo; q0 < q_hi; q0 += chunk) {
    hooks.check_cancel();
    const int64_t nb = std::min(chunk, q_hi - q0);
    if (use_t) {
      // the fused tcgen05 screen: FP16 GEMM tiles of the block against every
      // reference with the FP16-bound selection in the epilogue
      StcRun T;
      T.method = r.method; T.k = r.k; T.selfmode = r.selfmode; T.include_self = r.include_self;
      T.ld = rt->ld; T.nr = nr; T.q0 = q0; T.nq = nb;
      T.rdense = static_cast<const __half*>(rt->dense); T.qdense = static_cast<const __half*>(qt->dense);
      T.rnnz = rc->nnz; T.rnorm = (r.method == EUCLIDEAN) ? rc->cnorm : nullptr;
      T.rerr = rt->err; T.rbn = rt->bn; T.ref_mask = r.ref_mask;
      T.qnnz = qc->nnz; T.qnorm = (r.method == EUCLIDEAN) ? qc->cnorm : nullptr;
      T.qerr = qt->err; T.qbn = qt->bn;
      T.qry_blank = r.qry_blank; T.qry_force = force;
      const int64_t ld = rt->ld;
      SK((cudaError_t)stc_screen(T, s, cand, count, over, cap, hooks.time_begin, hooks.time_end));
      if (nrow <= RS_MAX_NROW) {
        RescreenArgs R;
        R.method = r.method; R.k = r.k; R.ref = ref; R.qry = qry; R.rf = rc->fval; R.qf = qc->fval;
        R.rnnz = rc->nnz; R.rnorm = (r.method == EUCLIDEAN) ? rc->cnorm : nullptr;
        R.qnnz = qc->nnz; R.qnorm = (r.method == EUCLIDEAN) ? qc->cnorm : nullptr;
        R.q_begin = q0; R.nq = nb; R.selfmode = r.selfmode; R.cap = cap; R.cand = cand; R.count = count;
        R.lo = rlo; R.hi = rhi;
        const size_t rsmem = (size_t)RS_MAX_QV * 4 + (size_t)((nrow + 31) / 32) * 8;
        if (rsmem > 48 * 1024)
          SK(cudaFuncSetAttribute(k_rescreen, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rsmem));
        k_rescreen<<<(unsigned)nb, RS_THREADS, rsmem, s>>>(R);
        const size_t ssm = sizeof(float) * (size_t)SELECT_WARPS * r.k;
        if (ssm > 48 * 1024)
          SK(cudaFuncSetAttribute(k_rescreen_select, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssm));
        k_rescreen_select<<<blocks_for(nb, SELECT_WARPS), SELECT_WARPS * 32, ssm, s>>>(R);
        SK(cudaGetLastError());
      }
      stats[6] += 2 * ld * nr * nb;
    } else {
    ScreenArgs A;
    int warps = 1;
    // stretches of the chunk's queries, by the query matrix's mean
    const int64_t chunk_units = nb + (int64_t)((double)qc->nnz_total * (double)nb / (double)nq / SCREEN_SEG);
    screen_shape(rc, nr, nrow, chunk_units, nsm, &A.part_subs, &warps);
    A.rows = rc->rows; A.ent = static_cast<const int2*>(rc->ent); A.exl = rc->exl;
    A.nsub = rc->nsub; A.lg = rc->sub_lg; A.nr = nr; A.ldS = ldS;
    A.qp = qry.p; A.qi = qry.i; A.qv = qc->fval; A.qxl = qc->fxl; A.q_begin = q0; A.nq = nb;
    A.nparts = (rc->nsub + A.part_subs - 1) / A.part_subs;
    // parts of a group: their entries (kScreenGroupBytes) stay in the L2
    A.group = (int)std::max<int64_t>(
        1, std::min<int64_t>(A.nparts, kScreenGroupBytes / std::max<int64_t>(1, rc->nnz_total * 8 / A.nparts)));
    A.S = S; A.work = work;
    SK(cudaMemsetAsync(work, 0, sizeof(*work), s));
    A.order = order; A.units = units;
    k_screen_order<<<1, 1024, 0, s>>>(qc->nnz, q0, nb, order, units);
    k_screen_zero<<<(unsigned)nb, 256, 0, s>>>(qc->nnz, q0, nr, ldS, S);
    const size_t smem = sizeof(float) * (size_t)warps * ((size_t)A.part_subs << A.lg);
    auto kernel = r.method == MANHATTAN ? k_screen_rows<1> : r.method == JS ? k_screen_rows<2> : k_screen_rows<0>;
    // a function attribute is per device: set on every call (cheap, thread-safe)
    SK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScreenAccBytes));
    const int64_t grid = std::min<int64_t>(nsm, (chunk_units * A.nparts + warps - 1) / warps);
    hooks.time_begin();
    kernel<<<(unsigned)grid, warps * 32, smem, s>>>(A);
    hooks.time_end();
    SK(cudaGetLastError());

    SelectScreenArgs B;
    B.method = r.method; B.k = r.k; B.S = S; B.nr = nr; B.ldS = ldS;
    const bool normed = r.method == EUCLIDEAN || r.method == MANHATTAN || r.method == JS;
    B.rnnz = rc->nnz; B.rnorm = normed ? rc->cnorm : nullptr;
    B.qnnz = qc->nnz; B.qnorm = normed ? qc->cnorm : nullptr;
    B.rsum = ra.xsum; B.qsum = qa.xsum;
    B.rs = ra.s; B.rss = ra.ss; B.qs = qa.s; B.qss = qa.ss; B.nrow = ref.nrow;
    B.ref_mask = r.ref_mask; B.qry_blank = r.qry_blank; B.qry_force_exact = force;
    B.q_begin = q0; B.nq = nb; B.selfmode = r.selfmode; B.include_self = r.include_self;
    B.cap = cap; B.cand = cand; B.count = count; B.overflow = over;
    // 32 warps on a query where eight would leave SMs without a block
    const bool wide = nb < 2 * nsm;
    const int nt = wide ? 1024 : 256;
    B.slices = std::max(1, (4 * r.k + nt - 1) / nt);
    const size_t ssmem = sizeof(uint32_t) * (size_t)std::max(B.slices * nt, cap);
    B.hi = reinterpret_cast<float*>(rvals);          // free until the exact values are written
    auto pick = [&](auto k8, auto k32) { return wide ? k32 : k8; };
    auto select = r.method == COSINE ? pick(k_screen_select<0, 8>, k_screen_select<0, 32>)
                  : r.method == BINARY ? pick(k_screen_select<2, 8>, k_screen_select<2, 32>)
                  : r.method == JS ? pick(k_screen_select<3, 8>, k_screen_select<3, 32>)
                  : (r.method == PEARSON || r.method == COVARIANCE)
                      ? pick(k_screen_select<4, 8>, k_screen_select<4, 32>)
                      : pick(k_screen_select<1, 8>, k_screen_select<1, 32>);
    select<<<(unsigned)nb, nt, ssmem, s>>>(B);
    SK(cudaGetLastError());
    }

    // exact FP64 values of the kept pairs, then the exact top-k
    SK((cudaError_t)launch_rerank(r.method, r.dist, ref, ra, qry, qa, cand, count, cap, nb, q0,
                                  r.selfmode && r.include_self && r.method != COVARIANCE, r.self_value, rvals, r.k,
                                  nr > 0 ? (double)rc->nnz_total / (double)nr : 0.0,
                                  nq > 0 ? (double)qc->nnz_total / (double)nq : 0.0, s));
    SelectArgs sa;
    sa.vals = rvals; sa.seg_stride = cap; sa.elem_stride = 1; sa.nseg = nb;
    sa.cand = cand; sa.cand_count = count; sa.cand_ld = cap;
    sa.seg_blank = r.qry_blank ? r.qry_blank + r.out_first : nullptr;
    sa.out_idx = d_idx; sa.out_val = d_val; sa.out_ld = out_ld; sa.out_row0 = q0 - r.out_first;
    sa.k = r.k; sa.decreasing = r.decreasing;
    launch_select(sa, s);
    SK(cudaGetLastError());

    std::vector<int32_t> h_over((size_t)nb), h_count((size_t)nb);
    SK(cudaMemcpyAsync(h_over.data(), over, sizeof(int32_t) * nb, cudaMemcpyDeviceToHost, s));
    SK(cudaMemcpyAsync(h_count.data(), count, sizeof(int32_t) * nb, cudaMemcpyDeviceToHost, s));
    SK(cudaStreamSynchronize(s));
    for (int64_t t = 0; t < nb; ++t) {
      if (h_over[(size_t)t]) overflow_queries.push_back((int)(q0 + t));
      stats[1] += h_count[(size_t)t];
    }
    stats[0] += nb * nr;
    stats[3] += 6;
  }
  std::sort(overflow_queries.begin(), overflow_queries.end());
  overflow_queries.erase(std::unique(overflow_queries.begin(), overflow_queries.end()),
                         overflow_queries.end());
  stats[2] += (int64_t)overflow_queries.size();
  buf.release();
  // queries the screen could not bound: the exact slab engine
  if (!overflow_queries.empty()) hooks.exact_list(overflow_queries);
  return 0;
}

const char* screen_error_site() { return g_screen_site; }

}  // namespace sdg
