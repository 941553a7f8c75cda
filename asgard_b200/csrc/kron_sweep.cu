// Terms acting in several dimensions, applied as a tree of one-dimensional
// passes ("sweeps") over vectors of the whole grid (n = 3).
//
// The operator of a term over all connected cell pairs is
//   y_r = sum_c (A_0[r_0, c_0] (x) ... (x) A_{d-1}[r_{d-1}, c_{d-1}]) x_c.
// Splitting each 1D operator at its diagonal, A_k = U_k + L_k (U: c_k >= r_k
// in the order of the 1D cells, L: c_k < r_k), every product of parts can be
// applied one dimension at a time without leaving the grid when the U parts
// come first and the L parts last: after the U parts a cell has only moved
// to coarser 1D cells, and what the L parts still have to reach is finer
// (the reference's upper/lower permutations, global_cpu,
// src/device/asgard_glkronmult_cpu.cpp:103-181, and its permutes,
// src/device/asgard_kronmult.hpp:152-224).  The one dimension between them
// takes its whole operator.  Needed of the grid: with a cell, the cells that
// replace one 1D index by a connected lower one are in it (sweep_build checks).
//
// Products that begin alike share their first passes and products that end
// alike their last ones: with X_0 = x, a pass X_{m + s} = U_s X_m for every
// subset m of the dimensions above s; then Y_m = A_0 X_m for every m; then
// Y_{m + s} += L_s Y_m, which leaves the term's product in the last Y.  That
// is 2^(m+1) - 2 half operators for a term of m dimensions, where the
// 2^(m-1) separate chains take (m + 1) 2^(m-1) half operators: 30 against 40
// at m = 4, 126 against 224 at m = 6.  The chains take fewer launches, though
// (m, all chains and terms side by side, against 2m - 1), which decides on
// grids of few values.
#include "internal.cuh"

#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <numeric>
#include <type_traits>

namespace asgk
{
enum sweep_fill
{
  kSweepUpper = 0,
  kSweepBoth  = 1,
  kSweepLower = 2
};

struct sweep_launch
{
  int job0 = 0, njobs = 0, blocks = 0; // blocks: the most of any job
};

// The units (a block each) of one dimension and fill.
struct sweep_units
{
  int first = 0, count = 0;
};

struct sweep_data
{
  int d = 0;
  int64_t N = 0; // values of one vector
  int4 *units = nullptr;
  int *index  = nullptr;
  int4 *recs  = nullptr;
  int4 *jobs  = nullptr;
  int *last   = nullptr; // [nresults] the vectors whose sum is the product
  double *work = nullptr;
  // Whose turn with work it is: one thread enqueues at a time, and an apply
  // waits for the one before it on another stream (done, once used is set; a
  // stream is told by its id, which unlike its handle is never used again).
  std::recursive_mutex turn;
  cudaEvent_t done = nullptr;
  bool used        = false;
  unsigned long long by = 0; // the stream of the last apply or solve
  int nresults = 0;
  bool chains  = false; // separate chains, not a tree
  sweep_units su[6][3];
  std::vector<sweep_launch> launches;
};

namespace
{
constexpr int ipow3w(int k) { return k == 0 ? 1 : 3 * ipow3w(k - 1); }

constexpr int kWarps = 8; // per block
constexpr int kSweepBlocks = 2;
// cells of a pencil that one thread holds in registers
constexpr int kSmall = 8;
// Entries of a row that one warp sums, and entries that one block takes: long
// blocks reuse the columns' values in L1 (d=4 level 7: 254 us with 16 and
// 128, 273 with 8 and single rounds, 307 with 16 and 512); a grid too small
// to fill the GPU wants short ones (d=3 level 6: 47 and 39 us).
constexpr int kRowEntries = 16, kBlockEntries = 128;
constexpr int kRowEntriesFew = 8, kBlockEntriesFew = 1;
constexpr int64_t kFewValues = 1 << 18;
// Where the terms run as separate chains: on a grid of few values, when the
// values of the passes that the tree would share and the products to add up
// stay few.  One FP64 apply of terms acting in every dimension, tree and
// chains: d=3 level 6, 2 terms 33.9 and 20.8 us; d=4 level 3, 1 term 38 and
// 25; d=5 level 4, 1 term (2.7 million extra values) 62 and 47, 3 terms (8.0
// million) 88 and 95; d=4 level 6, 2 terms (2.5 million) 79 and 76, 4 terms
// 122 and 130; d=6 level 1, 1 term (32 chains) 32 and 25, 3 terms (96) 34 and
// 36, 6 terms 39 and 59.
constexpr int64_t kChainExtra = int64_t(4) << 20;
constexpr int kChainSums      = 64;

template<typename TC> struct padW;
template<> struct padW<double> { static constexpr int value = 10; };
template<> struct padW<float> { static constexpr int value = 12; };

struct unit_tables
{
  sweep_units u[18]; // by 3 * dimension + fill
};

__device__ __forceinline__ void load_block(const double *b, double (&a)[9])
{
  const double2 *q = reinterpret_cast<const double2 *>(b);
#pragma unroll
  for (int i = 0; i < 4; i++)
  {
    double2 const t = __ldg(q + i);
    a[2 * i]        = t.x;
    a[2 * i + 1]    = t.y;
  }
  a[8] = __ldg(b + 8);
}
__device__ __forceinline__ void load_block(const float *b, float (&a)[9])
{
  const float4 *q = reinterpret_cast<const float4 *>(b);
  float4 const t0 = __ldg(q), t1 = __ldg(q + 1);
  a[0] = t0.x; a[1] = t0.y; a[2] = t0.z; a[3] = t0.w;
  a[4] = t1.x; a[5] = t1.y; a[6] = t1.z; a[7] = t1.w;
  a[8] = __ldg(b + 8);
}

// A launch of the tree may begin while the one before it drains: what does
// not change between applies (jobs, units, records, factors) is read before
// wait_previous, vectors after it.
__device__ __forceinline__ void let_next_begin()
{
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_previous()
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// acc += A v, A a column-major block: out_q += sum_p A(q, p) v_p, A(q, p) = a[q + 3p]
template<typename TC>
__device__ __forceinline__ void block_fma(TC const (&a)[9], TC v0, TC v1, TC v2, TC (&acc)[3])
{
  acc[0] = fma(a[6], v2, fma(a[3], v1, fma(a[0], v0, acc[0])));
  acc[1] = fma(a[7], v2, fma(a[4], v1, fma(a[1], v0, acc[1])));
  acc[2] = fma(a[8], v2, fma(a[5], v1, fma(a[2], v0, acc[2])));
}

__device__ __forceinline__ void shared_block(const double *b, double (&a)[9])
{
  const double2 *q = reinterpret_cast<const double2 *>(b);
#pragma unroll
  for (int i = 0; i < 4; i++)
  {
    double2 const t = q[i];
    a[2 * i]        = t.x;
    a[2 * i + 1]    = t.y;
  }
  a[8] = b[8];
}
__device__ __forceinline__ void shared_block(const float *b, float (&a)[9])
{
  const float4 *q = reinterpret_cast<const float4 *>(b);
  float4 const t0 = q[0], t1 = q[1];
  a[0] = t0.x; a[1] = t0.y; a[2] = t0.z; a[3] = t0.w;
  a[4] = t1.x; a[5] = t1.y; a[6] = t1.z; a[7] = t1.w;
  a[8] = b[8];
}

// Pencils of up to R cells for C columns of a lane: the fibre of every cell in
// registers, the cells' outputs one after the other, a factor read once for
// the C columns.  All warps of the block take the same class, whose factors
// (conn[r * R + c]: the connection of output r and input c, -1 none) they
// stage in shared memory while the fibres are on their way: read one by one
// where they are used, each would cost its connection's and its own L2
// latency.  cells: the cell table [member][pencil]; columns q0 + 32 i.
template<int R, int C, int D, typename TC, typename TI>
__device__ __forceinline__ void
small_pencils(int m, int np, const int *__restrict__ cells, int q0,
              const int *__restrict__ conn, const TC *__restrict__ P, int pstep,
              const TI *__restrict__ in, TC *__restrict__ out, bool add, int stride,
              TC *stage, int *on)
{
  constexpr int TS = ipow3w(D), F = TS / 3, PAD = padW<TC>::value;
  for (int e = threadIdx.x; e < R * R * 9; e += kWarps * 32)
  {
    int const pair = e / 9, i = e - 9 * pair;
    int const cn   = pair < m * R ? __ldg(conn + pair) : -1;
    if (i == 0)
      on[pair] = cn;
    if (cn >= 0)
      stage[pair * PAD + i] = __ldg(P + int64_t(cn) * pstep + i);
  }
  int at[C][R]; // where each cell's fibre begins, -1: none
  TC v[C][R][3];
#pragma unroll
  for (int i = 0; i < C; i++)
  {
    int const q      = q0 + 32 * i;
    int const pencil = q / F, f = q - pencil * F;
    int const base   = (f / stride) * 3 * stride + f % stride;
#pragma unroll
    for (int c = 0; c < R; c++)
      at[i][c] = (pencil < np && c < m) ? __ldg(cells + c * np + pencil) * TS + base : -1;
  }
  wait_previous();
#pragma unroll
  for (int i = 0; i < C; i++)
#pragma unroll
    for (int c = 0; c < R; c++)
    {
      v[i][c][0] = v[i][c][1] = v[i][c][2] = TC(0);
      if (at[i][c] >= 0)
      {
        const TI *p = in + at[i][c];
        v[i][c][0]  = static_cast<TC>(p[0]);
        v[i][c][1]  = static_cast<TC>(p[stride]);
        v[i][c][2]  = static_cast<TC>(p[2 * stride]);
      }
    }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; r++)
  {
    if (r >= m)
      break;
    TC acc[C][3];
#pragma unroll
    for (int i = 0; i < C; i++)
    {
      acc[i][0] = acc[i][1] = acc[i][2] = TC(0);
      if (add && at[i][r] >= 0)
      {
        const TC *o = out + at[i][r];
        acc[i][0]   = o[0];
        acc[i][1]   = o[stride];
        acc[i][2]   = o[2 * stride];
      }
    }
#pragma unroll
    for (int c = 0; c < R; c++)
      if (on[r * R + c] >= 0)
      {
        TC a[9];
        shared_block(stage + (r * R + c) * PAD, a);
#pragma unroll
        for (int i = 0; i < C; i++)
          block_fma(a, v[i][c][0], v[i][c][1], v[i][c][2], acc[i]);
      }
#pragma unroll
    for (int i = 0; i < C; i++)
      if (at[i][r] >= 0)
      {
        TC *o         = out + at[i][r];
        o[0]          = acc[i][0];
        o[stride]     = acc[i][1];
        o[2 * stride] = acc[i][2];
      }
  }
}

// Rounds of rows of large pencils for a tile of 32 columns (a lane each): in
// a round every warp sums up to kRowEntries entries of one row (a longer row
// takes 2, 4 or 8 warps, whose sums the first of them adds in order).
template<int TS, typename TC, typename TI>
__device__ __forceinline__ void
large_pencil(const int4 *__restrict__ recs, int rounds, const int *__restrict__ entries,
             const int *__restrict__ cells, int step, bool live, const TC *__restrict__ P,
             int pstep, const TI *__restrict__ in, TC *__restrict__ out, bool add, int base,
             int stride, TC (*part)[3][32])
{
  int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int2 *pairs = reinterpret_cast<const int2 *>(entries);
  // {row (-1: none), first entry, entries, warps of the row | warp << 8 |
  // some row of this round is split << 16}
  int4 next = __ldg(recs + warp);
  int2 ahead = lane < next.z ? __ldg(pairs + next.y + lane) : make_int2(0, 0);
  wait_previous();
  for (int q = 0; q < rounds; q++)
  {
    int4 const rec  = next;
    int const warps = rec.w & 255, sub = (rec.w >> 8) & 255;
    bool const split = (rec.w >> 16) != 0;
    if (q + 1 < rounds)
      next = __ldg(recs + (q + 1) * kWarps + warp);
    TC acc[3] = {TC(0), TC(0), TC(0)};
    for (int j0 = 0; j0 < rec.z; j0 += 32)
    {
      int const nj    = min(32, rec.z - j0);
      int2 const mine = ahead;
      if (j0 + 32 < rec.z)
        ahead = j0 + 32 + lane < rec.z ? __ldg(pairs + rec.y + j0 + 32 + lane) : make_int2(0, 0);
#pragma unroll 4
      for (int j = 0; j < nj; j++)
      {
        int const c = __shfl_sync(0xffffffffu, mine.x, j);
        int const n = __shfl_sync(0xffffffffu, mine.y, j);
        const TI *p = in + int64_t(__ldg(cells + c * step)) * TS + base;
        TC a[9];
        load_block(P + int64_t(n) * pstep, a);
        block_fma(a, static_cast<TC>(p[0]), static_cast<TC>(p[stride]),
                  static_cast<TC>(p[2 * stride]), acc);
      }
    }
    if (q + 1 < rounds && lane < next.z)
      ahead = __ldg(pairs + next.y + lane);
    if (split)
    {
      __syncthreads(); // the sums of the round before have been read
      part[warp][0][lane] = acc[0];
      part[warp][1][lane] = acc[1];
      part[warp][2][lane] = acc[2];
      __syncthreads();
      if (sub == 0)
        for (int w = 1; w < warps; w++)
        {
          acc[0] += part[warp + w][0][lane];
          acc[1] += part[warp + w][1][lane];
          acc[2] += part[warp + w][2][lane];
        }
    }
    if (rec.x >= 0 && sub == 0 && live)
    {
      TC *o = out + int64_t(__ldg(cells + rec.x * step)) * TS + base;
      if (add)
      {
        acc[0] += o[0];
        acc[1] += o[stride];
        acc[2] += o[2 * stride];
      }
      o[0]          = acc[0];
      o[stride]     = acc[1];
      o[2 * stride] = acc[2];
    }
  }
}

// One launch of the tree: blockIdx.y is a job (input vector, -1 the operator's
// x; 2 * output vector, odd to add to it; 3 * dimension + fill; term),
// blockIdx.x a range of the units of its dimension and fill.  Pencils that
// hold the same 1D cells form a class and share every index and factor below
// the cells themselves; a class's columns are its pencils' fibres (3^(d-1) each), 32 to a tile, one
// to a lane, so a warp's factors are uniform and no lane is idle whatever d.
// Pencils of up to kSmall cells: kSmall cell fibres per lane, the shorter the
// pencils the more tiles.  Bound by the latency of its loads at two blocks of
// 126 registers per SM, 23 % of the warps: the widest launches use the
// load/store pipe to 59 % (d=4 level 7) and 47 % (d=6 level 5, where DRAM moves
// 3.4 TB/s), narrow ones wait for one chain of loads.  One FP64 apply, all
// launches: d=4 level 7, 4 terms 254 us (5305 by the pair kernel); d=6 level
// 5, 6 terms 2.96 ms (21.8); d=3 level 6, 2 terms, as separate chains 26 us
// (129 with a kernel of a thread per output entry).  Two blocks per SM: more
// spill the fibres (d=4 277 -> 320-500 us with three or four).
template<int D, typename TC, typename TX>
__global__ void __launch_bounds__(kWarps * 32, kSweepBlocks)
    k_sweep(const int4 *__restrict__ units, unit_tables tab,
            const int *__restrict__ index, const int4 *__restrict__ recs,
            const int4 *__restrict__ jobs, const TC *__restrict__ P, int T,
            const TX *__restrict__ x, TC *__restrict__ work, int64_t N,
            const double *__restrict__ gate)
{
  if (gate_closed(gate))
    return;
  constexpr int TS = ipow3w(D), F = TS / 3;
  __shared__ TC part[kWarps][3][32];
  __shared__ __align__(16) TC stage[kSmall * kSmall * padW<TC>::value];
  __shared__ int on[kSmall * kSmall];
  int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  let_next_begin();
  int4 const job       = __ldg(jobs + blockIdx.y);
  sweep_units const su = tab.u[job.z];
  if (int(blockIdx.x) >= su.count)
    return;
  // {cells of a pencil, pencils, cell table [member][pencil], first tile},
  // {entries, first record, rounds} or {connections, cells at most, 0}
  int64_t const u = 2 * (int64_t(su.first) + blockIdx.x);
  int4 const ua = __ldg(units + u), ub = __ldg(units + u + 1);
  int const k = job.z / 3;
  int stride  = 1;
#pragma unroll
  for (int j = 1; j < D; j++)
    if (k < j)
      stride *= 3;
  const TC *Pk     = P + (int64_t(k) * T + job.w) * padW<TC>::value;
  int const pstep  = D * T * padW<TC>::value;
  TC *out          = work + int64_t(job.y >> 1) * N;
  const TC *in     = work + int64_t(job.x < 0 ? 0 : job.x) * N;
  bool const add   = (job.y & 1) != 0;
  auto go          = [&](auto *src) {
    const int *cells = index + ua.z, *list = index + ub.x;
    if (ub.z > 0)
    {
      int const column = ua.w * 32 + lane;
      bool const live  = column < ua.y * F;
      int const pencil = live ? column / F : 0, f = live ? column - pencil * F : 0;
      int const base   = (f / stride) * 3 * stride + f % stride;
      large_pencil<TS>(recs + ub.y, ub.z, list, cells + pencil, ua.y, live, Pk, pstep, src, out,
                       add, base, stride, part);
      return;
    }
    int const column = (ua.w + warp * (kSmall / ub.y)) * 32 + lane;
    switch (ub.y)
    {
    case 1:
      small_pencils<1, kSmall, D>(ua.x, ua.y, cells, column, list, Pk, pstep, src, out, add,
                                  stride, stage, on);
      break;
    case 2:
      small_pencils<2, kSmall / 2, D>(ua.x, ua.y, cells, column, list, Pk, pstep, src, out, add,
                                      stride, stage, on);
      break;
    case 4:
      small_pencils<4, kSmall / 4, D>(ua.x, ua.y, cells, column, list, Pk, pstep, src, out, add,
                                      stride, stage, on);
      break;
    default:
      small_pencils<8, kSmall / 8, D>(ua.x, ua.y, cells, column, list, Pk, pstep, src, out, add,
                                      stride, stage, on);
      break;
    }
  };
  if (job.x < 0)
    go(x);
  else
    go(in);
}

// y = beta y + alpha (sum of the terms' products, in term order) + ex x
template<typename TC, typename TX, typename TY>
__global__ void k_sweep_sum(int terms, const int *__restrict__ last,
                            const TC *__restrict__ work, int64_t N, double alpha,
                            const TX *__restrict__ x, double ex, double beta,
                            TY *__restrict__ y, const double *__restrict__ gate)
{
  wait_previous();
  if (gate_closed(gate))
    return;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < N;
       i += int64_t(gridDim.x) * blockDim.x)
  {
    double s = 0.0;
    for (int t = 0; t < terms; t++)
      s += static_cast<double>(work[int64_t(__ldg(last + t)) * N + i]);
    double v = alpha * s;
    if (ex != 0.0)
      v += ex * static_cast<double>(x[i]);
    if (beta != 0.0)
      v += beta * static_cast<double>(y[i]);
    y[i] = static_cast<TY>(v);
  }
}

template<int D, typename TC, typename TX, typename TY>
int launch_d(sweep_data const &w, const TC *P, int T, double alpha, const TX *x,
             double beta, TY *y, double ex, cudaStream_t s)
{
  TC *work = reinterpret_cast<TC *>(w.work);
  unit_tables tab;
  for (int k = 0; k < D; k++)
    for (int f = 0; f < 3; f++)
      tab.u[3 * k + f] = w.su[k][f];
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(kWarps * 32);
  cfg.stream   = s;
  cfg.attrs    = &early;
  cfg.numAttrs = g_recording ? 0 : 1; // a recorded cycle's nodes run in plain order
  for (auto const &l : w.launches)
  {
    cfg.gridDim = dim3(l.blocks, l.njobs);
    ASGK_CUDA(cudaLaunchKernelEx(&cfg, k_sweep<D, TC, TX>, static_cast<const int4 *>(w.units), tab,
                                 static_cast<const int *>(w.index),
                                 static_cast<const int4 *>(w.recs),
                                 static_cast<const int4 *>(w.jobs + l.job0), P, T, x, work, w.N, g_gate));
    count_launch();
  }
  cfg.gridDim = dim3(int(std::min<int64_t>((w.N + 255) / 256, 148 * 8)));
  ASGK_CUDA(cudaLaunchKernelEx(&cfg, k_sweep_sum<TC, TX, TY>, w.nresults,
                               static_cast<const int *>(w.last), static_cast<const TC *>(work),
                               w.N, alpha, x, ex, beta, y, g_gate));
  count_launch();
  return ASGK_OK;
}

template<typename TC, typename TX, typename TY>
int launch_t(sweep_data const &w, const TC *P, int T, double alpha, const TX *x,
             double beta, TY *y, double ex, cudaStream_t s)
{
  switch (w.d)
  {
  case 1: return launch_d<1>(w, P, T, alpha, x, beta, y, ex, s);
  case 2: return launch_d<2>(w, P, T, alpha, x, beta, y, ex, s);
  case 3: return launch_d<3>(w, P, T, alpha, x, beta, y, ex, s);
  case 4: return launch_d<4>(w, P, T, alpha, x, beta, y, ex, s);
  case 5: return launch_d<5>(w, P, T, alpha, x, beta, y, ex, s);
  case 6: return launch_d<6>(w, P, T, alpha, x, beta, y, ex, s);
  default: return ASGK_ERR_UNSUPPORTED;
  }
}

// ------------------------------------------------------------ host set-up

// Pencils of one dimension that hold the same 1D cells.
struct pencil_class
{
  std::vector<int> ids;   // 1D cells, ascending
  std::vector<int> first; // each pencil's first place in the cell order
  int cells = 0;          // cell table [member][pencil] in the index array
};

// The pencils of dimension k by class, larger classes first; order: the cells
// sorted by their other 1D cells, then by k's.  Empty when a cell is listed
// twice or (closed) a connected lower 1D cell of a member is missing.
std::vector<pencil_class> find_pencils(int d, int cells, const int *oned, const int *lut, int R1,
                                       int k, bool closed, std::vector<int> &order)
{
  std::iota(order.begin(), order.end(), 0);
  std::sort(order.begin(), order.end(), [&](int a, int b) {
    const int *x = oned + size_t(a) * d, *y = oned + size_t(b) * d;
    for (int j = 0; j < d; j++)
      if (j != k && x[j] != y[j])
        return x[j] < y[j];
    return x[k] < y[k];
  });
  auto same = [&](int a, int b) {
    for (int j = 0; j < d; j++)
      if (j != k && oned[size_t(a) * d + j] != oned[size_t(b) * d + j])
        return false;
    return true;
  };
  std::map<std::vector<int>, std::vector<int>> by;
  std::vector<int> ids;
  for (int p0 = 0; p0 < cells;)
  {
    int p1 = p0;
    ids.clear();
    for (; p1 < cells && same(order[p0], order[p1]); p1++)
    {
      ids.push_back(oned[size_t(order[p1]) * d + k]);
      if (p1 > p0 && ids[p1 - p0] == ids[p1 - p0 - 1])
        return {};
    }
    by[ids].push_back(p0);
    p0 = p1;
  }
  std::vector<pencil_class> out;
  std::vector<char> in(R1);
  for (auto const &c : by)
  {
    std::fill(in.begin(), in.end(), 0);
    for (int a : c.first)
      in[a] = 1;
    if (closed)
      for (int a : c.first)
        for (int b = 0; b < a; b++)
          if (!in[b] && (lut[size_t(a) * R1 + b] >= 0 || lut[size_t(b) * R1 + a] >= 0))
            return {};
    out.push_back({c.first, c.second, 0});
  }
  std::stable_sort(out.begin(), out.end(), [](pencil_class const &a, pencil_class const &b) {
    return a.ids.size() > b.ids.size();
  });
  return out;
}

// The units of one dimension and fill (see k_sweep).  Rows that a pass does
// not reach are left out when it adds to its output.
void build_units(std::vector<pencil_class> const &classes, const int *lut, int R1, int F, int fill,
                 bool adds, std::vector<int4> &units, std::vector<int> &index,
                 std::vector<int4> &recs, bool few, sweep_units &su)
{
  su.first = int(units.size() / 2);
  for (auto const &c : classes)
  {
    int const m = int(c.ids.size()), np = int(c.first.size());
    int const tiles = int((int64_t(np) * F + 31) / 32);
    auto conn       = [&](int r, int q) {
      bool const in = fill == kSweepBoth || (fill == kSweepUpper ? q >= r : q < r);
      return in ? lut[size_t(c.ids[r]) * R1 + c.ids[q]] : -1;
    };
    if (m <= kSmall)
    {
      int R = 1;
      while (R < m)
        R *= 2;
      int const at = int(index.size());
      bool any     = !adds;
      for (int r = 0; r < m; r++)
        for (int q = 0; q < R; q++)
        {
          index.push_back(q < m ? conn(r, q) : -1);
          any = any || index.back() >= 0;
        }
      if (any)
        for (int t = 0; t < tiles; t += kWarps * (kSmall / R))
        {
          units.push_back(make_int4(m, np, c.cells, t));
          units.push_back(make_int4(at, R, 0, 0));
        }
      continue;
    }
    // rows with their entries, those of many warps first
    struct row
    {
      int r, e0, n, warps;
    };
    std::vector<row> rows;
    if (index.size() % 2)
      index.push_back(0); // entries are read in pairs of words
    int const at = int(index.size());
    for (int r = 0; r < m; r++)
    {
      row w{r, int(index.size() - at) / 2, 0, 1};
      for (int q = 0; q < m; q++)
        if (conn(r, q) >= 0)
        {
          index.push_back(q);
          index.push_back(conn(r, q));
          ++w.n;
        }
      while (w.warps < kWarps && w.n > w.warps * (few ? kRowEntriesFew : kRowEntries))
        w.warps *= 2;
      if (w.n > 0 || !adds)
        rows.push_back(w);
    }
    std::stable_sort(rows.begin(), rows.end(), [](row const &a, row const &b) {
      return a.warps != b.warps ? a.warps > b.warps : a.n > b.n;
    });
    // rounds of kWarps warps; blocks of about kBlockEntries entries
    std::vector<std::pair<int, int>> parts; // first record, rounds
    size_t const recs0 = recs.size();
    int slot = kWarps, have = 0, r0 = int(recs0);
    for (auto const &w : rows)
    {
      if (slot + w.warps > kWarps)
      {
        if (have >= (few ? kBlockEntriesFew : kBlockEntries))
        {
          parts.emplace_back(r0, (int(recs.size()) - r0) / kWarps);
          r0   = int(recs.size());
          have = 0;
        }
        recs.resize(recs.size() + kWarps, make_int4(-1, 0, 0, 1));
        slot = 0;
      }
      int4 *rec = recs.data() + recs.size() - kWarps;
      for (int s = 0; s < w.warps; s++, slot++)
      {
        int const a = int(int64_t(w.n) * s / w.warps), b = int(int64_t(w.n) * (s + 1) / w.warps);
        rec[slot] = make_int4(w.r, w.e0 + a, b - a, w.warps | (s << 8));
      }
      have += w.n;
    }
    // all warps of a round with a split row meet at its barriers
    for (size_t i = recs0; i < recs.size(); i += kWarps)
    {
      bool split = false;
      for (int s = 0; s < kWarps; s++)
        split = split || (recs[i + s].w & 255) > 1;
      for (int s = 0; s < kWarps && split; s++)
        recs[i + s].w |= 1 << 16;
    }
    if (int(recs.size()) > r0)
      parts.emplace_back(r0, (int(recs.size()) - r0) / kWarps);
    for (int t = 0; t < tiles; t++)
      for (auto const &p : parts)
      {
        units.push_back(make_int4(m, np, c.cells, t));
        units.push_back(make_int4(at, p.first, p.second, 0));
      }
  }
  su.count = int(units.size() / 2) - su.first;
}

// The launches of the tree, with the vectors they use.  A level of the tree
// runs breadth first (one launch for all vectors of the level) while the
// vectors that this needs below it stay within `wide`, else depth first, so
// that at most two vectors per level wait.
struct tree_plan
{
  std::vector<int4> jobs;
  std::vector<sweep_launch> launches;
  std::vector<int> spare;
  int vectors = 0, wide = 0;
  sweep_units const (*su)[3] = nullptr;

  struct node
  {
    int vec;               // the vector holding X (-1: the operator's x)
    const std::vector<int> *term; // term, then its dimensions a_0 < a_1 < ...
  };
  int take()
  {
    if (!spare.empty())
    {
      int const v = spare.back();
      spare.pop_back();
      return v;
    }
    return vectors++;
  }
  void drop(int v)
  {
    if (v >= 0)
      spare.push_back(v);
  }
  void launch(std::vector<int4> const &js)
  {
    sweep_launch l;
    l.job0  = int(jobs.size());
    l.njobs = int(js.size());
    for (auto const &j : js)
      l.blocks = std::max(l.blocks, su[j.z / 3][j.z % 3].count);
    jobs.insert(jobs.end(), js.begin(), js.end());
    if (l.blocks > 0)
      launches.push_back(l);
  }
  // the products of dimensions a_0 .. a_s applied to every node's vector;
  // all nodes' terms act in the same number of dimensions
  std::vector<int> run(std::vector<node> const &in, int s)
  {
    std::vector<int4> js;
    std::vector<int> out;
    if (s == 0)
    {
      for (auto const &q : in)
      {
        out.push_back(take());
        js.push_back(make_int4(q.vec, 2 * out.back(), 3 * (*q.term)[1] + kSweepBoth, (*q.term)[0]));
      }
      launch(js);
      return out;
    }
    int64_t const need = int64_t(in.size()) << (s + 1);
    if (in.size() > 1 && need > wide)
    {
      for (auto const &q : in)
        out.push_back(run({q}, s)[0]);
      return out;
    }
    std::vector<node> up;
    for (auto const &q : in)
    {
      up.push_back({take(), q.term});
      js.push_back(make_int4(q.vec, 2 * up.back().vec, 3 * (*q.term)[1 + s] + kSweepUpper, (*q.term)[0]));
    }
    launch(js);
    std::vector<int> low;
    if (need <= wide)
    {
      std::vector<node> both(in);
      both.insert(both.end(), up.begin(), up.end());
      std::vector<int> const y = run(both, s - 1);
      low.assign(y.begin(), y.begin() + in.size());
      out.assign(y.begin() + in.size(), y.end());
      for (auto const &q : up)
        drop(q.vec);
    }
    else
    {
      out = run(up, s - 1);
      for (auto const &q : up)
        drop(q.vec);
      low = run(in, s - 1);
    }
    js.clear();
    for (size_t i = 0; i < in.size(); i++)
      js.push_back(make_int4(low[i], 2 * out[i] + 1, 3 * (*in[i].term)[1 + s] + kSweepLower,
                             (*in[i].term)[0]));
    launch(js);
    for (int v : low)
      drop(v);
    return out;
  }
  // Every term's chains: for each subset of the dimensions above a_0 their
  // upper parts from the last dimension down, the whole operator of a_0, the
  // lower parts of the other dimensions upwards.  A launch takes the next pass
  // of all of them; chains that begin alike are one until they part.
  std::vector<int> chains(std::vector<std::vector<int>> const &terms)
  {
    struct link
    {
      int vec; // -1: the operator's x
      const std::vector<int> *term;
      int q;                // the last upper part was dimension a_q's
      std::vector<int> low; // the dimensions left to their lower parts
      int lows;             // lower parts applied, -1 before a_0's operator
    };
    std::vector<link> now;
    std::vector<int> out;
    for (auto const &t : terms)
      now.push_back({-1, &t, int(t.size()) - 1, {}, -1});
    while (!now.empty())
    {
      std::vector<link> then;
      std::vector<int4> js;
      auto pass = [&](link const &l, int s, int fill, link child) {
        child.vec = take();
        js.push_back(make_int4(l.vec, 2 * child.vec, 3 * (*l.term)[1 + s] + fill, (*l.term)[0]));
        then.push_back(std::move(child));
      };
      std::vector<int> read;
      for (auto const &l : now)
      {
        if (l.lows == int(l.low.size()))
        {
          out.push_back(l.vec);
          continue;
        }
        read.push_back(l.vec);
        if (l.lows >= 0)
        {
          link child = l;
          child.lows++;
          pass(l, l.low[l.lows], kSweepLower, std::move(child));
          continue;
        }
        for (int s = l.q - 1; s >= 0; s--) // a_s next, those between go lower
        {
          link child = l;
          child.q    = s;
          for (int j = l.q - 1; j > s; j--)
            child.low.insert(child.low.begin(), j);
          child.lows = s == 0 ? 0 : -1;
          pass(l, s, s == 0 ? kSweepBoth : kSweepUpper, std::move(child));
        }
      }
      launch(js);
      for (int v : read)
        drop(v);
      now.swap(then);
    }
    return out;
  }
};

template<typename T>
int upload(T **dst, std::vector<T> const &src, int64_t &bytes)
{
  size_t const b = std::max<size_t>(src.size(), 1) * sizeof(T);
  if (cudaMalloc(reinterpret_cast<void **>(dst), b) != cudaSuccess)
  {
    cudaGetLastError();
    *dst = nullptr;
    return ASGK_ERR_ALLOC;
  }
  bytes += int64_t(b);
  if (!src.empty())
    ASGK_CUDA(cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice));
  return ASGK_OK;
}
} // namespace

void sweep_free(sweep_data *w)
{
  if (w == nullptr)
    return;
  cudaFree(w->units);
  cudaFree(w->index);
  cudaFree(w->recs);
  cudaFree(w->jobs);
  cudaFree(w->last);
  cudaFree(w->work);
  if (w->done)
    cudaEventDestroy(w->done);
  delete w;
}

// oned[cells][d]: the cells' 1D indices (< R1); lut[R1][R1]: the connection of
// (row, column) 1D cells or -1; terms: (term, its dimensions in increasing
// order) each.  ASGK_ERR_UNSUPPORTED with require_closed when the grid is not
// closed below in a dimension (the products' intermediate cells would be
// missing).
int sweep_build(int d, int cells, const int *oned, const int *lut, int R1,
                std::vector<std::vector<int>> const &terms, bool require_closed,
                sweep_data **out, int64_t &bytes)
{
  *out = nullptr;
  std::unique_ptr<sweep_data, void (*)(sweep_data *)> w(new (std::nothrow) sweep_data(), sweep_free);
  if (!w)
    return ASGK_ERR_ALLOC;
  w->d = d;
  w->N = int64_t(cells) * ipow3w(d);
  if (w->N >= int64_t(1) << 31) // places in a vector are 32-bit
    return ASGK_ERR_UNSUPPORTED;
  int64_t chains = 0, extra = 0; // passes of halves beyond the tree's
  for (auto const &t : terms)
  {
    int const m = int(t.size()) - 1;
    chains += int64_t(1) << (m - 1);
    extra += (int64_t(m + 1) << (m - 1)) - ((int64_t(2) << m) - 2);
  }
  w->chains = w->N < kFewValues && chains <= kChainSums && extra * w->N <= kChainExtra;
  bool used[6][3] = {};
  size_t widest   = 0;
  for (auto const &t : terms)
  {
    used[t[1]][kSweepBoth] = true;
    for (size_t i = 2; i < t.size(); i++)
      used[t[i]][kSweepUpper] = used[t[i]][kSweepLower] = true;
    widest = std::max(widest, t.size() - 1);
  }
  std::vector<int4> units, recs;
  std::vector<int> index, order(cells);
  for (int k = 0; k < d; k++)
  {
    if (!used[k][0] && !used[k][1] && !used[k][2])
      continue;
    auto classes = find_pencils(d, cells, oned, lut, R1, k, require_closed, order);
    if (classes.empty())
      return ASGK_ERR_UNSUPPORTED;
    for (auto &c : classes)
    {
      c.cells = int(index.size());
      for (size_t i = 0; i < c.ids.size(); i++)
        for (int p0 : c.first)
          index.push_back(order[p0 + i]);
    }
    for (int f = 0; f < 3; f++)
      if (used[k][f])
        build_units(classes, lut, R1, int(w->N / cells / 3), f, f == kSweepLower && !w->chains,
                    units, index, recs, w->N < kFewValues, w->su[k][f]);
    if (index.size() > size_t(1) << 30)
      return ASGK_ERR_UNSUPPORTED;
  }
  // as many vectors at once as keep the tree's working set in kSweepBytes
  tree_plan tp;
  tp.su   = w->su;
  tp.wide = int(std::min<int64_t>(1 << 20, kSweepBytes / (w->N * int64_t(sizeof(double)))));
  std::vector<int> last;
  if (w->chains)
    last = tp.chains(terms);
  for (size_t m = 1; m <= widest && !w->chains; m++)
  {
    std::vector<tree_plan::node> roots;
    for (auto const &t : terms)
      if (t.size() == m + 1)
        roots.push_back({-1, &t});
    if (roots.empty())
      continue;
    auto const r = tp.run(roots, int(m) - 1);
    last.insert(last.end(), r.begin(), r.end());
  }
  w->nresults = int(last.size());
  w->launches = tp.launches;
  int rc       = ASGK_OK;
  int64_t held = 0;
  if ((rc = upload(&w->units, units, held)) || (rc = upload(&w->index, index, held)) ||
      (rc = upload(&w->recs, recs, held)) ||
      (rc = upload(&w->jobs, tp.jobs, held)) || (rc = upload(&w->last, last, held)))
    return rc;
  size_t const b = size_t(tp.vectors) * size_t(w->N) * sizeof(double);
  if (cudaMalloc(reinterpret_cast<void **>(&w->work), b) != cudaSuccess)
  {
    cudaGetLastError();
    w->work = nullptr;
    return ASGK_ERR_ALLOC;
  }
  ASGK_CUDA(cudaEventCreateWithFlags(&w->done, cudaEventDisableTiming));
  bytes += held + int64_t(b);
  *out = w.release();
  return ASGK_OK;
}

namespace
{
int launch_tree(plan_data const &p, sweep_data const &w, int precision, double alpha,
                const void *x, bool f32, double beta, void *y, double ex, cudaStream_t s)
{
  if (f32)
    return launch_t<float, float, float>(w, p.vP32, p.terms, alpha, static_cast<const float *>(x),
                                         beta, static_cast<float *>(y), ex, s);
  const double *xd = static_cast<const double *>(x);
  double *yd       = static_cast<double *>(y);
  if (precision == ASGK_FP64)
    return launch_t<double, double, double>(w, p.vP64, p.terms, alpha, xd, beta, yd, ex, s);
  if (precision == ASGK_FP32)
    return launch_t<float, double, double>(w, p.vP32, p.terms, alpha, xd, beta, yd, ex, s);
  return ASGK_ERR_UNSUPPORTED;
}
} // namespace

sweep_turn::sweep_turn(sweep_data *w) : w_(w)
{
  if (w_)
    w_->turn.lock();
}
sweep_turn::~sweep_turn()
{
  if (w_)
    w_->turn.unlock();
}
int sweep_turn::wait(cudaStream_t s)
{
  if (w_ == nullptr)
    return ASGK_OK;
  unsigned long long id = 0;
  ASGK_CUDA(cudaStreamGetId(s, &id));
  if (w_->used && id != w_->by) // a wait of no use costs an apply 2 us
    ASGK_CUDA(cudaStreamWaitEvent(s, w_->done, 0));
  w_->by = id;
  return ASGK_OK;
}

// y = beta y + alpha (sum of the terms) x + ex x, the vectors of FP32
// (x_f32: arithmetic FP32) or FP64
int launch_sweep(plan_data const &p, sweep_data &w, int precision, double alpha, const void *x,
                 bool f32, double beta, void *y, double ex, cudaStream_t s)
{
  // what is recorded runs where the graph is launched
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusActive;
  if (!g_recording)
    ASGK_CUDA(cudaStreamIsCapturing(s, &capture));
  if (capture != cudaStreamCaptureStatusNone)
    return launch_tree(p, w, precision, alpha, x, f32, beta, y, ex, s);
  sweep_turn turn(&w);
  if (int rc = turn.wait(s))
    return rc;
  int const rc = launch_tree(p, w, precision, alpha, x, f32, beta, y, ex, s);
  ASGK_CUDA(cudaEventRecord(w.done, s));
  w.used = true;
  return rc;
}

} // namespace asgk
