// Sparse products over the symmetric exchange matrix and deterministic reductions.
//
// S x = S' x + delta A x, S' = 0.5 (A F + F^T A) (porerad/exchange.py:108-112).  A product
// is one kernel: the row sums of S' x followed by a per-row epilogue (the update of the
// solver that consumes the product) and block reductions in a fixed order, so every
// result is bitwise reproducible for a given operator.  Two row-sum schemes:
//  * the word stream (k_spmv_stream, kStream storage): each CTA streams its rows' entries column
//    block by column block, with that block of x in shared memory;
//  * warp per row (k_spmv_rows, the other modes): lanes stride over the row's entries (coalesced
//    32-bit column loads, gathers of x through L1/L2), partial sums meet in a fixed shuffle tree.
#pragma once
#include <algorithm>
#include <mutex>
#include <vector>
#include <type_traits>

#include "pr_objects.cuh"

namespace pr {

#define PR_FULL 0xffffffffu

struct SymView {
  const int64_t* __restrict__ row_ptr;
  const uint32_t* __restrict__ cols;
  const int32_t* __restrict__ cnt;
  const double* __restrict__ val;
  double factor;
  int64_t n;
};

inline SymView sym_view(const SymCsr& S) {
  SymView v;
  v.row_ptr = S.row_ptr.ptr;
  v.cols = S.cols.ptr;
  v.cnt = S.cnt.ptr;
  v.val = S.val.ptr;
  v.factor = S.factor;
  v.n = S.n_rows;
  return v;
}

// Coefficient and column of entry q (storage modes kCounts and kValues).
template <int kMode, typename Acc>
__device__ __forceinline__ void sym_entry(const SymView& S, int64_t q, Acc& c, uint32_t& col) {
  col = __ldg(S.cols + q);
  if constexpr (kMode == kCounts) c = (Acc)__ldg(S.cnt + q);
  else c = (Acc)__ldg(S.val + q);
}

// sum_j S'_ij x_j in precision Acc, the full sum on every lane of the warp.  Lane l adds
// entries b + l, b + l + 32, ... in that order; four of them are loaded before the first
// is added, so four word loads and four gathers are in flight per lane (the order of the
// additions, and so the result, does not depend on the unrolling).
template <int kMode, typename Acc, typename Tx>
__device__ __forceinline__ Acc sym_row_acc(const SymView& S, int64_t i, const Tx* __restrict__ x, int lane) {
  const int64_t b = S.row_ptr[i], e = S.row_ptr[i + 1];
  Acc acc = 0;
  int64_t q = b + lane;
  for (; q + 96 < e; q += 128) {
    Acc c0, c1, c2, c3;
    uint32_t j0, j1, j2, j3;
    sym_entry<kMode>(S, q, c0, j0);
    sym_entry<kMode>(S, q + 32, c1, j1);
    sym_entry<kMode>(S, q + 64, c2, j2);
    sym_entry<kMode>(S, q + 96, c3, j3);
    const Acc x0 = (Acc)__ldg(x + j0), x1 = (Acc)__ldg(x + j1), x2 = (Acc)__ldg(x + j2), x3 = (Acc)__ldg(x + j3);
    acc = fma(c0, x0, acc);
    acc = fma(c1, x1, acc);
    acc = fma(c2, x2, acc);
    acc = fma(c3, x3, acc);
  }
  for (; q < e; q += 32) {
    Acc c;
    uint32_t j;
    sym_entry<kMode>(S, q, c, j);
    acc = fma(c, (Acc)__ldg(x + j), acc);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(PR_FULL, acc, o);
  return kMode == kValues ? acc : acc * (Acc)S.factor;
}

// Calls fn(std::integral_constant<int, mode>) for the matrix's storage mode.
template <typename Fn>
inline void dispatch_mode(int mode, Fn&& fn) {
  if (mode == kStream) fn(std::integral_constant<int, kStream>());
  else if (mode == kCounts) fn(std::integral_constant<int, kCounts>());
  else fn(std::integral_constant<int, kValues>());
}

// atomic max of a non-negative double (bit patterns of non-negative doubles order as integers)
__device__ __forceinline__ void atomic_max_nonneg(double* addr, double v) {
  if (!(v >= 0.0)) v = __longlong_as_double(0x7ff0000000000000ll);  // NaN -> +inf
  atomicMax((unsigned long long*)addr, (unsigned long long)__double_as_longlong(v));
}

// Block-wide sum of K values per thread (fixed tree), the same in every thread.
template <int K>
__device__ __forceinline__ void block_sum(double (&v)[K]) {
  __shared__ double red[32][K];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k)
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(PR_FULL, v[k], o);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) red[wid][k] = v[k];
  __syncthreads();
  if (threadIdx.x < K) {
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += red[w][threadIdx.x];
    red[0][threadIdx.x] = s;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = red[0][k];
  __syncthreads();
}

// The same into partial[slot * K + k]; slot defaults to the block index.
template <int K>
__device__ __forceinline__ void block_sum_store(double (&v)[K], double* __restrict__ partial, int64_t slot = -1) {
  block_sum<K>(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) partial[(slot < 0 ? (int64_t)blockIdx.x : slot) * K + k] = v[k];
}

// Sum of a[b * stride + off] over b < count by one warp in a fixed order: lane l adds b = l,
// l + 32, ... in turn (eight loads at a time), then the lanes meet in a fixed shuffle tree; every lane
// gets the sum.
__device__ __forceinline__ double warp_sum_partials(const double* __restrict__ a, int count, int stride, int off,
                                                    int lane) {
  double s = 0.0;
  for (int b0 = lane; b0 < count; b0 += 256) {
    double v[8];
#pragma unroll
    for (int h = 0; h < 8; ++h) v[h] = b0 + 32 * h < count ? a[(int64_t)(b0 + 32 * h) * stride + off] : 0.0;
#pragma unroll
    for (int h = 0; h < 8; ++h) s += v[h];
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(PR_FULL, s, o);
  return s;
}

// True in every thread of the block that finishes last, which then sees what all the others wrote.
// Every thread of each of `blocks` blocks calls it once per launch; *ticket is 0 before and after.  A block's
// scalars are taken here instead of in a kernel of their own (3 us and a launch per step of a solver
// whose steps take 5 to 50).
__device__ __forceinline__ bool last_block(int* ticket, int blocks) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1) == blocks - 1;
    if (last) {
      *ticket = 0;
      __threadfence();
    }
  }
  __syncthreads();
  return last != 0;
}

// True in thread 0 of the block that finishes last, where v[k] is then the sum over the blocks of
// partial[b * K + k] (block_sum_store), in a fixed order: thread t adds b = t, t + T, .. in turn and the
// threads meet in block_sum_store's tree.  The loads are what it waits for, so the whole block makes
// them at once: one warp adding 592 partials in turn took 3 us of the 10 of a step's kernel on 64^3 cells.
template <int K>
__device__ __forceinline__ bool last_block_sums(double (&v)[K], double* partial, int* ticket, int blocks = gridDim.x) {
  if (!last_block(ticket, blocks)) return false;
  const int T = blockDim.x;
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = 0.0;
  for (int b0 = threadIdx.x; b0 < blocks; b0 += 4 * T) {
    double w[4][K];
#pragma unroll
    for (int h = 0; h < 4; ++h)
#pragma unroll
      for (int k = 0; k < K; ++k) w[h][k] = b0 + h * T < blocks ? __ldcg(partial + (int64_t)(b0 + h * T) * K + k) : 0.0;
#pragma unroll
    for (int h = 0; h < 4; ++h)
#pragma unroll
      for (int k = 0; k < K; ++k) v[k] += w[h][k];
  }
  block_sum<K>(v);
  return threadIdx.x == 0;
}

// out[k] = sum over blocks of partial[b * K + k] (one warp per k, warp_sum_partials order).
__global__ void k_sum_partials(const double* __restrict__ partial, int blocks, int K, double* __restrict__ out);

int sum_partials(const double* partial, int blocks, int K, double* out, cudaStream_t s);


// ------------------------------------------------------------------ generic products

// An epilogue Epi provides: a Red type of per-thread reduction state (value-initialised),
// bool skip() (the whole product is skipped, e.g. a converged solve), row(i, s, red) with
// s = (S' x)_i, and finish(red), called by every thread of the block once its rows are done.

// What bounds it: the latency of the gathers, so all 8 blocks an SM that the grid has for it have to fit,
// which takes 32 registers (the series' last-block sums had brought it to 40, and a second, mostly empty
// wave).  Binary64 values, 96^3 foam, 56 M entries: a series product 267 -> 232 us, a balancing one 257 -> 221;
// 128^3, 166 M: 722 -> 660 and 709 -> 659.
template <int kMode, typename Acc, typename Tx, class Epi>
__global__ void __launch_bounds__(256, 8) k_spmv_rows(SymView S, const Tx* __restrict__ x, Epi epi) {
  if (epi.skip()) return;
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  typename Epi::Red red{};
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < S.n; i += warps) {
    const Acc sum = sym_row_acc<kMode, Acc>(S, i, x, lane);
    if (lane == 0) epi.row(i, sum, red);
  }
  epi.finish(red);
}

// ------------------------------------------------------------------ word-stream products

constexpr int kStreamSmemMax = 220 * 1024;  // dynamic shared memory of a product

struct StreamView {
  const uint4* __restrict__ quads;
  const int64_t* __restrict__ cta_row;
  const int64_t* __restrict__ base;
  const int32_t* __restrict__ q;
  const int16_t* __restrict__ start;
  int64_t n;
  double factor;
  int W, nb, rows_cap, groups;
};

inline StreamView stream_view(const SymCsr& S) {
  const SymStream& T = S.stream;
  return StreamView{T.quads.ptr, T.cta_row.ptr, T.base.ptr, T.q.ptr, T.start.ptr,
                    S.n_rows,    S.factor,      T.W,        T.nb,    T.rows_cap, T.groups};
}

// Values a product of S leaves for its second kernel (its scratch `part`), 0 with one group.
inline int64_t stream_part(const SymCsr& S) {
  return S.mode == kStream && S.stream.groups > 1 ? S.stream.groups * S.n_rows : 0;
}

// Columns of a group and the most sums (rows times groups) a product in groups leaves (operator.cu).  A
// block of 12 224 values of x leaves room for the sums of 14 900 rows, twice what a CTA holds on average
// of 2^20.  Groups of 9152 and of 16 320 columns are within 2 % of it at 36 000 to 62 000 patches; of 4096,
// with three times the sums, 5 to 12 % slower (64^3 fibers at 64 rays 19.5 instead of 17.5 us).
constexpr int64_t kStreamGroup = 12224, kStreamPartMax = 1 << 20;

constexpr int kStreamPad = 16;  // places after a block of x: the first is 0 (the others keep the blocks aligned)

// Shared memory of a product: the row sums, every lane's part of the row its run begins in, the sums
// that came in over a warp boundary (with one stage they are added to the row sums); then one or two
// blocks of x.
template <typename T>
__host__ __device__ inline size_t stream_sums(int rows_cap, int nb) {
  return (((size_t)(nb > 1 ? 2 : 1) * rows_cap + kStreamThreads) * sizeof(T) + 15) / 16 * 16;
}
template <typename T>
inline size_t stream_smem(const SymStream& S) {
  return stream_sums<T>(S.rows_cap, S.nb) + (size_t)(S.nb > 1 ? 2 : 1) * (S.W + kStreamPad) * sizeof(T);
}

// Column block b of x into shared memory, every value to its stream_place, by asynchronous copies of
// one value each (W is a multiple of 64, so places stay inside the block).
template <typename T>
__device__ __forceinline__ void stream_load_x(const StreamView& S, const T* x, int b, T* xs) {
  const int64_t c0 = (int64_t)b * S.W;
  const int cols = (int)min((int64_t)S.W, S.n - c0);
  const T* src = x + c0;
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(xs);
  for (int t = threadIdx.x; t < cols; t += kStreamThreads)
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst + (uint32_t)sizeof(T) * stream_place(t)),
                 "l"(src + t), "n"(sizeof(T))
                 : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// Asks L2 for quads [from, to) of a stream.
__device__ __forceinline__ void stream_prefetch(const uint4* quads, int64_t from, int64_t to) {
  if (from < to)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(quads + from), "r"((unsigned)(to - from) * 16u) : "memory");
}

// n of a word as a number: an exact integer set under the exponent of 2^52 (2^23), less that power.
__device__ __forceinline__ void stream_count(uint32_t w, double& c) {
  c = __hiloint2double(0x43300000, (int)(w & kStreamCount)) - 0x1.0p52;
}
__device__ __forceinline__ void stream_count(uint32_t w, float& c) {
  c = __uint_as_float(0x4b000000u | (w & kStreamCount)) - 0x1.0p23f;
}

// a += the four entries of a quad, in order, x the staged block.
template <typename T>
__device__ __forceinline__ void stream_quad(const uint4& w, const T* xs, T& a) {
  const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    T c;
    stream_count(ws[e], c);
    a = fma(c, xs[ws[e] >> (32 - kStreamColBits)], a);
  }
}

// The sums that warps of a stage left for the row they began in: added to `in` by one warp, lane w
// holding warp w's; warps inside one long row are neighbours with the same row and are summed in
// warp order first.
template <typename T>
__device__ __forceinline__ void stream_fold(const T* heads, const int* rows, T* in, int lane) {
  T v = heads[lane];
  const int r = rows[lane];
  for (int o = 1; o < 32; o <<= 1) {
    const T u = __shfl_up_sync(PR_FULL, v, o);
    const int k = __shfl_up_sync(PR_FULL, r, o);
    if (lane >= o && k == r) v += u;
  }
  const int next = __shfl_down_sync(PR_FULL, r, 1);
  if (r >= 0 && (lane == 31 || next != r)) in[r] += v;
  __syncwarp();
}

// The work of CTA `cta` of a product.  Every lane sums its run of quads; at a row start it adds the
// finished sum to the row (its own: the row began in this lane) or, the first time, to the lane's own
// slot, as the part of the row its predecessors began.  The runs of a warp then meet in one segmented
// scan, and what belongs to a row begun in an earlier warp goes through `head`.  So in every stage
// exactly one lane adds to a row's sum, and one warp adds the heads, in an order fixed by the layout.
//
// What bounds it: the stream from HBM, then the gathers from shared memory and the copies of x.  Runs
// of equal length keep all lanes busy whatever the rows' lengths, which groups of 8 lanes per row
// segment did not (14 of 32 lanes active, 2.1 warp instructions per entry).  U quads per lane are in
// flight while the U before them are summed, and one thread asks L2 for the stream kAhead of these
// steps before its quads are loaded (without it the loads waited on DRAM).  128^3 foam, 257 094
// patches, 155 and 285 M entries, binary64: 204 and 296 us (groups of 8 lanes: 485 and 615 us; of
// these 148 and 234 us the stream alone, 30 us the copies of x, 20 us the row sums); binary32: 153
// and 220 us (315 and 424 us).
template <int U, typename T, class Epi>
__device__ __forceinline__ void spmv_stream_cta(const StreamView& S, const T* x, T* part, const Epi& epi, int cta) {
  extern __shared__ __align__(16) unsigned char stream_mem[];
  __shared__ T head[2][32];
  __shared__ int head_row[2][32];
  T* sum = reinterpret_cast<T*>(stream_mem);  // rows_cap rows, then one slot per lane
  T* in = S.nb > 1 ? sum + S.rows_cap + kStreamThreads : sum;
  T* xs = reinterpret_cast<T*>(stream_mem + stream_sums<T>(S.rows_cap, S.nb));
  const int64_t v0 = S.cta_row[cta];
  const int rows = (int)(S.cta_row[cta + 1] - v0);
  int b0 = 0;  // first column block of the CTA's group
  if (S.groups > 1) b0 = (int)((uint32_t)v0 / (uint32_t)S.n) * S.nb;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int own = S.rows_cap + tid;
  typename Epi::Red red{};
  if (rows > 0) {
    const int64_t d0 = (int64_t)cta * S.nb;
    constexpr int64_t kStep = (int64_t)U * kStreamThreads;
    constexpr int kAhead = 8 / U;
    int64_t asked = S.base[d0];
    const int64_t end = S.base[d0 + S.nb];
    const uint4* __restrict__ p = S.quads + asked + tid;
    if (tid == 0) {
      stream_prefetch(S.quads, asked, min(end, asked + 2 * kAhead * kStep));
      asked += 2 * kAhead * kStep;
    }
    int step = 0;
    int q1 = S.q[d0], start1 = S.start[d0 * kStreamThreads + tid];
    uint4 cur[U];
#pragma unroll
    for (int u = 0; u < U; ++u) cur[u] = __ldg(p + u * kStreamThreads);
    for (int i = tid; i < rows; i += kStreamThreads) sum[i] = in[i] = T(0);
    if (tid < min(S.nb, 2)) xs[(size_t)tid * (S.W + kStreamPad) + S.W] = T(0);
    previous_done();
    if (epi.skip()) return;
    stream_load_x(S, x, b0, xs);
    for (int b = 0; b < S.nb; ++b) {
      const int q = q1, start = start1;
      if (b + 1 < S.nb) {
        q1 = S.q[d0 + b + 1];
        start1 = S.start[(d0 + b + 1) * kStreamThreads + tid];
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();  // block b of x is staged, stage b - 1 is done
      if (b + 1 < S.nb) stream_load_x(S, x, b0 + b + 1, xs + (size_t)((b + 1) & 1) * (S.W + kStreamPad));
      if (b > 0 && warp == 0) stream_fold(head[(b - 1) & 1], head_row[(b - 1) & 1], in, lane);
      const T* xb = xs + (size_t)(b & 1) * (S.W + kStreamPad);
      int row = start, at = own;
      T a = 0;
      sum[own] = T(0);
      for (int t = 0; t < q; t += U) {
        uint4 nxt[U];
        p += kStep;  // the next U quads: of this stage, the next one or past the end
        if (tid == 0 && ++step == kAhead) {
          stream_prefetch(S.quads, asked, min(end, asked + kAhead * kStep));
          asked += kAhead * kStep;
          step = 0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) nxt[u] = __ldg(p + u * kStreamThreads);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (cur[u].x & kStreamRow) {
            sum[at] += a;
            at = ++row;
            a = 0;
          }
          stream_quad(cur[u], xb, a);
          cur[u] = nxt[u];
        }
      }
      // a: what the run leaves to its last row (or, with no row start, adds to the row it began in);
      // with the lanes before it, back to the last row start
      const unsigned m = __ballot_sync(PR_FULL, row != start);
      const unsigned upto = m & (0xffffffffu >> (31 - lane));
      const int from = upto ? 31 - __clz(upto) : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const T u = __shfl_up_sync(PR_FULL, a, o);
        if (lane - o >= from) a += u;
      }
      T c = __shfl_up_sync(PR_FULL, a, 1);  // what the lanes before leave to the row this one began in
      if (lane == 0) c = 0;
      const int fl = m ? __ffs(m) - 1 : 32;  // the first lane with a row start
      if (row != start) {
        c += sum[own];
        if (lane > fl) sum[start] += c;
        else head[b & 1][warp] = c;
      }
      if (lane == 0) head_row[b & 1][warp] = start;
      if (lane == 31) {
        if (m) sum[row] += a;
        else head[b & 1][warp] = a;
      }
    }
    __syncthreads();
    if (warp == 0) stream_fold(head[(S.nb - 1) & 1], head_row[(S.nb - 1) & 1], in, lane);
    __syncthreads();
    if (S.groups > 1) {
      for (int i = tid; i < rows; i += kStreamThreads) part[v0 + i] = sum[i];
    } else {
      for (int i = tid; i < rows; i += kStreamThreads)
        epi.row(v0 + i, (S.nb > 1 ? sum[i] + in[i] : sum[i]) * (T)S.factor, red);
    }
  }
  if (S.groups > 1) return;
  if (rows == 0) {
    previous_done();
    if (epi.skip()) return;
  }
  epi.finish(red);
}

// The rows of a product in groups: the sums of a row's groups, added in order.
template <typename T, class Epi>
__device__ __forceinline__ void spmv_stream_rows(const StreamView& S, const T* part, const Epi& epi) {
  typename Epi::Red red{};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < S.n; i += (int64_t)gridDim.x * blockDim.x) {
    T v[4], a = 0;
    for (int g = 0; g < S.groups; g += 4) {
#pragma unroll
      for (int h = 0; h < 4; ++h) v[h] = g + h < S.groups ? part[(g + h) * S.n + i] : T(0);
#pragma unroll
      for (int h = 0; h < 4; ++h) a += v[h];
    }
    epi.row(i, a * (T)S.factor, red);
  }
  epi.finish(red);
}

template <typename T, class Epi>
__global__ void __launch_bounds__(256) k_stream_rows(StreamView S, const T* part, Epi epi) {
  previous_done();
  if (epi.skip()) return;
  spmv_stream_rows(S, part, epi);
}

template <int U, typename T, class Epi>
__global__ void __launch_bounds__(kStreamThreads, 1) k_spmv_stream(StreamView S, const T* x, T* part, Epi epi) {
  spmv_stream_cta<U>(S, x, part, epi, blockIdx.x);
}

// One product of each of several operators in one launch: item k owns the CTAs
// [cta_begin_k, cta_begin_{k+1}) of the grid.  The epilogue must not index per-block storage by
// blockIdx (BalanceEpi reduces with atomics only).
template <typename T, class Epi>
struct StreamItem {
  StreamView S;
  const T* x;
  T* part;
  Epi epi;
  int cta_begin, unroll;
};

template <typename T, class Epi>
__global__ void __launch_bounds__(kStreamThreads, 1) k_spmv_stream_batch(const StreamItem<T, Epi>* __restrict__ items,
                                                                         int n_items) {
  int lo = 0, hi = n_items - 1;  // the last item whose first CTA is at or before this one
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (items[mid].cta_begin <= (int)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  const StreamItem<T, Epi> it = items[lo];
  const int cta = (int)blockIdx.x - it.cta_begin;
  if (it.unroll == 2) spmv_stream_cta<2>(it.S, it.x, it.part, it.epi, cta);
  else spmv_stream_cta<1>(it.S, it.x, it.part, it.epi, cta);
}

// The rows of those in groups, blockIdx.y counting the items.
template <typename T, class Epi>
__global__ void __launch_bounds__(256) k_stream_rows_batch(const StreamItem<T, Epi>* __restrict__ items) {
  const StreamItem<T, Epi>& it = items[blockIdx.y];
  if (it.S.groups == 1 || it.epi.skip()) return;
  spmv_stream_rows(it.S, (const T*)it.part, it.epi);
}

// Lets `kernel` use kStreamSmemMax of shared memory, once per device.
template <typename Kernel>
inline int allow_stream_smem(Kernel* kernel, bool (&done)[64]) {
  static std::mutex mu;
  int dev = 0;
  PR_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev >= 0 && dev < 64 && done[dev]) return PR_OK;
  PR_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmemMax));
  if (dev >= 0 && dev < 64) done[dev] = true;
  return PR_OK;
}

// Blocks of a product of S (the number of partial-sum slots its block reductions fill).
inline int spmv_slots(const SymCsr& S) {
  if (S.mode == kStream && S.stream.groups == 1) return S.stream.ctas;
  if (S.mode == kStream) return grid_for(S.n_rows, 256, sm_count() * 4);
  return grid_for(S.n_rows * 32, 256, sm_count() * 8);
}

// One product of S with x (device vector of n entries) and the epilogue epi; part: scratch of
// stream_part(S) values.
template <int kMode, typename T, class Epi>
inline int launch_spmv(const SymCsr& S, const T* x, T* part, const Epi& epi, cudaStream_t s) {
  if constexpr (kMode == kStream) {
    static bool done[2][64] = {};
    const size_t smem = stream_smem<T>(S.stream);
    auto go = [&](auto* kernel, bool (&ready)[64]) -> int {
      PR_TRY(allow_stream_smem(kernel, ready));
      ::pr::launch_mark();
      PR_CUDA(launch_early(kernel, S.stream.ctas, kStreamThreads, smem, s, stream_view(S), x, part, epi));
      return PR_OK;
    };
    PR_TRY(S.stream.unroll == 2 ? go(k_spmv_stream<2, T, Epi>, done[0]) : go(k_spmv_stream<1, T, Epi>, done[1]));
    if (S.stream.groups > 1) {
      ::pr::launch_mark();
      PR_CUDA(launch_early(k_stream_rows<T, Epi>, spmv_slots(S), 256, 0, s, stream_view(S), (const T*)part, epi));
    }
  } else {
    ::pr::launch_mark(), k_spmv_rows<kMode, T, T, Epi><<<spmv_slots(S), 256, 0, s>>>(sym_view(S), x, epi);
  }
  PR_CUDA(cudaGetLastError());
  return PR_OK;
}

// One product of each of the operators mats[k] (kStream) with xs[k], scratch parts[k] and epilogue
// epis[k], all in one launch (and one for the rows of those in groups).  items is device scratch for mats.size() items.
template <typename T, class Epi>
inline int launch_spmv_batch(const std::vector<const SymCsr*>& mats, const std::vector<const T*>& xs,
                             const std::vector<T*>& parts, const std::vector<Epi>& epis, StreamItem<T, Epi>* items, cudaStream_t s) {
  const int n = (int)mats.size();
  if (n == 0) return PR_OK;
  std::vector<StreamItem<T, Epi>> h(n);
  size_t smem = 0;
  int ctas = 0;
  int64_t rows = 0;  // of the largest operator in groups
  for (int i = 0; i < n; ++i) {
    const SymCsr& S = *mats[i];
    if (S.mode != kStream) {
      set_error("batched product: operator %d is not stored as a word stream", i);
      return PR_ERR_ARG;
    }
    h[i] = StreamItem<T, Epi>{stream_view(S), xs[i], parts[i], epis[i], ctas, S.stream.unroll};
    ctas += S.stream.ctas;
    smem = std::max(smem, stream_smem<T>(S.stream));
    if (S.stream.groups > 1) rows = std::max(rows, S.n_rows);
  }
  static bool done[64] = {};
  PR_TRY(allow_stream_smem(k_spmv_stream_batch<T, Epi>, done));
  PR_CUDA(cudaMemcpyAsync(items, h.data(), sizeof(StreamItem<T, Epi>) * n, cudaMemcpyHostToDevice, s));
  ::pr::launch_mark(), k_spmv_stream_batch<T, Epi><<<ctas, kStreamThreads, smem, s>>>(items, n);
  for (int c = 0; rows > 0 && c < n; c += 65535) {
    const dim3 grid((unsigned)grid_for(rows, 256, sm_count() * 4), (unsigned)std::min(n - c, 65535));
    ::pr::launch_mark(), k_stream_rows_batch<T, Epi><<<grid, 256, 0, s>>>(items + c);
  }
  PR_CUDA(cudaGetLastError());
  return PR_OK;
}

}  // namespace pr
