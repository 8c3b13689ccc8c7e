// Exchange operator on the device: pooling of arbitrary edge lists, the ray
// accounting check, the symmetric exchange matrix, diagonal balancing, the
// projected products and the reciprocity diagnostic.
//
// Follows porerad/exchange.py:37-197:
//   weight w_ij = n_ij / R_i                                       (exchange.py:72)
//   S = 0.5 (A F + F^T A) + delta A                                (exchange.py:108-112)
//   d > 0 with d * (S d) = A, found as y = log d from the residual
//   f(y) = y + log(S e^y) - log A; convergence when max|f| <= tol, acceptance when
//   the closure max|d (S d) / A - 1| <= min(max(10 tol, 10 eps), 1e-10); otherwise
//   the damped multiplicative iteration y += 0.5 (log A - log(d * S d)) until the
//   closure is <= min(tol, 1e-10) (exchange.py:153-197)
//   row_sum_error = max|F_p 1 - 1| <= 1e-10                       (exchange.py:78-80)
// The reference accelerates the log-residual with scipy.optimize.anderson; here it
// is type-II Anderson acceleration (Walker & Ni 2011) of the damped fixed-point map
// y <- y - beta f(y), history m = 10, beta = 1/2, least squares by the normal
// equations with a pseudo-inverse cut at 10 eps of the largest eigenvalue.  The
// solution d is defined by the equation, so the iterate path may differ from
// SciPy's; d itself agrees to the balancing tolerance.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_reduce.cuh>
#include <cub/device/device_scan.cuh>

#include <cmath>
#include <vector>

#include "pr_spmv.cuh"

namespace pr {

__global__ void k_sum_partials(const double* __restrict__ partial, int blocks, int K, double* __restrict__ out) {
  const int k = blockIdx.x;
  const double s = warp_sum_partials(partial, blocks, K, k, threadIdx.x & 31);
  if (threadIdx.x == 0) out[k] = s;
}

int sum_partials(const double* partial, int blocks, int K, double* out, cudaStream_t s) {
  ::pr::launch_mark(), k_sum_partials<<<K, 32, 0, s>>>(partial, blocks, K, out);
  PR_CUDA(cudaGetLastError());
  return PR_OK;
}


// ------------------------------------------------------------------ pooling

__global__ void k_edge_keys(const int32_t* __restrict__ o, const int32_t* __restrict__ r, int64_t m, int64_t n,
                            unsigned long long* __restrict__ key, unsigned int* __restrict__ bad) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = o[t], b = r[t];
    if (a < 0 || a >= n || b < 0 || b >= n) {
      atomicOr(bad, 1u);
      key[t] = 0;
    } else {
      key[t] = (unsigned long long)a * (unsigned long long)n + (unsigned long long)b;
    }
  }
}

__global__ void k_keys_to_csr(const unsigned long long* __restrict__ key, const int64_t* __restrict__ sum, int64_t m,
                              int64_t n, int32_t* __restrict__ col, int32_t* __restrict__ cnt,
                              int32_t* __restrict__ row_len, unsigned int* __restrict__ bad) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = (int64_t)(key[t] / (unsigned long long)n);
    col[t] = (int32_t)(key[t] % (unsigned long long)n);
    const int64_t c = sum[t];
    if (c < 0 || c > INT32_MAX) atomicOr(bad, 2u);
    cnt[t] = (int32_t)c;
    atomicAdd(row_len + row, 1);
  }
}

__global__ void k_zero_i32(int32_t* p, int64_t n) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) p[t] = 0;
}

__global__ void k_widen_scan_input(const int32_t* __restrict__ in, int64_t* __restrict__ out, int64_t n) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    out[t] = in[t];
}

// row_ptr[0] = 0, row_ptr[1..n] = inclusive sum of len (int64)
static int lengths_to_row_ptr(const int64_t* len, int64_t n, int64_t* row_ptr, cudaStream_t s) {
  PR_CUDA(cudaMemsetAsync(row_ptr, 0, sizeof(int64_t), s));
  if (n == 0) return PR_OK;
  size_t b = 0;
  PR_CUDA(cub::DeviceScan::InclusiveSum(nullptr, b, len, row_ptr + 1, n, s));
  DevBuf<uint8_t> tmp;
  PR_TRY(tmp.alloc(b + 16, s));
  PR_CUDA(cub::DeviceScan::InclusiveSum(tmp.ptr, b, len, row_ptr + 1, n, s));
  return PR_OK;
}

__global__ void k_row_sums(const int64_t* __restrict__ rp, const int32_t* __restrict__ cn, int64_t n,
                           int64_t* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    int64_t s = 0;
    for (int64_t q = rp[i] + lane; q < rp[i + 1]; q += 32) s += cn[q];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[i] = s;
  }
}

__global__ void k_merge_len(const int64_t* __restrict__ ap, const int32_t* __restrict__ ac,
                            const int64_t* __restrict__ bp, const int32_t* __restrict__ bc, int64_t n,
                            int64_t* __restrict__ len);
__global__ void k_merge_rank(const int64_t* __restrict__ ap, const int32_t* __restrict__ ac,
                             const int32_t* __restrict__ an, const int64_t* __restrict__ bp,
                             const int32_t* __restrict__ bc, const int32_t* __restrict__ bn, int64_t n,
                             const int64_t* __restrict__ op, int32_t* __restrict__ oc, int32_t* __restrict__ on,
                             unsigned int* __restrict__ bad);
__global__ void k_row_ptr_from_sorted(const uint32_t* __restrict__ keys, int64_t m, int64_t n,
                                      int64_t* __restrict__ row_ptr);

// Rows of counts with ascending columns.
struct RowsView {
  const int64_t* row_ptr;
  const int32_t* col;
  const int32_t* cnt;
};

// Rows of a and b merged, counts of equal columns added; *bad is set on a count above 2^31 - 1.
static int merge_rows(const RowsView& a, const RowsView& b, int64_t n, CountCsr& c, unsigned int* bad, cudaStream_t s) {
  c.n_rows = n;
  PR_TRY(c.row_ptr.alloc(n + 1, s));
  DevBuf<int64_t> len;
  PR_TRY(len.alloc(n > 0 ? n : 1, s));
  if (n > 0) {
    ::pr::launch_mark(), k_merge_len<<<grid_for(n * 32, 256), 256, 0, s>>>(a.row_ptr, a.col, b.row_ptr, b.col, n, len.ptr);
    PR_CUDA(cudaGetLastError());
  }
  PR_TRY(lengths_to_row_ptr(len.ptr, n, c.row_ptr.ptr, s));
  int64_t nnz = 0;
  PR_CUDA(cudaMemcpyAsync(&nnz, c.row_ptr.ptr + n, 8, cudaMemcpyDeviceToHost, s));
  PR_CUDA(cudaStreamSynchronize(s));
  c.nnz = nnz;
  PR_TRY(c.col.alloc(nnz, s));
  PR_TRY(c.cnt.alloc(nnz, s));
  if (n > 0) {
    ::pr::launch_mark(), k_merge_rank<<<grid_for(n * 32, 256), 256, 0, s>>>(a.row_ptr, a.col, a.cnt, b.row_ptr, b.col, b.cnt,
                                                                            n, c.row_ptr.ptr, c.col.ptr, c.cnt.ptr, bad);
    PR_CUDA(cudaGetLastError());
  }
  return PR_OK;
}

// What an edge list is: bit 0, ids outside [0, n); bit 1, a count outside int32 or negative; bit 2,
// not strictly ascending by (origin, receiver).  The counts are also narrowed to int32.
__global__ void k_edge_form(const int32_t* __restrict__ o, const int32_t* __restrict__ r, const int64_t* __restrict__ c,
                            int64_t m, int64_t n, int32_t* __restrict__ cnt, unsigned int* __restrict__ form) {
  unsigned f = 0;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x) {
    const int32_t a = o[t], b = r[t];
    const int64_t v = c[t];
    if (a < 0 || a >= n || b < 0 || b >= n) f |= 1u;
    if (v < 0 || v > INT32_MAX) f |= 2u;
    if (t > 0 && (o[t - 1] > a || (o[t - 1] == a && r[t - 1] >= b))) f |= 4u;
    cnt[t] = (int32_t)v;
  }
  f = __reduce_or_sync(PR_FULL, f);
  if ((threadIdx.x & 31) == 0 && f) atomicOr(form, f);
}

// Edge lists in any order pooled by a radix sort of (origin, receiver) keys and a sum per key.
static int pool_by_sort(const DevBuf<int32_t>& o, const DevBuf<int32_t>& r, const DevBuf<int64_t>& c, int64_t m, int64_t n,
                        CountCsr& csr, unsigned int* bad, cudaStream_t s) {
  DevBuf<int32_t> row_len;
  DevBuf<int64_t> c_sorted, sums, len64, nruns;
  DevBuf<unsigned long long> key, key_sorted, ukey;
  PR_TRY(csr.row_ptr.alloc(n + 1, s));
  PR_TRY(row_len.alloc(n > 0 ? n : 1, s));
  ::pr::launch_mark(), k_zero_i32<<<grid_for(n, 256), 256, 0, s>>>(row_len.ptr, n);
  int64_t u = 0;
  if (m > 0) {
    PR_TRY(key.alloc(m, s));
    PR_TRY(key_sorted.alloc(m, s));
    PR_TRY(c_sorted.alloc(m, s));
    ::pr::launch_mark(), k_edge_keys<<<grid_for(m, 256), 256, 0, s>>>(o.ptr, r.ptr, m, n, key.ptr, bad);
    PR_CUDA(cudaGetLastError());
    int end_bit = 1;
    while (end_bit < 64 && (((unsigned long long)1 << end_bit) < (unsigned long long)n * (unsigned long long)n)) ++end_bit;
    size_t b = 0;
    PR_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b, key.ptr, key_sorted.ptr, c.ptr, c_sorted.ptr, m, 0, end_bit, s));
    DevBuf<uint8_t> tmp;
    PR_TRY(tmp.alloc(b + 16, s));
    PR_CUDA(cub::DeviceRadixSort::SortPairs(tmp.ptr, b, key.ptr, key_sorted.ptr, c.ptr, c_sorted.ptr, m, 0, end_bit, s));
    PR_TRY(ukey.alloc(m, s));
    PR_TRY(sums.alloc(m, s));
    PR_TRY(nruns.alloc(1, s));
    size_t b2 = 0;
    PR_CUDA(cub::DeviceReduce::ReduceByKey(nullptr, b2, key_sorted.ptr, ukey.ptr, c_sorted.ptr, sums.ptr, nruns.ptr,
                                           cub::Sum(), m, s));
    DevBuf<uint8_t> tmp2;
    PR_TRY(tmp2.alloc(b2 + 16, s));
    PR_CUDA(cub::DeviceReduce::ReduceByKey(tmp2.ptr, b2, key_sorted.ptr, ukey.ptr, c_sorted.ptr, sums.ptr, nruns.ptr,
                                           cub::Sum(), m, s));
    unsigned int hbad = 0;
    PR_CUDA(cudaMemcpyAsync(&u, nruns.ptr, 8, cudaMemcpyDeviceToHost, s));
    PR_CUDA(cudaMemcpyAsync(&hbad, bad, 4, cudaMemcpyDeviceToHost, s));
    PR_CUDA(cudaStreamSynchronize(s));
    PR_ARG(!(hbad & 1u), "edge list holds patch ids outside [0, %lld)", (long long)n);  // before a row is taken from a key
  }
  csr.nnz = u;
  PR_TRY(csr.col.alloc(u, s));
  PR_TRY(csr.cnt.alloc(u, s));
  if (u > 0) {
    ::pr::launch_mark(), k_keys_to_csr<<<grid_for(u, 256), 256, 0, s>>>(ukey.ptr, sums.ptr, u, n, csr.col.ptr, csr.cnt.ptr, row_len.ptr,
                                                  bad);
    PR_CUDA(cudaGetLastError());
  }
  PR_TRY(len64.alloc(n > 0 ? n : 1, s));
  ::pr::launch_mark(), k_widen_scan_input<<<grid_for(n, 256), 256, 0, s>>>(row_len.ptr, len64.ptr, n);
  PR_TRY(lengths_to_row_ptr(len64.ptr, n, csr.row_ptr.ptr, s));
  return PR_OK;
}

// Pooled counts of edge lists.  The lists this library and pool_counts hand out ascend by (origin,
// receiver) without repeats; when every list does (and its counts fit int32), its rows are taken as
// they are and lists are pooled by row merges, in pairs, then pairs of results.  Lists in another order, with
// repeats or with counts outside int32 go through pool_by_sort, which gives the same table.  Two lists of
// 3.3e7 pairs each (96^3 fibers, 500 rays): 2.7 ms of merging against 14 ms of sorting and summing;
// one list of 6.1e7 pairs: 0.3 against 7 ms.
//
// A merge costs about 0.1 ms besides its pairs (launches and a look at its length) and every level of the
// tree reads all pairs again, while the sort costs 0.2 ms and 0.08 ms per 10^6 pairs however many lists
// there are.  So more than two lists are merged while they are at most 16 and hold 250 000 pairs for
// every list and every merge; merged / sorted, with their upload, in ms: 3 lists of 1.8 M pairs 0.84 / 0.90, of
// 0.6 M 0.59 / 0.48; 8 lists of 101 M 34.0 / 37.5, of 15.8 M 5.95 / 6.36, of 4.9 M 2.35 / 2.10; 16 lists of
// 202 M 70.8 / 74.0, of 31.6 M 14.9 / 12.2; 64 lists of 12.8 M 16.6 / 5.9 (the losing merges one after the other).
int counts_from_tables(const int32_t* const* origin, const int32_t* const* receiver, const int64_t* const* count,
                       const int64_t* n_edges, int n_tables, int64_t n, cudaStream_t s, pr_counts** out) {
  PR_ARG(n >= 0 && n < INT32_MAX, "n_patches %lld outside the int32 patch ids", (long long)n);
  PR_ARG(n_tables >= 0, "negative number of tables");
  int64_t m = 0, lists = 0;  // pairs, and lists with pairs
  for (int t = 0; t < n_tables; ++t) {
    PR_ARG(n_edges[t] >= 0, "negative edge count");
    PR_ARG(n_edges[t] == 0 || (origin[t] && receiver[t] && count[t]), "table %d has a NULL array", t);
    m += n_edges[t];
    lists += n_edges[t] > 0;
  }
  const bool merge = lists <= 2 || (lists <= 16 && m >= 250000 * lists * (lists - 1));
  std::unique_ptr<pr_counts> k(new pr_counts());
  cudaGetDevice(&k->device);
  k->csr = std::make_shared<CountCsr>();
  CountCsr& csr = *k->csr;
  csr.n_rows = n;
  DevBuf<int32_t> o, r, cnt;
  DevBuf<int64_t> c;
  DevBuf<unsigned int> bad;
  PR_TRY(bad.alloc(1, s));
  PR_CUDA(cudaMemsetAsync(bad.ptr, 0, 4, s));
  unsigned int form = 0;
  if (m > 0) {
    PR_TRY(o.alloc(m, s));
    PR_TRY(r.alloc(m, s));
    PR_TRY(c.alloc(m, s));
    if (merge) PR_TRY(cnt.alloc(m, s));
    // the tables one after the other into one device edge list
    int64_t at = 0;
    for (int t = 0; t < n_tables; ++t) {
      const int64_t mt = n_edges[t];
      if (mt == 0) continue;
      PR_TRY(copy_from_host(o.ptr + at, origin[t], (size_t)mt * 4, s));
      PR_TRY(copy_from_host(r.ptr + at, receiver[t], (size_t)mt * 4, s));
      PR_TRY(copy_from_host(c.ptr + at, count[t], (size_t)mt * 8, s));
      if (merge) {
        ::pr::launch_mark(), k_edge_form<<<grid_for(mt, 256), 256, 0, s>>>(o.ptr + at, r.ptr + at, c.ptr + at, mt, n,
                                                                          cnt.ptr + at, bad.ptr);
        PR_CUDA(cudaGetLastError());
      }
      at += mt;
    }
    if (merge) {
      PR_CUDA(cudaMemcpyAsync(&form, bad.ptr, 4, cudaMemcpyDeviceToHost, s));
      PR_CUDA(cudaStreamSynchronize(s));
      PR_ARG(!(form & 1u), "edge list holds patch ids outside [0, %lld)", (long long)n);
      PR_CUDA(cudaMemsetAsync(bad.ptr, 0, 4, s));
    }
  }
  unsigned int hbad = 0;
  if (m == 0 || form || !merge) {
    cnt.release();
    PR_TRY(pool_by_sort(o, r, c, m, n, csr, bad.ptr, s));
    PR_CUDA(cudaMemcpyAsync(&hbad, bad.ptr, 4, cudaMemcpyDeviceToHost, s));
    PR_CUDA(cudaStreamSynchronize(s));
    PR_ARG(!(hbad & 2u), "pooled counts must be non-negative and below 2^31");
  } else {
    c.release();
    struct Rows {
      CountCsr own;
      RowsView v;
    };
    std::vector<Rows> level;  // the lists with pairs, then their merges
    for (int64_t a = 0, t = 0; t < n_tables; a += n_edges[t++]) {
      if (n_edges[t] == 0) continue;
      level.emplace_back();
      Rows& q = level.back();
      PR_TRY(q.own.row_ptr.alloc(n + 1, s));
      ::pr::launch_mark(), k_row_ptr_from_sorted<<<grid_for(n + 1, 256), 256, 0, s>>>((const uint32_t*)o.ptr + a, n_edges[t],
                                                                                     n, q.own.row_ptr.ptr);
      PR_CUDA(cudaGetLastError());
      q.v = RowsView{q.own.row_ptr.ptr, r.ptr + a, cnt.ptr + a};
    }
    if (level.size() == 1) {
      csr.row_ptr = std::move(level[0].own.row_ptr);
      csr.nnz = m;
      csr.col = std::move(r);
      csr.cnt = std::move(cnt);
    } else {
      while (level.size() > 1) {
        std::vector<Rows> next;
        for (size_t t = 0; t + 1 < level.size(); t += 2) {
          next.emplace_back();
          Rows& q = next.back();
          PR_TRY(merge_rows(level[t].v, level[t + 1].v, n, q.own, bad.ptr, s));
          q.v = RowsView{q.own.row_ptr.ptr, q.own.col.ptr, q.own.cnt.ptr};
          level[t] = Rows();
          level[t + 1] = Rows();
        }
        if (level.size() & 1) next.push_back(std::move(level.back()));
        level = std::move(next);
      }
      csr = std::move(level[0].own);
      PR_CUDA(cudaMemcpyAsync(&hbad, bad.ptr, 4, cudaMemcpyDeviceToHost, s));
      PR_CUDA(cudaStreamSynchronize(s));
      PR_ARG(!hbad, "pooled counts must be non-negative and below 2^31");
    }
  }
  // rays per origin = row sums of the pooled counts (callers usually pass their own)
  PR_TRY(k->rays.alloc(n > 0 ? n : 1, s));
  ::pr::launch_mark(), k_row_sums<<<grid_for(n * 32, 256), 256, 0, s>>>(csr.row_ptr.ptr, csr.cnt.ptr, n, k->rays.ptr);
  PR_CUDA(cudaGetLastError());
  PR_CUDA(cudaStreamSynchronize(s));
  k->last_stream = s;
  *out = k.release();
  return PR_OK;
}

int counts_from_edges(const int32_t* origin, const int32_t* receiver, const int64_t* count, int64_t m, int64_t n,
                      cudaStream_t s, pr_counts** out) {
  return counts_from_tables(&origin, &receiver, &count, &m, 1, n, s, out);
}

__global__ void k_add_i64(const int64_t* __restrict__ a, const int64_t* __restrict__ b, int64_t n,
                          int64_t* __restrict__ out);

// pool_counts of two device tables (view_factors.py:290-300): rows merged, counts and rays summed.
int counts_merge(const pr_counts* A, const pr_counts* B, cudaStream_t s, pr_counts** out) {
  const CountCsr& a = *A->csr;
  const CountCsr& b = *B->csr;
  PR_ARG(a.n_rows == b.n_rows, "count tables of %lld and %lld patches", (long long)a.n_rows, (long long)b.n_rows);
  const int64_t n = a.n_rows;
  std::unique_ptr<pr_counts> k(new pr_counts());
  cudaGetDevice(&k->device);
  k->csr = std::make_shared<CountCsr>();
  DevBuf<unsigned int> bad;
  PR_TRY(bad.alloc(1, s));
  PR_CUDA(cudaMemsetAsync(bad.ptr, 0, 4, s));
  PR_TRY(merge_rows(RowsView{a.row_ptr.ptr, a.col.ptr, a.cnt.ptr}, RowsView{b.row_ptr.ptr, b.col.ptr, b.cnt.ptr}, n, *k->csr,
                    bad.ptr, s));
  PR_TRY(k->rays.alloc(n > 0 ? n : 1, s));
  if (n > 0) {
    ::pr::launch_mark(), k_add_i64<<<grid_for(n, 256), 256, 0, s>>>(A->rays.ptr, B->rays.ptr, n, k->rays.ptr);
    PR_CUDA(cudaGetLastError());
  }
  unsigned int hb = 0;
  PR_CUDA(cudaMemcpyAsync(&hb, bad.ptr, 4, cudaMemcpyDeviceToHost, s));
  PR_CUDA(cudaStreamSynchronize(s));
  PR_ARG(!hb, "pooled counts exceed 2^31");
  k->rays_traced = A->rays_traced + B->rays_traced;
  k->dda_steps = A->dda_steps + B->dda_steps;
  k->last_stream = s;
  *out = k.release();
  return PR_OK;
}

// ------------------------------------------------------------------ transpose / symmetric pattern

// (row << 32 | count) of every entry of F, in row order
__global__ void k_row_count_values(const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ cnt, int64_t n,
                                   unsigned long long* __restrict__ val) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps)
    for (int64_t q = row_ptr[i] + lane; q < row_ptr[i + 1]; q += 32)
      val[q] = ((unsigned long long)(uint32_t)i << 32) | (unsigned long long)(uint32_t)cnt[q];
}

__global__ void k_split_values(const unsigned long long* __restrict__ val, int64_t m, int32_t* __restrict__ col,
                               int32_t* __restrict__ cnt) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x) {
    col[t] = (int32_t)(val[t] >> 32);
    cnt[t] = (int32_t)(val[t] & 0xffffffffull);
  }
}

// row_ptr[c] = first position of key c in the sorted keys (lower bound), c = 0..n
__global__ void k_row_ptr_from_sorted(const uint32_t* __restrict__ keys, int64_t m, int64_t n,
                                      int64_t* __restrict__ row_ptr) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c <= n; c += (int64_t)gridDim.x * blockDim.x) {
    int64_t lo = 0, hi = m;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if ((int64_t)keys[mid] < c) lo = mid + 1;
      else hi = mid;
    }
    row_ptr[c] = lo;
  }
}

// F^T by one stable radix sort of F's entries (already in row order) keyed on the column
// alone: equal columns keep their row order, so every row of F^T comes out sorted.
int build_transpose(const CountCsr& F, CountCsr& T, cudaStream_t s) {
  const int64_t n = F.n_rows, m = F.nnz;
  T.n_rows = n;
  T.nnz = m;
  PR_TRY(T.row_ptr.alloc(n + 1, s));
  PR_TRY(T.col.alloc(m > 0 ? m : 1, s));
  PR_TRY(T.cnt.alloc(m > 0 ? m : 1, s));
  if (m == 0) {
    PR_CUDA(cudaMemsetAsync(T.row_ptr.ptr, 0, (n + 1) * sizeof(int64_t), s));
    return PR_OK;
  }
  DevBuf<uint32_t> keys_out;
  DevBuf<unsigned long long> val, val_out;
  PR_TRY(keys_out.alloc(m, s));
  PR_TRY(val.alloc(m, s));
  PR_TRY(val_out.alloc(m, s));
  ::pr::launch_mark(), k_row_count_values<<<grid_for(n * 32, 256), 256, 0, s>>>(F.row_ptr.ptr, F.cnt.ptr, n, val.ptr);
  PR_CUDA(cudaGetLastError());
  int bits = 1;
  while (bits < 32 && ((int64_t)1 << bits) < n) ++bits;
  const uint32_t* keys_in = (const uint32_t*)F.col.ptr;
  size_t b = 0;
  PR_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b, keys_in, keys_out.ptr, val.ptr, val_out.ptr, m, 0, bits, s));
  DevBuf<uint8_t> tmp;
  PR_TRY(tmp.alloc(b + 16, s));
  PR_CUDA(cub::DeviceRadixSort::SortPairs(tmp.ptr, b, keys_in, keys_out.ptr, val.ptr, val_out.ptr, m, 0, bits, s));
  ::pr::launch_mark(), k_split_values<<<grid_for(m, 256), 256, 0, s>>>(val_out.ptr, m, T.col.ptr, T.cnt.ptr);
  PR_CUDA(cudaGetLastError());
  ::pr::launch_mark(), k_row_ptr_from_sorted<<<grid_for(n + 1, 256), 256, 0, s>>>(keys_out.ptr, m, n, T.row_ptr.ptr);
  PR_CUDA(cudaGetLastError());
  return PR_OK;
}

// Row offsets of S: len_S(i) = len_F(i) + len_T(i).
__global__ void k_sym_row_ptr(const int64_t* __restrict__ fp, const int64_t* __restrict__ tp, int64_t n,
                              int64_t* __restrict__ sp) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= n; i += (int64_t)gridDim.x * blockDim.x)
    sp[i] = fp[i] + tp[i];
}

// Row i of S: the entries of row i of F (value 0.5 A_i n_ij / R_i) then those of row i of
// F^T (value 0.5 A_j n_ji / R_j); one warp per row, coalesced copies.
__global__ void k_sym_fill(const int64_t* __restrict__ fp, const int32_t* __restrict__ fc,
                           const int32_t* __restrict__ fn, const int64_t* __restrict__ tp,
                           const int32_t* __restrict__ tc, const int32_t* __restrict__ tn,
                           const int64_t* __restrict__ rays, const double* __restrict__ area, int64_t n,
                           const int64_t* __restrict__ sp, uint32_t* __restrict__ cols, double* __restrict__ val) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    const int64_t o = sp[i], fb = fp[i], lf = fp[i + 1] - fb, tb = tp[i], lt = tp[i + 1] - tb;
    for (int64_t e = lane; e < lf + lt; e += 32) {
      const bool f = e < lf;
      const int64_t src = f ? fb + e : tb + (e - lf);
      const uint32_t col = (uint32_t)(f ? fc[src] : tc[src]);
      const int32_t c = f ? fn[src] : tn[src];
      cols[o + e] = col;
      const int64_t owner = f ? i : (int64_t)col;
      val[o + e] = 0.5 * area[owner] * ((double)c / (double)rays[owner]);
    }
  }
}

// Merges of the rows of A and B rank every entry by a search in the other row.  Over the whole row in
// global memory that was nine scattered reads an entry, which L1 serves at about 3 lanes a clock: so a
// row pair of at most kMergeStage columns (all but the longest rows of 1000 rays) is copied to shared
// memory, and a tile's search is narrowed to where its values fall.  OF 128^3 at 500 rays per face (155 M
// merged entries, 2.5 GB): merge 1.87 -> 1.30 ms, lengths 0.76 -> 0.59 ms.
constexpr int kMergeStage = 1280, kMergeThreads = 256;

// Index in b[0 .. nb), ascending, of the first value >= x, for the warp's next values x (ascending over
// the lanes up to `last`); none of b[0 .. from) is that large.  The part of b that the tile's values fall
// in is found first, 64 values at a time, by reads that all lanes share.
__device__ __forceinline__ int tile_rank(const int32_t* b, int nb, int from, int32_t x, int last) {
  const int32_t most = __shfl_sync(0xffffffffu, x, last);
  int lo = from, hi = min(from + 64, nb);
  while (hi < nb && b[hi - 1] < most) hi = min(hi + 64, nb);
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (b[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// A warp's copy of a row, in shared memory.
__device__ __forceinline__ void stage_row(const int32_t* __restrict__ row, int n, int32_t* to, int lane) {
  for (int k = lane; k < n; k += 32) to[k] = row[k];
}

// |a intersect b|, every lane its share of a.
__device__ __forceinline__ int common_columns(const int32_t* __restrict__ a, int na, const int32_t* b, int nb, int lane) {
  int dup = 0, from = 0;
  for (int base = 0; base < na; base += 32) {
    const int k = base + lane, last = min(31, na - 1 - base);
    const int32_t x = k < na ? a[k] : 0;
    const int at = tile_rank(b, nb, from, x, last);
    dup += k < na && at < nb && b[at] == x;
    from = __shfl_sync(0xffffffffu, at, last);
  }
  return dup;
}

// |row i of A  union  row i of B| = |a| + |b| - |a intersect b|, one warp per row.
__global__ void __launch_bounds__(kMergeThreads) k_merge_len(const int64_t* __restrict__ ap, const int32_t* __restrict__ ac,
                                                             const int64_t* __restrict__ bp,
                                                             const int32_t* __restrict__ bc, int64_t n,
                                                             int64_t* __restrict__ len) {
  __shared__ int32_t staged[kMergeThreads / 32][kMergeStage];
  const int lane = threadIdx.x & 31;
  int32_t* sm = staged[threadIdx.x >> 5];
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    const int32_t *a = ac + ap[i], *b = bc + bp[i];
    const int na = (int)(ap[i + 1] - ap[i]), nb = (int)(bp[i + 1] - bp[i]);
    int dup;
    if (nb <= kMergeStage) {
      stage_row(b, nb, sm, lane);
      __syncwarp();
      dup = common_columns(a, na, sm, nb, lane);
      __syncwarp();
    } else {
      dup = common_columns(a, na, b, nb, lane);
    }
    for (int o = 16; o > 0; o >>= 1) dup += __shfl_xor_sync(0xffffffffu, dup, o);
    if (lane == 0) len[i] = (int64_t)na + nb - dup;
  }
}

// One row pooled by ranking: an entry of a lands at k + #(b < a_k) - #(common < a_k), an entry of b
// absent from a at m + #(a < b_m) - #(common < b_m); a common column carries both counts.  The
// common-prefix counts come from warp ballots over tiles of 32.
__device__ __forceinline__ void merge_row(const int32_t* a, const int32_t* __restrict__ an, int na, const int32_t* b,
                                          const int32_t* __restrict__ bn, int nb, int lane, int32_t* __restrict__ oc,
                                          int32_t* __restrict__ on, unsigned int* __restrict__ bad) {
  const unsigned lt = (1u << lane) - 1u;
  int carry = 0, from = 0;
  for (int base = 0; base < na; base += 32) {
    const int k = base + lane, last = min(31, na - 1 - base);
    const bool valid = k < na;
    const int32_t x = valid ? a[k] : 0;
    const int at = tile_rank(b, nb, from, x, last);
    from = __shfl_sync(0xffffffffu, at, last);
    const bool match = valid && at < nb && b[at] == x;
    const unsigned m = __ballot_sync(0xffffffffu, match);
    if (valid) {
      const int pos = k + at - (carry + __popc(m & lt));
      const int64_t c = (int64_t)an[k] + (match ? (int64_t)bn[at] : 0);
      if (c > INT32_MAX) atomicOr(bad, 1u);
      oc[pos] = x;
      on[pos] = (int32_t)c;
    }
    carry += __popc(m);
  }
  carry = from = 0;
  for (int base = 0; base < nb; base += 32) {
    const int k = base + lane, last = min(31, nb - 1 - base);
    const bool valid = k < nb;
    const int32_t y = valid ? b[k] : 0;
    const int at = tile_rank(a, na, from, y, last);
    from = __shfl_sync(0xffffffffu, at, last);
    const bool match = valid && at < na && a[at] == y;
    const unsigned m = __ballot_sync(0xffffffffu, match);
    if (valid && !match) {
      const int pos = k + at - (carry + __popc(m & lt));
      oc[pos] = y;
      on[pos] = bn[k];
    }
    carry += __popc(m);
  }
}

__global__ void __launch_bounds__(kMergeThreads) k_merge_rank(const int64_t* __restrict__ ap, const int32_t* __restrict__ ac,
                                                              const int32_t* __restrict__ an,
                                                              const int64_t* __restrict__ bp,
                                                              const int32_t* __restrict__ bc,
                                                              const int32_t* __restrict__ bn, int64_t n,
                                                              const int64_t* __restrict__ op, int32_t* __restrict__ oc,
                                                              int32_t* __restrict__ on, unsigned int* __restrict__ bad) {
  __shared__ int32_t staged[kMergeThreads / 32][kMergeStage];
  const int lane = threadIdx.x & 31;
  int32_t* sm = staged[threadIdx.x >> 5];
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    const int64_t a0 = ap[i], b0 = bp[i], o = op[i];
    const int na = (int)(ap[i + 1] - a0), nb = (int)(bp[i + 1] - b0);
    if (na <= kMergeStage && nb <= kMergeStage - na) {
      stage_row(ac + a0, na, sm, lane);
      stage_row(bc + b0, nb, sm + na, lane);
      __syncwarp();
      merge_row(sm, an + a0, na, sm + na, bn + b0, nb, lane, oc + o, on + o, bad);
      __syncwarp();
    } else {
      merge_row(ac + a0, an + a0, na, bc + b0, bn + b0, nb, lane, oc + o, on + o, bad);
    }
  }
}

__global__ void k_add_i64(const int64_t* __restrict__ a, const int64_t* __restrict__ b, int64_t n,
                          int64_t* __restrict__ out) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    out[t] = a[t] + b[t];
}

// Row sums of the counts must equal the rays of each origin (exchange.py:68-71).
__global__ void k_accounting(const int64_t* __restrict__ fp, const int32_t* __restrict__ fn,
                             const int64_t* __restrict__ rays, int64_t n, unsigned int* __restrict__ bad) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    int64_t s = 0;
    for (int64_t q = fp[i] + lane; q < fp[i + 1]; q += 32) s += fn[q];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(PR_FULL, s, o);
    if (lane == 0 && s != rays[i]) atomicOr(bad, 1u);
  }
}

// ------------------------------------------------------------------ balancing kernels

struct BalanceScalars {
  double max_f;      // max |f|
  double closure;    // max |d (S d) / A - 1|
  double bad;        // > 0 when S d is not finite and positive, or y left the log range
  int ticket, pad;   // last_block (the dots)
  double dots[20];   // dF_r . dF_c and dF_c . f (k_aa_dots)
};

#define PR_LOG_MAX 709.782712893384  // log(DBL_MAX)
#define PR_LOG_MIN -744.4400719213812  // log(smallest subnormal)

__global__ void k_exp_scale(const double* __restrict__ y, int64_t n, double* __restrict__ d, double* __restrict__ sc) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double v = y[i];
    if (!(v < PR_LOG_MAX && v > PR_LOG_MIN)) sc[2] = 1.0;  // benign race: any writer sets the flag
    d[i] = exp(v);
  }
}

// One balancing evaluation at y (d = e^y given, the vector of the product):  s = S d;
// f_new = y + log s - log A;  dF = f_new - f_old (when dF != nullptr);  closure
// |d s / A - 1|;  max |f_new|.  In multiplicative mode (mult = 1), also
// y_next = y + 0.5 (log A - log(d s)).
struct BalanceEpi {
  double delta;
  const double* area;
  const double* y;
  const double* d;
  double* f;
  double* dF;
  double* sc;
  int mult;
  double* y_next;
  struct Red {
    double mf = 0.0, mc = 0.0;
    bool bad = false;
  };
  __device__ bool skip() const { return false; }
  __device__ void row(int64_t i, double sp, Red& r) const {
    const double Ai = area[i];
    const double s = sp + delta * Ai * d[i];
    if (!(s > 0.0 && isfinite(s))) r.bad = true;
    const double fn = y[i] + log(s) - log(Ai);
    if (dF) dF[i] = fn - f[i];
    f[i] = fn;
    const double rowv = d[i] * s;
    r.mf = fmax(r.mf, fabs(fn));
    r.mc = fmax(r.mc, fabs(rowv / Ai - 1.0));
    if (mult) y_next[i] = y[i] + 0.5 * (log(Ai) - log(rowv));
  }
  __device__ void finish(Red& r) const {
    for (int o = 16; o > 0; o >>= 1) {
      r.mf = fmax(r.mf, __shfl_xor_sync(PR_FULL, r.mf, o));
      r.mc = fmax(r.mc, __shfl_xor_sync(PR_FULL, r.mc, o));
    }
    const bool bad = __any_sync(PR_FULL, r.bad);
    if ((threadIdx.x & 31) == 0) {
      atomic_max_nonneg(sc + 0, r.mf);
      atomic_max_nonneg(sc + 1, r.mc);
      if (bad) sc[2] = 1.0;
    }
  }
};

// One Anderson step of one operator: the update before the product and the dots after it.
struct AAStep {
  double gamma[10];
  int cols, cols_after;  // history columns before and after the step
  int slot;              // ring slot receiving the new differences
  int blocks;            // of the dots, by the operator's own rows: a batch gives it the same sums
  double beta;
  int64_t n;
  const double* y;
  const double* f;
  double *dY, *dF, *y_next, *d, *partial;
  BalanceScalars* sc;
};

// y_next = y - beta f - sum_c gamma_c (dY_c - beta dF_c);  dY_slot = y_next - y;  d = e^y_next, the
// vector of the next product (bad set when y_next leaves the log range).
__device__ __forceinline__ void aa_update(const AAStep& st) {
  const int64_t n = st.n;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double v = st.y[i] - st.beta * st.f[i];
#pragma unroll
    for (int c = 0; c < 10; ++c)
      if (c < st.cols) v -= st.gamma[c] * (st.dY[(int64_t)c * n + i] - st.beta * st.dF[(int64_t)c * n + i]);
    st.dY[(int64_t)st.slot * n + i] = v - st.y[i];
    st.y_next[i] = v;
    if (!(v < PR_LOG_MAX && v > PR_LOG_MIN)) st.sc->bad = 1.0;  // benign race: any writer sets the flag
    st.d[i] = exp(v);
  }
}

// Dots of the history: row `slot` of the Gram matrix (dF_slot . dF_c) and the right-hand side
// (dF_c . f) -> partial[block][2 * 10], summed by the last block into sc->dots.
__device__ __forceinline__ void aa_dots(const AAStep& st) {
  if ((int)blockIdx.x >= st.blocks) return;
  const int64_t n = st.n;
  double acc[20];
#pragma unroll
  for (int k = 0; k < 20; ++k) acc[k] = 0.0;
  const double* vr = st.dF + (int64_t)st.slot * n;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)st.blocks * blockDim.x) {
    const double a = vr[i], fi = st.f[i];
#pragma unroll
    for (int c = 0; c < 10; ++c) {
      if (c < st.cols_after) {
        const double v = st.dF[(int64_t)c * n + i];
        acc[c] = fma(a, v, acc[c]);
        acc[10 + c] = fma(v, fi, acc[10 + c]);
      }
    }
  }
  block_sum_store<20>(acc, st.partial);
  if (!last_block_sums<20>(acc, st.partial, &st.sc->ticket, st.blocks)) return;
#pragma unroll
  for (int k = 0; k < 20; ++k) st.sc->dots[k] = acc[k];
}

__global__ void __launch_bounds__(256) k_aa_update(AAStep st) { aa_update(st); }
__global__ void __launch_bounds__(256) k_aa_dots(AAStep st) { aa_dots(st); }

// The same for several operators, blockIdx.y counting them: one launch, where an operator's own takes
// a few microseconds with most of the GPU idle.
__global__ void __launch_bounds__(256) k_aa_update_batch(const AAStep* __restrict__ steps) { aa_update(steps[blockIdx.y]); }
__global__ void __launch_bounds__(256) k_aa_dots_batch(const AAStep* __restrict__ steps) { aa_dots(steps[blockIdx.y]); }

// Blocks of the dots over n rows: two rows a thread, and few enough partials (17 us a step at 64^3 with 592 blocks, 9 with these).
static int dots_grid(int64_t n) { return (int)std::min<int64_t>(std::max<int64_t>((n + 511) / 512, 1), sm_count() * 2); }

// ------------------------------------------------------------------ products

// y = S v (mode 0), (d / A) S v with v = d x (mode 1), d S v with v = d (x / A) (mode 2).
struct ApplyEpi {
  double delta;
  const double* area;
  const double* d;
  const double* v;
  int mode;
  double* y;
  struct Red {};
  __device__ bool skip() const { return false; }
  __device__ void row(int64_t i, double sp, Red&) const {
    const double s = sp + delta * area[i] * v[i];
    y[i] = mode == 0 ? s : (mode == 1 ? (d[i] / area[i]) * s : d[i] * s);
  }
  __device__ void finish(Red&) const {}
};

__global__ void k_prep_u(const double* __restrict__ d, const double* __restrict__ area, const double* __restrict__ x,
                         int64_t n, int mode, double* __restrict__ u) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    u[i] = mode == 1 ? d[i] * x[i] : d[i] * (x[i] / area[i]);
}

// F x (transposed = 0) or F^T x (transposed = 1, given the transposed CSR) with w = n / R of the origin.
__global__ void __launch_bounds__(256) k_raw_apply(const int64_t* __restrict__ rp, const int32_t* __restrict__ cl,
                                                   const int32_t* __restrict__ cn, const int64_t* __restrict__ rays,
                                                   int64_t n, int transposed, const double* __restrict__ x,
                                                   double* __restrict__ y) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    double acc = 0.0;
    for (int64_t q = rp[i] + lane; q < rp[i + 1]; q += 32) {
      const int32_t j = cl[q];
      const double w = (double)cn[q] / (double)rays[transposed ? j : i];
      acc = fma(w, x[j], acc);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(PR_FULL, acc, o);
    if (lane == 0) y[i] = acc;
  }
}

// Reciprocity defect over the sampled pairs (exchange.py:124-140).
__global__ void __launch_bounds__(256) k_reciprocity(const int64_t* __restrict__ fp, const int32_t* __restrict__ fc,
                                                     const int32_t* __restrict__ fn, const int64_t* __restrict__ rays,
                                                     const double* __restrict__ area, const double* __restrict__ d,
                                                     double delta, int64_t n, double* __restrict__ out) {
  double mdiff = 0.0, mjoint = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    for (int64_t q = fp[i]; q < fp[i + 1]; ++q) {
      const int32_t j = fc[q];
      const double w = (double)fn[q] / (double)rays[i];
      // n_ji by binary search in row j
      int64_t lo = fp[j], hi = fp[j + 1];
      while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (fc[mid] < i) lo = mid + 1;
        else hi = mid;
      }
      const double wr = (lo < fp[j + 1] && fc[lo] == (int32_t)i) ? (double)fn[lo] / (double)rays[j] : 0.0;
      const double Ai = area[i], Aj = area[j];
      double sij = 0.5 * (Ai * w + Aj * wr);
      double sji = 0.5 * (Aj * wr + Ai * w);
      if (j == (int32_t)i) {
        sij += delta * Ai;
        sji += delta * Aj;
      }
      const double jij = Ai * ((d[i] / Ai) * sij * d[j]);
      const double jji = Aj * ((d[j] / Aj) * sji * d[i]);
      mdiff = fmax(mdiff, fabs(jij - jji));
      mjoint = fmax(mjoint, fabs(jij));
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    mdiff = fmax(mdiff, __shfl_xor_sync(PR_FULL, mdiff, o));
    mjoint = fmax(mjoint, __shfl_xor_sync(PR_FULL, mjoint, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomic_max_nonneg(out + 0, mdiff);
    atomic_max_nonneg(out + 1, mjoint);
  }
}

__global__ void k_edges_out(const int64_t* __restrict__ fp, const int32_t* __restrict__ fn,
                            const int64_t* __restrict__ rays, int64_t n, int32_t* __restrict__ origin,
                            double* __restrict__ weight) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    for (int64_t q = fp[i] + lane; q < fp[i + 1]; q += 32) {
      if (origin) origin[q] = (int32_t)i;
      if (weight) weight[q] = (double)fn[q] / (double)rays[i];
    }
  }
}

// ------------------------------------------------------------------ host side

static int spmv_grid(int64_t rows) { return grid_for(rows * 32, 256, sm_count() * 8); }


// Symmetric eigen-decomposition (cyclic Jacobi) of a k x k matrix, k <= 10.
static void jacobi_eig(int k, double* a, double* v, double* w) {
  for (int i = 0; i < k; ++i)
    for (int j = 0; j < k; ++j) v[i * k + j] = i == j ? 1.0 : 0.0;
  for (int sweep = 0; sweep < 64; ++sweep) {
    double off = 0.0;
    for (int i = 0; i < k; ++i)
      for (int j = i + 1; j < k; ++j) off += a[i * k + j] * a[i * k + j];
    if (off < 1e-300) break;
    for (int p = 0; p < k; ++p)
      for (int q = p + 1; q < k; ++q) {
        const double apq = a[p * k + q];
        if (apq == 0.0) continue;
        const double theta = (a[q * k + q] - a[p * k + p]) / (2.0 * apq);
        const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
        const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
        for (int r = 0; r < k; ++r) {
          const double arp = a[r * k + p], arq = a[r * k + q];
          a[r * k + p] = c * arp - s * arq;
          a[r * k + q] = s * arp + c * arq;
        }
        for (int r = 0; r < k; ++r) {
          const double apr = a[p * k + r], aqr = a[q * k + r];
          a[p * k + r] = c * apr - s * aqr;
          a[q * k + r] = s * apr + c * aqr;
        }
        for (int r = 0; r < k; ++r) {
          const double vrp = v[r * k + p], vrq = v[r * k + q];
          v[r * k + p] = c * vrp - s * vrq;
          v[r * k + q] = s * vrp + c * vrq;
        }
      }
  }
  for (int i = 0; i < k; ++i) w[i] = a[i * k + i];
}

// Least-squares gamma = pinv(H) b for the k x k Gram matrix H.
static void solve_gram(int k, const double* H, const double* b, double* gamma) {
  double a[100], v[100], w[10];
  for (int i = 0; i < k * k; ++i) a[i] = H[i];
  jacobi_eig(k, a, v, w);
  double wmax = 0.0;
  for (int i = 0; i < k; ++i) wmax = fmax(wmax, fabs(w[i]));
  const double cut = 10.0 * 2.220446049250313e-16 * wmax;
  for (int i = 0; i < k; ++i) gamma[i] = 0.0;
  for (int e = 0; e < k; ++e) {
    if (!(fabs(w[e]) > cut)) continue;
    double proj = 0.0;
    for (int i = 0; i < k; ++i) proj += v[i * k + e] * b[i];
    proj /= w[e];
    for (int i = 0; i < k; ++i) gamma[i] += v[i * k + e] * proj;
  }
}

struct BalanceWork {
  int64_t n;
  DevBuf<double> y, y2, d, f, dY, dF, partial, part;
  DevBuf<BalanceScalars> own;
  BalanceScalars* sc;  // own, or this operator's place in a batch's array
  double* scalars() const { return (double*)sc; }
};

// One product at y with d = e^y: from y when exp_y, else d is there already (k_aa_update).
static int balance_eval(pr_operator* op, BalanceWork& w, const double* y, bool exp_y, double* dF, int mult, double* y_next,
                        cudaStream_t s) {
  const int64_t n = w.n;
  if (exp_y) {
    PR_CUDA(cudaMemsetAsync(w.sc, 0, sizeof(BalanceScalars), s));
    ::pr::launch_mark(), k_exp_scale<<<grid_for(n, 256), 256, 0, s>>>(y, n, w.d.ptr, w.scalars());
  }
  const BalanceEpi epi{op->delta, op->area.ptr, y, w.d.ptr, w.f.ptr, dF, w.scalars(), mult, y_next};
  int st = PR_OK;
  ::pr::timer_begin(kTimerBalance, s);
  dispatch_mode(op->S.mode, [&](auto u) { st = launch_spmv<decltype(u)::value, double>(op->S, w.d.ptr, w.part.ptr, epi, s); });
  ::pr::timer_end(kTimerBalance, s);
  PR_TRY(st);
  op->spmv_calls++;
  return PR_OK;
}

static int balance_scalars(const BalanceWork& w, BalanceScalars* out, cudaStream_t s) {
  PR_CUDA(cudaMemcpyAsync(out, w.sc, sizeof(BalanceScalars), cudaMemcpyDeviceToHost, s));
  return PR_OK;
}

static int balance_multiplicative(pr_operator* op, BalanceWork& w, double tol, cudaStream_t s);

// One Anderson iteration's host side, the same in balance() and balance_batch(): the step from the
// history, whose columns live in ring slots 0 .. cols - 1 (G and b are indexed by slot).
struct AAHistory {
  double G[10][10] = {{0}}, b[10] = {0};
  int cols = 0, oldest = 0;
  AAStep step(const BalanceWork& w, const double* y, double* y_next) {
    const int M = 10;
    AAStep st{};
    st.cols = cols;
    st.beta = 0.5;
    if (cols > 0) {
      double Hf[100], gamma[10] = {0};
      for (int i = 0; i < cols; ++i)
        for (int j = 0; j < cols; ++j) Hf[i * cols + j] = G[i][j];
      solve_gram(cols, Hf, b, gamma);
      for (int c = 0; c < cols; ++c) st.gamma[c] = gamma[c];
    }
    if (cols < M) {
      st.slot = cols++;
    } else {
      st.slot = oldest;
      oldest = (oldest + 1) % M;
    }
    st.cols_after = cols;
    st.blocks = dots_grid(w.n);
    st.n = w.n;
    st.y = y;
    st.f = w.f.ptr;
    st.dY = w.dY.ptr;
    st.dF = w.dF.ptr;
    st.y_next = y_next;
    st.d = w.d.ptr;
    st.partial = w.partial.ptr;
    st.sc = w.sc;
    return st;
  }
  void take(int slot, const double* dots) {
    for (int c = 0; c < cols; ++c) {
      G[slot][c] = dots[c];
      G[c][slot] = dots[c];
      b[c] = dots[10 + c];
    }
  }
};

static int balance_work(BalanceWork& w, const pr_operator* op, BalanceScalars* sc, cudaStream_t s) {
  const int64_t n = op->n;
  const int M = 10;
  w.n = n;
  PR_TRY(w.y.alloc(n, s));
  PR_TRY(w.y2.alloc(n, s));
  PR_TRY(w.d.alloc(n, s));
  PR_TRY(w.f.alloc(n, s));
  PR_TRY(w.dY.alloc((size_t)M * n, s));
  PR_TRY(w.dF.alloc((size_t)M * n, s));
  PR_TRY(w.part.alloc(stream_part(op->S), s));
  if (!sc) {
    PR_TRY(w.own.alloc(1, s));
    sc = w.own.ptr;
  }
  w.sc = sc;
  PR_TRY(w.partial.alloc((size_t)sm_count() * 2 * 20, s));
  PR_CUDA(cudaMemsetAsync(w.y.ptr, 0, n * sizeof(double), s));
  return PR_OK;
}

static int balance(pr_operator* op, double tol, cudaStream_t s) {
  const int64_t n = op->n;
  BalanceWork w;
  PR_TRY(balance_work(w, op, nullptr, s));
  BalanceScalars sc;
  PR_TRY(balance_eval(op, w, w.y.ptr, true, nullptr, 0, nullptr, s));
  PR_TRY(balance_scalars(w, &sc, s));
  PR_CUDA(cudaStreamSynchronize(s));
  const double eps = 2.220446049250313e-16;
  if (!(sc.bad > 0) && sc.closure <= tol) {  // exchange.py:157-159
    op->method = PR_BALANCE_NONE;
    op->iterations = 0;
    PR_CUDA(cudaMemcpyAsync(op->scale.ptr, w.d.ptr, n * 8, cudaMemcpyDeviceToDevice, s));
    return PR_OK;
  }
  // ---- Anderson acceleration
  bool aa_ok = false;
  int iters = 0;
  if (!(sc.bad > 0)) {
    AAHistory hist;
    double* y = w.y.ptr;
    double* y_next = w.y2.ptr;
    double max_f = sc.max_f;
    const int maxit = 500;  // scipy.optimize.anderson maxiter of exchange.py:177
    for (int it = 0; it < maxit && max_f > tol; ++it) {
      const AAStep st = hist.step(w, y, y_next);
      PR_CUDA(cudaMemsetAsync(w.sc, 0, sizeof(BalanceScalars), s));
      ::pr::launch_mark(), k_aa_update<<<grid_for(n, 256), 256, 0, s>>>(st);
      PR_CUDA(cudaGetLastError());
      PR_TRY(balance_eval(op, w, y_next, false, w.dF.ptr + (size_t)st.slot * n, 0, nullptr, s));
      ++iters;
      std::swap(y, y_next);
      ::pr::launch_mark(), k_aa_dots<<<st.blocks, 256, 0, s>>>(st);
      PR_CUDA(cudaGetLastError());
      PR_TRY(balance_scalars(w, &sc, s));
      PR_CUDA(cudaStreamSynchronize(s));
      if (sc.bad > 0 || !std::isfinite(sc.max_f)) break;
      hist.take(st.slot, sc.dots);
      max_f = sc.max_f;
    }
    if (y != w.y.ptr) PR_CUDA(cudaMemcpyAsync(w.y.ptr, y, n * 8, cudaMemcpyDeviceToDevice, s));
    const double accept = fmin(fmax(10.0 * tol, 10.0 * eps), 1.0e-10);  // exchange.py:180
    if (!(sc.bad > 0) && max_f <= tol && sc.closure <= accept) {
      aa_ok = true;
      // d = exp(y) is in w.d from the last evaluation
      PR_CUDA(cudaMemcpyAsync(op->scale.ptr, w.d.ptr, n * 8, cudaMemcpyDeviceToDevice, s));
      op->method = PR_BALANCE_ANDERSON;
      op->iterations = iters;
    }
  }
  if (aa_ok) return PR_OK;
  return balance_multiplicative(op, w, tol, s);
}

// Damped multiplicative iteration from y = 0 (exchange.py:185-196): the fallback when Anderson
// acceleration does not reach the acceptance tolerance.
static int balance_multiplicative(pr_operator* op, BalanceWork& w, double tol, cudaStream_t s) {
  const int64_t n = op->n;
  BalanceScalars sc;
  PR_CUDA(cudaMemsetAsync(w.y.ptr, 0, n * sizeof(double), s));
  double* y = w.y.ptr;
  double* y_next = w.y2.ptr;
  PR_TRY(balance_eval(op, w, y, true, nullptr, 1, y_next, s));
  PR_TRY(balance_scalars(w, &sc, s));
  PR_CUDA(cudaStreamSynchronize(s));
  for (int it = 1; it <= 20000; ++it) {
    if (sc.bad > 0) break;
    std::swap(y, y_next);
    // closure at the updated y, and the next multiplicative step from the same product
    PR_TRY(balance_eval(op, w, y, true, nullptr, 1, y_next, s));
    PR_TRY(balance_scalars(w, &sc, s));
    PR_CUDA(cudaStreamSynchronize(s));
    if (sc.bad > 0 || !std::isfinite(sc.closure)) break;
    if (sc.closure <= fmin(tol, 1.0e-10)) {
      PR_CUDA(cudaMemcpyAsync(op->scale.ptr, w.d.ptr, n * 8, cudaMemcpyDeviceToDevice, s));
      op->method = PR_BALANCE_MULTIPLICATIVE;
      op->iterations = it;
      return PR_OK;
    }
  }
  set_error("diagonal balancing of the exchange matrix did not converge");
  return PR_ERR_BALANCE;
}

// Anderson balancing of several operators in lockstep (the iteration of balance(), operator by
// operator the same steps): every iteration makes one product of each operator still iterating,
// all in one launch of the batched blocked product, and takes one host round trip for all of
// them.  A sweep of many small operators then fills the GPU with one grid per iteration instead
// of one operator's grid per stream.  Operators that Anderson does not settle fall back to the
// multiplicative iteration one at a time, as in balance().  Every operator must be stored as a word
// stream.
static int balance_batch(const std::vector<pr_operator*>& ops, double tol, cudaStream_t s) {
  const int m = (int)ops.size();
  if (m == 0) return PR_OK;
  const double eps = 2.220446049250313e-16;
  const double accept = fmin(fmax(10.0 * tol, 10.0 * eps), 1.0e-10);  // exchange.py:180
  struct State {
    BalanceWork w;
    AAHistory hist;
    int iters = 0;
    double* y = nullptr;
    double* y_next = nullptr;
    bool active = false, done = false;
    BalanceScalars sc{};
  };
  std::vector<State> st(m);
  DevBuf<BalanceScalars> scalars;
  DevBuf<AAStep> d_steps;
  std::vector<BalanceScalars> h_scalars(m);
  std::vector<AAStep> steps;
  PR_TRY(scalars.alloc(m, s));
  PR_TRY(d_steps.alloc(m, s));
  // the scalars of all operators in one copy; those of operators not listed are not looked at
  auto read_scalars = [&](const std::vector<int>& which) -> int {
    PR_CUDA(cudaMemcpyAsync(h_scalars.data(), scalars.ptr, sizeof(BalanceScalars) * m, cudaMemcpyDeviceToHost, s));
    PR_CUDA(cudaStreamSynchronize(s));
    for (int k : which) st[k].sc = h_scalars[k];
    return PR_OK;
  };
  for (int k = 0; k < m; ++k) {
    PR_TRY(balance_work(st[k].w, ops[k], scalars.ptr + k, s));
    st[k].y = st[k].w.y.ptr;
    st[k].y_next = st[k].w.y2.ptr;
  }
  DevBuf<StreamItem<double, BalanceEpi>> items;
  PR_TRY(items.alloc(m, s));
  // one product of each listed operator at y[k] (differences into dF_out[k] when given), d = e^y[k]
  auto products = [&](const std::vector<int>& which, const std::vector<double*>& ys,
                      const std::vector<double*>& dF_out) -> int {
    std::vector<const SymCsr*> mats;
    std::vector<const double*> xs;
    std::vector<double*> parts;
    std::vector<BalanceEpi> epis;
    for (size_t j = 0; j < which.size(); ++j) {
      pr_operator* op = ops[which[j]];
      BalanceWork& w = st[which[j]].w;
      mats.push_back(&op->S);
      xs.push_back(w.d.ptr);
      parts.push_back(w.part.ptr);
      epis.push_back(BalanceEpi{op->delta, op->area.ptr, ys[j], w.d.ptr, w.f.ptr, dF_out[j], w.scalars(), 0, nullptr});
      op->spmv_calls++;
    }
    PR_CUDA(cudaGetLastError());
    ::pr::timer_begin(kTimerBalance, s);
    const int rc = launch_spmv_batch<double>(mats, xs, parts, epis, items.ptr, s);
    ::pr::timer_end(kTimerBalance, s);
    PR_TRY(rc);
    return PR_OK;
  };
  // y = 0 for every operator
  {
    std::vector<int> all(m);
    std::vector<double*> ys(m), none(m, nullptr);
    PR_CUDA(cudaMemsetAsync(scalars.ptr, 0, sizeof(BalanceScalars) * m, s));
    for (int k = 0; k < m; ++k) {
      all[k] = k;
      ys[k] = st[k].y;
      BalanceWork& w = st[k].w;
      ::pr::launch_mark(), k_exp_scale<<<grid_for(ops[k]->n, 256), 256, 0, s>>>(ys[k], ops[k]->n, w.d.ptr, w.scalars());
    }
    PR_TRY(products(all, ys, none));
    PR_TRY(read_scalars(all));
  }
  for (int k = 0; k < m; ++k) {
    pr_operator* op = ops[k];
    if (!(st[k].sc.bad > 0) && st[k].sc.closure <= tol) {  // exchange.py:157-159
      op->method = PR_BALANCE_NONE;
      op->iterations = 0;
      PR_CUDA(cudaMemcpyAsync(op->scale.ptr, st[k].w.d.ptr, op->n * 8, cudaMemcpyDeviceToDevice, s));
      st[k].done = true;
    } else {
      st[k].active = !(st[k].sc.bad > 0) && st[k].sc.max_f > tol;
    }
  }
  for (int it = 0; it < 500; ++it) {  // scipy.optimize.anderson maxiter of exchange.py:177
    std::vector<int> which;
    std::vector<double*> ys, dFs;
    steps.clear();
    int64_t most = 0;
    for (int k = 0; k < m; ++k) {
      State& q = st[k];
      if (!q.active) continue;
      steps.push_back(q.hist.step(q.w, q.y, q.y_next));
      most = std::max(most, q.w.n);
      which.push_back(k);
      ys.push_back(q.y_next);
      dFs.push_back(q.w.dF.ptr + (size_t)steps.back().slot * q.w.n);
    }
    if (which.empty()) break;
    const int count = (int)which.size();
    PR_CUDA(cudaMemsetAsync(scalars.ptr, 0, sizeof(BalanceScalars) * m, s));
    PR_CUDA(cudaMemcpyAsync(d_steps.ptr, steps.data(), sizeof(AAStep) * count, cudaMemcpyHostToDevice, s));
    for (int c = 0; c < count; c += 65535) {
      const dim3 grid((unsigned)grid_for(most, 256), (unsigned)std::min(count - c, 65535));
      ::pr::launch_mark(), k_aa_update_batch<<<grid, 256, 0, s>>>(d_steps.ptr + c);
    }
    PR_CUDA(cudaGetLastError());
    PR_TRY(products(which, ys, dFs));
    for (int c = 0; c < count; c += 65535) {
      const dim3 grid((unsigned)dots_grid(most), (unsigned)std::min(count - c, 65535));
      ::pr::launch_mark(), k_aa_dots_batch<<<grid, 256, 0, s>>>(d_steps.ptr + c);
    }
    PR_CUDA(cudaGetLastError());
    PR_TRY(read_scalars(which));
    for (int j = 0; j < count; ++j) {
      State& q = st[which[j]];
      ++q.iters;
      std::swap(q.y, q.y_next);
      if (q.sc.bad > 0 || !std::isfinite(q.sc.max_f)) {
        q.active = false;
        continue;
      }
      q.hist.take(steps[j].slot, q.sc.dots);
      if (q.sc.max_f <= tol) q.active = false;
    }
  }
  for (int k = 0; k < m; ++k) {
    State& q = st[k];
    if (q.done) continue;
    pr_operator* op = ops[k];
    if (q.y != q.w.y.ptr) PR_CUDA(cudaMemcpyAsync(q.w.y.ptr, q.y, op->n * 8, cudaMemcpyDeviceToDevice, s));
    if (!(q.sc.bad > 0) && q.sc.max_f <= tol && q.sc.closure <= accept) {
      PR_CUDA(cudaMemcpyAsync(op->scale.ptr, q.w.d.ptr, op->n * 8, cudaMemcpyDeviceToDevice, s));
      op->method = PR_BALANCE_ANDERSON;
      op->iterations = q.iters;
    } else {
      PR_TRY(balance_multiplicative(op, q.w, tol, s));
    }
  }
  return PR_OK;
}

static bool all_equal_i64(const std::vector<int64_t>& v) {
  for (size_t i = 1; i < v.size(); ++i)
    if (v[i] != v[0]) return false;
  return true;
}
static bool all_equal_f64(const std::vector<double>& v) {
  for (size_t i = 1; i < v.size(); ++i)
    if (v[i] != v[0]) return false;
  return true;
}

// S' on the union of the patterns of F and F^T with the pair counts n_ij + n_ji (ranked
// row merge).
static int sym_union(const CountCsr& F, const CountCsr& T, pr_operator* op, cudaStream_t s) {
  SymCsr& S = op->S;
  const int64_t n = F.n_rows;
  DevBuf<int64_t> len;
  DevBuf<unsigned int> bad;
  PR_TRY(len.alloc(n, s));
  PR_TRY(bad.alloc(1, s));
  PR_CUDA(cudaMemsetAsync(bad.ptr, 0, 4, s));
  ::pr::launch_mark(), k_merge_len<<<grid_for(n * 32, 256), 256, 0, s>>>(F.row_ptr.ptr, F.col.ptr, T.row_ptr.ptr,
                                                                         T.col.ptr, n, len.ptr);
  PR_CUDA(cudaGetLastError());
  PR_TRY(lengths_to_row_ptr(len.ptr, n, S.row_ptr.ptr, s));
  int64_t nnz = 0;
  PR_CUDA(cudaMemcpyAsync(&nnz, S.row_ptr.ptr + n, 8, cudaMemcpyDeviceToHost, s));
  PR_CUDA(cudaStreamSynchronize(s));
  S.nnz = nnz;
  PR_TRY(S.cols.alloc(nnz, s));
  PR_TRY(S.cnt.alloc(nnz, s));
  ::pr::launch_mark(), k_merge_rank<<<grid_for(n * 32, 256), 256, 0, s>>>(
      F.row_ptr.ptr, F.col.ptr, F.cnt.ptr, T.row_ptr.ptr, T.col.ptr, T.cnt.ptr, n, S.row_ptr.ptr,
      (int32_t*)S.cols.ptr, S.cnt.ptr, bad.ptr);
  PR_CUDA(cudaGetLastError());
  unsigned int hb = 0;
  PR_CUDA(cudaMemcpyAsync(&hb, bad.ptr, 4, cudaMemcpyDeviceToHost, s));
  PR_CUDA(cudaStreamSynchronize(s));
  PR_ARG(!hb, "pair counts exceed 2^31");
  return PR_OK;
}

// Entries of a row as pieces of at most kStreamCount pairs, which is what a word holds (warp per row).
__device__ __forceinline__ int count_pieces(int32_t c) { return c > 0 ? (c - 1) / (int32_t)kStreamCount + 1 : 1; }

__global__ void k_piece_len(const int64_t* __restrict__ rp, const int32_t* __restrict__ cnt, int64_t n,
                            int64_t* __restrict__ len) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    int64_t s = 0;
    for (int64_t q = rp[i] + lane; q < rp[i + 1]; q += 32) s += count_pieces(cnt[q]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(PR_FULL, s, o);
    if (lane == 0) len[i] = s;
  }
}

__global__ void k_piece_fill(const int64_t* __restrict__ rp, const uint32_t* __restrict__ cols,
                             const int32_t* __restrict__ cnt, int64_t n, const int64_t* __restrict__ to,
                             uint32_t* __restrict__ piece_cols, int32_t* __restrict__ piece_cnt) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    const int64_t b = rp[i], e = rp[i + 1];
    int64_t at = to[i];
    for (int64_t base = b; base < e; base += 32) {
      const int64_t q = base + lane;
      int32_t left = q < e ? cnt[q] : 0;
      const int k = q < e ? count_pieces(left) : 0;
      int incl = k;
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(PR_FULL, incl, o);
        if (lane >= o) incl += v;
      }
      int64_t p = at + incl - k;
      for (int h = 0; h < k; ++h, ++p) {
        const int32_t c = min(left, (int32_t)kStreamCount);
        piece_cols[p] = cols[q];
        piece_cnt[p] = c;
        left -= c;
      }
      at += __shfl_sync(PR_FULL, incl, 31);
    }
  }
}

// Splits the entries whose counts do not fit a word, each into several of the same column (S.nnz stays the
// pairs of the union).  Where the words would outnumber the entries by more than two to one, and so take
// more bytes than columns and counts, S stays as it is, read by a warp per row (kCounts).  81 920 rays a
// patch: 64^3 foam, 389 M entries, 319 us a binary64 product from words and 744 by a warp per row;
// 40^3 fibers, 63.5 M, 60 and 107 us; 32^3 foam, 34 M, 40 and 65 us.
static int split_counts(SymCsr& S, cudaStream_t s) {
  const int64_t n = S.n_rows;
  DevBuf<int64_t> len, to;
  PR_TRY(len.alloc(n, s));
  PR_TRY(to.alloc(n + 1, s));
  ::pr::launch_mark(), k_piece_len<<<grid_for(n * 32, 256), 256, 0, s>>>(S.row_ptr.ptr, S.cnt.ptr, n, len.ptr);
  PR_CUDA(cudaGetLastError());
  PR_TRY(lengths_to_row_ptr(len.ptr, n, to.ptr, s));
  int64_t pieces = 0;
  PR_CUDA(cudaMemcpyAsync(&pieces, to.ptr + n, 8, cudaMemcpyDeviceToHost, s));
  PR_CUDA(cudaStreamSynchronize(s));
  if (pieces > 2 * S.nnz) S.mode = kCounts;
  if (pieces == S.nnz || S.mode == kCounts) return PR_OK;
  DevBuf<uint32_t> cols;
  DevBuf<int32_t> cnt;
  PR_TRY(cols.alloc(pieces, s));
  PR_TRY(cnt.alloc(pieces, s));
  ::pr::launch_mark(), k_piece_fill<<<grid_for(n * 32, 256), 256, 0, s>>>(S.row_ptr.ptr, S.cols.ptr, S.cnt.ptr, n, to.ptr,
                                                                          cols.ptr, cnt.ptr);
  PR_CUDA(cudaGetLastError());
  S.row_ptr = std::move(to);
  S.cols = std::move(cols);
  S.cnt = std::move(cnt);
  return PR_OK;
}

// CTA row boundaries of a word stream: boundary c is the first row r whose cost row_ptr[r] + r w
// reaches c / C of the total; w is what a row costs besides its entries.
__global__ void k_cta_rows(const int64_t* __restrict__ rp, int64_t n, int ctas, double w, int64_t* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > ctas) return;
  if (c == 0 || c == ctas) {
    out[c] = c == 0 ? 0 : n;
    return;
  }
  const double target = (double)c / (double)ctas * ((double)rp[n] + (double)n * w);
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if ((double)rp[mid] + (double)mid * w < target) lo = mid + 1;
    else hi = mid;
  }
  out[c] = lo;
}

// first[b n + i] = first entry of row i with column >= b W, relative to row_ptr[i] (b = 0 .. nb - 1);
// a row's columns ascend.
__global__ void k_block_first(const int64_t* __restrict__ rp, const uint32_t* __restrict__ cols, int64_t n, int nb,
                              int W, int32_t* __restrict__ first) {
  const int64_t total = n * (int64_t)nb;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t % n;
    const uint64_t key = (uint64_t)(t / n) * (uint64_t)W;
    int64_t lo = rp[i], hi = rp[i + 1];
    const int64_t base = lo;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (cols[mid] < key) lo = mid + 1;
      else hi = mid;
    }
    first[t] = (int32_t)(lo - base);
  }
}

// Quads of a row's segment in one column block: whole quads, at least one.
__device__ __forceinline__ int seg_quads(int len) { return len > 4 ? (len + 3) >> 2 : 1; }

// len[g n + i] = words of row i in column group g, of one block each.
__global__ void k_group_len(const int64_t* __restrict__ rp, const int32_t* __restrict__ first, int64_t n, int groups,
                            int64_t* __restrict__ len) {
  const int64_t total = n * (int64_t)groups;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < total; v += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = v % n;
    len[v] = 4 * seg_quads((v + n < total ? first[v + n] : (int32_t)(rp[i + 1] - rp[i])) - first[v]);
  }
}

// CTA boundaries of a word stream in groups: those of group g, group_cta[g] .. group_cta[g + 1] - 1,
// share its cost (words and w per row) evenly; cum[v] = words before row v of all groups' rows.
__global__ void k_group_rows(const int64_t* __restrict__ cum, const int32_t* __restrict__ group_cta, int64_t n,
                             int groups, double w, int64_t* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > group_cta[groups]) return;
  if (c == group_cta[groups]) {
    out[c] = groups * n;
    return;
  }
  int g = 0;
  while (group_cta[g + 1] <= c) ++g;
  const int64_t v0 = g * n, e0 = cum[v0];
  const double all = (double)(cum[v0 + n] - e0) + (double)n * w;
  const double target = (double)(c - group_cta[g]) / (double)(group_cta[g + 1] - group_cta[g]) * all;
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if ((double)(cum[v0 + mid] - e0) + (double)mid * w < target) lo = mid + 1;
    else hi = mid;
  }
  out[c] = v0 + lo;
}

// One block per (CTA, column block): off[b n + i] = the row's first quad within the stage, q = quads
// per lane, and the stage's size in quads.
__global__ void __launch_bounds__(256) k_stream_stage(const int64_t* __restrict__ rp, const int32_t* __restrict__ first,
                                                      const int64_t* __restrict__ cta_row, int64_t n, int nb,
                                                      int blocks, int unroll, int32_t* __restrict__ off, int32_t* __restrict__ q,
                                                      int64_t* __restrict__ size) {
  __shared__ int warp_sum[8];
  const int cta = blockIdx.x / nb, g = (int)(cta_row[cta] / n), b = g * nb + blockIdx.x % nb;
  const int64_t r0 = cta_row[cta] - g * n, r1 = cta_row[cta + 1] - g * n;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int carry = 0;
  for (int64_t base = r0; base < r1; base += 256) {
    const int64_t i = base + threadIdx.x;
    int len = 0;
    if (i < r1) {
      const int lo = first[(int64_t)b * n + i];
      const int hi = b + 1 < blocks ? first[(int64_t)(b + 1) * n + i] : (int)(rp[i + 1] - rp[i]);
      len = seg_quads(hi - lo);
    }
    int incl = len;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(PR_FULL, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) warp_sum[wid] = incl;
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < 8; ++w) {
      if (w < wid) before += warp_sum[w];
      total += warp_sum[w];
    }
    if (i < r1) off[(int64_t)b * n + i] = carry + before + incl - len;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const int unit = kStreamThreads * unroll, per = (carry + unit - 1) / unit * unroll;
    q[blockIdx.x] = per;
    size[blockIdx.x] = (int64_t)per * kStreamThreads;
  }
}

// start[l] of every lane of a stage (one block per stage): rows whose first quad lies before the
// lane's run, minus one.
__global__ void __launch_bounds__(256) k_stream_start(const int32_t* __restrict__ off, const int32_t* __restrict__ q,
                                                      const int64_t* __restrict__ cta_row, int64_t n, int nb,
                                                      int16_t* __restrict__ start) {
  const int cta = blockIdx.x / nb, g = (int)(cta_row[cta] / n), b = g * nb + blockIdx.x % nb;
  const int64_t r0 = cta_row[cta] - g * n, r1 = cta_row[cta + 1] - g * n;
  const int32_t* o = off + (int64_t)b * n;
  for (int l = threadIdx.x; l < kStreamThreads; l += blockDim.x) {
    const int key = l * q[blockIdx.x];
    int64_t lo = r0, hi = r1;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (o[mid] < key) lo = mid + 1;
      else hi = mid;
    }
    start[(int64_t)blockIdx.x * kStreamThreads + l] = (int16_t)(lo - r0 - 1);
  }
}

__global__ void k_stream_clear(uint4* __restrict__ quads, int64_t n, uint32_t word) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    quads[t] = make_uint4(word, word, word, word);
}

// The words of every row, one warp per row (its CTAs by binary search over cta_row).  The entries of
// the row's segment in block b fill the segment's slots (word e % 4 of quad off + e / 4 of the stage)
// 32 at a time, in an order that keeps the products' gathers apart: a half warp reads 16 eight-byte
// values of x at once from 16 pairs of banks, at quad l per + t of lane l, so slot e of quad k of lane
// l wants a place = l + 4 k + e modulo 16 (4 per + 1 is odd, so 16 lanes want 16 different places).
// Along the slots of a lane every 16 in a row want each place once: the first entry with a place takes
// its slot in the first 16, the second in the second 16, the others the slots left.
// What bounds it is the instructions around these exchanges: 2.2 ms for OF 128^3 at 500 rays per face
// (4.0 with lists of the slots of each place), where column order takes 0.9 but lengthens every
// product after it: 225 us against 206 at 500 rays, 335 against 297 at 1000, TL 160^3 279 against 248.
__global__ void __launch_bounds__(256) k_stream_fill(const int64_t* __restrict__ rp, const uint32_t* __restrict__ cols,
                                                     const int32_t* __restrict__ cnt, const int32_t* __restrict__ first,
                                                     const int32_t* __restrict__ off, const int32_t* __restrict__ q,
                                                     const int64_t* __restrict__ stage_base,
                                                     const int64_t* __restrict__ cta_row, int ctas, int64_t n, int nb,
                                                     int blocks, int W, uint32_t* __restrict__ words) {
  __shared__ uint32_t placed[8][32], others[8][32];
  const uint32_t none = (uint32_t)W << (32 - kStreamColBits);  // place W, n = 0
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + warp; i < n; i += warps) {
    const int64_t rb = rp[i];
    const int len = (int)(rp[i + 1] - rb);
    for (int b0 = 0; b0 < blocks; b0 += 32) {
      // lane k holds the segment of block b0 + k: its entries, first quad and stage
      int my_first = len, my_off = 0, my_per = 1;
      int64_t my_at = 0;
      if (b0 + lane < blocks) {
        const int g = (b0 + lane) / nb;
        const int64_t v = g * n + i;
        int lo = 0, hi = ctas - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (cta_row[mid] <= v) lo = mid;
          else hi = mid - 1;
        }
        const int64_t stage = (int64_t)lo * nb + (b0 + lane - g * nb), k = (int64_t)(b0 + lane) * n + i;
        my_first = first[k];
        my_off = off[k];
        my_per = q[stage];
        my_at = stage_base[stage];
      }
      const int after = b0 + 32 < blocks ? first[(int64_t)(b0 + 32) * n + i] : len;
      const int last = min(32, blocks - b0);
      for (int k = 0; k < last; ++k) {
        const int e0 = __shfl_sync(PR_FULL, my_first, k), up = __shfl_sync(PR_FULL, my_first, (k + 1) & 31);
        const int count = (k < 31 ? up : after) - e0, o = __shfl_sync(PR_FULL, my_off, k);
        const int per = __shfl_sync(PR_FULL, my_per, k);
        const int64_t at = __shfl_sync(PR_FULL, my_at, k);
        const float inv = 1.0f / (float)per;
        const uint32_t c0 = (uint32_t)(b0 + k) * (uint32_t)W;
        const int m = 4 * seg_quads(count);
        for (int base = 0; base < m; base += 32) {
          const int e = base + lane;
          uint32_t w = 0;
          int bank = 16 + lane;  // no entry: like no other
          if (e < count) {
            const int64_t j = rb + e0 + e;
            const uint32_t col = stream_place(cols[j] - c0);
            bank = (int)(col & 15u);
            w = (col << (32 - kStreamColBits)) | (uint32_t)cnt[j];
          }
          const int quad = o + (e >> 2);
          int l = (int)(((float)quad + 0.5f) * inv), t = quad - l * per;  // quad / per, at most one off
          if (t < 0) {
            --l;
            t += per;
          } else if (t >= per) {
            ++l;
            t -= per;
          }
          const int want = l + 4 * quad + (e & 3);
          const int want0 = __shfl_sync(PR_FULL, want, 0), want1 = __shfl_sync(PR_FULL, want, 16);
          const int rank = __popc(__match_any_sync(PR_FULL, bank) & lt);
          const int to = rank == 0 ? (bank - want0) & 15 : 16 + ((bank - want1) & 15);
          const bool fits = e < count && rank < 2 && base + to < m;
          const unsigned rest = __ballot_sync(PR_FULL, e < count && !fits);
          const unsigned taken = __reduce_or_sync(PR_FULL, fits ? 1u << to : 0u);
          if (fits) placed[warp][to] = w;
          else if (e < count) others[warp][__popc(rest & lt)] = w;
          __syncwarp();
          if (e < m) {
            uint32_t v = none;
            const int r = __popc(~taken & lt);
            if ((taken >> lane) & 1u) v = placed[warp][lane];
            else if (r < __popc(rest)) v = others[warp][r];
            words[4 * (at + (int64_t)t * kStreamThreads + l) + (e & 3)] = v | (e == 0 ? kStreamRow : 0u);
          }
          __syncwarp();
        }
      }
    }
  }
}

// The word stream of a union-stored S' in place of its columns and counts, unless its rows are too short
// for it (S.mode is then kCounts).
static int build_stream(SymCsr& S, cudaStream_t s) {
  SymStream& T = S.stream;
  const int64_t n = S.n_rows;
  const int64_t sms = sm_count();
  std::vector<int64_t> h;
  DevBuf<int32_t> first, off;
  auto rows_cap = [&](int64_t ctas) -> int {  // after the kernel that wrote cta_row
    h.resize(ctas + 1);
    PR_CUDA(cudaMemcpyAsync(h.data(), T.cta_row.ptr, (ctas + 1) * 8, cudaMemcpyDeviceToHost, s));
    PR_CUDA(cudaStreamSynchronize(s));
    int64_t cap = 1;
    for (int64_t c = 0; c < ctas; ++c) cap = std::max(cap, h[c + 1] - h[c]);
    T.ctas = (int)ctas;
    T.rows_cap = (int)std::min<int64_t>(cap, INT32_MAX);
    return PR_OK;
  };
  // Column groups of one block each, while one wave of CTAs holds the row sums of all groups.  A CTA
  // then copies one block of x instead of all of x, and has one stage instead of one per block, which
  // is what small operators spent their time on; the second kernel costs 3 to 4 us.  Product and
  // balancing step, binary64: 4 M entries on 44 676 patches 25.5 -> 17.5 us, 7.9 M on 35 882
  // 26.1 -> 19.4, 32 M on 62 034 51.5 -> 42.3.  Beyond 2^20 sums (110 000 patches) a wave no longer
  // holds them.
  T.nb = 1;
  T.groups = (int)std::min<int64_t>((n + kStreamGroup - 1) / kStreamGroup, INT32_MAX);
  bool grouped = T.groups > 1 && T.groups * n <= kStreamPartMax;
  if (grouped) {
    T.W = (int)(((n + T.groups - 1) / T.groups + 63) / 64 * 64);
    const int64_t room = ((int64_t)kStreamSmemMax - (int64_t)(T.W + kStreamPad) * 8 - 16) / 8 - kStreamThreads;
    DevBuf<int64_t> len, cum;
    DevBuf<int32_t> group_cta;
    PR_TRY(first.alloc((size_t)T.groups * n, s));
    PR_TRY(len.alloc((size_t)T.groups * n, s));
    PR_TRY(cum.alloc((size_t)T.groups * n + 1, s));
    PR_TRY(group_cta.alloc(T.groups + 1, s));
    ::pr::launch_mark(), k_block_first<<<grid_for(n * T.groups, 256), 256, 0, s>>>(S.row_ptr.ptr, S.cols.ptr, n, T.groups,
                                                                                  T.W, first.ptr);
    ::pr::launch_mark(), k_group_len<<<grid_for(n * T.groups, 256), 256, 0, s>>>(S.row_ptr.ptr, first.ptr, n, T.groups,
                                                                                len.ptr);
    PR_CUDA(cudaGetLastError());
    PR_TRY(lengths_to_row_ptr(len.ptr, n * T.groups, cum.ptr, s));
    std::vector<int64_t> ends(T.groups + 1);
    PR_CUDA(cudaMemcpy2DAsync(ends.data(), 8, cum.ptr, n * 8, 8, T.groups + 1, cudaMemcpyDeviceToHost, s));
    PR_CUDA(cudaStreamSynchronize(s));
    // w: what a row costs besides its quads, in entries; more while a CTA of rows with few entries holds
    // more of them than fit
    for (double w = 6.0; w < 2000.0; w *= 1.5) {
      // the CTAs one by one to the group with the most to do per CTA
      std::vector<int32_t> at(T.groups + 1, 0), per(T.groups, 1);
      auto load = [&](int g) { return ((double)(ends[g + 1] - ends[g]) + (double)n * w) / per[g]; };
      for (int64_t c = T.groups; c < sms; ++c) {
        int most = 0;
        for (int g = 1; g < T.groups; ++g)
          if (load(g) > load(most)) most = g;
        ++per[most];
      }
      for (int g = 0; g < T.groups; ++g) at[g + 1] = at[g] + per[g];
      const int ctas = at[T.groups];
      PR_TRY(T.cta_row.alloc(ctas + 1, s));
      PR_CUDA(cudaMemcpyAsync(group_cta.ptr, at.data(), (T.groups + 1) * 4, cudaMemcpyHostToDevice, s));
      ::pr::launch_mark(), k_group_rows<<<grid_for(ctas + 1, 256), 256, 0, s>>>(cum.ptr, group_cta.ptr, n, T.groups, w,
                                                                               T.cta_row.ptr);
      PR_CUDA(cudaGetLastError());
      PR_TRY(rows_cap(ctas));
      if (T.rows_cap <= room) break;
    }
    grouped = T.rows_cap <= room && T.rows_cap < (1 << 15);  // `start` holds 16 bits
  }
  if (!grouped) {
    // CTAs: a multiple of the SMs, with about kRows rows each at most, so that their sums leave room
    // for two blocks of x.  Where some hold far more rows than the average there are up to 8 an SM, and
    // then a row weighs more, which ends with n / ctas rows in each.  Half of kRows would make a second wave
    // of 128^3 foam and 160^3 layers (205 -> 250 us and 247 -> 302 us a product); 4000 would spare 170^3 foam its
    // second one (360 -> 299 us) at narrower blocks everywhere else, and has not been taken further.
    const int64_t kRows = 3000, kRowsMax = 6000, kPerSm = 8;
    T.groups = 1;
    // w: what a row costs besides its entries: in every column block about four entries' time for the
    // padding to whole quads and the row sum
    double w = 4.0 * ((double)n / 11000.0 + 1.0);
    for (int64_t k = (n + sms * kRows - 1) / (sms * kRows);;) {
      const int64_t ctas = std::min<int64_t>(sms * k, n);
      PR_TRY(T.cta_row.alloc(ctas + 1, s));
      ::pr::launch_mark(), k_cta_rows<<<grid_for(ctas + 1, 256), 256, 0, s>>>(S.row_ptr.ptr, n, (int)ctas, w, T.cta_row.ptr);
      PR_CUDA(cudaGetLastError());
      PR_TRY(rows_cap(ctas));
      if (T.rows_cap <= kRowsMax || ctas == n) break;
      if (2 * k <= kPerSm) k *= 2;
      else w *= 4.0;
    }
    const int64_t room = (((int64_t)kStreamSmemMax - (int64_t)stream_sums<double>(T.rows_cap, 2)) / 16 - kStreamPad) / 64 * 64;
    T.W = (int)std::min<int64_t>({room, ((int64_t)1 << kStreamColBits) - 64, (n + 63) / 64 * 64});
    T.nb = (int)((n + T.W - 1) / T.W);
    // A row costs a quad and a row sum in every block, so a stream's bytes (at least 16 n nb) and time grow
    // with n^2 while its entries grow with n.  Where there are more than 36 blocks, and more than 2 for every
    // 5 entries of a row, columns and counts stay as they are, read by a warp per row: 8 bytes an entry
    // whatever n.  us a balancing product, stream / warp per row (in brackets binary32), at entries per row:
    //   128^3 foam, 257 094 patches, 23 blocks: 13: 84 / 110 (71 / 59), 91: 99 / 145 (79 / 129), 605: 204 / 548
    //   150^3, 356 002, 33: 25: 130 / 157 (106 / 89), 91: 142 / 195 (114 / 178)
    //   170^3, 458 360, 39: 25: 266 / 198 (216 / 119), 92: 271 / 245 (220 / 227), 338: 360 / 604 (284 / 618)
    //   200^3, 637 508, 57: 92: 411 / 335 (336 / 316), 177: 455 / 499 (366 / 526), 341: 579 / 860 (424 / 878)
    //   256^3, 1 050 374, 98: 48: 1015 / 473 (841 / 360), 179: 1045 / 825 (838 / 880), 346: 1188 / 1464 (931 / 1472)
    if (T.nb > 36 && 5 * T.nb > 2 * (S.nnz / n)) {
      T = SymStream();
      S.mode = kCounts;
      return PR_OK;
    }
    PR_TRY(first.alloc((size_t)T.nb * n, s));
    ::pr::launch_mark(), k_block_first<<<grid_for(n * T.nb, 256), 256, 0, s>>>(S.row_ptr.ptr, S.cols.ptr, n, T.nb, T.W,
                                                                              first.ptr);
    PR_CUDA(cudaGetLastError());
  }
  const int blocks = T.groups * T.nb;
  const int64_t stages = (int64_t)T.ctas * T.nb;
  // quads in flight per lane: as many as keep the padding of a lane's run (half of them on average)
  // small against the run.  Two from runs of 2 on: 96^3 foam at 125 rays (64 us a product) and 128^3 at 64 (98) 4 %
  // slower; one always: 128^3 at 500 rays 3 us faster in binary64 (203), 6 slower in binary32 (149).
  const double run = ((double)S.nnz / 4.0 + 0.5 * (double)n * blocks) / (double)(stages * kStreamThreads);
  T.unroll = run >= 4.0 ? 2 : 1;
  DevBuf<int64_t> size;
  PR_TRY(off.alloc((size_t)blocks * n, s));
  PR_TRY(size.alloc(stages, s));
  PR_TRY(T.q.alloc(stages, s));
  PR_TRY(T.base.alloc(stages + 1, s));
  PR_TRY(T.start.alloc((size_t)stages * kStreamThreads, s));
  ::pr::launch_mark(), k_stream_stage<<<(int)stages, 256, 0, s>>>(S.row_ptr.ptr, first.ptr, T.cta_row.ptr, n, T.nb, blocks, T.unroll,
                                                                  off.ptr, T.q.ptr, size.ptr);
  ::pr::launch_mark(), k_stream_start<<<(int)stages, 256, 0, s>>>(off.ptr, T.q.ptr, T.cta_row.ptr, n, T.nb, T.start.ptr);
  PR_CUDA(cudaGetLastError());
  PR_TRY(lengths_to_row_ptr(size.ptr, stages, T.base.ptr, s));
  int64_t quads = 0;
  PR_CUDA(cudaMemcpyAsync(&quads, T.base.ptr + stages, 8, cudaMemcpyDeviceToHost, s));
  PR_CUDA(cudaStreamSynchronize(s));
  PR_TRY(T.quads.alloc(quads + (int64_t)T.unroll * kStreamThreads, s));
  const uint32_t none = (uint32_t)T.W << (32 - kStreamColBits);
  ::pr::launch_mark(), k_stream_clear<<<grid_for((int64_t)T.quads.n, 256), 256, 0, s>>>(T.quads.ptr, (int64_t)T.quads.n, none);
  ::pr::launch_mark(), k_stream_fill<<<grid_for(n * 32, 256), 256, 0, s>>>(
      S.row_ptr.ptr, S.cols.ptr, S.cnt.ptr, first.ptr, off.ptr, T.q.ptr, T.base.ptr, T.cta_row.ptr, T.ctas, n, T.nb, blocks, T.W,
      (uint32_t*)T.quads.ptr);
  PR_CUDA(cudaGetLastError());
  S.cols.release();
  S.cnt.release();
  return PR_OK;
}

int apply(const pr_operator* op, int which, const double* x_dev, double* y_dev, cudaStream_t s);

// Everything of operator_create before the balancing: accounting, transpose, S', column blocks.
static int operator_assemble(const pr_counts* k, const int64_t* rays, const double* area, double delta,
                             cudaStream_t s, std::unique_ptr<pr_operator>& op) {
  const int64_t n = k->csr->n_rows;
  op.reset(new pr_operator());
  cudaGetDevice(&op->device);
  op->n = n;
  op->F = k->csr;
  op->delta = delta;
  op->last_stream = s;
  PR_TRY(op->rays.alloc(n > 0 ? n : 1, s));
  PR_TRY(op->area.alloc(n > 0 ? n : 1, s));
  PR_TRY(op->scale.alloc(n > 0 ? n : 1, s));
  std::vector<int64_t> h_rays(n);
  std::vector<double> h_area(n);
  if (n > 0) {
    PR_CUDA(cudaMemcpyAsync(h_rays.data(), rays, n * 8, cudaMemcpyDefault, s));
    PR_CUDA(cudaMemcpyAsync(h_area.data(), area, n * 8, cudaMemcpyDefault, s));
    PR_CUDA(cudaStreamSynchronize(s));
    PR_CUDA(cudaMemcpyAsync(op->rays.ptr, h_rays.data(), n * 8, cudaMemcpyHostToDevice, s));
    PR_CUDA(cudaMemcpyAsync(op->area.ptr, h_area.data(), n * 8, cudaMemcpyHostToDevice, s));
  }
  const CountCsr& F = *op->F;
  // accounting (exchange.py:68-71)
  {
    DevBuf<unsigned int> bad;
    PR_TRY(bad.alloc(1, s));
    PR_CUDA(cudaMemsetAsync(bad.ptr, 0, 4, s));
    ::pr::launch_mark(), k_accounting<<<spmv_grid(n), 256, 0, s>>>(F.row_ptr.ptr, F.cnt.ptr, op->rays.ptr, n, bad.ptr);
    PR_CUDA(cudaGetLastError());
    unsigned int hb = 0;
    PR_CUDA(cudaMemcpyAsync(&hb, bad.ptr, 4, cudaMemcpyDeviceToHost, s));
    PR_CUDA(cudaStreamSynchronize(s));
    if (hb) {
      set_error("first-hit counts do not account for every emitted ray");
      return PR_ERR_ACCOUNTING;
    }
  }
  // symmetric matrix: row i = row i of F followed by row i of F^T
  {
    auto T = std::make_shared<CountCsr>();
    PR_TRY(build_transpose(F, *T, s));
    SymCsr& S = op->S;
    S.n_rows = n;
    PR_TRY(S.row_ptr.alloc(n + 1, s));
    const bool uniform = n > 0 && all_equal_i64(h_rays) && all_equal_f64(h_area) && h_rays[0] > 0;
    int64_t max_rays = 0;
    for (int64_t r : h_rays) max_rays = std::max(max_rays, r);
    if (uniform) {
      S.factor = 0.5 * h_area[0] / (double)h_rays[0];
      S.mode = kStream;
    } else {
      S.mode = kValues;
      S.nnz = F.nnz + T->nnz;
      PR_TRY(S.cols.alloc(S.nnz > 0 ? S.nnz : 1, s));
      PR_TRY(S.val.alloc(S.nnz > 0 ? S.nnz : 1, s));
    }
    if (n > 0 && S.mode == kValues) {
      ::pr::launch_mark(), k_sym_row_ptr<<<grid_for(n + 1, 256), 256, 0, s>>>(F.row_ptr.ptr, T->row_ptr.ptr, n,
                                                                              S.row_ptr.ptr);
      PR_CUDA(cudaGetLastError());
      ::pr::launch_mark(), k_sym_fill<<<grid_for(n * 32, 256), 256, 0, s>>>(
          F.row_ptr.ptr, F.col.ptr, F.cnt.ptr, T->row_ptr.ptr, T->col.ptr, T->cnt.ptr, op->rays.ptr, op->area.ptr, n,
          S.row_ptr.ptr, S.cols.ptr, S.val.ptr);
      PR_CUDA(cudaGetLastError());
    } else if (n > 0) {
      // equal areas and ray counts: S'_ij = factor (n_ij + n_ji) on the union of the patterns
      PR_TRY(sym_union(F, *T, op.get(), s));
      if (2 * max_rays > (int64_t)kStreamCount) PR_TRY(split_counts(op->S, s));  // n_ij + n_ji <= 2 R
      if (S.mode == kStream) PR_TRY(build_stream(op->S, s));
    }
    op->FT = T;  // kept for raw_rmatvec
  }
  return PR_OK;
}

// Row closure of F_p (exchange.py:78-80) after the balancing.
static int operator_closure(pr_operator* op, cudaStream_t s) {
  const int64_t n = op->n;
  if (n > 0) {
    DevBuf<double> ones, r;
    PR_TRY(ones.alloc(n, s));
    PR_TRY(r.alloc(n, s));
    std::vector<double> h1(n, 1.0);
    PR_CUDA(cudaMemcpyAsync(ones.ptr, h1.data(), n * 8, cudaMemcpyHostToDevice, s));
    PR_TRY(apply(op, PR_APPLY_MATVEC, ones.ptr, r.ptr, s));
    std::vector<double> hr(n);
    PR_CUDA(cudaMemcpyAsync(hr.data(), r.ptr, n * 8, cudaMemcpyDeviceToHost, s));
    PR_CUDA(cudaStreamSynchronize(s));
    double e = 0.0;
    for (int64_t i = 0; i < n; ++i) e = fmax(e, fabs(hr[i] - 1.0));
    op->row_sum_error = e;
    if (!(e <= 1.0e-10)) {
      set_error("projected rows do not close: %.3e", e);
      return PR_ERR_NOT_CLOSED;
    }
  }
  PR_CUDA(cudaStreamSynchronize(s));
  return PR_OK;
}

int operator_create(const pr_counts* k, const int64_t* rays, const double* area, double delta, double tol,
                    cudaStream_t s, pr_operator** out) {
  std::unique_ptr<pr_operator> op;
  PR_TRY(operator_assemble(k, rays, area, delta, s, op));
  if (op->n > 0) PR_TRY(balance(op.get(), tol, s));
  PR_TRY(operator_closure(op.get(), s));
  *out = op.release();
  return PR_OK;
}

// Several operators at once: each assembled as operator_create does, then those stored as word
// streams balanced together (balance_batch), the others one at a time; out[k] is
// set only when every operator succeeds.
int operators_create_batch(const pr_counts* const* counts, const int64_t* const* rays, const double* const* area,
                           int n_ops, double delta, double tol, cudaStream_t s, pr_operator** out) {
  std::vector<std::unique_ptr<pr_operator>> ops(n_ops);
  for (int k = 0; k < n_ops; ++k) PR_TRY(operator_assemble(counts[k], rays[k], area[k], delta, s, ops[k]));
  std::vector<pr_operator*> streams;
  for (int k = 0; k < n_ops; ++k) {
    pr_operator* op = ops[k].get();
    if (op->n == 0) continue;
    if (op->S.mode == kStream) streams.push_back(op);
    else PR_TRY(balance(op, tol, s));
  }
  PR_TRY(balance_batch(streams, tol, s));
  for (int k = 0; k < n_ops; ++k) PR_TRY(operator_closure(ops[k].get(), s));
  for (int k = 0; k < n_ops; ++k) out[k] = ops[k].release();
  return PR_OK;
}

// y = product(x) with x, y device vectors of length n.
int apply(const pr_operator* op, int which, const double* x, double* y, cudaStream_t s) {
  const int64_t n = op->n;
  if (n == 0) return PR_OK;
  const CountCsr& F = *op->F;
  if (which == PR_APPLY_RAW || which == PR_APPLY_RAW_T) {
    const CountCsr& M = which == PR_APPLY_RAW ? F : *op->FT;
    ::pr::launch_mark(), k_raw_apply<<<spmv_grid(n), 256, 0, s>>>(M.row_ptr.ptr, M.col.ptr, M.cnt.ptr, op->rays.ptr, n,
                                             which == PR_APPLY_RAW_T, x, y);
    PR_CUDA(cudaGetLastError());
    return PR_OK;
  }
  int mode = which == PR_APPLY_SYM ? 0 : (which == PR_APPLY_MATVEC ? 1 : 2);
  PR_ARG(which >= 0 && which <= PR_APPLY_RMATVEC, "unknown product %d", which);
  DevBuf<double> u, part;
  PR_TRY(part.alloc(stream_part(op->S), s));
  if (mode != 0) {
    PR_TRY(u.alloc(n, s));
    ::pr::launch_mark(), k_prep_u<<<grid_for(n, 256), 256, 0, s>>>(op->scale.ptr, op->area.ptr, x, n, mode, u.ptr);
    PR_CUDA(cudaGetLastError());
  }
  const double* v = mode == 0 ? x : u.ptr;
  const ApplyEpi epi{op->delta, op->area.ptr, op->scale.ptr, v, mode, y};
  int st = PR_OK;
  dispatch_mode(op->S.mode, [&](auto un) { st = launch_spmv<decltype(un)::value, double>(op->S, v, part.ptr, epi, s); });
  PR_TRY(st);
  op->spmv_calls++;
  return PR_OK;
}

int reciprocity_error(const pr_operator* op, double* out, cudaStream_t s) {
  const int64_t n = op->n;
  DevBuf<double> r;
  PR_TRY(r.alloc(2, s));
  PR_CUDA(cudaMemsetAsync(r.ptr, 0, 16, s));
  const CountCsr& F = *op->F;
  if (n > 0) {
    ::pr::launch_mark(), k_reciprocity<<<grid_for(n, 256), 256, 0, s>>>(F.row_ptr.ptr, F.col.ptr, F.cnt.ptr, op->rays.ptr, op->area.ptr,
                                                  op->scale.ptr, op->delta, n, r.ptr);
    PR_CUDA(cudaGetLastError());
  }
  double h[2];
  PR_CUDA(cudaMemcpyAsync(h, r.ptr, 16, cudaMemcpyDeviceToHost, s));
  PR_CUDA(cudaStreamSynchronize(s));
  const double tiny = 2.2250738585072014e-308;
  *out = h[0] / fmax(h[1], tiny);
  return PR_OK;
}

int operator_edges(const pr_operator* op, int32_t* origin, int32_t* receiver, double* weight, cudaStream_t s) {
  const CountCsr& F = *op->F;
  const int64_t m = F.nnz, n = op->n;
  if (m == 0) return PR_OK;
  DevBuf<int32_t> o;
  DevBuf<double> w;
  if (origin) PR_TRY(o.alloc(m, s));
  if (weight) PR_TRY(w.alloc(m, s));
  ::pr::launch_mark(), k_edges_out<<<spmv_grid(n), 256, 0, s>>>(F.row_ptr.ptr, F.cnt.ptr, op->rays.ptr, n, origin ? o.ptr : nullptr,
                                           weight ? w.ptr : nullptr);
  PR_CUDA(cudaGetLastError());
  if (origin) PR_CUDA(cudaMemcpyAsync(origin, o.ptr, m * 4, cudaMemcpyDefault, s));
  if (receiver) PR_CUDA(cudaMemcpyAsync(receiver, F.col.ptr, m * 4, cudaMemcpyDefault, s));
  if (weight) PR_CUDA(cudaMemcpyAsync(weight, w.ptr, m * 8, cudaMemcpyDefault, s));
  PR_CUDA(cudaStreamSynchronize(s));
  return PR_OK;
}

}  // namespace pr
