// Structural analysis on the device: CSC validation, the in-degree analyser,
// prefix scans, a stable radix sort, level sets, and the position-space
// layouts the executors read.
#include <algorithm>
#include <climits>
#include <cstdio>

#include "exec_common.cuh"
#include "internal.h"

namespace sptrsv {

namespace {
constexpr int kThreads = 256;

inline int grid_for(long long count, int threads = kThreads, int cap = 1 << 20) {
  long long g = (count + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return static_cast<int>(g);
}
}  // namespace

__device__ __forceinline__ int dir_of(const SysDesc& d, long long c) {
  return d.dir ? static_cast<int>(d.dir[c]) : d.substitution;
}

// ------------------------------------------------------------ validation
__global__ void k_validate_ptr(const int* __restrict__ col_ptr, int n, int nnz, int* flags) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c <= n; c += stride) {
    const int v = col_ptr[c];
    bool bad = v < 0 || v > nnz;
    if (c == 0 && v != 0) bad = true;
    if (c == n && v != nnz) bad = true;
    if (c < n && col_ptr[c + 1] < v) bad = true;
    if (bad) atomicOr(flags, SF_BAD_PTR);
  }
}

// One thread per column. A column whose pointers are not an in-range,
// non-decreasing pair is flagged SF_BAD_PTR and its rows are not read, so the
// kernel is safe on any column-pointer array (nnz = length of row_idx).
__global__ void k_validate_rows(const int* __restrict__ col_ptr, const int* __restrict__ row_idx, int n, int nnz,
                                SysDesc sd, int* flags) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += stride) {
    const int substitution = dir_of(sd, c);
    const int beg = col_ptr[c], end = col_ptr[c + 1];
    int f = 0;
    if (beg < 0 || end < beg || end > nnz) {
      f |= SF_BAD_PTR;
    } else if (beg == end) {
      f |= SF_MISSING_DIAG;
    } else {
      int prev = -1;
      bool has_diag = false;
      for (int e = beg; e < end; ++e) {
        const int r = row_idx[e];
        if (r < 0 || r >= n) { f |= SF_ROW_RANGE; break; }
        if (r <= prev) f |= SF_UNSORTED;
        prev = r;
        if (r == c) has_diag = true;
        if (substitution == 0 ? r < c : r > c) f |= SF_WRONG_TRIANGLE;
      }
      if (!(f & SF_ROW_RANGE)) {
        if (!has_diag) f |= SF_MISSING_DIAG;
        // The diagonal must open a forward column and close a backward one.
        const int edge = substitution == 0 ? row_idx[beg] : row_idx[end - 1];
        if (has_diag && edge != c) f |= SF_UNSORTED;
      }
    }
    if (f) atomicOr(flags, f);
  }
}

cudaError_t launch_validate_ptr(const int* col_ptr, int n, int nnz, int* flags, cudaStream_t s) {
  k_validate_ptr<<<grid_for((long long)n + 1), kThreads, 0, s>>>(col_ptr, n, nnz, flags);
  return cudaGetLastError();
}
cudaError_t launch_validate_rows(const int* col_ptr, const int* row_idx, int n, int nnz, const SysDesc& sd,
                                 int* flags, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_validate_rows<<<grid_for(n), kThreads, 0, s>>>(col_ptr, row_idx, n, nnz, sd, flags);
  return cudaGetLastError();
}

// ------------------------------------------------------------ batches
__device__ __forceinline__ int upper_bound_sys(const int* off, int count, long long v) {
  // largest s with off[s] <= v
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= v) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__global__ void k_batch_cols(const int* __restrict__ col_ptr_cat, int count, const int* __restrict__ sys_off,
                             const int* __restrict__ sys_eoff, const int* __restrict__ sys_sub, int n, int nnz,
                             int* col_ptr, unsigned char* dir, int* sys_of, int* flags) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  if (blockIdx.x == 0 && threadIdx.x == 0) col_ptr[n] = nnz;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += stride) {
    const int sy = upper_bound_sys(sys_off, count, c);
    const long long local = c - sys_off[sy];
    const int len = (sy + 1 < count ? sys_off[sy + 1] : n) - sys_off[sy];
    const int* cp = col_ptr_cat + sys_off[sy] + sy;
    const int enz = (sy + 1 < count ? sys_eoff[sy + 1] : nnz) - sys_eoff[sy];
    if (local == 0 && (cp[0] != 0 || cp[len] != enz)) atomicOr(flags, SF_BAD_PTR);
    col_ptr[c] = sys_eoff[sy] + cp[local];
    dir[c] = static_cast<unsigned char>(sys_sub[sy]);
    sys_of[c] = sy;
  }
}
__global__ void k_batch_rows(const int* __restrict__ row_idx_cat, int count, const int* __restrict__ sys_off,
                             const int* __restrict__ sys_eoff, int n, int nnz, int* row_idx, int* flags) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nnz; e += stride) {
    const int sy = upper_bound_sys(sys_eoff, count, e);
    const int local = row_idx_cat[e];
    const int len = (sy + 1 < count ? sys_off[sy + 1] : n) - sys_off[sy];
    if (local < 0 || local >= len) atomicOr(flags, SF_ROW_RANGE);
    row_idx[e] = sys_off[sy] + local;
  }
}
cudaError_t launch_batch_merge(const int* col_ptr_cat, const int* row_idx_cat, int count, const int* sys_off,
                               const int* sys_eoff, const int* sys_sub, int n, int nnz, int* col_ptr, int* row_idx,
                               unsigned char* dir, int* sys_of, int* flags, cudaStream_t s) {
  k_batch_cols<<<grid_for(n > 0 ? n : 1), kThreads, 0, s>>>(col_ptr_cat, count, sys_off, sys_eoff, sys_sub, n, nnz,
                                                            col_ptr, dir, sys_of, flags);
  if (nnz > 0)
    k_batch_rows<<<grid_for(nnz), kThreads, 0, s>>>(row_idx_cat, count, sys_off, sys_eoff, n, nnz, row_idx, flags);
  return cudaGetLastError();
}

__device__ __forceinline__ void nat_of(const SysDesc& sd, int n, long long r, long long* off, long long* nat) {
  if (!sd.sys_of) {
    *off = 0;
    *nat = sd.substitution == 0 ? r : n - 1 - r;
    return;
  }
  const int sy = sd.sys_of[r];
  *off = sd.sys_off[sy];
  const long long local = r - *off;
  *nat = sd.dir[r] == 0 ? local : sd.sys_n[sy] - 1 - local;
}

__global__ void k_nat_rows(SysDesc sd, int n, int* rows_nat) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n; r += stride) {
    long long off, nat;
    nat_of(sd, n, r, &off, &nat);
    rows_nat[off + nat] = static_cast<int>(r);
  }
}
cudaError_t launch_nat_rows(const SysDesc& sd, int n, int* rows_nat, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_nat_rows<<<grid_for(n), kThreads, 0, s>>>(sd, n, rows_nat);
  return cudaGetLastError();
}

// ------------------------------------------------------------ in-degree analyser
// inDeg[row] += 1 for every stored entry, diagonal included
// (reference: SpTRSV_cuda/sptrsv_syncfree_cuda.h:8-19). The caller zeroes inDeg.
// A row index outside [0, m) is skipped (never written) and, when `bad` is
// given, raises SF_ROW_RANGE there.
__global__ void k_in_degree(const int* __restrict__ row_idx, int m, int nnz, int* in_degree, int* bad) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nnz; e += stride) {
    const int r = row_idx[e];
    if (static_cast<unsigned>(r) < static_cast<unsigned>(m)) {
      atomicAdd(&in_degree[r], 1);
    } else if (bad) {
      atomicOr(bad, SF_ROW_RANGE);
    }
  }
}
cudaError_t launch_in_degree(const int* row_idx, int m, int nnz, int* in_degree, cudaStream_t s, int* bad) {
  if (nnz == 0) return cudaSuccess;
  k_in_degree<<<grid_for(nnz), kThreads, 0, s>>>(row_idx, m, nnz, in_degree, bad);
  return cudaGetLastError();
}

// ------------------------------------------------------------ exclusive scan
namespace {
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ int block_exclusive_scan(int v, int* s_warp, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    int w = lane < nw ? s_warp[lane] : 0;
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    if (lane < nw) s_warp[lane] = wi - w;
    if (lane == nw - 1) s_warp[32] = wi;
  }
  __syncthreads();
  const int excl = incl - v + s_warp[warp];
  *total = s_warp[32];
  __syncthreads();
  return excl;
}

__global__ void k_scan_tile_sums(const int* __restrict__ in, int count, int* sums) {
  __shared__ int s_warp[33];
  const long long base = (long long)blockIdx.x * kScanTile;
  int acc = 0;
  for (int i = 0; i < kScanItems; ++i) {
    const long long idx = base + (long long)i * kScanThreads + threadIdx.x;
    if (idx < count) acc += in[idx];
  }
  int total;
  block_exclusive_scan(acc, s_warp, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void k_scan_tiles(const int* __restrict__ in, int* out, int count, const int* __restrict__ carry,
                             int* total_out) {
  __shared__ int s_vals[kScanTile];
  __shared__ int s_warp[33];
  const long long base = (long long)blockIdx.x * kScanTile;
  for (int i = 0; i < kScanItems; ++i) {
    const int li = i * kScanThreads + threadIdx.x;
    const long long idx = base + li;
    s_vals[li] = idx < count ? in[idx] : 0;
  }
  __syncthreads();
  int local[kScanItems];
  int acc = 0;
  for (int i = 0; i < kScanItems; ++i) {
    local[i] = s_vals[threadIdx.x * kScanItems + i];
    acc += local[i];
  }
  int total;
  int run = block_exclusive_scan(acc, s_warp, &total) + (carry ? carry[blockIdx.x] : 0);
  for (int i = 0; i < kScanItems; ++i) {
    s_vals[threadIdx.x * kScanItems + i] = run;
    run += local[i];
  }
  __syncthreads();
  for (int i = 0; i < kScanItems; ++i) {
    const int li = i * kScanThreads + threadIdx.x;
    const long long idx = base + li;
    if (idx < count) out[idx] = s_vals[li];
  }
  if (total_out && blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanThreads - 1) {
    *total_out = run;  // last thread's running value after its items = grand total
  }
}
}  // namespace

cudaError_t exclusive_scan_int(const int* in, int* out, int count, bool with_total, cudaStream_t s) {
  if (count <= 0) {
    if (with_total) return cudaMemsetAsync(out, 0, sizeof(int), s);
    return cudaSuccess;
  }
  const int tiles = (count + kScanTile - 1) / kScanTile;
  int* total_ptr = with_total ? out + count : nullptr;
  if (tiles == 1) {
    k_scan_tiles<<<1, kScanThreads, 0, s>>>(in, out, count, nullptr, total_ptr);
    return cudaGetLastError();
  }
  int* sums = nullptr;
  cudaError_t err = cudaMallocAsync(reinterpret_cast<void**>(&sums), sizeof(int) * (size_t)(tiles + 1), s);
  if (err != cudaSuccess) return err;
  k_scan_tile_sums<<<tiles, kScanThreads, 0, s>>>(in, count, sums);
  err = cudaGetLastError();
  if (err == cudaSuccess) err = exclusive_scan_int(sums, sums, tiles, false, s);
  if (err == cudaSuccess) {
    k_scan_tiles<<<tiles, kScanThreads, 0, s>>>(in, out, count, sums, total_ptr);
    err = cudaGetLastError();
  }
  cudaError_t e2 = cudaFreeAsync(sums, s);
  return err != cudaSuccess ? err : e2;
}

// ------------------------------------------------------------ stable radix sort
namespace {
constexpr int kRsThreads = 256;
constexpr int kRsItems = 8;
constexpr int kRsTile = kRsThreads * kRsItems;
constexpr int kRsBins = 256;

__global__ void k_rs_hist(const unsigned* __restrict__ keys, int count, int shift, int* hist, int nblocks) {
  __shared__ int s_h[kRsBins];
  s_h[threadIdx.x] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * kRsTile;
  for (int i = 0; i < kRsItems; ++i) {
    const long long idx = base + (long long)i * kRsThreads + threadIdx.x;
    if (idx < count) atomicAdd(&s_h[(keys[idx] >> shift) & 0xFFu], 1);
  }
  __syncthreads();
  hist[threadIdx.x * nblocks + blockIdx.x] = s_h[threadIdx.x];
}

// Stable scatter: elements are ranked in index order within the tile (iteration
// by iteration, warp by warp, lane by lane), so equal digits keep input order.
__global__ void k_rs_scatter(const unsigned* __restrict__ keys_in, const int* __restrict__ vals_in,
                             unsigned* keys_out, int* vals_out, int count, int shift,
                             const int* __restrict__ offsets, int nblocks) {
  constexpr int kWarps = kRsThreads / 32;
  __shared__ int s_cnt[kWarps][kRsBins];
  __shared__ int s_off[kWarps][kRsBins];
  __shared__ int s_run[kRsBins];
  __shared__ int s_base[kRsBins];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  s_run[threadIdx.x] = 0;
  s_base[threadIdx.x] = offsets[threadIdx.x * nblocks + blockIdx.x];
  const long long base = (long long)blockIdx.x * kRsTile;
  for (int it = 0; it < kRsItems; ++it) {
    for (int w = 0; w < kWarps; ++w) s_cnt[w][threadIdx.x] = 0;
    __syncthreads();
    const long long idx = base + (long long)it * kRsThreads + threadIdx.x;
    const bool valid = idx < count;
    unsigned key = 0;
    int val = 0;
    int digit = kRsBins;  // out-of-range elements form their own group
    if (valid) {
      key = keys_in[idx];
      val = vals_in[idx];
      digit = static_cast<int>((key >> shift) & 0xFFu);
    }
    const unsigned peers = __match_any_sync(0xffffffffu, digit);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    const int leader = __ffs(peers) - 1;
    if (valid && lane == leader) s_cnt[warp][digit] = __popc(peers);
    __syncthreads();
    {
      int run = s_run[threadIdx.x];
      for (int w = 0; w < kWarps; ++w) {
        s_off[w][threadIdx.x] = run;
        run += s_cnt[w][threadIdx.x];
      }
      s_run[threadIdx.x] = run;
    }
    __syncthreads();
    if (valid) {
      const int pos = s_base[digit] + s_off[warp][digit] + rank;
      keys_out[pos] = key;
      vals_out[pos] = val;
    }
    __syncthreads();
  }
}
}  // namespace

size_t radix_sort_temp_bytes(int count) {
  const size_t nblocks = (size_t)((count + kRsTile - 1) / kRsTile);
  // histogram (+1 for the scan total), ping-pong keys and values
  return ((nblocks * kRsBins + 1) * sizeof(int) + 255) / 256 * 256 + (size_t)count * 8 + 512;
}

cudaError_t radix_sort_pairs(const unsigned* keys_in, const int* vals_in, unsigned* keys_out, int* vals_out,
                             int count, int key_bits, void* temp, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  const int nblocks = (count + kRsTile - 1) / kRsTile;
  int* hist = static_cast<int*>(temp);
  const size_t hist_bytes = (((size_t)nblocks * kRsBins + 1) * sizeof(int) + 255) / 256 * 256;
  unsigned* k_tmp = reinterpret_cast<unsigned*>(static_cast<char*>(temp) + hist_bytes);
  int* v_tmp = reinterpret_cast<int*>(k_tmp + count);
  int passes = (key_bits + 7) / 8;
  if (passes < 1) passes = 1;
  // Ping-pong so that the last pass lands in the output arrays.
  const unsigned* src_k = keys_in;
  const int* src_v = vals_in;
  for (int p = 0; p < passes; ++p) {
    const bool to_out = ((passes - 1 - p) % 2) == 0;
    unsigned* dk = to_out ? keys_out : k_tmp;
    int* dv = to_out ? vals_out : v_tmp;
    k_rs_hist<<<nblocks, kRsThreads, 0, s>>>(src_k, count, p * 8, hist, nblocks);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    err = exclusive_scan_int(hist, hist, nblocks * kRsBins, false, s);
    if (err != cudaSuccess) return err;
    k_rs_scatter<<<nblocks, kRsThreads, 0, s>>>(src_k, src_v, dk, dv, count, p * 8, hist, nblocks);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    src_k = dk;
    src_v = dv;
  }
  return cudaSuccess;
}

// ------------------------------------------------------------ small helpers
__global__ void k_iota(int* out, int count, int start, int step) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += stride)
    out[i] = start + static_cast<int>(i) * step;
}
cudaError_t launch_iota(int* out, int count, int start, int step, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  k_iota<<<grid_for(count), kThreads, 0, s>>>(out, count, start, step);
  return cudaGetLastError();
}

__global__ void k_expand_cols(const int* __restrict__ col_ptr, int n, int* col_of) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += stride)
    for (int e = col_ptr[c]; e < col_ptr[c + 1]; ++e) col_of[e] = static_cast<int>(c);
}
cudaError_t launch_expand_cols(const int* col_ptr, int n, int* col_of, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_expand_cols<<<grid_for(n), kThreads, 0, s>>>(col_ptr, n, col_of);
  return cudaGetLastError();
}

constexpr int kRankMax = 1024;  // longest list sorted by rank (k_rank_lists)

// Column of every entry, and the entries dealt to their rows in any order:
// (entry, column) at the next free slot of row r (cursor[r], row pointers on
// entry). A warp takes 32 columns, whose entries are one contiguous range.
__global__ void __launch_bounds__(kThreads) k_scatter_rows(const int* __restrict__ col_ptr,
                                                           const int* __restrict__ row_idx, int n, int* cursor,
                                                           int* col_of, int* entry_out, int* col_out) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long groups = ((long long)n + 31) / 32;
  for (long long g = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; g < groups; g += nwarps) {
    const long long c = g * 32 + lane;
    const int start = c < n ? col_ptr[c] : INT_MAX;
    const int end = c < n ? col_ptr[c + 1] : 0;
    const unsigned lo = static_cast<unsigned>(__shfl_sync(kFull, start, 0));
    const unsigned hi = static_cast<unsigned>(__reduce_max_sync(kFull, end));
    for (unsigned base = lo; base < hi; base += 32) {
      const unsigned e = base + lane;
      int own = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const int t = __shfl_sync(kFull, start, own + step);
        if (static_cast<unsigned>(t) <= e) own += step;
      }
      if (e >= hi) continue;
      const int col = static_cast<int>(g * 32) + own;
      const int slot = atomicAdd(&cursor[row_idx[e]], 1);
      col_of[e] = col;
      entry_out[slot] = static_cast<int>(e);
      col_out[slot] = col;
    }
  }
}

// CSR rows from CSC columns by a counting transpose: scatter, then each row's
// entries sorted by their CSC index (ascending column). row_ptr = exclusive
// scan of the row counts, no row longer than kRankMax entries. (The stable
// radix sort of all entries on their row took 0.65 ms for 3M entries.)
bool transpose_by_rank(int longest_row) { return longest_row <= kRankMax; }

cudaError_t launch_transpose_pattern(const int* col_ptr, const int* row_idx, const int* row_ptr, int n, int nnz,
                                     int* col_of, int* src_out, int* col_out, cudaStream_t s) {
  if (n <= 0 || nnz <= 0) return cudaSuccess;
  int *cursor = nullptr, *entry = nullptr, *col = nullptr;
  auto run = [&]() -> cudaError_t {
    cudaError_t e;
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&cursor), sizeof(int) * n, s)) != cudaSuccess) return e;
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&entry), sizeof(int) * nnz, s)) != cudaSuccess) return e;
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&col), sizeof(int) * nnz, s)) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(cursor, row_ptr, sizeof(int) * n, cudaMemcpyDeviceToDevice, s)) != cudaSuccess) return e;
    k_scatter_rows<<<grid_for(n), kThreads, 0, s>>>(col_ptr, row_idx, n, cursor, col_of, entry, col);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return launch_rank_lists(row_ptr, entry, col, n, false, src_out, col_out, s);
  };
  const cudaError_t e = run();
  if (cursor) cudaFreeAsync(cursor, s);
  if (entry) cudaFreeAsync(entry, s);
  if (col) cudaFreeAsync(col, s);
  return e;
}

__global__ void k_copy_keys(const int* __restrict__ in, unsigned* out, int count) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += stride)
    out[i] = static_cast<unsigned>(in[i]);
}
cudaError_t launch_copy_keys(const int* in, unsigned* out, int count, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  k_copy_keys<<<grid_for(count), kThreads, 0, s>>>(in, out, count);
  return cudaGetLastError();
}

__global__ void k_gather_int(const int* __restrict__ src, const int* __restrict__ idx, int* out, int count) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += stride)
    out[i] = src[idx[i]];
}
cudaError_t launch_gather_int(const int* src, const int* idx, int* out, int count, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  k_gather_int<<<grid_for(count), kThreads, 0, s>>>(src, idx, out, count);
  return cudaGetLastError();
}

// ------------------------------------------------------------ ready-order lists
// The fast (non-exact) executors consume a dependency list in batches and only
// move to the next batch once the current one has arrived. Listing each
// position's dependencies in the order they complete (ascending position for a
// forward walk, descending for the reverse walk) leaves only the final batch
// waiting on the last publication, instead of whatever followed it in the
// serial (column) order.
__global__ void k_rank_keys(const int* __restrict__ pos, int count, int n, int descending, unsigned* keys) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += stride)
    keys[i] = static_cast<unsigned>(descending ? n - 1 - pos[i] : pos[i]);
}
__global__ void k_owner_keys(const int* __restrict__ owner, const int* __restrict__ idx, int count, unsigned* keys) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += stride)
    keys[i] = static_cast<unsigned>(owner[idx[i]]);
}

// Lists up to kRankMax entries are sorted by rank: an entry's place in its list
// is the number of smaller keys there (keys are distinct inside a list). A warp
// takes the lists of 32 consecutive owners, one contiguous range; its lanes walk
// the entries and, as neighbours mostly share a list, read each list's keys as
// broadcasts. Two stable radix sorts of all entries (by position, then by owner)
// took 0.80 ms for the lists of a 2.7M-entry system and 8.1 ms for those of 33M
// entries (lists up to 1,000).
__global__ void __launch_bounds__(kThreads) k_rank_lists(const int* __restrict__ ptr, const int* __restrict__ key,
                                                         const int* __restrict__ src, int n, int descending,
                                                         int* key_out, int* src_out) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long groups = ((long long)n + 31) / 32;
  for (long long g = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; g < groups; g += nwarps) {
    const long long p = g * 32 + lane;
    const int start = p < n ? ptr[p] : INT_MAX;
    const int end = p < n ? ptr[p + 1] : 0;
    const unsigned lo = static_cast<unsigned>(__shfl_sync(kFull, start, 0));
    const unsigned hi = static_cast<unsigned>(__reduce_max_sync(kFull, end));
    for (unsigned base = lo; base < hi; base += 32) {
      const unsigned e = base + lane;
      // the last list that starts at or before e owns it (empty lists share
      // their successor's start)
      int own = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const int t = __shfl_sync(kFull, start, own + step);
        if (static_cast<unsigned>(t) <= e) own += step;
      }
      const int s0 = __shfl_sync(kFull, start, own), s1 = __shfl_sync(kFull, end, own);
      if (e >= hi) continue;
      const int k = key[e];
      int rank = 0;
#pragma unroll 4
      for (int j = s0; j < s1; ++j) rank += key[j] < k ? 1 : 0;
      if (descending) rank = s1 - s0 - 1 - rank;
      key_out[s0 + rank] = k;
      src_out[s0 + rank] = src[e];
    }
  }
}

cudaError_t launch_rank_lists(const int* ptr, const int* key, const int* src, int n, bool descending, int* key_out,
                              int* src_out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_rank_lists<<<grid_for(n), kThreads, 0, s>>>(ptr, key, src, n, descending ? 1 : 0, key_out, src_out);
  return cudaGetLastError();
}

cudaError_t launch_sort_lists(const int* ptr, const int* pos, const int* src, int n, int count, int longest,
                              bool descending, int* pos_out, int* src_out, cudaStream_t s) {
  if (count <= 0 || n <= 0) return cudaSuccess;
  if (longest <= kRankMax) return launch_rank_lists(ptr, pos, src, n, descending, pos_out, src_out, s);
  int bits = 1;
  while (bits < 31 && (1u << bits) <= static_cast<unsigned>(n - 1)) ++bits;
  unsigned *k1 = nullptr, *k2 = nullptr;
  int *v1 = nullptr, *v2 = nullptr;
  void* temp = nullptr;
  auto run = [&]() -> cudaError_t {
    cudaError_t err;
    if ((err = cudaMallocAsync(reinterpret_cast<void**>(&k1), sizeof(unsigned) * count, s)) != cudaSuccess) return err;
    if ((err = cudaMallocAsync(reinterpret_cast<void**>(&k2), sizeof(unsigned) * count, s)) != cudaSuccess) return err;
    if ((err = cudaMallocAsync(reinterpret_cast<void**>(&v1), sizeof(int) * count, s)) != cudaSuccess) return err;
    if ((err = cudaMallocAsync(reinterpret_cast<void**>(&v2), sizeof(int) * count, s)) != cudaSuccess) return err;
    if ((err = cudaMallocAsync(&temp, radix_sort_temp_bytes(count), s)) != cudaSuccess) return err;
    // entries by position of the dependency, then (stable) by owning position
    k_rank_keys<<<grid_for(count), kThreads, 0, s>>>(pos, count, n, descending ? 1 : 0, k1);
    if ((err = launch_iota(v1, count, 0, 1, s)) != cudaSuccess) return err;
    if ((err = radix_sort_pairs(k1, v1, k2, v2, count, bits, temp, s)) != cudaSuccess) return err;
    if ((err = launch_expand_cols(ptr, n, v1, s)) != cudaSuccess) return err;
    k_owner_keys<<<grid_for(count), kThreads, 0, s>>>(v1, v2, count, k1);
    if ((err = radix_sort_pairs(k1, v2, k2, v1, count, bits, temp, s)) != cudaSuccess) return err;
    if ((err = launch_gather_int(pos, v1, pos_out, count, s)) != cudaSuccess) return err;
    if ((err = launch_gather_int(src, v1, src_out, count, s)) != cudaSuccess) return err;
    return cudaGetLastError();
  };
  const cudaError_t err = run();
  // temporaries are released on every path (stream-ordered after their last use)
  if (k1) cudaFreeAsync(k1, s);
  if (k2) cudaFreeAsync(k2, s);
  if (v1) cudaFreeAsync(v1, s);
  if (v2) cudaFreeAsync(v2, s);
  if (temp) cudaFreeAsync(temp, s);
  return err;
}

// ------------------------------------------------------------ schedule heuristics
// The plan's counters (PlanCounter, summed or maximised into count[]). Grids of
// a few CTAs per SM with one atomic per CTA and counter: with one per warp the
// same-address atomics took 130-200 us of a 6-10M-entry analysis.
namespace {
constexpr int kStatGrid = 152 * 8;

__device__ __forceinline__ unsigned long long block_sum(unsigned long long v, unsigned long long* s_warp) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned long long t = 0;
  for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) t += s_warp[w];
  return t;
}
}  // namespace

// Longest dependency list (CSR rows) and longest dependent list (CSC columns),
// and the entries of lists longer than `cut` on either side (diagonals excluded).
__global__ void k_list_stats(const int* __restrict__ row_ptr, const int* __restrict__ col_ptr, int n, int cut,
                             unsigned long long* count) {
  __shared__ unsigned long long s_warp[kThreads / 32];
  __shared__ int s_max[2];
  if (threadIdx.x < 2) s_max[threadIdx.x] = 0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  unsigned long long row_long = 0, col_long = 0;
  int row_max = 0, col_max = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    const int r = row_ptr[i + 1] - row_ptr[i] - 1, c = col_ptr[i + 1] - col_ptr[i] - 1;
    row_max = max(row_max, r);
    col_max = max(col_max, c);
    if (r > cut) row_long += r;
    if (c > cut) col_long += c;
  }
  row_max = __reduce_max_sync(0xffffffffu, row_max);
  col_max = __reduce_max_sync(0xffffffffu, col_max);
  row_long = block_sum(row_long, s_warp);
  col_long = block_sum(col_long, s_warp);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&s_max[0], row_max);
    atomicMax(&s_max[1], col_max);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMax(&count[PC_ROW_MAX], static_cast<unsigned long long>(s_max[0]));
    atomicMax(&count[PC_COL_MAX], static_cast<unsigned long long>(s_max[1]));
    if (row_long) atomicAdd(&count[PC_ROW_LONG], row_long);
    if (col_long) atomicAdd(&count[PC_COL_LONG], col_long);
  }
}

cudaError_t launch_list_stats(const int* row_ptr, const int* col_ptr, int n, int cut, unsigned long long* count,
                              cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_list_stats<<<grid_for(n, kThreads, kStatGrid), kThreads, 0, s>>>(row_ptr, col_ptr, n, cut, count);
  return cudaGetLastError();
}

// How unlike the lists of neighbouring positions are: over windows of kVarietyWindow
// segments of 32 positions, the squared deviations of the segments' entries from their
// window's mean (count[0]) and the squared means (count[1]), rounded per window, so that
// the sums do not depend on their order. A last part of a segment is left out.
constexpr int kVarietyWindow = 64;
__global__ void __launch_bounds__(kVarietyWindow) k_list_variety(const int* __restrict__ ptr, int nseg,
                                                                 unsigned long long* count) {
  __shared__ double s_sum[2], s_square[2];
  const int g = blockIdx.x * kVarietyWindow + threadIdx.x;
  const double v = g < nseg ? static_cast<double>(ptr[(g + 1) * 32] - ptr[g * 32]) : 0.0;
  double sum = v, square = v * v;
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    square += __shfl_xor_sync(0xffffffffu, square, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s_sum[threadIdx.x >> 5] = sum;
    s_square[threadIdx.x >> 5] = square;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  const double total = s_sum[0] + s_sum[1];
  const double mean2 = total * total / min(kVarietyWindow, nseg - static_cast<int>(blockIdx.x) * kVarietyWindow);
  atomicAdd(&count[0], static_cast<unsigned long long>(llrint(fmax(s_square[0] + s_square[1] - mean2, 0.0))));
  atomicAdd(&count[1], static_cast<unsigned long long>(llrint(mean2)));
}

cudaError_t launch_list_variety(const int* ptr, int n, unsigned long long* count, cudaStream_t s) {
  const int nseg = n / 32;
  if (nseg <= 0) return cudaSuccess;
  k_list_variety<<<(nseg + kVarietyWindow - 1) / kVarietyWindow, kVarietyWindow, 0, s>>>(ptr, nseg, count);
  return cudaGetLastError();
}

// Off-diagonal entries whose row and column fall in the same block of `block`
// unknowns of the natural execution order (ascending for a forward solve,
// descending for a backward one): how much of the DAG a blocked order keeps
// inside one CTA.
__global__ void k_block_locality(const int* __restrict__ row, const int* __restrict__ col, int nnz, int n,
                                 int block, int backward, unsigned long long* count) {
  __shared__ unsigned long long s_warp[kThreads / 32];
  const long long stride = (long long)gridDim.x * blockDim.x;
  unsigned local = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nnz; i += stride) {
    const int r = row[i], c = col[i];
    if (r == c) continue;
    const int pr = backward ? n - 1 - r : r, pc = backward ? n - 1 - c : c;
    local += (pr / block == pc / block) ? 1u : 0u;
  }
  const unsigned long long total = block_sum(local, s_warp);
  if (threadIdx.x == 0 && total) atomicAdd(&count[PC_LOCAL], total);
}

cudaError_t launch_block_locality(const int* row, const int* col, int nnz, int n, int block, bool backward,
                                  unsigned long long* count, cudaStream_t s) {
  if (nnz <= 0) return cudaSuccess;
  k_block_locality<<<grid_for(nnz, kThreads, kStatGrid), kThreads, 0, s>>>(row, col, nnz, n, block, backward ? 1 : 0,
                                                                           count);
  return cudaGetLastError();
}

// Unknowns with two or more dependencies on the level just before their own
// (in a warp-synchronous loop those dependencies land in the same iteration)
// and unknowns with any dependency, over the CSR rows (diagonal included in
// each row and skipped here).
__global__ void k_coarrival(const int* __restrict__ row_ptr, const int* __restrict__ col,
                            const int* __restrict__ depth, int n, unsigned long long* count) {
  __shared__ unsigned long long s_warp[kThreads / 32];
  const long long stride = (long long)gridDim.x * blockDim.x;
  unsigned co = 0, any = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    const int prev = depth[i] - 1;
    int k = 0, deps = 0;
    for (int e = row_ptr[i]; e < row_ptr[i + 1]; ++e) {
      const int c = col[e];
      if (c == i) continue;
      ++deps;
      k += depth[c] == prev ? 1 : 0;
    }
    co += k >= 2 ? 1u : 0u;
    any += deps > 0 ? 1u : 0u;
  }
  const unsigned long long co_total = block_sum(co, s_warp), any_total = block_sum(any, s_warp);
  if (threadIdx.x == 0) {
    if (co_total) atomicAdd(&count[PC_COARRIVE], co_total);
    if (any_total) atomicAdd(&count[PC_DEPENDENT], any_total);
  }
}

cudaError_t launch_coarrival(const int* row_ptr, const int* col, const int* depth, int n, unsigned long long* count,
                             cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_coarrival<<<grid_for(n, kThreads, kStatGrid), kThreads, 0, s>>>(row_ptr, col, depth, n, count);
  return cudaGetLastError();
}

// ------------------------------------------------------------ level sets
// Breadth-first peeling of the in-degree, one grid barrier per level
// (the level definition of SpTRSV_cuda/findlevel.h:6-69): level 0 holds rows
// whose only entry is the diagonal; a row joins level l+1 when the last of its
// dependencies is visited at level l. Cooperative launch (all CTAs resident).
__global__ void k_levels(const int* __restrict__ col_ptr, const int* __restrict__ row_idx,
                         const int* __restrict__ in_degree, int n, int* cnt, int* front_a, int* front_b,
                         int* depth, int* level_sizes, DeviceCtl* ctl, unsigned long long timeout_ns,
                         int* tails /* [4]: three rotating tails + level count */, unsigned smin, unsigned smax) {
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = tid; i < n; i += stride) {
    const int d = in_degree[i];
    cnt[i] = d;
    if (d == 1) {
      const int slot = atomicAdd(&tails[0], 1);
      front_a[slot] = static_cast<int>(i);
      depth[i] = 0;
    }
  }
  if (!grid_barrier(ctl, timeout_ns, smin, smax)) return;
  int* cur = front_a;
  int* nxt = front_b;
  for (int level = 0;; ++level) {
    const int cur_tail = level % 3, nxt_tail = (level + 1) % 3, free_tail = (level + 2) % 3;
    const int size = *reinterpret_cast<volatile int*>(&tails[cur_tail]);
    if (size == 0) {
      if (tid == 0) tails[3] = level;
      break;
    }
    if (tid == 0) {
      level_sizes[level] = size;
      tails[free_tail] = 0;
    }
    // one warp per frontier node, lanes over the node's column entries
    const long long warp = tid >> 5;
    const long long nwarps = stride >> 5;
    const int lane = static_cast<int>(tid & 31);
    for (long long q = warp; q < size; q += nwarps) {
      const int node = cur[q];
      for (int e = col_ptr[node] + lane; e < col_ptr[node + 1]; e += 32) {
        const int r = row_idx[e];
        if (r == node) continue;
        const int old = atomicSub(&cnt[r], 1);
        if (old == 2) {
          const int slot = atomicAdd(&tails[nxt_tail], 1);
          nxt[slot] = r;
          depth[r] = level + 1;
        }
      }
    }
    if (!grid_barrier(ctl, timeout_ns, smin, smax)) return;
    int* t = cur;
    cur = nxt;
    nxt = t;
  }
}

cudaError_t launch_levels(const int* col_ptr, const int* row_idx, const int* in_degree, int n, int* cnt_scratch,
                          int* front_a, int* front_b, int* depth, int* level_sizes, DeviceCtl* ctl,
                          unsigned long long timeout_ns, cudaStream_t s) {
  // tails live right after level_sizes[n+1]
  int* tails = level_sizes + n + 1;
  cudaError_t err = cudaMemsetAsync(tails, 0, 4 * sizeof(int), s);
  if (err != cudaSuccess) return err;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // one CTA per SM and a short back-off in the per-level grid barrier: deep
  // DAGs pay one barrier per level (2M-row mesh, 2,827 levels: analysis 41.1
  // ms with four CTAs per SM and 32-256 ns back-off, 36.4 with this; a
  // 200k-row chain 973 vs 694 ms; wide power-law levels unchanged)
  unsigned smin = 16, smax = 64;
  int grid = sms;
  void* args[] = {(void*)&col_ptr, (void*)&row_idx, (void*)&in_degree, (void*)&n, (void*)&cnt_scratch,
                  (void*)&front_a, (void*)&front_b, (void*)&depth, (void*)&level_sizes, (void*)&ctl,
                  (void*)&timeout_ns, (void*)&tails, (void*)&smin, (void*)&smax};
  return cudaLaunchCooperativeKernel((void*)k_levels, dim3(grid), dim3(kThreads), args, 0, s);
}

// Level sets without a barrier per level: depth[r] = 1 + the deepest of its
// dependencies, rows in natural order, one lane per row, a warp's 32 rows in
// lockstep as in the solve executors (value-as-flag words, -1 = not known yet;
// chunk-local dependencies through shared memory). A level then costs one poll
// (or one shared-memory hop) instead of the peeling kernel's chain of dependent
// accesses and its grid barrier (~4 us a level).
//
// Three CTAs of 256 rows per SM and a 100 ns nap after 16 idle iterations: how
// many rows are in flight bounds systems whose levels spread over all rows (a
// mesh row is one long chain), and polls of rows far ahead slow the others.
// Whole analysis, ms, peeling -> 1 / 2 CTAs without naps / 3 with 100 ns / 4
// with 200: 2M-row mesh (2,827 levels) 15.1 -> 15.6 / 10.9 / 9.2 / 8.5; 1M-row
// band (1,232) 8.5 -> 4.1 / 4.2 / 4.5 / 5.1; 150k-row narrow band (8,814) 34.9 ->
// 7.7 / 8.2 / 8.7 / 8.8; 30 independent bands of 39,000 rows one after the other
// 5.8 -> 6.6 / 5.4 / 5.0 / 5.0; a 300,000-row chain 1,046 -> 80 / 90 / 101 / 107.
// (Eight CTAs without naps: the pollers starve the rows they wait for.)
constexpr int kLevelChunk = 256;  // rows per CTA at a time, one per thread
constexpr int kLevelCtas = 3;
constexpr unsigned kLevelNap = 100;

__global__ void __launch_bounds__(kLevelChunk) k_levels_pull(const int* __restrict__ row_ptr,
                                                             const int* __restrict__ col, int n, int backward,
                                                             int nchunks, int* depth, int* deepest, DeviceCtl* ctl,
                                                             unsigned long long timeout_ns) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int U = 4;
  __shared__ int s_depth[kLevelChunk];
  __shared__ unsigned s_chunk;
  const int last = n - 1;
  int mine = 0;
  for (;;) {
    const unsigned c = next_chunk(ctl, nchunks, &s_chunk);
    if (c >= (unsigned)nchunks) break;
    const int base = static_cast<int>(c) * kLevelChunk;
    volatile int* s_d = s_depth;
    s_d[threadIdx.x] = -1;
    __syncthreads();
    const int w = base + threadIdx.x;  // walk index
    const int r = backward ? last - w : w;
    bool done = w >= n, fail = false;
    // entries e, e + step, ... (left of them): farthest dependency first
    int e = 0, left = 0;
    const int step = backward ? -1 : 1;
    if (!done) {
      const int b0 = row_ptr[r], b1 = row_ptr[r + 1];
      left = b1 - b0 - 1;
      e = backward ? b1 - 1 : b0;
    }
    int d = 0, q[U], v[U];
    unsigned todo = 0u;
    auto poll = [&](int u) {
      const int wq = (backward ? last - q[u] : q[u]) - base;
      v[u] = wq >= 0 ? s_d[wq] : static_cast<int>(ld_relaxed_u32(reinterpret_cast<const unsigned*>(&depth[q[u]])));
    };
    auto load = [&]() {
      todo = 0u;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        q[u] = u < left ? col[e + u * step] : -1;
        v[u] = -1;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (q[u] >= 0) {
          poll(u);
          todo |= 1u << u;
        }
    };
    if (!done) load();
    WaitBudget wb(timeout_ns);
    unsigned idle = 0u;
    bool work = __any_sync(kFull, !done);  // the last chunk may leave a warp without rows
    while (work) {
      bool progress = false;
      if (!done) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if ((todo & (1u << u)) && v[u] >= 0) {
            d = max(d, v[u] + 1);
            todo &= ~(1u << u);
            progress = true;
          }
        if (!todo) {
          e += U * step;
          left -= U;
          progress = true;
          if (left > 0) {
            load();
          } else {
            s_d[threadIdx.x] = d;
            st_relaxed_u32(reinterpret_cast<unsigned*>(&depth[r]), static_cast<unsigned>(d));
            mine = max(mine, d);
            done = true;
          }
        } else {
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (todo & (1u << u)) poll(u);
        }
      }
      if (__any_sync(kFull, progress)) {
        idle = 0u;
        work = __any_sync(kFull, !done);
      } else {
        if (idle >= 16u) __nanosleep(kLevelNap);
        if ((++idle & 15u) == 0u && __any_sync(kFull, !wb.poll<true>(ctl, r))) {
          fail = true;
          break;
        }
      }
    }
    if (__syncthreads_or(fail)) break;
  }
  mine = __reduce_max_sync(kFull, mine);
  if ((threadIdx.x & 31) == 0 && mine > 0) atomicMax(deepest, mine);
  leave(ctl);
}

cudaError_t launch_levels_pull(const int* row_ptr, const int* col, int n, bool backward, int* depth, int* deepest,
                               DeviceCtl* ctl, unsigned long long timeout_ns, int num_sms, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(depth, 0xFF, sizeof(int) * (size_t)n, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(deepest, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  const int nchunks = (n + kLevelChunk - 1) / kLevelChunk;
  const int grid = std::min(nchunks, num_sms * kLevelCtas);
  k_levels_pull<<<grid, kLevelChunk, 0, s>>>(row_ptr, col, n, backward ? 1 : 0, nchunks, depth, deepest, ctl,
                                             timeout_ns);
  return cudaGetLastError();
}

// level_ptr[l] = first index of key l in the sorted keys (every level is non-empty)
__global__ void k_level_starts(const unsigned* __restrict__ keys, int n, int nlevels, int* level_ptr) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    if (i == 0 || keys[i] != keys[i - 1]) level_ptr[keys[i]] = static_cast<int>(i);
    if (i == n - 1) level_ptr[nlevels] = n;
  }
}
cudaError_t launch_level_starts(const unsigned* keys, int n, int nlevels, int* level_ptr, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_level_starts<<<grid_for(n), kThreads, 0, s>>>(keys, n, nlevels, level_ptr);
  return cudaGetLastError();
}

// ------------------------------------------------------------ schedule
// mode 0: key = depth (level order); mode 1: key = natural position / block
// (second, stable pass of the blocked level order).
// mode 0: key = depth (level order); mode 1: key = (natural position inside its
// system / block) * count + system (second, stable pass of the blocked level
// order; batches interleave their systems block by block).
__global__ void k_schedule_keys(const int* __restrict__ rows, const int* __restrict__ depth, int n, SysDesc sd,
                                int block, int mode, unsigned* keys, const int* __restrict__ sys_depth,
                                int max_depth) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    const int r = rows[i];
    if (mode == 0) {
      keys[i] = static_cast<unsigned>(depth[r]);
    } else if (mode == 2) {
      // the level stretched to max(D_s, T) keys, T = max_depth (the stretch
      // target): floor(level * max(D_s, T) / D_s) grows strictly with the
      // level inside system s
      const long long ds = sys_depth[sd.sys_of[r]] > 0 ? sys_depth[sd.sys_of[r]] : 1;
      const long long span = ds > max_depth ? ds : max_depth;
      keys[i] = static_cast<unsigned>((long long)depth[r] * span / ds);
    } else {
      long long off, nat;
      nat_of(sd, n, r, &off, &nat);
      const long long sy = sd.sys_of ? sd.sys_of[r] : 0;
      keys[i] = static_cast<unsigned>((nat / block) * sd.count + sy);
    }
  }
}
cudaError_t launch_schedule_keys(const int* rows, const int* depth, int n, const SysDesc& sd, int block, int mode,
                                 unsigned* keys, cudaStream_t s, const int* sys_depth, int max_depth) {
  if (n <= 0) return cudaSuccess;
  k_schedule_keys<<<grid_for(n), kThreads, 0, s>>>(rows, depth, n, sd, block, mode, keys, sys_depth, max_depth);
  return cudaGetLastError();
}

// sys_depth[s] = 1 + the deepest level of system s (zeroed by the caller)
__global__ void k_sys_depth(const int* __restrict__ depth, const int* __restrict__ sys_of, int n, int* sys_depth) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n; r += stride)
    atomicMax(&sys_depth[sys_of[r]], depth[r] + 1);
}
cudaError_t launch_sys_depth(const int* depth, const int* sys_of, int n, int* sys_depth, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_sys_depth<<<grid_for(n), kThreads, 0, s>>>(depth, sys_of, n, sys_depth);
  return cudaGetLastError();
}

__global__ void k_long_keys(const int* __restrict__ rows, const int* __restrict__ in_degree, int n, int threshold,
                            unsigned* keys) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride)
    keys[i] = in_degree[rows[i]] - 1 > threshold ? 0u : 1u;
}
cudaError_t launch_long_keys(const int* rows, const int* in_degree, int n, int threshold, unsigned* keys,
                             cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_long_keys<<<grid_for(n), kThreads, 0, s>>>(rows, in_degree, n, threshold, keys);
  return cudaGetLastError();
}

__global__ void k_inverse_perm(const int* __restrict__ perm, int n, int* iperm) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += stride)
    iperm[perm[p]] = static_cast<int>(p);
}
cudaError_t launch_inverse_perm(const int* perm, int n, int* iperm, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_inverse_perm<<<grid_for(n), kThreads, 0, s>>>(perm, n, iperm);
  return cudaGetLastError();
}

__global__ void k_dep_counts(const int* __restrict__ perm, const int* __restrict__ in_degree, int n, int* counts) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += stride)
    counts[p] = in_degree[perm[p]] - 1;
}
cudaError_t launch_dep_counts(const int* perm, const int* in_degree, int n, int* counts, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_dep_counts<<<grid_for(n), kThreads, 0, s>>>(perm, in_degree, n, counts);
  return cudaGetLastError();
}

__global__ void k_out_counts(const int* __restrict__ perm, const int* __restrict__ col_ptr, int n, int* counts) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += stride) {
    const int c = perm[p];
    counts[p] = col_ptr[c + 1] - col_ptr[c] - 1;
  }
}
cudaError_t launch_out_counts(const int* perm, const int* col_ptr, int n, int* counts, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_out_counts<<<grid_for(n), kThreads, 0, s>>>(perm, col_ptr, n, counts);
  return cudaGetLastError();
}

// Dependencies of position p in the order the serial executor accumulates
// them: ascending column for a forward solve, descending for a backward one
// (SpTRSV_cuda/sptrsv_syncfree_serialref.h:76-103 and :105-133).
__global__ void k_fill_pull(const int* __restrict__ perm, const int* __restrict__ iperm,
                            const int* __restrict__ csr_ptr, const int* __restrict__ csr_col,
                            const int* __restrict__ csr_src, const int* __restrict__ dep_ptr, int n,
                            SysDesc sd, int* dep_pos, int* dep_src, int* dep_col, int* diag_src) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += stride) {
    const int r = perm[p];
    const int substitution = dir_of(sd, r);
    const int beg = csr_ptr[r], end = csr_ptr[r + 1];
    int out = dep_ptr[p];
    if (substitution == 0) {
      for (int k = beg; k < end - 1; ++k, ++out) {
        dep_pos[out] = iperm[csr_col[k]];
        dep_src[out] = csr_src[k];
        dep_col[out] = csr_col[k];
      }
      diag_src[p] = csr_src[end - 1];
    } else {
      for (int k = end - 1; k > beg; --k, ++out) {
        dep_pos[out] = iperm[csr_col[k]];
        dep_src[out] = csr_src[k];
        dep_col[out] = csr_col[k];
      }
      diag_src[p] = csr_src[beg];
    }
  }
}
cudaError_t launch_fill_pull(const int* perm, const int* iperm, const int* csr_ptr, const int* csr_col,
                             const int* csr_src, const int* dep_ptr, int n, const SysDesc& sd, int* dep_pos,
                             int* dep_src, int* dep_col, int* diag_src, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_fill_pull<<<grid_for(n), kThreads, 0, s>>>(perm, iperm, csr_ptr, csr_col, csr_src, dep_ptr, n, sd,
                                                dep_pos, dep_src, dep_col, diag_src);
  return cudaGetLastError();
}

// Dependents of position p (its column's off-diagonal entries), listed in the
// order the serial executor run on the transpose accumulates them: descending
// row for a lower triangle (its transpose is solved backward), ascending for an
// upper one. The push executor is order-agnostic; the adjoint solve relies on it.
__global__ void k_fill_push(const int* __restrict__ perm, const int* __restrict__ iperm,
                            const int* __restrict__ col_ptr, const int* __restrict__ row_idx,
                            const int* __restrict__ out_ptr, int n, SysDesc sd, int* out_pos, int* out_src) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += stride) {
    const int c = perm[p];
    const int substitution = dir_of(sd, c);
    int out = out_ptr[p];
    if (substitution == 0) {
      for (int e = col_ptr[c + 1] - 1; e > col_ptr[c]; --e, ++out) {
        out_pos[out] = iperm[row_idx[e]];
        out_src[out] = e;
      }
    } else {
      for (int e = col_ptr[c]; e < col_ptr[c + 1] - 1; ++e, ++out) {
        out_pos[out] = iperm[row_idx[e]];
        out_src[out] = e;
      }
    }
  }
}
cudaError_t launch_fill_push(const int* perm, const int* iperm, const int* col_ptr, const int* row_idx,
                             const int* out_ptr, int n, const SysDesc& sd, int* out_pos, int* out_src,
                             cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_fill_push<<<grid_for(n), kThreads, 0, s>>>(perm, iperm, col_ptr, row_idx, out_ptr, n, sd, out_pos,
                                                out_src);
  return cudaGetLastError();
}

// ------------------------------------------------------------ value staging
template <typename TV>
__device__ __forceinline__ TV value_at(const TV* val, int i) {
  return __ldg(val + i);
}
__device__ __forceinline__ float value_at(const LatestValues& val, int i) {
  return *val.latest ? val.f32[i] : static_cast<float>(val.f64[i]);
}

// Gathers the values of one list set (out[e] = val[src[e]], scaled by the
// reciprocal of the owning position's diagonal for SCALE: x_p = b_p/d_p - sum_j
// w_j x_j then needs one fused multiply-add per dependency). DIAG first stages
// the diagonal and its reciprocal of the same positions; `flags` (a word of
// pinned host memory, or null) is set to SF_ZERO_DIAG on a zero or non-finite one.
//
// A warp takes 32 positions at a time: their lists are one contiguous range, so
// its lanes walk entries, coalesced, and find an entry's owner among the 32 list
// starts they hold by a binary search over shuffles. Bound by the gather of
// 8-byte values from 32-byte sectors. (One thread per list, as before, strides
// its loads and stores over 32 lists: the 5M-entry band system's pull weights
// took 66 us, the FP64 diagonal 11 more; with the copy of the values into the handle
// and the checks, all of set_values takes 90 us now.)
template <typename Source, typename T, bool DIAG, bool SCALE>
__global__ void __launch_bounds__(256) k_stage_lists(const int* __restrict__ ptr, const int* __restrict__ src,
                                                     const Source val, const int* __restrict__ diag_src, T* diag,
                                                     T* rcp, T* out, int n, int* flags, int* latest) {
  using TV = decltype(value_at(val, 0));
  constexpr unsigned kFull = 0xffffffffu;
  if (DIAG && latest && blockIdx.x == 0 && threadIdx.x == 0) *latest = sizeof(TV) == 4;
  constexpr int U = 4;
  const int lane = threadIdx.x & 31;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long groups = ((long long)n + 31) / 32;
  for (long long g = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; g < groups; g += nwarps) {
    const long long p = g * 32 + lane;
    T r = T(0);
    int start = INT_MAX, end = 0;
    if (p < n) {
      start = ptr[p];
      end = ptr[p + 1];
      if (DIAG) {
        const T d = static_cast<T>(value_at(val, diag_src[p]));
        r = T(1) / d;
        diag[p] = d;
        rcp[p] = r;
        if (flags && (!(d != T(0)) || !isfinite(d))) *reinterpret_cast<volatile int*>(flags) = SF_ZERO_DIAG;
      } else if (SCALE) {
        r = rcp[p];
      }
    }
    if (!out) continue;
    // entry indices as unsigned: a batch may reach past the last entry a 32-bit count can hold
    const unsigned lo = static_cast<unsigned>(__shfl_sync(kFull, start, 0));
    const unsigned hi = static_cast<unsigned>(__reduce_max_sync(kFull, end));
    for (unsigned base = lo; base < hi; base += 32 * U) {
      TV v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned e = base + u * 32 + lane;
        v[u] = e < hi ? value_at(val, src[e]) : TV(0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned e = base + u * 32 + lane;
        T w = static_cast<T>(v[u]);
        if (SCALE) {
          // the last list that starts at or before e owns it (empty lists share
          // their successor's start)
          int own = 0;
#pragma unroll
          for (int step = 16; step > 0; step >>= 1) {
            const int t = __shfl_sync(kFull, start, own + step);
            if (static_cast<unsigned>(t) <= e) own += step;
          }
          w *= __shfl_sync(kFull, r, own);
        }
        if (e < hi) out[e] = w;
      }
    }
  }
}

template <typename Source, typename T>
cudaError_t launch_stage_values(const Layout& L, Source val, Values<T>& V, unsigned forms, int* flags, cudaStream_t s,
                                int* latest) {
  if (L.n <= 0) return cudaSuccess;
  const int grid = grid_for(L.n);
  const bool dep = (forms & FORM_DEP_W) && L.ndep > 0;
  // the diagonal with the pull weights where both are wanted
  if (forms & FORM_DIAG) {
    k_stage_lists<Source, T, true, true><<<grid, kThreads, 0, s>>>(L.dep_ptr, L.dep_src_f, val, L.diag_src, V.diag,
                                                                   V.rcp, dep ? V.dep_w : nullptr, L.n, flags, latest);
  } else if (dep) {
    k_stage_lists<Source, T, false, true><<<grid, kThreads, 0, s>>>(L.dep_ptr, L.dep_src_f, val, nullptr, nullptr,
                                                                    V.rcp, V.dep_w, L.n, nullptr, nullptr);
  }
  if (L.ndep > 0) {
    if (forms & FORM_OUT_W)
      k_stage_lists<Source, T, false, true><<<grid, kThreads, 0, s>>>(L.out_ptr, L.out_src_f, val, nullptr, nullptr,
                                                                      V.rcp, V.out_w, L.n, nullptr, nullptr);
    if (forms & FORM_DEP_VAL)
      k_stage_lists<Source, T, false, false><<<grid, kThreads, 0, s>>>(L.dep_ptr, L.dep_src, val, nullptr, nullptr,
                                                                       nullptr, V.dep_val, L.n, nullptr, nullptr);
    if (forms & FORM_OUT_VAL)
      k_stage_lists<Source, T, false, false><<<grid, kThreads, 0, s>>>(L.out_ptr, L.out_src, val, nullptr, nullptr,
                                                                       nullptr, V.out_val, L.n, nullptr, nullptr);
  }
  if constexpr (sizeof(T) == 8)
    if (forms & FORM_DEP_SPLIT) return launch_split_weights(V.dep_w, L.ndep, V.dep_split, s);
  return cudaGetLastError();
}

template cudaError_t launch_stage_values<const double*, double>(const Layout&, const double*, Values<double>&,
                                                                 unsigned, int*, cudaStream_t, int*);
template cudaError_t launch_stage_values<const double*, float>(const Layout&, const double*, Values<float>&,
                                                                unsigned, int*, cudaStream_t, int*);
template cudaError_t launch_stage_values<const float*, float>(const Layout&, const float*, Values<float>&, unsigned,
                                                               int*, cudaStream_t, int*);
template cudaError_t launch_stage_values<LatestValues, float>(const Layout&, LatestValues, Values<float>&, unsigned,
                                                              int*, cudaStream_t, int*);

}  // namespace sptrsv
