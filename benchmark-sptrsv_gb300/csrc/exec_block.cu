// Blocked layouts (deep, narrow DAGs such as a mesh triangle): the walks over short
// lists for one right-hand side (k_pull_block), and the tables of the units, built on
// the device.
//
// A unit is one CTA's work, and a solve costs its levels times what one level
// takes, plus a hop from unit to unit. With lockstep lanes that poll for their
// dependencies (k_pull_wsync_imp) an iteration carries polls, votes and divergent
// multiply-adds, ~600 cycles. k_pull_block has one consumer warp walk the unit's
// levels in order, 32 unknowns of one level at a time, so every dependency inside
// the unit is there when it is read: a level is U loads from shared memory, U
// multiply-adds (64 cycles each in FP64) and a store. Everything else is taken off
// that warp:
//   12 loader warps bring the segments' first terms, weights and addresses into a
//     ring in shared memory, wait for dependencies on other units and fold them
//     in (they come first in ready order). They sit on the other three
//     sub-partitions (warp index mod 4), where an FP64 product does not hold the
//     consumer's pipe;
//   2 storer warps write the value words that other units poll, and x.
// The consumer takes the next segment's operands early if they are there and does
// not wait for them before its own level is out. With 9 loaders the 2M-row mesh
// takes 729 us (its lists no longer come from L2), with one storer 1,088.
//
// Whole solves, before (k_pull_wsync_imp) and after: meshes of 300 x 300 185 and
// 141 us, 1000 x 1000 592 and 447, 1414 x 1414 860 and 664 (FP32 635 and 495),
// 300 x 3000 1,071 and 738; transposed (k_pull_wsync before) 300 x 300 323 and 140,
// 1000 x 1000 1,061 and 446, 1414 x 1414 1,512 and 677.
#include <algorithm>
#include <climits>

#include "exec_common.cuh"
#include "internal.h"

namespace sptrsv {

namespace {

constexpr int kBlockThreads = 512;
constexpr int kStorers = 2;   // warps 4 and 8
constexpr int kLoaders = 12;  // warps 1-3, 5-7, 9-11, 13-15
constexpr int kRing = 16;     // segments the loaders may be ahead (a power of two)

template <typename T>
struct BlockArgs {
  int nunits, width;
  const int* unit;      // [nunits+1] first position
  const int* useg;      // [nunits+1] first segment
  const int* seg;       // [segments+1] first position
  const int* perm;
  const int* dep_ptr;
  const int* dep_pos;   // ready order
  const T* w;
  const T* rcp;
  const T* b;
  T* x;
  T* xw;
  DeviceCtl* ctl;
  unsigned long long timeout_ns;
};

__device__ __forceinline__ int ld_acquire_shared(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared.s32 %0, [%1];"
               : "=r"(v)
               : "r"(static_cast<unsigned>(__cvta_generic_to_shared(p)))
               : "memory");
  return v;
}
__device__ __forceinline__ void st_release_shared(int* p, int v) {
  asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(p))), "r"(v)
               : "memory");
}
__device__ __forceinline__ double ld_word(unsigned a, double) {
  double v;
  asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float ld_word(unsigned a, float) {
  float v;
  asm volatile("ld.volatile.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_word(unsigned a, double v) {
  asm volatile("st.volatile.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_word(unsigned a, float v) {
  asm volatile("st.volatile.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// multiply-adds that stay where they are written among the shared-memory accesses
__device__ __forceinline__ void fma_here(double& acc, double a, double b) {
  asm volatile("fma.rn.f64 %0, %1, %2, %0;" : "+d"(acc) : "d"(a), "d"(b));
}
__device__ __forceinline__ void fma_here(float& acc, float a, float b) {
  asm volatile("fma.rn.f32 %0, %1, %2, %0;" : "+f"(acc) : "f"(a), "f"(b));
}

// One segment's operands, 32 lanes: the first term with the imported
// dependencies taken off it, and for the others negated weight and shared-memory
// address; dst = address of the result (lanes without an unknown read the zero
// word and write the spare one).
template <typename T, int U>
struct RingSlot {
  T acc[32];
  T w[U][32];
  unsigned src[U][32];
  unsigned dst[32];
};

// ADJ: the transposed walk, units and segments from the last to the first over the
// lists of dependents.
template <typename T, int U, bool ADJ>
__global__ void __launch_bounds__(kBlockThreads) k_pull_block(BlockArgs<T> a) {
  using F = Flag<T>;
  using Bits = typename F::Bits;
  constexpr unsigned kFull = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto* ring = reinterpret_cast<RingSlot<T, U>*>(smem_raw);
  T* s_x = reinterpret_cast<T*>(ring + kRing);  // [width] unit, zero, spare
  const unsigned s_xa = static_cast<unsigned>(__cvta_generic_to_shared(s_x));
  __shared__ unsigned s_chunk;
  __shared__ int s_ready[kRing];  // 1 + the segment a ring slot holds
  __shared__ int s_done;          // segments the consumer is through with
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned zero = s_xa + (unsigned)a.width * (unsigned)sizeof(T), spare = zero + (unsigned)sizeof(T);
  for (;;) {
    const unsigned c = next_chunk(a.ctl, a.nunits, &s_chunk);
    if (c >= (unsigned)a.nunits) break;
    const int unit = ADJ ? a.nunits - 1 - (int)c : (int)c;
    const int base = a.unit[unit], end = ADJ ? a.unit[unit + 1] : 0, nseg = a.useg[unit + 1] - a.useg[unit];
    // first position of the k-th segment, first past it
    const int g0 = ADJ ? a.useg[unit + 1] - 1 : a.useg[unit];
    auto lo_of = [&](int k) { return a.seg[ADJ ? g0 - k : g0 + k]; };
    auto hi_of = [&](int k) { return a.seg[(ADJ ? g0 - k : g0 + k) + 1]; };
    auto other_unit = [&](int q) { return ADJ ? q >= end && q != INT_MAX : q < base; };
    if (threadIdx.x < kRing) s_ready[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
      s_done = 0;
      s_x[a.width] = T(0);
    }
    __syncthreads();
    bool fail = false;
    WaitBudget wb(a.timeout_ns);
    unsigned idle = 0u;
    // false once the wait must end; the first failure of any warp ends the others' waits too
    auto keep_waiting = [&]() {
      if ((++idle & 63u) == 0u && __any_sync(kFull, !wb.poll<true>(a.ctl, base))) fail = true;
      return !fail;
    };
    // whether the consumer is through with `count` segments, seen by every lane (each
    // looks for itself, a vote keeps the warp together; one lane's look and a shuffle
    // take the 2M-row mesh 666 instead of 663 us)
    auto consumed = [&](int count) { return __all_sync(kFull, ld_acquire_shared(&s_done) >= count); };
    if (warp == 0) {
      T acc = T(0), w[U];
      unsigned src[U], dst = spare;
      auto take = [&](int k) {  // segment k from the ring
        const RingSlot<T, U>& r = ring[k & (kRing - 1)];
        acc = r.acc[lane];
        dst = r.dst[lane];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          w[u] = r.w[u][lane];
          src[u] = r.src[u][lane];
        }
      };
      int loaded = 0;  // segments known to be in the ring
      auto look = [&](int k) {  // one look at all its slots
        const int s = k + lane;
        const bool in = lane < kRing && s < nseg && ld_acquire_shared(&s_ready[s & (kRing - 1)]) == s + 1;
        loaded = k + __ffs(~__ballot_sync(kFull, in)) - 1;
        __syncwarp();  // every lane reads slots whose flag another one acquired
        return loaded > k;
      };
      auto wait_loaded = [&](int k) {
        wb.start = 0;  // the budget is a single wait's
        while (!look(k))
          if (!keep_waiting()) break;
      };
      if (nseg > 0) {
        wait_loaded(0);
        if (!fail) take(0);
      }
      for (int k = 0; k < nseg && !fail; ++k) {
        T cur = acc, cw[U], v[U];
        const unsigned to = dst;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          cw[u] = w[u];
          v[u] = ld_word(src[u], T(0));
        }
        // the next segment's operands, if they are there, while the products run
        fma_here(cur, cw[0], v[0]);
        const bool have = k + 1 < nseg && (loaded > k + 1 || look(k + 1));
        if (have) take(k + 1);
#pragma unroll
        for (int u = 1; u < U; ++u) fma_here(cur, cw[u], v[u]);
        st_word(to, cur);
        __syncwarp();
        st_release_shared(&s_done, k + 1);
        if (!have && k + 1 < nseg) {
          wait_loaded(k + 1);
          if (!fail) take(k + 1);
        }
      }
    } else if (warp % 4 == 0) {
      // results out: the value words other units poll, and x. Rows are loaded one
      // of this warp's segments ahead, segment bounds two (used as loaded only, so
      // that nothing waits for them here)
      const int k0 = warp / 4 <= kStorers ? warp / 4 - 1 : nseg;
      int n_lo = 0, n_hi = 0, b_lo = 0, b_hi = 0, n_row = 0;
      auto bounds = [&](int k) {
        if (k >= nseg) return;
        b_lo = lo_of(k);
        b_hi = hi_of(k);
      };
      auto fetch = [&]() {
        n_lo = b_lo;
        n_hi = b_hi;
        if (n_lo + lane < n_hi) n_row = a.perm[n_lo + lane];
      };
      bounds(k0);
      fetch();
      bounds(k0 + kStorers);
      for (int k = k0; k < nseg; k += kStorers) {
        const int p = n_lo + lane, hi = n_hi, row = n_row;
        if (k + kStorers < nseg) fetch();
        bounds(k + 2 * kStorers);
        wb.start = 0;
        while (!consumed(k + 1))
          if (!keep_waiting()) break;
        if (fail) break;
        if (p < hi) {
          const T v = ld_word(s_xa + (unsigned)(p - base) * (unsigned)sizeof(T), T(0));
          F::store(&a.xw[p], v);
          a.x[row] = v;
        }
      }
    } else {
      for (int k = warp / 4 * 3 + warp % 4 - 1; k < nseg; k += kLoaders) {
        const int p = lo_of(k) + lane, hi = hi_of(k);
        T acc = T(0), w[U];
        unsigned src[U];
        int q[U];
        Bits v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          w[u] = T(0);
          src[u] = zero;
          q[u] = INT_MAX;
          v[u] = 0;
        }
        if (p < hi) {
          const int e = a.dep_ptr[p], e1 = a.dep_ptr[p + 1], row = a.perm[p];
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (e + u < e1) {
              w[u] = a.w[e + u];
              q[u] = a.dep_pos[e + u];
            }
          acc = a.b[row] * a.rcp[p];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (other_unit(q[u])) v[u] = F::load(&a.xw[q[u]]);
            else if (q[u] != INT_MAX) src[u] = s_xa + (unsigned)(q[u] - base) * (unsigned)sizeof(T);
          }
        }
        unsigned imported[U];
#pragma unroll
        for (int u = 0; u < U; ++u) imported[u] = __ballot_sync(kFull, other_unit(q[u]));
        wb.start = 0;
        while (!consumed(k + 1 - kRing))
          if (!keep_waiting()) break;
        if (fail) break;
        RingSlot<T, U>& r = ring[k & (kRing - 1)];
        r.dst[lane] = p < hi ? s_xa + (unsigned)(p - base) * (unsigned)sizeof(T) : spare;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          r.w[u][lane] = other_unit(q[u]) ? -T(0) : -w[u];  // -0 x 0 added changes no value
          r.src[u][lane] = src[u];
        }
        // imported dependencies come first in ready order
        wb.start = 0;
        for (;;) {
          bool pending = false;
#pragma unroll
          for (int u = 0; u < U; ++u) pending = pending || (other_unit(q[u]) && v[u] == F::EMPTY);
          if (!__any_sync(kFull, pending)) break;
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (other_unit(q[u]) && v[u] == F::EMPTY) v[u] = F::load(&a.xw[q[u]]);
          if (!keep_waiting()) break;
        }
        if (fail) break;
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (imported[u])
            if (other_unit(q[u])) acc = fma(-w[u], F::value(v[u]), acc);
        r.acc[lane] = acc;
        __syncwarp();
        if (lane == 0) st_release_shared(&s_ready[k & (kRing - 1)], k + 1);
      }
    }
    if (__syncthreads_or(fail)) break;
  }
  leave(a.ctl);
}

// ------------------------------------------------------------------ tables
// The unit position p lies in.
__device__ __forceinline__ int unit_of(const int* unit, int nunits, int p) {
  int lo = 0, hi = nunits - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (unit[mid] <= p) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Slots of in-unit dependencies; the others are counted, and with `ext` given
// listed in any order as (position, unit, entry).
__global__ void k_import_split(const int* __restrict__ ptr, const int* __restrict__ pos, int n,
                               const int* __restrict__ unit, int nunits, int* dep_slot, int* count, unsigned* ext_q,
                               int* ext_u, int* ext_e) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += stride) {
    const int u = unit_of(unit, nunits, static_cast<int>(p)), base = unit[u];
    for (int e = ptr[p]; e < ptr[p + 1]; ++e) {
      const int q = pos[e];
      if (q >= base) {
        if (!ext_q) dep_slot[e] = q - base;
        continue;
      }
      const int at = atomicAdd(count, 1);
      if (ext_q) {
        ext_q[at] = static_cast<unsigned>(q);
        ext_u[at] = u;
        ext_e[at] = e;
      }
    }
  }
}
__global__ void k_gather_keys(const int* __restrict__ src, const int* __restrict__ idx, int count, unsigned* keys) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += stride)
    keys[i] = static_cast<unsigned>(src[idx[i]]);
}
// flag[i] = 1 where the (unit, position) pair differs from the one before it
__global__ void k_import_flags(const unsigned* __restrict__ su, const unsigned* __restrict__ q,
                               const int* __restrict__ idx, int count, int* flag) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += stride)
    flag[i] = i == 0 || su[i] != su[i - 1] || q[idx[i]] != q[idx[i - 1]] ? 1 : 0;
}
// im_ptr[u] = first import of unit u (rank[i] = pairs before i, rank[count] = all of them)
__global__ void k_import_starts(const unsigned* __restrict__ su, const int* __restrict__ rank, int count, int nunits,
                                int* im_ptr) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u > nunits) return;
  int lo = 0, hi = count;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (su[mid] < static_cast<unsigned>(u)) lo = mid + 1;
    else hi = mid;
  }
  im_ptr[u] = rank[lo];
}
__global__ void k_import_fill(const unsigned* __restrict__ su, const unsigned* __restrict__ q,
                              const int* __restrict__ ext_e, const int* __restrict__ idx, const int* __restrict__ rank,
                              const int* __restrict__ im_ptr, int count, int width, int* im_q, int* dep_slot) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += stride) {
    const int g = rank[i + 1] - 1;  // the pair i belongs to
    im_q[g] = static_cast<int>(q[idx[i]]);
    dep_slot[ext_e[idx[i]]] = width + g - im_ptr[su[i]];
  }
}

// Segments of a unit: runs of at most 32 consecutive positions of one level. One
// warp per unit; first pass (seg null) counts them, and the levels of all units.
__global__ void k_unit_segments(const int* __restrict__ perm, const int* __restrict__ depth,
                                const int* __restrict__ unit, int nunits, const int* __restrict__ first, int* count,
                                int* levels, int* seg) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (u >= nunits) return;
  const int base = unit[u], end = unit[u + 1];
  int total = 0, runs = 0, run = base, before = -1;  // start of the level's run, level of the position before
  for (int p0 = base; p0 < end; p0 += 32) {
    const int p = p0 + lane;
    const int d = p < end ? depth[perm[p]] : -1;
    int prev = __shfl_up_sync(kFull, d, 1);
    if (lane == 0) prev = before;
    const unsigned changes = __ballot_sync(kFull, p < end && d != prev);
    const unsigned upto = changes & ((2u << lane) - 1u);
    const int start = upto ? p0 + 31 - __clz(upto) : run;
    const bool opens = p < end && ((p - start) & 31) == 0;
    const unsigned opening = __ballot_sync(kFull, opens);
    if (seg && opens) seg[first[u] + total + __popc(opening & ((1u << lane) - 1u))] = p;
    total += __popc(opening);
    runs += __popc(changes);
    if (changes) run = p0 + 31 - __clz(changes);
    before = __shfl_sync(kFull, d, 31);
  }
  if (!seg && lane == 0) {
    count[u] = total;
    atomicAdd(levels, runs);
  }
}

inline int grid_1d(long long count) { return static_cast<int>(std::min<long long>((count + 255) / 256, 1 << 20)); }

}  // namespace

cudaError_t launch_import_split(const Layout& L, const int* unit, int nunits, int* dep_slot, int* count,
                                unsigned* ext_q, int* ext_u, int* ext_e, cudaStream_t s) {
  if (L.n <= 0) return cudaSuccess;
  k_import_split<<<grid_1d(L.n), 256, 0, s>>>(L.dep_ptr, L.dep_pos_f, L.n, unit, nunits, dep_slot, count, ext_q, ext_u,
                                              ext_e);
  return cudaGetLastError();
}

cudaError_t launch_import_tables(const unsigned* ext_q, const int* ext_u, const int* ext_e, int count, int n,
                                 int nunits, int width, int* im_ptr, int* im_q, int* dep_slot, cudaStream_t s) {
  if (count <= 0) return cudaMemsetAsync(im_ptr, 0, sizeof(int) * ((size_t)nunits + 1), s);
  auto bits = [](int v) {
    int b = 1;
    while (b < 31 && (1 << b) <= v) ++b;
    return b;
  };
  unsigned *keys = nullptr, *sorted = nullptr;
  int *iota = nullptr, *by_q = nullptr, *idx = nullptr, *rank = nullptr;
  void* temp = nullptr;
  auto run = [&]() -> cudaError_t {
    cudaError_t e;
    const size_t bytes = sizeof(int) * (size_t)count;
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&keys), bytes, s)) != cudaSuccess) return e;
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&sorted), bytes, s)) != cudaSuccess) return e;
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&iota), bytes, s)) != cudaSuccess) return e;
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&by_q), bytes, s)) != cudaSuccess) return e;
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&idx), bytes, s)) != cudaSuccess) return e;
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&rank), bytes + sizeof(int), s)) != cudaSuccess) return e;
    if ((e = cudaMallocAsync(&temp, radix_sort_temp_bytes(count), s)) != cudaSuccess) return e;
    // by position, then (stable) by unit
    if ((e = launch_iota(iota, count, 0, 1, s)) != cudaSuccess) return e;
    if ((e = radix_sort_pairs(ext_q, iota, sorted, by_q, count, bits(n - 1), temp, s)) != cudaSuccess) return e;
    k_gather_keys<<<grid_1d(count), 256, 0, s>>>(ext_u, by_q, count, keys);
    if ((e = radix_sort_pairs(keys, by_q, sorted, idx, count, bits(nunits - 1), temp, s)) != cudaSuccess) return e;
    k_import_flags<<<grid_1d(count), 256, 0, s>>>(sorted, ext_q, idx, count, rank);
    if ((e = exclusive_scan_int(rank, rank, count, true, s)) != cudaSuccess) return e;
    k_import_starts<<<(nunits + 256) / 256, 256, 0, s>>>(sorted, rank, count, nunits, im_ptr);
    k_import_fill<<<grid_1d(count), 256, 0, s>>>(sorted, ext_q, ext_e, idx, rank, im_ptr, count, width, im_q, dep_slot);
    return cudaGetLastError();
  };
  const cudaError_t e = run();
  for (void* b : {(void*)keys, (void*)sorted, (void*)iota, (void*)by_q, (void*)idx, (void*)rank, temp})
    if (b) cudaFreeAsync(b, s);
  return e;
}

cudaError_t launch_level_walk(const int* perm, const int* depth, int n, int nlevels, int* walk, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  unsigned *keys = nullptr, *sorted = nullptr;
  int* iota = nullptr;
  void* temp = nullptr;
  int bits = 1;
  while (bits < 31 && (1 << bits) < nlevels) ++bits;
  const size_t bytes = sizeof(int) * (size_t)n;
  cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&keys), bytes, s);
  if (e == cudaSuccess) e = cudaMallocAsync(reinterpret_cast<void**>(&sorted), bytes, s);
  if (e == cudaSuccess) e = cudaMallocAsync(reinterpret_cast<void**>(&iota), bytes, s);
  if (e == cudaSuccess) e = cudaMallocAsync(&temp, radix_sort_temp_bytes(n), s);
  if (e == cudaSuccess) e = launch_iota(iota, n, 0, 1, s);
  if (e == cudaSuccess) {
    k_gather_keys<<<grid_1d(n), 256, 0, s>>>(depth, perm, n, keys);
    e = radix_sort_pairs(keys, iota, sorted, walk, n, bits, temp, s);
  }
  for (void* b : {(void*)keys, (void*)sorted, (void*)iota, temp})
    if (b) cudaFreeAsync(b, s);
  return e;
}

cudaError_t launch_unit_segments(const int* perm, const int* depth, const int* unit, int nunits, const int* first,
                                 int* count, int* levels, int* seg, cudaStream_t s) {
  if (nunits <= 0) return cudaSuccess;
  k_unit_segments<<<(nunits + 3) / 4, 128, 0, s>>>(perm, depth, unit, nunits, first, count, levels, seg);
  return cudaGetLastError();
}

namespace {
template <typename T>
size_t slot_bytes(int u) {
  return u == 1 ? sizeof(RingSlot<T, 1>) : (u == 2 ? sizeof(RingSlot<T, 2>) : (u == 3 ? sizeof(RingSlot<T, 3>) : sizeof(RingSlot<T, 4>)));
}
}  // namespace

template <typename T>
size_t block_smem_bytes(int width, int longest) {
  return slot_bytes<T>(longest) * kRing + (size_t)(width + 2) * sizeof(T);
}
template size_t block_smem_bytes<double>(int, int);
template size_t block_smem_bytes<float>(int, int);

template <typename T>
cudaError_t launch_pull_block(const Layout& L, const Values<T>& V, const VecView<T>& v, T* xw, DeviceCtl* ctl,
                              const UnitTable& units, int longest, unsigned long long timeout_ns, int num_sms,
                              cudaStream_t s, bool adj) {
  if (L.n == 0) return cudaSuccess;
  BlockArgs<T> a{};
  a.nunits = units.count;
  a.width = units.width;
  a.unit = units.start;
  a.useg = units.seg_ptr;
  a.seg = units.seg;
  a.perm = L.perm;
  a.dep_ptr = adj ? L.out_ptr : L.dep_ptr;
  a.dep_pos = adj ? L.out_pos_f : L.dep_pos_f;
  a.w = adj ? V.out_w : V.dep_w;
  a.rcp = V.rcp;
  a.b = v.b;
  a.x = v.x;
  a.xw = xw;
  a.ctl = ctl;
  a.timeout_ns = timeout_ns;
  const size_t smem = block_smem_bytes<T>(units.width, longest);
  auto run = [&](auto kernel) -> cudaError_t {
    const cudaError_t e = allow_shared(kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<std::min(num_sms, a.nunits), kBlockThreads, smem, s>>>(a);
    return cudaGetLastError();
  };
  switch (longest) {
    case 1: return adj ? run(k_pull_block<T, 1, true>) : run(k_pull_block<T, 1, false>);
    case 2: return adj ? run(k_pull_block<T, 2, true>) : run(k_pull_block<T, 2, false>);
    case 3: return adj ? run(k_pull_block<T, 3, true>) : run(k_pull_block<T, 3, false>);
    case 4: return adj ? run(k_pull_block<T, 4, true>) : run(k_pull_block<T, 4, false>);
    default: return cudaErrorInvalidValue;
  }
}
template cudaError_t launch_pull_block<double>(const Layout&, const Values<double>&, const VecView<double>&, double*,
                                               DeviceCtl*, const UnitTable&, int, unsigned long long, int,
                                               cudaStream_t, bool);
template cudaError_t launch_pull_block<float>(const Layout&, const Values<float>&, const VecView<float>&, float*,
                                              DeviceCtl*, const UnitTable&, int, unsigned long long, int,
                                              cudaStream_t, bool);

}  // namespace sptrsv
