// Level-order executor with lists staged ahead, several right-hand sides.
//
// The loop of k_pull_ahead (exec_ahead.cu) for blocks: G lanes hold an unknown,
// each R adjacent right-hand sides (one two-word load per pair), and every lane
// walks the unknown's list on its own. The next chunk's lists are copied to
// shared memory with cp.async and its first terms loaded while the CTA works on
// the current one; the next entry's address is worked out while a poll is in
// flight, and finished lanes do not poll. Chunks are 256 / G unknowns, claimed
// two ahead, with a CTA barrier between them: it holds back the warps that
// would otherwise poll far ahead of the wave. As many CTAs per SM as fit: the
// lanes of a group poll adjacent words, so polls are cheap and throughput (one
// dependency per iteration and lane) counts.
//
// FP64, 500k-row band of 9 entries per column, k_pull_wsync_multi -> this kernel
// (forward / transposed, us): 2 right-hand sides 610 / 641 -> 430 / 495, 4 557 /
// 596 -> 365 / 444, 8 573 / 575 -> 375 / 484, 16 568 / 605 -> 472 / 565, 32 723 /
// 797 -> 602 / 724, 64 987 / 1,030 -> 945 / 1,018 (there the FP64 pipe: 20 M
// warp-wide multiply-adds per 1M rows hold it ~1.1 ms); FP32 at 64 840 / 829 ->
// 534 / 657.
#include <algorithm>

#include "exec_ahead.cuh"
#include "internal.h"

namespace sptrsv {

namespace {

template <typename T>
struct AheadMultiArgs {
  int n, rhs, nchunks, cap;
  const int* perm;
  const int* ptr;   // dependency lists in ready order (dependents, for the transposed walk)
  const int* pos;
  const T* w;
  const T* rcp;
  const T* b;
  T* x;
  long long b_si, b_sk, x_si, x_sk;
  T* xw;  // [n * rhs in whole lanes], position-major
  DeviceCtl* ctl;
  unsigned long long timeout_ns;
};

// How a block reaches the kernel: rows or columns of whole lanes; not whole lanes
// (words past the last right-hand side repeat it); rows of whole lanes that
// launch_columns_in made of a column-major block, scaled by the diagonal there, where
// memory is the bound (1M rows of 9 entries, 64 right-hand sides: 1,684 us here
// instead of 1,772; whole solves 2,148 -> 2,086, at 32 on 500k rows 682 -> 662, FP32
// 664 -> 638). Laid out like the value words the rows scatter: 90 us longer.
// kWalk: a blocked layout in level order, through `walk` (positions by level). Its
// lists come from global memory, every dependency from the value words.
enum { kWhole, kPad, kStaged, kWalk };

// G lanes per unknown, R adjacent right-hand sides per lane, 256 / G unknowns per
// chunk.
template <typename T, bool ADJ, int G, int R, int MODE>
__global__ void __launch_bounds__(256) k_pull_ahead_multi(AheadMultiArgs<T> a, int words, const int* walk) {
  using F = Flag<T>;
  using Bits = typename F::Bits;
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kUnknowns = 256 / G;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned s_ticket;
  T* s_win = reinterpret_cast<T*>(smem_raw);  // [kUnknowns * G * R] values of the chunk in hand
  T* s_w = s_win + kUnknowns * G * R;         // [2][cap]
  int* s_q = reinterpret_cast<int*>(s_w + 2 * a.cap);
  const unsigned s_wina = static_cast<unsigned>(__cvta_generic_to_shared(s_win));
  const unsigned s_wa = static_cast<unsigned>(__cvta_generic_to_shared(s_w));
  const unsigned s_qa = static_cast<unsigned>(__cvta_generic_to_shared(s_q));
  const int j = threadIdx.x / G, k = (threadIdx.x % G) * R;  // unknown of the chunk, first right-hand side
  const int last = a.n - 1, rhs = MODE == kWhole ? a.rhs : words;
  const bool col = k < rhs;
  // two chunks ahead: rows and list bounds
  int f_row = 0, f_e = 0, f_e1 = 0, f_lo = 0, f_hi = 0, f_p = 0;
  auto fetch = [&](int c) {
    f_e = f_e1 = f_lo = f_hi = 0;
    if (c >= a.nchunks) return;
    const int base = c * kUnknowns, end = min(base + kUnknowns, a.n);
    const int pr = base + j;
    if (pr < a.n) {
      const int p = MODE == kWalk ? walk[ADJ ? last - pr : pr] : (ADJ ? last - pr : pr);
      if (MODE == kWalk) f_p = p;
      f_row = a.perm[p];
      f_e = a.ptr[p];
      f_e1 = a.ptr[p + 1];
    }
    if (MODE == kWalk) return;  // no lists to stage
    f_lo = a.ptr[ADJ ? last - (end - 1) : base];
    f_hi = a.ptr[ADJ ? last - base + 1 : end];
  };
  // one chunk ahead: first terms, and the lists on their way to shared memory
  int n_row = 0, n_e = 0, n_e1 = 0, n_lo = 0, n_p = 0;
  T n_acc[R];
  auto stage = [&](int c, int buf) {
    n_row = f_row;
    n_e = f_e;
    n_e1 = f_e1;
    n_lo = f_lo;
    n_p = f_p;
    if (c >= a.nchunks) return;
    const int pr = c * kUnknowns + j;
    if (pr < a.n && col) {
      const int p = MODE == kWalk ? n_p : (ADJ ? last - pr : pr);
      if (MODE == kStaged) {
#pragma unroll
        for (int i = 0; i < R; ++i) n_acc[i] = a.b[(long long)n_row * rhs + k + i];
      } else {
        const T r = a.rcp[p];
#pragma unroll
        for (int i = 0; i < R; ++i)
          n_acc[i] = a.b[(long long)n_row * a.b_si + (long long)(MODE == kPad || MODE == kWalk ? min(k + i, a.rhs - 1) : k + i) * a.b_sk] * r;
      }
    }
    const int hi = min(f_hi, f_lo + a.cap);
    for (int e = f_lo + threadIdx.x; e < hi; e += 256) {
      copy_async(s_qa + (unsigned)(buf * a.cap + e - f_lo) * 4u, a.pos + e);
      copy_async(s_wa + (unsigned)(buf * a.cap + e - f_lo) * (unsigned)sizeof(T), a.w + e);
    }
  };
  // chunks are claimed two ahead; the earliest unfinished one is always in hand
  auto claim = [&]() {
    if (threadIdx.x == 0) s_ticket = ctl_failed(a.ctl) ? a.nchunks : atomicAdd(&a.ctl->ticket, 1u);
  };
  auto claimed = [&]() { return static_cast<int>(min(s_ticket, (unsigned)a.nchunks)); };
  claim();
  __syncthreads();
  int c = claimed();
  __syncthreads();
  claim();
  __syncthreads();
  int c1 = claimed();
  __syncthreads();
  claim();
  fetch(c);
  stage(c, 0);
  fetch(c1);
  for (int buf = 0; c < a.nchunks; buf ^= 1) {
    const int base = c * kUnknowns, pr = base + j;
    bool done = pr >= a.n || !col;
    const int p = MODE == kWalk ? n_p : (ADJ ? last - pr : pr);
    const int row = n_row, lo = n_lo;
    int e = n_e;
    const int e1 = n_e1;
    T acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      acc[i] = n_acc[i];
      *reinterpret_cast<volatile Bits*>(&s_win[threadIdx.x * R + i]) = F::EMPTY;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int c2 = claimed();
    stage(c1, buf ^ 1);
    fetch(c2);
    const T* lw = s_w + buf * a.cap - lo;
    const int* lq = s_q + buf * a.cap - lo;
    const int hi = lo + a.cap;
    const T *word = a.xw, *nword = a.xw;
    unsigned local = s_wina, nlocal = s_wina;
    bool mine = true, nmine = true;
    T w = T(0), nw = T(0);
    int nq = 0;
    int left = e1 - e - 1;
    auto next = [&](int ee) {
      nq = MODE != kWalk && ee < hi ? lq[ee] : a.pos[ee];
      nw = MODE != kWalk && ee < hi ? lw[ee] : a.w[ee];
    };
    auto target = [&](int q) {
      const int off = (ADJ ? last - q : q) - base;
      nmine = MODE != kWalk && off >= 0;
      nlocal = s_wina + (unsigned)((off & (kUnknowns - 1)) * (G * R) + k) * (unsigned)sizeof(T);
      nword = a.xw + (long long)q * rhs + k;
    };
    auto publish = [&]() {
      Bits v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        v[i] = F::bits(acc[i]);
        F::store_shared(&s_win[threadIdx.x * R + i], acc[i]);
      }
      publish_words(&a.xw[(long long)p * rhs + k], v);
      done = true;
    };
    if (!done) {
      if (left < 0) {
        publish();
      } else {
        next(e);
        w = nw;
        target(nq);
        word = nword;
        local = nlocal;
        mine = nmine;
        if (left > 0) next(++e);
      }
    }
    bool fail = false;
    unsigned idle = 0u;
    int seen = 0;
    WaitBudget wb(a.timeout_ns);
    while (!__all_sync(kFull, done)) {
      Bits bits[R];
      poll_words(bits, local, word, mine, !done);
      target(nq);  // in the poll's shadow
      bool hit = true;
#pragma unroll
      for (int i = 0; i < R; ++i) hit = hit && bits[i] != F::EMPTY;
      if (hit) {
#pragma unroll
        for (int i = 0; i < R; ++i) acc[i] = fma(-w, F::value(bits[i]), acc[i]);
        if (left > 0) {
          w = nw;
          word = nword;
          local = nlocal;
          mine = nmine;
          if (--left > 0) next(++e);
        } else {
          publish();
        }
      }
      if ((++idle & 255u) == 0u) {
        // (a flag of its own keeps the padded quadruples within 64 registers, four CTAs per
        // SM: FP32, 33 right-hand sides on 1M rows 1,298 us without, 1,146 with it)
        bool lost = false;
        if (!lockstep_wait(wb, left - done, seen, MODE == kPad && R == 4 ? lost : fail, a.ctl, p)) {
          fail = true;
          break;
        }
      }
    }
    if (!fail && pr < a.n && col) {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (MODE == kStaged) a.x[(long long)row * rhs + k + i] = acc[i];
        else a.x[(long long)row * a.x_si + (long long)(MODE == kPad || MODE == kWalk ? min(k + i, a.rhs - 1) : k + i) * a.x_sk] = acc[i];
      }
    }
    if (__syncthreads_or(fail)) break;
    claim();
    c = c1;
    c1 = c2;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  leave(a.ctl);
}

}  // namespace

template <typename T, bool ADJ>
cudaError_t launch_ahead_multi(AheadMultiArgs<T>& a, int avg, bool narrow, int num_sms, cudaStream_t s, const int* walk) {
  const int words = ahead_multi_words(a.rhs, sizeof(T), narrow);
  auto run = [&](auto kernel, int g, int r) -> cudaError_t {
    const int unknowns = 256 / g;
    a.nchunks = (a.n + unknowns - 1) / unknowns;
    // twice the average chunk's lists (longer ones read the rest from global memory)
    a.cap = walk ? 0 : std::min(1024, std::max(64, (2 * avg * unknowns / 32 + 31) / 32 * 32));
    const size_t smem = (size_t)256 * r * sizeof(T) + (size_t)2 * a.cap * (sizeof(T) + sizeof(int));
    const cudaError_t e = allow_shared(kernel, smem);
    if (e != cudaSuccess) return e;
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 256, smem);
    if (per < 1) per = 1;
    const int grid = static_cast<int>(std::min<long long>((long long)num_sms * per, a.nchunks));
    kernel<<<grid, 256, smem, s>>>(a, words, walk);
    return cudaGetLastError();
  };
  // quadruples are FP32's, pairs over 32 lanes FP64's (forward, or along a level walk),
  // and a level walk starts at 9 right-hand sides in FP32 (ahead_multi_shape,
  // use_ahead_multi, use_level_walk)
  constexpr bool half = sizeof(T) == 4;
  const bool pad = a.rhs != words, staged = a.b_si == 0;
  const int shape = ahead_multi_shape(a.rhs, sizeof(T), narrow);
  if (walk) {
    switch (shape) {
      case 16 * 8 + 1: return run(k_pull_ahead_multi<T, ADJ, 16, 1, kWalk>, 16, 1);
      case 8 * 8 + 2: return run(k_pull_ahead_multi<T, ADJ, 8, 2, kWalk>, 8, 2);
      case 16 * 8 + 2: return run(k_pull_ahead_multi<T, ADJ, 16, 2, kWalk>, 16, 2);
    }
    if constexpr (half) {
      if (shape == 16 * 8 + 4) return run(k_pull_ahead_multi<T, ADJ, 16, 4, kWalk>, 16, 4);
    } else {
      if (shape == 8 * 8 + 1) return run(k_pull_ahead_multi<T, ADJ, 8, 1, kWalk>, 8, 1);
      if (shape == 32 * 8 + 2) return run(k_pull_ahead_multi<T, ADJ, 32, 2, kWalk>, 32, 2);
    }
    return cudaErrorInvalidValue;
  }
  switch (shape) {
    case 2 * 8 + 1: return run(k_pull_ahead_multi<T, ADJ, 2, 1, kWhole>, 2, 1);
    case 4 * 8 + 1: return run(k_pull_ahead_multi<T, ADJ, 4, 1, kWhole>, 4, 1);
    case 8 * 8 + 1: return run(k_pull_ahead_multi<T, ADJ, 8, 1, kWhole>, 8, 1);
    case 16 * 8 + 1: return run(k_pull_ahead_multi<T, ADJ, 16, 1, kWhole>, 16, 1);
    case 8 * 8 + 2:
      return pad ? run(k_pull_ahead_multi<T, ADJ, 8, 2, kPad>, 8, 2) : run(k_pull_ahead_multi<T, ADJ, 8, 2, kWhole>, 8, 2);
    case 16 * 8 + 2:
      return staged ? run(k_pull_ahead_multi<T, ADJ, 16, 2, kStaged>, 16, 2)
                    : (pad ? run(k_pull_ahead_multi<T, ADJ, 16, 2, kPad>, 16, 2)
                           : run(k_pull_ahead_multi<T, ADJ, 16, 2, kWhole>, 16, 2));
  }
  if constexpr (half) {
    if (shape == 16 * 8 + 4)
      return staged ? run(k_pull_ahead_multi<T, ADJ, 16, 4, kStaged>, 16, 4)
                    : (pad ? run(k_pull_ahead_multi<T, ADJ, 16, 4, kPad>, 16, 4)
                           : run(k_pull_ahead_multi<T, ADJ, 16, 4, kWhole>, 16, 4));
  } else if constexpr (!ADJ) {
    if (shape == 32 * 8 + 2)
      return staged ? run(k_pull_ahead_multi<T, ADJ, 32, 2, kStaged>, 32, 2)
                    : (pad ? run(k_pull_ahead_multi<T, ADJ, 32, 2, kPad>, 32, 2)
                           : run(k_pull_ahead_multi<T, ADJ, 32, 2, kWhole>, 32, 2));
  }
  return cudaErrorInvalidValue;
}

namespace {

// Columns of a right-hand-side block (n entries each) to rows of `words` first
// terms b / d, in 32 x 32 tiles through shared memory (whole lines on both sides).
// Zeros past the last right-hand side.
template <typename T>
__global__ void __launch_bounds__(256) k_columns_in(const T* __restrict__ b, const T* __restrict__ rcp,
                                                    const int* __restrict__ iperm, T* __restrict__ out, int n, int rhs,
                                                    int words) {
  __shared__ T tile[32][33];
  __shared__ T scale[32];
  const int r0 = blockIdx.x * 32, k0 = blockIdx.y * 32, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0 && r0 + lane < n) scale[lane] = rcp[iperm[r0 + lane]];
  if (r0 + lane < n) {
#pragma unroll
    for (int i = 0; i < 32; i += 8)
      tile[warp + i][lane] = k0 + warp + i < rhs ? b[(long long)(k0 + warp + i) * n + r0 + lane] : T(0);
  }
  __syncthreads();
#pragma unroll
  for (int i = warp; i < 32; i += 8)
    if (r0 + i < n && k0 + lane < words) out[(long long)(r0 + i) * words + k0 + lane] = tile[lane][i] * scale[i];
}
// The solution's columns from rows of `words` values.
template <typename T>
__global__ void __launch_bounds__(256) k_columns_out(const T* __restrict__ in, T* __restrict__ x, int n, int rhs,
                                                     int words) {
  __shared__ T tile[32][33];
  const int r0 = blockIdx.x * 32, k0 = blockIdx.y * 32, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = warp; i < 32; i += 8)
    if (r0 + i < n && k0 + lane < rhs) tile[lane][i] = in[(long long)(r0 + i) * words + k0 + lane];
  __syncthreads();
#pragma unroll
  for (int i = warp; i < 32; i += 8)
    if (r0 + lane < n && k0 + i < rhs) x[(long long)(k0 + i) * n + r0 + lane] = tile[i][lane];
}

}  // namespace

template <typename T>
cudaError_t launch_columns_in(const Layout& L, const Values<T>& V, const T* b, T* out, int rhs, int words,
                              cudaStream_t s) {
  if (L.n == 0) return cudaSuccess;
  k_columns_in<T><<<dim3((L.n + 31) / 32, (words + 31) / 32), 256, 0, s>>>(b, V.rcp, L.iperm, out, L.n, rhs, words);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_columns_out(const Layout& L, const T* in, T* x, int rhs, int words, cudaStream_t s) {
  if (L.n == 0) return cudaSuccess;
  k_columns_out<T><<<dim3((L.n + 31) / 32, (rhs + 31) / 32), 256, 0, s>>>(in, x, L.n, rhs, words);
  return cudaGetLastError();
}
template cudaError_t launch_columns_in<double>(const Layout&, const Values<double>&, const double*, double*, int, int,
                                               cudaStream_t);
template cudaError_t launch_columns_in<float>(const Layout&, const Values<float>&, const float*, float*, int, int,
                                              cudaStream_t);
template cudaError_t launch_columns_out<double>(const Layout&, const double*, double*, int, int, cudaStream_t);
template cudaError_t launch_columns_out<float>(const Layout&, const float*, float*, int, int, cudaStream_t);

template <typename T>
cudaError_t launch_pull_ahead_multi(const Layout& L, const Values<T>& V, int rhs, const VecView<T>& v, T* xw,
                                    DeviceCtl* ctl, bool narrow, unsigned long long timeout_ns, int num_sms,
                                    cudaStream_t s, bool adj, const int* walk) {
  if (L.n == 0) return cudaSuccess;
  AheadMultiArgs<T> a{};
  a.n = L.n;
  a.rhs = rhs;
  a.perm = L.perm;
  a.ptr = adj ? L.out_ptr : L.dep_ptr;
  a.pos = adj ? L.out_pos_f : L.dep_pos_f;
  a.w = adj ? V.out_w : V.dep_w;
  a.rcp = V.rcp;
  a.b = v.b;
  a.x = v.x;
  a.b_si = v.b_si;
  a.b_sk = v.b_sk;
  a.x_si = v.x_si;
  a.x_sk = v.x_sk;
  a.xw = xw;
  a.ctl = ctl;
  a.timeout_ns = timeout_ns;
  const int avg = static_cast<int>(32LL * L.ndep / L.n);
  return adj ? launch_ahead_multi<T, true>(a, avg, narrow, num_sms, s, walk)
             : launch_ahead_multi<T, false>(a, avg, narrow, num_sms, s, walk);
}
template cudaError_t launch_pull_ahead_multi<double>(const Layout&, const Values<double>&, int, const VecView<double>&,
                                                     double*, DeviceCtl*, bool, unsigned long long, int, cudaStream_t,
                                                     bool, const int*);
template cudaError_t launch_pull_ahead_multi<float>(const Layout&, const Values<float>&, int, const VecView<float>&,
                                                    float*, DeviceCtl*, bool, unsigned long long, int, cudaStream_t,
                                                    bool, const int*);

}  // namespace sptrsv
