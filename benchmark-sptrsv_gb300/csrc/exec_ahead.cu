// Level-order executor with lists staged ahead (one right-hand side).
//
// As k_pull_wsync: a warp takes 32 consecutive walk indices, one unknown per lane,
// and advances in lockstep; values are value-as-flag words in global memory.
// What a level costs is how long a lockstep iteration takes once its last
// dependency is published, and there a list entry fetched from global memory
// costs all 32 lanes its latency on top of the poll's. So the warp claims its
// segments by ticket one ahead (no CTA barrier between them) and copies the next
// segment's lists, one contiguous range, to shared memory with cp.async while it
// works on the current one. An iteration is then one poll (~285 cycles to L2)
// plus the multiply-add of the lanes that consumed. Dependencies inside the
// segment go through a 32-word window in shared memory. Lanes that are done do
// not poll: a poll of 32 scattered words holds the SM's load path for ~32 cycles,
// which the other warps' polls wait for, and a 128-byte line of L1 each, so the
// list buffers must leave L1 room (two CTAs with 107 KB of buffers each: 2,767 us
// on a split power-law walk, 2,127 with 86 KB).
//
// U = entries polled per iteration. One (the next entry's address is worked out
// during the poll) is the shortest iteration; two consume lists that have
// largely arrived twice as fast. Work per level, t = dependencies + 4 per unknown,
// decides how many lanes are needed (us, forward / transposed):
//   t < 21,000        one CTA per SM, U = 1 forward, 2 transposed: 1M-row band
//                     (9,700) 893 / 897, with U the other way 905 / 1,011; 200k rows
//                     of 40 entries (6,700) 1,010 / 1,084 vs 1,073 / 1,181
//   t <= 34,000       one CTA, U = 2: 4M-row power law (30,100) 1,363 forward, 1,459
//                     with U = 1, 1,403 with two CTAs; FP32, 25,000, 373 vs 410
//   t <= 120,000      two CTAs, U = 2: 2M-row band (49,700) 413 / 479, one CTA 496 / 548;
//                     2M rows of 9 entries (66,300) 393 / 493, three 409 / 580. But
//                     three where the lists leave L1 to the polls: FP32 of more than 6
//                     entries (the same 385 / 517, two 481 / 641), transposed FP64 of at
//                     most 6 (2M rows of 4, 38,900, 456, two 605; 2M of 6, 101,000, 335,
//                     two 439), and from 90,000 on at most 6 (the same 277, two 346);
//                     and one transposed where a segment is longer than two CTAs' buffers
//                     (1M rows of 20, 40,700, 704, two 726; FP32 678, two 1,060)
//   beyond            three CTAs: 4M rows of 4 entries (230,000) 270 / 279, two 299 / 313
// k_pull_wsync on these: 1,103 / 1,354, 1,187 / 1,383, 1,687, 490 (FP32), 510 / 578,
// 323 / 297.
//
// A warp works through its segments in walk order and holds at most two claimed
// ones it has not started, so the earliest unfinished segment is always being
// worked on: every dependency lies earlier in the walk.
#include <algorithm>

#include "exec_ahead.cuh"
#include "internal.h"

namespace sptrsv {

namespace {

template <typename T>
struct AheadArgs {
  int n, nseg, cap;
  const int* perm;
  const int* ptr;   // dependency lists in ready order (dependents, for the transposed walk)
  const int* pos;
  const T* w;
  const T* rcp;
  const T* b;
  T* x;
  T* xw;
  DeviceCtl* ctl;
  unsigned long long timeout_ns;
};

template <typename T, bool ADJ, int U>
__global__ void __launch_bounds__(256) k_pull_ahead(AheadArgs<T> a) {
  using F = Flag<T>;
  using Bits = typename F::Bits;
  constexpr unsigned kFull = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  // values of the segment in hand, then this warp's two list buffers
  T* s_win = reinterpret_cast<T*>(smem_raw) + warp * 32;
  T* s_w = reinterpret_cast<T*>(smem_raw) + nwarps * 32 + (size_t)warp * 2 * a.cap;
  int* s_q = reinterpret_cast<int*>(reinterpret_cast<T*>(smem_raw) + nwarps * 32 + (size_t)nwarps * 2 * a.cap) +
             warp * 2 * a.cap;
  const unsigned s_wina = static_cast<unsigned>(__cvta_generic_to_shared(s_win));
  const unsigned s_wa = static_cast<unsigned>(__cvta_generic_to_shared(s_w));
  const unsigned s_qa = static_cast<unsigned>(__cvta_generic_to_shared(s_q));
  const int last = a.n - 1;
  unsigned raw = 0u;  // the next segment's number, in lane 0 until it is needed
  auto claim = [&]() {
    if (lane == 0) raw = atomicAdd(&a.ctl->ticket, 1u);
  };
  auto claimed = [&]() { return static_cast<int>(min(__shfl_sync(kFull, raw, 0), (unsigned)a.nseg)); };
  int f_row = 0, f_e = 0, f_e1 = 0;
  auto fetch = [&](int sg) {
    const int pr = sg < a.nseg ? sg * 32 + lane : a.n;
    f_e = f_e1 = 0;
    if (pr < a.n) {
      const int p = ADJ ? last - pr : pr;
      f_row = a.perm[p];
      f_e = a.ptr[p];
      f_e1 = a.ptr[p + 1];
    }
  };
  int n_row = 0, n_e = 0, n_e1 = 0, n_lo = 0;
  T n_acc = T(0);
  auto stage = [&](int sg, int buf) {
    n_row = f_row;
    n_e = f_e;
    n_e1 = f_e1;
    if (sg >= a.nseg) return;
    const int pr = sg * 32 + lane;
    if (pr < a.n) n_acc = a.b[n_row] * a.rcp[ADJ ? last - pr : pr];
    const int cnt = min(32, a.n - sg * 32);
    const int lo = __shfl_sync(kFull, f_e, ADJ ? cnt - 1 : 0);
    const int hi = min(__shfl_sync(kFull, f_e1, ADJ ? 0 : cnt - 1), lo + a.cap);
    n_lo = lo;
    for (int e = lo + lane; e < hi; e += 32) {
      copy_async(s_qa + (unsigned)(buf * a.cap + e - lo) * 4u, a.pos + e);
      copy_async(s_wa + (unsigned)(buf * a.cap + e - lo) * (unsigned)sizeof(T), a.w + e);
    }
  };
  claim();
  int sg = claimed();
  claim();
  int sg1 = claimed();
  claim();
  fetch(sg);
  stage(sg, 0);
  fetch(sg1);
  bool fail = false;
  for (int buf = 0; sg < a.nseg; buf ^= 1) {
    const int base = sg * 32, pr = base + lane;
    bool done = pr >= a.n;
    const int p = ADJ ? last - pr : pr;
    const int row = n_row, lo = n_lo;
    int e = n_e;
    const int e1 = n_e1;
    T acc = n_acc;
    *reinterpret_cast<volatile Bits*>(&s_win[lane]) = F::EMPTY;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    stage(sg1, buf ^ 1);
    const int sg2 = claimed();
    claim();
    fetch(sg2);
    const T* lw = s_w + buf * a.cap - lo;
    const int* lq = s_q + buf * a.cap - lo;
    const int hi = lo + a.cap;
    // the U entries polled, in list order, and for U = 1 the one after it
    const T *word0 = a.xw, *word1 = a.xw;
    unsigned local0 = s_wina, local1 = s_wina;
    bool mine0 = true, mine1 = true;
    T w0 = T(0), w1 = T(0);
    int q1 = 0;
    int left = e1 - e;  // entries from the first polled on
    auto target = [&](int q, const T*& word, unsigned& local, bool& mine) {
      const int off = (ADJ ? last - q : q) - base;
      mine = off >= 0;
      local = s_wina + (unsigned)(off & 31) * (unsigned)sizeof(T);
      word = a.xw + q;
    };
    auto entry = [&](int ee, int& q, T& w) {
      q = ee < hi ? lq[ee] : a.pos[ee];
      w = ee < hi ? lw[ee] : a.w[ee];
    };
    auto second = [&]() {
      entry(e + 1, q1, w1);
      if (U == 2) target(q1, word1, local1, mine1);
    };
    auto first = [&]() {
      int q0;
      entry(e, q0, w0);
      target(q0, word0, local0, mine0);
      if (left > 1) second();
    };
    auto publish = [&]() {
      F::store_shared(&s_win[lane], acc);
      F::store(&a.xw[p], acc);
      done = true;
    };
    if (!done) {
      if (left <= 0) publish();
      else first();
    }
    unsigned idle = 0u;
    int seen = 0;
    WaitBudget wb(a.timeout_ns);
    while (!__all_sync(kFull, done)) {
      Bits bits0[1], bits1[1];
      poll_words(bits0, local0, word0, mine0, !done);
      if (U == 2) poll_words(bits1, local1, word1, mine1, !done && left > 1);
      if (U == 1) target(q1, word1, local1, mine1);  // in the poll's shadow
      if (bits0[0] != F::EMPTY) {
        acc = fma(-w0, F::value(bits0[0]), acc);
        if (U == 2 && bits1[0] != F::EMPTY) {
          acc = fma(-w1, F::value(bits1[0]), acc);
          left -= 2;
          e += 2;
          if (left > 0) first();
        } else {
          --left;
          ++e;
          w0 = w1;
          word0 = word1;
          local0 = local1;
          mine0 = mine1;
          if (left > 1) second();
        }
        if (left <= 0) publish();
      }
      if ((++idle & 255u) == 0u) {
        // lockstep_wait written out: other registers make the transposed walk slower (a
        // 1M-row band 1,077 -> 1,217 us)
        if (__any_sync(kFull, left != seen)) wb.start = 0;
        seen = left;
        if (!wb.poll<true>(a.ctl, p)) fail = true;
        if (__any_sync(kFull, fail)) {
          fail = true;
          break;
        }
      }
    }
    if (fail) break;
    if (pr < a.n) a.x[row] = acc;
    sg = sg1;
    sg1 = sg2;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  leave(a.ctl);
}

}  // namespace

namespace {
// Work per level (see above).
double level_work(const Layout& L, int nlevels) {
  return (static_cast<double>(L.ndep) + 4.0 * L.n) / std::max(1, nlevels);
}
}  // namespace

int ahead_entries(const Layout& L, int nlevels, bool adj) { return !adj && level_work(L, nlevels) < 21000.0 ? 1 : 2; }

template <typename T>
cudaError_t launch_pull_ahead(const Layout& L, const Values<T>& V, const VecView<T>& v, T* xw, DeviceCtl* ctl,
                              int nlevels, unsigned long long timeout_ns, int num_sms, cudaStream_t s, bool adj) {
  if (L.n == 0) return cudaSuccess;
  constexpr int block = 256;
  const double t = level_work(L, nlevels);
  int ctas = t <= 34000.0 ? 1 : (t <= 120000.0 ? 2 : 3);
  if (ctas == 2) {
    const double segment = 32.0 * L.ndep / L.n;  // entries
    if (adj && segment > 400.0) ctas = 1;
    else if (segment > 200.0) ctas = sizeof(T) == 8 ? 2 : 3;
    else if ((adj && sizeof(T) == 8) || t > 90000.0) ctas = 3;
  }
  const bool one = ahead_entries(L, nlevels, adj) == 1;
  // list buffers hold twice the average segment (longer ones read the rest from
  // global memory), as far as the CTAs and L1 leave room
  const int avg = static_cast<int>(32LL * L.ndep / L.n);
  const int cap = std::min(ctas == 1 ? 640 : (ctas == 2 ? 400 : 200), std::max(64, (2 * avg + 31) / 32 * 32));
  AheadArgs<T> a{};
  a.n = L.n;
  a.nseg = (L.n + 31) / 32;
  a.cap = cap;
  a.perm = L.perm;
  a.ptr = adj ? L.out_ptr : L.dep_ptr;
  a.pos = adj ? L.out_pos_f : L.dep_pos_f;
  a.w = adj ? V.out_w : V.dep_w;
  a.rcp = V.rcp;
  a.b = v.b;
  a.x = v.x;
  a.xw = xw;
  a.ctl = ctl;
  a.timeout_ns = timeout_ns;
  const size_t smem = (size_t)(block / 32) * (32 * sizeof(T) + 2 * cap * (sizeof(T) + sizeof(int)));
  auto kernel = one ? k_pull_ahead<T, false, 1> : (adj ? k_pull_ahead<T, true, 2> : k_pull_ahead<T, false, 2>);
  const cudaError_t e = allow_shared(kernel, smem);
  if (e != cudaSuccess) return e;
  int per = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, block, smem);
  per = std::max(1, std::min(per, ctas));
  const int grid = std::min(num_sms * per, (a.nseg + block / 32 - 1) / (block / 32));
  kernel<<<grid, block, smem, s>>>(a);
  return cudaGetLastError();
}
template cudaError_t launch_pull_ahead<double>(const Layout&, const Values<double>&, const VecView<double>&, double*,
                                               DeviceCtl*, int, unsigned long long, int, cudaStream_t, bool);
template cudaError_t launch_pull_ahead<float>(const Layout&, const Values<float>&, const VecView<float>&, float*,
                                              DeviceCtl*, int, unsigned long long, int, cudaStream_t, bool);

}  // namespace sptrsv
