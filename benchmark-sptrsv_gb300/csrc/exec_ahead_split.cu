// Level-order executor with lists staged ahead and long lists split over lanes
// (one right-hand side).
//
// k_pull_ahead's loop, two entries polled per iteration, over pieces: a list
// longer than the split length takes up to 32 adjacent lanes of a segment,
// interleaved, and once all of them are through, a segmented suffix sum hands
// the head lane the value to publish (as k_pull_wsync_split, from where the
// completion test comes). Segments are packed on the device.
//
// Power-law upper triangles, k_pull_wsync_split -> this kernel (us): 20,000 rows
// 128 -> 104, 200,000 rows (13,300 units of work per level: dependencies plus 4 per
// unknown) 215 -> 191, 1M rows of band 5,000 (3,600) 3,728 -> 2,870. Wider levels
// need more lanes than list buffers leave room for (1M rows, 25,000: 614 -> 856),
// so beyond kSplitAheadWork the plan keeps k_pull_wsync_split.
#include <algorithm>

#include "exec_ahead.cuh"
#include "internal.h"

namespace sptrsv {

namespace {

constexpr int kPackBlock = 1024;  // unknowns packed into segments together

// Lanes an unknown of `len` dependencies takes.
__device__ __forceinline__ int lanes_of(int len, int split) {
  return len > split ? min(32, (len + split - 1) / split) : 1;
}

// Segments of 32 lanes, each lane one piece, no unknown over two segments: one
// thread packs a block of kPackBlock consecutive walk indices, starting on a
// fresh segment. First pass (walk null): segments per block; second: the walk
// index of every piece (-1: padding) from the block's first segment on.
template <bool ADJ>
__global__ void k_pack_pieces(const int* __restrict__ ptr, int n, int split, const int* __restrict__ first, int* count,
                              int* walk) {
  const int blk = blockIdx.x * blockDim.x + threadIdx.x;
  const int nblk = (n + kPackBlock - 1) / kPackBlock;
  if (blk >= nblk) return;
  const int i0 = blk * kPackBlock, i1 = min(i0 + kPackBlock, n);
  int* out = walk ? walk + (long long)first[blk] * 32 : nullptr;
  int seg = 0, lane = 0;
  for (int i = i0; i < i1; ++i) {
    const int p = ADJ ? n - 1 - i : i;
    const int k = lanes_of(ptr[p + 1] - ptr[p], split);
    if (lane + k > 32) {
      if (out)
        for (; lane < 32; ++lane) out[seg * 32 + lane] = -1;
      ++seg;
      lane = 0;
    }
    if (out)
      for (int j = 0; j < k; ++j) out[seg * 32 + lane + j] = i;
    lane += k;
  }
  if (out)
    for (; lane < 32; ++lane) out[seg * 32 + lane] = -1;
  if (count) count[blk] = seg + 1;
}

template <typename T>
struct SplitArgs {
  int n, nseg, cap;
  const int* walk;  // [nseg * 32]
  const int* perm;
  const int* ptr;
  const int* pos;
  const T* w;
  const T* rcp;
  const T* b;
  T* x;
  T* xw;
  DeviceCtl* ctl;
  unsigned long long timeout_ns;
};

template <typename T, bool ADJ>
__global__ void __launch_bounds__(256) k_pull_ahead_split(SplitArgs<T> a) {
  using F = Flag<T>;
  using Bits = typename F::Bits;
  constexpr unsigned kFull = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  // values of the segment in hand by lane of the unknown's head, then this warp's two list buffers
  T* s_win = reinterpret_cast<T*>(smem_raw) + warp * 32;
  T* s_w = reinterpret_cast<T*>(smem_raw) + nwarps * 32 + (size_t)warp * 2 * a.cap;
  int* s_q = reinterpret_cast<int*>(reinterpret_cast<T*>(smem_raw) + nwarps * 32 + (size_t)nwarps * 2 * a.cap) +
             warp * 2 * a.cap;
  const unsigned s_wina = static_cast<unsigned>(__cvta_generic_to_shared(s_win));
  const unsigned s_wa = static_cast<unsigned>(__cvta_generic_to_shared(s_w));
  const unsigned s_qa = static_cast<unsigned>(__cvta_generic_to_shared(s_q));
  const unsigned at_or_below = (2u << lane) - 1u;
  const int last = a.n - 1;
  unsigned raw = 0u;
  auto claim = [&]() {
    if (lane == 0) raw = atomicAdd(&a.ctl->ticket, 1u);
  };
  auto claimed = [&]() { return static_cast<int>(min(__shfl_sync(kFull, raw, 0), (unsigned)a.nseg)); };
  auto pieces = [&](int sg) { return sg < a.nseg ? a.walk[sg * 32 + lane] : -1; };
  int f_walk = -1, f_row = 0, f_e = 0, f_e1 = 0;
  auto fetch = [&](int walk) {
    f_walk = walk;
    f_e = f_e1 = 0;
    if (walk >= 0) {
      const int p = ADJ ? last - walk : walk;
      f_row = a.perm[p];
      f_e = a.ptr[p];
      f_e1 = a.ptr[p + 1];
    }
  };
  int n_walk = -1, n_row = 0, n_e = 0, n_e1 = 0, n_lo = 0;
  T n_acc = T(0);
  auto stage = [&](int buf) {
    n_walk = f_walk;
    n_row = f_row;
    n_e = f_e;
    n_e1 = f_e1;
    const unsigned valid = __ballot_sync(kFull, f_walk >= 0);
    if (!valid) return;
    if (f_walk >= 0) n_acc = a.b[n_row] * a.rcp[ADJ ? last - f_walk : f_walk];
    const int end = 31 - __clz(valid);
    const int lo = __shfl_sync(kFull, f_e, ADJ ? end : 0);
    const int hi = min(__shfl_sync(kFull, f_e1, ADJ ? 0 : end), lo + a.cap);
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
  int sg2 = claimed();
  claim();
  fetch(pieces(sg));
  stage(0);
  fetch(pieces(sg1));
  int g_walk = pieces(sg2);  // pieces two segments ahead
  bool fail = false;
  for (int buf = 0; sg < a.nseg; buf ^= 1) {
    const int walk = n_walk, row = n_row, lo = n_lo;
    const bool valid = walk >= 0;
    const int p = ADJ ? last - walk : walk;
    int e = n_e;
    const int e1 = n_e1;
    T acc = n_acc;
    *reinterpret_cast<volatile Bits*>(&s_win[lane]) = F::EMPTY;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    stage(buf ^ 1);
    const int sg3 = claimed();
    claim();
    fetch(g_walk);
    g_walk = pieces(sg3);
    // the lanes of this lane's unknown: gs (its head) to ge
    const int prev = __shfl_up_sync(kFull, walk, 1);
    const bool head = valid && (lane == 0 || prev != walk);
    const unsigned heads = __ballot_sync(kFull, head), valids = __ballot_sync(kFull, valid);
    const unsigned above = heads & ~at_or_below;
    const int ge = above ? __ffs(above) - 2 : 31 - __clz(valids);
    const int gs = valid ? 31 - __clz(heads & at_or_below) : lane;
    const int step = valid ? ge - gs + 1 : 1;
    // unknowns over several lanes, and the rounds of a sum over the widest of them
    const unsigned multi = __ballot_sync(kFull, head && step > 1);
    const unsigned span = __reduce_max_sync(kFull, static_cast<unsigned>(step));
    const int base = __shfl_sync(kFull, walk, 0);
    if (!head) acc = T(0);
    e += lane - gs;
    const T* lw = s_w + buf * a.cap - lo;
    const int* lq = s_q + buf * a.cap - lo;
    const int hi = lo + a.cap;
    // the two entries polled, in list order; `left` entries from the first on
    const T *word0 = a.xw, *word1 = a.xw;
    unsigned local0 = s_wina, local1 = s_wina;
    bool mine0 = true, mine1 = true;
    T w0 = T(0), w1 = T(0);
    int q1 = 0;
    int left = valid ? (e1 - e + step - 1) / step : 0;
    auto entry = [&](int ee, int& q, T& w) {
      q = ee < hi ? lq[ee] : a.pos[ee];
      w = ee < hi ? lw[ee] : a.w[ee];
    };
    auto target = [&](int q, const T*& word, unsigned& local, bool& mine) {
      const int off = (ADJ ? last - q : q) - base;
      mine = off >= 0;
      local = s_wina + (unsigned)(off & 31) * (unsigned)sizeof(T);
      word = a.xw + q;
    };
    auto first = [&]() {
      int q0;
      entry(e, q0, w0);
      target(q0, word0, local0, mine0);
      if (left > 1) {
        entry(e + step, q1, w1);
        target(q1, word1, local1, mine1);
      }
    };
    auto publish = [&](T xi) {
      F::store_shared(&s_win[(walk - base) & 31], xi);
      F::store(&a.xw[p], xi);
    };
    bool done = !valid;  // this lane's piece is consumed
    if (valid) {
      if (left <= 0) {
        done = true;
        if (head && step == 1) publish(acc);
      } else {
        first();
      }
    }
    unsigned idle = 0u, waiting = multi;  // split unknowns not yet published
    int seen = 0;
    WaitBudget wb(a.timeout_ns);
    while (!__all_sync(kFull, done)) {
      Bits bits0[1], bits1[1];
      poll_words(bits0, local0, word0, mine0, !done);
      poll_words(bits1, local1, word1, mine1, left > 1);
      if (bits0[0] != F::EMPTY) {
        acc = fma(-w0, F::value(bits0[0]), acc);
        if (bits1[0] != F::EMPTY) {
          acc = fma(-w1, F::value(bits1[0]), acc);
          left -= 2;
          e += 2 * step;
          if (left > 0) first();
        } else {
          --left;
          e += step;
          w0 = w1;
          word0 = word1;
          local0 = local1;
          mine0 = mine1;
          if (left > 1) {
            entry(e + step, q1, w1);
            target(q1, word1, local1, mine1);
          }
        }
        if (left <= 0) {
          left = 0;
          done = true;
          if (step == 1) publish(acc);
        }
      }
      if (waiting) {
        // a split unknown is complete once none of its lanes is pending: a
        // segmented OR from its last lane down to its head, the same in every lane
        const unsigned pending = ~__ballot_sync(kFull, done);
        unsigned v = pending, f = (heads >> 1) | 0x80000000u;  // f: last lane of an unknown
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const unsigned open = ~f;
          v |= (v >> d) & open;
          f |= (f >> d) & open;
        }
        const unsigned ready = waiting & ~v;
        if (ready) {
          T xi = acc;
          for (unsigned off = 1; off < span; off <<= 1) {
            const T t = __shfl_down_sync(kFull, xi, off);
            if (lane + static_cast<int>(off) <= ge) xi += t;
          }
          if ((ready >> lane) & 1u) {
            acc = xi;
            publish(xi);
          }
          waiting &= ~ready;
        }
      }
      if ((++idle & 255u) == 0u) {
        if (!lockstep_wait(wb, left, seen, fail, a.ctl, p)) break;
      }
    }
    if (fail) break;
    if (head) a.x[row] = acc;
    sg = sg1;
    sg1 = sg2;
    sg2 = sg3;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  leave(a.ctl);
}

}  // namespace

cudaError_t launch_pack_count(const int* ptr, int n, int split, bool adj, int* count, cudaStream_t s) {
  const int nblk = (n + kPackBlock - 1) / kPackBlock;
  auto kernel = adj ? k_pack_pieces<true> : k_pack_pieces<false>;
  kernel<<<(nblk + 63) / 64, 64, 0, s>>>(ptr, n, split, nullptr, count, nullptr);
  return cudaGetLastError();
}
cudaError_t launch_pack_fill(const int* ptr, int n, int split, bool adj, const int* first, int* walk, cudaStream_t s) {
  const int nblk = (n + kPackBlock - 1) / kPackBlock;
  auto kernel = adj ? k_pack_pieces<true> : k_pack_pieces<false>;
  kernel<<<(nblk + 63) / 64, 64, 0, s>>>(ptr, n, split, first, nullptr, walk);
  return cudaGetLastError();
}
namespace {

// Pieces of k_pull_wsync_split (see PieceTable). Chunks start at every multiple of
// `chunk` walk indices, so each such range is packed by a thread of its own: pass 1
// (walk null) counts its segments and chunks, pass 2 fills them from their first
// ones. On the host the 4M-row power-law triangle's pieces took 33 ms.
__global__ void k_pieces(const int* __restrict__ ptr, const int* __restrict__ perm, int n, bool reversed, int split,
                         int chunk, int shift, int nranges, int* nseg, int* nchunk, int* walk, int* row, int* lo, int* hi,
                         int* cseg, int* cbase, unsigned char* seg_split) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nranges) return;
  const int seg_cap = max(1, (chunk + 31) / 32);
  const int i0 = static_cast<int>(max(0LL, (long long)b * chunk - shift));
  const int i1 = static_cast<int>(min((long long)n, (long long)(b + 1) * chunk - shift));
  const int seg0 = walk ? nseg[b] : 0;
  int used = 0, chunk_seg = 0, chunks = walk ? nchunk[b] : 0;  // pieces placed (with padding), first segment in hand
  for (int i = i0; i < i1; ++i) {
    const int p = reversed ? n - 1 - i : i;
    const int e0 = ptr[p], e1 = ptr[p + 1], c = e1 - e0;
    const int k = c > split ? min(32, (c + split - 1) / split) : 1;
    const int padded = (used + 31) & ~31;
    const bool full = (used & 31) + k > 32;
    const int after = ((full ? padded : used) + k - 1) / 32 + 1;
    if (i == i0 || after - chunk_seg > seg_cap) {
      used = padded;
      chunk_seg = used / 32;
      if (walk) {
        cseg[chunks] = seg0 + chunk_seg;
        cbase[chunks] = i;
      }
      ++chunks;
    } else if (full) {
      used = padded;
    }
    if (walk) {
      const long long at = 32LL * seg0 + used;
      if (k > 1) seg_split[at / 32] = 1;
      const int r = perm[p];
      for (int j = 0; j < k; ++j) {
        walk[at + j] = i;
        row[at + j] = r;
        lo[at + j] = e0 + j;
        hi[at + j] = e1;
      }
    }
    used += k;
  }
  if (!walk) {
    nseg[b] = (used + 31) / 32;
    nchunk[b] = chunks;
  }
}

}  // namespace

cudaError_t launch_pieces(const int* ptr, const int* perm, int n, bool reversed, int split, int chunk, int shift,
                          int nranges, int* nseg, int* nchunk, const PieceTable& t, cudaStream_t s) {
  if (nranges <= 0) return cudaSuccess;
  k_pieces<<<(nranges + 31) / 32, 32, 0, s>>>(ptr, perm, n, reversed, split, chunk, shift, nranges, nseg, nchunk, t.walk,
                                             t.row, t.lo, t.hi, t.cseg, t.cbase, t.seg_split);
  return cudaGetLastError();
}

int pack_blocks(int n) { return (n + kPackBlock - 1) / kPackBlock; }

template <typename T>
cudaError_t launch_pull_ahead_split(const Layout& L, const Values<T>& V, const VecView<T>& v, T* xw, DeviceCtl* ctl,
                                    const SplitTable& tab, unsigned long long timeout_ns, int num_sms, cudaStream_t s,
                                    bool adj) {
  if (L.n == 0) return cudaSuccess;
  SplitArgs<T> a{};
  a.n = L.n;
  a.nseg = tab.nseg;
  a.walk = tab.walk;
  a.cap = 640;
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
  constexpr int block = 256;
  const size_t smem = (size_t)(block / 32) * (32 * sizeof(T) + 2 * a.cap * (sizeof(T) + sizeof(int)));
  auto kernel = adj ? k_pull_ahead_split<T, true> : k_pull_ahead_split<T, false>;
  const cudaError_t e = allow_shared(kernel, smem);
  if (e != cudaSuccess) return e;
  const int grid = std::min(num_sms, (a.nseg + block / 32 - 1) / (block / 32));
  kernel<<<grid, block, smem, s>>>(a);
  return cudaGetLastError();
}
template cudaError_t launch_pull_ahead_split<double>(const Layout&, const Values<double>&, const VecView<double>&,
                                                     double*, DeviceCtl*, const SplitTable&, unsigned long long, int,
                                                     cudaStream_t, bool);
template cudaError_t launch_pull_ahead_split<float>(const Layout&, const Values<float>&, const VecView<float>&, float*,
                                                    DeviceCtl*, const SplitTable&, unsigned long long, int, cudaStream_t,
                                                    bool);

}  // namespace sptrsv
