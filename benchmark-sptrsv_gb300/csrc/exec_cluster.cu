// One-cluster executor for narrow dependency DAGs (one right-hand side).
//
// Where the level sets hold a few hundred dependencies, a solve keeps few lanes
// busy and costs what its hops from level to level cost. Through a global
// value-as-flag word a hop is a store to L2 plus the poll that notices it; here
// the whole solution vector lives in the shared memory of one thread block
// cluster of 16 CTAs, a dependency is polled in this CTA's shared memory or in
// a peer's (a distributed-shared-memory load takes ~220 cycles, a flag hop by
// such polls ~410), and nothing is polled in global memory, so the solve needs
// no flag words there and no clearing pass: one launch.
//
// Walk indices are dealt to the CTAs in runs of 1 << cshift; inside a CTA its
// warps take 32 consecutive ones at a time, in order, one unknown per lane, in
// lockstep (as k_pull_wsync). Every CTA of a cluster is resident, each warp
// works through its segments in walk order, and every dependency lies earlier
// in the walk, so the wait for the earliest unfinished unknown always ends. A
// lane consumes one dependency per iteration, in ready order; the next entry's
// address is worked out while the poll is in flight. A segment's lists (one
// contiguous range) are copied to shared memory with cp.async while the warp
// works on the segment before, because a list entry fetched from global memory
// inside the loop stalls all 32 lanes on it.
//
// Measured (FP64, kernel and launch, forward / transposed, against k_pull_wsync):
// 10,000 rows / 147 levels 67.2 / 75.7 vs 118.9 / 145.3 us; 50,000 rows / 380
// levels 145 / 192 vs 295 / 377; 100,000 rows / 438 levels of 2,051 dependencies
// 213 / 250 vs 369 / 457; 150,001 rows / 8,814 levels 2,921 / 3,721 vs 5,050 /
// 7,215. Bound by the hop: a lockstep iteration is one remote poll
// (~220 cycles) plus the multiply-add of the lanes that consumed (64 cycles in
// FP64; FP32 runs 10 % faster). One CTA instead of 16 loses (10,000 rows: 113
// us): an FP64 warp instruction holds its sub-partition's pipe for 64 cycles
// whatever lanes are active, so one SM's four pipes bind first.
#include "exec_common.cuh"
#include "internal.h"

namespace sptrsv {

namespace {

constexpr int kRankShift = ClusterPlan::kRankShift;

template <typename T>
struct ClusterArgs {
  int n;
  int cshift;   // walk indices [c << cshift, (c + 1) << cshift) belong to CTA c mod 16
  int slots;    // shared-memory slots per CTA
  int cap;      // list entries per warp buffer
  const int* perm;
  const int* ptr;   // dependency lists in ready order (dependents, for the transposed walk)
  const int* pos;
  const T* w;
  const T* rcp;
  const T* b;
  T* x;
  DeviceCtl* ctl;
  unsigned long long timeout_ns;
};

__device__ __forceinline__ unsigned map_shared(unsigned addr, unsigned rank) {
  unsigned v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(v) : "r"(addr), "r"(rank));
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// One poll of a value word: from this CTA's shared memory when `mine`, else
// from a peer's (one predicated load each, so a warp that holds both kinds
// waits for the longer of the two, not for their sum). Lanes that do not `look`
// get the empty pattern and load nothing: distributed-shared-memory loads of
// scattered words are served at well under one a cycle per SM.
__device__ __forceinline__ unsigned long long poll_word(unsigned addr, unsigned remote, bool mine, bool look, double) {
  unsigned long long v;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\tsetp.ne.u32 q, %4, 0;\n\tmov.u64 %0, -1;\n\t"
      "@p ld.relaxed.cluster.shared::cta.u64 %0, [%1];\n\t"
      "@q ld.relaxed.cluster.shared::cluster.u64 %0, [%2];\n\t}"
      : "=&l"(v) : "r"(addr), "r"(remote), "r"((unsigned)(mine && look)), "r"((unsigned)(!mine && look)) : "memory");
  return v;
}
__device__ __forceinline__ unsigned poll_word(unsigned addr, unsigned remote, bool mine, bool look, float) {
  unsigned v;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\tsetp.ne.u32 q, %4, 0;\n\tmov.u32 %0, -1;\n\t"
      "@p ld.relaxed.cluster.shared::cta.u32 %0, [%1];\n\t"
      "@q ld.relaxed.cluster.shared::cluster.u32 %0, [%2];\n\t}"
      : "=&r"(v) : "r"(addr), "r"(remote), "r"((unsigned)(mine && look)), "r"((unsigned)(!mine && look)) : "memory");
  return v;
}
__device__ __forceinline__ void publish_word(unsigned addr, unsigned long long v) {
  asm volatile("st.relaxed.cluster.shared::cta.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
__device__ __forceinline__ void publish_word(unsigned addr, unsigned v) {
  asm volatile("st.relaxed.cluster.shared::cta.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

template <typename T, bool ADJ>
__global__ void __launch_bounds__(512) k_pull_cluster(ClusterArgs<T> a) {
  using F = Flag<T>;
  using Bits = typename F::Bits;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* s_x = reinterpret_cast<T*>(smem_raw);
  const unsigned s_base = static_cast<unsigned>(__cvta_generic_to_shared(s_x));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int rank = blockIdx.x;  // one cluster: the block index is the cluster rank
  const int rmask = (1 << kRankShift) - 1, cmask = (1 << a.cshift) - 1;
  // this warp's two list buffers
  T* s_w = s_x + a.slots + (size_t)warp * 2 * a.cap;
  int* s_q = reinterpret_cast<int*>(s_x + a.slots + (size_t)nwarps * 2 * a.cap) + warp * 2 * a.cap;
  const unsigned s_wa = static_cast<unsigned>(__cvta_generic_to_shared(s_w));
  const unsigned s_qa = static_cast<unsigned>(__cvta_generic_to_shared(s_q));
  for (int i = threadIdx.x; i < a.slots; i += blockDim.x) *reinterpret_cast<Bits*>(&s_x[i]) = F::EMPTY;
  const int last = a.n - 1;
  const int nseg = a.slots >> 5;
  // local segment ls covers 32 walk indices from here
  auto seg_start = [&](int ls) {
    const int sc = ls >> (a.cshift - 5);
    return (((sc << kRankShift) + rank) << a.cshift) + ((ls & ((1 << (a.cshift - 5)) - 1)) << 5);
  };
  int f_row = 0, f_e = 0, f_e1 = 0;  // bounds, two segments ahead
  auto fetch = [&](int ls) {
    const int pr = ls < nseg ? seg_start(ls) + lane : a.n;
    f_e = f_e1 = 0;
    if (pr < a.n) {
      const int p = ADJ ? last - pr : pr;
      f_row = a.perm[p];
      f_e = a.ptr[p];
      f_e1 = a.ptr[p + 1];
    }
  };
  // staged, one segment ahead: the scaled right-hand side, and the segment's
  // (contiguous) lists on their way into the warp's other buffer
  int n_row = 0, n_e = 0, n_e1 = 0, n_lo = 0;
  T n_acc = T(0);
  auto stage = [&](int ls, int buf) {
    const int pr = ls < nseg ? seg_start(ls) + lane : a.n;
    n_row = f_row;
    n_e = f_e;
    n_e1 = f_e1;
    if (pr < a.n) n_acc = a.b[n_row] * a.rcp[ADJ ? last - pr : pr];
    const int cnt = min(32, a.n - (pr - lane));
    if (ls >= nseg || cnt <= 0) return;
    const int lo = __shfl_sync(0xffffffffu, f_e, ADJ ? cnt - 1 : 0);
    const int hi = min(__shfl_sync(0xffffffffu, f_e1, ADJ ? 0 : cnt - 1), lo + a.cap);
    n_lo = lo;
    for (int e = lo + lane; e < hi; e += 32) {
      copy_async(s_qa + (unsigned)(buf * a.cap + e - lo) * 4u, a.pos + e);
      copy_async(s_wa + (unsigned)(buf * a.cap + e - lo) * (unsigned)sizeof(T), a.w + e);
    }
  };
  fetch(warp);
  stage(warp, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  fetch(warp + nwarps);
  __syncwarp();  // the cluster barrier's aligned form takes whole warps
  cluster_sync();
  bool fail = false;
  int buf = 0;
  for (int ls = warp; ls < nseg && !fail; ls += nwarps, buf ^= 1) {
    const int pr = seg_start(ls) + lane;
    bool done = pr >= a.n;
    const int p = ADJ ? last - pr : pr;
    const int row = n_row, lo = n_lo;
    int e = n_e;
    const int e1 = n_e1;
    T acc = n_acc;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    stage(ls + nwarps, buf ^ 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    fetch(ls + 2 * nwarps);
    const T* lw = s_w + buf * a.cap - lo;
    const int* lq = s_q + buf * a.cap - lo;
    const int hi = lo + a.cap;
    const unsigned own = s_base + (unsigned)((ls << 5) + lane) * (unsigned)sizeof(T);
    unsigned addr = own, remote = own, naddr = own, nremote = own;
    bool mine = true, nmine = true;
    T w = T(0), nw = T(0);
    int nq = 0;
    // entries left after the one being polled
    int left = e1 - e - 1;
    auto next = [&](int ee) {
      nq = ee < hi ? lq[ee] : a.pos[ee];
      nw = ee < hi ? lw[ee] : a.w[ee];
    };
    auto target = [&](int q) {
      const int qr = ADJ ? last - q : q;
      const int c = qr >> a.cshift;
      const int rk = c & rmask;
      naddr = s_base + ((((c >> kRankShift) << a.cshift) + (qr & cmask)) * (unsigned)sizeof(T));
      nmine = rk == rank;
      nremote = map_shared(naddr, rk);
    };
    if (left < 0) {
      if (!done) publish_word(own, F::bits(acc));
      done = true;
    } else {
      next(e);
      w = nw;
      target(nq);
      addr = naddr;
      remote = nremote;
      mine = nmine;
      if (left > 0) next(++e);
    }
    unsigned idle = 0u;
    int seen = 0;
    WaitBudget wb(a.timeout_ns);
    while (!__all_sync(0xffffffffu, done)) {
      const Bits bits = poll_word(addr, remote, mine, !done, T(0));
      target(nq);  // in the poll's shadow
      if (bits != F::EMPTY) {
        acc = fma(-w, F::value(bits), acc);
        if (left > 0) {
          w = nw;
          addr = naddr;
          remote = nremote;
          mine = nmine;
          if (--left > 0) next(++e);
        } else {
          publish_word(own, F::bits(acc));
          done = true;
        }
      }
      if ((++idle & 255u) == 0u) {
        if (!lockstep_wait(wb, left - done, seen, fail, a.ctl, p)) break;
      }
    }
    if (pr < a.n && !fail) a.x[row] = acc;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  // peers may still poll this CTA's words
  __syncwarp();
  cluster_sync();
  if (rank == 0 && threadIdx.x == 0) ctl_report(a.ctl, *reinterpret_cast<volatile int*>(&a.ctl->code));
}

// Launch configuration of the executor; the attribute must outlive it.
void cluster_config(const ClusterPlan& plan, size_t smem, cudaStream_t s, cudaLaunchConfig_t& cfg,
                    cudaLaunchAttribute& at) {
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = 1u << kRankShift;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = 1;
  cfg.gridDim = dim3(1u << kRankShift);
  cfg.blockDim = dim3(plan.block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
}

template <typename T>
constexpr auto cluster_kernel(bool adj) {
  return adj ? k_pull_cluster<T, true> : k_pull_cluster<T, false>;
}

}  // namespace

template <typename T>
bool cluster_fits(const ClusterPlan& plan, int n) {
  int dev = 0, limit = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t smem = plan.smem(n, sizeof(T));
  if (smem > (size_t)limit) return false;
  for (bool adj : {false, true}) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    int clusters = 0;
    auto kernel = cluster_kernel<T>(adj);
    cluster_config(plan, smem, nullptr, cfg, at);
    // set once per plan, to the device's limit whatever this plan needs, so that
    // no launch has to set them
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
      cudaGetLastError();
      return false;
    }
  }
  return true;
}

template <typename T>
cudaError_t launch_pull_cluster(const Layout& L, const Values<T>& V, const VecView<T>& v, DeviceCtl* ctl,
                                const ClusterPlan& plan, unsigned long long timeout_ns, cudaStream_t s, bool adj) {
  if (L.n == 0) return cudaSuccess;
  ClusterArgs<T> a{};
  a.n = L.n;
  a.cshift = plan.cshift;
  a.slots = plan.slots(L.n);
  a.cap = plan.cap;
  a.perm = L.perm;
  a.ptr = adj ? L.out_ptr : L.dep_ptr;
  a.pos = adj ? L.out_pos_f : L.dep_pos_f;
  a.w = adj ? V.out_w : V.dep_w;
  a.rcp = V.rcp;
  a.b = v.b;
  a.x = v.x;
  a.ctl = ctl;
  a.timeout_ns = timeout_ns;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  cluster_config(plan, plan.smem(L.n, sizeof(T)), s, cfg, at);
  return cudaLaunchKernelEx(&cfg, cluster_kernel<T>(adj), a);
}
template bool cluster_fits<double>(const ClusterPlan&, int);
template bool cluster_fits<float>(const ClusterPlan&, int);
template cudaError_t launch_pull_cluster<double>(const Layout&, const Values<double>&, const VecView<double>&,
                                                 DeviceCtl*, const ClusterPlan&, unsigned long long, cudaStream_t, bool);
template cudaError_t launch_pull_cluster<float>(const Layout&, const Values<float>&, const VecView<float>&,
                                                DeviceCtl*, const ClusterPlan&, unsigned long long, cudaStream_t, bool);

}  // namespace sptrsv
