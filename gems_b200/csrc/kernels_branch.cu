// kernels_branch.cu -- the branch terms on the host: which kernels of branch_kernels.cuh a session
// uses, their launches, and the time-out probes of the Newton loop's waits.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>

#include "branch_kernels.cuh"

namespace gems {

namespace {

// The exchange's time-out path on purpose: each block publishes and waits for one more than
// there are, so it gives up after kPollLimit polls and the flag reads GEMS_ERR_TIMEOUT.
__global__ void k_exchange_probe(ulonglong2 *slots, int *flag) {
  if (threadIdx.x == 0) {
    publish(slots + kSlotStride * blockIdx.x, 1.0, 1);
    publish(slots + kSlotStride * blockIdx.x + 1, 2.0, 1);
  }
  double a, b;
  const bool ok = gather(slots, gridDim.x + 1, 1, a, b);
  if (threadIdx.x == 0) atomicExch(flag, ok ? GEMS_OK : GEMS_ERR_TIMEOUT);
}

// The cluster wait's time-out path on purpose: two blocks send each other a pair and wait for one
// more, so each gives up after the clock budget.  The flag reads GEMS_ERR_TIMEOUT when they did
// and the pairs that were sent have come.
__global__ void k_cluster_probe(int *flag) {
  __shared__ __align__(16) double2 recv[2];
  __shared__ __align__(8) uint64_t bar;
  const uint32_t s_bar = tc::sptr(&bar);
  const int rank = blockIdx.x & 1;
  if (threadIdx.x == 0) {
    tc::mbar_init(s_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc::mbar_expect_tx(s_bar, 3 * sizeof(double2));
    recv[0] = recv[1] = make_double2(0.0, 0.0);
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (threadIdx.x < 2)
    send_pair(cluster_addr(tc::sptr(&recv[rank]), threadIdx.x), cluster_addr(s_bar, threadIdx.x),
              1.0, 2.0);
  const bool ok = cluster_wait(s_bar, 0);
  // the other block has given up too: nothing is on its way to this one
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const volatile double *v = &recv[0].x;
  if (threadIdx.x == 0 && blockIdx.x == 0)
    atomicExch(flag, !ok && v[0] + v[1] + v[2] + v[3] == 6.0 ? GEMS_ERR_TIMEOUT : GEMS_OK);
}

BranchFns memory_kernels(int e2) {
  return e2 <= 2 ? branch_memory_4(e2) : e2 <= 5 ? branch_memory_20(e2) : branch_memory_wide(e2);
}
BranchFns kernels_for(const Session *s, bool from_partials, int e2) {
  const bool safe = s->desc.scaling == GEMS_SCALE_SAFE;
  if (!from_partials) return memory_kernels(e2);
  if (s->desc.precision == GEMS_PREC_MIXED) return branch_mixed_4(safe, e2);
  switch (s->desc.nstates) {
    case 4: return branch_f64_4(safe, e2);
    case 20: return branch_f64_20(safe, e2);
    default: return e2 <= 5 ? branch_f64_61(safe, e2) : branch_f64_61_wide(safe, e2);
  }
}

}  // namespace

bool theta_in_kernel(const Session *s) {
  return s->desc.precision == GEMS_PREC_FP64 || s->desc.nstates == 4;
}

static bool mixed_of(const Session *s) { return s->desc.precision == GEMS_PREC_MIXED; }

// Op lists that a branch call runs in its own launch: few of them, and few enough patterns that
// the launches around them cost more than the lanes' own loads (from about 2^15 on, the traversal
// kernels' staged tables and one thread per pattern are the faster way).
bool small_ops(const Session *s, int nops) {
  return s->desc.nstates == 4 && s->desc.ncat >= 2 && nops >= 1 && nops <= kSmallOps &&
         nops * s->desc.ncat <= 64 && s->P <= kSmallPatterns && s->force_shape < 0;
}
static SmallOps small_list(const gems_op *ops, int nops) {
  SmallOps o;
  std::memset(&o, 0, sizeof(o));
  o.n = nops;
  if (nops) std::memcpy(o.op, ops, sizeof(DevOp) * nops);
  return o;
}

// br: theta from the branch's partials; null: theta as stored.  The two results are in
// s->h_result once the stream has completed.
static int launch_terms(Session *s, const gems_branch *br, int flags, int id, double length,
                        const gems_op *ops, int nops) {
  DevCtx c = s->ctx();
  SmallOps o = small_list(ops, nops);
  Split sp = split_of(s->block, s->desc.ncat);
  const BranchFns f = kernels_for(s, br != nullptr, sp.E2);
  const long per = kThreadsT / sp.L;
  const int grid = (int)std::min<long>(s->nsm * ctas_t(sp.E2), (s->P + per - 1) / per);
  gems_branch b{};
  if (br) b = *br;
  const size_t smem = sizeof(double) * (2 * sp.L * sp.E2 * (flags & kDerv ? 3 : 1) +
                                        small_doubles(nops, s->desc.ncat, mixed_of(s)));
  unsigned int *ticket = s->d_bar;
  double *out = s->h_result;
  void *args[] = {&c, &b, &length, &sp.L, &flags, &ticket, &out, &o};
  cudaEvent_t ev0;
  if (int st = prof_begin(s, id, &ev0)) return st;
  GEMS_CUDA(cudaLaunchKernel(f.terms, dim3(grid), dim3(kThreadsT), args, smem, s->stream));
  s->launches++;
  return prof_end(s, id, ev0);
}

int enqueue_terms(Session *s, const gems_branch *br, bool store, bool lnl, double length,
                  const gems_op *ops, int nops) {
  return launch_terms(s, br, (store ? kStore : 0) | (lnl ? kLnl : kDerv), lnl ? (br ? 1 : 4) : 3,
                      length, ops, nops);
}

int enqueue_theta(Session *s, const gems_branch *br) {
  return launch_terms(s, br, kStore, 2, br->length, nullptr, 0);
}

// a non-finite total: the sum with non-finite pattern values clamped to 4 log(2^-256)
// (phylokernelnew.h:3168-3184)
double terms_lnl(const Session *s) {
  return std::isfinite(s->h_result[0]) ? s->h_result[0] : s->h_result[1];
}

int launch_derv(Session *s, const gems_branch *br, double length, double *df, double *ddf,
                const gems_op *ops, int nops) {
  if (int st = enqueue_terms(s, br, br != nullptr, false, length, ops, nops)) return st;
  GEMS_CUDA(cudaStreamSynchronize(s->stream));
  *df = s->h_result[0];
  *ddf = s->h_result[1];
  if (!std::isfinite(*df)) *df = *ddf = 0.0;  // phylokernelnew.h:2646-2649
  return GEMS_OK;
}

int launch_from_buffer(Session *s, double length, double *lnl) {
  if (int st = enqueue_terms(s, nullptr, false, true, length, nullptr, 0)) return st;
  GEMS_CUDA(cudaStreamSynchronize(s->stream));
  *lnl = terms_lnl(s);
  return GEMS_OK;
}

size_t newton_slot_bytes() { return sizeof(ulonglong2) * 2 * kMaxClusters * kSlotStride; }

int newton_result(Session *s, double *opt_len, int *nevals) {
  GEMS_CUDA(cudaStreamSynchronize(s->stream));
  *opt_len = s->h_result[0];
  *nevals = (int)s->h_result[1];
  return (int)s->h_result[2];
}

int launch_newton_async(Session *s, const gems_branch *br, double guess, double min_len,
                        double max_len, double xacc, int max_steps, const gems_op *ops,
                        int nops) {
  DevCtx c = s->ctx();
  const Split sp = split_of(s->block, s->desc.ncat);
  const void *fn = kernels_for(s, br != nullptr, sp.E2).newton;
  const int nsm = s->nsm;
  const size_t table = sizeof(double) * 2 * sp.L * sp.E2;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;  // all clusters of a launch resident together
  attr[1].val.cooperative = 1;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(newton_threads(sp.E2));
  cfg.dynamicSmemBytes =
      3 * table + sizeof(double) * small_doubles(nops, s->desc.ncat, mixed_of(s));
  cfg.stream = s->stream;
  cfg.attrs = attr;
  auto fit = [&](int &n, int size) {  // clusters of this launch that the GPU holds at once
    if (n >= 0) return n;
    if (size == 16 && cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                           1) != cudaSuccess) {
      cudaGetLastError();
      return n = 0;
    }
    attr[0].val.clusterDim.x = size;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(size);
    int m = 0;
    if (cudaOccupancyMaxActiveClusters(&m, fn, &cfg) != cudaSuccess) {
      cudaGetLastError();
      m = 0;
    }
    return n = m;
  };
  // One block per SM at most, two patterns a thread where that fills them (a pair costs little
  // more than one): one cluster of up to 16 blocks, which also holds up to the register rows of
  // its threads, else clusters of 8, as many as the GPU takes at once.
  long per = cfg.blockDim.x / sp.L;
  const long held = sp.E2 <= 2 ? 4 : 2;
  int *fits = s->newton_fit[br != nullptr];
  const int most = std::max(1, nsm / s->newton_share);
  const long want = (s->P + 2 * per - 1) / (2 * per);
  const int one = most >= 16 && fit(fits[1], 16) > 0 ? 16 : 8;  // the largest single cluster
  int cluster = 1, clusters = 1;
  if (s->P <= one * per * held || most < 16 || fit(fits[0], 8) < 2) {
    while (cluster < want && 2 * cluster <= std::min(most, one)) cluster *= 2;
  } else {
    cluster = 8;
    clusters = (int)std::min<long>({(want + 7) / 8, most / 8, fits[0], kMaxClusters});
  }
  // A share of the GPU that does not hold all rows reads the others again in every evaluation.
  // Blocks that hold none have more threads to an SM, and the same share of them is on more SMs;
  // theta is formed before, by the whole GPU.  Clusters as small as the slots allow, so that few
  // blocks of the share are lost to rounding.  A 16th of the GPU, blocks that hold rows / that
  // hold none: 60,000 patterns of 4 states and 4 categories 221 / 102 us, 100,000 of 20 states
  // 1,964 / 757, 8,000 of 61 states and 9 categories 5,232 / 1,396; a quarter 81 / 61, 520 / 253,
  // 1,392 / 457.  Up to twice the rows that are held the extra launch outweighs it (18,501 patterns
  // of 4 states on a quarter: 45.7 / 46.6).
  if (s->newton_share > 1 && s->P > 2 * cluster * clusters * per * held) {
    if (br)
      if (int st = launch_terms(s, br, kStore, 2, br->length, ops, nops)) return st;
    br = nullptr;
    nops = 0;
    fn = memory_kernels(sp.E2).stream;
    cfg.blockDim = dim3(stream_threads(sp.E2));
    cfg.dynamicSmemBytes = 5 * table;
    per = cfg.blockDim.x / sp.L;
    const int share = std::max(1, stream_ctas(sp.E2) * nsm / s->newton_share);
    cluster = 1;
    while (cluster < 8 && share > kMaxClusters * cluster) cluster *= 2;
    clusters = (int)std::min<long>({(s->P + 2 * cluster * per - 1) / (2 * cluster * per),
                                    share / cluster, kMaxClusters});
    if (fit(s->stream_fit, 8) > 0) clusters = std::min(clusters, s->stream_fit * 8 / cluster);
  }
  attr[0].val.clusterDim.x = cluster;
  cfg.numAttrs = clusters > 1 ? 2 : 1;
  cfg.gridDim = dim3(cluster * clusters);
  SmallOps o = small_list(ops, nops);
  NewtonArgs a{};
  if (br) a.br = *br;
  a.guess = guess;
  a.x1 = min_len;
  a.x2 = max_len;
  a.xacc = xacc;
  a.maxstep = max_steps;
  a.L = sp.L;
  a.cluster = cluster;
  a.slots = reinterpret_cast<ulonglong2 *>(s->d_slots);
  a.tag0 = (unsigned long long)(++s->newton_launches) << 32;
  a.result = s->h_result;
  void *args[] = {&c, &a, &o};
  cudaEvent_t ev0;
  if (int st = prof_begin(s, 5, &ev0)) return st;
  GEMS_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
  s->launches++;
  return prof_end(s, 5, ev0);
}

int check_barrier_timeout(int device, int *status) {
  GEMS_CUDA(cudaSetDevice(device));
  ulonglong2 *slots = nullptr;
  int *flag = nullptr;
  GEMS_CUDA(cudaMalloc((void **)&slots, newton_slot_bytes()));
  cudaError_t e = cudaMalloc((void **)&flag, 2 * sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(slots, 0, newton_slot_bytes());
  if (e == cudaSuccess) e = cudaMemset(flag, 0, 2 * sizeof(int));
  if (e == cudaSuccess) {
    void *args[] = {&slots, &flag};
    e = cudaLaunchCooperativeKernel((void *)k_exchange_probe, dim3(2), dim3(32), args, 0, nullptr);
  }
  if (e == cudaSuccess) {
    int *second = flag + 1;
    void *args[] = {&second};
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(32);
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelExC(&cfg, (void *)k_cluster_probe, args);
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  int h[2] = {-1, -1};
  if (e == cudaSuccess) e = cudaMemcpy(h, flag, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(slots);
  cudaFree(flag);
  if (e != cudaSuccess) return cuda_status(e, "exchange probe");
  *status = h[0] == GEMS_ERR_TIMEOUT ? h[1] : h[0];
  return GEMS_OK;
}

}  // namespace gems
