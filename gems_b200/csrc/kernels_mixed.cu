// kernels_mixed.cu -- mixed-precision form: FP32 real-space partials, FP64 everywhere else.
//
// Partials are stored as non-negative real-space vectors (FP32), pattern-major like the FP64
// form.  One node update per category c is
//      out[c] = (P_c(t_L) . L[c]) (*) (P_c(t_R) . R[c]),   P_c(t) = evec diag(exp(eval r_c t)) inv_evec
// with P built in FP64 and rounded once to FP32 (4n^2 flops instead of the eigen-space 6n^2;
// no cancellation since every term is >= 0).  Underflow is handled per pattern (NORM) or per
// (pattern, category) (SAFE): below 2^-64 the values are multiplied by 2^64 and a uint16
// counter is incremented; each count is worth 64*log(2) in the log-likelihood.
// The branch terms are FP64: both partials are lifted to the eigen basis in FP64
// (inv_evec . real), and theta / the log-likelihood reduction / the derivative sums / Newton
// are the FP64 kernels' (kernels_branch.cu), so every accepted length is re-evaluated in FP64.
#include <algorithm>
#include <climits>
#include <cmath>
#include <string>

#include "gems_internal.cuh"

namespace gems {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float group_maxf(float v, int G) {
  for (int o = 1; o < G; o <<= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// P_c(t) for both children of every op (FP64 -> FP32), and tip tables P_c . indicator.
// opmats (as float): [op][side][C][n][n] then [op][side][unknown+1][C][n]; grid (nops, 2).
__global__ void k_prep_ops_mixed(DevCtx c, const DevOp *ops, float *opm, size_t stride_f) {
  extern __shared__ double ex[];  // [C][n] exp terms
  const int k = blockIdx.x, side = blockIdx.y;
  const DevOp op = ops[k];
  const int kind = side ? op.r_kind : op.l_kind;
  const double len = side ? op.r_len : op.l_len;
  const int n = c.n, C = c.C, nn = n * n;
  for (int idx = threadIdx.x; idx < C * n; idx += blockDim.x) {
    const int cc = idx / n, i = idx - cc * n;
    ex[idx] = exp(c.eval[i] * (c.rates[cc] * len));
  }
  __syncthreads();
  float *Pm = opm + (size_t)k * stride_f + (size_t)side * C * nn;
  for (int idx = threadIdx.x; idx < C * nn; idx += blockDim.x) {
    const int cc = idx / nn, r = idx - cc * nn, x = r / n, y = r - x * n;
    double acc = 0.0;
    for (int i = 0; i < n; i++) acc = fma(c.evec[x * n + i] * ex[cc * n + i], c.inv_evec[i * n + y], acc);
    Pm[idx] = (float)fmax(acc, 0.0);
  }
  if (kind != GEMS_CHILD_TIP) return;
  __syncthreads();
  float *leaf = opm + (size_t)k * stride_f + (size_t)2 * C * nn + (size_t)side * (c.unknown + 1) * c.block;
  const int rows = (c.unknown + 1) * c.block;
  for (int idx = threadIdx.x; idx < rows; idx += blockDim.x) {
    const int s = idx / c.block, r = idx - s * c.block, cc = r / n, x = r - cc * n;
    const double *ind = c.tip_real + (size_t)s * n;
    const float *prow = Pm + (size_t)cc * nn + (size_t)x * n;
    float acc = 0.f;
    for (int y = 0; y < n; y++) acc = fmaf(prow[y], (float)ind[y], acc);
    leaf[idx] = acc;
  }
}

// N states of one (pattern, category) row; cs = floats between 4-state chunks (mix_cs)
template <int N>
__device__ __forceinline__ void load_vecf(const float *__restrict__ src, float (&v)[N], int cs) {
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N / 4; i++) {
      float4 t = __ldcg(reinterpret_cast<const float4 *>(src + (size_t)i * cs));
      v[4 * i] = t.x;
      v[4 * i + 1] = t.y;
      v[4 * i + 2] = t.z;
      v[4 * i + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = __ldcg(src + (size_t)(i / 4) * cs + i % 4);
  }
}

template <int N>
__device__ __forceinline__ void store_vecf(float *__restrict__ dst, const float (&v)[N], int cs) {
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N / 4; i++)
      *reinterpret_cast<float4 *>(dst + (size_t)i * cs) =
          make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  } else {
    // whole 4-state chunks; in the tile-major form the padding states are stored as zeros
    // (they meet zero rows of P in the tensor-core products)
#pragma unroll
    for (int i = 0; i < (N + 3) / 4; i++) {
      float4 w;
      w.x = v[4 * i];
      w.y = 4 * i + 1 < N ? v[4 * i + 1] : 0.f;
      w.z = 4 * i + 2 < N ? v[4 * i + 2] : 0.f;
      w.w = 4 * i + 3 < N ? v[4 * i + 3] : 0.f;
      if (mix_k<N>() > 0) {
        *reinterpret_cast<float4 *>(dst + (size_t)i * cs) = w;
      } else {
        dst[4 * i] = w.x;
        if (4 * i + 1 < N) dst[4 * i + 1] = w.y;
        if (4 * i + 2 < N) dst[4 * i + 2] = w.z;
        if (4 * i + 3 < N) dst[4 * i + 3] = w.w;
      }
    }
  }
}

template <int N, bool SAFE>
__device__ __forceinline__ void child_msg_f(const DevCtx &c, int kind, int id, const float *Pm,
                                            const float *leaf, long p, int gl, float (&v)[N],
                                            int &s) {
  if (kind == GEMS_CHILD_TIP) {
    const int st = c.tips[(size_t)id * c.P + p];
    const float *lt = leaf + (size_t)st * c.block + gl * N;
#pragma unroll
    for (int x = 0; x < N; x++) v[x] = __ldg(lt + x);
    s = 0;
  } else {
    const float *src = static_cast<const float *>(c.partials) + (size_t)id * c.slot_elems +
                       mix_off<N>(c, p, gl);
    float L[N];
    load_vecf<N>(src, L, mix_cs<N>());
    const float *pm = Pm + (size_t)gl * N * N;
#pragma unroll
    for (int x = 0; x < N; x++) {
      float acc = 0.f;
#pragma unroll
      for (int y = 0; y < N; y++) acc = fmaf(__ldg(pm + x * N + y), L[y], acc);
      v[x] = acc;
    }
    const uint16_t *sc = c.scale + (size_t)id * c.slot_scale;
    s = SAFE ? sc[(size_t)p * c.C + gl] : sc[p];
  }
}

template <int N, bool SAFE>
__global__ void __launch_bounds__(kThreads) k_traverse_mixed(DevCtx c, const DevOp *__restrict__ ops,
                                                             int nops, const float *__restrict__ opm,
                                                             size_t stride_f, int p0, int p1) {
  const int G = c.G;
  const int gl = threadIdx.x & (G - 1);
  const long p = p0 + ((long)blockIdx.x * blockDim.x + threadIdx.x) / G;
  const bool act = p < p1 && gl < c.C;
  const int C = c.C;
  const size_t nnC = (size_t)C * N * N;
  float *part = static_cast<float *>(c.partials);
  for (int k = 0; k < nops; k++) {
    const DevOp op = ops[k];
    const float *mats = opm + (size_t)k * stride_f;
    const bool tiptip = op.l_kind == GEMS_CHILD_TIP && op.r_kind == GEMS_CHILD_TIP;
    float out[N];
    float lh_max = 0.f;
    int sl = 0, sr = 0;
    if (act) {
      float vl[N], vr[N];
      child_msg_f<N, SAFE>(c, op.l_kind, op.l_id, mats, mats + 2 * nnC, p, gl, vl, sl);
      child_msg_f<N, SAFE>(c, op.r_kind, op.r_id, mats + nnC,
                           mats + 2 * nnC + (size_t)(c.unknown + 1) * c.block, p, gl, vr, sr);
#pragma unroll
      for (int x = 0; x < N; x++) {
        out[x] = vl[x] * vr[x];
        lh_max = fmaxf(lh_max, out[x]);
      }
    }
    if (!SAFE) lh_max = group_maxf(lh_max, G);
    int s_out = sl + sr;
    if (act) {
      if (!tiptip && lh_max < kScaleThrF && c.invar[p] == 0.0) {
#pragma unroll
        for (int x = 0; x < N; x++) out[x] *= 18446744073709551616.0f;  // 2^64
        s_out += 1;
      }
      store_vecf<N>(part + (size_t)op.dst_slot * c.slot_elems + mix_off<N>(c, p, gl), out, mix_cs<N>());
      uint16_t *sc = c.scale + (size_t)op.dst_slot * c.slot_scale;
      if (SAFE)
        sc[(size_t)p * C + gl] = (uint16_t)s_out;
      else if (gl == 0)
        sc[p] = (uint16_t)s_out;
    }
    __syncwarp();
  }
}

// ----------------------------------------------------------------------------------------
// theta (FP64, eigen basis) of a 20- or 61-state branch from its FP32 real partials, and its lnL.
// Lifting a row to the eigen basis is a product with inv_evec, done on the FP64 mma (m8n8k4) for
// the 8 patterns of a warp, both ends of the branch on the same fragments of inv_evec.  Lane
// (g, t) = (lane / 4, lane % 4) holds the states 4s + t of pattern g as A fragments (K steps s) and,
// with column n = 2 t' + e of N tile m standing for state 8m + 4e + t', the same states of the
// result; a warp reads 128 contiguous bytes of the tile-major partials per K step, and the sums
// run in index order.
// Bound by FP64 throughput, 2 x 8 x 16 mma a category and 8 patterns for 61 states: 23 us for
// 3,780 patterns of 61 states and 50 us for 98,762 of 20 (4 categories), where one thread per
// (pattern, category) with its rows in local memory took 65 and 74.  The last block adds the
// blocks' sums in index order and writes them to pinned host memory.
// ----------------------------------------------------------------------------------------
constexpr int kWarpsL = 4;

template <int N, bool SAFE>
__device__ __forceinline__ void theta_mixed(const DevCtx &c, const gems_branch &br, int nblocks,
                                            int want_lnl, int store_theta, unsigned int *ticket,
                                            double *out) {
  constexpr int S = (N + 3) / 4, M = (N + 7) / 8;
  static_assert(mix_k<N>() == S, "K steps are the chunks of the tile-major rows");
  extern __shared__ double sm[];  // inv_evec as B fragments [S][M][32], then val [C][N]
  __shared__ double sh[2][32];
  __shared__ bool last;
  double *val = sm + S * M * 32;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  for (int i = threadIdx.x; i < S * M * 32; i += blockDim.x) {
    const int l = i & 31, m = (i >> 5) % M, k = 4 * ((i >> 5) / M) + (l & 3), n = l >> 2;
    const int x = 8 * m + 4 * (n & 1) + (n >> 1);
    sm[i] = k < N && x < N ? c.inv_evec[x * N + k] : 0.0;
  }
  if (want_lnl)
    for (int i = threadIdx.x; i < c.block; i += blockDim.x)
      val[i] = exp(c.eval[i % N] * (c.rates[i / N] * br.length)) * c.props[i / N];
  __syncthreads();
  const float *part = static_cast<const float *>(c.partials);
  const float *dad = part + (size_t)br.dad_slot * c.slot_elems;
  const float *node = part + (size_t)br.node_id * c.slot_elems;
  const uint16_t *sd = c.scale + (size_t)br.dad_slot * c.slot_scale;
  const uint16_t *sn = c.scale + (size_t)br.node_id * c.slot_scale;
  const bool is_tip = br.node_kind == GEMS_CHILD_TIP;
  // P is a multiple of 64: whole warps of patterns.  nblocks sums whatever the grid is: a batched
  // call adds in the order of the session's own.
  for (int vb = blockIdx.x; vb < nblocks; vb += gridDim.x) {
    double v[2] = {0.0, 0.0};
    for (long p0 = 8l * ((long)vb * kWarpsL + (threadIdx.x >> 5)); p0 < c.P;
         p0 += 8l * kWarpsL * nblocks) {
      const long p = p0 + g;
      const int st = is_tip ? min((int)c.tips[(size_t)br.node_id * c.P + p], c.unknown) : 0;
      int ms;
      if (SAFE) {
        ms = INT_MAX;
        for (int cc = t; cc < c.C; cc += 4)
          ms = min(ms, (int)sd[p * c.C + cc] + (is_tip ? 0 : (int)sn[p * c.C + cc]));
        ms = min(ms, __shfl_xor_sync(0xffffffffu, ms, 1));
        ms = min(ms, __shfl_xor_sync(0xffffffffu, ms, 2));
      } else {
        ms = (int)sd[p] + (is_tip ? 0 : (int)sn[p]);
      }
      double lh = 0.0;
      for (int cc = 0; cc < c.C; cc++) {
        const size_t o = mix_off<N>(c, p, cc) + t;
        float a[S], b[S];
#pragma unroll
        for (int s = 0; s < S; s++) {
          a[s] = __ldcg(dad + o + (size_t)s * mix_cs<N>());
          b[s] = is_tip ? 0.f : __ldcg(node + o + (size_t)s * mix_cs<N>());
        }
        int ss = ms;
        if (SAFE) ss = (int)sd[p * c.C + cc] + (is_tip ? 0 : (int)sn[p * c.C + cc]);
        double x[M][2], y[M][2];
#pragma unroll
        for (int m = 0; m < M; m++) x[m][0] = x[m][1] = y[m][0] = y[m][1] = 0.0;
        __syncwarp();
#pragma unroll
        for (int s = 0; s < S; s++) {
          double f[M];
#pragma unroll
          for (int m = 0; m < M; m++) f[m] = sm[(s * M + m) * 32 + lane];
#pragma unroll
          for (int m = 0; m < M; m++) dmma(x[m], (double)a[s], f[m]);
          if (!is_tip) {
#pragma unroll
            for (int m = 0; m < M; m++) dmma(y[m], (double)b[s], f[m]);
          }
        }
        // a category one count above the minimum is 2^-64 smaller; two or more: negligible
        const double up = ss == ms ? 1.0 : 5.421010862427522e-20;
        double *dst = c.theta + (size_t)p * c.block + cc * N + t;
#pragma unroll
        for (int s = 0; s < S; s++) {
          if (4 * s + t >= N) continue;
          const double e =
              is_tip ? __ldg(c.tip + (size_t)st * N + 4 * s + t) : y[s >> 1][s & 1];
          double th = e * x[s >> 1][s & 1];
          if (SAFE) th = ss > ms + 1 ? 0.0 : th * up;
          if (store_theta) dst[4 * s] = th;
          if (want_lnl) lh = fma(val[cc * N + 4 * s + t], th, lh);
        }
      }
      if (store_theta && t == 0) c.scale_all[p] = (double)ms * kLogScaleThrF;
      if (!want_lnl) continue;
      lh += __shfl_xor_sync(0xffffffffu, lh, 1);
      lh += __shfl_xor_sync(0xffffffffu, lh, 2);
      if (t == 0) {
        const double plh = log(fabs(lh) + c.invar[p]) + ms * kLogScaleThrF;
        c.pattern_lh[p] = plh;
        if (p < c.nptn) {
          const double f = c.freq[p];
          v[0] += plh * f;
          v[1] += (isfinite(plh) ? plh : 4.0 * kLogScaleThr) * f;
        }
      }
    }
    if (!want_lnl) continue;
    block_sum<2>(v, sh);
    if (threadIdx.x == 0) {
      __stcg(c.red + 2 * vb, v[0]);
      __stcg(c.red + 2 * vb + 1, v[1]);
    }
  }
  if (!want_lnl) return;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double v[2] = {0.0, 0.0};
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
    v[0] += __ldcg(c.red + 2 * b);
    v[1] += __ldcg(c.red + 2 * b + 1);
  }
  block_sum<2>(v, sh);
  if (threadIdx.x == 0) {
    out[0] = v[0];
    out[1] = v[1];
    *ticket = 0;  // ready for the next launch
  }
}
template <int N, bool SAFE>
__global__ void __launch_bounds__(32 * kWarpsL, N == 61 ? 3 : 5)
    k_theta_mixed(DevCtx c, gems_branch br, int want_lnl, int store_theta, unsigned int *ticket,
                  double *out) {
  theta_mixed<N, SAFE>(c, br, gridDim.x, want_lnl, store_theta, ticket, out);
}

// the lnL of one branch of each of many sessions (candidate models), blockIdx.y its number
constexpr int kLiftBatch = 32;
struct LiftJob {
  DevCtx c;
  gems_branch br;
  unsigned int *ticket;
  double *out;
};
struct LiftBatch {
  LiftJob job[kLiftBatch];
};
template <int N, bool SAFE>
__global__ void __launch_bounds__(32 * kWarpsL, N == 61 ? 3 : 5)
    k_lnl_mixed_batch(const __grid_constant__ LiftBatch b, int nblocks) {
  const LiftJob &j = b.job[blockIdx.y];
  theta_mixed<N, SAFE>(j.c, j.br, nblocks, 1, 0, j.ticket, j.out);
}

}  // namespace

#define GEMS_DISPATCH_NM(n, NAME, ...)                                  \
  switch (n) {                                                          \
    case 4: { constexpr int NS = 4; __VA_ARGS__; } break;               \
    case 20: { constexpr int NS = 20; __VA_ARGS__; } break;             \
    case 61: { constexpr int NS = 61; __VA_ARGS__; } break;             \
    default: set_error(std::string(NAME) + ": unsupported state count"); \
      return GEMS_ERR_BAD_ARG;                                          \
  }

int launch_prep_ops_mixed(Session *s, int nops) {
  if (nops <= 0) return GEMS_OK;
  DevCtx c = s->ctx();
  const size_t smem = sizeof(double) * s->desc.ncat * s->desc.nstates;
  k_prep_ops_mixed<<<dim3(nops, 2), 256, smem, s->stream>>>(
      c, s->d_ops, reinterpret_cast<float *>(s->d_opmats), s->op_stride);
  s->launches++;
  GEMS_CUDA(cudaGetLastError());
  return GEMS_OK;
}

int launch_traverse_mixed(Session *s, int nops, int p0, int p1) {
  if (nops <= 0 || p1 <= p0) return GEMS_OK;
  DevCtx c = s->ctx();
  const int grid = (int)(((long)(p1 - p0) * s->G + kThreads - 1) / kThreads);
  const bool safe = s->desc.scaling == GEMS_SCALE_SAFE;
  const float *opm = reinterpret_cast<const float *>(s->d_opmats);
  cudaEvent_t ev0;
  if (int st = prof_begin(s, 0, &ev0)) return st;
  GEMS_DISPATCH_NM(s->desc.nstates, "traverse_mixed",
    if (safe) k_traverse_mixed<NS, true><<<grid, kThreads, 0, s->stream>>>(c, s->d_ops, nops, opm, s->op_stride, p0, p1);
    else k_traverse_mixed<NS, false><<<grid, kThreads, 0, s->stream>>>(c, s->d_ops, nops, opm, s->op_stride, p0, p1));
  s->launches++;
  GEMS_CUDA(cudaGetLastError());
  return prof_end(s, 0, ev0);
}

// blocks of k_theta_mixed: at most one wave
static int lift_blocks(const Session *s) {
  return std::min(s->nsm * (s->desc.nstates == 61 ? 3 : 5), (s->P / 8 + kWarpsL - 1) / kWarpsL);
}

// theta (and optionally the branch lnL) from the two FP32 partials of br, 20 or 61 states
int enqueue_theta_mixed(Session *s, const gems_branch *br, bool want_lnl, bool store_theta) {
  DevCtx c = s->ctx();
  const int n = s->desc.nstates;
  const bool safe = s->desc.scaling == GEMS_SCALE_SAFE;
  const size_t smem =
      sizeof(double) * ((size_t)((n + 3) / 4) * ((n + 7) / 8) * 32 + (want_lnl ? s->block : 0));
  const int grid = lift_blocks(s);
  cudaEvent_t ev0;
  if (int st = prof_begin(s, want_lnl ? 1 : 2, &ev0)) return st;
  const int wl = want_lnl ? 1 : 0, stt = store_theta ? 1 : 0;
  auto *fn = n == 20 ? (safe ? k_theta_mixed<20, true> : k_theta_mixed<20, false>)
                     : (safe ? k_theta_mixed<61, true> : k_theta_mixed<61, false>);
  fn<<<grid, 32 * kWarpsL, smem, s->stream>>>(c, *br, wl, stt, s->d_bar, s->h_result);
  s->launches++;
  GEMS_CUDA(cudaGetLastError());
  return prof_end(s, want_lnl ? 1 : 2, ev0);
}

// the lnL of a branch of each session (as enqueue_theta_mixed; 20 or 61 states, one state,
// category and pattern count and one scaling), 32 sessions a launch (their contexts fit a
// launch's parameters), on the first one's stream.  A session of a few thousand patterns fills
// a quarter of the GPU for 23 us: with its own launch, and its own copy of the op list before it,
// 32 codon models of 3,780 patterns took 12.6 ms an evaluation, with both shared 12.0.
int enqueue_lnl_mixed_batch(Session *const *ss, const gems_branch *br, int n) {
  Session *s0 = ss[0];
  const int ns = s0->desc.nstates;
  const bool safe = s0->desc.scaling == GEMS_SCALE_SAFE;
  const size_t smem =
      sizeof(double) * ((size_t)((ns + 3) / 4) * ((ns + 7) / 8) * 32 + s0->block);
  auto *fn = ns == 20 ? (safe ? k_lnl_mixed_batch<20, true> : k_lnl_mixed_batch<20, false>)
                      : (safe ? k_lnl_mixed_batch<61, true> : k_lnl_mixed_batch<61, false>);
  for (int i0 = 0; i0 < n; i0 += kLiftBatch) {
    const int m = std::min(kLiftBatch, n - i0);
    LiftBatch b{};
    for (int i = 0; i < m; i++) {
      Session *s = ss[i0 + i];
      b.job[i] = {s->ctx(), br[i0 + i], s->d_bar, s->h_result};
    }
    // about one wave of blocks over all sessions: each block lays out its inv_evec once
    const int most = lift_blocks(s0);
    const int per = std::min(most, std::max(1, s0->nsm * (ns == 61 ? 3 : 5) / m));
    cudaEvent_t ev0;
    if (int st = prof_begin(s0, 1, &ev0)) return st;
    fn<<<dim3(per, m), 32 * kWarpsL, smem, s0->stream>>>(b, most);
    s0->launches++;
    GEMS_CUDA(cudaGetLastError());
    if (int st = prof_end(s0, 1, ev0)) return st;
  }
  return GEMS_OK;
}

}  // namespace gems
