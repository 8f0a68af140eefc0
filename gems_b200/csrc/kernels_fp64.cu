// kernels_fp64.cu -- FP64 eigen-space likelihood kernels for sm_100a.
//
// Layout in HBM (per partial slot): pattern-major, then category, then state:
//   partial[p][c][x] at ((p * C) + c) * n + x, doubles.  One pattern's block of C*n values is
//   contiguous, so a group of G (= next pow2 >= C) adjacent lanes handles one pattern, lane c
//   owning category c: a warp covers 32/G consecutive patterns and reads/writes one
//   contiguous span (coalesced), and the per-pattern max / min / sums are warp shuffles.
//
// Arithmetic follows tree/phylokernelnew.h (reversible, non-site-specific kernel):
//   E_c(t)[x][i]   = evec[x][i] * exp(eval[i] * r_c * t)                          (:1043-1062)
//   tip table      = sum_i E_c[x][i] * tip[state][i], unknown row = 1                (:1064-1088)
//   partial        = inv_evec . ((E_L . L) * (E_R . R)) per category               (:1911-2035)
//   NORM scaling   : max |partial| over the pattern's block < 2^-256 and ptn_invar == 0
//                    -> ldexp(.,256), scale_num[p] += 1; tip-tip never scaled     (:2019-2034)
//   SAFE scaling   : the same per (pattern, category)                             (:1997-2013)
// The branch terms are in kernels_branch.cu.
#include <cmath>
#include <string>

#include "gems_internal.cuh"

namespace gems {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ double group_max(double v, int G) {
  for (int o = 1; o < G; o <<= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// ----------------------------------------------------------------------------------------
// Per-op transition tables (computePartialInfo): E_L, E_R and tip tables for tip children.
// grid = (nops, 2 sides)
// ----------------------------------------------------------------------------------------
__global__ void k_prep_ops(DevCtx c, const DevOp *ops, double *opmats, size_t stride) {
  const int k = blockIdx.x, side = blockIdx.y;
  const DevOp op = ops[k];
  const int kind = side ? op.r_kind : op.l_kind;
  const double len = side ? op.r_len : op.l_len;
  const int n = c.n, C = c.C, nn = n * n;
  double *E = opmats + (size_t)k * stride + (size_t)side * C * nn;
  for (int idx = threadIdx.x; idx < C * nn; idx += blockDim.x) {
    const int cc = idx / nn, r = idx - cc * nn, x = r / n, i = r - x * n;
    E[idx] = c.evec[x * n + i] * exp(c.eval[i] * (c.rates[cc] * len));
  }
  if (kind != GEMS_CHILD_TIP) return;
  __syncthreads();
  double *leaf = opmats + (size_t)k * stride + (size_t)2 * C * nn +
                 (size_t)side * (c.unknown + 1) * c.block;
  const int nrow = c.unknown * c.block;
  for (int idx = threadIdx.x; idx < nrow; idx += blockDim.x) {
    const int s = idx / c.block, r = idx - s * c.block;
    const double *e = E + (size_t)r * n;
    const double *t = c.tip + (size_t)s * n;
    double acc = 0.0;
    for (int i = 0; i < n; i++) acc = fma(e[i], t[i], acc);
    leaf[idx] = acc;
  }
  for (int idx = threadIdx.x; idx < c.block; idx += blockDim.x) leaf[nrow + idx] = 1.0;
}

// Real-space message from one child for category gl: E_c . child (internal) or the tip row.
template <int N, bool SAFE>
__device__ __forceinline__ void child_msg(const DevCtx &c, int kind, int id, const double *E,
                                          const double *leaf, long p, int gl, double (&v)[N],
                                          int &s) {
  if (kind == GEMS_CHILD_TIP) {
    const int st = c.tips[(size_t)id * c.P + p];
    const double *lt = leaf + (size_t)st * c.block + gl * N;
#pragma unroll
    for (int x = 0; x < N; x++) v[x] = __ldg(lt + x);
    s = 0;
  } else {
    const double *slot = static_cast<const double *>(c.partials) + (size_t)id * c.slot_elems;
    double L[N];
    load_row<N>(slot, c, p, gl, L);
    const double *e = E + (size_t)gl * N * N;
#pragma unroll
    for (int x = 0; x < N; x++) {
      double acc = 0.0;
#pragma unroll
      for (int i = 0; i < N; i++) acc = fma(__ldg(e + x * N + i), L[i], acc);
      v[x] = acc;
    }
    const uint16_t *sc = c.scale + (size_t)id * c.slot_scale;
    s = SAFE ? sc[(size_t)p * c.C + gl] : sc[p];
  }
}

// Whole traversal for the patterns [p0, p1) of this launch, p1 <= P: every op in postorder.
// A pattern is always handled by the same lane group, so children written by an earlier op are
// read back by the same warp (ordered by __syncwarp); no inter-CTA dependency exists.
template <int N, bool SAFE>
__global__ void __launch_bounds__(kThreads) k_traverse(DevCtx c, const DevOp *__restrict__ ops,
                                                       int nops, const double *__restrict__ opmats,
                                                       size_t stride, int p0, int p1) {
  const int G = c.G;
  const int gl = threadIdx.x & (G - 1);
  const long p = p0 + ((long)blockIdx.x * blockDim.x + threadIdx.x) / G;
  const bool act = p < p1 && gl < c.C;
  const int C = c.C;
  const size_t nnC = (size_t)C * N * N;
  double *part = static_cast<double *>(c.partials);
  for (int k = 0; k < nops; k++) {
    const DevOp op = ops[k];
    const double *mats = opmats + (size_t)k * stride;
    const bool tiptip = op.l_kind == GEMS_CHILD_TIP && op.r_kind == GEMS_CHILD_TIP;
    double out[N];
    double lh_max = 0.0;
    int sl = 0, sr = 0;
    if (act) {
      double tmp[N];
      {
        double vl[N];
        child_msg<N, SAFE>(c, op.l_kind, op.l_id, mats, mats + 2 * nnC, p, gl, vl, sl);
        double vr[N];
        child_msg<N, SAFE>(c, op.r_kind, op.r_id, mats + nnC,
                           mats + 2 * nnC + (size_t)(c.unknown + 1) * c.block, p, gl, vr, sr);
#pragma unroll
        for (int x = 0; x < N; x++) tmp[x] = vl[x] * vr[x];
      }
#pragma unroll
      for (int j = 0; j < N; j++) {
        double acc = 0.0;
#pragma unroll
        for (int x = 0; x < N; x++) acc = fma(__ldg(c.inv_evec + j * N + x), tmp[x], acc);
        out[j] = acc;
        lh_max = fmax(lh_max, fabs(acc));
      }
    }
    if (!SAFE) lh_max = group_max(lh_max, G);
    int s_out = sl + sr;
    if (act) {
      if (!tiptip && lh_max < kScaleThr && c.invar[p] == 0.0) {
#pragma unroll
        for (int j = 0; j < N; j++) out[j] = ldexp(out[j], kScaleExp);
        s_out += 1;
      }
      store_row<N>(part + (size_t)op.dst_slot * c.slot_elems, c, p, gl, out);
      uint16_t *sc = c.scale + (size_t)op.dst_slot * c.slot_scale;
      if (SAFE)
        sc[(size_t)p * C + gl] = (uint16_t)s_out;
      else if (gl == 0)
        sc[p] = (uint16_t)s_out;
    }
    __syncwarp();
  }
}

}  // namespace

// ---- dispatch helpers over the state count -----------------------------------------------
#define GEMS_DISPATCH_N(n, NAME, ...)                                  \
  switch (n) {                                                         \
    case 4: { constexpr int NS = 4; __VA_ARGS__; } break;              \
    case 20: { constexpr int NS = 20; __VA_ARGS__; } break;            \
    case 61: { constexpr int NS = 61; __VA_ARGS__; } break;            \
    default: set_error(std::string(NAME) + ": unsupported state count"); \
      return GEMS_ERR_BAD_ARG;                                         \
  }

int launch_prep_ops(Session *s, int nops) {
  if (nops <= 0) return GEMS_OK;
  DevCtx c = s->ctx();
  k_prep_ops<<<dim3(nops, 2), 256, 0, s->stream>>>(c, s->d_ops, s->d_opmats, s->op_stride);
  s->launches++;
  GEMS_CUDA(cudaGetLastError());
  return GEMS_OK;
}

int launch_traverse(Session *s, int nops, int p0, int p1) {
  if (nops <= 0 || p1 <= p0) return GEMS_OK;
  DevCtx c = s->ctx();
  const int grid = (int)(((long)(p1 - p0) * s->G + kThreads - 1) / kThreads);
  const bool safe = s->desc.scaling == GEMS_SCALE_SAFE;
  cudaEvent_t ev0;
  if (int st = prof_begin(s, 0, &ev0)) return st;
  GEMS_DISPATCH_N(s->desc.nstates, "traverse",
    if (safe) k_traverse<NS, true><<<grid, kThreads, 0, s->stream>>>(c, s->d_ops, nops, s->d_opmats, s->op_stride, p0, p1);
    else k_traverse<NS, false><<<grid, kThreads, 0, s->stream>>>(c, s->d_ops, nops, s->d_opmats, s->op_stride, p0, p1));
  s->launches++;
  GEMS_CUDA(cudaGetLastError());
  return prof_end(s, 0, ev0);
}

}  // namespace gems
