// branch_kernels.cuh -- the kernels of the branch terms: log-likelihood, theta, derivatives, lnL from
// theta, and the Newton loop on the device (phylokernelnew.h:2053-3495, utils/optimization.cpp:422-499).
//
// Every term is a dot product over the C * n elements of a pattern's theta = node (*) dad (eigen
// space) with tables of exp(eval_i r_c t):
//      lh = sum theta v0,   d1 = sum theta v1,   d2 = sum theta v2
// so one layout serves all state counts: L lanes share a pattern (a power of two, at least C),
// each lane taking a few element pairs (pair_of): a warp reads whole lines of the pattern-major
// theta and partials whatever n is.  (One lane per category row, the form before, read n = 20 and 61
// with a stride of n doubles: two to four times the sectors.)
//
// Theta is formed by the kernel that uses it, from the two partials, and stored for the calls
// after it; the tables are computed by every block; the last block to finish adds the per-block
// sums in index order and writes the result to pinned host memory.  One launch per call instead
// of a table, a theta, a term and a reduction kernel and a copy: lnL and the derivatives of 29
// branches of a 16-taxon, 3,801-pattern tree, bound by launches, take 0.93 ms instead of 1.29 ms;
// the lnL of a 450,000-pattern tree from its partials and 256 replicates 141 us instead of 170.
//
// Reductions over patterns are deterministic: a fixed tree per block, then index order.
//
// A translation unit instantiates the kernels of one source of theta (branch_*.cu): a process loads
// a unit's module whole when it first launches one of its kernels, 0.3 ms a kernel, so that the
// first branch call of a process took 18 ms with all of them in one unit.
#pragma once

#include <climits>
#include <cmath>
#include <type_traits>

#include "gems_internal.cuh"
#include "tc_common.cuh"

namespace gems {

// k_terms and k_newton of one source of theta, state count and split; of theta in memory also the
// streaming k_newton
struct BranchFns {
  const void *terms, *newton, *stream;
};

namespace {

// where theta comes from
enum : int {
  kMem = 0,  // c.theta
  kT4,       // FP64 partials, 4 states (tile-major)
  kR20,      // FP64 partials, 20 states (pattern-major)
  kR61,      // FP64 partials, 61 states
  kM4        // FP32 real-space partials, 4 states: lifted to the eigen basis in FP64
};
enum : int { kStore = 1, kLnl = 2, kDerv = 4 };
constexpr int kSmallOps = 16;           // ops of a list that a branch call runs itself
constexpr int kSmallPatterns = 1 << 15;

template <int SRC>
__host__ __device__ constexpr int src_states() {
  return SRC == kR20 ? 20 : (SRC == kR61 ? 61 : 4);
}

// Lanes per pattern and pairs per lane for a block of B = C * n elements: at least C lanes (the
// SAFE counters of a pattern, one per lane), more until a lane holds at most five pairs.
struct Split {
  int L, E2;
};
inline Split split_of(int B, int C) {
  const int u = (B + 1) / 2;
  int L = 2;
  while (L < C) L *= 2;
  while (L < 32 && (u + L - 1) / L > 5) L *= 2;
  const int need = (u + L - 1) / L;
  for (int e : {1, 2, 3, 4, 5, 8, 12})
    if (need <= e) return {L, e};
  return {L, 16};  // 61 states, 16 categories: 488 pairs on 32 lanes
}

// the pair that lane l holds at q: strided, so that a warp reads whole lines, except for one or two
// pairs per lane (4 states), where a lane holds a category's row (one 16- or 32-byte piece)
template <int E2>
__device__ __forceinline__ int pair_of(int q, int l, int L) {
  return E2 <= 2 ? l * E2 + q : q * L + l;
}

// two elements j, j + 1 (j even) of a pattern-major row of `block` doubles
__device__ __forceinline__ void row_pair(const double *row, int j, int block, double &a,
                                         double &b) {
  if (block % 2 == 0) {
    const double2 v = __ldcg(reinterpret_cast<const double2 *>(row + j));
    a = v.x, b = v.y;
  } else {
    a = __ldcg(row + j), b = j + 1 < block ? __ldcg(row + j + 1) : 0.0;
  }
}

// elements i, i + 1 of inv_evec . v (4 states)
__device__ __forceinline__ void lift2(const DevCtx &c, int i, float4 v, double &x, double &y) {
  const double *r = c.inv_evec + i * 4;
  auto row = [&](const double *q) {
    double s = fma(__ldg(q), (double)v.x, 0.0);
    s = fma(__ldg(q + 1), (double)v.y, s);
    s = fma(__ldg(q + 2), (double)v.z, s);
    return fma(__ldg(q + 3), (double)v.w, s);
  };
  x = row(r);
  y = row(r + 4);
}

// This lane's theta elements of two patterns p[0], p[1], SAFE rows brought to the pattern's
// smallest count (+1: times the scaling threshold, more: zero), and that count.  All loads are
// issued before the first is used.  All lanes of a warp call it.
template <int SRC, bool SAFE, int E2>
__device__ __forceinline__ void load_theta(const DevCtx &c, const gems_branch &br, int L, int l,
                                           const long (&p)[2], double (&th)[2][2 * E2],
                                           int (&ms)[2]) {
  constexpr int N = src_states<SRC>();
  const bool act[2] = {p[0] < c.P, p[1] < c.P};
  ms[0] = ms[1] = 0;
  if constexpr (SRC == kMem) {
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int q = 0; q < E2; q++) {
        const int j = 2 * pair_of<E2>(q, l, L);
        th[u][2 * q] = th[u][2 * q + 1] = 0.0;
        if (act[u] && j < c.block)
          row_pair(c.theta + (size_t)p[u] * c.block, j, c.block, th[u][2 * q], th[u][2 * q + 1]);
      }
    return;
  }
  const bool is_tip = br.node_kind == GEMS_CHILD_TIP;
  int tip[2] = {0, 0}, sd[2] = {0, 0}, sn[2] = {0, 0};
#pragma unroll
  for (int u = 0; u < 2; u++) {
    if (!act[u]) continue;
    if (is_tip) tip[u] = c.tips[(size_t)br.node_id * c.P + p[u]];
    if (!SAFE || l < c.C) {
      const size_t o = SAFE ? (size_t)p[u] * c.C + l : (size_t)p[u];
      sd[u] = c.scale[(size_t)br.dad_slot * c.slot_scale + o];
      if (!is_tip) sn[u] = c.scale[(size_t)br.node_id * c.slot_scale + o];
    }
  }
  if constexpr (SRC == kM4) {
    const float *part = static_cast<const float *>(c.partials);
    float4 d[2][E2], n[2][E2];
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int q = 0; q < E2; q++) {
        const int j = 2 * pair_of<E2>(q, l, L);
        d[u][q] = n[u][q] = make_float4(0.f, 0.f, 0.f, 0.f);
        // (two pairs: both of one category's row, which is read once)
        if (!act[u] || j >= c.block || (E2 == 2 && q == 1)) continue;
        const size_t o = mix_off<4>(c, p[u], j >> 2);
        d[u][q] = __ldcg(reinterpret_cast<const float4 *>(part + (size_t)br.dad_slot * c.slot_elems + o));
        if (!is_tip)
          n[u][q] = __ldcg(reinterpret_cast<const float4 *>(part + (size_t)br.node_id * c.slot_elems + o));
      }
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int q = 0; q < E2; q++) {
        const int i = 2 * pair_of<E2>(q, l, L) & 3, qq = E2 == 2 ? 0 : q;
        double dx, dy, nx, ny;
        lift2(c, i, d[u][qq], dx, dy);
        if (is_tip) {
          const double2 v = __ldg(reinterpret_cast<const double2 *>(c.tip + (size_t)tip[u] * 4 + i));
          nx = v.x, ny = v.y;
        } else {
          lift2(c, i, n[u][qq], nx, ny);
        }
        th[u][2 * q] = nx * dx;
        th[u][2 * q + 1] = ny * dy;
      }
  } else {
    const double *part = static_cast<const double *>(c.partials);
    const double *dad = part + (size_t)br.dad_slot * c.slot_elems;
    const double *node = part + (size_t)br.node_id * c.slot_elems;
    double n[2][2 * E2];
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int q = 0; q < E2; q++) {
        const int j = 2 * pair_of<E2>(q, l, L);
        double &a = th[u][2 * q], &b = th[u][2 * q + 1];
        a = b = n[u][2 * q] = n[u][2 * q + 1] = 0.0;
        if (!act[u] || j >= c.block) continue;
        if constexpr (SRC == kT4) {
          const size_t o = f64_off<4>(c, p[u], j >> 2, j & 3);
          const double2 v = __ldcg(reinterpret_cast<const double2 *>(dad + o));
          a = v.x, b = v.y;
          if (!is_tip) {
            const double2 w = __ldcg(reinterpret_cast<const double2 *>(node + o));
            n[u][2 * q] = w.x, n[u][2 * q + 1] = w.y;
          }
        } else {
          row_pair(dad + (size_t)p[u] * c.block, j, c.block, a, b);
          if (!is_tip)
            row_pair(node + (size_t)p[u] * c.block, j, c.block, n[u][2 * q], n[u][2 * q + 1]);
        }
      }
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int q = 0; q < E2; q++) {
        if (is_tip) {
          const int j = 2 * pair_of<E2>(q, l, L);
          n[u][2 * q] = __ldg(c.tip + (size_t)tip[u] * N + j % N);
          n[u][2 * q + 1] = __ldg(c.tip + (size_t)tip[u] * N + (j + 1) % N);
        }
        th[u][2 * q] *= n[u][2 * q];
        th[u][2 * q + 1] *= n[u][2 * q + 1];
      }
  }
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const int ss = sd[u] + sn[u];
    ms[u] = ss;
    if (!SAFE) continue;
    if (!act[u] || l >= c.C) ms[u] = INT_MAX;
    for (int o = 1; o < L; o <<= 1) ms[u] = min(ms[u], __shfl_xor_sync(0xffffffffu, ms[u], o));
    if (!__any_sync(0xffffffffu, act[u] && l < c.C && ss != ms[u])) continue;
    const double thr = SRC == kM4 ? 5.421010862427522e-20 /* 2^-64 */ : kScaleThr;
    const int base = (threadIdx.x & 31) & ~(L - 1);
#pragma unroll
    for (int e = 0; e < 2 * E2; e++) {
      const int j = 2 * pair_of<E2>(e >> 1, l, L) + (e & 1);
      const int k = __shfl_sync(0xffffffffu, ss, base + min(j / N, c.C - 1));
      if (k == ms[u] + 1)
        th[u][e] *= thr;
      else if (k > ms[u] + 1)
        th[u][e] = 0.0;
    }
  }
}

template <int E2>
__device__ __forceinline__ void store_theta(const DevCtx &c, int L, int l, long p,
                                            const double (&th)[2 * E2]) {
#pragma unroll
  for (int q = 0; q < E2; q++) {
    const int j = 2 * pair_of<E2>(q, l, L);
    if (j >= c.block) continue;
    double *d = c.theta + (size_t)p * c.block + j;
    if (c.block % 2 == 0) {
      *reinterpret_cast<double2 *>(d) = make_double2(th[2 * q], th[2 * q + 1]);
    } else {
      d[0] = th[2 * q];
      if (j + 1 < c.block) d[1] = th[2 * q + 1];
    }
  }
}

// eval_i r_c and prop_c of element j of the block (zero past it)
__device__ __forceinline__ void table_factors(const DevCtx &c, int j, double &cof, double &prop) {
  cof = prop = 0.0;
  if (j < c.block) {
    const int cc = j / c.n, i = j - cc * c.n;
    cof = c.eval[i] * c.rates[cc];
    prop = c.props[cc];
  }
}
// v0 = exp(eval_i r_c t) prop_c, v1 = (eval_i r_c) v0, v2 = (eval_i r_c) v1 (`len` elements each,
// nt tables)
__device__ __forceinline__ void put_tables(double t, int j, double cof, double prop, int len,
                                           int nt, double *v) {
  const double a = exp(cof * t) * prop, b = cof * a;
  v[j] = a;
  if (nt > 1) {
    v[len + j] = b;
    v[2 * len + j] = cof * b;
  }
}

// dot product of this lane's elements with a table, then the sum over the pattern's lanes
template <int E2>
__device__ __forceinline__ double dot(const double (&th)[2 * E2], const double *v, int L, int l) {
  double s = 0.0;
#pragma unroll
  for (int q = 0; q < E2; q++) {
    const double2 w = *reinterpret_cast<const double2 *>(v + 2 * pair_of<E2>(q, l, L));
    s = fma(w.x, th[2 * q], s);
    s = fma(w.y, th[2 * q + 1], s);
  }
  return s;
}
// the same of two patterns' elements, with one read of the table
template <int E2>
__device__ __forceinline__ void dot2(const double (&a)[2 * E2], const double (&b)[2 * E2],
                                     const double *v, int L, int l, double &x, double &y) {
  x = y = 0.0;
#pragma unroll
  for (int q = 0; q < E2; q++) {
    const double2 w = *reinterpret_cast<const double2 *>(v + 2 * pair_of<E2>(q, l, L));
    x = fma(w.x, a[2 * q], x);
    y = fma(w.x, b[2 * q], y);
    x = fma(w.y, a[2 * q + 1], x);
    y = fma(w.y, b[2 * q + 1], y);
  }
}
// x of the first pattern, y of the second: even lanes end with x's sum over the pattern's lanes,
// odd lanes with y's (one exchange fewer than two sums)
__device__ __forceinline__ double lanes_sum2(double x, double y, int L, int l) {
  const double keep = l & 1 ? y : x, give = l & 1 ? x : y;
  double s = keep + __shfl_xor_sync(0xffffffffu, give, 1);
  for (int o = 2; o < L; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// sums of two values over the block in a fixed tree; valid in the first warp's lane 0
template <int NW>
__device__ __forceinline__ void block_pair(double &a, double &b, double (*sh)[2]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  if (lane == 0) sh[w][0] = a, sh[w][1] = b;
  __syncthreads();
  if (w == 0) {
    a = lane < NW ? sh[lane][0] : 0.0;
    b = lane < NW ? sh[lane][1] : 0.0;
    for (int o = NW / 2; o > 0; o >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, o);
      b += __shfl_down_sync(0xffffffffu, b, o);
    }
  }
}

// ---- short op lists of 4-state sessions ---------------------------------------------------
// A branch call that needs a few node updates first (the partials between the last branch and
// this one) runs them in its own launch: with two pairs per lane (2 or more categories) a lane
// holds one category's row of a pattern, which is all that a node update needs beside the
// pattern's maximum.  The op list travels as a kernel parameter, the exponentials (mixed: P_c) are
// made in shared memory by each block, the row that the last op wrote is kept, and everything is
// stored as the traversal kernels store it: the same sums in the same order, the same bits.
// This takes an op-list copy, a table launch and a traversal launch off the chain of a call: per
// optimised branch of a 50-taxon tree with 18,501 patterns (FP64) 39 us -> 32, of NNI evaluations
// of 4,703 (mixed) 49 -> 43, per branch derivative of 3,801 (FP64) 31 -> 23.
struct SmallOps {
  int n;
  int pad;
  DevOp op[kSmallOps];
};
template <int SRC, int E2>
__host__ __device__ constexpr bool small_form() {
  return (SRC == kT4 || SRC == kM4) && E2 == 2;
}
// doubles of dynamic shared memory: evec, inv_evec, exponentials [op][side][C][4], mixed: P_c
// [op][side][C][16] floats
__host__ __device__ inline int small_doubles(int n, int C, bool mixed) {
  return n ? 32 + n * 2 * C * (mixed ? 12 : 4) : 0;
}

// by all threads of the block, followed by a barrier
template <int SRC>
__device__ __forceinline__ void small_tables(const DevCtx &c, const SmallOps &o, double *sm) {
  const int C = c.C, n = o.n * 2 * C * 4;
  double *ex = sm + 32;
  for (int i = threadIdx.x; i < 32; i += blockDim.x) sm[i] = i < 16 ? c.evec[i] : c.inv_evec[i - 16];
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int j = i & 3, cc = (i >> 2) % C, ks = (i >> 2) / C;
    const DevOp &op = o.op[ks >> 1];
    ex[i] = exp(c.eval[j] * (c.rates[cc] * (ks & 1 ? op.r_len : op.l_len)));
  }
  if constexpr (SRC == kM4) {
    __syncthreads();
    float *P = reinterpret_cast<float *>(ex + n);
    for (int i = threadIdx.x; i < 4 * n; i += blockDim.x) {
      const int y = i & 3, x = (i >> 2) & 3;
      const double *e = ex + (i >> 4) * 4;
      double acc = 0.0;
#pragma unroll
      for (int j = 0; j < 4; j++) acc = fma(sm[x * 4 + j] * e[j], sm[16 + j * 4 + y], acc);
      P[i] = (float)fmax(acc, 0.0);
    }
  }
}

// the node updates of patterns p[0], p[1] (this lane: category l); all lanes of a warp call it
template <int SRC, bool SAFE>
__device__ __forceinline__ void small_traverse(const DevCtx &c, const SmallOps &o,
                                               const double *sm, int L, int l,
                                               const long (&p)[2]) {
  using R = std::conditional_t<SRC == kM4, float, double>;
  const int C = c.C, cat = l < C ? l : 0;
  const bool act[2] = {p[0] < c.P && l < C, p[1] < c.P && l < C};
  const bool inv0[2] = {act[0] && c.invar[p[0]] == 0.0, act[1] && c.invar[p[1]] == 0.0};
  const double *ev = sm, *iv = sm + 16, *ex = sm + 32;
  const float *Pm = reinterpret_cast<const float *>(ex + o.n * 2 * C * 4);
  R *part = static_cast<R *>(c.partials);
  R last[2][4];  // the row that the last op wrote, and its counter
  int slast[2] = {0, 0}, slot = -1;
#pragma unroll
  for (int u = 0; u < 2; u++)
#pragma unroll
    for (int x = 0; x < 4; x++) last[u][x] = 0;
  for (int k = 0; k < o.n; k++) {
    const DevOp &op = o.op[k];
    R v[2][2][4];  // [side][pattern][state]
    int sc[2] = {0, 0};
#pragma unroll
    for (int side = 0; side < 2; side++) {
      const int kind = side ? op.r_kind : op.l_kind, id = side ? op.r_id : op.l_id;
      const double *d = ex + ((2 * k + side) * C + cat) * 4;
      const float4 *P = reinterpret_cast<const float4 *>(Pm) + ((2 * k + side) * C + cat) * 4;
      R row[2][4];
      if (kind == GEMS_CHILD_TIP) {
        int st[2] = {0, 0};
#pragma unroll
        for (int u = 0; u < 2; u++)
          if (act[u]) st[u] = min((int)c.tips[(size_t)id * c.P + p[u]], c.unknown);
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
          for (int x = 0; x < 4; x++)
            row[u][x] = (R)__ldg((SRC == kM4 ? c.tip_real : c.tip) + st[u] * 4 + x);
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
          for (int x = 0; x < 4; x++) {
            if constexpr (SRC == kM4) {
              const float4 r = P[x];
              v[side][u][x] = fmaf(r.w, row[u][3], fmaf(r.z, row[u][2], fmaf(r.y, row[u][1], fmaf(r.x, row[u][0], 0.f))));
            } else {
              double acc = 0.0;
#pragma unroll
              for (int i = 0; i < 4; i++) acc = fma(ev[x * 4 + i] * d[i], row[u][i], acc);
              v[side][u][x] = st[u] == c.unknown ? 1.0 : acc;
            }
          }
        continue;
      }
      const bool kept = id == slot;
#pragma unroll
      for (int u = 0; u < 2; u++) {
#pragma unroll
        for (int x = 0; x < 4; x++) row[u][x] = last[u][x];
        if (kept) {
          sc[u] += slast[u];
        } else if (act[u]) {
          const R *src = part + (size_t)id * c.slot_elems;
          if constexpr (SRC == kM4) {
            const float4 r = __ldcg(reinterpret_cast<const float4 *>(src + mix_off<4>(c, p[u], cat)));
            row[u][0] = r.x, row[u][1] = r.y, row[u][2] = r.z, row[u][3] = r.w;
          } else {
            const double2 a = __ldcg(reinterpret_cast<const double2 *>(src + f64_off<4>(c, p[u], cat, 0)));
            const double2 b = __ldcg(reinterpret_cast<const double2 *>(src + f64_off<4>(c, p[u], cat, 2)));
            row[u][0] = a.x, row[u][1] = a.y, row[u][2] = b.x, row[u][3] = b.y;
          }
          sc[u] += c.scale[(size_t)id * c.slot_scale + (SAFE ? (size_t)p[u] * C + cat : (size_t)p[u])];
        }
      }
#pragma unroll
      for (int u = 0; u < 2; u++)
#pragma unroll
        for (int x = 0; x < 4; x++) {
          if constexpr (SRC == kM4) {
            const float4 r = P[x];
            v[side][u][x] = fmaf(r.w, row[u][3], fmaf(r.z, row[u][2], fmaf(r.y, row[u][1], fmaf(r.x, row[u][0], 0.f))));
          } else {
            double acc = 0.0;
#pragma unroll
            for (int i = 0; i < 4; i++) acc = fma(ev[x * 4 + i], row[u][i] * d[i], acc);
            v[side][u][x] = acc;
          }
        }
    }
    const bool tiptip = op.l_kind == GEMS_CHILD_TIP && op.r_kind == GEMS_CHILD_TIP;
#pragma unroll
    for (int u = 0; u < 2; u++) {
      // the row's maximum as bits that compare like it (FP64: the high word; NaN counts as zero)
      int h = 0;
      if constexpr (SRC == kM4) {
        float m = 0.f;
#pragma unroll
        for (int x = 0; x < 4; x++) {
          last[u][x] = v[0][u][x] * v[1][u][x];
          m = fmaxf(m, last[u][x]);
        }
        h = __float_as_int(m);
      } else {
        double t[4];
#pragma unroll
        for (int x = 0; x < 4; x++) t[x] = v[0][u][x] * v[1][u][x];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          double acc = 0.0;
#pragma unroll
          for (int x = 0; x < 4; x++) acc = fma(iv[j * 4 + x], t[x], acc);
          last[u][j] = acc;
          const int w = __double2hiint(acc) & 0x7fffffff;
          h = max(h, w > 0x7ff00000 ? 0 : w);
        }
      }
      if (!SAFE) {
        if (!act[u]) h = 0;
        for (int q = 1; q < L; q <<= 1) h = max(h, __shfl_xor_sync(0xffffffffu, h, q));
      }
      // 2^-256, or 2^-64 as a float
      const int thr = SRC == kM4 ? 0x1f800000 : 0x2FF00000;
      if (!tiptip && h < thr && inv0[u]) {
#pragma unroll
        for (int x = 0; x < 4; x++) last[u][x] *= (R)(SRC == kM4 ? 0x1p64 : 0x1p256);
        sc[u] += 1;
      }
      slast[u] = sc[u];
      if (!act[u]) continue;
      R *dst = part + (size_t)op.dst_slot * c.slot_elems;
      if constexpr (SRC == kM4) {
        *reinterpret_cast<float4 *>(dst + mix_off<4>(c, p[u], cat)) =
            make_float4(last[u][0], last[u][1], last[u][2], last[u][3]);
      } else {
        *reinterpret_cast<double2 *>(dst + f64_off<4>(c, p[u], cat, 0)) =
            make_double2(last[u][0], last[u][1]);
        *reinterpret_cast<double2 *>(dst + f64_off<4>(c, p[u], cat, 2)) =
            make_double2(last[u][2], last[u][3]);
      }
      uint16_t *scd = c.scale + (size_t)op.dst_slot * c.slot_scale;
      if (SAFE)
        scd[(size_t)p[u] * C + cat] = (uint16_t)sc[u];
      else if (l == 0)
        scd[p[u]] = (uint16_t)sc[u];
    }
    slot = op.dst_slot;
    __syncwarp();  // NORM: the counter that lane 0 wrote is read by its pattern's lanes
  }
}

constexpr int kThreadsT = 256;
// resident blocks per SM (the registers of two patterns' elements)
constexpr int ctas_t(int e2) { return e2 <= 2 ? 3 : (e2 <= 5 ? 2 : 1); }

// One evaluation at length t: flags kStore (theta and scale_all kept), kLnl (pattern_lh; out =
// lnL, lnL with non-finite patterns clamped) or kDerv (df_frac, ddf_term; out = df, ddf); kStore
// alone: theta only.
template <int SRC, bool SAFE, int E2>
__global__ void __launch_bounds__(kThreadsT, ctas_t(E2))
    k_terms(DevCtx c, gems_branch br, double t, int L, int flags, unsigned int *ticket,
            double *out, const __grid_constant__ SmallOps ops) {
  extern __shared__ __align__(16) double tab[];
  __shared__ double sh[kThreadsT / 32][2];
  __shared__ bool last;
  const int len = 2 * L * E2;
  for (int j = threadIdx.x; j < len; j += kThreadsT) {
    double cof, prop;
    table_factors(c, j, cof, prop);
    put_tables(t, j, cof, prop, len, flags & kDerv ? 3 : 1, tab);
  }
  double *small = tab + (flags & kDerv ? 3 : 1) * len;
  if constexpr (small_form<SRC, E2>())
    if (ops.n) small_tables<SRC>(c, ops, small);
  __syncthreads();
  const int l = threadIdx.x & (L - 1);
  const long per = blockDim.x / L, step = per * gridDim.x;
  double v0 = 0.0, v1 = 0.0;
  constexpr double thr = SRC == kM4 ? kLogScaleThrF : kLogScaleThr;
  // two patterns at a time: their loads overlap, and the logarithm or the division of the first
  // is the even lanes', of the second the odd lanes'
  for (long b = (long)blockIdx.x * per; b < c.P; b += 2 * step) {
    const long pu[2] = {b + threadIdx.x / L, b + step + threadIdx.x / L};
    const long p = l & 1 ? pu[1] : pu[0];
    double th[2][2 * E2], iv = 0.0, f = 0.0, sc = 0.0;
    int ms[2];
    if (l < 2 && p < c.P) {
      iv = c.invar[p];
      f = c.freq[p];
      if (SRC == kMem && (flags & kLnl)) sc = c.scale_all[p];
    }
    if constexpr (small_form<SRC, E2>())
      if (ops.n) small_traverse<SRC, SAFE>(c, ops, small, L, l, pu);
    load_theta<SRC, SAFE, E2>(c, br, L, l, pu, th, ms);
    if (flags & kStore) {
#pragma unroll
      for (int u = 0; u < 2; u++)
        if (pu[u] < c.P) {
          store_theta<E2>(c, L, l, pu[u], th[u]);
          if (l == 0) c.scale_all[pu[u]] = (double)ms[u] * thr;
        }
      if (flags == kStore) continue;
    }
    const double lh = lanes_sum2(dot<E2>(th[0], tab, L, l), dot<E2>(th[1], tab, L, l), L, l);
    double d1 = 0.0, d2 = 0.0;
    if (flags & kDerv) {
      const double *t1 = tab + len, *t2 = t1 + len;
      d1 = lanes_sum2(dot<E2>(th[0], t1, L, l), dot<E2>(th[1], t1, L, l), L, l);
      d2 = lanes_sum2(dot<E2>(th[0], t2, L, l), dot<E2>(th[1], t2, L, l), L, l);
    }
    if (l >= 2 || p >= c.P) continue;
    const double like = fabs(lh) + iv;
    if (flags & kDerv) {
      if (p >= c.nptn) continue;
      const double inv = 1.0 / like;
      const double dff = d1 * inv, ddff = d2 * inv;
      const double t1 = dff * f, t2 = ddff * f;
      v0 += t1;
      v1 += fma(-t1, dff, t2);
      c.df_frac[p] = dff;
      c.ddf_term[p] = fma(-dff, dff, ddff);
    } else {
      const double plh = log(like) + (SRC == kMem ? sc : (l ? ms[1] : ms[0]) * thr);
      c.pattern_lh[p] = plh;
      if (p < c.nptn) {
        v0 += plh * f;
        v1 += (isfinite(plh) ? plh : 4.0 * kLogScaleThr) * f;
      }
    }
  }
  block_pair<kThreadsT / 32>(v0, v1, sh);
  if (threadIdx.x == 0) {
    __stcg(c.red + 2 * blockIdx.x, v0);
    __stcg(c.red + 2 * blockIdx.x + 1, v1);
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  v0 = v1 = 0.0;
  for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
    v0 += __ldcg(c.red + 2 * b);
    v1 += __ldcg(c.red + 2 * b + 1);
  }
  __syncthreads();
  block_pair<kThreadsT / 32>(v0, v1, sh);
  if (threadIdx.x == 0) {
    out[0] = v0;
    out[1] = v1;
    *ticket = 0;  // ready for the next launch
  }
}

// ----------------------------------------------------------------------------------------
// Device-side Newton (Optimization::minimizeNewton) as one launch.  Each evaluation is a sum of
// (df, ddf) over all patterns; every thread then runs the same scalar update on the same sums, so
// all follow one iterate sequence.  A thread keeps its first patterns' theta in registers over
// all evaluations, the others are read again each time.
//
// An evaluation is a chain of latencies (exponentials, dot products, sums over lanes, warps and
// blocks, one division), so the exchange between blocks is what its design is about:
// - Within a cluster, every warp sends its sums to each block's shared memory (st.async, counted
//   by that block's mbarrier), and every warp adds all of them in one order: no barrier of the
//   block, no leader, no broadcast.  Up to 16 blocks (8,192 patterns of 4 states and 4
//   categories) need nothing else.
// - Beyond that, each cluster of 8 publishes its sums in global memory, each with a tag (launch
//   number, evaluation) in one 16-byte store, and the first warp of every block polls all
//   clusters' slots until they carry the tag: one trip through L2.  Tags of earlier launches
//   never match, so nothing is cleared.  Two sets of slots (and of shared-memory buffers) in
//   turn: a set is written again only by who has seen everyone's next sums, which each sends
//   after reading this set.
// Every wait is bounded; who gives up sends nothing more, so the others give up too, and all
// reach the cluster barrier at the end.
// Measured, a loop of five evaluations (theta of 4,703 / 18,501 patterns of 4 states, 9,707 of 20,
// 4 categories): 31.1 / 37.2 / 47.8 us with a counting barrier over 74 / 290 / 152 blocks and a
// theta launch of 4.8 / 4.5 / 9.6 us before it; 28.9 / 39.7 / 46.3 us, theta included, with an
// all-to-all exchange of every block's sums through L2 (4,000 to 7,200 cycles of an evaluation);
// 25.6 / 27.0 / 32.1 us, theta included, as here.
// ----------------------------------------------------------------------------------------
constexpr int kPollLimit = 1 << 20;  // each poll is an L2 round trip or two: a second or so
constexpr int kMaxClusters = 32;
constexpr int kMaxCluster = 16;

__device__ __forceinline__ void publish(ulonglong2 *slot, double v, unsigned long long tag) {
  asm volatile(
      "{\n\t.reg .b128 r;\n\tmov.b128 r, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], r;\n\t}\n" ::"l"(
          slot),
      "l"(__double_as_longlong(v)), "l"(tag)
      : "memory");
}
__device__ __forceinline__ bool peek(const ulonglong2 *slot, unsigned long long tag, double &v) {
  unsigned long long a, b;
  asm volatile(
      "{\n\t.reg .b128 r;\n\tld.relaxed.gpu.global.b128 r, [%2];\n\tmov.b128 {%0, %1}, r;\n\t}\n"
      : "=l"(a), "=l"(b)
      : "l"(slot)
      : "memory");
  v = __longlong_as_double(a);
  return b == tag;
}

// Sums of n <= 32 published pairs (slot pairs 128 bytes apart), by one warp: the same bits in
// every lane of every caller; false when they have not all come in time.
constexpr int kSlotStride = 8;  // ulonglong2 per pair
__device__ __forceinline__ bool gather(const ulonglong2 *slots, int n, unsigned long long tag,
                                       double &a, double &b) {
  const int lane = threadIdx.x & 31;
  bool ok = false;
  for (int k = 0; k < kPollLimit && !ok; k++) {
    a = b = 0.0;
    bool mine = true;
    if (lane < n) {
      const bool u = peek(slots + kSlotStride * lane, tag, a);
      const bool v = peek(slots + kSlotStride * lane + 1, tag, b);
      mine = u && v;
    }
    ok = __all_sync(0xffffffffu, mine);
  }
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  return ok;
}

// address of this CTA's shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void send_pair(uint32_t dst, uint32_t bar, double a, double b) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
      "l"(__double_as_longlong(a)), "l"(__double_as_longlong(b)), "r"(bar)
      : "memory");
}
// Bounded wait for what the blocks of the cluster sent, false when it has not all come in time.
// The senders are other blocks: the acquire is at cluster scope (tc::mbar_wait's, for copies and
// MMAs of the block itself, is at the block's).
__device__ __forceinline__ bool cluster_wait(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > tc::kWaitCycles) return false;
  }
}

struct NewtonArgs {
  gems_branch br;
  double guess, x1, x2, xacc;
  int maxstep, L, cluster;   // blocks per cluster
  ulonglong2 *slots;         // two sets of kMaxClusters pairs
  unsigned long long tag0;   // launch number, shifted
  double *result;            // pinned host memory: length, evaluations, status
};

// threads of a block that takes an SM's registers: more than five pairs per lane need more than
// 128 each
__host__ __device__ constexpr int newton_threads(int e2) { return e2 <= 5 ? 512 : 256; }
template <int E2>
__host__ __device__ constexpr int held_rows() {
  return E2 <= 2 ? 4 : 2;  // an even number
}
// the same of blocks that hold no rows, and how many of them an SM takes
__host__ __device__ constexpr int stream_threads(int e2) { return e2 <= 5 ? 256 : 128; }
__host__ __device__ constexpr int stream_ctas(int e2) {
  return e2 <= 2 || e2 == 8 || e2 == 12 ? 4 : 3;
}

// HELD: the first rows of each thread in registers, one block to an SM; else none (launched for
// small shares of the GPU)
template <int SRC, bool SAFE, int E2, bool HELD>
__global__ void __launch_bounds__(HELD ? newton_threads(E2) : stream_threads(E2),
                                  HELD ? 1 : stream_ctas(E2))
    k_newton(DevCtx c, const NewtonArgs a, const __grid_constant__ SmallOps ops) {
  extern __shared__ __align__(16) double tab[];
  constexpr int nt = HELD ? newton_threads(E2) : stream_threads(E2), nw = nt / 32;
  __shared__ __align__(16) double2 recv[2][kMaxCluster * nw];
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ double tot[2];
  __shared__ bool tot_ok;
  constexpr int RH = HELD ? held_rows<E2>() : 0, RA = RH ? RH : 2;
  constexpr double thr = SRC == kM4 ? kLogScaleThrF : kLogScaleThr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int CS = a.cluster, nclusters = gridDim.x / CS, rank = blockIdx.x % CS;
  const int L = a.L, len = 2 * L * E2, l = threadIdx.x & (L - 1);
  const long per = nt / L, step = per * gridDim.x;
  const long b0 = (long)blockIdx.x * per;
  const int sub = threadIdx.x / L;
  // (this block's receive address is kept, not made in each evaluation: mixed, 4 states, 8 categories,
  // 250,000 patterns 87.4 us a loop of one evaluation instead of 94.5)
  const uint32_t s_recv = tc::sptr(&recv[0][0]), s_bars = tc::sptr(&bars[0]);
  const uint32_t expect = CS * nw * sizeof(double2);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; i++) {
      tc::mbar_init(s_bars + 8 * i, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int i = 0; i < 2; i++) tc::mbar_expect_tx(s_bars + 8 * i, expect);
  }
  // the others' barriers are ready once all blocks have been here (waited for below)
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");

  const double *small = tab + 3 * len;
  if constexpr (small_form<SRC, E2>())
    if (ops.n) {
      small_tables<SRC>(c, ops, tab + 3 * len);
      __syncthreads();
    }
  auto updates = [&](const long (&p)[2]) {
    if constexpr (small_form<SRC, E2>())
      if (ops.n) small_traverse<SRC, SAFE>(c, ops, small, L, l, p);
  };

  // theta of this thread's rows: formed and stored (or read), the first ones kept; of each two
  // patterns, even lanes hold the first's +I term and weight and odd lanes the second's
  double th[RA][2 * E2], inva[RA / 2], fr[RA / 2];
  auto weights = [&](long p, double &iv, double &f) {
    iv = f = 0.0;
    if (l < 2 && p < c.nptn) iv = c.invar[p], f = c.freq[p];
  };
  auto keep = [&](const long (&p)[2], const double (&v)[2][2 * E2], const int (&m)[2]) {
    if constexpr (SRC != kMem) {
#pragma unroll
      for (int u = 0; u < 2; u++)
        if (p[u] < c.P) {
          store_theta<E2>(c, L, l, p[u], v[u]);
          if (l == 0) c.scale_all[p[u]] = (double)m[u] * thr;
        }
    }
  };
#pragma unroll
  for (int r = 0; r < RH; r += 2) {
    const long p[2] = {b0 + r * step + sub, b0 + (r + 1) * step + sub};
    inva[r / 2] = fr[r / 2] = 0.0;
#pragma unroll
    for (int e = 0; e < 2 * E2; e++) th[r][e] = th[r + 1][e] = 0.0;
    if (b0 + r * step >= c.P) continue;
    double v[2][2 * E2];
    int m[2];
    weights(l & 1 ? p[1] : p[0], inva[r / 2], fr[r / 2]);
    updates(p);
    load_theta<SRC, SAFE, E2>(c, a.br, L, l, p, v, m);
    keep(p, v, m);
#pragma unroll
    for (int e = 0; e < 2 * E2; e++) th[r][e] = v[0][e], th[r + 1][e] = v[1][e];
  }
  if (SRC != kMem)
    for (long b = b0 + RH * step; b < c.P; b += 2 * step) {
      const long p[2] = {b + sub, b + step + sub};
      double v[2][2 * E2];
      int m[2];
      updates(p);
      load_theta<SRC, SAFE, E2>(c, a.br, L, l, p, v, m);
      keep(p, v, m);
    }

  // this thread's table elements: eval_i r_c and prop_c (HELD: at most 2 x 32 x E2 of them, else
  // behind the tables)
  constexpr int kTab = HELD ? (64 * E2 + nt - 1) / nt : 1;
  double cof[kTab], prop[kTab];
  double2 *fac = reinterpret_cast<double2 *>(tab + 3 * len);
  if constexpr (HELD) {
#pragma unroll
    for (int i = 0; i < kTab; i++) table_factors(c, threadIdx.x + i * nt, cof[i], prop[i]);
  } else {
    for (int j = threadIdx.x; j < len; j += nt) table_factors(c, j, fac[j].x, fac[j].y);
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");

  int nevals = 0;
  // f = -dlnL/dt and df = -d2lnL/dt2 at t (computeFuncDerv, phylotree.cpp:2555).  Tables of the
  // last evaluation may be overwritten: its sums have come, so every warp had read them.
  auto eval = [&](double t, double &f, double &df) -> bool {
    if constexpr (HELD) {
#pragma unroll
      for (int i = 0; i < kTab; i++)
        if (threadIdx.x + i * nt < len)
          put_tables(t, threadIdx.x + i * nt, cof[i], prop[i], len, 3, tab);
    } else {
      for (int j = threadIdx.x; j < len; j += nt) put_tables(t, j, fac[j].x, fac[j].y, len, 3, tab);
    }
    __syncthreads();
    double v0 = 0.0, v1 = 0.0;
    // two patterns' terms, b and b + step from this block's start
    auto add = [&](const double (&x)[2 * E2], const double (&y)[2 * E2], long b, double iv,
                   double w) {
      const double *t1 = tab + len, *t2 = t1 + len;
      double h, d, g;
      if constexpr (HELD) {
        h = lanes_sum2(dot<E2>(x, tab, L, l), dot<E2>(y, tab, L, l), L, l);
        d = lanes_sum2(dot<E2>(x, t1, L, l), dot<E2>(y, t1, L, l), L, l);
        g = lanes_sum2(dot<E2>(x, t2, L, l), dot<E2>(y, t2, L, l), L, l);
      } else {
        double p, q;
        dot2<E2>(x, y, tab, L, l, p, q), h = lanes_sum2(p, q, L, l);
        dot2<E2>(x, y, t1, L, l, p, q), d = lanes_sum2(p, q, L, l);
        dot2<E2>(x, y, t2, L, l, p, q), g = lanes_sum2(p, q, L, l);
      }
      if (l < 2 && b + l * step + sub < c.nptn) {
        const double inv = 1.0 / (fabs(h) + iv);
        const double dff = d * inv, q = dff * w;
        v0 += q;
        v1 += fma(-q, dff, g * inv * w);
      }
    };
#pragma unroll
    for (int r = 0; r < RH; r += 2)
      if (b0 + r * step < c.P) add(th[r], th[r + 1], b0 + r * step, inva[r / 2], fr[r / 2]);
    for (long b = b0 + RH * step; b < c.P; b += 2 * step) {
      const long p[2] = {b + sub, b + step + sub};
      double v[2][2 * E2], iv, w;
      int m[2];
      weights(l & 1 ? p[1] : p[0], iv, w);
      load_theta<kMem, SAFE, E2>(c, a.br, L, l, p, v, m);
      add(v[0], v[1], b, iv, w);
    }
    for (int o = 16; o > 0; o >>= 1) {
      v0 += __shfl_xor_sync(0xffffffffu, v0, o);
      v1 += __shfl_xor_sync(0xffffffffu, v1, o);
    }
    const int set = nevals & 1, use = (nevals >> 1) & 1;  // buffers; how often they were used, mod 2
    nevals++;
    const uint32_t bar = s_bars + 8 * set;
    if (lane < CS)
      send_pair(cluster_addr(s_recv + (set * kMaxCluster * nw + rank * nw + warp) * 16, lane),
                cluster_addr(bar, lane), v0, v1);
    bool ok = cluster_wait(bar, use);
    v0 = v1 = 0.0;
    if (ok)
      for (int i = lane; i < CS * nw; i += 32) {
        const double2 v = recv[set][i];
        v0 += v.x;
        v1 += v.y;
      }
    // armed again for the evaluation after next, whose sums are sent after this one's were read
    if (threadIdx.x == 0 && ok) tc::mbar_expect_tx(bar, expect);
    for (int o = 16; o > 0; o >>= 1) {
      v0 += __shfl_xor_sync(0xffffffffu, v0, o);
      v1 += __shfl_xor_sync(0xffffffffu, v1, o);
    }
    ok = __all_sync(0xffffffffu, ok);
    if (nclusters > 1) {
      if (warp == 0) {
        ulonglong2 *slots = a.slots + set * kMaxClusters * kSlotStride;
        const unsigned long long tag = a.tag0 + (unsigned)nevals;
        if (ok && rank == 0 && lane < 2)
          publish(slots + kSlotStride * (blockIdx.x / CS) + lane, lane ? v1 : v0, tag);
        ok = gather(slots, nclusters, tag, v0, v1) && ok;
        if (lane == 0) tot[0] = v0, tot[1] = v1, tot_ok = ok;
      }
      __syncthreads();
      v0 = tot[0];
      v1 = tot[1];
      ok = tot_ok;
    } else {
      ok = __syncthreads_and(ok);
    }
    if (!ok) return false;
    if (!isfinite(v0)) v0 = v1 = 0.0;
    f = -v0;
    df = -v1;
    return true;
  };

  const double x1 = a.x1, x2 = a.x2, xacc = a.xacc;
  double f, df, dx, temp, xh, xl, rts, rts_old;
  double ret = 0.0;
  int status = GEMS_OK;
  rts = a.guess;
  if (rts < x1) rts = x1;
  if (rts > x2) rts = x2;
  do {
    if (!eval(rts, f, df)) { status = GEMS_ERR_TIMEOUT; ret = rts; break; }
    if (!isfinite(f) || !isfinite(df)) { status = GEMS_ERR_NUMERIC_UNDERFLOW; ret = rts; break; }
    if (df >= 0.0 && fabs(f) < xacc) { ret = rts; break; }
    if (f < 0.0) { xl = rts; xh = x2; } else { xh = rts; xl = x1; }
    dx = fabs(xh - xl);
    bool done = false;
    for (int j = 1; j <= a.maxstep && !done; j++) {
      rts_old = rts;
      const double newton = f / df;  // beside the bracket test, not after it
      if ((df <= 0.0) || (((rts - xh) * df - f) * ((rts - xl) * df - f) >= 0.0)) {
        dx = 0.5 * (xh - xl);
        rts = xl + dx;
        if (xl == rts) { ret = rts; done = true; break; }
      } else {
        dx = newton;
        temp = rts;
        rts -= dx;
        if (temp == rts) { ret = rts; done = true; break; }
      }
      if (fabs(dx) < xacc || (j == a.maxstep)) { ret = rts_old; done = true; break; }
      if (!eval(rts, f, df)) { status = GEMS_ERR_TIMEOUT; ret = rts; done = true; break; }
      if (!isfinite(f) || !isfinite(df)) {
        status = GEMS_ERR_NUMERIC_UNDERFLOW; ret = rts; done = true; break;
      }
      if (df > 0.0 && fabs(f) < xacc) { ret = rts; done = true; break; }
      if (f < 0.0) xl = rts;
      else if (f > 0.0) xh = rts;
    }
    if (!done) ret = 0.0;
  } while (false);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.result[0] = ret;
    a.result[1] = (double)nevals;
    a.result[2] = (double)status;
  }
  // no block leaves while another may still send to its shared memory
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---- kernel tables -------------------------------------------------------------------------
template <int SRC, bool SAFE, int E2>
BranchFns branch_fns() {
  return {(const void *)k_terms<SRC, SAFE, E2>, (const void *)k_newton<SRC, SAFE, E2, true>, nullptr};
}
template <int E2>
BranchFns memory_fns() {
  BranchFns f = branch_fns<kMem, false, E2>();
  f.stream = (const void *)k_newton<kMem, false, E2, false>;
  return f;
}

}  // namespace

// The tables, by the pairs per lane that split_of gives: 4 states one or two, 20 states three to
// five, 61 states three and more (wide: eight and more).
BranchFns branch_f64_4(bool safe, int e2);
BranchFns branch_mixed_4(bool safe, int e2);
BranchFns branch_f64_20(bool safe, int e2);
BranchFns branch_f64_61(bool safe, int e2);
BranchFns branch_f64_61_wide(bool safe, int e2);
BranchFns branch_memory_4(int e2);
BranchFns branch_memory_20(int e2);
BranchFns branch_memory_wide(int e2);

}  // namespace gems
