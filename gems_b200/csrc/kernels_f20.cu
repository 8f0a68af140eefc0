// kernels_f20.cu -- FP64 20-state traversal on the FP64 tensor instructions (mma.sync m8n8k4).
//
// Node update per category c (eigen space, the reference's form, phylokernelnew.h:1911-2035):
//      out = inv_evec . ((evec . (d_L (*) L)) (*) (evec . (d_R (*) R))),  d[i] = exp(eval_i r_c t)
// A warp owns 8 patterns and all their categories for the whole op list.  Each product is
// D[8 patterns x 20] = A[8 x 20] . B^T with B = evec or inv_evec, which depend on neither the
// category nor the op: both matrices are laid out as B fragments in shared memory once per CTA
// (7.5 KB), and one read of a fragment serves the categories of a pass.
//
// Fragments chain without a shuffle.  Lane (g, t) = (lane / 4, lane % 4) of an m8n8k4 holds
// A[g][k = t], B[k = t][n = g] and C[g][2t], C[g][2t + 1].  With the K and N orders below, the C
// fragment of one product is the A fragment of the next:
//      K step s = 2m + e (m, e in {0, 1}): k = t is state 8m + 2t + e;    step 4: state 16 + t
//      N tile m < 2: column n is state 8m + n;   tile 2: even n is state 16 + n / 2, odd n unused
// so lane (g, t) always holds the five states {2t, 2t + 1, 8 + 2t, 9 + 2t, 16 + t} of pattern g:
// no K padding, and 20 of 24 columns used.  The same lane stores and re-reads those elements, so
// a child written by an earlier op needs no synchronisation, and a warp's accesses of a row fill
// whole 32-byte sectors.  The product of the next op's child that this op wrote starts from
// registers (the plan's forward bit).
//
// Bound by FP64 throughput (mma and FMA have the same rate on sm_100a, 64 FMA per clock and SM
// measured): 30 mma per category and pattern group of an op with one internal child, 2.65 ms of
// them for 126 ops over 98,762 patterns with 4 categories.  That evaluation takes 3.97 ms (the
// FP64 pipe 71% active); it took 8.66 ms with one thread per (pattern, category) and the matrices
// as constant operands.  Measured splits of the work: both matrices in registers, 8 warps per SM
// 4.59 ms; in shared memory, four categories a pass at 2 / 3 CTAs per SM 5.46 / 4.24 ms, two a
// pass at 3 / 4 CTAs 4.49 / 3.97 ms, one a pass at 4 CTAs 4.34 ms.
#include <string>

#include "gems_internal.cuh"

namespace gems {

namespace {

constexpr int kN = 20;
constexpr int kWarpsF = 4;           // warps per CTA
constexpr int kPatF = 8;             // patterns per warp
constexpr int kPassF = 2;            // categories per pass
constexpr int kCtasF = 4;            // resident CTAs per SM (128 registers)
constexpr int kThrHi = 0x2FF00000;   // high word of 2^-256

// the state of K step s at lane position t
__device__ __forceinline__ int state_of(int s, int t) {
  return s < 4 ? 8 * (s >> 1) + 2 * t + (s & 1) : 16 + t;
}

// v <- M . v for CH categories of the warp's 8 patterns; b: this lane's fragments of M, 32 lanes
// apart in shared memory
template <int CH>
__device__ __forceinline__ void apply(const double *b, double (&v)[CH][5]) {
  __syncwarp();
  double acc[CH][3][2];
#pragma unroll
  for (int c = 0; c < CH; c++)
#pragma unroll
    for (int m = 0; m < 3; m++) acc[c][m][0] = acc[c][m][1] = 0.0;
#pragma unroll
  for (int s = 0; s < 5; s++) {
    double f[3];
#pragma unroll
    for (int m = 0; m < 3; m++) f[m] = b[(s * 3 + m) * 32];
#pragma unroll
    for (int c = 0; c < CH; c++)
#pragma unroll
      for (int m = 0; m < 3; m++) dmma(acc[c][m], v[c][s], f[m]);
  }
#pragma unroll
  for (int c = 0; c < CH; c++) {
#pragma unroll
    for (int s = 0; s < 4; s++) v[c][s] = acc[c][s >> 1][s & 1];
    v[c][4] = acc[c][2][0];
  }
}

// this lane's elements of the rows of categories c0.. of one pattern
template <int CH>
__device__ __forceinline__ void load_rows(const double *row, int t, int nc,
                                          double (&v)[CH][5]) {
#pragma unroll
  for (int c = 0; c < CH; c++) {
    if (c >= nc) continue;
    const double2 a = __ldcg(reinterpret_cast<const double2 *>(row + c * kN + 2 * t));
    const double2 b = __ldcg(reinterpret_cast<const double2 *>(row + c * kN + 8 + 2 * t));
    v[c][0] = a.x, v[c][1] = a.y, v[c][2] = b.x, v[c][3] = b.y;
    v[c][4] = __ldcg(row + c * kN + 16 + t);
  }
}
template <int CH>
__device__ __forceinline__ void store_rows(double *row, int t, int nc,
                                           const double (&v)[CH][5]) {
#pragma unroll
  for (int c = 0; c < CH; c++) {
    if (c >= nc) continue;
    *reinterpret_cast<double2 *>(row + c * kN + 2 * t) = make_double2(v[c][0], v[c][1]);
    *reinterpret_cast<double2 *>(row + c * kN + 8 + 2 * t) = make_double2(v[c][2], v[c][3]);
    row[c * kN + 16 + t] = v[c][4];
  }
}
// Table rows (exp factors, tip messages) are stored in lane order, [5][C / w][4 lanes][w] with
// w = 2 for an even C and 1 for an odd one: the four lanes of a pattern read 32 w contiguous
// bytes of the row of its state.
__host__ __device__ constexpr int table_width(int C) { return C % 2 == 0 ? 2 : 1; }

// this lane's five states of a table row, categories c0 .. c0 + nc (even c0 for an even C)
template <int CH>
__device__ __forceinline__ void load_table(const double *__restrict__ tab, int C, int c0, int t,
                                           int nc, double (&v)[CH][5]) {
  if (CH % 2 == 0 && table_width(C) == 2) {
#pragma unroll
    for (int s = 0; s < 5; s++)
#pragma unroll
      for (int c = 0; c + 1 < CH; c += 2)
        if (c < nc) {
          const double2 a =
              __ldg(reinterpret_cast<const double2 *>(tab) + (s * (C / 2) + (c0 + c) / 2) * 4 + t);
          v[c][s] = a.x, v[c + 1][s] = a.y;
        }
  } else {
    const int w = table_width(C);
#pragma unroll
    for (int s = 0; s < 5; s++)
#pragma unroll
      for (int c = 0; c < CH; c++)
        if (c < nc) v[c][s] = __ldg(tab + (s * (C / w) + (c0 + c) / w) * 4 * w + t * w + (c0 + c) % w);
  }
}

// |x| as its high word, NaN as 0 (a maximum over them ignores NaN, as fmax does; 2^-256 is a
// power of two, so the high words decide the comparison with it)
__device__ __forceinline__ int abs_hi(double x) {
  const int h = __double2hiint(x) & 0x7fffffff;
  return h > 0x7ff00000 ? 0 : h;
}

// Warps of a CTA, and CTAs on an SM, when W warps share a group of patterns
__host__ __device__ constexpr int warps_f(int w) { return w == 3 ? 3 : kWarpsF; }
__host__ __device__ constexpr int ctas_f(int w) { return w == 3 ? 5 : kCtasF; }

// KC categories held in registers, CB of them per pass.  W warps share 8 patterns: 1: C == KC;
// more: C > KC, `share` categories to each (the pattern's maximum, NORM, is exchanged in shared
// memory); 0: C > KC and one warp for all, KC at a time (nothing forwarded: they share the
// registers).
template <bool SAFE, int KC, int W>
__global__ void __launch_bounds__(32 * warps_f(W), ctas_f(W))
    k_traverse_f20(DevCtx c, const DevOp *__restrict__ ops, int nops,
                   const double *__restrict__ tab, size_t stride, int p0, int p1, int share) {
  constexpr bool MULTI = W == 0;
  constexpr int kGroups = W > 1 ? warps_f(W) / W : kWarpsF;
  constexpr int CB = KC < kPassF ? KC : kPassF;
  __shared__ double frag[2][15][32];  // evec, inv_evec as B fragments
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  __shared__ int group_max[W > 1 ? kGroups : 1][W > 1 ? W : 1][kPatF];
  const int warp = threadIdx.x >> 5, group = W > 1 ? warp / W : warp;
  const long p = p0 + ((long)blockIdx.x * kGroups + group) * kPatF + g;
  const bool act = p < p1;
  const int C = W == 1 ? KC : c.C, blk = C * kN;
  const int first_c = W > 1 ? warp % W * share : 0;             // this warp's categories
  const int mine = W > 1 ? min(share, C - first_c) : KC;
  for (int i = threadIdx.x; i < 2 * 15 * 32; i += 32 * warps_f(W)) {
    const int l = i & 31, sm = (i >> 5) % 15, s = sm / 3, m = sm % 3, n = l >> 2;
    // column n of tile m
    const int x = m < 2 ? 8 * m + n : 16 + (n >> 1);
    const double *src = i < 15 * 32 ? c.evec : c.inv_evec;
    (&frag[0][0][0])[i] = m < 2 || !(n & 1) ? src[x * kN + state_of(s, l & 3)] : 0.0;
  }
  __syncthreads();
  const double *be = &frag[0][0][lane], *bi = &frag[1][0][lane];
  const bool inv0 = act && c.invar[p] == 0.0;
  double *part = static_cast<double *>(c.partials);

  double x[KC][5];          // the op's first child, then its output
  int sx[SAFE ? KC : 1];    // its counters
#pragma unroll
  for (int j = 0; j < KC; j++)
#pragma unroll
    for (int s = 0; s < 5; s++) x[j][s] = 0.0;
#pragma unroll
  for (int j = 0; j < (SAFE ? KC : 1); j++) sx[j] = 0;

  DevOp op = ops[0];
  // tip bytes of an op, fetched while the op before it computes
  auto tip_byte = [&](int kind, int id) {
    return kind == GEMS_CHILD_TIP && act ? (int)c.tips[(size_t)id * c.P + p] : 0;
  };
  int tl = tip_byte(op.l_kind, op.l_id), tr = tip_byte(op.r_kind, op.r_id);
  for (int k = 0; k < nops; k++) {
    const DevOp nxt = ops[k + 1 < nops ? k + 1 : k];
    const double *tk = tab + (size_t)k * stride;
    const bool tiptip = op.l_kind == GEMS_CHILD_TIP && op.r_kind == GEMS_CHILD_TIP;
    // the forwarded child comes first: it is in registers while the other one loads
    const bool fwd_r = !MULTI && op.r_kind == GEMS_CHILD_PARTIAL && plan_rsrc(op.pad_) == kSrcFwd;
    const bool fwd = fwd_r || (!MULTI && op.l_kind == GEMS_CHILD_PARTIAL &&
                               plan_lsrc(op.pad_) == kSrcFwd);
    const int first = fwd_r ? 1 : 0;
    const int kind[2] = {first ? op.r_kind : op.l_kind, first ? op.l_kind : op.r_kind};
    const int id[2] = {first ? op.r_id : op.l_id, first ? op.l_id : op.r_id};
    const int tip[2] = {first ? tr : tl, first ? tl : tr};
    int s_norm = 0, hmax = 0;  // NORM: counters; largest |out| of the pattern, as a high word
    if (!SAFE && act) {
      if (fwd) s_norm = sx[0];
#pragma unroll
      for (int i = 0; i < 2; i++)
        if (kind[i] == GEMS_CHILD_PARTIAL && !(i == 0 && fwd))
          s_norm += c.scale[(size_t)id[i] * c.slot_scale + p];
    }
    double *dst = part + (size_t)op.dst_slot * c.slot_elems + (size_t)p * blk;
    for (int c0 = first_c; c0 < (MULTI ? C : first_c + 1); c0 += KC) {
#pragma unroll
      for (int cb = 0; cb < KC; cb += CB) {
        // categories c0 + cb .. + nc of this pass (CB of them unless the last of an odd KC or C)
        const int cc = c0 + cb;
        const int nc = MULTI   ? min(CB, C - cc)
                       : W > 1 ? min(CB, mine - cb)
                               : (KC - cb < CB ? KC - cb : CB);
        if (W != 1 && nc <= 0) break;
        double v[2][CB][5];
        int sc[CB];
#pragma unroll
        for (int j = 0; j < CB; j++) sc[j] = 0;
        // raw elements (and SAFE counters) of both children
#pragma unroll
        for (int i = 0; i < 2; i++) {
#pragma unroll
          for (int j = 0; j < CB; j++)
#pragma unroll
            for (int q = 0; q < 5; q++) v[i][j][q] = 0.0;
          if (i == 0 && fwd) {
#pragma unroll
            for (int j = 0; j < CB; j++)
              if (cb + j < KC) {
                if (SAFE) sc[j] = sx[SAFE ? (cb + j) % KC : 0];
#pragma unroll
                for (int q = 0; q < 5; q++) v[0][j][q] = x[(cb + j) % KC][q];
              }
          } else if (act) {
            if (kind[i] == GEMS_CHILD_TIP) {
              const int st = min(tip[i], c.unknown);
              load_table<CB>(tk + 2 * blk + ((size_t)(i ^ first) * (c.unknown + 1) + st) * blk, C,
                             cc, t, nc, v[i]);
            } else {
              load_rows<CB>(part + (size_t)id[i] * c.slot_elems + (size_t)p * blk + cc * kN, t, nc,
                            v[i]);
              if (SAFE) {
                const uint16_t *q = c.scale + (size_t)id[i] * c.slot_scale + (size_t)p * C + cc;
#pragma unroll
                for (int j = 0; j < CB; j++)
                  if (j < nc) sc[j] += q[j];
              }
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
          if (kind[i] != GEMS_CHILD_PARTIAL) continue;
          double d[CB][5];
#pragma unroll
          for (int j = 0; j < CB; j++)
#pragma unroll
            for (int q = 0; q < 5; q++) d[j][q] = 0.0;
          load_table<CB>(tk + (i ^ first) * blk, C, cc, t, nc, d);
#pragma unroll
          for (int j = 0; j < CB; j++)
#pragma unroll
            for (int q = 0; q < 5; q++) v[i][j][q] *= d[j][q];
          apply<CB>(be, v[i]);
        }
#pragma unroll
        for (int j = 0; j < CB; j++)
#pragma unroll
          for (int q = 0; q < 5; q++) v[0][j][q] *= v[1][j][q];
        apply<CB>(bi, v[0]);
#pragma unroll
        for (int j = 0; j < CB; j++) {
          if (cb + j >= KC) continue;
          constexpr int kk = KC;
          double(&o)[5] = x[(cb + j) % kk];
          int h = 0;
#pragma unroll
          for (int q = 0; q < 5; q++) {
            o[q] = v[0][j][q];
            h = max(h, abs_hi(o[q]));
          }
          if (SAFE) {
            h = max(h, __shfl_xor_sync(0xffffffffu, h, 1));
            h = max(h, __shfl_xor_sync(0xffffffffu, h, 2));
            const bool up = !tiptip && h < kThrHi && inv0;
            if (up) {
#pragma unroll
              for (int q = 0; q < 5; q++) o[q] *= 0x1p256;
            }
            sx[SAFE ? (cb + j) % kk : 0] = sc[j] + (up ? 1 : 0);
          } else {
            hmax = max(hmax, h);
          }
        }
      }
      if (!SAFE && !MULTI) {
        hmax = max(hmax, __shfl_xor_sync(0xffffffffu, hmax, 1));
        hmax = max(hmax, __shfl_xor_sync(0xffffffffu, hmax, 2));
        if constexpr (W > 1) {
          if (t == 0) group_max[group][warp % W][g] = hmax;
          __syncthreads();
#pragma unroll
          for (int i = 0; i < W; i++) hmax = max(hmax, group_max[group][i][g]);
        }
        sx[0] = s_norm;
        if (!tiptip && hmax < kThrHi && inv0) {
#pragma unroll
          for (int j = 0; j < KC; j++)
#pragma unroll
            for (int q = 0; q < 5; q++) x[j][q] *= 0x1p256;
          sx[0] += 1;
        }
        s_norm = sx[0];
      }
      if (act) {
        const int nc = MULTI ? min(KC, C - c0) : mine;
        store_rows<KC>(dst + c0 * kN, t, nc, x);
        if (SAFE && t == 0) {
          uint16_t *q = c.scale + (size_t)op.dst_slot * c.slot_scale + (size_t)p * C + c0;
#pragma unroll
          for (int j = 0; j < KC; j++)
            if (j < nc) q[j] = (uint16_t)sx[SAFE ? j : 0];
        }
      }
    }
    if (!SAFE && MULTI) {
      // the pattern's maximum is known after the last pass: rows below the threshold (rare) are
      // scaled where they were stored, each lane its own elements
      hmax = max(hmax, __shfl_xor_sync(0xffffffffu, hmax, 1));
      hmax = max(hmax, __shfl_xor_sync(0xffffffffu, hmax, 2));
      if (!tiptip && hmax < kThrHi && inv0) {
        for (int cc = 0; cc < C; cc++)
#pragma unroll
          for (int q = 0; q < 5; q++) dst[cc * kN + state_of(q, t)] *= 0x1p256;
        s_norm += 1;
      }
    }
    if (!SAFE && act && t == 0 && first_c == 0)
      c.scale[(size_t)op.dst_slot * c.slot_scale + p] = (uint16_t)s_norm;
    // the counters that lane t = 0 wrote are read by its pattern's four lanes, with NORM by those
    // of all the group's warps
    if (!SAFE && W > 1)
      __syncthreads();
    else
      __syncwarp();
    op = nxt;
    tl = tip_byte(op.l_kind, op.l_id);
    tr = tip_byte(op.r_kind, op.r_id);
  }
}

// Op tables, grid (nops, 2 sides, tip-row groups): d[side] (exp factors of an internal child),
// then the tip messages [side][state code] = sum_i evec[x][i] d[i] tip[state][i] of a tip child
// (1 for the unknown state), rows in lane order.
__global__ void k_prep_ops_f20(DevCtx c, const DevOp *ops, double *tab, size_t stride) {
  extern __shared__ double sm[];  // exp factors [C][20], evec (rows of 21: 20 rows in 20 banks)
  const int k = blockIdx.x, side = blockIdx.y, C = c.C, blk = c.block, w = table_width(C);
  const DevOp op = ops[k];
  const bool is_tip = (side ? op.r_kind : op.l_kind) == GEMS_CHILD_TIP;
  if (!is_tip && blockIdx.z > 0) return;
  const double len = side ? op.r_len : op.l_len;
  double *ev = sm + blk;
  for (int i = threadIdx.x; i < blk; i += blockDim.x)
    sm[i] = exp(c.eval[i % kN] * (c.rates[i / kN] * len));
  if (is_tip)
    for (int i = threadIdx.x; i < kN * kN; i += blockDim.x) ev[i / kN * (kN + 1) + i % kN] = c.evec[i];
  __syncthreads();
  // element r of a row in lane order: state and category
  auto place = [&](int r, int &x, int &cc) {
    const int e = r % w, t = (r / w) % 4, q = r / (4 * w);
    cc = q % (C / w) * w + e;
    x = state_of(q / (C / w), t);
  };
  double *tk = tab + (size_t)k * stride;
  int x, cc;
  if (!is_tip) {
    for (int r = threadIdx.x; r < blk; r += blockDim.x) {
      place(r, x, cc);
      tk[side * blk + r] = sm[cc * kN + x];
    }
    return;
  }
  double *leaf = tk + 2 * blk + (size_t)side * (c.unknown + 1) * blk;
  const int per = (c.unknown + gridDim.z) / gridDim.z, s0 = blockIdx.z * per;
  const int s1 = min(s0 + per, c.unknown + 1);
  for (int i = s0 * blk + threadIdx.x; i < s1 * blk; i += blockDim.x) {
    const int s = i / blk;
    place(i - s * blk, x, cc);
    double acc = 0.0;
    if (s == c.unknown) {
      acc = 1.0;
    } else {
      const double *tp = c.tip + (size_t)s * kN;
#pragma unroll
      for (int j = 0; j < kN; j++) acc = fma(ev[x * (kN + 1) + j] * sm[cc * kN + j], __ldg(tp + j), acc);
    }
    leaf[i] = acc;
  }
}

template <bool SAFE>
const void *kernel_f20(int C, int w) {
  switch (w) {
    case 0: return (const void *)k_traverse_f20<SAFE, 4, 0>;
    case 2: return (const void *)k_traverse_f20<SAFE, 4, 2>;
    case 3: return (const void *)k_traverse_f20<SAFE, 4, 3>;
    case 4: return (const void *)k_traverse_f20<SAFE, 4, 4>;
  }
  switch (C) {
    case 1: return (const void *)k_traverse_f20<SAFE, 1, 1>;
    case 2: return (const void *)k_traverse_f20<SAFE, 2, 1>;
    case 3: return (const void *)k_traverse_f20<SAFE, 3, 1>;
    default: return (const void *)k_traverse_f20<SAFE, 4, 1>;
  }
}

// Warps that share a group of 8 patterns of n (W).  One warp for more than four categories is a
// chain several times as long, with every child read back: 24 taxa, 16 categories, 100 patterns
// 312 us (NORM; SAFE 345) against 121 (128) with four warps, 3,000 patterns 327 (362) against 168
// (172); 5 categories, 100 patterns 134 (149) against 107.  Once the groups alone fill the GPU the
// one warp, which reads each fragment of the matrices for more categories, is the faster: 100,000
// patterns of 5 categories 1,012 us against 1,403, of 9 categories 1,674 against 2,042.  So the
// warps share while all of them are resident at once.
int warps_per_group(const Session *s, int n) {
  const int C = s->desc.ncat, w = (C + 3) / 4;
  if (w == 1) return 1;
  const long groups = ((long)n + kPatF - 1) / kPatF;
  return groups * w <= (long)s->nsm * kCtasF * kWarpsF ? w : 0;
}

}  // namespace

const void *traverse_f20_kernel(const Session *s, int n, int *threads, int *patterns) {
  const int w = warps_per_group(s, n);
  *threads = 32 * warps_f(w);
  *patterns = kPatF * (w > 1 ? warps_f(w) / w : kWarpsF);
  return s->desc.scaling == GEMS_SCALE_SAFE ? kernel_f20<true>(s->desc.ncat, w)
                                            : kernel_f20<false>(s->desc.ncat, w);
}

int launch_prep_ops_f20(Session *s, int nops) {
  if (nops <= 0) return GEMS_OK;
  DevCtx c = s->ctx();
  const size_t smem = sizeof(double) * (s->block + kN * (kN + 1));
  k_prep_ops_f20<<<dim3(nops, 2, 4), 256, smem, s->stream>>>(c, s->d_ops, s->d_opmats,
                                                            s->op_stride);
  s->launches++;
  GEMS_CUDA(cudaGetLastError());
  return GEMS_OK;
}

int launch_traverse_f20(Session *s, int nops, int p0, int p1) {
  DevCtx c = s->ctx();
  int threads = 0, per = 0;
  const void *fn = traverse_f20_kernel(s, p1 - p0, &threads, &per);
  const int grid = (p1 - p0 + per - 1) / per;
  const DevOp *ops = s->d_ops;
  const double *tab = s->d_opmats;
  size_t stride = s->op_stride;
  // categories of a warp that shares its patterns: even counts of an even C (load_table)
  const int C = s->desc.ncat, w = (C + 3) / 4;
  int share = C % 2 ? (C + w - 1) / w : 4;
  void *args[] = {&c, &ops, &nops, &tab, &stride, &p0, &p1, &share};
  GEMS_CUDA(cudaLaunchKernel(fn, dim3(grid), dim3(threads), args, 0, s->stream));
  s->launches++;
  return GEMS_OK;
}

}  // namespace gems
