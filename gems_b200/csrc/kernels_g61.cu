// kernels_g61.cu -- FP64 traversal for 61 states (codon models) as register-tiled GEMMs.
//
// The node update of the reference (tree/phylokernelnew.h:1911-2035) per (pattern, category)
// row is
//     out = inv_evec . ((E_L,c . L) * (E_R,c . R)),   E_c = evec . diag(exp(eval r_c t)).
// Over a tile of rows each product is a GEMM: V = L . E_c^T (K = N = 61) for the rows of
// category c, and out = T . inv_evec^T for all rows.  The products and their summation order
// are those of the per-row form (fma over the contraction index in ascending order), so the
// values are the generic kernel's bit for bit.  (The factored form evec . (d (*) L) of the 4- and
// 20-state kernels was tried here: with 61 states the eigen-space sums cancel heavily, and on
// a 160-taxon tree with long branches it moved partials by up to 2.5e-8 of their pattern's
// largest value, measured in plain FP64 numpy as well.)
//
// - k_traverse_g61w (SAFE scaling, the usual one for 61 states): warps of 8 patterns of one
//   category with chained products on the FP64 mma (below).
// - k_traverse_g61 (NORM scaling, whose per-pattern maximum spans the categories): FP64 FMA,
//   one CTA per tile of up to 64 rows = tp patterns x C categories (tp = 64 / C rounded down to
//   a multiple of 8), stored category-major (row = c * tp + pattern), 128 threads as 8 x 16:
//   thread (ty, tx) owns rows ty*8..ty*8+7 -- all of one category -- and columns tx, tx+16,
//   tx+32, tx+48 (32 FP64 accumulators); two CTAs per SM; the A operand of a child (its partial
//   rows) staged k-major in shared memory, inv_evec^T there for the whole traversal, E_c^T read
//   through L1 from the op table ([side][c][k][64 columns]) and prefetched into L1 while the
//   child's rows load; a tip child's V is a row of the op's leaf table, gathered by state.
// The mma sums come out bit-identical to the FMA ones (the tests compare every partial).
// Measured on one 200-taxon codon model (3,780 patterns, +G4), a from-scratch traversal: per-row
// kernel 26.6 ms; FMA tiles of 128 rows 7.0 ms, with the L1 prefetch 5.9 ms, 64-row tiles at two
// CTAs per SM 5.3 ms; mma over rows staged in shared memory between products 4.7 ms; chained in
// registers 2.05 ms.  lnL and eight branch derivatives of that model: 11.6 -> 5.0 ms with the last
// form, its op tables (mma as well, 17 us where one thread per element took 234) included.
#include <string>

#include "gems_internal.cuh"

namespace gems {

namespace {

constexpr int kN = 61;
constexpr int kK = 64;       // padded contraction length (MMA k-steps of 4)
constexpr int kNC = 64;      // padded output columns
constexpr int kRows = 64;    // rows per tile
constexpr int kSaLd = kRows + 2;
constexpr int kMaxCatG = 8;
constexpr int kThreadsG = 2 * kRows;  // 8 rows x 4 columns per thread
constexpr size_t kSmemG = sizeof(double) * ((size_t)kK * kNC + (size_t)kK * kSaLd + kRows);

// patterns per tile: 64 / C rounded down to a multiple of 8, so that the 8 rows of a thread
// (category-major rows) belong to one category
__host__ __device__ constexpr int tile_patterns(int C) { return kRows / C / 8 * 8; }

// per-op table (doubles): Et[2][C][kK][kNC] (Et[side][c][i][x] = E_c[x][i], zero padded), then
// leaf[2][unknown + 1][C][61]
__host__ __device__ constexpr size_t et_doubles(int C) { return (size_t)C * kK * kNC; }

__global__ void k_prep_ops_g61(DevCtx c, const DevOp *ops, double *tab, size_t stride) {
  __shared__ double dsh[kMaxCatG * kN];
  const int k = blockIdx.x, side = blockIdx.y;
  const DevOp op = ops[k];
  const int kind = side ? op.r_kind : op.l_kind;
  const double len = side ? op.r_len : op.l_len;
  const int C = c.C, blk = C * kN;
  for (int idx = threadIdx.x; idx < blk; idx += blockDim.x) {
    const int cc = idx / kN, i = idx - cc * kN;
    dsh[idx] = exp(c.eval[i] * (c.rates[cc] * len));
  }
  __syncthreads();
  double *et = tab + (size_t)k * stride + (size_t)side * et_doubles(C);
  for (int idx = threadIdx.x; idx < (int)et_doubles(C); idx += blockDim.x) {
    const int cc = idx / (kK * kNC), r = idx - cc * (kK * kNC), i = r / kNC, x = r - i * kNC;
    et[idx] = (i < kN && x < kN) ? c.evec[x * kN + i] * dsh[cc * kN + i] : 0.0;
  }
  if (kind != GEMS_CHILD_TIP) return;
  double *leaf = tab + (size_t)k * stride + 2 * et_doubles(C) + (size_t)side * (c.unknown + 1) * blk;
  const int rows = c.unknown * blk;
  for (int idx = threadIdx.x; idx < rows; idx += blockDim.x) {
    const int s = idx / blk, r = idx - s * blk, cc = r / kN, x = r - cc * kN;
    const double *t = c.tip + (size_t)s * kN;
    double acc = 0.0;
    for (int i = 0; i < kN; i++) acc = fma(c.evec[x * kN + i] * dsh[cc * kN + i], t[i], acc);
    leaf[idx] = acc;
  }
  for (int idx = threadIdx.x; idx < blk; idx += blockDim.x) leaf[rows + idx] = 1.0;
}

// acc[j][q] = sum_k sA[k][ty*8 + j] * B[k][tx + 16 q], k ascending; B in global memory (read
// through L1) or shared memory
template <bool GLOBAL_B>
__device__ __forceinline__ void gemm_tile(const double *__restrict__ sA,
                                          const double *__restrict__ B, int ty, int tx,
                                          double (&acc)[8][4]) {
#pragma unroll
  for (int j = 0; j < 8; j++)
#pragma unroll
    for (int q = 0; q < 4; q++) acc[j][q] = 0.0;
#pragma unroll 2
  for (int k = 0; k < kK; k++) {
    double b[4];
#pragma unroll
    for (int q = 0; q < 4; q++) b[q] = GLOBAL_B ? __ldg(B + k * kNC + tx + 16 * q) : B[k * kNC + tx + 16 * q];
    const double2 *a2 = reinterpret_cast<const double2 *>(sA + k * kSaLd + ty * 8);
    double a[8];
#pragma unroll
    for (int h = 0; h < 4; h++) {
      const double2 t = a2[h];
      a[2 * h] = t.x;
      a[2 * h + 1] = t.y;
    }
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[j][q] = fma(a[j], b[q], acc[j][q]);
  }
}

// tile row -> (category, pattern within the tile) and back to the slot's pattern-major rows
struct TileMap {
  int C, tp, nrow;
  long p0, P;
  __device__ int cat(int r) const { return r / tp; }
  __device__ long pattern(int r) const { return p0 + (r - (r / tp) * tp); }
  __device__ bool valid(int r) const { return r < nrow && pattern(r) < P; }
  // offset of the row's first state in the slot
  __device__ size_t off(int r) const { return ((size_t)pattern(r) * C + cat(r)) * kN; }
};

// V of one child for the thread's rows and columns, and their patterns' scale counts.  A partial
// child's GEMM leaves sA in use: the caller synchronises before the next write of sA.
__device__ __forceinline__ void child_v(const DevCtx &c, const TileMap &tm, int kind, int id,
                                        const double *et, const double *leaf, double *sA, int ty,
                                        int tx, double (&v)[8][4], int (&s)[8]) {
  if (kind == GEMS_CHILD_TIP) {
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int r = ty * 8 + j;
      const bool ok = tm.valid(r);
      const int st = ok ? min((int)c.tips[(size_t)id * c.P + tm.pattern(r)], c.unknown) : 0;
      const double *row = leaf + ((size_t)st * tm.C + tm.cat(r)) * kN;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int col = tx + 16 * q;
        v[j][q] = ok && col < kN ? __ldg(row + col) : 0.0;
      }
      s[j] = 0;
    }
    return;
  }
  // the rows of E_c^T this CTA will read, pulled into L1 while the child's rows load (the
  // GEMM's first touch of each row otherwise waits on L2: 7.0 -> 5.9 ms with 128-row tiles)
  {
    const char *e0 = reinterpret_cast<const char *>(et);
    const int lines = (int)(et_doubles(tm.C) * sizeof(double) / 128);
    for (int l = threadIdx.x; l < lines; l += blockDim.x)
      asm volatile("prefetch.global.L1 [%0];" ::"l"(e0 + (size_t)l * 128));
  }
  // sA[k][r] = L[r][k] for k < 61, zero elsewhere.  idx runs over (pattern, category, k) in
  // the slot's order, so consecutive threads read consecutive doubles; every load of a thread
  // is issued before the first store.
  const double *src = static_cast<const double *>(c.partials) + (size_t)id * c.slot_elems;
  constexpr int kPer = kRows * kK / kThreadsG;
  static_assert(kRows * kK % kThreadsG == 0, "whole loads per thread");
  double a[kPer];
#pragma unroll
  for (int u = 0; u < kPer; u++) {
    const int idx = threadIdx.x + u * kThreadsG;
    const int g = idx / kK, k = idx - g * kK;  // g = pattern-major row within the tile
    const int lp = g / tm.C, cc = g - lp * tm.C;
    a[u] = (g < tm.nrow && tm.p0 + lp < tm.P && k < kN)
               ? __ldcg(src + ((size_t)(tm.p0 + lp) * tm.C + cc) * kN + k)
               : 0.0;
  }
#pragma unroll
  for (int u = 0; u < kPer; u++) {
    const int idx = threadIdx.x + u * kThreadsG;
    const int g = idx / kK, k = idx - g * kK;
    const int lp = g / tm.C, cc = g - lp * tm.C;
    if (g < tm.nrow) sA[k * kSaLd + cc * tm.tp + lp] = a[u];
  }
  const uint16_t *sc = c.scale + (size_t)id * c.slot_scale;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const int r = ty * 8 + j;
    s[j] = tm.valid(r) ? sc[tm.pattern(r)] : 0;
  }
  __syncthreads();
  // rows past the tile's (64 % C) have no category: any table will do, their A rows are zero
  const int cat = min(tm.cat(ty * 8), tm.C - 1);
  gemm_tile<true>(sA, et + (size_t)cat * kK * kNC, ty, tx, v);
}

__global__ void __launch_bounds__(kThreadsG, 2)
    k_traverse_g61(DevCtx c, const DevOp *__restrict__ ops, int nops,
                   const double *__restrict__ tab, size_t stride, int tile0) {
  extern __shared__ __align__(16) double smem[];
  double *sIv = smem;                  // [kK][kNC]: inv_evec[j][x] at [x][j]
  double *sA = sIv + kK * kNC;         // [kK][kSaLd]
  double *sMax = sA + kK * kSaLd;      // [kRows] row maxima
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  TileMap tm;
  tm.C = c.C;
  tm.tp = tile_patterns(c.C);
  tm.nrow = tm.tp * c.C;
  tm.p0 = (long)(tile0 + blockIdx.x) * tm.tp;
  tm.P = c.P;
  for (int idx = tid; idx < kK * kNC; idx += blockDim.x) {
    const int k = idx / kNC, x = idx - k * kNC;
    sIv[idx] = (k < kN && x < kN) ? c.inv_evec[x * kN + k] : 0.0;
  }
  // rows of sA past the tile's rows (64 % C) are never written: zero them once
  for (int idx = tid; idx < kK * kSaLd; idx += blockDim.x) sA[idx] = 0.0;
  double *part = static_cast<double *>(c.partials);
  const int blk = c.C * kN;
  for (int kop = 0; kop < nops; kop++) {
    const DevOp op = ops[kop];
    const double *tk = tab + (size_t)kop * stride;
    const double *leafL = tk + 2 * et_doubles(c.C);
    const double *leafR = leafL + (size_t)(c.unknown + 1) * blk;
    const bool tiptip = op.l_kind == GEMS_CHILD_TIP && op.r_kind == GEMS_CHILD_TIP;
    double vl[8][4], o[8][4];
    int sl[8], sr[8];
    __syncthreads();  // sA free (previous op's last GEMM, or the set-up)
    child_v(c, tm, op.l_kind, op.l_id, tk, leafL, sA, ty, tx, vl, sl);
    __syncthreads();
    child_v(c, tm, op.r_kind, op.r_id, tk + et_doubles(c.C), leafR, sA, ty, tx, o, sr);
    __syncthreads();
    // T = V_L (*) V_R into sA (k-major); columns >= 61 of V are zero, so row 61 of T is zero
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int x = tx + 16 * q;
      if (x < kK) {
#pragma unroll
        for (int j = 0; j < 8; j++) sA[x * kSaLd + ty * 8 + j] = vl[j][q] * o[j][q];
      }
    }
    __syncthreads();
    gemm_tile<false>(sA, sIv, ty, tx, o);
    double m[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      double x = 0.0;
#pragma unroll
      for (int q = 0; q < 4; q++) x = fmax(x, fabs(o[j][q]));
      for (int off = 1; off < 16; off <<= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, off));
      m[j] = x;
    }
    // the pattern's maximum over its C rows (rows c * tp + lp, in other threads)
    if (tx == 0) {
#pragma unroll
      for (int j = 0; j < 8; j++) sMax[ty * 8 + j] = m[j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int lp = (ty * 8 + j) % tm.tp;
      double x = 0.0;
      for (int u = 0; u < tm.C; u++) x = fmax(x, sMax[u * tm.tp + lp]);
      m[j] = x;
    }
    uint16_t *scd = c.scale + (size_t)op.dst_slot * c.slot_scale;
    double *dst = part + (size_t)op.dst_slot * c.slot_elems;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int r = ty * 8 + j;
      if (!tm.valid(r)) continue;
      const long p = tm.pattern(r);
      const int cat = tm.cat(r);
      int s_out = sl[j] + sr[j];
      if (!tiptip && m[j] < kScaleThr && c.invar[p] == 0.0) {
#pragma unroll
        for (int q = 0; q < 4; q++) o[j][q] = ldexp(o[j][q], kScaleExp);
        s_out += 1;
      }
      double *row = dst + tm.off(r);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int col = tx + 16 * q;
        if (col < kN) row[col] = o[j][q];
      }
      if (tx == 0 && cat == 0) scd[p] = (uint16_t)s_out;
    }
  }
}

// ---------------------------------------------------------------------------------------
// SAFE scaling: categories are independent, so a CTA owns 64 patterns of ONE category and its
// warps 8 patterns each, for the whole op list, with the products on the FP64 mma (m8n8k4).
//
// Lane (g, t) = (lane / 4, lane % 4) holds A[g][k = t], B[k = t][n = g] and C[g][2t], C[g][2t + 1].
// K step s covers states 4s .. 4s + 3 (the sums run in index order, as in the per-row kernel);
// column n = 2 t' + e of N tile m stands for state 8m + 4e + t', so lane t's C fragment of a
// product holds states 4s + t, s = 2m + e: the A fragments of the next one.  Products chain in
// registers, a lane always holds the states {4s + t} of pattern g (it stores and re-reads those
// elements itself: no synchronisation between ops), and the child that the last op wrote comes
// from registers (the plan's forward bit).
//
// Both operands' B fragments lie in shared memory in lane order (one 16-byte read gives two):
// inv_evec for the whole traversal, E_c of the next two internal children in a ring of two 32 KB
// slots filled by cp.async while the product before runs; one barrier per product.
// Bound by FP64 throughput: 256 mma per 8 patterns and op with one internal child.
// ---------------------------------------------------------------------------------------
constexpr int kFrag = kK * kNC;               // doubles of one matrix in fragment order
constexpr int kWarpsW = 8, kThreadsW = 32 * kWarpsW;
constexpr size_t kSmemW = sizeof(double) * 3 * (size_t)kFrag;
static_assert(kWarpsW * 8 == kRows, "a warp holds 8 patterns");

// element i of a matrix in fragment order, [16 K steps][4 pairs of N tiles][32 lanes][2]: its
// contraction index k and output state x
__device__ __forceinline__ void frag_place(int i, int &k, int &x) {
  const int lane = (i >> 1) & 31, m = 2 * ((i >> 6) & 3) + (i & 1), n = lane >> 2;
  k = 4 * (i >> 8) + (lane & 3);
  x = 8 * m + 4 * (n & 1) + (n >> 1);
}
// v <- M . v for the warp's 8 patterns
__device__ __forceinline__ void product(const double *frag, int lane, double (&v)[16]) {
  __syncwarp();
  double acc[8][2];
#pragma unroll
  for (int m = 0; m < 8; m++) acc[m][0] = acc[m][1] = 0.0;
  const double2 *f = reinterpret_cast<const double2 *>(frag) + lane;
#pragma unroll
  for (int s = 0; s < 16; s++) {
    double2 b[4];
#pragma unroll
    for (int q = 0; q < 4; q++) b[q] = f[(s * 4 + q) * 32];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      dmma(acc[2 * q], v[s], b[q].x);
      dmma(acc[2 * q + 1], v[s], b[q].y);
    }
  }
#pragma unroll
  for (int s = 0; s < 16; s++) v[s] = acc[s >> 1][s & 1];
}

// Op tables of the SAFE form, grid (nops, 2 sides, C): per side and category, an internal child's
// E_c in fragment order, or a tip child's messages [state code][8][4 lanes][2] (E_c . tip vector,
// 1 for the unknown state) in the order its rows are read.
constexpr int kTipRow = 64;  // doubles per state code
__global__ void __launch_bounds__(256) k_prep_ops_g61w(DevCtx c, const DevOp *ops, double *tab,
                                                       size_t stride) {
  extern __shared__ __align__(16) double sE[];  // [kFrag]
  __shared__ double d[kK];
  const int k = blockIdx.x, side = blockIdx.y, cc = blockIdx.z;
  const DevOp op = ops[k];
  const double len = side ? op.r_len : op.l_len;
  for (int i = threadIdx.x; i < kN; i += blockDim.x) d[i] = exp(c.eval[i] * (c.rates[cc] * len));
  __syncthreads();
  double *out = tab + (size_t)k * stride + ((size_t)side * c.C + cc) * kFrag;
  const bool tip = (side ? op.r_kind : op.l_kind) == GEMS_CHILD_TIP;
  for (int i = threadIdx.x; i < kFrag; i += blockDim.x) {
    int kk, x;
    frag_place(i, kk, x);
    const double v = kk < kN && x < kN ? c.evec[x * kN + kk] * d[kk] : 0.0;
    if (tip)
      sE[i] = v;
    else
      out[i] = v;
  }
  if (!tip) return;
  __syncthreads();
  // a warp's 8 state codes: rows of tip vectors times E_c, summed in index order
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int st = 8 * (threadIdx.x >> 5) + g;
  double v[16];
#pragma unroll
  for (int s = 0; s < 16; s++)
    v[s] = st < c.unknown && 4 * s + t < kN ? c.tip[(size_t)st * kN + 4 * s + t] : 0.0;
  product(sE, lane, v);
  if (st > c.unknown) return;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const double a = st == c.unknown ? 1.0 : v[2 * q], b = st == c.unknown ? 1.0 : v[2 * q + 1];
    reinterpret_cast<double2 *>(out + st * kTipRow)[q * 4 + t] = make_double2(a, b);
  }
}

__global__ void __launch_bounds__(kThreadsW, 2)
    k_traverse_g61w(DevCtx c, const DevOp *__restrict__ ops, int nops,
                    const double *__restrict__ tab, size_t stride, int tile0) {
  extern __shared__ __align__(16) double smem[];
  double *sInv = smem, *sE = smem + kFrag;
  const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int cat = blockIdx.x % c.C;
  const long p = (long)(tile0 + blockIdx.x / c.C) * kRows + 8 * (tid >> 5) + g;
  const bool act = p < c.P;
  const size_t row = ((size_t)p * c.C + cat) * kN;
  for (int i = tid; i < kFrag; i += kThreadsW) {
    int kk, x;
    frag_place(i, kk, x);
    sInv[i] = kk < kN && x < kN ? c.inv_evec[x * kN + kk] : 0.0;
  }
  double *part = static_cast<double *>(c.partials);
  const bool inv0 = act && c.invar[p] == 0.0;

  // the side of an op that is worked on first: the forwarded child, which is in registers
  auto first_side = [](const DevOp &o) {
    return o.r_kind == GEMS_CHILD_PARTIAL && plan_rsrc(o.pad_) == kSrcFwd ? 1 : 0;
  };
  // the next internal child in working order from (op k, position i), and its E_c into a slot
  int nk = 0, ni = 0, nslot = 0;
  auto fetch_next = [&]() {
    for (; nk < nops; nk++, ni = 0) {
      const DevOp o = ops[nk];
      for (; ni < 2; ni++) {
        const int side = ni ^ first_side(o);
        if ((side ? o.r_kind : o.l_kind) != GEMS_CHILD_PARTIAL) continue;
        const double *src =
            tab + (size_t)nk * stride + ((size_t)side * c.C + cat) * kFrag + 2 * tid;
        const uint32_t dst = static_cast<uint32_t>(
            __cvta_generic_to_shared(sE + (size_t)(nslot & 1) * kFrag + 2 * tid));
#pragma unroll
        for (int j = 0; j < kFrag / 2 / kThreadsW; j++)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                           dst + j * kThreadsW * 16),
                       "l"(src + j * kThreadsW * 2)
                       : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
        nslot++;
        ni++;
        return;
      }
    }
  };
  fetch_next();
  int slot = 0;
  // message of an internal child: its E_c has come for every warp, and every warp is done with
  // the slot before it, which the next one's copy may fill
  auto message = [&](double (&v)[16]) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    fetch_next();
    product(sE + (size_t)(slot & 1) * kFrag, lane, v);
    slot++;
  };

  __syncthreads();  // sInv, before any warp's first product
  double x[16];
  int sx = 0;  // counter of x
#pragma unroll
  for (int s = 0; s < 16; s++) x[s] = 0.0;
  for (int k = 0; k < nops; k++) {
    const DevOp op = ops[k];
    const double *tk = tab + (size_t)k * stride;
    const int first = first_side(op);
    const bool fwd = first || (op.l_kind == GEMS_CHILD_PARTIAL && plan_lsrc(op.pad_) == kSrcFwd);
    const bool tiptip = op.l_kind == GEMS_CHILD_TIP && op.r_kind == GEMS_CHILD_TIP;
    // a child's elements and counter
    auto load = [&](int side, double (&v)[16], int &s) {
      const int kind = side ? op.r_kind : op.l_kind, id = side ? op.r_id : op.l_id;
      s = 0;
#pragma unroll
      for (int q = 0; q < 16; q++) v[q] = 0.0;
      if (!act) return;
      if (kind == GEMS_CHILD_TIP) {
        const int st = min((int)c.tips[(size_t)id * c.P + p], c.unknown);
        const double2 *q = reinterpret_cast<const double2 *>(
                               tk + ((size_t)side * c.C + cat) * kFrag + st * kTipRow) + t;
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const double2 a = __ldg(q + 4 * j);
          v[2 * j] = a.x, v[2 * j + 1] = a.y;
        }
      } else {
        const double *q = part + (size_t)id * c.slot_elems + row + t;
#pragma unroll
        for (int j = 0; j < 15; j++) v[j] = __ldcg(q + 4 * j);
        if (t == 0) v[15] = __ldcg(q + 60);
        s = c.scale[(size_t)id * c.slot_scale + (size_t)p * c.C + cat];
      }
    };
    double y[16];
    int sy;
    if (!fwd) load(first, x, sx);
    if ((first ? op.r_kind : op.l_kind) == GEMS_CHILD_PARTIAL) message(x);
    load(1 - first, y, sy);
    if ((first ? op.l_kind : op.r_kind) == GEMS_CHILD_PARTIAL) message(y);
#pragma unroll
    for (int s = 0; s < 16; s++) x[s] *= y[s];
    product(sInv, lane, x);
    // |x| by its high word, NaN as 0: a maximum that ignores NaN, compared with a power of two
    int h = 0;
#pragma unroll
    for (int s = 0; s < 16; s++) {
      const int w = __double2hiint(x[s]) & 0x7fffffff;
      h = max(h, w > 0x7ff00000 ? 0 : w);
    }
    h = max(h, __shfl_xor_sync(0xffffffffu, h, 1));
    h = max(h, __shfl_xor_sync(0xffffffffu, h, 2));
    sx += sy;
    if (!tiptip && h < 0x2FF00000 /* 2^-256 */ && inv0) {
#pragma unroll
      for (int s = 0; s < 16; s++) x[s] *= 0x1p256;
      sx += 1;
    }
    if (act) {
      double *q = part + (size_t)op.dst_slot * c.slot_elems + row + t;
#pragma unroll
      for (int j = 0; j < 15; j++) q[4 * j] = x[j];
      if (t == 0) {
        q[60] = x[15];
        c.scale[(size_t)op.dst_slot * c.slot_scale + (size_t)p * c.C + cat] = (uint16_t)sx;
      }
    }
    __syncwarp();  // the counter that lane t = 0 wrote is read by its pattern's four lanes
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

}  // namespace

size_t g61_op_doubles(int ncat, int unknown) {
  return 2 * et_doubles(ncat) + 2 * (size_t)(unknown + 1) * ncat * kN;
}

bool g61_supported(const Session *s) {
  const int C = s->desc.ncat;
  return s->g61_enabled && s->desc.precision == GEMS_PREC_FP64 && s->desc.nstates == kN &&
         C >= 1 && C <= kMaxCatG;
}

int launch_prep_ops_g61(Session *s, int nops) {
  if (nops <= 0) return GEMS_OK;
  if (s->desc.scaling == GEMS_SCALE_SAFE)
    k_prep_ops_g61w<<<dim3(nops, 2, s->desc.ncat), 256, sizeof(double) * kFrag, s->stream>>>(
        s->ctx(), s->d_ops, s->d_opmats, s->op_stride);
  else
    k_prep_ops_g61<<<dim3(nops, 2), 256, 0, s->stream>>>(s->ctx(), s->d_ops, s->d_opmats,
                                                          s->op_stride);
  s->launches++;
  GEMS_CUDA(cudaGetLastError());
  return GEMS_OK;
}

int g61_pattern_granule(const Session *s) {
  return s->desc.scaling == GEMS_SCALE_SAFE ? kRows : tile_patterns(s->desc.ncat);
}

int launch_traverse_g61(Session *s, int nops, int p0, int p1) {
  if (nops <= 0 || p1 <= p0) return GEMS_OK;
  const bool safe = s->desc.scaling == GEMS_SCALE_SAFE;
  const int gran = g61_pattern_granule(s);
  if (p0 % gran != 0 || (p1 % gran != 0 && p1 != s->P)) {
    set_error("FP64 61-state traversal: pattern range not aligned to its pattern tiles");
    return GEMS_ERR_BAD_ARG;
  }
  cudaEvent_t ev0;
  if (int st = prof_begin(s, 0, &ev0)) return st;
  const int tile0 = p0 / gran, tiles = (p1 + gran - 1) / gran - tile0;
  // the limit is a per-kernel attribute shared by every thread of the process: always the same
  // value
  if (safe) {  // FP64 tensor cores, one category per tile
    GEMS_CUDA(cudaFuncSetAttribute(k_traverse_g61w, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kSmemW));
    k_traverse_g61w<<<tiles * s->desc.ncat, kThreadsW, kSmemW, s->stream>>>(
        s->ctx(), s->d_ops, nops, s->d_opmats, s->op_stride, tile0);
  } else {  // NORM: a pattern's categories in one tile, FP64 FMA
    GEMS_CUDA(cudaFuncSetAttribute(k_traverse_g61, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kSmemG));
    k_traverse_g61<<<tiles, kThreadsG, kSmemG, s->stream>>>(s->ctx(), s->d_ops, nops, s->d_opmats,
                                                            s->op_stride, tile0);
  }
  s->launches++;
  GEMS_CUDA(cudaGetLastError());
  return prof_end(s, 0, ev0);
}

}  // namespace gems
