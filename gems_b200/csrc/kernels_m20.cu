// kernels_m20.cu -- mixed-precision 20-state traversal (FP32 real-space partials, 4n^2-flop form).
//
// Node update per category c:  out = (P_c(t_L) . L) (*) (P_c(t_R) . R), FP32 throughout.
// The 20 x 20 products are small and each op depends on the one before it, so what counts is how
// little stands between two of them.  Here an op is register work of single warps:
// - A warp owns 2 x 32 / G patterns (G = categories rounded up to a power of two); lane
//   (category, j) holds the rows of its category of two patterns.  Rows live in registers as f32
//   pairs, and the dot products run on fma.rn.f32x2: two multiply-adds an issue, the pairs of a
//   row of P and of a child row as they lie in memory.
// - P_c comes from shared memory: the lanes of a category read the same 16 bytes, with those of
//   the other categories beside them, so one read of all categories is one wavefront and serves
//   eight multiply-adds a lane.
// - The child that the last op wrote is in registers (the plan's forward bit); others are read
//   from their slot, each lane its own elements.  Row maxima span a pattern's lanes by shuffles.
// - The op tables (descriptor, an internal child's P_c, a tip child's rows of every state code)
//   come into a ring of shared-memory slots by one bulk copy each, counted by mbarriers: no warp
//   waits at a CTA barrier.  16 KB an op, where the split TF32 images that tensor-core operands
//   need are 48.
// This form took the place of a tcgen05 one (split TF32 products, one 128-pattern tile per CTA,
// two CTAs per SM at most): its op was one chain of copy, split, MMA, TMEM load, rescaling and
// store across the whole CTA, 6,400 cycles for 128 patterns, with the tensor pipe 9% busy.
// Protein +G4, 128 taxa, 98,762 patterns: evaluation 2.66 -> 1.61 ms, |error of lnL| 2e-7 ->
// 1e-8 of it.  Bound by shared-memory reads (a tip row per lane conflicts 2.4 ways: 0.3 ms), the
// FP32 rate (0.55 ms) and the latencies between them.  Measured shapes: one pattern per lane, 24
// warps per SM 2.28 ms; two, with tables staged by every thread between CTA barriers 1.89 ms; in
// the ring, 128 threads x 3 CTAs per SM 1.71, 256 x 2 1.93 (spills), 384 x 1 1.90, 192 x 2 1.61.
// Every wait is bounded; a warp that gives up makes the others leave, and the host reports it at
// its next wait for the session.
#include <algorithm>
#include <string>

#include "gems_internal.cuh"
#include "tc_common.cuh"

namespace gems {

namespace {

constexpr int kN = 20;
constexpr int kThreadsM = 192;
constexpr int kCtasM = 2;       // resident CTAs per SM
constexpr int kNP = 2;          // patterns per lane
constexpr int kRing = 4;        // op tables in shared memory (fewer where they do not fit)

typedef unsigned long long f2;  // two packed FP32

__host__ __device__ constexpr int lanes_of(int C) {
  return C <= 1 ? 1 : (C <= 2 ? 2 : (C <= 4 ? 4 : (C <= 8 ? 8 : 16)));
}
// floats between the tip rows of consecutive state codes: an odd number of 16-byte units
__host__ __device__ constexpr int tip_stride(int C) { return 4 * ((C * kN / 4) | 1); }
// floats of a side's table: P_c as [row][quad][G categories][4] (an internal child), or the tip
// rows of every state code
__host__ __device__ constexpr int p_floats(int C) { return lanes_of(C) * kN * kN; }
__host__ __device__ constexpr int tip_floats(int C, int unknown) {
  return (unknown + 1) * tip_stride(C);
}
__host__ __device__ constexpr int side_floats(int C, int unknown) {
  return p_floats(C) > tip_floats(C, unknown) ? p_floats(C) : tip_floats(C, unknown);
}
// an op's table: a descriptor {slot, children, flags}, then the two sides
constexpr int kHeadM = 4;
enum : int { kTipL = 1, kTipR = 2, kFwdL = 4, kFwdR = 8 };  // tip child; the last op's output
__host__ __device__ constexpr int op_floats(int C, int unknown) {
  return kHeadM + 2 * side_floats(C, unknown);
}

__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float sum2(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return x + y;
}
__device__ __forceinline__ f2 pack2(float x, float y) {
  f2 a;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(x), "f"(y));
  return a;
}

// P_c(t) of internal children and the messages of tip children, FP64 sums rounded once; grid
// (nops, 2 sides, C)
__global__ void k_prep_ops_m20(DevCtx c, const DevOp *ops, float *tab, size_t stride_f, int R) {
  __shared__ double ex[kN], ev[kN * (kN + 1)], iv[kN * kN];
  __shared__ float P[kN * kN];
  const int k = blockIdx.x, side = blockIdx.y, cc = blockIdx.z;
  const DevOp op = ops[k];
  const double len = side ? op.r_len : op.l_len;
  if (threadIdx.x == 0 && side == 0 && cc == 0) {
    int f = (op.l_kind == GEMS_CHILD_TIP ? kTipL : 0) | (op.r_kind == GEMS_CHILD_TIP ? kTipR : 0);
    if (!(f & kTipL) && plan_lsrc(op.pad_) == kSrcFwd) f |= kFwdL;
    if (!(f & kTipR) && plan_rsrc(op.pad_) == kSrcFwd) f |= kFwdR;
    *reinterpret_cast<int4 *>(tab + (size_t)k * stride_f) =
        make_int4(op.dst_slot, op.l_id, op.r_id, f);
  }
  if (threadIdx.x < kN) ex[threadIdx.x] = exp(c.eval[threadIdx.x] * (c.rates[cc] * len));
  for (int i = threadIdx.x; i < kN * kN; i += blockDim.x) {
    ev[i / kN * (kN + 1) + i % kN] = c.evec[i];
    iv[i] = c.inv_evec[i];
  }
  __syncthreads();
  float *out = tab + (size_t)k * stride_f + kHeadM + (size_t)side * R;
  const bool tip = (side ? op.r_kind : op.l_kind) == GEMS_CHILD_TIP;
  for (int i = threadIdx.x; i < kN * kN; i += blockDim.x) {
    const int x = i / kN, y = i - x * kN;
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < kN; j++) acc = fma(ev[x * (kN + 1) + j] * ex[j], iv[j * kN + y], acc);
    const float v = (float)fmax(acc, 0.0);
    if (tip)
      P[i] = v;
    else
      out[((i / 4) * lanes_of(c.C) + cc) * 4 + i % 4] = v;
  }
  if (!tip) return;
  __syncthreads();
  const int ts = tip_stride(c.C);
  for (int i = threadIdx.x; i < (c.unknown + 1) * kN; i += blockDim.x) {
    const int s = i / kN, x = i - s * kN;
    float acc = 0.f;
#pragma unroll
    for (int y = 0; y < kN; y++) acc = fmaf(P[x * kN + y], (float)__ldg(c.tip_real + s * kN + y), acc);
    out[s * ts + cc * kN + x] = acc;
  }
}

struct RingM {
  uint64_t full[kRing], empty[kRing];
  int err;  // a wait expired: every warp leaves
};

template <int G, bool SAFE>
__global__ void __launch_bounds__(kThreadsM, kCtasM)
    k_traverse_m20(DevCtx c, const float *__restrict__ tab, size_t stride_f, int nops, int slots,
                   int R, int p0, int p1, int *flag) {
  extern __shared__ __align__(16) float sm[];  // ring of op tables
  __shared__ RingM ring;
  constexpr int LP = 32 / G;  // lanes per category
  const int lane = threadIdx.x & 31, C = c.C;
  const int cat = lane / LP;
  // this lane's patterns, LP apart
  const int warps = blockDim.x >> 5;
  const int pa = p0 + (blockIdx.x * warps + (threadIdx.x >> 5)) * kNP * LP + lane % LP;
  bool act[kNP], inv0[kNP];
#pragma unroll
  for (int j = 0; j < kNP; j++) {
    act[j] = pa + j * LP < p1 && cat < C;
    inv0[j] = act[j] && c.invar[pa + j * LP] == 0.0;
  }
  float *part = static_cast<float *>(c.partials);
  const int ts = tip_stride(C), tcat = cat < C ? cat : 0;
  const int opf = kHeadM + 2 * R, lag = slots > 2 ? 2 : 1;
  if (threadIdx.x == 0) {
    for (int i = 0; i < slots; i++) {
      tc::mbar_init(tc::sptr(&ring.full[i]), 1);
      tc::mbar_init(tc::sptr(&ring.empty[i]), warps);
    }
    ring.err = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // the table of op k into its slot (one thread; the slot is free)
  auto fetch = [&](int k) {
    const uint32_t bar = tc::sptr(&ring.full[k % slots]);
    const uint32_t bytes = (uint32_t)opf * 4;
    tc::mbar_expect_tx(bar, bytes);
    tc::bulk_g2s(tc::sptr(sm + (size_t)(k % slots) * opf), tab + (size_t)k * stride_f, bytes, bar);
  };
  int fetched = 0;  // thread 0: op tables asked for
  if (threadIdx.x == 0)
    for (; fetched < slots && fetched < nops; fetched++) fetch(fetched);
  // tip state codes of an op: left, right of the first pattern, then of the second
  auto tip_bytes = [&](const int4 &d) {
    int b = 0;
#pragma unroll
    for (int j = 0; j < kNP; j++) {
      if (!act[j]) continue;
      const uint8_t *t = c.tips + pa + j * LP;
      if (d.w & kTipL) b |= min((int)t[(size_t)d.y * c.P], c.unknown) << (16 * j);
      if (d.w & kTipR) b |= min((int)t[(size_t)d.z * c.P], c.unknown) << (16 * j + 8);
    }
    return b;
  };
  // the table of op k has come (false: a wait expired, here or in another warp)
  auto ready = [&](int k) {
    const bool ok = tc::ws_wait(tc::sptr(&ring.full[k % slots]), (k / slots) & 1, &ring.err);
    return __all_sync(0xffffffffu, ok) != 0;
  };

  f2 x[kNP][kN / 2];  // the last op's output
  int sx[kNP] = {};
#pragma unroll
  for (int j = 0; j < kNP; j++)
#pragma unroll
    for (int i = 0; i < kN / 2; i++) x[j][i] = 0ull;
  bool ok = ready(0);
  int tips = ok ? tip_bytes(*reinterpret_cast<const int4 *>(sm)) : 0;
  for (int k = 0; k < nops && ok; k++) {
    // the next table of the ring, into the slot of the op two (with two slots: one) before
    if (threadIdx.x == 0 && k >= lag && fetched < nops) {
      ok = tc::ws_wait(tc::sptr(&ring.empty[fetched % slots]), (fetched / slots - 1) & 1,
                       &ring.err);
      if (ok) fetch(fetched++);
    }
    const float *tk = sm + (size_t)(k % slots) * opf + kHeadM;
    const int4 op = *reinterpret_cast<const int4 *>(tk - kHeadM);
    // the forwarded child first: it is in registers
    const bool fwd_r = op.w & kFwdR, fwd = op.w & (kFwdL | kFwdR);
    float t[kNP][kN];
    int sc[kNP] = {};
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int side = fwd_r ? 1 - i : i;
      const float *ms = tk + (size_t)side * R;
      if (op.w >> side & 1) {
#pragma unroll
        for (int j = 0; j < kNP; j++) {
          const int st = tips >> (16 * j + 8 * side) & 255;
          const float4 *row = reinterpret_cast<const float4 *>(ms + st * ts + tcat * kN);
#pragma unroll
          for (int q = 0; q < kN / 4; q++) {
            const float4 v = row[q];
            t[j][4 * q] = i ? t[j][4 * q] * v.x : v.x;
            t[j][4 * q + 1] = i ? t[j][4 * q + 1] * v.y : v.y;
            t[j][4 * q + 2] = i ? t[j][4 * q + 2] * v.z : v.z;
            t[j][4 * q + 3] = i ? t[j][4 * q + 3] * v.w : v.w;
          }
        }
        continue;
      }
      if (i == 0 && fwd) {
#pragma unroll
        for (int j = 0; j < kNP; j++) sc[j] = sx[j];
      } else {
        const int id = side ? op.z : op.y;
        const float *slot = part + (size_t)id * c.slot_elems;
        const uint16_t *scale = c.scale + (size_t)id * c.slot_scale;
#pragma unroll
        for (int j = 0; j < kNP; j++) {
          if (!act[j]) continue;
          const int p = pa + j * LP;
          const float *row = slot + mix_off<kN>(c, p, cat);
#pragma unroll
          for (int q = 0; q < kN / 4; q++) {
            const ulonglong2 v =
                __ldcg(reinterpret_cast<const ulonglong2 *>(row + (size_t)q * mix_cs<kN>()));
            x[j][2 * q] = v.x;
            x[j][2 * q + 1] = v.y;
          }
          sc[j] += SAFE ? scale[(size_t)p * C + cat] : scale[p];
        }
      }
      const ulonglong2 *P = reinterpret_cast<const ulonglong2 *>(ms) + tcat;
#pragma unroll
      for (int r = 0; r < kN; r++) {
        f2 a[kNP] = {};
#pragma unroll
        for (int q = 0; q < kN / 4; q++) {
          const ulonglong2 m = P[(r * (kN / 4) + q) * G];
#pragma unroll
          for (int j = 0; j < kNP; j++) a[j] = fma2(m.x, x[j][2 * q], a[j]);
#pragma unroll
          for (int j = 0; j < kNP; j++) a[j] = fma2(m.y, x[j][2 * q + 1], a[j]);
        }
#pragma unroll
        for (int j = 0; j < kNP; j++) {
          const float u = sum2(a[j]);
          t[j][r] = i ? t[j][r] * u : u;
        }
      }
    }
    // this warp is done with the table; the next op's tip state codes come under the rest
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(tc::sptr(&ring.empty[k % slots]));
    int next_tips = 0;
    if (k + 1 < nops && (ok = ready(k + 1) && ok))
      next_tips = tip_bytes(*reinterpret_cast<const int4 *>(sm + (size_t)((k + 1) % slots) * opf));
#pragma unroll
    for (int j = 0; j < kNP; j++) {
      float mx = 0.f;
#pragma unroll
      for (int i = 0; i < kN; i++) mx = fmaxf(mx, t[j][i]);
      if (!SAFE) {
        if (cat >= C) mx = 0.f;
#pragma unroll
        for (int o = LP; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      }
      sx[j] = sc[j];
      if ((op.w & 3) != 3 && mx < kScaleThrF && inv0[j]) {
#pragma unroll
        for (int i = 0; i < kN; i++) t[j][i] *= 18446744073709551616.0f;  // 2^64
        sx[j] += 1;
      }
#pragma unroll
      for (int i = 0; i < kN / 2; i++) x[j][i] = pack2(t[j][2 * i], t[j][2 * i + 1]);
      if (!act[j]) continue;
      const int p = pa + j * LP;
      float *row = part + (size_t)op.x * c.slot_elems + mix_off<kN>(c, p, cat);
#pragma unroll
      for (int q = 0; q < kN / 4; q++)
        *reinterpret_cast<ulonglong2 *>(row + (size_t)q * mix_cs<kN>()) =
            make_ulonglong2(x[j][2 * q], x[j][2 * q + 1]);
      uint16_t *scale = c.scale + (size_t)op.x * c.slot_scale;
      if (SAFE)
        scale[(size_t)p * C + cat] = (uint16_t)sx[j];
      else if (cat == 0)
        scale[p] = (uint16_t)sx[j];
    }
    __syncwarp();  // NORM: the counter that a pattern's first lane wrote is read by its others
    tips = next_tips;
    ok = __all_sync(0xffffffffu, ok) != 0;
  }
  if (!ok) {
    *(volatile int *)&ring.err = 1;
    if (lane == 0) *(volatile int *)flag = GEMS_ERR_TIMEOUT;
    // the copies issued must land before the CTA's shared memory is released
    if (threadIdx.x == 0)
      for (int k = fetched > slots ? fetched - slots : 0; k < fetched; k++)
        tc::mbar_wait(tc::sptr(&ring.full[k % slots]), (k / slots) & 1);
  }
}

template <bool SAFE>
const void *kernel_m20(int G) {
  switch (G) {
    case 1: return (const void *)k_traverse_m20<1, SAFE>;
    case 2: return (const void *)k_traverse_m20<2, SAFE>;
    case 4: return (const void *)k_traverse_m20<4, SAFE>;
    case 8: return (const void *)k_traverse_m20<8, SAFE>;
    default: return (const void *)k_traverse_m20<16, SAFE>;
  }
}
// slots of the ring: at most 72 KB a CTA (two per SM beside the L1 cache), at least two
int slots_m20(int C, int unknown) {
  const size_t one = sizeof(float) * op_floats(C, unknown);
  return (int)std::max<size_t>(2, std::min<size_t>(kRing, (72 << 10) / one));
}
size_t smem_m20(int C, int unknown) {
  return sizeof(float) * slots_m20(C, unknown) * op_floats(C, unknown);
}

}  // namespace

size_t m20_op_floats(int ncat, int unknown) { return op_floats(ncat, unknown); }

const void *traverse_m20_kernel(const Session *s, int *threads, int *patterns, size_t *smem) {
  const int G = lanes_of(s->desc.ncat);
  *threads = kThreadsM;
  *patterns = kThreadsM / 32 * kNP * (32 / G);
  *smem = smem_m20(s->desc.ncat, s->unknown);
  const void *fn =
      s->desc.scaling == GEMS_SCALE_SAFE ? kernel_m20<true>(G) : kernel_m20<false>(G);
  // the limit is a property of the kernel, shared by every session and host thread: always set
  // to the largest size that its category counts need
  size_t most = 0;
  for (int c = G / 2 + 1; c <= G; c++) most = std::max(most, smem_m20(c, s->unknown));
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) !=
      cudaSuccess)
    return nullptr;
  return fn;
}

int launch_prep_ops_m20(Session *s, int nops) {
  if (nops <= 0) return GEMS_OK;
  k_prep_ops_m20<<<dim3(nops, 2, s->desc.ncat), 128, 0, s->stream>>>(
      s->ctx(), s->d_ops, reinterpret_cast<float *>(s->d_opmats), s->op_stride_tc,
      side_floats(s->desc.ncat, s->unknown));
  s->launches++;
  GEMS_CUDA(cudaGetLastError());
  return GEMS_OK;
}

int launch_traverse_m20(Session *s, int nops, int p0, int p1) {
  DevCtx c = s->ctx();
  int threads = 0, per = 0;
  size_t smem = 0;
  const void *fn = traverse_m20_kernel(s, &threads, &per, &smem);
  if (!fn) return cuda_status(cudaGetLastError(), "cudaFuncSetAttribute");
  // fewer warps per CTA where six would leave SMs without one, though fewer then share a copy of
  // an op's table (64 taxa, 3,000 patterns, one category: 8 CTAs of 6 warps 207 us, 47 of one
  // 181 us)
  const int one = per / (threads / 32), most = (p1 - p0 + one - 1) / one;
  threads = 32 * std::max(1, std::min(threads / 32, most / 148));
  per = one * (threads / 32);
  const int grid = (p1 - p0 + per - 1) / per;
  const float *tab = reinterpret_cast<const float *>(s->d_opmats);
  size_t stride = s->op_stride_tc;
  int R = side_floats(s->desc.ncat, s->unknown), slots = slots_m20(s->desc.ncat, s->unknown);
  int *flag = s->h_status;  // pinned: read by the host at its next wait
  void *args[] = {&c, &tab, &stride, &nops, &slots, &R, &p0, &p1, &flag};
  GEMS_CUDA(cudaLaunchKernel(fn, dim3(grid), dim3(threads), args, smem, s->stream));
  s->launches++;
  return GEMS_OK;
}

}  // namespace gems
