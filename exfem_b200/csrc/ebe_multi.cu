// Stored-Ke product for several right-hand sides on the CUDA cores, and the
// multi-load-case Jacobi PCG built on it.
//
// Y = opA(V) for nrhs = 1..16 right-hand sides at once, with the element matrices
// Ke (ne, nd, nd) stored in BF16, FP32 or FP64 (the output of
// exfem_element_stiffness) and V, Y (ndof, nrhs) with the right-hand sides fastest:
// FP32 for BF16 / FP32 Ke, FP64 for FP64 Ke.  This is the multi-load-case form of
// the reference's stored-Ke product (gfem/model.py:264-267 gather_matvec inside
// opA; gfem/optimize.py:116-143 vmaps it, with Jacobi PCG, over the load cases):
// one read of Ke serves every right-hand side.
//
// Per element the work is Ke (nd x nd) times U_e (nd x nrhs): 2 FMA per byte of
// BF16 Ke at four right-hand sides, far below what the tensor cores need to be the
// bound, so the contraction runs on the CUDA cores and the kernel is bound by
// streaming Ke.  The element rows are then summed per node through the gather plan in
// the reference's order (gfem/model.py:241-267) and opA's prescribed rows applied
// (gather_multi_kernel).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "async_copy.cuh"
#include "internal.h"
#include "solver.h"

namespace exfem {

namespace {

template <class KT>
__device__ __forceinline__ float to_acc(KT v, float) { return (float)v; }
template <>
__device__ __forceinline__ float to_acc<__nv_bfloat16>(__nv_bfloat16 v, float) { return __bfloat162float(v); }
__device__ __forceinline__ double to_acc(double v, double) { return v; }

}  // namespace

// ys[(e*nd + i)*NR + r] = sum_j Ke[e, i, j] * (free * V)[dof(e, j), r]
//
// One warp takes 4 C3D8 or 3 C3D10, one lane per element node: the lane forms the
// node's three rows, so that a value of U read from shared memory serves three rows of
// up to four elements at once (their lanes read different elements' values together).
// Ke comes into shared memory by bulk copies, in the same order as it is stored where
// the lanes' rows then lie in different banks (3 rows = an odd number of access
// widths), else with a padded copy per lane; the element values of V are gathered in
// 16-byte vectors meanwhile.  The rows leave through shared memory as one bulk store.
// B200, 131,072 C3D8 in BF16, four right-hand sides: 46 us; one lane per row with
// every value of U broadcast to one element's lanes took 55 us (the L1 pipe 79% busy:
// 87 wavefronts an element against 27 here).
template <int ET, int NR, class KT, class VT>
struct MultiSmem {
  using Ke = KT;
  static constexpr int NN = ElemTraits<ET>::nnode, ND = 3 * NN, EPW = 32 / NN;
  static constexpr int CHUNK = 3 * ND * (int)sizeof(KT);  // a lane's rows
  static constexpr int AW = CHUNK % 16 == 0 ? 16 : (CHUNK % 8 == 0 ? 8 : 4);
  static constexpr bool PAD = (CHUNK / AW) % 2 == 0;      // rows would share banks: padded copies
  static constexpr int KP = PAD ? CHUNK + 16 : CHUNK;
  static constexpr int W = 16 / (int)sizeof(VT), NRP = (NR + W - 1) / W * W;
  static constexpr int US = ND * NRP + W;                 // element stride of U: different banks
  static constexpr int KB = (EPW * NN * KP + 15) / 16 * 16;
  alignas(16) unsigned char k[KB];
  alignas(16) VT u[EPW * US];                             // U, then the rows
  uint64_t bar;
};

// right-hand sides R0 .. R0 + RG - 1 of a node's three rows; kr: the rows of Ke, ue: the
// element's values
template <int R0, int RG, class S, class VT>
__device__ __forceinline__ void node_rows(const unsigned char* kr, const VT* ue, VT (&y)[3][S::NRP]) {
  using KT = typename S::Ke;
  constexpr int ND = S::ND, W = S::W, NRP = S::NRP, AW = S::AW, CW = AW / (int)sizeof(KT);  // columns per read of Ke
  static_assert(RG % W == 0 && R0 + RG <= NRP, "whole vectors of right-hand sides");
  VT acc[3][RG];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int j = 0; j < RG; ++j) acc[r][j] = VT(0);
#pragma unroll
  for (int c0 = 0; c0 < ND; c0 += CW) {
    KT k[3][CW];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      using L = std::conditional_t<AW == 16, uint4, std::conditional_t<AW == 8, uint2, unsigned>>;
      const L t = *reinterpret_cast<const L*>(kr + (r * ND + c0) * sizeof(KT));
      memcpy(k[r], &t, AW);
    }
#pragma unroll
    for (int c = 0; c < CW; ++c) {
      VT u[RG];
#pragma unroll
      for (int h = 0; h < RG / W; ++h) {
        const uint4 t = *reinterpret_cast<const uint4*>(ue + (c0 + c) * NRP + R0 + h * W);
        memcpy(u + h * W, &t, 16);
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const VT kc = to_acc(k[r][c], VT(0));
        if constexpr (sizeof(VT) == 4) {
#pragma unroll
          for (int j = 0; j < RG; j += 2) {
            const float2 t =
                __ffma2_rn(make_float2(kc, kc), make_float2(u[j], u[j + 1]), make_float2(acc[r][j], acc[r][j + 1]));
            acc[r][j] = t.x;
            acc[r][j + 1] = t.y;
          }
        } else {
#pragma unroll
          for (int j = 0; j < RG; ++j) acc[r][j] += kc * u[j];
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int j = 0; j < RG; ++j) y[r][R0 + j] = acc[r][j];
}

template <int ET, int NR, class KT, class VT, int NW>
__global__ void __launch_bounds__(32 * NW)
ebe_multi_kernel(int64_t ne, const int32_t* __restrict__ conn, const KT* __restrict__ Ke, const VT* __restrict__ V,
                 const uint8_t* __restrict__ fixed, VT* __restrict__ ys, int vecv, int aligned, int* __restrict__ err) {
  using S = MultiSmem<ET, NR, KT, VT>;
  constexpr int NN = S::NN, ND = S::ND, EPW = S::EPW, W = S::W, NRP = S::NRP;
  constexpr int EB = ND * ND * (int)sizeof(KT);  // bytes of an element's matrix
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  S& sm = reinterpret_cast<S*>(smem_raw)[warp];
  const int64_t e0 = ((int64_t)blockIdx.x * NW + warp) * EPW;
  if (e0 >= ne) return;
  const int cnt = ne - e0 < EPW ? (int)(ne - e0) : EPW;
  const int el = lane / NN, node = lane - el * NN;
  const bool on = el < cnt;  // C3D10: el = 3 for the two spare lanes
  // ---- Ke: bulk copies need 16-byte boundaries and sizes
  const unsigned char* src = reinterpret_cast<const unsigned char*>(Ke) + e0 * EB;
  const bool bulk = aligned && (e0 * EB) % 16 == 0 && (cnt * EB) % 16 == 0;
  if (bulk) {
    if (lane == 0) {
      mbar_init(&sm.bar, 1);
      fence_mbar_init();
      mbar_expect_tx(&sm.bar, cnt * EB);
    }
    __syncwarp();
    if constexpr (S::PAD) {
      if (on) bulk_g2s(sm.k + lane * S::KP, src + lane * S::CHUNK, S::CHUNK, &sm.bar);
    } else {
      if (lane == 0) bulk_g2s(sm.k, src, cnt * EB, &sm.bar);
    }
  } else {
    for (int i = lane; i < cnt * EB / 4; i += 32)
      cp_async<4>(sm.k + (S::PAD ? i * 4 / S::CHUNK * (S::KP - S::CHUNK) : 0) + i * 4, src + i * 4, 4);
  }
  // ---- element values of V, prescribed DOFs zeroed
#pragma unroll
  for (int i0 = 0; i0 < EPW * ND; i0 += 32) {
    const int i = i0 + lane;
    if (i < cnt * ND) {
      const int64_t d = 3 * (int64_t)__ldg(conn + e0 * NN + i / 3) + i % 3;
      const bool off = fixed && __ldg(fixed + d);
      const VT* v = V + d * NR;
      VT* dst = sm.u + (i / ND) * S::US + (i % ND) * NRP;
      if (NR % W == 0 && vecv) {  // V 16-byte aligned (checked on the host)
#pragma unroll
        for (int h = 0; h < NRP / W; ++h) {
          uint4 t = __ldg(reinterpret_cast<const uint4*>(v) + h);
          if (off) t = make_uint4(0, 0, 0, 0);
          reinterpret_cast<uint4*>(dst)[h] = t;
        }
      } else {
#pragma unroll
        for (int j = 0; j < NRP; ++j) dst[j] = j < NR && !off ? __ldg(v + j) : VT(0);
      }
    }
  }
  if (bulk) {
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&sm.bar, 0, err))) return;
  } else {
    cp_async_wait_all();
  }
  __syncwarp();
  // ---- the node's three rows, at most eight FP64 right-hand sides at a time (registers)
  const unsigned char* kr = sm.k + (on ? lane : 0) * S::KP;
  const VT* ue = sm.u + (on ? el : 0) * S::US;
  constexpr int R1 = sizeof(VT) == 8 && NRP > 8 ? 8 : NRP;
  VT y[3][NRP];
  node_rows<0, R1, S>(kr, ue, y);
  if constexpr (R1 < NRP) node_rows<R1, NRP - R1, S>(kr, ue, y);
  __syncwarp();  // every lane has read U: its place takes the rows, as they are stored
  if (on) {
    VT* o = sm.u + lane * 3 * NR;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int j = 0; j < NR; j += (NR % W == 0 ? W : 1)) {
        if constexpr (NR % W == 0) {
          uint4 t;
          memcpy(&t, &y[r][j], 16);
          *reinterpret_cast<uint4*>(o + r * NR + j) = t;
        } else {
          o[r * NR + j] = y[r][j];
        }
      }
  }
  const int bytes = cnt * ND * NR * (int)sizeof(VT);
  VT* out = ys + e0 * (ND * NR);
  if (bytes % 16 == 0 && (uintptr_t)out % 16 == 0) {
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) {
      bulk_s2g(out, sm.u, bytes);
      bulk_commit();
      bulk_wait_read<0>();
    }
  } else {
    __syncwarp();
    for (int i = lane; i < cnt * ND * NR; i += 32) out[i] = sm.u[i];
  }
}

// Y[3n+c, r] = fixed ? V : sum over node n's gather-plan slots of the element rows, the
// slots in the plan's order (slot s holds rows 3s .. 3s+2).  One thread per RW rows (1 or
// the node's 3) and NV groups of W right-hand sides (W = 16 bytes' worth where their number
// and the addresses allow it, else 1); K plan slots and their values are requested before
// any is added.  Bound by the latency of the plan -> row chain with few right-hand sides
// and by the L1 pipe with many, where the plan's own reads count (once per thread).
template <class VT, int W, int NV, int RW, int K>
__global__ void __launch_bounds__(256)
gather_multi_kernel(int64_t nitem, int vmax, const int32_t* __restrict__ plan, int32_t sentinel,
                    const VT* __restrict__ ys, const uint8_t* __restrict__ fixed, const VT* __restrict__ V, int nrhs,
                    VT* __restrict__ Y) {
  struct alignas(W * sizeof(VT)) Vec {
    VT v[W];
  };
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int nq = nrhs / (W * NV);
  const int64_t item = nq == 1 ? t : t / nq;  // degree of freedom, or node (RW = 3)
  if (item >= nitem) return;
  const int r = (int)(t - item * nq) * (W * NV);
  const int64_t n = RW == 3 ? item : item / 3, d = RW == 3 ? 3 * item : item;
  const int c = (int)(d - 3 * n);
  const int32_t* row = plan + n * vmax;
  Vec s[RW][NV];
#pragma unroll
  for (int i = 0; i < RW; ++i)
#pragma unroll
    for (int h = 0; h < NV; ++h)
#pragma unroll
      for (int j = 0; j < W; ++j) s[i][h].v[j] = VT(0);
  for (int k0 = 0; k0 < vmax; k0 += K) {
    int32_t slot[K];
    Vec w[K][RW][NV];
#pragma unroll
    for (int k = 0; k < K; ++k) slot[k] = k0 + k < vmax ? row[k0 + k] : sentinel;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (slot[k] != sentinel)
#pragma unroll
        for (int i = 0; i < RW; ++i)
#pragma unroll
          for (int h = 0; h < NV; ++h)
            w[k][i][h] = reinterpret_cast<const Vec*>(ys + (3 * (int64_t)slot[k] + c + i) * nrhs + r)[h];
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (slot[k] != sentinel)
#pragma unroll
        for (int i = 0; i < RW; ++i)
#pragma unroll
          for (int h = 0; h < NV; ++h)
#pragma unroll
            for (int j = 0; j < W; ++j) s[i][h].v[j] += w[k][i][h].v[j];
    if (slot[K - 1] == sentinel) break;  // slots are listed without gaps
  }
#pragma unroll
  for (int i = 0; i < RW; ++i) {
    const bool pass = fixed && fixed[d + i];
#pragma unroll
    for (int h = 0; h < NV; ++h) {
      const int64_t o = (d + i) * nrhs + r;
      reinterpret_cast<Vec*>(Y + o)[h] = pass ? reinterpret_cast<const Vec*>(V + o)[h] : s[i][h];
    }
  }
}

template <class VT>
int launch_gather_multi(exfem_block_s* b, const VT* ys, const VT* V, VT* Y, int nrhs, bool bc, cudaStream_t s) {
  constexpr int W = 16 / (int)sizeof(VT);
  if (!b->nn) return EXFEM_OK;
  const uint8_t* fx = bc ? b->fixed.p : nullptr;
  const int32_t sentinel = (int32_t)(b->ne * b->nnode);
  const bool vec = nrhs % W == 0 && ((uintptr_t)V | (uintptr_t)Y | (uintptr_t)ys) % 16 == 0;
#define EXF_GATHER(W, NV, RW, K)                                                                                  \
  do {                                                                                                            \
    const int64_t nitem = RW == 3 ? b->nn : b->ndof(), work = nitem * (nrhs / (W * NV));                          \
    gather_multi_kernel<VT, W, NV, RW, K><<<(unsigned)((work + 255) / 256), 256, 0, s>>>(nitem, b->vmax, b->plan.p, \
                                                                                         sentinel, ys, fx, V, nrhs, Y); \
  } while (0)
  // B200, us with the rows cold, 256,000 C3D8 / 96,000 C3D10; in brackets one row and one
  // group per thread with K = 8 for every count.  FP32: 4 right-hand sides 26 / 16, 8
  // 41 / 23 (47 / 27), 12 55 / 32 (68 / 39), 16 67 / 35 (85 / 49); FP64: 8 67 / 36 (86 / 49),
  // 16 126 / 65 (166 / 95).  Counts without 16-byte groups take a node's three rows per
  // thread, which read the plan once: FP32 7 40 / 24 (72 / 44), FP64 15 126 / 72 (184 / 106);
  // with one or two right-hand sides there is too little to read for that.
  if (vec && nrhs % (2 * W) == 0) EXF_GATHER(W, 2, 1, 4);
  else if (vec && nrhs > W) EXF_GATHER(W, 1, 1, 4);
  else if (vec) EXF_GATHER(W, 1, 1, 8);
  else if (nrhs >= 3) EXF_GATHER(1, 1, 3, 4);
  else EXF_GATHER(1, 1, 1, (sizeof(VT) == 4 ? 4 : 8));
#undef EXF_GATHER
  EX_LAUNCH_CHECK();
  return EXFEM_OK;
}

template int launch_gather_multi<float>(exfem_block_s*, const float*, const float*, float*, int, bool, cudaStream_t);
template int launch_gather_multi<double>(exfem_block_s*, const double*, const double*, double*, int, bool,
                                         cudaStream_t);

namespace {

template <int ET, int NR, class KT, class VT>
int multi_go(exfem_block_s* b, const KT* Ke, const VT* V, VT* ys, const uint8_t* fx, cudaStream_t s) {
  using S = MultiSmem<ET, NR, KT, VT>;
  constexpr int NW = sizeof(S) > 16 * 1024 ? 2 : 4;  // small blocks where a warp's share is large
  constexpr size_t smem = NW * sizeof(S);
  constexpr int64_t per = NW * S::EPW;
  auto kern = ebe_multi_kernel<ET, NR, KT, VT, NW>;
  if constexpr (smem > 48 * 1024)
    EX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<(unsigned)((b->ne + per - 1) / per), 32 * NW, smem, s>>>(b->ne, b->conn.p, Ke, V, fx, ys,
                                                                   (uintptr_t)V % 16 == 0, (uintptr_t)Ke % 16 == 0,
                                                                   b->dev_err.p);
  EX_LAUNCH_CHECK();
  return EXFEM_OK;
}

template <int ET, class KT, class VT>
int multi_launch(exfem_block_s* b, const KT* Ke, int nrhs, const VT* V, VT* ys, const uint8_t* fx, cudaStream_t s) {
#define EXF_MULTI(NR) \
  case NR:            \
    return multi_go<ET, NR, KT, VT>(b, Ke, V, ys, fx, s);
  switch (nrhs) {
    EXF_MULTI(1) EXF_MULTI(2) EXF_MULTI(3) EXF_MULTI(4) EXF_MULTI(5) EXF_MULTI(6) EXF_MULTI(7) EXF_MULTI(8)
    EXF_MULTI(9) EXF_MULTI(10) EXF_MULTI(11) EXF_MULTI(12) EXF_MULTI(13) EXF_MULTI(14) EXF_MULTI(15)
    EXF_MULTI(16)
    default:
      set_error("the multi-right-hand-side stored-Ke product takes 1..16 right-hand sides, got %d", nrhs);
      return EXFEM_ERR_ARG;
  }
#undef EXF_MULTI
}

template <class KT, class VT>
int multi_dispatch(exfem_block_s* b, const KT* Ke, int nrhs, const VT* V, VT* Y, bool bc, DevBuf<VT>& rows,
                   cudaStream_t s) {
  if (nrhs < 1 || nrhs > 16) {
    set_error("the multi-right-hand-side stored-Ke product takes 1..16 right-hand sides, got %d", nrhs);
    return EXFEM_ERR_ARG;
  }
  int st;
  const size_t need = (size_t)b->ne * b->nd * nrhs;
  if (rows.n < need && (st = rows.alloc(need))) return st;
  if (b->ne) {
    const uint8_t* fx = bc ? b->fixed.p : nullptr;
    st = b->etype == EXFEM_C3D8 ? multi_launch<EXFEM_C3D8>(b, Ke, nrhs, V, rows.p, fx, s)
                                : multi_launch<EXFEM_C3D10>(b, Ke, nrhs, V, rows.p, fx, s);
    if (st) return st;
  }
  return launch_gather_multi<VT>(b, rows.p, V, Y, nrhs, bc, s);
}

}  // namespace

int launch_ebe_matvec_multi(exfem_block_s* b, const void* Ke, int ke_dtype, int nrhs, const void* V, void* Y,
                            bool bc, cudaStream_t s) {
  switch (ke_dtype) {
    case EXFEM_BF16:
      return multi_dispatch<__nv_bfloat16, float>(b, (const __nv_bfloat16*)Ke, nrhs, (const float*)V, (float*)Y, bc,
                                                  b->ys_tc, s);
    case EXFEM_F32:
      return multi_dispatch<float, float>(b, (const float*)Ke, nrhs, (const float*)V, (float*)Y, bc, b->ys_tc, s);
    case EXFEM_F64:
      return multi_dispatch<double, double>(b, (const double*)Ke, nrhs, (const double*)V, (double*)Y, bc, b->ys_m64,
                                            s);
    default:
      set_error("unknown element-matrix type %d", ke_dtype);
      return EXFEM_ERR_ARG;
  }
}

// ---------------------------------------------------------------- multi-case Jacobi PCG
//
// gfem/optimize.py:116-143: linalg.pcg (gfem/linalg.py:21-47) vmapped over the load
// cases, with A(v) = free K (free v) + (1 - free) v, the right-hand sides free * f
// and the preconditioner inv = free ? 1 / (d != 0 ? d : 1) : 1 from the assembled
// diagonal d.  Here every case is a column of (ndof, NR) arrays and each iteration
// issues one stored-Ke product for all of them; every case keeps its own scalars and
// stops on its own test (r.r <= tol^2 max(b.b, 1e-300) or k >= maxiter), after
// which its column is left as it is — the iterates of a vmapped while loop, whose
// finished lanes stop changing.  Reductions: per-block partial sums of each column
// in a fixed order, then the last block sums the partials in block order
// (deterministic for a given grid).

namespace {

constexpr int MP_T = 256;           // threads per reduction block
constexpr int MP_MAX_BLOCKS = 592;  // 4 per SM

struct MultiScal {
  double rz[16], rr[16], bb[16], tol2[16], alpha[16], beta[16];
  int k[16], done[16], act[16];
  int maxiter, loops;
};

enum MpOp { MP_INIT = 0, MP_ALPHA, MP_XR, MP_RZ };

// per-column block sums of `acc`, then the final sums (in block order) handed to fin
template <int NR, class Fin>
__device__ __forceinline__ void mp_finish(double (&acc)[NR], double* partial, unsigned* counter, Fin fin) {
  __shared__ double sw[MP_T / 32][NR];
  __shared__ int last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < NR; ++j) {
    double v = acc[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) sw[warp][j] = v;
  }
  __syncthreads();
  if (threadIdx.x < NR) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < MP_T / 32; ++w) t += sw[w][threadIdx.x];
    partial[(int64_t)blockIdx.x * NR + threadIdx.x] = t;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  __syncthreads();
  if (last) {
    __threadfence();
    if (threadIdx.x < NR) {
      double t = 0.0;
      for (unsigned b = 0; b < gridDim.x; ++b) t += ((volatile double*)partial)[(int64_t)b * NR + threadIdx.x];
      fin(threadIdx.x, t);
    }
    __syncthreads();
    if (threadIdx.x == 0) *counter = 0u;
  }
}

// MP_INIT:  what 0: sums B.B; 1: R = B, P = dinv R, sums R.P; 2: sums R.R (and the
//           first stopping test)
// MP_ALPHA: sums P.Q -> alpha, act = !done
// MP_XR:    X += alpha P, R -= alpha Q (active columns); sums R.R
// MP_RZ:    sums R.(dinv R) -> beta, rz, k, done
template <int NR, int OP>
__global__ void __launch_bounds__(MP_T)
mp_reduce_kernel(int64_t n, const double* __restrict__ B, const double* __restrict__ dinv, double* __restrict__ X,
                 double* __restrict__ R, double* __restrict__ P, const double* __restrict__ Q, MultiScal* sc,
                 double* partial, unsigned* counter, int what) {
  double acc[NR];
  double al[NR];
  bool on[NR];
#pragma unroll
  for (int j = 0; j < NR; ++j) {
    acc[j] = 0.0;
    al[j] = OP == MP_XR ? sc->alpha[j] : 0.0;
    on[j] = OP == MP_XR ? sc->act[j] != 0 : true;
  }
  for (int64_t i = blockIdx.x * (int64_t)MP_T + threadIdx.x; i < n; i += (int64_t)gridDim.x * MP_T) {
    const double di = dinv[i];
#pragma unroll
    for (int j = 0; j < NR; ++j) {
      const int64_t q = i * NR + j;
      if constexpr (OP == MP_INIT) {
        const double b = B[q];
        if (what == 1) {
          R[q] = b;
          P[q] = di * b;
          acc[j] += b * (di * b);
        } else {
          acc[j] += b * b;
        }
      } else if constexpr (OP == MP_ALPHA) {
        acc[j] += P[q] * Q[q];
      } else if constexpr (OP == MP_XR) {
        double r = R[q];
        if (on[j]) {
          X[q] += al[j] * P[q];
          r -= al[j] * Q[q];
          R[q] = r;
        }
        acc[j] += r * r;
      } else {
        const double r = R[q];
        acc[j] += r * (di * r);
      }
    }
  }
  mp_finish<NR>(acc, partial, counter, [&](int j, double t) {
    if constexpr (OP == MP_INIT) {
      if (what == 0) {
        sc->bb[j] = fmax(t, 1e-300);
      } else if (what == 1) {
        sc->rz[j] = t;
      } else {
        sc->rr[j] = t;
        sc->k[j] = 0;
        sc->done[j] = !(t > sc->tol2[j] && 0 < sc->maxiter);
      }
    } else if constexpr (OP == MP_ALPHA) {
      sc->act[j] = !sc->done[j];
      sc->alpha[j] = sc->act[j] ? sc->rz[j] / t : 0.0;
    } else if constexpr (OP == MP_XR) {
      if (sc->act[j]) sc->rr[j] = t;
    } else {
      if (sc->act[j]) {
        sc->beta[j] = t / sc->rz[j];
        sc->rz[j] = t;
        sc->k[j] += 1;
        sc->done[j] = !(sc->rr[j] > sc->tol2[j] && sc->k[j] < sc->maxiter);
      }
    }
  });
}

// P = dinv R + beta P on the columns active in this iteration
template <int NR>
__global__ void mp_update_p_kernel(int64_t n, const double* __restrict__ dinv, const double* __restrict__ R,
                                   double* __restrict__ P, const MultiScal* sc) {
  double be[NR];
  bool on[NR];
#pragma unroll
  for (int j = 0; j < NR; ++j) {
    be[j] = sc->beta[j];
    on[j] = sc->act[j] != 0;
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double di = dinv[i];
#pragma unroll
    for (int j = 0; j < NR; ++j)
      if (on[j]) P[i * NR + j] = di * R[i * NR + j] + be[j] * P[i * NR + j];
  }
}

__global__ void mp_scal_init_kernel(MultiScal* sc, int maxiter) {
  for (int j = 0; j < 16; ++j) {
    sc->rz[j] = sc->rr[j] = sc->bb[j] = sc->tol2[j] = sc->alpha[j] = sc->beta[j] = 0.0;
    sc->k[j] = 0;
    sc->done[j] = 1;
    sc->act[j] = 0;
  }
  sc->maxiter = maxiter;
  sc->loops = 0;
}

__global__ void mp_tol_kernel(MultiScal* sc, int nr, double tol) {
  for (int j = 0; j < nr; ++j) sc->tol2[j] = tol * tol * sc->bb[j];
}

// inverse diagonal of the reference's preconditioner: free ? 1 / (d != 0 ? d : 1) : 1
__global__ void mp_dinv_kernel(int64_t n, const double* __restrict__ d, const uint8_t* __restrict__ fixed,
                               double* __restrict__ dinv) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const bool fr = !(fixed && fixed[i]);
    dinv[i] = fr ? 1.0 / (fabs(d[i]) > 0.0 ? d[i] : 1.0) : 1.0;
  }
}

// loop condition: another pass while some column is active, at most maxiter + 2 passes
__global__ void mp_cond_kernel(cudaGraphConditionalHandle h, MultiScal* sc, int nr, int head) {
  if (head) sc->loops = 0;
  else sc->loops += 1;
  bool any = false;
  for (int j = 0; j < nr; ++j) any = any || !sc->done[j];
  cudaGraphSetConditional(h, (any && (long long)sc->loops <= (long long)sc->maxiter + 1) ? 1u : 0u);
}

template <int NR>
int mp_iteration(exfem_block_s* b, const double* Ke, const double* dinv, double* X, double* R, double* P, double* Q,
                 MultiScal* sc, double* partial, unsigned* counter, unsigned grid, cudaStream_t s) {
  const int64_t n = b->ndof();
  int st;
  if ((st = launch_ebe_matvec_multi(b, Ke, EXFEM_F64, NR, P, Q, true, s))) return st;
  mp_reduce_kernel<NR, MP_ALPHA><<<grid, MP_T, 0, s>>>(n, nullptr, dinv, X, R, P, Q, sc, partial, counter, 0);
  mp_reduce_kernel<NR, MP_XR><<<grid, MP_T, 0, s>>>(n, nullptr, dinv, X, R, P, Q, sc, partial, counter, 0);
  mp_reduce_kernel<NR, MP_RZ><<<grid, MP_T, 0, s>>>(n, nullptr, dinv, X, R, P, Q, sc, partial, counter, 0);
  mp_update_p_kernel<NR><<<grid_for(n, 256), 256, 0, s>>>(n, dinv, R, P, sc);
  EX_LAUNCH_CHECK();
  return EXFEM_OK;
}

template <int NR>
int mp_solve(exfem_block_s* b, const double* Ke, const double* Bm, double* X, double tol, int maxiter, int* iters,
             double* relres, cudaStream_t s) {
  const int64_t n = b->ndof();
  int st;
  // workspace: dinv (n), R, P, Q (n NR each), partial sums, scalars, counter
  // (every array starts on 256 bytes: the product reads P with 16-byte loads)
  DevBuf<double>& w = b->mp_work;
  const int64_t np = (n + 31) / 32 * 32;
  const size_t need = (size_t)np * (1 + 3 * NR) + (size_t)MP_MAX_BLOCKS * 16 + sizeof(MultiScal) / 8 + 64;
  if (w.n < need && (st = w.alloc(need))) return st;
  double* dinv = w.p;
  double* R = dinv + np;
  double* P = R + np * NR;
  double* Q = P + np * NR;
  double* partial = Q + np * NR;
  MultiScal* sc = reinterpret_cast<MultiScal*>(partial + MP_MAX_BLOCKS * 16);
  unsigned* counter = reinterpret_cast<unsigned*>(sc + 1);
  const unsigned grid =
      (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + MP_T * 4 - 1) / (MP_T * 4), MP_MAX_BLOCKS));
  // element rows of the product, allocated before the capture below
  const size_t nrows = (size_t)b->ne * b->nd * NR;
  if (b->ys_m64.n < nrows && (st = b->ys_m64.alloc(nrows))) return st;
  EX_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned), s));
  if ((st = launch_ebe_diagonal(b, Ke, Q, s))) return st;
  mp_dinv_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, Q, b->fixed.p, dinv);
  mp_scal_init_kernel<<<1, 1, 0, s>>>(sc, maxiter);
  EX_CUDA(cudaMemsetAsync(X, 0, sizeof(double) * n * NR, s));
  for (int what = 0; what < 3; ++what) {
    mp_reduce_kernel<NR, MP_INIT><<<grid, MP_T, 0, s>>>(n, Bm, dinv, X, R, P, nullptr, sc, partial, counter, what);
    if (what == 0) mp_tol_kernel<<<1, 1, 0, s>>>(sc, NR, tol);
  }
  EX_LAUNCH_CHECK();
  // the iteration loop as one graph: a conditional while node repeats one captured
  // iteration while some column is active
  cudaGraph_t g = nullptr;
  EX_CUDA(cudaGraphCreate(&g, 0));
  cudaGraphExec_t ge = nullptr;
  auto fail = [&](cudaError_t e, const char* what) {
    if (ge) cudaGraphExecDestroy(ge);
    cudaGraphDestroy(g);
    set_error("multi-case PCG graph: %s: %s", what, cudaGetErrorString(e));
    return EXFEM_ERR_CUDA;
  };
  cudaGraphConditionalHandle h;
  cudaError_t e = cudaGraphConditionalHandleCreate(&h, g, 0, 0);
  if (e != cudaSuccess) return fail(e, "condition handle");
  int nr = NR, head = 1;
  void* args[] = {&h, &sc, &nr, &head};
  cudaKernelNodeParams kp = {};
  kp.func = (void*)mp_cond_kernel;
  kp.gridDim = dim3(1);
  kp.blockDim = dim3(1);
  kp.kernelParams = args;
  cudaGraphNode_t n_head, n_loop;
  if ((e = cudaGraphAddKernelNode(&n_head, g, nullptr, 0, &kp)) != cudaSuccess) return fail(e, "head node");
  cudaGraphNodeParams cp = {};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  if ((e = cudaGraphAddNode(&n_loop, g, &n_head, 1, &cp)) != cudaSuccess) return fail(e, "while node");
  {
    CaptureScope cap;
    if ((e = cudaStreamBeginCaptureToGraph(s, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                           cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
      return fail(e, "capture of the loop body");
    int cs = mp_iteration<NR>(b, Ke, dinv, X, R, P, Q, sc, partial, counter, grid, s);
    if (!cs) {
      mp_cond_kernel<<<1, 1, 0, s>>>(h, sc, NR, 0);
      if (cudaGetLastError() != cudaSuccess) cs = EXFEM_ERR_CUDA;
    }
    cudaGraph_t captured = nullptr;
    e = cudaStreamEndCapture(s, &captured);
    if (cs) {
      cudaGraphDestroy(g);
      return cs;
    }
    if (e != cudaSuccess) return fail(e, "end of the body capture");
  }
  if ((e = cudaGraphInstantiate(&ge, g, 0)) != cudaSuccess) return fail(e, "instantiation");
  if ((e = cudaGraphLaunch(ge, s)) != cudaSuccess) return fail(e, "launch");
  MultiScal hs;
  e = cudaMemcpyAsync(&hs, sc, sizeof(MultiScal), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaGraphExecDestroy(ge);
  cudaGraphDestroy(g);
  EX_CUDA(e);
  bool all = true;
  for (int j = 0; j < NR; ++j) {
    const double rel = std::sqrt(hs.rr[j] / hs.bb[j]);
    if (iters) iters[j] = hs.k[j];
    if (relres) relres[j] = rel;
    all = all && std::isfinite(rel) && hs.rr[j] <= hs.tol2[j];
  }
  return all ? EXFEM_OK : EXFEM_NOT_CONVERGED;
}

}  // namespace

int multi_pcg(exfem_block_s* b, const double* Ke, int nrhs, const double* B, double* X, double tol, int maxiter,
              int* iters, double* relres, cudaStream_t s) {
  switch (nrhs) {
    case 1: return mp_solve<1>(b, Ke, B, X, tol, maxiter, iters, relres, s);
    case 2: return mp_solve<2>(b, Ke, B, X, tol, maxiter, iters, relres, s);
    case 3: return mp_solve<3>(b, Ke, B, X, tol, maxiter, iters, relres, s);
    case 4: return mp_solve<4>(b, Ke, B, X, tol, maxiter, iters, relres, s);
    case 8: return mp_solve<8>(b, Ke, B, X, tol, maxiter, iters, relres, s);
    case 16: return mp_solve<16>(b, Ke, B, X, tol, maxiter, iters, relres, s);
    default:
      set_error("the multi-case PCG takes 1, 2, 3, 4, 8 or 16 load cases per call, got %d", nrhs);
      return EXFEM_ERR_ARG;
  }
}

}  // namespace exfem
