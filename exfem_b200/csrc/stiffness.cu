// Element tangents Ke = sum_g vol_g G_g^T C_g G_g (gfem/model.py:70-111, 479-483) and
// their diagonals, FP64 arithmetic, stored as FP64, FP32 or BF16.
//
// With g_a the gradient of shape function a at a Gauss point, the stress of a unit
// displacement of node b along k under the (consistent) tangent
//   C = K I (x) I + 2 mu c1 dev + c2 n (x) n
// contracts with the strain of a unit displacement of node a along i to
//   Ke[ai, bk] = delta_ik tr P_ab + P_ab[k][i] - 2/3 P_ab[i][k] + R_ab[i][k],
//   P_ab[i][k] = sum_g vol mu c1 g_a[i] g_b[k],
//   R_ab[i][k] = sum_g vol c2 m_a[i] m_b[k] + (volumetric part),  m_a = n g_a,
// where the volumetric part is sum_g vol K g_a[i] g_b[k] (C3D10) or, under B-bar
// (C3D8), (sum_g vol) K g0_a[i] g0_b[k] with g0 the gradients at the centre, and m_a
// has the B-bar correction (g0_a - g_a) tr n / 3.  P and R are Gram matrices of the
// element's gradients over its 4 or 8 Gauss points: a contraction, done with the
// FP64 matrix instruction.  For every pair of components (i, k) one 8 x 8 tile over
// the node pairs (a, b) is accumulated (two node tiles per side for ten nodes), so
// that P_ab[i][k] and P_ab[k][i] sit in the same lane and Ke follows without any
// exchange; the lane that holds row a and columns b, b+1 has six consecutive entries
// of three rows of Ke.
#include <cuda_bf16.h>

#include "gauss_warp.cuh"
#include "internal.h"

namespace exfem {

namespace {

// store two consecutive entries of Ke
__device__ __forceinline__ void put2(double* p, double a, double b) { *reinterpret_cast<double2*>(p) = make_double2(a, b); }
__device__ __forceinline__ void put2(float* p, double a, double b) {
  *reinterpret_cast<float2*>(p) = make_float2((float)a, (float)b);
}
__device__ __forceinline__ void put2(__nv_bfloat16* p, double a, double b) {
  *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn((float)a, (float)b);
}

// shared memory of one warp
template <int ET, bool J2, int MODE, class OutT>
struct StiffSmem {
  using Tr = ElemTraits<ET>;
  static constexpr int NN = Tr::nnode, NG = Tr::ngp, ND = 3 * NN, EPW = 32 / NG;
  union {                  // node values (first part), then the matrix being put together
    alignas(16) OutT stage[MODE == 0 ? ND * ND : 8];
    struct {
      NodeSmem<ET, J2> nd;
      double st[J2 ? 32 * 19 : 1];  // Gauss-point states: the lanes' odd stride of 19 meets no bank conflict
    };
  };
  double iJ[9][32];        // inverse Jacobian of Gauss point `lane`
  double vol[32];          // weighted volume
  double al[32], be[32];   // vol mu c1, vol c2
  double n[J2 ? 6 : 1][32];
  double iJ0[ET == EXFEM_C3D8 ? 9 : 1][EPW];
};

// One warp takes EPW = 32 / ngp elements: first one lane per Gauss point evaluates
// the inverse Jacobian, volume and material tangent into the warp's shared memory
// (node values read once per element, broadcast), then the warp forms the elements'
// matrices one after the other on the matrix unit.  Each Ke is put together in
// shared memory and leaves as one bulk store, so that global memory sees whole lines.
// MODE 1 writes the diagonal entries only.
//
// Measured on B200: 40,000 J2 C3D8 (184 MB of Ke) 64 us, 72,450 C3D10 (522 MB) 109 us
// = 0.73 of the copy bandwidth; one thread per node, which formed every gradient again
// for each node pair and stored single entries, took 1,273 and 1,418 us.  C3D10 is
// bound by the stores; C3D8 by the latency of the material phase at 12 warps an SM:
// four blocks' worth of registers (128 a thread) spill there and take 88 us, two take
// 94 us; the elastic kernels fit four without spills (C3D10: 115 us at two or three).
template <int ET, bool J2, int MODE, class OutT, int NW>
__global__ void __launch_bounds__(32 * NW, J2 ? 3 : 4)
stiffness_kernel(int64_t ne, const double* __restrict__ X, const int32_t* __restrict__ conn,
                 const double* __restrict__ u, const double* __restrict__ scale, const double* __restrict__ st_old,
                 const double* __restrict__ tan_in, const __grid_constant__ MatDev mat,
                 const double* __restrict__ lam_e, const double* __restrict__ mu_e, OutT* __restrict__ Ke,
                 double* __restrict__ ediag, const int32_t* __restrict__ tpos, int tile, int bulk) {
  using S = StiffSmem<ET, J2, MODE, OutT>;
  constexpr int NN = S::NN, NG = S::NG, ND = S::ND, EPW = S::EPW, XS = DnTable<ET>::XS;
  constexpr int NT = NN > 8 ? 2 : 1, KS = NG / 4;  // node tiles per side, matrix steps over the Gauss points
  constexpr bool BBAR = ET == EXFEM_C3D8;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double* tab = reinterpret_cast<double*>(smem_raw);  // dN_b / dxi_i at every Gauss point, rows of XS
  constexpr int TAB = (NG * XS + 15) / 16 * 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  S& sm = reinterpret_cast<S*>(tab + TAB)[warp];
  for (int k = threadIdx.x; k < NG * XS; k += 32 * NW) tab[k] = dn_table<ET>()[k];
  __syncthreads();
  const int row = lane >> 2, q = lane & 3;  // this lane's row and Gauss point (matrix A), or column pair (C)
  double dNl[KS][NT][3];
#pragma unroll
  for (int s = 0; s < KS; ++s)
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int a = 8 * t + row;
        dNl[s][t][i] = a < NN ? tab[(4 * s + q) * XS + 3 * a + i] : 0.0;
      }
  const int64_t e0 = ((int64_t)blockIdx.x * NW + warp) * EPW;
  if (e0 >= ne) return;
  const int cnt = ne - e0 < EPW ? (int)(ne - e0) : EPW;

  // ---- Gauss-point states and node values of the warp's elements
  if (J2 && !tan_in && st_old) {
    for (int k = lane; k < cnt * NG * 19; k += 32) cp_async<8>(sm.st + k, st_old + e0 * (NG * 19) + k, 8);
  }
  const int le = lane / NG, g = lane % NG;
  gather_nodes<ET, J2>(sm.nd, X, conn, u, nullptr, e0 + (le < cnt ? le : 0), cnt, [&](int el) { return e0 + el; },
                       [] {});
  if constexpr (J2) cp_async_wait_all();
  __syncwarp();

  // ---- one lane per Gauss point: geometry and material
  bool plastic = false;
  if (le < cnt) {
    const int64_t e = e0 + le;
    const bool own = lam_e != nullptr;  // per-element Lame parameters override the material's
    const double lam_k = own ? lam_e[e] : mat.lam, mu_k = own ? mu_e[e] : mat.mu;
    double J[9], G[9], J0[9], G0[9], iJ[9], iJ0[9];
    gauss_gradients<ET, J2>(sm.nd, tab, le, g, J, G, J0, G0);
    const double detJ = inv3(J, iJ);
    if constexpr (BBAR) {
      inv3(J0, iJ0);
      if (g == 0)
#pragma unroll
        for (int k = 0; k < 9; ++k) sm.iJ0[k][le] = iJ0[k];
    }
    double tn[8] = {0, 0, 0, 0, 0, 0, 1.0, 0.0};
    if constexpr (J2) {
      if (tan_in) {
        const int64_t tp = tpos[e];
#pragma unroll
        for (int k = 0; k < 8; ++k) tn[k] = tan_in[tile_index(tp, g * 8 + k, NG * 8, tile)];
      } else {
        double H[9], sig[6], st[19];
        matmul3(G, iJ, H);
        if constexpr (BBAR) {
          double tr0 = 0.0;
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int i = 0; i < 3; ++i) tr0 += G0[3 * c + i] * iJ0[3 * i + c];
          const double bb = (tr0 - (H[0] + H[4] + H[8])) * (1.0 / 3.0);
          H[0] += bb;
          H[4] += bb;
          H[8] += bb;
        }
#pragma unroll
        for (int k = 0; k < 19; ++k) st[k] = st_old ? sm.st[lane * 19 + k] : 0.0;
        material_stress(mat, lam_k, mu_k, H, st, nullptr, sig, tn);
      }
    }
    const double vol = (ET == EXFEM_C3D8 ? 1.0 : 1.0 / 24.0) * detJ * (scale ? scale[e] : 1.0);
#pragma unroll
    for (int k = 0; k < 9; ++k) sm.iJ[k][lane] = iJ[k];
    sm.vol[lane] = vol;
    sm.al[lane] = vol * mu_k * tn[6];
    if constexpr (J2) {
      sm.be[lane] = vol * tn[7];
#pragma unroll
      for (int k = 0; k < 6; ++k) sm.n[k][lane] = tn[k];
      plastic = !(tn[6] == 1.0 && tn[7] == 0.0);
    }
  }
  const unsigned pl = J2 ? __ballot_sync(0xffffffffu, plastic) : 0u;
  __syncwarp();

  // ---- the warp's elements one after the other
  for (int w = 0; w < cnt; ++w) {
    const int64_t e = e0 + w;
    const bool own = lam_e != nullptr;
    const double mu_k = own ? mu_e[e] : mat.mu;
    const double Kb = own ? lam_e[e] + 2.0 * mu_k / 3.0 : mat.K;
    const bool full = J2 && ((pl >> (w * NG)) & ((1u << NG) - 1u)) != 0;  // some Gauss point is plastic
    double ga[KS][NT][3], al[KS], ma[KS][NT][3], be[KS], ga0[3], vsum = 0.0;
    if constexpr (BBAR) {
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) s += hex_sign(row, i) > 0 ? sm.iJ0[3 * i + j][w] : -sm.iJ0[3 * i + j][w];
        ga0[j] = 0.125 * s;
      }
#pragma unroll
      for (int p = 0; p < NG; ++p) vsum += sm.vol[w * NG + p];
    }
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      const int p = w * NG + 4 * s + q;
      double iJ[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) iJ[k] = sm.iJ[k][p];
      al[s] = sm.al[p];
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          ga[s][t][j] = dNl[s][t][0] * iJ[j] + dNl[s][t][1] * iJ[3 + j] + dNl[s][t][2] * iJ[6 + j];
      if (full) {
        double n[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) n[k] = sm.n[J2 ? k : 0][p];
        be[s] = sm.be[p];
        const double tr3 = (n[0] + n[1] + n[2]) * (1.0 / 3.0);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const double(&x)[3] = ga[s][t];
          ma[s][t][0] = n[0] * x[0] + n[3] * x[1] + n[5] * x[2];
          ma[s][t][1] = n[3] * x[0] + n[1] * x[1] + n[4] * x[2];
          ma[s][t][2] = n[5] * x[0] + n[4] * x[1] + n[2] * x[2];
          if constexpr (BBAR)
#pragma unroll
            for (int j = 0; j < 3; ++j) ma[s][t][j] += (ga0[j] - x[j]) * tr3;
        }
      }
    }
    if constexpr (MODE == 1) {
      // diagonal entries: sums over this lane's Gauss points, then over the four
      // lanes that share the row
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        double d[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          const double(&x)[3] = ga[s][t];
          const double xx = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
          const double kv = BBAR ? 0.0 : sm.vol[w * NG + 4 * s + q] * Kb;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            d[k] += al[s] * (xx + x[k] * x[k] / 3.0) + kv * x[k] * x[k];
            if (full) d[k] += be[s] * ma[s][t][k] * ma[s][t][k];
          }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          d[k] += __shfl_xor_sync(0xffffffffu, d[k], 1);
          d[k] += __shfl_xor_sync(0xffffffffu, d[k], 2);
          if constexpr (BBAR) d[k] += Kb * vsum * ga0[k] * ga0[k];
        }
        const int a = 8 * t + row;
        if (a < NN && q < 3) ediag[(e * NN + a) * 3 + q] = q == 0 ? d[0] : (q == 1 ? d[1] : d[2]);
      }
      continue;
    }
    OutT* stage = sm.stage;
#pragma unroll
    for (int ta = 0; ta < NT; ++ta)
#pragma unroll
      for (int tb = 0; tb < NT; ++tb) {
        double P[3][3][2], R[3][3][2];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int k = 0; k < 3; ++k) P[i][k][0] = P[i][k][1] = R[i][k][0] = R[i][k][1] = 0.0;
#pragma unroll
        for (int s = 0; s < KS; ++s)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const double a = al[s] * ga[s][ta][i];
#pragma unroll
            for (int k = 0; k < 3; ++k) dmma(P[i][k], a, ga[s][tb][k]);
          }
        if (full) {
#pragma unroll
          for (int s = 0; s < KS; ++s) {
            const double kg = BBAR ? 0.0 : sm.vol[w * NG + 4 * s + q] * Kb;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              const double a = be[s] * ma[s][ta][i];
#pragma unroll
              for (int k = 0; k < 3; ++k) dmma(R[i][k], a, ma[s][tb][k]);
              if constexpr (!BBAR) {
                const double v = kg * ga[s][ta][i];
#pragma unroll
                for (int k = 0; k < 3; ++k) dmma(R[i][k], v, ga[s][tb][k]);
              }
            }
          }
        }
        // C3D10 without plastic points: one modulus for all of them, R = (K / mu) P
        const double rp = BBAR || full ? 0.0 : Kb / mu_k;
        const int a = 8 * ta + row, b0 = 8 * tb + 2 * q;
        double g0b[2][3];
        if constexpr (BBAR)
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int k = 0; k < 3; ++k) g0b[c][k] = __shfl_sync(0xffffffffu, ga0[k], 4 * (2 * q + c));
        if (bulk && ta == 0 && tb == 0) {  // the previous element's bulk store has read the buffer
          if (lane == 0) bulk_wait_read<0>();
          __syncwarp();
        }
        if (a < NN && b0 < NN) {
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            double o[6];
            const double ka = BBAR ? Kb * vsum * ga0[i] : 0.0;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const double tr = P[0][0][c] + P[1][1][c] + P[2][2][c];
#pragma unroll
              for (int k = 0; k < 3; ++k) {
                double v = P[k][i][c] - (2.0 / 3.0) * P[i][k][c] + (i == k ? tr : 0.0);
                if constexpr (BBAR) v += ka * g0b[c][k] + R[i][k][c];
                else v += R[i][k][c] + rp * P[i][k][c];
                o[3 * c + k] = v;
              }
            }
            OutT* d = stage + (3 * a + i) * ND + 3 * b0;
#pragma unroll
            for (int c = 0; c < 3; ++c) put2(d + 2 * c, o[2 * c], o[2 * c + 1]);
          }
        }
      }
    if (bulk) {
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        bulk_s2g(Ke + e * (ND * ND), stage, ND * ND * (uint32_t)sizeof(OutT));
        bulk_commit();
      }
    } else {  // matrices that are no multiple of 16 bytes, or start off a 16-byte boundary
      __syncwarp();
      for (int k = lane; k < ND * ND; k += 32) Ke[e * (ND * ND) + k] = stage[k];
      __syncwarp();
    }
  }
  if (MODE == 0 && bulk && lane == 0) bulk_wait_read<0>();
}

template <int ET, bool J2, int MODE, class OutT>
int stiffness_go(exfem_block_s* b, const double* u, const double* st_old, const double* tan_in, OutT* Ke,
                 double* ediag, cudaStream_t s) {
  using S = StiffSmem<ET, J2, MODE, OutT>;
  constexpr int NW = 4;
  constexpr size_t smem = (size_t)((S::NG * DnTable<ET>::XS + 15) / 16 * 16) * sizeof(double) + NW * sizeof(S);
  auto kern = stiffness_kernel<ET, J2, MODE, OutT, NW>;
  if constexpr (smem > 48 * 1024)
    EX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // No preferred split of the on-chip memory is set: a launch that wants another split than
  // the running kernels' waits for them to leave, and under other streams' solves (device
  // loops) that is the end of their backlog.  J2 Newton corrections take their diagonal
  // from here: mean J2 service at 2,000 requests/s on 24 streams 20 s with the preference,
  // 2.4 s without.  Alone the kernel is no slower (40,000 J2 C3D8: 65.5 and 63.5 us).
  constexpr size_t bytes = (size_t)S::ND * S::ND * sizeof(OutT);
  const int bulk = MODE == 0 && bytes % 16 == 0 && (uintptr_t)Ke % 16 == 0;
  const int64_t per = NW * S::EPW;
  kern<<<(unsigned)((b->ne + per - 1) / per), 32 * NW, smem, s>>>(b->ne, b->X.p, b->conn.p, u, b->scale.p, st_old,
                                                                   tan_in, b->mat, b->lam_e.p, b->mu_e.p, Ke, ediag,
                                                                   b->tpos.p, b->tile, bulk);
  EX_LAUNCH_CHECK();
  return EXFEM_OK;
}

template <int ET, class OutT>
int stiffness_et(exfem_block_s* b, const double* u, const double* st_old, const double* tan_in, OutT* Ke,
                 double* ediag, cudaStream_t s) {
  const bool j2 = b->mat.kind == EXFEM_J2;
  if constexpr (sizeof(OutT) == 8) {
    if (ediag)
      return j2 ? stiffness_go<ET, true, 1, double>(b, u, st_old, tan_in, Ke, ediag, s)
                : stiffness_go<ET, false, 1, double>(b, u, st_old, tan_in, Ke, ediag, s);
  }
  return j2 ? stiffness_go<ET, true, 0, OutT>(b, u, st_old, tan_in, Ke, nullptr, s)
            : stiffness_go<ET, false, 0, OutT>(b, u, st_old, tan_in, Ke, nullptr, s);
}

template <class OutT>
int stiffness_out(exfem_block_s* b, const double* u, const double* st_old, const double* tan_in, void* Ke,
                  double* ediag, cudaStream_t s) {
  return b->etype == EXFEM_C3D8 ? stiffness_et<EXFEM_C3D8, OutT>(b, u, st_old, tan_in, (OutT*)Ke, ediag, s)
                                : stiffness_et<EXFEM_C3D10, OutT>(b, u, st_old, tan_in, (OutT*)Ke, ediag, s);
}

}  // namespace

// Ke (FP64, FP32 or BF16), or with `ediag` its diagonal entries (ne, nnode, 3).  The
// J2 tangent data come from u and st_old, or from `tan_in` (the stored tangent).
int launch_stiffness(exfem_block_s* b, const double* u, const double* st_old, int dtype, void* Ke, double* ediag,
                     cudaStream_t s, const double* tan_in) {
  if (b->ne == 0) return EXFEM_OK;
  if (dtype == EXFEM_F64) return stiffness_out<double>(b, u, st_old, tan_in, Ke, ediag, s);
  if (dtype == EXFEM_F32) return stiffness_out<float>(b, u, st_old, tan_in, Ke, ediag, s);
  if (dtype == EXFEM_BF16) return stiffness_out<__nv_bfloat16>(b, u, st_old, tan_in, Ke, ediag, s);
  set_error("unsupported Ke dtype %d", dtype);
  return EXFEM_ERR_ARG;
}

}  // namespace exfem
