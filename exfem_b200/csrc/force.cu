// FP64 internal force with the J2 return map and the consistent-tangent data it
// produces, the tangent data alone, element-averaged stresses, and the element vectors
// of the FP64 tangent product (gfem/model.py:35-81, 129-137, 466-490).
//
// One warp takes 32 / ngp elements (4 C3D8, 8 C3D10), one lane per Gauss point (elastic
// stresses and the elastic forces of larger C3D8 meshes one thread per element:
// elastic_kernel).  Node values are gathered once per element and Gauss-point states in
// whole lines into the warp's shared memory; a lane evaluates its point's kinematics and
// material; the element forces
//   f_a = sum_g sum_i dN_a/dxi_i(g) Q_g[:, i],  Q_g = vol sigma J^-T,
// are one small product of the constant dN table with the Q of all the warp's elements
// side by side, done with the FP64 matrix instruction, which also sums over the lanes;
// under B-bar (C3D8) the mean stress acts through the gradients at the centre, three
// more rows of the same product.  New states and forces leave in whole lines.
//
// J2 blocks are walked in tile order, in which the tangent data of neighbouring
// elements are neighbours in memory; otherwise elements are taken as they are numbered.
//
// Measured on B200, with the assembly: 40,000 J2 C3D8 49 us, 125,550 J2 C3D10 88 us
// (states read and written, tangent data written); one thread per element, which read
// each state entry with a stride of a whole element, took 170 and 212 us, and copying
// states entry by entry instead of in bulk 63 and 104 us.
#include "gauss_warp.cuh"
#include "internal.h"

namespace exfem {

namespace {

enum BulkArrays { BULK_OLD = 1, BULK_NEW = 2, BULK_FE = 4 };

// shared memory of one warp
template <int ET, bool J2>
struct ForceSmem {
  using Tr = ElemTraits<ET>;
  static constexpr int NN = Tr::nnode, NG = Tr::ngp, ND = 3 * NN, EPW = 32 / NG, ST = NG * 19;
  static constexpr bool BBAR = ET == EXFEM_C3D8;
  alignas(16) double st[J2 ? 32 * 19 : 2];  // Gauss-point states: the lanes' stride of 19 meets no bank conflict
  union {                                   // node values, then Q of every Gauss point, then element forces
    NodeSmem<ET, true> nd;
    double Q[9][33];  // odd stride for the gathers of the matrix product
    alignas(16) double F[EPW * ND];
  };
  double c0[BBAR ? EPW : 1][9];  // mean stress times the inverse Jacobian of the centre
  uint64_t bar;                  // arrival of the states
};

// an element's stress output from the volume sums of its points (any of S, mises, peeq may
// be NULL)
template <int N>
__device__ __forceinline__ void store_stress(int64_t e, const double (&sum)[N], double vol, double vol_alpha,
                                             double* __restrict__ S, double* __restrict__ mises,
                                             double* __restrict__ peeq) {
  double s[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) s[k] = sum[k] / vol;
  if (S) {
    double* o = S + e * 9;
    o[0] = s[0]; o[1] = s[3]; o[2] = s[5];
    o[3] = s[3]; o[4] = s[1]; o[5] = s[4];
    o[6] = s[5]; o[7] = s[4]; o[8] = s[2];
  }
  const double m3 = (s[0] + s[1] + s[2]) / 3.0;
  const double d0 = s[0] - m3, d1 = s[1] - m3, d2 = s[2] - m3;
  if (mises)
    mises[e] = sqrt(1.5 * (d0 * d0 + d1 * d1 + d2 * d2 + 2.0 * (s[3] * s[3] + s[4] * s[4] + s[5] * s[5])));
  if (peeq) peeq[e] = vol_alpha / vol;
}

// warps an SM holds: the products need few enough registers for 20 (with the node sums, 16
// and 20 warps: 116,000 C3D8 55.2 / 53.2 us, 329,232 C3D10 125 / 116), except the J2 C3D8's,
// which spill (116,000 elements 73.4 / 76.7)
template <int ET, bool J2, int MODE>
constexpr int force_warps() {
  return MODE == FORCE_PRODUCT && !(J2 && ET == EXFEM_C3D8) ? 20 : 16;
}

template <int ET, bool J2, int MODE, int NW>
__global__ void __launch_bounds__(32 * NW, force_warps<ET, J2, MODE>() / NW)
force_kernel(int64_t ne, const double* __restrict__ X, const int32_t* __restrict__ conn,
             const double* u, const double* __restrict__ scale, const double* st_old, double* st_new,
             double* fe, double* tan64, float* __restrict__ tan32, double* __restrict__ S,
             double* __restrict__ mises, double* __restrict__ peeq, const __grid_constant__ MatDev mat,
             const double* __restrict__ lam_e, const double* __restrict__ mu_e, const int32_t* __restrict__ order,
             int tile_log2, int bulk, int* __restrict__ err, const uint8_t* __restrict__ nf,
             const int* skip) {
  using SM = ForceSmem<ET, J2 && MODE != FORCE_PRODUCT>;
  constexpr int NN = SM::NN, NG = SM::NG, ND = SM::ND, EPW = SM::EPW, ST = SM::ST, XS = DnTable<ET>::XS;
  constexpr bool BBAR = SM::BBAR;
  constexpr bool TILED = J2 && MODE != FORCE_STRESS;  // walked in tile order
  constexpr bool PRODUCT = MODE == FORCE_PRODUCT, OUT = MODE == FORCE_FULL || PRODUCT, STATES = J2 && !PRODUCT;
  constexpr int MT = NN > 8 ? 2 : 1, NTC = (3 * EPW + 7) / 8, KS = NG * 3 / 4 + (BBAR ? 1 : 0);
  if (PRODUCT && skip) {
    chain_wait();
    if (*skip) return;
  }
  __shared__ __align__(16) double tab[NG * XS];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  SM& sm = reinterpret_cast<SM*>(smem_raw)[warp];
  for (int k = threadIdx.x; k < NG * XS; k += 32 * NW) tab[k] = dn_table<ET>()[k];
  __syncthreads();
  const int64_t p0 = ((int64_t)blockIdx.x * NW + warp) * EPW;
  if (p0 >= ne) return;
  const int cnt = ne - p0 < EPW ? (int)(ne - p0) : EPW;
  const int le = lane / NG, g = lane % NG;
  const bool valid = le < cnt;
  const int64_t pos = p0 + (valid ? le : 0);
  const int32_t eid = TILED ? order[pos] : (int32_t)pos;  // this lane's element
  // element of the warp's el-th position, on every lane
  auto elem = [&](int el) { return TILED ? (int64_t)__shfl_sync(0xffffffffu, eid, el * NG) : p0 + el; };

  // ---- states (whole elements, one bulk copy each) and node values
  if (STATES && st_old) {
    if (bulk & BULK_OLD) {
      if (lane == 0) {
        mbar_init(&sm.bar, 1);
        fence_mbar_init();
        mbar_expect_tx(&sm.bar, cnt * ST * (uint32_t)sizeof(double));
      }
      __syncwarp();
      if (valid && g == 0)
        bulk_g2s(sm.st + le * ST, st_old + (int64_t)eid * ST, ST * (uint32_t)sizeof(double), &sm.bar);
    } else {
      for (int k0 = 0; k0 < 32 * 19; k0 += 32) {
        const int k = k0 + lane, el = k / ST;
        const int64_t e = elem(el);
        if (el < cnt) cp_async<8>(sm.st + k, st_old + e * ST + (k - el * ST), 8);
      }
    }
  }
  gather_nodes<ET, true>(sm.nd, X, conn, u, nf, eid, cnt, elem, [&] {
    if (PRODUCT && !skip) chain_wait();  // products are chained launches: u is the vector of the one ahead
  });
  // tile_index(pos, 8 g + k, 8 ngp, tile) for a power of two
  const int64_t tan0 =
      TILED ? (((pos >> tile_log2) * (NG * 8) + g * 8) << tile_log2) + (pos & ((1 << tile_log2) - 1)) : 0;
  double tn[8];
  if constexpr (J2 && PRODUCT) {
#pragma unroll
    for (int k = 0; k < 8; ++k) tn[k] = tan64[tan0 + (k << tile_log2)];
  }
  __syncwarp();

  // ---- this lane's Gauss point
  const double lam_k = lam_e ? lam_e[eid] : mat.lam, mu_k = lam_e ? mu_e[eid] : mat.mu;
  double J[9], G[9], J0[9], G0[9], iJ[9], iJ0[9], H[9];
  gauss_gradients<ET, true>(sm.nd, tab, le, g, J, G, J0, G0);
  const double detJ = inv3(J, iJ);
  matmul3(G, iJ, H);
  if constexpr (BBAR) {
    inv3(J0, iJ0);
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
  double sig[6], alpha = 0.0;
  if constexpr (J2 && PRODUCT) {
    double e[6];
    sym_from_grad(H, e);
    tangent_stress(mat.K, mat.mu, tn, e, sig);
  } else if constexpr (J2) {
    double* st = sm.st + lane * 19;
    if (!st_old) {
#pragma unroll
      for (int k = 0; k < 19; ++k) st[k] = 0.0;
    } else if (bulk & BULK_OLD) {
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&sm.bar, 0, err))) return;
    } else {
      cp_async_wait_all();
      __syncwarp();
    }
    double e[6], sn[19];
    sym_from_grad(H, e);
    j2_return(mat, e, st, MODE == FORCE_TANGENT ? nullptr : sn, sig, tn);
    alpha = sn[9];
    if (MODE == FORCE_FULL)
#pragma unroll
      for (int k = 0; k < 19; ++k) st[k] = sn[k];
  } else {
    double e[6];
    sym_from_grad(H, e);
    elastic_stress(lam_k, mu_k, e, sig);
    if (MODE == FORCE_FULL && st_new && valid)
      st_new[(int64_t)eid * NG + g] = st_old ? st_old[(int64_t)eid * NG + g] : 0.0;
  }
  const double vol = (BBAR ? 1.0 : 1.0 / 24.0) * detJ * (MODE != FORCE_STRESS && scale ? scale[eid] : 1.0);

  if constexpr (TILED && !PRODUCT) {
    if (valid) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int64_t o = tan0 + (k << tile_log2);
        tan64[o] = tn[k];
        tan32[o] = (float)tn[k];
      }
    }
  }

  if constexpr (MODE == FORCE_STRESS) {
    // volume averages over the element's lanes
    double a[8];
#pragma unroll
    for (int k = 0; k < 6; ++k) a[k] = vol * sig[k];
    a[6] = vol;
    a[7] = vol * alpha;
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int o = NG / 2; o > 0; o >>= 1) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
    if (valid && g == 0) {
      store_stress(eid, a, a[6], a[7], S, mises, peeq);
    }
  }

  if constexpr (OUT) {
    // Q = vol sigma J^-T; under B-bar the deviatoric part, and the mean stress of the
    // element times the gradients at its centre
    double t = 0.0;
    if constexpr (BBAR) {
      t = vol * (sig[0] + sig[1] + sig[2]) * (1.0 / 3.0);
      double tacc = t;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) tacc += __shfl_xor_sync(0xffffffffu, tacc, o);
      if (g == 0)
#pragma unroll
        for (int k = 0; k < 9; ++k) sm.c0[le][k] = tacc * iJ0[k];
    }
    const double r[3][3] = {{vol * sig[0] - t, vol * sig[3], vol * sig[5]},
                            {vol * sig[3], vol * sig[1] - t, vol * sig[4]},
                            {vol * sig[5], vol * sig[4], vol * sig[2] - t}};
    __syncwarp();  // node values read by every lane; new states in place
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int i = 0; i < 3; ++i)
        sm.Q[3 * c + i][lane] = r[c][0] * iJ[3 * i] + r[c][1] * iJ[3 * i + 1] + r[c][2] * iJ[3 * i + 2];
    if (STATES && st_new) {
      if (bulk & BULK_NEW) {
        fence_proxy_async();
        __syncwarp();
        if (valid && g == 0) {
          bulk_s2g(st_new + (int64_t)eid * ST, sm.st + le * ST, ST * (uint32_t)sizeof(double));
          bulk_commit();
        }
      } else {
        for (int k0 = 0; k0 < 32 * 19; k0 += 32) {
          const int k = k0 + lane, el = k / ST;
          const int64_t e = elem(el);
          if (el < cnt) st_new[e * ST + (k - el * ST)] = sm.st[k];
        }
      }
    }
    __syncwarp();
    const int row = lane >> 2, q = lane & 3;
    double f[MT][NTC][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NTC; ++n) f[m][n][0] = f[m][n][1] = 0.0;
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      const bool centre = BBAR && s == KS - 1;  // k: the three rows of the centre, one empty
      const int kk = 4 * s + q, gk = kk / 3, i = centre ? q : kk % 3;
      double a[MT], b[NTC];
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const int node = 8 * m + row;
        if (centre) a[m] = q < 3 ? 0.125 * hex_sign(node & 7, q) : 0.0;
        else a[m] = node < NN ? tab[gk * XS + 3 * node + i] : 0.0;
      }
#pragma unroll
      for (int n = 0; n < NTC; ++n) {
        const int col = 8 * n + row, el = col / 3, c = col % 3;
        if (centre) b[n] = q < 3 && el < EPW ? sm.c0[el < EPW ? el : 0][3 * i + c] : 0.0;
        else b[n] = el < EPW ? sm.Q[3 * c + i][el * NG + gk] : 0.0;
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NTC; ++n) dmma(f[m][n], a[m], b[n]);
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NTC; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int node = 8 * m + row, col = 8 * n + 2 * q + h;
          if (node < NN && col < 3 * EPW) sm.F[(col / 3) * ND + 3 * node + col % 3] = f[m][n][h];
        }
    if (bulk & BULK_FE) {
      fence_proxy_async();
      __syncwarp();
      if (valid && g == 0) {
        bulk_s2g(fe + (int64_t)eid * ND, sm.F + le * ND, ND * (uint32_t)sizeof(double));
        bulk_commit();
      }
    } else {
      __syncwarp();
      for (int k0 = 0; k0 < EPW * ND; k0 += 32) {
        const int k = k0 + lane, el = k / ND < EPW ? k / ND : EPW - 1;
        const int64_t e = elem(el);
        if (k < cnt * ND) fe[e * ND + (k - el * ND)] = sm.F[k];
      }
    }
    bulk_wait_read<0>();  // shared memory stays until the copies have read it
  }
}

// Elastic stresses, and elastic forces of C3D8 meshes that fill the chip: one thread per
// element.  An elastic point has no state and little arithmetic, so the warp's transforms,
// node values in shared memory and sums over an element's points are most of force_kernel's
// time there; a thread that takes its element's points one after the other has none of them.
// B200, us a call, warp / thread: stresses 40,000 C3D8 16.7 / 12.5, 432,000 142 / 58, 125,550
// C3D10 37 / 23, 1,080,000 316 / 156 (equal up to some 10,000 elements, where a call is
// its launch); C3D8 forces with the node sums 40,000 24.5 / 20.7, 128,000 63 / 41, 432,000
// 218 / 129.
template <int ET, int MODE>
__global__ void __launch_bounds__(128)
elastic_kernel(int64_t ne, const double* __restrict__ X, const int32_t* __restrict__ conn,
               const double* __restrict__ u, const double* __restrict__ scale, const double* __restrict__ st_old,
               double* __restrict__ st_new, double* __restrict__ fe, double* __restrict__ S,
               double* __restrict__ mises, double* __restrict__ peeq, double lam_m, double mu_m,
               const double* __restrict__ lam_e, const double* __restrict__ mu_e) {
  constexpr int NN = ElemTraits<ET>::nnode, NG = ElemTraits<ET>::ngp;
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const double lam = lam_e ? lam_e[e] : lam_m, mu = lam_e ? mu_e[e] : mu_m;
  int32_t nod[NN];
#pragma unroll
  for (int a = 0; a < NN; ++a) nod[a] = conn[e * NN + a];
  double acc[6] = {0, 0, 0, 0, 0, 0}, vsum = 0.0;
  if constexpr (ET == EXFEM_C3D8) {
    const double sc = MODE == FORCE_FULL && scale ? scale[e] : 1.0;
    double cm[7][3], um[7][3];
    {
      double xa[8][3], ua[8][3];
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          xa[a][c] = X[3 * (int64_t)nod[a] + c];
          ua[a][c] = u[3 * (int64_t)nod[a] + c];
        }
#pragma unroll
      for (int a = 7; a >= 0; --a)  // relative to the first node, as in gather_nodes
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          xa[a][c] -= xa[0][c];
          ua[a][c] -= ua[0][c];
        }
      hex_to_modal(xa, cm);
      hex_to_modal(ua, um);
    }
    double J0[9], iJ0[9], tr0 = 0.0, Fm[7][3], tacc = 0.0;
#pragma unroll
    for (int n = 0; n < 3; ++n)
#pragma unroll
      for (int i = 0; i < 3; ++i) J0[3 * n + i] = cm[i][n];
    inv3(J0, iJ0);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int i = 0; i < 3; ++i) tr0 += um[i][c] * iJ0[3 * i + c];
#pragma unroll
    for (int k = 0; k < 7; ++k) Fm[k][0] = Fm[k][1] = Fm[k][2] = 0.0;
#pragma unroll 1
    for (int g = 0; g < NG; ++g) {
      const double x = HEX_GQ * hex_sign(g, 0), y = HEX_GQ * hex_sign(g, 1), z = HEX_GQ * hex_sign(g, 2);
      double J[9], iJ[9], G[9], H[9], eps[6], sig[6];
      hex_modal_grad(cm, x, y, z, J);
      const double detJ = inv3(J, iJ);
      hex_modal_grad(um, x, y, z, G);
      matmul3(G, iJ, H);
      const double bb = (tr0 - (H[0] + H[4] + H[8])) * (1.0 / 3.0);
      H[0] += bb;
      H[4] += bb;
      H[8] += bb;
      sym_from_grad(H, eps);
      elastic_stress(lam, mu, eps, sig);
      if constexpr (MODE == FORCE_STRESS) {
#pragma unroll
        for (int k = 0; k < 6; ++k) acc[k] += detJ * sig[k];
        vsum += detJ;
      } else {
        const double vol = detJ * sc, t = vol * (sig[0] + sig[1] + sig[2]) * (1.0 / 3.0);
        tacc += t;
        const double r[3][3] = {{vol * sig[0] - t, vol * sig[3], vol * sig[5]},
                                {vol * sig[3], vol * sig[1] - t, vol * sig[4]},
                                {vol * sig[5], vol * sig[4], vol * sig[2] - t}};
        double Q[9];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int i = 0; i < 3; ++i)
            Q[3 * c + i] = r[c][0] * iJ[3 * i] + r[c][1] * iJ[3 * i + 1] + r[c][2] * iJ[3 * i + 2];
        hex_modal_grad_adj(Q, x, y, z, Fm);
        if (st_new) st_new[e * NG + g] = st_old ? st_old[e * NG + g] : 0.0;
      }
    }
    if constexpr (MODE == FORCE_FULL) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int i = 0; i < 3; ++i) Fm[i][c] += tacc * iJ0[3 * i + c];
      double f[8][3];
      hex_from_modal(Fm, f);
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) fe[(e * 8 + a) * 3 + c] = f[a][c];
    }
  } else {
    static_assert(MODE == FORCE_STRESS, "C3D10 forces are taken by force_kernel at every size");
#pragma unroll 1
    for (int g = 0; g < NG; ++g) {
      double J[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, G[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, iJ[9], H[9], eps[6], sig[6];
#pragma unroll
      for (int a = 0; a < NN; ++a) {
        const int64_t n3 = 3 * (int64_t)nod[a];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double dn = elem_dN(ET, g, a, i);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            J[3 * c + i] += X[n3 + c] * dn;
            G[3 * c + i] += u[n3 + c] * dn;
          }
        }
      }
      const double w = inv3(J, iJ) * (1.0 / 24.0);
      matmul3(G, iJ, H);
      sym_from_grad(H, eps);
      elastic_stress(lam, mu, eps, sig);
#pragma unroll
      for (int k = 0; k < 6; ++k) acc[k] += w * sig[k];
      vsum += w;
    }
  }
  if constexpr (MODE == FORCE_STRESS) store_stress(e, acc, vsum, 0.0, S, mises, peeq);
}

template <int ET, bool J2, int MODE>
int force_go(exfem_block_s* b, const double* u, const double* st_old, double* st_new, double* fe, double* S,
             double* mises, double* peeq, cudaStream_t s, const uint8_t* nf = nullptr, const int* skip = nullptr) {
  constexpr int NW = 4;
  using SM = ForceSmem<ET, J2 && MODE != FORCE_PRODUCT>;
  constexpr size_t smem = NW * sizeof(SM);
  constexpr int64_t per = NW * SM::EPW;
  // bulk copies need 16-byte boundaries: elements' states and forces are multiples of
  // 16 bytes, so it takes the arrays themselves to start on one
  const int bulk = ((uintptr_t)st_old % 16 == 0 ? BULK_OLD : 0) | ((uintptr_t)st_new % 16 == 0 ? BULK_NEW : 0) |
                   ((uintptr_t)fe % 16 == 0 ? BULK_FE : 0);
  auto kern = force_kernel<ET, J2, MODE, NW>;
  const unsigned grid = (unsigned)((b->ne + per - 1) / per);
  if constexpr (MODE == FORCE_PRODUCT)
    launch_chained(kern, grid, 32 * NW, smem, s, b->ne, b->X.p, b->conn.p, u, b->scale.p, st_old, st_new, fe, b->tan64.p,
                   b->tan32.p, S, mises, peeq, b->mat, b->lam_e.p, b->mu_e.p, b->order_dev.p, b->tile == 128 ? 7 : 8,
                   bulk, b->dev_err.p, nf, skip);
  else
    kern<<<grid, 32 * NW, smem, s>>>(b->ne, b->X.p, b->conn.p, u, b->scale.p, st_old, st_new, fe, b->tan64.p, b->tan32.p,
                                     S, mises, peeq, b->mat, b->lam_e.p, b->mu_e.p, b->order_dev.p,
                                     b->tile == 128 ? 7 : 8, bulk, b->dev_err.p, nf, skip);
  EX_LAUNCH_CHECK();
  return EXFEM_OK;
}

template <int ET, int MODE>
int elastic_go(exfem_block_s* b, const double* u, const double* st_old, double* st_new, double* fe, double* S,
               double* mises, double* peeq, cudaStream_t s) {
  elastic_kernel<ET, MODE><<<(unsigned)((b->ne + 127) / 128), 128, 0, s>>>(
      b->ne, b->X.p, b->conn.p, u, b->scale.p, st_old, st_new, fe, S, mises, peeq, b->mat.lam, b->mat.mu, b->lam_e.p,
      b->mu_e.p);
  EX_LAUNCH_CHECK();
  return EXFEM_OK;
}

// a thread takes eight times as long over its element as the lanes of a warp, and its blocks
// cover the chip from some 19,000 elements on (148 x 128); forces, us a call, warp / thread:
// 4,000 elements 8.5 / 11.1, 8,000 10.4 / 12.5, 12,000 12.5 / 12.5, 16,000 14.5 / 12.5
bool elastic_force_by_threads(int64_t ne) { return ne > 12000; }

template <int ET>
int force_et(exfem_block_s* b, int mode, const double* u, const double* st_old, double* st_new, double* fe, double* S,
             double* mises, double* peeq, cudaStream_t s) {
  if (b->mat.kind == EXFEM_J2) {
    if (mode == FORCE_FULL) return force_go<ET, true, FORCE_FULL>(b, u, st_old, st_new, fe, S, mises, peeq, s);
    if (mode == FORCE_TANGENT) return force_go<ET, true, FORCE_TANGENT>(b, u, st_old, st_new, fe, S, mises, peeq, s);
    return force_go<ET, true, FORCE_STRESS>(b, u, st_old, st_new, fe, S, mises, peeq, s);
  }
  if (mode == FORCE_TANGENT) return EXFEM_OK;  // an elastic tangent does not change
  if (mode == FORCE_STRESS) return elastic_go<ET, FORCE_STRESS>(b, u, st_old, st_new, fe, S, mises, peeq, s);
  if constexpr (ET == EXFEM_C3D8)
    if (elastic_force_by_threads(b->ne)) return elastic_go<ET, FORCE_FULL>(b, u, st_old, st_new, fe, S, mises, peeq, s);
  return force_go<ET, false, FORCE_FULL>(b, u, st_old, st_new, fe, S, mises, peeq, s);
}

}  // namespace

int launch_force(exfem_block_s* b, int mode, const double* u, const double* st_old, double* st_new, double* fe,
                 double* S, double* mises, double* peeq, cudaStream_t s) {
  if (b->ne == 0) return EXFEM_OK;
  return b->etype == EXFEM_C3D8 ? force_et<EXFEM_C3D8>(b, mode, u, st_old, st_new, fe, S, mises, peeq, s)
                                : force_et<EXFEM_C3D10>(b, mode, u, st_old, st_new, fe, S, mises, peeq, s);
}

// element vectors fe (ne, nnode, 3) of the FP64 tangent product K (free v): the force
// kernel on v with the linear stress, elastic or of the stored tangent data
int launch_product_elements(exfem_block_s* b, const double* v, double* fe, bool bc, const int* skip, cudaStream_t s) {
  if (b->ne == 0) return EXFEM_OK;
  const uint8_t* nf = bc ? b->node_fixed.p : nullptr;
  const bool j2 = b->mat.kind == EXFEM_J2;
#define EXF_GO(ET, J2) \
  force_go<ET, J2, FORCE_PRODUCT>(b, v, nullptr, nullptr, fe, nullptr, nullptr, nullptr, s, nf, skip)
  if (b->etype == EXFEM_C3D8) return j2 ? EXF_GO(EXFEM_C3D8, true) : EXF_GO(EXFEM_C3D8, false);
  return j2 ? EXF_GO(EXFEM_C3D10, true) : EXF_GO(EXFEM_C3D10, false);
#undef EXF_GO
}

}  // namespace exfem
