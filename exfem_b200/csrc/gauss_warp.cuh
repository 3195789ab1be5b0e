// Kinematics of the warp-per-elements FP64 kernels (force, tangents): one warp holds
// 32 / ngp elements (4 C3D8, 8 C3D10), one lane per Gauss point, lane = element * ngp +
// point.  Node values meet in the warp's shared memory once per element.
#pragma once
#include "async_copy.cuh"
#include "element_math.cuh"

namespace exfem {

// dN_b / dxi_i at every Gauss point in rows of XS: even, so that pairs load with one
// 16-byte access, and such that the points' rows fall into different banks
template <int ET>
struct DnTable {
  static constexpr int NN = ElemTraits<ET>::nnode, NG = ElemTraits<ET>::ngp, XS = ET == EXFEM_C3D8 ? 26 : 30;
  double v[NG * XS];
  constexpr DnTable() : v{} {
    for (int g = 0; g < NG; ++g)
      for (int b = 0; b < NN; ++b)
        for (int i = 0; i < 3; ++i) v[g * XS + 3 * b + i] = ET == EXFEM_C3D8 ? hex_dN(g, b, i) : tet10_dN(g, b, i);
  }
};
static __device__ const DnTable<EXFEM_C3D8> dn_hex{};
static __device__ const DnTable<EXFEM_C3D10> dn_tet{};
template <int ET>
__device__ __forceinline__ const double* dn_table() {
  if constexpr (ET == EXFEM_C3D8) return dn_hex.v;
  else return dn_tet.v;
}

// Node values of a warp's elements: W = 3 (coordinates) or 6 (coordinates and
// displacements) per node of a C3D10 or per trilinear mode of a C3D8.  The element
// stride keeps 16-byte accesses of the elements' lanes in different banks.
template <int ET, bool U>
struct NodeSmem {
  static constexpr int W = U ? 6 : 3, EPW = 32 / ElemTraits<ET>::ngp;
  static constexpr int ES = ET == EXFEM_C3D8 ? 8 * W + 2 : (U ? 62 : 30);
  alignas(16) double v[EPW * ES];
};

// Gather of X and u (u may be NULL: zeros) at the nodes of the warp's elements.
// `eid`: this lane's element; `elem(el)`: the warp's el-th element, called by all lanes;
// `cnt`: elements of this warp; `nf` (or NULL): per node, the components of u taken as
// zero (bits); `ready()`: called by all lanes once, after the loads that depend on the
// mesh alone and before those of u.  The caller synchronises the warp afterwards.
//
// C3D8: a lane loads one of its element's eight nodes and a Walsh-Hadamard transform
// over the element's lanes turns the corner values into the modal ones (corner signs
// are the characters of the lane's three bits), so the Gauss points need 7 modes
// instead of 8 nodes and the centre's gradients are modes themselves.
template <int ET, bool U, class Elem, class Ready>
__device__ __forceinline__ void gather_nodes(NodeSmem<ET, U>& nd, const double* __restrict__ X,
                                             const int32_t* __restrict__ conn, const double* u,
                                             const uint8_t* __restrict__ nf, int64_t eid, int cnt, Elem elem,
                                             Ready ready) {
  constexpr int W = NodeSmem<ET, U>::W, EPW = NodeSmem<ET, U>::EPW, ES = NodeSmem<ET, U>::ES;
  const int lane = threadIdx.x & 31;
  if constexpr (ET == EXFEM_C3D8) {
    const int j = lane & 7, a = j ^ ((j >> 1) & 1);  // bits of j: the corner lies on the + side of each axis
    const int32_t node = conn[eid * 8 + a];
    const int64_t n3 = 3 * (int64_t)node;
    const unsigned off = U && nf ? nf[node] : 0u;
    double v[W];
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] = X[n3 + c];
    ready();
    if constexpr (U)
#pragma unroll
      for (int c = 0; c < 3; ++c) v[3 + c] = u && !((off >> c) & 1u) ? u[n3 + c] : 0.0;
    // relative to the first node: the sums below then carry no rounding of the
    // distance from the origin
#pragma unroll
    for (int k = 0; k < W; ++k) v[k] -= __shfl_sync(0xffffffffu, v[k], lane & 24);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
      for (int k = 0; k < W; ++k) {
        const double p = __shfl_xor_sync(0xffffffffu, v[k], o);
        v[k] = (j & o) ? v[k] - p : v[k] + p;
      }
#pragma unroll
    for (int k = 0; k < W; ++k) nd.v[(lane >> 3) * ES + j * W + k] = 0.125 * v[k];
  } else {
    constexpr int NN = 10, P = (EPW * NN + 31) / 32;
    int32_t node[P];
    unsigned off[P];
    int at[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int k = 32 * p + lane, el = k / NN < EPW ? k / NN : EPW - 1, a = k - el * NN;
      const int64_t e = elem(el);
      at[p] = k < cnt * NN ? el * ES + a * W : -1;
      node[p] = at[p] >= 0 ? conn[e * NN + a] : 0;
    }
#pragma unroll
    for (int p = 0; p < P; ++p) {
      off[p] = U && nf && at[p] >= 0 ? nf[node[p]] : 0u;
      if (at[p] >= 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) nd.v[at[p] + c] = X[3 * (int64_t)node[p] + c];
    }
    ready();
    if constexpr (U)
#pragma unroll
      for (int p = 0; p < P; ++p)
        if (at[p] >= 0)
#pragma unroll
          for (int c = 0; c < 3; ++c)
            nd.v[at[p] + 3 + c] = u && !((off[p] >> c) & 1u) ? u[3 * (int64_t)node[p] + c] : 0.0;
  }
}

// J = dX/dxi and G = du/dxi at this lane's Gauss point (m[3c + i]); J0, G0: at the
// centre (C3D8 only)
template <int ET, bool U>
__device__ __forceinline__ void gauss_gradients(const NodeSmem<ET, U>& nd, const double* __restrict__ tab, int le,
                                                int g, double (&J)[9], double (&G)[9], double (&J0)[9],
                                                double (&G0)[9]) {
  constexpr int W = NodeSmem<ET, U>::W, ES = NodeSmem<ET, U>::ES;
  const double2* p = reinterpret_cast<const double2*>(nd.v + le * ES);
  if constexpr (ET == EXFEM_C3D8) {
    const double x = hex_sign(g, 0) > 0 ? HEX_GQ : -HEX_GQ, y = hex_sign(g, 1) > 0 ? HEX_GQ : -HEX_GQ,
                 z = hex_sign(g, 2) > 0 ? HEX_GQ : -HEX_GQ;
    double m[8 * W];  // modes 1, x, y, xy, z, xz, yz, xyz
#pragma unroll
    for (int k = W / 2; k < 8 * W / 2; ++k) {
      const double2 t = p[k];
      m[2 * k] = t.x;
      m[2 * k + 1] = t.y;
    }
#pragma unroll
    for (int f = 0; f < W / 3; ++f) {
      double(&D)[9] = f ? G : J;
      double(&D0)[9] = f ? G0 : J0;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int o = 3 * f + c;
        const double mx = m[W + o], my = m[2 * W + o], mxy = m[3 * W + o], mz = m[4 * W + o], mxz = m[5 * W + o],
                     myz = m[6 * W + o], mxyz = m[7 * W + o];
        D0[3 * c] = mx;
        D0[3 * c + 1] = my;
        D0[3 * c + 2] = mz;
        D[3 * c] = mx + y * mxy + z * mxz + (y * z) * mxyz;
        D[3 * c + 1] = my + x * mxy + z * myz + (x * z) * mxyz;
        D[3 * c + 2] = mz + y * myz + x * mxz + (x * y) * mxyz;
      }
    }
  } else {
    const double2* dn = reinterpret_cast<const double2*>(tab + g * DnTable<ET>::XS);
#pragma unroll
    for (int k = 0; k < 9; ++k) J[k] = G[k] = 0.0;
#pragma unroll
    for (int b = 0; b < 10; b += 2) {  // two nodes: 2 W values and 6 table entries in 16-byte loads
      double v[2 * W], d[6];
#pragma unroll
      for (int k = 0; k < W; ++k) {
        const double2 t = p[b * W / 2 + k];
        v[2 * k] = t.x;
        v[2 * k + 1] = t.y;
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double2 t = dn[3 * b / 2 + k];
        d[2 * k] = t.x;
        d[2 * k + 1] = t.y;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            J[3 * c + i] += v[h * W + c] * d[3 * h + i];
            if constexpr (U) G[3 * c + i] += v[h * W + 3 + c] * d[3 * h + i];
          }
    }
  }
}

}  // namespace exfem
