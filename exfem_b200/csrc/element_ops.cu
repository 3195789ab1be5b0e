// FP64 element operations: deterministic assembly of element vectors (gather plan or
// colour scatter), the geometry streams of the matrix-free operator, initial-stress
// stiffness, and the stored-Ke element-by-element product and diagonals.
//
// Reference: gfem/model.py:113-117 (geo_stiff), 162-173 (ops_matvec / ops_diagonal),
// 241-267 (gather plan assembly), 466-486 (Model.internal_force / element_stiffness).
#include "internal.h"

namespace exfem {

// ---------------------------------------------------------------- assembly
// f[3n+c] = sum over the gather plan of node n (reference order); optional opA
// finalisation y = fixed ? v : sum.  One thread per degree of freedom: the three of a
// node read neighbouring entries, and eight plan slots and their entries are requested
// before any is added (in the plan's order), because the kernel is bound by the latency
// of the plan -> entry chain: one thread per node with one slot in flight took 10 us
// for 44,541 nodes of C3D8 and 27 us for 176,715 of C3D10.
__global__ void __launch_bounds__(256)
gather_assemble_kernel(int64_t ndof, int vmax, const int32_t* __restrict__ plan, int32_t sentinel,
                       const double* ys, const __grid_constant__ RowOut<double> out,
                       const uint8_t* __restrict__ fixed, const double* v, const int* skip) {
  constexpr int K = 8;
  const int64_t d = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool in = d < ndof;
  const int64_t n = in ? d / 3 : 0;
  const int c = in ? (int)(d - 3 * n) : 0;
  const int32_t* row = plan + n * vmax;
  const bool pass = in && v && fixed && fixed[d];
  int32_t slot[K];  // the plan is constant: its first slots are requested before the wait
#pragma unroll
  for (int k = 0; k < K; ++k) slot[k] = k < vmax ? row[k] : sentinel;
  chain_wait();
  if (!in || (skip && *skip)) return;
  double s = 0.0;
  for (int k0 = 0; k0 < vmax; k0 += K) {
    double w[K];
    if (k0 > 0)
#pragma unroll
      for (int k = 0; k < K; ++k) slot[k] = k0 + k < vmax ? row[k0 + k] : sentinel;
#pragma unroll
    for (int k = 0; k < K; ++k) w[k] = slot[k] != sentinel ? ys[3 * (int64_t)slot[k] + c] : 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (slot[k] != sentinel) s += w[k];
    if (slot[K - 1] == sentinel) break;  // slots are listed without gaps
  }
  row_out(out, d, pass ? v[d] : s);
}

int launch_gather_assemble(exfem_block_s* b, const double* ys, double* f, const double* v_opa,
                           const int* skip, cudaStream_t s, const RowOut<double>* out) {
  RowOut<double> o;
  if (out) o = *out;
  else o.y = f;
  if (b->nn == 0) return EXFEM_OK;
  const int threads = 256;
  launch_chained(gather_assemble_kernel, (unsigned)((b->ndof() + threads - 1) / threads), threads, 0, s, b->ndof(),
                 b->vmax, b->plan.p, (int32_t)(b->ne * b->nnode), ys, o,
                 (const uint8_t*)(v_opa ? b->fixed.p : nullptr), v_opa, skip);
  EX_LAUNCH_CHECK();
  return EXFEM_OK;
}

// one colour: elements of the colour share no node, so plain read-modify-write is exact
__global__ void colour_scatter_kernel(int64_t cnt, const int32_t* __restrict__ elems,
                                      const int32_t* __restrict__ conn, int nnode,
                                      const double* __restrict__ fe, double* __restrict__ f) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= cnt) return;
  const int64_t e = elems[i];
  for (int a = 0; a < nnode; ++a) {
    const int64_t n = conn[e * nnode + a];
    for (int c = 0; c < 3; ++c) f[3 * n + c] += fe[(e * nnode + a) * 3 + c];
  }
}

int launch_colour_assemble(exfem_block_s* b, const double* fe, double* f, cudaStream_t s) {
  EX_CUDA(cudaMemsetAsync(f, 0, sizeof(double) * b->ndof(), s));
  for (int c = 0; c < b->ncolour; ++c) {
    const int64_t a0 = b->colour_ptr[c], cnt = b->colour_ptr[c + 1] - a0;
    if (!cnt) continue;
    colour_scatter_kernel<<<(unsigned)((cnt + 127) / 128), 128, 0, s>>>(cnt, b->colour_elems.p + a0,
                                                                        b->conn.p, b->nnode, fe, f);
    EX_LAUNCH_CHECK();
  }
  return EXFEM_OK;
}

// ---------------------------------------------------------------- geometry streams
// Per element: C3D8 the 7 modal coordinate vectors (21) and the stiffness scale;
// C3D10 the inverse Jacobian (9) and vol * scale; then, only for blocks with
// per-element Lame parameters, lambda and mu (the matrix-free kernels otherwise
// take the material's from their arguments).
template <int ET>
__global__ void geometry_kernel(int64_t ne, const double* __restrict__ X, const int32_t* __restrict__ conn_tile,
                                const int32_t* __restrict__ order, const double* __restrict__ scale,
                                const double* __restrict__ lam_e, const double* __restrict__ mu_e, int GS,
                                double* __restrict__ g64, float* __restrict__ g32, int tile) {
  using Tr = ElemTraits<ET>;
  constexpr int NN = Tr::nnode, GF = Tr::geo_stride;
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;   // tile position
  if (p >= ne) return;
  const int64_t e = order[p];
  const int32_t* cn = conn_tile + p * NN;                              // this position's nodes
  const double sc = scale ? scale[e] : 1.0;
  double out[GF];
#pragma unroll
  for (int k = 0; k < GF; ++k) out[k] = 0.0;
  if constexpr (ET == EXFEM_C3D8) {
    double xa[8][3], cm[7][3];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int c = 0; c < 3; ++c) xa[a][c] = X[3 * (int64_t)cn[a] + c];
    hex_to_modal(xa, cm);
#pragma unroll
    for (int k = 0; k < 7; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) out[3 * k + c] = cm[k][c];
    out[21] = sc;
  } else {
    double J[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, iJ[9];
#pragma unroll
    for (int a = 0; a < 10; ++a) {
      const int64_t n3 = 3 * (int64_t)cn[a];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) J[3 * c + i] += X[n3 + c] * tet10_dN(0, a, i);
    }
    const double det = inv3(J, iJ);
#pragma unroll
    for (int k = 0; k < 9; ++k) out[k] = iJ[k];
    out[9] = det / 24.0 * sc;
  }
  if (lam_e) {
    out[GF - 2] = lam_e[e];
    out[GF - 1] = mu_e[e];
  }
  for (int k = 0; k < GS; ++k) {
    g64[tile_index(p, k, GS, tile)] = out[k];
    g32[tile_index(p, k, GS, tile)] = (float)out[k];
  }
}

int build_geometry(exfem_block_s* b) {
  const int GF = b->etype == EXFEM_C3D8 ? ElemTraits<EXFEM_C3D8>::geo_stride : ElemTraits<EXFEM_C3D10>::geo_stride;
  const int GS = b->lam_e.p ? GF : GF - 2;
  int st;
  const int64_t padded = b->ntile * b->tile * GS;
  if (b->geo64.n != (size_t)padded || b->geo_stride != GS) {
    if ((st = b->geo64.alloc(padded))) return st;
    if ((st = b->geo32.alloc(padded))) return st;
    EX_CUDA(cudaMemset(b->geo64.p, 0, b->geo64.bytes()));
    EX_CUDA(cudaMemset(b->geo32.p, 0, b->geo32.bytes()));
  }
  b->geo_stride = GS;
  if (b->ne == 0) return EXFEM_OK;
  const int threads = 128;
  const unsigned grid = (unsigned)((b->ne + threads - 1) / threads);
  if (b->etype == EXFEM_C3D8)
    geometry_kernel<EXFEM_C3D8><<<grid, threads>>>(b->ne, b->X.p, b->conn_tile.p, b->order_dev.p, b->scale.p,
                                                   b->lam_e.p, b->mu_e.p, GS, b->geo64.p, b->geo32.p, b->tile);
  else
    geometry_kernel<EXFEM_C3D10><<<grid, threads>>>(b->ne, b->X.p, b->conn_tile.p, b->order_dev.p, b->scale.p,
                                                    b->lam_e.p, b->mu_e.p, GS, b->geo64.p, b->geo32.p, b->tile);
  EX_LAUNCH_CHECK();
  // the legacy stream only: a device-wide synchronisation would invalidate a graph
  // capture in progress on another host thread
  EX_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
  return EXFEM_OK;
}

// ---------------------------------------------------------------- initial-stress stiffness
// K_sigma of an element under a constant Cauchy stress sigma (gfem/model.py:113-117
// geo_stiff): k_ab = sum_g vol_g dN_a/dX . sigma . dN_b/dX with the plain
// (not B-bar) shape-function gradients and vol_g = w_g det J, expanded as
// K[3a+i, 3b+j] = k_ab delta_ij.  One thread per (element, node a) writes rows
// 3a .. 3a+2.
template <int ET>
__global__ void __launch_bounds__(128)
geo_stiffness_kernel(int64_t ne, const double* __restrict__ X, const int32_t* __restrict__ conn,
                     const double* __restrict__ S, double* __restrict__ Kg) {
  constexpr int NN = ElemTraits<ET>::nnode, NG = ElemTraits<ET>::ngp, ND = 3 * NN;
  const double w = ET == EXFEM_C3D8 ? 1.0 : 1.0 / 24.0;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < ne * NN; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = t / NN;
    const int a = (int)(t - e * NN);
    const int32_t* ce = conn + e * NN;
    double sg[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) sg[k] = S[e * 9 + k];
    double k_ab[NN];
#pragma unroll
    for (int b = 0; b < NN; ++b) k_ab[b] = 0.0;
    for (int g = 0; g < NG; ++g) {
      double J[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, iJ[9];
      for (int c = 0; c < NN; ++c) {
        const double* xc = X + 3 * (int64_t)ce[c];
#pragma unroll
        for (int n = 0; n < 3; ++n)
#pragma unroll
          for (int i = 0; i < 3; ++i) J[3 * n + i] += xc[n] * elem_dN(ET, g, c, i);
      }
      const double vol = w * inv3(J, iJ);
      double ga[3], sa[3];                                   // dN_a/dX and sigma . dN_a/dX
#pragma unroll
      for (int j = 0; j < 3; ++j)
        ga[j] = elem_dN(ET, g, a, 0) * iJ[j] + elem_dN(ET, g, a, 1) * iJ[3 + j] + elem_dN(ET, g, a, 2) * iJ[6 + j];
#pragma unroll
      for (int j = 0; j < 3; ++j) sa[j] = ga[0] * sg[j] + ga[1] * sg[3 + j] + ga[2] * sg[6 + j];
      for (int b = 0; b < NN; ++b) {
        double gb[3];
#pragma unroll
        for (int j = 0; j < 3; ++j)
          gb[j] = elem_dN(ET, g, b, 0) * iJ[j] + elem_dN(ET, g, b, 1) * iJ[3 + j] + elem_dN(ET, g, b, 2) * iJ[6 + j];
        k_ab[b] += vol * (sa[0] * gb[0] + sa[1] * gb[1] + sa[2] * gb[2]);
      }
    }
    double* K = Kg + e * (int64_t)ND * ND;
    for (int i = 0; i < 3; ++i)
      for (int b = 0; b < NN; ++b)
#pragma unroll
        for (int j = 0; j < 3; ++j) K[(int64_t)(3 * a + i) * ND + 3 * b + j] = i == j ? k_ab[b] : 0.0;
  }
}

int launch_geo_stiffness(exfem_block_s* b, const double* S, double* Kg, cudaStream_t s) {
  if (b->ne == 0) return EXFEM_OK;
  const int64_t work = b->ne * b->nnode;
  const unsigned grid = (unsigned)std::min<int64_t>((work + 127) / 128, 1 << 20);
  if (b->etype == EXFEM_C3D8) geo_stiffness_kernel<EXFEM_C3D8><<<grid, 128, 0, s>>>(b->ne, b->X.p, b->conn.p, S, Kg);
  else geo_stiffness_kernel<EXFEM_C3D10><<<grid, 128, 0, s>>>(b->ne, b->X.p, b->conn.p, S, Kg);
  EX_LAUNCH_CHECK();
  return EXFEM_OK;
}

// ---------------------------------------------------------------- stored-Ke products
// ys[e, r] = sum_j Ke[e, r, j] * (free*v)[dofs[e, j]]
//
// Bound by streaming Ke.  One warp per element: four lanes share a row and read it in
// 16-byte pieces 64 contiguous bytes at a time (8 rows of an element per load
// instruction, every sector whole), all pieces of an element requested before the
// first is used; the lanes' v come from one gather of the element's DOFs by shuffles,
// and a row is summed over its four lanes.  40,641 C3D8 (187 MB of Ke) on B200: 30 us
// against 77 us for one thread per row, whose loads were a row apart.
template <int ET, bool VEC>
__global__ void __launch_bounds__(256)
ebe_rows_kernel(int64_t ne, const int32_t* __restrict__ conn, const double* __restrict__ Ke,
                const double* __restrict__ v, const uint8_t* __restrict__ fixed, double* __restrict__ ys,
                const int* __restrict__ skip) {
  constexpr int NN = ElemTraits<ET>::nnode, ND = 3 * NN, NP = ND / 2;  // pieces of 16 bytes per row
  constexpr int RP = (ND + 7) / 8, PL = (NP + 3) / 4;                  // passes over the rows, pieces per lane
  if (skip && *skip) return;
  const int lane = threadIdx.x & 31, row = lane >> 2, q = lane & 3;
  const int64_t e = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (e >= ne) return;
  const double* K = Ke + e * (ND * ND);
  double2 k[RP][PL];
#pragma unroll
  for (int r = 0; r < RP; ++r)
#pragma unroll
    for (int p = 0; p < PL; ++p) {
      const int i = 8 * r + row, j = q + 4 * p;
      k[r][p] = make_double2(0.0, 0.0);
      if (i < ND && j < NP) {
        const double* src = K + i * ND + 2 * j;
        if constexpr (VEC) k[r][p] = __ldcs(reinterpret_cast<const double2*>(src));
        else k[r][p] = make_double2(src[0], src[1]);
      }
    }
  double vl = 0.0;
  if (lane < ND) {
    const int64_t d = 3 * (int64_t)conn[e * NN + lane / 3] + lane % 3;
    vl = (fixed && fixed[d]) ? 0.0 : v[d];
  }
  double s[RP];
#pragma unroll
  for (int r = 0; r < RP; ++r) s[r] = 0.0;
#pragma unroll
  for (int p = 0; p < PL; ++p) {
    const double va = __shfl_sync(0xffffffffu, vl, 2 * (q + 4 * p)), vb = __shfl_sync(0xffffffffu, vl, 2 * (q + 4 * p) + 1);
    const bool in = q + 4 * p < NP;
#pragma unroll
    for (int r = 0; r < RP; ++r)
      if (in) s[r] = fma(k[r][p].y, vb, fma(k[r][p].x, va, s[r]));
  }
#pragma unroll
  for (int r = 0; r < RP; ++r) {
    s[r] += __shfl_xor_sync(0xffffffffu, s[r], 1);
    s[r] += __shfl_xor_sync(0xffffffffu, s[r], 2);
    if (q == 0 && 8 * r + row < ND) ys[e * ND + 8 * r + row] = s[r];
  }
}

int launch_ebe_matvec(exfem_block_s* b, const double* Ke, const double* v, double* y,
                      const int* skip, cudaStream_t s, bool bc, const RowOut<double>* out) {
  int st;
  if (b->ys.n < (size_t)(b->ne * b->nnode * 3) && (st = b->ys.alloc(b->ne * b->nnode * 3))) return st;
  if (b->ne) {
    const unsigned grid = (unsigned)((b->ne + 7) / 8);
    const uint8_t* fx = bc ? b->fixed.p : nullptr;
    const bool vec = (uintptr_t)Ke % 16 == 0;  // element matrices are multiples of 16 bytes
#define EXF_ROWS(ET, VEC) ebe_rows_kernel<ET, VEC><<<grid, 256, 0, s>>>(b->ne, b->conn.p, Ke, v, fx, b->ys.p, skip)
    if (b->etype == EXFEM_C3D8) {
      if (vec) EXF_ROWS(EXFEM_C3D8, true);
      else EXF_ROWS(EXFEM_C3D8, false);
    } else {
      if (vec) EXF_ROWS(EXFEM_C3D10, true);
      else EXF_ROWS(EXFEM_C3D10, false);
    }
#undef EXF_ROWS
    EX_LAUNCH_CHECK();
  }
  return launch_gather_assemble(b, b->ys.p, y, bc ? v : nullptr, skip, s, out);
}

__global__ void ebe_diag_kernel(int64_t nn, int vmax, int nnode, const int32_t* __restrict__ plan,
                                int64_t sentinel, const double* __restrict__ Ke, const double* __restrict__ ediag,
                                double* __restrict__ diag) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= nn) return;
  const int nd = 3 * nnode;
  double s[3] = {0, 0, 0};
  for (int k = 0; k < vmax; ++k) {
    const int64_t slot = plan[n * vmax + k];
    if (slot == sentinel) break;
    const int64_t e = slot / nnode;
    const int a = (int)(slot - e * nnode);
    for (int c = 0; c < 3; ++c)
      s[c] += Ke ? Ke[e * nd * nd + (3 * a + c) * (int64_t)nd + 3 * a + c] : ediag[slot * 3 + c];
  }
  for (int c = 0; c < 3; ++c) diag[3 * n + c] = s[c];
}

int launch_ebe_diagonal(exfem_block_s* b, const double* Ke, double* diag, cudaStream_t s) {
  if (b->nn == 0) return EXFEM_OK;
  ebe_diag_kernel<<<(unsigned)((b->nn + 255) / 256), 256, 0, s>>>(b->nn, b->vmax, b->nnode, b->plan.p,
                                                                  b->ne * b->nnode, Ke, nullptr, diag);
  EX_LAUNCH_CHECK();
  return EXFEM_OK;
}

int launch_mf_diagonal(exfem_block_s* b, double* diag, cudaStream_t s) {
  int st;
  if (b->ys.n < (size_t)(b->ne * b->nnode * 3) && (st = b->ys.alloc(b->ne * b->nnode * 3))) return st;
  // element diagonals of the current matrix-free tangent: the stiffness kernel
  // in diagonal-only mode reading the stored per-Gauss-point tangent data (the
  // displacement enters the tangent only through that data)
  if (b->ne) {
    const double* tan_in = b->mat.kind == EXFEM_J2 ? b->tan64.p : nullptr;
    if ((st = launch_stiffness(b, nullptr, nullptr, EXFEM_F64, nullptr, b->ys.p, s, tan_in))) return st;
  }
  ebe_diag_kernel<<<(unsigned)((b->nn + 255) / 256), 256, 0, s>>>(b->nn, b->vmax, b->nnode, b->plan.p,
                                                                  b->ne * b->nnode, nullptr, b->ys.p, diag);
  EX_LAUNCH_CHECK();
  return EXFEM_OK;
}

}  // namespace exfem
