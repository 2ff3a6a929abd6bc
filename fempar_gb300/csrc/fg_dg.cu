// fg_dg.cu -- discontinuous Galerkin (symmetric interior penalty) Poisson on the device: the
// second formulation of tutorial_01 (tutorial_01_poisson_sharp_circular_wave_modules.f90:146-322).
//
// Space: every dof is a cell-interior dof, numbered cell by cell in local order (id =
// c*nn + a + 1); boundary data enter weakly, so there are no strong Dirichlet dofs.  The row
// of dof (c, a) holds the dofs of c and of its face neighbours, blocks in increasing cell id.
//
// Numeric phase: the volume integrals come from the continuous path's element matrices (identity
// node table, no lifting).  Then one block per cell owns the cell's rows: it starts from the
// cell's element matrix and, face by face, integrates the facet terms that land in its rows
//   interior facet, cell side I, other side J (n_1 = n, n_2 = -n, n outward of the smaller
//   cell id, as the reference's first cell around the facet):
//     A(i_I, j_J) += w|J_F| ( -1/2 (grad phi_j^J . n_I) phi_i^I - 1/2 (grad phi_i^I . n_J) phi_j^J
//                             + C_IP/h phi_j^J phi_i^I (n_I . n_J) )
//   boundary facet:  A(i, j) += w|J_F| ( -(grad phi_j . n) phi_i - (grad phi_i . n) phi_j
//                                         + C_IP/h phi_i phi_j ),
//                    b(i) += w|J_F| ( -g (grad phi_i . n) + C_IP/h g phi_i )
// with C_IP = 10 p^2 and h = min over the facet's cells of 2 (prod_i |grad xi_i|^-1)^(1/3)
// (sbm_cell_map.i90:429-461, sbm_facet_integrator.i90:248-264).  Facet geometry per facet
// Gauss point ((p+1)^2 points, sbm_facet_map.i90:74-128): |J_F| n is the cofactor row of the cell's
// Jacobian for the face's direction, outward of the cell; the other cell evaluates its Jacobian
// at its own reference point of the facet point (through the face's shared corners).  Each cell
// computes its facets in its own frame and keeps the rows it owns: deterministic, no facet
// matrices in HBM, no atomics.  The reference sums a diagonal entry's contributions in facet id
// order, this kernel in local face order: entries agree to rounding.
#include <cub/cub.cuh>

#include "fg_internal.h"

namespace fg {

static inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// local face lf (0..5) of the hex = n-face 20 + lf in the reference order: xy(z=0), xy(z=1),
// xz(y=0), xz(y=1), yz(x=0), yz(x=1)
__host__ __device__ __forceinline__ void dg_face(int lf, int& d1, int& d2, int& dn, int& anchor) {
  const int dn_of[6] = {2, 2, 1, 1, 0, 0};
  dn = dn_of[lf];
  anchor = (lf & 1) << dn;
  d1 = dn == 0 ? 1 : 0;
  d2 = dn == 2 ? 1 : 2;
}

// ---- space ---------------------------------------------------------------------------
__global__ void k_dg_nbr_struct(int nx, int ny, int nz, int32_t* nbr, int8_t* nbrface) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t nc = (int64_t)nx * ny * nz;
  if (idx >= nc * 6) return;
  const int64_t c = idx / 6;
  const int lf = (int)(idx % 6);
  int d1, d2, dn, a;
  dg_face(lf, d1, d2, dn, a);
  const int n[3] = {nx, ny, nz};
  int ijk[3] = {(int)(c % nx), (int)((c / nx) % ny), (int)(c / ((int64_t)nx * ny))};
  const int side = (a >> dn) & 1;
  ijk[dn] += side ? 1 : -1;
  if (ijk[dn] < 0 || ijk[dn] >= n[dn]) {
    nbr[idx] = -1;
    nbrface[idx] = -1;
  } else {
    nbr[idx] = (int32_t)(ijk[0] + (int64_t)nx * (ijk[1] + (int64_t)ny * ijk[2]));
    nbrface[idx] = (int8_t)(lf ^ 1);
  }
}

// unstructured: the face's first cell is known (vowner); the other holder registers itself
__global__ void k_dg_second(int64_t nc, int64_t nv, const int32_t* cellvef, const int64_t* vowner, int64_t* second) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= nc * 6) return;
  const int64_t c = idx / 6;
  const int lf = (int)(idx % 6);
  const int64_t gid = cellvef[c * 26 + 20 + lf];
  if ((vowner[gid - nv] >> 5) != c) second[gid - nv] = c * 32 + 20 + lf;
}
__global__ void k_dg_nbr_unst(int64_t nc, int64_t nv, const int32_t* cellvef, const int64_t* vowner,
                              const int64_t* second, int32_t* nbr, int8_t* nbrface) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= nc * 6) return;
  const int64_t c = idx / 6;
  const int lf = (int)(idx % 6);
  const int64_t gid = cellvef[c * 26 + 20 + lf];
  const int64_t o = vowner[gid - nv];
  const int64_t s = (o >> 5) == c ? second[gid - nv] : o;
  nbr[idx] = s < 0 ? -1 : (int32_t)(s >> 5);
  nbrface[idx] = s < 0 ? (int8_t)-1 : (int8_t)((s & 31) - 20);
}

__global__ void k_dg_ids(int64_t n, int32_t* cellnode, int32_t* latdof, int32_t* free2lat) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  cellnode[i] = (int32_t)i;
  latdof[i] = (int32_t)(i + 1);
  free2lat[i] = (int32_t)i;
}

// blocks of a cell's rows: the cell and its neighbours, ascending
__device__ __forceinline__ int dg_blocks(int64_t c, const int32_t* nbr, int64_t* blk) {
  int nb = 0;
  blk[nb++] = c;
  for (int lf = 0; lf < 6; ++lf)
    if (nbr[c * 6 + lf] >= 0) blk[nb++] = nbr[c * 6 + lf];
  for (int i = 1; i < nb; ++i) {
    int64_t v = blk[i];
    int j = i - 1;
    while (j >= 0 && blk[j] > v) { blk[j + 1] = blk[j]; --j; }
    blk[j + 1] = v;
  }
  return nb;
}

__global__ void k_dg_rowlen(int64_t nc, int nn, const int32_t* nbr, int64_t* rowlen) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= nc * nn) return;
  const int64_t c = r / nn;
  int nb = 1;
  for (int lf = 0; lf < 6; ++lf) nb += nbr[c * 6 + lf] >= 0;
  rowlen[r] = (int64_t)nb * nn;
}

__global__ void k_dg_cols(int64_t nc, int nn, const int32_t* nbr, const int64_t* rowptr, int32_t* col) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= nc * nn) return;
  const int64_t c = r / nn;
  int64_t blk[7];
  const int nb = dg_blocks(c, nbr, blk);
  int64_t p = rowptr[r];
  for (int k = 0; k < nb; ++k)
    for (int b = 0; b < nn; ++b) col[p++] = (int32_t)(blk[k] * nn + b);
}

fg_status dg_space_build(fg_space* sp) {
  fg_mesh* m = sp->mesh;
  fg_ctx* ctx = m->ctx;
  const int64_t nc = m->ncells, nn = sp->tab.nn, n = nc * nn;
  if (n >= (int64_t)0x7fffffff) {
    set_error("dof count exceeds int32 ids");
    return FG_ERR_UNSUPPORTED;
  }
  sp->nlat = n;
  sp->nfree = n;
  sp->ndir = 0;
  FG_TRY(dev_alloc(ctx, (void**)&sp->d_cellnode, sizeof(int32_t) * n));
  FG_TRY(dev_alloc(ctx, (void**)&sp->d_latdof, sizeof(int32_t) * n));
  FG_TRY(dev_alloc(ctx, (void**)&sp->d_free2lat, sizeof(int32_t) * n));
  FG_TRY(dev_alloc(ctx, (void**)&sp->d_dir2lat, sizeof(int32_t)));
  k_dg_ids<<<nblk(n, 256), 256, 0, ctx->stream>>>(n, sp->d_cellnode, sp->d_latdof, sp->d_free2lat);
  FG_TRY(dev_alloc(ctx, (void**)&sp->d_dgnbr, sizeof(int32_t) * nc * 6));
  FG_TRY(dev_alloc(ctx, (void**)&sp->d_dgnbrface, sizeof(int8_t) * nc * 6));
  if (m->unst) {
    const int64_t nef = m->nedges + m->nfaces;
    int64_t* second = nullptr;
    FG_TRY(dev_alloc(ctx, (void**)&second, sizeof(int64_t) * (nef > 0 ? nef : 1)));
    FG_CUDA_TRY(cudaMemsetAsync(second, 0xff, sizeof(int64_t) * (nef > 0 ? nef : 1), ctx->stream));
    k_dg_second<<<nblk(nc * 6, 256), 256, 0, ctx->stream>>>(nc, m->nverts, m->d_cellvef, m->d_vowner, second);
    k_dg_nbr_unst<<<nblk(nc * 6, 256), 256, 0, ctx->stream>>>(nc, m->nverts, m->d_cellvef, m->d_vowner, second,
                                                               sp->d_dgnbr, sp->d_dgnbrface);
    FG_CUDA_TRY(cudaGetLastError());
    FG_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    dev_free(ctx, second);
  } else {
    k_dg_nbr_struct<<<nblk(nc * 6, 256), 256, 0, ctx->stream>>>(m->n[0], m->n[1], m->n[2], sp->d_dgnbr,
                                                                 sp->d_dgnbrface);
    FG_CUDA_TRY(cudaGetLastError());
  }
  FG_TRY(dev_alloc(ctx, (void**)&sp->d_rowptr, sizeof(int64_t) * (n + 1)));
  k_dg_rowlen<<<nblk(n, 256), 256, 0, ctx->stream>>>(nc, (int)nn, sp->d_dgnbr, sp->d_rowptr);
  FG_CUDA_TRY(cudaGetLastError());
  int64_t nnz = 0;
  FG_TRY(scan_i64(ctx, sp->d_rowptr, n, &nnz));
  FG_CUDA_TRY(cudaMemcpyAsync(sp->d_rowptr + n, &nnz, sizeof(int64_t), cudaMemcpyHostToDevice, ctx->stream));
  sp->nnz = nnz;
  FG_TRY(dev_alloc(ctx, (void**)&sp->d_col, sizeof(int32_t) * nnz));
  k_dg_cols<<<nblk(n, 256), 256, 0, ctx->stream>>>(nc, (int)nn, sp->d_dgnbr, sp->d_rowptr, sp->d_col);
  FG_CUDA_TRY(cudaGetLastError());
  sp->row_cap = 0;
  FG_TRY(space_count_upper(sp));
  ctx->launches += 6;
  return FG_OK;
}

// ---- solver layout ------------------------------------------------------------------------
// Cell blocks: a row holds its 7 blocks (the cell and its neighbours in ascending order, zero
// blocks on the cell itself where it has fewer) of nn columns, padded to a multiple of 4; rows in
// natural order, slices of 32, entries 4-wide per lane as in the other layouts.  A block's
// columns are consecutive, so one first column per cell and block replaces a column index per
// entry: 4 B per FP32 entry instead of 8 (196 entries per Q2 row against 192), and the rows of a
// cell gather the same addresses.
__global__ void k_dg_block_table(int64_t nc, int nn, const int32_t* nbr, int32_t* blk, int32_t* ident) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= nc) return;
  int64_t b[7];
  const int nb = dg_blocks(c, nbr, b);
  for (int k = 0; k < 8; ++k) blk[c * 8 + k] = (int32_t)((k < nb ? b[k] : c) * nn);
  for (int a = 0; a < nn; ++a) ident[c * nn + a] = (int32_t)(c * nn + a);
}

fg_status dg_space_build_layout(fg_space* sp) {
  fg_ctx* ctx = sp->mesh->ctx;
  const int64_t nc = sp->mesh->ncells, nn = sp->tab.nn;
  sp->nslices = (sp->nfree + 31) / 32;
  sp->sell_nnz = sp->nslices * 32 * 7 * ((nn + 3) / 4 * 4);
  FG_TRY(dev_alloc(ctx, (void**)&sp->d_dgblk, sizeof(int32_t) * nc * 8));
  FG_TRY(dev_alloc(ctx, (void**)&sp->d_iperm, sizeof(int32_t) * sp->nfree));
  k_dg_block_table<<<nblk(nc, 256), 256, 0, ctx->stream>>>(nc, (int)nn, sp->d_dgnbr, sp->d_dgblk, sp->d_iperm);
  FG_CUDA_TRY(cudaGetLastError());
  ctx->launches += 1;
  return FG_OK;
}

// CSR values -> cell blocks, FP64 and FP32; a block per slice (its CSR rows are one contiguous
// piece that stays in L1 over the passes)
__global__ void __launch_bounds__(256)
    k_dg_vals(int64_t n, int nn, const int64_t* __restrict__ rowptr, const double* __restrict__ val,
              double* __restrict__ sval, float* __restrict__ sval32) {
  __shared__ int64_t s_start[32];
  __shared__ int s_len[32];
  const int64_t s = blockIdx.x;
  if (threadIdx.x < 32) {
    const int64_t r = s * 32 + threadIdx.x;
    s_start[threadIdx.x] = r < n ? rowptr[r] : 0;
    s_len[threadIdx.x] = r < n ? (int)(rowptr[r + 1] - rowptr[r]) : 0;
  }
  __syncthreads();
  const int g = (nn + 3) >> 2, total = 7 * g * 32;  // groups of 4 entries
  for (int e = threadIdx.x; e < total; e += 256) {
    const int l = e & 31, gr = e >> 5, k = gr / g, b = 4 * (gr - k * g);
    double v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int j = k * nn + b + t;
      v[t] = b + t < nn && j < s_len[l] ? val[s_start[l] + j] : 0.0;
    }
    const int64_t o = (s * total + e) * 4;
    double2* d = reinterpret_cast<double2*>(sval + o);
    d[0] = make_double2(v[0], v[1]);
    d[1] = make_double2(v[2], v[3]);
    *reinterpret_cast<float4*>(sval32 + o) = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
  }
}

fg_status dg_system_fill(fg_system* sys) {
  fg_space* sp = sys->space;
  fg_ctx* ctx = sp->mesh->ctx;
  k_dg_vals<<<(unsigned)sp->nslices, 256, 0, ctx->stream>>>(sp->nfree, sp->tab.nn, sp->d_rowptr, sys->d_val,
                                                            sys->d_sval, sys->d_sval32);
  FG_CUDA_TRY(cudaGetLastError());
  ctx->launches += 1;
  return FG_OK;
}

// ---- numeric phase ------------------------------------------------------------------------
// weak Dirichlet data g at a facet point (the analytic functions of the drivers)
__device__ double dg_boundary_value(int fn, const double* prm, const double* x) {
  switch (fn) {
    case FG_FN_CONST: return prm[0];
    case FG_FN_LINEAR: return x[0] + x[1] + x[2];
    case FG_FN_SHARP_WAVE: {
      const double dx = x[0] - prm[2], dy = x[1] - prm[3], dz = x[2] - prm[4];
      return atan(prm[0] * (sqrt(dx * dx + dy * dy + dz * dz) - prm[1]));
    }
    default: return 0.0;
  }
}

struct DgParams {
  int nx, ny;             // structured lattice (vertex ids); unused on unstructured meshes
  const int32_t* cellvert;  // unstructured meshes (null on the lattice)
  double x1[4], w1[4];    // facet Gauss-Legendre rule, p+1 points
  double cip;             // 10 p^2
  int bfn;                // boundary function (weak Dirichlet data)
  double prm[8];
};

__device__ __forceinline__ int64_t dg_vertex(const DgParams& q, int64_t c, int k) {
  if (q.cellvert) return q.cellvert[c * 8 + k];
  const int64_t nx = q.nx, ny = q.ny;
  const int64_t ci = c % nx, cj = (c / nx) % ny, ck = c / (nx * ny);
  return (ci + (k & 1)) + (nx + 1) * ((cj + ((k >> 1) & 1)) + (ny + 1) * (ck + ((k >> 2) & 1)));
}

// A block owns a cell's rows.  The facet terms of its rows, in the cell's own frame of each face
// (tangential directions 0 and 1, layers l of nodes along the normal):
//  * on a face a shape function is nonzero only for the face's nodes, where it is the 2D shape
//    Phi_alpha; its gradient has the tangential parts there too and a normal part
//    L_l'(+-1) Phi_alpha in every layer;
//  * with w = w_q |J_F| J^-1 n per side (tangential w_0, w_1, normal w_n) the facet therefore needs
//    five (p+1)^2 x (p+1)^2 matrices, sums over its Gauss points of Phi_alpha(q) times
//      N: w_n Phi_beta   M: pen Phi_beta   T: w_0 d_0 Phi_beta + w_1 d_1 Phi_beta
//    and N, T of the other side (its nodes renumbered into this frame), and every entry of the
//    diagonal and neighbour blocks is a combination of at most five of their entries.
// That is ~5 (p+1)^6 FMAs per face where summing all node pairs took 8 (p+1)^8.  The geometry of
// all 6 (p+1)^2 facet points is computed at once, a thread per point and side (three threads did
// it point after point: an FP64 warp instruction holds the SM's FP64 pipe for 16 cycles however
// few lanes are active).  n |J_F| is a cofactor row of J, so no normalisation is needed.
// FP64-bound; 32^3 Q2: 66.1 -> 3.9 ms.
template <int P>
struct DgShape {
  static constexpr int NP1 = P + 1, NN = NP1 * NP1 * NP1, NQF = NP1 * NP1, NF = NQF * NQF, NG = 6 * NQF;
  static constexpr int NT = P == 1 ? 32 : (P == 2 ? 96 : 256);
  // table: Phi, d_0 Phi, d_1 Phi [node][point], L'(-1), L'(1)
  static constexpr int TAB = 3 * NF + 2 * NP1;
  // D, O, r, vertices and edge differences of 7 cells, per facet point n[3], own w[3], other
  // w[3], pen, s; five scaled tables
  static constexpr int DOUBLES = TAB + 2 * NN * NN + NN + 7 * (24 + 36) + 11 * NG + 5 * NF;
  static constexpr size_t SMEM = sizeof(double) * DOUBLES;
};

// J of the trilinear map at xi from the 12 edge differences (3 directions x 4 edges), its cofactors
// C[k][i] = det d xi_k / d x_i and determinant
__device__ __forceinline__ double dg_cofactors(const double* ed, const double* xi, double (&C)[3][3]) {
  double J[3][3];  // [d][i] = d x_i / d xi_d
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double a = xi[d == 0 ? 1 : 0], b = xi[d == 2 ? 1 : 2];
    const double am = 0.125 * (1.0 - a), ap = 0.125 * (1.0 + a), bm = 1.0 - b, bp = 1.0 + b;
    const double w[4] = {am * bm, ap * bm, am * bp, ap * bp};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      double v = 0.0;
#pragma unroll
      for (int e = 0; e < 4; ++e) v = fma(w[e], ed[d * 12 + e * 3 + i], v);
      J[d][i] = v;
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int u = (k + 1) % 3, v = (k + 2) % 3;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int x = (i + 1) % 3, y = (i + 2) % 3;
      C[k][i] = J[u][x] * J[v][y] - J[u][y] * J[v][x];
    }
  }
  return J[0][0] * C[0][0] + J[0][1] * C[0][1] + J[0][2] * C[0][2];
}
// prod_k |grad xi_k|^2
__device__ __forceinline__ double dg_grad_product(const double (&C)[3][3], double inv) {
  double s = 1.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) s *= (C[k][0] * C[k][0] + C[k][1] * C[k][1] + C[k][2] * C[k][2]) * (inv * inv);
  return s;
}

template <int P>
__global__ void __launch_bounds__(DgShape<P>::NT)
    k_dg_rows(int64_t nc, DgParams q, const double* __restrict__ table, const double* __restrict__ coords,
              const int32_t* __restrict__ nbr, const int8_t* __restrict__ nbrface, const double* __restrict__ E,
              const double* __restrict__ EV, const int64_t* __restrict__ rowptr, double* __restrict__ val,
              float* __restrict__ val32, double* __restrict__ rhs) {
  using S = DgShape<P>;
  constexpr int NP1 = S::NP1, NN = S::NN, NQF = S::NQF, NF = S::NF, NG = S::NG, NT = S::NT;
  extern __shared__ double sm[];
  double* Phi = sm;             // [node][point]
  double* D0 = Phi + NF;
  double* D1 = D0 + NF;
  double* dL = D1 + NF;         // [side][layer]
  double* D = dL + 2 * NP1;
  double* O = D + NN * NN;
  double* rv = O + NN * NN;
  double* xv = rv + NN;         // [7][24]
  double* ed = xv + 7 * 24;     // [7][36]
  double* gn = ed + 7 * 36;     // [NG][3] |J_F| n, outward
  double* gw = gn + 3 * NG;     // [NG][3] own side: tangential 0, 1, normal
  double* go = gw + 3 * NG;     // [NG][3] other side in this frame
  double* gp = go + 3 * NG;     // [NG] pen
  double* gs = gp + NG;         // [NG] gradient product of the own side; boundary value
  double* pre = gs + NG;        // [5][node][point]
  __shared__ int s_o[6], s_ax[6], s_k[6];  // neighbour, packed orientation, block of the neighbour
  __shared__ int s_nb, s_kc;
  const int tid = threadIdx.x;
  const int64_t c = blockIdx.x;
  for (int i = tid; i < S::TAB; i += NT) sm[i] = table[i];
  for (int i = tid; i < NN * NN; i += NT) D[i] = E[(size_t)c * NN * NN + i];
  for (int i = tid; i < NN; i += NT) rv[i] = EV[c * NN + i];
  // orientation of each neighbour: its face axes in this cell's face frame, through the shared corners
  if (tid < 6) {
    const int lf = tid;
    const int64_t o = nbr[c * 6 + lf];
    int packed = 0;
    if (o >= 0) {
      int d1, d2, dn, a, r1, r2, rn, ra;
      dg_face(lf, d1, d2, dn, a);
      dg_face(nbrface[c * 6 + lf], r1, r2, rn, ra);
      int M[3];
      for (int bs = 0; bs < 3; ++bs) {  // corners (0,0), (1,0), (0,1) of the neighbour's face
        const int64_t gv = dg_vertex(q, o, ra | ((bs & 1) << r1) | ((bs >> 1) << r2));
        M[bs] = 0;
        for (int bl = 0; bl < 4; ++bl)
          if (dg_vertex(q, c, a | ((bl & 1) << d1) | ((bl >> 1) << d2)) == gv) M[bs] = bl;
      }
      const int ax0 = ((M[0] ^ M[1]) & 1) ? 0 : 1, ax1 = ((M[0] ^ M[2]) & 1) ? 0 : 1;
      // bits: axis of r1, axis of r2, flips, neighbour's local face
      packed = ax0 | (ax1 << 1) | (((M[0] >> ax0) & 1) << 2) | (((M[0] >> ax1) & 1) << 3) | (nbrface[c * 6 + lf] << 4);
    }
    s_o[lf] = (int)o;
    s_ax[lf] = packed;
  }
  for (int t = tid; t < 7 * 24; t += NT) {
    const int m = t / 24, k = (t % 24) / 3, l = t % 3;
    const int64_t cc = m == 0 ? c : nbr[c * 6 + m - 1];
    xv[t] = cc >= 0 ? coords[dg_vertex(q, cc, k) * 3 + l] : 0.0;
  }
  if (tid == 0) {
    int64_t blk[7];
    const int nb = dg_blocks(c, nbr, blk);
    for (int k = 0; k < nb; ++k) {
      if (blk[k] == c) s_kc = k;
      for (int lf = 0; lf < 6; ++lf)
        if (nbr[c * 6 + lf] == blk[k]) s_k[lf] = k;
    }
    s_nb = nb;
  }
  __syncthreads();
  for (int t = tid; t < 7 * 36; t += NT) {
    const int m = t / 36, d = (t % 36) / 12, e = (t % 12) / 3, l = t % 3;
    const int p1 = d == 0 ? 1 : 0, p2 = d == 2 ? 1 : 2;
    const int lo = ((e & 1) << p1) | ((e >> 1) << p2);
    ed[t] = xv[m * 24 + (lo | (1 << d)) * 3 + l] - xv[m * 24 + lo * 3 + l];
  }
  __syncthreads();
  // own side of every facet point
  for (int t = tid; t < NG; t += NT) {
    const int lf = t / NQF, qp = t % NQF;
    int d1, d2, dn, a;
    dg_face(lf, d1, d2, dn, a);
    const double u0 = q.x1[qp % NP1], u1 = q.x1[qp / NP1], wq = q.w1[qp % NP1] * q.w1[qp / NP1];
    const bool side = (a >> dn) & 1, boundary = s_o[lf] < 0;
    double xi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) xi[d] = d == d1 ? u0 : (d == d2 ? u1 : (side ? 1.0 : -1.0));
    double C[3][3];
    const double det = dg_cofactors(ed, xi, C);
    const double inv = 1.0 / det;
    const double sg = side == (det > 0.0) ? 1.0 : -1.0;  // outward
    double n[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      n[i] = sg * (dn == 0 ? C[0][i] : (dn == 1 ? C[1][i] : C[2][i]));
      gn[t * 3 + i] = n[i];
    }
    const double f = (boundary ? wq : 0.5 * wq) * inv;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double w = f * (C[k][0] * n[0] + C[k][1] * n[1] + C[k][2] * n[2]);
      gw[t * 3 + (k == d1 ? 0 : (k == d2 ? 1 : 2))] = w;
    }
    const double s = dg_grad_product(C, inv);
    // C_IP / h = C_IP / 2 (prod |grad xi|)^(1/3)
    if (boundary) {
      gp[t] = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]) * wq * (0.5 * q.cip) * cbrt(sqrt(s));
      double x[3] = {0.0, 0.0, 0.0};
      for (int k = 0; k < 4; ++k) {
        const int v = a | ((k & 1) << d1) | ((k >> 1) << d2);
        const double fs = 0.5 * ((k & 1) ? 1.0 + u0 : 1.0 - u0), ft = 0.5 * ((k & 2) ? 1.0 + u1 : 1.0 - u1);
        for (int l = 0; l < 3; ++l) x[l] = x[l] + fs * ft * xv[v * 3 + l];
      }
      gs[t] = dg_boundary_value(q.bfn, q.prm, x);
    } else {
      gs[t] = s;
    }
  }
  __syncthreads();
  // other side of every interior facet point
  for (int t = tid; t < NG; t += NT) {
    const int lf = t / NQF, qp = t % NQF;
    if (s_o[lf] < 0) continue;
    const int pk = s_ax[lf], ax0 = pk & 1, ax1 = (pk >> 1) & 1;
    int r1, r2, rn, ra;
    dg_face(pk >> 4, r1, r2, rn, ra);
    const double u[2] = {q.x1[qp % NP1], q.x1[qp / NP1]}, wq = q.w1[qp % NP1] * q.w1[qp / NP1];
    const double f1 = (pk & 4) ? -1.0 : 1.0, f2 = (pk & 8) ? -1.0 : 1.0;
    const double v1 = f1 * (ax0 ? u[1] : u[0]), v2 = f2 * (ax1 ? u[1] : u[0]), vn = ((ra >> rn) & 1) ? 1.0 : -1.0;
    double xi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) xi[d] = d == r1 ? v1 : (d == r2 ? v2 : vn);
    double C[3][3];
    const double det = dg_cofactors(ed + (lf + 1) * 36, xi, C);
    const double inv = 1.0 / det;
    const double n0 = gn[t * 3], n1 = gn[t * 3 + 1], n2 = gn[t * 3 + 2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double w = 0.5 * wq * inv * (C[k][0] * n0 + C[k][1] * n1 + C[k][2] * n2);
      if (k == r1) go[t * 3 + ax0] = f1 * w;
      else if (k == r2) go[t * 3 + ax1] = f2 * w;
      else go[t * 3 + 2] = w;
    }
    const double s = fmax(gs[t], dg_grad_product(C, inv));  // h = min over the two cells
    gp[t] = sqrt(n0 * n0 + n1 * n1 + n2 * n2) * wq * (0.5 * q.cip) * cbrt(sqrt(s));
  }
  __syncthreads();
  const int nb = s_nb;
  const int64_t row0 = rowptr[c * NN];
  const int st[3] = {1, NP1, NP1 * NP1};
  for (int lf = 0; lf < 6; ++lf) {
    int d1, d2, dn, a;
    dg_face(lf, d1, d2, dn, a);
    const int side = (a >> dn) & 1, fl = side ? P : 0;
    const bool boundary = s_o[lf] < 0;
    const int g0 = lf * NQF;
    const int sd1 = st[d1], sd2 = st[d2], sdn = st[dn];
    // tables scaled by the facet's weights; the neighbour block cleared
    for (int t = tid; t < NF; t += NT) {
      const int g = g0 + t % NQF;
      const double ph = Phi[t], e0 = D0[t], e1 = D1[t];
      pre[t] = gw[g * 3 + 2] * ph;
      pre[NF + t] = gp[g] * ph;
      pre[2 * NF + t] = gw[g * 3] * e0 + gw[g * 3 + 1] * e1;
      if (!boundary) {
        pre[3 * NF + t] = go[g * 3 + 2] * ph;
        pre[4 * NF + t] = go[g * 3] * e0 + go[g * 3 + 1] * e1;
      }
    }
    if (!boundary)
      for (int t = tid; t < NN * NN; t += NT) O[t] = 0.0;
    __syncthreads();
    if (boundary) {  // right-hand side: -g (grad phi . n) + pen g phi
      for (int i = tid; i < NN; i += NT) {
        const int l = (i / sdn) % NP1, al = (i / sd1) % NP1 + NP1 * ((i / sd2) % NP1);
        double v = 0.0;
        for (int qp = 0; qp < NQF; ++qp) {
          double k = dL[side * NP1 + l] * pre[al * NQF + qp];
          if (l == fl) k += pre[2 * NF + al * NQF + qp] - pre[NF + al * NQF + qp];
          v = fma(gs[g0 + qp], k, v);
        }
        rv[i] -= v;
      }
    }
    double N[(NF + NT - 1) / NT], T[(NF + NT - 1) / NT];
    int lp = 0, s1 = 0, s2 = 0, sn = 0, side2 = 0, pk = 0;
    if (!boundary) {
      pk = s_ax[lf];
      int r1, r2, rn, ra;
      dg_face(pk >> 4, r1, r2, rn, ra);
      side2 = (ra >> rn) & 1;
      lp = side2 ? P : 0;
      s1 = st[r1]; s2 = st[r2]; sn = st[rn];
    }
    // node of this frame's tangential index in the neighbour, without its layer
    auto other = [&](int al) {
      const int b0 = al % NP1, b1 = al / NP1;
      const int x = (pk & 1) ? b1 : b0, y = (pk & 2) ? b1 : b0;
      return ((pk & 4) ? P - x : x) * s1 + ((pk & 8) ? P - y : y) * s2;
    };
#pragma unroll
    for (int r = 0; r < (NF + NT - 1) / NT; ++r) {
      const int t = tid + r * NT;
      N[r] = T[r] = 0.0;
      if (t >= NF) continue;
      const int x = t / NQF, y = t % NQF;
      double M = 0.0, NO = 0.0, TO = 0.0;
      for (int qp = 0; qp < NQF; ++qp) {
        const double ph = Phi[x * NQF + qp];
        const double* pr = pre + y * NQF + qp;
        N[r] = fma(ph, pr[0], N[r]);
        M = fma(ph, pr[NF], M);
        T[r] = fma(ph, pr[2 * NF], T[r]);
        if (!boundary) {
          NO = fma(ph, pr[3 * NF], NO);
          TO = fma(ph, pr[4 * NF], TO);
        }
      }
      // rows of face node x, columns of node (l, y)
      const int ix = fl * sdn + (x % NP1) * sd1 + (x / NP1) * sd2;
      const int jy = (y % NP1) * sd1 + (y / NP1) * sd2;
#pragma unroll
      for (int l = 0; l < NP1; ++l) {
        double v = dL[side * NP1 + l] * N[r];
        if (l == fl) v += T[r] - M;
        D[ix * NN + jy + l * sdn] -= v;
      }
      if (!boundary) {
        const int oy = other(y);
#pragma unroll
        for (int l = 0; l < NP1; ++l) {
          double v = dL[side2 * NP1 + l] * NO;
          if (l == lp) v += TO + M;
          O[ix * NN + oy + l * sn] = -v;
        }
      }
    }
    __syncthreads();
    // the transposed terms: rows of node (l, y), columns of face node x
#pragma unroll
    for (int r = 0; r < (NF + NT - 1) / NT; ++r) {
      const int t = tid + r * NT;
      if (t >= NF) continue;
      const int x = t / NQF, y = t % NQF;
      const int jx = (x % NP1) * sd1 + (x / NP1) * sd2 + fl * sdn;
      const int iy = (y % NP1) * sd1 + (y / NP1) * sd2;
      const int ox = boundary ? 0 : other(x) + lp * sn;
#pragma unroll
      for (int l = 0; l < NP1; ++l) {
        double v = dL[side * NP1 + l] * N[r];
        if (l == fl) v += T[r];
        const int i = iy + l * sdn;
        D[i * NN + jx] -= v;
        if (!boundary) O[i * NN + ox] = l == fl ? O[i * NN + ox] + v : v;
      }
    }
    __syncthreads();
    if (!boundary) {
      const int k = s_k[lf];
      for (int t = tid; t < NN * NN; t += NT) {
        const int i = t / NN, j = t - i * NN;
        const int64_t pos = row0 + ((int64_t)i * nb + k) * NN + j;
        val[pos] = O[t];
        if (val32) val32[pos] = (float)O[t];
      }
      __syncthreads();
    }
  }
  for (int t = tid; t < NN * NN; t += NT) {
    const int i = t / NN, j = t - i * NN;
    const int64_t pos = row0 + ((int64_t)i * nb + s_kc) * NN + j;
    val[pos] = D[t];
    if (val32) val32[pos] = (float)D[t];
  }
  for (int i = tid; i < NN; i += NT) rhs[c * NN + i] = rv[i];
}

template <int P>
static fg_status launch_dg_rows(fg_system* sys) {
  using S = DgShape<P>;
  fg_space* sp = sys->space;
  fg_mesh* m = sp->mesh;
  fg_ctx* ctx = m->ctx;
  DgParams q;
  q.nx = m->n[0];
  q.ny = m->n[1];
  q.cellvert = m->unst ? m->d_cellvert : nullptr;
  gl_rule(P + 1, q.x1, q.w1);
  q.cip = 10.0 * P * P;
  q.bfn = sys->integ.boundary_fn;
  for (int i = 0; i < 8; ++i) q.prm[i] = sys->integ.fn_param[i];
  if (!sp->d_dgtab) {
    // 2D shapes of a face and their derivatives at its Gauss points, and L_l'(-1), L_l'(1)
    std::vector<double> h(S::TAB);
    double v[4][4], dv[4][4];
    for (int j = 0; j <= P; ++j)
      for (int k = 0; k <= P; ++k) lagrange_1d(P, j, q.x1[k], v[j][k], dv[j][k]);
    for (int al = 0; al < S::NQF; ++al)
      for (int qp = 0; qp < S::NQF; ++qp) {
        const int a0 = al % S::NP1, a1 = al / S::NP1, q0 = qp % S::NP1, q1 = qp / S::NP1;
        h[al * S::NQF + qp] = v[a0][q0] * v[a1][q1];
        h[S::NF + al * S::NQF + qp] = dv[a0][q0] * v[a1][q1];
        h[2 * S::NF + al * S::NQF + qp] = v[a0][q0] * dv[a1][q1];
      }
    for (int l = 0; l <= P; ++l) {
      double val;
      lagrange_1d(P, l, -1.0, val, h[3 * S::NF + l]);
      lagrange_1d(P, l, 1.0, val, h[3 * S::NF + S::NP1 + l]);
    }
    FG_TRY(dev_alloc(ctx, (void**)&sp->d_dgtab, sizeof(double) * h.size()));
    FG_CUDA_TRY(cudaMemcpyAsync(sp->d_dgtab, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice, ctx->stream));
    FG_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  }
  FG_CUDA_TRY(cudaFuncSetAttribute((const void*)k_dg_rows<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
  k_dg_rows<P><<<(unsigned)m->ncells, S::NT, S::SMEM, ctx->stream>>>(
      m->ncells, q, sp->d_dgtab, m->d_coords, sp->d_dgnbr, sp->d_dgnbrface, sys->d_elmat, sys->d_elvec, sp->d_rowptr, sys->d_val,
      sys->d_val32, sys->d_rhs);
  ctx->launches += 1;
  FG_CUDA_TRY(cudaGetLastError());
  return FG_OK;
}

fg_status dg_assemble_rows(fg_system* sys) {
  switch (sys->space->order) {
    case 1: return launch_dg_rows<1>(sys);
    case 2: return launch_dg_rows<2>(sys);
    case 3: return launch_dg_rows<3>(sys);
    default: set_error("dG order %d not built", sys->space->order); return FG_ERR_UNSUPPORTED;
  }
}

}  // namespace fg
