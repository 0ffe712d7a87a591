// Thermal diffusion half step (diffusion3d_p.m with the reference's default options): linear
// elements on the 8-child split of every P2 tetrahedron, double-Jacobian element integrals,
// lumped capacity, theta scheme, Dirichlet temperatures, Jacobi-preconditioned Polak-Ribiere CG.
//
// Layout: split elements `sub` [4][nsub] (node ids), packed conductivity C [10][nsub] (entries (i,j), i >= j,
// in the order 00 10 11 20 21 22 30 31 32 33) and a node -> (local, element) list in element order. The
// conductivity is assembled into rows (node -> neighbour columns, values) once per set-up: a product then
// reads 12 B per nonzero, about 15 a node, where the element form read and wrote 160 B per split element,
// about 6 a node (98 us per product at 338k nodes; now 29 us). Sums run in a fixed order, no atomics.
//
// The CG keeps its scalars on the device: three launches per iteration (direction; product and q.Aq; step
// with r.r and the dots of the next direction), whose kernels do nothing once a flag says that the
// iteration has ended, so the host looks at it every DIFF_CHECK iterations only (it read four scalars per
// iteration, each a wait).
#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "common.cuh"

namespace m3sph {

unsigned red_blocks(size_t n);
const double *slm_x90(m3sph_mesh *M);

// children of a P2 tetrahedron (local node numbers 0..9) for the three interior diagonals, and the
// diagonals' end nodes (tetmesh_p2_to_p1.m): the table that the reference's split follows
static const int EL2CHILD[3][8][4] = {
    {{0, 4, 8, 7}, {4, 1, 5, 9}, {8, 5, 2, 6}, {7, 9, 6, 3}, {9, 7, 6, 4}, {5, 8, 4, 6}, {7, 6, 4, 8}, {9, 4, 6, 5}},
    {{0, 4, 8, 7}, {4, 1, 5, 9}, {8, 5, 2, 6}, {7, 9, 6, 3}, {4, 8, 7, 5}, {9, 6, 5, 7}, {8, 7, 5, 6}, {4, 5, 7, 9}},
    {{0, 4, 8, 7}, {4, 1, 5, 9}, {8, 5, 2, 6}, {7, 9, 6, 3}, {7, 4, 8, 9}, {6, 5, 9, 8}, {4, 8, 9, 5}, {8, 9, 6, 7}}};
static const int DIAG2NOD[3][2] = {{4, 6}, {5, 7}, {8, 9}};

struct DiffState {
  int nsub = 0, nnod = 0, nfix = 0;
  double kappa = 0.0, theta = 1.0, tol = 1e-8;
  int itmax = 500;
  int *sub = nullptr;                  // [4][nsub]
  uint8_t *cls = nullptr;              // [nsub]
  double *C = nullptr;                 // [10][nsub]
  double *Me = nullptr;                // [4][nsub] lumped element capacities
  int *gptr = nullptr, *gidx = nullptr;  // [nnod+1], [4 nsub]: local * nsub + element
  // rows of the assembled conductivity, columns sorted: entry k of row n is at sptr[n / 32] + 32 k + n % 32
  int *sptr = nullptr, *rlen = nullptr, *rcol = nullptr;  // [slices of 32 rows], [nnod], [padded nonzeros]
  double *rval = nullptr;              // [padded nonzeros]
  double *ML = nullptr, *Cdiag = nullptr, *Mi = nullptr;  // [nnod]; Mi: inverse diagonal, 0 on fixed nodes
  uint8_t *fixmask = nullptr;          // [nnod]
  int *ifix = nullptr;                 // [nfix]
  double *vfix = nullptr;              // [nfix]
  double *rhs = nullptr, *r = nullptr, *q = nullptr, *Aq = nullptr, *T = nullptr;
  int fixcap = 0;
  double *scal = nullptr;              // CG scalars (DS_*)
  int *err = nullptr;
  bool ready = false;                  // a set-up has run to its end
};

static DiffState *diff_state(m3sph_mesh *M) { return reinterpret_cast<DiffState *>(M->diff); }

static void diff_free(void *p) {
  DiffState *D = reinterpret_cast<DiffState *>(p);
  for (void *q : {(void *)D->sub, (void *)D->cls, (void *)D->C, (void *)D->Me, (void *)D->gptr, (void *)D->gidx,
                  (void *)D->sptr, (void *)D->rlen, (void *)D->rcol, (void *)D->rval, (void *)D->ML, (void *)D->Mi, (void *)D->Cdiag, (void *)D->fixmask,
                  (void *)D->ifix, (void *)D->vfix, (void *)D->rhs, (void *)D->r, (void *)D->q, (void *)D->Aq,
                  (void *)D->T, (void *)D->scal, (void *)D->err})
    if (q) cudaFree(q);
  delete D;
}

// element integrals of one split element (assembly_diffusion_els_*_opt.m): vertex (theta, phi, r)
// in the element's frame (X-90 coordinates from the location tables), J_SL from them, J_CS at each of the 4
// points of ip_tetrahedron(4). FP64 issue bounds it, so the gradients are multiplied in the spherical basis,
// where the metric is diagonal and the linear element's derivatives are constant: 3.7 ms at 2.0M split elements
// with Cartesian gradients at every point and the X-90 frame formed per element; now 0.82 ms.
__global__ void k_diff_setup(int nsub, const int *__restrict__ sub, const uint8_t *__restrict__ cls,
                             const double *__restrict__ SX, const double *__restrict__ S, int nnod, double kappa,
                             double *__restrict__ C, double *__restrict__ Me, int *err) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nsub) return;
  const int c = cls[e];
  double V[3][4];
  for (int i = 0; i < 4; ++i) {
    const int n = sub[(size_t)i * nsub + e];
    if (c <= 1) {
      V[0][i] = S[n];
      V[1][i] = S[nnod + n];
      V[2][i] = S[2 * (size_t)nnod + n];
      if (c == 1) {
        V[1][i] += M_PI;
        if (V[1][i] > 2.0 * M_PI) V[1][i] -= 2.0 * M_PI;
      }
    } else {   // X-90-rotated frame: (x, -z, y)
      V[0][i] = SX[n];
      V[1][i] = SX[nnod + n];
      V[2][i] = SX[2 * (size_t)nnod + n];
    }
  }
  // J_SL[j][k] = d sph_k / d loc_j with dN4 = [I; -1 -1 -1]
  double J[3][3];
  for (int j = 0; j < 3; ++j)
    for (int k = 0; k < 3; ++k) J[j][k] = V[k][j] - V[k][3];
  const double det = J[0][0] * (J[1][1] * J[2][2] - J[1][2] * J[2][1]) - J[0][1] * (J[1][0] * J[2][2] - J[1][2] * J[2][0]) +
                     J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
  if (det < 0.0) atomicOr(err, 1);
  // cofactors: d N_i / d sph_k = cf[k][i] / det, constant over the element (sum_i = 0)
  double cf[3][4];
  cf[0][0] = J[1][1] * J[2][2] - J[1][2] * J[2][1];
  cf[0][1] = J[0][2] * J[2][1] - J[0][1] * J[2][2];
  cf[0][2] = J[0][1] * J[1][2] - J[0][2] * J[1][1];
  cf[1][0] = J[1][2] * J[2][0] - J[1][0] * J[2][2];
  cf[1][1] = J[0][0] * J[2][2] - J[0][2] * J[2][0];
  cf[1][2] = J[0][2] * J[1][0] - J[0][0] * J[1][2];
  cf[2][0] = J[1][0] * J[2][1] - J[1][1] * J[2][0];
  cf[2][1] = J[0][1] * J[2][0] - J[0][0] * J[2][1];
  cf[2][2] = J[0][0] * J[1][1] - J[0][1] * J[1][0];
#pragma unroll
  for (int k = 0; k < 3; ++k) cf[k][3] = -(cf[k][0] + cf[k][1] + cf[k][2]);
  // det J_CS = r^2 sin(theta) and grad N_i . grad N_j = d_r d_r + d_th d_th / r^2 + d_ph d_ph / (r sin(theta))^2:
  // the points enter through three sums only
  const double a = (5.0 + 3.0 * sqrt(5.0)) / 20.0, b = (5.0 - sqrt(5.0)) / 20.0;
  const double bt = b * (V[0][0] + V[0][1] + V[0][2] + V[0][3]), br = b * (V[2][0] + V[2][1] + V[2][2] + V[2][3]);
  double st[4], wp[4];
#pragma unroll
  for (int ip = 0; ip < 4; ++ip) {
    const double th = bt + (a - b) * V[0][ip], rr = br + (a - b) * V[2][ip];
    if (th == 0.0) atomicOr(err, 2);
    st[ip] = sin(th);
    wp[ip] = rr * rr * st[ip];
  }
  const double hr = wp[0] + wp[1] + wp[2] + wp[3], ht = st[0] + st[1] + st[2] + st[3];
  const double s01 = st[0] * st[1], s23 = st[2] * st[3];
  const double hp = ((st[0] + st[1]) * s23 + (st[2] + st[3]) * s01) / (s01 * s23);   // sum of 1 / sin(theta)
  const double f = 0.25 * kappa / det;
  const double h[3] = {f * ht, f * hp, f * hr};
  double Cp[10], Ml[4];
  int k = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double a0 = h[0] * cf[0][i], a1 = h[1] * cf[1][i], a2 = h[2] * cf[2][i];
#pragma unroll
    for (int j = 0; j <= i; ++j, ++k) Cp[k] = a0 * cf[0][j] + a1 * cf[1][j] + a2 * cf[2][j];
    Ml[i] = 0.25 * det * (b * hr + (a - b) * wp[i]);   // row sum of w N_i N_j (sum_j N_j = 1)
  }
  for (int k = 0; k < 10; ++k) C[(size_t)k * nsub + e] = Cp[k];
  for (int i = 0; i < 4; ++i) Me[(size_t)i * nsub + e] = Ml[i];
}

__device__ __forceinline__ int pk(int i, int j) { return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i; }

// lumped capacity: per node the sum of its elements' values in element order
__global__ void k_diff_lump(int nnod, const int *__restrict__ gptr, const int *__restrict__ gidx,
                            const double *__restrict__ Me, double *__restrict__ ML) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nnod) return;
  double s = 0.0;
  for (int k = gptr[n]; k < gptr[n + 1]; ++k) s += Me[gidx[k]];
  ML[n] = s;
}

// Row pattern, one warp per node: its neighbours (itself included) through a hash table in shared memory.
// With rcol null the row lengths; then the columns, sorted. At most 128 elements share a vertex (the mesh
// set-up's colour limit), so a node of the split has fewer than 400 neighbours.
constexpr int DP_WARPS = 4, DP_TAB = 1024;
__global__ void __launch_bounds__(DP_WARPS * 32) k_diff_pattern(int nnod, int nsub, const int *__restrict__ sub,
                                                                const int *__restrict__ gptr, const int *__restrict__ gidx,
                                                                int *__restrict__ rlen, const int *__restrict__ sptr,
                                                                int *__restrict__ rcol) {
  __shared__ int tab[DP_WARPS][DP_TAB];
  __shared__ int list[DP_WARPS][DP_TAB];
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * DP_WARPS + wl;
  if (n >= nnod) return;
  int *h = tab[wl], *out = list[wl];
  for (int i = lane; i < DP_TAB; i += 32) h[i] = -1;
  __syncwarp();
  const int b = gptr[n], m = 4 * (gptr[n + 1] - b);
  for (int t = lane; t < m; t += 32) {
    const int e = gidx[b + (t >> 2)] % nsub, v = sub[(size_t)(t & 3) * nsub + e];
    int s = (int)(((unsigned)v * 2654435761u) >> 22);
    for (int probe = 0; probe < DP_TAB; ++probe) {
      const int old = atomicCAS(&h[s], -1, v);
      if (old == -1 || old == v) break;
      s = (s + 1) & (DP_TAB - 1);
    }
  }
  __syncwarp();
  int cnt = 0;
  for (int i = lane; i < DP_TAB; i += 32) {
    const int v = h[i];
    const unsigned mask = __ballot_sync(0xffffffffu, v >= 0);
    if (v >= 0) out[cnt + __popc(mask & ((1u << lane) - 1u))] = v;
    cnt += __popc(mask);
  }
  __syncwarp();
  if (!rcol) {
    if (lane == 0) rlen[n] = cnt;
    return;
  }
  for (int i = lane; i < cnt; i += 32) {
    const int v = out[i];
    int rank = 0;
    for (int k = 0; k < cnt; ++k) rank += out[k] < v;
    rcol[(size_t)sptr[n >> 5] + 32 * rank + (n & 31)] = v;
  }
}
// Row values, 16 lanes per node: a lane sums its column's entries over the node's elements in element order.
// FP64 additions (pipe 74 % busy), L1 (63 %) and the latency of the three dependent loads per element bound it:
// 0.41 ms at 338k nodes one element at a time, 0.37 ms with four in flight
__global__ void __launch_bounds__(256) k_diff_rows(int nnod, int nsub, const int *__restrict__ sub,
                                                   const double *__restrict__ C, const int *__restrict__ gptr,
                                                   const int *__restrict__ gidx, const int *__restrict__ sptr,
                                                   const int *__restrict__ rlen, const int *__restrict__ rcol,
                                                   double *__restrict__ rval,
                                                   double *__restrict__ Cdiag) {
  const int n = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 4), lane = threadIdx.x & 15;
  if (n >= nnod) return;
  const int b = gptr[n], f = gptr[n + 1];
  const size_t r0 = (size_t)sptr[n >> 5] + (n & 31);
  const int len = rlen[n];
  for (int k = lane; k < len; k += 16) {
    const int col = rcol[r0 + 32 * k];
    double v = 0.0;
#pragma unroll 4
    for (int g = b; g < f; ++g) {
      const int o = gidx[g], i = (o >= nsub) + (o >= 2 * nsub) + (o >= 3 * nsub), e = o - i * nsub;
      int j = -1;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (sub[(size_t)q * nsub + e] == col) j = q;
      if (j >= 0) v += C[(size_t)pk(i, j) * nsub + e];
    }
    rval[r0 + 32 * k] = v;
    if (col == n) Cdiag[n] = v;
  }
}

// CG scalars on the device
enum { DS_RD = 0, DS_BETA, DS_ALPHA, DS_TOL2, DS_RR, DS_DONE, DS_IT, DS_BAD, DS_N };

// Row products, a thread per row on slices of 32 rows: s_n = sum C_nm x_m, and with it
//   DP_RHS    y = ML x + c s                                (right-hand side)
//   DP_RESID  y = rhs - (ML x + c s) on free nodes, 0 on fixed ones, q = 0, Mi = 1 / diag; r.r and the dots
//             of the first direction: the scalars of a CG from this residual
//   DP_CG     y = ML x + c s on free nodes, 0 on fixed ones; alpha = rd / x.y
// With 8 lanes per row the shuffles' additions and the one lane that finishes a row were most of the FP64
// issue: 61 us at 338k rows, 5.2M nonzeros; now 29 us.
enum { DP_RHS = 0, DP_RESID = 1, DP_CG = 2 };
template <int MODE>
__global__ void __launch_bounds__(256) k_diff_rowprod(int nnod, const int *__restrict__ sptr, const int *__restrict__ rlen,
                                                      const int *__restrict__ rcol, const double *__restrict__ rval,
                                                      const double *__restrict__ ML, const double *__restrict__ x, double c,
                                                      const uint8_t *__restrict__ fixmask, double *__restrict__ y,
                                                      const double *__restrict__ rhs, const double *__restrict__ Cdiag,
                                                      double *__restrict__ Mi, double *__restrict__ q, double tol,
                                                      double *scal, double *partials, unsigned *cnt) {
  if (MODE == DP_CG && scal[DS_DONE] != 0.0) return;
  double v[2] = {0.0, 0.0};
  for (int n = blockIdx.x * 256 + threadIdx.x; n < nnod; n += gridDim.x * 256) {
    const int len = rlen[n];
    const size_t r0 = (size_t)sptr[n >> 5] + (n & 31);
    double s = 0.0;
#pragma unroll 4
    for (int k = 0; k < len; ++k) s += rval[r0 + 32 * k] * x[rcol[r0 + 32 * k]];
    const double m = ML[n], a = m * x[n] + c * s;
    const bool fixed = MODE != DP_RHS && fixmask[n];
    if (MODE == DP_RHS) {
      y[n] = a;
    } else if (MODE == DP_RESID) {
      const double r = fixed ? 0.0 : rhs[n] - a, mi = fixed ? 0.0 : 1.0 / (m + c * Cdiag[n]);
      y[n] = r;
      Mi[n] = mi;
      q[n] = 0.0;
      v[0] += r * r;
      v[1] += r * (r * mi);
    } else {
      const double t = fixed ? 0.0 : a;
      y[n] = t;
      v[0] += x[n] * t;
    }
  }
  if (MODE == DP_RHS) return;
  if (!block_reduce_last<2>(v, partials, cnt) || threadIdx.x) return;
  if (MODE == DP_RESID) {
    // pcg_solver_p.m: the tolerance is relative to the initial residual. A residual that is exactly zero
    // (a field the step leaves unchanged) or below it is converged; a NaN one is an error
    scal[DS_RR] = v[0];
    scal[DS_TOL2] = tol * tol * v[0];
    scal[DS_RD] = v[1];
    scal[DS_BETA] = 0.0;
    scal[DS_DONE] = (v[0] < tol * tol * v[0] || v[0] == 0.0 || isnan(v[0])) ? 1.0 : 0.0;
    scal[DS_IT] = 0.0;
    scal[DS_BAD] = isnan(v[0]) ? 1.0 : 0.0;
  } else {
    scal[DS_ALPHA] = scal[DS_RD] / v[0];
  }
}
// q = d + beta q, d = r / diag on free nodes
__global__ void k_diff_dir(int n, const double *__restrict__ r, const double *__restrict__ Mi, double *__restrict__ q,
                           const double *__restrict__ scal) {
  if (scal[DS_DONE] != 0.0) return;
  const double beta = scal[DS_BETA];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    q[i] = r[i] * Mi[i] + beta * q[i];
}
// x += alpha q ; r -= alpha Aq ; then r.r and for the next direction d = r / diag: r.d and Aq.d, which give
// beta = (r - rlast).d / rdlast = -alpha Aq.d / rdlast (Polak-Ribiere)
__global__ void __launch_bounds__(256) k_diff_step(int n, const double *__restrict__ q, const double *__restrict__ Aq,
                                                   double *__restrict__ x, double *__restrict__ r,
                                                   const double *__restrict__ Mi, double *scal, int itmax,
                                                   double *partials, unsigned *cnt) {
  if (scal[DS_DONE] != 0.0) return;
  const double alpha = scal[DS_ALPHA];
  double v[3] = {0.0, 0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double a = Aq[i], ri = r[i] - alpha * a, d = ri * Mi[i];
    x[i] += alpha * q[i];
    r[i] = ri;
    v[0] += ri * ri;
    v[1] += ri * d;
    v[2] += a * d;
  }
  if (!block_reduce_last<3>(v, partials, cnt) || threadIdx.x) return;
  const double it = scal[DS_IT] + 1.0;
  scal[DS_IT] = it;
  scal[DS_RR] = v[0];
  scal[DS_BETA] = -alpha * v[2] / scal[DS_RD];
  scal[DS_RD] = v[1];
  if (isnan(v[0])) scal[DS_BAD] = 1.0;
  if (isnan(v[0]) || v[0] < scal[DS_TOL2] || it >= itmax) scal[DS_DONE] = 1.0;
}
__global__ void k_diff_setfix(const int *ifix, const double *vfix, int nfix, double *x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nfix) x[ifix[i]] = vfix[i];
}
static int dalloc_d(void **p, size_t bytes) {
  M3_CUDA(cudaMalloc(p, bytes ? bytes : 1));
  return M3SPH_OK;
}

static int diff_build(m3sph_mesh *M, DiffState *D, double theta_cone) {
  cudaStream_t s = M->stream;
  Level &L0 = M->lev[0];
  const int nel = L0.nel, nnod = L0.nnod;
  std::vector<double> X(3 * (size_t)nnod), S(3 * (size_t)nnod);
  M3_CUDA(cudaMemcpyAsync(X.data(), M->fin.gcoord, X.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
  M3_CUDA(cudaMemcpyAsync(S.data(), M->fin.gcoord_sph, S.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
  M3_CUDA(cudaStreamSynchronize(s));
  const std::vector<int> &el = L0.h_el2nod_orig;   // [nel][10]
  const size_t nsub = 8 * (size_t)nel;
  if (nsub > (size_t)(1u << 31) / 4) {
    set_error("mesh too large for the diffusion split");
    return M3SPH_ERR_BAD_INPUT;
  }
  std::vector<int> sub(4 * nsub);
  std::vector<uint8_t> cls(nsub);
  const double tc = theta_cone * M_PI / 180.0;
  for (int e = 0; e < nel; ++e) {
    const int *en = &el[(size_t)e * 10];
    // shortest interior diagonal (Cartesian), the first on ties (tetmesh_p2_to_p1.m)
    int isp = 0;
    double best = 0.0;
    for (int k = 0; k < 3; ++k) {
      const int a = en[DIAG2NOD[k][0]], b = en[DIAG2NOD[k][1]];
      double d2 = 0.0;
      for (int c = 0; c < 3; ++c) {
        const double dd = X[(size_t)c * nnod + a] - X[(size_t)c * nnod + b];
        d2 += dd * dd;
      }
      const double len = std::sqrt(d2);
      if (k == 0 || len < best) {
        best = len;
        isp = k;
      }
    }
    for (int k = 0; k < 8; ++k) {
      const size_t se = 8 * (size_t)e + k;
      int nin = 0;
      bool cross = false;
      double ph[4];
      for (int i = 0; i < 4; ++i) {
        const int n = en[EL2CHILD[isp][k][i]];
        sub[(size_t)i * nsub + se] = n;
        const double th = S[n];
        ph[i] = S[nnod + n];
        nin += (th <= tc || th >= M_PI - tc) ? 1 : 0;
      }
      const int pairs[6][2] = {{0, 1}, {1, 2}, {2, 0}, {0, 3}, {1, 3}, {2, 3}};
      for (const auto &pp : pairs) cross |= std::fabs(ph[pp[0]] - ph[pp[1]]) > M_PI;
      // check_els_in_cone.m / check_phi.m on the split elements
      cls[se] = (uint8_t)(nin == 0 ? (cross ? 1 : 0) : (nin < 3 ? 3 : 2));
    }
  }
  // node -> (local, element) entries in element order
  std::vector<int> ptr(nnod + 1, 0), idx(4 * nsub);
  for (size_t e = 0; e < nsub; ++e)
    for (int i = 0; i < 4; ++i) ptr[sub[(size_t)i * nsub + e] + 1]++;
  for (int n = 0; n < nnod; ++n) ptr[n + 1] += ptr[n];
  std::vector<int> fill(ptr.begin(), ptr.end() - 1);
  for (size_t e = 0; e < nsub; ++e)
    for (int i = 0; i < 4; ++i) idx[fill[sub[(size_t)i * nsub + e]]++] = (int)((size_t)i * nsub + e);
  D->nsub = (int)nsub;
  D->nnod = nnod;
  int st;
  if ((st = dalloc_d((void **)&D->sub, sub.size() * sizeof(int))) ||
      (st = dalloc_d((void **)&D->cls, cls.size())) || (st = dalloc_d((void **)&D->C, 10 * nsub * sizeof(double))) ||
      (st = dalloc_d((void **)&D->Me, 4 * nsub * sizeof(double))) ||
      (st = dalloc_d((void **)&D->scal, DS_N * sizeof(double))) ||
      (st = dalloc_d((void **)&D->rlen, (size_t)nnod * sizeof(int))) ||
      (st = dalloc_d((void **)&D->sptr, ((size_t)nnod + 31) / 32 * sizeof(int))) ||
      (st = dalloc_d((void **)&D->gptr, ptr.size() * sizeof(int))) ||
      (st = dalloc_d((void **)&D->gidx, idx.size() * sizeof(int))) ||
      (st = dalloc_d((void **)&D->ML, nnod * sizeof(double))) || (st = dalloc_d((void **)&D->Cdiag, nnod * sizeof(double))) ||
      (st = dalloc_d((void **)&D->fixmask, nnod)) || (st = dalloc_d((void **)&D->err, sizeof(int))))
    return st;
  for (double **p : {&D->Mi, &D->rhs, &D->r, &D->q, &D->Aq, &D->T})
    if ((st = dalloc_d((void **)p, nnod * sizeof(double)))) return st;
  M3_CUDA(cudaMemcpyAsync(D->sub, sub.data(), sub.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  M3_CUDA(cudaMemcpyAsync(D->cls, cls.data(), cls.size(), cudaMemcpyHostToDevice, s));
  M3_CUDA(cudaMemcpyAsync(D->gptr, ptr.data(), ptr.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  M3_CUDA(cudaMemcpyAsync(D->gidx, idx.data(), idx.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  // row pattern: lengths, starts of the slices (on the host), columns
  const unsigned g = (unsigned)((nnod + DP_WARPS - 1) / DP_WARPS);
  k_diff_pattern<<<g, DP_WARPS * 32, 0, s>>>(nnod, D->nsub, D->sub, D->gptr, D->gidx, D->rlen, nullptr, nullptr); count_launch();
  M3_CUDA(cudaGetLastError());
  std::vector<int> rlen(nnod), sptr((nnod + 31) / 32);
  M3_CUDA(cudaMemcpyAsync(rlen.data(), D->rlen, nnod * sizeof(int), cudaMemcpyDeviceToHost, s));
  M3_CUDA(cudaStreamSynchronize(s));
  size_t nnz = 0;
  for (size_t b = 0; b < sptr.size(); ++b) {
    sptr[b] = (int)nnz;
    nnz += 32 * (size_t)*std::max_element(rlen.begin() + 32 * b, rlen.begin() + std::min<size_t>(nnod, 32 * b + 32));
    if (nnz > 2147483647ull) {
      set_error("mesh too large for the diffusion rows");
      return M3SPH_ERR_BAD_INPUT;
    }
  }
  if ((st = dalloc_d((void **)&D->rcol, nnz * sizeof(int))) || (st = dalloc_d((void **)&D->rval, nnz * sizeof(double))))
    return st;
  M3_CUDA(cudaMemcpyAsync(D->sptr, sptr.data(), sptr.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  k_diff_pattern<<<g, DP_WARPS * 32, 0, s>>>(nnod, D->nsub, D->sub, D->gptr, D->gidx, nullptr, D->sptr, D->rcol); count_launch();
  M3_CUDA(cudaGetLastError());
  M3_CUDA(cudaStreamSynchronize(s));
  return M3SPH_OK;
}

// element integrals, lumped capacity and conductivity diagonal for the diffusivity kappa
static int diff_integrate(m3sph_mesh *M, DiffState *D) {
  cudaStream_t s = M->stream;
  const int nsub = D->nsub, nnod = D->nnod;
  M3_CUDA(cudaMemsetAsync(D->err, 0, sizeof(int), s));
  k_diff_setup<<<(nsub + 127) / 128, 128, 0, s>>>(nsub, D->sub, D->cls, slm_x90(M), M->fin.gcoord_sph, nnod, D->kappa, D->C,
                                                  D->Me, D->err); count_launch();
  k_diff_lump<<<(nnod + 127) / 128, 128, 0, s>>>(nnod, D->gptr, D->gidx, D->Me, D->ML); count_launch();
  k_diff_rows<<<(unsigned)(((size_t)nnod * 16 + 255) / 256), 256, 0, s>>>(nnod, nsub, D->sub, D->C, D->gptr, D->gidx, D->sptr,
                                                                         D->rlen, D->rcol, D->rval, D->Cdiag); count_launch();
  M3_CUDA(cudaGetLastError());
  int herr = 0;
  M3_CUDA(cudaMemcpyAsync(&herr, D->err, sizeof(int), cudaMemcpyDeviceToHost, s));
  M3_CUDA(cudaStreamSynchronize(s));
  if (herr & 1) {
    set_error("negative Jacobi");
    return M3SPH_ERR_NEGATIVE_JACOBIAN;
  }
  if (herr & 2) {
    set_error("integration point with theta = 0 (det(J_CS) = Inf)");
    return M3SPH_ERR_BAD_INPUT;
  }
  return M3SPH_OK;
}

// one diffusion3d_p step on the device-resident T (nnod) over dt; *nit = PCG iterations
int diffusion_resident(m3sph_mesh *M, double *T, double dt, int *nit) {
  DiffState *D = diff_state(M);
  if (!D || !D->ready) {
    set_error("diffusion not set up (call m3sph_diffusion_setup)");
    return M3SPH_ERR_BAD_INPUT;
  }
  cudaStream_t s = M->stream;
  const int n = D->nnod;
  const double c = dt * D->theta;
  const unsigned gr = (unsigned)std::min((n + 255) / 256, 2048);   // two partial sums per block
  // rhs = M T - dt (1 - theta) C T (diffusion3d_p.m:96-97)
  k_diff_rowprod<DP_RHS><<<gr, 256, 0, s>>>(n, D->sptr, D->rlen, D->rcol, D->rval, D->ML, T, -dt * (1.0 - D->theta), nullptr,
                                            D->rhs, nullptr, nullptr, nullptr, nullptr, 0.0, nullptr, nullptr,
                                            nullptr); count_launch();
  // T(ifix) = vfix; r = rhs - A T on the free rows (A(:,ifix) vfix moves to the rhs through T)
  if (D->nfix) {
    k_diff_setfix<<<(D->nfix + 255) / 256, 256, 0, s>>>(D->ifix, D->vfix, D->nfix, T); count_launch();
  }
  k_diff_rowprod<DP_RESID><<<gr, 256, 0, s>>>(n, D->sptr, D->rlen, D->rcol, D->rval, D->ML, T, c, D->fixmask, D->r, D->rhs,
                                              D->Cdiag, D->Mi, D->q, D->tol, D->scal, M->red, M->red_cnt); count_launch();
  // iterations are launched DIFF_CHECK at a time; those past the end do nothing
  constexpr int DIFF_CHECK = 6;
  double h[DS_N];
  for (int it = 0;; it += DIFF_CHECK) {
    M3_CUDA(cudaGetLastError());
    M3_CUDA(cudaMemcpyAsync(h, D->scal, sizeof(h), cudaMemcpyDeviceToHost, s));
    M3_CUDA(cudaStreamSynchronize(s));
    if (h[DS_DONE] != 0.0) break;
    for (int k = 0; k < DIFF_CHECK; ++k) {
      k_diff_dir<<<red_blocks(n), 256, 0, s>>>(n, D->r, D->Mi, D->q, D->scal); count_launch();
      k_diff_rowprod<DP_CG><<<gr, 256, 0, s>>>(n, D->sptr, D->rlen, D->rcol, D->rval, D->ML, D->q, c, D->fixmask, D->Aq,
                                               nullptr, nullptr, nullptr, nullptr, 0.0, D->scal, M->red,
                                               M->red_cnt); count_launch();
      k_diff_step<<<red_blocks(n), 256, 0, s>>>(n, D->q, D->Aq, T, D->r, D->Mi, D->scal, D->itmax, M->red,
                                                M->red_cnt); count_launch();
    }
  }
  if (h[DS_BAD] != 0.0) {
    set_error("NaN in the diffusion solve");
    return M3SPH_ERR_NAN;
  }
  if (nit) *nit = (int)h[DS_IT];
  return M3SPH_OK;
}

}  // namespace m3sph

using namespace m3sph;

extern "C" int m3sph_diffusion_setup(m3sph_mesh *M, const m3sph_diffusion_opts *o, const int32_t *ifix,
                                     const double *vfix, int32_t nfix) {
  if (!M || !o || nfix < 0 || (nfix > 0 && (!ifix || !vfix)) || !(o->kappa >= 0.0)) {
    set_error("m3sph_diffusion_setup: bad arguments");
    return M3SPH_ERR_BAD_INPUT;
  }
  M3_CUDA(cudaSetDevice(M->device));
  cudaStream_t s = M->stream;
  // the list is checked first: a set-up refused for it leaves an earlier one as it was
  const int nnod = M->lev[0].nnod;
  std::vector<int> fx(nfix);
  std::vector<uint8_t> mask(nnod, 0);
  for (int i = 0; i < nfix; ++i) {
    if (ifix[i] < 1 || ifix[i] > nnod) {
      set_error("m3sph_diffusion_setup: ifix entry out of range");
      return M3SPH_ERR_BAD_INPUT;
    }
    fx[i] = ifix[i] - 1;
    mask[fx[i]] = 1;
  }
  DiffState *D = diff_state(M);
  if (!D) {
    // a state that could not be built is not kept, so that no later call takes it for a set-up
    D = new DiffState();
    const int st = diff_build(M, D, o->theta_cone > 0 ? o->theta_cone : 45.0);
    if (st) {
      diff_free(D);
      return st;
    }
    M->diff = D;
    M->diff_free = diff_free;
  }
  D->ready = false;                    // until every array below holds this set-up
  D->kappa = o->kappa;
  D->theta = o->theta;
  D->tol = o->tol > 0 ? o->tol : 1e-8;
  D->itmax = o->itmax > 0 ? o->itmax : 500;
  D->nfix = nfix;
  if (nfix > D->fixcap || !D->ifix) {
    if (D->ifix) cudaFree(D->ifix);
    if (D->vfix) cudaFree(D->vfix);
    D->ifix = nullptr;
    D->vfix = nullptr;
    D->fixcap = std::max(1, nfix);
    M3_TRY(dalloc_d((void **)&D->ifix, D->fixcap * sizeof(int)));
    M3_TRY(dalloc_d((void **)&D->vfix, D->fixcap * sizeof(double)));
  }
  if (nfix) {
    M3_CUDA(cudaMemcpyAsync(D->ifix, fx.data(), nfix * sizeof(int), cudaMemcpyHostToDevice, s));
    M3_CUDA(cudaMemcpyAsync(D->vfix, vfix, nfix * sizeof(double), cudaMemcpyHostToDevice, s));
  }
  M3_CUDA(cudaMemcpyAsync(D->fixmask, mask.data(), D->nnod, cudaMemcpyHostToDevice, s));
  M3_TRY(diff_integrate(M, D));
  M3_CUDA(cudaStreamSynchronize(s));
  D->ready = true;
  return M3SPH_OK;
}

extern "C" int m3sph_diffusion3d(m3sph_mesh *M, double *T, double dt, int32_t *nit) {
  if (!M || !T) {
    set_error("m3sph_diffusion3d: bad arguments");
    return M3SPH_ERR_BAD_INPUT;
  }
  M3_CUDA(cudaSetDevice(M->device));
  DiffState *D = diff_state(M);
  if (!D || !D->ready) {
    set_error("m3sph_diffusion3d: call m3sph_diffusion_setup first");
    return M3SPH_ERR_BAD_INPUT;
  }
  cudaStream_t s = M->stream;
  double *Td = D->T;
  int st = M3SPH_OK, it = 0;
  if (cudaMemcpyAsync(Td, T, D->nnod * sizeof(double), cudaMemcpyHostToDevice, s) != cudaSuccess)
    st = cuda_fail(cudaGetLastError(), "m3sph_diffusion3d upload");
  if (!st && D->kappa > 0.0) st = diffusion_resident(M, Td, dt, &it);
  if (!st && (cudaMemcpyAsync(T, Td, D->nnod * sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
              cudaStreamSynchronize(s) != cudaSuccess))
    st = cuda_fail(cudaGetLastError(), "m3sph_diffusion3d download");
  if (nit) *nit = it;
  return st;
}
