// Vector kernels (warp-shuffle FP64 reductions, fused CG updates), multigrid transfer
// (intermesh_transfer_matrix / Ic2f' restriction), Jacobi smoothing and the dense coarse
// solve that stands in for cholesky_factorization / cholesky_solve.
#include "common.cuh"
#include "tc.cuh"

namespace m3sph {

constexpr int RED_THREADS = 256;
constexpr int RED_BLOCKS = 608;      // 4 CTAs per SM on 152 SMs
// blocks of a reduction over n values: at least 4 values per thread (a fixed number for a given n)
unsigned red_blocks(size_t n) {
  return (unsigned)std::max<size_t>(1, std::min<size_t>(RED_BLOCKS, (n + 4 * RED_THREADS - 1) / (4 * RED_THREADS)));
}

// out[0] = a.b
__global__ void k_dot(const double *__restrict__ a, const double *__restrict__ b, size_t n, double *partials,
                      unsigned *cnt, double *out) {
  grid_dep();
  double v[1] = {0.0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    v[0] += a[i] * b[i];
  if (block_reduce_last<1>(v, partials, cnt) && threadIdx.x == 0) out[0] = v[0];
}
// out[0] = a.b, out[1] = c.b (b in the precision of the preconditioner)
template <typename T>
__global__ void k_dot2(const double *__restrict__ a, const double *__restrict__ c, const T *__restrict__ b, size_t n,
                       double *partials, unsigned *cnt, double *out) {
  grid_dep();
  double v[2] = {0.0, 0.0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const double bi = (double)b[i];
    v[0] += a[i] * bi;
    v[1] += c[i] * bi;
  }
  if (block_reduce_last<2>(v, partials, cnt) && threadIdx.x == 0) {
    out[0] = v[0];
    out[1] = v[1];
  }
}
// out[0] = sum(a)
__global__ void k_sum(const double *__restrict__ a, size_t n, double *partials, unsigned *cnt, double *out) {
  grid_dep();
  double v[1] = {0.0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) v[0] += a[i];
  if (block_reduce_last<1>(v, partials, cnt) && threadIdx.x == 0) out[0] = v[0];
}

int dot(const double *a, const double *b, size_t n, double *partials, unsigned *cnt, double *out, cudaStream_t s) {
  launch_pdl(k_dot, red_blocks(n), RED_THREADS, 0, s, a, b, n, partials, cnt, out); count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}
template <typename T>
int dot2(const double *a, const double *c, const T *b, size_t n, double *partials, unsigned *cnt, double *out, cudaStream_t s) {
  launch_pdl(k_dot2<T>, red_blocks(n), RED_THREADS, 0, s, a, c, b, n, partials, cnt, out); count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}
template int dot2<double>(const double *, const double *, const double *, size_t, double *, unsigned *, double *, cudaStream_t);
template int dot2<float>(const double *, const double *, const float *, size_t, double *, unsigned *, double *, cudaStream_t);
int vsum(const double *a, size_t n, double *partials, unsigned *cnt, double *out, cudaStream_t s) {
  launch_pdl(k_sum, red_blocks(n), RED_THREADS, 0, s, a, n, partials, cnt, out); count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}

// ---------------------------------------------------------------------------------------
// flexible PCG updates with device-resident scalars
// scal layout used by the CG: [0] rd, [1] Kqprev.d, [2] qKq, [3] rr, [4] rdlast, [5] alpha_prev,
// [6] first iteration. The V-cycle's result is read in its own precision and the residual is handed to it
// the same way, and a reduction's last block finishes it (and the scalars), so that an iteration's vector
// work is three launches beside the outer product (it was eleven, 3-6 us each at 130,662 dofs).
// ---------------------------------------------------------------------------------------
// q = d + beta q, beta = -alpha_prev * (Kq_prev . d) / rdlast (Polak-Ribiere: (r - rlast).d / rdlast)
template <typename T>
__global__ void k_cg_dir(const T *__restrict__ d, double *__restrict__ q, size_t n, const double *scal) {
  grid_dep();
  const bool first = scal[6] != 0.0;
  double beta = 0.0;
  if (!first) beta = -scal[5] * scal[1] / scal[4];
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    q[i] = first ? (double)d[i] : (double)d[i] + beta * q[i];
}
// alpha = rd / qKq ; x += alpha q ; r -= alpha Kq (and its FP32 copy) ; rr, rdlast, alpha_prev, first = 0.
// A NaN step (a NaN right-hand side, or a breakdown) leaves x as it is; the NaN residual then ends the loop.
// Then whether the loop goes on: it ends when a bounded wait of the iteration's kernels gave up (their error
// words, wait_err; the products are then wrong), when the residual is below the tolerance or NaN, at the
// iteration limit, or, with the learned smoother, at a contraction factor above 0.95 (or growth). `loop` is the
// condition of the captured loop around the iteration (0: the host runs it).
__global__ void k_cg_update(double *__restrict__ x, double *__restrict__ r, const double *__restrict__ q,
                            const double *__restrict__ Kq, float *__restrict__ r32, size_t n, double *scal,
                            double *partials, unsigned *cnt, WaitWords wait_err, cudaGraphConditionalHandle loop) {
  grid_dep();
  const double rd = scal[0], alpha = rd / scal[2];
  const bool step = !isnan(alpha);
  double v[1] = {0.0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    if (step) x[i] += alpha * q[i];
    const double ri = r[i] - alpha * Kq[i];
    r[i] = ri;
    if (r32) r32[i] = (float)ri;
    v[0] += ri * ri;
  }
  if (block_reduce_last<1>(v, partials, cnt) && threadIdx.x == 0) {
    scal[3] = v[0];
    scal[4] = rd;
    scal[5] = alpha;
    scal[6] = 0.0;
    const double rrms = sqrt(v[0]) / scal[CG_SQ], it = scal[CG_IT] + 1.0, prev = scal[CG_PREV];
    const bool last = it >= scal[CG_LIMIT], stalled = it > 1.0 && rrms > 0.95 * prev;
    bool gave_up = false;
    for (const int *w : wait_err.w) gave_up |= w && __ldcg(w) != 0;
    const int status = gave_up ? CG_WAIT_ERROR
                       : isnan(rrms) ? CG_NAN
                       : rrms < scal[CG_TOL] ? CG_CONVERGED
                       : scal[CG_LEARNED] != 0.0 && (stalled || last) ? CG_STALLED
                       : last ? CG_LIMIT_REACHED : CG_RUN;
    scal[CG_PREV] = rrms;
    scal[CG_IT] = it;
    scal[CG_STATUS] = (double)status;
    if (loop) cudaGraphSetConditional(loop, status == CG_RUN && (long long)it % CG_LOOP_MAX != 0);
  }
}

template <typename T>
int cg_dir(const T *d, double *q, size_t n, const double *scal, cudaStream_t s) {
  launch_pdl(k_cg_dir<T>, red_blocks(n), RED_THREADS, 0, s, d, q, n, scal); count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}
template int cg_dir<double>(const double *, double *, size_t, const double *, cudaStream_t);
template int cg_dir<float>(const float *, double *, size_t, const double *, cudaStream_t);
int cg_update(double *x, double *r, const double *q, const double *Kq, float *r32, size_t n, double *scal,
              double *partials, unsigned *cnt, WaitWords wait_err, cudaGraphConditionalHandle loop, cudaStream_t s) {
  launch_pdl(k_cg_update, red_blocks(n), RED_THREADS, 0, s, x, r, q, Kq, r32, n, scal, partials, cnt, wait_err, loop);
  count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}

// ---------------------------------------------------------------------------------------
// generic elementwise kernels
// ---------------------------------------------------------------------------------------
// y = (b - y) masked: residual r = b - Kx on free dofs, its FP32 copy and out[0] = r.r
__global__ void k_residual(const double *__restrict__ b, double *__restrict__ y, const uint8_t *__restrict__ mask,
                           float *__restrict__ y32, size_t n, double *partials, unsigned *cnt, double *out) {
  grid_dep();
  double v[1] = {0.0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const double r = mask[i] ? b[i] - y[i] : 0.0;
    y[i] = r;
    if (y32) y32[i] = (float)r;
    v[0] += r * r;
  }
  if (block_reduce_last<1>(v, partials, cnt) && threadIdx.x == 0) out[0] = v[0];
}
int residual(const double *b, double *y, const uint8_t *mask, float *y32, size_t n, double *partials, unsigned *cnt,
             double *out, cudaStream_t s) {
  launch_pdl(k_residual, red_blocks(n), RED_THREADS, 0, s, b, y, mask, y32, n, partials, cnt, out); count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}
__global__ void k_mask(double *__restrict__ y, const uint8_t *__restrict__ mask, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    if (!mask[i]) y[i] = 0.0;
}
int apply_mask(double *y, const uint8_t *mask, size_t n, cudaStream_t s) {
  k_mask<<<RED_BLOCKS, RED_THREADS, 0, s>>>(y, mask, n); count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}
template <typename A, typename B>
__global__ void k_convert(const A *__restrict__ a, B *__restrict__ b, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    b[i] = (B)a[i];
}
int d2f(const double *a, float *b, size_t n, cudaStream_t s) {
  k_convert<double, float><<<RED_BLOCKS, RED_THREADS, 0, s>>>(a, b, n); count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}
int f2d(const float *a, double *b, size_t n, cudaStream_t s) {
  k_convert<float, double><<<RED_BLOCKS, RED_THREADS, 0, s>>>(a, b, n); count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}

// ---------------------------------------------------------------------------------------
// Jacobi smoothing pieces (MG_V_cycle_v2, mgpcg_solver_p.m:397-437, 525-550)
// ---------------------------------------------------------------------------------------
// first down sweep: d = w * r0 * Dinv
template <typename T>
__global__ void k_jac_first(T w, const T *__restrict__ r0, const T *__restrict__ Di, T *__restrict__ d, size_t n) {
  grid_dep();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    d[i] = w * r0[i] * Di[i];
}
// d += w * (r0 - Kd) * Dinv
template <typename T>
__global__ void k_jac(T w, const T *__restrict__ r0, const T *__restrict__ Kd, const T *__restrict__ Di,
                      T *__restrict__ d, size_t n) {
  grid_dep();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    d[i] += w * (r0[i] - Kd[i]) * Di[i];
}
template <typename T>
int jac_first(T w, const T *r0, const T *Di, T *d, size_t n, cudaStream_t s) {
  launch_pdl(k_jac_first<T>, RED_BLOCKS, RED_THREADS, 0, s, w, r0, Di, d, n); count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}
template <typename T>
int jac(T w, const T *r0, const T *Kd, const T *Di, T *d, size_t n, cudaStream_t s) {
  launch_pdl(k_jac<T>, RED_BLOCKS, RED_THREADS, 0, s, w, r0, Kd, Di, d, n); count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}
template int jac_first<double>(double, const double *, const double *, double *, size_t, cudaStream_t);
template int jac_first<float>(float, const float *, const float *, float *, size_t, cudaStream_t);
template int jac<double>(double, const double *, const double *, const double *, double *, size_t, cudaStream_t);
template int jac<float>(float, const float *, const float *, const float *, float *, size_t, cudaStream_t);

// ---------------------------------------------------------------------------------------
// transfer: restriction rc = Ic2f' (r0 - Kd) (gather over coarse rows), prolongation
// d_f += Ic2f d_c (gather over fine rows); both masked to free dofs
// ---------------------------------------------------------------------------------------
// one warp per coarse row: lane l takes fine entries ptr[i] + l, + 32, ... (coarse rows gather ~40
// fine nodes), then a shuffle sum. On the way down the coarse residual is also handed to what comes
// next: the first Jacobi sweep from zero, d = w Di r (Di, d), or the operand of the coarsest-level solve
// on its free dofs (cmap, xfree).
template <typename T>
__global__ void __launch_bounds__(256) k_restrict(const int *__restrict__ ptr, const int *__restrict__ col,
                                                  const float *__restrict__ w, int nrow, const T *__restrict__ a,
                                                  const T *__restrict__ b, const uint8_t *__restrict__ mask,
                                                  T *__restrict__ out, T wj, const T *__restrict__ Di, T *__restrict__ d,
                                                  const int *__restrict__ cmap, T *__restrict__ xfree) {
  const int i = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  const bool row = i < nrow;
  const int kb = row ? ptr[i] + lane : 0, ke = row ? ptr[i + 1] : 0;
  int j = kb < ke ? col[kb] : 0;
  T wk = kb < ke ? (T)w[kb] : T(0);
  grid_dep();
  if (!row) return;
  T s0 = 0, s1 = 0, s2 = 0;
  for (int k = kb; k < ke; k += 32) {
    if (k != kb) {
      j = col[k];
      wk = (T)w[k];
    }
    if (b) {
      s0 += wk * (a[3 * j] - b[3 * j]);
      s1 += wk * (a[3 * j + 1] - b[3 * j + 1]);
      s2 += wk * (a[3 * j + 2] - b[3 * j + 2]);
    } else {
      s0 += wk * a[3 * j];
      s1 += wk * a[3 * j + 1];
      s2 += wk * a[3 * j + 2];
    }
  }
  const T t = lane_sum3<32>(s0, s1, s2);
  if (lane % 8 == 0 && lane < 24) {
    const size_t q = 3 * (size_t)i + lane / 8;
    const T v = mask[q] ? t : T(0);
    out[q] = v;
    if (d) d[q] = wj * v * Di[q];
    if (cmap) {
      const int f = cmap[q];
      if (f >= 0) xfree[f] = v;
    }
  }
}
// out = add + P xc (masked); add may alias out; pc: also the Cartesian copy of out
template <typename T>
__global__ void k_prolong(const int *__restrict__ ptr, const int *__restrict__ col, const float *__restrict__ w,
                          int nrow, const T *__restrict__ xc, const T *add, const uint8_t *__restrict__ mask, T *out,
                          PaCart pc) {
  grid_dep();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nrow) return;
  T t[3] = {0, 0, 0};
  for (int k = ptr[i]; k < ptr[i + 1]; ++k) {
    const int j = col[k];
    const T wk = (T)w[k];
#pragma unroll
    for (int c = 0; c < 3; ++c) t[c] += wk * xc[3 * j + c];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const T base = add ? add[3 * i + c] : T(0);
    t[c] = mask[3 * i + c] ? base + t[c] : T(0);
    out[3 * i + c] = t[c];
  }
  if (pc.xc) pc.xc[i] = pa_to_cart(pc.trig[i], (float)t[0], (float)t[1], (float)t[2]);
}
template <typename T>
int restrict_(const Level &F, const Level &C, const T *a, const T *b, T *out, cudaStream_t s, T wj, const T *Di, T *d,
              const int *cmap, T *xfree) {
  launch_pdl(k_restrict<T>, (unsigned)(((size_t)C.nnod * 32 + 255) / 256), 256, 0, s, F.R_ptr, F.R_col, F.R_w, C.nnod,
             a, b,
                                                                             C.freemask, out, wj, Di, d, cmap, xfree);
  count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}
template <typename T>
int prolong(const Level &F, const Level &C, const T *xc, const T *add, T *out, const PaCart &pc, cudaStream_t s) {
  launch_pdl(k_prolong<T>, (F.nnod + 255) / 256, 256, 0, s, F.P_ptr, F.P_col, F.P_w, F.nnod, xc, add, F.freemask, out,
             pc);
  count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}
template int restrict_<double>(const Level &, const Level &, const double *, const double *, double *, cudaStream_t,
                               double, const double *, double *, const int *, double *);
template int restrict_<float>(const Level &, const Level &, const float *, const float *, float *, cudaStream_t, float,
                              const float *, float *, const int *, float *);
template int prolong<double>(const Level &, const Level &, const double *, const double *, double *, const PaCart &,
                             cudaStream_t);
template int prolong<float>(const Level &, const Level &, const float *, const float *, float *, const PaCart &,
                            cudaStream_t);

// ---------------------------------------------------------------------------------------
// coarsest level: dense assembly, in-place Gauss-Jordan inverse (SPD, no pivoting), GEMV
// ---------------------------------------------------------------------------------------
// dense matrix from the level's 3x3-block rows (blocks [9][nnzb]): every entry is written once, so
// the result does not depend on the order in which threads run
// rows and columns of fixed dofs are left out: the matrix is the free-dof block, nf x nf, through
// the compact map cmap (-1 for a fixed dof)
template <typename T>
__global__ void k_dense_from_bsr(const int *__restrict__ ptr, const int *__restrict__ col, const T *__restrict__ B,
                                 int nrow, size_t nnzb, const int *__restrict__ cmap, int ld, T *__restrict__ A) {
  const int i = blockIdx.x;
  if (i >= nrow) return;
  for (int k = ptr[i] + threadIdx.x; k < ptr[i + 1]; k += blockDim.x) {
    const int j = col[k];
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const int a = cmap[3 * i + p];
      if (a < 0) continue;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int b = cmap[3 * j + q];
        if (b >= 0) A[(size_t)a * ld + b] = B[(size_t)(p * 3 + q) * nnzb + k];
      }
    }
  }
}
// ---------------------------------------------------------------------------------------
// blocked Gauss-Jordan inverse of the SPD coarsest matrix, panels of NB (no pivoting). Per panel k, with
// D = A_kk, C = A_:k and R = D^-1 A_k: :
//   A_ij -= C_i R_j (i, j outside panel k), A_kj = R_j, A_ik = -C_i D^-1, A_kk = D^-1.
// The matrix stays symmetric up to sign -- A_ij = A_ji' when both or neither of panels i, j have been
// swept, A_ij = -A_ji' when one has -- so only tiles on and below the diagonal are kept and updated (half
// the work of the full form): C_i of an unswept panel i is the stored tile, of a swept one minus the
// transpose of tile (k, i), and R_j = +-D^-1 C_j'. The upper triangle is filled in at the end.
//
// Three launches per panel, and from 48 FP32 panels on k_gjb_diag of the next panel beside the update of this
// one (gj_blocked_inverse):
//  * k_gjb_diag inverts D in one CTA, the block held in registers (an RT x RT piece per thread), by
//    16-wide sub-panels: the 16 x 16 pivot block by one warp through shuffles, the rest as rank-16
//    updates. (One pivot at a time in shared memory took 975 us per panel in FP32 and 3,941 us in FP64;
//    now 74 us, and 129 us for the 64-wide FP64 block.)
//  * k_gjb_panels saves C (transposed), forms R and writes panel k of the matrix (its products summed by
//    chunks of 16: 2 to 3 % less error of the inverse);
//  * FP32: k_gjb_update_tc, on the tensor cores. FP64: k_gjb_update, a tile GEMM of NB x NB tiles, 256
//    threads, an RT x RT register block per thread read from shared memory as 16-byte vectors, chunks of the
//    inner dimension brought in by 16-byte asynchronous copies two chunks ahead (panels are padded to whole
//    tiles with zeros, so the copies need no bounds); FP64 issue bounds it.
// NB is 64 in FP64: the diagonal block is inverted on one SM, whose FP64 rate (2 FMA a cycle) makes a
// 128-wide block cost 0.5 ms.
// ---------------------------------------------------------------------------------------
template <typename T> struct Gj;
template <> struct Gj<float> { static constexpr int NB = 128, KC = 16; using V = float4; static constexpr int VN = 4; };
template <> struct Gj<double> { static constexpr int NB = 64, KC = 8; using V = double2; static constexpr int VN = 2; };
constexpr int GJ_ST = 3;             // chunk stages
// tensor-core update (FP32): operand images of a 128 x 128 panel block, three BF16 parts whose sum is the FP32
// value, K-major and 128-byte swizzled: [half of K][part][128 rows][64 K]
namespace gu {
constexpr int NB = 128, ATOM = NB * 128, HALF = 3 * ATOM, IMAGE = 2 * HALF;
constexpr int WARPS = 16, THREADS = (WARPS + 2) * 32;     // two groups of 8 epilogue warps, a copy warp, an MMA warp
constexpr int STAGE_LD = 20;                               // floats per row of a warp's staging tile of 16 rows
constexpr int OFF_A = 0, OFF_B = IMAGE, OFF_ST = OFF_B + 2 * HALF;
constexpr int OFF_BAR = OFF_ST + WARPS * 16 * STAGE_LD * 4;  // a_full, b_full[2], b_empty[2], acc_full[4], acc_empty[2], drain
// The accumulators round towards zero. In a half of K the large product comes last, in four instructions of
// K = 16, and after each the sum is cut; for terms of one sign the sums are 1/4, 1/2, 3/4 and all of the result, a
// cut takes half a unit of the last place on average, and that is 2^-24 / (2 ln 2) = 4.3e-8 of the value:
// 2.5 x 4.3e-8 = 1.07e-7 of the result is lost. The third part of C gives 1e-7 back. Error of a V-cycle with
// the inverse of 3,210 free dofs: 5.2e-7 with nothing given back, 3.6e-7 with half of it, 2.4e-7 with this;
// 3.3e-7 with an update by FP32 multiply-adds (tests: 1 to 48 panels).
constexpr float ROUNDING = 1e-7f;
constexpr int OFF_TM = OFF_BAR + 12 * 8;
constexpr int SMEM = OFF_TM + 8, SMEM_ALLOC = SMEM + 1024;
static_assert(OFF_BAR % 8 == 0 && OFF_ST % 16 == 0 && SMEM_ALLOC <= 232448, "one CTA per SM");
}  // namespace gu
constexpr int GJ_SB = 16;            // sub-panel width of the diagonal block

// values of the work array: D^-1, its transpose, the saved column panel and the row panel
// FP32: also the operand images of the two panels and an error word
template <typename T> size_t gj_work(int n) {
  const size_t NB = Gj<T>::NB, npad = (n + NB - 1) / NB * NB;
  return 2 * NB * NB + 2 * NB * npad + (sizeof(T) == 4 ? 2 * (npad / NB) * (gu::IMAGE / 4) + 4 : 0);
}
size_t dense_inverse_work64(int n) { return gj_work<double>(n); }
size_t dense_inverse_work32(int n) { return gj_work<float>(n); }
// row stride of the dense inverse: whole 16-byte vectors
int dense_ld(int n) { return (n + 3) & ~3; }


// acc = sum_m X[m][row] Y[m][col] over m < NB, X and Y with row strides ldx, ldy (16-byte aligned).
// Thread (ty, tx) owns rows and columns in groups of four consecutive indices: gj_idx
template <typename T>
__device__ __forceinline__ int gj_idx(int t, int a) {
  constexpr int NG = Gj<T>::NB / 64;                 // groups per thread
  return (a >> 2) * (Gj<T>::NB / NG) + 4 * t + (a & 3);
}
__device__ __forceinline__ void gj_ld4(const float *p, float *v) {
  const float4 q = *reinterpret_cast<const float4 *>(p);
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void gj_ld4(const double *p, double *v) {
  const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void gj_st4(float *p, const float *v) {
  *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void gj_st4(double *p, const double *v) {
  *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
  *reinterpret_cast<double2 *>(p + 2) = make_double2(v[2], v[3]);
}
template <typename T> constexpr size_t gj_smem() { return sizeof(T) * GJ_ST * 2 * Gj<T>::KC * Gj<T>::NB; }
template <typename T, int RT, int CT>
__device__ __forceinline__ void gj_tile(T (&acc)[RT][CT], const T *X, size_t ldx, const T *Y, size_t ldy) {
  constexpr int NB = Gj<T>::NB, KC = Gj<T>::KC, NCH = NB / KC, VN = 16 / sizeof(T), PR = NB / VN, PY = 16 * CT / VN;
  extern __shared__ __align__(16) unsigned char gj_raw[];
  T(*sm)[2][KC][NB] = reinterpret_cast<T(*)[2][KC][NB]>(gj_raw);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int a = 0; a < RT; ++a)
#pragma unroll
    for (int b = 0; b < CT; ++b) acc[a][b] = T(0);
  auto issue = [&](int ch) {
    if (ch < NCH) {
      for (int q = threadIdx.x; q < KC * PR; q += 256) {
        const int m = q / PR, v = (q % PR) * VN, k = ch * KC + m;
        const uint32_t dx = (uint32_t)__cvta_generic_to_shared(&sm[ch % GJ_ST][0][m][v]);
        const uint32_t dy = (uint32_t)__cvta_generic_to_shared(&sm[ch % GJ_ST][1][m][v]);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dx), "l"(X + k * ldx + v) : "memory");
        if (PY == PR || q % PR < PY)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dy), "l"(Y + k * ldy + v) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int ch = 0; ch < GJ_ST - 1; ++ch) issue(ch);
  for (int ch = 0; ch < NCH; ++ch) {
    asm volatile("cp.async.wait_group %0;" ::"n"(GJ_ST - 2) : "memory");
    __syncthreads();                     // chunk ch has landed, everyone is done with chunk ch - 1
    issue(ch + GJ_ST - 1);
    const T(*xs)[NB] = sm[ch % GJ_ST][0], (*ys)[NB] = sm[ch % GJ_ST][1];
    T part[RT][CT];                      // a chunk's sum by itself: shorter chains of roundings
#pragma unroll
    for (int a = 0; a < RT; ++a)
#pragma unroll
      for (int b = 0; b < CT; ++b) part[a][b] = T(0);
#pragma unroll
    for (int m = 0; m < KC; ++m) {
      T xv[RT], yv[CT];
#pragma unroll
      for (int g = 0; g < RT; g += 4) gj_ld4(&xs[m][gj_idx<T>(ty, g)], xv + g);
#pragma unroll
      for (int g = 0; g < CT; g += 4) gj_ld4(&ys[m][gj_idx<T>(tx, g)], yv + g);
#pragma unroll
      for (int a = 0; a < RT; ++a)
#pragma unroll
        for (int b = 0; b < CT; ++b) (sizeof(T) == 4 ? part : acc)[a][b] += xv[a] * yv[b];
    }
    if (sizeof(T) == 4)
#pragma unroll
      for (int a = 0; a < RT; ++a)
#pragma unroll
        for (int b = 0; b < CT; ++b) acc[a][b] += part[a][b];
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <typename T>
__global__ void __launch_bounds__(256) k_gjb_diag(const T *__restrict__ A, int ld, int kb, int nb, T *__restrict__ Dinv,
                                                  T *__restrict__ DinvT, const T *Ct, const T *R, size_t npad) {
  constexpr int NB = Gj<T>::NB, RT = NB / 16, SB = GJ_SB;
  __shared__ T sC[NB][SB + 1], sK[SB][NB], sR[SB][NB], sD[SB][SB + 1];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16, r0 = ty * RT, c0 = tx * RT;
  T a[RT][RT];
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < RT; ++j) {
      const int r = r0 + i, c = c0 + j;
      a[i][j] = (r < nb && c < nb) ? A[(size_t)(kb + r) * ld + kb + c] : (r == c ? T(1) : T(0));
    }
  if (sizeof(T) == 4 && Ct) {            // A - C R of the panel before, padded rows and columns are zero
    T u[RT][RT];
    gj_tile<T, RT, RT>(u, Ct + kb, npad, R + kb, npad);
    // its threads hold groups of four rows and columns 64 apart: through shared memory to whole pieces
    extern __shared__ __align__(16) unsigned char gj_raw[];
    T(*su)[NB] = reinterpret_cast<T(*)[NB]>(gj_raw);
    for (int h = 0; h < NB / 16; ++h) {
      __syncthreads();
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < RT; ++j)
          if (gj_idx<T>(ty, i) / 16 == h) su[gj_idx<T>(ty, i) % 16][gj_idx<T>(tx, j)] = u[i][j];
      __syncthreads();
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < RT; ++j)
          if ((r0 + i) / 16 == h) a[i][j] -= su[(r0 + i) % 16][c0 + j];
    }
    __syncthreads();
  }
  for (int p0 = 0; p0 < NB; p0 += SB) {
    const bool inr = r0 >= p0 && r0 < p0 + SB, inc = c0 >= p0 && c0 < p0 + SB;    // RT divides SB
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int j = 0; j < RT; ++j) {
        if (inc) sC[r0 + i][c0 + j - p0] = a[i][j];
        if (inr) sK[r0 + i - p0][c0 + j] = a[i][j];
      }
    __syncthreads();
    if (threadIdx.x < 32) {
      // 16 x 16 pivot block: lane (h, c) holds rows 8h..8h+7 of column c
      const int lane = threadIdx.x, c = lane & 15, h = lane >> 4;
      T d[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) d[r] = sK[8 * h + r][p0 + c];
#pragma unroll
      for (int p = 0; p < SB; ++p) {
        const int hp = p >> 3;
        const T piv = __shfl_sync(0xffffffffu, d[p & 7], p + 16 * hp);
        const T rp = __shfl_sync(0xffffffffu, d[p & 7], c + 16 * hp);
        const T inv = T(1) / piv, row = c == p ? inv : rp * inv;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const T cv = __shfl_sync(0xffffffffu, d[r], p + 16 * h);
          if (8 * h + r == p) d[r] = row;
          else d[r] = c == p ? -cv * inv : d[r] - cv * row;
        }
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) sD[8 * h + r][c] = d[r];
    }
    __syncthreads();
    // R = D^-1 A_k: , with D^-1 itself in the panel's own columns
    for (int q = threadIdx.x; q < SB * NB; q += 256) {
      const int r = q / NB, c = q % NB;
      T v = T(0);
      if (c >= p0 && c < p0 + SB) {
        v = sD[r][c - p0];
      } else {
#pragma unroll
        for (int m = 0; m < SB; ++m) v += sD[r][m] * sK[m][c];
      }
      sR[r][c] = v;
    }
    __syncthreads();
    if (inr) {
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < RT; ++j) a[i][j] = sR[r0 + i - p0][c0 + j];
    } else {
      if (inc) {
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
          for (int j = 0; j < RT; ++j) a[i][j] = T(0);
      }
#pragma unroll 4
      for (int m = 0; m < SB; ++m) {
        T x[RT], y[RT];
#pragma unroll
        for (int i = 0; i < RT; ++i) x[i] = sC[r0 + i][m];
#pragma unroll
        for (int j = 0; j < RT; ++j) y[j] = sR[m][c0 + j];
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
          for (int j = 0; j < RT; ++j) a[i][j] -= x[i] * y[j];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < RT; ++j) {
      Dinv[(r0 + i) * NB + c0 + j] = a[i][j];
      DinvT[(c0 + j) * NB + r0 + i] = a[i][j];
    }
}

// rows c0 .. c0 + 63 of the operand image of block column j0 of a panel S (128 K-rows of npad values): row c =
// column j0 + c of S, times 1 + up
__device__ __forceinline__ void gj_image(const float *S, size_t npad, int j0, int c0, float up, unsigned char *img) {
  for (int q = threadIdx.x; q < 64 * 16; q += 256) {
    const int c = c0 + (q & 63), ch = q >> 6;
    uint32_t w[3][4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      float v[2], p[3][2];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const float x = S[(size_t)(8 * ch + 2 * h + t) * npad + j0 + c];
        v[t] = x;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (k == 2) v[t] += up * x;
          p[k][t] = __bfloat162float(__float2bfloat16_rn(v[t]));
          v[t] -= p[k][t];               // exact: 8 of the 24 bits each time
        }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) w[k][h] = tc_pack(p[k][0], p[k][1]);
    }
    unsigned char *o = img + (ch >> 3) * gu::HALF + tc_sw(c, ch & 7);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      *reinterpret_cast<uint4 *>(o + k * gu::ATOM) = make_uint4(w[k][0], w[k][1], w[k][2], w[k][3]);
  }
}

// block j, columns c0 .. c0 + NW - 1 of it: saved column panel Ct[m][i] = C_i[m] for its rows i and row panel
// R = +-D^-1 C_j' for its columns (minus for panels already swept, j < kblk), zero padding past n; then panel k of
// the matrix itself: its row R, its column -C D^-1 = -R' and its diagonal block D^-1. FP32: the operand images of
// C and R as well, and two CTAs per block (70 -> 50 us at 14.8k free dofs: a CTA's share is a serial chain of loads,
// product and stores).
template <typename T> constexpr int GJ_PANEL_CTAS = sizeof(T) == 4 ? 2 : 1;
template <typename T>
__global__ void __launch_bounds__(256) k_gjb_panels(T *__restrict__ A, int ld, int n, int kblk, int nb,
                                                    const T *__restrict__ Dinv, const T *__restrict__ DinvT, size_t npad,
                                                    T *R, T *Ct, unsigned char *imgC, unsigned char *imgR) {
  constexpr int NB = Gj<T>::NB, RT = NB / 16, NW = NB / GJ_PANEL_CTAS<T>, CT = NW / 16;
  __shared__ T tr[32][33];
  const int j = blockIdx.x, c0 = blockIdx.y * NW, j0 = j * NB + c0, kb = kblk * NB;
  const bool swept = j < kblk;
  if (j == kblk) {
    for (int q = threadIdx.x; q < NB * NW; q += 256) {
      const int r = q / NW, c = c0 + q % NW;
      if (r < nb && c < nb) A[(size_t)(kb + r) * ld + kb + c] = Dinv[r * NB + c];
    }
    return;
  }
  if (swept) {
    // C_i = -A_ki' : row m of tile (k, j) is column m of C
    for (int q = threadIdx.x; q < NB * NW; q += 256) {
      const int m = q / NW, c = q % NW;
      Ct[m * npad + j0 + c] = (m < nb) ? -A[(size_t)(kb + m) * ld + j0 + c] : T(0);
    }
  } else {
    // tile (j, k), transposed 32 x 32 at a time
    const int lx = threadIdx.x % 32, ly = threadIdx.x / 32;
    for (int b = 0; b < (NW / 32) * (NB / 32); ++b) {
      const int i0 = (b / (NB / 32)) * 32, m0 = (b % (NB / 32)) * 32;
      __syncthreads();
      for (int y = ly; y < 32; y += 8) {
        const int i = j0 + i0 + y, m = m0 + lx;
        tr[y][lx] = (i < n && m < nb) ? A[(size_t)i * ld + kb + m] : T(0);
      }
      __syncthreads();
      for (int y = ly; y < 32; y += 8) Ct[(size_t)(m0 + y) * npad + j0 + i0 + lx] = tr[lx][y];
    }
  }
  __syncthreads();
  T acc[RT][CT];
  gj_tile<T, RT, CT>(acc, DinvT, NB, Ct + j0, npad);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int a = 0; a < RT; ++a)
#pragma unroll
    for (int g = 0; g < CT; g += 4) {
      T v[4];
#pragma unroll
      for (int b = 0; b < 4; ++b) v[b] = swept ? -acc[a][g + b] : acc[a][g + b];
      const int m = gj_idx<T>(ty, a), c = j0 + gj_idx<T>(tx, g);
      gj_st4(&R[m * npad + c], v);
      if (swept && m < nb) gj_st4(&A[(size_t)(kb + m) * ld + c], v);
    }
  __syncthreads();
  if (!swept) {
    const int lx = threadIdx.x % 32, ly = threadIdx.x / 32;
    for (int b = 0; b < (NW / 32) * (NB / 32); ++b) {
      const int r0 = (b / (NB / 32)) * 32, m0 = (b % (NB / 32)) * 32;
      __syncthreads();
      for (int y = ly; y < 32; y += 8) tr[y][lx] = R[(size_t)(m0 + y) * npad + j0 + r0 + lx];
      __syncthreads();
      for (int y = ly; y < 32; y += 8) {
        const int i = j0 + r0 + y, m = m0 + lx;
        if (i < n && m < nb) A[(size_t)i * ld + kb + m] = -tr[lx][y];
      }
    }
  }
  if constexpr (sizeof(T) == 4) {
    gj_image(Ct, npad, j * NB, c0, gu::ROUNDING, imgC + (size_t)j * gu::IMAGE);
    gj_image(R, npad, j * NB, c0, 0.f, imgR + (size_t)j * gu::IMAGE);
  }
}

// tile t of the lower triangle without panel k: block row and column
__device__ __forceinline__ void gj_tile_of(size_t t, int kblk, int &bi, int &bj) {
  bi = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
  while ((size_t)bi * (bi + 1) / 2 > t) --bi;
  while ((size_t)(bi + 1) * (bi + 2) / 2 <= t) ++bi;
  bj = (int)(t - (size_t)bi * (bi + 1) / 2);
  bi += bi >= kblk;
  bj += bj >= kblk;
}

// A - C R on a tile outside panel k (FP64)
template <typename T>
__global__ void __launch_bounds__(256, 2) k_gjb_update(T *__restrict__ A, int ld, int n, int kblk, size_t npad,
                                                       const T *__restrict__ R, const T *__restrict__ Ct) {
  constexpr int NB = Gj<T>::NB, RT = NB / 16;
  int bi, bj;
  gj_tile_of(blockIdx.x, kblk, bi, bj);
  const int i0 = bi * NB, j0 = bj * NB;
  T acc[RT][RT];
  gj_tile<T, RT, RT>(acc, Ct + i0, npad, R + j0, npad);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int a = 0; a < RT; ++a) {
    const int i = i0 + gj_idx<T>(ty, a);
    if (i >= n) continue;
#pragma unroll
    for (int g = 0; g < RT; g += 4) {
      const int j = j0 + gj_idx<T>(tx, g);
      if (j >= ld) continue;                         // ld is a multiple of 4: whole vectors
      T *p = A + (size_t)i * ld + j, v[4];
      gj_ld4(p, v);
#pragma unroll
      for (int b = 0; b < 4; ++b) v[b] -= acc[a][g + b];
      gj_st4(p, v);
    }
  }
}

// The same for FP32 on the tensor cores. A product of two FP32 values is the six largest of the nine products of
// their BF16 parts (the rest is below 2^-26 of it); the accumulators are FP32. An accumulator takes a half of K,
// first the five small products and then the large one, so that the roundings of the former are 2^-8 smaller,
// the two halves are added in FP32, and what rounding towards zero takes is given back (gu::ROUNDING). Against
// FP64 inverses of difference matrices of 129 to 14,801 unknowns and contrasts of 1e2 to 1e4 the error of the
// whole inverse is 0 to 10 % below that of FP32 multiply-adds (without ROUNDING 1 to 4 % above); on the coarsest
// levels of shells, 378 to 17,334 dofs, a V-cycle's error from the inverse is 5 % above to 50 % below.
// A persistent CTA takes a run of tiles of the triangle, row by row: the row's operand stays in shared memory
// (96 KB), the column's comes in halves of 48 KB through a ring of two, and the accumulators of two tiles
// alternate in TMEM between two groups of epilogue warps, which subtract through a staging tile. At 14.8k free
// dofs 223 us per panel (248 us on 151 SMs with the next diagonal block beside it), FP32 multiply-adds 589 us; the triangle read and written at the copy rate would be
// 130 us, the MMAs alone are 82 us: what is left is the latency of the A accesses (272 us with chunks fetched when
// they were needed, 255 us without the prefetch of the next tile into L2).
__global__ void __launch_bounds__(gu::THREADS, 1) k_gjb_update_tc(float *__restrict__ A, int ld, int n, int kblk,
                                                                  int done, size_t ntile, const unsigned char *__restrict__ imgC,
                                                                  const unsigned char *__restrict__ imgR, int *err) {
  using namespace gu;
  extern __shared__ __align__(16) unsigned char gj_raw[];
  unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(gj_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sbase = tc_smem_u32(sm);
  const uint32_t a_full = sbase + OFF_BAR, b_full = a_full + 8, b_empty = a_full + 24, acc_full = a_full + 40,
                 acc_empty = a_full + 72, drain = a_full + 88;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + OFF_TM);
  if (tid == 0) {
    tc_bar_init(a_full, 1);
    tc_bar_init(drain, 1);
    for (int b = 0; b < 2; ++b) {
      tc_bar_init(b_full + 8 * b, 1);
      tc_bar_init(b_empty + 8 * b, 1);
    }
    for (int b = 0; b < 4; ++b) tc_bar_init(acc_full + 8 * b, 1);
    for (int b = 0; b < 2; ++b) tc_bar_init(acc_empty + 8 * b, WARPS / 2);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(tslot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const size_t t0 = ntile * blockIdx.x / gridDim.x, t1 = ntile * (blockIdx.x + 1) / gridDim.x;
  int bi, bj;
  if (warp == WARPS) {
    // ---------------- copies ----------------
    if (lane == 0) {
      int row = -1, na = 0, nbt[2] = {0, 0};        // copies issued per barrier
      bool ok = true;
      uint32_t it = 0;
      for (size_t t = t0; t < t1 && ok; ++t, ++it) {
        gj_tile_of(t, kblk, bi, bj);
        for (int h = 0; h < 2 && ok; ++h) {
          if (it) ok = tc_bar_wait(b_empty + 8 * h, (it - 1) & 1);
          // a new row: its operand goes where the last tile's MMAs read, so both halves must be done
          if (h == 0 && bi != row) {
            if (it) ok = ok && tc_bar_wait(b_empty + 8, (it - 1) & 1);
            if (ok) {
              tc_bulk_load(sbase + OFF_A, imgC + (size_t)bi * IMAGE, IMAGE, a_full);
              ++na;
              row = bi;
            }
          }
          if (!ok) break;
          tc_bulk_load(sbase + OFF_B + h * HALF, imgR + (size_t)bj * IMAGE + h * HALF, HALF, b_full + 8 * h);
          ++nbt[h];
        }
      }
      if (!ok) atomicOr(err, 1);
      // no copy may be in flight when the block ends, whichever warp gave up
      if (na) tc_bar_wait(a_full, (na - 1) & 1);
      for (int h = 0; h < 2; ++h)
        if (nbt[h]) tc_bar_wait(b_full + 8 * h, (nbt[h] - 1) & 1);
    }
    __syncwarp();
  } else if (warp == WARPS + 1) {
    // ---------------- MMAs ----------------
    if (lane == 0) {
      // products of parts (A, B), smallest first
      constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
      int row = -1, na = 0;
      bool ok = true;
      uint32_t it = 0;
      for (size_t t = t0; t < t1 && ok; ++t, ++it) {
        gj_tile_of(t, kblk, bi, bj);
        const int buf = it & 1;
        if (it >= 2) ok = tc_bar_wait(acc_empty + 8 * buf, ((it >> 1) - 1) & 1);
        if (ok && bi != row) {
          ok = tc_bar_wait(a_full, na & 1);
          ++na;
          row = bi;
        }
        for (int h = 0; h < 2 && ok; ++h) {
          ok = tc_bar_wait(b_full + 8 * h, it & 1);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = sbase + OFF_A + h * HALF, sb = sbase + OFF_B + h * HALF, d = tmem + 256 * buf + 128 * h;
#pragma unroll
          for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              tc_mma(d, tc_sdesc(sa + PA[p] * ATOM + 32 * k), tc_sdesc(sb + PB[p] * ATOM + 32 * k), tc_idesc(NB, NB),
                     p > 0 || k > 0);
          tc_commit(b_empty + 8 * h);
          tc_commit(acc_full + 8 * (2 * buf + h));
        }
      }
      if (!ok) atomicOr(err, 2);
      tc_commit(drain);                      // nor an MMA when TMEM is given back
      tc_bar_wait(drain, 0);
    }
    __syncwarp();
  } else {
    // ---------------- epilogue: groups take every other tile; in a group warp w has rows 32 (w % 4) .. + 31 and
    // columns 64 (w / 4) .. + 63, 16 at a time ----------------
    const int grp = warp >> 3, r0 = 32 * (warp & 3), c0 = 64 * ((warp >> 2) & 1), lr = lane >> 2, lc = 4 * (lane & 3);
    float *st = reinterpret_cast<float *>(sm + OFF_ST) + warp * 16 * STAGE_LD;
    const uint32_t trow = tmem + ((uint32_t)r0 << 16) + c0 + 256 * grp;
    // a tile's part into L2, half a row of 256 bytes at a time (a load's own prefetch would bring 32)
    auto prefetch = [&](size_t t) {
      if (t >= t1) return;
      int pi, pj;
      gj_tile_of(t, kblk, pi, pj);
      const int i = pi * NB + r0 + lane, j = pj * NB + c0;
      if (i < n && j < ld)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(A + (size_t)i * ld + j),
                     "r"(4 * min(64, ld - j)));
    };
    // 16 columns of A ahead: while a chunk is worked on, the next one (of the group's next tile after the last) is
    // on its way
    int i0 = 0, j0 = 0;
    float *p = nullptr;
    auto locate = [&](size_t t) {
      gj_tile_of(t, kblk, bi, bj);
      i0 = bi * NB + r0 + lr;
      j0 = bj * NB + c0 + lc;
      p = A + (size_t)i0 * ld + j0;
    };
    auto fetch = [&](float4(&v)[4], int q) {   // rows lr + 8 a
#pragma unroll
      for (int a = 0; a < 4; ++a)
        if (j0 + 16 * q < ld && i0 + 8 * a < n) v[a] = *reinterpret_cast<const float4 *>(p + (size_t)(8 * a) * ld + 16 * q);
    };
    uint32_t use = 0;
    float4 v[2][4];
    prefetch(t0 + grp);
    if (t0 + grp < t1) {
      locate(t0 + grp);
      fetch(v[0], 0);
    }
    for (size_t t = t0 + grp; t < t1; t += 2, ++use) {
      prefetch(t + 2);
      bool ok = tc_bar_wait(acc_full + 8 * (2 * grp), use & 1) && tc_bar_wait(acc_full + 8 * (2 * grp + 1), use & 1);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicOr(err, 4);
        break;
      }
      tc_fence_after();
      const bool skip = bi == done && bj == done;      // the block k_gjb_diag updates itself
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int ic = i0;
        const bool jin = j0 + 16 * q < ld && !skip;
        float *pc = p + 16 * q;
        if (q < 3) {
          fetch(v[(q + 1) & 1], q + 1);
        } else if (t + 2 < t1) {
          locate(t + 2);
          fetch(v[0], 0);
        }
        float x[16], y[16];
        tc_ld16(trow + 16 * q, x);
        tc_ld16(trow + 128 + 16 * q, y);
        if (q == 3) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) tc_arrive(acc_empty + 8 * grp);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {          // 16 rows at a time through the staging tile
          __syncwarp();
          if ((lane >> 4) == h)
#pragma unroll
            for (int c = 0; c < 16; c += 4)
              *reinterpret_cast<float4 *>(st + (lane & 15) * STAGE_LD + c) =
                  make_float4(x[c] + y[c], x[c + 1] + y[c + 1], x[c + 2] + y[c + 2], x[c + 3] + y[c + 3]);
          __syncwarp();
#pragma unroll
          for (int a = 2 * h; a < 2 * h + 2; ++a) {
            const float4 u = *reinterpret_cast<const float4 *>(st + (lr + 8 * (a & 1)) * STAGE_LD + lc), w = v[q & 1][a];
            if (jin && ic + 8 * a < n)
              *reinterpret_cast<float4 *>(pc + (size_t)(8 * a) * ld) =
                  make_float4(w.x - u.x, w.y - u.y, w.z - u.z, w.w - u.w);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// upper triangle from the lower one
template <typename T>
__global__ void __launch_bounds__(256) k_gjb_mirror(T *__restrict__ A, int ld, int n) {
  __shared__ T tr[32][33];
  const int bi = blockIdx.y, bj = blockIdx.x;
  if (bj > bi) return;
  const int lx = threadIdx.x % 32, ly = threadIdx.x / 32;
  for (int y = ly; y < 32; y += 8) {
    const int i = bi * 32 + y, j = bj * 32 + lx;
    if (i < n && j < n) tr[y][lx] = A[(size_t)i * ld + j];
  }
  __syncthreads();
  for (int y = ly; y < 32; y += 8) {
    const int i = bj * 32 + y, j = bi * 32 + lx;
    if (i < n && j < n && j > i) A[(size_t)i * ld + j] = tr[lx][y];
  }
}

// second stream of an inversion and its two events
struct GjSide {
  cudaStream_t stream = nullptr;
  cudaEvent_t panel = nullptr, inverted = nullptr;
  int open() {
    M3_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    M3_CUDA(cudaEventCreateWithFlags(&panel, cudaEventDisableTiming));
    M3_CUDA(cudaEventCreateWithFlags(&inverted, cudaEventDisableTiming));
    return M3SPH_OK;
  }
  ~GjSide() {
    if (stream) {
      cudaStreamSynchronize(stream);
      cudaStreamDestroy(stream);
    }
    if (panel) cudaEventDestroy(panel);
    if (inverted) cudaEventDestroy(inverted);
  }
};

// in-place inverse of the n x n SPD matrix A with row stride ld; work holds gj_work(n) values
template <typename T>
int gj_blocked_inverse(T *A, int ld, int n, T *work, cudaStream_t s) {
  if (n == 0) return M3SPH_OK;         // every dof prescribed: nothing to invert, and no grid to launch
  constexpr int NB = Gj<T>::NB;
  const int nbk = (n + NB - 1) / NB;
  const size_t npad = (size_t)nbk * NB;
  T *Dinv = work, *DinvT = Dinv + NB * NB, *R = DinvT + NB * NB, *Ct = R + NB * npad;
  const size_t ntile = (size_t)nbk * (nbk - 1) / 2;        // lower tiles outside a panel
  unsigned char *imgC = nullptr, *imgR = nullptr;
  int *err = nullptr;
  M3_CUDA(cudaFuncSetAttribute(k_gjb_diag<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gj_smem<T>()));
  M3_CUDA(cudaFuncSetAttribute(k_gjb_panels<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gj_smem<T>()));
  if constexpr (sizeof(T) == 4) {
    imgC = reinterpret_cast<unsigned char *>(Ct + NB * npad);
    imgR = imgC + (size_t)nbk * gu::IMAGE;
    err = reinterpret_cast<int *>(imgR + (size_t)nbk * gu::IMAGE);
    M3_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
    M3_CUDA(cudaFuncSetAttribute(k_gjb_update_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, gu::SMEM_ALLOC));
  } else {
    M3_CUDA(cudaFuncSetAttribute(k_gjb_update<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gj_smem<T>()));
  }
  // Large matrices: the next diagonal block is updated and inverted on a second stream while the other tiles are
  // updated on all SMs but one. That pays when the update (223 us at 116 blocks, with their square) is longer than the
  // extra product of the diagonal block's CTA (35 us): from 48 blocks on.
  GjSide side;
  const bool ahead = sizeof(T) == 4 && nbk >= 48;
  if (ahead) M3_TRY(side.open());
  for (int k = 0; k < nbk; ++k) {
    const int kb = k * NB, nb = std::min(NB, n - kb);
    if (!ahead || k == 0) {
      k_gjb_diag<T><<<1, 256, 0, s>>>(A, ld, kb, nb, Dinv, DinvT, nullptr, nullptr, npad); count_launch();
    } else {
      M3_CUDA(cudaStreamWaitEvent(s, side.inverted, 0));
    }
    k_gjb_panels<T><<<dim3(nbk, GJ_PANEL_CTAS<T>), 256, gj_smem<T>(), s>>>(A, ld, n, k, nb, Dinv, DinvT, npad, R, Ct, imgC,
                                                                            imgR); count_launch();
    if (nbk == 1) break;
    if (ahead && k + 1 < nbk) {
      const int kb1 = kb + NB, nb1 = std::min(NB, n - kb1);
      M3_CUDA(cudaEventRecord(side.panel, s));
      M3_CUDA(cudaStreamWaitEvent(side.stream, side.panel, 0));
      k_gjb_diag<T><<<1, 256, gj_smem<T>(), side.stream>>>(A, ld, kb1, nb1, Dinv, DinvT, Ct, R, npad); count_launch();
      M3_CUDA(cudaEventRecord(side.inverted, side.stream));
    }
    if constexpr (sizeof(T) == 4) {
      k_gjb_update_tc<<<(unsigned)std::min<size_t>(ntile, ahead ? 151 : 152), gu::THREADS, gu::SMEM_ALLOC, s>>>(
          A, ld, n, k, ahead ? k + 1 : -1, ntile, imgC, imgR, err);
    } else {
      k_gjb_update<T><<<(unsigned)ntile, 256, gj_smem<T>(), s>>>(A, ld, n, k, npad, R, Ct);
    }
    count_launch();
  }
  const unsigned g = (unsigned)((n + 31) / 32);
  k_gjb_mirror<T><<<dim3(g, g), 256, 0, s>>>(A, ld, n); count_launch();
  M3_CUDA(cudaGetLastError());
  if (err) {
    int h = 0;
    M3_CUDA(cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, s));
    M3_CUDA(cudaStreamSynchronize(s));
    if (h) {
      set_error("coarse inverse: a bounded wait gave up (code " + std::to_string(h) + ")");
      return M3SPH_ERR_CUDA;
    }
  }
  return M3SPH_OK;
}

// free-dof inverse of the level matrix (from its block rows): A (nf rows of dense_ld(nf) values) = (K
// restricted to the free dofs)^-1
template <typename T>
int dense_inverse_blocked(const Level &L, const T *B, T *A, T *work, const int *cmap, int nf, cudaStream_t s) {
  const int ld = dense_ld(nf);
  M3_CUDA(cudaMemsetAsync(A, 0, sizeof(T) * (size_t)nf * ld, s));
  k_dense_from_bsr<T><<<L.nnod, 64, 0, s>>>(L.bsr_ptr, L.bsr_col, B, L.nnod, (size_t)L.nnzb, cmap, ld, A); count_launch();
  return gj_blocked_inverse<T>(A, ld, nf, work, s);
}
template int dense_inverse_blocked<double>(const Level &, const double *, double *, double *, const int *, int,
                                           cudaStream_t);
template int dense_inverse_blocked<float>(const Level &, const float *, float *, float *, const int *, int,
                                          cudaStream_t);

// y[i] (+)= sum_j A[cmap[i]][j] x[j], x compact on the free dofs (zero padded to the row stride), 0 on fixed
// dofs: one warp per dof, 16-byte loads of both (the rows are 16-byte aligned), so a row of 2,430 values is
// 19 independent loads a lane. (Scalar loads with the operand read through the dof list, after a
// memset of y: 9.0 us at 2.3k free dofs; now 4.6.)
template <typename T, typename X>
__global__ void __launch_bounds__(256) k_dense_gemv(const T *__restrict__ A, int ld, int n, const int *__restrict__ cmap,
                                                    const X *__restrict__ x, X *__restrict__ y, int accumulate) {
  grid_dep();
  const int i = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= n) return;
  const int row = cmap[i];
  if (row < 0) {
    if (lane == 0) y[i] = X(0);
    return;
  }
  const T *a = A + (size_t)row * ld;
  X s = 0;
#pragma unroll 4
  for (int j = 4 * lane; j < ld; j += 128) {
    T av[4];
    X xv[4];
    gj_ld4(a + j, av);
    gj_ld4(x + j, xv);
#pragma unroll
    for (int k = 0; k < 4; ++k) s += (X)av[k] * xv[k];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) y[i] = accumulate ? y[i] + s : s;
}
// a - b on the free dofs, compact
__global__ void k_sub_compact(const double *a, const double *b, const int *cmap, double *out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && cmap[i] >= 0) out[cmap[i]] = a[i] - b[i];
}
template <typename T> int bsr_apply(const Level &L, const T *B, const T *x, T *y, cudaStream_t s);

// FP64 coarse solve d = A^-1 r from the FP32 inverse A32 and the FP64 operator B64 of the coarsest
// level: d = A32 r, then `sweeps` steps of iterative refinement d += A32 (r - A d); xfree holds r on the
// free dofs (compact) and is overwritten
int coarse_refined(const Level &L, const float *A32, const double *B64, const double *r, double *d, double *t,
                   int sweeps, const int *cmap, double *xfree, int nf, cudaStream_t s) {
  const int n = L.ndof, ld = dense_ld(nf);
  const unsigned g = (unsigned)((n + 7) / 8);
  launch_pdl(k_dense_gemv<float, double>, g, 256, 0, s, A32, ld, n, cmap, xfree, d, 0); count_launch();
  for (int k = 0; k < sweeps; ++k) {
    M3_TRY(bsr_apply<double>(L, B64, d, t, s));
    k_sub_compact<<<(n + 255) / 256, 256, 0, s>>>(r, t, cmap, xfree, n); count_launch();
    launch_pdl(k_dense_gemv<float, double>, g, 256, 0, s, A32, ld, n, cmap, xfree, d, 1); count_launch();
  }
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}

__global__ void k_d2f_n(const double *a, float *b, size_t n) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}
// FP32 inverse of the FP64 coarsest operator (its blocks rounded to FP32)
int dense_inverse_from64(const Level &L, const double *B64, float *B32tmp, float *A, float *work, const int *cmap,
                         int nf, cudaStream_t s) {
  const size_t nb = 9 * (size_t)L.nnzb;
  k_d2f_n<<<(unsigned)((nb + 255) / 256), 256, 0, s>>>(B64, B32tmp, nb); count_launch();
  return dense_inverse_blocked<float>(L, B32tmp, A, work, cmap, nf, s);
}

// d = A^-1 r on the free dofs (r compact in xfree), 0 on the fixed ones
template <typename T>
int dense_gemv(const T *A, int n, int nf, const int *cmap, const T *xfree, T *y, cudaStream_t s) {
  launch_pdl(k_dense_gemv<T, T>, (n + 7) / 8, 256, 0, s, A, dense_ld(nf), n, cmap, xfree, y, 0);
  count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}
template int dense_gemv<double>(const double *, int, int, const int *, const double *, double *, cudaStream_t);
template int dense_gemv<float>(const float *, int, int, const int *, const float *, float *, cudaStream_t);

}  // namespace m3sph
