// Shared device/host declarations of the m3sph CUDA library (sm_103a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <string>
#include <utility>
#include <vector>

#include "../../include/m3sph.h"

struct m3sph_mesh;

namespace m3sph {

constexpr int NNODEL = 10;        // P2 velocity nodes per element
constexpr int NUDOF = 30;         // velocity dofs per element
constexpr int NPACK = 465;        // packed lower triangle of a 30x30 symmetric matrix
constexpr int NIP = 14;           // quadrature points (ip_tetrahedron.m:100-123)
constexpr int MAX_COLORS = 128;

// packed lower-triangle index of (r, c), r >= c, column-major (MUTILS sparse_create layout)
__host__ __device__ constexpr int pack_idx(int r, int c) { return c * (2 * NUDOF - c + 1) / 2 + (r - c); }

// Element matrices are stored as vectorised SoA: packed entry k of element e of a level with nel
// elements lives at ((k / V) * nel + e) * V + k % V with V = 4 (float) or 2 (double), so one
// thread loads 16 bytes at a time and a warp's loads stay contiguous (512 B per load).
template <typename T> struct KVec;
template <> struct KVec<float> { static constexpr int V = 4; };
template <> struct KVec<double> { static constexpr int V = 2; };
template <typename T>
__host__ __device__ __forceinline__ size_t kidx(int k, size_t e, size_t nel) {
  constexpr int V = KVec<T>::V;
  return ((size_t)(k / V) * nel + e) * V + (k % V);
}
// packed entry k -> (row r, column c) of the lower triangle, column-major (k = 0: (0,0), 1: (1,0), ...)
__host__ __device__ constexpr int unpack_c(int k) {
  int c = 0;
  while (k >= 30 - c) { k -= 30 - c; ++c; }
  return c;
}
__host__ __device__ constexpr int unpack_r(int k) {
  int c = 0;
  while (k >= 30 - c) { k -= 30 - c; ++c; }
  return c + k;
}
// y_hi + y_lo += (v_hi + v_lo)(x_hi + x_lo) in double-float: the product's rounding error by FMA,
// the sum's by Knuth's two-sum (used by the FP64-accurate outer operator built from FP32 parts)
__device__ __forceinline__ void df_mac(float vh, float vl, float xh, float xl, float &sh, float &sl) {
  const float p = vh * xh;
  float e = fmaf(vh, xh, -p);
  e = fmaf(vh, xl, e);
  e = fmaf(vl, xh, e);
  const float s = sh + p;
  const float bb = s - sh;
  const float err = (sh - (s - bb)) + (p - bb);
  sh = s;
  sl += err + e;
}

#ifdef __CUDACC__
// two FP32 values in one 64-bit register, and one instruction for both
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// Sums of three values over groups of W lanes (all lanes of a warp call it): the lanes that start quarter c of a
// group get sum c. Two exchanges split the values over the quarters, so it takes 2 + 1 + log2(W / 4) additions
// and not 3 log2(W).
template <int W, typename T>
__device__ __forceinline__ T lane_sum3(T s0, T s1, T s2) {
  const int lane = threadIdx.x % W;
  const bool h = lane & (W / 2), q = lane & (W / 4);
  T a = (h ? s2 : s0) + __shfl_xor_sync(0xffffffffu, h ? s0 : s2, W / 2);
  const T t = __shfl_xor_sync(0xffffffffu, h ? s1 : T(0), W / 2);
  const T b = (h ? T(0) : s1) + t;
  a = (q ? b : a) + __shfl_xor_sync(0xffffffffu, q ? a : b, W / 4);
#pragma unroll
  for (int o = W / 8; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}
#endif

// Block reduction whose last block finishes it: v[k] summed over the grid in a fixed order (threads of a
// block by shuffles, then blocks in order), so the result does not depend on scheduling. `cnt` is 0 before
// and after. Returns true in the last block, whose thread 0 holds the sums. Blocks of up to 256 threads.
#ifdef __CUDACC__
template <int NV>
__device__ __forceinline__ bool block_reduce_last(double (&v)[NV], double *partials, unsigned *cnt) {
  __shared__ double sh[NV][8];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  auto block_sum = [&]() {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
      if (lane == 0) sh[k][wid] = v[k];
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        double t = lane < nw ? sh[k][lane] : 0.0;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        v[k] = t;
      }
    }
  };
  block_sum();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) partials[k * gridDim.x + blockIdx.x] = v[k];
    __threadfence();
    last = atomicInc(cnt, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    v[k] = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x) v[k] += __ldcg(partials + k * gridDim.x + i);
  }
  block_sum();
  return true;
}
#endif

template <typename T> constexpr int kpad() { return ((NPACK + KVec<T>::V - 1) / KVec<T>::V) * KVec<T>::V; }

void set_error(const std::string &msg);
// host-side count of kernel launches issued by this library (reported by m3sph_launch_count)
void count_launch();
int cuda_fail(cudaError_t e, const char *what);

#define M3_TRY(call)                 \
  do {                               \
    int _s = (call);                 \
    if (_s != M3SPH_OK) return _s;   \
  } while (0)

#define M3_CUDA(call)                                  \
  do {                                                 \
    cudaError_t _e = (call);                           \
    if (_e != cudaSuccess) return cuda_fail(_e, #call); \
  } while (0)

// Programmatic dependent launch. A kernel started with launch_pdl may be placed on the chip before the one ahead
// of it in its stream has finished; grid_dep() waits for that. Before grid_dep() a kernel may read only what the
// kernel right ahead of it does not write (operator data, connectivity, weights): that one has passed its own
// grid_dep() or run to its end, so all earlier ones have finished.
// A grid that leaves half of the SMs free allows its successor's start at once; with larger ones the early
// blocks take room and bandwidth from it (one velocity solve at 30,720 elements: 161 ms if they do, 144 if not),
// and the successor starts as its blocks end. An iteration of the velocity solve is about 30 short kernels, whose
// gaps and start-up latencies were a quarter of its time: 156 -> 148 ms at 30,720 elements, 87 -> 75 ms at 3,840.
#ifdef __CUDACC__
constexpr unsigned PDL_EARLY_GRID = 76;
__device__ __forceinline__ void grid_dep() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
  if (gridDim.x <= PDL_EARLY_GRID) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
void launch_pdl(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, k, std::forward<A>(a)...);   // its error is picked up by the caller's cudaGetLastError
}
#endif

// quadrature / shape-function tables (computed on the host, copied to constant memory)
struct ShapeTables {
  double ipw[NIP];
  double NP[NIP][4];
  double NU[NIP][10];
  double dNU[NIP][10][3];
  double N20[NIP][20];
  double dN20[NIP][20][3];
};
void build_shape_tables(ShapeTables &t);
int upload_shape_tables();

// device buffers of one multigrid level
struct Level {
  int nel = 0, nnod = 0, nvnod = 0, ndof = 0;
  int nfree = 0;
  std::vector<int> cstart;            // colour ranges of `corder` (host)
  int *el2nod = nullptr;              // [10][nel], 0-based
  int *corder = nullptr;              // [nel] element ids sorted by colour (per-colour kernels)
  uint8_t *freemask = nullptr;        // [ndof], 1 = free dof
  double *K64 = nullptr;              // [465][nel] rotated, masked element matrices
  float *K32 = nullptr;
  float *KL32 = nullptr;              // K64 - K32 rounded to FP32 (finest level, mixed precision)
  double *Dinv64 = nullptr;           // [ndof] inverse diagonal (0 on fixed dofs)
  float *Dinv32 = nullptr;
  // children (coarse levels): fine index of child k, and parent-local vertex indices
  int *child = nullptr;               // [8][nel]
  uint32_t *child_vloc = nullptr;     // [8][nel], 4 x 4-bit parent-local node index (0..9)
  // transfer to the next coarser level (levels 0..nmg-2)
  int *P_ptr = nullptr, *P_col = nullptr;   // fine node rows
  float *P_w = nullptr;
  int *R_ptr = nullptr, *R_col = nullptr;   // coarse node rows (transpose)
  float *R_w = nullptr;
  // assembled 3x3-block CSR of the level operator (coarse levels): one launch per application
  int nnzb = 0;
  int *bsr_ptr = nullptr, *bsr_col = nullptr;   // [nnod+1], [nnzb]
  int *bsr_cptr = nullptr, *bsr_contrib = nullptr;   // per block: contributions e*100 + a*10 + b
  double *B64 = nullptr;                         // [nnzb][9]
  float *B32 = nullptr;
  // streamed apply (finest level): phase 1 streams the element matrices in chunks of 32
  // elements and writes element outputs Ye; phase 2 sums them per node in a fixed order
  int nchunk = 0, sa_grid = 0;
  int *chunk_conn = nullptr;          // [nchunk][10][32] node ids of the chunk's elements (0: unused lane)
  float *ye32 = nullptr;              // [nel][30] element outputs
  int nchunk8 = 0;                    // FP64-accurate operators: chunks of 8 elements
  int *chunk_conn8 = nullptr;         // [nchunk8][10][8]
  double *ye64 = nullptr;             // [nel][30]
  int *g_ptr = nullptr;               // [nnod + 1] node -> incident (element, local node) entries
  int *g_idx = nullptr;               // [10 nel] offsets e * 30 + 3 * local node into Ye, element order
  int *sa_err = nullptr;              // bounded waits of the streamed apply that gave up (bit mask)
  // partially assembled FP32 operator (finest level): per integration point the 3x3 factor
  // sqrt(w eta) d xi / d x, tiles of 64 elements [tile][NIP][9][32][2] (lane, lane + 32); per node RR's angles; slots: the
  // nodes of every tile
  float *pa32 = nullptr;
  float4 *pa_trig = nullptr;          // [nnod] (cos theta, sin theta, cos phi, sin phi)
  float4 *pa_xc = nullptr;            // [nnod] operand, masked, global Cartesian components
  float4 *pa_yb = nullptr;            // [slots] sums of a tile's element outputs, node-major
  int *pa_tptr = nullptr;             // [tiles + 1] first slot of a tile
  int2 *pa_slot = nullptr;            // [slots] {position in pa_yb, begin | end << 16 of its entries}
  uint16_t *pa_ent = nullptr;         // [tiles][640] entries: 3 a * 65 + element of the tile
  int *pa_nptr = nullptr;             // [nnod + 1] a node's range of pa_yb
  bool pa_ready = false;              // pa32 written by the last operator set-up
  // host copies needed at set-up
  std::vector<int> h_el2nod_orig;     // [nel][10], 0-based
};

struct Finest {
  double *gcoord = nullptr;           // [3][nnod]
  double *gcoord_sph = nullptr;       // [3][nnod]
  double *RR = nullptr;               // [9][nnod] (theta,phi,r)->(x,y,z), row-major 3x3
  uint8_t *cls = nullptr;             // [nel]
  int *iso_slot = nullptr;            // [nel], -1 if not iso
  double *cubic = nullptr;            // [60][niso] (theta,phi,r) x 20 nodes, X-90 frame
  int niso = 0;
  double *visc = nullptr, *dens = nullptr;  // [nvnod]
  double *G64 = nullptr;              // [120][nel]: G[p][3n+c]
  double *M64 = nullptr;              // [10][nel] packed lower 4x4
  double *Fbe = nullptr;              // [nel][30]
  double *BCe = nullptr;              // [nel][30] K_unmasked * Ufix per element
  double *Fb = nullptr;               // [ndof] assembled, rotated
  double *LiMM = nullptr;             // [nvnod] inverse lumped M
  int *err = nullptr;                 // device error flags
};

// state of a velocity solve's CG, at scal + CG_STATE: the host sets it, the step kernel ends the loop
enum { CG_STATE = 24, CG_TOL = 24, CG_SQ, CG_PREV, CG_IT, CG_LIMIT, CG_LEARNED, CG_STATUS, CG_RR0, CG_STATE_END };
enum { CG_RUN = 0, CG_CONVERGED, CG_NAN, CG_STALLED, CG_LIMIT_REACHED, CG_WAIT_ERROR };
constexpr int CG_LOOP_MAX = 256;    // iterations of a captured loop before the host looks at it

struct Coarse {
  int n = 0;                          // dofs of the coarsest level
  int nf = 0;                         // its free dofs: the dense inverse is nf rows of dense_ld(nf) values
  int *cmap = nullptr;                // [n] level dof -> compact index, -1 for a fixed dof
  double *A64 = nullptr;              // dense inverse
  float *A32 = nullptr;
  bool refine64 = false;              // FP64 path: FP32 inverse + iterative refinement against B64
  float *B32tmp = nullptr;            // [9][nnzb] FP32 copy of the coarsest FP64 blocks (refinement)
  double *t64 = nullptr;              // [n] refinement residual
  double *x64 = nullptr;              // [dense_ld(nf)] operand of the coarse solve on the free dofs (compact)
  float *x32 = nullptr;
};

// Cartesian copy of a nodal vector for the partially assembled operator: a pass that writes (theta,
// phi, r) values of a node also writes xc[node] when xc is set
struct PaCart {
  const float4 *trig = nullptr;       // [nnod] (cos theta, sin theta, cos phi, sin phi)
  float4 *xc = nullptr;
};
// masked local (theta, phi, r) values of a node -> global Cartesian components
__device__ __forceinline__ float4 pa_to_cart(const float4 tr, float x0, float x1, float x2) {
  const float a = tr.x * x0 + tr.y * x2;             // ct x0 + st x2
  return make_float4(tr.z * a - tr.w * x1, tr.w * a + tr.z * x1, tr.x * x2 - tr.y * x0, 0.f);
}

// threads of a node-sum pass that go to the nv vertices, four each, in whole warps; edge nodes follow, one
// thread each
__host__ __device__ __forceinline__ int gather_threads4(int nv) { return (4 * nv + 31) & ~31; }

// error words that bounded waits set when they give up (either may be null)
struct WaitWords {
  const int *w[2];
};

// scratch of a grid reduction
struct Reduction {
  double *partials;
  unsigned *cnt;
};

struct SetupArgs {
  int nel, nnod;
  const int *el2nod;        // [10][nel]
  const uint8_t *cls;
  const int *iso_slot;
  const double *cubic;      // [60][niso]
  int niso;
  const double *gcoord, *gcoord_sph, *RR;
  const double *visc, *dens;
  const uint8_t *freemask;
  double g, Bscale, Dens0, minVisc, maxVisc;
  double *K64; float *K32; double *G64; double *M64; double *Fbe;
  float *KL32;              // low FP32 part of K64 - K32 (double-float outer operator) or nullptr
  float *PA32;              // [tile][NIP][9][32][2] partially assembled factors or nullptr
  const double *ufix;       // [3*nnod] prescribed values (rotated frame) or nullptr
  double *BCe;              // [nel][30] element K_unmasked * ufix (when ufix != nullptr)
  int *err;
};

int slm_build(m3sph_mesh *M, const m3sph_level &f0);
int slm_advect_resident(m3sph_mesh *M, const double *U_soa, double *T, double dt, const m3sph_slm_opts *o,
                        bool first_step, m3sph_locate_info *info);
int stokes_velocity_soa(m3sph_mesh *M, double *dst);
int stokes_resident_solve(m3sph_mesh *M, const m3sph_opts *opts, bool zero_p, m3sph_info &inf);
int stokes_calc_dt(m3sph_mesh *M, double dt_adv_limit, double dtmax, double *dt, double *dt_adv);
int diffusion_resident(m3sph_mesh *M, double *T, double dt, int *nit);
int stokes_set_pressure(m3sph_mesh *M, const double *P);
int ml_build(m3sph_mesh *M);
int ml_features(m3sph_mesh *M, const double *h_visc);
template <typename T>
int ml_sweep(m3sph_mesh *M, int j, const T *r0, const T *kd, const T *Dinv, T *tmp, T *d, const PaCart &pc, bool first);
int ml_init_kernels();
int ml_set_infer(int v);
int ml_check(m3sph_mesh *M);
int *ml_error_word(m3sph_mesh *M);
bool ml_ready(m3sph_mesh *M);
int ml_add_samples(m3sph_mesh *M, const double *r, const double *err, int stride, int offset);
int ml_reserve(m3sph_mesh *M, long cap);
int ml_set_params(m3sph_mesh *M, const float *h);
int ml_get_params(m3sph_mesh *M, float *h);
int ml_epoch(m3sph_mesh *M, int batch, float lr, unsigned long long seed, double *mse);
int ml_gradients(m3sph_mesh *M, const float *hX, const float *hT, int n, float *hgrad, double *loss);
int ml_forward(m3sph_mesh *M, const float *hX, int n, float *hY);
int ml_nparam();
long ml_count(m3sph_mesh *M);
void ml_mark_trained(m3sph_mesh *M, bool t);

}  // namespace m3sph

struct m3sph_mesh {
  int device = 0;
  int nmg = 0;
  cudaStream_t stream = nullptr;
  std::vector<m3sph::Level> lev;
  m3sph::Finest fin;
  m3sph::Coarse coarse;
  int precision = 0;                  // 0 fp64, 1 fp32 V-cycle
  m3sph_physics phys{};
  double last_setup_ms = 0.0;
  bool have_operator = false;
  std::vector<int> h_ifix;            // 0-based fixed dofs (rotated frame)
  std::vector<double> h_vfix;
  double *Ufix = nullptr;             // [ndof0] prescribed values (rotated frame)
  double *bc_rhs = nullptr;           // K1_full * Ufix
  bool has_nonzero_fix = false;
  bool bc_stale = false;              // prescribed values changed since the last operator rebuild
  // scratch
  std::vector<void *> work;           // device buffers owned by the workspace
  void *wk = nullptr;                 // host-side workspace descriptor
  void (*wk_free)(void *) = nullptr;
  struct CgGraph { double *key; cudaGraphExec_t exec; unsigned long long kernels; };
  std::vector<CgGraph> graphs;        // captured MG-PCG loops and their kernels per iteration
  bool use_graphs = true;
  bool df_outer = true;               // double-float outer operator on the mixed path
  bool split_apply = true;            // 4-warp split element products where the streamed ones are off
  int ml_schedule = 1;                // learned smoothing per side: 0 learned-Jacobi-learned, 1 one learned sweep
  float ml_omega = 1.0f;              // relaxation weight of the learned correction
  void *ml = nullptr;                 // learned smoother state
  void (*ml_free)(void *) = nullptr;
  int smoother = 0;                   // 0 Jacobi, 1 learned smoother on the two finest levels
  bool smoother_active = false;       // learned smoother in use for the current solve
  int smoother_fallbacks = 0;
  double r_min = 0.0, r_max = 0.0;    // shell radii (features)
  double Lx = 0.0, Ly = 0.0, Lz = 0.0; // extents of the finest mesh (MESH.Lx/Ly/Lz, init_mesh_curved_p.m:264-272)
  double rad_max = 0.0;               // largest node radius sqrt(x^2+y^2+z^2) (rock_prop.m:10-11)
  double *T = nullptr;                // [nnod] resident temperature of the time step
  double *Usoa = nullptr;             // [3][nnod] Cartesian velocity handed to the advection
  long long ts_steps = 0;             // time steps taken since the temperature was set
  double ts_time = 0.0;               // model time accumulated by the time steps
  void *diff = nullptr;               // thermal-diffusion state
  void (*diff_free)(void *) = nullptr;
  void *slm = nullptr;                // advection / point-location state
  void (*slm_free)(void *) = nullptr;
  double *red = nullptr;              // reduction partials
  unsigned *red_cnt = nullptr;        // finished blocks of a reduction (0 between kernels)
  double *scal = nullptr;             // device scalars
  double *h_scal = nullptr;           // pinned host mirror
};
