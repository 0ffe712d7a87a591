// Partially assembled FP32 operator of the finest level (the V-cycle operator).
//
// The stored form streams the 465 packed entries of every element matrix (1,860 B per element in
// FP32). This form stores, per element and integration point, only the 3x3 factor
//   A_q = sqrt(w_q eta_q) R_cls^T J_dbl,q      (A[c][j] = d xi_j / d x_c, global Cartesian)
// (J_dbl and w = detJ_CS detJ_SL w_ip as in assembly_stokes_els_*_opt.m:134-164, eta the
// vertex-interpolated viscosity of calc_element_visc.m:5-7, R_cls the element's frame rotation
// undone), 14 x 9 FP32 = 504 B per element, and forms the product on the fly: with u the element's
// velocities in global Cartesian components (node dofs rotated by RR, make_rotation_matrix.m),
//   L = grad u (scaled by sqrt(w eta)),  S = L + L^T - 2/3 tr(L) I,
//   y_n += S grad N_n (scaled)
// which is K = sum_q w eta B^T D B with the deviatoric "23rd" D (C1 = 4/3, C2 = -2/3) of
// assembly_stokes_els_*_opt.m:201-317, written in the rotation-invariant tensor form. The reference
// gradient of a P2 field is linear in the barycentric coordinates, so the element's velocities are
// turned once into the 12 coefficients per component of
//   g_j = d u / d xi_j = sum_m lam_m E_jm        (j < 3, m < 4)
// and the result is accumulated as the moments F_jm += lam_m T_j of the same form: 36 + 36 FMA per
// point in place of 90 + 90 with the 10 nodal derivatives.
//
// Node work is done once per node, not once per element and node (10 nodes an element, about 7
// entries a node): the passes that write a velocity vector also write it masked and rotated to
// global Cartesian components as one float4 per node (xc), and the rotation back and the mask of the
// result are in the node sums.
//
// Elements: one warp per tile of 64 consecutive elements, two per lane held in packed registers
// (fma.rn.f32x2), so one instruction works on both: a version with one element per lane issued
// 3,700 instructions per 32 elements and kept the schedulers busier than the FMA pipe. Lane 0 streams
// the tile's factors (stored tile by tile, 2-point chunks) through a private ring of 4 stages with bulk
// copies while the lanes gather u (one 16-byte load per node). The 64 elements are the children of 8
// neighbouring parents, so their 640 node entries fall on about 190 nodes: the warp sums its element
// outputs per node in shared memory in a fixed order and writes one float4 per tile node (a "slot").
// Node sums then add about 2 slots per node in tile order, so the result does not depend on
// scheduling.
//
// Measured (tiles + node sums): 104.9 + 27.7 us -> 68.7 + 7.8 us at 491,520 elements, 54.3 + 14.8 ->
// 35.7 + 5.9 at 245,760, 11.0 + 7.9 -> 8.3 + 4.3 at 30,720 (before: one element per thread, 64 KB factor
// tile per 128 elements, rotations and masks per element, 120 B of outputs per element summed by 7
// entries a node). 210 registers and 25 KB of shared memory leave 8 warps (512 elements) per SM: FMA pipe
// 41 %, DRAM 54 %; a quarter of a warp's time is the wait for the gathers at its start.
// Waits on the copies are bounded in time; one that gives up sets a bit of the level's error word.
#include <vector>

#include "common.cuh"

namespace m3sph {

__constant__ uint64_t c_pa_lam2[NIP][4];  // barycentric coordinates of the integration points, FP32 pairs

// end vertices of the edge nodes 4..9 (edges 1-2, 2-3, 3-4, 4-1, 1-3, 2-4 of the P2 numbering)
__device__ __forceinline__ constexpr int pa_ea(int k) { return k == 1 ? 1 : k == 2 ? 2 : k == 5 ? 1 : 0; }
__device__ __forceinline__ constexpr int pa_eb(int k) { return k == 0 ? 1 : k == 1 ? 2 : k == 4 ? 2 : 3; }

int pa_upload_tables() {
  ShapeTables t;
  build_shape_tables(t);
  float lam[NIP][4][2];
  for (int q = 0; q < NIP; ++q)
    for (int v = 0; v < 4; ++v) lam[q][v][0] = lam[q][v][1] = (float)t.NP[q][v];
  static_assert(sizeof(lam) == sizeof(uint64_t) * NIP * 4, "pairs");
  M3_CUDA(cudaMemcpyToSymbol(c_pa_lam2, lam, sizeof(lam)));
  return M3SPH_OK;
}

// per node (cos theta, sin theta, cos phi, sin phi) from the rotation blocks RR (row-major
// 3x3, [9][nnod]): RR = [cp ct, -sp, cp st; sp ct, cp, sp st; -st, 0, ct]
__global__ void k_pa_trig(const double *__restrict__ RR, int nnod, float4 *__restrict__ trig) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nnod) return;
  const double ct = RR[8 * (size_t)nnod + n], st = -RR[6 * (size_t)nnod + n];
  const double cp = RR[4 * (size_t)nnod + n], sp = -RR[1 * (size_t)nnod + n];
  trig[n] = make_float4((float)ct, (float)st, (float)cp, (float)sp);
}

constexpr int PA_E = 64;                             // elements per tile: lane l works on l and l + 32
constexpr int PA_CHUNK_IP = 2;                       // integration points per ring stage
constexpr int PA_NCHUNK = NIP / PA_CHUNK_IP;
constexpr int PA_CHUNK = PA_CHUNK_IP * 9 * PA_E;     // floats
constexpr int PA_STAGES = 4;
constexpr int PA_LD = PA_E + 1;                      // staging stride of the element outputs
constexpr unsigned long long PA_TIMEOUT_NS = 1000000000ull;
static_assert(NIP % PA_CHUNK_IP == 0 && PA_CHUNK * 4 % 16 == 0, "whole chunks, 16-byte copies");
static_assert(30 * PA_LD <= PA_STAGES * PA_CHUNK, "element outputs fit in the ring");
static_assert(10 * PA_E <= 32767 && 27 * PA_LD + PA_E <= 65535, "16-bit tile tables");

// floats of the factor array: whole tiles
size_t pa_factor_floats(int nel) { return (size_t)((nel + PA_E - 1) / PA_E) * NIP * 9 * PA_E; }

// Tile tables. A tile's slots are its nodes, those with most entries first (lanes of a round then have
// loops of similar length), else in order of first occurrence; a slot lists the tile's (element, local
// node) entries of its node in that order. Slots are written to node-major positions: the sums of a
// node are contiguous, in tile order.
int pa_build(Level &L, const double *RR, cudaStream_t s) {
  const int nel = L.nel, nnod = L.nnod, ntile = (nel + PA_E - 1) / PA_E;
  const int *en = L.h_el2nod_orig.data();
  std::vector<int> tptr(ntile + 1, 0), last(nnod, -1), pos(nnod), nptr(nnod + 1, 0);
  for (int t = 0; t < ntile; ++t) {
    const size_t b = (size_t)t * PA_E * 10, f = std::min((size_t)(t + 1) * PA_E, (size_t)nel) * 10;
    int ns = 0;
    for (size_t i = b; i < f; ++i)
      if (last[en[i]] != t) {
        last[en[i]] = t;
        nptr[en[i] + 1]++;
        ++ns;
      }
    tptr[t + 1] = tptr[t] + ns;
  }
  for (int n = 0; n < nnod; ++n) nptr[n + 1] += nptr[n];
  const size_t nslot = tptr[ntile];
  std::vector<int> fill(nptr.begin(), nptr.end() - 1);
  std::vector<int2> slot(nslot);
  std::vector<uint16_t> ent((size_t)ntile * 10 * PA_E, 0);
  std::fill(last.begin(), last.end(), -1);
  int node[10 * PA_E], cnt[10 * PA_E], order[10 * PA_E], nxt[10 * PA_E], byc[10 * PA_E + 2];
  for (int t = 0; t < ntile; ++t) {
    const size_t b = (size_t)t * PA_E * 10, f = std::min((size_t)(t + 1) * PA_E, (size_t)nel) * 10;
    int ns = 0;
    for (size_t i = b; i < f; ++i) {
      const int n = en[i];
      if (last[n] != t) {
        last[n] = t;
        pos[n] = ns;
        node[ns] = n;
        cnt[ns++] = 0;
      }
      cnt[pos[n]]++;
    }
    // stable counting sort, largest count first
    std::fill(byc, byc + 10 * PA_E + 2, 0);
    for (int k = 0; k < ns; ++k) byc[10 * PA_E - cnt[k] + 1]++;
    for (int c = 0; c <= 10 * PA_E; ++c) byc[c + 1] += byc[c];
    for (int k = 0; k < ns; ++k) order[byc[10 * PA_E - cnt[k]]++] = k;
    int beg = 0;
    for (int i = 0; i < ns; ++i) {
      const int k = order[i];
      slot[tptr[t] + i] = make_int2(fill[node[k]]++, beg | ((beg + cnt[k]) << 16));
      nxt[k] = beg;
      beg += cnt[k];
    }
    for (size_t i = b; i < f; ++i)
      ent[b + nxt[pos[en[i]]]++] = (uint16_t)(3 * ((i - b) % 10) * PA_LD + (i - b) / 10);
  }
  M3_CUDA(cudaMalloc(&L.pa_tptr, sizeof(int) * tptr.size()));
  M3_CUDA(cudaMalloc(&L.pa_slot, sizeof(int2) * nslot));
  M3_CUDA(cudaMalloc(&L.pa_ent, sizeof(uint16_t) * ent.size()));
  M3_CUDA(cudaMalloc(&L.pa_nptr, sizeof(int) * nptr.size()));
  M3_CUDA(cudaMalloc(&L.pa_yb, sizeof(float4) * nslot));
  M3_CUDA(cudaMalloc(&L.pa_xc, sizeof(float4) * (size_t)nnod));
  M3_CUDA(cudaMalloc(&L.pa_trig, sizeof(float4) * (size_t)nnod));
  M3_CUDA(cudaMemcpyAsync(L.pa_tptr, tptr.data(), sizeof(int) * tptr.size(), cudaMemcpyHostToDevice, s));
  M3_CUDA(cudaMemcpyAsync(L.pa_slot, slot.data(), sizeof(int2) * nslot, cudaMemcpyHostToDevice, s));
  M3_CUDA(cudaMemcpyAsync(L.pa_ent, ent.data(), sizeof(uint16_t) * ent.size(), cudaMemcpyHostToDevice, s));
  M3_CUDA(cudaMemcpyAsync(L.pa_nptr, nptr.data(), sizeof(int) * nptr.size(), cudaMemcpyHostToDevice, s));
  k_pa_trig<<<(nnod + 255) / 256, 256, 0, s>>>(RR, nnod, L.pa_trig);
  count_launch();
  M3_CUDA(cudaGetLastError());
  M3_CUDA(cudaStreamSynchronize(s));                 // the copies above read host vectors of this function
  return M3SPH_OK;
}

__device__ __forceinline__ uint32_t pa_smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long pa_gtime() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool pa_mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool pa_mbar_wait(uint32_t bar, uint32_t parity) {
  if (pa_mbar_test(bar, parity)) return true;
  const unsigned long long t0 = pa_gtime();
  for (;;) {
    for (int i = 0; i < 32; ++i)
      if (pa_mbar_test(bar, parity)) return true;
    if (pa_gtime() - t0 > PA_TIMEOUT_NS) return false;
  }
}
__device__ __forceinline__ void pa_bulk_load(uint32_t dst, const float *src, uint32_t bar, uint64_t pol) {
  asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(bar),
               "r"((uint32_t)(PA_CHUNK * 4))
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst),
      "l"(src), "r"((uint32_t)(PA_CHUNK * 4)), "r"(bar), "l"(pol)
      : "memory");
}

__global__ void __launch_bounds__(32, 8)
k_pa_tile(const float *__restrict__ pa, const int *__restrict__ el2nod, int nel, const float4 *__restrict__ xc,
          const int *__restrict__ tptr, const int2 *__restrict__ slot, const uint16_t *__restrict__ ent,
          float4 *__restrict__ yb, int *__restrict__ err) {
  __shared__ __align__(128) float ring[PA_STAGES * PA_CHUNK];
  __shared__ __align__(16) uint16_t s_ent[10 * PA_E];
  __shared__ __align__(8) int2 s_slot[10 * PA_E];
  __shared__ __align__(8) unsigned long long bars[PA_STAGES];
  const int tile = blockIdx.x, lane = threadIdx.x;
  const float *src = pa + (size_t)tile * (NIP * 9 * PA_E);
  const uint32_t bar0 = pa_smem_u32(bars);
  uint64_t pol = 0;
  if (lane == 0) {
    for (int i = 0; i < PA_STAGES; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * i) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    for (int i = 0; i < PA_STAGES; ++i) pa_bulk_load(pa_smem_u32(ring + i * PA_CHUNK), src + i * PA_CHUNK, bar0 + 8 * i, pol);
  }
  // gradient coefficients of both elements: with Z_jj = u_j and Z_jm the velocity of edge node (j, m),
  // d u / d L_j = 4 sum_m lam_m Z_jm - u_j and g_j = d u / d L_j - d u / d L_3
  uint64_t E[3][3][4];                               // [component][j][m]
  {
    const int e0 = min(tile * PA_E + lane, nel - 1), e1 = min(tile * PA_E + 32 + lane, nel - 1);
    int n0[10], n1[10];
#pragma unroll
    for (int n = 0; n < 10; ++n) {
      n0[n] = el2nod[(size_t)n * nel + e0];
      n1[n] = el2nod[(size_t)n * nel + e1];
    }
    // the tile's tables arrive while the points are worked on
    const int s0 = tptr[tile], ns = tptr[tile + 1] - s0;
    for (int i = lane; i < 10 * PA_E / 8; i += 32)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(pa_smem_u32(s_ent + 8 * i)),
                   "l"(ent + (size_t)tile * (10 * PA_E) + 8 * i)
                   : "memory");
    for (int i = lane; i < ns; i += 32)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(pa_smem_u32(s_slot + i)), "l"(slot + s0 + i) : "memory");
    grid_dep();                        // factors, connectivity and tables are constants, the operand is not
    uint64_t v[10][3];
#pragma unroll
    for (int n = 0; n < 10; ++n) {
      const float4 a = xc[n0[n]], b = xc[n1[n]];
      v[n][0] = f2_pack(a.x, b.x);
      v[n][1] = f2_pack(a.y, b.y);
      v[n][2] = f2_pack(a.z, b.z);
    }
    const uint64_t m1 = f2_pack(-1.f, -1.f), c4 = f2_pack(4.f, 4.f);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const uint64_t z3[4] = {v[7][p], v[9][p], v[6][p], v[3][p]};      // Z_3m
      const uint64_t z[3][4] = {{v[0][p], v[4][p], v[8][p], v[7][p]},
                                {v[4][p], v[1][p], v[5][p], v[9][p]},
                                {v[8][p], v[5][p], v[2][p], v[6][p]}};
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const uint64_t d = f2_fma(m1, v[j][p], v[3][p]);                  // u_3 - u_j
#pragma unroll
        for (int m = 0; m < 4; ++m) E[p][j][m] = f2_fma(c4, f2_fma(m1, z3[m], z[j][m]), d);
      }
    }
  }
  uint64_t F[3][3][4];
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int m = 0; m < 4; ++m) F[p][j][m] = 0;
  __syncwarp();                                      // barriers initialised before anyone waits
#pragma unroll 1
  for (int c = 0; c < PA_NCHUNK; ++c) {
    const int st = c % PA_STAGES;
    if (!__all_sync(0xffffffffu, pa_mbar_wait(bar0 + 8 * st, (c / PA_STAGES) & 1))) {
      if (lane == 0) atomicOr(err, 32);
      asm volatile("cp.async.wait_all;" ::: "memory");
      for (int i = c; i < min(c + PA_STAGES, PA_NCHUNK); ++i)      // copies still in flight
        pa_mbar_wait(bar0 + 8 * (i % PA_STAGES), (i / PA_STAGES) & 1);
      return;
    }
    const uint64_t *stage = reinterpret_cast<const uint64_t *>(ring + st * PA_CHUNK) + lane;
#pragma unroll
    for (int h = 0; h < PA_CHUNK_IP; ++h) {
      uint64_t a[9], lam[4];
#pragma unroll
      for (int k = 0; k < 9; ++k) a[k] = stage[(h * 9 + k) * 32];
#pragma unroll
      for (int m = 0; m < 4; ++m) lam[m] = c_pa_lam2[c * PA_CHUNK_IP + h][m];
      uint64_t L[3][3];                              // L[p][c] = sum_j g_j A[c][j]
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        uint64_t g[3];
#pragma unroll
        for (int j = 0; j < 3; ++j)
          g[j] = f2_fma(lam[0], E[p][j][0], f2_fma(lam[1], E[p][j][1], f2_fma(lam[2], E[p][j][2], f2_mul(lam[3], E[p][j][3]))));
#pragma unroll
        for (int k = 0; k < 3; ++k) L[p][k] = f2_fma(g[0], a[3 * k], f2_fma(g[1], a[3 * k + 1], f2_mul(g[2], a[3 * k + 2])));
      }
      const uint64_t two = f2_pack(2.f, 2.f), mt = f2_pack(-2.f / 3.f, -2.f / 3.f);
      const uint64_t tr = f2_mul(mt, f2_add(f2_add(L[0][0], L[1][1]), L[2][2]));
      uint64_t S[3][3];
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        S[p][p] = f2_fma(two, L[p][p], tr);
#pragma unroll
        for (int k = 0; k < p; ++k) S[p][k] = S[k][p] = f2_add(L[p][k], L[k][p]);
      }
      // back to the reference directions: T[p][j] = sum_c S[p][c] A[c][j], and its moments
#pragma unroll
      for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const uint64_t t = f2_fma(S[p][0], a[j], f2_fma(S[p][1], a[3 + j], f2_mul(S[p][2], a[6 + j])));
#pragma unroll
          for (int m = 0; m < 4; ++m) F[p][j][m] = f2_fma(lam[m], t, F[p][j][m]);
        }
    }
    __syncwarp();                                    // every lane done with the stage
    if (lane == 0 && c + PA_STAGES < PA_NCHUNK)
      pa_bulk_load(pa_smem_u32(ring + st * PA_CHUNK), src + (c + PA_STAGES) * PA_CHUNK, bar0 + 8 * st, pol);
  }
  // element outputs over the ring (every copy has landed), then the sums of the tile's nodes. With
  // W_jm = sum lam_m T_j (T_3 = -sum_j T_j): vertex v: 4 W_vv - sum_m W_vm; edge (j, m): 4 (W_jm + W_mj)
  const uint64_t m1 = f2_pack(-1.f, -1.f), c4 = f2_pack(4.f, 4.f);
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    uint64_t W[4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
#pragma unroll
      for (int j = 0; j < 3; ++j) W[j][m] = F[p][j][m];
      W[3][m] = f2_mul(m1, f2_add(f2_add(W[0][m], W[1][m]), W[2][m]));
    }
    float *o = ring + p * PA_LD + lane;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 r = f2_unpack(f2_fma(c4, W[k][k], f2_mul(m1, f2_add(f2_add(W[k][0], W[k][1]), f2_add(W[k][2], W[k][3])))));
      o[3 * k * PA_LD] = r.x;
      o[3 * k * PA_LD + 32] = r.y;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const float2 r = f2_unpack(f2_mul(c4, f2_add(W[pa_ea(k)][pa_eb(k)], W[pa_eb(k)][pa_ea(k)])));
      o[3 * (4 + k) * PA_LD] = r.x;
      o[3 * (4 + k) * PA_LD + 32] = r.y;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  const int ns = tptr[tile + 1] - tptr[tile];
  for (int i = lane; i < ns; i += 32) {
    const int2 sl = s_slot[i];
    const int b = sl.y & 0xffff, f = sl.y >> 16;
    float t0 = 0.f, t1 = 0.f, t2 = 0.f;
#pragma unroll 4
    for (int k = b; k < f; ++k) {
      const float *y = ring + s_ent[k];
      t0 += y[0];
      t1 += y[PA_LD];
      t2 += y[2 * PA_LD];
    }
    yb[sl.x] = make_float4(t0, t1, t2, 0.f);
  }
}

// ---- node passes ----
// sum of a node's slots rotated back to its local frame, 0 on fixed dofs
__device__ __forceinline__ void pa_node_sum(const int *__restrict__ nptr, const float4 *__restrict__ yb, const float4 tr,
                                            const uint8_t *__restrict__ mask, int n, float (&y)[3]) {
  float t0 = 0.f, t1 = 0.f, t2 = 0.f;
  const int b = nptr[n], e = nptr[n + 1];
#pragma unroll 4
  for (int k = b; k < e; ++k) {
    const float4 v = yb[k];
    t0 += v.x;
    t1 += v.y;
    t2 += v.z;
  }
  const float c = tr.z * t0 + tr.w * t1;             // cp yx + sp yy
  const size_t i = 3 * (size_t)n;
  y[0] = mask[i] ? tr.x * c - tr.y * t2 : 0.f;
  y[1] = mask[i + 1] ? tr.z * t1 - tr.w * t0 : 0.f;
  y[2] = mask[i + 2] ? tr.y * c + tr.x * t2 : 0.f;
}
__global__ void k_pa_cart(int nnod, const float4 *__restrict__ trig, const uint8_t *__restrict__ mask,
                          const float *__restrict__ x, float4 *__restrict__ xc) {
  grid_dep();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nnod) return;
  const size_t i = 3 * (size_t)n;
  xc[n] = pa_to_cart(trig[n], mask[i] ? x[i] : 0.f, mask[i + 1] ? x[i + 1] : 0.f, mask[i + 2] ? x[i + 2] : 0.f);
}
__global__ void k_pa_gather(int nnod, const int *__restrict__ nptr, const float4 *__restrict__ yb,
                            const float4 *__restrict__ trig,
                            const uint8_t *__restrict__ mask, float *__restrict__ y) {
  grid_dep();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nnod) return;
  float v[3];
  pa_node_sum(nptr, yb, trig[n], mask, n, v);
#pragma unroll
  for (int c = 0; c < 3; ++c) y[3 * (size_t)n + c] = v[c];
}
// d += w (r - K d) / diag and the new d in Cartesian components (Di is 0 on fixed dofs)
__global__ void k_pa_gather_jac(int nnod, const int *__restrict__ nptr, const float4 *__restrict__ yb,
                                const float4 *__restrict__ trig,
                                const uint8_t *__restrict__ mask, float w, const float *__restrict__ r,
                                const float *__restrict__ Di, float *__restrict__ d, float4 *__restrict__ xc) {
  grid_dep();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nnod) return;
  const float4 tr = trig[n];
  float y[3], dn[3];
  pa_node_sum(nptr, yb, tr, mask, n, y);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const size_t i = 3 * (size_t)n + c;
    dn[c] = d[i] + w * (r[i] - y[c]) * Di[i];
    d[i] = dn[c];
    dn[c] = mask[i] ? dn[c] : 0.f;
  }
  xc[n] = pa_to_cart(tr, dn[0], dn[1], dn[2]);
}
// first sweep from zero, d = w r / diag, and d in Cartesian components
__global__ void k_pa_jac_first(int nnod, const float4 *__restrict__ trig, const uint8_t *__restrict__ mask, float w,
                               const float *__restrict__ r, const float *__restrict__ Di, float *__restrict__ d,
                               float4 *__restrict__ xc) {
  grid_dep();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nnod) return;
  float dn[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const size_t i = 3 * (size_t)n + c;
    dn[c] = w * r[i] * Di[i];
    d[i] = dn[c];
    dn[c] = mask[i] ? dn[c] : 0.f;
  }
  xc[n] = pa_to_cart(trig[n], dn[0], dn[1], dn[2]);
}

static void pa_tiles(const Level &L, cudaStream_t s) {
  launch_pdl(k_pa_tile, (L.nel + PA_E - 1) / PA_E, 32, 0, s, L.pa32, L.el2nod, L.nel, L.pa_xc, L.pa_tptr, L.pa_slot,
             L.pa_ent,
                                                       L.pa_yb, L.sa_err);
  count_launch();
}
constexpr int PA_NT = 128;                           // node passes: threads per block
static unsigned pa_ngrid(const Level &L) { return (unsigned)((L.nnod + PA_NT - 1) / PA_NT); }

int pa_jac_first_f32(const Level &L, float w, const float *r, const float *Di, float *d, cudaStream_t s) {
  launch_pdl(k_pa_jac_first, pa_ngrid(L), PA_NT, 0, s, L.nnod, L.pa_trig, L.freemask, w, r, Di, d, L.pa_xc);
  count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}

// y = K x; have_cart: xc already holds x (written by the pass that made x)
int pa_apply_f32(const Level &L, const float *x, float *y, bool have_cart, cudaStream_t s) {
  if (!have_cart) {
    launch_pdl(k_pa_cart, pa_ngrid(L), PA_NT, 0, s, L.nnod, L.pa_trig, L.freemask, x, L.pa_xc);
    count_launch();
  }
  pa_tiles(L, s);
  launch_pdl(k_pa_gather, pa_ngrid(L), PA_NT, 0, s, L.nnod, L.pa_nptr, L.pa_yb, L.pa_trig, L.freemask, y);
  count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}

// d += w (r - K d) / diag (one weighted Jacobi sweep); leaves the new d in xc
int pa_apply_jac_f32(const Level &L, float w, const float *r, const float *Di, float *d, bool have_cart, cudaStream_t s) {
  if (!have_cart) {
    launch_pdl(k_pa_cart, pa_ngrid(L), PA_NT, 0, s, L.nnod, L.pa_trig, L.freemask, d, L.pa_xc);
    count_launch();
  }
  pa_tiles(L, s);
  launch_pdl(k_pa_gather_jac, pa_ngrid(L), PA_NT, 0, s, L.nnod, L.pa_nptr, L.pa_yb, L.pa_trig, L.freemask, w, r, Di, d,
                                                L.pa_xc);
  count_launch();
  M3_CUDA(cudaGetLastError());
  return M3SPH_OK;
}

}  // namespace m3sph
