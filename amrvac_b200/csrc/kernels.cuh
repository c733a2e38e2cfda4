// Kernel launchers shared by the per-physics translation units.
#pragma once

#include <cuda_runtime.h>

#include "stage.cuh"

namespace amrvac {

// ---------------------------------------------------------------- setdt tail
// After the CFL reduction: dt = courantpar / max (src/mod_dt.t:233-235), the
// dtmin check (55-60), the slowsteps ramp (64-67), final_dt_reduction (69-79)
// and the output-interval cap (88-99).  scal: [0]=dt [1]=cmax_global
// [2]=global_time [3]=time_max [4]=dtsave [5]=dtmin [6]=courantpar
// [7]=final_exit flag [8]=slowsteps [9]=steps since set_time (it - it_init).
__device__ __forceinline__ void setdt_finalize(volatile unsigned long long *red, volatile double *scal,
                                               uint32_t *status) {
  const double smalldouble = 1.0e-12, bigdouble = 1.0e99;
  const double x = __longlong_as_double((long long)red[0]);
  const double cm = __longlong_as_double((long long)red[1]);
  red[0] = 0ull;
  red[1] = 0ull;
  double dt = bigdouble;
  if (x > smalldouble) dt = fmin(dt, scal[6] / x);
  if (dt < scal[5]) atomicOr(status, ST_DT_TOO_SMALL);
  if (scal[8] > scal[9] + 1.0) {
    const double q = 1.0 - (scal[9] + 1.0) / scal[8];
    dt = dt * (1.0 - q * q);
  }
  const double t = scal[2], tmax = scal[3], dtsave = scal[4];
  if (tmax - t <= scal[5]) scal[7] = 1.0;
  dt = fmin(dt, tmax - t);
  if (dtsave > 0.0) {
    double dtmax = ceil(t / dtsave) * dtsave;
    const double other = t > 0.0 ? ceil(t / bigdouble) * bigdouble : 0.0;
    dtmax = fmin(dtmax, other) - t;
    if (dtmax > smalldouble) dt = fmin(dt, dtmax);
    else dt = fmin(dt, dtsave);
  }
  scal[0] = dt;
  scal[1] = cm;
}

// ---------------------------------------------------------------- getdt
// getdt_courant (src/mod_dt.t:160-287) per block, reduced over all blocks.
// red[0] <- max over blocks of the block's courant sum (maxsum: max_cells
// sum_d cmax_d/dx_d; summax / minimum per the reference), red[1] <- max cmax.
struct GetdtArgs {
  const double *u;
  const double *dxb;
  int nblocks;
  int bn;  // block edge
  int type_courant;
  unsigned long long *red;
  PhysParams P;
  uint32_t *status;  // the context's status word: the small-value check of getdt
  const uint32_t *skip;  // 'average': blocks flagged ST_SV_AVG are reduced by sv_getdt_kernel
  // setdt in the same launch: the last CTA to finish (counted in *ticket)
  // turns the maxima into dt (scal non-null), and with advance also moves
  // global_time and the step count on (nothing between here and the end of
  // an unsplit step reads them)
  double *scal;
  unsigned *ticket;
  int advance;
  // amrvac_gpu_getdt: the last CTA writes the two maxima to the host's memory
  // (mapped), sets scal's cmax_global and clears the words for the next call
  double *host;
  bool dependent;  // launch: the predecessor on the stream allows a dependent launch
  int nsm;         // launch: SMs of the device
};

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Non-negative doubles order like their bit patterns.
__device__ __forceinline__ void atomic_max_pos(unsigned long long *a, double v) {
  if (v > 0.0) atomicMax(a, (unsigned long long)__double_as_longlong(v));
}

// Work items: up to GETDT_CHUNK cells of one block, x fastest (coalesced), 256
// threads at a time.  With 'maxsum' only two maxima leave a block, so the
// CTAs (one wave of four per SM, 64 registers) stride over the items of all
// blocks and reduce once at the end; 'summax' and 'minimum' combine the
// directions' maxima of a block, so there an item is a whole block and each is
// reduced on its own.  The kernel is bound by its loads' latency: one CTA per
// block at two per SM measured 53 us at 128^3 MHD (151 MB).
constexpr int GETDT_CHUNK = 1024;
template <bool MHD, int NDIR, bool GLM, int NDIM>
__global__ void __launch_bounds__(256, 4) getdt_kernel(const GetdtArgs A) {
  using V = Vars<MHD, NDIR, GLM>;
  constexpr int NW = V::NW;
  const int bn = A.bn;
  const int ncell = bn * (NDIM >= 2 ? bn : 1) * (NDIM == 3 ? bn : 1);
  const int t = threadIdx.x;
  const bool maxsum = A.type_courant == 1;
  const int chunk = maxsum ? GETDT_CHUNK : ncell;
  const int parts = (ncell + chunk - 1) / chunk, nitem = A.nblocks * parts;
  __shared__ double red[5][8];
  const int lane = t & 31, wid = t >> 5;
  pdl_wait();
  pdl_trigger();
  double mtot = 0.0, mcm = 0.0, mdim[3] = {0.0, 0.0, 0.0};
  // the maxima of all threads into red[0]; adds them to the global words
  auto reduce = [&]() {
    const double v[5] = {mtot, mcm, mdim[0], mdim[1], mdim[2]};
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const double w = warp_max(v[q]);
      if (lane == 0) red[q][wid] = w;
    }
    __syncthreads();
    if (t == 0) {
      double m[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
      for (int q = 0; q < 5; ++q)
        for (int w = 0; w < 8; ++w) m[q] = fmax(m[q], red[q][w]);
      double x = m[0];
      if (!maxsum) {
        double courantmax = 0.0, tot = 0.0;
        for (int d = 0; d < NDIM; ++d) {
          courantmax = fmax(courantmax, m[2 + d]);
          tot = tot + courantmax;
        }
        x = A.type_courant == 2 ? tot : courantmax;
      }
      atomic_max_pos(A.red + 0, x);
      atomic_max_pos(A.red + 1, m[1]);
    }
    __syncthreads();
  };
  for (int it = blockIdx.x; it < nitem; it += gridDim.x) {
    const int b = it / parts, c0 = (it - b * parts) * chunk, c1 = min(c0 + chunk, ncell);
    if (A.skip && (A.skip[b] & ST_SV_AVG)) continue;
    double dxinv[3];
#pragma unroll
    for (int d = 0; d < NDIM; ++d) dxinv[d] = 1.0 / A.dxb[b * 3 + d];
    // c is the cell's index within its block-variable row (cell_offset's layout)
    const double *ub = A.u + (size_t)b * NW * ncell;
#pragma unroll 1
    for (int c = c0 + t; c < c1; c += 256) {
      double w[NW];
#pragma unroll
      for (int v = 0; v < NW; ++v) w[v] = ub[(size_t)v * ncell + c];
      // getdt_courant takes the primitives through phys_to_primitive, small-value
      // fix included (src/mod_dt.t:189-191)
      if (A.P.fix_small_values) {
        if (small_values<double, MHD, NDIR, GLM>(w, false, A.P) && A.P.small_values_method != 1 && A.status)
          atomicOr(A.status, ST_SMALL_VALUE);
      }
      to_primitive<MHD, NDIR, GLM>(w, A.P);
      double tot = 0.0;
#pragma unroll
      for (int d = 0; d < NDIM; ++d) {
        double cm;
        if constexpr (MHD) {
          double cf;
          if (d == 0) cf = fast_speed<double, NDIR, V::B0 + 0>(w, A.P);
          else if (d == 1) cf = fast_speed<double, NDIR, V::B0 + (NDIR > 1 ? 1 : 0)>(w, A.P);
          else cf = fast_speed<double, NDIR, V::B0 + (NDIR > 2 ? 2 : 0)>(w, A.P);
          cm = fabs(w[V::M0 + d]) + cf;
        } else {
          cm = fabs(w[V::M0 + d]) + sqrt(A.P.gamma * w[V::E] / w[V::RHO]);
        }
        const double cd = cm * dxinv[d];
        tot = d == 0 ? cd : tot + cd;
        mdim[d] = fmax(mdim[d], cd);
        mcm = fmax(mcm, cm);
      }
      mtot = fmax(mtot, tot);
    }
    if (!maxsum) {
      reduce();
      mtot = mcm = mdim[0] = mdim[1] = mdim[2] = 0.0;
    }
  }
  if (maxsum) reduce();
  if (t == 0 && A.scal) {
    __threadfence();
    if (atomicAdd(A.ticket, 1u) == gridDim.x - 1) {
      __threadfence();
      *A.ticket = 0u;
      if (A.host) {
        volatile unsigned long long *red = A.red;
        const double x = __longlong_as_double((long long)red[0]), cm = __longlong_as_double((long long)red[1]);
        red[0] = 0ull;
        red[1] = 0ull;
        A.scal[1] = cm;
        A.host[0] = x;
        A.host[1] = cm;
        __threadfence_system();
      } else {
        setdt_finalize(A.red, A.scal, A.status);
        if (A.advance) {
          A.scal[2] = A.scal[2] + A.scal[0];
          A.scal[9] = A.scal[9] + 1.0;
        }
      }
    }
  }
}

// ---------------------------------------------------------------- points
struct PointArgs {
  int n;
  const double *a, *b, *c, *d;  // inputs (state-major [n][nw])
  double *out, *out2;
  double cg;
  PhysParams P;
};

template <bool MHD, int NDIR, bool GLM, int NDIM, int SOLVER, int D>
__global__ void riemann_points_kernel(const PointArgs A) {
  using V = Vars<MHD, NDIR, GLM>;
  constexpr int NW = V::NW;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= A.n) return;
  double wL[NW], wR[NW], F[NW];
#pragma unroll
  for (int v = 0; v < NW; ++v) {
    const int ov = orig_index<MHD, NDIR, D>(v);
    wL[v] = A.a[(size_t)p * NW + ov];
    wR[v] = A.b[(size_t)p * NW + ov];
  }
  face_from_states<double, MHD, NDIR, GLM, NDIM, SOLVER, 0>(wL, wR, A.P, A.cg, F);
#pragma unroll
  for (int v = 0; v < NW; ++v) A.out[(size_t)p * NW + orig_index<MHD, NDIR, D>(v)] = F[v];
}

template <bool MHD, int NDIR, bool GLM, int D>
__global__ void flux_points_kernel(const PointArgs A) {
  using V = Vars<MHD, NDIR, GLM>;
  constexpr int NW = V::NW;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= A.n) return;
  double wc[NW], w[NW], f[NW];
#pragma unroll
  for (int v = 0; v < NW; ++v) { wc[v] = A.a[(size_t)p * NW + v]; w[v] = A.b[(size_t)p * NW + v]; }
  phys_flux<double, MHD, NDIR, GLM, D>(wc, w, A.cg, f);
#pragma unroll
  for (int v = 0; v < NW; ++v) A.out[(size_t)p * NW + v] = f[v];
}

template <bool MHD, int NDIR, bool GLM, int D>
__global__ void cbounds_points_kernel(const PointArgs A) {
  using V = Vars<MHD, NDIR, GLM>;
  constexpr int NW = V::NW;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= A.n) return;
  double lc[NW], rc[NW], lp[NW], rp[NW];
#pragma unroll
  for (int v = 0; v < NW; ++v) {
    lc[v] = A.a[(size_t)p * NW + v]; rc[v] = A.b[(size_t)p * NW + v];
    lp[v] = A.c[(size_t)p * NW + v]; rp[v] = A.d[(size_t)p * NW + v];
  }
  double cmax, cmin = 0.0;
  if (A.out2) cbounds<double, MHD, NDIR, GLM, D, true>(lc, rc, lp, rp, A.P, cmax, cmin);
  else cbounds<double, MHD, NDIR, GLM, D, false>(lc, rc, lp, rp, A.P, cmax, cmin);
  A.out[p] = cmax;
  if (A.out2) A.out2[p] = cmin;
}

// ---------------------------------------------------------------- a2max
// phys_get_a2max (hd_get_a2max src/hd/mod_hd_phys.t:813-833; MHD the same,
// src/mhd/mod_mhd_phys.t:2678-2698) reduced as getdt_courant and setdt do
// for schmid1 (src/mod_dt.t:193-197, 130): per block and direction d the
// maximum over its cells and conserved variables of
// |-w(i+2) + 16 w(i+1) - 30 w(i) + 16 w(i-1) - w(i-2)|, / 12 / dx_d^2, then
// the maximum over blocks into out[d].  One CTA per z-plane of a block.
template <int NW, int NDIM, int BN = BN16>
__global__ void __launch_bounds__(256) a2max_kernel(const StageArgs A, double *out) {
  constexpr int PL = NDIM == 3 ? BN : 1;
  const int b = blockIdx.x / PL, k = blockIdx.x - (blockIdx.x / PL) * PL;
  auto w = [&](int ii, int jj, int kk, int v) {
    uint32_t flip;
    const int blk = resolve_cell<NDIM>(A, b, ii, jj, kk, flip, BN);
    const double x = blk >= 0 ? __ldg(A.uin + cell_offset<NDIM>(blk, NW, v, ii, jj, kk, BN))
                              : __ldg(A.gbuf + ghost_offset<NDIM>(-2 - blk, NW, v, ii, jj, kk, BN));
    return ((flip >> v) & 1u) ? -x : x;
  };
  __shared__ double red[8];
#pragma unroll 1
  for (int d = 0; d < NDIM; ++d) {
    const int e0 = d == 0, e1 = d == 1, e2 = d == 2;
    double m = 0.0;
    for (int c = threadIdx.x; c < BN * BN; c += 256) {  // the cells of the plane
      const int i = c % BN, j = c / BN;
#pragma unroll
      for (int v = 0; v < NW; ++v) {
        const double a = fabs(((((-w(i + 2 * e0, j + 2 * e1, k + 2 * e2, v) + 16.0 * w(i + e0, j + e1, k + e2, v)) -
                                 30.0 * w(i, j, k, v)) +
                                16.0 * w(i - e0, j - e1, k - e2, v)) -
                               w(i - 2 * e0, j - 2 * e1, k - 2 * e2, v)));
        m = fmax(m, a);
      }
    }
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      double mm = red[0];
      for (int q = 1; q < 8; ++q) mm = fmax(mm, red[q]);
      const double dx = A.dxb[b * 3 + d];
      atomic_max_pos(reinterpret_cast<unsigned long long *>(out + d), mm / 12.0 / (dx * dx));
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- Linde, 3-D
// add_source_linde (src/mhd/mod_mhd_phys.t:5599-5665) for 3-D blocks, run
// after the stage kernel on its output: w(B_d) += g_d, w(e) += wCT(B_d) g_d
// with g_d = divbdiff / sum_d(1/dx_d^2) * d(divB)/dx_d (central), divB of wCT
// (central, get_divb with mhd_divb_nth = 1), leaving out the cell layers next
// to level-jump faces; then the small-value check of mhd_add_source.  Its
// stencil (divB at the six neighbours: B two cells out and across the z
// planes' halos) is gathered here through the stage's neighbour resolution
// (and the level-jump ghost buffers); one CTA per z-plane of a block.
template <int NDIR, int BN = BN16>
__global__ void __launch_bounds__(256) linde3d_kernel(const StageArgs A) {
  using V = Vars<true, NDIR, false>;
  constexpr int NW = V::NW;
  const int b = blockIdx.x / BN, k = blockIdx.x - (blockIdx.x / BN) * BN;
  if (b >= A.nblocks) return;
  const int m = A.amr_face ? A.amr_face[b] : 0;
  for (int c = threadIdx.x; c < BN * BN; c += 256) {  // the cells of the plane
  const int i = c % BN, j = c / BN;
  if (m && (((m & 1) && i == 0) || ((m & 2) && i == BN - 1) || ((m & 4) && j == 0) || ((m & 8) && j == BN - 1) ||
            ((m & 16) && k == 0) || ((m & 32) && k == BN - 1)))
    continue;
  double dx[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) dx[d] = A.dxb[b * 3 + d];
  auto bct = [&](int ii, int jj, int kk, int c) -> double {  // wCT's B_c, up to two cells outside
    uint32_t flip;
    const int blk = resolve_cell<3>(A, b, ii, jj, kk, flip, BN);
    const int v = V::B0 + c;
    const double x = blk >= 0 ? __ldg(A.uin + cell_offset<3>(blk, NW, v, ii, jj, kk, BN))
                              : __ldg(A.gbuf + ghost_offset<3>(-2 - blk, NW, v, ii, jj, kk, BN));
    return ((flip >> v) & 1u) ? -x : x;
  };
  auto divb = [&](int ii, int jj, int kk) {
    double d = 0.5 * (bct(ii + 1, jj, kk, 0) - bct(ii - 1, jj, kk, 0)) * (1.0 / dx[0]);
    d = d + 0.5 * (bct(ii, jj + 1, kk, 1) - bct(ii, jj - 1, kk, 1)) * (1.0 / dx[1]);
    d = d + 0.5 * (bct(ii, jj, kk + 1, 2) - bct(ii, jj, kk - 1, 2)) * (1.0 / dx[2]);
    return d;
  };
  const double inv2 = (1.0 / (dx[0] * dx[0]) + 1.0 / (dx[1] * dx[1])) + 1.0 / (dx[2] * dx[2]);
  double w[NW];
#pragma unroll
  for (int v = 0; v < NW; ++v) w[v] = A.uout[cell_offset<3>(b, NW, v, i, j, k, BN)];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double dp = d == 0 ? divb(i + 1, j, k) : (d == 1 ? divb(i, j + 1, k) : divb(i, j, k + 1));
    const double dm = d == 0 ? divb(i - 1, j, k) : (d == 1 ? divb(i, j - 1, k) : divb(i, j, k - 1));
    double g = (dp - dm) * 0.5;
    g = g / dx[d];
    g = g * A.P.divbdiff / inv2;
    w[V::B0 + d] = w[V::B0 + d] + g;
    w[V::E] = w[V::E] + __ldg(A.uin + cell_offset<3>(b, NW, V::B0 + d, i, j, k, BN)) * g;
  }
  if (A.P.fix_small_values) {
    if (small_values<double, true, NDIR, false>(w, false, A.P) && A.P.small_values_method != 1)
      atomicOr(A.status, ST_SMALL_VALUE);
  }
#pragma unroll
  for (int v = 0; v < NW; ++v) A.uout[cell_offset<3>(b, NW, v, i, j, k, BN)] = w[v];
  }  // cells of the plane
}

// ---------------------------------------------------------------- dispatch
struct KernelSet {
  cudaError_t (*prepare)() = nullptr;
  int (*hancock_ctas_per_sm)() = nullptr;
  cudaError_t (*stage)(const StageArgs &, int nctas, cudaStream_t) = nullptr;
  // MUSCL-Hancock predictor of twostep Predictor_Corrector (tvdlf sets only)
  cudaError_t (*hancock)(const StageArgs &, int nctas, cudaStream_t) = nullptr;
  // the 3-D Linde divB source after a stage (3-D MHD sets without GLM)
  cudaError_t (*linde3d)(const StageArgs &, cudaStream_t) = nullptr;
  // a2max_global of schmid1 (every set)
  cudaError_t (*a2max)(const StageArgs &, double *out, cudaStream_t) = nullptr;
  cudaError_t (*getdt)(const GetdtArgs &, cudaStream_t) = nullptr;
  cudaError_t (*riemann_points)(const PointArgs &, int idim, cudaStream_t) = nullptr;
  cudaError_t (*flux_points)(const PointArgs &, int idim, cudaStream_t) = nullptr;
  cudaError_t (*cbounds_points)(const PointArgs &, int idim, cudaStream_t) = nullptr;
  size_t stage_smem = 0;
  int bn = BN16;  // the block edge the stage kernels were built for
  // Stage-kernel variants the autotuner times (variant 0 is `stage`): per
  // variant the launch, its occupancy query, threads per CTA, the CTAs per
  // SM its registers are capped for, and asynchronous plane staging.
  static constexpr int MAXVAR = 4;
  int nvar = 1;
  cudaError_t (*stage_v[MAXVAR])(const StageArgs &, int nctas, cudaStream_t) = {};
  int (*ctas_v[MAXVAR])() = {};
  cudaError_t (*prepare_v[MAXVAR])() = {};
  int var_threads[MAXVAR] = {}, var_minb[MAXVAR] = {}, var_async[MAXVAR] = {};
  // threads per CTA and CTAs per SM of variant 0 on a grid (Launch::build)
  void (*shape)(int nblocks, int nsm, int *threads, int *minb) = nullptr;
};

// One stage-kernel variant of a scheme (see stage_variant).
template <bool MHD, int NDIR, bool GLM, int NDIM, int SOLVER, int LIM, int BS, class TF, int BN, int VAR>
struct StageVar {
  using V = Vars<MHD, NDIR, GLM>;
  using O = StageOcc<TF, MHD, NDIM, LIM, BN, VAR>;
  static constexpr size_t SMEM = Tile<TF, V::NW, NDIM, HaloW<LIM>::value, tile_edge(BN)>::BYTES;
  static cudaError_t prepare() {
    return cudaFuncSetAttribute(fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOLVER, LIM, BS, BN, VAR>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
  }
  static cudaError_t stage(const StageArgs &A, int nctas, cudaStream_t s) {
    return launch_dependent<StageArgs>(&fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOLVER, LIM, BS, BN, VAR>, nctas,
                                       O::THREADS, SMEM, s, A.dependent, A);
  }
  static int ctas_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &n, fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOLVER, LIM, BS, BN, VAR>, O::THREADS, SMEM) != cudaSuccess)
      return 1;
    return n > 0 ? n : 1;
  }
  static void add(KernelSet &k, int slot) {
    k.stage_v[slot] = &stage;
    k.ctas_v[slot] = &ctas_per_sm;
    k.prepare_v[slot] = &prepare;
    k.var_threads[slot] = O::THREADS;
    k.var_minb[slot] = O::MINB;
    k.var_async[slot] = O::ASYNC && sizeof(TF) == 8 && NDIM == 3 && tile_edge(BN) == BN && HaloW<LIM>::value == 2;
    if (slot + 1 > k.nvar) k.nvar = slot + 1;
  }
};

template <bool MHD, int NDIR, bool GLM, int NDIM, int SOLVER, int LIM = 0, int BS = 0, class TF = double,
          int BN = BN16>
struct Launch {
  using V = Vars<MHD, NDIR, GLM>;
  static constexpr int THREADS = StageOcc<TF, MHD, NDIM, LIM, BN>::THREADS;
  static constexpr size_t SMEM = Tile<TF, V::NW, NDIM, HaloW<LIM>::value, tile_edge(BN)>::BYTES;
  // The 2-D hydrodynamics tile is small (30 KB) and its kernel waits for its
  // block's loads and barriers: four CTAs per SM (64 registers) instead of two
  // hide them, 2048^2 HLLC + vanleer FP64 0.37 -> 0.31 ms per stage.  So they do
  // for the other solvers and limiters (1024^2, us a step: HLL + cada3 292 -> 252,
  // Roe 293 -> 265, TVDLF 223 -> 193, HLL + WENO3 560 -> 424, HLL + Venkatakrishnan
  // 639 -> 521).  A grid that the two-CTA kernel holds in one wave has no second
  // CTA to hide behind, and runs the kernel that spills least (64^2: 28 -> 26 us a
  // step; 272^2 in blocks of 8, 1156 tiles at eight CTAs per SM: 53 -> 35).
  static constexpr bool HAS_DENSE = !MHD && NDIM == 2 && sizeof(TF) == 8 && HaloW<LIM>::value == 2;
  static constexpr int VMAIN = HAS_DENSE ? VAR_DENSE : 0;
  static constexpr int NTILE = (BN / tile_edge(BN)) * (BN / tile_edge(BN));
  // Up to one tile per SM there is no other work to hide a tile's latency, and
  // a block edge of 16 takes a thread per face (576 threads: one round of
  // faces instead of three; 64^2 HLLC 24.9 -> 21.7 us a step).  At two tiles per
  // SM half of them (288) measured no gain over 256 (256^2 31.8 -> 32.2).
  static constexpr bool HAS_WIDE = HAS_DENSE && BN == 16;
  // the build that runs nblocks blocks on nsm SMs
  static int build(int nblocks, int nsm) {
    if (HAS_WIDE && nblocks <= nsm) return VAR_WIDE;
    return HAS_DENSE && nblocks * NTILE > StageOcc<TF, MHD, NDIM, LIM, BN>::MINB * nsm ? VAR_DENSE : 0;
  }
  static void shape(int nblocks, int nsm, int *threads, int *minb) {
    const int var = build(nblocks, nsm);
    *threads = var == VAR_WIDE ? StageOcc<TF, MHD, NDIM, LIM, BN, VAR_WIDE>::THREADS : THREADS;
    *minb = var == VAR_WIDE    ? StageOcc<TF, MHD, NDIM, LIM, BN, VAR_WIDE>::MINB
            : var == VAR_DENSE ? StageOcc<TF, MHD, NDIM, LIM, BN, VAR_DENSE>::MINB
                               : StageOcc<TF, MHD, NDIM, LIM, BN>::MINB;
  }
  // typepred1 = fs_hancock for tvdlf and tvdmu (src/io/mod_input_output.t:787-797),
  // in a wave of its own: it is less dense than the stage's and, at small block
  // edges, has more CTAs per SM than two (512^2 in blocks of 8, tvdlf: 72 us a
  // step; with 296 CTAs, two per SM, 131)
  static constexpr bool HAS_HANCOCK = (SOLVER == SOLVER_TVDLF || SOLVER == SOLVER_TVDMU) && sizeof(TF) == 8;
  static cudaError_t prepare() {
    cudaError_t e = cudaFuncSetAttribute(fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOLVER, LIM, BS, BN>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    if constexpr (HAS_DENSE) {
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOLVER, LIM, BS, BN, VAR_DENSE>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    }
    if constexpr (HAS_WIDE) {
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOLVER, LIM, BS, BN, VAR_WIDE>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    }
    if constexpr (HAS_HANCOCK) {
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOLVER_HANCOCK, LIM, BS, BN>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    }
    return e;
  }
  static cudaError_t stage(const StageArgs &A, int nctas, cudaStream_t s) {
    [[maybe_unused]] const int var = build(A.nblocks, A.nsm);
    if constexpr (HAS_WIDE) {
      if (var == VAR_WIDE)
        return launch_dependent<StageArgs>(
            &fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOLVER, LIM, BS, BN, VAR_WIDE>, nctas,
            StageOcc<TF, MHD, NDIM, LIM, BN, VAR_WIDE>::THREADS, SMEM, s, A.dependent, A);
    }
    if constexpr (HAS_DENSE) {
      if (var == VAR_DENSE)
        return launch_dependent<StageArgs>(&fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOLVER, LIM, BS, BN, VAR_DENSE>,
                                           nctas, THREADS, SMEM, s, A.dependent, A);
    }
    return launch_dependent<StageArgs>(&fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOLVER, LIM, BS, BN>, nctas, THREADS,
                                       SMEM, s, A.dependent, A);
  }
  static cudaError_t a2max(const StageArgs &A, double *out, cudaStream_t s) {
    a2max_kernel<V::NW, NDIM, BN><<<A.nblocks * (NDIM == 3 ? BN : 1), 256, 0, s>>>(A, out);
    return cudaGetLastError();
  }
  static cudaError_t linde3d(const StageArgs &A, cudaStream_t s) {
    if constexpr (MHD && NDIM == 3 && !GLM) {
      linde3d_kernel<NDIR, BN><<<A.nblocks * BN, 256, 0, s>>>(A);
      return cudaGetLastError();
    } else {
      return cudaErrorNotSupported;
    }
  }
  static cudaError_t hancock(const StageArgs &A, int nctas, cudaStream_t s) {
    if constexpr (HAS_HANCOCK) {
      return launch_dependent<StageArgs>(&fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOLVER_HANCOCK, LIM, BS, BN>, nctas,
                                         THREADS, SMEM, s, A.dependent, A);
    } else {
      return cudaErrorNotSupported;
    }
  }
  template <int SOL, int VAR>
  static int resident() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &n, fv_stage_kernel<TF, MHD, NDIR, GLM, NDIM, SOL, LIM, BS, BN, VAR>, THREADS, SMEM) != cudaSuccess)
      return 1;
    return n > 0 ? n : 1;
  }
  static int ctas_per_sm() { return resident<SOLVER, VMAIN>(); }
  static int hancock_ctas_per_sm() {
    if constexpr (HAS_HANCOCK) return resident<SOLVER_HANCOCK, 0>();
    else return 1;
  }
  static cudaError_t getdt(const GetdtArgs &A, cudaStream_t s) {
    int ncell = 1;
    for (int d = 0; d < NDIM; ++d) ncell *= A.bn;
    const long items = (long)A.nblocks * (A.type_courant == 1 ? (ncell + GETDT_CHUNK - 1) / GETDT_CHUNK : 1);
    const int nctas = (int)(items < 4 * A.nsm ? items : 4 * A.nsm);
    return launch_dependent<GetdtArgs>(&getdt_kernel<MHD, NDIR, GLM, NDIM>, nctas, 256, 0, s, A.dependent, A);
  }
  template <int D>
  static void rp(const PointArgs &A, cudaStream_t s) {
    riemann_points_kernel<MHD, NDIR, GLM, NDIM, SOLVER, D><<<(A.n + 127) / 128, 128, 0, s>>>(A);
  }
  static cudaError_t riemann_points(const PointArgs &A, int idim, cudaStream_t s) {
    if (idim == 1) rp<0>(A, s);
    else if (idim == 2 && NDIM >= 2) rp<NDIM >= 2 ? 1 : 0>(A, s);
    else if (idim == 3 && NDIM >= 3) rp<NDIM >= 3 ? 2 : 0>(A, s);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
  }
  template <int D>
  static void fp(const PointArgs &A, cudaStream_t s) {
    flux_points_kernel<MHD, NDIR, GLM, D><<<(A.n + 127) / 128, 128, 0, s>>>(A);
  }
  static cudaError_t flux_points(const PointArgs &A, int idim, cudaStream_t s) {
    if (idim == 1) fp<0>(A, s);
    else if (idim == 2 && NDIR >= 2) fp<NDIR >= 2 ? 1 : 0>(A, s);
    else if (idim == 3 && NDIR >= 3) fp<NDIR >= 3 ? 2 : 0>(A, s);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
  }
  template <int D>
  static void cp(const PointArgs &A, cudaStream_t s) {
    cbounds_points_kernel<MHD, NDIR, GLM, D><<<(A.n + 127) / 128, 128, 0, s>>>(A);
  }
  static cudaError_t cbounds_points(const PointArgs &A, int idim, cudaStream_t s) {
    if (idim == 1) cp<0>(A, s);
    else if (idim == 2 && NDIR >= 2) cp<NDIR >= 2 ? 1 : 0>(A, s);
    else if (idim == 3 && NDIR >= 3) cp<NDIR >= 3 ? 2 : 0>(A, s);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
  }
  static KernelSet set() {
    KernelSet k;
    k.prepare = &prepare;
    k.hancock_ctas_per_sm = &hancock_ctas_per_sm;
    k.stage = &stage;
    if (HAS_HANCOCK) k.hancock = &hancock;
    if (MHD && NDIM == 3 && !GLM) k.linde3d = &linde3d;
    k.a2max = &a2max;
    k.getdt = &getdt;
    k.riemann_points = &riemann_points;
    k.flux_points = &flux_points;
    k.cbounds_points = &cbounds_points;
    k.stage_smem = SMEM;
    k.bn = BN;
    StageVar<MHD, NDIR, GLM, NDIM, SOLVER, LIM, BS, TF, BN, 0>::add(k, 0);
    k.stage_v[0] = &stage;
    k.ctas_v[0] = &ctas_per_sm;
    k.shape = &shape;
    return k;
  }
};

// Lookup key for one physics / dimension / solver combination.
struct KernelKey {
  bool mhd;
  int ndim, ndir;
  bool glm;
  int solver;
  int limiter;     // used to pick a compile-time specialised stage kernel
  int boundspeed;
  bool mixed;      // FP32 face arithmetic (mixed form)
  int bn;          // block edge (block_nx)
};

bool lookup_hd(const KernelKey &k, KernelSet *out);
// small_values_method 'average' (smallavg.cu): detection, whole-block stage
// and getdt of the flagged blocks; scratch per CTA (SvScratch).
struct SvScratch;
struct SvSet {
  cudaError_t (*detect)(const StageArgs &, const double *reg, cudaStream_t) = nullptr;
  cudaError_t (*stage)(const StageArgs &, const double *snap_base, const double *snap_in, SvScratch, int nctas,
                       cudaStream_t) = nullptr;
  cudaError_t (*getdt)(const StageArgs &, const double *reg, int type_courant, unsigned long long *red, SvScratch,
                       int nctas, cudaStream_t) = nullptr;
};
struct SvScratch {
  double *base;
  size_t per_cta;  // doubles per CTA
};
bool lookup_sv(const KernelKey &k, SvSet *out);
// The variants 1..3 of the benchmark schemes' stage kernels (k_tune.cu).
bool add_stage_variants(const KernelKey &k, KernelSet *out);
// block edges other than 16 (k_blocks.cuh, one unit per edge)
bool lookup_bn8(const KernelKey &k, KernelSet *out);
bool lookup_bn10(const KernelKey &k, KernelSet *out);
bool lookup_bn12(const KernelKey &k, KernelSet *out);
bool lookup_bn32(const KernelKey &k, KernelSet *out);
bool lookup_mp5_hd(const KernelKey &k, KernelSet *out);
bool lookup_mp5_mhd(const KernelKey &k, KernelSet *out);
bool lookup_mhd2(const KernelKey &k, KernelSet *out);
bool lookup_mhd3(const KernelKey &k, KernelSet *out);

}  // namespace amrvac
