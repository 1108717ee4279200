// Quad2D (2D tensor-product element) forms of the BP5/BP6 path: the element
// operator, the forcing, the lumped mass and the Jacobi diagonal.
//
//   Aq_e = Dr^T (G00 ur + G01 us) + Ds^T (G01 ur + G11 us) + lambda wJ q,
//   (ur, us) = (Dr, Ds) q
// (okl/bp5AxQuad2D.okl, okl/bp5AxAffineQuad2D.okl, okl/bp6AxQuad2D.okl with
// Nfields = dim = 2).  Stored factors carry the GLL weights; affine factors are
// per element and the weights w_i w_j are applied here.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "bp_cg_device.cuh"
#include "bp_internal.hpp"

namespace bp {

// The line form from the warps per SM on at which it overtakes the node form:
// tenths of a warp by degree, measured at 1 to 40 warps per SM over all degrees,
// precisions, factor storages and field counts (1200 meshes; the form chosen
// takes 1.003 of the better one's time on average, 1.16 at the most, where one
// figure for all degrees, 8 warps stored and 3 affine, took 1.02 and 3.4).  The
// line form comes late at low degrees in FP32 (stored p=2 at 8 warps 3.3 us against
// 2.9) and early at high ones, where the node form's block holds one element
// (FP64 p=14 at 8 warps 10 us against 35).  Affine, its loads are fewer and it
// comes sooner; with two fields, whose factors the node form reads once, later.
bool quad_line_form(int N, int affine, int Nfields, int bytes, int32_t Nelements) {
  static const short stored64[15] = {80, 100, 80, 80, 80, 40, 60, 50, 60, 50, 60, 35, 40, 15, 35};
  static const short stored32[15] = {80, 140, 100, 100, 90, 70, 70, 80, 60, 80, 70, 60, 50, 40, 40};
  static const short aff[15] = {40, 60, 40, 30, 40, 20, 30, 30, 30, 30, 35, 30, 25, 15, 25};
  const int hundredths = (affine ? aff : bytes == 8 ? stored64 : stored32)[N - 1] * (Nfields == 1 ? 10 : affine ? 12 : 13);
  return (int64_t)100 * Nelements * Nfields >= (int64_t)hundredths * sm_count() * (32 / (N + 1));
}

namespace {

// One warp serves SPW element(-field)s of NQ lines each; a thread owns column x
// of its element in registers (q, then the result) and row y of the r-steps.
// Shared memory carries what crosses between rows and columns (ten accesses of
// a value per node); D and its transpose are read as warp-uniform pairs
// (broadcasts), and a row of D serves both the s-derivative and the s-part of
// the divergence.  Warps are independent: no block barrier after D is there.
//
// Before, one thread per node read a row and a column of q, of the r- and
// s-fluxes and of D for every node (66 shared-memory accesses; 93% of the L1
// pipe, 0.45 of HBM); affine factors took a column form with block barriers.
// BK5 p=7 700x500 curved: 373 -> 252 us.
template <int NQ>
struct QuadShape {
  static constexpr int SPW = 32 / NQ;                     // element(-field)s per warp
  static constexpr int WARPS = 4, THREADS = 32 * WARPS;
  static constexpr int EPB = SPW * WARPS;
  static constexpr int RS = NQ % 2 ? NQ : NQ + 1;         // odd row stride: rows fall in distinct banks
  static constexpr int NP = NQ * NQ;
  static constexpr int DS = NQ + NQ % 2;                  // rows of D padded to whole pairs
};

// sum of the NQ products d[n] r[n], d read in pairs
template <int NQ, class F>
__device__ __forceinline__ F quad_dot(const F* d, const F (&r)[NQ]) {
  using V2 = typename std::conditional<sizeof(F) == 8, double2, float2>::type;
  F a = 0;
#pragma unroll
  for (int n = 0; n + 1 < NQ; n += 2) {
    const V2 v = *reinterpret_cast<const V2*>(d + n);
    a += v.x * r[n];
    a += v.y * r[n + 1];
  }
  if (NQ % 2) a += d[NQ - 1] * r[NQ - 1];
  return a;
}

template <int NQ, bool AFFINE, bool DOT, class F>
__global__ void __launch_bounds__(QuadShape<NQ>::THREADS)
ax_quad_kernel(int Nelements, int Nfields, const int32_t* __restrict__ elementList, const int32_t* __restrict__ G2L,
               const F* __restrict__ wJ, const F* __restrict__ ggeo, const F* __restrict__ gllw,
               const F* __restrict__ Dg, F lambda, const F* __restrict__ q, F* __restrict__ Aq,
               const int* __restrict__ skip, CgFuse fuse) {
  if (skip && *skip) return;
  using Sh = QuadShape<NQ>;
  constexpr int RS = Sh::RS, NP = Sh::NP, DS = Sh::DS, SPW = Sh::SPW;
  __shared__ __align__(16) F s_D[NQ * DS];    // row o of D
  __shared__ __align__(16) F s_Dt[NQ * DS];   // row o of D^T
  __shared__ F s_U[Sh::EPB][NQ * RS];
  __shared__ F s_R[Sh::EPB][NQ * RS];
  __shared__ double s_red[Sh::WARPS];
  for (int n = threadIdx.x; n < NP; n += Sh::THREADS) {
    const F d = Dg[n];
    s_D[n / NQ * DS + n % NQ] = d;
    s_Dt[n % NQ * DS + n / NQ] = d;
  }
  const int lane = threadIdx.x & 31, sl = lane / NQ;
  const bool on = sl < SPW;                               // the last lanes own no line
  const int slot = (threadIdx.x >> 5) * SPW + (on ? sl : 0), x = on ? lane - sl * NQ : 0;
  // element-major (element, field): one or two fields of fewer than 2^31 elements
  // are counted in 32 bits (in 64 the p=7 curved case took 257 us against 251)
  const unsigned v = blockIdx.x * Sh::EPB + slot;
  const bool valid = on && v < (unsigned)Nelements * (unsigned)Nfields;
  const int eidx = (int)(v >> (Nfields - 1)), f = (int)(v & (Nfields - 1));
  const int e = valid ? elementList[eidx] : 0;
  const size_t lbase = ((size_t)e * Nfields + f) * NP;
  const F* const ge = ggeo + 3 * (size_t)e * (AFFINE ? 1 : NP);
  const F* const we = wJ + (size_t)e * (AFFINE ? 1 : NP);
  if (!AFFINE && NQ > 4 && valid && x == 0) {   // (smaller elements: more requests than they save)
    l2_prefetch(ge, 3 * NP);
    l2_prefetch(we, NP);
  }
  F* const U = s_U[slot];
  F* const R = s_R[slot];
  F u[NQ];   // column x
  {
    int32_t id[NQ];
#pragma unroll
    for (int j = 0; j < NQ; ++j) id[j] = valid ? __ldg(G2L + lbase + j * NQ + x) : -1;
#pragma unroll
    for (int j = 0; j < NQ; ++j) u[j] = id[j] >= 0 ? __ldg(q + id[j]) : F(0);
  }
  if (on) {
#pragma unroll
    for (int j = 0; j < NQ; ++j) U[j * RS + x] = u[j];
  }
  __syncthreads();   // D is there
  double pdot = 0.0;
  if (on) {   // r-derivative on row x
    F r[NQ];
#pragma unroll
    for (int n = 0; n < NQ; ++n) r[n] = U[x * RS + n];
#pragma unroll
    for (int o = 0; o < NQ; ++o) R[x * RS + o] = quad_dot<NQ>(s_D + o * DS, r);
  }
  __syncwarp();
  if (on) {   // column x: s-derivative, fluxes, s-part of the divergence
    F ga[3] = {0, 0, 0}, wa = 0;
    if (AFFINE && valid) {
      const F wx = __ldg(gllw + x);
#pragma unroll
      for (int c = 0; c < 3; ++c) ga[c] = __ldg(ge + c) * wx;
      wa = __ldg(we) * wx;
    }
    const F* const gp = (valid ? ge : ggeo) + 3 * x;
    const F* const wp = (valid ? we : wJ) + x;
    F acc[NQ];
#pragma unroll
    for (int n = 0; n < NQ; ++n) acc[n] = 0;
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
      F g0, g1, g2, w;
      if (AFFINE) {
        const F wj = __ldg(gllw + j);
        g0 = ga[0] * wj; g1 = ga[1] * wj; g2 = ga[2] * wj;
        w = wa * wj;
      } else {
        g0 = __ldg(gp + 3 * j * NQ); g1 = __ldg(gp + 3 * j * NQ + 1); g2 = __ldg(gp + 3 * j * NQ + 2);
        w = __ldg(wp + j * NQ);
      }
      const F ur = R[j * RS + x], us = quad_dot<NQ>(s_D + j * DS, u);
      const F fr = g0 * ur + g1 * us, fs = g1 * ur + g2 * us, mq = lambda * w * u[j];
      R[j * RS + x] = fr;
      acc[j] += mq;
      if (DOT && valid)
        pdot += (double)ur * (double)fr + (double)us * (double)fs + (double)mq * (double)u[j];
#pragma unroll
      for (int n = 0; n < NQ; ++n) acc[n] += s_D[j * DS + n] * fs;
    }
#pragma unroll
    for (int n = 0; n < NQ; ++n) U[n * RS + x] = acc[n];
  }
  __syncwarp();
  if (on) {   // r-part of the divergence on row x
    F r[NQ];
#pragma unroll
    for (int n = 0; n < NQ; ++n) r[n] = R[x * RS + n];
#pragma unroll
    for (int o = 0; o < NQ; ++o) U[x * RS + o] += quad_dot<NQ>(s_Dt + o * DS, r);
  }
  __syncwarp();
  if (valid) {   // out by columns: whole sectors
#pragma unroll
    for (int j = 0; j < NQ; ++j) Aq[lbase + j * NQ + x] = U[j * RS + x];
  }
  if (DOT) {
    pdot = warp_tree_sum(pdot);
    if (lane == 0) s_red[threadIdx.x >> 5] = pdot;
    __syncthreads();
    if (threadIdx.x == 0) {
      double r = 0.0;
      for (int w = 0; w < Sh::WARPS; ++w) r += s_red[w];
      fuse.partials[blockIdx.x] = r;
    }
  }
}

// Node form, for meshes too small to fill the chip with warps: one thread per
// node, so an element takes Nq dependent steps where the line form takes Nq^2
// per thread (BK5 p=15, 42 elements: 6.7 us against 12; 100,000 elements 60
// against 39 us the other way).
template <int NQ>
struct QuadNodeShape {
  static constexpr int EPB0 = 256 / (NQ * NQ);
  static constexpr int EPB = EPB0 < 1 ? 1 : (EPB0 > 16 ? 16 : EPB0);   // element slots per block
  static constexpr int RS = NQ + 1;                                     // padded row
  static constexpr int THREADS = NQ * NQ * EPB;
};

template <int NQ, int NF, bool AFFINE, bool DOT, class F>
__global__ void __launch_bounds__(QuadNodeShape<NQ>::THREADS)
ax_quad_node_kernel(int Nelements, const int32_t* __restrict__ elementList, const int32_t* __restrict__ G2L,
               const F* __restrict__ wJ, const F* __restrict__ ggeo, const F* __restrict__ gllw,
               const F* __restrict__ Dg, F lambda, const F* __restrict__ q, F* __restrict__ Aq,
               const int* __restrict__ skip, CgFuse fuse) {
  if (skip && *skip) return;
  using Sh = QuadNodeShape<NQ>;
  constexpr int EPB = Sh::EPB, RS = Sh::RS, NP = NQ * NQ;
  __shared__ F s_D[NQ][RS];
  __shared__ F s_w[NQ];
  __shared__ F s_q[EPB][NF][NQ][RS];
  __shared__ F s_Gr[EPB][NF][NQ][RS];
  __shared__ F s_Gs[EPB][NF][NQ][RS];
  __shared__ double s_red[Sh::THREADS];

  const int i = threadIdx.x, j = threadIdx.y, es = threadIdx.z;
  const int t = i + NQ * (j + NQ * es);
  const int eidx = blockIdx.x * EPB + es;
  const bool active = eidx < Nelements;
  const int e = active ? elementList[eidx] : 0;
  for (int n = t; n < NP; n += Sh::THREADS) s_D[n / NQ][n % NQ] = Dg[n];
  if (AFFINE && t < NQ) s_w[t] = gllw[t];
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    const int32_t id = active ? G2L[((size_t)e * NF + f) * NP + j * NQ + i] : -1;
    s_q[es][f][j][i] = (id != -1) ? q[id] : F(0);
  }
  __syncthreads();

  F G00, G01, G11, GwJ;
  if (AFFINE) {
    const F w = s_w[i] * s_w[j];
    G00 = active ? ggeo[3 * (size_t)e + 0] * w : F(0);
    G01 = active ? ggeo[3 * (size_t)e + 1] * w : F(0);
    G11 = active ? ggeo[3 * (size_t)e + 2] * w : F(0);
    GwJ = active ? wJ[e] * w : F(0);
  } else {
    const size_t gb = (size_t)e * NP + j * NQ + i;
    G00 = active ? ggeo[3 * gb + 0] : F(0);
    G01 = active ? ggeo[3 * gb + 1] : F(0);
    G11 = active ? ggeo[3 * gb + 2] : F(0);
    GwJ = active ? wJ[gb] : F(0);
  }
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    F ur = 0, us = 0;
#pragma unroll
    for (int m = 0; m < NQ; ++m) {
      ur += s_D[i][m] * s_q[es][f][j][m];
      us += s_D[j][m] * s_q[es][f][m][i];
    }
    s_Gr[es][f][j][i] = G00 * ur + G01 * us;
    s_Gs[es][f][j][i] = G01 * ur + G11 * us;
  }
  __syncthreads();
  double pdot = 0.0;
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    const F qn = s_q[es][f][j][i];
    F ap = qn * lambda * GwJ;
#pragma unroll
    for (int m = 0; m < NQ; ++m) {
      ap += s_D[m][i] * s_Gr[es][f][j][m];
      ap += s_D[m][j] * s_Gs[es][f][m][i];
    }
    if (active) Aq[((size_t)e * NF + f) * NP + j * NQ + i] = ap;
    if (DOT) pdot += (double)qn * (double)ap;
  }
  if (DOT) fuse_pap(pdot, fuse, s_red);
}

template <int NQ, class F>
static int launch_quad_nq(const bp_ax_desc_t& d, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                          const F* wJ, const F* ggeo, const F* gllw, const F* D, F lambda, const F* q, F* Aq,
                          const int* skip, const CgFuse* fuse, cudaStream_t s, int* nblocks) {
  using Sh = QuadShape<NQ>;
  const CgFuse Fz = fuse ? *fuse : CgFuse{};
  if (!quad_line_form(d.N, d.affine, d.Nfields, (int)sizeof(F), Nelements)) {
    using Nd = QuadNodeShape<NQ>;
    const dim3 grid((Nelements + Nd::EPB - 1) / Nd::EPB), block(NQ, NQ, Nd::EPB);
    if (nblocks) *nblocks = (int)grid.x;
#define BP_QUAD_NODE(NF)                                                                                             \
  (d.affine ? (fuse ? ax_quad_node_kernel<NQ, NF, true, true, F> : ax_quad_node_kernel<NQ, NF, true, false, F>)       \
            : (fuse ? ax_quad_node_kernel<NQ, NF, false, true, F> : ax_quad_node_kernel<NQ, NF, false, false, F>))
    auto kn = d.Nfields == 1 ? BP_QUAD_NODE(1) : BP_QUAD_NODE(2);
#undef BP_QUAD_NODE
    kn<<<grid, block, 0, s>>>(Nelements, elementList, G2L, wJ, ggeo, gllw, D, lambda, q, Aq, skip, Fz);
    BP_CUDA_TRY(cudaGetLastError());
    return BP_SUCCESS;
  }
  const dim3 grid((unsigned)(((int64_t)Nelements * d.Nfields + Sh::EPB - 1) / Sh::EPB));
  if (nblocks) *nblocks = (int)grid.x;
  auto k = d.affine ? (fuse ? ax_quad_kernel<NQ, true, true, F> : ax_quad_kernel<NQ, true, false, F>)
                    : (fuse ? ax_quad_kernel<NQ, false, true, F> : ax_quad_kernel<NQ, false, false, F>);
  k<<<grid, Sh::THREADS, 0, s>>>(Nelements, d.Nfields, elementList, G2L, wJ, ggeo, gllw, D, lambda, q, Aq, skip, Fz);
  BP_CUDA_TRY(cudaGetLastError());
  return BP_SUCCESS;
}

template <class F>
static int launch_quad_t(const bp_ax_desc_t& d, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                         const F* wJ, const F* ggeo, const F* gllw, const F* D, F lambda, const F* q, F* Aq,
                         const int* skip, const CgFuse* fuse, cudaStream_t s, int* nblocks) {
  if (nblocks) *nblocks = 0;
  if (d.Nfields != 1 && d.Nfields != 2) return fail(BP_ERROR_ARG, "Quad2D operator: Nfields must be 1 or 2");
  if (fuse && fuse->dir) return 1;
  if (Nelements == 0) return BP_SUCCESS;
  switch (d.N + 1) {
#define BP_QUAD_CASE(nq) \
  case nq:               \
    return launch_quad_nq<nq, F>(d, Nelements, elementList, G2L, wJ, ggeo, gllw, D, lambda, q, Aq, skip, fuse, s, nblocks);
    BP_QUAD_CASE(2) BP_QUAD_CASE(3) BP_QUAD_CASE(4) BP_QUAD_CASE(5) BP_QUAD_CASE(6) BP_QUAD_CASE(7)
    BP_QUAD_CASE(8) BP_QUAD_CASE(9) BP_QUAD_CASE(10) BP_QUAD_CASE(11) BP_QUAD_CASE(12) BP_QUAD_CASE(13)
    BP_QUAD_CASE(14) BP_QUAD_CASE(15) BP_QUAD_CASE(16)
#undef BP_QUAD_CASE
    default:
      return fail(BP_ERROR_ARG, "Quad2D operator: degree N must be in 1..15");
  }
}

// Forcing of okl/rhsQuad2D.okl (rhsQuad2D, rhsAffineQuad2D) at the GLL nodes
// of the bilinear map (meshPhysicalNodesQuad2D.cpp)
__global__ void rhs_analytic_quad_kernel(int Nq, int affine, int Nfields, int E, const double* __restrict__ EX,
                                         const double* __restrict__ EY, const double* __restrict__ gllz,
                                         const double* __restrict__ gllw, const double* __restrict__ wJ,
                                         double lambda, double* __restrict__ rL) {
  const int Np = Nq * Nq;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long long)E * Np) return;
  const int e = (int)(gid / Np), n = (int)(gid % Np);
  const int i = n % Nq, j = n / Nq;
  const double r = gllz[i], s = gllz[j];
  const double* ex = EX + 4 * (size_t)e;
  const double* ey = EY + 4 * (size_t)e;
  const double x = 0.25 * (1 - r) * (1 - s) * ex[0] + 0.25 * (1 + r) * (1 - s) * ex[1] +
                   0.25 * (1 + r) * (1 + s) * ex[2] + 0.25 * (1 - r) * (1 + s) * ex[3];
  const double y = 0.25 * (1 - r) * (1 - s) * ey[0] + 0.25 * (1 + r) * (1 - s) * ey[1] +
                   0.25 * (1 + r) * (1 + s) * ey[2] + 0.25 * (1 - r) * (1 + s) * ey[3];
  const double w = affine ? wJ[e] * gllw[i] * gllw[j] : wJ[gid];
  const double pi = 3.14159265358979323846;
  if (Nfields == 1) {
    rL[gid] = w * ((2 * pi * pi + lambda) * sin(pi * x) * sin(pi * y));
  } else {
    const size_t base = (size_t)e * Np * 2 + n;
    rL[base] = w * ((3 * pi * pi + lambda) * sin(2.0 * pi * x) * sin(pi * y));
    rL[base + Np] = w * ((3 * pi * pi + lambda) * sin(pi * x) * sin(2.0 * pi * y));
  }
}

// rL[l] = wJ_l f[G2L[l]] (0 on masked nodes), Quad2D weights
__global__ void mass_local_quad_kernel(int Nq, int affine, int Nfields, int E, const int32_t* __restrict__ G2L,
                                       const double* __restrict__ gllw, const double* __restrict__ wJ,
                                       const double* __restrict__ f, double* __restrict__ rL) {
  const int Np = Nq * Nq;
  const long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= (long long)E * Np * Nfields) return;
  const int e = (int)(l / ((long long)Np * Nfields));
  const int n = (int)(l % Np);
  const double w = affine ? wJ[e] * gllw[n % Nq] * gllw[n / Nq] : wJ[(size_t)e * Np + n];
  const int32_t id = G2L[l];
  rL[l] = (id != -1) ? w * f[id] : 0.0;
}

// Element diagonal of the Quad2D operator (Jacobi): the two 1D stiffness
// directions, the mixed term at the node and lambda wJ
__global__ void diag_local_quad_kernel(int Nq, int affine, int Nfields, int E, const double* __restrict__ ggeo,
                                       const double* __restrict__ wJ, const double* __restrict__ gllw,
                                       const double* __restrict__ D, double lambda, double* __restrict__ dL) {
  const int Np = Nq * Nq;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long long)E * Np) return;
  const int e = (int)(gid / Np), n = (int)(gid % Np);
  const int i = n % Nq, j = n / Nq;
  auto G = [&](int ii, int jj, int c) -> double {
    if (affine) return ggeo[3 * (size_t)e + c] * gllw[ii] * gllw[jj];
    return ggeo[3 * ((size_t)e * Np + ii + jj * Nq) + c];
  };
  double d = 0.0;
  for (int m = 0; m < Nq; ++m) {
    d += G(m, j, 0) * D[m * Nq + i] * D[m * Nq + i];
    d += G(i, m, 2) * D[m * Nq + j] * D[m * Nq + j];
  }
  d += 2 * G(i, j, 1) * D[i * Nq + i] * D[j * Nq + j];
  d += lambda * (affine ? wJ[e] * gllw[i] * gllw[j] : wJ[gid]);
  for (int f = 0; f < Nfields; ++f) dL[(size_t)e * Np * Nfields + (size_t)f * Np + n] = d;
}

}  // namespace

int launch_ax_quad(const bp_ax_desc_t& d, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                   const double* wJ, const double* ggeo, const double* gllw, const double* D, double lambda,
                   const double* q, double* Aq, const int* skip, const CgFuse* fuse, cudaStream_t s, int* nblocks) {
  return launch_quad_t<double>(d, Nelements, elementList, G2L, wJ, ggeo, gllw, D, lambda, q, Aq, skip, fuse, s,
                               nblocks);
}

int launch_ax_quad(const bp_ax_desc_t& d, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                   const float* wJ, const float* ggeo, const float* gllw, const float* D, float lambda,
                   const float* q, float* Aq, const int* skip, const CgFuse* fuse, cudaStream_t s, int* nblocks) {
  return launch_quad_t<float>(d, Nelements, elementList, G2L, wJ, ggeo, gllw, D, lambda, q, Aq, skip, fuse, s,
                              nblocks);
}

int launch_rhs_analytic_quad(int N, int affine, int Nfields, int E, const double* EX, const double* EY,
                             const double* gllz, const double* gllw, const double* wJ, double lambda, double* rL,
                             cudaStream_t s) {
  const int Nq = N + 1;
  const long long tot = (long long)E * Nq * Nq;
  if (tot == 0) return BP_SUCCESS;
  rhs_analytic_quad_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(Nq, affine, Nfields, E, EX, EY, gllz, gllw,
                                                                           wJ, lambda, rL);
  BP_CUDA_TRY(cudaGetLastError());
  return BP_SUCCESS;
}

int launch_mass_local_quad(int N, int affine, int Nfields, int E, const int32_t* G2L, const double* gllw,
                           const double* wJ, const double* f, double* rL, cudaStream_t s) {
  const int Nq = N + 1;
  const long long tot = (long long)E * Nq * Nq * Nfields;
  if (tot == 0) return BP_SUCCESS;
  mass_local_quad_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(Nq, affine, Nfields, E, G2L, gllw, wJ, f,
                                                                         rL);
  BP_CUDA_TRY(cudaGetLastError());
  return BP_SUCCESS;
}

int launch_diag_local_quad(int N, int affine, int Nfields, int E, const double* ggeo, const double* wJ,
                           const double* gllw, const double* D, double lambda, double* dL, cudaStream_t s) {
  const int Nq = N + 1;
  const long long tot = (long long)E * Nq * Nq;
  if (tot == 0) return BP_SUCCESS;
  diag_local_quad_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(Nq, affine, Nfields, E, ggeo, wJ, gllw, D,
                                                                         lambda, dL);
  BP_CUDA_TRY(cudaGetLastError());
  return BP_SUCCESS;
}

}  // namespace bp
