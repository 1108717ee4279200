// Over-integrated element operators of BP1-BP4 (mass, and stiffness + lambda
// mass, evaluated at N+2 Gauss points per direction).  Included once by
// bp_ax_cub64.cu (BP_CUB_REAL = double) and once by bp_ax_cub32.cu
// (BP_CUB_REAL = float, the mixed-precision CG); each inclusion is its own
// CUDA module with its own constant bank.
//
// Forms (reference kernels):
//   CUB_MASS_AFFINE   wJ_e (MM x MM x MM) q                  okl/bp1AxAffineHex3D.okl:29-135
//   CUB_MASS          I^T (cubwJ . (I q))                     okl/bp1AxHex3D.okl
//   CUB_STIFF_AFFINE  invV^T (S_modal + lambda wJ_e) invV q   okl/bp3AxAffineHex3D.okl:29-258
//   CUB_STIFF         I^T (S_cub + lambda cubwJ) I q          okl/bp3AxHex3D.okl:29-340
// with S = Dr^T(G00 Dr + G01 Ds + G02 Dt) + Ds^T(...) + Dt^T(...) on the
// quadrature grid.  BP2/BP4 apply the same operator to each of the 3 fields.
//
// Work mapping.  Every 1D step (interpolation, derivative, projection, weak
// derivative) is a small matrix applied along lines of the element's grid.  A
// thread owns one line of every step: it reads the line into registers and
// writes all of its outputs, so the matrix index of every multiply-add is the
// same in all threads of the warp and the matrices live in the constant bank
// (c_cub below); shared memory only carries the field between steps whose line
// direction changes.  The steps of one (element, field):
//   b-lines of nodes (a, c), a-lines (j, c), c-lines (i, j)   interpolation
//   rows (y, z), columns (x, z)                                r-, s-derivative
//   columns (x, y)     t-derivative, fluxes, t-part of the weak divergence
//   rows, columns                                              r-, s-part added
//   columns (x, z), (x, b), rows (b, c)                        projection
// The mass forms go from the c-line to the points and back in registers.
//
// What bounds it: the FP64 stiffness at p=7 moves 50 KB of factors and values
// and 25 passes of 8 bytes per point through shared memory; DRAM, the shared-
// memory pipe and FP64 arithmetic need 0.49, 0.3 and 0.3 ms of a 40^3 launch.
// What it takes is many independent warps with few registers: one element per
// block of three warps keeps 18-24 warps per SM resident, and a bulk prefetch
// asks L2 for the element's factors while q is gathered and interpolated, so
// the flux loop reads them without a trip to DRAM.  Measured at 40^3 curved
// p=7 (before: three elements in lockstep per block of 243 threads, outer
// loops rolled for registers, 16 warps): BK3 FP64 1.376 -> 0.79 ms, BK1 at
// 32^3 365 -> 131 us, FP32 BK3 at 19x19x20 87 -> 61 us; BK4 p=5 on 21x18x23
// 221 -> 147 us.
#pragma once

#ifndef BP_CUB_REAL
#error "define BP_CUB_REAL (double or float) before including bp_ax_cub.cuh"
#endif

#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "bp_cg_device.cuh"
#include "bp_internal.hpp"

namespace bp {
namespace {

using CubReal = BP_CUB_REAL;

enum CubForm { CUB_MASS_AFFINE = 0, CUB_MASS = 1, CUB_STIFF_AFFINE = 2, CUB_STIFF = 3 };

// Constant-bank table, three groups of one slot per degree: the curved forms
// (T = cubInterp [G x NQ], then cubD [G x G]; mass and stiffness share the
// slot, both write the mesh's cubInterp), the affine stiffness forms of
// BP3/BP4 (T = invV [NQ x NQ], then the modal cubD [NQ x NQ]) and the affine
// mass forms of BP1/BP2 (T = MM [NQ x NQ]).  Each launch first copies its
// operands into its slot on the launch stream (once per slot and source in a
// stream capture: const_slot_copy), so two launches of the same
// degree and group on different streams must pass the same matrices (every
// caller that passes its mesh's own matrices does); operators of different
// groups never share a slot.
__host__ __device__ constexpr int cub_curved_size(int nq) { return (nq + 1) * nq + (nq + 1) * (nq + 1); }
__host__ __device__ constexpr int cub_affine_size(int nq) { return 2 * nq * nq; }
__host__ __device__ constexpr int cub_mass_affine_size(int nq) { return nq * nq; }
__host__ __device__ constexpr int cub_slot(int nq, int form) {
  const int group = (form == CUB_MASS || form == CUB_STIFF) ? 0 : form == CUB_STIFF_AFFINE ? 1 : 2;
  int off = 0;
  for (int n = 2; n < (group == 0 ? nq : 17); ++n) off += cub_curved_size(n);
  if (group >= 1)
    for (int n = 2; n < (group == 1 ? nq : 17); ++n) off += cub_affine_size(n);
  if (group == 2)
    for (int n = 2; n < nq; ++n) off += cub_mass_affine_size(n);
  return off;
}
constexpr int kCubTable = cub_slot(17, CUB_MASS_AFFINE);
static_assert(kCubTable * sizeof(double) <= 64 * 1024, "constant table exceeds the 64 KB bank");

static __constant__ CubReal c_cub[kCubTable];

// Slots per block, registers a thread may take and unrolling, by the points G
// per direction (sweeps over 8,000 to 2.5 million nodes, one and three fields,
// with and without q.Aq; times below are the geometric mean over these).
// Several slots only where one leaves the block small (a mass element of 9
// threads: 28 slots 2940 GB/s, 7 slots 1950; curved, 14 slots take 0.97 of 21's
// time, affine 1.19; FP64 stiffness 0.92 with 48 registers) or a warp half empty
// (G = 6: 36 threads).  Registers: few, for more resident blocks, where a few
// spilled values cost less than these give (FP64 stiffness G = 9: 96 registers
// 4002, 80 3726 GB/s; G = 10: 96 3855, 128 3620).  Outputs of a line are unrolled
// but for FP64 G = 13 and 17 and the curved FP32 G = 13 (spills).  The flux loop runs three points at a time in FP64 and, in
// FP32, as a whole up to G = 7 (0.87-0.95 of the time of three at a time, or of
// one at a time at G = 6).  FP32 G = 12: unrolled outputs 0.82 (curved) and 0.70
// (affine) of rolled ones; G = 13 and 14, with 80 and 128 registers, 0.85-0.95
// and 0.83-0.89.  The mass columns run as a whole (FP64 G = 11: 3083 against
// 2946 GB/s by three), except where that spills (G = 16: 350 against 62 us).
template <int NQ, int FORM>
struct CubRule {
  static constexpr bool CURVED = (FORM == CUB_MASS || FORM == CUB_STIFF);
  static constexpr bool STIFF = (FORM == CUB_STIFF_AFFINE || FORM == CUB_STIFF);
  static constexpr bool D = sizeof(CubReal) == 8;
  static constexpr int G = CURVED ? NQ + 1 : NQ;
  static constexpr int EPB =
      G == 2   ? 24
      : G == 3 ? (STIFF || CURVED ? 14 : 21)
      : STIFF  ? (G == 4 ? (D ? 6 : 8) : G == 5 ? 5 : G == 6 ? (D ? 5 : 3) : G == 8 && D ? 2 : 1)
               : (G == 4 ? (CURVED ? 8 : 12) : G <= 6 ? 5 : G == 7 ? 3 : G == 8 ? 2 : 1);
  static constexpr int WARPS = (G * G * EPB + 31) / 32;
  static constexpr int REGS = !D       ? (G <= 7 ? 48 : G == 13 && STIFF ? 80 : G == 14 && STIFF ? 128 : 3 * G + 26)
                              : !STIFF ? 4 * G + 24
                              : G == 3 ? 48
                              : G <= 6 ? 64
                              : G == 7 ? 80
                              : G <= 13 ? 100
                              : G <= 16 ? 128 : 170;
  static constexpr int minb(bool dot) {   // resident blocks to allow for (the q.Aq form takes 8 registers more)
    const int n = 65536 / (WARPS * 32 * (REGS + (dot ? 8 : 0)));
    return n < 1 ? 1 : n * WARPS > 64 ? 64 / WARPS : n > 32 ? 32 : n;
  }
  static constexpr int UN = !STIFF ? G : D ? (G == 13 || G == 17 ? 3 : G) : (G == 13 && CURVED ? 4 : G);
  static constexpr int UK = !STIFF ? (G == 16 ? 3 : G)
                            : D    ? (G == 6 ? 1 : 3)
                                   : (G <= 7 ? G : G == 13 || G == 14 ? 4 : 3);
};

// One element (of one field) per slot of G x G threads, EPB slots per block.
template <int NQ, int FORM>
struct CubShape {
  static constexpr bool CURVED = (FORM == CUB_MASS || FORM == CUB_STIFF);
  static constexpr bool STIFF = (FORM == CUB_STIFF_AFFINE || FORM == CUB_STIFF);
  static constexpr int G = CURVED ? NQ + 1 : NQ;   // quadrature points per direction
  static constexpr int G2 = G * G, GP = G * G2, NP = NQ * NQ * NQ;
  // row and plane strides of a G^3 field: the rows, columns and lines that a
  // warp's threads walk fall in distinct banks where that is possible (strides
  // chosen by counting the wavefronts of every access of the kernel for all
  // row strides G..G+2 and plane pads 0..15; at even G a stride of G + 1 or a
  // pad cuts them by 5-20%)
  static constexpr int RS = (G % 2 || G == 6 || G == 10 || G == 14) ? G : G + 1;
  static constexpr int PAD = G == 6 ? 1 : G == 7 ? 5 : G == 10 ? 5 : G == 14 ? 9 : G == 16 ? 15 : 0;
  static constexpr int PL = G * RS + PAD;
  static constexpr int FIELD = G * PL;
  static constexpr int NBUF = STIFF ? 3 : 1;        // u, and the r and s buffers of the stiffness
  static constexpr int EPB = CubRule<NQ, FORM>::EPB;
  static constexpr int THREADS = (G2 * EPB + 31) / 32 * 32;   // whole warps; the last threads own no line
  static constexpr size_t FIELDS = sizeof(CubReal) * (size_t)NBUF * FIELD * EPB;
  static constexpr size_t SMEM = FIELDS < sizeof(double) * THREADS ? sizeof(double) * THREADS : FIELDS;
  static constexpr int SLOT = cub_slot(NQ, FORM);
  static constexpr int TSIZE = G * NQ;              // T rows = output points
  static constexpr int DSIZE = STIFF ? G * G : 0;
};

// The 1D matrices of a form in the constant bank: T(o, i) maps NQ nodes to G
// points (MASS_AFFINE applies MM^T), D(a, b) is G x G.
#define CUB_T(o, i) \
  (FORM == CUB_MASS_AFFINE ? c_cub[Sh::SLOT + (i) * NQ + (o)] : c_cub[Sh::SLOT + (o) * NQ + (i)])
#define CUB_D(a, b) c_cub[Sh::SLOT + Sh::TSIZE + (a) * Sh::G + (b)]

// A line of NI values through the NO x NI matrix mat(o, n): store(o, value).
template <int NI, int NO, int UN, class F, class Mat, class Store>
__device__ __forceinline__ void cub_line(const F (&r)[NI], Mat mat, Store store) {
#pragma unroll UN
  for (int o = 0; o < NO; ++o) {
    F a = 0;
#pragma unroll
    for (int n = 0; n < NI; ++n) a += mat(o, n) * r[n];
    store(o, a);
  }
}
template <int N, int STRIDE, class F>
__device__ __forceinline__ void cub_load(const F* p, F (&r)[N]) {
#pragma unroll
  for (int n = 0; n < N; ++n) r[n] = p[n * STRIDE];
}

template <int NQ, int FORM, bool DOT>
__global__ void __launch_bounds__((CubShape<NQ, FORM>::THREADS), (CubRule<NQ, FORM>::minb(DOT)))
ax_cub_kernel(int Nelements, int Nfields, const int32_t* __restrict__ elementList, const int32_t* __restrict__ G2L,
              const CubReal* __restrict__ wJ, const CubReal* __restrict__ ggeo, CubReal lambda,
              const CubReal* __restrict__ q, CubReal* __restrict__ Aq, const int* __restrict__ skip,
              double* __restrict__ partials) {
  pdl_wait();
  pdl_release();
  if (skip && *skip) return;
  using F = CubReal;
  using Sh = CubShape<NQ, FORM>;
  using V2 = typename std::conditional<sizeof(F) == 8, double2, float2>::type;
  constexpr int G = Sh::G, G2 = Sh::G2, GP = Sh::GP, NQ2 = NQ * NQ, NP = Sh::NP, RS = Sh::RS, PL = Sh::PL;
  constexpr int EPB = Sh::EPB, UN = CubRule<NQ, FORM>::UN, UK = CubRule<NQ, FORM>::UK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // The guards t < G2 (hi < G, ...) are also what keeps the steps apart: as one
  // straight line of code the scheduler moved loads and addresses of later
  // steps up and spilled (BK3 p=7: 854 against 752 us).
  const int slot = EPB == 1 || threadIdx.x >= G2 * EPB ? 0 : threadIdx.x / G2;
  const int t = threadIdx.x - slot * G2;      // >= G2: no line
  F* const U = reinterpret_cast<F*>(smem_raw) + (size_t)slot * Sh::NBUF * Sh::FIELD;   // the field
  F* const R = U + Sh::FIELD;                                // r-derivative / r-flux
  F* const S = R + Sh::FIELD;                                // s-derivative / s-flux
  const int64_t v = (int64_t)blockIdx.x * EPB + slot;        // element-major (element, field)
  const bool valid = v < (int64_t)Nelements * Nfields;
  const int eidx = Nfields == 1 ? (int)v : (int)(v / Nfields), f = (int)(v - (int64_t)eidx * Nfields);
  const int element = valid ? elementList[eidx] : 0;
  const size_t lbase = ((size_t)element * Nfields + f) * NP;
  const F* const ge = ggeo + 6 * (size_t)element * (Sh::CURVED ? GP : 1);
  const F* const we = wJ + (size_t)element * (Sh::CURVED ? GP : 1);
  if (Sh::CURVED && valid && t == 0) {   // the element's factors, while q is gathered and interpolated
    if (Sh::STIFF) l2_prefetch(ge, 6 * GP);
    l2_prefetch(we, GP);
  }
  // line (y, z), (x, z) or (x, y) of this thread in the roles of the steps
  // G x G lines hi < G; G x NQ lines hi < NQ; NQ x NQ lines hn < NQ
  const int hi = t / G, lo = t - hi * G, hn = t / NQ, ln = t - hn * NQ;
  const auto T = [](int o, int i) { return CUB_T(o, i); };
  const auto Tt = [](int o, int i) { return CUB_T(i, o); };
  const auto D = [](int o, int i) { return CUB_D(o, i); };
  const auto Dt = [](int o, int i) { return CUB_D(i, o); };
  double pdot = 0.0;
  // q.A_e q, where its factors are in registers: at the points, lambda w (I q)^2
  // and the gradient times the flux (the affine mass has no such place and
  // gathers q again)

  // interpolation: along b from the gathered nodes (a, c) = (ln, hn)
  if (hn < NQ) {
    int32_t id[NQ];
    F r[NQ];
#pragma unroll
    for (int b = 0; b < NQ; ++b) id[b] = valid ? __ldg(G2L + lbase + hn * NQ2 + b * NQ + ln) : -1;
#pragma unroll
    for (int b = 0; b < NQ; ++b) r[b] = id[b] >= 0 ? __ldg(q + id[b]) : F(0);
    F* const p = U + hn * PL + ln;
    cub_line<NQ, G, UN>(r, T, [&](int o, F x) { p[o * RS] = x; });
  }
  __syncthreads();
  // along a, rows (j, c) = (lo, hi)
  if (hi < NQ) {
    F* const p = U + hi * PL + lo * RS;
    F r[NQ];
    cub_load<NQ, 1>(p, r);
    cub_line<NQ, G, UN>(r, T, [&](int o, F x) { p[o] = x; });
  }
  __syncthreads();

  F* const col = U + hi * RS + lo;            // column (i, j) = (lo, hi), this thread's own
  if constexpr (FORM == CUB_MASS_AFFINE) {
    if (t < G2 && valid) {
      F r[NQ];
      cub_load<NQ, PL>(col, r);
      const F wa = __ldg(we);
      cub_line<NQ, NQ, UN>(r, T, [&](int o, F x) {
        const size_t l = lbase + o * NQ2 + t;
        const F y = wa * x;
        Aq[l] = y;
        if (DOT) {
          const int32_t id = __ldg(G2L + l);
          pdot += (double)(id >= 0 ? __ldg(q + id) : F(0)) * (double)y;
        }
      });
    }
  } else if constexpr (FORM == CUB_MASS) {
    // along c to the points, the weights, and back along c: row k of T serves both
    if (t < G2) {
      F r[NQ], a[NQ];
      cub_load<NQ, PL>(col, r);
#pragma unroll
      for (int n = 0; n < NQ; ++n) a[n] = 0;
      const F* const wp = (valid ? we : wJ) + t;
#pragma unroll UK
      for (int k = 0; k < G; ++k) {
        F o = 0, m[NQ];
#pragma unroll
        for (int n = 0; n < NQ; ++n) {
          m[n] = CUB_T(k, n);
          o += m[n] * r[n];
        }
        const F w = __ldg(wp + k * G2);
        if (DOT && valid) pdot += (double)(w * o) * (double)o;
        o *= w;
#pragma unroll
        for (int n = 0; n < NQ; ++n) a[n] += m[n] * o;
      }
#pragma unroll
      for (int n = 0; n < NQ; ++n) col[n * PL] = a[n];
    }
    __syncthreads();
    if (hi < NQ) {   // along a, rows (j, c)
      F* const p = U + hi * PL + lo * RS;
      F s[G];
      cub_load<G, 1>(p, s);
      cub_line<G, NQ, UN>(s, Tt, [&](int o, F x) { p[o] = x; });
    }
    __syncthreads();
    if (hn < NQ && valid) {   // along b, columns (a, c)
      F s[G];
      cub_load<G, RS>(U + hn * PL + ln, s);
      cub_line<G, NQ, UN>(s, Tt, [&](int o, F x) { Aq[lbase + hn * NQ2 + o * NQ + ln] = x; });
    }
  } else {
    if (t < G2) {   // along c to the points
      F r[NQ];
      cub_load<NQ, PL>(col, r);
      cub_line<NQ, G, UN>(r, T, [&](int o, F x) { col[o * PL] = x; });
    }
    __syncthreads();
    const int row = hi * PL + lo * RS, scol = hi * PL + lo;   // row (y, z), column (x, z) = (lo, hi)
    if (t < G2) {
      F r[G];
      cub_load<G, 1>(U + row, r);
      cub_line<G, G, UN>(r, D, [&](int o, F x) { R[row + o] = x; });
      cub_load<G, RS>(U + scol, r);
      cub_line<G, G, UN>(r, D, [&](int o, F x) { S[scol + o * RS] = x; });
    }
    __syncthreads();
    if (t < G2) {   // the fluxes at the points of the column, the t-derivative and the t-part of the
                    // divergence: row k of D serves both
      F ga[6] = {0, 0, 0, 0, 0, 0}, wa = 0;
      if (!Sh::CURVED && valid) {
#pragma unroll
        for (int c = 0; c < 6; ++c) ga[c] = __ldg(ge + c);
        wa = __ldg(we);
      }
      const F* const gp = (valid ? ge : ggeo) + 6 * t;
      const F* const wp = (valid ? we : wJ) + t;
      F u[G], acc[G];
      cub_load<G, PL>(col, u);
#pragma unroll
      for (int n = 0; n < G; ++n) acc[n] = 0;
      F *pr = R + hi * RS + lo, *ps = S + hi * RS + lo;
#pragma unroll UK
      for (int k = 0; k < G; ++k) {
        F g[6], w;
        if (Sh::CURVED) {
          const V2* gv = reinterpret_cast<const V2*>(gp + 6 * k * G2);
          const V2 a0 = __ldg(gv), a1 = __ldg(gv + 1), a2 = __ldg(gv + 2);
          g[0] = a0.x; g[1] = a0.y; g[2] = a1.x; g[3] = a1.y; g[4] = a2.x; g[5] = a2.y;
          w = __ldg(wp + k * G2);
        } else {
#pragma unroll
          for (int c = 0; c < 6; ++c) g[c] = ga[c];
          w = wa;
        }
        F m[G], d0 = 0, d1 = 0;   // two chains: the sum is on the critical path
#pragma unroll
        for (int n = 0; n < G; ++n) {
          m[n] = CUB_D(k, n);
          if (n & 1) d1 += m[n] * u[n];
          else d0 += m[n] * u[n];
        }
        const F dr = pr[k * PL], ds = ps[k * PL], dt = d0 + d1, qk = col[k * PL];
        const F fr = g[0] * dr + g[1] * ds + g[2] * dt, fs = g[1] * dr + g[3] * ds + g[4] * dt;
        const F gt = g[2] * dr + g[4] * ds + g[5] * dt, mq = lambda * w * qk;
        col[k * PL] = mq;
        pr[k * PL] = fr;
        ps[k * PL] = fs;
        if (DOT && valid)   // products in FP64: their range is that of the squares
          pdot += (double)dr * (double)fr + (double)ds * (double)fs + (double)dt * (double)gt + (double)mq * (double)qk;
#pragma unroll
        for (int n = 0; n < G; ++n) acc[n] += m[n] * gt;
      }
#pragma unroll
      for (int n = 0; n < G; ++n) col[n * PL] += acc[n];
    }
    __syncthreads();
    if (t < G2) {   // the r-part, added on rows
      F r[G];
      cub_load<G, 1>(R + row, r);
      cub_line<G, G, UN>(r, Dt, [&](int o, F x) { U[row + o] += x; });
    }
    __syncthreads();
    if (t < G2) {   // the s-part, added on columns (x, z), and the projection along b of the same columns
      F r[G];
      cub_load<G, RS>(S + scol, r);
      cub_line<G, G, UN>(r, Dt, [&](int o, F x) { U[scol + o * RS] += x; });
      cub_load<G, RS>(U + scol, r);
      cub_line<G, NQ, UN>(r, Tt, [&](int o, F x) { U[scol + o * RS] = x; });
    }
    __syncthreads();
    if (hi < NQ) {   // along c, columns (x, b) = (lo, hi)
      F r[G];
      cub_load<G, PL>(col, r);
      cub_line<G, NQ, UN>(r, Tt, [&](int o, F x) { col[o * PL] = x; });
    }
    __syncthreads();
    if (hn < NQ) {   // along a, rows (b, c) = (ln, hn)
      F* const p = U + hn * PL + ln * RS;
      F r[G];
      cub_load<G, 1>(p, r);
      cub_line<G, NQ, UN>(r, Tt, [&](int o, F x) { p[o] = x; });
    }
    __syncthreads();
    if (valid && t < G2)   // out in node order: whole sectors
      for (int n = t; n < NP; n += G2) {
        const int c = n / NQ2, m = n - c * NQ2, b = m / NQ, a = m - b * NQ;
        Aq[lbase + n] = U[c * PL + b * RS + a];
      }
  }
  if (DOT) {
    const double bs = fuse_block_sum(pdot, reinterpret_cast<double*>(smem_raw));
    if (threadIdx.x == 0) partials[blockIdx.x] = bs;
  }
}
#undef CUB_D
#undef CUB_T

// device address of the constant table on the current device
static CubReal* cub_table_address() {
  static DeviceSymbol sym(c_cub);
  return static_cast<CubReal*>(sym.address());
}

template <int NQ, int FORM>
static int launch_cub_form(int32_t Nelements, int Nfields, const int32_t* elementList, const int32_t* G2L,
                           const CubOperands<CubReal>& o, CubReal lambda, const CubReal* q, CubReal* Aq,
                           const int* skip, cudaStream_t s, double* partials, int* nblocks) {
  using Sh = CubShape<NQ, FORM>;
  if (Sh::CURVED && Sh::STIFF && (reinterpret_cast<uintptr_t>(o.ggeo) % (2 * sizeof(CubReal))))
    return fail(BP_ERROR_ARG, "over-integrated operator: cubggeo must be aligned to two elements");
  CubReal* tab = cub_table_address();
  if (!tab) return fail(BP_ERROR_CUDA, "over-integrated operator: constant table address lookup failed");
  // this launch's 1D operands into its slot of the constant bank, in stream order
  BP_TRY(const_slot_copy(tab + Sh::SLOT, o.T, sizeof(CubReal) * Sh::TSIZE, s));
  if (Sh::STIFF)
    BP_TRY(const_slot_copy(tab + Sh::SLOT + Sh::TSIZE, o.D, sizeof(CubReal) * Sh::DSIZE, s));
  auto k = partials ? ax_cub_kernel<NQ, FORM, true> : ax_cub_kernel<NQ, FORM, false>;
  if (Sh::SMEM > 48 * 1024)
    BP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::SMEM));
  const dim3 grid((unsigned)(((int64_t)Nelements * Nfields + Sh::EPB - 1) / Sh::EPB));
  if (nblocks) *nblocks = (int)grid.x;
  BP_CUDA_TRY(launch_pdl(k, grid, dim3(Sh::THREADS), Sh::SMEM, s, Nelements, Nfields, elementList,
                         G2L, o.wJ, o.ggeo, lambda, q, Aq, skip, partials));
  return BP_SUCCESS;
}

template <int NQ>
static int launch_cub_nq(const bp_ax_desc_t& d, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                         const CubOperands<CubReal>& o, CubReal lambda, const CubReal* q, CubReal* Aq,
                         const int* skip, cudaStream_t s, double* partials, int* nblocks) {
  const bool stiff = d.bp >= 3;
#define BP_CUB(FORM) \
  return launch_cub_form<NQ, FORM>(Nelements, d.Nfields, elementList, G2L, o, lambda, q, Aq, skip, s, partials, nblocks)
  if (d.affine) {
    if (stiff) BP_CUB(CUB_STIFF_AFFINE);
    BP_CUB(CUB_MASS_AFFINE);
  }
  if (stiff) BP_CUB(CUB_STIFF);
  BP_CUB(CUB_MASS);
#undef BP_CUB
}

int launch_ax_cub_impl(const bp_ax_desc_t& d, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                       const CubOperands<CubReal>& o, CubReal lambda, const CubReal* q, CubReal* Aq,
                       const int* skip, cudaStream_t s, const CgFuse* fuse, int* nblocks) {
  if (nblocks) *nblocks = 0;
  if (d.bp < 1 || d.bp > 4) return fail(BP_ERROR_ARG, "over-integrated operator: bp must be 1..4");
  if (d.Nfields != ((d.bp % 2) ? 1 : 3))
    return fail(BP_ERROR_ARG, "over-integrated operator: BP1/BP3 take 1 field, BP2/BP4 3");
  if (Nelements == 0) return BP_SUCCESS;
  double* partials = fuse ? fuse->partials : nullptr;
  switch (d.N + 1) {
#define BP_CUB_CASE(nq) \
  case nq:              \
    return launch_cub_nq<nq>(d, Nelements, elementList, G2L, o, lambda, q, Aq, skip, s, partials, nblocks);
    BP_CUB_CASE(2) BP_CUB_CASE(3) BP_CUB_CASE(4) BP_CUB_CASE(5) BP_CUB_CASE(6) BP_CUB_CASE(7) BP_CUB_CASE(8)
    BP_CUB_CASE(9) BP_CUB_CASE(10) BP_CUB_CASE(11) BP_CUB_CASE(12) BP_CUB_CASE(13) BP_CUB_CASE(14)
    BP_CUB_CASE(15) BP_CUB_CASE(16)
#undef BP_CUB_CASE
    default:
      return fail(BP_ERROR_ARG, "over-integrated operator: degree N must be in 1..15");
  }
}

}  // namespace
}  // namespace bp
