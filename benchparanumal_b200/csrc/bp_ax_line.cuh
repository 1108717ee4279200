// BP5/BP6 element operator (GLL collocation) in the line-per-thread form of
// bp_ax_cub.cuh: every 1D derivative is a constant-bank matrix applied along
// whole lines owned by single threads.  Included once by bp_ax_line64.cu
// (BP_LINE_REAL = double) and once by bp_ax_line32.cu (float).
//
//   Aq_e = Dr^T(G00 ur + G01 us + G02 ut) + Ds^T(G01 ur + G11 us + G12 ut)
//        + Dt^T(G02 ur + G12 us + G22 ut) + lambda wJ q,  (ur,us,ut) = (Dr,Ds,Dt) q
// (okl/bp5AxHex3D.okl:415-569, okl/bp5AxAffineHex3D.okl:419-579,
// okl/bp6AxHex3D.okl:50-255).  Stored factors carry the GLL weights; affine
// factors are per element and the weights w_i w_j w_k are applied here.
//
#pragma once

#ifndef BP_LINE_REAL
#error "define BP_LINE_REAL (double or float) before including bp_ax_line.cuh"
#endif

#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "bp_cg_device.cuh"
#include "bp_internal.hpp"
#include "bp_pack.cuh"

namespace bp {
namespace {

using LineReal = BP_LINE_REAL;

// constant table: per degree D [NQ x NQ] then gllw [NQ]
__host__ __device__ constexpr int line_slot(int nq) {
  int off = 0;
  for (int n = 2; n < nq; ++n) off += n * n + n;
  return off;
}
constexpr int kLineTable = line_slot(17);
static __constant__ LineReal c_line[kLineTable];

// Packed values (PK right-hand sides per node): elements per block, and the
// registers a thread may take.  Small blocks that do not wait for one another
// beat elements in lockstep (four per block of 256 threads before), as for one
// value per node below.
template <int NQ, class T>
struct LineShape {
  static constexpr int G2 = NQ * NQ;
  // 16-byte values: eight threads of a row or column walk fall in distinct
  // bank groups at an odd row stride
  static constexpr int RS = (NQ % 2) ? NQ : NQ + 1;
  static constexpr int PLANE = NQ * RS;
  static constexpr int FIELD = NQ * PLANE;
  static constexpr int EPB = NQ == 2 ? 16 : NQ == 3 ? 7 : NQ == 4 ? 4 : NQ == 5 ? 5 : NQ == 6 ? 3 : 1;
  static constexpr int THREADS = (G2 * EPB + 31) / 32 * 32;   // whole warps; the last threads own no line
  static constexpr int SLOT = line_slot(NQ);
  static constexpr size_t SMEM0 = sizeof(T) * (size_t)3 * FIELD * EPB;
  static constexpr size_t RED = sizeof(double) * PackTraits<T>::R * THREADS;   // the block sums' scratch
  static constexpr size_t smem() { return SMEM0 < RED ? RED : SMEM0; }
};

template <int NQ, class T>
struct LineMinBlocks {
  static constexpr int REGS = PackTraits<T>::R >= 4 ? (NQ <= 8 ? 128 : NQ <= 11 ? 168 : 200) : (NQ <= 8 ? 96 : 128);
  static constexpr int V0 = 65536 / (LineShape<NQ, T>::THREADS * REGS);
  static constexpr int V = V0 < 1 ? 1 : V0;
};

// T = Pack<LineReal, PK>: PK right-hand sides of one mesh in lockstep, one pack
// per node; p.Ap partials per lane at partials[lane * gridDim.x + blockIdx.x].
// The lines are the same as with one value per node, but the t-part of the
// result stays with the thread of column (x, y), whose q is still in shared
// memory at the end: forming p.Ap from q and the result takes two conversions
// to FP64 per lane and node, from gradients and fluxes eight.
//
// Each value crosses shared memory once per step (17 16-byte accesses per
// node; the TMA form's row and column reads take 32 and more).
// The body works on element block `blk` of `nblk` (partials[lane * nblk +
// blk]) in the dynamic shared memory smem_raw: the kernel below and the
// persistent CG step share it.
template <int NQ, bool AFFINE, class T>
__device__ __forceinline__ void ax_line_body(int blk, int nblk, int Nelements,
                                             const int32_t* __restrict__ elementList,
                                             const int32_t* __restrict__ G2L, const LineReal* __restrict__ wJ,
                                             const LineReal* __restrict__ ggeo, const LineReal* __restrict__ gllw,
                                             LineReal lambda, const T* __restrict__ q, T* __restrict__ Aq,
                                             double* __restrict__ partials, unsigned char* smem_raw) {
  using F = LineReal;
  using Sh = LineShape<NQ, T>;
  using V2 = typename std::conditional<sizeof(F) == 8, double2, float2>::type;
  constexpr int RS = Sh::RS, PLANE = Sh::PLANE, EPB = Sh::EPB, NQ2 = NQ * NQ, NP = NQ * NQ * NQ;
  constexpr int SLOT = Sh::SLOT, LANES = PackTraits<T>::R;
#define D_(a, b) c_line[SLOT + (a) * NQ + (b)]
#define W_(a) c_line[SLOT + NQ * NQ + (a)]

  __syncthreads();   // a previous call's last uses of this shared memory are done (persistent use)
  T* const sbase = reinterpret_cast<T*>(smem_raw);
  const int es = EPB == 1 || threadIdx.x >= NQ2 * EPB ? 0 : threadIdx.x / NQ2;
  const int t = threadIdx.x - es * NQ2;       // >= NQ2: no line
  T* const U = sbase + (size_t)es * 3 * Sh::FIELD;
  T* const R = U + Sh::FIELD;
  T* const S = R + Sh::FIELD;
  const int eidx = blk * EPB + es;
  const bool valid = eidx < Nelements;
  const int element = valid ? elementList[eidx] : 0;
  const size_t lbase = (size_t)element * NP;
  const F* const ge = ggeo + 6 * (size_t)element * (AFFINE ? 1 : NP);
  const F* const we = wJ + (size_t)element * (AFFINE ? 1 : NP);
  if (!AFFINE && valid && t == 0) {
    l2_prefetch(ge, 6 * NP);
    l2_prefetch(we, NP);
  }
  const int hi = t / NQ, lo = t - hi * NQ;
  const int row = hi * PLANE + lo * RS, scol = hi * PLANE + lo, tcol = hi * RS + lo;
  double pdot[LANES];
#pragma unroll
  for (int l = 0; l < LANES; ++l) pdot[l] = 0.0;
  // in place or not: a line's outputs replace values that only its thread reads
  const auto line = [&](const T* in, T* out, int stride, bool trans) {
    T r[NQ];
#pragma unroll
    for (int n = 0; n < NQ; ++n) r[n] = in[n * stride];
#pragma unroll
    for (int o = 0; o < NQ; ++o) {
      T a = pack_zero<T>();
#pragma unroll
      for (int n = 0; n < NQ; ++n) a += (trans ? D_(n, o) : D_(o, n)) * r[n];
      out[o * stride] = a;
    }
  };
  if (t < NQ2) {
    int32_t id[NQ];
#pragma unroll
    for (int k = 0; k < NQ; ++k) id[k] = valid ? __ldg(G2L + lbase + k * NQ2 + t) : -1;
#pragma unroll
    for (int k = 0; k < NQ; ++k) U[tcol + k * PLANE] = id[k] >= 0 ? q[id[k]] : pack_zero<T>();
  }
  __syncthreads();
  if (t < NQ2) {   // r-derivative on rows, s-derivative on columns (x, z)
    line(U + row, R + row, 1, false);
    line(U + scol, S + scol, RS, false);
  }
  __syncthreads();
  T acc[NQ];       // the t-part of the result column, through the r- and s-parts
#pragma unroll
  for (int n = 0; n < NQ; ++n) acc[n] = pack_zero<T>();
  if (t < NQ2) {   // t-derivative, fluxes, t-part: row k of D serves both
    F ga[6] = {0, 0, 0, 0, 0, 0}, wxy = 0;
    if (AFFINE && valid) {
#pragma unroll
      for (int c = 0; c < 6; ++c) ga[c] = __ldg(ge + c);
      wxy = __ldg(gllw + lo) * __ldg(gllw + hi);
    }
    const F* const gp = (valid ? ge : ggeo) + 6 * t;
    T u[NQ];
#pragma unroll
    for (int n = 0; n < NQ; ++n) u[n] = U[tcol + n * PLANE];
#pragma unroll 2
    for (int k = 0; k < NQ; ++k) {
      F g[6];
      if (AFFINE) {
        const F wk = wxy * W_(k);
#pragma unroll
        for (int c = 0; c < 6; ++c) g[c] = ga[c] * wk;
      } else {
        const V2* gv = reinterpret_cast<const V2*>(gp + 6 * k * NQ2);
        const V2 a0 = __ldg(gv), a1 = __ldg(gv + 1), a2 = __ldg(gv + 2);
        g[0] = a0.x; g[1] = a0.y; g[2] = a1.x; g[3] = a1.y; g[4] = a2.x; g[5] = a2.y;
      }
      F m[NQ];
      T dt = pack_zero<T>();
#pragma unroll
      for (int n = 0; n < NQ; ++n) {
        m[n] = D_(k, n);
        dt += m[n] * u[n];
      }
      T *pr = R + tcol + k * PLANE, *ps = S + tcol + k * PLANE;
      const T dr = *pr, ds = *ps;
      *pr = g[0] * dr + g[1] * ds + g[2] * dt;
      *ps = g[1] * dr + g[3] * ds + g[4] * dt;
      const T ft = g[2] * dr + g[4] * ds + g[5] * dt;
#pragma unroll
      for (int n = 0; n < NQ; ++n) acc[n] += m[n] * ft;
    }
  }
  __syncthreads();
  if (t < NQ2) {   // r-part on rows, s-part on columns, in place
    line(R + row, R + row, 1, true);
    line(S + scol, S + scol, RS, true);
  }
  __syncthreads();
  if (t < NQ2 && valid) {
    const F wa = AFFINE ? __ldg(we) * (__ldg(gllw + lo) * __ldg(gllw + hi)) : F(0);
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const T qk = U[tcol + k * PLANE];
      const F w = AFFINE ? wa * W_(k) : __ldg(we + k * NQ2 + t);
      const T out = (lambda * w) * qk + acc[k] + R[tcol + k * PLANE] + S[tcol + k * PLANE];
      Aq[lbase + k * NQ2 + t] = out;
      lane_dot(pdot, qk, out);
    }
  }
  if (partials) {
    double bs[LANES];
    fuse_block_sum_lanes<LANES>(pdot, reinterpret_cast<double*>(sbase), bs);
    if (threadIdx.x == 0)
#pragma unroll
      for (int l = 0; l < LANES; ++l) partials[(size_t)l * nblk + blk] = bs[l];
  }
#undef W_
#undef D_
}

template <int NQ, bool AFFINE, class T>
__global__ void __launch_bounds__(LineShape<NQ, T>::THREADS, (LineMinBlocks<NQ, T>::V))
ax_line_kernel(int Nelements, const int32_t* __restrict__ elementList, const int32_t* __restrict__ G2L,
               const LineReal* __restrict__ wJ, const LineReal* __restrict__ ggeo,
               const LineReal* __restrict__ gllw, LineReal lambda, const T* __restrict__ q,
               T* __restrict__ Aq, const int* __restrict__ skip, double* __restrict__ partials) {
  pdl_wait();
  pdl_release();
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ax_line_body<NQ, AFFINE, T>(blockIdx.x, gridDim.x, Nelements, elementList, G2L, wJ, ggeo, gllw, lambda, q,
                              Aq, partials, smem_raw);
}

// device address of the constant table on the current device
static LineReal* line_table_address() {
  static DeviceSymbol sym(c_line);
  return static_cast<LineReal*>(sym.address());
}

// ---- one value per node: the operator proper -------------------------------
// One element (of one field) per slot of NQ x NQ threads, EPB slots per block;
// a thread owns one line of every step and the steps pass the field through
// shared memory:
//   columns (x, y)  q gathered;  rows, columns (x, z): r-, s-derivative;
//   columns (x, y)  t-derivative, fluxes, t-part of the weak divergence;
//   rows, columns (x, z): r-part added, s-part added and written out.
// p.Ap is formed at the fluxes, where q.A_e q = sum of (dr fr + ds fs + dt ft +
// lambda w q^2) has every factor in registers.
//
// Bound by latency in its former shape (Nq^2 threads per element, two to eight
// elements in lockstep per block, qk, gt and the result line held through the
// steps: 128 registers with spills, 16 warps per SM; 0.26 of HBM at BK5 p=10).
// Short-lived lines, one element per block and a bulk prefetch of the factors
// to L2 took BK5 p=10 on 19x23x17 from 331 to 154 us.
template <int NQ>
struct LinesShape {
  static constexpr bool D = sizeof(LineReal) == 8;
  static constexpr int G2 = NQ * NQ, NP = NQ * G2;
  // strides without bank conflicts where possible (as the over-integrated kernels')
  static constexpr int RS = (NQ % 2 || NQ == 6 || NQ == 10 || NQ == 14) ? NQ : NQ + 1;
  static constexpr int PL = NQ * RS + (NQ == 6 ? 1 : NQ == 7 ? 5 : NQ == 10 ? 5 : NQ == 14 ? 9 : NQ == 16 ? 15 : 0);
  static constexpr int FIELD = NQ * PL;
  // slots, registers and unrolling from sweeps over 8,000 to 2.5 million nodes,
  // both factor storages, one and three fields, with and without p.Ap (times are
  // the geometric mean over these): FP64 Nq = 5 the flux loop as a whole 0.96 of
  // three points at a time (with three slots 0.93, but then more partials: 16^3
  // elements at p=4 would keep the alpha kernel, 100 CG iterations 2.86 against
  // 2.66 ms); Nq = 2 with p.Ap 40 registers 0.83 of 64; FP32 the flux loop as a
  // whole at Nq = 4, 11, 13 0.92-0.96; Nq = 12 outputs unrolled 0.89
  static constexpr int EPB = NQ == 2 ? 24 : NQ == 3 ? 21 : NQ == 4 ? 6 : NQ <= 6 ? 5 : NQ == 8 && D ? 2 : 1;
  static constexpr int WARPS = (G2 * EPB + 31) / 32;
  static constexpr int THREADS = WARPS * 32;   // whole warps; the last threads own no line
  // registers a thread may take: few, for more resident blocks, where spills cost less than these give
  static constexpr int regs(bool dot) {   // (the p.Ap form takes 8 more)
    if (D && NQ == 2) return dot ? 48 : 64;
    if (!D && NQ == 12) return dot ? 70 : 96;
    return (!D ? (NQ <= 7 ? 48 : 3 * NQ + 26) : NQ <= 6 ? 64 : NQ == 7 ? 80 : NQ <= 13 ? 100 : 128) + (dot ? 8 : 0);
  }
  static constexpr int minb(bool dot) {   // resident blocks to allow for
    const int n = 65536 / (THREADS * regs(dot));
    return n < 1 ? 1 : n * WARPS > 64 ? 64 / WARPS : n > 32 ? 32 : n;
  }
  static constexpr int UN = D ? (NQ == 13 ? 3 : NQ) : (NQ == 13 ? 4 : NQ == 14 ? 3 : NQ);
  static constexpr int UK = D ? (NQ == 5 ? NQ : 3) : (NQ == 4 || NQ == 11 || NQ == 13 ? NQ : 3);   // flux loop
  static constexpr int SLOT = line_slot(NQ);
  static constexpr size_t SMEM0 = sizeof(LineReal) * (size_t)3 * FIELD * EPB;
  static constexpr size_t SMEM = SMEM0 < sizeof(double) * THREADS ? sizeof(double) * THREADS : SMEM0;
};

#define LINE_D(a, b) c_line[Sh::SLOT + (a) * NQ + (b)]

template <int NQ, int UN, int STRIDE, class F, class Mat, class Store>
__device__ __forceinline__ void line_apply(const F* p, Mat mat, Store store) {
  F r[NQ];
#pragma unroll
  for (int n = 0; n < NQ; ++n) r[n] = p[n * STRIDE];
#pragma unroll UN
  for (int o = 0; o < NQ; ++o) {
    F a = 0;
#pragma unroll
    for (int n = 0; n < NQ; ++n) a += mat(o, n) * r[n];
    store(o, a);
  }
}

template <int NQ, bool AFFINE, bool DOT>
__global__ void __launch_bounds__(LinesShape<NQ>::THREADS, LinesShape<NQ>::minb(DOT))
ax_lines_kernel(int Nelements, int Nfields, const int32_t* __restrict__ elementList, const int32_t* __restrict__ G2L,
                const LineReal* __restrict__ wJ, const LineReal* __restrict__ ggeo,
                const LineReal* __restrict__ gllw, LineReal lambda, const LineReal* __restrict__ q,
                LineReal* __restrict__ Aq, const int* __restrict__ skip, double* __restrict__ partials) {
  pdl_wait();
  pdl_release();
  if (skip && *skip) return;
  using F = LineReal;
  using Sh = LinesShape<NQ>;
  using V2 = typename std::conditional<sizeof(F) == 8, double2, float2>::type;
  constexpr int G2 = Sh::G2, NP = Sh::NP, RS = Sh::RS, PL = Sh::PL, EPB = Sh::EPB, UN = Sh::UN, UK = Sh::UK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int slot = EPB == 1 || threadIdx.x >= G2 * EPB ? 0 : threadIdx.x / G2;
  const int t = threadIdx.x - slot * G2;      // >= G2: no line
  F* const U = reinterpret_cast<F*>(smem_raw) + (size_t)slot * 3 * Sh::FIELD;
  F* const R = U + Sh::FIELD;
  F* const S = R + Sh::FIELD;
  const int64_t v = (int64_t)blockIdx.x * EPB + slot;        // element-major (element, field)
  const bool valid = v < (int64_t)Nelements * Nfields;
  const int eidx = Nfields == 1 ? (int)v : (int)(v / Nfields), f = (int)(v - (int64_t)eidx * Nfields);
  const int element = valid ? elementList[eidx] : 0;
  const size_t lbase = ((size_t)element * Nfields + f) * NP;
  const F* const ge = ggeo + 6 * (size_t)element * (AFFINE ? 1 : NP);
  const F* const we = wJ + (size_t)element * (AFFINE ? 1 : NP);
  if (!AFFINE && valid && t == 0) {
    l2_prefetch(ge, 6 * NP);
    l2_prefetch(we, NP);
  }
  const int hi = t / NQ, lo = t - hi * NQ;
  const int row = hi * PL + lo * RS, scol = hi * PL + lo, tcol = hi * RS + lo;
  const auto D = [](int o, int i) { return LINE_D(o, i); };
  const auto Dt = [](int o, int i) { return LINE_D(i, o); };
  double pdot = 0.0;
  if (t < G2) {
    int32_t id[NQ];
#pragma unroll
    for (int k = 0; k < NQ; ++k) id[k] = valid ? __ldg(G2L + lbase + k * G2 + t) : -1;
#pragma unroll
    for (int k = 0; k < NQ; ++k) U[tcol + k * PL] = id[k] >= 0 ? __ldg(q + id[k]) : F(0);
  }
  __syncthreads();
  if (t < G2) {
    line_apply<NQ, UN, 1>(U + row, D, [&](int o, F x) { R[row + o] = x; });
    line_apply<NQ, UN, RS>(U + scol, D, [&](int o, F x) { S[scol + o * RS] = x; });
  }
  __syncthreads();
  if (t < G2) {   // row k of D serves the t-derivative and the t-part of the divergence
    F ga[6] = {0, 0, 0, 0, 0, 0}, wa = 0, wxy = 0;
    if (AFFINE && valid) {
#pragma unroll
      for (int c = 0; c < 6; ++c) ga[c] = __ldg(ge + c);
      wa = __ldg(we);
      wxy = __ldg(gllw + lo) * __ldg(gllw + hi);
    }
    const F* const gp = (valid ? ge : ggeo) + 6 * t;
    const F* const wp = (valid ? we : wJ) + t;
    F u[NQ], acc[NQ];
#pragma unroll
    for (int n = 0; n < NQ; ++n) {
      u[n] = U[tcol + n * PL];
      acc[n] = 0;
    }
#pragma unroll UK
    for (int k = 0; k < NQ; ++k) {
      F g[6], w;
      if (AFFINE) {
        const F wk = wxy * c_line[Sh::SLOT + NQ * NQ + k];
#pragma unroll
        for (int c = 0; c < 6; ++c) g[c] = ga[c] * wk;
        w = wa * wk;
      } else {
        const V2* gv = reinterpret_cast<const V2*>(gp + 6 * k * G2);
        const V2 a0 = __ldg(gv), a1 = __ldg(gv + 1), a2 = __ldg(gv + 2);
        g[0] = a0.x; g[1] = a0.y; g[2] = a1.x; g[3] = a1.y; g[4] = a2.x; g[5] = a2.y;
        w = __ldg(wp + k * G2);
      }
      F m[NQ], d0 = 0, d1 = 0;   // two chains: the sum is on the critical path
#pragma unroll
      for (int n = 0; n < NQ; ++n) {
        m[n] = LINE_D(k, n);
        if (n & 1) d1 += m[n] * u[n];
        else d0 += m[n] * u[n];
      }
      F *pr = R + tcol + k * PL, *ps = S + tcol + k * PL, *pu = U + tcol + k * PL;
      const F dr = *pr, ds = *ps, dt = d0 + d1, qk = *pu;
      const F fr = g[0] * dr + g[1] * ds + g[2] * dt, fs = g[1] * dr + g[3] * ds + g[4] * dt;
      const F ft = g[2] * dr + g[4] * ds + g[5] * dt, mq = lambda * w * qk;
      *pr = fr;
      *ps = fs;
      *pu = mq;
      if (DOT && valid)   // products in FP64: their range is that of the squares
          pdot += (double)dr * (double)fr + (double)ds * (double)fs + (double)dt * (double)ft + (double)mq * (double)qk;
#pragma unroll
      for (int n = 0; n < NQ; ++n) acc[n] += m[n] * ft;
    }
#pragma unroll
    for (int n = 0; n < NQ; ++n) U[tcol + n * PL] += acc[n];
  }
  __syncthreads();
  if (t < G2) line_apply<NQ, UN, 1>(R + row, Dt, [&](int o, F x) { U[row + o] += x; });
  __syncthreads();
  if (t < G2 && valid)
    line_apply<NQ, UN, RS>(S + scol, Dt,
                           [&](int o, F x) { Aq[lbase + hi * G2 + o * NQ + lo] = U[scol + o * RS] + x; });
  if (DOT) {
    const double bs = fuse_block_sum(pdot, reinterpret_cast<double*>(smem_raw));
    if (threadIdx.x == 0) partials[blockIdx.x] = bs;
  }
}
#undef LINE_D

template <int NQ>
static int launch_lines_nq(const bp_ax_desc_t& d, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                           const LineReal* wJ, const LineReal* ggeo, const LineReal* gllw, const LineReal* D,
                           LineReal lambda, const LineReal* q, LineReal* Aq, const int* skip, cudaStream_t s,
                           double* partials, int* nblocks) {
  using Sh = LinesShape<NQ>;
  if (!d.affine && (reinterpret_cast<uintptr_t>(ggeo) % (2 * sizeof(LineReal)))) return 1;   // the pencil form's
  LineReal* tab = line_table_address();
  if (!tab) return fail(BP_ERROR_CUDA, "element operator: constant table address lookup failed");
  BP_TRY(const_slot_copy(tab + Sh::SLOT, D, sizeof(LineReal) * NQ * NQ, s));
  if (d.affine)
    BP_TRY(const_slot_copy(tab + Sh::SLOT + NQ * NQ, gllw, sizeof(LineReal) * NQ, s));
  auto k = d.affine ? (partials ? ax_lines_kernel<NQ, true, true> : ax_lines_kernel<NQ, true, false>)
                    : (partials ? ax_lines_kernel<NQ, false, true> : ax_lines_kernel<NQ, false, false>);
  if (Sh::SMEM > 48 * 1024)
    BP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::SMEM));
  const dim3 grid((unsigned)(((int64_t)Nelements * d.Nfields + Sh::EPB - 1) / Sh::EPB));
  if (nblocks) *nblocks = (int)grid.x;
  BP_CUDA_TRY(launch_pdl(k, grid, dim3(Sh::THREADS), Sh::SMEM, s, Nelements, d.Nfields, elementList, G2L, wJ, ggeo,
                         gllw, lambda, q, Aq, skip, partials));
  return BP_SUCCESS;
}

template <int NQ, class T>
static int launch_line_nq(const bp_ax_desc_t& d, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                          const LineReal* wJ, const LineReal* ggeo, const LineReal* gllw, const LineReal* D,
                          LineReal lambda, const T* q, T* Aq, const int* skip, cudaStream_t s,
                          double* partials, int* nblocks) {
  using Sh = LineShape<NQ, T>;
  constexpr size_t SMEM = Sh::smem();
  if (!d.affine && (reinterpret_cast<uintptr_t>(ggeo) % (2 * sizeof(LineReal))))
    return fail(BP_ERROR_ARG, "element operator: ggeo must be aligned to two elements");
  LineReal* tab = line_table_address();
  if (!tab) return fail(BP_ERROR_CUDA, "element operator: constant table address lookup failed");
  BP_TRY(const_slot_copy(tab + Sh::SLOT, D, sizeof(LineReal) * NQ * NQ, s));
  if (d.affine)
    BP_TRY(const_slot_copy(tab + Sh::SLOT + NQ * NQ, gllw, sizeof(LineReal) * NQ, s));
  const dim3 block(Sh::THREADS);
  const dim3 grid((Nelements + Sh::EPB - 1) / Sh::EPB);
  if (nblocks) *nblocks = (int)grid.x;
  if (d.affine) {
    if (SMEM > 48 * 1024)
      BP_CUDA_TRY(cudaFuncSetAttribute(ax_line_kernel<NQ, true, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)SMEM));
    BP_CUDA_TRY(launch_pdl(ax_line_kernel<NQ, true, T>, grid, block, SMEM, s, Nelements, elementList, G2L,
                           wJ, ggeo, gllw, lambda, q, Aq, skip, partials));
  } else {
    if (SMEM > 48 * 1024)
      BP_CUDA_TRY(cudaFuncSetAttribute(ax_line_kernel<NQ, false, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)SMEM));
    BP_CUDA_TRY(launch_pdl(ax_line_kernel<NQ, false, T>, grid, block, SMEM, s, Nelements, elementList,
                           G2L, wJ, ggeo, gllw, lambda, q, Aq, skip, partials));
  }
  BP_CUDA_TRY(cudaGetLastError());
  return BP_SUCCESS;
}

int launch_ax_line_impl(const bp_ax_desc_t& d, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                        const LineReal* wJ, const LineReal* ggeo, const LineReal* gllw, const LineReal* D,
                        LineReal lambda, const LineReal* q, LineReal* Aq, const int* skip, cudaStream_t s,
                        const CgFuse* fuse, int* nblocks) {
  if (nblocks) *nblocks = 0;
  if (Nelements == 0) return BP_SUCCESS;
  double* partials = fuse ? fuse->partials : nullptr;
  switch (d.N + 1) {
#define BP_LINE_CASE(nq) \
  case nq:               \
    return launch_lines_nq<nq>(d, Nelements, elementList, G2L, wJ, ggeo, gllw, D, lambda, q, Aq, skip, s, partials, nblocks);
    BP_LINE_CASE(2) BP_LINE_CASE(3) BP_LINE_CASE(4) BP_LINE_CASE(5) BP_LINE_CASE(6) BP_LINE_CASE(7)
    BP_LINE_CASE(8) BP_LINE_CASE(9) BP_LINE_CASE(10) BP_LINE_CASE(11) BP_LINE_CASE(12) BP_LINE_CASE(13)
    BP_LINE_CASE(14) BP_LINE_CASE(15) BP_LINE_CASE(16)
#undef BP_LINE_CASE
    default:
      return fail(BP_ERROR_ARG, "element operator: degree N must be in 1..15");
  }
}

// the same operator on PK right-hand sides packed per node (one field)
template <int PK>
int launch_ax_line_pk(const bp_ax_desc_t& d, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                      const LineReal* wJ, const LineReal* ggeo, const LineReal* gllw, const LineReal* D,
                      LineReal lambda, const LineReal* q, LineReal* Aq, const int* skip, cudaStream_t s,
                      const CgFuse* fuse, int* nblocks) {
  using T = Pack<LineReal, PK>;
  if (nblocks) *nblocks = 0;
  if (d.Nfields != 1) return fail(BP_ERROR_ARG, "packed element operator: one field only");
  if (Nelements == 0) return BP_SUCCESS;
  double* partials = fuse ? fuse->partials : nullptr;
  const T* qp = reinterpret_cast<const T*>(q);
  T* ap = reinterpret_cast<T*>(Aq);
  switch (d.N + 1) {
#define BP_LINE_PK_CASE(nq) \
  case nq:                  \
    return launch_line_nq<nq, T>(d, Nelements, elementList, G2L, wJ, ggeo, gllw, D, lambda, qp, ap, skip, s, partials, nblocks);
    BP_LINE_PK_CASE(2) BP_LINE_PK_CASE(3) BP_LINE_PK_CASE(4) BP_LINE_PK_CASE(5) BP_LINE_PK_CASE(6)
    BP_LINE_PK_CASE(7) BP_LINE_PK_CASE(8) BP_LINE_PK_CASE(9) BP_LINE_PK_CASE(10) BP_LINE_PK_CASE(11)
    BP_LINE_PK_CASE(12)
#undef BP_LINE_PK_CASE
    default:
      return fail(BP_ERROR_ARG, "packed element operator: degree N must be in 1..11");
  }
}

}  // namespace
}  // namespace bp
