// Simplex (affine Tri2D and Tet3D) BP5 element operator, forcings and Jacobi
// diagonal.
//
// The reference's affine simplex operators (okl/bp5AxAffineTri2D.okl:27-89,
// okl/bp5AxAffineTet3D.okl) apply dense Np x Np reference matrices per element:
//   Aq_e = sum_ab G_ab S_ab q_e + lambda J MM q_e
// over ab = rr, rs, ss (triangles: NSM = 3) or rr, rs, rt, ss, st, tt
// (tetrahedra: NSM = 6), with per-element factors G_ab and J.  Np is not a
// tensor product, so there is no sum factorisation: a batched product of the
// four stacked matrices with the elements' gathered values (in shared memory),
// the matrices read with node-fastest layout (X[k*Np + n] is the weight of
// node k in output n: the reference's device copies o_S and o_MM), so the
// threads of a node group read consecutive words for every k.  The matrices (4*Np^2
// doubles, 41 KB at p = 7) are shared by all elements and stay in L1/L2.
// Sums over k run in increasing k, the output combines the four sums in the
// reference's order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "bp_cg_device.cuh"
#include "bp_internal.hpp"

namespace bp {
namespace {

constexpr int kTriThreads = 256;

// nodes of the degree-N triangle (dim 2) or tetrahedron (dim 3)
int simplex_np(int dim, int N) { return dim == 2 ? (N + 1) * (N + 2) / 2 : (N + 1) * (N + 2) * (N + 3) / 6; }

// node groups per block (element slots for the forcing) and threads per block
// (whole warps, at most kTriThreads + 32: tetrahedra of degree 11..15 have
// 364..816 nodes, and their threads walk the nodes of the element in strides)
static void tri_shape(int Np, int* epb, int* threads) {
  *epb = Np >= kTriThreads ? 1 : kTriThreads / Np;
  *threads = std::min((*epb * Np + 31) / 32 * 32, kTriThreads + 32);
}

// Thread (n, g) of a block computes node n of the kTriElems elements of group
// g, so every matrix entry it loads serves kTriElems elements (four FMAs per
// element).  Measured on 400x400 boxes (320,000 triangles): one element per
// thread 6.1 TFLOP/s (reference flop model) at p=7 and 36.7 ms for 100 CG
// iterations at p=5; four 7.3 TFLOP/s and 26.2 ms; eight 7.8 TFLOP/s but
// 43.4 ms (132 registers in the CG form with the p.Ap sum).
constexpr int kTriElems = 4;

// Triangles are held to three blocks per SM (72 registers instead of 82,
// a few words of spills): ncu showed two blocks (16 warps) waiting on the
// matrix loads (long scoreboard); three gave BK5 p=5 5.29 -> 6.18 and p=7
// 7.46 -> 8.14 TFLOP/s and 100 CG iterations at p=5 32.1 -> 29.4 ms (400x400,
// the same box).  Tetrahedra need their 110 registers (seven sums of four
// elements).
template <class F, int NSM, bool DOT>
__global__ void __launch_bounds__(kTriThreads + 32, NSM == 3 ? 3 : 1)
ax_simplex_kernel(int Nelements, int Np, int groups, const int32_t* __restrict__ elementList,
              const int32_t* __restrict__ G2L, const F* __restrict__ wJ, const F* __restrict__ ggeo,
              const F* __restrict__ S, const F* __restrict__ MM, F lambda, const F* __restrict__ q,
              F* __restrict__ Aq, const int* __restrict__ skip, double* __restrict__ partials) {
  pdl_wait();
  pdl_release();
  if (skip && *skip) return;
  // [groups*kTriElems][Np] values; the block sum reuses it (sized for doubles)
  extern __shared__ __align__(16) double s_raw[];
  F* const s_q = reinterpret_cast<F*>(s_raw);
  const int t = threadIdx.x;
  const int slots = groups * kTriElems;
  const int e0 = blockIdx.x * slots;
  for (int i = t; i < slots * Np; i += blockDim.x) {
    const int j = i / Np, m = i - j * Np;
    F v = 0;
    if (e0 + j < Nelements) {
      const int32_t id = G2L[(size_t)elementList[e0 + j] * Np + m];
      if (id >= 0) v = q[id];
    }
    s_q[i] = v;
  }
  __syncthreads();
  // one node per thread; with more nodes than threads (one group), the
  // threads take the element's nodes in strides of the block
  const int g = t / Np;
  double pdot = 0.0;
  for (int n = t - g * Np; g < groups && n < Np; n += blockDim.x) {
    const F* sq = s_q + (size_t)g * kTriElems * Np;
    const size_t NP2 = (size_t)Np * Np;
    F acc[NSM + 1][kTriElems];   // the S_ab sums, then the mass sum
#pragma unroll
    for (int a = 0; a <= NSM; ++a)
#pragma unroll
      for (int j = 0; j < kTriElems; ++j) acc[a][j] = 0;
    for (int k = 0; k < Np; ++k) {
      const size_t o = (size_t)k * Np + n;
      F w[NSM + 1];
#pragma unroll
      for (int a = 0; a < NSM; ++a) w[a] = __ldg(S + a * NP2 + o);
      w[NSM] = __ldg(MM + o);
#pragma unroll
      for (int j = 0; j < kTriElems; ++j) {
        const F qk = sq[j * Np + k];
#pragma unroll
        for (int a = 0; a <= NSM; ++a) acc[a][j] += w[a] * qk;
      }
    }
#pragma unroll
    for (int j = 0; j < kTriElems; ++j) {
      const int eidx = e0 + g * kTriElems + j;
      if (eidx < Nelements) {
        const int element = elementList[eidx];
        const F* gg = ggeo + NSM * (size_t)element;
        F out = gg[0] * acc[0][j];
#pragma unroll
        for (int a = 1; a < NSM; ++a) out += gg[a] * acc[a][j];
        out += wJ[element] * lambda * acc[NSM][j];
        Aq[(size_t)element * Np + n] = out;
        if (DOT) pdot += (double)sq[j * Np + n] * (double)out;
      }
    }
  }
  if (DOT) {
    const double bs = fuse_block_sum(pdot, s_raw);
    if (t == 0) partials[blockIdx.x] = bs;
  }
}

// FP64 operator on the tensor cores (mma.sync m8n8k4 f64, the FP64 tensor
// instruction; tcgen05 has no FP64 kind).  Per matrix X_c (S_ab.., MM) the
// product P_c(n, e) = sum_k X_c(n, k) q(k, e) over M = Np nodes and N = elements,
// then out = sum_c f_c(e) P_c: the reference's order, so each sum is Np terms
// long (one sum over c and k together, the factors in the streamed operand, is
// C Np terms and measured four times the rounding error).  A warp holds MT
// m-tiles of 8 nodes by NT n-tiles of 8 elements; matrix fragments come from
// global memory (node-fastest rows: 64 contiguous bytes per k, L1/L2 hits
// after the first block) a group of KU k steps ahead of their use (an element
// batch too small to fill the chip waits for L2 once per group), each serving
// NT tiles; q comes from shared memory.  Rows past Np are computed on clamped
// loads and not stored; k past Np multiplies zeros.  blockIdx.y takes every
// gridDim.y-th set of rows.  Bound by the DMMA pipe and, at Np = 35, by the
// gather ahead of it.  BK5 tetrahedra p=4 (93,600) 177 -> 122 us, p=7 (7,986)
// 147 -> 84, p=15 (6) 590 -> 100; triangles p=15 (3,200) 69 -> 37 us, against
// one thread per node on the FP64 cores.
constexpr int kMmaWarps = 4;

__device__ __forceinline__ void simplex_dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// words per element of the q tile: k padded to whole steps of 4, and 4 or 12
// mod 16 so that the 4 x 4 fragment reads of a half-warp fall in distinct banks
__host__ __device__ constexpr int simplex_kp(int Np) { return (Np + 3) / 4 * 4 + ((Np + 3) / 4 % 2 ? 0 : 4); }

template <int C, int MT, int NT, bool DOT>
__global__ void __launch_bounds__(kMmaWarps * 32)
ax_simplex_mma_kernel(int Nelements, int Np, int wm, const int32_t* __restrict__ elementList,
                      const int32_t* __restrict__ G2L, const double* __restrict__ wJ,
                      const double* __restrict__ ggeo, const double* __restrict__ S, const double* __restrict__ MM,
                      double lambda, const double* __restrict__ q, double* __restrict__ Aq,
                      const int* __restrict__ skip, double* __restrict__ partials) {
  pdl_wait();
  pdl_release();
  if (skip && *skip) return;
  extern __shared__ __align__(16) double s_raw[];
  const int KP = simplex_kp(Np), KT = (Np + 3) / 4;
  const int wn = kMmaWarps / wm;                 // warps along the elements
  const int EB = wn * NT * 8;                    // elements per block
  double* const s_q = s_raw;                     // [EB][KP]
  const int t = threadIdx.x, lane = t & 31, w = t >> 5, g = lane >> 2, t4 = lane & 3;
  const int e0 = blockIdx.x * EB;
  // gather in batches: the index loads of a batch in flight together, then its values
  constexpr int GB = 6;
  for (int i0 = t; i0 < EB * KP; i0 += GB * kMmaWarps * 32) {
    int32_t id[GB];
#pragma unroll
    for (int u = 0; u < GB; ++u) {
      const int i = i0 + u * kMmaWarps * 32, j = i / KP, m = i - j * KP;
      id[u] = i < EB * KP && m < Np && e0 + j < Nelements ? G2L[(size_t)elementList[e0 + j] * Np + m] : -1;
    }
    double v[GB];
#pragma unroll
    for (int u = 0; u < GB; ++u) v[u] = id[u] >= 0 ? q[id[u]] : 0.0;
#pragma unroll
    for (int u = 0; u < GB; ++u)
      if (i0 + u * kMmaWarps * 32 < EB * KP) s_q[i0 + u * kMmaWarps * 32] = v[u];
  }
  __syncthreads();
  const int mw = w % wm, eb = (w / wm) * NT * 8;   // this warp's row of m-sets and first element
  // the elements of this lane's accumulator columns nt*8 + 2 t4 + h (-1: none)
  int el[NT][2];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int eidx = e0 + eb + nt * 8 + 2 * t4 + h;
      el[nt][h] = eidx < Nelements ? elementList[eidx] : -1;
    }
  const size_t NP2 = (size_t)Np * Np;
  const double* const sq = s_q + (size_t)(eb + g) * KP + t4;
  double pdot = 0.0;
  for (int m0 = (blockIdx.y * wm + mw) * MT * 8; m0 < Np; m0 += gridDim.y * wm * MT * 8) {
    double tot[MT][NT][2];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) tot[mt][nt][0] = tot[mt][nt][1] = 0.0;
    int row[MT];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) row[mt] = min(m0 + mt * 8 + g, Np - 1) + t4 * Np;
    // fragments of the matrix X at the KU k steps from kt on (past the end: zeros)
    constexpr int KU = NT == 2 ? 1 : 4;
    auto load_a = [&](const double* X, int kt, double (&a)[KU][MT]) {
#pragma unroll
      for (int u = 0; u < KU; ++u)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
          a[u][mt] = (kt + u) * 4 + t4 < Np ? __ldg(X + (size_t)(kt + u) * 4 * Np + row[mt]) : 0.0;
    };
    double nxt[KU][MT];
    load_a(S, 0, nxt);
#pragma unroll 1
    for (int c = 0; c < C; ++c) {
      const double* const X = c < C - 1 ? S + c * NP2 : MM;
      const double* const Xn = c + 1 < C - 1 ? X + NP2 : MM;   // the next matrix
      double acc[MT][NT][2];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[mt][nt][0] = acc[mt][nt][1] = 0.0;
#pragma unroll(KU == 1 ? 2 : 1)
      for (int kt = 0; kt < KT; kt += KU) {
        double a[KU][MT];
#pragma unroll
        for (int u = 0; u < KU; ++u)
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) a[u][mt] = nxt[u][mt];
        const bool last = kt + KU >= KT;
        load_a(last ? Xn : X, last ? 0 : kt + KU, nxt);
#pragma unroll
        for (int u = 0; u < KU; ++u) {
          if (u > 0 && kt + u >= KT) break;
          double b[NT];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) b[nt] = sq[nt * 8 * KP + (kt + u) * 4];
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) simplex_dmma(acc[mt][nt], a[u][mt], b[nt]);
        }
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const size_t e = el[nt][h] < 0 ? 0 : el[nt][h];
          const double f = el[nt][h] < 0 ? 0.0 : c < C - 1 ? __ldg(ggeo + (C - 1) * e + c) : __ldg(wJ + e) * lambda;
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) tot[mt][nt][h] += f * acc[mt][nt][h];
        }
    }
    // accumulator of lane (g, t4): node m0 + mt*8 + g, elements nt*8 + 2 t4 + {0, 1}
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (el[nt][h] >= 0) {
          const int j = eb + nt * 8 + 2 * t4 + h;
          double* const o = Aq + (size_t)el[nt][h] * Np;
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            const int n = m0 + mt * 8 + g;
            if (n < Np) {
              o[n] = tot[mt][nt][h];
              if (DOT) pdot += s_q[(size_t)j * KP + n] * tot[mt][nt][h];
            }
          }
        }
      }
  }
  if (DOT) {
    const double bs = fuse_block_sum(pdot, s_raw);
    if (t == 0) partials[blockIdx.y * gridDim.x + blockIdx.x] = bs;
  }
}

// b_e = J_e MM f_e with f scattered through GlobalToLocal (masked nodes 0)
__global__ void __launch_bounds__(kTriThreads + 32)
tri_mass_local_kernel(int Nelements, int Np, int epb, const int32_t* __restrict__ G2L,
                      const double* __restrict__ wJ, const double* __restrict__ MM, const double* __restrict__ f,
                      double* __restrict__ bL) {
  extern __shared__ __align__(16) double s_f[];
  for (int i = threadIdx.x; i < epb * Np; i += blockDim.x) {
    const int es = i / Np, n = i - es * Np, e = blockIdx.x * epb + es;
    if (e < Nelements) {
      const int32_t id = G2L[(size_t)e * Np + n];
      s_f[i] = id >= 0 ? f[id] : 0.0;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < epb * Np; i += blockDim.x) {
    const int es = i / Np, n = i - es * Np, e = blockIdx.x * epb + es;
    if (e >= Nelements) continue;
    double acc = 0.0;
    for (int k = 0; k < Np; ++k) acc += __ldg(MM + (size_t)k * Np + n) * s_f[es * Np + k];
    bL[(size_t)e * Np + n] = wJ[e] * acc;
  }
}

// diagonal of A_e: sum_ab G_ab S_ab(n,n) + lambda J MM(n,n)
__global__ void simplex_diag_local_kernel(int Nelements, int Np, int nsm, const double* __restrict__ wJ,
                                          const double* __restrict__ ggeo, const double* __restrict__ S,
                                          const double* __restrict__ MM, double lambda, double* __restrict__ dL) {
  const size_t NP2 = (size_t)Np * Np;
  const size_t total = (size_t)Nelements * Np;
  for (size_t l = blockIdx.x * (size_t)blockDim.x + threadIdx.x; l < total; l += (size_t)blockDim.x * gridDim.x) {
    const size_t e = l / Np, n = l - e * Np;
    const size_t dn = n * Np + n;
    const double* g = ggeo + nsm * e;
    double d = g[0] * S[dn];
    for (int a = 1; a < nsm; ++a) d += g[a] * S[a * NP2 + dn];
    dL[l] = d + lambda * wJ[e] * MM[dn];
  }
}

// rhsAffineTri2D / rhsAffineTet3D (okl/rhsTri2D.okl, okl/rhsTet3D.okl):
// b_e = MM (J_e f) with f = (2 pi^2 + lambda) sin(pi x) sin(pi y) on triangles,
// (3 pi^2 + lambda) sin(pi x) sin(pi y) sin(pi z) on tetrahedra (z given)
__global__ void __launch_bounds__(kTriThreads + 32)
simplex_rhs_analytic_kernel(int Nelements, int Np, int epb, const double* __restrict__ wJ,
                            const double* __restrict__ MM, const double* __restrict__ x, const double* __restrict__ y,
                            const double* __restrict__ z, double lambda, double* __restrict__ bL) {
  extern __shared__ __align__(16) double s_f[];
  const double pi = 3.14159265358979323846;
  for (int i = threadIdx.x; i < epb * Np; i += blockDim.x) {
    const int es = i / Np, e = blockIdx.x * epb + es;
    if (e < Nelements) {
      const size_t id = (size_t)e * Np + (i - es * Np);
      const double f = z ? (3 * pi * pi + lambda) * sin(pi * x[id]) * sin(pi * y[id]) * sin(pi * z[id])
                         : (2 * pi * pi + lambda) * sin(pi * x[id]) * sin(pi * y[id]);
      s_f[i] = wJ[e] * f;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < epb * Np; i += blockDim.x) {
    const int es = i / Np, n = i - es * Np, e = blockIdx.x * epb + es;
    if (e >= Nelements) continue;
    double acc = 0.0;
    for (int m = 0; m < Np; ++m) acc += __ldg(MM + (size_t)m * Np + n) * s_f[es * Np + m];
    bL[(size_t)e * Np + n] = acc;
  }
}

}  // namespace

int launch_rhs_analytic_simplex(int dim, int N, int32_t Nelements, const double* wJ, const double* MM,
                                const double* x, const double* y, const double* z, double lambda, double* bL,
                                cudaStream_t s) {
  if (Nelements == 0) return BP_SUCCESS;
  const int Np = simplex_np(dim, N);
  int epb = 0, threads = 0;
  tri_shape(Np, &epb, &threads);
  const int grid = (Nelements + epb - 1) / epb;
  simplex_rhs_analytic_kernel<<<grid, threads, sizeof(double) * epb * Np, s>>>(Nelements, Np, epb, wJ, MM, x, y,
                                                                              dim == 3 ? z : nullptr, lambda, bL);
  BP_CUDA_TRY(cudaGetLastError());
  return BP_SUCCESS;
}

// Warps along the nodes (wm of kMmaWarps; the others along the elements),
// m-tiles and n-tiles per warp, blocks along the nodes.
struct SimplexMmaPlan {
  int mt, nt, wm, gy;
  int eb() const { return kMmaWarps / wm * nt * 8; }
  size_t smem(int Np) const { return sizeof(double) * (size_t)eb() * simplex_kp(Np); }
};

// A batch that leaves the chip idle spreads its rows over blockIdx.y, to at most
// about two blocks per SM.  Two estimates of a plan's time:
//
// rough: the rounds of row sets a warp runs, times the tile products, fragment
// loads and latency of a k step, times the waves beyond three blocks per SM.
//
// fine: a block alone on its SM takes the k steps of its rounds, each with its
// tile products, fragment loads and a latency, after the gather of its q tile in
// batches of dependent loads; the n blocks of an SM (between the average one and
// the busiest) follow one another at the pace of the more limiting of their
// residency (registers or shared memory) and of the SM's DMMA and load pipes.
// Weights in DMMA issue slots, fitted to the timings of every plan at 985
// problems, triangles p = 3..15 and tetrahedra p = 2..12, 6 to 400,000 elements,
// with and without p.Ap.
//
// The fine estimate decides where the roughly best plan splits the rows (it
// ranks splits poorly); elsewhere it has to put another plan 8% below that one.
// Over the 985 problems this takes 1.031 of the best plan's time on average, 297
// of them over 5% faster than the rough choice alone (which takes 1.11, and at
// 700-2,100 elements more than one thread per node: tetrahedra p=8, 750: 49 us
// against 44 there and 30 now; an FP64 CG iteration at p=7, 2,058: 74, 56 and 51),
// 6 over 5% slower, 1.10 at the most.  The fine estimate alone: 1.028, but 38
// slower, up to 1.39.
static SimplexMmaPlan simplex_mma_plan(int C, int Np, int32_t E, int sms, bool dot) {
  const int tiles = (Np + 7) / 8;
  const double steps1 = C * ((Np + 3) / 4);
  SimplexMmaPlan rough{1, 1, 1, 1}, fine = rough;
  double rough_cost = 1e300, rough_fine = 1e300, fine_cost = 1e300;
  for (int nt = 2; nt >= 1; --nt)
    for (int wm = 1; wm <= kMmaWarps; wm *= 2)
      for (int mt = 1; mt <= 5; ++mt) {
        SimplexMmaPlan p{mt, nt, wm, 1};
        if (p.smem(Np) > 48 * 1024 && (nt > 1 || wm < kMmaWarps)) continue;
        const int sets = (tiles + mt * wm - 1) / (mt * wm);
        const int bx = (E + p.eb() - 1) / p.eb();
        p.gy = std::max(1, std::min(sets, 2 * sms / bx));
        const int rounds = (sets + p.gy - 1) / p.gy;
        const int64_t blocks = bx * (int64_t)p.gy;
        const double per_sm = (double)blocks / sms;
        const double r = std::max(per_sm / 3, 1.0) * rounds * (mt * nt + 0.6 * mt + 0.3 * nt + 1.5);

        // registers a thread of the kernel takes (p.Ap: more with one or four tiles)
        const int regs = mt == 1 ? (nt == 1 ? (dot ? 72 : 64) : dot ? 96 : 72)
                         : mt == 2 ? 96 : mt == 3 || (mt == 4 && !dot) ? 128 : 168;
        const int resident = (int)std::min<size_t>(65536 / (regs * 32 * kMmaWarps), 227 * 1024 / (p.smem(Np) + 1024));
        const double n = 0.4 * ((blocks + sms - 1) / sms) + 0.6 * std::max(per_sm, 1.0);
        const double gathers = p.eb() * ((Np + 3) / 4 * 4) / (6.0 * 32 * kMmaWarps);
        const double steps = rounds * steps1;
        const double alone = steps * (0.8 * mt * nt + mt + 3.6 * nt + 8) + 80 * std::ceil(gathers);
        const double pipes = steps * (mt * nt + 0.2 * mt + 0.08) + 4 * gathers;
        const double f = alone + (n - 1) * std::max(alone / resident, pipes);
        if (r < rough_cost) {
          rough_cost = r;
          rough_fine = f;
          rough = p;
        }
        if (f < fine_cost) {
          fine_cost = f;
          fine = p;
        }
      }
  return fine_cost < (rough.gy > 1 ? 1.0 : 0.92) * rough_fine ? fine : rough;
}

template <int C, int MT, int NT>
static int launch_simplex_mma(const SimplexMmaPlan& p, int Np, int32_t E, const int32_t* elementList,
                              const int32_t* G2L, const double* wJ, const double* ggeo, const double* S,
                              const double* MM, double lambda, const double* q, double* Aq, const int* skip,
                              cudaStream_t s, double* partials, int* nblocks) {
  const dim3 grid((E + p.eb() - 1) / p.eb(), p.gy);
  if (nblocks) *nblocks = (int)(grid.x * grid.y);
  const size_t smem = p.smem(Np);
  auto k = partials ? ax_simplex_mma_kernel<C, MT, NT, true> : ax_simplex_mma_kernel<C, MT, NT, false>;
  if (smem > 48 * 1024) BP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  BP_CUDA_TRY(launch_pdl(k, grid, kMmaWarps * 32, smem, s, (int)E, Np, p.wm, elementList, G2L, wJ, ggeo, S, MM, lambda,
                         q, Aq, skip, partials));
  return BP_SUCCESS;
}

template <int C>
static int launch_ax_simplex_mma(int N, int32_t E, const int32_t* elementList, const int32_t* G2L, const double* wJ,
                                 const double* ggeo, const double* S, const double* MM, double lambda,
                                 const double* q, double* Aq, const int* skip, cudaStream_t s, double* partials,
                                 int* nblocks) {
  const int Np = simplex_np(C == 4 ? 2 : 3, N);
  const SimplexMmaPlan p = simplex_mma_plan(C, Np, E, sm_count(), partials != nullptr);
#define BP_SIMPLEX_MMA(MT, NT)                                                                                     \
  if (p.mt == MT && p.nt == NT)                                                                                    \
    return launch_simplex_mma<C, MT, NT>(p, Np, E, elementList, G2L, wJ, ggeo, S, MM, lambda, q, Aq, skip, s, partials, \
                                         nblocks);
#define BP_SIMPLEX_MMA_NT(MT) BP_SIMPLEX_MMA(MT, 1) BP_SIMPLEX_MMA(MT, 2)
  BP_SIMPLEX_MMA_NT(1) BP_SIMPLEX_MMA_NT(2) BP_SIMPLEX_MMA_NT(3) BP_SIMPLEX_MMA_NT(4) BP_SIMPLEX_MMA_NT(5)
#undef BP_SIMPLEX_MMA_NT
#undef BP_SIMPLEX_MMA
  return fail(BP_ERROR_ARG, "simplex operator: no tile shape");
}

template <class F, int NSM>
static int launch_ax_simplex_t(int N, int32_t Nelements, const int32_t* elementList, const int32_t* G2L, const F* wJ,
                               const F* ggeo, const F* S, const F* MM, F lambda, const F* q, F* Aq, const int* skip,
                               cudaStream_t s, double* partials, int* nblocks) {
  if (nblocks) *nblocks = 0;
  if (N < 1 || N > 15) return fail(BP_ERROR_ARG, "simplex operator: degree N must be in 1..15");
  if (Nelements == 0) return BP_SUCCESS;
  const int Np = simplex_np(NSM == 3 ? 2 : 3, N);
  // an element of less than one m-tile of nodes is mostly padding there (triangles
  // p=1: 42 us scalar against 81; p=2 and tetrahedra p=1 the same in both)
  if constexpr (sizeof(F) == 8)
    if (Np >= 8)
      return launch_ax_simplex_mma<NSM + 1>(N, Nelements, elementList, G2L, wJ, ggeo, S, MM, lambda, q, Aq, skip, s,
                                            partials, nblocks);
  int groups = 0, threads = 0;
  tri_shape(Np, &groups, &threads);
  const int slots = groups * kTriElems;
  const int grid = (Nelements + slots - 1) / slots;
  if (nblocks) *nblocks = grid;
  const size_t smem = sizeof(double) * (size_t)(slots * Np > threads ? slots * Np : threads);
  if (partials)
    BP_CUDA_TRY(launch_pdl(ax_simplex_kernel<F, NSM, true>, grid, threads, smem, s, (int)Nelements, Np, groups, elementList,
                           G2L, wJ, ggeo, S, MM, lambda, q, Aq, skip, partials));
  else
    BP_CUDA_TRY(launch_pdl(ax_simplex_kernel<F, NSM, false>, grid, threads, smem, s, (int)Nelements, Np, groups, elementList,
                           G2L, wJ, ggeo, S, MM, lambda, q, Aq, skip, (double*)nullptr));
  return BP_SUCCESS;
}

template <class F>
static int launch_ax_simplex_any(int dim, int N, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                                 const F* wJ, const F* ggeo, const F* S, const F* MM, F lambda, const F* q, F* Aq,
                                 const int* skip, cudaStream_t s, double* partials, int* nblocks) {
  if (dim == 2)
    return launch_ax_simplex_t<F, 3>(N, Nelements, elementList, G2L, wJ, ggeo, S, MM, lambda, q, Aq, skip, s,
                                     partials, nblocks);
  return launch_ax_simplex_t<F, 6>(N, Nelements, elementList, G2L, wJ, ggeo, S, MM, lambda, q, Aq, skip, s, partials,
                                   nblocks);
}

void simplex_plan(int dim, int N, int32_t Nelements, int32_t* plan) {
  const int Np = simplex_np(dim, N);
  const SimplexMmaPlan p =
      Np < 8 ? SimplexMmaPlan{0, 0, 0, 0} : simplex_mma_plan(dim == 2 ? 4 : 7, Np, Nelements, sm_count(), false);
  plan[0] = p.mt;
  plan[1] = p.nt;
  plan[2] = p.wm;
  plan[3] = p.gy;
}

int launch_ax_simplex(int dim, int N, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                      const double* wJ, const double* ggeo, const double* S, const double* MM, double lambda,
                      const double* q, double* Aq, const int* skip, cudaStream_t s, double* partials, int* nblocks) {
  return launch_ax_simplex_any<double>(dim, N, Nelements, elementList, G2L, wJ, ggeo, S, MM, lambda, q, Aq, skip, s,
                                       partials, nblocks);
}

int launch_ax_simplex(int dim, int N, int32_t Nelements, const int32_t* elementList, const int32_t* G2L,
                      const float* wJ, const float* ggeo, const float* S, const float* MM, float lambda,
                      const float* q, float* Aq, const int* skip, cudaStream_t s, double* partials, int* nblocks) {
  return launch_ax_simplex_any<float>(dim, N, Nelements, elementList, G2L, wJ, ggeo, S, MM, lambda, q, Aq, skip, s,
                                      partials, nblocks);
}

int launch_mass_local_simplex(int dim, int N, int32_t Nelements, const int32_t* G2L, const double* wJ,
                              const double* MM, const double* f, double* bL, cudaStream_t s) {
  if (Nelements == 0) return BP_SUCCESS;
  const int Np = simplex_np(dim, N);
  int epb = 0, threads = 0;
  tri_shape(Np, &epb, &threads);
  const int grid = (Nelements + epb - 1) / epb;
  tri_mass_local_kernel<<<grid, threads, sizeof(double) * epb * Np, s>>>(Nelements, Np, epb, G2L, wJ, MM, f, bL);
  BP_CUDA_TRY(cudaGetLastError());
  return BP_SUCCESS;
}

int launch_diag_local_simplex(int dim, int N, int32_t Nelements, const double* wJ, const double* ggeo,
                              const double* S, const double* MM, double lambda, double* dL, cudaStream_t s) {
  if (Nelements == 0) return BP_SUCCESS;
  const int Np = simplex_np(dim, N);
  const size_t total = (size_t)Nelements * Np;
  const int grid = (int)((total + 255) / 256 < 65535 ? (total + 255) / 256 : 65535);
  simplex_diag_local_kernel<<<grid, 256, 0, s>>>(Nelements, Np, dim == 2 ? 3 : 6, wJ, ggeo, S, MM, lambda, dL);
  BP_CUDA_TRY(cudaGetLastError());
  return BP_SUCCESS;
}

}  // namespace bp
