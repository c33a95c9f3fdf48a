// FP64 kernels of the FR residual-and-update path (plain form).
//
// One CTA owns one element ("cell") and gathers every correction that lands on
// it in ascending face-color order, so the sum order per cell is the order in
// which the reference's colored Numba kernels scatter into that cell
// (core/fr_residual/inviscid_kernel_colored.py:43-236,
// core/fr_residual/viscous_flux_kernel.py:292-520): no atomics, bit-stable
// results run to run.
//
// Template dims: S solution points, FN over-integration points, NP flux points
// per face, N1D points per direction.
#pragma once
#include "afr_device.cuh"

namespace afr {

struct StageArgs {
  const double* Ucur;   // state the residual is evaluated on (N,S,nv)
  const double* U0;     // step-start state (RK combination)
  double* Unext;        // output state (N,S,nv); may be Ucur or U0: a warp or CTA writes only the cells it read
  const double* PF;     // (N,S,16) point fields of Ucur (k_pre)
  const double* nut;    // (N,S) kinematic eddy viscosity or null
  const double* dt;     // (N,S)
  double* Rinv;         // residual-only mode outputs (N,S,nv), may be null
  double* Rvisc;
  double* norm_part;    // (N) per-cell sum of squares of dU/dt (stage 0)
  double* norm_rho_part;  // (N) per-cell sum of squares of the density column of dU/dt (stage 0)
  int nv;
  int stage;            // 0,1,2 RK stage, -1 residual only
  int inviscid_only;
  double mu;
  unsigned* status;
  int N;                     // cells
  const int32_t* slot_flags; // (n_slots) flags of the residual slots (see SlotTable)
  int cell_base, cell_end;   // cell range of this launch (one cell type)
};

__device__ __forceinline__ int cell_type(const Geom& g, int e) { return e < g.n_prism ? 0 : 1; }

// Doubles per point of a state tile staged in shared memory (n_vars <= 7 used).
// Odd, so that threads reading consecutive points' rows hit different banks.
constexpr int US = 9;

// asynchronous 8-byte copy global -> shared (both 8-byte aligned); completed
// by cp_async_wait_all before the block barrier that publishes the data
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
// 16-byte asynchronous copy global -> shared (both 16-byte aligned)
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// one m8n8k4 FP64 step: lane (g = lane/4, t = lane%4) supplies A[g][t] and
// B[t][g] and holds D[g][2t], D[g][2t+1]
__device__ __forceinline__ void dmma884(double& d0, double& d1, double a0, double b0) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a0), "d"(b0));
}


// Small FP64 products C (M x N) = A (M x K) * B (K x N) on the FP64 tensor
// path: mma.sync m8n8k4 .f64, one 8 x 8 output tile per warp at a time, K in
// steps of 4.  A is read from a fragment-major image (layout in Ops): one
// contiguous 256-byte load per warp and k-step, the image's zeros standing for
// the rows and columns outside the operator; b(k, n) fetches B (padding reads
// as zero) and c(m, n, value) stores results; block-wide work split by warp,
// no barrier inside.  The sum order over k is the unit's, so results can
// differ from a sequential FP64 sum in the last bits.
template <class FB, class FC>
__device__ __forceinline__ void dmma_product_f(int M, int N, int K, const double* __restrict__ Af, FB b, FC c) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nw = blockDim.x >> 5;
  const int mt = (M + 7) >> 3, nt = (N + 7) >> 3, KS = (K + 3) >> 2;
  for (int tile = threadIdx.x >> 5; tile < mt * nt; tile += nw) {
    const int mi = tile / nt, m = mi * 8 + g, n0 = (tile % nt) * 8;
    const double* ap = Af + (size_t)mi * KS * 32 + lane;
    double c0 = 0.0, c1 = 0.0;
    for (int ks = 0; ks < KS; ++ks) {
      const int k = ks * 4 + t;
      const double a0 = __ldg(ap + ks * 32);
      const double b0 = (k < K && n0 + g < N) ? b(k, n0 + g) : 0.0;
      dmma884(c0, c1, a0, b0);
    }
    const int n = n0 + 2 * t;
    if (m < M) {
      if (n < N) c(m, n, c0);
      if (n + 1 < N) c(m, n + 1, c1);
    }
  }
}

// dmma_product_f with each warp computing all column tiles of a row tile
// (at most NT of them): the A fragment is loaded once per k-step and the NT
// accumulations are independent, so their tensor-core latencies overlap.  Per
// element the k-steps accumulate in the same order as dmma_product_f.  Pays
// when the row tiles keep every warp busy (measured: slower than
// dmma_product_f for the 27-row filter and SST divergence with 4 row tiles).
template <int NT, class FB, class FC>
__device__ __forceinline__ void dmma_product_rb(int M, int N, int K, const double* __restrict__ Af, FB b, FC c) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nw = blockDim.x >> 5;
  const int mt = (M + 7) >> 3, KS = (K + 3) >> 2;
  for (int mi = threadIdx.x >> 5; mi < mt; mi += nw) {
    const double* ap = Af + (size_t)mi * KS * 32 + lane;
    double acc[NT][2];
#pragma unroll
    for (int ni = 0; ni < NT; ++ni) acc[ni][0] = acc[ni][1] = 0.0;
    for (int ks = 0; ks < KS; ++ks) {
      const int k = ks * 4 + t;
      const double a0 = __ldg(ap + ks * 32);
#pragma unroll
      for (int ni = 0; ni < NT; ++ni) {
        const int n = ni * 8 + g;
        const double b0 = (k < K && n < N) ? b(k, n) : 0.0;
        dmma884(acc[ni][0], acc[ni][1], a0, b0);
      }
    }
    const int m = mi * 8 + g;
    if (m < M) {
#pragma unroll
      for (int ni = 0; ni < NT; ++ni) {
        const int n = ni * 8 + 2 * t;
        if (n < N) c(m, n, acc[ni][0]);
        if (n + 1 < N) c(m, n + 1, acc[ni][1]);
      }
    }
  }
}

// Median-based outlier zeroing (core/fr_operators/troubled_cell.py:346-408):
// per cell and variable, |R| > 1e4 * max(median |R|, 1e-9 mean|U|, 1e-300)
// is set to zero.  A column has nothing to zero when that threshold is at
// least max |R|.  Two lower bounds of the median prove that without ranking:
// the minimum, and p = max|R| * 1e-4 (raised until 1e4 * p >= max|R|) when at
// least as many elements as lie at or above the median's rank are >= p.
// Such columns (no NaN) skip the O(S^2) rank pass; the others take it, so the
// result is the same element for element.
constexpr int OUT_WORK = 25;  // [0,5) median or bound, [5,10) mean|U|, [10,20) middle pair, [20,25) rank flag

// per column v of one block: mean |U| (rows Ur, stride ldU), the bound and the rank flag
template <int S>
__device__ __forceinline__ void outlier_column(const double* R, const double* Ur, int ldU, int v, double* w) {
  constexpr int NEED = S - ((S & 1) ? S / 2 : S / 2 - 1);  // elements at or above the (lower) middle rank
  double acc = 0.0, lo = INFINITY, hi = 0.0;
  bool nan = false;
  for (int s = 0; s < S; ++s) {
    acc += fabs(Ur[s * ldU + v]);
    const double x = fabs(R[s * 5 + v]);
    lo = fmin(lo, x);
    hi = fmax(hi, x);
    nan = nan || isnan(x);
  }
  w[5 + v] = acc / S;
  const double fl = 1e-9 * w[5 + v];
  bool skip = !nan && hi <= 1e4 * fmax(fmax(lo, fl), 1e-300);
  double bound = lo;
  if (!nan && !skip) {
    double p = hi * 1e-4;
    // next double up (p is finite and >= 0 here: its bit pattern plus one)
    for (int it = 0; it < 4 && 1e4 * p < hi; ++it) p = __longlong_as_double(__double_as_longlong(p) + 1);
    if (1e4 * p >= hi) {
      int cnt = 0;
      for (int s = 0; s < S; ++s) cnt += fabs(R[s * 5 + v]) >= p;
      if (cnt >= NEED) {
        skip = true;
        bound = p;
      }
    }
  }
  w[v] = bound;
  w[20 + v] = skip ? 0.0 : 1.0;
}

// stable rank of |R[s,v]| in its column; the middle one(s) into w
template <int S>
__device__ __forceinline__ void outlier_rank(const double* R, int s, int v, double* w) {
  const double x = fabs(R[s * 5 + v]);
  int rank = 0;
  for (int j = 0; j < S; ++j) {
    const double y = fabs(R[j * 5 + v]);
    rank += (y < x) || (y == x && j < s);
  }
  if (S & 1) {
    if (rank == S / 2) w[v] = x;
  } else {
    if (rank == S / 2 - 1) w[10 + v] = x;
    if (rank == S / 2) w[15 + v] = x;
  }
}

__device__ __forceinline__ void outlier_zero(double* R, int r, int v, const double* w, bool odd) {
  const double med = odd ? w[v] : 0.5 * (w[10 + v] + w[15 + v]);
  const double ref = fmax(fmax(med, 1e-9 * w[5 + v]), 1e-300);
  if (fabs(R[r]) > 1e4 * ref) R[r] = 0.0;
}

// nb contiguous (S,5) blocks R + b*S*5 in shared memory, reference rows
// Uref + b*S*ldU (first 5 columns), all blocks in one pass per phase.  work >= OUT_WORK doubles per block.
template <int S>
__device__ void suppress_outliers_blocks(double* R, const double* Uref, int ldU, int nb, double* work) {
  int flagged = 0;
  for (int t = threadIdx.x; t < nb * 5; t += blockDim.x) {
    const int b = t / 5, v = t % 5;
    outlier_column<S>(R + b * S * 5, Uref + b * S * ldU, ldU, v, work + b * OUT_WORK);
    flagged |= work[b * OUT_WORK + 20 + v] != 0.0;
  }
  if (!__syncthreads_or(flagged)) return;  // no column takes the rank pass: nothing is zeroed
  for (int t = threadIdx.x; t < nb * S * 5; t += blockDim.x) {
    const int b = t / (S * 5), r = t % (S * 5), s = r / 5, v = r % 5;
    double* w = work + b * OUT_WORK;
    if (w[20 + v] != 0.0) outlier_rank<S>(R + b * S * 5, s, v, w);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nb * S * 5; t += blockDim.x) {
    const int b = t / (S * 5), r = t % (S * 5), v = r % 5;
    const double* w = work + b * OUT_WORK;
    if (w[20 + v] != 0.0) outlier_zero(R + b * S * 5, r, v, w, S & 1);
  }
  __syncthreads();
}

// The same for the inviscid and viscous residuals of nc cells at once: block
// b < nc is sRi of cell b, block nc + b is sRv of cell b; cell rows of the
// reference field at sU + b*S*US.  work >= OUT_WORK doubles per block.
template <int S>
__device__ void suppress_outliers_cells(double* sRi, double* sRv, const double* sU, int nc, bool visc, double* work) {
  const int nb = nc * (visc ? 2 : 1);
  int flagged = 0;
  for (int t = threadIdx.x; t < nb * 5; t += blockDim.x) {
    const int bb = t / 5, v = t % 5;
    const double* R = bb < nc ? sRi + bb * S * 5 : sRv + (bb - nc) * S * 5;
    outlier_column<S>(R, sU + (bb % nc) * S * US, US, v, work + bb * OUT_WORK);
    flagged |= work[bb * OUT_WORK + 20 + v] != 0.0;
  }
  if (!__syncthreads_or(flagged)) return;  // no column takes the rank pass: nothing is zeroed
  for (int t = threadIdx.x; t < nb * S * 5; t += blockDim.x) {
    const int bb = t / (S * 5), r = t % (S * 5), s = r / 5, v = r % 5;
    double* w = work + bb * OUT_WORK;
    if (w[20 + v] != 0.0) outlier_rank<S>(bb < nc ? sRi + bb * S * 5 : sRv + (bb - nc) * S * 5, s, v, w);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nb * S * 5; t += blockDim.x) {
    const int bb = t / (S * 5), r = t % (S * 5), v = r % 5;
    const double* w = work + bb * OUT_WORK;
    if (w[20 + v] != 0.0) outlier_zero(bb < nc ? sRi + bb * S * 5 : sRv + (bb - nc) * S * 5, r, v, w, S & 1);
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// per-point pre-pass: PF (N,S,16) = primitive q(5) (no pressure floor,
// core/fr_residual/inviscid.py:38-47), symmetric velocity gradient (6: the
// viscous flux holds no other combination) and grad T (3)
// (core/fr_operators/gradients.py:23-64 as used by
// core/fr_residual/viscous_flux.py:161-166), mu_t = max(rho,1e-10) * nu_t (1),
// one unused (128-byte rows)
// ---------------------------------------------------------------------------
constexpr int PFW = 16;
constexpr int PFS = 17;  // row stride in shared memory (odd: consecutive rows on distinct banks)

template <int S>
struct PreTile {
  static constexpr int CPB = S <= 8 ? 16 : (S <= 27 ? 4 : 2);  // cells per CTA
};

// CPB cells per CTA; cells [cell_base, cell_end) share one cell type.  The
// reference-space gradients are one FP64 tensor-core product (rows s*3+m of
// D3g, columns (cell, field)); the tile's PF rows are assembled in shared
// memory and stored as one contiguous block.
template <int S>
__global__ void __launch_bounds__(128) k_pre(Geom g, Ops ops, const double* __restrict__ U, int nv,
                                             const double* __restrict__ nut, int want_grads,
                                             double* __restrict__ PF, int cell_base, int cell_end) {
  constexpr int CPB = PreTile<S>::CPB;
  __shared__ double sPF[CPB * S * PFS];
  __shared__ double f[CPB * S * 4];
  __shared__ double gc[CPB * S * 3 * 4];
  const int e0 = cell_base + blockIdx.x * CPB;
  const int nc = min(CPB, cell_end - e0);
  const int ct = cell_type(g, e0);
  for (int t = threadIdx.x; t < nc * S; t += blockDim.x) {
    const size_t p = (size_t)e0 * S + t;
    double q[5];
    const double* u = U + p * nv;
    cons_to_prim(u, q);
    double* o = sPF + t * PFS;
    for (int v = 0; v < 5; ++v) o[v] = q[v];
    o[15] = 0.0;
    o[14] = nut ? fmax(u[0], 1e-10) * nut[p] : 0.0;
    f[t * 4 + 0] = q[1];
    f[t * 4 + 1] = q[2];
    f[t * 4 + 2] = q[3];
    f[t * 4 + 3] = q[4] / (fmax(q[0], 1e-10) * R_AIR);
  }
  __syncthreads();
  if (want_grads) {
    dmma_product_rb<(4 * CPB + 7) / 8>(
        3 * S, 4 * nc, S, ops.fD3g[ct], [&](int j, int col) { return f[((col >> 2) * S + j) * 4 + (col & 3)]; },
        [&](int r, int col, double x) { gc[((col >> 2) * S * 3 + r) * 4 + (col & 3)] = x; });
    __syncthreads();
    for (int t = threadIdx.x; t < nc * S; t += blockDim.x) {
      double inv[9];
      if (e0 >= g.inv0) {
        const double* ip = g.inv + ((size_t)(e0 - g.inv0) * S + t) * 9;
        for (int k = 0; k < 9; ++k) inv[k] = __ldg(ip + k);
      } else {  // adjugate planes of a structured prism
        const double* ap = g.adj + (size_t)(e0 + t / S) * 9 * S + t % S;
        const double rd = 1.0 / __ldg(g.det + (size_t)e0 * S + t);
        for (int k = 0; k < 9; ++k) inv[k] = __ldg(ap + k * S) * rd;
      }
      double gr[4][3];  // rows u, v, w, T
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int n = 0; n < 3; ++n) {
          double acc = 0.0;
          for (int m = 0; m < 3; ++m) acc += gc[(t * 3 + m) * 4 + q] * inv[m * 3 + n];
          gr[q][n] = acc;
        }
      double* o = sPF + t * PFS + 5;
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        o[n] = gr[n][n];
        o[6 + n] = gr[3][n];
      }
      o[3] = 0.5 * (gr[0][1] + gr[1][0]);
      o[4] = 0.5 * (gr[0][2] + gr[2][0]);
      o[5] = 0.5 * (gr[1][2] + gr[2][1]);
    }
  } else {
    for (int t = threadIdx.x; t < nc * S * 9; t += blockDim.x) sPF[(t / 9) * PFS + 5 + t % 9] = 0.0;
  }
  __syncthreads();
  double* out = PF + (size_t)e0 * S * PFW;
  for (int t = threadIdx.x; t < nc * S * PFW; t += blockDim.x) out[t] = sPF[(t / PFW) * PFS + t % PFW];
}

// ---------------------------------------------------------------------------
// face kernel: one thread per (slot, flux point).  A slot is one side of one
// face record whose own extrapolation + correction lifting lands on a cell
// (core/fr_residual/inviscid_kernel_colored.py:86-157 owner side, :159-236
// neighbour side; core/fr_residual/viscous_flux_kernel.py:335-520).  Writes
// the inviscid and viscous flux jumps J (n_slots, 9, NP).
// Slot flags: bit0 neighbour side, bit1 boundary face, bits2-3 axis, bit4 side>0.
// ---------------------------------------------------------------------------
struct SlotTable {
  int32_t n;                // number of slots
  const int32_t* flags;     // (n)
  // mixed form
  const int32_t* face;      // (n)
  const int32_t* cell;      // (n) cell the slot lifts into
  const int32_t* c0;        // (n) first interpolation source cell, -1 if none
  const int32_t* c1;        // (n) second source cell, -1 if none
  const int32_t* i1;        // (n) row of the compact second-source table
  // plain form: (n, 2) what a slot's face points need: source cells and matrix
  // rows (c0, m0, c1, m1), then face, flags, cell, row of tnormal and bc_group
  int4* rec;
};



// one warp's m8n8k4 FP64 product C (M x N) = A (M x K) * B (K x N) with
// every tile's accumulators held in registers (MT row tiles, NT column
// tiles): each k-step loads the A fragments of all row tiles and the B
// fragments of all column tiles, so the operand loads of the whole product
// are independent of one another and of the products.  a(m, k), b(k, n)
// fetch operands (padding reads as zero), c(m, n, value) stores results.
template <int MT, int NT, int K, class FA, class FB, class FC>
__device__ __forceinline__ void dmma_warp_rb(int M, int N, FA a, FB b, FC c) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double acc[MT][NT][2];
#pragma unroll
  for (int mi = 0; mi < MT; ++mi)
#pragma unroll
    for (int ni = 0; ni < NT; ++ni) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
#pragma unroll
  for (int k0 = 0; k0 < K; k0 += 4) {
    const int k = k0 + t;
    double av[MT], bv[NT];
#pragma unroll
    for (int mi = 0; mi < MT; ++mi) {
      const int m = mi * 8 + g;
      av[mi] = (m < M && k < K) ? a(m, k) : 0.0;
    }
#pragma unroll
    for (int ni = 0; ni < NT; ++ni) {
      const int n = ni * 8 + g;
      bv[ni] = (n < N && k < K) ? b(k, n) : 0.0;
    }
#pragma unroll
    for (int mi = 0; mi < MT; ++mi)
#pragma unroll
      for (int ni = 0; ni < NT; ++ni) dmma884(acc[mi][ni][0], acc[mi][ni][1], av[mi], bv[ni]);
  }
#pragma unroll
  for (int mi = 0; mi < MT; ++mi)
#pragma unroll
    for (int ni = 0; ni < NT; ++ni) {
      const int m = mi * 8 + g, n = ni * 8 + 2 * t;
      if (m < M) {
        if (n < N) c(m, n, acc[mi][ni][0]);
        if (n + 1 < N) c(m, n + 1, acc[mi][ni][1]);
      }
    }
}

// dmma_warp_rb with A read from a fragment-major image (layout in Ops) of an
// operator with at most MT * 8 rows and K columns
template <int MT, int NT, int K, class FB, class FC>
__device__ __forceinline__ void dmma_warp_rb_f(int M, int N, const double* __restrict__ Af, FB b, FC c) {
  constexpr int KS = (K + 3) / 4;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double acc[MT][NT][2];
#pragma unroll
  for (int mi = 0; mi < MT; ++mi)
#pragma unroll
    for (int ni = 0; ni < NT; ++ni) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
#pragma unroll
  for (int ks = 0; ks < KS; ++ks) {
    const int k = ks * 4 + t;
    double av[MT], bv[NT];
#pragma unroll
    for (int mi = 0; mi < MT; ++mi) av[mi] = __ldg(Af + (mi * KS + ks) * 32 + lane);
#pragma unroll
    for (int ni = 0; ni < NT; ++ni) {
      const int n = ni * 8 + g;
      bv[ni] = (n < N && k < K) ? b(k, n) : 0.0;
    }
#pragma unroll
    for (int mi = 0; mi < MT; ++mi)
#pragma unroll
      for (int ni = 0; ni < NT; ++ni) dmma884(acc[mi][ni][0], acc[mi][ni][1], av[mi], bv[ni]);
  }
#pragma unroll
  for (int mi = 0; mi < MT; ++mi)
#pragma unroll
    for (int ni = 0; ni < NT; ++ni) {
      const int m = mi * 8 + g, n = ni * 8 + 2 * t;
      if (m < M) {
        if (n < N) c(m, n, acc[mi][ni][0]);
        if (n + 1 < N) c(m, n + 1, acc[mi][ni][1]);
      }
    }
}

// the jumps of one slot point from its own side and the other side's fields; f:
// the slot's row of tnormal and bc_group (read by boundary and fallback slots)
template <int S, int NP, bool VISC, int NF>
__device__ __forceinline__ void face_jump(const Geom& g, const Faces& fc, const Bc& bc, int sl, int i, int e, int f,
                                          bool is_owner, bool bnd, double side, const double (&ow)[NF],
                                          double (&ot)[NF], const double4* __restrict__ arow, double mu,
                                          double* __restrict__ J) {
  const double* tn = fc.tnormal + ((size_t)f * NP + i) * 3;
  if (bnd) {
    double n[3], gq[5];
    for (int d = 0; d < 3; ++d) n[d] = tn[d];
    ghost_state(bc, fc.bc_group[f], ow, n, gq);
#pragma unroll
    for (int v = 0; v < 5; ++v) ot[v] = gq[v];
#pragma unroll
    for (int k = 5; k < NF; ++k) ot[k] = ow[k];
  }
  // pointwise fluxes; the own adjugate row and its norm are geometry, formed at
  // create (a negative norm marks the alignment fallback)
  const double4 ar = arow[(size_t)sl * NP + i];
  const double a0 = ar.x, a1 = ar.y, a2 = ar.z;
  const double mag = fabs(ar.w);
  double dir[3] = {a0 / mag * side, a1 / mag * side, a2 / mag * side};
  if (ar.w < 0.0) {
    const double sg = is_owner ? 1.0 : -1.0;
    dir[0] = sg * tn[0];
    dir[1] = sg * tn[1];
    dir[2] = sg * tn[2];
  }
  double Fc[5], Fp[3][5];
  ausm_up(ow, ot, dir, Fc);
  euler_flux(ow, Fp);
  double* Jo = J + (size_t)sl * 9 * NP + i;
  for (int v = 0; v < 5; ++v) Jo[v * NP] = Fc[v] * mag * side - (a0 * Fp[0][v] + a1 * Fp[1][v] + a2 * Fp[2][v]);
  if constexpr (VISC) {
    double av[NF];  // the common flux: both sides' averages
#pragma unroll
    for (int k = 1; k < NF; ++k) av[k] = 0.5 * (ow[k] + ot[k]);
    double Gc[3][4], Go[3][4];
    viscous_flux_sym(av + 1, av + 5, av + 11, mu, av[14], Gc);
    viscous_flux_sym(ow + 1, ow + 5, ow + 11, mu, ow[14], Go);
    double jv[4];
    for (int v = 0; v < 4; ++v)
      jv[v] = (a0 * Gc[0][v] + a1 * Gc[1][v] + a2 * Gc[2][v]) - (a0 * Go[0][v] + a1 * Go[1][v] + a2 * Go[2][v]);
    if (bnd) {
      // interior-penalty term on boundary faces (core/fr_operators/flux_kernels.py:140-200);
      // cell volume scale = mean of det over the cell's points (viscous_flux_kernel.py:344-347)
      double vol_o = 0.0;
      for (int s = 0; s < S; ++s) vol_o += g.det[(size_t)e * S + s];
      vol_o /= S;
      double h = pow(vol_o, 1.0 / 3.0);
      if (h < 1e-300) h = 1e-300;
      const double eta = C_IP * (mu + ow[14]) / h;
      const double scale = eta * sqrt(a0 * a0 + a1 * a1 + a2 * a2) * side;
      for (int v = 0; v < 3; ++v) jv[v] += -scale * (ow[1 + v] - ot[1 + v]);
    }
    for (int v = 0; v < 4; ++v) Jo[(5 + v) * NP] = jv[v];
  }
}

// Face kernels.  A slot is one side of one face record whose correction lifts
// into a cell; lane = (slot, flux point) forms the own side by extrapolation, the
// other side with the record's matrix (the second source added to the first),
// the ghost state, AUSM+up with the alignment fallback and the BR1 common flux
// with the boundary penalty
// (core/fr_residual/inviscid_kernel_colored.py:86-236,
// core/fr_residual/viscous_flux_kernel.py:335-520), and writes the jumps
// J (n_slots, 9, NP: inviscid 5, viscous momentum and energy 4).
// A weight of zero contributes nothing while the state is finite (the reference
// skips zero weights, inviscid_kernel_colored.py:117-121; a non-finite state
// makes the step non-finite either way).
//
// k_face (orders 2, 3): a warp per group of SPW = 32 / NP slots; both sides'
// products are register-blocked on the FP64 tensor path, their operands
// gathered straight from global memory.  ROWS: the own side from the nonzeros of
// its extrapolation row instead (Ops::ex_*), by the lane itself.  That pays only
// without viscosity, where the product's five columns leave three of a tile's
// eight idle, and where the rows are sparse: step of 17,280 P2 prisms (5.1
// nonzeros of 27 on average) 728 us with, 746 without; residual of 10,368 P2 tets
// (15.9) 245 and 224.  With viscosity the rows cost more on every mesh: 17,280 P2
// prisms 1,144 and 1,090 us per step, 1,332 and 1,275 with SST; both residuals of
// 10,368 P2 tets 593 and 511, of 10,080 P3 prisms 1,386 and 1,182, of 6,000 P3
// tets 910 and 629.
// k_face_staged (order 1, 8 x 4 matrices that fill a quarter of the tensor
// tiles): a warp per cell, the own side from the row's nonzeros; the rows of the cell and of its slots' source cells
// arrive in shared memory by 16-byte asynchronous copies, all in flight at
// once, and the products are plain multiply-adds.  24,576 P1 tets, inviscid: 83 us on
// the tensor path, 64 us staged; 17,280 P2 prisms, viscous: 268 us staged.
// Slot flags: bit0 neighbour side, bit1 boundary face, bits2-3 axis, bit4 side>0.
constexpr int FACE_WARPS = 4;
constexpr int FW_F = 15;  // fields per face point and side

template <int S, int NP, bool VISC>
struct FaceSmem {
  static constexpr int SPW = 32 / NP;        // slots in flight per warp
  static constexpr int RQ = VISC ? 8 : 3;    // 16-byte pieces of a point row (without viscosity only q)
  static constexpr int RW = VISC ? 18 : 6;   // row stride: 16-byte accesses to eight rows hit distinct banks
  static constexpr int warp = (1 + SPW) * S * RW;  // doubles: the cell's rows, then each slot's source rows
  static constexpr int total = FACE_WARPS * warp * 8;
};

template <int S, int NP, bool VISC>
__global__ void __launch_bounds__(32 * FACE_WARPS, VISC ? 3 : 4)
    k_face_staged(Geom g, Ops ops, Faces fc, Bc bc, SlotTable st, const double* __restrict__ PF,
                  const double4* __restrict__ arow, double mu, double* __restrict__ J) {
  using L = FaceSmem<S, NP, VISC>;
  constexpr int SPW = L::SPW, RQ = L::RQ, RW = L::RW, NF = VISC ? FW_F : 5;
  extern __shared__ __align__(16) double smf64[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e = blockIdx.x * FACE_WARPS + warp;
  if (e >= g.N) return;  // whole warps; warp-level synchronisation only
  double* own = smf64 + warp * L::warp;
  double* nb = own + S * RW;
  auto stage = [&](double* dst, int c) {
    const double* pf = PF + (size_t)c * S * PFW;
    for (int t = lane; t < S * RQ; t += 32) {
      const int r = t / RQ, q = t - r * RQ;
      cp_async16(dst + r * RW + 2 * q, pf + r * PFW + 2 * q);
    }
  };
  stage(own, e);
  const int k0 = __ldg(fc.slot_ptr + e), k1 = __ldg(fc.slot_ptr + e + 1);
  const int ct = cell_type(g, e);
  const int j = lane / NP, i = lane % NP;
  for (int kb = k0; kb < k1; kb += SPW) {
    const int nsl = min(SPW, k1 - kb);
    const bool live = j < nsl;  // lanes past the last slot follow it
    const int sl = kb + (live ? j : 0);
    const int4 r0 = __ldg(st.rec + 2 * (size_t)sl), r1 = __ldg(st.rec + 2 * (size_t)sl + 1);
    for (int q = 0; q < nsl; ++q) {
      const int c = __shfl_sync(0xffffffffu, r0.x, q * NP);
      if (c >= 0) stage(nb + q * S * RW, c);
    }
    cp_async_wait_all();
    __syncwarp();
    const int f = r1.w, fl = r1.y;
    const bool is_owner = (fl & 1) == 0;
    const bool bnd = (fl & 2) != 0;
    const double side = (fl & 16) ? 1.0 : -1.0;
    double ow[NF], ot[NF];
#pragma unroll
    for (int k = 0; k < NF; ++k) ow[k] = ot[k] = 0.0;
    auto add = [&](double (&o)[NF], double w, const double* row) {
      const double2* x = reinterpret_cast<const double2*>(row);
#pragma unroll
      for (int q = 0; q < (NF + 1) / 2; ++q) {
        const double2 v = x[q];
        o[2 * q] += w * v.x;
        if (2 * q + 1 < NF) o[2 * q + 1] += w * v.y;
      }
    };
    {
      const int gr = (ct * 3 + ((fl >> 2) & 3)) * 2 + ((fl & 16) ? 1 : 0);
      const int n = __ldg(ops.ex_n + gr * NP + i);
      const size_t at = (size_t)gr * S * NP + i;
#pragma unroll 3
      for (int k = 0; k < n; ++k)
        add(ow, __ldg(ops.ex_w + at + (size_t)k * NP), own + __ldg(ops.ex_i + at + (size_t)k * NP) * RW);
    }
    const double* nr = nb + (live ? j : 0) * S * RW;
    if (r0.x >= 0) {
      const double* M = (is_owner ? fc.nb_m0 : fc.ow_m0) + (size_t)r0.y * S * NP + i;
#pragma unroll 8
      for (int s = 0; s < S; ++s) add(ot, __ldg(M + s * NP), nr + s * RW);
    }
    if (__any_sync(0xffffffffu, r0.z >= 0)) {
      // second sources, into the same rows
      __syncwarp();
      for (int q = 0; q < nsl; ++q) {
        const int c = __shfl_sync(0xffffffffu, r0.z, q * NP);
        if (c >= 0) stage(nb + q * S * RW, c);
      }
      cp_async_wait_all();
      __syncwarp();
      if (r0.z >= 0) {
        const double* M = (is_owner ? fc.nb_m1 : fc.ow_m1) + (size_t)r0.w * S * NP + i;
#pragma unroll 8
        for (int s = 0; s < S; ++s) add(ot, __ldg(M + s * NP), nr + s * RW);
      }
    }
    __syncwarp();  // the rows are consumed
    if (live && lane < SPW * NP)
      face_jump<S, NP, VISC>(g, fc, bc, sl, i, e, f, is_owner, bnd, side, ow, ot, arow, mu, J);
  }
}

template <int S, int NP, bool VISC, bool ROWS>
__global__ void __launch_bounds__(32 * FACE_WARPS, 4)
    k_face(Geom g, Ops ops, Faces fc, Bc bc, SlotTable st, const double* __restrict__ PF,
           const double4* __restrict__ arow, double mu, double* __restrict__ J) {
  constexpr int SPW = 32 / NP, MT = (NP + 7) / 8, NF = VISC ? FW_F : 5, NT = (NF + 7) / 8;
  __shared__ double sOt[FACE_WARPS][SPW * NP * NF];
  __shared__ double sOw[ROWS ? 1 : FACE_WARPS][ROWS ? 1 : SPW * NP * NF];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sl0 = (blockIdx.x * FACE_WARPS + warp) * SPW;
  if (sl0 >= st.n) return;  // whole warps; warp-level synchronisation only
  const int nsl = min(SPW, st.n - sl0);
  double* ot_s = sOt[warp];
  for (int j = 0; j < nsl; ++j) {
    const int4 r0 = __ldg(st.rec + 2 * (size_t)(sl0 + j)), r1 = __ldg(st.rec + 2 * (size_t)(sl0 + j) + 1);
    const bool is_owner = (r1.y & 1) == 0;
    double* ot = ot_s + j * NP * NF;
    if constexpr (!ROWS) {
      const int gr = (cell_type(g, r1.z) * 3 + ((r1.y >> 2) & 3)) * 2 + ((r1.y & 16) ? 1 : 0);
      const double* pf = PF + (size_t)r1.z * S * PFW;
      double* ow = sOw[warp] + j * NP * NF;
      dmma_warp_rb_f<MT, NT, S>(
          NP, NF, ops.fextrap + (size_t)gr * (MT * ((S + 3) / 4) * 32),
          [&](int s, int n) { return __ldg(pf + s * PFW + n); }, [&](int i, int n, double x) { ow[i * NF + n] = x; });
    }
    for (int src = 0; src < 2; ++src) {
      const int c = src == 0 ? r0.x : r0.z;
      if (c < 0) {
        if (src == 0)
          for (int t = lane; t < NP * NF; t += 32) ot[t] = 0.0;
        continue;
      }
      const double* M = (src == 0 ? (is_owner ? fc.nb_m0 : fc.ow_m0) : (is_owner ? fc.nb_m1 : fc.ow_m1)) +
                        (size_t)(src == 0 ? r0.y : r0.w) * S * NP;
      const double* pc = PF + (size_t)c * S * PFW;
      __syncwarp();
      dmma_warp_rb<MT, NT, S>(
          NP, NF, [&](int i, int s) { return __ldg(M + s * NP + i); },
          [&](int s, int n) { return __ldg(pc + s * PFW + n); },
          [&](int i, int n, double x) {
            if (src == 0) ot[i * NF + n] = x;
            else ot[i * NF + n] += x;
          });
    }
  }
  __syncwarp();
  const int j = lane / NP, i = lane % NP;
  if (j >= nsl || lane >= SPW * NP) return;
  const int sl = sl0 + j;
  const int4 r1 = __ldg(st.rec + 2 * (size_t)sl + 1);
  const int fl = r1.y, e = r1.z;
  double ow[NF], ot[NF];
#pragma unroll
  for (int k = 0; k < NF; ++k) {
    ow[k] = ROWS ? 0.0 : sOw[ROWS ? 0 : warp][ROWS ? 0 : (j * NP + i) * NF + k];
    ot[k] = ot_s[(j * NP + i) * NF + k];
  }
  if constexpr (ROWS) {
    const int gr = (cell_type(g, e) * 3 + ((fl >> 2) & 3)) * 2 + ((fl & 16) ? 1 : 0);
    const int n = __ldg(ops.ex_n + gr * NP + i);
    const size_t at = (size_t)gr * S * NP + i;
    const double* pf = PF + (size_t)e * S * PFW;
#pragma unroll 3
    for (int k = 0; k < n; ++k) {
      const double w = __ldg(ops.ex_w + at + (size_t)k * NP);
      const double2* x = reinterpret_cast<const double2*>(pf + __ldg(ops.ex_i + at + (size_t)k * NP) * PFW);
#pragma unroll
      for (int q = 0; q < (NF + 1) / 2; ++q) {
        const double2 v = __ldg(x + q);
        ow[2 * q] += w * v.x;
        if (2 * q + 1 < NF) ow[2 * q + 1] += w * v.y;
      }
    }
  }
  face_jump<S, NP, VISC>(g, fc, bc, sl, i, e, r1.w, (fl & 1) == 0, (fl & 2) != 0, (fl & 16) ? 1.0 : -1.0, ow, ot, arow,
                         mu, J);
}

// own adjugate row of the face's axis at every slot flux point (E * adj) and
// its norm, negative where the row's direction falls back to the face normal
// (alignment below 0.5, core/fr_residual/inviscid_kernel_colored.py:104-108);
// normals (F, P, 3); fallback: set where an interior slot does
template <int S, int NP>
__global__ void k_slot_rows(Geom g, Ops ops, const double* __restrict__ normals, SlotTable st,
                            double4* __restrict__ arow, unsigned* fallback) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)st.n * NP) return;
  const int sl = (int)(t / NP), i = (int)(t % NP);
  const int4 rc = __ldg(st.rec + 2 * (size_t)sl + 1);
  const int f = rc.x, fl = rc.y, e = rc.z;
  const int ax = (fl >> 2) & 3, sb = (fl & 16) ? 1 : 0;
  const double* Er = ops.extrap + ((((size_t)cell_type(g, e) * 3 + ax) * 2 + sb) * NP + i) * S;
  double a0 = 0.0, a1 = 0.0, a2 = 0.0;
  for (int s = 0; s < S; ++s) {
    const double w = Er[s];
    const double* ad = g.adj + ((size_t)e * S + s) * 9 + ax * 3;
    a0 += w * ad[0];
    a1 += w * ad[1];
    a2 += w * ad[2];
  }
  double mag = sqrt(a0 * a0 + a1 * a1 + a2 * a2);
  if (mag < 1e-300) mag = 1e-300;
  const double side = sb ? 1.0 : -1.0, sg = (fl & 1) == 0 ? 1.0 : -1.0;
  const double* tn = normals + ((size_t)f * NP + i) * 3;
  const double al = a0 / mag * side * (sg * tn[0]) + a1 / mag * side * (sg * tn[1]) + a2 / mag * side * (sg * tn[2]);
  arow[t] = make_double4(a0, a1, a2, al < 0.5 ? -mag : mag);
  if (al < 0.5 && !(fl & 2)) *fallback = 1u;
}

// every slot's normals at its face's row
__global__ void k_slot_face_rows(SlotTable st) {
  const int sl = blockIdx.x * blockDim.x + threadIdx.x;
  if (sl < st.n) st.rec[2 * (size_t)sl + 1].w = st.rec[2 * (size_t)sl + 1].x;
}

// ---------------------------------------------------------------------------
// cell kernel: CPB cells per CTA (structured prisms of orders 1 and 2 take
// k_px_cell and k_update).  Volume terms (inviscid over-integrated
// divergence with W = f2c * D_fine folded at create, viscous divergence),
// lifting of the face jumps of each cell's slots in ascending color order,
// outlier suppression, then (stage >= 0) the SSP-RK3 Shu-Osher combination,
// positivity projection and modal filter (core/time_integration/base.py:250-335,
// core/time_integration/positivity.py:13-45, core/fr_solver/filter.py:29-42).
// ---------------------------------------------------------------------------
constexpr int CELL_THREADS = 256;
constexpr int CELL_MAXSLOT = 6;  // slots per cell staged in shared memory (more: read from global)

// Doubles of each block.  Without viscosity only q of the point fields, the
// inviscid jumps and residuals are held, so more CTAs fit an SM.
template <int S, int FN, int CPB, int NPMAX, bool VISC>
struct CellSmem {
  static constexpr int PS = VISC ? PFS : 5;        // point-field row stride
  static constexpr int JF = VISC ? 9 : 5;          // jump fields
  static constexpr int oPF = 0;                    // CPB*S*PS
  static constexpr int oAdj = oPF + CPB * S * PS;  // CPB*S*9
  static constexpr int oU = oAdj + (VISC ? CPB * S * 9 : 0);  // CPB*S*US
  static constexpr int oDet = oU + CPB * S * US;   // CPB*S: det, then 1 / det
  static constexpr int oRi = oDet + CPB * S;       // CPB*S*5
  static constexpr int oRv = oRi + CPB * S * 5;    // CPB*S*5
  static constexpr int oQf = oRv + (VISC ? CPB * S * 5 : 0);  // CPB*FN*5
  static constexpr int oFt = oQf + CPB * FN * 5;   // CPB*FN*15
  static constexpr int oGt = oFt + CPB * FN * 15;  // CPB*S*15; with or without viscosity the norm terms (2*CPB*S)
  static constexpr int oJ = oGt + (VISC ? CPB * S * 15 : CPB * S * 2);  // staged jumps of the CTA's slots
  static constexpr int oAf = oJ + CPB * CELL_MAXSLOT * NPMAX * JF;      // CPB*FN*9 adjugates at the fine points
  static constexpr int work = oAf + CPB * FN * 9;  // CPB*2*OUT_WORK (outliers)
  static constexpr int oG = work + CPB * 2 * OUT_WORK;  // g_left, g_right (8)
  static constexpr int oI = oG + 8;                // ints: lifting maps (6*S), slot flags, slot pointers
  static constexpr int total = oI + (6 * S + CPB * CELL_MAXSLOT + CPB + 2) / 2 + 1;
};

template <int S, int FN, int NP, int CPB, bool VISC>
__global__ void __launch_bounds__(CELL_THREADS, 3) k_cell(Geom g, Ops ops, Faces fc, StageArgs a,
                                                          const double* __restrict__ J) {
  using L = CellSmem<S, FN, CPB, NP, VISC>;
  extern __shared__ double sm[];
  double* sPF = sm + L::oPF;
  double* sAdj = sm + L::oAdj;
  double* sU = sm + L::oU;
  double* sDet = sm + L::oDet;
  double* sRi = sm + L::oRi;
  double* sRv = sm + L::oRv;
  double* sQf = sm + L::oQf;
  double* sFt = sm + L::oFt;
  double* sGt = sm + L::oGt;
  double* work = sm + L::work;
  double* sG = sm + L::oG;
  int* sDfp = reinterpret_cast<int*>(sm + L::oI);
  int* sDco = sDfp + 3 * S;
  int* sFl = sDco + 3 * S;
  int* sPtr = sFl + CPB * CELL_MAXSLOT;
  const int e0 = a.cell_base + blockIdx.x * CPB;
  const int nc = min(CPB, a.cell_end - e0);
  const int ct = cell_type(g, e0);  // a launch covers cells of one type
  const int nv = a.nv;
  constexpr bool visc = VISC;
  constexpr int PS = L::PS;
  const int tid = threadIdx.x;

  double* sAf = sm + L::oAf;
  // ---- load: asynchronous 8-byte copies, all in flight at once ----
  for (int t = tid; t < nc * S * (VISC ? PFW : 5); t += blockDim.x) {
    const int p = t / (VISC ? PFW : 5), k = t % (VISC ? PFW : 5);
    cp_async8(sPF + p * PS + k, a.PF + ((size_t)e0 * S + p) * PFW + k);
  }
  if (VISC)
    for (int t = tid; t < nc * S * 9; t += blockDim.x) cp_async8(sAdj + t, g.adj + (size_t)e0 * S * 9 + t);
  for (int t = tid; t < nc * S * nv; t += blockDim.x)
    cp_async8(sU + (t / nv) * US + t % nv, a.Ucur + (size_t)e0 * S * nv + t);
  for (int t = tid; t < nc * S; t += blockDim.x) cp_async8(sDet + t, g.det + (size_t)e0 * S + t);
  for (int t = tid; t < nc * FN * 9; t += blockDim.x) cp_async8(sAf + t, g.adj_fine + (size_t)e0 * FN * 9 + t);
  // the jumps of this CTA's slots are contiguous (slots are stored cell-major)
  const int k_beg = fc.slot_ptr[e0], k_end = fc.slot_ptr[e0 + nc];
  const bool staged = (k_end - k_beg) <= CPB * CELL_MAXSLOT;
  double* sJ = sm + L::oJ;
  constexpr int JF = L::JF;
  if (staged) {
    for (int t = tid; t < (k_end - k_beg) * NP * JF; t += blockDim.x) {
      const int k = t / (NP * JF), r = t - k * (NP * JF);
      cp_async8(sJ + t, J + (size_t)(k_beg + k) * 9 * NP + r);
    }
    for (int t = tid; t < k_end - k_beg; t += blockDim.x) sFl[t] = __ldg(a.slot_flags + k_beg + t);
  }
  // the lifting's maps: read per slot and point below, where each was a chain
  // of dependent global loads
  constexpr int N1D = S == 8 ? 2 : (S == 27 ? 3 : 4);
  for (int t = tid; t < 3 * S; t += blockDim.x) {
    sDfp[t] = __ldg(ops.dist_fp + t);
    sDco[t] = __ldg(ops.dist_co + t);
  }
  if (tid < N1D) {
    sG[tid] = ops.g_left[tid];
    sG[4 + tid] = ops.g_right[tid];
  }
  if (tid <= nc) sPtr[tid] = __ldg(fc.slot_ptr + e0 + tid);
  cp_async_wait_all();
  __syncthreads();

  // ---- Q at fine points (c2f, an FP64 tensor-core product: rows the fine
  // points, columns (cell, variable)) and viscous contravariant fluxes ----
  {
    dmma_product_rb<(5 * CPB + 7) / 8>(
        FN, 5 * nc, S, ops.fc2f[ct],
        [&](int s, int col) { return sPF[((col / 5) * S + s) * PS + col % 5]; },
        [&](int i, int col, double x) { sQf[((col / 5) * FN + i) * 5 + col % 5] = x; });
  }
  if constexpr (VISC) {
    for (int t = tid; t < nc * S; t += blockDim.x) {
      double G[3][4];
      const double* p = sPF + t * PS;
      viscous_flux_sym(p + 1, p + 5, p + 11, a.mu, p[14], G);
      const double* am = sAdj + t * 9;
      for (int m = 0; m < 3; ++m) {
        sGt[(t * 3 + m) * 5] = 0.0;
        for (int v = 0; v < 4; ++v)
          sGt[(t * 3 + m) * 5 + 1 + v] = am[m * 3 + 0] * G[0][v] + am[m * 3 + 1] * G[1][v] + am[m * 3 + 2] * G[2][v];
      }
    }
  }
  __syncthreads();
  for (int t = tid; t < nc * S; t += blockDim.x) sDet[t] = 1.0 / sDet[t];  // each use within an ulp of a division
  // ---- Euler fluxes at fine points, contravariant with adj_fine ----
  for (int t = tid; t < nc * FN; t += blockDim.x) {
    const int b = t / FN, i = t % FN;
    double q[5], F[3][5];
    for (int v = 0; v < 5; ++v) q[v] = sQf[t * 5 + v];
    euler_flux(q, F);
    const double* ad = sAf + (size_t)(b * FN + i) * 9;
    double am[9];
    for (int k = 0; k < 9; ++k) am[k] = ad[k];
    for (int m = 0; m < 3; ++m)
      for (int v = 0; v < 5; ++v)
        sFt[(t * 3 + m) * 5 + v] = am[m * 3 + 0] * F[0][v] + am[m * 3 + 1] * F[1][v] + am[m * 3 + 2] * F[2][v];
  }
  __syncthreads();
  // ---- divergences on the FP64 tensor path: inviscid W (S x 3FN) applied to
  // the fine-point fluxes, viscous D3 (S x 3S) to the point fluxes; rows the
  // solution points, columns (cell, variable) ----
  {
    auto fb = [&](int k, int col) { return sFt[(col / 5) * FN * 15 + k * 5 + col % 5]; };
    auto fo = [&](int s, int col, double x) {
      const int b = col / 5;
      sRi[(b * S + s) * 5 + col % 5] = -x * sDet[b * S + s];
    };
    // with as many row tiles as warps, each warp keeps its operator fragment for
    // every column tile
    if constexpr ((S + 7) / 8 >= CELL_THREADS / 32 && 5 * CPB > 8)
      dmma_product_rb<(5 * CPB + 7) / 8>(S, 5 * nc, FN * 3, ops.fW[ct], fb, fo);
    else
      dmma_product_f(S, 5 * nc, FN * 3, ops.fW[ct], fb, fo);
    if constexpr (VISC) {
      dmma_product_f(
          S, 5 * nc, S * 3, ops.fD3[ct],
          [&](int k, int col) { return sGt[(col / 5) * S * 15 + k * 5 + col % 5]; },
          [&](int s, int col, double x) {
            const int b = col / 5;
            sRv[(b * S + s) * 5 + col % 5] = x * sDet[b * S + s];
          });
    }
  }
  __syncthreads();
  // ---- lift the face jumps of each cell's slots, ascending color order ----
  for (int t = tid; t < nc * S * 5; t += blockDim.x) {
    const int b = t / (S * 5), r = t % (S * 5), s = r / 5, v = r % 5;
    const double rdj = sDet[b * S + s];  // each term within an ulp of g' J / det
    double ci = 0.0, cv = 0.0;
    for (int k = sPtr[b]; k < sPtr[b + 1]; ++k) {
      const int fl = staged ? sFl[k - k_beg] : a.slot_flags[k];
      const int ax = (fl >> 2) & 3;
      const int fp = sDfp[ax * S + s];
      const double gw = sG[((fl & 16) ? 4 : 0) + sDco[ax * S + s]];
      const double* Jk = staged ? sJ + (k - k_beg) * JF * NP + fp : J + (size_t)k * 9 * NP + fp;
      ci += -(gw * Jk[v * NP]) * rdj;
      if (VISC && v > 0) cv += (gw * Jk[(4 + v) * NP]) * rdj;
    }
    sRi[t] = sRi[t] + ci;
    if constexpr (VISC) sRv[t] = sRv[t] + cv;
  }
  __syncthreads();
  suppress_outliers_cells<S>(sRi, sRv, sU, nc, visc, work);

  if (a.stage < 0) {
    for (int t = tid; t < nc * S * nv; t += blockDim.x) {
      const int p = t / nv, v = t % nv;
      if (a.Rinv) a.Rinv[(size_t)e0 * S * nv + t] = v < 5 ? sRi[p * 5 + v] : 0.0;
      if (a.Rvisc) a.Rvisc[(size_t)e0 * S * nv + t] = (v < 5 && visc) ? sRv[p * 5 + v] : 0.0;
    }
    return;
  }

  // ---- RK stage combination + positivity (per point) ----
  double* Up = sQf;  // (CPB*S, US) reuses the fine-point scratch (and the flux scratch after it)
  static_assert(CPB * S * US <= CPB * FN * 20, "RK tile must fit the fine-point and flux scratch");
  double* part = sGt;  // (CPB*S) squared dU/dt per point (stage 0)
  // loops over the 8 possible variables, unrolled, so the arrays stay in registers
  for (int p = tid; p < nc * S; p += blockDim.x) {
    double Lr[8], un[8];
    double sq_sum = 0.0;
#pragma unroll
    for (int v = 0; v < 8; ++v) Lr[v] = v < 5 ? sRi[p * 5 + v] + (visc ? sRv[p * 5 + v] : 0.0) : 0.0;
#pragma unroll
    for (int v = 0; v < 8; ++v)
      if (v < nv) sq_sum += Lr[v] * Lr[v];
    const size_t gp = (size_t)e0 * S + p;
    const double dts = a.dt[gp];
    const double* u0 = a.U0 + gp * nv;
    const double* uc = sU + p * US;
    if (a.stage == 0) {
#pragma unroll
      for (int v = 0; v < 8; ++v) un[v] = v < nv ? u0[v] + dts * Lr[v] : 0.0;
    } else if (a.stage == 1) {
#pragma unroll
      for (int v = 0; v < 8; ++v) un[v] = v < nv ? (0.75 * u0[v] + 0.25 * uc[v]) + (0.25 * dts) * Lr[v] : 0.0;
    } else {
      // 1/3 U0 + 0 U1 + 2/3 U2 + 2/3 dt L; the 0*U1 term is dropped: it can only
      // turn a finite value into NaN where U1 is non-finite, and U2 (filtered
      // from U1) is then non-finite at the same cell already.
#pragma unroll
      for (int v = 0; v < 8; ++v)
        un[v] = v < nv ? (1.0 / 3.0 * u0[v] + 2.0 / 3.0 * uc[v]) + (2.0 / 3.0 * dts) * Lr[v] : 0.0;
    }
    const double rho = fmax(un[0], 1e-6);
    un[0] = rho;
    double vel[3] = {un[1] / rho, un[2] / rho, un[3] / rho};
    const double vm = sqrt(vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2]);
    if (vm > 1e4) {
      const double cf = 1e4 / vm;
      for (int d = 0; d < 3; ++d) { vel[d] *= cf; un[1 + d] = rho * vel[d]; }
    }
    const double ke = 0.5 * rho * (vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2]);
    const double pr = (GAMMA - 1.0) * (un[4] - ke);
    if (pr < 1.0) un[4] = 1.0 / (GAMMA - 1.0) + ke;
    if (nv > 5) un[5] = fmax(un[5], 0.0);
    if (nv > 6) un[6] = fmax(un[6], 1e-8);
#pragma unroll
    for (int v = 0; v < 8; ++v)
      if (v < nv) Up[p * US + v] = un[v];
    part[p] = sq_sum;
    part[CPB * S + p] = Lr[0] * Lr[0];
  }
  __syncthreads();
  // modal filter on the first five variables as an FP64 tensor-core product
  // (rows s, columns (cell, variable), K the cell's points)
  dmma_product_f(
      S, 5 * nc, S, ops.ffilt[ct],
      [&](int j, int col) { return Up[((col / 5) * S + j) * US + col % 5]; },
      [&](int s, int col, double x) { a.Unext[((size_t)(e0 + col / 5) * S + s) * nv + col % 5] = x; });
  for (int p = tid; p < nc * S; p += blockDim.x)
    for (int v = 5; v < nv; ++v) a.Unext[((size_t)e0 * S + p) * nv + v] = Up[p * US + v];
  if (a.stage == 0 && tid < nc) {
    double acc = 0.0;  // fixed order per cell: points ascending
    for (int s = 0; s < S; ++s) acc += part[tid * S + s];
    a.norm_part[e0 + tid] = acc;
    double acc_rho = 0.0;
    for (int s = 0; s < S; ++s) acc_rho += part[CPB * S + tid * S + s];
    a.norm_rho_part[e0 + tid] = acc_rho;
    // a non-finite dU/dt anywhere in the cell makes its partial non-finite
    if (!isfinite(acc) && a.status) atomicOr(a.status, (unsigned)DS_NONFINITE);
  }
}

}  // namespace afr
