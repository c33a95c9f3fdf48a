// Mixed-precision form of the FR residual-and-update stage.
//
// Prisms whose operators are tensor products take the FP32 cell kernel
// (afr_prism.cuh) in place of k_mx_pre and k_mx_vol.  Elsewhere (tets, P3) the
// operator contractions run on the tensor cores (tcgen05, BF16 inputs, FP32
// accumulation in tensor memory) as three-term hi+lo split products,
// D = A_hi*B_hi + A_hi*B_lo + A_lo*B_hi, which carry about 16 significant bits
// of each factor.  Pointwise fluxes are FP32.  FP64 is kept for the state, the
// geometry metrics, the primitive recovery from the conserved state, the
// residual sums and RK update, the norm and the force coefficients.
//
// Four kernels per stage (same data flow as the reference's residual,
// core/fr_residual/inviscid.py:139-345 and core/fr_residual/viscous_flux.py:113-302):
//   k_mx_pre   per 8-cell tile: gradients of (u,v,w,T) (D_3d as a GEMM) and the
//              extrapolation of all point fields to every face point of the
//              cell (boundary_extrap of all six faces stacked as one GEMM);
//   k_mx_face  per pair of slot flux points: AUSM+up and BR1 jumps.  Where the
//              other side's interpolation row equals one of that cell's own
//              extrapolation rows (matched once at create: every prism face
//              point, most tet face points) the other side is read from its
//              face-point fields; elsewhere it is interpolated from the source
//              cells' FP32 point fields with the reference's matrices;
//   k_mx_vol   per C-cell tile (persistent): c2f, viscous D_3d and the folded
//              W = f2c*D_fine divergence as GEMMs -> volume terms (FP32);
//   k_update a warp per few cells: lifting in ascending color order, outlier
//              zeroing, SSP-RK3 combination, positivity (FP64), filter (an
//              FP64 product on the tensor path).
//
// Contraction inputs are deviations from the cell mean where the operator
// reproduces constants (c2f, extrapolation, derivatives), so the split error is
// relative to the variation inside the cell, not to the free-stream level.  The
// inviscid flux is split as F(q) = F(qbar) + dF: the W contraction acts on the
// contravariant dF (formed algebraically, without cancellation), and
// W*(adj_fine (x) F(qbar)) = MD*F(qbar) uses the FP64 metric divergence
// MD[c,s,n] = sum_{i,m} W[s,(i,m)] adj_fine[c,i,m,n] formed at create.
//
// Shared-memory operand images are K-major without swizzle (afr_tc.cuh).  Row
// orders are chosen so that lanes of a warp write eight consecutive 16-byte
// rows (conflict-free 2-byte stores): A rows are (field, cell) with the cell
// index fastest in groups of eight.
#pragma once
#include "afr_kernels.cuh"
#include "afr_tc.cuh"

namespace afr {

constexpr int MX_THREADS = 512;  // pre-pass CTA
constexpr int MX_PRE_CELLS = 8;

__host__ __device__ constexpr int pad16(int x) { return (x + 15) / 16 * 16; }
__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }
__host__ __device__ constexpr int pow2_cols(int x) { return x <= 32 ? 32 : (x <= 64 ? 64 : (x <= 128 ? 128 : 256)); }
// Copies of the face-point rows in the 128-row extrapolation image: with 6*NP
// face points <= 32 (P1) every 32-lane quarter of tensor memory holds a copy,
// <= 64 (P2) two halves do; each copy's readout serves its share of the tile's
// cells, so every warp of the CTA takes part in the readout.
__host__ __device__ constexpr int mx_ext_dup(int nfp) { return nfp <= 32 ? 4 : (nfp <= 64 ? 2 : 1); }

// Operator images, K-major canonical, BF16 bit patterns.  "cat" images stack
// the hi rows over the lo rows (2N rows, one image); the others are [hi | lo].
struct MxOps {
  const uint16_t* c2f[2];  // B cat: rows i < Fq (fine point), K = Sq (solution point)
  const uint16_t* W[2];    // B cat: rows s < Sq, K = 3*Fq, k = m*Fq + i
  const uint16_t* D3[2];   // B cat: rows s < Sq, K = 3*Sq, k = m*Sq + j
  const uint16_t* D3g[2];  // B: rows m*Sq + s, K = Sq (j)
  const uint16_t* E[2];    // A: rows j*(128/DUP) + fp, fp = (ax*2+side)*NP + i, copies j < DUP = mx_ext_dup(6*NP); K = Sq
  const double* MD;        // (N, S, 3) metric divergence of the folded W
  const float4* adjf;      // (N, FN, 3) FP32 fine-point adjugate rows (4th entry zero)
  const float4* adjs;      // (N, S, 3) FP32 solution-point adjugate rows
  const float4* invs;      // (N, S, 3) FP32 inverse-Jacobian rows
  const double* rdet;      // (N, S) 1 / det, FP64
  const double* hcell;     // (N) interior-penalty length, cube root of the mean det
};

constexpr uint8_t MX_OFP_GENERAL = 255;  // other side by interpolation from point fields

struct MxFace {
  // (n_slots*NP) own adjugate row at the flux point, and its norm; the norm is
  // negative where the alignment fallback replaces the row's direction by the
  // face normal (both are geometry: decided once)
  const float4* arow;
  const uint8_t* ofp;   // (n_slots*NP) face point of the other side, (ax*2+side)*NP + j, or MX_OFP_GENERAL
};

// A matched pair of slot points: everything the paired face kernel needs to
// find its data, in one 16-byte load (the chain pair -> slot -> face -> cells
// was three dependent loads).  Rows are (cell*6 + face)*NP + point with the
// slot's side in the sign bit.
struct MxPair {
  int32_t t, t2;        // owner- and neighbour-side slot points
  uint32_t row, row2;   // their own face-point rows
};

// Point fields: q (5), symmetric velocity gradient (S00, S11, S22, S01, S02,
// S12: the viscous flux holds no other combination), grad T (3), mu_t.
constexpr int MX_XF = 15;  // fields per face point, in that order
constexpr int MX_PF = 16;  // floats per solution point: gradients (9), mu_t, q (5), 1 unused

struct MxBuf {
  float* XF;   // (N, 6, FW, NP) point fields at the face points, one contiguous block per face of the cell
  float* PFm;  // (N, S, MX_PF)
  float* Jm;   // (n_slots, 9, NP) jumps: inviscid (5), viscous momentum and energy (4)
  float* RV;   // (N, 9, S) volume terms, in the same order
  int FW;      // MX_XF (orders 1, 2) or 5 (order 3: inviscid only)
};

namespace mxd {

__device__ __forceinline__ void st_split(uint16_t* img, int img_elems, int idx, float x) {
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  const __nv_bfloat16 l = __float2bfloat16_rn(x - __bfloat162float(h));
  img[idx] = __bfloat16_as_ushort(h);
  img[img_elems + idx] = __bfloat16_as_ushort(l);
}

// n floats, 16-byte vector accesses when both ends allow them
__device__ __forceinline__ void copy_f32(float* dst, const float* src, int n) {
  if (((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u) == 0) {
    const float4* s4 = reinterpret_cast<const float4*>(src);
    float4* d4 = reinterpret_cast<float4*>(dst);
    for (int t = threadIdx.x; t < n / 4; t += blockDim.x) d4[t] = s4[t];
    for (int t = (n / 4) * 4 + threadIdx.x; t < n; t += blockDim.x) dst[t] = src[t];
  } else {
    for (int t = threadIdx.x; t < n; t += blockDim.x) dst[t] = src[t];
  }
}

// L2 prefetch of bytes [off, off + bytes) of an array of total bytes (bulk
// copy engine, no data returned to the SM); the range is clipped to 16-byte
// boundaries inside the array.  A hint: issued by one thread.
__device__ __forceinline__ void prefetch_l2(const void* base, size_t total, size_t off, size_t bytes) {
  const size_t lo = off & ~size_t(15);
  size_t hi = off + bytes;
  hi = (hi + 15) & ~size_t(15);
  const size_t cap = total & ~size_t(15);
  if (hi > cap) hi = cap;
  const uintptr_t b = reinterpret_cast<uintptr_t>(base);
  for (size_t p = lo; p < hi; p += 32768) {
    const uint32_t n = (uint32_t)((hi - p) < 32768 ? (hi - p) : 32768);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(b + p), "r"(n) : "memory");
  }
}

using afr::cp_async8;
using afr::cp_async_wait_all;

// 16-byte copy global -> shared of an operator image
__device__ __forceinline__ void copy_img(void* dst, const void* src, int bytes) {
  const uint4* s = reinterpret_cast<const uint4*>(src);
  uint4* d = reinterpret_cast<uint4*>(dst);
  for (int t = threadIdx.x; t < bytes / 16; t += blockDim.x) d[t] = __ldg(s + t);
}

// D (tensor memory) = A * B^T over K with the three-term split; A has 128
// rows, B has nb rows.  Issued by one thread.
__device__ __forceinline__ void mma_split(uint32_t tmem, const uint16_t* A, const uint16_t* B, int nb, int K) {
  const uint32_t a_hi = tc::smem_u32(A), a_lo = a_hi + 128u * K * 2u;
  const uint32_t b_hi = tc::smem_u32(B), b_lo = b_hi + (uint32_t)nb * K * 2u;
  const uint32_t idesc = tc::idesc_bf16(128, nb);
  for (int ks = 0; ks < K / 16; ++ks) {
    const uint32_t ao = ks * 2u * 128u * 16u, bo = ks * 2u * (uint32_t)nb * 16u;
    const uint64_t ah = tc::make_desc(a_hi + ao, 128 * 16, 128), al = tc::make_desc(a_lo + ao, 128 * 16, 128);
    const uint64_t bh = tc::make_desc(b_hi + bo, nb * 16, 128), bl = tc::make_desc(b_lo + bo, nb * 16, 128);
    tc::mma_bf16(tmem, ah, bh, idesc, ks > 0 ? 1u : 0u);
    tc::mma_bf16(tmem, ah, bl, idesc, 1u);
    tc::mma_bf16(tmem, al, bh, idesc, 1u);
  }
}

// D (tensor memory, 2n columns) with the three-term split against a stacked
// operator image Bcat = [B_hi; B_lo] (2n rows): columns [0, n) collect
// A_hi*B_hi + A_lo*B_hi and columns [n, 2n) collect A_hi*B_lo; the sum of the
// two blocks is the product.  Two MMAs per K step, A_hi read once.
__device__ __forceinline__ void mma_cat(uint32_t tmem, const uint16_t* A, const uint16_t* Bcat, int n, int K) {
  const uint32_t a_hi = tc::smem_u32(A), a_lo = a_hi + 128u * K * 2u;
  const uint32_t b = tc::smem_u32(Bcat);
  const uint32_t id2 = tc::idesc_bf16(128, 2 * n), id1 = tc::idesc_bf16(128, n);
  for (int ks = 0; ks < K / 16; ++ks) {
    const uint32_t ao = ks * 2u * 128u * 16u, bo = ks * 2u * 2u * (uint32_t)n * 16u;
    const uint64_t ah = tc::make_desc(a_hi + ao, 128 * 16, 128), al = tc::make_desc(a_lo + ao, 128 * 16, 128);
    const uint64_t bc = tc::make_desc(b + bo, 2 * n * 16, 128);  // all 2n rows; the first n are B_hi
    tc::mma_bf16(tmem, ah, bc, id2, ks > 0 ? 1u : 0u);
    tc::mma_bf16(tmem, al, bc, id1, 1u);
  }
}

// (cell, point) enumeration with the cell fastest in groups of 8: lanes of a
// warp cover 8 cells x 4 consecutive points.
__device__ __forceinline__ void cell_point(int idx, int npts, int& c, int& p) {
  const int rest = idx >> 3;
  p = rest % npts;
  c = (rest / npts) * 8 + (idx & 7);
}

// F(qbar + dq) - F(qbar) for the Euler flux, written as telescoped products so
// that no large terms cancel (qbar, dq primitive: rho, u, v, w, p).
template <class T>
__device__ __forceinline__ void euler_flux_delta(const T qb[5], const T dq[5], T dF[3][5]) {
  const T rb = qb[0], dr = dq[0], dp = dq[4];
  const T ub[3] = {qb[1], qb[2], qb[3]}, du[3] = {dq[1], dq[2], dq[3]};
  const T u[3] = {ub[0] + du[0], ub[1] + du[1], ub[2] + du[2]};
  const T g1 = T(GAMMA / (GAMMA - 1.0));
  const T uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
  const T d_uu = (u[0] + ub[0]) * du[0] + (u[1] + ub[1]) * du[1] + (u[2] + ub[2]) * du[2];
  const T p = qb[4] + dp;
  const T r = rb + dr;
  const T e = g1 * p + T(0.5) * r * uu;                 // rho H
  const T de = g1 * dp + T(0.5) * (dr * uu + rb * d_uu);
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    const T dm = dr * u[n] + rb * du[n];              // delta(rho u_n)
    const T mb = rb * ub[n];
    dF[n][0] = dm;
#pragma unroll
    for (int j = 0; j < 3; ++j) dF[n][1 + j] = dm * u[j] + mb * du[j] + (n == j ? dp : T(0));
    dF[n][4] = du[n] * e + ub[n] * de;
  }
}

// primitives (rho, u, v, w, p) without pressure floor (core/fr_residual/inviscid.py:38-47)
// and T = p / (rho R), with one reciprocal of rho (the mixed form has no bitwise target)
__device__ __forceinline__ void prim_T(const double* U, double q[6]) {
  const double rho = fmax(U[0], 1e-10);
  const double r = 1.0 / rho;
  const double u = U[1] * r, v = U[2] * r, w = U[3] * r;
  const double p = (GAMMA - 1.0) * rho * (U[4] * r - 0.5 * (u * u + v * v + w * w));
  q[0] = rho; q[1] = u; q[2] = v; q[3] = w; q[4] = p;
  q[5] = p * r * (1.0 / R_AIR);
}

__device__ __forceinline__ bool wait_commit(uint64_t* bar, uint32_t& phase, unsigned* status) {
  const bool ok = tc::mbar_wait(bar, phase);
  phase ^= 1u;
  if (!ok) atomicOr(status, (unsigned)DS_TC_TIMEOUT);
  return ok;
}

}  // namespace mxd

// ---------------------------------------------------------------------------
// pre-pass: gradients and face-point extrapolation of one 8-cell tile
// ---------------------------------------------------------------------------
template <int S, int NP>
struct MxPreSmem {
  static constexpr int Sq = pad16(S), NFP = 6 * NP, NB1 = 3 * Sq, NB2MAX = 128;
  static constexpr int oB1 = 0;                        // D3g image (hi|lo)
  static constexpr int oA2 = oB1 + NB1 * Sq * 4;       // E image
  static constexpr int oA1 = oA2 + 128 * Sq * 4;       // gradient inputs, rows phi*8 + c
  static constexpr int oB2 = oA1 + 128 * Sq * 4;       // face-field inputs, rows f*8 + c
  static constexpr int oG = oB2 + NB2MAX * Sq * 4;     // reference-space gradients [c][s][m][phi]
  static constexpr int oQ = oG + MX_PRE_CELLS * S * 12 * 4;  // q and T (FP64) [c][s][6]
  static constexpr int oM = oQ + MX_PRE_CELLS * S * 6 * 8;   // means (FP64) [c][9]
  // the next tile's state rows (stride nv <= 8) and nu_t, copied asynchronously
  // (P1, P2; at P3 the tile's loads are direct: no room)
  static constexpr bool STG = S <= 27;
  static constexpr int oStg = oM + MX_PRE_CELLS * 9 * 8;
  // and the next tile's FP32 inverse-Jacobian rows (float4 x 3 per point), 16-byte aligned
  static constexpr int oInv = (oStg + (STG ? MX_PRE_CELLS * S * 9 * 8 : 0) + 15) / 16 * 16;
  static constexpr int total = oInv + (STG ? MX_PRE_CELLS * S * 48 : 0);
  static constexpr int NCOL = pow2_cols(cmax(NB1, NB2MAX));
};

template <int S, int NP>
__global__ void __launch_bounds__(MX_THREADS, 2)  // 64 registers: two CTAs per SM (tensor memory allows two)
    k_mx_pre(Geom g, MxOps mo, MxBuf mb, const double* __restrict__ U, int nv, const double* __restrict__ nut,
             int visc, int cell_base, int cell_end, unsigned* status) {
  using L = MxPreSmem<S, NP>;
  constexpr int Sq = L::Sq, NFP = L::NFP, C = MX_PRE_CELLS;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t bar;
  __shared__ uint32_t tbase;
  __shared__ int abort_flag;
  uint16_t* sB1 = reinterpret_cast<uint16_t*>(smem + L::oB1);
  uint16_t* sA2 = reinterpret_cast<uint16_t*>(smem + L::oA2);
  uint16_t* sA1 = reinterpret_cast<uint16_t*>(smem + L::oA1);
  uint16_t* sB2 = reinterpret_cast<uint16_t*>(smem + L::oB2);
  float* sG = reinterpret_cast<float*>(smem + L::oG);
  double* sQ = reinterpret_cast<double*>(smem + L::oQ);
  double* sM = reinterpret_cast<double*>(smem + L::oM);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int FW = mb.FW;
  visc = visc && FW >= MX_XF;
  const int nfw = visc ? MX_XF : 5;  // fields extrapolated by this call
  const int NB2 = pad16(nfw * C);
  const int ct = cell_type(g, cell_base);

  if (visc) mxd::copy_img(sB1, (ct ? mo.D3g[1] : mo.D3g[0]), L::NB1 * Sq * 4);
  mxd::copy_img(sA2, (ct ? mo.E[1] : mo.E[0]), 128 * Sq * 4);
  // operand padding (K columns s >= S, rows never written) stays zero
  for (int t = tid; t < 128 * Sq * 4 / 16; t += MX_THREADS) reinterpret_cast<uint4*>(sA1)[t] = make_uint4(0, 0, 0, 0);
  for (int t = tid; t < L::NB2MAX * Sq * 4 / 16; t += MX_THREADS)
    reinterpret_cast<uint4*>(sB2)[t] = make_uint4(0, 0, 0, 0);
  if (warp == 0) tc::tmem_alloc(&tbase, L::NCOL);
  if (tid == 0) {
    tc::mbar_init(&bar, 1);
    tc::fence_mbar_init();
    abort_flag = 0;
  }
  tc::fence_async_smem();
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tbase;
  uint32_t phase = 0;
  const int ntiles = (cell_end - cell_base + C - 1) / C;

  // asynchronous copies of a tile's contiguous state and nu_t blocks into the
  // staging buffer; issued one tile ahead, so they overlap the tile before
  double* sStg = reinterpret_cast<double*>(smem + L::oStg);
  float4* sInvs = reinterpret_cast<float4*>(smem + L::oInv);
  auto stage = [&](int tl) {
    if constexpr (L::STG) {
      const size_t eb = (size_t)cell_base + (size_t)tl * C;
      const int nn = min(C, cell_end - (int)eb);
      const double* ub = U + eb * S * nv;
      for (int t = tid; t < nn * S * nv; t += MX_THREADS) cp_async8(sStg + t, ub + t);
      if (nut)
        for (int t = tid; t < nn * S; t += MX_THREADS) cp_async8(sStg + C * S * 8 + t, nut + eb * S + t);
      cp_async_commit();
    }
  };
  // the tile's inverse-Jacobian rows: read by the gradient phase, so the next
  // tile's copies are issued only once that phase of the current tile is over
  auto stage_inv = [&](int tl) {
    if constexpr (L::STG) {
      if (visc) {
        const size_t eb = (size_t)cell_base + (size_t)tl * C;
        const int nn = min(C, cell_end - (int)eb);
        const float4* ib = mo.invs + eb * S * 3;
        for (int t = tid; t < nn * S * 3; t += MX_THREADS) cp_async16(sInvs + t, ib + t);
        cp_async_commit();
      }
    }
  };
  if (blockIdx.x < ntiles) {
    stage(blockIdx.x);
    stage_inv(blockIdx.x);
  }

  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int e0 = cell_base + tile * C;
    const int nc = min(C, cell_end - e0);
    if (tid == 0 && tile + (int)gridDim.x < ntiles) {
      // the next tile's remaining inputs (contiguous cell ranges) into L2 while this one runs
      const size_t en = (size_t)cell_base + (size_t)(tile + gridDim.x) * C;
      const size_t nn = min((size_t)C, (size_t)cell_end - en), NS = (size_t)g.N * S;
      if (!L::STG) mxd::prefetch_l2(U, NS * nv * 8, en * S * nv * 8, nn * S * nv * 8);
      if (visc && !L::STG) mxd::prefetch_l2(mo.invs, NS * 48, en * S * 48, nn * S * 48);
      if (nut && !L::STG) mxd::prefetch_l2(nut, NS * 8, en * S * 8, nn * S * 8);
    }
    if constexpr (L::STG) {
      cp_async_wait0();  // this thread's copies of the tile
      __syncthreads();   // everyone's
    }
    // nu_t of the tile's point t = c*S + s
    auto nut_at = [&](int c, int s) -> double {
      return L::STG ? sStg[C * S * 8 + c * S + s] : nut[(size_t)(e0 + c) * S + s];
    };
    // primitives and temperature in FP64
    for (int t = tid; t < C * S; t += MX_THREADS) {
      const int c = t % C, s = t / C;
      double q[6] = {1.0, 0.0, 0.0, 0.0, 1.0, 1.0};
      if (c < nc) mxd::prim_T(L::STG ? sStg + (c * S + s) * nv : U + ((size_t)(e0 + c) * S + s) * nv, q);
#pragma unroll
      for (int v = 0; v < 6; ++v) sQ[(c * S + s) * 6 + v] = q[v];
    }
    __syncthreads();
    // cell means of q (5) and of u, v, w, T (4)
    for (int t = tid; t < C * 9; t += MX_THREADS) {
      const int c = t / 9, k = t % 9;
      const int col = k < 5 ? k : (k < 8 ? k - 4 : 5);
      double acc = 0.0;
      for (int s = 0; s < S; ++s) acc += sQ[(c * S + s) * 6 + col];
      sM[c * 9 + k] = acc * (1.0 / S);
    }
    __syncthreads();
    for (int t = tid; t < C * S; t += MX_THREADS) {
      const int c = t % C, s = t / C;
      const double* q = sQ + (c * S + s) * 6;
      if (c < nc) {
        const float mutf = (visc && nut) ? float(q[0] * nut_at(c, s)) : 0.f;
        float* o = mb.PFm + ((size_t)(e0 + c) * S + s) * MX_PF;
        *reinterpret_cast<float2*>(o + 10) = make_float2(float(q[0]), float(q[1]));
        *reinterpret_cast<float4*>(o + 12) = make_float4(float(q[2]), float(q[3]), float(q[4]), 0.f);
        o[9] = mutf;
      }
      if (visc) {
        const double phi[4] = {q[1], q[2], q[3], q[5]};
#pragma unroll
        for (int f = 0; f < 4; ++f)
          mxd::st_split(sA1, 128 * Sq, tc::kmajor_index(f * C + c, s, 128), float(phi[f] - sM[c * 9 + 5 + f]));
        const double mut = (c < nc && nut) ? q[0] * nut_at(c, s) : 0.0;
        mxd::st_split(sB2, NB2 * Sq, tc::kmajor_index(14 * C + c, s, NB2), float(mut));
      }
#pragma unroll
      for (int v = 0; v < 5; ++v)
        mxd::st_split(sB2, NB2 * Sq, tc::kmajor_index(v * C + c, s, NB2), float(q[v] - sM[c * 9 + v]));
    }
    tc::fence_async_smem();
    __syncthreads();
    if (tile + (int)gridDim.x < ntiles) stage(tile + (int)gridDim.x);  // the staging buffer is free again
    if (visc) {
      if (tid == 0) {
        tc::fence_after();
        mxd::mma_split(tmem, sA1, sB1, L::NB1, Sq);
        tc::commit(&bar);
        if (!mxd::wait_commit(&bar, phase, status)) abort_flag = 1;
      }
      __syncthreads();
      if (abort_flag) break;
      tc::fence_after();
      // rows phi*8 + c live in TMEM lanes 0..31: warps 0 and 4 split the columns
      if ((warp & 3) == 0) {
        const int f = lane / C, c = lane % C;
        for (int ch = warp >> 2; ch < L::NB1 / 8; ch += MX_THREADS / 128) {
          float v8[8];
          tc::tmem_ld8(tmem + ch * 8, v8);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int n = ch * 8 + j, m = n / Sq, s = n % Sq;
            if (s < S) sG[((c * S + s) * 3 + m) * 4 + f] = v8[j];
          }
        }
      }
      __syncthreads();
      // physical gradients (core/fr_operators/gradients.py:23-64) and mu_t
      for (int t = tid; t < C * S; t += MX_THREADS) {
        const int c = t % C, s = t / C;
        float gr[12], pf[9];
        if (c < nc) {
          const float4* inv = L::STG ? sInvs + (c * S + s) * 3 : mo.invs + ((size_t)(e0 + c) * S + s) * 3;
          float iv[9];
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const float4 x = L::STG ? inv[m] : __ldg(inv + m);
            iv[m * 3 + 0] = x.x;
            iv[m * 3 + 1] = x.y;
            iv[m * 3 + 2] = x.z;
          }
          const float* gs = sG + (c * S + s) * 12;
#pragma unroll
          for (int f = 0; f < 4; ++f)
#pragma unroll
            for (int n = 0; n < 3; ++n)
              gr[f * 3 + n] = gs[0 * 4 + f] * iv[0 * 3 + n] + gs[1 * 4 + f] * iv[1 * 3 + n] + gs[2 * 4 + f] * iv[2 * 3 + n];
          pf[0] = gr[0];
          pf[1] = gr[4];
          pf[2] = gr[8];
          pf[3] = 0.5f * (gr[1] + gr[3]);
          pf[4] = 0.5f * (gr[2] + gr[6]);
          pf[5] = 0.5f * (gr[5] + gr[7]);
#pragma unroll
          for (int n = 0; n < 3; ++n) pf[6 + n] = gr[9 + n];
          float* o = mb.PFm + ((size_t)(e0 + c) * S + s) * MX_PF;
          *reinterpret_cast<float4*>(o) = make_float4(pf[0], pf[1], pf[2], pf[3]);
          *reinterpret_cast<float4*>(o + 4) = make_float4(pf[4], pf[5], pf[6], pf[7]);
          o[8] = pf[8];
        } else {
#pragma unroll
          for (int k = 0; k < 9; ++k) pf[k] = 0.f;
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) mxd::st_split(sB2, NB2 * Sq, tc::kmajor_index((5 + k) * C + c, s, NB2), pf[k]);
      }
      tc::fence_async_smem();
      __syncthreads();
      if (tile + (int)gridDim.x < ntiles) stage_inv(tile + (int)gridDim.x);  // the rows are consumed
    }
    // extrapolation of every field to all face points: D[fp][f*8+c]
    if (tid == 0) {
      tc::fence_after();
      mxd::mma_split(tmem, sA2, sB2, NB2, Sq);
      tc::commit(&bar);
      if (!mxd::wait_commit(&bar, phase, status)) abort_flag = 1;
    }
    __syncthreads();
    if (abort_flag) break;
    tc::fence_after();
    {
      // copy j of the face-point rows (lanes j*128/DUP ...) serves cells
      // [j*C/DUP, (j+1)*C/DUP); the quarters of one copy split its face points
      constexpr int DUP = mx_ext_dup(NFP), QPC = 4 / DUP, CPC = C / DUP;
      const int q4 = warp & 3, j = q4 / QPC, fp = (q4 % QPC) * 32 + lane;
      if ((q4 % QPC) * 32 < NFP) {
        for (int f = warp >> 2; f < nfw; f += MX_THREADS / 128) {
          float vc[CPC];  // this copy's cells only (fixed register indices)
          tc::tmem_ldn<CPC>(tmem + ((uint32_t)(q4 * 32) << 16) + f * 8 + j * CPC, vc);
          if (fp < NFP) {
#pragma unroll
            for (int cc = 0; cc < CPC; ++cc) {
              const int c = j * CPC + cc;
              if (c < nc) {
                const float val = f < 5 ? float(sM[c * 9 + f] + (double)vc[cc]) : vc[cc];
                mb.XF[(((size_t)(e0 + c) * 6 + fp / NP) * FW + f) * NP + fp % NP] = val;
              }
            }
          }
        }
      }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
  }
  if constexpr (L::STG) cp_async_wait0();  // copies still in flight after an aborted tile
  tc::fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, L::NCOL);
  }
}

// ---------------------------------------------------------------------------
// face kernel: one thread per pair of slot points (or single slot point), fields read at face points
// ---------------------------------------------------------------------------
// The jumps of slot point t from its own face-point fields ow and the other
// side's ot (core/fr_residual/inviscid_kernel_colored.py:86-236,
// core/fr_residual/viscous_flux_kernel.py:335-520)
template <int NP>
__device__ __forceinline__ void mx_face_jump(const Faces& fc, const SlotTable& st, const MxFace& mf, const MxBuf& mb,
                                             const double* __restrict__ hcell, float mu, int visc, int t, float side,
                                             bool bnd, const float (&ow)[MX_XF], const float (&ot)[MX_XF]) {
  const int sl = t / NP, i = t % NP;
  const float4 ar = mf.arow[t];
  const float a0 = ar.x, a1 = ar.y, a2 = ar.z;
  const float mag = fmaxf(fabsf(ar.w), 1e-30f);
  // divided, not multiplied by 1 / mag: the second rounding would show in the
  // step's error (P1: 6.8e-9 -> 7.3e-9)
  float dir[3] = {a0 / mag * side, a1 / mag * side, a2 / mag * side};
  if (ar.w < 0.f) {  // alignment fallback: the face normal, outward from this side
    const int f = st.face[sl];
    const double* tnp = fc.tnormal + ((size_t)f * NP + i) * 3;
    const float sg = (st.flags[sl] & 1) == 0 ? 1.f : -1.f;
#pragma unroll
    for (int d = 0; d < 3; ++d) dir[d] = sg * float(tnp[d]);
  }
  float Fc[5], Fp[3][5];
  ausm_up<float>(ow, ot, dir, Fc);
  euler_flux<float>(ow, Fp);
  float* Jo = mb.Jm + (size_t)sl * 9 * NP + i;
#pragma unroll
  for (int v = 0; v < 5; ++v) Jo[v * NP] = Fc[v] * mag * side - (a0 * Fp[0][v] + a1 * Fp[1][v] + a2 * Fp[2][v]);
  if (visc) {
    float av[MX_XF];  // the common flux: both sides' averages
#pragma unroll
    for (int k = 1; k < MX_XF; ++k) av[k] = 0.5f * (ow[k] + ot[k]);
    float Gc[3][4], Go[3][4];
    viscous_flux_sym<float>(av + 1, av + 5, av + 11, mu, av[14], Gc);
    viscous_flux_sym<float>(ow + 1, ow + 5, ow + 11, mu, ow[14], Go);
    float jv[4];  // momentum and energy (no viscous mass flux)
#pragma unroll
    for (int v = 0; v < 4; ++v)
      jv[v] = (a0 * Gc[0][v] + a1 * Gc[1][v] + a2 * Gc[2][v]) - (a0 * Go[0][v] + a1 * Go[1][v] + a2 * Go[2][v]);
    if (bnd) {
      // interior penalty (core/fr_operators/flux_kernels.py:140-200)
      const float eta = float(C_IP) * (mu + ow[14]) / float(hcell[st.cell[sl]]);
      const float scale = eta * fabsf(ar.w) * side;
#pragma unroll
      for (int v = 0; v < 3; ++v) jv[v] += -scale * (ow[1 + v] - ot[1 + v]);
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) Jo[(5 + v) * NP] = jv[v];
  }
}

// face point fp = (axis*2+side)*NP + i of cell e: field k at [k * NP]
template <int NP>
__device__ __forceinline__ const float* mx_face_row(const MxBuf& mb, int e, int fp) {
  return mb.XF + ((size_t)e * 6 + fp / NP) * mb.FW * NP + fp % NP;
}

// a slot point outside the pairs (boundary, interpolated or without a matched
// partner)
template <int S, int NP>
__device__ __forceinline__ void mx_face_single(const Faces& fc, const Bc& bc, const SlotTable& st, const MxFace& mf,
                                               const MxBuf& mb, const double* __restrict__ hcell, float mu, int visc,
                                               int t) {
  const int sl = t / NP, i = t % NP;
  const int f = st.face[sl];
  const int e = st.cell[sl];
  const int fl = st.flags[sl];
  const bool is_owner = (fl & 1) == 0;
  const bool bnd = (fl & 2) != 0;
  const int ax = (fl >> 2) & 3;
  const int nf = visc ? MX_XF : 5;
  float ow[MX_XF], ot[MX_XF];
  {
    const float* xo = mx_face_row<NP>(mb, e, (ax * 2 + ((fl & 16) ? 1 : 0)) * NP + i);
#pragma unroll
    for (int k = 0; k < MX_XF; ++k) ow[k] = k < nf ? __ldg(xo + k * NP) : 0.f;
  }
  const double* tnp = fc.tnormal + ((size_t)f * NP + i) * 3;
  const float tn[3] = {float(tnp[0]), float(tnp[1]), float(tnp[2])};
  if (bnd) {
    float gq[5];
    ghost_state<float>(bc, fc.bc_group[f], ow, tn, gq);
#pragma unroll
    for (int v = 0; v < 5; ++v) ot[v] = gq[v];
#pragma unroll
    for (int k = 5; k < MX_XF; ++k) ot[k] = ow[k];
  } else if (mf.ofp[t] != MX_OFP_GENERAL) {
    // matched rows come from the record's other cell (either source slot may hold them)
    const int oc = is_owner ? fc.neighbor[f] : fc.owner[f];
    const float* xn = mx_face_row<NP>(mb, oc, mf.ofp[t]);
#pragma unroll
    for (int k = 0; k < MX_XF; ++k) ot[k] = k < nf ? __ldg(xn + k * NP) : 0.f;
  } else {
    // interpolation from the source cells' point fields (sum src0 then src1,
    // zero weights skipped as in core/fr_residual/inviscid_kernel_colored.py:117-121)
#pragma unroll
    for (int k = 0; k < MX_XF; ++k) ot[k] = 0.f;
    for (int src = 0; src < 2; ++src) {
      const int c = src == 0 ? st.c0[sl] : st.c1[sl];
      if (c < 0) continue;
      const double* M = src == 0 ? (is_owner ? fmat(fc.nb_m0, fc.nb_m0i, f, i, NP, S)
                                             : fmat(fc.ow_m0, fc.ow_m0i, f, i, NP, S))
                                 : (is_owner ? fmat(fc.nb_m1, fc.nb_m1i, st.i1[sl], i, NP, S)
                                             : fmat(fc.ow_m1, fc.ow_m1i, st.i1[sl], i, NP, S));
      const float* pf = mb.PFm + (size_t)c * S * MX_PF;
      for (int s = 0; s < S; ++s) {
        const float w = float(__ldg(M + s * NP));
        if (w == 0.f) continue;
        const float4* p4 = reinterpret_cast<const float4*>(pf + s * MX_PF);
        const float4 x2 = __ldg(p4 + 2), x3 = __ldg(p4 + 3);
        ot[0] += w * x2.z; ot[1] += w * x2.w; ot[2] += w * x3.x; ot[3] += w * x3.y; ot[4] += w * x3.z;
        if (visc) {
          const float4 x0 = __ldg(p4), x1 = __ldg(p4 + 1);
          ot[5] += w * x0.x;  ot[6] += w * x0.y;  ot[7] += w * x0.z;  ot[8] += w * x0.w;
          ot[9] += w * x1.x;  ot[10] += w * x1.y; ot[11] += w * x1.z; ot[12] += w * x1.w;
          ot[13] += w * x2.x; ot[14] += w * x2.y;
        }
      }
    }
  }
  mx_face_jump<NP>(fc, st, mf, mb, hcell, mu, visc, t, (fl & 16) ? 1.f : -1.f, bnd, ow, ot);
}

// Matched interior face points in pairs: slot point t (owner side) and its
// partner t2 (the neighbour side's slot point at the matched face point) read
// the same two face-point rows, own and other swapped; one thread loads them
// once and forms both jumps.  The first rest_blocks CTAs take the points
// outside the pairs: one launch, so that their longer load chains run under
// the pairs instead of after them.  80 registers (three 256-thread CTAs).
template <int S, int NP>
__global__ void __launch_bounds__(256, 3) k_mx_face(Faces fc, Bc bc, SlotTable st, MxFace mf, MxBuf mb,
                                                    const double* __restrict__ hcell, float mu, int visc,
                                                    const int32_t* __restrict__ rest, int n_rest, int rest_blocks,
                                                    const MxPair* __restrict__ pairs, int n_pairs) {
  if ((int)blockIdx.x < rest_blocks) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n_rest) mx_face_single<S, NP>(fc, bc, st, mf, mb, hcell, mu, visc, rest[j]);
    return;
  }
  const int idx = ((int)blockIdx.x - rest_blocks) * blockDim.x + threadIdx.x;
  if (idx >= n_pairs) return;
  const int4 pr = __ldg(reinterpret_cast<const int4*>(pairs) + idx);
  const int nf = visc ? MX_XF : 5;
  float ra[MX_XF], rb[MX_XF];
  {
    const uint32_t r0 = (uint32_t)pr.z & 0x7fffffffu, r1 = (uint32_t)pr.w & 0x7fffffffu;
    const float* xa = mb.XF + (size_t)(r0 / NP) * mb.FW * NP + r0 % NP;
    const float* xb = mb.XF + (size_t)(r1 / NP) * mb.FW * NP + r1 % NP;
#pragma unroll
    for (int k = 0; k < MX_XF; ++k) {
      ra[k] = k < nf ? __ldg(xa + k * NP) : 0.f;
      rb[k] = k < nf ? __ldg(xb + k * NP) : 0.f;
    }
  }
  mx_face_jump<NP>(fc, st, mf, mb, hcell, mu, visc, pr.x, pr.z < 0 ? 1.f : -1.f, false, ra, rb);
  mx_face_jump<NP>(fc, st, mf, mb, hcell, mu, visc, pr.y, pr.w < 0 ? 1.f : -1.f, false, rb, ra);
}

// ---------------------------------------------------------------------------
// volume kernel: persistent over C-cell tiles, tensor-core contractions.
// Writes the volume terms RV (N, 9, S) FP32: inviscid -(W*Ft + MD*F(qbar))/det
// (5) and the momentum and energy rows of the viscous D_3d*Gt/det (4).
// ---------------------------------------------------------------------------
constexpr int MX_VOL_THREADS = 512;

template <int S, int FN, int C>
struct MxVolSmem {
  static constexpr int Sq = pad16(S), Fq = pad16(FN);
  static constexpr bool VP = S <= 27;  // viscous terms built in (P1, P2)
  static constexpr int QS = Fq * 5 + 4;  // floats per cell of the fine-point deviations
  static constexpr int oBc = 0;
  static constexpr int oBW = oBc + Fq * Sq * 4;
  static constexpr int oBD = oBW + Sq * 3 * Fq * 4;
  static constexpr int oR1 = oBD + (VP ? Sq * 3 * Sq * 4 : 0);
  static constexpr int szAc = 128 * Sq * 4, szAD = VP ? 128 * 3 * Sq * 4 : 0, szAW = 128 * 3 * Fq * 4;
  static constexpr int szR1 = cmax(szAc + szAD, szAW);
  static constexpr int oR2 = oR1 + szR1;  // q (FP64) before the first product, then dq, then the RV tile
  static constexpr int szR2 = cmax(cmax(C * QS * 4, C * S * 5 * 8), C * S * 9 * 4);
  static constexpr int oX = oR2 + szR2;
  // doubles: qbar, F(qbar); with VP also det and the metric divergence of the tile
  static constexpr int nX = C * 5 + C * 15 + (VP ? C * S * 4 : 0);
  // the next tile's state rows (stride nv <= 8), 1/det and MD, copied
  // asynchronously (P1, P2; at P3 the tile's loads are direct: no room)
  static constexpr bool STG = VP;
  static constexpr int oStg = oX + nX * 8;
  static constexpr int nStg = STG ? C * S * 12 : 0;
  static constexpr int total = oStg + nStg * 8;
  // TMEM columns: each product holds two column blocks (stacked hi / lo operand)
  static constexpr int cFq = 0, cD3 = 2 * Fq, cW = 2 * Fq + (VP ? 2 * Sq : 0);
  static constexpr int NCOL = pow2_cols(cW + 2 * Sq);
  static_assert(cW + 2 * Sq <= NCOL, "tensor memory columns");
};

template <int S, int FN, int C>
__global__ void __launch_bounds__(MX_VOL_THREADS, 1)
    k_mx_vol(Geom g, MxOps mo, const double* __restrict__ Ucur, int nv, int inviscid_only, float mu,
             const float* __restrict__ PFm, float* __restrict__ RV, int cell_base, int cell_end, unsigned* status) {
  using L = MxVolSmem<S, FN, C>;
  constexpr int Sq = L::Sq, Fq = L::Fq, QS = L::QS, NT = MX_VOL_THREADS;
  static_assert(C % 8 == 0 && 5 * C <= 128, "tile rows (v, c) must fit 128 lanes in groups of 8 cells");
  static_assert(L::NCOL <= 256 && L::total <= 227 * 1024, "tensor memory / shared memory budget");
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t bar;
  __shared__ uint32_t tbase;
  __shared__ int abort_flag;
  uint16_t* sBc = reinterpret_cast<uint16_t*>(smem + L::oBc);
  uint16_t* sBW = reinterpret_cast<uint16_t*>(smem + L::oBW);
  uint16_t* sBD = reinterpret_cast<uint16_t*>(smem + L::oBD);
  uint16_t* sAc = reinterpret_cast<uint16_t*>(smem + L::oR1);
  uint16_t* sAD = reinterpret_cast<uint16_t*>(smem + L::oR1 + L::szAc);
  uint16_t* sAW = reinterpret_cast<uint16_t*>(smem + L::oR1);
  double* sQ = reinterpret_cast<double*>(smem + L::oR2);
  float* sQf = reinterpret_cast<float*>(smem + L::oR2);
  float* sR = reinterpret_cast<float*>(smem + L::oR2);
  double* sQb = reinterpret_cast<double*>(smem + L::oX);  // [c][5]
  double* sFb = sQb + C * 5;                              // [c][n][v] Euler flux at qbar
  double* sDet = sFb + C * 15;                            // [c][s] 1/det (VP)
  double* sMD = sDet + C * S;                             // [c][s][3] (VP)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool visc = L::VP && !inviscid_only;
  const int ct = cell_type(g, cell_base);

  mxd::copy_img(sBc, (ct ? mo.c2f[1] : mo.c2f[0]), Fq * Sq * 4);
  mxd::copy_img(sBW, (ct ? mo.W[1] : mo.W[0]), Sq * 3 * Fq * 4);
  if (visc) mxd::copy_img(sBD, (ct ? mo.D3[1] : mo.D3[0]), Sq * 3 * Sq * 4);
  if (warp == 0) tc::tmem_alloc(&tbase, L::NCOL);
  if (tid == 0) {
    tc::mbar_init(&bar, 1);
    tc::fence_mbar_init();
    abort_flag = 0;
  }
  tc::fence_async_smem();
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tbase;
  uint32_t phase = 0;
  const int ntiles = (cell_end - cell_base + C - 1) / C;
  const int q4 = warp & 3;                      // TMEM lane quarter of this warp
  const int lrow = q4 * 32 + lane;              // TMEM lane of this thread
  const uint32_t lane_base = (uint32_t)(q4 * 32) << 16;
  const int wsplit = warp >> 2, nsplit = NT / 128;  // warps sharing a lane quarter split the columns

  // asynchronous copies of a tile's contiguous state, 1/det and MD blocks into
  // the staging buffer; issued one tile ahead, so they overlap the tile before
  double* sStg = reinterpret_cast<double*>(smem + L::oStg);
  auto stage = [&](int tl) {
    if constexpr (L::STG) {
      const size_t eb = (size_t)cell_base + (size_t)tl * C;
      const int nn = min(C, cell_end - (int)eb);
      const double* ub = Ucur + eb * S * nv;
      for (int t = tid; t < nn * S * nv; t += NT) cp_async8(sStg + t, ub + t);
      for (int t = tid; t < nn * S; t += NT) cp_async8(sStg + C * S * 8 + t, mo.rdet + eb * S + t);
      for (int t = tid; t < nn * S * 3; t += NT) cp_async8(sStg + C * S * 9 + t, mo.MD + eb * S * 3 + t);
      cp_async_commit();
    }
  };
  if (blockIdx.x < ntiles) stage(blockIdx.x);

  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int e0 = cell_base + tile * C;
    const int nc = min(C, cell_end - e0);
    if (tid == 0 && tile + (int)gridDim.x < ntiles) {
      // the next tile's remaining inputs (contiguous cell ranges) into L2 while this one runs
      const size_t en = (size_t)cell_base + (size_t)(tile + gridDim.x) * C;
      const size_t nn = min((size_t)C, (size_t)cell_end - en), NS = (size_t)g.N * S;
      mxd::prefetch_l2(mo.adjf, (size_t)g.N * FN * 48, en * FN * 48, nn * FN * 48);
      if (!L::STG) mxd::prefetch_l2(Ucur, NS * nv * 8, en * S * nv * 8, nn * S * nv * 8);
      if (visc) {
        mxd::prefetch_l2(PFm, NS * MX_PF * 4, en * S * MX_PF * 4, nn * S * MX_PF * 4);
        mxd::prefetch_l2(mo.adjs, NS * 48, en * S * 48, nn * S * 48);
      }
    }
    if constexpr (L::STG) {
      cp_async_wait0();  // this thread's copies of the tile
      __syncthreads();   // everyone's
    }
    // ---- primitives (FP64), det and metric divergence of the tile ----
    for (int t = tid; t < C * S; t += NT) {
      const int c = t / S;
      double q[6] = {1.0, 0.0, 0.0, 0.0, 1.0, 1.0};
      if (c < nc) {
        mxd::prim_T(L::STG ? sStg + t * nv : Ucur + ((size_t)e0 * S + t) * nv, q);
        if (L::VP) {
          sDet[t] = sStg[C * S * 8 + t];  // reciprocal: the readouts multiply
          sMD[t * 3 + 0] = sStg[C * S * 9 + t * 3 + 0];
          sMD[t * 3 + 1] = sStg[C * S * 9 + t * 3 + 1];
          sMD[t * 3 + 2] = sStg[C * S * 9 + t * 3 + 2];
        }
      }
#pragma unroll
      for (int v = 0; v < 5; ++v) sQ[t * 5 + v] = q[v];
    }
    __syncthreads();
    if (tile + (int)gridDim.x < ntiles) stage(tile + (int)gridDim.x);  // the staging buffer is free again
    for (int t = tid; t < C * 5; t += NT) {
      const int c = t / 5, v = t % 5;
      double acc = 0.0;
      for (int s = 0; s < S; ++s) acc += sQ[(c * S + s) * 5 + v];
      sQb[t] = acc * (1.0 / S);
    }
    __syncthreads();
    for (int c = tid; c < C; c += NT) {
      double F[3][5];
      euler_flux<double>(sQb + c * 5, F);
#pragma unroll
      for (int n = 0; n < 3; ++n)
#pragma unroll
        for (int v = 0; v < 5; ++v) sFb[c * 15 + n * 5 + v] = F[n][v];
    }
    // ---- A operands: q - qbar at the solution points; contravariant viscous flux ----
    for (int idx = tid; idx < C * Sq; idx += NT) {
      int c, s;
      mxd::cell_point(idx, Sq, c, s);
      const bool live = c < nc && s < S;
#pragma unroll
      for (int v = 0; v < 5; ++v)
        mxd::st_split(sAc, 128 * Sq, tc::kmajor_index(v * C + c, s, 128),
                      live ? float(sQ[(c * S + s) * 5 + v] - sQb[c * 5 + v]) : 0.f);
      if (visc) {
        float Gt[3][5];
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
          for (int v = 0; v < 5; ++v) Gt[m][v] = 0.f;
        if (live) {
          const size_t p = (size_t)(e0 + c) * S + s;
          const float4* pf = reinterpret_cast<const float4*>(PFm + p * MX_PF);
          const float4 g0 = __ldg(pf), g1 = __ldg(pf + 1), g2 = __ldg(pf + 2);
          const float4* am = mo.adjs + p * 3;
          float vel[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) vel[d] = float(sQ[(c * S + s) * 5 + 1 + d]);
          const float sg[6] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y};
          const float gT[3] = {g1.z, g1.w, g2.x};
          float G[3][4];
          viscous_flux_sym<float>(vel, sg, gT, mu, g2.y, G);
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const float4 x = __ldg(am + m);
#pragma unroll
            for (int v = 0; v < 4; ++v) Gt[m][1 + v] = x.x * G[0][v] + x.y * G[1][v] + x.z * G[2][v];
          }
        }
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
          for (int v = 0; v < 5; ++v)
            mxd::st_split(sAD, 128 * 3 * Sq, tc::kmajor_index(v * C + c, m * Sq + s, 128), Gt[m][v]);
      }
    }
    // the fine-point adjugate rows of this thread's flux items, loaded now so
    // that their latency overlaps the products and the readout below
    constexpr int NFI = (C * Fq + NT - 1) / NT;
    float4 adf[NFI][3];
#pragma unroll
    for (int k = 0; k < NFI; ++k) {
      const int idx = tid + k * NT;
      int c, i;
      mxd::cell_point(idx, Fq, c, i);
      const bool live = idx < C * Fq && c < nc && i < FN;
      const float4* ad = mo.adjf + ((size_t)(e0 + (live ? c : 0)) * FN + (live ? i : 0)) * 3;
#pragma unroll
      for (int m = 0; m < 3; ++m) adf[k][m] = live ? __ldg(ad + m) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    tc::fence_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc::fence_after();
      mxd::mma_cat(tmem + L::cFq, sAc, sBc, Fq, Sq);
      if (visc) mxd::mma_cat(tmem + L::cD3, sAD, sBD, Sq, 3 * Sq);
      tc::commit(&bar);
      if (!mxd::wait_commit(&bar, phase, status)) abort_flag = 1;
    }
    __syncthreads();
    if (abort_flag) break;
    tc::fence_after();
    // ---- fine-point deviations dq = c2f*(q - qbar): TMEM -> shared ----
    if (q4 * 32 < 5 * C) {
      for (int ch = wsplit; ch < Fq / 8; ch += nsplit) {
        float v8[8], w8[8];
        tc::tmem_ld8(tmem + lane_base + L::cFq + ch * 8, v8);
        tc::tmem_ld8(tmem + lane_base + L::cFq + Fq + ch * 8, w8);
        if (lrow < 5 * C) {
          const int v = lrow / C, c = lrow % C;
#pragma unroll
          for (int j = 0; j < 8; ++j) sQf[c * QS + (ch * 8 + j) * 5 + v] = v8[j] + w8[j];
        }
      }
    }
    __syncthreads();
    // ---- contravariant Euler flux deviations at the fine points -> A_W ----
#pragma unroll
    for (int k = 0; k < NFI; ++k) {
      const int idx = tid + k * NT;
      if (idx >= C * Fq) break;
      int c, i;
      mxd::cell_point(idx, Fq, c, i);
      float Ft[3][5];
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int v = 0; v < 5; ++v) Ft[m][v] = 0.f;
      if (c < nc && i < FN) {
        float qb[5], dq[5], dF[3][5];
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          qb[v] = float(sQb[c * 5 + v]);
          dq[v] = sQf[c * QS + i * 5 + v];
        }
        mxd::euler_flux_delta(qb, dq, dF);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          const float4 x = adf[k][m];
#pragma unroll
          for (int v = 0; v < 5; ++v) Ft[m][v] = x.x * dF[0][v] + x.y * dF[1][v] + x.z * dF[2][v];
        }
      }
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int v = 0; v < 5; ++v)
          mxd::st_split(sAW, 128 * 3 * Fq, tc::kmajor_index(v * C + c, m * Fq + i, 128), Ft[m][v]);
    }
    tc::fence_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc::fence_after();
      mxd::mma_cat(tmem + L::cW, sAW, sBW, Sq, 3 * Fq);
      tc::commit(&bar);
    }
    // viscous divergence while the W product runs (its columns are complete);
    // the dq tile is consumed, so the RV tile reuses its space
    if (q4 * 32 < 5 * C) {
      for (int ch = wsplit; ch < Sq / 8; ch += nsplit) {
        float v8[8], w8[8];
        if (visc) {
          tc::tmem_ld8(tmem + lane_base + L::cD3 + ch * 8, v8);
          tc::tmem_ld8(tmem + lane_base + L::cD3 + Sq + ch * 8, w8);
        }
        if (lrow < 5 * C) {
          const int v = lrow / C, c = lrow % C;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int s = ch * 8 + j;
            if (s < S && c < nc && v > 0)
              sR[(c * 9 + 4 + v) * S + s] = visc ? float(double(v8[j] + w8[j]) * sDet[c * S + s]) : 0.f;
          }
        }
      }
    }
    if (tid == 0 && !mxd::wait_commit(&bar, phase, status)) abort_flag = 1;
    __syncthreads();
    if (abort_flag) break;
    tc::fence_after();
    // ---- inviscid volume term: -(W*dFt + MD*F(qbar)) / det ----
    if (q4 * 32 < 5 * C) {
      for (int ch = wsplit; ch < Sq / 8; ch += nsplit) {
        float v8[8], w8[8];
        tc::tmem_ld8(tmem + lane_base + L::cW + ch * 8, v8);
        tc::tmem_ld8(tmem + lane_base + L::cW + Sq + ch * 8, w8);
        if (lrow < 5 * C) {
          const int v = lrow / C, c = lrow % C;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int s = ch * 8 + j;
            if (s < S && c < nc) {
              const size_t p = (size_t)(e0 + c) * S + s;
              const double* md = L::VP ? sMD + (c * S + s) * 3 : mo.MD + p * 3;
              const double rdj = L::VP ? sDet[c * S + s] : __ldg(mo.rdet + p);
              const double mdf = md[0] * sFb[c * 15 + v] + md[1] * sFb[c * 15 + 5 + v] + md[2] * sFb[c * 15 + 10 + v];
              sR[(c * 9 + v) * S + s] = float(-(double(v8[j] + w8[j]) + mdf) * rdj);
            }
          }
        }
      }
    }
    __syncthreads();
    // coalesced store of the tile's volume terms (cells e0 .. e0+nc are contiguous)
    mxd::copy_f32(RV + (size_t)e0 * S * 9, sR, nc * S * 9);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
  }
  if constexpr (L::STG) cp_async_wait0();  // copies still in flight after an aborted tile
  tc::fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, L::NCOL);
  }
}

// ---------------------------------------------------------------------------
// update kernel: a warp owns CW whole cells from load to store.  Lifting of the
// face jumps in ascending color order, outlier zeroing, then the SSP-RK3
// combination, positivity and filter in FP64 (or the residual-only outputs).
//
// A lane owns a solution point (S <= 27; two at S = 64; four cells side by
// side at S = 8), so the residual, the outlier test and the RK combination
// stay in registers and the phases need no block barrier: the block-wide form
// of this kernel spent 2,600 instructions per P2 cell, most of them index
// arithmetic around shared-memory tiles.  The volume terms and the jumps are
// stored field-major (planes of points), so every load of a lane's values is
// one coalesced access.  CW = 3 at P2 and P3 makes the filter's 5*CW = 15
// columns two nearly full column tiles of the FP64 tensor product.
// ---------------------------------------------------------------------------
constexpr int MX_UPD_SLOTS = 5;  // slots of a prism, whose jumps are loaded together (other counts: one by one)

template <int S>
struct MxUpd {
  static constexpr int PL = (S + 31) / 32;            // points per lane
  static constexpr int CPR = S < 32 ? 32 / S : 1;     // cells side by side in a warp
  static constexpr int CW = S == 8 ? 8 : 3;           // cells per warp
  static constexpr int PR = CW / CPR;                 // rounds
  static_assert(CW % CPR == 0, "whole rounds");
  // shared memory: g' per (side, axis, point), face point per (axis, point);
  // per warp two state tiles (current state, then the filtered one; step-start state, then the output)
  static constexpr int tab = 6 * S * 8 + (3 * S * 4 + 15) / 16 * 16;
  __host__ __device__ static constexpr int warp_bytes(int nv) { return 2 * CW * S * nv * 8; }
  static constexpr int bytes(int nv, int warps) { return tab + warps * warp_bytes(nv); }
};

namespace mxd {

// maximum over the lanes of a cell
template <int S>
__device__ __forceinline__ unsigned cell_max(unsigned x) {
  if constexpr (S == 8) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) x = max(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
  } else {
    return __reduce_max_sync(0xffffffffu, x);
  }
}

// lanes of this cell where p holds
template <int S>
__device__ __forceinline__ unsigned cell_ballot(bool p, int grp) {
  const unsigned b = __ballot_sync(0xffffffffu, p);
  return S == 8 ? (b >> (8 * grp)) & 0xffu : b;
}

template <int S>
__device__ __forceinline__ double cell_sum(double x) {
#pragma unroll
  for (int o = 1; o < (S == 8 ? 8 : 32); o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// True when the outlier rule (|R| > 1e4 * max(median |R|, 1e-9 mean |U|,
// 1e-300) is zeroed, core/fr_operators/troubled_cell.py:346-408) provably
// zeroes nothing of a column: at least as many values as lie at or above the
// median's rank reach 1e-4 of an upper bound of the largest one.  The bound is
// the largest high word plus one, so one integer maximum and one ballot
// decide; columns that fail (or hold a NaN or infinity) take outlier_exact.
template <int S, int PL>
__device__ __forceinline__ bool outlier_clear(const double (&x)[PL], const bool (&on)[PL], int grp) {
  constexpr int NEED = S - ((S & 1) ? S / 2 : S / 2 - 1);
  unsigned hw = 0u;
#pragma unroll
  for (int l = 0; l < PL; ++l) hw = max(hw, on[l] ? (unsigned)__double2hiint(x[l]) & 0x7fffffffu : 0u);
  hw = cell_max<S>(hw);
  const bool finite = hw < 0x7fe00000u;  // no early return: every lane of the warp takes part in the ballots
  const double hi = __hiloint2double((int)hw + 1, 0);
  const double p = hi * 1.0000000001e-4;  // 1e4 * p >= hi after rounding
  int cnt = 0;
#pragma unroll
  for (int l = 0; l < PL; ++l) cnt += __popc(cell_ballot<S>(on[l] && fabs(x[l]) >= p, grp));
  return finite && (cnt >= NEED || hi <= 1e-297);
}

// the rule itself: stable ranks over the cell's points, median, zeroing
// (a call: kept out of the registers of the common path)
template <int PL>
struct Vals {
  double v[PL];
};
template <int S, int PL>
__device__ __noinline__ Vals<PL> outlier_exact(Vals<PL> X, Vals<PL> u, int grp, int s0, bool live) {
  double(&x)[PL] = X.v;
  bool on[PL];
#pragma unroll
  for (int l = 0; l < PL; ++l) on[l] = live && s0 + 32 * l < S;
  double acc = 0.0;
#pragma unroll
  for (int l = 0; l < PL; ++l) acc += on[l] ? fabs(u.v[l]) : 0.0;
  const double mean = cell_sum<S>(acc) / S;
  int rank[PL];
#pragma unroll
  for (int l = 0; l < PL; ++l) rank[l] = 0;
  for (int j = 0; j < S; ++j) {
    double src = x[0];
    if constexpr (PL > 1) src = j >= 32 ? x[PL - 1] : x[0];
    const double y = fabs(__shfl_sync(0xffffffffu, src, (S == 8 ? 8 * grp : 0) + (j & 31)));
#pragma unroll
    for (int l = 0; l < PL; ++l) {
      const double a = fabs(x[l]);
      rank[l] += (y < a) || (y == a && j < s0 + 32 * l);
    }
  }
  auto at_rank = [&](int r) {  // |x| of the point with rank r (0 where a NaN leaves none)
    double v = 0.0;
#pragma unroll
    for (int l = 0; l < PL; ++l) {
      const unsigned b = cell_ballot<S>(on[l] && rank[l] == r, grp);
      const double y = fabs(__shfl_sync(0xffffffffu, x[l], (S == 8 ? 8 * grp : 0) + (b ? __ffs(b) - 1 : 0)));
      if (b) v = y;
    }
    return v;
  };
  const double med = (S & 1) ? at_rank(S / 2) : 0.5 * (at_rank(S / 2 - 1) + at_rank(S / 2));
  const double thr = 1e4 * fmax(fmax(med, 1e-9 * mean), 1e-300);
#pragma unroll
  for (int l = 0; l < PL; ++l)
    if (fabs(x[l]) > thr) x[l] = 0.0;
  return X;
}
}  // namespace mxd

// T: float (mixed form) or double (plain form of structured prisms).  Register
// caps from timing four, five and six CTAs per SM: P2 float 203 us at five (214
// at six, 221 at four; 91,200 prisms), P1 float 131 us at six (135 at five; 256,000),
// P2 double 54 us at four (60 at three; 17,280).
template <int S, int NP, class T>
__global__ void __launch_bounds__(128, S == 64 ? 3 : (sizeof(T) == 8 ? 4 : (S == 8 ? 6 : 5)))
    k_update(Ops ops, Faces fc, StageArgs a, int ct, const T* __restrict__ RV, const T* __restrict__ Jm,
             const double* __restrict__ rdet) {
  using L = MxUpd<S>;
  constexpr int PL = L::PL, CPR = L::CPR, CW = L::CW, PR = L::PR;
  extern __shared__ __align__(16) uint8_t smb[];
  double* sG = reinterpret_cast<double*>(smb);
  int* sFp = reinterpret_cast<int*>(smb + 6 * S * 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nv = a.nv;
  for (int t = threadIdx.x; t < 3 * S; t += blockDim.x) {
    const int co = ops.dist_co[t];
    sG[t] = ops.g_left[co];
    sG[3 * S + t] = ops.g_right[co];
    sFp[t] = ops.dist_fp[t];
  }
  __syncthreads();
  const int e0 = a.cell_base + (blockIdx.x * (blockDim.x >> 5) + warp) * CW;
  const int nc = min(CW, a.cell_end - e0);
  if (nc <= 0) return;  // whole warps; no block barrier below
  double* sU = reinterpret_cast<double*>(smb + L::tab + warp * L::warp_bytes(nv));
  double* s0 = sU + CW * S * nv;
  const bool visc = !a.inviscid_only;
  const bool step = a.stage >= 0;
  if (step) {
    const double* uc = a.Ucur + (size_t)e0 * S * nv;
    for (int t = lane; t < nc * S * nv; t += 32) cp_async8(sU + t, uc + t);
    if (a.stage > 0) {  // stage 0 starts from the current state
      const double* u0 = a.U0 + (size_t)e0 * S * nv;
      for (int t = lane; t < nc * S * nv; t += 32) cp_async8(s0 + t, u0 + t);
    }
    cp_async_commit();
  }
  const int grp = S < 32 ? lane / S : 0;  // cell side of the warp
  const int sp = S < 32 ? lane % S : lane;
  // slot ranges (lane c: cell c's first slot) and flags (lane j: slots kb + j and kb + 32 + j)
  const int ptr = __ldg(fc.slot_ptr + e0 + min(lane, nc));
  const int kb = __shfl_sync(0xffffffffu, ptr, 0), ke = __shfl_sync(0xffffffffu, ptr, nc);
  const bool flags_held = ke - kb <= (CW * MX_UPD_SLOTS > 32 ? 64 : 32);
  const int fl = kb + lane < ke ? __ldg(a.slot_flags + kb + lane) : 0;
  const int fl2 = kb + 32 + lane < ke ? __ldg(a.slot_flags + kb + 32 + lane) : 0;
#pragma unroll 1
  for (int r = 0; r < PR; ++r) {
    const int c = r * CPR + (grp < CPR ? grp : 0);
    const bool live = grp < CPR && c < nc;
    const int e = e0 + (c < nc ? c : 0);  // lanes without a cell read one that exists
    double x[9][PL];  // dU/dt: inviscid 0..4, viscous momentum and energy 5..8
    double rd[PL];
    bool on[PL];
#pragma unroll
    for (int l = 0; l < PL; ++l) on[l] = live && sp + 32 * l < S;
    double cx[9][PL];
#pragma unroll
    for (int v = 0; v < 9; ++v)
#pragma unroll
      for (int l = 0; l < PL; ++l) cx[v][l] = 0.0;
    const int k0 = __shfl_sync(0xffffffffu, ptr, c < nc ? c : 0);
    const int n = __shfl_sync(0xffffffffu, ptr, (c < nc ? c : 0) + 1) - k0;
    T rv[9][PL];
#pragma unroll
    for (int l = 0; l < PL; ++l) {
      rd[l] = __ldg(rdet + (size_t)e * S + sp + 32 * l);
#pragma unroll
      for (int v = 0; v < 9; ++v)
        rv[v][l] = v < 5 || visc ? __ldg(RV + ((size_t)e * 9 + v) * S + sp + 32 * l) : T(0);
    }
    // jumps of the cell's slots, ascending color order
    if (flags_held && __all_sync(0xffffffffu, n == MX_UPD_SLOTS)) {
      // five slots, as every prism has: all loads of a point in flight at once
#pragma unroll
      for (int l = 0; l < PL; ++l) {
        T jv[MX_UPD_SLOTS][9];
        int gi[MX_UPD_SLOTS];
#pragma unroll
        for (int j = 0; j < MX_UPD_SLOTS; ++j) {
          const int q = k0 - kb + j;
          int f = __shfl_sync(0xffffffffu, fl, q & 31);
          if constexpr (CW * MX_UPD_SLOTS > 32) {
            const int f2 = __shfl_sync(0xffffffffu, fl2, q & 31);
            f = q < 32 ? f : f2;
          }
          const int as = ((f >> 2) & 3) * S + sp + 32 * l;
          gi[j] = ((f & 16) ? 3 * S : 0) + as;
          const T* Jk = Jm + (size_t)(k0 + j) * 9 * NP + sFp[as];
#pragma unroll
          for (int v = 0; v < 9; ++v) jv[j][v] = v < 5 || visc ? __ldg(Jk + v * NP) : T(0);
        }
#pragma unroll
        for (int j = 0; j < MX_UPD_SLOTS; ++j) {
          const double gw = sG[gi[j]];
#pragma unroll
          for (int v = 0; v < 9; ++v) cx[v][l] += gw * double(jv[j][v]);
        }
      }
    } else {
      for (int j = 0; j < n; ++j) {
        const int f = __ldg(a.slot_flags + k0 + j);
#pragma unroll
        for (int l = 0; l < PL; ++l) {
          const int as = ((f >> 2) & 3) * S + sp + 32 * l;
          const double gw = sG[((f & 16) ? 3 * S : 0) + as];
          const T* Jk = Jm + (size_t)(k0 + j) * 9 * NP + sFp[as];
#pragma unroll
          for (int v = 0; v < 9; ++v)
            if (v < 5 || visc) cx[v][l] += gw * double(__ldg(Jk + v * NP));
        }
      }
    }
#pragma unroll
    for (int l = 0; l < PL; ++l)
#pragma unroll
      for (int v = 0; v < 9; ++v)  // inviscid corrections enter with -g', viscous with +g'
        x[v][l] = double(rv[v][l]) + (v < 5 ? -cx[v][l] : cx[v][l]) * rd[l];
    // outliers: a column that is not provably free of them takes the exact rule
    unsigned bad = 0u;
#pragma unroll
    for (int v = 0; v < 9; ++v)
      if (v < 5 || visc) bad |= mxd::outlier_clear<S, PL>(x[v], on, grp) ? 0u : 1u << v;
    bad = S == 8 ? __reduce_or_sync(0xffffffffu, bad) : bad;
    if (bad) {
#pragma unroll
      for (int v = 0; v < 9; ++v)
        if (bad >> v & 1u) {
          mxd::Vals<PL> u, X;
#pragma unroll
          for (int l = 0; l < PL; ++l) {
            X.v[l] = x[v][l];
            u.v[l] = on[l] ? a.Ucur[((size_t)e * S + sp + 32 * l) * nv + (v < 5 ? v : v - 4)] : 0.0;
          }
          X = mxd::outlier_exact<S, PL>(X, u, grp, sp, live);
#pragma unroll
          for (int l = 0; l < PL; ++l) x[v][l] = X.v[l];
        }
    }
    if (!step) {
      // residual-only outputs: assembled as rows, stored as blocks below
#pragma unroll
      for (int l = 0; l < PL; ++l)
        if (on[l]) {
          double* ri = sU + (c * S + sp + 32 * l) * nv;
          double* rw = s0 + (c * S + sp + 32 * l) * nv;
#pragma unroll
          for (int v = 0; v < 7; ++v)
            if (v < nv) {
              ri[v] = v < 5 ? x[v < 5 ? v : 0][l] : 0.0;
              rw[v] = (v > 0 && v < 5 && visc) ? x[v > 0 && v < 5 ? 4 + v : 0][l] : 0.0;
            }
        }
      continue;
    }
    if (r == 0) {
      cp_async_wait0();
      __syncwarp();
    }
    // RK stage combination + positivity, in place over the state tile
    double sq = 0.0, sr = 0.0;
#pragma unroll
    for (int l = 0; l < PL; ++l)
      if (on[l]) {
        double Lr[5], un[7];
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          Lr[v] = x[v][l] + (v > 0 ? x[v > 0 ? 4 + v : 0][l] : 0.0);
          sq += Lr[v] * Lr[v];
        }
        sr += Lr[0] * Lr[0];
        const double dts = __ldg(a.dt + (size_t)e * S + sp + 32 * l);
        double* uc = sU + (c * S + sp + 32 * l) * nv;
        const double* u0 = a.stage > 0 ? s0 + (c * S + sp + 32 * l) * nv : uc;
        const double w0 = a.stage == 0 ? 0.0 : (a.stage == 1 ? 0.75 : 1.0 / 3.0);
        const double w1 = a.stage == 0 ? 1.0 : (a.stage == 1 ? 0.25 : 2.0 / 3.0);
#pragma unroll
        for (int v = 0; v < 7; ++v) {
          const double b = v < nv ? (a.stage == 0 ? uc[v] : w0 * u0[v] + w1 * uc[v]) : 0.0;
          un[v] = v < 5 ? b + (w1 * dts) * Lr[v < 5 ? v : 0] : b;
        }
        // positivity (core/time_integration/positivity.py:13-45), one reciprocal of rho
        const double rho = fmax(un[0], 1e-6);
        un[0] = rho;
        const double rr = 1.0 / rho;
        double vel[3] = {un[1] * rr, un[2] * rr, un[3] * rr};
        const double v2 = vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2];
        double ke = 0.5 * rho * v2;
        if (v2 > 9.9e7) {  // near or above the speed limit of 1e4
          const double vm = sqrt(v2);
          if (vm > 1e4) {
            const double cf = 1e4 / vm;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              vel[d] *= cf;
              un[1 + d] = rho * vel[d];
            }
          }
          ke = 0.5 * rho * (vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2]);
        }
        const double pr = (GAMMA - 1.0) * (un[4] - ke);
        if (pr < 1.0) un[4] = 1.0 / (GAMMA - 1.0) + ke;
        un[5] = fmax(un[5], 0.0);
        un[6] = fmax(un[6], 1e-8);
#pragma unroll
        for (int v = 0; v < 7; ++v)
          if (v < nv) uc[v] = un[v];
      }
    if (a.stage == 0) {
      const double acc = mxd::cell_sum<S>(sq), acc_rho = mxd::cell_sum<S>(sr);
      if (live && sp == 0) {
        a.norm_part[e] = acc;
        a.norm_rho_part[e] = acc_rho;
        // a non-finite dU/dt anywhere in the cell makes its partial non-finite
        if (!isfinite(acc) && a.status) atomicOr(a.status, (unsigned)DS_NONFINITE);
      }
    }
  }
  __syncwarp();
  const int nst = nc * S * nv;
  if (!step) {
    if (a.Rinv)
      for (int t = lane; t < nst; t += 32) a.Rinv[(size_t)e0 * S * nv + t] = sU[t];
    if (a.Rvisc)
      for (int t = lane; t < nst; t += 32) a.Rvisc[(size_t)e0 * S * nv + t] = s0[t];
    return;
  }
  // modal filter of the first five variables: one FP64 tensor-core product per
  // warp (rows s, columns (cell, variable), K = the cell's points) into the
  // step-start tile, which the stage no longer needs
  if (nv > 5)
    for (int p = lane; p < nc * S; p += 32) {
      s0[p * nv + 5] = sU[p * nv + 5];
      if (nv > 6) s0[p * nv + 6] = sU[p * nv + 6];
    }
  dmma_warp_rb_f<(S + 7) / 8, (5 * CW + 7) / 8, S>(
      S, 5 * nc, ops.ffilt[ct], [&](int j, int col) { return sU[((col / 5) * S + j) * nv + col % 5]; },
      [&](int m, int col, double v) { s0[((col / 5) * S + m) * nv + col % 5] = v; });
  __syncwarp();
  double* out = a.Unext + (size_t)e0 * S * nv;
  for (int t = lane; t < nst; t += 32) out[t] = s0[t];
}

// ---------------------------------------------------------------------------
// set-up kernels of the mixed form
// ---------------------------------------------------------------------------
// own adjugate row at each slot flux point (E * adj, FP64 then rounded) and the
// face point of the other side whose extrapolation row equals the slot's
// interpolation row to tol relative (MX_OFP_GENERAL where none does).  used: bit
// axis*2 + side of every face whose face-point fields a slot reads, and MX_GENERAL
// where some point interpolates from point fields
constexpr unsigned MX_GENERAL = 1u << 8;
template <int S, int NP>
__global__ void k_mx_match(Geom g, Ops ops, Faces fc, SlotTable st, float4* arow, uint8_t* ofp, unsigned* used,
                           double tol) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= st.n * NP) return;
  const int sl = t / NP, i = t % NP;
  const int f = st.face[sl], e = st.cell[sl], fl = st.flags[sl];
  const bool is_owner = (fl & 1) == 0, bnd = (fl & 2) != 0;
  const int ax = (fl >> 2) & 3, sb = (fl & 16) ? 1 : 0;
  const int ct = cell_type(g, e);
  const double* Er = ops.extrap + (((size_t)ct * 3 + ax) * 2 + sb) * NP * S + (size_t)i * S;
  double a0 = 0.0, a1 = 0.0, a2 = 0.0;
  for (int s = 0; s < S; ++s) {
    const double w = Er[s];
    const double* ad = g.adj + ((size_t)e * S + s) * 9 + ax * 3;
    a0 += w * ad[0];
    a1 += w * ad[1];
    a2 += w * ad[2];
  }
  {
    // the direction is compared with the face normal in the face kernel's own FP32 arithmetic
    const float4 ar = make_float4(float(a0), float(a1), float(a2), float(sqrt(a0 * a0 + a1 * a1 + a2 * a2)));
    const float mag = fmaxf(ar.w, 1e-30f), sd = sb ? 1.f : -1.f, sg = is_owner ? 1.f : -1.f;
    const double* tn = fc.tnormal + ((size_t)f * NP + i) * 3;
    const float al = ar.x / mag * sd * (sg * float(tn[0])) + ar.y / mag * sd * (sg * float(tn[1])) +
                     ar.z / mag * sd * (sg * float(tn[2]));
    arow[t] = make_float4(ar.x, ar.y, ar.z, al < 0.5f ? -mag : ar.w);
  }
  auto mark = [used](unsigned bits) {
    if (bits & ~*(volatile unsigned*)used) atomicOr(used, bits);  // few threads find a bit unset
  };
  mark(1u << (ax * 2 + sb));
  if (bnd) {
    ofp[t] = 0;
    return;
  }
  // the other side's interpolation row; the reference may split one cell's
  // row over its two source slots, so same-cell rows are added first
  const int c0 = st.c0[sl], c1 = st.c1[sl];
  const int expect = is_owner ? fc.neighbor[f] : fc.owner[f];
  const bool one_cell = (c0 == expect || c0 < 0) && (c1 == expect || c1 < 0) && (c0 >= 0 || c1 >= 0);
  if (!one_cell) {
    mark(MX_GENERAL);
    ofp[t] = MX_OFP_GENERAL;
    return;
  }
  const double* M0 =
      c0 >= 0 ? (is_owner ? fmat(fc.nb_m0, fc.nb_m0i, f, i, NP, S) : fmat(fc.ow_m0, fc.ow_m0i, f, i, NP, S)) : nullptr;
  const double* M1 = c1 >= 0 ? (is_owner ? fmat(fc.nb_m1, fc.nb_m1i, st.i1[sl], i, NP, S)
                                         : fmat(fc.ow_m1, fc.ow_m1i, st.i1[sl], i, NP, S))
                             : nullptr;
  const int oax = is_owner ? fc.n_axis[f] : fc.o_axis[f];
  const int osb = (is_owner ? fc.n_side[f] : fc.o_side[f]) > 0.0 ? 1 : 0;
  const int oct = cell_type(g, expect);
  double mmax = 0.0;
  for (int s = 0; s < S; ++s) mmax = fmax(mmax, fabs((M0 ? M0[s * NP] : 0.0) + (M1 ? M1[s * NP] : 0.0)));
  int best = -1;
  double best_err = INFINITY;
  for (int j = 0; j < NP; ++j) {
    const double* Eo = ops.extrap + (((size_t)oct * 3 + oax) * 2 + osb) * NP * S + (size_t)j * S;
    double err = 0.0;
    for (int s = 0; s < S && err <= best_err; ++s)
      err = fmax(err, fabs((M0 ? M0[s * NP] : 0.0) + (M1 ? M1[s * NP] : 0.0) - Eo[s]));
    if (err < best_err) {
      best_err = err;
      best = j;
    }
  }
  const bool matched = best >= 0 && best_err <= tol * fmax(mmax, 1e-300);
  mark(matched ? 1u << (oax * 2 + osb) : MX_GENERAL);
  ofp[t] = matched ? (uint8_t)((oax * 2 + osb) * NP + best) : MX_OFP_GENERAL;
}

// the records of matched slot points: their face-point rows and sides
__global__ void k_mx_pairs(SlotTable st, const int2* __restrict__ pts, int n, int NP, MxPair* __restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int2 t = pts[j];
  auto row = [&](int p) -> uint32_t {
    const int sl = p / NP, fl = st.flags[sl], face = ((fl >> 2) & 3) * 2 + ((fl & 16) ? 1 : 0);
    return (((uint32_t)st.cell[sl] * 6 + face) * NP + p % NP) | ((fl & 16) ? 0x80000000u : 0u);
  };
  out[j] = MxPair{t.x, t.y, row(t.x), row(t.y)};
}

// 1 / det per solution point
__global__ void k_mx_rdet(const double* __restrict__ det, size_t n, double* __restrict__ out) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) out[t] = 1.0 / det[t];
}

// FP32 copies of 3 x 3 metric rows (adjugates, inverse Jacobians: the mixed
// kernels round them to FP32 before use); one row of 3 per float4
__global__ void k_mx_rows_f32(const double* __restrict__ adj_fine, size_t nrows, float4* __restrict__ out) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nrows) return;
  const double* a = adj_fine + t * 3;
  out[t] = make_float4(float(a[0]), float(a[1]), float(a[2]), 0.f);
}

// MD[c,s,n] = sum_{i,m} W[s, i*3+m] adj_fine[c,i,m,n]  (W's columns follow D_fine: i*3+m),
// rounded once: every stage multiplies the same MD with a flux of the pressure's
// size, so its error would add up over a step where those of the divergence
// average out (FP64 P2 RANS step, momentum against 64 bits: 8.7e-16 with a plain
// sum, 8.0e-16 so)
template <int S, int FN>
__global__ void k_mx_md(Geom g, Ops ops, size_t ncells, double* MD) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ncells * S * 3) return;
  const int n = (int)(t % 3);
  const int s = (int)((t / 3) % S);
  const size_t c = t / (3 * S);
  const int ct = cell_type(g, (int)c);
  const double* w = ops.W[ct] + (size_t)s * FN * 3;
  const double* ad = g.adj_fine + c * FN * 9;
  double acc = 0.0, low = 0.0;  // sum, and the rounding errors of its products and additions
  for (int i = 0; i < FN; ++i)
    for (int m = 0; m < 3; ++m) {
      const double x = w[i * 3 + m], y = ad[i * 9 + m * 3 + n];
      const double p = __dmul_rn(x, y), sum = __dadd_rn(acc, p), b = __dadd_rn(sum, -acc);
      low += __fma_rn(x, y, -p) + (__dadd_rn(acc, -__dadd_rn(sum, -b)) + __dadd_rn(p, -b));
      acc = sum;
    }
  MD[t] = acc + low;
}

template <int S>
__global__ void k_mx_hcell(Geom g, double* hcell) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= g.N) return;
  double vol = 0.0;
  for (int s = 0; s < S; ++s) vol += g.det[(size_t)e * S + s];
  vol /= S;
  double h = pow(vol, 1.0 / 3.0);
  if (h < 1e-300) h = 1e-300;
  hcell[e] = h;
}

}  // namespace afr
