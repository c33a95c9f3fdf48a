// Cell kernel of prisms, FP32 (mixed form) and FP64 (plain form), whose operators
// have tensor-product structure in the collapsed coordinates (a, b, c): point s = (a*N1 + b)*N1 + c.
//
//   D_3d[.,.,0]  couples points of one a-line (same b, c), the same weights on
//   every line; D_3d[.,.,2] likewise along c; D_3d[.,.,1] couples the points of
//   one triangle plane (same c).
//   boundary_extrap reads one a-line (axis 0), one triangle plane (axis 1) or
//   one c-line (axis 2) per face point.
//   c2f and the folded W = f2c*D_fine (per reference axis m) are Kronecker
//   products triangle (x) c-line.
//
// The reference's prism operators have this structure to rounding: entries
// outside it are at most 2e-15 of the largest in D_3d, boundary_extrap and c2f,
// and W is off by 6e-15 (P1) and 1.1e-13 (P2) of its rows' l1 norms.  afr_create
// tests for it (px_operators) and takes this kernel instead of k_mx_pre +
// k_mx_vol (mixed) or k_pre + k_cell's volume terms (plain), which stay for every
// other operator set (tets, P3).
//
// Why: with the structure a P2 cell needs 9 k multiply-adds instead of the
// 45 k of the dense products, so plain FP32 (whose products carry 24 bits
// instead of the 16 of a BF16 hi+lo pair) is no longer bound by arithmetic,
// and everything a cell needs for the face-point fields, the viscous and the
// inviscid volume terms is formed in one pass over the state: 9.7 KB per P2
// cell instead of 19 KB for the two tensor-core kernels.
//
// A warp owns CW whole cells from load to store, so the phases are separated
// by __syncwarp only and the warps of an SM drift apart and overlap one
// another's loads and arithmetic.  CW is chosen so that the items of the
// phases fill the 32 lanes: P2, CW = 2: 27 + 27 points, 30 (cell, variable,
// c-level), 32 (cell, fine triangle point), 30 (cell, field); P1, CW = 6: 48,
// 60, 54 and 90 in two or three rounds.  The operators of the extrapolation, c2f
// and W arrive as a kernel parameter: every index into them is a compile-time
// constant, so they are operands from the constant bank and cost no loads.  The
// derivatives differ from point to point; a lane loads its point's rows once.
#pragma once
#include "afr_mixed.cuh"

namespace afr {

// warps per CTA: P1's 16 KB per warp fill an SM better in pairs (14 warps instead
// of 12; 256,000 prisms: 319 -> 298 us), P2 is limited by registers
__host__ __device__ constexpr int px_warps(int n1) { return n1 == 2 ? 2 : 4; }

template <class T, int N1, int NF>
struct PxOps {
  static constexpr int NT = N1 * N1, MT = NF * NF;
  T E02[2][2][N1];   // extrapolation along a (0) and c (1): [which][side][point of the line]
  T E1[2][N1][NT];   // extrapolation to the b faces: [side][a of the face point][triangle point]
  // The factors below start at an odd entry, where the compiler cannot combine
  // their loads.  102,660 P2 prisms, step: 2,028 us there, 2,058 aligned to four
  // entries, 2,086 at an even one (registers and spills are the same).
  T odd[1];
  T Ct[MT][NT], Cc[NF][N1];        // c2f = Ct (x) Cc
  T Wt[3][NT][MT], Wc[3][N1][NF];  // W per axis = Wt (x) Wc
};

// per-cell metrics in the order the lanes read them
template <class T>
struct PxGeom {
  const T* adjs;       // (n_prism, 9, S) solution-point adjugates, entry m*3 + n
  // fine-point adjugates (fine point = triangle point * NF + c-level): FP32
  // (n_prism, 9, MT, NF), a lane's c-line in one vector; FP64 (n_prism, NF, 9, MT), level by level
  const T* adjf;
  const double* MD;    // (N, S, 3)
  const double* rdet;  // (N, S)
  const T* rows;       // derivative rows of the points, see px_rows
};

template <class T>
struct alignas(4 * sizeof(T)) Vec4 {
  T x, y, z, w;
};
template <class T>
struct alignas(16) VecN {  // 16 bytes
  static constexpr int N = 16 / sizeof(T);
  T v[N];
};

template <class T, int N1, int NF, int CW>
struct PxSmem {
  static constexpr bool D = sizeof(T) == 8;
  static constexpr int S = N1 * N1 * N1, NT = N1 * N1, MT = NF * NF;
  // triangle row stride: 16-byte rows on distinct banks
  static constexpr int TP = D ? (MT == 16 ? 18 : 10) : (MT == 16 ? 20 : 12);
  static constexpr int FS = S | 1;               // field row stride (odd)
  static constexpr int oDev = 64 * S / sizeof(T), oG = oDev + 4 * S;  // inside H, after the staged state (8 doubles per point)
  static constexpr int need = D ? oG + 12 * S : cmax(oG + 12 * S, 6 * MX_XF * NT);
  // c-contracted fluxes; before: state, gradient inputs, viscous fluxes; FP32: face fields
  static constexpr int nH = cmax(15 * N1 * TP, need);
  static constexpr int nX = MX_XF * FS, nY = 5 * N1 * TP;
  static constexpr int oX = (nH + 3) / 4 * 4, oY = (oX + nX + 3) / 4 * 4, oRef = oY + nY, oF = oRef + 8;
  static constexpr int cell = (oF + 120 / (int)sizeof(T) + 3) / 4 * 4;  // T values per cell
  static constexpr int total = px_warps(N1) * CW * cell * (int)sizeof(T);
};

// rho H of the Euler flux, rho * (p / (0.4 max(rho, 1e-10)) + |u|^2 / 2) + p over
// max(rho, 1e-10) times rho (core/fr_operators/flux_kernels.py:28-68)
__device__ __forceinline__ double px_rhoH(double rho, double p, double u2) {
  if (rho >= 1e-10) return GAMMA / (GAMMA - 1.0) * p + 0.5 * rho * u2;
  const double rs = 1e-10;
  const double rhoE = rho * (p / ((GAMMA - 1.0) * rs) + 0.5 * u2);
  return rho * ((rhoE + p) / rs);
}

// T = float: the mixed form (face-point fields XF by extrapolation, point
// fields PF only where a face point interpolates from them).  T = double: the
// plain form; it writes the point fields, from which k_face extrapolates and
// interpolates with every entry of the mesh's own operators.
template <class T, int N1, int NF, int CW, bool VISC>
__global__ void __launch_bounds__(32 * px_warps(N1), sizeof(T) == 8 ? (N1 == 3 ? 2 : 4) : (N1 == 3 ? 4 : 7))
    k_px_cell(const __grid_constant__ PxOps<T, N1, NF> op, PxGeom<T> pg, float* __restrict__ XF, T* __restrict__ PF,
              T* __restrict__ RV, int FW, unsigned face_mask, const double* __restrict__ U, int nv,
              const double* __restrict__ nut, T mu, int cell_base, int cell_end) {
  using L = PxSmem<T, N1, NF, CW>;
  constexpr bool D = sizeof(T) == 8;
  constexpr int S = L::S, NT = L::NT, MT = L::MT, TP = L::TP, FS = L::FS, NP = NT;
  constexpr int CPR = 32 / S;                 // cells per round of the point phases
  constexpr int PR = (CW + CPR - 1) / CPR;    // rounds
  constexpr int VN = VecN<T>::N;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* smf = reinterpret_cast<T*>(smraw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e0 = cell_base + (blockIdx.x * px_warps(N1) + warp) * CW;
  const int nc = min(CW, cell_end - e0);
  if (nc <= 0) return;  // whole warps; no block barrier below
  T* sw = smf + warp * CW * L::cell;
  // point lanes: the same solution point every round
  const int s = lane % S, pc = lane / S;
  const int cc = s % N1;

  // ---- state and nu_t of the warp's cells ----
  for (int c = 0; c < nc; ++c) {
    double* d = reinterpret_cast<double*>(sw + c * L::cell);
    const double* ub = U + (size_t)(e0 + c) * S * nv;
    for (int t = lane; t < S * nv; t += 32) cp_async8(d + t, ub + t);
    if (VISC && nut)
      for (int t = lane; t < S; t += 32) cp_async8(d + 7 * S + t, nut + (size_t)(e0 + c) * S + t);
  }
  cp_async_wait_all();
  __syncwarp();

  // ---- primitives; deviations from the cell's reference point ----
  T uf[PR][3], mut[PR];
#pragma unroll
  for (int r = 0; r < PR; ++r) {
    const int c = r * CPR + pc;
    const bool in = pc < CPR && c < CW;
    T* sc = sw + (in ? c : 0) * L::cell;
    double q[6] = {1.0, 0.0, 0.0, 0.0, 1.0, 1.0};
    mut[r] = T(0);
    if (in && c < nc) {
      const double* d = reinterpret_cast<const double*>(sc);
      if constexpr (D) {  // quotients as in k_pre: a reciprocal of rho would round twice
        cons_to_prim(d + s * nv, q);
        q[5] = q[4] / (q[0] * R_AIR);
      } else {
        mxd::prim_T(d + s * nv, q);
      }
      if (VISC && nut) mut[r] = T(q[0] * d[7 * S + s]);
    }
    // FP32: deviations from the value at the cell's middle point, which carry
    // the variation in 24 bits.  FP64 keeps the values; the reference state
    // only enters the inviscid flux (below), and any finite one serves: zero
    // where the middle point's value is beyond FP32's range.
    T dev[6];
    constexpr int MID = S / 2;
#pragma unroll
    for (int v = 0; v < 6; ++v) {
      if (v == 5 && (D || !VISC)) {  // the temperature: gradients only
        dev[5] = T(q[5]);
        continue;
      }
      float ref = __shfl_sync(0xffffffffu, float(q[v]), (pc < CPR ? pc : 0) * S + MID);
      if (D && !isfinite(ref)) ref = 0.f;
      dev[v] = D ? T(q[v]) : T(q[v] - double(ref));
      if (in && s == MID) sc[L::oRef + v] = T(ref);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) uf[r][d] = T(q[1 + d]);
    if (in) {
#pragma unroll
      for (int v = 0; v < 5; ++v) sc[L::oX + v * FS + s] = dev[v];
      if (VISC) *reinterpret_cast<Vec4<T>*>(sc + L::oDev + 4 * s) = Vec4<T>{dev[1], dev[2], dev[3], dev[5]};
    }
    if (!D && PF && in && c < nc) {
      T* o = PF + ((size_t)(e0 + c) * S + s) * MX_PF;
#pragma unroll
      for (int v = 0; v < 5; ++v) o[10 + v] = T(q[v]);
    }
  }
  __syncwarp();

  T vis[PR][4];
  if constexpr (VISC) {
    // this lane's rows of the derivative operators
    T d0[N1], d1[NT], d2[N1];
#pragma unroll
    for (int l = 0; l < N1; ++l) {
      d0[l] = __ldg(pg.rows + l * S + s);
      d2[l] = __ldg(pg.rows + (N1 + NT + l) * S + s);
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) d1[t] = __ldg(pg.rows + (N1 + t) * S + s);
    T rd[PR];
#pragma unroll
    for (int r = 0; r < PR; ++r) {
      const int c = r * CPR + pc;
      const bool in = pc < CPR && c < CW;
      T* sc = sw + (in ? c : 0) * L::cell;
      T aj[9];
      rd[r] = T(0);
#pragma unroll
      for (int k = 0; k < 9; ++k) aj[k] = T(0);
      if (in && c < nc) {
#pragma unroll
        for (int k = 0; k < 9; ++k) aj[k] = __ldg(pg.adjs + ((size_t)(e0 + c) * 9 + k) * S + s);
        rd[r] = T(__ldg(pg.rdet + (size_t)(e0 + c) * S + s));
      }
      // reference-space gradients of u, v, w, T
      const Vec4<T>* dv = reinterpret_cast<const Vec4<T>*>(sc + L::oDev);
      T g[3][4];
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int f = 0; f < 4; ++f) g[m][f] = T(0);
      auto acc = [](T (&o)[4], T w, const Vec4<T>& x) {
        o[0] += w * x.x;
        o[1] += w * x.y;
        o[2] += w * x.z;
        o[3] += w * x.w;
      };
#pragma unroll
      for (int l = 0; l < N1; ++l) {
        acc(g[0], d0[l], dv[l * NT + s % NT]);
        acc(g[2], d2[l], dv[s - cc + l]);
      }
#pragma unroll
      for (int t = 0; t < NT; ++t) acc(g[1], d1[t], dv[t * N1 + cc]);
      // physical gradients: inverse Jacobian = adjugate / det
      T gr[4][3];
#pragma unroll
      for (int f = 0; f < 4; ++f)
#pragma unroll
        for (int n = 0; n < 3; ++n)
          gr[f][n] = rd[r] * (g[0][f] * aj[n] + g[1][f] * aj[3 + n] + g[2][f] * aj[6 + n]);
      const T sym[6] = {gr[0][0], gr[1][1], gr[2][2], T(0.5) * (gr[0][1] + gr[1][0]), T(0.5) * (gr[0][2] + gr[2][0]),
                        T(0.5) * (gr[1][2] + gr[2][1])};
      T G[3][4];
      viscous_flux_sym(uf[r], sym, gr[3], mu, mut[r], G);
      if (in) {
        T* x = sc + L::oX + 5 * FS + s;
#pragma unroll
        for (int k = 0; k < 6; ++k) x[k * FS] = sym[k];
#pragma unroll
        for (int k = 0; k < 3; ++k) x[(6 + k) * FS] = gr[3][k];
        x[9 * FS] = mut[r];
        Vec4<T>* gt = reinterpret_cast<Vec4<T>*>(sc + L::oG);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          T h[4];
#pragma unroll
          for (int v = 0; v < 4; ++v) h[v] = aj[m * 3] * G[0][v] + aj[m * 3 + 1] * G[1][v] + aj[m * 3 + 2] * G[2][v];
          gt[m * S + s] = Vec4<T>{h[0], h[1], h[2], h[3]};
        }
      }
      if (!D && PF && in && c < nc) {
        T* o = PF + ((size_t)(e0 + c) * S + s) * MX_PF;
#pragma unroll
        for (int k = 0; k < 6; ++k) o[k] = sym[k];
#pragma unroll
        for (int k = 0; k < 3; ++k) o[6 + k] = gr[3][k];
        o[9] = mut[r];
      }
    }
    __syncwarp();
    // viscous divergence / det (the mass component is zero)
#pragma unroll
    for (int r = 0; r < PR; ++r) {
      const int c = r * CPR + pc;
      const T* sc = sw + (pc < CPR && c < CW ? c : 0) * L::cell;
      const Vec4<T>* gt = reinterpret_cast<const Vec4<T>*>(sc + L::oG);
      T o[4] = {T(0), T(0), T(0), T(0)};
      auto acc = [&](T w, const Vec4<T>& x) {
        o[0] += w * x.x;
        o[1] += w * x.y;
        o[2] += w * x.z;
        o[3] += w * x.w;
      };
#pragma unroll
      for (int l = 0; l < N1; ++l) {
        acc(d0[l], gt[l * NT + s % NT]);
        acc(d2[l], gt[2 * S + s - cc + l]);
      }
#pragma unroll
      for (int t = 0; t < NT; ++t) acc(d1[t], gt[S + t * N1 + cc]);
#pragma unroll
      for (int v = 0; v < 4; ++v) vis[r][v] = o[v] * rd[r];
    }
    __syncwarp();  // H is reused for the face-point fields
  }

  if constexpr (D) {
    // point fields of the face kernel: one contiguous block of 128-byte rows per cell
    for (int c = 0; c < nc; ++c) {
      const T* sc = sw + c * L::cell;
      T* dst = PF + (size_t)(e0 + c) * S * PFW;
      for (int t = lane; t < S * PFW; t += 32) {
        const int j = t / PFW, f = t % PFW;
        if (f < (VISC ? MX_XF : 5)) dst[t] = sc[L::oX + f * FS + j];
      }
    }
    __syncwarp();
  } else {
    // ---- extrapolation: one lane per (cell, field), the field in registers ----
    constexpr int NFL = VISC ? MX_XF : 5;
    for (int it = lane; it < CW * NFL; it += 32) {
      const int c = it / NFL, f = it - c * NFL;
      T* sc = sw + c * L::cell;
      float x[S];
      const float* xs = sc + L::oX + f * FS;
#pragma unroll
      for (int j = 0; j < S; ++j) x[j] = xs[j];
      const float base = f < 5 ? sc[L::oRef + f] : 0.f;  // the extrapolation reproduces constants
      float* o = sc + f * NP;                            // face k's point i at o[k * MX_XF * NP + i]
#pragma unroll
      for (int sd = 0; sd < 2; ++sd) {
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          float a0 = 0.f, a2 = 0.f;
#pragma unroll
          for (int l = 0; l < N1; ++l) {
            a0 += op.E02[0][sd][l] * x[l * NT + i];
            a2 += op.E02[1][sd][l] * x[i * N1 + l];
          }
          o[sd * MX_XF * NP + i] = base + a0;
          o[(4 + sd) * MX_XF * NP + i] = base + a2;
        }
        if (face_mask >> (2 + sd) & 1) {
#pragma unroll
          for (int i = 0; i < NP; ++i) {
            float a1 = 0.f;
#pragma unroll
            for (int t = 0; t < NT; ++t) a1 += op.E1[sd][i / N1][t] * x[t * N1 + i % N1];
            o[(2 + sd) * MX_XF * NP + i] = base + a1;
          }
        }
      }
    }
    __syncwarp();
    // face-point fields of the faces that some slot reads, one contiguous block per face
    for (int c = 0; c < nc; ++c) {
      const T* sc = sw + c * L::cell;
      float* dst = XF + (size_t)(e0 + c) * 6 * FW * NP;
      if (VISC && FW == MX_XF) {
        constexpr int HB = MX_XF * NP;  // floats per face block
        for (int t = lane; t < 6 * HB / 2; t += 32) {
          const bool use = (face_mask >> (2 * t / HB) & 1) | (face_mask >> ((2 * t + 1) / HB) & 1);
          if (use) reinterpret_cast<float2*>(dst)[t] = reinterpret_cast<const float2*>(sc)[t];
        }
      } else {
        for (int t = lane; t < 6 * 5 * NP; t += 32) {
          const int k = t / (5 * NP), j = t - k * (5 * NP);
          if (face_mask >> k & 1) dst[k * FW * NP + j] = sc[k * MX_XF * NP + j];
        }
      }
    }
  }
  if constexpr (VISC) {
    // the gradient fields are consumed: their rows park the viscous terms
#pragma unroll
    for (int r = 0; r < PR; ++r) {
      const int c = r * CPR + pc;
      if (pc < CPR && c < CW) {
#pragma unroll
        for (int v = 0; v < 4; ++v) sw[c * L::cell + L::oX + (5 + v) * FS + s] = vis[r][v];
      }
    }
  }

  // ---- c2f, triangle part: one lane per (cell, variable, c-level) ----
  for (int it = lane; it < CW * 5 * N1; it += 32) {
    const int c = it / (5 * N1), vk = it - c * (5 * N1), v = vk / N1, k = vk - v * N1;
    T* sc = sw + c * L::cell;
    T x[NT];
    const T base = D ? sc[L::oRef + v] : T(0);
#pragma unroll
    for (int t = 0; t < NT; ++t) x[t] = sc[L::oX + v * FS + t * N1 + k] - base;
    T* y = sc + L::oY + vk * TP;
#pragma unroll
    for (int tv = 0; tv < (MT + VN - 1) / VN; ++tv) {
      VecN<T> z;
#pragma unroll
      for (int j = 0; j < VN; ++j) {
        z.v[j] = T(0);
        if (tv * VN + j < MT) {
#pragma unroll
          for (int t = 0; t < NT; ++t) z.v[j] += op.Ct[tv * VN + j][t] * x[t];
        }
      }
      *reinterpret_cast<VecN<T>*>(y + tv * VN) = z;
    }
  }
  // Euler flux at the reference state, FP64: lane = (cell, direction)
  if (lane < 3 * CW) {
    const int c = lane / 3, n = lane % 3;
    T* sc = sw + c * L::cell;
    const T* rf = sc + L::oRef;
    const double q[5] = {rf[0], rf[1], rf[2], rf[3], rf[4]};
    const double un = n == 0 ? q[1] : (n == 1 ? q[2] : q[3]);
    const double m = q[0] * un;
    double* F = reinterpret_cast<double*>(sc + L::oF) + n * 5;
    F[0] = m;
    F[1] = m * q[1] + (n == 0 ? q[4] : 0.0);
    F[2] = m * q[2] + (n == 1 ? q[4] : 0.0);
    F[3] = m * q[3] + (n == 2 ? q[4] : 0.0);
    F[4] = un * px_rhoH(q[0], q[4], q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
  }
  __syncwarp();

  // ---- fine points: one lane per (cell, fine triangle point) walks the
  // c-line: c2f along c, flux deviation, contravariant components, and the
  // c part of W accumulated in registers ----
  for (int it = lane; it < CW * MT; it += 32) {
    const int c = it / MT, t = it - c * MT;
    T* sc = sw + c * L::cell;
    T af[D ? 1 : 9][D ? 1 : NF], an[D ? 9 : 1];
    const T* ap = pg.adjf + (size_t)(e0 + (c < nc ? c : 0)) * NF * 9 * MT + t;
    if constexpr (D) {
#pragma unroll
      for (int k = 0; k < 9; ++k) an[k] = __ldg(ap + k * MT);
    }
    if constexpr (!D) {
      const float* ap = pg.adjf + ((size_t)(e0 + (c < nc ? c : 0)) * 9 * MT + t) * NF;
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        if constexpr (NF == 4) {
          const float4 x = __ldg(reinterpret_cast<const float4*>(ap + (size_t)k * MT * NF));
          af[k][0] = x.x;
          af[k][1] = x.y;
          af[k][2] = x.z;
          af[k][NF - 1] = x.w;
        } else {
#pragma unroll
          for (int l = 0; l < NF; ++l) af[k][l] = __ldg(ap + (size_t)k * MT * NF + l);
        }
      }
    }
    T y[5][N1], qb[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      qb[v] = sc[L::oRef + v];
#pragma unroll
      for (int k = 0; k < N1; ++k) y[v][k] = sc[L::oY + (v * N1 + k) * TP + t];
    }
    T h[3][5][N1];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int v = 0; v < 5; ++v)
#pragma unroll
        for (int k = 0; k < N1; ++k) h[m][v][k] = T(0);
#pragma unroll
    for (int l = 0; l < NF; ++l) {
      T dq[5], dF[3][5];
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        dq[v] = T(0);
#pragma unroll
        for (int k = 0; k < N1; ++k) dq[v] += op.Cc[l][k] * y[v][k];
      }
      T al[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        if constexpr (D) {
          al[k] = an[k];  // loaded one level ahead
          if (l + 1 < NF) an[k] = __ldg(ap + ((l + 1) * 9 + k) * MT);
        } else {
          al[k] = af[k][l];
        }
      }
      if constexpr (D) {
        // the flux itself (density floored as in the plain Euler flux), less
        // the flux of the reference state
        const double* Fr = reinterpret_cast<const double*>(sc + L::oF);
        const T rho = qb[0] + dq[0], p = qb[4] + dq[4];
        const T u[3] = {qb[1] + dq[1], qb[2] + dq[2], qb[3] + dq[3]};
        const T rH = px_rhoH(rho, p, u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
#pragma unroll
        for (int n = 0; n < 3; ++n) {
          const T m = rho * u[n];
          dF[n][0] = m - Fr[n * 5];
#pragma unroll
          for (int j = 0; j < 3; ++j) dF[n][1 + j] = m * u[j] + (n == j ? p : T(0)) - Fr[n * 5 + 1 + j];
          dF[n][4] = rH * u[n] - Fr[n * 5 + 4];
        }
      } else {
        mxd::euler_flux_delta<T>(qb, dq, dF);
      }
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          const T ft = al[m * 3] * dF[0][v] + al[m * 3 + 1] * dF[1][v] + al[m * 3 + 2] * dF[2][v];
#pragma unroll
          for (int k = 0; k < N1; ++k) h[m][v][k] += op.Wc[m][k][l] * ft;
        }
    }
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int v = 0; v < 5; ++v)
#pragma unroll
        for (int k = 0; k < N1; ++k) sc[((m * 5 + v) * N1 + k) * TP + t] = h[m][v][k];
  }
  __syncwarp();

  // ---- W, triangle part: one lane per (cell, variable, c-level) ----
  for (int it = lane; it < CW * 5 * N1; it += 32) {
    const int c = it / (5 * N1), vk = it - c * (5 * N1), v = vk / N1, k = vk - v * N1;
    T* sc = sw + c * L::cell;
    T o[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) o[j] = T(0);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const VecN<T>* hp = reinterpret_cast<const VecN<T>*>(sc + (m * 5 * N1 + vk) * TP);
#pragma unroll
      for (int tv = 0; tv < (MT + VN - 1) / VN; ++tv) {
        const VecN<T> xv = hp[tv];
#pragma unroll
        for (int i = 0; i < VN; ++i)
          if (tv * VN + i < MT) {
#pragma unroll
            for (int j = 0; j < NT; ++j) o[j] += op.Wt[m][j][tv * VN + i] * xv.v[i];
          }
      }
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) sc[L::oX + v * FS + j * N1 + k] = o[j];  // the deviations are consumed
  }
  __syncwarp();

  // ---- volume terms: -(W*dFt + MD*F(ref)) / det and the viscous part ----
#pragma unroll
  for (int r = 0; r < PR; ++r) {
    const int c = r * CPR + pc;
    if (pc < CPR && c < nc) {
      T* sc = sw + c * L::cell;
      const size_t p = (size_t)(e0 + c) * S + s;
      const double md0 = __ldg(pg.MD + p * 3), md1 = __ldg(pg.MD + p * 3 + 1), md2 = __ldg(pg.MD + p * 3 + 2);
      const double rdet = __ldg(pg.rdet + p);
      const double* F = reinterpret_cast<const double*>(sc + L::oF);
      const T* x = sc + L::oX + s;
      T* o = RV + (size_t)(e0 + c) * 9 * S + s;
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        const double mdf = md0 * F[v] + md1 * F[5 + v] + md2 * F[10 + v];
        o[v * S] = T(-(double(x[v * FS]) + mdf) * rdet);
        if (VISC && v > 0) o[(4 + v) * S] = x[(4 + v) * FS];
      }
    }
  }
}

// FP64 3 x 3 metric entries (npts <= 64 per cell, 9 each) -> planes (N, 9, npts),
// or with levels > 1 (N, levels, 9, npts / levels), point = j * levels + level.
// A CTA per cell, through shared memory: out may be adj (a second copy of the
// metrics would be a quarter of a P2 handle).
template <class T>
__global__ void __launch_bounds__(128) k_px_planes(const double* adj, int npts, int levels, T* out) {
  __shared__ double sh[64 * 9];
  const size_t base = (size_t)blockIdx.x * npts * 9;
  for (int t = threadIdx.x; t < npts * 9; t += blockDim.x) sh[t] = adj[base + t];
  __syncthreads();
  const int w = npts / levels;
  for (int t = threadIdx.x; t < npts * 9; t += blockDim.x) {
    const int j = t % w, k = t / w % 9, l = t / (w * 9);
    out[base + t] = T(sh[(j * levels + l) * 9 + k]);
  }
}

// ---- host: operator structure ----
// Each test returns its worst deviation relative to the operator's largest
// entry (infinity where the structure is absent altogether).

// Kronecker factors of an (R*r) x (K*k) operator at a(row, col): A = T (R x K) (x) c (r x k)
template <class Get>
inline double px_kron(int R, int r, int K, int k, Get a, std::vector<double>& T, std::vector<double>& c) {
  double big = 0.0, dev = 0.0;
  int pi = 0, pj = 0;
  for (int i = 0; i < R * r; ++i)
    for (int j = 0; j < K * k; ++j) {
      const double x = std::fabs(a(i, j));
      if (!(x <= 1e300)) return INFINITY;
      if (x > big) {
        big = x;
        pi = i;
        pj = j;
      }
    }
  if (big == 0.0) return INFINITY;
  T.assign((size_t)R * K, 0.0);
  c.assign((size_t)r * k, 0.0);
  for (int i = 0; i < R; ++i)
    for (int j = 0; j < K; ++j) T[i * K + j] = a(i * r + pi % r, j * k + pj % k);
  for (int i = 0; i < r; ++i)
    for (int j = 0; j < k; ++j) c[i * k + j] = a(pi / r * r + i, pj / k * k + j) / a(pi, pj);
  for (int i = 0; i < R * r; ++i)
    for (int j = 0; j < K * k; ++j)
      dev = std::max(dev, std::fabs(a(i, j) - T[(i / r) * K + j / k] * c[(i % r) * k + j % k]));
  return dev / big;
}

// Line and plane factors of a derivative operator D (S, S, 3), S = n^3
template <int n>
inline double px_lines(const double* D, double (&D0)[n][n], double (&D1)[n * n][n * n], double (&D2)[n][n]) {
  constexpr int NT = n * n, S = NT * n;
  auto d = [&](int s, int j, int m) { return D[((size_t)s * S + j) * 3 + m]; };
  double big = 0.0, dev = 0.0;
  for (int s = 0; s < S; ++s)
    for (int j = 0; j < S; ++j) {
      const double w[3] = {s % NT == j % NT ? d(s / NT * NT, j / NT * NT, 0) : 0.0,
                           s % n == j % n ? d(s / n * n, j / n * n, 1) : 0.0,
                           s / n == j / n ? d(s % n, j % n, 2) : 0.0};
      for (int m = 0; m < 3; ++m) {
        if (!(std::fabs(d(s, j, m)) <= 1e300)) return INFINITY;
        big = std::max(big, std::fabs(d(s, j, m)));
        dev = std::max(dev, std::fabs(d(s, j, m) - w[m]));
      }
    }
  if (big == 0.0) return INFINITY;
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      D0[i][j] = d(i * NT, j * NT, 0);
      D2[i][j] = d(i, j, 2);
    }
  for (int i = 0; i < NT; ++i)
    for (int j = 0; j < NT; ++j) D1[i][j] = d(i * n, j * n, 1);
  return dev / big;
}

// Derivative rows of every point for the FP64 kernels: (2*n + n*n, S), the
// point's weights along its a-line, triangle plane and c-line; each line also
// takes an equal share of the row's entries outside the structure.
template <int n>
inline std::vector<double> px_rows(const double* D) {
  constexpr int NT = n * n, S = NT * n;
  std::vector<double> out((size_t)(2 * n + NT) * S);
  for (int s = 0; s < S; ++s)
    for (int m = 0; m < 3; ++m) {
      const int cnt = m == 1 ? NT : n;
      std::vector<double> w(cnt, 0.0);
      double rest = 0.0;
      for (int j = 0; j < S; ++j) {
        const double x = D[((size_t)s * S + j) * 3 + m];
        if (m == 0 && j % NT == s % NT) w[j / NT] = x;
        else if (m == 1 && j % n == s % n) w[j / n] = x;
        else if (m == 2 && j / n == s / n) w[j % n] = x;
        else rest += x;
      }
      const int base = m == 0 ? 0 : (m == 1 ? n : n + NT);
      for (int l = 0; l < cnt; ++l) out[(size_t)(base + l) * S + s] = w[l] + rest / cnt;
    }
  return out;
}

// The structured operators of a prism set and their worst deviation from the
// given ones: D (S, S, 3), E (3, 2, P, S), c2f (Fn, S), relative to the largest
// entry, and the folded W = f2c * Df (S, Fn, 3), as the row's summed deviation
// over its l1 norm: what the contraction can be off by, in terms of its input.
// f2c (S, Fn) and Df (Fn, Fn, 3) only give W's factors: neither is applied by
// itself, and noise that is small in each can add up in their product.
template <int N1, int NF>
inline double px_operators(const double* D, const double* E, const double* c2f, const double* f2c, const double* Df,
                           const double* W, PxOps<double, N1, NF>& o) {
  constexpr int NT = N1 * N1, S = NT * N1, MT = NF * NF, FN = MT * NF, P = NT;
  double d0[N1][N1], d1[NT][NT], d2[N1][N1];  // the kernels take px_rows instead
  double dev = px_lines<N1>(D, d0, d1, d2);
  auto e = [&](int ax, int sd, int i, int s) { return E[(((size_t)ax * 2 + sd) * P + i) * S + s]; };
  double big = 0.0, de = 0.0;
  for (int i = 0; i < 6 * P * S; ++i) {
    if (!(std::fabs(E[i]) <= 1e300)) return INFINITY;
    big = std::max(big, std::fabs(E[i]));
  }
  if (big == 0.0) return INFINITY;
  for (int sd = 0; sd < 2; ++sd) {
    for (int i = 0; i < P; ++i)
      for (int s = 0; s < S; ++s) {
        const double w0 = s % NT == i ? e(0, sd, 0, s / NT * NT) : 0.0;
        const double w1 = s % N1 == i % N1 ? e(1, sd, i / N1 * N1, s / N1 * N1) : 0.0;
        const double w2 = s / N1 == i ? e(2, sd, 0, s % N1) : 0.0;
        de = std::max(de, std::max(std::fabs(e(0, sd, i, s) - w0),
                                   std::max(std::fabs(e(1, sd, i, s) - w1), std::fabs(e(2, sd, i, s) - w2))));
      }
    for (int l = 0; l < N1; ++l) {
      o.E02[0][sd][l] = e(0, sd, 0, l * NT);
      o.E02[1][sd][l] = e(2, sd, 0, l);
    }
    for (int a = 0; a < N1; ++a)
      for (int t = 0; t < NT; ++t) o.E1[sd][a][t] = e(1, sd, a * N1, t * N1);
  }
  dev = std::max(dev, de / big);
  std::vector<double> T, c;
  dev = std::max(dev, px_kron(MT, NF, NT, N1, [&](int i, int j) { return c2f[(size_t)i * S + j]; }, T, c));
  if (!(dev < 1.0)) return INFINITY;
  for (int i = 0; i < MT * NT; ++i) o.Ct[i / NT][i % NT] = T[i];
  for (int i = 0; i < NF * N1; ++i) o.Cc[i / N1][i % N1] = c[i];
  // W's factors from those of f2c and D_fine: (T (x) c) * (a-line, plane, c-line)
  double f0[NF][NF], f1[MT][MT], f2[NF][NF];
  if (!(px_kron(NT, N1, MT, NF, [&](int i, int j) { return f2c[(size_t)i * FN + j]; }, T, c) < 1.0) ||
      !(px_lines<NF>(Df, f0, f1, f2) < 1.0))
    return INFINITY;
  for (int r = 0; r < NT; ++r)
    for (int t = 0; t < MT; ++t) {
      double w0 = 0.0, w1 = 0.0;
      for (int l = 0; l < NF; ++l) w0 += T[r * MT + l * NF + t % NF] * f0[l][t / NF];
      for (int l = 0; l < MT; ++l) w1 += T[r * MT + l] * f1[l][t];
      o.Wt[0][r][t] = w0;
      o.Wt[1][r][t] = w1;
      o.Wt[2][r][t] = T[r * MT + t];
    }
  for (int k = 0; k < N1; ++k)
    for (int l = 0; l < NF; ++l) {
      double w2 = 0.0;
      for (int j = 0; j < NF; ++j) w2 += c[k * NF + j] * f2[j][l];
      o.Wc[0][k][l] = o.Wc[1][k][l] = c[k * NF + l];
      o.Wc[2][k][l] = w2;
    }
  for (int s = 0; s < S; ++s) {
    double off = 0.0, l1 = 0.0;
    for (int i = 0; i < FN; ++i)
      for (int m = 0; m < 3; ++m) {
        const double w = W[((size_t)s * FN + i) * 3 + m];
        off += std::fabs(w - o.Wt[m][s / N1][i / NF] * o.Wc[m][s % N1][i % NF]);
        l1 += std::fabs(w);
      }
    if (!(l1 <= 1e300) || l1 == 0.0) return INFINITY;
    dev = std::max(dev, off / l1);
  }
  return dev;
}

template <int N1, int NF>
inline PxOps<float, N1, NF> px_float(const PxOps<double, N1, NF>& d) {
  PxOps<float, N1, NF> f;
  static_assert(sizeof(f) * 2 == sizeof(d), "the same fields");
  const double* x = reinterpret_cast<const double*>(&d);
  float* y = reinterpret_cast<float*>(&f);
  for (size_t i = 0; i < sizeof(f) / sizeof(float); ++i) y[i] = (float)x[i];
  return f;
}

}  // namespace afr
