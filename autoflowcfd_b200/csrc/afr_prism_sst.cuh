// SST kernels of prisms with tensor-product operators (afr_prism.cuh): a warp
// owns its cells, a lane a solution point, derivatives along lines and planes
// in plain FP64 multiply-adds.
//
// The generic kernels form the gradients and the transport divergence as dense
// FP64 tensor products, of whose 81 x 27 entries 15 in 81 are nonzero for
// these operators, and read the cells' metrics and point values twice.  Here
// the point kernel also forms the volume part of the transport, so the update
// kernel reads five numbers per point and the face corrections.
#pragma once
#include "afr_prism.cuh"
#include "afr_sst.cuh"

namespace afr {

constexpr int PXS_WARPS = 4;

// rows: (2*N1 + N1*N1, S) derivative weights of each point along its a-line,
// triangle plane and c-line, with the operator's entries outside the structure
// (rounding noise of its construction) added to the row's own, so that
// constants are differentiated exactly as the full operator does
template <int N1>
struct PxsSmem {
  static constexpr int S = N1 * N1 * N1, CPR = 32 / S;
  static constexpr int cell = 18 * S;  // doubles: state (7) then fluxes (6), inverse Jacobian (9), k, omega
  static constexpr int total = PXS_WARPS * CPR * cell * 8;
};

// pt of a structured prism, field-major (N, 5, S): source increments of k and
// omega (point-implicit), volume transport of k and omega over rho, 1 / (rho det)
template <int N1>
__global__ void __launch_bounds__(32 * PXS_WARPS)
    k_pxs_point(const double* __restrict__ rows, Geom g, SstArgs a, int cell_base, int cell_end) {
  using L = PxsSmem<N1>;
  constexpr int S = L::S, NT = N1 * N1, CPR = L::CPR;
  extern __shared__ __align__(16) double smd[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e0 = cell_base + (blockIdx.x * PXS_WARPS + warp) * CPR;
  const int nc = min(CPR, cell_end - e0);
  if (nc <= 0) return;  // whole warps; no block barrier below
  const int s = lane % S, c = lane / S < CPR ? lane / S : 0;
  const bool on = lane / S < nc;
  const int cc = s % N1;
  const int nv = a.nv;
  double* sw = smd + warp * CPR * L::cell;
  for (int b = 0; b < nc; ++b) {
    double* sc = sw + b * L::cell;
    const double* ub = a.U + (size_t)(e0 + b) * S * nv;
    for (int t = lane; t < S * nv; t += 32) cp_async8(sc + t, ub + t);
    const double* ib = g.inv + (size_t)(e0 + b) * S * 9;
    for (int t = lane; t < S * 9; t += 32) cp_async8(sc + 7 * S + t, ib + t);
    for (int t = lane; t < S; t += 32) {
      cp_async8(sc + 16 * S + 2 * t, a.k + (size_t)(e0 + b) * S + t);
      cp_async8(sc + 16 * S + 2 * t + 1, a.w + (size_t)(e0 + b) * S + t);
    }
  }
  cp_async_commit();
  const size_t p = (size_t)(e0 + (c < nc ? c : 0)) * S + s;
  const double wd = __ldg(g.wall_dist + p), dts = __ldg(a.dt + p), det = __ldg(g.det + p);
  double d0[N1], d1[NT], d2[N1];  // this point's rows of the derivative operators
#pragma unroll
  for (int l = 0; l < N1; ++l) {
    d0[l] = __ldg(rows + l * S + s);
    d2[l] = __ldg(rows + (N1 + NT + l) * S + s);
  }
#pragma unroll
  for (int t = 0; t < NT; ++t) d1[t] = __ldg(rows + (N1 + t) * S + s);
  cp_async_wait0();
  __syncwarp();
  double* sc = sw + c * L::cell;
  const double* kw = sc + 16 * S;
  double gp[5][3];
  {
    double r[3][5];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int q = 0; q < 5; ++q) r[m][q] = 0.0;
    auto acc = [&](double (&o)[5], double w, int j) {
#pragma unroll
      for (int q = 0; q < 3; ++q) o[q] += w * sc[j * nv + 1 + q];
      o[3] += w * kw[2 * j];
      o[4] += w * kw[2 * j + 1];
    };
#pragma unroll
    for (int l = 0; l < N1; ++l) {
      acc(r[0], d0[l], l * NT + s % NT);
      acc(r[2], d2[l], s - cc + l);
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) acc(r[1], d1[t], t * N1 + cc);
    const double* inv = sc + 7 * S + 9 * s;
#pragma unroll
    for (int q = 0; q < 5; ++q)
#pragma unroll
      for (int n = 0; n < 3; ++n) gp[q][n] = r[0][q] * inv[n] + r[1][q] * inv[3 + n] + r[2][q] * inv[6 + n];
  }
  double u[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) u[v] = sc[s * nv + v];
  const double kf = kw[2 * s], wf = kw[2 * s + 1];
  const double graw[2][3] = {{gp[3][0], gp[3][1], gp[3][2]}, {gp[4][0], gp[4][1], gp[4][2]}};
  const double rho = fmax(u[0], 1e-10), rrho = 1.0 / rho;
  const double vel[3] = {u[1] * rrho, u[2] * rrho, u[3] * rrho};
  const SstPoint o = sst_closure(gp, rho, kf, wf, wd, a.mu);
  __syncwarp();  // the state rows are consumed: their space receives the fluxes
  {
    const double* inv = sc + 7 * S + 9 * s;
    double* F = sc + 2 * s;  // [m][point][k, omega]
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const double a0 = det * inv[m * 3], a1 = det * inv[m * 3 + 1], a2 = det * inv[m * 3 + 2];
      const double vm = rho * (a0 * vel[0] + a1 * vel[1] + a2 * vel[2]);
      const double fk = vm * kf + o.gk * (a0 * graw[0][0] + a1 * graw[0][1] + a2 * graw[0][2]);
      const double fw = vm * wf + o.gw * (a0 * graw[1][0] + a1 * graw[1][1] + a2 * graw[1][2]);
      if (lane / S < CPR) {
        F[2 * m * S] = fk;
        F[2 * m * S + 1] = fw;
      }
    }
  }
  __syncwarp();
  double dk = 0.0, dw = 0.0;
  {
    const double2* F = reinterpret_cast<const double2*>(sc);
    auto acc = [&](double w, const double2& x) {
      dk += w * x.x;
      dw += w * x.y;
    };
#pragma unroll
    for (int l = 0; l < N1; ++l) {
      acc(d0[l], F[l * NT + s % NT]);
      acc(d2[l], F[2 * S + s - cc + l]);
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) acc(d1[t], F[S + t * N1 + cc]);
  }
  if (!on) return;
  const double rr = rrho / det;
  const double wo = fmax(wf, 1e-10);
  double* pt = a.pt + (size_t)(e0 + c) * 5 * S + s;
  pt[0] = dfinite((o.Sk * rrho) / (1.0 + dts * (SST_BSTAR * wo)));
  pt[S] = dfinite((o.Sw * rrho) / (1.0 + dts * (o.beta * wo)));
  pt[2 * S] = -dk * rr;
  pt[3 * S] = -dw * rr;
  pt[4 * S] = rr;
  a.nut[p] = o.nut;
  double2* o8 = reinterpret_cast<double2*>(a.sp8 + p * 8);
  o8[0] = make_double2(rho, vel[0]);
  o8[1] = make_double2(vel[1], vel[2]);
  o8[2] = make_double2(kf, wf);
  o8[3] = make_double2(o.gk, o.gw);
  if (a.dbg) {
    a.dbg[p * 4 + 0] = o.Sk;
    a.dbg[p * 4 + 1] = o.Sw;
  }
}

constexpr int PXS_SLOTS = 8;  // transport slots of a prism (3 split quads, 2 triangles), loaded together

// face corrections in ascending color order, outliers, update of k and omega
template <int S, int NP>
__global__ void __launch_bounds__(32 * PXS_WARPS) k_pxs_update(Ops ops, Faces fc, SstArgs a, int cell_base,
                                                               int cell_end) {
  constexpr int CPR = 32 / S;
  __shared__ double sG[6 * S];
  __shared__ int sFp[3 * S];
  for (int t = threadIdx.x; t < 3 * S; t += blockDim.x) {
    const int co = ops.dist_co[t];
    sG[t] = ops.g_left[co];
    sG[3 * S + t] = ops.g_right[co];
    sFp[t] = ops.dist_fp[t];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e0 = cell_base + (blockIdx.x * PXS_WARPS + warp) * CPR;
  const int nc = min(CPR, cell_end - e0);
  if (nc <= 0) return;  // whole warps
  const int grp = lane / S, s = lane % S;
  const bool on[1] = {grp < nc};
  const int c = on[0] ? grp : 0, e = e0 + c;
  const size_t p = (size_t)e * S + s;
  const double* pt = a.pt + (size_t)e * 5 * S + s;
  const double dkd = __ldg(pt), dwd = __ldg(pt + S), tk0 = __ldg(pt + 2 * S), tw0 = __ldg(pt + 3 * S),
               rr = __ldg(pt + 4 * S);
  const double kf = a.k[p], wf = a.w[p], dts = __ldg(a.dt + p);
  const int ptr = __ldg(fc.tslot_ptr + e0 + min(lane, nc));
  const int kb = __shfl_sync(0xffffffffu, ptr, 0), ke = __shfl_sync(0xffffffffu, ptr, nc);
  const int code = kb + lane < ke ? __ldg(fc.tslot + kb + lane) : 0;
  const int k0 = __shfl_sync(0xffffffffu, ptr, c), n = __shfl_sync(0xffffffffu, ptr, c + 1) - k0;
  const double2* cfp = reinterpret_cast<const double2*>(a.cfp);
  double ck = 0.0, cw = 0.0;
  if (__all_sync(0xffffffffu, n == PXS_SLOTS)) {  // then at most CPR * 8 <= 32 slots: every code is held by a lane
    double2 cv[PXS_SLOTS];
    int gi[PXS_SLOTS];
#pragma unroll
    for (int j = 0; j < PXS_SLOTS; ++j) {
      const int q = __shfl_sync(0xffffffffu, code, k0 - kb + j);
      const int as = ((q >> 2) & 3) * S + s;
      gi[j] = (((q & 1) ? 3 * S : 0) + as) | ((q & 2) ? 0x40000000 : 0);
      cv[j] = __ldg(cfp + (size_t)(q >> 4) * NP + sFp[as]);
    }
#pragma unroll
    for (int j = 0; j < PXS_SLOTS; ++j) {
      const double g = sG[gi[j] & 0x3fffffff];
      const double gw = (gi[j] & 0x40000000) ? g : -g;
      ck += gw * cv[j].x;
      cw += gw * cv[j].y;
    }
  } else {
    for (int j = 0; j < n; ++j) {
      const int q = __ldg(fc.tslot + k0 + j);
      const int as = ((q >> 2) & 3) * S + s;
      const double g = sG[((q & 1) ? 3 * S : 0) + as];
      const double gw = (q & 2) ? g : -g;
      const double2 cv = __ldg(cfp + (size_t)(q >> 4) * NP + sFp[as]);
      ck += gw * cv.x;
      cw += gw * cv.y;
    }
  }
  double x[2][1] = {{tk0 + ck * rr}, {tw0 + cw * rr}};
  unsigned bad = 0u;
#pragma unroll
  for (int q = 0; q < 2; ++q) bad |= mxd::outlier_clear<S, 1>(x[q], on, grp) ? 0u : 1u << q;
  bad = S == 8 ? __reduce_or_sync(0xffffffffu, bad) : bad;
#pragma unroll
  for (int q = 0; q < 2; ++q)
    if (bad >> q & 1u) {
      mxd::Vals<1> X, ref;
      X.v[0] = x[q][0];
      ref.v[0] = on[0] ? (q == 0 ? kf : wf) : 0.0;
      X = mxd::outlier_exact<S, 1>(X, ref, grp < CPR ? grp : 0, s, on[0]);
      x[q][0] = X.v[0];
    }
  if (!on[0]) return;
  const double tk = dfinite(x[0][0]), tw = dfinite(x[1][0]);
  double kn = kf + dts * dfinite(dkd + tk);
  double wn = wf + dts * dfinite(dwd + tw);
  if (!isfinite(kn)) kn = 1e-12;
  if (!isfinite(wn)) wn = 1e-12;
  a.k[p] = fmax(kn, 1e-12);
  a.w[p] = fmax(wn, 1e-12);
  if (a.dbg) {
    a.dbg[p * 4 + 2] = tk;
    a.dbg[p * 4 + 3] = tw;
  }
}

}  // namespace afr
