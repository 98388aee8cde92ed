// Discrete adjoint of one SSP-RK3 stage: the transpose of the linearised
// right-hand side L(u) = M^{-1} R(u) applied to an adjoint vector, fused with
// the reversed stage combination.  The forward operator is the one of
// dgp_kernels.cuh / dgp_elem.cuh (DGCell::computeVolumeContribution,
// DGCell.cc:184-249; DGBoundaryCell::computeBoundaryContributions,
// DGCell.cc:639-732; RungeKuttaTVD3::advanceInTime, TimeIntegrator.cc:838-990).
//
// With nu = mu / |J| per cell (the inverse mass is diagonal):
//   faces   per face point, the traces of nu on both sides give the flux
//           cotangent Fbar = (nu_R - nu_L) |J_f| w; the Jacobians dF^/dU_L and
//           dF^/dU_R come from evaluating the law's numerical (or boundary)
//           flux on dual numbers (the Roe flux: its own reverse pass,
//           roe_vjp); U_L^bar = Fbar dF^/dU_L is written into the
//           left cell's face slot, U_R^bar into the right cell's (no atomics,
//           the forward slot layout);
//   volume  H[(cell,j)][(q,r)] = sum_k dphi_(q,r),k nu[j][k] (the transposed
//           contraction), flux cotangent Fbar_ji = sum_r H_jr J^{-1}_ir |J| w_q,
//           U^bar_m(q) = sum_ji Fbar_ji dF_ji/dU_m(U(q)) (dual numbers), and
//           w[m][k] = sum_q phi_k(q) U^bar_m(q) + sum_s slot_s[m] phi_s,k (the
//           same lift as the forward face term).
// Stage combination (per row, FP64): out = ca mu + cb dt w + cc acc and
// acc <- cd acc + ce mu, which runs the three reversed stages
//   lambda2 = 2/3 lambda3 + 2/3 dt L'(u2)^T lambda3,  acc = 1/3 lambda3
//   lambda1 = 1/4 lambda2 + 1/4 dt L'(u1)^T lambda2,  acc += 3/4 lambda2
//   lambda_n = acc + lambda1 + dt L'(u_n)^T lambda1.
#pragma once

#include "dgp_dual.cuh"
#include "dgp_stage.cuh"

namespace dgp {

template <typename T>
struct AdjArgs {
  StageArgs<T> s;      // forward state of the stage in s.C, tables, geometry, slots
  const double* mu;    // adjoint input [cell][field][mode] (internal order)
  double* out;         // adjoint output
  double* acc;         // running sum of the reversed stages (read and/or written)
  double ca, cb, cc, cd, ce;
  double dt;
  const double* t_seg; // device: time at the start of the step
  double t_factor;     // stage time = *t_seg + t_factor * dt (as the forward stage)
};

// input directions per dual-number pass of the face Jacobians: the 2M
// directions of both sides in as few passes of at most 8 lanes as possible,
// split evenly (one pass for the 2D Euler law: 0.90x the backward time of two
// lanes a pass on the adjoint workload); two lanes for the exact Riemann
// solver, whose iteration would otherwise carry 8-lane dual numbers
template <class K>
constexpr int adj_lanes() {
  constexpr int dirs = 2 * K::M, passes = (dirs + 7) / 8;
  return K::FLUX == DGP_FLUX_GODUNOV ? 2 : (dirs + passes - 1) / passes;
}

// numerical fluxes with a hand-written reverse pass (flux_vjp); boundary faces
// of the others and theirs run on dual numbers
template <class K>
constexpr bool flux_vjp_built() {
  return K::LAW == DGP_LAW_EULER2D && K::FLUX == DGP_FLUX_ROE;
}

// gL = fb dF^/dU_L, gR = fb dF^/dU_R of the Roe flux (numerical_flux): the
// reverse pass of its own steps, ~350 operations where 8-lane dual numbers carry
// nine times the flux's 250 (P2 Euler, 32768 cells: 49 -> 29 us a launch; the
// whole gradient 6.92 -> 5.88 ms at three blocks a SM, 6.02 at four, 6.06 at two).
// x_ stands for the cotangent of x.
template <typename T>
__device__ __forceinline__ void roe_vjp(T g, const T* n, const T* u0, const T* u1, const T* fb, T* gL, T* gR) {
  const T half = (T)0.5, gm1 = g - (T)1, n0 = n[0], n1 = n[1];
  struct Side {
    T rho, is, r, ir, u, v, p, H;     // 1 / sqrt(rho), sqrt(rho), 1 / rho
    T rho_, m1_, m2_, E_, u_, v_, p_, H_, r_;
  } a, b;
  auto state = [&](const T* U, Side& s) {
    s.rho = U[0];
    s.is = inv_sqrt(s.rho);
    s.r = s.rho * s.is;
    s.ir = s.is * s.is;
    s.u = U[1] * s.ir;
    s.v = U[2] * s.ir;
    s.p = gm1 * (U[3] - half * (U[1] * U[1] + U[2] * U[2]) * s.ir);
    s.H = (U[3] + s.p) * s.ir;
    // the half of the physical flux: (m.n, m1 vn + p n0, m2 vn + p n1, (E + p) vn)
    const T h0 = half * fb[0], h1 = half * fb[1], h2 = half * fb[2], h3 = half * fb[3];
    const T vn = s.u * n0 + s.v * n1, vn_ = h1 * U[1] + h2 * U[2] + h3 * (U[3] + s.p);
    s.p_ = h1 * n0 + h2 * n1 + h3 * vn;
    s.m1_ = h0 * n0 + h1 * vn;
    s.m2_ = h0 * n1 + h2 * vn;
    s.E_ = h3 * vn;
    s.u_ = vn_ * n0;
    s.v_ = vn_ * n1;
    s.rho_ = s.H_ = s.r_ = (T)0;
  };
  state(u0, a);
  state(u1, b);
  const T D = (T)1 / (a.r + b.r), rA = a.r * b.r, w0 = a.r * D, w1 = b.r * D;
  const T uA = a.u * w0 + b.u * w1, vA = a.v * w0 + b.v * w1, HA = a.H * w0 + b.H * w1;
  const T q2 = uA * uA + vA * vA, qq = HA - half * q2;
  if (qq > (T)0) {
    const T c2 = gm1 * qq, ic = inv_sqrt(c2), c = c2 * ic, ic2 = ic * ic;
    const T vn = uA * n0 + vA * n1;
    const T e1 = fabs(vn), e3 = fabs(vn + c), e4 = fabs(vn - c);
    const T dr = b.rho - a.rho, dp = b.p - a.p, du = b.u - a.u, dv = b.v - a.v;
    const T dun = n0 * du + n1 * dv, dut = n1 * du - n0 * dv, k = half * rA * ic;
    // wave strengths and their cotangents
    const T a1 = dr - dp * ic2, a3 = k * dun + half * dp * ic2, a4 = half * dp * ic2 - k * dun;
    const T s1 = e1 * a1, s2 = e1 * dut * rA, s3 = e3 * a3, s4 = e4 * a4;
    const T R0 = -half * fb[0], R1 = -half * fb[1], R2 = -half * fb[2], R3 = -half * fb[3];
    const T S_ = R0 + R1 * uA + R2 * vA, T_ = R1 * n0 + R2 * n1 + R3 * vn;
    const T s1_ = S_ + R3 * half * q2, s2_ = R1 * n1 - R2 * n0 + R3 * (uA * n1 - vA * n0);
    const T s3_ = S_ + R3 * HA + T_ * c, s4_ = S_ + R3 * HA - T_ * c;
    const T S = s1 + s3 + s4, d34 = s3 - s4;
    T c_ = T_ * d34, vn_ = R3 * d34 * c, H_ = R3 * (s3 + s4);
    T u_ = R1 * S + R3 * (s1 * uA + s2 * n1), v_ = R2 * S + R3 * (s1 * vA - s2 * n0);
    const T e1_ = s1_ * a1 + s2_ * dut * rA, e3_ = s3_ * a3, e4_ = s4_ * a4;
    const T a1_ = s1_ * e1, a3_ = s3_ * e3, a4_ = s4_ * e4;
    const T g1 = vn < (T)0 ? -e1_ : e1_, g3 = vn + c < (T)0 ? -e3_ : e3_, g4 = vn - c < (T)0 ? -e4_ : e4_;
    vn_ += g1 + g3 + g4;
    c_ += g3 - g4;
    const T d_ = a3_ - a4_, m_ = half * (a3_ + a4_);
    const T dp_ = (m_ - a1_) * ic2, ic2_ = (m_ - a1_) * dp;
    const T dun_ = d_ * k, dut_ = s2_ * e1 * rA, k_ = d_ * dun;
    const T rA_ = s2_ * e1 * dut + half * ic * k_;
    const T c2_ = half * ic * (c_ - half * rA * k_ * ic2) - ic2 * ic2 * ic2_;
    const T q_ = gm1 * c2_;
    H_ += q_;
    u_ += vn_ * n0 - q_ * uA;
    v_ += vn_ * n1 - q_ * vA;
    const T du_ = n0 * dun_ + n1 * dut_, dv_ = n1 * dun_ - n0 * dut_;
    auto side = [&](Side& s, T w, T other, T sign) {
      s.u_ += u_ * w + sign * du_;
      s.v_ += v_ * w + sign * dv_;
      s.H_ += H_ * w;
      s.r_ += D * (u_ * (s.u - uA) + v_ * (s.v - vA) + H_ * (s.H - HA)) + rA_ * other;
      s.rho_ += sign * a1_;
      s.p_ += sign * dp_;
    };
    side(a, w0, b.r, (T)-1);
    side(b, w1, a.r, (T)1);
  }
  auto conserved = [&](Side& s, T* gs) {
    s.rho_ += half * s.r_ * s.is - s.H_ * s.H * s.ir;
    s.E_ += s.H_ * s.ir;
    s.p_ += s.H_ * s.ir;
    const T P = gm1 * s.p_;
    gs[0] = s.rho_ + P * half * (s.u * s.u + s.v * s.v) - (s.u_ * s.u + s.v_ * s.v) * s.ir;
    gs[1] = s.m1_ - P * s.u + s.u_ * s.ir;
    gs[2] = s.m2_ - P * s.v + s.v_ * s.ir;
    gs[3] = s.E_ + P;
  };
  conserved(a, gL);
  conserved(b, gR);
}

// trace of nu = mu / |J| at one face point
template <class K>
__device__ __forceinline__ void nu_trace(const double* __restrict__ mu, double inv_detj,
                                         const typename K::T* phi, typename K::T* V) {
  // (the vector of the previous launch: plain loads, not the read-only path)
  using T = typename K::T;
  constexpr int NP = K::NP;
#pragma unroll
  for (int j = 0; j < K::M; ++j) {
    T acc = 0;
    if constexpr (NP % 2 == 0) {
#pragma unroll
      for (int k = 0; k < NP; k += 2) {
        const double2 v = *reinterpret_cast<const double2*>(mu + j * NP + k);
        acc += phi[k] * (T)v.x;
        acc += phi[k + 1] * (T)v.y;
      }
    } else {
#pragma unroll
      for (int k = 0; k < NP; ++k) acc += phi[k] * (T)mu[j * NP + k];
    }
    V[j] = acc * (T)inv_detj;
  }
}

template <class K>
__global__ void __launch_bounds__(K::FACE_BLOCK, flux_vjp_built<K>() ? 3 : 1)
    adj_face_kernel(const __grid_constant__ AdjArgs<typename K::T> a) {
  using T = typename K::T;
  constexpr int M = K::M, NP = K::NP, NQF = K::NQF, DIM = K::DIM, MNP = K::MNP;
  __shared__ T s_phif[K::NLF * NQF * NP];
  __shared__ T s_fqw[NQF];
  __shared__ int s_qmap[K::NPERM * NQF];
  face_tables<K>(a.s, s_phif, s_fqw, s_qmap);
  const int tid = threadIdx.x;
  const int fl = tid / NQF, q = tid - (tid / NQF) * NQF;
  const int f = blockIdx.x * K::FPB + fl;
  pdl_wait();  // (tables and weights are constant; a trigger after the wait keeps the
  pdl_trigger();  //  stage states that cell_trace reads complete before the kernel starts)
  if (fl >= K::FPB || f >= a.s.mesh.F) return;
  const auto& m = a.s.mesh;
  const int eL = m.fel[2 * f], eR = m.fel[2 * f + 1];
  const int code = m.fcode[f];
  const int lfL = code & 15, lfR = (code >> 4) & 15, perm = code >> 8;
  T n[DIM];
#pragma unroll
  for (int i = 0; i < DIM; ++i) n[i] = m.fnrm[f * DIM + i];
  const T jw = m.fj[f] * s_fqw[q];
  T UL[M], UR[M], VL[M], VR[M], gL[M], gR[M];
  const T* phiL = s_phif + (lfL * NQF + q) * NP;
  cell_trace<K>(a.s.C + (size_t)eL * MNP, phiL, UL);
  nu_trace<K>(a.mu + (size_t)eL * MNP, 1.0 / m.detjd[eL], phiL, VL);
  if (eR >= 0) {
    const int qR = s_qmap[perm * NQF + q];
    const T* phiR = s_phif + (lfR * NQF + qR) * NP;
    cell_trace<K>(a.s.C + (size_t)eR * MNP, phiR, UR);
    nu_trace<K>(a.mu + (size_t)eR * MNP, 1.0 / m.detjd[eR], phiR, VR);
    T fb[M];
#pragma unroll
    for (int j = 0; j < M; ++j) fb[j] = (VR[j] - VL[j]) * jw;
    if constexpr (flux_vjp_built<K>()) {
      roe_vjp<T>((T)a.s.law.p[7], n, UL, UR, fb, gL, gR);
    } else {
      // the Jacobian W input directions per pass (narrow dual numbers keep the
      // flux in registers); direction c < M is d/dU_L[c], c >= M is d/dU_R[c - M]
      constexpr int W = adj_lanes<K>();
      using D = Dual<T, W>;
#pragma unroll 1
      for (int c0 = 0; c0 < 2 * M; c0 += W) {
        D dl[M], dr[M], nd[DIM], F[M];
#pragma unroll
        for (int j = 0; j < M; ++j) {
          dl[j] = D::var(UL[j], j - c0);
          dr[j] = D::var(UR[j], M + j - c0);
        }
#pragma unroll
        for (int i = 0; i < DIM; ++i) nd[i] = D(n[i]);
        numerical_flux<K::LAW, K::FLUX, DIM, D>(a.s.law, nd, dl, dr, F);
#pragma unroll
        for (int w = 0; w < W; ++w) {
          T g = 0;
#pragma unroll
          for (int j = 0; j < M; ++j) g += fb[j] * F[j].d[w];
          const int c = c0 + w;
#pragma unroll
          for (int k = 0; k < M; ++k) {
            if (k == c) gL[k] = g;
            if (k + M == c) gR[k] = g;
          }
        }
      }
    }
    T* sr = a.s.slots + slot_index<K>(eR, lfR * NQF + qR, 0);
#pragma unroll
    for (int c = 0; c < M; ++c) sr[c] = gR[c];
  } else {
    constexpr int W = flux_vjp_built<K>() ? 2 : adj_lanes<K>();
    using D = Dual<T, W>;
    const int b = -eR - 1;
    const double* x = m.bpts + ((size_t)b * NQF + q) * 3;
    const double time = __fma_rn(a.t_factor, a.dt, *a.t_seg);
#pragma unroll 1
    for (int c0 = 0; c0 < M; c0 += W) {
      D dl[M], nd[DIM], F[M];
#pragma unroll
      for (int j = 0; j < M; ++j) dl[j] = D::var(UL[j], j - c0);
#pragma unroll
      for (int i = 0; i < DIM; ++i) nd[i] = D(n[i]);
      boundary_flux<K::LAW, K::FLUX, DIM, D>(a.s.law, m.bbid[b], nd, x, time, dl, F);
#pragma unroll
      for (int w = 0; w < W; ++w) {
        T g = 0;
#pragma unroll
        for (int j = 0; j < M; ++j) g += -VL[j] * jw * F[j].d[w];
#pragma unroll
        for (int k = 0; k < M; ++k)
          if (k == c0 + w) gL[k] = g;
      }
    }
  }
  T* sl = a.s.slots + slot_index<K>(eL, lfL * NQF + q, 0);
#pragma unroll
  for (int c = 0; c < M; ++c) sl[c] = gL[c];
}

// shared memory of the element kernel: values at the volume points (then
// U^bar) and H, field-major rows as in the stage kernel
template <class K>
struct AdjSmem {
  using T = typename K::T;
  using S = StageShape<K>;
  static constexpr size_t oH = (size_t)S::VQ * S::LDR * sizeof(T);
  static constexpr size_t bytes = oH + (size_t)S::KV * S::LDR * sizeof(T) + 16;
};

template <class K>
constexpr size_t adj_elem_smem() {
  return AdjSmem<K>::bytes;
}

// Element part of a reversed stage, the work mapping of the stage kernel: one
// thread per (cell, field) row contracts the stage state and nu from registers
// against constant-bank tables (U at the volume points, H), thread (cell,
// point) the flux cotangents on dual numbers, then the rows again.  Linear
// laws: the volume points are the modes of degree < p (stage kernel), the
// transposed table and U^bar's modes directly.  P2 Euler on 32768 cells:
// 30 -> 13 us a launch (tables and rows read from shared memory before).
template <class K>
__global__ void __launch_bounds__(K::BLOCK) adj_elem_kernel(const __grid_constant__ AdjArgs<typename K::T> a,
                                                            const __grid_constant__ StageTab<K> tb) {
  using T = typename K::T;
  using S = StageShape<K>;
  constexpr int M = K::M, NP = K::NP, DIM = K::DIM, TS = K::TS, BLOCK = K::BLOCK;
  constexpr int NS = K::NS, VQ = S::VQ, KV = S::KV, LDR = S::LDR, TEP = S::TEP;
  constexpr int RALIGN = pow2_div(NP * 8) < 16 ? pow2_div(NP * 8) : 16;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T* sU = reinterpret_cast<T*>(smem_raw);
  T* sH = reinterpret_cast<T*>(smem_raw + AdjSmem<K>::oH);
  const int tid = threadIdx.x;
  const int e0 = blockIdx.x * TS;
  const auto& m = a.s.mesh;
  const int ne = min(TS, m.E - e0);
  const int row = tid, cell = row / M, field = row - cell * M, prow = field * TEP + cell;
  const bool live = row < ne * M;
  const size_t gbase = ((size_t)e0 * M + row) * NP;
  const double det = live ? m.detjd[e0 + cell] : 1.0;
  // a cell's geometry for its points' threads
  constexpr int NG = BLOCK / TS;
  const int ve = tid % TS, vg = tid / TS;
  const bool vlive = vg < NG && ve < ne;
  T J[DIM * DIM], vdet = 0;
  if (vlive) {
#pragma unroll
    for (int i = 0; i < DIM * DIM; ++i) J[i] = m.jinv[(size_t)(e0 + ve) * DIM * DIM + i];
    vdet = (T)m.detjd[e0 + ve];
  }
  pdl_wait();
  pdl_trigger();

  if (live) {
    constexpr int UV = table_unroll(VQ > 0 ? VQ : 1, NP), UK = table_unroll(KV > 0 ? KV : 1, NP);
    double v[NP];
    T c[NP];
    ld_row_pinned<NP, RALIGN>(a.s.C + gbase, v);
#pragma unroll
    for (int k = 0; k < NP; ++k) c[k] = (T)v[k];
#pragma unroll UV
    for (int q = 0; q < VQ; ++q) {
      if constexpr (S::LINEAR)
        sU[q * LDR + prow] = c[q];
      else
        sU[q * LDR + prow] = table_dot<NP, false, T>(c, tb.phi + q * NP, 0);
    }
    // H[(direction, point)][row] = sum_k dv[(direction, point)][k] nu[row][k]
    ld_row_pinned<NP, RALIGN>(a.mu + gbase, v);
#pragma unroll
    for (int k = 0; k < NP; ++k) c[k] = (T)(v[k] / det);
#pragma unroll UK
    for (int kk = 0; kk < KV; ++kk) sH[kk * LDR + prow] = table_dot<NP, false, T>(c, tb.dv + kk * NP, 0);
  }
  __syncthreads();

  // U^bar_m(q) = sum_ji Fbar_ji dF_ji/dU_m at each volume point
  if (vlive) {
    using D = Dual<T, M>;
#pragma unroll 1
    for (int q = vg; q < VQ; q += NG) {
      D U[M];
#pragma unroll
      for (int j = 0; j < M; ++j) U[j] = D::var(sU[q * LDR + j * TEP + ve], j);
      D F[M][DIM];
      volume_flux<K::LAW, DIM, D>(a.s.law, U, F);
      T jw = vdet;
      if constexpr (!S::LINEAR) jw = vdet * tb.qw[q];
      T ub[M];
#pragma unroll
      for (int c = 0; c < M; ++c) ub[c] = 0;
#pragma unroll
      for (int j = 0; j < M; ++j) {
        T h[DIM];
#pragma unroll
        for (int r = 0; r < DIM; ++r) h[r] = sH[(r * VQ + q) * LDR + j * TEP + ve];
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
          T fb = 0;
#pragma unroll
          for (int r = 0; r < DIM; ++r) fb += h[r] * J[i * DIM + r];
          fb *= jw;
#pragma unroll
          for (int c = 0; c < M; ++c) ub[c] += fb * F[j][i].d[c];
        }
      }
#pragma unroll
      for (int c = 0; c < M; ++c) sU[q * LDR + c * TEP + ve] = ub[c];
    }
  }
  __syncthreads();

  // w = sum_q phi_k(q) U^bar(q) + lift of the adjoint face slots, then the
  // reversed stage combination in FP64
  if (live) {
    double mu[NP], ac[NP];
    ld_row_pinned<NP, RALIGN>(a.mu + gbase, mu);
    const bool use_acc = a.cc != 0.0 || a.cd != 0.0;
    if (use_acc) ld_row_pinned<NP, RALIGN>(a.acc + gbase, ac);
    T acc[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) acc[k] = 0;
    constexpr int UV = table_unroll(VQ > 0 ? VQ : 1, NP), UF = table_unroll(NS, NP);
    if constexpr (S::LINEAR) {
#pragma unroll
      for (int q = 0; q < VQ; ++q) acc[q] = sU[q * LDR + prow];
    } else {
#pragma unroll UV
      for (int q = 0; q < VQ; ++q) {
        const T ub = sU[q * LDR + prow];
#pragma unroll
        for (int k = 0; k < NP; ++k) acc[k] += ub * tb.phi[q * NP + k];
      }
    }
    const T* sl = a.s.slots + slot_index<K>(e0 + cell, 0, field);
#pragma unroll UF
    for (int s = 0; s < NS; ++s) {
      const T sv = sl[(size_t)s * K::ROWS];
#pragma unroll
      for (int k = 0; k < NP; ++k) acc[k] += sv * tb.phif[s * NP + k];
    }
    double o[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      o[k] = a.ca * mu[k] + a.cb * a.dt * (double)acc[k];
      if (a.cc != 0.0) o[k] += a.cc * ac[k];
    }
    st_row<NP, RALIGN>(a.out + gbase, o);
    if (a.cd != 0.0 || a.ce != 0.0) {
#pragma unroll
      for (int k = 0; k < NP; ++k) o[k] = (a.cd != 0.0 ? a.cd * ac[k] : 0.0) + a.ce * mu[k];
      st_row<NP, RALIGN>(a.acc + gbase, o);
    }
  }
}

// ---- objective: J = sum_r (rho(x_r) - obs_r)^2 at receiver points ----------
struct Receivers {
  int n;
  const int* cell;       // internal cell of each receiver
  const double* phi;     // [n][NP] basis at the receiver's reference point
  const double* obs;     // [n]
  int np, mnp;
};

// rho at the receivers (field 0) and J, one block of 256 threads
static __global__ void receiver_values_kernel(Receivers r, const double* C, double* rho, double* J) {
  __shared__ double red[32];
  double acc = 0.0;
  for (int i = threadIdx.x; i < r.n; i += blockDim.x) {
    const double* c = C + (size_t)r.cell[i] * r.mnp;
    double v = 0.0;
    for (int k = 0; k < r.np; ++k) v += r.phi[(size_t)i * r.np + k] * c[k];
    rho[i] = v;
    const double d = v - r.obs[i];
    acc += d * d;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    *J = s;
  }
}

// dJ/du_T: 2 (rho_r - obs_r) phi_k(x_r) in row (cell_r, field 0); one thread
// walks the receivers in order (receivers may share a cell)
static __global__ void receiver_seed_kernel(Receivers r, const double* rho, double* lam) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  for (int i = 0; i < r.n; ++i) {
    const double g = 2.0 * (rho[i] - r.obs[i]);
    double* l = lam + (size_t)r.cell[i] * r.mnp;
    for (int k = 0; k < r.np; ++k) l[k] += g * r.phi[(size_t)i * r.np + k];
  }
}

}  // namespace dgp
