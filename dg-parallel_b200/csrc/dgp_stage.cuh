// Fused stage kernel: one CTA per tile of TS cells computes every face flux
// that touches the tile, the volume term, the lift of the face slots, the
// diagonal inverse mass and the SSP-RK3 stage combination, with the last
// stage's residual and CFL reductions fused in.
//
// Work mapping.  The state is contracted with small constant tables four times
// (face traces, volume values, gradients, lift).  All four run as one thread
// per (cell, field) row with the row in registers and the table as the
// multiply-add's constant-bank operand: the tables travel as kernel
// parameters (StageTab), so an entry costs no shared-memory access and no
// register.  Measured on B200, FP64 multiply-adds with a table operand run at
// 12.4e12/s from the constant bank and 7.5e12/s from shared memory (18.4e12/s
// without a table); FP32 24e12/s against 8.2e12/s.  Between the row phases the
// values pass through shared memory, field-major at an odd pitch, so that both
// the rows (consecutive lanes: consecutive rows) and the points (consecutive
// lanes: consecutive cells) access it without bank conflicts:
//   A  rows: traces of every face point into the slots sS, values at the
//      volume points into sV; the halo rows (the neighbours across the tile's
//      outer faces) are contracted straight from global memory, only at the
//      points of the face they share
//   B  points: the law's numerical, periodic or boundary flux of every face
//      point, written over the own traces; the volume flux mapped to reference
//      directions, written over the volume values
//   D  rows: gradients and lift, then FP64 dt/|J| and the stage combination
// P3 Euler Roe, 131072 triangles, stages 1 / 2 / 3: FP64 89 / 91 / 110 us
// (with the tables and rows read from shared memory: 117 / 117 / 142), mixed
// 59 / 60 / 76 us (94 / 94 / 117).  What bounds it: no unit above 45 % busy
// (FP64 pipe 38-40 %, shared memory 40 %); the flux of a face point is a chain of
// ~50 dependent FP64 operations at 16 resident warps a SM.
//
// Laws with a linear flux (advection, Maxwell) need no volume quadrature on
// affine cells: the flux of a mode is the mode of the flux, and the volume
// integral of grad(phi_k) phi_l is a table.  Their volume "points" are the
// modes l of degree < p, the table rows int d_r phi_k phi_l, and entries with
// deg(phi_k) <= deg(phi_l) vanish (every rule here integrates degree 2p - 1
// exactly, so this is the quadrature's own result up to rounding).  P2 tets:
// 81 multiply-adds a row instead of 560.
//
// The own rows, the face records and (tensor cores) the B operand arrive by
// bulk copies on an mbarrier.  A face between two tiles is evaluated by both,
// from identical inputs with identical arithmetic, so each side receives the
// same flux it would get from a separate face pass.  The stage writes a
// different buffer from the one it reads (u_n -> u1 -> u2 -> u_n in place,
// own rows only), so no tile reads a row another tile is writing.
//
// Replaces DGBoundaryCell::computeBoundaryContributions (DGCell.cc:639-732),
// DGCell::computeVolumeContribution (DGCell.cc:184-249) and the
// RungeKuttaTVD3::advanceInTime update loops (TimeIntegrator.cc:838-990).
//
// P0 fallback (DGCell::setToZero, DGCell.cc:785-811; DGAnalysis.cc:392-417,
// and the correction inside DGCell::computeVolumeContribution,
// DGCell.cc:197-221): a cell is marked when its value at any of its volume
// quadrature points or its trace at any of its face points is not physical.
// Each tile checks its own cells at their face and volume points in phase B
// and its halo cells at all of theirs, so it knows every mark that reaches its
// faces without a grid-wide pass; a tile that sees one repeats phases A and B
// with the marked rows' modes k >= 1 at zero.  Marks of stage 1 persist into
// u_n for stages 2 and 3 (bad[e]).
#pragma once

#include <type_traits>

#include "dgp_elem.cuh"
#include "dgp_host.h"
#include "dgp_round.h"
#include "dgp_umma.cuh"

namespace dgp {

constexpr int modes_upto(int dim, int degree) {
  return degree < 0 ? 0
         : dim == 2 ? (degree + 1) * (degree + 2) / 2
                    : (degree + 1) * (degree + 2) * (degree + 3) / 6;
}

constexpr int mode_degree(int dim, int k) {
  int d = 0;
  while (modes_upto(dim, d) <= k) ++d;
  return d;
}

// laws whose flux is linear in the state with constant coefficients
constexpr bool linear_flux(int law) {
  return law == DGP_LAW_SCALAR || law == DGP_LAW_MAXWELL2D || law == DGP_LAW_MAXWELL3D;
}

// laws whose state can be non-physical (is_physical)
constexpr bool has_physical_range(int law) { return law == DGP_LAW_EULER2D || law == DGP_LAW_EULER3D; }

// laws whose largest eigenvalue depends on the state (max_eigen)
constexpr bool state_dependent_speed(int law) { return law == DGP_LAW_EULER2D || law == DGP_LAW_EULER3D; }

// Pitch between the fields of a shared-memory row (element (cell e, field j)
// at j * pitch + e): consecutive lanes hold consecutive rows (e = row / M,
// j = row % M), so the pitch is the one of [TE, TE + 4] that brings the fewest
// of a wavefront's lanes (16 for 8-byte, 32 for 4-byte elements) to one bank.
constexpr int field_pitch(int TE, int M, int esize) {
  if (M == 1) return TE;
  const int lanes = 128 / esize;
  int best = TE, best_hits = 1 << 30;
  for (int p = TE; p <= TE + 4; ++p) {
    int worst = 0;
    for (int r0 = 0; r0 < 4 * lanes && r0 + lanes <= TE * M; r0 += lanes) {
      int hits[32] = {};
      for (int r = r0; r < r0 + lanes; ++r) {
        const int b = ((r % M) * p + r / M) % lanes;
        if (++hits[b] > worst) worst = hits[b];
      }
    }
    if (worst < best_hits) {
      best_hits = worst;
      best = p;
    }
  }
  return best;
}

template <class K>
struct StageShape {
  using T = typename K::T;
  static constexpr bool LINEAR = linear_flux(K::LAW);
  // volume points: quadrature points, or the modes of degree < p
  static constexpr int VQ = LINEAR ? modes_upto(K::DIM, K::ORDER - 1) : K::NQ;
  static constexpr int KV = VQ * K::DIM;
  static constexpr int TEP = field_pitch(K::TS, K::M, sizeof(T));
  // pitch of a face or volume point: the points of a face (consecutive lanes
  // of phase B) fall on banks apart
  static constexpr int LANES = 128 / (int)sizeof(T);
  static constexpr int SPREAD = LANES / K::NQF > 0 ? LANES / K::NQF : 1;
  static constexpr int LDR0 = K::M * TEP;
  static constexpr int LDR = LDR0 + ((SPREAD - LDR0) % LANES + LANES) % LANES;
  // halo traces [side][point][field], sides apart by 16 bytes times an odd number
  static constexpr int LDH0 = K::NQF * K::M;
  static constexpr int HV = 16 / (int)sizeof(T);
  static constexpr int LDH = ((LDH0 + HV - 1) / HV | 1) * HV;
  // first mode with a gradient against volume point q
  __host__ __device__ static constexpr int k_first(int q) {
    return LINEAR ? modes_upto(K::DIM, mode_degree(K::DIM, q)) : 1;
  }
};

// The reference tables as the kernel's parameters, on 16 bytes whatever comes
// before them: the wide constant loads of neighbouring entries need it.
template <class K>
struct alignas(16) StageTab {
  using T = typename K::T;
  using S = StageShape<K>;
  T phif[K::NS * K::NP];                       // face traces [local face, point][mode]
  T dv[(S::KV > 0 ? S::KV : 1) * K::NP];       // gradients [direction, volume point][mode]
  T phi[(S::LINEAR ? 1 : S::VQ) * K::NP];      // volume values [point][mode]
  T qw[S::LINEAR ? 1 : S::VQ];
  T fqw[K::NQF];
  T phimax[K::NP];                             // largest |phi_k| over the volume and face points
  double phiv[(K::NV > 1 ? K::NV - 1 : 1) * K::NP];  // values at the vertices (CFL)
};

template <class K>
size_t stage_tab_bytes() {
  static_assert(sizeof(StageTab<K>) + sizeof(StageArgs<typename K::T>) <= 32764, "kernel parameters");
  return sizeof(StageTab<K>);
}

template <class K>
void fill_stage_tab(const RefTables& t, const double* phimax, void* out) {
  using T = typename K::T;
  using S = StageShape<K>;
  constexpr int NP = K::NP;
  auto& tb = *static_cast<StageTab<K>*>(out);
  tb = StageTab<K>{};
  for (int i = 0; i < K::NS * NP; ++i) tb.phif[i] = (T)t.phif[i];
  for (int r = 0; r < K::DIM; ++r)
    for (int q = 0; q < S::VQ; ++q)
      for (int k = 0; k < NP; ++k) {
        double v;
        if constexpr (S::LINEAR) {
          long double s = 0.0L;
          for (int p = 0; p < K::NQ; ++p)
            s += (long double)t.qw[p] * t.dphi[((size_t)p * K::DIM + r) * NP + k] * t.phi[(size_t)p * NP + q];
          v = (double)s;
        } else {
          v = t.dphi[((size_t)q * K::DIM + r) * NP + k];
        }
        tb.dv[(r * S::VQ + q) * NP + k] = (T)v;
      }
  if constexpr (!S::LINEAR) {
    for (int i = 0; i < S::VQ * NP; ++i) tb.phi[i] = (T)t.phi[i];
    for (int q = 0; q < S::VQ; ++q) tb.qw[q] = (T)t.qw[q];
  }
  for (int q = 0; q < K::NQF; ++q) tb.fqw[q] = (T)t.fqw[q];
  for (int k = 0; k < NP; ++k) tb.phimax[k] = (T)phimax[k];
  for (int i = 0; i < (K::NV - 1) * NP; ++i) tb.phiv[i] = t.phiv[i];
}

template <class K, bool TC = false>
struct FusedSmem {
  using T = typename K::T;
  using S = StageShape<K>;
  static constexpr size_t r16(size_t n) { return (n + 15) / 16 * 16; }
  static constexpr bool MIXED = sizeof(T) == 4;
  // The mixed form's volume contraction on the tensor cores (tcgen05, TF32
  // with split operands) where TC asks for it: one M = 128 MMA tile covers
  // the tile's rows, N = 16 the modes, K = KPAD the (direction, point) pairs
  // padded to whole k-steps.  UMMA_OK: the shape allows it.
  static constexpr bool UMMA_OK = MIXED && K::BLOCK == 128 && K::TS * K::M <= 128 && K::NP <= 16;
  static constexpr bool UMMA = UMMA_OK && TC;
  static constexpr int KPAD = S::KV > 0 ? (S::KV + 7) / 8 * 8 : 8;
  static constexpr int UN = 16;
  static constexpr size_t a_bytes = (size_t)128 * KPAD * 4;  // one split part of A
  static constexpr size_t b_bytes = (size_t)UN * KPAD * 4;   // one split part of B
  // device blob of the tensor-core form: B = the gradient table as TF32 high
  // and low parts in the MMA layout
  static constexpr size_t fblob_elems = UMMA_OK ? 2 * b_bytes / 4 : 1;
  // one-field laws keep the volume values in registers
  static constexpr bool VREG = K::M == 1 && !UMMA;
  static constexpr size_t rows_bytes = (size_t)K::TS * K::MNP * 8;
  static constexpr bool bulk_rows = rows_bytes % 16 == 0;  // every tile starts on a 16-byte boundary
  static constexpr size_t max2(size_t a, size_t b) { return a > b ? a : b; }
  // slots (later the CFL states, FP64) | volume values (r = 0 of G) |
  // union {staged rows FP64; G of the other directions, or A} | J^{-1} |
  // |J| FP64 | B | face records | halo traces | halo P0 bounds | P0 marks
  static constexpr size_t oS = 0;
  static constexpr size_t oV = oS + r16(max2((size_t)K::NS * S::LDR * sizeof(T),
                                             state_dependent_speed(K::LAW) ? (size_t)K::NV * S::LDR * 8 : 0));
  static constexpr size_t oX = oV + (VREG ? 0 : r16((size_t)S::VQ * S::LDR * sizeof(T)));
  static constexpr size_t oJ =
      oX + r16(max2(r16(rows_bytes), UMMA ? 2 * a_bytes
                                          : VREG ? 0 : (size_t)(K::DIM - 1) * S::VQ * S::LDR * sizeof(T)));
  static constexpr size_t oDet = oJ + r16((size_t)K::TS * K::DIM * K::DIM * sizeof(T));
  static constexpr size_t oB = oDet + r16((size_t)K::TS * 8);
  static constexpr size_t oF = oB + (UMMA ? r16(2 * b_bytes) : 0);
  static constexpr bool P0 = has_physical_range(K::LAW);
  __host__ __device__ static constexpr size_t oH(int nf) { return oF + (size_t)nf * sizeof(FaceRec<K::DIM>); }
  __host__ __device__ static constexpr size_t oP(int nf, int nh) {
    return oH(nf) + r16((size_t)nh * S::LDH * sizeof(T));
  }
  __host__ __device__ static constexpr size_t oM(int nf, int nh) {
    return oP(nf, nh) + (P0 ? r16((size_t)nh * K::M * 2 * sizeof(T)) : 0);
  }
  static constexpr size_t bytes(int nf, int nh) { return oM(nf, nh) + (P0 ? r16((size_t)K::TS + nh) : 0); }
  // at most 128 registers a thread (FP32: 80), so that four (six) CTAs of 128
  // threads fit; P3 Euler Roe on 131072 cells, a stage: FP64 89 us at 128 and
  // 89 at 168 (three CTAs), FP32 58 at 80, 61 at 100, 67 at 128.  FP32 takes 128
  // where 80 cost more in spills than the CTAs gain: rows of 15 modes and more
  // (P4 triangles, P3 tets), and the tensor-core form whose A operand leaves no
  // room for more than four CTAs (P3 and P4).
  static constexpr int SMEM_CTAS = (int)(227 * 1024 / (bytes(2 * K::TS, K::TS) + 1024));
  static constexpr int REGS = MIXED && K::NP < 15 && !(UMMA && SMEM_CTAS <= 4) ? 80 : 128;
  static constexpr int MIN_BLOCKS = 65536 / (K::BLOCK * REGS) > 0 ? 65536 / (K::BLOCK * REGS) : 1;
};

// host: the tensor-core form's B[n][kk] = dv of row kk at mode n, as FP32
// split into TF32 high and low parts, zero beyond the modes and the rows
template <class K>
void fill_fused_blob(const void* tab, double* blob) {
  using FS = FusedSmem<K>;
  if constexpr (FS::UMMA_OK) {
    const auto& tb = *static_cast<const StageTab<K>*>(tab);
    for (int n = 0; n < FS::UN; ++n)
      for (int kk = 0; kk < FS::KPAD; ++kk) {
        float v = 0.0f;
        if (kk < FS::S::KV && n < K::NP) v = (float)tb.dv[kk * K::NP + n];
        const float hi = host_tf32(v), lo = host_tf32(v - hi);
        const uint32_t o = umma_off(n, kk, FS::KPAD) / 4;
        blob[o] = hi;
        blob[FS::b_bytes / 4 + o] = lo;
      }
  }
}

// Rounding probe (error decomposition of the mixed form): with RND, the terms
// whose bit is set in the mask are rounded to FP32 inside the FP64 kernel.
// Bits: geometry (J^{-1}, |J| w, face normals, |J_f| w), face-point traces,
// volume-point values, volume flux products G, face slots, the contraction's
// result, the reference tables.
enum : int {
  kRndGeometry = 1, kRndTraces = 2, kRndVolumeValues = 4, kRndVolumeFlux = 8, kRndSlots = 16,
  kRndContraction = 32, kRndTables = 64
};

template <bool RND, typename T>
__device__ __forceinline__ T probe(T x, int mask, int bit) {
  if constexpr (RND) {
    if (mask & bit) return (T)(float)x;
  }
  return x;
}

// the one configuration the probe is built for: the FP64 P3 Euler vortex
// workload with Roe flux and 128-thread tiles
template <class K>
constexpr bool probe_built() {
  return sizeof(typename K::T) == 8 && K::LAW == DGP_LAW_EULER2D && K::FLUX == DGP_FLUX_ROE && K::DIM == 2 &&
         K::ORDER == 3 && K::BLOCK == 128;
}

constexpr int kFinalizeThreads = 1024;

// loops over table rows are unrolled completely while the code stays within
// the instruction cache (the tables' constant offsets then cost no address
// arithmetic: 27 us against 39 us for the P3 contractions of 131072 cells
// unrolled by four), and by four beyond (P3 tets: 4000 multiply-adds)
constexpr int table_unroll(int rows, int np) { return rows * np <= 700 ? rows : 4; }

// loads that stay where they are written (before a barrier, so that they
// are in flight while the CTA works up to it)
__device__ __forceinline__ double ld_pinned(const double* p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double2 ld_pinned2(const double* p) {
  double2 v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

__device__ __forceinline__ int2 ld_pinned_i2(const int2* p) {
  int2 v;
  asm volatile("ld.global.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// a row of N FP64 values at p, aligned to ALIGN bytes
template <int N, int ALIGN>
__device__ __forceinline__ void ld_row_pinned(const double* p, double (&out)[N]) {
  if constexpr (ALIGN == 16) {
#pragma unroll
    for (int i = 0; i + 1 < N; i += 2) {
      const double2 v = ld_pinned2(p + i);
      out[i] = v.x;
      out[i + 1] = v.y;
    }
    if constexpr (N % 2 == 1) out[N - 1] = ld_pinned(p + N - 1);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = ld_pinned(p + i);
  }
}

template <int N, int ALIGN>
__device__ __forceinline__ void st_row(double* p, const double (&v)[N]) {
  if constexpr (ALIGN == 16) {
#pragma unroll
    for (int i = 0; i + 1 < N; i += 2) *reinterpret_cast<double2*>(p + i) = make_double2(v[i], v[i + 1]);
    if constexpr (N % 2 == 1) p[N - 1] = v[N - 1];
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = v[i];
  }
}

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// a tile that computes nothing in the last stage (its instance has finished,
// or its copies gave up) leaves neutral partials
template <class K>
__device__ __forceinline__ void fused_tile_idle(const StageArgs<typename K::T>& a, int tile) {
  if (a.stage != 3 || threadIdx.x != 0) return;
  const int ntiles = (a.mesh.E + K::TS - 1) / K::TS;
  a.partials[tile] = 0.0;
  a.partials[ntiles + tile] = 1e300;
}

// an own cell's state in shared memory (its fields a pitch apart): counts a
// non-physical one and, with the P0 fallback on, marks its cell (true then)
template <class K>
__device__ __noinline__ bool check_trace(const StageArgs<typename K::T>& a, const typename K::T* p, int e0, int l,
                                         unsigned char* s_mark) {
  using T = typename K::T;
  T U[K::M];
  for (int j = 0; j < K::M; ++j) U[j] = p[j * StageShape<K>::TEP];
  if (is_physical<K::LAW, T>(a.law, U)) return false;
  flag_nonphysical(a.status, e0 + l);
  if (!a.p0) return false;
  s_mark[l] = 1;
  return true;
}

// One face point: traces of both sides, the law's numerical or boundary flux,
// and the slots of the own sides.  CHECK: count non-physical own traces and,
// with the P0 fallback on, mark their cells (returns true when it marked one).
template <class K, bool ENS, bool RND>
__device__ __forceinline__ bool fused_face_point(const StageArgs<typename K::T>& a, const TimeCtl* c, int inst, int e0,
                                                 const FaceRec<K::DIM>& fr, int q, const typename K::T* s_fqw,
                                                 const int* s_qmap, typename K::T* sS, const typename K::T* sHt,
                                                 unsigned char* s_mark, bool check) {
  using T = typename K::T;
  using S = StageShape<K>;
  constexpr int M = K::M, NQF = K::NQF, DIM = K::DIM, TS = K::TS;
  const int refL = fr.side & 0xffff, refR = (unsigned)fr.side >> 16;
  const int kind = (fr.code >> 3) & 3;
  T n[DIM];
#pragma unroll
  for (int i = 0; i < DIM; ++i) n[i] = probe<RND, T>((T)fr.n[i], a.round_mask, kRndGeometry);
  const T jw = probe<RND, T>((T)fr.fj * s_fqw[q], a.round_mask, kRndGeometry);
  // an own side's trace lies in the slots, a halo side's in its own list
  const bool ownL = !(refL & kHaloRef);
  const int lfL = refL / TS, lL = refL - lfL * TS;
  T* pL = sS + (lfL * NQF + q) * S::LDR + lL;
  bool marked = false;
  T UL[M], UR[M], flux[M];
  if (ownL) {
#pragma unroll
    for (int j = 0; j < M; ++j) UL[j] = pL[j * S::TEP];
  } else {
    const T* h = sHt + (refL & (kHaloRef - 1)) * S::LDH + q * M;
    load_vec<T, M>(h, UL);
  }
  bool ownR = false;
  T* pR = nullptr;
  int lR = 0;
  if (kind != kFaceBoundary) {
    ownR = !(refR & kHaloRef);
    // a periodic partner's trace is stored in the left cell's point order
    int qR = q;
    if (kind == kFaceInterior) {
      const int perm = fr.code & 7;
      if constexpr (DIM == 2)
        qR = perm ? NQF - 1 - q : q;
      else
        qR = s_qmap[perm * NQF + q];
    }
    if (ownR) {
      const int lfR = refR / TS;
      lR = refR - lfR * TS;
      pR = sS + (lfR * NQF + qR) * S::LDR + lR;
#pragma unroll
      for (int j = 0; j < M; ++j) UR[j] = pR[j * S::TEP];
    } else {
      const T* h = sHt + (refR & (kHaloRef - 1)) * S::LDH + qR * M;
      load_vec<T, M>(h, UR);
    }
    // periodic edges (DGCell.cc:687-705): the numerical flux, to the left cell only
    numerical_flux<K::LAW, K::FLUX, DIM, T>(a.law, n, UL, UR, flux);
  } else {
    const int b = fr.code >> 5;
    const double* x = a.mesh.bpts + ((size_t)b * NQF + q) * 3;
    const double time = __fma_rn(a.stage_time_factor, c->dt, c->t);
    if constexpr (ENS)
      boundary_flux<K::LAW, K::FLUX, DIM, T>(a.laws[inst], a.mesh.bbid[b], n, x, time, UL, flux);
    else
      boundary_flux<K::LAW, K::FLUX, DIM, T>(a.law, a.mesh.bbid[b], n, x, time, UL, flux);
  }
  if constexpr (has_physical_range(K::LAW)) {
    // one test of both own traces beside the flux; the marks and counts of a
    // non-physical one are off the main path
    const bool bad = (ownL && !surely_physical<K::LAW, T>(a.law, UL)) || (ownR && !surely_physical<K::LAW, T>(a.law, UR));
    if (bad && check) {
      if (ownL) marked |= check_trace<K>(a, pL, e0, lL, s_mark);
      if (ownR) marked |= check_trace<K>(a, pR, e0, lR, s_mark);
    }
  }
  if (ownL) {
#pragma unroll
    for (int j = 0; j < M; ++j) pL[j * S::TEP] = probe<RND, T>(-flux[j] * jw, a.round_mask, kRndSlots);
  }
  if (ownR) {
#pragma unroll
    for (int j = 0; j < M; ++j) pR[j * S::TEP] = probe<RND, T>(flux[j] * jw, a.round_mask, kRndSlots);
  }
  return marked;
}

// dot product of a row in registers with one table row (constant bank)
template <int NP, bool RND, typename T>
__device__ __forceinline__ T table_dot(const T (&c)[NP], const T* t, int mask) {
  T acc = 0;
#pragma unroll
  for (int k = 0; k < NP; ++k) acc += probe<RND, T>(t[k], mask, kRndTables) * c[k];
  return acc;
}

// traces of one halo row at the points of local face LF
template <class K, int LF, bool RND>
__device__ __forceinline__ void halo_traces(const StageTab<K>& tb, const typename K::T (&c)[K::NP],
                                            typename K::T* out, int mask, int z) {
  using T = typename K::T;
  constexpr int UN = table_unroll(K::NQF, K::NP);
#pragma unroll UN
  for (int q = 0; q < K::NQF; ++q)
    out[q * K::M] = probe<RND, T>(
        table_dot<K::NP, RND, T>(c, tb.phif + z + (LF * K::NQF + q) * K::NP, mask), mask, kRndTraces);
}

// The P0 check of one halo cell: true when its value at a volume quadrature
// point or its trace at a face point is not physical.  bnd: mean and bound
// per field; a cell whose modes k >= 1 cannot move a field past the limit
// anywhere (physical_bound) is cleared without evaluating its points.
template <class K>
__device__ bool halo_cell_bad(const StageArgs<typename K::T>& a, const StageTab<K>& tb, const int2* side,
                              const typename K::T* bnd) {
  using T = typename K::T;
  constexpr int M = K::M, NP = K::NP;
  T mean[M], B[M];
#pragma unroll
  for (int j = 0; j < M; ++j) {
    mean[j] = bnd[2 * j];
    B[j] = bnd[2 * j + 1];
  }
  if (physical_bound<K::LAW, T>(a.law, mean, B)) return false;
  const int cell = side->x;
#pragma unroll 1
  for (int p = 0; p < StageShape<K>::VQ + K::NS; ++p) {
    const T* t = p < StageShape<K>::VQ ? tb.phi + p * NP : tb.phif + (p - StageShape<K>::VQ) * NP;
    T U[M];
    for (int j = 0; j < M; ++j) {
      T acc = 0;
      for (int k = 0; k < NP; ++k) acc += t[k] * (T)a.C[((size_t)cell * M + j) * NP + k];
      U[j] = acc;
    }
    if (!is_physical<K::LAW, T>(a.law, U)) return true;
  }
  return false;
}

// phase A of an own row: face traces, then (VOL) volume values
template <class K, bool RND, bool VOL>
__device__ __forceinline__ void own_points(const StageTab<K>& tb, const typename K::T (&c)[K::NP], typename K::T* sS,
                                           typename K::T* sV, int prow, int mask) {
  using T = typename K::T;
  using S = StageShape<K>;
  constexpr int NP = K::NP, NS = K::NS, VQ = S::VQ;
  constexpr int UF = table_unroll(NS, NP), UV = table_unroll(VQ > 0 ? VQ : 1, NP);
#pragma unroll UF
  for (int s = 0; s < NS; ++s)
    sS[s * S::LDR + prow] = probe<RND, T>(table_dot<NP, RND, T>(c, tb.phif + s * NP, mask), mask, kRndTraces);
  if constexpr (VOL) {
#pragma unroll UV
    for (int q = 0; q < VQ; ++q) {
      if constexpr (S::LINEAR)
        sV[q * S::LDR + prow] = c[q];
      else
        sV[q * S::LDR + prow] = probe<RND, T>(table_dot<NP, RND, T>(c, tb.phi + q * NP, mask), mask, kRndVolumeValues);
    }
  }
}

template <class K, bool ENS, bool TC = false, bool RND = false>
__global__ void __launch_bounds__(K::BLOCK, FusedSmem<K, TC>::MIN_BLOCKS)
    stage_kernel(const __grid_constant__ StageArgs<typename K::T> a, const __grid_constant__ StageTab<K> tb) {
  using T = typename K::T;
  using S = StageShape<K>;
  using FS = FusedSmem<K, TC>;
  constexpr int M = K::M, NP = K::NP, MNP = K::MNP, NS = K::NS, NQF = K::NQF, DIM = K::DIM;
  constexpr int TS = K::TS, NT = K::BLOCK, VQ = S::VQ, KV = S::KV, LDR = S::LDR, TEP = S::TEP, NV = K::NV;
  constexpr bool PHYS = has_physical_range(K::LAW);
  constexpr int RALIGN = pow2_div(NP * 8) < 16 ? pow2_div(NP * 8) : 16;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T* sS = reinterpret_cast<T*>(smem_raw + FS::oS);
  T* sV = reinterpret_cast<T*>(smem_raw + FS::oV);
  T* sX = reinterpret_cast<T*>(smem_raw + FS::oX);
  double* sRow = reinterpret_cast<double*>(smem_raw + FS::oX);
  T* sJi = reinterpret_cast<T*>(smem_raw + FS::oJ);
  double* sDet = reinterpret_cast<double*>(smem_raw + FS::oDet);
  const FaceRec<DIM>* sF = reinterpret_cast<const FaceRec<DIM>*>(smem_raw + FS::oF);
  __shared__ __align__(8) uint64_t bar;
  __shared__ double red[2 * (NT / 32)];
  __shared__ T s_fqw[NQF];
  __shared__ int s_qmap[DIM == 3 ? K::NPERM * NQF : 1];
  __shared__ __align__(8) uint64_t mma_bar;
  __shared__ uint32_t s_tmem;

  const int tid = threadIdx.x;
  const int tile = blockIdx.x;
  const int e0 = tile * TS;
  const int nfm = a.tm.nf_max, nhm = a.tm.nh_max;
  T* sHt = reinterpret_cast<T*>(smem_raw + FS::oH(nfm));
  T* sBnd = reinterpret_cast<T*>(smem_raw + FS::oP(nfm, nhm));
  unsigned char* s_mark = smem_raw + FS::oM(nfm, nhm);

  // What the tile reads from global memory is requested here, before anything
  // is waited for; the solver's constant data even before the previous kernel
  // of the stream has ended (pdl_wait).  Bulk copies on one mbarrier: the face
  // records, the own rows (where their bytes are whole 16-byte units: not at a
  // last tile with an odd number of values, nor from a base on an odd 8 bytes,
  // a stored state of an odd length), B of the tensor cores.  A bound on the
  // first wait (a.mbar_polls) counts polls from the rows' issue.
  if (!late_start<K>(a)) pdl_trigger();
  const int nrow = min(TS, a.mesh.E - e0);
  const bool bulk = FS::bulk_rows && (nrow * MNP) % 2 == 0 && (reinterpret_cast<uintptr_t>(a.C) & 15) == 0;
  const uint32_t rb = bulk ? (uint32_t)(nrow * MNP * 8) : 0u;
  bool failed = false;
  if (tid == 0) {
    mbar_init(&bar, 1);
    if constexpr (FS::UMMA) mbar_init(&mma_bar, 1);
    const uint32_t fb = (uint32_t)(nfm * sizeof(FaceRec<DIM>));
    mbar_arrive_expect_tx(&bar, fb + rb + (FS::UMMA ? (uint32_t)(2 * FS::b_bytes) : 0));
    bulk_g2s(smem_raw + FS::oF, static_cast<const FaceRec<DIM>*>(a.tm.tf_rec) + (size_t)tile * nfm, fb, &bar);
    if constexpr (FS::UMMA) bulk_g2s(smem_raw + FS::oB, a.tab.blob, (uint32_t)(2 * FS::b_bytes), &bar);
  }
  // the thread's first halo side
  int2 hs = make_int2(-1, 0);
  if (tid < nhm * M) hs = ld_pinned_i2(a.tm.th_side + (size_t)tile * nhm + tid / M);
  const int2 cnt = ld_pinned_i2(a.tm.count + tile);
  for (int i = tid; i < nrow * DIM * DIM; i += NT) {
    if constexpr (sizeof(T) == 8)
      cp_async8(sJi + i, a.mesh.jinv + (size_t)e0 * DIM * DIM + i);
    else
      cp_async4(sJi + i, a.mesh.jinv + (size_t)e0 * DIM * DIM + i);
  }
  for (int i = tid; i < nrow; i += NT) cp_async8(sDet + i, a.mesh.detjd + e0 + i);
  if constexpr (DIM == 3)
    for (int i = tid; i < K::NPERM * NQF; i += NT) cp_async4(s_qmap + i, a.tab.qmap + i);
  double csz = 0.0;
  if (!state_dependent_speed(K::LAW) && a.stage == 3 && a.fuse_cfl && tid < nrow)
    csz = ld_pinned(a.mesh.csize + e0 + tid);
  if (tid < NQF) s_fqw[tid] = tb.fqw[tid];
  if constexpr (PHYS)
    for (int i = tid; i < TS + nhm; i += NT) s_mark[i] = 0;
  int inst = 0, eend = a.mesh.E;
  if constexpr (ENS) {  // the tile belongs to one instance
    inst = a.cell_inst[e0];
    eend = a.inst_end[inst];
  }
  if constexpr (FS::UMMA) {
    // 32 columns of tensor memory for D, freed on every way out of the kernel
    if (tid < 32) tmem_alloc(&s_tmem, 32);
    tc_fence_before();
  }
  pdl_wait();
  if (tid == 0) {
    if (bulk) bulk_g2s(sRow, a.C + (size_t)e0 * MNP, rb, &bar);
    if (a.mbar_polls > 0 && !mbar_test_polls(&bar, 0, a.mbar_polls)) failed = true;
  }
  TimeCtl* c = a.ctl + inst;
  const int all_done = a.gctl->done, inst_done = ENS ? c->done : 0;
  const double dt = c->dt;
  __syncthreads();  // the barrier's initialisation
  if (all_done || inst_done) {
    // nothing to do: leave once the copies have landed
    if (tid == 0) mbar_wait(&bar, 0, kMbarPolls);
    cp_async_wait_all();
    if (!all_done) fused_tile_idle<K>(a, tile);
    if constexpr (FS::UMMA) {
      tc_fence_after();
      __syncthreads();
      if (tid < 32) tmem_dealloc(s_tmem, 32);
    }
    return;
  }
  const int ne = min(TS, eend - e0), nf = cnt.x, nh = cnt.y;

  const int row = tid;
  const bool live = row < ne * M;
  const int cell = row / M, field = row - (row / M) * M;
  const int prow = field * TEP + cell;
  const size_t gbase = ((size_t)e0 * M + row) * NP;
  // volume point owner (laws with several fields): cell ve, points vg, vg + NG, ...
  constexpr int NG = NT / TS;
  const int ve = tid % TS, vg = tid / TS;
  T accv[FS::VREG ? NP : 1];  // volume term of a one-field law's row

  // a second round only when the P0 fallback dropped a cell of the tile
#pragma unroll 1
  for (int round = 0;; ++round) {
    // ---- A: own rows -> face traces and volume values ----------------------
    T cr[NP];
    if (round == 0) {
      if (!mbar_wait(&bar, 0, kMbarPolls)) failed = true;
      if (live) {
        if (bulk) {
          double v[NP];
          if constexpr (RALIGN == 16) {
            load_vec<double, NP>(sRow + (size_t)row * NP, v);
          } else {
#pragma unroll
            for (int k = 0; k < NP; ++k) v[k] = sRow[(size_t)row * NP + k];
          }
#pragma unroll
          for (int k = 0; k < NP; ++k) cr[k] = (T)v[k];
        } else {
#pragma unroll
          for (int k = 0; k < NP; ++k) cr[k] = (T)a.C[gbase + k];
        }
      }
    } else if (live) {
      const bool drop = PHYS && s_mark[cell];
#pragma unroll
      for (int k = 0; k < NP; ++k) cr[k] = (k > 0 && drop) ? (T)0 : (T)a.C[gbase + k];
    }
    if (live) {
      own_points<K, RND, !FS::VREG>(tb, cr, sS, sV, prow, a.round_mask);
    }
    // halo rows, one (side, field) a thread
#pragma unroll 1
    for (int base = 0; base < nh * M; base += NT) {
      const int it = base + tid;
      if (it >= nh * M) break;
      // a zero that the compiler cannot see through, uniform and of this
      // round of the loop: without it the table's constants are hoisted out
      // of the loop into registers that are not there
      const int z = base & a.tab.zero;
      const int h = it / M, j = it - (it / M) * M;
      if (base > 0 || round > 0) hs = a.tm.th_side[(size_t)tile * nhm + h];
      double hrow[NP];
      ld_row_pinned<NP, RALIGN>(a.C + ((size_t)hs.x * M + j) * NP, hrow);
      T hc[NP];
#pragma unroll
      for (int k = 0; k < NP; ++k) hc[k] = (T)hrow[k];
      if constexpr (PHYS) {
        if (round > 0) {
          if (s_mark[TS + h])
#pragma unroll
            for (int k = 1; k < NP; ++k) hc[k] = (T)0;
        } else if (a.p0) {
          T b = 0;
#pragma unroll
          for (int k = 1; k < NP; ++k) b += fabs(hc[k]) * tb.phimax[k];
          sBnd[2 * it] = hc[0] * tb.phi[0];
          sBnd[2 * it + 1] = b;
        }
      }
      T* out = sHt + h * S::LDH + j;
      switch (hs.y & 7) {
        case 0: halo_traces<K, 0, RND>(tb, hc, out, a.round_mask, z); break;
        case 1: halo_traces<K, 1, RND>(tb, hc, out, a.round_mask, z); break;
        case 2: halo_traces<K, 2, RND>(tb, hc, out, a.round_mask, z); break;
        case 3:
          if constexpr (K::NLF == 4) halo_traces<K, 3, RND>(tb, hc, out, a.round_mask, z);
          break;
        default: {
          // periodic partner: its basis at the mirrored points
          const T* ph = a.mesh.bpphi + (size_t)(hs.y >> 3) * NQF * NP;
          for (int q = 0; q < NQF; ++q) {
            T u = 0;
#pragma unroll
            for (int k = 0; k < NP; ++k) u += __ldg(ph + q * NP + k) * hc[k];
            out[q * M] = u;
          }
        }
      }
    }
    if (round == 0) {
      cp_async_wait_all();
      if (__syncthreads_or(failed)) {
        // record the failure, wait once more (bounded) for the copies this CTA
        // issued before its shared memory is released; the tile's output is not
        // written, the last stage still leaves neutral partials
        if (tid == 0) {
          atomicAdd(&a.status->timeouts, 1);
          mbar_wait(&bar, 0, kMbarPolls);
        }
        fused_tile_idle<K>(a, tile);
        if constexpr (FS::UMMA) {
          tc_fence_after();
          __syncthreads();
          if (tid < 32) tmem_dealloc(s_tmem, 32);
        }
        return;
      }
    } else {
      __syncthreads();
    }

    // ---- B: face points and volume points ------------------------------------
    bool mk = false;
    for (int t = tid; t < nf * NQF; t += NT) {
      const int f = t / NQF, q = t - f * NQF;
      mk |= fused_face_point<K, ENS, RND>(a, c, inst, e0, sF[f], q, s_fqw, s_qmap, sS, sHt, s_mark, round == 0);
    }
    if constexpr (PHYS) {
      if (a.p0 && round == 0) {
        for (int h = tid; h < nh; h += NT)
          if (halo_cell_bad<K>(a, tb, a.tm.th_side + (size_t)tile * nhm + h, sBnd + 2 * h * M)) {
            s_mark[TS + h] = 1;
            mk = true;
          }
      }
    }
    if constexpr (FS::VREG) {
#pragma unroll
      for (int k = 0; k < NP; ++k) accv[k] = 0;
      if (live && VQ > 0) {
        T J[DIM * DIM];
#pragma unroll
        for (int i = 0; i < DIM * DIM; ++i) J[i] = sJi[row * DIM * DIM + i];
        const T det = (T)sDet[row];
        // linear laws whole: the entries that vanish are then known when the
        // kernel is compiled (P3 tets, 381 of 600: left in a loop, their test
        // cost 1124 us a step of 93750 cells in FP64 against 466, 728 / 251 mixed)
        constexpr int UV = S::LINEAR ? (VQ > 0 ? VQ : 1) : table_unroll(VQ > 0 ? VQ : 1, NP * (1 + DIM));
#pragma unroll UV
        for (int q = 0; q < VQ; ++q) {
          T U[1], F[1][DIM];
          if constexpr (S::LINEAR)
            U[0] = cr[q];
          else
            U[0] = table_dot<NP, false, T>(cr, tb.phi + q * NP, 0);
          volume_flux<K::LAW, DIM, T>(a.law, U, F);
          T jw = det;
          if constexpr (!S::LINEAR) jw = det * tb.qw[q];
#pragma unroll
          for (int r = 0; r < DIM; ++r) {
            T g = 0;
#pragma unroll
            for (int i = 0; i < DIM; ++i) g += F[0][i] * J[i * DIM + r];
            g *= jw;
#pragma unroll
            for (int k = 0; k < NP; ++k)
              if (k >= S::k_first(q)) accv[k] += g * tb.dv[(r * VQ + q) * NP + k];
          }
        }
      }
    } else if (vg < NG && ve < ne) {
      T J[DIM * DIM];
#pragma unroll
      for (int i = 0; i < DIM * DIM; ++i) J[i] = probe<RND, T>(sJi[ve * DIM * DIM + i], a.round_mask, kRndGeometry);
      const T det = (T)sDet[ve];
#pragma unroll 1
      for (int q = vg; q < VQ; q += NG) {
        T U[M];
#pragma unroll
        for (int j = 0; j < M; ++j) U[j] = sV[q * LDR + j * TEP + ve];
        if constexpr (PHYS) {
          if (!surely_physical<K::LAW, T>(a.law, U)) {
            const bool m = check_trace<K>(a, sV + q * LDR + ve, e0, ve, s_mark);
            mk |= m && round == 0;
          }
        }
        T F[M][DIM];
        volume_flux<K::LAW, DIM, T>(a.law, U, F);
        T jw = det;
        if constexpr (!S::LINEAR)
          jw = probe<RND, T>(det * probe<RND, T>(tb.qw[q], a.round_mask, kRndTables), a.round_mask, kRndGeometry);
#pragma unroll
        for (int j = 0; j < M; ++j)
#pragma unroll
          for (int r = 0; r < DIM; ++r) {
            T g = 0;
#pragma unroll
            for (int i = 0; i < DIM; ++i) g += F[j][i] * J[i * DIM + r];
            if constexpr (FS::UMMA) {
              // A[(cell, field)][r * VQ + q] as TF32 high and low parts
              uint32_t hi, lo;
              tf32_split((float)(g * jw), hi, lo);
              const uint32_t o = umma_off(ve * M + j, r * VQ + q, FS::KPAD);
              *reinterpret_cast<uint32_t*>(smem_raw + FS::oX + o) = hi;
              *reinterpret_cast<uint32_t*>(smem_raw + FS::oX + FS::a_bytes + o) = lo;
            } else {
              const T gv = probe<RND, T>(g * jw, a.round_mask, kRndVolumeFlux);
              if (r == 0)
                sV[q * LDR + j * TEP + ve] = gv;
              else
                sX[((r - 1) * VQ + q) * LDR + j * TEP + ve] = gv;
            }
          }
      }
    }
    if constexpr (PHYS) {
      if (a.p0 && round == 0) {
        if (__syncthreads_or(mk)) continue;
        break;
      }
    }
    __syncthreads();
    break;
  }
  if constexpr (PHYS) {
    // stage 1: the marks persist into u_n for stages 2 and 3
    if (a.p0 && a.stage == 1)
      for (int l = tid; l < ne; l += NT) a.bad[e0 + l] = s_mark[l];
  }
  if constexpr (FS::UMMA) {
    // the padding columns of A are zero (the padding rows of B are): then the
    // generic writes of A are ordered before the tensor cores read it
    constexpr int NPAD = FS::KPAD - KV;
    if constexpr (NPAD > 0) {
      for (int i = tid; i < 128 * NPAD; i += NT) {
        const uint32_t o = umma_off(i / NPAD, KV + i % NPAD, FS::KPAD);
        *reinterpret_cast<uint32_t*>(smem_raw + FS::oX + o) = 0u;
        *reinterpret_cast<uint32_t*>(smem_raw + FS::oX + FS::a_bytes + o) = 0u;
      }
    }
    fence_proxy_async_smem();
    __syncthreads();
    // D[row][mode] = sum over K of A B: per k-step of 8, the products
    // hi hi + hi lo + lo hi (TF32), accumulated in FP32 in tensor memory; the
    // CUDA cores lift the face slots meanwhile
    tc_fence_after();
    if (tid == 0) {
      constexpr uint32_t idesc = umma_idesc_tf32(128, FS::UN);
      constexpr uint32_t SBO = (FS::KPAD / 4) * 128;
      const unsigned char* A = smem_raw + FS::oX;
      const unsigned char* B = smem_raw + FS::oB;
      uint32_t accum = 0;
#pragma unroll
      for (int kb = 0; kb < FS::KPAD / 8; ++kb) {
        const uint32_t ko = (uint32_t)kb * 256;
        const uint64_t ahi = umma_desc(A + ko, 128, SBO), alo = umma_desc(A + FS::a_bytes + ko, 128, SBO);
        const uint64_t bhi = umma_desc(B + ko, 128, SBO), blo = umma_desc(B + FS::b_bytes + ko, 128, SBO);
        umma_tf32(s_tmem, ahi, bhi, idesc, accum);
        accum = 1;
        umma_tf32(s_tmem, ahi, blo, idesc, 1);
        umma_tf32(s_tmem, alo, bhi, idesc, 1);
      }
      umma_commit(&mma_bar);
    }
  }

  pdl_trigger();  // late at the latest
  // ---- D: gradients + lift + inverse mass + stage combination --------------
  // the FP64 row and u_n (stages 2, 3) come from global memory meanwhile
  double out[NP], u0[NP];
  bool drop0 = false;  // u_n of a cell that stage 1 dropped to its mean
  if (live && a.stage >= 1) {
    ld_row_pinned<NP, RALIGN>(a.C + gbase, out);
    if (a.stage >= 2) {
      ld_row_pinned<NP, RALIGN>(a.U0 + gbase, u0);
      if constexpr (PHYS) drop0 = a.p0 && a.bad[e0 + cell];
    }
  }
  const double dtj = live ? dt / sDet[cell] : 0.0;
  T acc[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) acc[k] = FS::VREG ? accv[FS::VREG ? k : 0] : (T)0;
  if (live) {
    constexpr int UK = table_unroll(VQ > 0 ? VQ : 1, NP * DIM), UF = table_unroll(NS, NP);
    if constexpr (!FS::UMMA && !FS::VREG) {
#pragma unroll
      for (int r = 0; r < DIM; ++r) {
#pragma unroll UK
        for (int q = 0; q < VQ; ++q) {
          const T gv = r == 0 ? sV[q * LDR + prow] : sX[((r - 1) * VQ + q) * LDR + prow];
#pragma unroll
          for (int k = 0; k < NP; ++k)
            if (k >= S::k_first(q))
              acc[k] += gv * probe<RND, T>(tb.dv[(r * VQ + q) * NP + k], a.round_mask, kRndTables);
        }
      }
    }
#pragma unroll UF
    for (int s = 0; s < NS; ++s) {
      const T sv = sS[s * LDR + prow];
#pragma unroll
      for (int k = 0; k < NP; ++k)
        acc[k] += sv * probe<RND, T>(tb.phif[s * NP + k], a.round_mask, kRndTables);
    }
  }
  if constexpr (FS::UMMA) {
    if (!mbar_wait(&mma_bar, 0, kMbarPolls)) {
      // never expected: record it, then wait once more (bounded) so that the
      // tensor memory is not read or freed under a running MMA
      if (tid == 0) atomicAdd(&a.status->timeouts, 1);
      mbar_wait(&mma_bar, 0, kMbarPolls);
    }
    tc_fence_after();
    float dv[16];
    tmem_ld16(s_tmem + ((uint32_t)(tid & ~31) << 16), dv);
#pragma unroll
    for (int k = 0; k < NP; ++k) acc[k] += (k < 16 ? dv[k < 16 ? k : 0] : (T)0);
  }
  double rsum = 0.0;
  if (live) {
    if constexpr (PHYS) {
      if (a.p0 && a.stage >= 1) {
        if (s_mark[cell]) {
#pragma unroll
          for (int k = 1; k < NP; ++k) out[k] = 0.0;
        }
        if (drop0) {
#pragma unroll
          for (int k = 1; k < NP; ++k) u0[k] = 0.0;
        }
      }
    }
    if constexpr (RND) {
#pragma unroll
      for (int k = 0; k < NP; ++k) acc[k] = probe<RND, T>(acc[k], a.round_mask, kRndContraction);
    }
    // the stage combination in the reference's operation order
    if (a.stage == 1) {
      if (a.U0out) st_row<NP, RALIGN>(a.U0out + gbase, out);
#pragma unroll
      for (int k = 0; k < NP; ++k) out[k] = out[k] + (double)acc[k] * dtj;
    } else if (a.stage == 2) {
#pragma unroll
      for (int k = 0; k < NP; ++k) out[k] = 0.25 * (out[k] + (double)acc[k] * dtj + 3. * u0[k]);
    } else if (a.stage == 3) {
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        out[k] = third(2.0 * (out[k] + (double)acc[k] * dtj) + u0[k]);
        const double dd = out[k] - u0[k];
        rsum += dd * dd;
      }
    } else {
#pragma unroll
      for (int k = 0; k < NP; ++k) out[k] = (double)acc[k];
    }
  }
  if constexpr (FS::UMMA) {
    tc_fence_before();
    __syncthreads();
    if (tid < 32) tmem_dealloc(s_tmem, 32);
  }
  if (live) st_row<NP, RALIGN>(a.Cout + gbase, out);
  if (a.stage != 3) return;

  // ---- last stage: residual partial of the tile and the smallest CFL step of
  // its cells (DGCell::computeMAXEV, DGCell.cc:1155-1207: eigenvalue at the
  // mean and, on triangles, at the three reference vertices), written to
  // partials[tile] and partials[ntiles + tile] for stage_finalize_kernel
  const int ntiles = (a.mesh.E + TS - 1) / TS;
  double dtl = 1e300;
  if (a.fuse_cfl) {
    if constexpr (state_dependent_speed(K::LAW)) {
      // the rows evaluate the states, field-major in place of the slots; then
      // NV neighbouring lanes take a cell's states and combine their
      // eigenvalues in the order of computeMAXEV
      double* sE = reinterpret_cast<double*>(smem_raw + FS::oS);
      __syncthreads();
      if (live) {
        sE[prow] = out[0] * a.tab.phi0;
#pragma unroll
        for (int v = 1; v < NV; ++v) {
          double s = 0;
#pragma unroll
          for (int k = 0; k < NP; ++k) s += tb.phiv[(v - 1) * NP + k] * out[k];
          sE[v * LDR + prow] = s;
        }
      }
      __syncthreads();
      for (int i0 = 0; i0 < TS * NV; i0 += NT) {
        const int e = (i0 + tid) / NV, v = (i0 + tid) % NV;
        double am = 0.0;
        if (e < ne) {
          double val[M];
#pragma unroll
          for (int j = 0; j < M; ++j) val[j] = sE[v * LDR + j * TEP + e];
          am = max_eigen<K::LAW, double>(a.law, val);
        }
#pragma unroll
        for (int w = 1; w < NV; ++w) {
          const double b = __shfl_down_sync(0xffffffffu, am, w, NV);
          if (v == 0) am = (b > am ? b : am);
        }
        if (v == 0 && e < ne) dtl = fmin(dtl, a.mesh.csize[e0 + e] * c->cfl / (am * (2. * K::ORDER + 1.0)));
      }
    } else if (tid < ne) {
      double val[M] = {};
      dtl = csz * c->cfl / (max_eigen<K::LAW, double>(a.law, val) * (2. * K::ORDER + 1.0));
    }
  }
  // both reductions of the tile with one barrier
  for (int o = 16; o > 0; o >>= 1) {
    rsum += __shfl_xor_sync(0xffffffffu, rsum, o);
    dtl = fmin(dtl, __shfl_xor_sync(0xffffffffu, dtl, o));
  }
  if ((tid & 31) == 0) {
    red[tid >> 5] = rsum;
    red[NT / 32 + (tid >> 5)] = dtl;
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < NT / 32; ++w) {
      rsum += red[w];
      dtl = fmin(dtl, red[NT / 32 + w]);
    }
    a.partials[tile] = rsum;
    if (a.fuse_cfl) a.partials[ntiles + tile] = dtl;
  }
}

// After the last stage: one CTA sums the tiles' residual partials in tile
// order, takes the minimum of their CFL steps, advances the time and, with the
// fused CFL, finalizes the next step (per instance for ensembles).  Keeping
// this out of the stage kernel spares every tile a fence and an atomic round
// trip on one address.
template <class K>
__global__ void __launch_bounds__(kFinalizeThreads) stage_finalize_kernel(
    const __grid_constant__ StageArgs<typename K::T> a, int ntiles) {
  constexpr int NT = kFinalizeThreads;
  __shared__ double red[NT / 32], redd[NT / 32];
  if (!late_start<K>(a)) pdl_trigger();
  pdl_wait();
  if (a.gctl->done) return;
  const double* part = a.partials;
  const double* dtp = a.partials + ntiles;
  const int tid = threadIdx.x;
  if (a.cell_inst) {
    // a warp per instance (a thread each took a round trip per few tiles)
    for (int i = tid / 32; i < a.ninst; i += NT / 32) {
      TimeCtl* c = a.ctl + i;
      if (c->done) continue;
      double r = 0.0, d = 1e300;
      for (int b = a.tile_first[i] + (tid & 31); b < a.tile_first[i + 1]; b += 32) {
        r += part[b];
        d = fmin(d, dtp[b]);
      }
      for (int o = 16; o > 0; o >>= 1) {
        r += __shfl_xor_sync(0xffffffffu, r, o);
        d = fmin(d, __shfl_xor_sync(0xffffffffu, d, o));
      }
      __syncwarp();
      if ((tid & 31) == 0) {
        c->resid = r;
        c->t = c->t + c->dt;
        c->steps += 1;
        if (a.fuse_cfl) {
          ctl_finalize(c, d);
          if (c->done) c->t_mark_ns = device_clock_ns();
        }
      }
    }
    __syncthreads();
    if (tid == 0) {
      int all = 1;
      for (int i = 0; i < a.ninst; ++i) all &= (*(volatile int*)&a.ctl[i].done) != 0;
      a.gctl->done = all;
    }
    return;
  }
  // one round trip for the partials and the time control, one barrier
  TimeCtl now;
  if (tid == 0) now = *a.ctl;
  double r = 0.0, d = 1e300;
  for (int b = tid; b < ntiles; b += NT) {
    r += part[b];
    d = fmin(d, dtp[b]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    r += __shfl_xor_sync(0xffffffffu, r, o);
    d = fmin(d, __shfl_xor_sync(0xffffffffu, d, o));
  }
  if ((tid & 31) == 0) {
    red[tid >> 5] = r;
    redd[tid >> 5] = d;
  }
  __syncthreads();
  if (tid < 32) {
    r = tid < NT / 32 ? red[tid] : 0.0;
    d = tid < NT / 32 ? redd[tid] : 1e300;
    for (int o = 16; o > 0; o >>= 1) {
      r += __shfl_xor_sync(0xffffffffu, r, o);
      d = fmin(d, __shfl_xor_sync(0xffffffffu, d, o));
    }
  }
  if (tid == 0) {
    now.resid = r;
    now.t = now.t + now.dt;
    now.steps += 1;
    if (a.fuse_cfl) ctl_finalize(&now, d);
    *a.ctl = now;
  }
}

}  // namespace dgp
