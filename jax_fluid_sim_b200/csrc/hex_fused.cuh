// Fused right-hand side of the sum-factorised hexahedron path: three launches per evaluation
// instead of six.
//
//   k_hex_traces   (hex_kernels.cuh): face traces of U, of the viscous variables and of
//                  their raw gradients, per face side.
//   k_hex_face     one thread per face point, the points of a face in consecutive threads:
//                  HLLC (or the boundary ghost) minus each side's anchor flux, the BR2 jump,
//                  then each side's local lift at the face points, r_f = M^-1[slab_f] B_f^T jump
//                  seen through B_f (hybrid/navier_stokes.py:138-188), and the averaged viscous
//                  normal flux (hybrid/navier_stokes.py:210-324).  The local lift is a fixed linear
//                  map of the face's jumps: for an affine element br2 coef m1i[end][end] (K (x) K)
//                  with K = bf m1i bf^T, otherwise a QF^2 x QF^2 operator per element face built
//                  once from M^-1 (k_hex_lop).  This replaces k_face_flux, the per-face part of
//                  k_hex_lift and k_face_visc, and the traces are read once.
//   k_hex_element  one CTA per element (128 threads at P3, one warp at P1 and P2): the nodal lift
//                  M^-1 sum_f B_f^T jump_f, the volume terms (U, grad v and lift at the volume points; inviscid and viscous fluxes), the face
//                  terms and M^-1 with the stage update.  The lift and the residuals stay in shared
//                  memory (no nodal-lift or residual buffers in HBM); M^-1 is read by the lift and
//                  by the final product.
// Summation order inside each phase is that of the six-launch kernels; the local
// lift is summed as one operator instead of three factors, which moves results by round-off.
#pragma once
#include "hex_kernels.cuh"
#include "mlp_kernels.cuh"

namespace dgb {

// Local face of each face side of the hexahedron block: face_lf[f * 2 + side] (set-up).
static __global__ void k_hex_face_lf(const DevPlan P_, int8_t* face_lf) {
  const BlockDev& B = P_.blk[0];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= B.E * 6) return;
  int ft, f, side;
  decode_face(B.elem_face[t], ft, f, side);
  face_lf[(size_t)f * 2 + side] = (int8_t)(t % 6);
}

// Local-lift operator of every face of the non-affine elements (set-up), in the canonical face-point
// order of that face: L[c][c'] = sum_{i,j in slab} BF[c][i] M^-1[node i][node j] BF[c'][j], BF the
// face interpolation bf (x) bf, stored as [c'][c].  One CTA per (listed element, local face).  Mt is M^-1 transposed
// in element node order (the hexahedron path's layout).
template <int P, typename T>
__global__ void k_hex_lop(const DevPlan P_, const HexTables tables, const int* __restrict__ elems, int count,
                          T* __restrict__ lop) {
  using D = HexDims<P>;
  constexpr int N = D::N, QF = D::QF, N2 = D::N2, N3 = D::N3, QF2 = D::QF2;
  __shared__ double ms[N2][N2];
  __shared__ double t1[N2][QF2];     // Mslab BF^T
  const int item = blockIdx.x;
  if (item >= count * 6) return;
  const int e = elems[item / 6], lf = item % 6;
  int a0, end, a1, a2;
  hex_face_axes(lf, a0, end, a1, a2);
  const int st0 = axis_stride<N>(a0), st1 = axis_stride<N>(a1), st2 = axis_stride<N>(a2);
  const double* Mt = P_.blk[0].minv + (size_t)e * N3 * N3;
  for (int idx = threadIdx.x; idx < N2 * N2; idx += blockDim.x) {
    const int si = idx / N2, sj = idx % N2;
    const int ni = tables.lex2node[end * st0 + (si % N) * st1 + (si / N) * st2];
    const int nj = tables.lex2node[end * st0 + (sj % N) * st1 + (sj / N) * st2];
    ms[si][sj] = Mt[(size_t)nj * N3 + ni];
  }
  __syncthreads();
  // BF[c][s] = bf[c % QF][s % N] bf[c / QF][s / N] (canonical face point c, slab node s)
  for (int idx = threadIdx.x; idx < N2 * QF2; idx += blockDim.x) {
    const int si = idx / QF2, c = idx % QF2;
    double acc = 0.0;
    for (int sj = 0; sj < N2; ++sj)
      acc += ms[si][sj] * tables.bf[(c % QF) * N + sj % N] * tables.bf[(c / QF) * N + sj / N];
    t1[si][c] = acc;
  }
  __syncthreads();
  T* out = lop + ((size_t)(item / 6) * 6 + lf) * QF2 * QF2;
  for (int idx = threadIdx.x; idx < QF2 * QF2; idx += blockDim.x) {
    const int c = idx / QF2, cp = idx % QF2;
    double acc = 0.0;
    for (int si = 0; si < N2; ++si)
      acc += tables.bf[(c % QF) * N + si % N] * tables.bf[(c / QF) * N + si / N] * t1[si][cp];
    out[cp * QF2 + c] = (T)acc;       // transposed: a face's lanes then read one row together
  }
}

// Inputs of the fused face kernel beyond the plan: the local face of each face side, the lift
// operators of the non-affine elements (lop_index[e] >= 0 selects one) and its precision.
struct HexFaceArgs {
  const int8_t* face_lf;      // [F][2]
  const int* lop_index;       // [E], -1 for affine elements
  const double* lop;          // [count][6][QF2][QF2] (transposed), float64 plans
  const float* lop32;         // the same in float32, mixed-precision plans
};

// R: arithmetic of the local lifts and the viscous face flux (float in precision mode 1; HLLC and
// the jumps are float64 in both modes).  F32: the viscous traces come from trV32 / trG32.
template <int P, int NV, typename R = double, bool F32 = false>
__global__ void __launch_bounds__(kThreads, NV <= 5 ? 6 : 1) k_hex_face(const DevPlan P_, const HexTables tables,
                                                                       const HexCodes codes, const HexFaceArgs A) {
  using D = HexDims<P>;
  constexpr int N = D::N, QF = D::QF, QF2 = D::QF2;
  constexpr int FPC = kThreads / QF2;                // faces per CTA
  constexpr bool RF = sizeof(R) == sizeof(float);    // float32 face fluxes and jumps (mixed precision)
  // jumps of each face's points, [face][point][12]; the face stride is padded to a 16-byte
  // multiple (two doubles or four floats) so that a point's 12 jumps are read by 16-byte loads
  constexpr int JS = QF2 * 12 + (sizeof(R) == sizeof(float) ? 4 : 2);
  __shared__ __align__(16) R jmp[FPC * JS];
  __shared__ R K[QF][QF];                            // bf m1i bf^T
  const FaceDev& fd = P_.face[1];
  const int slot = threadIdx.x / QF2, q = threadIdx.x % QF2;
  const int f = blockIdx.x * FPC + slot;
  const bool live = slot < FPC && f < fd.F;
  if (threadIdx.x < QF * QF) {
    const int a = threadIdx.x / QF, c = threadIdx.x % QF;
    double acc = 0.0;
    for (int j = 0; j < N; ++j)
      for (int k = 0; k < N; ++k) acc += tables.bf[a * N + j] * tables.m1i[j * N + k] * tables.bf[c * N + k];
    K[a][c] = (R)acc;
  }
  int nb = -1;
  double n[3] = {0.0, 0.0, 0.0}, w = 0.0;
  size_t so = 0, sn = 0;
  double UL[NV];
  if (live) {
    nb = fd.nb[f];
    n[0] = fd.n[face_at(f, 3, 0, QF2, q)], n[1] = fd.n[face_at(f, 3, 1, QF2, q)], n[2] = fd.n[face_at(f, 3, 2, QF2, q)];
    w = fd.w[(size_t)f * QF2 + q];
    so = (size_t)f * 2;
    sn = so + 1;
    double UR[NV], Fh[NV], Fa[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) UL[v] = fd.trA[face_at(so, NV, v, QF2, q)];
    if (nb >= 0) {
#pragma unroll
      for (int v = 0; v < NV; ++v) UR[v] = fd.trA[face_at(sn, NV, v, QF2, q)];
    } else if (P_.ph.has_boundary) {
      ghost_state<NV>(P_.ph, case_view(P_.ph, P_.blk[0].ecase, fd.ol[f]).far, UL, n, fd.tag[f], UR);
    } else {
#pragma unroll
      for (int v = 0; v < NV; ++v) UR[v] = UL[v];
    }
    hllc<NV>(P_.ph, UL, UR, n, Fh);
    {
      double a[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) a[v] = fd.anc[((size_t)f * 2 + 0) * NV + v];
      normal_flux<NV>(P_.ph, a, n, Fa);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        if (RF) fd.fluxI32[face_at(so, NV, v, QF2, q)] = (float)((Fh[v] - Fa[v]) * w);
        else fd.fluxI[face_at(so, NV, v, QF2, q)] = (Fh[v] - Fa[v]) * w;
      }
    }
    if (nb >= 0) {
      double a[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) a[v] = fd.anc[((size_t)f * 2 + 1) * NV + v];
      normal_flux<NV>(P_.ph, a, n, Fa);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        if (RF) fd.fluxI32[face_at(sn, NV, v, QF2, q)] = (float)((Fh[v] - Fa[v]) * w);
        else fd.fluxI[face_at(sn, NV, v, QF2, q)] = (Fh[v] - Fa[v]) * w;
      }
    }
  }
  if (!P_.viscous) return;
  double vo[4], vn[4];
  auto load_v = [&](size_t side, double* out) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      if constexpr (F32) out[m] = __ldg(fd.trV32 + face_at(side, 4, m, QF2, q));
      else out[m] = fd.trV[face_at(side, 4, m, QF2, q)];
    }
  };
  if (live) {
    load_v(so, vo);
    if (nb >= 0) {
      load_v(sn, vn);
    } else if (P_.ph.has_boundary) {
      const CaseView cv = case_view(P_.ph, P_.blk[0].ecase, fd.ol[f]);
      viscous_ghost<NV>(P_.ph, cv.far, cv.wall_T, UL, n, fd.tag[f], vn);
    } else {
      viscous_vars<NV>(P_.ph, UL, vn);
    }
    // a point's 12 jumps are a row of jmp: 16-byte stores
    R jr[12];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int d = 0; d < 3; ++d) jr[m * 3 + d] = (R)(0.5 * w * (vn[m] - vo[m]) * n[d]);
    R* js = &jmp[slot * JS + q * 12];
    if constexpr (RF) {
      float4* s4 = reinterpret_cast<float4*>(js);
#pragma unroll
      for (int k = 0; k < 3; ++k) s4[k] = make_float4(jr[4 * k], jr[4 * k + 1], jr[4 * k + 2], jr[4 * k + 3]);
    } else {
      double2* s2 = reinterpret_cast<double2*>(js);
#pragma unroll
      for (int k = 0; k < 6; ++k) s2[k] = make_double2(jr[2 * k], jr[2 * k + 1]);
    }
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      if constexpr (RF) fd.jumpW32[face_at(f, 12, k, QF2, q)] = jr[k];
      else fd.jumpW[face_at(f, 12, k, QF2, q)] = jr[k];
    }
  }
  __syncthreads();
  if (!live) return;
  const BlockDev& B = P_.blk[0];
  const CaseView cv = case_view(P_.ph, B.ecase, fd.ol[f]);
  const R* jf = &jmp[slot * JS];
  R Fo[3 * NV];
  const int nsides = nb >= 0 ? 2 : 1;
  for (int s = 0; s < nsides; ++s) {
    const int e = s == 0 ? fd.ol[f] : fd.nl[f];
    const int code = s == 0 ? fd.oc[f] : fd.nc[f];
    const uint8_t* perm = codes.perm + (size_t)code * QF2;
    const int lf = A.face_lf[(size_t)f * 2 + s];
    const int cq = perm[q];
    // the side's face-point permutation in registers (one 16-byte load for P3 faces), so that the
    // operator loads of the lift loop do not wait on the permutation loads one by one
    unsigned wd[4] = {0u, 0u, 0u, 0u};
    if constexpr (QF2 == 16) {
      const uint4 raw = __ldg(reinterpret_cast<const uint4*>(perm));
      wd[0] = raw.x, wd[1] = raw.y, wd[2] = raw.z, wd[3] = raw.w;
    }
    auto pm = [&](int k) -> int {
      if constexpr (QF2 == 16) return (int)((wd[k / 4] >> (8 * (k % 4))) & 0xFFu);
      else return perm[k];
    };
    // the 12 jumps of face point qp (16-byte loads from the padded rows)
    auto jrow = [&](int qp, R* r) {
      if constexpr (sizeof(R) == sizeof(float)) {
        const float4* p4 = reinterpret_cast<const float4*>(jf + qp * 12);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float4 v = p4[k];
          r[4 * k] = v.x, r[4 * k + 1] = v.y, r[4 * k + 2] = v.z, r[4 * k + 3] = v.w;
        }
      } else {
        const double2* p2 = reinterpret_cast<const double2*>(jf + qp * 12);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          const double2 v = p2[k];
          r[2 * k] = v.x, r[2 * k + 1] = v.y;
        }
      }
    };
    R lift[12];
#pragma unroll
    for (int c = 0; c < 12; ++c) lift[c] = R(0);
    const int li = A.lop_index ? A.lop_index[e] : -1;
    if (li < 0) {
      // affine: br2 coef m1i[end][end] (K (x) K) in this side's canonical order
      int a0, end, a1, a2;
      hex_face_axes(lf, a0, end, a1, a2);
      const R scale = (R)(P_.ph.br2 * B.acoef[e] * tables.m1i[end * N + end]);
      const int c1 = cq % QF, c2 = cq / QF;
#pragma unroll
      for (int qp = 0; qp < QF2; ++qp) {
        const int cp = pm(qp);
        const R kk = K[c1][cp % QF] * K[c2][cp / QF];
        R jv[12];
        jrow(qp, jv);
#pragma unroll
        for (int c = 0; c < 12; ++c) lift[c] += kk * jv[c];
      }
#pragma unroll
      for (int c = 0; c < 12; ++c) lift[c] *= scale;
    } else {
      const size_t lo = ((size_t)li * 6 + lf) * QF2 * QF2 + cq;
#pragma unroll
      for (int qp = 0; qp < QF2; ++qp) {
        R kk;
        if constexpr (sizeof(R) == sizeof(float)) kk = __ldg(A.lop32 + lo + pm(qp) * QF2);
        else kk = (R)__ldg(A.lop + lo + pm(qp) * QF2);
        R jv[12];
        jrow(qp, jv);
#pragma unroll
        for (int c = 0; c < 12; ++c) lift[c] += kk * jv[c];
      }
#pragma unroll
      for (int c = 0; c < 12; ++c) lift[c] *= (R)P_.ph.br2;
    }
    const size_t ss = s == 0 ? so : sn;
    // the owner's lift at boundary faces stays in the face buffers for the wall-force integral
    // (dgb_wall_forces reads the viscous traction there)
    if (nb < 0)
#pragma unroll
      for (int c = 0; c < 12; ++c) fd.liftF[face_at(ss, 12, c, QF2, q)] = (double)lift[c];
    R U[NV], g[12];
#pragma unroll
    for (int v = 0; v < NV; ++v) U[v] = (R)fd.trP[face_at(ss, NV, v, QF2, q)];
#pragma unroll
    for (int c = 0; c < 12; ++c) {
      if constexpr (F32) g[c] = (R)__ldg(fd.trG32 + face_at(ss, 12, c, QF2, q));
      else g[c] = (R)fd.trG[face_at(ss, 12, c, QF2, q)];
    }
#pragma unroll
    for (int c = 0; c < 12; ++c) g[c] += lift[c];
    if (s == 0) {
      viscous_flux<NV>(P_.ph, cv.mu, cv.kappa, U, g, Fo);
    } else {
      R Fn[3 * NV];
      viscous_flux<NV>(P_.ph, cv.mu, cv.kappa, U, g, Fn);
#pragma unroll
      for (int k = 0; k < 3 * NV; ++k) Fo[k] = R(0.5) * (Fo[k] + Fn[k]);
    }
  }
  R out[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v)
    out[v] = Fo[0 * NV + v] * (R)n[0] + Fo[1 * NV + v] * (R)n[1] + Fo[2 * NV + v] * (R)n[2];
  if (nb < 0 && P_.ph.has_boundary && tag_in(fd.tag[f], P_.ph.wall, P_.ph.n_wall)) out[4] = R(0);
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    if (RF) fd.fluxV32[face_at(f, NV, v, QF2, q)] = (float)(out[v] * (R)w);
    else fd.fluxV[face_at(f, NV, v, QF2, q)] = (double)(out[v] * (R)w);
  }
}

// K consecutive shared-memory values at p (16-byte aligned) into r: 16-byte loads, then an 8-byte
// load of a float pair, then single values.
template <int K, typename T>
__device__ __forceinline__ void lds_vec(const T* p, T* r) {
  constexpr int VA = 16 / sizeof(T), K16 = K / VA * VA;
#pragma unroll
  for (int k = 0; k < K16; k += VA) load16(p + k, r + k);
  constexpr int K8 = (sizeof(T) == sizeof(float) && K - K16 >= 2) ? K16 + 2 : K16;
  if constexpr (K8 > K16) {
    const float2 v = *reinterpret_cast<const float2*>(p + K16);
    r[K16] = v.x;
    r[K16 + 1] = v.y;
  }
#pragma unroll
  for (int k = K8; k < K; ++k) r[k] = p[k];
}

__host__ __device__ constexpr int up4(int n) { return (n + 3) / 4 * 4; }

// Shared-memory layout of k_hex_element, in units of R.  Nodal arrays hold N planes of PS values a channel, the
// point arrays Q3 values a channel.  The nodal U, V and lift LF stand side by side, so that their planes are
// one list; the point arrays come over them once the planes have been read.
template <int P, int NV, bool SPLIT, typename R>
struct HexElemSmem {
  using D = HexDims<P>;
  static constexpr int N = D::N, Q = D::Q, QF = D::QF, N2 = D::N2, N3 = D::N3, Q3 = D::Q3, QF2 = D::QF2;
  static constexpr int C = SPLIT ? 2 * NV : NV;          // residual channels
  static constexpr int PS = plane_stride<R>(N2), NS = N * PS, FP = plane_stride<R>(QF2), QQ = Q * Q;
  static constexpr int U = 0, V = U + NV * NS, LF = V + 4 * NS, NODAL = up4(LF + 12 * NS);
  // phase B, beyond the nodal arrays: face planes of the jumps (contracted in place), the nodal sums (or the
  // non-affine elements' rows of two groups of 6 channels, LR apart)
  static constexpr int LR = (6 * (int)sizeof(R) + 15) / 16 * 16 / (int)sizeof(R);
  static constexpr int JC = NODAL, BALL = up4(JC + 72 * FP), B_END = BALL + cmax(12 * NS, 2 * LR * N3);
  // phase C: U - anchor uq [NV][Q3], gradients of v gq [12][Q3] and the lift lq [12][Q3] (later Gi, Gv [3][NV][Q3]
  // each) at the points; half-contracted planes beyond them: U, V, LF (T2), then the two y and x derivatives of v
  static constexpr int UQ = 0, GQ = UQ + NV * Q3, LQ = GQ + 12 * Q3;
  static constexpr int T2 = up4(cmax(LQ + 12 * Q3, NODAL)), TBD = T2 + (NV + 16) * N * QQ, TDB = TBD + 4 * N * QQ;
  static constexpr int T_END = TDB + 4 * N * QQ;
  static constexpr int GI = LQ, GVI = GI + 3 * NV * Q3, G_END = up4(GI + (SPLIT ? 6 : 3) * NV * Q3);
  // residuals [C][NS]: over uq and gq, dead by then, where they fit
  static constexpr bool RR_IN = C * NS <= LQ;
  // phase D: face planes hc [6][C][FP] (later the results in memory order), then the non-affine elements' rows
  // of residuals and the M^-1 partial sums
  static constexpr int CSH = (NV + 16 / (int)sizeof(R) - 1) / (16 / (int)sizeof(R)) * (16 / (int)sizeof(R));
  static constexpr int CS = SPLIT ? 2 * CSH : CSH;
  static constexpr int D_SIZE = up4(6 * C * FP) + up4(CS * N3) + 4 * NV * N3;
  static constexpr int RR = RR_IN ? 0 : up4(cmax(G_END, D_SIZE)), RR_END = RR + up4(C * NS);
  static constexpr int HC = RR_IN ? RR_END : 0, RT = HC + up4(6 * C * FP), PART = RT + up4(CS * N3);
  static constexpr int D_END = cmax(HC + D_SIZE, RR_END);
  static_assert(C * N3 <= 6 * C * FP, "the results take the face planes' place");
  static constexpr int TOTAL = up4(cmax(cmax(B_END, T_END), cmax(G_END, D_END)));
};

// Sums over the faces of each node: put(c, l, first(c, l) + sum of fv[lf][c][node's place on lf]) for C channels.
// N = 4: a value per step, its node and places by shifts and masks.  Else a thread keeps one node, whose (at most
// three) places are found once for its channels: with 3 nodes a side the index arithmetic of every value made the
// two sums 15 % of the element kernel.  P2 element kernel, a stage: 4k elements 44.2 -> 41.9 us, 13k non-affine
// 132.6 -> 129.2, 7k with 16 variables 238 -> 229; P3 that way 3,352 -> 3,376 us (202k, mixed), so N = 4 keeps its own.
template <int N, int C, int FP, int NT, typename R, typename Put, typename First>
__device__ __forceinline__ void node_faces(const R* fv, Put put, First first) {
  constexpr int N2 = N * N, N3 = N2 * N, PAD = N == 2 ? 8 : 32;
  constexpr int G = NT / PAD < 1 ? 1 : NT / PAD > C ? C : NT / PAD, CG = (C + G - 1) / G;      // channels: G groups of CG
  if constexpr (N == 4) {
    for (int idx = threadIdx.x; idx < C * N3; idx += NT) {
      const int c = idx / N3, l = idx % N3;
      const int xyz[3] = {l % N, (l / N) % N, l / N2};
      R acc = first(c, l);
#pragma unroll
      for (int lf = 0; lf < 6; ++lf) {
        int a0, end, a1, a2;
        hex_face_axes(lf, a0, end, a1, a2);
        if (xyz[a0] == end) acc += fv[(lf * C + c) * FP + xyz[a2] * N + xyz[a1]];
      }
      put(c, l, acc);
    }
    return;
  }
  for (int t = threadIdx.x; t < PAD * G; t += NT) {
    const int l = t % PAD, c0 = t / PAD * CG;
    if (l >= N3) continue;
    const int xyz[3] = {l % N, (l / N) % N, l / N2};
    int at[6];
#pragma unroll
    for (int lf = 0; lf < 6; ++lf) {
      int a0, end, a1, a2;
      hex_face_axes(lf, a0, end, a1, a2);
      at[lf] = xyz[a0] == end ? (lf * C + c0) * FP + xyz[a2] * N + xyz[a1] : -1;
    }
#pragma unroll
    for (int k = 0; k < CG; ++k) {
      if (C % G != 0 && c0 + k >= C) break;
      R acc = first(c0 + k, l);
#pragma unroll
      for (int lf = 0; lf < 6; ++lf)
        if (at[lf] >= 0) acc += fv[at[lf] + k * FP];
      put(c0 + k, l, acc);
    }
  }
}

// Lift + volume + finalize of hexahedron e by one CTA (see the file comment).  SPLIT keeps the inviscid
// and viscous residuals apart (right-hand-side outputs, the MOOD step's viscous residual).
template <int P, int NV, bool SPLIT, typename R>
__device__ __forceinline__ void hex_element(const DevPlan& P_, const StatePtrs& S, const HexTablesT<R>& tables,
                                            const HexCodes& codes, const FinalizeArgs& A, const int e) {
  using D = HexDims<P>;
  using L = HexElemSmem<P, NV, SPLIT, R>;
  constexpr int N = D::N, Q = D::Q, QF = D::QF, N2 = D::N2, N3 = D::N3, Q3 = D::Q3, QF2 = D::QF2, NT = D::NTE;
  constexpr int C = L::C;
  constexpr int b = 0;
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  R* smem = reinterpret_cast<R*>(dyn_smem);
  constexpr int PS = L::PS, NS = L::NS, FP = L::FP, QQ = L::QQ;
  R* U = smem + L::U;            // [NV][NS] minus anchor
  R* V = smem + L::V;            // [4][NS]
  R* Lf = smem + L::LF;          // [12][NS] nodal lift
  R* Rr = smem + L::RR;          // [C][NS] residuals (inviscid, then viscous)
  auto nod = [](int l) { return l / N2 * PS + l % N2; };      // node l of a channel
  __shared__ int node2lex[64], lex2node[64], fslot[6], fperm[6], fface[6];
  __shared__ R anchor[NV], w1[Q];
  const BlockDev& B = P_.blk[b];
  const FaceDev& fd = P_.face[1];
  const CaseView cv = case_view(P_.ph, B.ecase, e);
  const double* Ug = S.b[b] + (size_t)e * N3 * NV;
  // the state arrives in one coalesced sweep (raw: beyond the nodal arrays) and is spread from shared memory
  double* raw = reinterpret_cast<double*>(smem + L::NODAL);
  static_assert((L::TOTAL - L::NODAL) * (int)sizeof(R) >= N3 * NV * (int)sizeof(double) && L::NODAL * sizeof(R) % 8 == 0,
                "raw state");
  for (int idx = threadIdx.x; idx < N3 * NV; idx += NT) raw[idx] = Ug[idx];
  if (threadIdx.x < 6) {
    int ft, f, side;
    decode_face(B.elem_face[e * 6 + threadIdx.x], ft, f, side);
    fslot[threadIdx.x] = (f * 2 + side) * QF2;
    fperm[threadIdx.x] = B.elem_code[e * 6 + threadIdx.x] * QF2;
    fface[threadIdx.x] = (f << 1) | side;
  }
  for (int l = threadIdx.x; l < N3; l += NT) {
    const int node = codes.lex2node[l];
    lex2node[l] = node;
    node2lex[node] = l;
  }
  __syncthreads();
  // what the element reads later, on its way to L2: the faces' jumps and fluxes and the stage's base
  for (int it = threadIdx.x; it < 6 * 3; it += NT) {
    const int lf = it % 6, f = fface[lf] >> 1;
    constexpr int fb = QF2 * (int)sizeof(R);
    const char* p;
    int bytes = NV * fb;
    if (it < 6) {
      p = (const char*)(sizeof(R) == 4 ? (const void*)fd.fluxI32 : (const void*)fd.fluxI) + (size_t)fslot[lf] * NV * sizeof(R);
    } else if (!P_.viscous) {
      break;
    } else if (it < 12) {
      p = (const char*)(sizeof(R) == 4 ? (const void*)fd.jumpW32 : (const void*)fd.jumpW) + (size_t)f * 12 * fb;
      bytes = 12 * fb;
    } else {
      p = (const char*)(sizeof(R) == 4 ? (const void*)fd.fluxV32 : (const void*)fd.fluxV) + (size_t)f * NV * fb;
    }
    for (int o = 0; o < bytes; o += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
  }
  if (A.stage) prefetch_l2<NT>(A.base[b] + (size_t)e * N3 * NV, N3 * NV * 8);
  if (threadIdx.x < NV) anchor[threadIdx.x] = (R)raw[threadIdx.x];
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < Q; ++k) w1[k] = tables.w1[k];
  const bool visc = P_.viscous;
  const bool aff = B.affine && B.affine[e];
  // a predicted troubled element: only its viscous residual is used (the subcell scheme replaces
  // its update), so the inviscid volume and face terms are not formed
  const bool skip_inv = SPLIT && A.skip_inviscid && A.skip_inviscid[e];
  const double* MT = B.minv + (size_t)e * N3 * N3;
  const float* MT32 = (sizeof(R) == sizeof(float) && B.minv32) ? B.minv32 + (size_t)e * N3 * N3 : nullptr;
  if (!aff) {
    // the element's M^-1, inverse Jacobians and w|det J| on their way to L2 while the nodal work runs
    if (MT32) prefetch_l2<NT>(MT32, N3 * N3 * 4);
    else prefetch_l2<NT>(MT, N3 * N3 * 8);
    if (sizeof(R) == sizeof(float) && B.jinv32) prefetch_l2<NT>(B.jinv32 + (size_t)e * Q3 * 9, Q3 * 9 * 4);
    else prefetch_l2<NT>(B.jinv + (size_t)e * Q3 * 9, Q3 * 9 * 8);
    prefetch_l2<NT>(B.wdet + (size_t)e * Q3, Q3 * 8);
  }
  for (int l = threadIdx.x; l < N3; l += NT) {
    const double* un = raw + lex2node[l] * NV;
    double u[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      u[v] = un[v];
      U[v * NS + nod(l)] = (R)(u[v] - raw[v]);
    }
    if (visc) {
      double vv[4];
      viscous_vars<NV>(P_.ph, u, vv);
#pragma unroll
      for (int m = 0; m < 4; ++m) V[m * NS + nod(l)] = (R)vv[m];
    }
  }
  if (visc) {
    __syncthreads();                    // raw is dead
    // ---- phase B: nodal lift M^-1 sum_f B_f^T jump_f
    R* jc = smem + L::JC;             // [6][12][FP] jumps at the canonical face points, then their sums at the face nodes
    R* ball = smem + L::BALL;         // [12][NS]
    constexpr int LR = L::LR;
    // one face point per thread: its 12 jump components to the canonical point
    for (int it = threadIdx.x; it < 6 * QF2; it += NT) {
      const int lf = it / QF2, q = it % QF2;
      const int cp = codes.perm[fperm[lf] + q];
      const size_t jo = face_at(fface[lf] >> 1, 12, 0, QF2, q);
#pragma unroll
      for (int k = 0; k < 12; ++k) {
        if constexpr (sizeof(R) == sizeof(float)) jc[(lf * 12 + k) * FP + cp] = fd.jumpW32[jo + k * QF2];
        else jc[(lf * 12 + k) * FP + cp] = (R)fd.jumpW[jo + k * QF2];
      }
    }
    __syncthreads();
    planes<QF, N, FP, FP, NT>(jc, jc, 72, tables.bfT, tables.bfT, threadIdx.x);
    __syncthreads();
    // non-affine elements: rows of two 16-byte aligned groups of 6 channels (LR apart) in element
    // node order, for 16-byte loads in the dense M^-1 (summed in node order)
    node_faces<N, 12, FP, NT>(jc, [&](int c, int l, R acc) {
      ball[aff ? c * NS + nod(l) : lex2node[l] * 2 * LR + (c / 6) * LR + c % 6] = acc;
    }, [](int, int) { return R(0); });
    __syncthreads();
    if (aff) {
      planes<N, N, PS, PS, NT>(ball, ball, 12 * N, tables.m1i, tables.m1i, threadIdx.x);
      __syncthreads();
      const R cf = (R)B.acoef[e];
      for (int line = threadIdx.x; line < 12 * N2; line += NT) {
        R x[N];
        line_load<N, N2, PS, NS>(ball, line, x);
#pragma unroll
        for (int o = 0; o < N; ++o) {
          R acc = R(0);
#pragma unroll
          for (int i = 0; i < N; ++i) acc += tables.m1i[o * N + i] * x[i];
          Lf[line / N2 * NS + o * PS + line % N2] = acc * cf;
        }
      }
    } else {
      auto dense_lift = [&](const auto* M) {
        for (int idx = threadIdx.x; idx < 2 * N3; idx += NT) {
          const int i = idx % N3, g = idx / N3, c0 = g * 6;
          R sacc[6] = {R(0), R(0), R(0), R(0), R(0), R(0)};
#pragma unroll 8
          for (int j = 0; j < N3; ++j) {
            const R m = (R)__ldg(M + (size_t)j * N3 + i);
            R bj[6];
            lds_vec<6>(ball + j * 2 * LR + g * LR, bj);
#pragma unroll
            for (int k = 0; k < 6; ++k) sacc[k] += m * bj[k];
          }
          const int li = nod(node2lex[i]);
#pragma unroll
          for (int k = 0; k < 6; ++k) Lf[(c0 + k) * NS + li] = sacc[k];
        }
      };
      if (MT32) dense_lift(MT32); else dense_lift(MT);
    }
  }
  __syncthreads();
  // ---- phase C: volume terms (k_hex_volume's arithmetic with the lift from shared memory)
  {
    R* uq = smem + L::UQ;                // [NV][Q3]   U - anchor at volume points
    R* gq = smem + L::GQ;                // [3][4][Q3] reference gradients of v
    R* lq = smem + L::LQ;                // [12][Q3]   nodal lift at the points; Gi, Gv reuse this region
    R* t2 = smem + L::T2;                // planes of U, V, LF contracted along x and y
    R* tbd = smem + L::TBD;              // the same of V with the y derivative, and with the x derivative
    R* tdb = smem + L::TDB;
    // U, V and the lift as one list of planes, then V's derivatives; three directions share the planes:
    // each gradient goes through the same three 1-D products as a contraction of its own
    planes<N, Q, PS, QQ, NT>(U, t2, (visc ? NV + 16 : NV) * N, tables.bq, tables.bq, rotated<NT>(0));
    if (visc) {
      planes<N, Q, PS, QQ, NT>(V, tbd, 4 * N, tables.bq, tables.dq, rotated<NT>((NV + 16) * N));
      planes<N, Q, PS, QQ, NT>(V, tdb, 4 * N, tables.dq, tables.bq, rotated<NT>((NV + 20) * N));
    }
    __syncthreads();
    constexpr int CQ = N * QQ;
    lines<N, Q, QQ, QQ, CQ, QQ, Q3, NT>(t2, uq, NV * QQ, tables.bq, rotated<NT>(0));
    if (visc) {
      lines<N, Q, QQ, QQ, CQ, QQ, Q3, NT>(t2 + (NV + 4) * CQ, lq, 12 * QQ, tables.bq, rotated<NT>(NV * QQ));
      lines<N, Q, QQ, QQ, CQ, QQ, Q3, NT>(tdb, gq, 4 * QQ, tables.bq, rotated<NT>((NV + 12) * QQ));
      lines<N, Q, QQ, QQ, CQ, QQ, Q3, NT>(tbd, gq + 4 * Q3, 4 * QQ, tables.bq, rotated<NT>((NV + 16) * QQ));
      lines<N, Q, QQ, QQ, CQ, QQ, Q3, NT>(t2 + NV * CQ, gq + 8 * Q3, 4 * QQ, tables.dq, rotated<NT>((NV + 20) * QQ));
    }
    __syncthreads();
    const double* jinv = B.jinv + (size_t)e * Q3 * 9;
    const float* jinv32 = (sizeof(R) == sizeof(float) && B.jinv32) ? B.jinv32 + (size_t)e * Q3 * 9 : nullptr;
    const double* wdet = B.wdet + (size_t)e * Q3;
    R Ja[9], deta = R(0);
    if (aff) {
#pragma unroll
      for (int k = 0; k < 9; ++k) Ja[k] = (R)B.ajinv[(size_t)e * 9 + k];
      deta = (R)B.adet[e];
    }
    // a point's Gi and Gv take the place of its own lift (and later channels): no other thread reads there
    R* Gi = smem + L::GI;                // [3][NV][Q3]
    R* Gv = smem + L::GVI;               // [3][NV][Q3] (SPLIT only)
    R Fa[3][NV];
    {
      const R ex[3] = {R(1), R(0), R(0)}, ey[3] = {R(0), R(1), R(0)}, ez[3] = {R(0), R(0), R(1)};
      normal_flux<NV>(P_.ph, anchor, ex, Fa[0]);
      normal_flux<NV>(P_.ph, anchor, ey, Fa[1]);
      normal_flux<NV>(P_.ph, anchor, ez, Fa[2]);
    }
    for (int q = threadIdx.x; q < Q3; q += NT) {
      R J[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) J[k] = aff ? Ja[k] : (jinv32 ? (R)jinv32[k * Q3 + q] : (R)jinv[k * Q3 + q]);
      const R wq = aff ? w1[q / (Q * Q)] * w1[(q / Q) % Q] * w1[q % Q] * deta : (R)wdet[q];
      R Uq[NV], F[3][NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) Uq[v] = anchor[v] + uq[v * Q3 + q];
      if (skip_inv) {
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
          for (int v = 0; v < NV; ++v) F[d][v] = Fa[d][v];
      } else {
        const R ex[3] = {R(1), R(0), R(0)}, ey[3] = {R(0), R(1), R(0)}, ez[3] = {R(0), R(0), R(1)};
        normal_flux<NV>(P_.ph, Uq, ex, F[0]);
        normal_flux<NV>(P_.ph, Uq, ey, F[1]);
        normal_flux<NV>(P_.ph, Uq, ez, F[2]);
      }
      R Fv[3 * NV];
#pragma unroll
      for (int k = 0; k < 3 * NV; ++k) Fv[k] = R(0);
      if (visc) {
        // reference -> physical gradient, plus the lift
        R grad[12];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const R g0 = gq[m * Q3 + q], g1 = gq[(4 + m) * Q3 + q], g2 = gq[(8 + m) * Q3 + q];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            R x = g0 * J[0 * 3 + d] + g1 * J[1 * 3 + d] + g2 * J[2 * 3 + d];
            x += lq[(m * 3 + d) * Q3 + q];
            grad[m * 3 + d] = x;
          }
        }
        viscous_flux<NV>(P_.ph, cv.mu, cv.kappa, Uq, grad, Fv);
      }
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const R gi = (J[r * 3 + 0] * (F[0][v] - Fa[0][v]) + J[r * 3 + 1] * (F[1][v] - Fa[1][v]) +
                        J[r * 3 + 2] * (F[2][v] - Fa[2][v])) * wq;
          const R gv = -(J[r * 3 + 0] * Fv[0 * NV + v] + J[r * 3 + 1] * Fv[1 * NV + v] +
                         J[r * 3 + 2] * Fv[2 * NV + v]) * wq;
          if (SPLIT) {
            Gi[(r * NV + v) * Q3 + q] = gi;
            Gv[(r * NV + v) * Q3 + q] = gv;
          } else {
            Gi[(r * NV + v) * Q3 + q] = gi + gv;
          }
        }
    }
    __syncthreads();
    // weak divergence: planes along x and y in place (dqT along the direction of the component), then along z,
    // where the three components' terms are summed as (t0 + t1) + t2
    auto divergence = [&](R* G, R* out) {
      planes<Q, N, QQ, QQ, NT>(G, G, NV * Q, tables.dqT, tables.bqT, rotated<NT>(0));
      planes<Q, N, QQ, QQ, NT>(G + NV * Q3, G + NV * Q3, NV * Q, tables.bqT, tables.dqT, rotated<NT>(NV * Q));
      planes<Q, N, QQ, QQ, NT>(G + 2 * NV * Q3, G + 2 * NV * Q3, NV * Q, tables.bqT, tables.bqT, rotated<NT>(2 * NV * Q));
      __syncthreads();
      for (int line = threadIdx.x; line < NV * N2; line += NT) {
        R x0[Q], x1[Q], x2[Q];
        line_load<Q, N2, QQ, Q3>(G, line, x0);
        line_load<Q, N2, QQ, Q3>(G + NV * Q3, line, x1);
        line_load<Q, N2, QQ, Q3>(G + 2 * NV * Q3, line, x2);
#pragma unroll
        for (int o = 0; o < N; ++o) {
          R s0 = R(0), s1 = R(0), s2 = R(0);
#pragma unroll
          for (int i = 0; i < Q; ++i) s0 += tables.bqT[o * Q + i] * x0[i];
#pragma unroll
          for (int i = 0; i < Q; ++i) s1 += tables.bqT[o * Q + i] * x1[i];
#pragma unroll
          for (int i = 0; i < Q; ++i) s2 += tables.dqT[o * Q + i] * x2[i];
          R acc = s0;
          acc += s1;
          acc += s2;
          out[line / N2 * NS + o * PS + line % N2] = acc;
        }
      }
      __syncthreads();
    };
    R* Rv = Rr + NV * NS;
    if (skip_inv) {
      for (int idx = threadIdx.x; idx < NV * NS; idx += NT) Rr[idx] = R(0);
      __syncthreads();
    } else {
      divergence(Gi, Rr);
    }
    if (SPLIT) {
      if (visc) {
        divergence(Gv, Rv);
      } else {
        for (int idx = threadIdx.x; idx < NV * NS; idx += NT) Rv[idx] = R(0);
        __syncthreads();
      }
    }
  }
  // ---- phase D: face terms, M^-1, stage update (k_hex_finalize with the residuals in shared memory)
  R* hc = smem + L::HC;                         // [6][C][FP] face flux at canonical points, then at the face nodes
  const size_t base = (size_t)e * N3 * NV;
  // one face point per thread: its NV inviscid and NV viscous flux values (contiguous)
  for (int it = threadIdx.x; it < 6 * QF2; it += NT) {
    const int lf = it / QF2, q = it % QF2;
    const int f = fface[lf] >> 1, side = fface[lf] & 1;
    const double si = side == 0 ? -1.0 : 1.0;
    const int c = codes.perm[fperm[lf] + q];
    const size_t ki = (size_t)fslot[lf] * NV + q, kv = (size_t)f * QF2 * NV + q;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      if constexpr (sizeof(R) == sizeof(float)) {
        // float32 fluxes of the mixed-precision face kernel
        const R hi = skip_inv ? R(0) : (R)si * fd.fluxI32[ki + v * QF2];
        const R hv = visc ? -(R)si * fd.fluxV32[kv + v * QF2] : R(0);
        if (SPLIT) {
          hc[(lf * C + v) * FP + c] = hi;
          hc[(lf * C + NV + v) * FP + c] = hv;
        } else {
          hc[(lf * C + v) * FP + c] = hi + hv;
        }
      } else {
        const double hi = skip_inv ? 0.0 : si * fd.fluxI[ki + v * QF2];
        const double hv = visc ? -si * fd.fluxV[kv + v * QF2] : 0.0;
        if (SPLIT) {
          hc[(lf * C + v) * FP + c] = (R)hi;
          hc[(lf * C + NV + v) * FP + c] = (R)hv;
        } else {
          hc[(lf * C + v) * FP + c] = (R)(hi + hv);
        }
      }
    }
  }
  __syncthreads();
  planes<QF, N, FP, FP, NT>(hc, hc, 6 * C, tables.bfT, tables.bfT, threadIdx.x);
  __syncthreads();
  // non-affine elements: the residuals go to rows RrT [N3][CS] in element node order (inviscid
  // channels, then from CSH the viscous ones) beyond hc, for pair loads in the
  // dense M^-1
  constexpr int CSH = L::CSH, CS = L::CS;
  R* RrT = smem + L::RT;
  node_faces<N, C, FP, NT>(hc, [&](int c, int l, R acc) {
    if (aff)
      Rr[c * NS + nod(l)] = acc;
    else
      RrT[lex2node[l] * CS + (c < NV ? c : CSH + c - NV)] = acc;
  }, [&](int c, int l) { return Rr[c * NS + nod(l)]; });
  __syncthreads();
  // values idx (node-major, as in memory) of the residuals, inviscid and viscous: coalesced stores
  auto emit = [&](const R* inv, const R* vis, R cf) {
    for (int idx = threadIdx.x; idx < NV * N3; idx += NT) {
      const size_t o = base + idx;
      const double ri = (double)(cf * inv[idx]), rv = SPLIT ? (double)(cf * vis[idx]) : 0.0;
      if (!A.stage) {
        if (A.out_inv[b]) A.out_inv[b][o] = ri;
        if (SPLIT && A.out_vis[b]) A.out_vis[b][o] = rv;
      } else {
        const double total = SPLIT ? ri + rv : ri;
        const double eul = S.b[b][o] + A.dt * total;
        if (SPLIT && A.out_vis[b]) A.out_vis[b][o] = rv;
        if (A.euler[b]) A.euler[b][o] = eul;
        A.dst[b][o] = A.alpha * A.base[b][o] + A.beta * eul;
      }
    }
  };
  R* rows = hc;                                       // [C / NV][N3][NV] results in memory order (hc is dead)
  if (aff) {
    planes<N, N, PS, PS, NT>(Rr, Rr, C * N, tables.m1i, tables.m1i, threadIdx.x);
    __syncthreads();
    for (int line = threadIdx.x; line < C * N2; line += NT) {
      R x[N];
      line_load<N, N2, PS, NS>(Rr, line, x);
      const int c = line / N2;
#pragma unroll
      for (int o = 0; o < N; ++o) {
        R acc = R(0);
#pragma unroll
        for (int i = 0; i < N; ++i) acc += tables.m1i[o * N + i] * x[i];
        rows[(c / NV) * NV * N3 + lex2node[o * N2 + line % N2] * NV + c % NV] = acc;
      }
    }
    __syncthreads();
    emit(rows, rows + NV * N3, (R)B.acoef[e]);
    return;
  }
  constexpr int VB = NV < 8 ? NV : 8;
  constexpr int NG = (NV + VB - 1) / VB;
  constexpr int HALVES = NG * N3 * 2 <= kThreads ? 2 : 1;
  constexpr int JH = (N3 + HALVES - 1) / HALVES;
  R* part = smem + L::PART;                           // [HALVES][2][NV][N3]
  auto apply = [&](const auto* M) {
    for (int idx = threadIdx.x; idx < HALVES * NG * N3; idx += NT) {
      const int i = idx % N3, g = (idx / N3) % NG, h = idx / (NG * N3);
      const int v0 = g * VB;
      R ri[VB], rv[VB];
#pragma unroll
      for (int k = 0; k < VB; ++k) ri[k] = rv[k] = R(0);
      const int j1 = (h + 1) * JH < N3 ? (h + 1) * JH : N3;
#pragma unroll 8
      for (int j = h * JH; j < j1; ++j) {
        const R m = (R)__ldg(M + (size_t)j * N3 + i);
        R xi[VB], xv[VB];
        lds_vec<VB>(RrT + j * CS + v0, xi);
        if (SPLIT) lds_vec<VB>(RrT + j * CS + CSH + v0, xv);
#pragma unroll
        for (int k = 0; k < VB; ++k) {
          if (v0 + k < NV) {
            ri[k] += m * xi[k];
            if (SPLIT) rv[k] += m * xv[k];
          }
        }
      }
#pragma unroll
      for (int k = 0; k < VB; ++k) {
        if (v0 + k >= NV) continue;
        part[((h * 2 + 0) * NV + v0 + k) * N3 + i] = ri[k];
        part[((h * 2 + 1) * NV + v0 + k) * N3 + i] = rv[k];
      }
    }
  };
  if (MT32) apply(MT32); else apply(MT);
  __syncthreads();
  for (int idx = threadIdx.x; idx < NV * N3; idx += NT) {
    const int v = idx / N3, i = idx % N3;
    R si = part[(0 * NV + v) * N3 + i], sv = part[(1 * NV + v) * N3 + i];
    if (HALVES == 2) {
      si += part[(2 * NV + v) * N3 + i];
      sv += part[(3 * NV + v) * N3 + i];
    }
    rows[i * NV + v] = si;
    if (SPLIT) rows[NV * N3 + i * NV + v] = sv;
  }
  __syncthreads();
  emit(rows, rows + NV * N3, R(1));
}

template <int P, int NV, bool SPLIT, typename R>
constexpr int hex_element_ctas() { return sizeof(R) == sizeof(float) ? (SPLIT || NV > 5 ? 6 : 7) * kThreads / HexDims<P>::NTE : 1; }

// Every element, except those flagged in A.skip.
template <int P, int NV, bool SPLIT, typename R>
__global__ void __launch_bounds__(HexDims<P>::NTE, hex_element_ctas<P, NV, SPLIT, R>())
    k_hex_element(const __grid_constant__ DevPlan P_, const StatePtrs S, const __grid_constant__ HexTablesT<R> tables,
                  const HexCodes codes, const __grid_constant__ FinalizeArgs A) {
  prefetch_ahead<P, NV, HexDims<P>::NTE>(P_.blk[0], S.b[0]);
  if (A.skip && A.skip[blockIdx.x]) return;     // uniform across the CTA
  hex_element<P, NV, SPLIT, R>(P_, S, tables, codes, A, blockIdx.x);
}

// The listed elements, taken in turn by the CTAs.
template <int P, int NV, typename R>
__global__ void __launch_bounds__(HexDims<P>::NTE, hex_element_ctas<P, NV, true, R>())
    k_hex_element_list(const __grid_constant__ DevPlan P_, const StatePtrs S, const __grid_constant__ HexTablesT<R> tables,
                       const HexCodes codes, const __grid_constant__ FinalizeArgs A, const unsigned* __restrict__ list,
                       const unsigned* __restrict__ count) {
  const unsigned n = *count;
  for (unsigned i = blockIdx.x; i < n; i += gridDim.x) {
    hex_element<P, NV, true, R>(P_, S, tables, codes, A, (int)list[i]);
    __syncthreads();
  }
}

// Predictor statistics of the hexahedron block (the layout of k_elem_stats), one warp per element:
// the Persson fractions use the tensor-product P1 projector (three N x N pencil passes, as the
// troubled-cell sensor) instead of the dense Np x Np projector, whose rows every warp would
// stream from L2 for every element.
template <int P, int NV>
__global__ void __launch_bounds__(kThreads) k_hex_elem_stats(const DevPlan P_, const StatePtrs S,
                                                            const HexTables tables, float* __restrict__ stats) {
  using D = HexDims<P>;
  constexpr int N = D::N, N3 = D::N3;
  __shared__ double work[kThreads / 32][4 * 2 * N3];   // per warp: Mon, Low, t1, t2
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e = blockIdx.x * (kThreads / 32) + warp;
  if (e >= P_.blk[0].E) return;
  const double* Ug = S.b[0] + (size_t)e * N3 * NV;
  double* Mon = work[warp];
  double* Low = Mon + 2 * N3;
  double* t1 = Low + 2 * N3;
  double* t2 = t1 + 2 * N3;
  double srho = 0, sp = 0, rmin = INFINITY, rmax = -INFINITY, pmin = INFINITY, pmax = -INFINITY;
  for (int l = lane; l < N3; l += 32) {
    double u[NV], W[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) u[v] = Ug[tables.lex2node[l] * NV + v];
    primitive<NV>(P_.ph, u, W);
    Mon[l] = W[0];
    Mon[N3 + l] = W[4];
    srho += W[0];
    sp += W[4];
    rmin = fmin(rmin, W[0]);
    rmax = fmax(rmax, W[0]);
    pmin = fmin(pmin, W[4]);
    pmax = fmax(pmax, W[4]);
  }
  __syncwarp();
  double h0 = 0, h1 = 0, s0 = 0, s1 = 0;
  if (P >= 2) {
    warp_tensor3<2, N>(Mon, Low, t1, t2, tables.p1d);
    for (int i = lane; i < N3; i += 32) {
      const double m0 = Mon[i], m1 = Mon[N3 + i];
      const double d0 = m0 - Low[i], d1 = m1 - Low[N3 + i];
      h0 += d0 * d0;
      h1 += d1 * d1;
      s0 += m0 * m0;
      s1 += m1 * m1;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    srho += __shfl_xor_sync(0xffffffff, srho, o);
    sp += __shfl_xor_sync(0xffffffff, sp, o);
    rmin = fmin(rmin, __shfl_xor_sync(0xffffffff, rmin, o));
    rmax = fmax(rmax, __shfl_xor_sync(0xffffffff, rmax, o));
    pmin = fmin(pmin, __shfl_xor_sync(0xffffffff, pmin, o));
    pmax = fmax(pmax, __shfl_xor_sync(0xffffffff, pmax, o));
    h0 += __shfl_xor_sync(0xffffffff, h0, o);
    h1 += __shfl_xor_sync(0xffffffff, h1, o);
    s0 += __shfl_xor_sync(0xffffffff, s0, o);
    s1 += __shfl_xor_sync(0xffffffff, s1, o);
  }
  if (lane == 0) {
    float* st = stats + (size_t)e * kMlpStats;
    st[0] = (float)(srho / N3);
    st[1] = (float)(sp / N3);
    st[2] = (float)(rmin / fmax(fabs(rmax), 1e-30));
    st[3] = (float)(pmin / fmax(fabs(pmax), 1e-30));
    st[4] = (float)(h0 / fmax(s0, 1e-12));
    st[5] = (float)(h1 / fmax(s1, 1e-12));
  }
}

}  // namespace dgb
