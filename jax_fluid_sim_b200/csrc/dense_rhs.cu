// Right-hand side of the dense path (hybrid meshes: hexahedra, wedges, tetrahedra) in two launches per
// evaluation (hybrid/spatial.py:47-72,137-249, hybrid/navier_stokes.py:27-347), as one residual:
//
//   k_dense_faces    face traces and HLLC flux: one thread per face point.  The traces are formed from
//                    the nodes on the face (the basis of every other node is zero there), read
//                    from the element states, so no trace buffer goes through memory.  With viscous
//                    terms also the gradients, the BR2 jump, both sides' local lifts (M^-1 over the face's
//                    nodes alone, 9 to 16 times fewer products than over all nodes) and the viscous flux.
//   k_dense_update   one CTA per NE elements: (nodal lift,) volume residual, face terms, M^-1 and the
//                    stage update, with everything between them in shared memory.
//
// The residual of a 4^3 P2 hybrid box with viscous terms took nine launches and three additions of the
// split residuals, 122 us, and takes these two, 51 us.  Split residuals (MOOD, the separate right-hand
// sides) and mixed viscous plans keep the general kernels of dg_kernels.cuh.
//
// The element kernel is bound by the operand loads of its contractions, not by their arithmetic: with
// one accumulator row per table value and broadcast operand (one element per CTA, one value per
// load) the load pipe runs at three times the FP64 pipe's time.  So a thread keeps a tile: EB elements x
// NV variables of one point while it interpolates, IB nodes x EB2 elements x NV variables of one chunk
// of points while it sums the residual, with 16-byte shared-memory loads; a table value from L1/L2 then
// serves EB * NV products instead of NV.  NE is chosen so that both phases fill kThreads.
// Checked Euler steps of hybrid boxes, general kernels against these two: 16^3 P3 1860 -> 952 us, 32^3 P1
// 1308 -> 499 us, 23^3 P2 mixed 2776 -> 1433 us.
// A nodal value that is not finite reaches a neighbour through the faces that the node lies on; the general kernels
// multiply it by the zeros of the other faces' tables as well, so it is a ring of elements further after a step.  Either
// way the element itself is not finite and the step's status refuses the state.
// Sums run in the order of the one-value-per-thread form: per output the nodes (points) ascend, and
// the residual is summed per chunk of points, then over the chunks.
#include "dense_rhs.h"

namespace dgb {

namespace {

// Shapes of an element of type T (0 hexahedron, 1 wedge, 2 tetrahedron) at degree P.
template <int P, int T>
struct Shape {
  static constexpr int N1 = P + 1, TRI = (P + 1) * (P + 2) / 2, QUAD = N1 * N1;
  static constexpr int Np = T == 0 ? N1 * N1 * N1 : T == 1 ? TRI * N1 : (P + 1) * (P + 2) * (P + 3) / 6;
  static constexpr int Nq = T == 0 ? (P == 1 ? 8 : P == 2 ? 27 : 125) : T == 1 ? (P == 1 ? 6 : 125) : (P == 1 ? 4 : 125);
  static constexpr int nlf = T == 0 ? 6 : T == 1 ? 5 : 4;
  static constexpr int ntri = T == 0 ? 0 : T == 1 ? 2 : 4;         // the triangles come first
  static constexpr int NQT = P == 1 ? 3 : P == 2 ? 16 : 25, NQQ = (P + 1) * (P + 1);
  static constexpr int Nf = ntri * NQT + (nlf - ntri) * NQQ;        // face points
  static constexpr int Nj = ntri * TRI + (nlf - ntri) * QUAD;       // face nodes, per face
  __host__ __device__ static constexpr int nq(int lf) { return lf < ntri ? NQT : NQQ; }
  __host__ __device__ static constexpr int nfn(int lf) { return lf < ntri ? TRI : QUAD; }
  __host__ __device__ static constexpr int poff(int lf) { return lf <= ntri ? lf * NQT : ntri * NQT + (lf - ntri) * NQQ; }
  __host__ __device__ static constexpr int joff(int lf) { return lf <= ntri ? lf * TRI : ntri * TRI + (lf - ntri) * QUAD; }
};

// Work split: NE elements per CTA; EB elements per thread while interpolating, IB nodes x EB2
// elements per thread in the residual sum.  P2 and P3 volume rules of 125 points take one thread per
// point over four elements; the 27 points of a P2 hexahedron leave room for four pairs; P1 elements
// are one thread per (element, point).
// With viscous terms an element has about four times the work and shared memory: one P2 or P3 element per CTA
// (two 27-point hexahedra), tiles of one element.
template <int P, int T, bool VISC>
struct Split {
  static constexpr bool one = P == 1;
  static constexpr int NE = VISC ? (one ? (T == 0 ? 8 : T == 1 ? 10 : 16) : (P == 2 && T == 0 ? 2 : 1))
                                 : (one ? (T == 0 ? 16 : T == 1 ? 20 : 32) : (P == 2 && T == 0 ? 8 : 4));
  static constexpr int EB = one || VISC ? 1 : (P == 2 && T == 0 ? 2 : 4);
  static constexpr int EB2 = one || VISC ? 1 : 2;
  static constexpr int IB = one || VISC || Shape<P, T>::Np % 2 ? 1 : 2;
};

__host__ __device__ constexpr int round_up(int a, int b) { return (a + b - 1) / b * b; }

// Shared memory of k_dense_update in units of R.
template <int P, int T, int NV, typename R, bool VISC>
struct Smem {
  using S = Shape<P, T>;
  using W = Split<P, T, VISC>;
  static constexpr int VA = 16 / (int)sizeof(R);
  static constexpr int UE = round_up(W::EB * NV, VA);                  // one node of EB elements
  static constexpr int UG = S::Np * UE;                                 // one group of EB elements
  static constexpr int GP = round_up(W::EB2 * 3 * NV, VA);             // one point of EB2 elements
  // point stride of a group: an odd number of 16-byte units, so that a warp's stores (one point per
  // lane) fall on distinct banks
  static constexpr int GQ0 = W::EB / W::EB2 * GP, GQ = (GQ0 / VA) % 2 ? GQ0 : GQ0 + VA;
  static constexpr int GG0 = S::Nq * GQ, GG = (GG0 / VA) % 2 ? GG0 : GG0 + VA;
  // at the front: anchors (double), their fluxes, and two ints per (element, face)
  static constexpr int AN = W::NE * NV * (8 / (int)sizeof(R)), FA = W::NE * 3 * NV;
  static constexpr int FI = (2 * W::NE * S::nlf * 4 + (int)sizeof(R) - 1) / (int)sizeof(R);
  static constexpr int U = round_up(AN + FA + FI, VA);
  // viscous plans: nodal viscous variables [NE][Np][4] and lift [NE][Np][12]; before the points are worked, the
  // jumps [NE][Nf][12] and their nodal sums [NE][Np][12] where G goes
  static constexpr int V = U + W::NE / W::EB * UG, LF = V + (VISC ? W::NE * S::Np * 4 : 0);
  static constexpr int Gs = LF + (VISC ? W::NE * S::Np * 12 : 0);
  static constexpr int JS = Gs, BS = JS + W::NE * S::Nf * 12, B_END = VISC ? BS + W::NE * S::Np * 12 : 0;
  static constexpr int G = W::NE / W::EB * GG;
  // over G once it is dead: chunk sums, fluxes, face sums, totals, results
  static constexpr int FS = round_up(NV, VA);                          // one row of NV values
  static constexpr int chunk_max = kThreads / S::Np > 0 ? kThreads / S::Np : 1;
  static constexpr int Pc = W::one ? W::NE * S::Np * FS : chunk_max * W::NE * S::Np * FS;
  static constexpr int Fl = Gs + round_up(Pc, VA), Fp = Fl + W::NE * S::Nf * FS;
  // totals: over the fluxes, which are dead by then, except at P1 (in the chunk sums' place: each
  // thread reads its own sums before it writes its total)
  static constexpr int Tt = W::one ? Gs : Fl;
  static constexpr int End = Fp + (W::one ? 0 : W::NE * S::Nj * FS);   // P1: no face sums
  static_assert(S::Np <= S::Nf, "the totals take the fluxes' place");
  static constexpr int most = Gs + G > End ? Gs + G : End, total = most > B_END ? most : B_END;
};

// n values at p (16-byte aligned)
template <int K, typename R>
__device__ __forceinline__ void lds16(const R* p, R* r) {
  constexpr int VA = 16 / (int)sizeof(R);
  if constexpr (sizeof(R) == 8) {
#pragma unroll
    for (int k = 0; k < K / VA; ++k) {
      const double2 v = reinterpret_cast<const double2*>(p)[k];
      r[2 * k] = v.x, r[2 * k + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < K / VA; ++k) {
      const float4 v = reinterpret_cast<const float4*>(p)[k];
      r[4 * k] = v.x, r[4 * k + 1] = v.y, r[4 * k + 2] = v.z, r[4 * k + 3] = v.w;
    }
  }
#pragma unroll
  for (int k = K / VA * VA; k < K; ++k) r[k] = p[k];
}
template <int K, typename R>
__device__ __forceinline__ void sts16(R* p, const R* r) {
  constexpr int VA = 16 / (int)sizeof(R);
  if constexpr (sizeof(R) == 8) {
#pragma unroll
    for (int k = 0; k < K / VA; ++k) reinterpret_cast<double2*>(p)[k] = make_double2(r[2 * k], r[2 * k + 1]);
  } else {
#pragma unroll
    for (int k = 0; k < K / VA; ++k)
      reinterpret_cast<float4*>(p)[k] = make_float4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
  }
#pragma unroll
  for (int k = K / VA * VA; k < K; ++k) p[k] = r[k];
}

// ------------------------------------------------------------------------------------ element kernel
template <int P, int T, int NV, typename R, bool VISC>
__device__ __forceinline__ void update_body(const DevPlan& D, const StatePtrs& St, const FinalizeArgs& A,
                                            const DenseBlock& X, int b, int cta, bool volume_done, R* sm) {
  using S = Shape<P, T>;
  using W = Split<P, T, VISC>;
  using L = Smem<P, T, NV, R, VISC>;
  constexpr int Np = S::Np, Nq = S::Nq, nlf = S::nlf, NE = W::NE, EB = W::EB, EB2 = W::EB2, IB = W::IB;
  double* anchor = reinterpret_cast<double*>(sm);
  R* Fanc = sm + L::AN;                                                // flux of the anchor states
  int* fslot = reinterpret_cast<int*>(Fanc + L::FA);
  int* fcode = fslot + NE * nlf;
  const BlockDev& B = D.blk[b];
  const int e0 = cta * NE, ne = B.E - e0 < NE ? B.E - e0 : NE;     // elements of this CTA
  const double* Ug = St.b[b] + (size_t)e0 * Np * NV;
  const int C = X.chunks;
  // every load of a phase is issued before its first use: at three CTAs per SM a loop of dependent
  // load and store pairs waits out each latency in turn
  auto faces = [&]() {
    for (int t = threadIdx.x; t < ne * nlf; t += kThreads) {
      int ft, f, side;
      decode_face(B.elem_face[(size_t)e0 * nlf + t], ft, f, side);
      fslot[t] = (f << 1) | side;
      fcode[t] = side == 0 ? D.face[ft].oc[f] : D.face[ft].nc[f];
    }
  };
  constexpr int VALS = NE * Np * NV, VR = (VALS + kThreads - 1) / kThreads;
  if (!volume_done) {
    for (int t = threadIdx.x; t < NE * NV; t += kThreads)
      anchor[t] = t / NV < ne ? Ug[(size_t)(t / NV) * Np * NV + t % NV] : 1.0;
    R* U = sm + L::U;
    R* G = sm + L::Gs;
    // U minus the anchor; the slots past the last element hold zeros (and unit anchors), so that their
    // points stay finite
    R x[VR];
#pragma unroll
    for (int k = 0; k < VR; ++k) {
      const int t = k * kThreads + threadIdx.x, e = t / (Np * NV);
      x[k] = t < VALS && e < ne ? (R)(Ug[t] - Ug[(size_t)e * Np * NV + t % NV]) : (R)0;
    }
    faces();
#pragma unroll
    for (int k = 0; k < VR; ++k) {
      const int t = k * kThreads + threadIdx.x;
      const int e = t / (Np * NV), i = (t / NV) % Np, v = t % NV;
      if (t < VALS) U[(e / EB) * L::UG + i * L::UE + (e % EB) * NV + v] = x[k];
    }
    if constexpr (VISC)
      for (int t = threadIdx.x; t < NE * Np; t += kThreads) {
        double u[NV], vv[4] = {0.0, 0.0, 0.0, 0.0};
        if (t / Np < ne) {
#pragma unroll
          for (int v = 0; v < NV; ++v) u[v] = Ug[t * NV + v];
          viscous_vars<NV>(D.ph, u, vv);
        }
        sts16<4>(sm + L::V + t * 4, vv);
      }
    __syncthreads();
    if constexpr (VISC) {
      // ---- nodal lift M^-1 sum_f B_f^T jump_f (hybrid/navier_stokes.py:138-188)
      double* Js = sm + L::JS;
      double* Bs = sm + L::BS;
      for (int t = threadIdx.x; t < NE * S::Nf * 12; t += kThreads) {
        const int e = t / (S::Nf * 12), r = t % (S::Nf * 12);
        int lf = 0;
#pragma unroll
        for (int m = 1; m < nlf; ++m) lf += r >= S::poff(m) * 12;
        const int nq = S::nq(lf), k = (r - S::poff(lf) * 12) / nq, q = (r - S::poff(lf) * 12) % nq;
        double x = 0.0;
        if (e < ne) x = D.face[lf < S::ntri ? 0 : 1].jumpW[face_at(fslot[e * nlf + lf] >> 1, 12, k, nq, q)];
        Js[(e * S::Nf + S::poff(lf) + q) * 12 + k] = x;
      }
      __syncthreads();
      // thread = (element, node, four of the twelve components)
      for (int t = threadIdx.x; t < ne * Np * 3; t += kThreads) {
        const int e = t / (Np * 3), i = t % Np, g = t / Np % 3 * 4;
        double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int lf = 0; lf < nlf; ++lf) {
          const int ft = lf < S::ntri ? 0 : 1, nq = S::nq(lf), nfn = S::nfn(lf);
          const int j = X.finv[ft][fcode[e * nlf + lf] * Np + i];
          if (j < 0) continue;
          const double* cB = static_cast<const double*>(X.cB[ft]) + (size_t)fcode[e * nlf + lf] * nq * nfn + j;
          const double* js = Js + (e * S::Nf + S::poff(lf)) * 12 + g;
#pragma unroll 4
          for (int q = 0; q < nq; ++q) {
            const double bt = __ldg(cB + q * nfn);
            double x[4];
            lds16<4>(js + q * 12, x);
#pragma unroll
            for (int k = 0; k < 4; ++k) s[k] += bt * x[k];
          }
        }
        sts16<4>(Bs + (e * Np + i) * 12 + g, s);
      }
      __syncthreads();
      for (int t = threadIdx.x; t < ne * Np * 3; t += kThreads) {
        const int e = t / (Np * 3), i = t % Np, g = t / Np % 3 * 4;
        const bool aff = B.affine != nullptr && B.affine[e0 + e];
        const double* Mi = (aff ? B.mref_inv : B.minv + (size_t)(e0 + e) * Np * Np) + i;
        const double ms = aff ? B.acoef[e0 + e] : 1.0;
        double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
        for (int j = 0; j < Np; ++j) {
          const double m = __ldg(Mi + j * Np);
          double x[4];
          lds16<4>(Bs + (e * Np + j) * 12 + g, x);
#pragma unroll
          for (int k = 0; k < 4; ++k) s[k] += m * x[k];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) s[k] *= ms;
        sts16<4>(sm + L::LF + (e * Np + i) * 12 + g, s);
      }
      for (int t = threadIdx.x; t < (NE - ne) * Np * 12; t += kThreads) sm[L::LF + ne * Np * 12 + t] = 0.0;
      __syncthreads();
    }
    for (int t = threadIdx.x; t < NE * 3; t += kThreads) {
      const int d = t % 3;
      const R n[3] = {(R)(d == 0), (R)(d == 1), (R)(d == 2)};
      R a[NV], F[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) a[v] = (R)anchor[t / 3 * NV + v];
      normal_flux<NV>(D.ph, a, n, F);
#pragma unroll
      for (int v = 0; v < NV; ++v) Fanc[t * NV + v] = F[v];
    }
    __syncthreads();
    // ---- fluxes at the volume points: thread = (point, group of EB elements)
    const R* Bt = static_cast<const R*>(X.Bt);
    for (int t = threadIdx.x; t < NE / EB * Nq; t += kThreads) {
      const int q = t % Nq, g = t / Nq;
      R acc[EB * NV];
#pragma unroll
      for (int k = 0; k < EB * NV; ++k) acc[k] = (R)0;
      double gr[VISC ? 12 : 1], lq[VISC ? 12 : 1];     // reference gradients of v, lift (EB = 1)
      if constexpr (VISC)
#pragma unroll
        for (int k = 0; k < 12; ++k) gr[k] = lq[k] = 0.0;
      const R* Ur = U + g * L::UG;
#pragma unroll 4
      for (int i = 0; i < Np; ++i) {
        const R bq = __ldg(Bt + i * Nq + q);
        R x[EB * NV];
        lds16<EB * NV>(Ur + i * L::UE, x);
#pragma unroll
        for (int k = 0; k < EB * NV; ++k) acc[k] += bq * x[k];
        if constexpr (VISC) {
          const double* gd = B.dBq + (size_t)i * 3 * Nq + q;
          const double d0 = __ldg(gd), d1 = __ldg(gd + Nq), d2 = __ldg(gd + 2 * Nq);
          double v[4], l[12];
          lds16<4>(sm + L::V + (g * Np + i) * 4, v);
          lds16<12>(sm + L::LF + (g * Np + i) * 12, l);
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            gr[m] += d0 * v[m];
            gr[4 + m] += d1 * v[m];
            gr[8 + m] += d2 * v[m];
          }
#pragma unroll
          for (int k = 0; k < 12; ++k) lq[k] += bq * l[k];
        }
      }
      R* Gq = G + g * L::GG + q * L::GQ;
#pragma unroll
      for (int h = 0; h < EB / EB2; ++h) {
        R out[EB2 * 3 * NV];                                         // [r][element][v]
#pragma unroll
        for (int k = 0; k < EB2; ++k) {
          const int el = g * EB + h * EB2 + k;
          const size_t e = (size_t)e0 + (el < ne ? el : 0);
          const bool aff = B.affine != nullptr && B.affine[e];
          const double* Jd = aff ? B.ajinv + e * 9 : B.jinv + e * 9 * Nq + q;
          const int js = aff ? 1 : Nq;
          R J[9];
#pragma unroll
          for (int m = 0; m < 9; ++m) J[m] = (R)Jd[m * js];
          const R wq = aff ? (R)(B.wref[q] * B.adet[e]) : (R)(B.wdet[e * Nq + q] * 1.0);
          R Uq[NV], F[3][NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) Uq[v] = (R)(anchor[el * NV + v] + (double)acc[(h * EB2 + k) * NV + v]);
          const R* Fa = Fanc + el * 3 * NV;
          const R ex[3] = {(R)1, (R)0, (R)0}, ey[3] = {(R)0, (R)1, (R)0}, ez[3] = {(R)0, (R)0, (R)1};
          normal_flux<NV>(D.ph, Uq, ex, F[0]);
          normal_flux<NV>(D.ph, Uq, ey, F[1]);
          normal_flux<NV>(D.ph, Uq, ez, F[2]);
#pragma unroll
          for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int v = 0; v < NV; ++v)
              out[(r * EB2 + k) * NV + v] = (J[r * 3 + 0] * (F[0][v] - Fa[v]) + J[r * 3 + 1] * (F[1][v] - Fa[NV + v]) +
                                             J[r * 3 + 2] * (F[2][v] - Fa[2 * NV + v])) * wq;
        }
        if constexpr (VISC) {
          // minus the viscous flux of the lifted gradients
          const int el = g < ne ? g : 0;
          const size_t e = (size_t)e0 + el;
          const bool aff = B.affine != nullptr && B.affine[e];
          const double* Jd = aff ? B.ajinv + e * 9 : B.jinv + e * 9 * Nq + q;
          const int js = aff ? 1 : Nq;
          double J[9], grad[12], Uq[NV], Fv[3 * NV];
#pragma unroll
          for (int m = 0; m < 9; ++m) J[m] = Jd[m * js];
          const double wq = aff ? B.wref[q] * B.adet[e] : B.wdet[e * Nq + q];
#pragma unroll
          for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int d = 0; d < 3; ++d)
              grad[m * 3 + d] = gr[m] * J[d] + gr[4 + m] * J[3 + d] + gr[8 + m] * J[6 + d] + lq[m * 3 + d];
#pragma unroll
          for (int v = 0; v < NV; ++v) Uq[v] = anchor[g * NV + v] + acc[v];
          const CaseView cv = case_view(D.ph, B.ecase, e);
          viscous_flux<NV>(D.ph, cv.mu, cv.kappa, Uq, grad, Fv);
#pragma unroll
          for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int v = 0; v < NV; ++v)
              out[r * NV + v] -= (J[r * 3] * Fv[v] + J[r * 3 + 1] * Fv[NV + v] + J[r * 3 + 2] * Fv[2 * NV + v]) * wq;
        }
        sts16<EB2 * 3 * NV>(Gq + h * L::GP, out);
      }
    }
    __syncthreads();
    // ---- residual: thread = (IB nodes, chunk of points, EB2 elements); P1 elements keep the chunks
    // in one thread.  At most ROUNDS items per thread, kept in registers until G is dead.
    const R* dBi = static_cast<const R*>(X.dBi);
    constexpr int NI = Np / IB;
    constexpr int items_max = (W::one ? 1 : L::chunk_max) * NI * (NE / EB2);
    constexpr int ROUNDS = (items_max + kThreads - 1) / kThreads;
    const int items = (W::one ? 1 : C) * NI * (NE / EB2);
    R sum[ROUNDS][IB * EB2 * NV];
#pragma unroll
    for (int rd = 0; rd < ROUNDS; ++rd) {
      const int t = rd * kThreads + threadIdx.x;
#pragma unroll
      for (int k = 0; k < IB * EB2 * NV; ++k) sum[rd][k] = (R)0;
      if (t >= items) continue;
      const int i = t % NI * IB, ep = (t / NI) % (NE / EB2), c0 = t / (NI * (NE / EB2));
      const R* Gr = G + (ep * EB2 / EB) * L::GG + (ep % (EB / EB2)) * L::GP;
      const int clo = W::one ? 0 : c0, chi = W::one ? C : c0 + 1;
      for (int c = clo; c < chi; ++c) {
        const int q0 = c * Nq / C, q1 = (c + 1) * Nq / C;
        R s[IB * EB2 * NV];
#pragma unroll
        for (int k = 0; k < IB * EB2 * NV; ++k) s[k] = (R)0;
        // the next point's table values are loaded before this point's products: they come from L2 (a
        // block's dBi is 12 to 192 KB), whose latency the few warps do not cover by themselves
        R g[3 * IB];
        const R* gd = dBi + q0 * 3 * Np + i;
#pragma unroll
        for (int m = 0; m < 3 * IB; ++m) g[m] = __ldg(gd + m / IB * Np + m % IB);
#pragma unroll 1
        for (int q = q0; q < q1; ++q) {
          R gn[3 * IB];
          gd += q + 1 < q1 ? 3 * Np : 0;
#pragma unroll
          for (int m = 0; m < 3 * IB; ++m) gn[m] = __ldg(gd + m / IB * Np + m % IB);
          R x[EB2 * 3 * NV];
          lds16<EB2 * 3 * NV>(Gr + q * L::GQ, x);
#pragma unroll
          for (int n = 0; n < IB; ++n)
#pragma unroll
            for (int k = 0; k < EB2 * NV; ++k) {
              R& acc = s[n * EB2 * NV + k];
              if constexpr (sizeof(R) == sizeof(double)) {
                acc += g[n] * x[k];
                acc += g[IB + n] * x[EB2 * NV + k];
                acc += g[2 * IB + n] * x[2 * EB2 * NV + k];
              } else {
                acc += g[n] * x[k] + g[IB + n] * x[EB2 * NV + k] + g[2 * IB + n] * x[2 * EB2 * NV + k];
              }
            }
#pragma unroll
          for (int m = 0; m < 3 * IB; ++m) g[m] = gn[m];
        }
#pragma unroll
        for (int k = 0; k < IB * EB2 * NV; ++k) sum[rd][k] += s[k];
      }
    }
    __syncthreads();                                                   // G is dead
    R* Pc = sm + L::Gs;                                                // [C][NE][Np][FS]
#pragma unroll
    for (int rd = 0; rd < ROUNDS; ++rd) {
      const int t = rd * kThreads + threadIdx.x;
      if (t >= items) continue;
      const int i = t % NI * IB, ep = (t / NI) % (NE / EB2), c0 = t / (NI * (NE / EB2));
#pragma unroll
      for (int n = 0; n < IB; ++n)
#pragma unroll
        for (int k = 0; k < EB2; ++k)
          sts16<NV>(Pc + ((c0 * NE + ep * EB2 + k) * Np + i + n) * L::FS, &sum[rd][(n * EB2 + k) * NV]);
    }
  } else {
    faces();
    __syncthreads();
  }
  // ---- face terms: the fluxes of the element's face points, then thread = (element, face, face node)
  R* Fl = sm + L::Fl;                                                  // [NE][Nf][FS]
  {
    constexpr int FR = (NE * S::Nf + kThreads - 1) / kThreads;
    double x[FR][NV];
#pragma unroll
    for (int k = 0; k < FR; ++k) {
      const int t = k * kThreads + threadIdx.x, e = t / S::Nf, pt = t % S::Nf;
      if (t >= ne * S::Nf) continue;
      int lf = 0;
#pragma unroll
      for (int m = 1; m < nlf; ++m) lf += pt >= S::poff(m);
      const FaceDev& fd = D.face[lf < S::ntri ? 0 : 1];
      const int nq = S::nq(lf);
      const double* src = fd.fluxI + face_at((size_t)fslot[e * nlf + lf], NV, 0, nq, pt - S::poff(lf));
#pragma unroll
      for (int v = 0; v < NV; ++v) x[k][v] = src[v * nq];
      if constexpr (VISC) {
        const double* vis = fd.fluxV + face_at(fslot[e * nlf + lf] >> 1, NV, 0, nq, pt - S::poff(lf));
#pragma unroll
        for (int v = 0; v < NV; ++v) x[k][v] -= vis[v * nq];
      }
    }
#pragma unroll
    for (int k = 0; k < FR; ++k) {
      const int t = k * kThreads + threadIdx.x;
      if (t >= ne * S::Nf) continue;
      R y[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) y[v] = (R)x[k][v];
      sts16<NV>(Fl + t * L::FS, y);
    }
  }
  __syncthreads();
  R* Fp = sm + L::Fp;                                                  // [NE][Nj][FS]
  // face lf's contribution to its node j: the points in order, then the side's sign
  auto face_sum = [&](int e, int lf, int j, R* s) {
    const int ft = lf < S::ntri ? 0 : 1, nq = S::nq(lf), nfn = S::nfn(lf);
    const R* cB = static_cast<const R*>(X.cB[ft]) + (size_t)fcode[e * nlf + lf] * nq * nfn + j;
    const R* fl = Fl + (e * S::Nf + S::poff(lf)) * L::FS;
#pragma unroll
    for (int v = 0; v < NV; ++v) s[v] = (R)0;
#pragma unroll 4
    for (int q = 0; q < nq; ++q) {
      const R bt = __ldg(cB + q * nfn);
      R x[NV];
      lds16<NV>(fl + q * L::FS, x);
#pragma unroll
      for (int v = 0; v < NV; ++v) s[v] += bt * x[v];
    }
    const R sgn = (fslot[e * nlf + lf] & 1) == 0 ? (R)-1 : (R)1;
#pragma unroll
    for (int v = 0; v < NV; ++v) s[v] = sgn * s[v];
  };
  if constexpr (!W::one) {             // P1 sums a node's faces in the totals pass (three faces a node)
    for (int t = threadIdx.x; t < ne * S::Nj; t += kThreads) {
      const int e = t / S::Nj, jt = t % S::Nj;
      int lf = 0;
#pragma unroll
      for (int m = 1; m < nlf; ++m) lf += jt >= S::joff(m);
      R s[NV];
      face_sum(e, lf, jt - S::joff(lf), s);
      sts16<NV>(Fp + t * L::FS, s);
    }
    __syncthreads();
  }
  // ---- totals: chunk sums, then the faces in local order; thread = (element, node)
  R* Tt = sm + L::Tt;                                                  // [NE][Np][FS]
  {
    const R* Pc = sm + L::Gs;
    const int nc = W::one ? 1 : C;
    for (int t = threadIdx.x; t < ne * Np; t += kThreads) {
      const int e = t / Np, i = t % Np;
      R s[NV];
      if (volume_done) {
        const double* Ri = B.Rinv + ((size_t)(e0 + e) * Np + i) * NV;
#pragma unroll
        for (int v = 0; v < NV; ++v) s[v] = (R)Ri[v];
      } else {
#pragma unroll
        for (int v = 0; v < NV; ++v) s[v] = (R)0;
        for (int c = 0; c < nc; ++c) {
          R x[NV];
          lds16<NV>(Pc + ((c * NE + e) * Np + i) * L::FS, x);
#pragma unroll
          for (int v = 0; v < NV; ++v) s[v] += x[v];
        }
      }
#pragma unroll
      for (int lf = 0; lf < nlf; ++lf) {
        const int j = X.finv[lf < S::ntri ? 0 : 1][fcode[e * nlf + lf] * Np + i];
        if (j < 0) continue;
        R x[NV];
        if constexpr (W::one) face_sum(e, lf, j, x);
        else lds16<NV>(Fp + (e * S::Nj + S::joff(lf) + j) * L::FS, x);
#pragma unroll
        for (int v = 0; v < NV; ++v) s[v] += x[v];
      }
      sts16<NV>(Tt + t * L::FS, s);
    }
  }
  __syncthreads();
  // ---- M^-1 (symmetric: read by columns, one node per lane); the results go over the chunk sums
  R* Rs = sm + (W::one ? L::Fl : L::Gs);                               // [NE][Np][NV]
  for (int t = threadIdx.x; t < ne * Np; t += kThreads) {
    const int e = t / Np, i = t % Np;
    const bool aff = B.affine != nullptr && B.affine[e0 + e];
    const R* Mi = (aff ? static_cast<const R*>(X.mref) : static_cast<const R*>(X.minv) + (size_t)(e0 + e) * Np * Np) + i;
    const R ms = (R)(aff ? B.acoef[e0 + e] : 1.0);
    R r[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] = (R)0;
#pragma unroll 8
    for (int j = 0; j < Np; ++j) {
      const R m = __ldg(Mi + j * Np);
      R x[NV];
      lds16<NV>(Tt + (e * Np + j) * L::FS, x);
#pragma unroll
      for (int v = 0; v < NV; ++v) r[v] += m * x[v];
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) Rs[t * NV + v] = ms * r[v];
  }
  __syncthreads();
  // ---- stage update or outputs, along the elements' contiguous values
  const size_t base = (size_t)e0 * Np * NV;
  const int vals = ne * Np * NV;
  if (!A.stage) {
    for (int t = threadIdx.x; t < vals; t += kThreads) {
      if (A.out_inv[b]) A.out_inv[b][base + t] = (double)Rs[t];
      if (A.out_vis[b]) A.out_vis[b][base + t] = 0.0;
    }
    return;
  }
  double u[VR], w[VR];
#pragma unroll
  for (int k = 0; k < VR; ++k) {
    const int t = k * kThreads + threadIdx.x;
    if (t < vals) {
      u[k] = Ug[t];
      w[k] = A.base[b][base + t];
    }
  }
#pragma unroll
  for (int k = 0; k < VR; ++k) {
    const int t = k * kThreads + threadIdx.x;
    if (t < vals) {
      const double eul = u[k] + A.dt * (double)Rs[t];
      if (A.out_vis[b]) A.out_vis[b][base + t] = 0.0;
      if (A.euler[b]) A.euler[b][base + t] = eul;
      A.dst[b][base + t] = A.alpha * w[k] + A.beta * eul;
    }
  }
}

struct UpdateGrid {
  int cta0[DGB_MAX_BLOCKS + 1];
  bool volume_done[DGB_MAX_BLOCKS];
};

template <int P, int NV, typename R, bool VISC>
__global__ void __launch_bounds__(kThreads, VISC ? 3 : sizeof(R) == sizeof(float) || P == 1 ? 5 : 3)
    k_dense_update(const __grid_constant__ DevPlan D, const StatePtrs St, const __grid_constant__ FinalizeArgs A,
                   const __grid_constant__ DenseTables X, const UpdateGrid L) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  R* sm = reinterpret_cast<R*>(dyn_smem);
  int b = 0;
  while (b + 1 < D.nblocks && (int)blockIdx.x >= L.cta0[b + 1]) ++b;
  const int cta = blockIdx.x - L.cta0[b];
  if (D.blk[b].type == 0) update_body<P, 0, NV, R, VISC>(D, St, A, X.b[b], b, cta, L.volume_done[b], sm);
  else if (D.blk[b].type == 1) update_body<P, 1, NV, R, VISC>(D, St, A, X.b[b], b, cta, L.volume_done[b], sm);
  else update_body<P, 2, NV, R, VISC>(D, St, A, X.b[b], b, cta, L.volume_done[b], sm);
}

// --------------------------------------------------------------------------------------- face kernel
// One face type's CTA: kThreads / nq faces, one thread per face point.  The face's nodes on both
// sides come from the element states into shared memory (minus the side's anchor, node 0).
template <int P, int FT, int NV, typename R, bool VISC>
struct FaceSmem {
  static constexpr int nq = FT == 0 ? Shape<P, 1>::NQT : Shape<P, 1>::NQQ, nfn = FT == 0 ? Shape<P, 1>::TRI : Shape<P, 1>::QUAD;
  static_assert(nfn <= nq, "the local lift has one thread per face node");
  static constexpr int FPC = kThreads / nq, FS = round_up(NV, 16 / (int)sizeof(R));
  static constexpr int NPM = FT == 0 ? Shape<P, 1>::Np : Shape<P, 0>::Np;      // nodes of the largest element with such faces
  // in R: anchors (double), face nodes [FPC][2][nfn][FS]; viscous: all nodes' viscous variables [FPC][2][NPM][4],
  // later the lift's nodal rows b and r [FPC][nfn][12] each, and the jumps [FPC][nq][12]
  static constexpr int AN = round_up(FPC * 2 * NV * (8 / (int)sizeof(R)), 4), N = AN + FPC * 2 * nfn * FS;
  static constexpr int V = N, BB = V, RR = BB + FPC * nfn * 12;
  static constexpr int vis = FPC * 2 * NPM * 4 > FPC * nfn * 24 ? FPC * 2 * NPM * 4 : FPC * nfn * 24;
  static constexpr int J = V + (VISC ? vis : 0), total = J + (VISC ? FPC * nq * 12 : 0);
};

template <int P, int FT, int NV, typename R, bool VISC>
__device__ __forceinline__ void faces_body(const DevPlan& D, const StatePtrs& St, const DenseTables& X, int cta,
                                           bool store_traces, R* smem) {
  using L = FaceSmem<P, FT, NV, R, VISC>;
  constexpr int nq = L::nq, nfn = L::nfn, FPC = L::FPC, FS = L::FS;
  double* anc = reinterpret_cast<double*>(smem);
  R* sm = smem + L::AN;
  const FaceDev& fd = D.face[FT];
  const int f0 = cta * FPC, nf = fd.F - f0 < FPC ? fd.F - f0 : FPC;
  for (int t = threadIdx.x; t < nf * 2 * nfn; t += kThreads) {
    const int j = t % nfn;
    const int3 side = X.side[FT][f0 * 2 + t / nfn];
    const int blk = side.x, code = side.z;
    if (blk < 0) continue;
    const double* u = St.b[blk] + (size_t)side.y * D.blk[blk].Np * NV;
    const double* un = u + (int)X.b[blk].fnode[FT][code * nfn + j] * NV;
    R x[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const double a = u[v];
      if (j == 0) anc[(t / nfn) * NV + v] = a;
      x[v] = (R)(un[v] - a);
    }
    sts16<NV>(sm + t * FS, x);
  }
  if constexpr (VISC) {
    for (int t = threadIdx.x; t < nf * 2 * L::NPM; t += kThreads) {
      const int i = t % L::NPM;
      const int3 side = X.side[FT][f0 * 2 + t / L::NPM];
      if (side.x < 0 || i >= D.blk[side.x].Np) continue;
      const double* un = St.b[side.x] + ((size_t)side.y * D.blk[side.x].Np + i) * NV;
      double u[NV], vv[4];
#pragma unroll
      for (int v = 0; v < NV; ++v) u[v] = un[v];
      viscous_vars<NV>(D.ph, u, vv);
      sts16<4>(smem + L::V + t * 4, vv);
    }
  }
  __syncthreads();
  const int slot = threadIdx.x / nq, q = threadIdx.x % nq;
  const int f = f0 + slot;
  const bool live = slot < nf;
  if (!VISC && !live) return;
  const int nb = live ? fd.nb[f] : -1;
  const size_t so = (size_t)f * 2, sn = so + 1;
  double n[3] = {0.0, 0.0, 0.0}, w = 0.0;
  double UL[NV], UR[NV];
  auto trace = [&](int side, int blk, int code, double* out) {
    const R* cBt = static_cast<const R*>(X.b[blk].cBt[FT]) + (size_t)code * nfn * nq + q;
    const R* row = sm + (slot * 2 + side) * nfn * FS;
    R acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = (R)0;
#pragma unroll
    for (int j = 0; j < nfn; ++j) {
      const R bt = __ldg(cBt + j * nq);
      R x[NV];
      lds16<NV>(row + j * FS, x);
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[v] += bt * x[v];
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) out[v] = anc[(slot * 2 + side) * NV + v] + (double)acc[v];
  };
  if (live) {
    n[0] = fd.n[face_at(f, 3, 0, nq, q)], n[1] = fd.n[face_at(f, 3, 1, nq, q)], n[2] = fd.n[face_at(f, 3, 2, nq, q)];
    w = fd.w[(size_t)f * nq + q];
    double Fh[NV], Fa[NV];
    trace(0, fd.ob[f], fd.oc[f], UL);
    if (nb >= 0) {
      trace(1, nb, fd.nc[f], UR);
    } else if (D.ph.has_boundary) {
      ghost_state<NV>(D.ph, case_view(D.ph, D.blk[fd.ob[f]].ecase, fd.ol[f]).far, UL, n, fd.tag[f], UR);
    } else {
#pragma unroll
      for (int v = 0; v < NV; ++v) UR[v] = UL[v];
    }
    if (store_traces) {
#pragma unroll
      for (int v = 0; v < NV; ++v) fd.trA[face_at(so, NV, v, nq, q)] = UL[v];
      if (nb >= 0)
#pragma unroll
        for (int v = 0; v < NV; ++v) fd.trA[face_at(sn, NV, v, nq, q)] = UR[v];
    }
    hllc<NV>(D.ph, UL, UR, n, Fh);
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      if (side == 1 && nb < 0) break;
      double a[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) a[v] = anc[(slot * 2 + side) * NV + v];
      normal_flux<NV>(D.ph, a, n, Fa);
      double* out = fd.fluxI + face_at(side ? sn : so, NV, 0, nq, q);
#pragma unroll
      for (int v = 0; v < NV; ++v) out[v * nq] = (Fh[v] - Fa[v]) * w;
    }
  }
  if constexpr (VISC) {
    // ---- viscous traces and raw gradients of both sides, the BR2 jump
    double* jmp = smem + L::J;
    double gs[2][12], vt[2][4];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      if (!live || (s == 1 && nb < 0)) continue;
      const int blk = s ? nb : fd.ob[f], code = s ? fd.nc[f] : fd.oc[f];
      const BlockDev& B = D.blk[blk];
      const int Np = B.Np;
      const double* Bt = B.trBt[FT] + (size_t)code * Np * nq + q;
      const double* dBt = B.trdBt[FT] + (size_t)code * Np * 3 * nq + q;
      const double* row = smem + L::V + (slot * 2 + s) * L::NPM * 4;
      double gr[12];
#pragma unroll
      for (int k = 0; k < 12; ++k) gr[k] = 0.0;
#pragma unroll
      for (int m = 0; m < 4; ++m) vt[s][m] = 0.0;
#pragma unroll 4
      for (int i = 0; i < Np; ++i) {
        const double bt = __ldg(Bt + i * nq);
        const double d0 = __ldg(dBt + i * 3 * nq), d1 = __ldg(dBt + (i * 3 + 1) * nq), d2 = __ldg(dBt + (i * 3 + 2) * nq);
        double v[4];
        lds16<4>(row + i * 4, v);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          vt[s][m] += bt * v[m];
          gr[m] += d0 * v[m];
          gr[4 + m] += d1 * v[m];
          gr[8 + m] += d2 * v[m];
        }
      }
      double J[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) J[k] = fd.jinv[face_at(so + s, 9, k, nq, q)];
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int d = 0; d < 3; ++d) gs[s][m * 3 + d] = gr[m] * J[d] + gr[4 + m] * J[3 + d] + gr[8 + m] * J[6 + d];
    }
    const CaseView cv = case_view(D.ph, D.blk[live ? fd.ob[f] : 0].ecase, live ? fd.ol[f] : 0);
    if (live) {
      if (nb < 0) {
        if (D.ph.has_boundary) viscous_ghost<NV>(D.ph, cv.far, cv.wall_T, UL, n, fd.tag[f], vt[1]);
        else viscous_vars<NV>(D.ph, UL, vt[1]);
      }
      double jr[12];
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          jr[m * 3 + d] = 0.5 * w * (vt[1][m] - vt[0][m]) * n[d];
          fd.jumpW[face_at(f, 12, m * 3 + d, nq, q)] = jr[m * 3 + d];
        }
      sts16<12>(jmp + (slot * nq + q) * 12, jr);
    }
    __syncthreads();
    // ---- each side's local lift br2 B_f M^-1 B_f^T jump, over the nodes of the face alone (the basis of the
    // others vanishes there)
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const bool on = live && (s == 0 || nb >= 0);
      double* bb = smem + L::BB + slot * nfn * 12;
      double* rr = smem + L::RR + slot * nfn * 12;
      const int blk = !on ? 0 : s ? nb : fd.ob[f], code = !on ? 0 : s ? fd.nc[f] : fd.oc[f], el = !on ? 0 : s ? fd.nl[f] : fd.ol[f];
      const BlockDev& B = D.blk[blk];
      const DenseBlock& Xb = X.b[blk];
      if (on && q < nfn) {
        const double* cB = static_cast<const double*>(Xb.cB[FT]) + (size_t)code * nq * nfn + q;
        double x[12];
#pragma unroll
        for (int k = 0; k < 12; ++k) x[k] = 0.0;
#pragma unroll 4
        for (int p = 0; p < nq; ++p) {
          const double bt = __ldg(cB + p * nfn);
          double j[12];
          lds16<12>(jmp + (slot * nq + p) * 12, j);
#pragma unroll
          for (int k = 0; k < 12; ++k) x[k] += bt * j[k];
        }
        sts16<12>(bb + q * 12, x);
      }
      __syncthreads();
      if (on && q < nfn) {
        const bool aff = B.affine != nullptr && B.affine[el];
        const int Np = B.Np;
        const uint8_t* fn = Xb.fnode[FT] + code * nfn;
        const double* M = (aff ? B.mref_inv : B.minv + (size_t)el * Np * Np) + fn[q];
        const double ms = D.ph.br2 * (aff ? B.acoef[el] : 1.0);
        double x[12];
#pragma unroll
        for (int k = 0; k < 12; ++k) x[k] = 0.0;
#pragma unroll 4
        for (int p = 0; p < nfn; ++p) {
          const double m = __ldg(M + (int)fn[p] * Np);
          double j[12];
          lds16<12>(bb + p * 12, j);
#pragma unroll
          for (int k = 0; k < 12; ++k) x[k] += m * j[k];
        }
#pragma unroll
        for (int k = 0; k < 12; ++k) x[k] *= ms;
        sts16<12>(rr + q * 12, x);
      }
      __syncthreads();
      if (on) {
        const double* cBt = static_cast<const double*>(Xb.cBt[FT]) + (size_t)code * nfn * nq + q;
#pragma unroll 4
        for (int p = 0; p < nfn; ++p) {
          const double bt = __ldg(cBt + p * nq);
          double j[12];
          lds16<12>(rr + p * 12, j);
#pragma unroll
          for (int k = 0; k < 12; ++k) gs[s][k] += bt * j[k];
        }
      }
    }
    if (!live) return;
    double Fo[3 * NV];
    viscous_flux<NV>(D.ph, cv.mu, cv.kappa, UL, gs[0], Fo);
    if (nb >= 0) {
      double Fn[3 * NV];
      viscous_flux<NV>(D.ph, cv.mu, cv.kappa, UR, gs[1], Fn);
#pragma unroll
      for (int k = 0; k < 3 * NV; ++k) Fo[k] = 0.5 * (Fo[k] + Fn[k]);
    }
    double out[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) out[v] = Fo[v] * n[0] + Fo[NV + v] * n[1] + Fo[2 * NV + v] * n[2];
    if (nb < 0 && D.ph.has_boundary && tag_in(fd.tag[f], D.ph.wall, D.ph.n_wall)) out[4] = 0.0;
#pragma unroll
    for (int v = 0; v < NV; ++v) fd.fluxV[face_at(f, NV, v, nq, q)] = out[v] * w;
  }
}

template <int P, int NV, typename R, bool VISC>
constexpr int faces_smem() {
  constexpr int t = FaceSmem<P, 0, NV, R, VISC>::total, q = FaceSmem<P, 1, NV, R, VISC>::total;
  return t > q ? t : q;
}

template <int P, int NV, typename R, bool VISC>
__global__ void __launch_bounds__(kThreads, VISC ? 3 : 4)
    k_dense_faces(const __grid_constant__ DevPlan D, const StatePtrs St, const __grid_constant__ DenseTables X,
                  int tri_ctas, bool store_traces) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  R* sm = reinterpret_cast<R*>(dyn_smem);
  if ((int)blockIdx.x < tri_ctas) faces_body<P, 0, NV, R, VISC>(D, St, X, blockIdx.x, store_traces, sm);
  else faces_body<P, 1, NV, R, VISC>(D, St, X, blockIdx.x - tri_ctas, store_traces, sm);
}

// -------------------------------------------------------------------------------------------- launch
template <typename K>
cudaError_t allow_smem(K kernel, size_t smem) {
  return smem > 40 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaSuccess;
}

template <int P, int NV, typename R, bool VISC>
cudaError_t launch_faces(const DevPlan& D, const StatePtrs& S, const DenseTables& T, bool store_traces, cudaStream_t st) {
  constexpr int ft = kThreads / Shape<P, 1>::NQT, fq = kThreads / Shape<P, 1>::NQQ;
  constexpr size_t smem = sizeof(R) * (size_t)faces_smem<P, NV, R, VISC>();
  const int tri = (D.face[0].F + ft - 1) / ft, quad = (D.face[1].F + fq - 1) / fq;
  if (tri + quad == 0) return cudaSuccess;
  const cudaError_t e = allow_smem(k_dense_faces<P, NV, R, VISC>, smem);
  if (e != cudaSuccess) return e;
  k_dense_faces<P, NV, R, VISC><<<tri + quad, kThreads, smem, st>>>(D, S, T, tri, store_traces);
  return cudaGetLastError();
}

template <int P, int NV, typename R, bool VISC>
cudaError_t launch_update(const DevPlan& D, const StatePtrs& S, const FinalizeArgs& A, const DenseTables& T,
                          const bool* volume_done, cudaStream_t st) {
  UpdateGrid L;
  L.cta0[0] = 0;
  size_t smem = 0;
  for (int b = 0; b < D.nblocks; ++b) {
    const int type = D.blk[b].type;
    const int ne = type == 0 ? Split<P, 0, VISC>::NE : type == 1 ? Split<P, 1, VISC>::NE : Split<P, 2, VISC>::NE;
    const size_t need = sizeof(R) * (size_t)(type == 0   ? Smem<P, 0, NV, R, VISC>::total
                                             : type == 1 ? Smem<P, 1, NV, R, VISC>::total
                                                         : Smem<P, 2, NV, R, VISC>::total);
    smem = need > smem ? need : smem;
    L.cta0[b + 1] = L.cta0[b] + (D.blk[b].E + ne - 1) / ne;
    L.volume_done[b] = volume_done != nullptr && volume_done[b];
  }
  if (L.cta0[D.nblocks] == 0) return cudaSuccess;
  const cudaError_t e = allow_smem(k_dense_update<P, NV, R, VISC>, smem);
  if (e != cudaSuccess) return e;
  k_dense_update<P, NV, R, VISC><<<L.cta0[D.nblocks], kThreads, smem, st>>>(D, S, A, T, L);
  return cudaGetLastError();
}

template <int P>
DenseShape shape_of(int type) {
  auto make = [](auto s) {
    using S = decltype(s);
    return DenseShape{S::Np, S::Nq, S::nlf, {S::NQT, S::NQQ}, {S::TRI, S::QUAD}};
  };
  return type == 0 ? make(Shape<P, 0>()) : type == 1 ? make(Shape<P, 1>()) : make(Shape<P, 2>());
}

}  // namespace

DenseShape dense_shape(int P, int type) {
  return P == 1 ? shape_of<1>(type) : P == 2 ? shape_of<2>(type) : shape_of<3>(type);
}

// viscous terms: float64 only (the caller keeps the general kernels for mixed plans)
#define DGB_DENSE_DISPATCH(CALL)                                                                                   \
  if (D.nv != 5 || (D.viscous && f32)) return cudaErrorInvalidValue;                                               \
  if (D.viscous) return D.degree == 1 ? CALL(1, 5, double, true) : D.degree == 2 ? CALL(2, 5, double, true) : CALL(3, 5, double, true); \
  if (f32) return D.degree == 1 ? CALL(1, 5, float, false) : D.degree == 2 ? CALL(2, 5, float, false) : CALL(3, 5, float, false); \
  return D.degree == 1 ? CALL(1, 5, double, false) : D.degree == 2 ? CALL(2, 5, double, false) : CALL(3, 5, double, false)

cudaError_t dense_face_flux(const DevPlan& D, const StatePtrs& S, const DenseTables& T, bool f32, bool store_traces,
                            cudaStream_t st) {
#define DGB_CALL(P, NV, R, V) (launch_faces<P, NV, R, V>(D, S, T, store_traces, st))
  DGB_DENSE_DISPATCH(DGB_CALL);
#undef DGB_CALL
}

cudaError_t dense_update(const DevPlan& D, const StatePtrs& S, const FinalizeArgs& A, const DenseTables& T, bool f32,
                         const bool* volume_done, cudaStream_t st) {
#define DGB_CALL(P, NV, R, V) (launch_update<P, NV, R, V>(D, S, A, T, volume_done, st))
  DGB_DENSE_DISPATCH(DGB_CALL);
#undef DGB_CALL
}

}  // namespace dgb
