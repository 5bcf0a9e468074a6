// MOOD subcell finite-volume recompute (float64, any element type).
//
// Reference: hybrid/subcell.py:442-950 and hybrid/limiter.py:267-343.  The reference runs
// the subcell scheme on every element and selects with `where`; here only troubled
// elements (flags from k_troubled on the unlimited candidate) and the parent faces they
// touch do work:
//   k_mood_screen  one thread per parent face: lists the faces with a troubled side, the
//                  troubled elements, and the elements on such faces (troubled or not).
//   k_mood_fv      troubled elements: subcell means (projection), Green-Gauss gradients,
//                  constant/TVD/CWENO-Z face states with admissibility clamps, HLLC on the
//                  internal subfaces, internal residual per subcell (gather, no atomics).
//   k_mood_faces   listed faces, one warp each (mood_face): lanes 0-15 the 16
//                  DG-FV coupling subfaces (FV mean on a troubled side, DG value at the
//                  subface centre otherwise), lanes 16-31 the DG face flux integrated with
//                  the face rule; stores subface fluxes and (new - old) face flux.
//   k_mood_update  listed elements.  Troubled: subface fluxes added in local-face order,
//                  FV update (+ projected viscous rhs), bound-limited reconstruction to DG; others:
//                  the candidate plus the conservative correction from active faces on which they are not
//                  troubled.  In place on the candidate, or out of place over every element.
// The lists hold every block's elements (and both face types), so each kernel is one launch whose CTAs
// take entries in turn.  Before, every kernel was a launch per block with a CTA per element, which on a
// shocked flow of 202,752 hexahedra (1 % of them troubled) left 99 % of the CTAs to start and return:
// 532 us a stage for the three and the flagged elements' viscous pass.  The order of the
// lists changes from run to run; no result depends on it.
#pragma once
#include "aux_kernels.cuh"
#include "dg_kernels.cuh"

namespace dgb {

constexpr int kSub = 16;   // boundary subfaces per parent face at 4 divisions

struct SubcellBlockDev {
  int S, NI, NB;
  const double* P;        // [E][S][Np] projection
  const double* R;        // [E][Np][S] reconstruction
  const double* vol;      // [E][S]
  const double* cen;      // [E][S][3]
  const double* in_n;     // [E][NI][3]
  const double* in_a;     // [E][NI]
  const double* bd_n;     // [E][NB][3]
  const double* bd_a;     // [E][NB]
  const int32_t* iown;    // [NI]
  const int32_t* inbr;    // [NI]
  const int32_t* csr_ptr; // [S+1]
  const int32_t* csr_face;// [2 NI]
  const double* bbasis;   // [NB][Np] basis at the boundary subface centres
  const int32_t* gather;  // [NB] subcell read for a subface
  const int32_t* scatter; // [NB] subcell written for a subface (-1: none)
  double* ubar;           // [E][S][NV] scratch
  double* rsub;           // [E][S][NV] scratch
};

struct SubcellFaceDev {
  const int32_t* osub;    // [F][16] owner boundary subfaces
  const int32_t* nsub;    // [F][16] neighbour boundary subfaces matched to the owner's
  double* fsub;           // [F][16][NV] subface fluxes (times area)
  double* dflux;          // [F][NV]     new - old integrated face flux
  uint8_t* active;        // [F]
};

struct MoodDev {
  SubcellBlockDev blk[DGB_MAX_BLOCKS];
  SubcellFaceDev face[2];
  int recon;              // 0 constant, 1 tvd, 2 weno
};

struct FlagPtrs {
  const uint8_t* f[DGB_MAX_BLOCKS];
};

// Work lists of one recompute.  count: troubled elements, touched elements, active faces; the counts and the
// marks after them are cleared before the faces are screened.
struct MoodLists {
  unsigned* troubled;   // block << 28 | element
  unsigned* touched;    // the same
  unsigned* faces;      // face type << 30 | face
  unsigned* mark[DGB_MAX_BLOCKS];   // [E] 1 once an element is on the touched list
  unsigned* count;
};
enum { kMoodTroubled, kMoodTouched, kMoodFaces, kMoodCounts };

// Appends the lanes with want set to list (one atomic per warp).
__device__ __forceinline__ void append(unsigned* list, unsigned* count, bool want, unsigned entry) {
  const unsigned votes = __ballot_sync(0xffffffffu, want), lane = threadIdx.x & 31;
  if (votes == 0) return;
  unsigned at = 0;
  if (lane == (unsigned)(__ffs(votes) - 1)) at = atomicAdd(count, __popc(votes));
  at = __shfl_sync(0xffffffffu, at, __ffs(votes) - 1);
  if (want) list[at + __popc(votes & ((1u << lane) - 1))] = entry;
}

// Admissibility clamps of reconstructed subcell traces (hybrid/subcell.py:645-663)
template <int NV>
__device__ __forceinline__ void clamp_state(double* U) {
  U[0] = fmax(U[0], 1.0e-14);
  const double ek = 0.5 * (U[1] * U[1] + U[2] * U[2] + U[3] * U[3]) / U[0];
  U[4] = fmax(U[4], ek + 1.0e-12);
#pragma unroll
  for (int v = 5; v < NV; ++v) U[v] = fmax(U[v], 0.0);
}

// --------------------------------------------------------------------------------------------
// One thread per parent face of both types (whole warps).
static __global__ void __launch_bounds__(kThreads) k_mood_screen(const DevPlan P, const MoodDev M, const FlagPtrs Fl,
                                                                const MoodLists L) {
  const int F0 = P.face[0].F, F = F0 + P.face[1].F;
  const int t = blockIdx.x * kThreads + threadIdx.x;
  bool active = false, tr[2] = {false, false}, first[2] = {false, false};
  unsigned entry[2] = {0, 0};
  const int ft = t >= F0 ? 1 : 0, f = t - (ft ? F0 : 0);
  if (t < F) {
    const FaceDev& fd = P.face[ft];
    const int blk[2] = {fd.ob[f], fd.nb[f]}, el[2] = {fd.ol[f], fd.nl[f]};
#pragma unroll
    for (int s = 0; s < 2; ++s)
      if (blk[s] >= 0) {
        tr[s] = Fl.f[blk[s]][el[s]] != 0;
        entry[s] = (unsigned)blk[s] << 28 | (unsigned)el[s];
      }
    active = tr[0] || tr[1];
    M.face[ft].active[f] = active;
    if (active)
#pragma unroll
      for (int s = 0; s < 2; ++s) first[s] = blk[s] >= 0 && atomicExch(&L.mark[blk[s]][el[s]], 1u) == 0u;
  }
  append(L.faces, L.count + kMoodFaces, active, (unsigned)ft << 30 | (unsigned)f);
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    append(L.touched, L.count + kMoodTouched, first[s], entry[s]);
    append(L.troubled, L.count + kMoodTroubled, first[s] && tr[s], entry[s]);
  }
}

// Shared memory of k_mood_fv (doubles): the nodal state, the subcell means, then either the element's projection
// rows or the gradients and both traces of the internal subfaces.
__host__ __device__ inline int mood_fv_smem(int NV, int Np, int S, int NI) {
  const int work = 3 * S * NV + 2 * NI * NV;
  return Np * NV + S * NV + (S * Np > work ? S * Np : work);
}

template <int NV>
__global__ void __launch_bounds__(kThreads) k_mood_fv(const DevPlan P, const MoodDev M, const StatePtrs S,
                                                     const MoodLists L) {
  extern __shared__ double smem[];
  const unsigned n = L.count[kMoodTroubled];
  for (unsigned item = blockIdx.x; item < n; item += gridDim.x) {
    const int b = L.troubled[item] >> 28, e = L.troubled[item] & 0xfffffffu;
    const BlockDev& B = P.blk[b];
    const SubcellBlockDev& C = M.blk[b];
    const int Np = B.Np, Sn = C.S, NI = C.NI;
    double* U = smem;                     // [Np][NV]
    double* ub = U + Np * NV;             // [S][NV]
    double* Pr = ub + Sn * NV;            // [S][Np] projection
    double* g = Pr;                       // [S][3][NV]
    double* tl = g + 3 * Sn * NV;         // [NI][NV] owner-side trace, later the flux
    double* tr = tl + NI * NV;            // [NI][NV] neighbour-side trace
    const double* Ug = S.b[b] + (size_t)e * Np * NV;
    const double* Pe = C.P + (size_t)e * Sn * Np;
    for (int i = threadIdx.x; i < Np * NV; i += kThreads) U[i] = Ug[i];
#pragma unroll 8
    for (int i = threadIdx.x; i < Sn * Np; i += kThreads) Pr[i] = Pe[i];
    __syncthreads();
    for (int idx = threadIdx.x; idx < Sn * NV; idx += kThreads) {
      const int s = idx / NV, v = idx % NV;
      double acc = 0.0;
      for (int i = 0; i < Np; ++i) acc += Pr[s * Np + i] * U[i * NV + v];
      ub[idx] = acc;
      C.ubar[(size_t)e * Sn * NV + idx] = acc;
    }
    __syncthreads();
    const double* nrm = C.in_n + (size_t)e * NI * 3;
    const double* ar = C.in_a + (size_t)e * NI;
    const double* vol = C.vol + (size_t)e * Sn;
    const double* cen = C.cen + (size_t)e * Sn * 3;
    if (M.recon != 0) {
      // Green-Gauss gradient per subcell: sum over its internal subfaces of 0.5 n A (U_nbr - U_own) / V
      for (int idx = threadIdx.x; idx < Sn * 3 * NV; idx += kThreads) {
        const int s = idx / (3 * NV), d = (idx / NV) % 3, v = idx % NV;
        double acc = 0.0;
        for (int k = C.csr_ptr[s]; k < C.csr_ptr[s + 1]; ++k) {
          const int f = C.csr_face[k];
          acc += (0.5 * nrm[f * 3 + d] * ar[f]) * (ub[C.inbr[f] * NV + v] - ub[C.iown[f] * NV + v]);
        }
        g[idx] = acc / fmax(vol[s], 1.0e-14);
      }
      __syncthreads();
    }
    // both traces of every internal subface, one (subface, variable) per thread
    for (int idx = threadIdx.x; idx < NI * NV; idx += kThreads) {
      const int f = idx / NV, v = idx % NV;
      const int o = C.iown[f], nb = C.inbr[f];
      const double uo = ub[o * NV + v], un = ub[nb * NV + v];
      double ul = uo, ur = un;
      if (M.recon != 0) {
        const double dU = un - uo;
        double duo = 0.0, dun = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const double dc = cen[nb * 3 + d] - cen[o * 3 + d];
          duo += g[(o * 3 + d) * NV + v] * dc;
          dun -= g[(nb * 3 + d) * NV + v] * dc;
        }
        if (M.recon == 1) {
          // smooth Venkatakrishnan-type TVD limiter (subcell.py:578-606)
          const double eps = 1.0e-12;
          const double ro = dU / (duo + (duo >= 0.0 ? eps : -eps));
          const double rn = (-dU) / (dun + (dun >= 0.0 ? eps : -eps));
          const double po = ro > 0.0 ? (ro * ro + 2.0 * ro) / (ro * ro + ro + 2.0) : 0.0;
          const double pn = rn > 0.0 ? (rn * rn + 2.0 * rn) / (rn * rn + rn + 2.0) : 0.0;
          ul = uo + 0.5 * fmin(fmax(po, 0.0), 1.0) * duo;
          ur = un + 0.5 * fmin(fmax(pn, 0.0), 1.0) * dun;
        } else {
          // CWENO-Z (subcell.py:608-641)
          const double so = duo, sn = -dun;
          const double ph = 0.5 * (uo + un) + 0.125 * (so - sn);
          const double po = uo + 0.5 * so, pn = un - 0.5 * sn;
          const double es = 1.0e-12;
          const double bh = (sn - so) * (sn - so) + 0.1 * dU * dU;
          const double bo = (dU - so) * (dU - so) + 0.1 * dU * dU;
          const double bn = (dU - sn) * (dU - sn) + 0.1 * dU * dU;
          const double bc = dU * dU;
          const double tau = fabs(bc - bh);
          const double th = tau / (bh + es), to = tau / (bo + es), tn = tau / (bn + es), tc = tau / (bc + es);
          const double a0 = 0.70 * (1.0 + th * th), a1 = 0.28 * (1.0 + to * to), a2 = 0.02 * (1.0 + tc * tc);
          const double sl = a0 + a1 + a2;
          ul = (a0 / sl) * ph + (a1 / sl) * po + (a2 / sl) * uo;
          const double a1r = 0.28 * (1.0 + tn * tn);
          const double sr = a0 + a1r + a2;
          ur = (a0 / sr) * ph + (a1r / sr) * pn + (a2 / sr) * un;
        }
      }
      tl[idx] = ul;
      tr[idx] = ur;
    }
    __syncthreads();
    for (int f = threadIdx.x; f < NI; f += kThreads) {
      double UL[NV], UR[NV], Fl[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        UL[v] = tl[f * NV + v];
        UR[v] = tr[f * NV + v];
      }
      if (M.recon != 0) {
        clamp_state<NV>(UL);
        clamp_state<NV>(UR);
      }
      hllc<NV>(P.ph, UL, UR, nrm + f * 3, Fl);
#pragma unroll
      for (int v = 0; v < NV; ++v) tl[f * NV + v] = Fl[v] * ar[f];
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < Sn * NV; idx += kThreads) {
      const int s = idx / NV, v = idx % NV;
      double acc = 0.0;
      for (int k = C.csr_ptr[s]; k < C.csr_ptr[s + 1]; ++k) {
        const int f = C.csr_face[k];
        acc += C.iown[f] == s ? -tl[f * NV + v] : tl[f * NV + v];
      }
      C.rsub[(size_t)e * Sn * NV + idx] = acc;
    }
    __syncthreads();
  }
}

// --------------------------------------------------------------------------------------------
template <int NV>
__device__ void dg_at_subface(const double* Ue, const double* basis_row, int Np, double* out) {
#pragma unroll
  for (int v = 0; v < NV; ++v) out[v] = 0.0;
  for (int i = 0; i < Np; ++i) {
    const double bi = basis_row[i];
#pragma unroll
    for (int v = 0; v < NV; ++v) out[v] += bi * Ue[i * NV + v];
  }
}

// One parent face with a troubled side, worked by a whole warp (lane: see k_mood_faces).
template <int NV>
__device__ __forceinline__ void mood_face(const DevPlan& P, const MoodDev& M, const StatePtrs& S, int ft, int f,
                                          const FlagPtrs& Fl, int lane) {
  const FaceDev& fd = P.face[ft];
  const SubcellFaceDev& sf = M.face[ft];
  const int ob = fd.ob[f], ol = fd.ol[f], nb = fd.nb[f], nl = fd.nl[f];
  const bool tro = Fl.f[ob][ol] != 0;
  const bool trn = nb >= 0 && Fl.f[nb][nl] != 0;
  double Fv[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) Fv[v] = 0.0;
  if (lane < kSub) {
    const SubcellBlockDev& Co = M.blk[ob];
    const BlockDev& Bo = P.blk[ob];
    const int os = sf.osub[f * kSub + lane];
    double UL[NV], UR[NV];
    if (tro) {
      const double* ub = Co.ubar + ((size_t)ol * Co.S + Co.gather[os]) * NV;
#pragma unroll
      for (int v = 0; v < NV; ++v) UL[v] = ub[v];
    } else {
      dg_at_subface<NV>(S.b[ob] + (size_t)ol * Bo.Np * NV, Co.bbasis + (size_t)os * Bo.Np, Bo.Np, UL);
    }
    const double* n = Co.bd_n + ((size_t)ol * Co.NB + os) * 3;
    const double A = Co.bd_a[(size_t)ol * Co.NB + os];
    if (nb >= 0) {
      const SubcellBlockDev& Cn = M.blk[nb];
      const BlockDev& Bn = P.blk[nb];
      const int ns = sf.nsub[f * kSub + lane];
      if (trn) {
        const double* ub = Cn.ubar + ((size_t)nl * Cn.S + Cn.gather[ns]) * NV;
#pragma unroll
        for (int v = 0; v < NV; ++v) UR[v] = ub[v];
      } else {
        dg_at_subface<NV>(S.b[nb] + (size_t)nl * Bn.Np * NV, Cn.bbasis + (size_t)ns * Bn.Np, Bn.Np, UR);
      }
    } else if (P.ph.has_boundary) {
      ghost_state<NV>(P.ph, case_view(P.ph, P.blk[ob].ecase, ol).far, UL, n, fd.tag[f], UR);
    } else {
#pragma unroll
      for (int v = 0; v < NV; ++v) UR[v] = UL[v];
    }
    clamp_state<NV>(UL);
    clamp_state<NV>(UR);
    double H[NV];
    hllc<NV>(P.ph, UL, UR, n, H);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      Fv[v] = H[v] * A;
      sf.fsub[((size_t)f * kSub + lane) * NV + v] = Fv[v];
    }
  } else {
    // DG face flux at the face rule points, integrated (hybrid/subcell.py:690-746); lanes
    // 16-31 stride over the face points.  It enters (new - old) with a minus sign.
    for (int q = lane - kSub; q < fd.nq; q += 32 - kSub) {
      const int nq = fd.nq;
      const size_t so = (size_t)f * 2, sn = so + 1;
      const double n[3] = {fd.n[face_at(f, 3, 0, nq, q)], fd.n[face_at(f, 3, 1, nq, q)], fd.n[face_at(f, 3, 2, nq, q)]};
      double UL[NV], UR[NV], H[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) UL[v] = fd.trA[face_at(so, NV, v, nq, q)];
      if (nb >= 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) UR[v] = fd.trA[face_at(sn, NV, v, nq, q)];
      } else if (P.ph.has_boundary) {
        ghost_state<NV>(P.ph, case_view(P.ph, P.blk[ob].ecase, ol).far, UL, n, fd.tag[f], UR);
      } else {
#pragma unroll
        for (int v = 0; v < NV; ++v) UR[v] = UL[v];
      }
      clamp_state<NV>(UL);
      clamp_state<NV>(UR);
      hllc<NV>(P.ph, UL, UR, n, H);
      const double w = fd.w[(size_t)f * fd.nq + q];
#pragma unroll
      for (int v = 0; v < NV; ++v) Fv[v] -= H[v] * w;
    }
  }
  // warp sum: lanes 0-15 contribute new subface fluxes, lanes 16.. minus the old flux
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    double x = Fv[v];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffff, x, o);
    if (lane == 0) sf.dflux[(size_t)f * NV + v] = x;
  }
}

// The listed faces, one warp each.
template <int NV>
__global__ void __launch_bounds__(kThreads) k_mood_faces(const DevPlan P, const MoodDev M, const StatePtrs S,
                                                        const FlagPtrs Fl, const MoodLists L) {
  const unsigned n = L.count[kMoodFaces], warps = gridDim.x * (kThreads / 32);
  for (unsigned item = (blockIdx.x * kThreads + threadIdx.x) >> 5; item < n; item += warps)
    mood_face<NV>(P, M, S, L.faces[item] >> 30, (int)(L.faces[item] & 0x3fffffffu), Fl, threadIdx.x & 31);
}

// --------------------------------------------------------------------------------------------
// Shared memory of k_mood_update (doubles): residuals, FV means, the raw reconstruction, then the element's
// projection and later its reconstruction rows.
__host__ __device__ inline int mood_update_smem(int NV, int Np, int S) { return 2 * S * NV + Np * NV + S * Np; }

// out = troubled ? bound-limited reconstruction of the FV update : candidate + corrections.  ALL = false: the touched
// elements, in place (out is the candidate); else every one of the plan's `elements`.  This kernel is the first to
// write out, an element once what it reads of that element has been read, so out may also be the base state or visc.
template <int NV, bool ALL>
__global__ void __launch_bounds__(kThreads) k_mood_update(const DevPlan P, const MoodDev M, const FlagPtrs Fl,
                                                         const StatePtrs visc, double dt, const StatePtrs cand_,
                                                         const StatePtrs out_, const MoodLists L, unsigned elements) {
  extern __shared__ double smem[];
  __shared__ double vtot, corr[DGB_MAX_VARS];
  const unsigned n = ALL ? elements : L.count[kMoodTouched];
  for (unsigned item = blockIdx.x; item < n; item += gridDim.x) {
    int b = 0, e = (int)item;
    if constexpr (ALL)
      for (; e >= P.blk[b].E; ++b) e -= P.blk[b].E;
    else
      b = L.touched[item] >> 28, e = L.touched[item] & 0xfffffffu;
    const BlockDev& B = P.blk[b];
    const SubcellBlockDev& C = M.blk[b];
    const int Np = B.Np, Sn = C.S;
    const size_t base = (size_t)e * Np * NV;
    const double* vol = C.vol + (size_t)e * Sn;
    double* out = out_.b[b];
    const double* cand = ALL ? cand_.b[b] : out;
    if (ALL && !L.mark[b][e]) {
      for (int idx = threadIdx.x; idx < Np * NV; idx += kThreads) out[base + idx] = cand[base + idx];
      continue;
    }
    if (!Fl.f[b][e]) {
      // conservative correction from the active faces, in local-face order
      if (threadIdx.x == 0) {
        double s = 0.0;
        for (int k = 0; k < Sn; ++k) s += vol[k];
        vtot = s;
      }
      __syncthreads();
      if (threadIdx.x < NV) {
        double c = 0.0;
        for (int lf = 0; lf < B.nlf; ++lf) {
          int ft, f, side;
          decode_face(B.elem_face[e * B.nlf + lf], ft, f, side);
          if (!M.face[ft].active[f]) continue;
          const double d = M.face[ft].dflux[(size_t)f * NV + threadIdx.x];
          c += side == 0 ? -dt * d / vtot : dt * d / vtot;
        }
        corr[threadIdx.x] = c;
      }
      __syncthreads();
      for (int idx = threadIdx.x; idx < Np * NV; idx += kThreads) out[base + idx] = cand[base + idx] + corr[idx % NV];
      __syncthreads();
      continue;
    }
    double* res = smem;                    // [S][NV]
    double* fv = res + Sn * NV;            // [S][NV]
    double* raw = fv + Sn * NV;            // [Np][NV]
    double* rows = raw + Np * NV;          // [S][Np] projection, then [Np][S] reconstruction
    const double* vis = visc.b[b];
    for (int idx = threadIdx.x; idx < Sn * NV; idx += kThreads) res[idx] = C.rsub[(size_t)e * Sn * NV + idx];
    if (vis) {
      const double* Pe = C.P + (size_t)e * Sn * Np;
#pragma unroll 8
      for (int i = threadIdx.x; i < Sn * Np; i += kThreads) rows[i] = Pe[i];
      for (int i = threadIdx.x; i < Np * NV; i += kThreads) raw[i] = vis[base + i];
    }
    for (int lf = 0; lf < B.nlf; ++lf) {
      int ft, f, side;
      decode_face(B.elem_face[e * B.nlf + lf], ft, f, side);
      const SubcellFaceDev& sf = M.face[ft];
      const int32_t* sub = side == 0 ? sf.osub : sf.nsub;
      __syncthreads();
      for (int idx = threadIdx.x; idx < kSub * NV; idx += kThreads) {
        const int j = idx / NV, v = idx % NV;
        const int sc = C.scatter[sub[f * kSub + j]];
        if (sc < 0) continue;
        const double h = sf.fsub[((size_t)f * kSub + j) * NV + v];
        res[sc * NV + v] += side == 0 ? -h : h;
      }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < Sn * NV; idx += kThreads) {
      const int s = idx / NV, v = idx % NV;
      double x = C.ubar[(size_t)e * Sn * NV + idx] + dt * res[idx] / vol[s];
      if (vis) {
        double pv = 0.0;
        for (int i = 0; i < Np; ++i) pv += rows[s * Np + i] * raw[i * NV + v];
        x += dt * pv;
      }
      fv[idx] = x;
    }
    __syncthreads();
    const double* Re = C.R + (size_t)e * Np * Sn;
#pragma unroll 8
    for (int i = threadIdx.x; i < Np * Sn; i += kThreads) rows[i] = Re[i];
    __syncthreads();
    for (int idx = threadIdx.x; idx < Np * NV; idx += kThreads) {
      const int i = idx / NV, v = idx % NV;
      double acc = 0.0;
      for (int s = 0; s < Sn; ++s) acc += rows[i * Sn + s] * fv[s * NV + v];
      raw[idx] = acc;
    }
    __syncthreads();
    // Zhang-Shu bound limiting per variable (hybrid/subcell.py:406-439)
    if (threadIdx.x < NV) {
      const int v = threadIdx.x;
      double ms = 0.0, vs = 0.0, smin = INFINITY, smax = -INFINITY, dmin = INFINITY, dmax = -INFINITY;
      for (int s = 0; s < Sn; ++s) {
        ms += fv[s * NV + v] * vol[s];
        vs += vol[s];
        smin = fmin(smin, fv[s * NV + v]);
        smax = fmax(smax, fv[s * NV + v]);
      }
      const double mean = ms / fmax(vs, 1.0e-14);
      for (int i = 0; i < Np; ++i) {
        dmin = fmin(dmin, raw[i * NV + v]);
        dmax = fmax(dmax, raw[i * NV + v]);
      }
      const double eps = 1.0e-12;
      const double tmax = dmax > mean + eps ? (smax - mean) / (dmax - mean + eps) : 1.0;
      const double tmin = dmin < mean - eps ? (mean - smin) / (mean - dmin + eps) : 1.0;
      corr[v] = fmin(fmax(fmin(tmax, tmin), 0.0), 1.0);
      res[v] = mean;                       // res is dead
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < Np * NV; idx += kThreads) {
      const double mean = res[idx % NV];
      out[base + idx] = mean + corr[idx % NV] * (raw[idx] - mean);
    }
    __syncthreads();
  }
}

static __global__ void k_blend(const double* base, const double* x, double alpha, double beta, double* out, size_t n) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] = alpha * base[i] + beta * x[i];
}

}  // namespace dgb
