// Element-local limiter, detector and reduction kernels (float64).
//
//   k_positivity    Zhang-Shu scaling toward the cell mean: density theta in closed form,
//                   pressure theta by 30 bisection steps over node, volume-point and
//                   face-point samples (hybrid/limiter.py:69-147).
//   k_troubled      Persson-type high-mode sensor on (rho, p) plus the MOOD admissibility
//                   test at samples and the mean (hybrid/limiter.py:165-185, 285-300).
//   k_rate          CFL rate per element and, by the last CTA, dt
//                   (hybrid/time_integration.py:93-169).
//   k_adm   finite check and min rho / min p over all nodes
//                   (hybrid/time_integration.py:291-312), combined across stages.
#pragma once
#include "dg_kernels.cuh"

namespace dgb {

struct LimiterConst {
  double density_floor, pressure_floor, relative_floor;   // positivity limiter
  double adm_density_floor, adm_pressure_floor;           // integrator admissibility
  double sensor_threshold;
  double lebesgue;   // max over the limiter's sample points of sum_i |B_i(x)|; 0: no nodal certificate
};

template <int NV>
__device__ __forceinline__ double pressure_of(const Physics& ph, const double* U) {
  const double srho = fmax(U[0], kRhoFloor);
  const double ke = 0.5 * (U[1] * U[1] + U[2] * U[2] + U[3] * U[3]) / srho;
  return (ph.gamma - 1.0) * (U[4] - ke);
}

// Certificate, from the nodal values alone, that density and pressure are admissible at every
// limiter sample of the element and at its cell mean.  A sample u(x) = sum_i B_i(x) U_i, with
// sum_i B_i = 1, obeys |u(x) - c| <= L h, for c and h the midpoint and half-range of the nodal
// values and L the largest sum_i |B_i| over the sample points (their Lebesgue constant).  Intervals of
// rho, m and E then bound rho and p = (gamma - 1)(E - |m|^2 / 2 rho) from below at every sample.
// The cell mean is a positive combination of samples, so its rho lies in the same interval and
// its p is at least the smallest sample p (p is concave in the conserved variables).  The margins
// tol_r and tol_p cover the rounding of the computed samples many times over.  True when
//   rho_lo - tol_r >= max(rho_floor, rel (rho_hi + tol_r)),
//   p_lo - tol_p >= max(p_floor, rel pmean_hi + tol_p),
// with rho_lo >= 1e-3 rho_hi, so that the relative rounding of |m|^2 / rho stays small.
// A non-finite nodal value gives false.  Every thread returns the same value.
// The bound check of the certificate, from the smallest and largest nodal value of rho, m and E.
__device__ __forceinline__ bool certificate_from_range(const double (&mn)[5], const double (&mx)[5],
                                                       const Physics& ph, double L, double rho_floor,
                                                       double p_floor, double rel) {
  if (!(L >= 1.0)) return false;
  double a[5], b[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    const double c = 0.5 * (mn[v] + mx[v]), h = 0.5 * (mx[v] - mn[v]);
    a[v] = c - L * h;
    b[v] = c + L * h;
  }
  const double tol_r = 1.0e-12 * L * fmax(fabs(a[0]), fabs(b[0]));
  if (!(a[0] - tol_r > 0.0) || !(a[0] >= 1.0e-3 * b[0])) return false;
  double m2hi = 0.0, m2lo = 0.0;
#pragma unroll
  for (int d = 1; d <= 3; ++d) {
    m2hi += fmax(a[d] * a[d], b[d] * b[d]);
    m2lo += (a[d] <= 0.0 && b[d] >= 0.0) ? 0.0 : fmin(a[d] * a[d], b[d] * b[d]);
  }
  const double g1 = ph.gamma - 1.0;
  const double ke_hi = 0.5 * m2hi / a[0], ke_lo = 0.5 * m2lo / b[0];
  const double p_lo = g1 * (a[4] - ke_hi), pmean_hi = g1 * (b[4] - ke_lo);
  const double tol_p = 1.0e-6 * g1 * (L * fmax(fabs(a[4]), fabs(b[4])) + ke_hi);
  return (a[0] - tol_r >= fmax(rho_floor, rel * (b[0] + tol_r))) &&
         (p_lo - tol_p >= fmax(p_floor, rel * pmean_hi + tol_p));
}

// Smallest and largest value over the warp of each lane's minima and maxima, in every lane, through the warp's
// integer reduction: a float's or a double's bits, with the lower ones of negative values inverted, order as an
// integer does.  EXACT: the extreme upper half of the doubles, then the extreme lower half of the lanes that have it.
// Else the minima rounded down and the maxima up to float32, half the reductions.
// (Shuffles took 100 of them and 50 float64 comparisons, which bound these kernels.)
template <bool EXACT>
__device__ __forceinline__ void warp_range(double (&mn)[5], double (&mx)[5]) {
  if constexpr (EXACT) {
    auto ordered = [](long long i) { return i ^ ((i >> 63) & 0x7fffffffffffffffLL); };
    auto value = [&](int hi, unsigned lo) { return __longlong_as_double(ordered((long long)hi << 32 | lo)); };
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const long long a = ordered(__double_as_longlong(mn[v])), b = ordered(__double_as_longlong(mx[v]));
      const int ah = __reduce_min_sync(0xffffffff, (int)(a >> 32)), bh = __reduce_max_sync(0xffffffff, (int)(b >> 32));
      const unsigned al = __reduce_min_sync(0xffffffff, (int)(a >> 32) == ah ? (unsigned)a : 0xffffffffu);
      const unsigned bl = __reduce_max_sync(0xffffffff, (int)(b >> 32) == bh ? (unsigned)b : 0u);
      mn[v] = value(ah, al);
      mx[v] = value(bh, bl);
    }
  } else {
    auto ordered = [](int i) { return i ^ ((i >> 31) & 0x7fffffff); };
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const int lo = __reduce_min_sync(0xffffffff, ordered(__float_as_int(__double2float_rd(mn[v]))));
      const int hi = __reduce_max_sync(0xffffffff, ordered(__float_as_int(__double2float_ru(mx[v]))));
      mn[v] = (double)__int_as_float(ordered(lo));
      mx[v] = (double)__int_as_float(ordered(hi));
    }
  }
}

// The nodal values [NP][NV] of one element in a warp's registers: lane l holds nodes l, l + 32.
template <int NV, int NP>
struct WarpNodes {
  static constexpr int K = (NP + 31) / 32;
  double u[K][NV];
  __device__ __forceinline__ void load(const double* Ug) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int l = k * 32 + (threadIdx.x & 31);
      if (l < NP)
#pragma unroll
        for (int v = 0; v < NV; ++v) u[k][v] = Ug[l * NV + v];
    }
  }
  // whether every value is finite and the certificate clears the element, the same in every lane: most elements by
  // their range rounded outward, which contains the exact one and so clears no more than it does; the others by
  // the exact one, from the values in memory (Ug, as loaded or stored by these lanes), so that no register is kept for it
  __device__ __forceinline__ bool certified(const double* Ug, const Physics& ph, double L, double rho_floor, double p_floor,
                                            double rel) const {
    double mn[5], mx[5];
    auto clear = [&]() {
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        mn[v] = INFINITY;
        mx[v] = -INFINITY;
      }
    };
    auto include = [&](int v, double x) {
      mn[v] = fmin(mn[v], x);
      mx[v] = fmax(mx[v], x);
    };
    auto cleared = [&]() -> bool {
      bool ok = false;
      if ((threadIdx.x & 31) == 0) ok = certificate_from_range(mn, mx, ph, L, rho_floor, p_floor, rel);
      return __any_sync(0xffffffff, ok);
    };
    bool fin = true;
    clear();
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (k * 32 + (threadIdx.x & 31) < NP)
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          fin &= isfinite(u[k][v]);
          if (v < 5) include(v, u[k][v]);
        }
    if (!__all_sync(0xffffffff, fin)) return false;
    warp_range<false>(mn, mx);
    if (cleared()) return true;
    clear();
#pragma unroll 1
    for (int l = threadIdx.x & 31; l < NP; l += 32)
#pragma unroll
      for (int v = 0; v < 5; ++v) include(v, Ug[l * NV + v]);
    __syncwarp();
    warp_range<true>(mn, mx);
    return cleared();
  }
};

// The certificate worked by a whole block for one element: each thread takes nodes in a stride,
// warps combine by shuffles and every thread combines the warps.  Every thread returns the same
// value.
template <int NV>
__device__ bool nodal_certificate(const double* __restrict__ Ug, int Np, const Physics& ph, double L,
                                  double rho_floor, double p_floor, double rel) {
  __shared__ double red[10][kThreads / 32];
  double mn[5], mx[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    mn[v] = INFINITY;
    mx[v] = -INFINITY;
  }
  bool fin = true;
  for (int l = threadIdx.x; l < Np; l += blockDim.x) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const double x = Ug[l * NV + v];
      fin &= isfinite(x);
      if (v < 5) {
        mn[v] = fmin(mn[v], x);
        mx[v] = fmax(mx[v], x);
      }
    }
  }
#pragma unroll
  for (int v = 0; v < 5; ++v)
    for (int o = 16; o > 0; o >>= 1) {
      mn[v] = fmin(mn[v], __shfl_xor_sync(0xffffffff, mn[v], o));
      mx[v] = fmax(mx[v], __shfl_xor_sync(0xffffffff, mx[v], o));
    }
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      red[v][threadIdx.x >> 5] = mn[v];
      red[5 + v][threadIdx.x >> 5] = mx[v];
    }
  const bool all_finite = __syncthreads_and(fin);
  if (!all_finite) return false;
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    mn[v] = red[v][0];
    mx[v] = red[5 + v][0];
    for (int k = 1; k < kThreads / 32; ++k) {
      mn[v] = fmin(mn[v], red[v][k]);
      mx[v] = fmax(mx[v], red[5 + v][k]);
    }
  }
  return certificate_from_range(mn, mx, ph, L, rho_floor, p_floor, rel);
}

// Limits of the certificate and the list of the elements that it does not clear.
struct CertifyArgs {
  double L, rho_floor, p_floor, rel;
  int* list;
  int* count;
};

// Certificate pre-pass, one warp per element of NP nodes: elements of block U that the
// certificate does not clear are appended to list (in no fixed order; each is then processed on
// its own, so results do not depend on it).  *count must be zero before the launch.
template <int NV, int NP>
__global__ void __launch_bounds__(kThreads) k_certify(const double* __restrict__ U, int E, const Physics ph,
                                                     const CertifyArgs C) {
  const long long e = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (e >= E) return;
  WarpNodes<NV, NP> x;
  x.load(U + e * NP * NV);
  if (!x.certified(U + e * NP * NV, ph, C.L, C.rho_floor, C.p_floor, C.rel) && (threadIdx.x & 31) == 0)
    C.list[atomicAdd(C.count, 1)] = (int)e;
}

// The SSP-RK stage blend out = alpha * base + beta * x (as k_blend forms it) between its two certificates, one warp
// per element.  LIST = false, every element: x is certified; an element that is not cleared goes to Cx's list and is
// blended after its positivity step, by the second form; a cleared one is blended and the blend certified
// (not cleared: Co's list).  LIST = true: the elements of Cx's list, blended and certified.  x is read once for its
// certificate and the blend: 202k P3 elements, 178 + 340 us as two passes, 265 us as one (memory: 1.55 GB).
// out may be base.
template <int NV, int NP, bool LIST>
__global__ void __launch_bounds__(kThreads) k_blend_certify(const double* base, const double* x, double alpha,
                                                           double beta, double* out, int E, const Physics ph,
                                                           const CertifyArgs Cx, const CertifyArgs Co) {
  const int warps = gridDim.x * (kThreads / 32), lane = threadIdx.x & 31;
  const int n = LIST ? *Cx.count : E;
  for (int item = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); item < n; item += warps) {
    const int e = LIST ? Cx.list[item] : item;
    const size_t o = (size_t)e * NP * NV;
    WarpNodes<NV, NP> u, w;
    u.load(x + o);
    w.load(base + o);
    if (!LIST && !u.certified(x + o, ph, Cx.L, Cx.rho_floor, Cx.p_floor, Cx.rel)) {
      if (lane == 0) Cx.list[atomicAdd(Cx.count, 1)] = e;
      continue;
    }
#pragma unroll
    for (int k = 0; k < WarpNodes<NV, NP>::K; ++k) {
      const int l = k * 32 + lane;
      if (l < NP)
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          u.u[k][v] = alpha * w.u[k][v] + beta * u.u[k][v];
          out[o + l * NV + v] = u.u[k][v];
        }
    }
    if (!u.certified(out + o, ph, Co.L, Co.rho_floor, Co.p_floor, Co.rel) && lane == 0) Co.list[atomicAdd(Co.count, 1)] = e;
  }
}

// BlockDev::elem_code from the faces' records (set-up).
static __global__ void k_elem_codes(const DevPlan P, int b, uint8_t* __restrict__ out) {
  const BlockDev& B = P.blk[b];
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)B.E * B.nlf) return;
  int ft, f, side;
  decode_face(B.elem_face[t], ft, f, side);
  out[t] = (uint8_t)(side == 0 ? P.face[ft].oc[f] : P.face[ft].nc[f]);
}

// samples = [U at nodes; B U at volume points; Bfs U at face points]  -> S[Ns_total][NV]
template <int NV>
__device__ void build_samples(const BlockDev& B, const double* U, double* S) {
  const int Np = B.Np, Nq = B.Nq, Ns = B.Ns;
  const int total = (Np + Nq + Ns) * NV;
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int r = idx / NV, v = idx % NV;
    double val;
    if (r < Np) {
      val = U[r * NV + v];
    } else {
      const double* row = r < Np + Nq ? B.B + (size_t)(r - Np) * Np : B.fsB + (size_t)(r - Np - Nq) * Np;
      double s = 0.0;
      for (int i = 0; i < Np; ++i) s += row[i] * U[i * NV + v];
      val = s;
    }
    S[idx] = val;
  }
}

// Cell mean: sum_q wdet (B U) / sum_q wdet, from the volume samples [q][v], worked by all threads
// (a strided sum per thread, shuffles per warp, the warps added in order by thread 0); ends with
// the block synchronised and mean[] set.
template <int NV>
__device__ void cell_mean(const BlockDev& B, int e, const double* Svol, double* mean) {
  __shared__ double part[kThreads / 32][NV + 1];
  const double* wdet = B.wdet + (size_t)e * B.Nq;
  double s[NV + 1];
#pragma unroll
  for (int v = 0; v <= NV; ++v) s[v] = 0.0;
  for (int q = threadIdx.x; q < B.Nq; q += blockDim.x) {
    const double w = wdet[q];
#pragma unroll
    for (int v = 0; v < NV; ++v) s[v] += Svol[q * NV + v] * w;
    s[NV] += w;
  }
#pragma unroll
  for (int v = 0; v <= NV; ++v)
    for (int o = 16; o > 0; o >>= 1) s[v] += __shfl_xor_sync(0xffffffff, s[v], o);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int v = 0; v <= NV; ++v) part[threadIdx.x >> 5][v] = s[v];
  __syncthreads();
  if (threadIdx.x < NV) {
    double a = 0.0, w = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      a += part[k][threadIdx.x];
      w += part[k][NV];
    }
    mean[threadIdx.x] = a / w;
  }
  __syncthreads();
}

template <int NV>
__global__ void __launch_bounds__(kThreads) k_positivity(const DevPlan P, const StatePtrs S, int b,
                                                        const LimiterConst L) {
  extern __shared__ double smem[];
  __shared__ double mean[NV];
  __shared__ double sh_theta_rho;
  const BlockDev& B = P.blk[b];
  const int e = blockIdx.x;
  const int Np = B.Np, Nq = B.Nq;
  const int Nt = Np + Nq + B.Ns;
  double* U = smem;
  double* Smp = U + Np * NV;
  double* Ug = S.b[b] + (size_t)e * Np * NV;
  // nodal certificate of theta = 1: the state stays as it is (mean + 1 * (U - mean) is U to rounding)
  if (nodal_certificate<NV>(Ug, Np, P.ph, B.lebesgue, L.density_floor, L.pressure_floor, L.relative_floor)) return;
  for (int i = threadIdx.x; i < Np * NV; i += blockDim.x) U[i] = Ug[i];
  __syncthreads();
  build_samples<NV>(B, U, Smp);
  __syncthreads();
  cell_mean<NV>(B, e, Smp + Np * NV, mean);
  __syncthreads();
  double Wm[NV];
  primitive<NV>(P.ph, mean, Wm);
  const double rfloor = fmax(L.density_floor, L.relative_floor * Wm[0]);
  const double pfloor = fmax(L.pressure_floor, L.relative_floor * Wm[4]);
  // minimum sampled density
  double rmin = INFINITY;
  bool nan_seen = false;
  for (int r = threadIdx.x; r < Nt; r += blockDim.x) {
    const double d = Smp[r * NV];
    nan_seen |= isnan(d);
    rmin = fmin(rmin, d);
  }
  // block min (NaN propagates like a jnp.min)
  __shared__ double red[kThreads / 32];
  __shared__ int red_nan;
  if (threadIdx.x == 0) red_nan = 0;
  for (int o = 16; o > 0; o >>= 1) rmin = fmin(rmin, __shfl_xor_sync(0xffffffff, rmin, o));
  __syncthreads();
  if (nan_seen) atomicOr(&red_nan, 1);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = rmin;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = red[0];
    for (int k = 1; k < kThreads / 32; ++k) m = fmin(m, red[k]);
    if (red_nan) m = NAN;
    const double denom = mean[0] - m;
    const double th = (m < rfloor) ? (mean[0] - rfloor) / fmax(denom, 1.0e-30) : 1.0;
    // jnp.clip(x, 0, 1) keeps NaN as NaN
    sh_theta_rho = isnan(th) ? th : fmin(fmax(th, 0.0), 1.0);
  }
  __syncthreads();
  const double upper = sh_theta_rho;
  // pressure admissibility of mean + theta*(sample - mean) at every sample
  auto pressure_ok = [&](double theta) -> bool {
    bool ok = true;
    for (int r = threadIdx.x; r < Nt; r += blockDim.x) {
      double s[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) s[v] = mean[v] + theta * (Smp[r * NV + v] - mean[v]);
      ok &= (pressure_of<NV>(P.ph, s) >= pfloor);
    }
    return __syncthreads_and(ok);
  };
  // theta = upper when the pressure is admissible there; only otherwise is the reference's
  // 30-step bisection result used, so it is computed only in that case (same theta)
  double theta = upper;
  if (!pressure_ok(upper)) {
    double lo = 0.0, hi = upper;
    for (int it = 0; it < 30; ++it) {
      const double mid = 0.5 * (lo + hi);
      const bool ok = pressure_ok(mid);
      lo = ok ? mid : lo;
      hi = ok ? hi : mid;
    }
    theta = lo;
  }
  for (int idx = threadIdx.x; idx < Np * NV; idx += blockDim.x) {
    const int v = idx % NV;
    Ug[idx] = mean[v] + theta * (U[idx] - mean[v]);
  }
}

// Learned-predictor hooks of the troubled-cell kernels.  mode 1 (learned): an element whose
// predicted flag is set goes to the subcell scheme without the a-posteriori test; mode 2
// (evaluate): every element is tested and the flag is the test's, the prediction is only
// counted.  counts: [1] predicted, [2] missed (tested troubled, not predicted),
// [3] false positive and [4] hit (mode 2 only).
struct PredictArgs {
  const uint8_t* pred;
  int mode;
  unsigned long long* counts;
};

__device__ __forceinline__ bool predicted_skip(const PredictArgs& pa, int e, uint8_t* flag_out) {
  if (pa.mode != 1 || !pa.pred || !pa.pred[e]) return false;
  if (threadIdx.x == 0) {
    if (flag_out) flag_out[e] = 1;
    if (pa.counts) atomicAdd(pa.counts + 1, 1ULL);
  }
  return true;
}

__device__ __forceinline__ void count_prediction(const PredictArgs& pa, int e, bool detected) {
  if (!pa.counts || !pa.pred || pa.mode == 0) return;
  const bool pr = pa.pred[e] != 0;
  if (pa.mode == 2 && pr) atomicAdd(pa.counts + 1, 1ULL);
  if (detected && !pr) atomicAdd(pa.counts + 2, 1ULL);
  if (pa.mode == 2 && pr && !detected) atomicAdd(pa.counts + 3, 1ULL);
  if (pa.mode == 2 && pr && detected) atomicAdd(pa.counts + 4, 1ULL);
}

template <int NV>
__global__ void __launch_bounds__(kThreads) k_troubled(const DevPlan P, const StatePtrs S, int b, const LimiterConst L,
                                                      double* sensor_out, uint8_t* flag_out, const PredictArgs pa) {
  extern __shared__ double smem[];
  __shared__ double mean[NV];
  __shared__ double red[4][kThreads / 32];
  const BlockDev& B = P.blk[b];
  const int e = blockIdx.x;
  if (predicted_skip(pa, e, flag_out)) return;
  const int Np = B.Np, Nq = B.Nq;
  const int Nt = Np + Nq + B.Ns;
  double* U = smem;
  double* Smp = U + Np * NV;
  double* Mon = Smp + Nt * NV;   // [Np][2] monitored (rho, p)
  const double* Ug = S.b[b] + (size_t)e * Np * NV;
  // nodal certificate of admissible samples and mean: then only the sensor needs computing
  const bool certified = nodal_certificate<NV>(Ug, Np, P.ph, B.lebesgue, L.density_floor, L.pressure_floor, 0.0);
  for (int i = threadIdx.x; i < Np * NV; i += blockDim.x) U[i] = Ug[i];
  __syncthreads();
  if (!certified) build_samples<NV>(B, U, Smp);
  for (int i = threadIdx.x; i < Np; i += blockDim.x) {
    double W[NV];
    primitive<NV>(P.ph, U + i * NV, W);
    Mon[i * 2 + 0] = W[0];
    Mon[i * 2 + 1] = W[4];
  }
  __syncthreads();
  if (!certified) cell_mean<NV>(B, e, Smp + Np * NV, mean);
  // sensor: sum_i (m - Pi m)^2 / max(sum_i m^2, 1e-12), max over (rho, p)
  double hi0 = 0.0, hi1 = 0.0, sc0 = 0.0, sc1 = 0.0;
  if (P.degree >= 2) {
    for (int i = threadIdx.x; i < Np; i += blockDim.x) {
      double l0 = 0.0, l1 = 0.0;
      for (int j = 0; j < Np; ++j) {
        l0 += B.p1proj[(size_t)i * Np + j] * Mon[j * 2 + 0];
        l1 += B.p1proj[(size_t)i * Np + j] * Mon[j * 2 + 1];
      }
      const double d0 = Mon[i * 2 + 0] - l0, d1 = Mon[i * 2 + 1] - l1;
      hi0 += d0 * d0;
      hi1 += d1 * d1;
      sc0 += Mon[i * 2 + 0] * Mon[i * 2 + 0];
      sc1 += Mon[i * 2 + 1] * Mon[i * 2 + 1];
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    hi0 += __shfl_xor_sync(0xffffffff, hi0, o);
    hi1 += __shfl_xor_sync(0xffffffff, hi1, o);
    sc0 += __shfl_xor_sync(0xffffffff, sc0, o);
    sc1 += __shfl_xor_sync(0xffffffff, sc1, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = hi0;
    red[1][threadIdx.x >> 5] = hi1;
    red[2][threadIdx.x >> 5] = sc0;
    red[3][threadIdx.x >> 5] = sc1;
  }
  __syncthreads();
  // invalid samples (including the cell mean)
  bool bad = false;
  for (int r = threadIdx.x; r <= (certified ? -1 : Nt); r += blockDim.x) {
    const double* s = r < Nt ? Smp + r * NV : mean;
    double W[NV];
    primitive<NV>(P.ph, s, W);
    bool finite = true;
#pragma unroll
    for (int v = 0; v < NV; ++v) finite &= isfinite(W[v]);
    bad |= !finite || (W[0] < L.density_floor) || (W[4] < L.pressure_floor);
  }
  const bool any_bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    double h0 = 0, h1 = 0, s0 = 0, s1 = 0;
    for (int k = 0; k < kThreads / 32; ++k) {
      h0 += red[0][k]; h1 += red[1][k]; s0 += red[2][k]; s1 += red[3][k];
    }
    double value = 0.0;
    if (P.degree >= 2) {
      const double r0 = h0 / fmax(s0, 1.0e-12), r1 = h1 / fmax(s1, 1.0e-12);
      value = (isnan(r0) || isnan(r1)) ? NAN : fmax(r0, r1);
    }
    const bool detected = (value > L.sensor_threshold) || any_bad;
    if (sensor_out) sensor_out[e] = value;
    if (flag_out) flag_out[e] = (uint8_t)detected;
    count_prediction(pa, e, detected);
  }
}

// ---------------------------------------------------------------- reductions
struct Partial {
  double a, b;   // (max rate) or (rho_min, p_min)
  int flag;      // finite / nan seen
  int pad;
};

// The reductions over the whole state are one launch over all blocks: CTAs [cta0[b], cta0[b + 1]) take block b,
// every CTA leaves a partial, and the one that finishes last (by the ticket counter, which wraps to zero for
// the next launch) reduces them.  A launch per block and one for the final reduction cost about 5 us each
// on states of any size that stays in L2, a tenth of a small step.
// Each kind of reduction has partials and a counter of its own, and its CTAs are the same number in every launch
// of the plan: whatever launches overlap (calls of one plan on two streams, which may spoil one another's result
// as they always could), each adds `ctas` to a counter that wraps at `ctas`, so it ends at zero and later
// results are right.
struct Reduction {
  int cta0[DGB_MAX_BLOCKS + 1];
  int ctas;                // launched: cta0[nblocks], at least one
  Partial* partials;       // [ctas]
  unsigned* ticket;
};

__device__ __forceinline__ int reduce_block(const Reduction& G, int nblocks) {
  int b = 0;
  while (b + 1 < nblocks && (int)blockIdx.x >= G.cta0[b + 1]) ++b;
  return b;
}

// Thread 0 has written the CTA's partial: true in every thread of the CTA that is the last to do so.
__device__ __forceinline__ bool last_cta(unsigned* ticket) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  return last;
}

// max over elements of the reference's rate, then dt = clip(cfl / max)
template <int NV>
__global__ void __launch_bounds__(kThreads) k_rate(const DevPlan P, const StatePtrs S, const Reduction G, double cp,
                                                  double cfl, double* dt_out) {
  // one warp per element; grid-stride over the block's elements
  const int b = reduce_block(G, P.nblocks);
  const BlockDev& B = P.blk[b];
  const int lane = threadIdx.x & 31;
  const int warp = ((blockIdx.x - G.cta0[b]) * kThreads + threadIdx.x) >> 5;
  const int nwarps = ((G.cta0[b + 1] - G.cta0[b]) * kThreads) >> 5;
  const double df = 2.0 * P.degree + 1.0;
  double best = -INFINITY;
  for (int e = warp; e < B.E; e += nwarps) {
    const double* U = S.b[b] + (size_t)e * B.Np * NV;
    double smax = -INFINITY, rsum = 0.0;
    bool en = false;
    for (int i = lane; i < B.Np; i += 32) {
      double W[NV];
      primitive<NV>(P.ph, U + i * NV, W);
      // jnp.maximum propagates NaN where fmax drops it: a NaN density or pressure makes the
      // reference's rate NaN (then 1e7), so it is flagged before the floors
      const double rho = fmax(W[0], 1.0e-14), p = fmax(W[4], 1.0e-14);
      const double sp = sqrt(W[1] * W[1] + W[2] * W[2] + W[3] * W[3]) + sqrt(P.ph.gamma * p / rho);
      en |= isnan(W[0]) || isnan(W[4]) || isnan(sp);
      smax = fmax(smax, sp);
      rsum += rho;
    }
    for (int o = 16; o > 0; o >>= 1) {
      smax = fmax(smax, __shfl_xor_sync(0xffffffff, smax, o));
      rsum += __shfl_xor_sync(0xffffffff, rsum, o);
    }
    en = __any_sync(0xffffffff, en);
    const double h = B.length[e];
    double rate = en ? NAN : df * smax / h;
    if (P.viscous) {
      const double rmin = fmax(rsum / B.Np, 0.1);
      const CaseView cv = case_view(P.ph, B.ecase, e);
      const double diff = fmax((4.0 / 3.0) * cv.mu / rmin, cv.kappa / (rmin * cp));
      const double vl = fmax(h, 0.01);
      rate = rate + 2.0 * P.ph.br2 * df * df * diff / (vl * vl);
    }
    // jnp.nan_to_num(rate, nan=1e7, posinf=1e7)
    if (isnan(rate) || (isinf(rate) && rate > 0.0)) rate = 1.0e7;
    else if (isinf(rate)) rate = -1.7976931348623157e308;
    best = fmax(best, rate);
  }
  __shared__ double red[kThreads / 32];
  if (lane == 0) red[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = red[0];
    for (int k = 1; k < kThreads / 32; ++k) m = fmax(m, red[k]);
    __stcg(&G.partials[blockIdx.x].a, m);
  }
  if (!last_cta(G.ticket)) return;
  double m = -INFINITY;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += kThreads) m = fmax(m, __ldcg(&G.partials[i].a));
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffff, m, o));
  if (lane == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 0; k < kThreads / 32; ++k) m = fmax(m, red[k]);
    const double dt = cfl / fmax(m, 1.0e-12);
    *dt_out = fmin(fmax(dt, 1.0e-7), 1.0e-3);
  }
}

template <int NV>
__global__ void __launch_bounds__(kThreads) k_adm(const DevPlan P, const StatePtrs S, const Reduction G, double rho_floor,
                                                 double p_floor, int combine, dgb_status* status) {
  const int b = reduce_block(G, P.nblocks);
  const BlockDev& B = P.blk[b];
  const size_t nodes = (size_t)B.E * B.Np;
  double rmin = INFINITY, pmin = INFINITY;
  int finite = 1, rnan = 0, pnan = 0;
  const size_t stride = (size_t)(G.cta0[b + 1] - G.cta0[b]) * kThreads;
  for (size_t k = (blockIdx.x - G.cta0[b]) * (size_t)kThreads + threadIdx.x; k < nodes; k += stride) {
    const double* U = S.b[b] + k * NV;
#pragma unroll
    for (int v = 0; v < NV; ++v) finite &= isfinite(U[v]) ? 1 : 0;
    const double p = pressure_of<NV>(P.ph, U);
    rnan |= isnan(U[0]);
    pnan |= isnan(p);
    rmin = fmin(rmin, U[0]);
    pmin = fmin(pmin, p);
  }
  // (rho_min, p_min, finite) over the CTA; fmin drops a NaN where the reference keeps it
  __shared__ double r1[kThreads / 32], r2[kThreads / 32];
  auto reduce = [&]() {
    for (int o = 16; o > 0; o >>= 1) {
      rmin = fmin(rmin, __shfl_xor_sync(0xffffffff, rmin, o));
      pmin = fmin(pmin, __shfl_xor_sync(0xffffffff, pmin, o));
    }
    finite = __syncthreads_and(finite);
    rnan = __syncthreads_or(rnan);
    pnan = __syncthreads_or(pnan);
    if ((threadIdx.x & 31) == 0) {
      r1[threadIdx.x >> 5] = rmin;
      r2[threadIdx.x >> 5] = pmin;
    }
    __syncthreads();
    for (int k = 0; k < kThreads / 32; ++k) {
      rmin = fmin(rmin, r1[k]);
      pmin = fmin(pmin, r2[k]);
    }
    rmin = rnan ? NAN : rmin;
    pmin = pnan ? NAN : pmin;
  };
  reduce();
  if (threadIdx.x == 0) {
    __stcg(&G.partials[blockIdx.x].a, rmin);
    __stcg(&G.partials[blockIdx.x].b, pmin);
    __stcg(&G.partials[blockIdx.x].flag, finite);
  }
  if (!last_cta(G.ticket)) return;
  rmin = pmin = INFINITY;
  finite = 1, rnan = pnan = 0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += kThreads) {
    const double a = __ldcg(&G.partials[i].a), c = __ldcg(&G.partials[i].b);
    rnan |= isnan(a);
    pnan |= isnan(c);
    rmin = fmin(rmin, a);
    pmin = fmin(pmin, c);
    finite &= __ldcg(&G.partials[i].flag);
  }
  reduce();
  if (threadIdx.x != 0) return;
  const int valid = finite && (rmin >= rho_floor) && (pmin >= p_floor);
  // combine: the first stage overwrites the status, later stages AND / min into it
  if (combine) {
    status->valid = status->valid && valid;
    status->rho_min = (isnan(status->rho_min) || isnan(rmin)) ? NAN : fmin(status->rho_min, rmin);
    status->p_min = (isnan(status->p_min) || isnan(pmin)) ? NAN : fmin(status->p_min, pmin);
  } else {
    status->valid = valid;
    status->rho_min = rmin;
    status->p_min = pmin;
  }
}

}  // namespace dgb
