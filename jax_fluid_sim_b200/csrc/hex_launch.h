// Launches of the fused hexahedron kernels (hex_fused.cuh), compiled in hex_rhs_f64.cu and hex_rhs_f32.cu.
#pragma once
#include <cuda_runtime.h>

#include "hex_fused.cuh"

namespace dgb {

// Face traces of every hexahedron; F32: the viscous ones in float32 (mixed-precision plans).
template <int P, int NV, typename R, bool F32>
cudaError_t launch_hex_traces(const DevPlan& D, const StatePtrs& S, const HexTablesT<R>& T, const HexCodes& codes,
                              cudaStream_t st);
template <int P, int NV, typename R, bool F32>
cudaError_t launch_hex_face(const DevPlan& D, const HexTables& T, const HexCodes& codes, const HexFaceArgs& A,
                            cudaStream_t st);
template <int P, int NV, bool SPLIT, typename R>
cudaError_t launch_hex_element(const DevPlan& D, const StatePtrs& S, const HexTablesT<R>& T, const HexCodes& codes,
                               const FinalizeArgs& A, cudaStream_t st);

// The same, split residuals, of the elements list[0 .. *count), at most `most` of them.
template <int P, int NV, typename R>
cudaError_t launch_hex_element_list(const DevPlan& D, const StatePtrs& S, const HexTablesT<R>& T, const HexCodes& codes,
                                    const FinalizeArgs& A, const unsigned* list, const unsigned* count, int most,
                                    cudaStream_t st);

// The launches of one precision, as explicit instantiations (PREFIX: extern, or nothing to define them).
#define DGB_HEX_LAUNCHES_NV(PREFIX, P, NV, R, F32)                                                                    \
  PREFIX template cudaError_t launch_hex_traces<P, NV, R, F32>(const DevPlan&, const StatePtrs&, const HexTablesT<R>&, \
                                                               const HexCodes&, cudaStream_t);                        \
  PREFIX template cudaError_t launch_hex_face<P, NV, R, F32>(const DevPlan&, const HexTables&, const HexCodes&,       \
                                                             const HexFaceArgs&, cudaStream_t);
#define DGB_HEX_LIST(PREFIX, P, NV, R)                                                                              \
  PREFIX template cudaError_t launch_hex_element_list<P, NV, R>(const DevPlan&, const StatePtrs&,                   \
                                                                const HexTablesT<R>&, const HexCodes&,              \
                                                                const FinalizeArgs&, const unsigned*,               \
                                                                const unsigned*, int, cudaStream_t);
#define DGB_HEX_ELEMENT(PREFIX, P, NV, SPLIT, R)                                                                    \
  PREFIX template cudaError_t launch_hex_element<P, NV, SPLIT, R>(const DevPlan&, const StatePtrs&,                 \
                                                                  const HexTablesT<R>&, const HexCodes&,            \
                                                                  const FinalizeArgs&, cudaStream_t);
#define DGB_HEX_DEGREE(PREFIX, P, R)            \
  DGB_HEX_LAUNCHES_NV(PREFIX, P, 5, R, false)   \
  DGB_HEX_LAUNCHES_NV(PREFIX, P, 16, R, false)  \
  DGB_HEX_ELEMENT(PREFIX, P, 5, false, R)       \
  DGB_HEX_ELEMENT(PREFIX, P, 5, true, R)        \
  DGB_HEX_ELEMENT(PREFIX, P, 16, false, R)      \
  DGB_HEX_ELEMENT(PREFIX, P, 16, true, R)       \
  DGB_HEX_LIST(PREFIX, P, 5, R)                 \
  DGB_HEX_LIST(PREFIX, P, 16, R)
#define DGB_HEX_LAUNCHES(PREFIX, R) DGB_HEX_DEGREE(PREFIX, 1, R) DGB_HEX_DEGREE(PREFIX, 2, R) DGB_HEX_DEGREE(PREFIX, 3, R)
#define DGB_HEX_LAUNCHES_F32(PREFIX)             \
  DGB_HEX_LAUNCHES(PREFIX, float)                \
  DGB_HEX_LAUNCHES_NV(PREFIX, 1, 5, float, true) \
  DGB_HEX_LAUNCHES_NV(PREFIX, 1, 16, float, true) \
  DGB_HEX_LAUNCHES_NV(PREFIX, 2, 5, float, true) \
  DGB_HEX_LAUNCHES_NV(PREFIX, 2, 16, float, true) \
  DGB_HEX_LAUNCHES_NV(PREFIX, 3, 5, float, true) \
  DGB_HEX_LAUNCHES_NV(PREFIX, 3, 16, float, true)

}  // namespace dgb
