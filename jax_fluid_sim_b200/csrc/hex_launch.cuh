// Definitions of the launches declared in hex_launch.h (included by the two units that compile them).
#pragma once
#include "hex_launch.h"

namespace dgb {

template <typename K>
cudaError_t allow_smem(K kernel, size_t smem) {
  return smem > 40 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaSuccess;
}

template <int P, int NV, typename R, bool F32>
cudaError_t launch_hex_traces(const DevPlan& D, const StatePtrs& S, const HexTablesT<R>& T, const HexCodes& codes,
                              cudaStream_t st) {
  constexpr size_t smem = sizeof(R) * (size_t)HexSmem<P, NV, R>::TRACES;
  const cudaError_t e = allow_smem(k_hex_traces<P, NV, R, F32>, smem);
  if (e != cudaSuccess || D.blk[0].E == 0) return e;
  k_hex_traces<P, NV, R, F32><<<D.blk[0].E, HexDims<P>::NT, smem, st>>>(D, S, 0, T, codes);
  return cudaGetLastError();
}

template <int P, int NV, typename R, bool F32>
cudaError_t launch_hex_face(const DevPlan& D, const HexTables& T, const HexCodes& codes, const HexFaceArgs& A,
                            cudaStream_t st) {
  constexpr int per = kThreads / HexDims<P>::QF2;
  if (D.face[1].F == 0) return cudaSuccess;
  k_hex_face<P, NV, R, F32><<<(D.face[1].F + per - 1) / per, kThreads, 0, st>>>(D, T, codes, A);
  return cudaGetLastError();
}

template <int P, int NV, bool SPLIT, typename R>
cudaError_t launch_hex_element(const DevPlan& D, const StatePtrs& S, const HexTablesT<R>& T, const HexCodes& codes,
                               const FinalizeArgs& A, cudaStream_t st) {
  constexpr size_t smem = sizeof(R) * (size_t)HexElemSmem<P, NV, SPLIT, R>::TOTAL;
  const cudaError_t e = allow_smem(k_hex_element<P, NV, SPLIT, R>, smem);
  if (e != cudaSuccess || D.blk[0].E == 0) return e;
  k_hex_element<P, NV, SPLIT, R><<<D.blk[0].E, HexDims<P>::NTE, smem, st>>>(D, S, T, codes, A);
  return cudaGetLastError();
}

template <int P, int NV, typename R>
cudaError_t launch_hex_element_list(const DevPlan& D, const StatePtrs& S, const HexTablesT<R>& T, const HexCodes& codes,
                                    const FinalizeArgs& A, const unsigned* list, const unsigned* count, int most,
                                    cudaStream_t st) {
  constexpr size_t smem = sizeof(R) * (size_t)HexElemSmem<P, NV, true, R>::TOTAL;
  const cudaError_t e = allow_smem(k_hex_element_list<P, NV, R>, smem);
  if (e != cudaSuccess || most == 0) return e;
  // about one resident wave
  const int ctas = 148 * 4 * kThreads / HexDims<P>::NTE;
  k_hex_element_list<P, NV, R><<<most < ctas ? most : ctas, HexDims<P>::NTE, smem, st>>>(D, S, T, codes, A, list, count);
  return cudaGetLastError();
}

}  // namespace dgb
