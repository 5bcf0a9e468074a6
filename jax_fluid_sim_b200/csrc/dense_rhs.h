// Right-hand side of the dense blocks in two launches (dense_rhs.cu).
#pragma once
#include <cuda_runtime.h>

#include "dg_kernels.cuh"

namespace dgb {

// What the kernels of one block read besides BlockDev, in the arithmetic type of the plan's
// precision (double, or float in mixed plans; the tables are the double ones rounded once).
struct DenseBlock {
  const void* Bt;            // [Np][Nq]
  const void* dBi;           // [Nq][3][Np]
  const void* minv;          // [E][Np][Np]
  const void* mref;          // [Np][Np] (affine blocks; else null)
  // per face type: the nodes on the face of each trace code, ascending, and the basis at the face
  // points over those nodes alone (the other nodes' values are zero there)
  const uint8_t* fnode[2];   // [codes][nfn]
  const int8_t* finv[2];     // [codes][Np]: position in fnode, -1 off the face
  const void* cB[2];         // [codes][nq][nfn]
  const void* cBt[2];        // [codes][nfn][nq]
  int chunks;                // point chunks of the residual sum (volume_chunks of the block's width)
};

struct DenseTables {
  bool ready;                // every block has the shapes and the face-node structure below
  DenseBlock b[DGB_MAX_BLOCKS];
  const int3* side[2];       // per face type [F][2]: block (-1: none), element, trace code of each side
};

// Expected shapes of a block at degree P: 0 hexahedron, 1 wedge, 2 tetrahedron.
struct DenseShape {
  int Np, Nq, nlf, nq[2], nfn[2];   // [0] triangle, [1] quadrilateral faces
};
DenseShape dense_shape(int P, int type);

// rhs of S with the stage update or outputs of A.  store_traces: also write the face traces (the MOOD
// face kernel and the wall forces read them).  volume_done[b]: block b's volume residual is already in Rinv.
cudaError_t dense_face_flux(const DevPlan& P, const StatePtrs& S, const DenseTables& T, bool f32, bool store_traces,
                            cudaStream_t st);
cudaError_t dense_update(const DevPlan& P, const StatePtrs& S, const FinalizeArgs& A, const DenseTables& T, bool f32,
                         const bool* volume_done, cudaStream_t st);

}  // namespace dgb
