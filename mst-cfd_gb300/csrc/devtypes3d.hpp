// Device-side views of the 3D residual path (kernels3d.inc).
#pragma once
#include <cuda_runtime.h>

#include "devtypes.hpp"

namespace mst {

// Gradient record per cell: [3][5] plus one pad, so that a cell's gradient
// is 64 B (FP32) or 128 B (FP64), loaded and stored as aligned vectors.
constexpr int kGrad3 = 16;
constexpr int kNoFace3 = 0x7fffffff;

// 3D mesh in device order (mesh3d.hpp DevLayout3D): FP64 vectors of 3
// packed (x, y, z) per face or cell-face (FP64 paths), FP32 tables (FP32 path)
struct DevMesh3 {
  int n_cells, n_faces;
  bool in_turn;  // every launch after the end of the one before
  const int2* f_c0c1;
  const int* f_info;
  const double *f_dir, *f_r0, *f_r1, *f_eta;
  // FP32 copies packed for one 16-byte load each: (S, eta0), (r0, 0), (r1, 0)
  // and (r0 - r1, 0)
  const float4 *f_dir_eta32, *f_r0_32, *f_r1_32, *f_d32;
  const double* c_vol;
  const double* c_ivol;     // 1/V
  const float2* c_ivol_ff;  // 1/V as a float pair
  const int* c_ptr;
  const int* cf_face;       // device face, ~face where the cell is its c1
  const int* cf_nb;         // neighbour device cell, -1 on boundary faces
  const double* cf_w;       // [tot][2] face-value weights (self, neighbour)
  const double* cf_dir;     // [tot][3] outward area vector
  // FP32 path: the cell-face tables by face position, [e_deg][n_cells]: the
  // neighbour (boundary and absent faces: the cell itself), (outward S, self
  // weight), the neighbour weight (boundary 1 and 0, absent all zero), the
  // device face as cf_face (absent: kNoFace3).  A warp's loads are contiguous.
  int e_deg;
  const int* e_nb;
  const float4* e_dw;
  const float* e_w1;
  const int* e_face;
};

// One stage of the 3D path.  FP64 state: q [nC][5].  FP32 path: the state
// as float pairs, hi parts (h4 = rho, rho u, rho v, rho w; h1 = E) and lo
// parts (l4, l1).
struct Step3Args {
  const double* q;        // state the residual is evaluated on (FP64)
  double* qn;             // updated state (FP64)
  const double* q0;       // Q^n for the second RK stage (FP64)
  const float4* h4;
  const float* h1;
  const float4* l4;
  const float* l1;
  float4* nh4;
  float* nh1;
  float4* nl4;
  float* nl1;
  const float4* ph4;      // Q^n hi / lo for the second stage
  const float* ph1;
  const float4* pl4;
  const float* pl1;
  const void* grad;       // [nC][kGrad3] in the path's precision ([3][5] + pad)
  double* r_out;          // [nC][5] residual (residual-only launches)
  double* fx;             // FP64 paths: face-flux buffer, [nF][6] (production:
                          // projected on the area vector) or [nF][16] (exact)
  float4* fx4;            // FP32 path: the projected flux, components 0-3
  float* fx1;             // and 4
  const double* scal;     // device [0] = dt (FP64 paths)
  const float* dt_ff;     // device dt as a float pair (FP32 path)
  int stage;              // 0: Q - dt/V R;  1: 0.5 Q0 + 0.5 (Q - dt/V R)
  int limiter;
  double mu, lam, kappa, cv;
  float mu_f, lam_f, kappa_f, cv_f;
  double inlet[5];
  float inlet_f[5];
};

}  // namespace mst
