// Element buffers and their gather (gather.cu).
#pragma once
#include "common.cuh"

namespace igap {

constexpr int NPAIRS = NB * (NB + 1) / 2;  // 378 basis pairs b <= c
constexpr int EBUF = NPAIRS * 9;           // doubles of one element's matrix: 3 x 3 blocks [pair][d][e]

// Number of pair (b, c), b <= c, row by row.
__host__ __device__ constexpr int pair_index(int b, int c) { return b * NB - b * (b - 1) / 2 + c - b; }

struct GatherMap {
  DevMesh m;
  const int64_t *rowptr;
  int64_t ndof;
  // batches: mesh and first element of every instance, instance of every control point
  const DevMesh *meshes;
  const int64_t *eoff;
  const int *cpinst;
  // Dirichlet DOFs (or null): index + 1 in the list of prescribed values, 0 otherwise; the state
  const int *dir;
  const double *dir_g, *U;
  int parts;       // partial sums per element residual, [element][part][81]
  const int *err;  // error word of the element kernel: NaN is written when it is set (or null)
};

// Buffers of the context ([element][EBUF], [element][NE]); false: not available.
bool ensure_ebuf(Context *c);
bool ensure_fbuf(Context *c);  // FP32 [element][27][243]
bool ensure_rbuf(Context *c);  // FP64 [element][res_parts][81]
// blocks per element of the projection of precomputed laws: more than one only
// while the elements leave SMs idle (two blocks of 8 warps fill an SM)
inline int res_parts(int64_t nel) { return nel >= 304 ? 1 : (int)(608 / nel < 8 ? 608 / nel : 8); }
// The gathers apply the Dirichlet rows (RR = U - g) and rows and columns (unit
// diagonal).
int launch_tangent_gather(Context *c, double *vals, const int *err = nullptr);
int launch_tangent_gather_f32(Context *c, double *vals);
int launch_residual_gather(Context *c, double *RR, int parts, const int *err = nullptr);
void batch_gather_map(Context *c, GatherMap *a);

}  // namespace igap
