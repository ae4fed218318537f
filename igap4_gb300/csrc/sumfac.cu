// FP64 tangent of the reference's laws by sum factorisation, from the law
// outputs of every point (64 Gauss points, degree 2):
//   K[(b,d),(c,e)] = sum_q sum_kl R_q[b,k] D_q[(d,k),(e,l)] R_q[c,l]
// (src/assmcore_iga.c:722-750).  The FP64 pipe (2 FMA per clock and SM) bounds
// the direct form: 3.65 M FMA an element.  The rational basis's physical
// derivatives are a linear image of the tensor-product B-spline's parametric
// ones, R_q[b,k] = w_b sum_l T_q[k,l] N_b^(l), with T (73 entries that do not
// vanish: quotient rule and chain rule) independent of b, so with
//   D^_q = T_q^T D_q T_q                                      (10 x 10 per d <= e)
// the sum over the points factors direction by direction:
//   A1[(ky,kz),(ly,lz)][bx,cx](qy,qz) = sum_qx N_bx^kx N_cx^lx D^
//   A2[kz,lz][bx,cx][by,cy](qz)       = sum_qy N_by^ky N_cy^ly A1
//   K[b,c]                            = w_b w_c sum_qz N_bz^kz N_cz^lz A2
// for the six blocks d <= e (K and D are symmetric; the diagonal blocks take
// the upper half of D^, of the index groups and of the pairs): 1.10 M FMA.
// T is built once per context (37 KB an element).
//
// One CTA of 640 threads per element: thread = point x derivative in the
// transform, (group pair, bx) x (qy, qz) in x, (kz, lz, bx, cx, by) x qz in y, a
// pair (b, c) in z; D^, A1 and A2 in shared memory, the next block's moduli in
// registers before they are needed.  Results go to the element buffers
// (gather.cu).
#include <cuda_runtime.h>

#include "common.cuh"
#include "element.cuh"
#include "gather.cuh"

namespace igap {

namespace {
constexpr int SF_THREADS = 640;
constexpr int SF_Q = 64;               // Gauss points
constexpr int SF_NT = 73;              // entries of T
constexpr int SF_A1 = 20;              // stride of A1's (qy, qz), 16 used (bank spread)

struct SfSmem {
  double T[SF_NT * SF_Q];
  double M[36 * 9 * SF_A1];            // M = D T [9][10][64], then A1 [36][9][20]
  double Dh[100 * SF_Q];               // D^ [10][10][64], then A2 [9][9][9][4]
  double Kb[EBUF];
  double P[3][81 * 4];                 // per direction N_b^k N_c^l [k][l][b][c][q]
  double w[NB];
};

// index of T[k][l] (k physical, l parametric derivative)
__host__ __device__ constexpr int t_index(int k, int l)
{
  return l == 0 ? k : (l < 4 ? 10 + 9 * (l - 1) + k - 1 : 37 + 6 * (l - 4) + k - 4);
}

// derivative index of (kx, ky, kz) grouped by (ky, kz): group g's variant v has
// kx = v; grouped by kz: groups with ky = their place
__constant__ signed char c_group[6][3] = {{0, 1, 4}, {2, 5, -1}, {3, 6, -1}, {7, -1, -1}, {8, -1, -1}, {9, -1, -1}};
__constant__ signed char c_gn[6] = {3, 2, 2, 1, 1, 1};
__constant__ signed char c_zgroup[3][3] = {{0, 1, 3}, {2, 4, -1}, {5, -1, -1}};
__constant__ signed char c_zn[3] = {3, 2, 1};
// group pairs (g, h), largest products first, so that the two halves of a warp
// do equal work; the pairs g <= h among them
__constant__ signed char c_pairs[36][2] = {{0, 0}, {0, 1}, {0, 2}, {1, 0}, {2, 0}, {1, 1}, {1, 2}, {2, 1}, {2, 2},
                                           {0, 3}, {0, 4}, {0, 5}, {3, 0}, {4, 0}, {5, 0}, {1, 3}, {1, 4}, {1, 5},
                                           {2, 3}, {2, 4}, {2, 5}, {3, 1}, {4, 1}, {5, 1}, {3, 2}, {4, 2}, {5, 2},
                                           {3, 3}, {3, 4}, {3, 5}, {4, 3}, {4, 4}, {4, 5}, {5, 3}, {5, 4}, {5, 5}};
__constant__ signed char c_upairs[21][2] = {{0, 0}, {0, 1}, {0, 2}, {1, 1}, {1, 2}, {2, 2}, {0, 3},
                                            {0, 4}, {0, 5}, {1, 3}, {1, 4}, {1, 5}, {2, 3}, {2, 4},
                                            {2, 5}, {3, 3}, {3, 4}, {3, 5}, {4, 4}, {4, 5}, {5, 5}};
__constant__ signed char c_zpairs[9][2] = {{0, 0}, {0, 1}, {1, 0}, {1, 1}, {0, 2}, {2, 0}, {1, 2}, {2, 1}, {2, 2}};
__constant__ signed char c_uzpairs[6][2] = {{0, 0}, {0, 1}, {1, 1}, {0, 2}, {1, 2}, {2, 2}};
}  // namespace

// T of every point: point_geometry's steps (quotient rule, chain rule) applied
// to the unit vector of each parametric derivative.  A warp per point.
__global__ void __launch_bounds__(256) sumfac_t_kernel(DevMesh m, double *__restrict__ T)
{
  __shared__ ElemData E;
  __shared__ PointScratch Pt[8];
  __shared__ double R[8][NB * NDD];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t e = blockIdx.x;
  const int ez = (int)(e % m.nelem[2]), ey = (int)((e / m.nelem[2]) % m.nelem[1]),
            ex = (int)(e / ((int64_t)m.nelem[1] * m.nelem[2]));
  load_element(E, m, 0, nullptr, ex, ey, ez, tid, 256);
  __syncthreads();
  for (int q = warp; q < SF_Q; q += 8) {
    point_geometry(E, Pt[warp], m, ex, ey, ez, q, lane, R[warp]);
    if (lane < NDD) {
      const double *W = Pt[warp].W, *Xg = Pt[warp].Xg;
      double G[9], Gi[9];
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) G[3 * i + j] = Xg[NDD * i + 1 + j];
      const double c0 = G[4] * G[8] - G[5] * G[7], c1 = G[2] * G[7] - G[1] * G[8], c2 = G[1] * G[5] - G[2] * G[4];
      const double c3 = G[5] * G[6] - G[3] * G[8], c4 = G[0] * G[8] - G[2] * G[6], c5 = G[2] * G[3] - G[0] * G[5];
      const double c6 = G[3] * G[7] - G[4] * G[6], c7 = G[1] * G[6] - G[0] * G[7], c8 = G[0] * G[4] - G[1] * G[3];
      const double id = 1.0 / (G[0] * c0 + G[1] * c3 + G[2] * c6);
      Gi[0] = c0 * id; Gi[1] = c1 * id; Gi[2] = c2 * id;
      Gi[3] = c3 * id; Gi[4] = c4 * id; Gi[5] = c5 * id;
      Gi[6] = c6 * id; Gi[7] = c7 * id; Gi[8] = c8 * id;
      double r[NDD], n[NDD];
      for (int k = 0; k < NDD; k++) r[k] = k == lane ? 1.0 / W[0] : 0.0;
      for (int k = 1; k < NDD; k++) r[k] -= r[0] * W[k] / W[0];
      int a = 4;
      for (int i = 1; i < 4; i++)
        for (int j = i; j < 4; j++) { r[a] -= (r[j] * W[i] + r[i] * W[j]) / W[0]; a++; }
      for (int k = 0; k < NDD; k++) n[k] = r[k];
      for (int i = 0; i < 3; i++) {
        double s = 0.0;
        for (int j = 0; j < 3; j++) s += n[1 + j] * Gi[3 * j + i];
        r[1 + i] = s;
      }
      for (int k = 4; k < NDD; k++)
        for (int i = 0; i < 3; i++) n[k] -= r[1 + i] * Xg[NDD * i + k];
      const double Hs[3][3] = {{n[4], n[5], n[6]}, {n[5], n[7], n[8]}, {n[6], n[8], n[9]}};
      a = 4;
      for (int i = 0; i < 3; i++)
        for (int j = i; j < 3; j++) {
          double s = 0.0;
          for (int mm = 0; mm < 3; mm++) {
            double t = 0.0;
            for (int l = 0; l < 3; l++) t += Hs[mm][l] * Gi[3 * l + j];
            s += Gi[3 * mm + i] * t;
          }
          r[a++] = s;
        }
      double *o = T + e * (SF_NT * SF_Q) + q;
      const int k0 = lane == 0 ? 0 : (lane < 4 ? 1 : 4);
      for (int k = k0; k < NDD; k++) o[t_index(k, lane) * SF_Q] = r[k];
    }
    __syncwarp();
  }
}

// Block (d, e) of the element matrix from its moduli in registers (`row`: this
// thread's row r of D, thread = (r, q)); SYM: d = e.
template <bool SYM>
__device__ __forceinline__ void sumfac_block(SfSmem &S, const double (&row)[9], double mass, int d, int e)
{
  const int tid = threadIdx.x, q = tid & 63, r = (tid >> 6) + 1;  // r: 1..9 (10: idle)
  if (r <= 9) {  // M[r][l] = sum_k D[r][k] T[k][l]
    double *o = S.M + (r - 1) * 10 * SF_Q + q;
#pragma unroll
    for (int l = 0; l < 10; l++) {
      double s = 0.0;
#pragma unroll
      for (int k = l < 4 ? 1 : 4; k < 10; k++) s = fma(row[k - 1], S.T[t_index(k, l) * SF_Q + q], s);
      o[l * SF_Q] = s;
    }
  }
  __syncthreads();
  {  // D^[l'][l] = sum_r T[r][l'] M[r][l], thread = (l, q); SYM: l' <= l
    const int l = tid >> 6;
    double mc[9];
#pragma unroll
    for (int k = 0; k < 9; k++) mc[k] = S.M[(k * 10 + l) * SF_Q + q];
#pragma unroll
    for (int lp = 0; lp < 10; lp++) {
      if (SYM && lp > l) break;
      double s = lp == 0 && l == 0 ? S.T[q] * S.T[q] * mass : 0.0;  // the value slots' inertia
#pragma unroll
      for (int k = lp < 4 ? 1 : 4; k < 10; k++) s = fma(S.T[t_index(k, lp) * SF_Q + q], mc[k - 1], s);
      S.Dh[(lp * 10 + l) * SF_Q + q] = s;
    }
  }
  __syncthreads();
  // x: a half warp per (group pair, bx), lane = (qy, qz)
  {
    constexpr int NP = SYM ? 21 : 36;
    const int yz = tid & 15;
    for (int t = tid >> 4; t < NP * 3; t += SF_THREADS / 16) {
      const int p = t / 3, bx = t - 3 * p;
      const int g = SYM ? c_upairs[p][0] : c_pairs[p][0], h = SYM ? c_upairs[p][1] : c_pairs[p][1];
      double a0 = 0.0, a1 = 0.0, a2 = 0.0;
      const int ng = c_gn[g], nh = c_gn[h];
      for (int kx = 0; kx < ng; kx++)
        for (int lx = 0; lx < nh; lx++) {
          const int k = c_group[g][kx], l = c_group[h][lx];
          const double *dh = S.Dh + (SYM && k > l ? l * 10 + k : k * 10 + l) * SF_Q + yz;
          const double *P = S.P[0] + ((kx * 3 + lx) * 9 + bx * 3) * 4;
#pragma unroll
          for (int qx = 0; qx < 4; qx++) {
            const double v = dh[16 * qx];
            a0 = fma(P[qx], v, a0);
            a1 = fma(P[4 + qx], v, a1);
            a2 = fma(P[8 + qx], v, a2);
          }
        }
      double *o = S.M + ((g * 6 + h) * 9 + bx * 3) * SF_A1 + yz;
      o[0] = a0;
      o[SF_A1] = a1;
      o[2 * SF_A1] = a2;
    }
  }
  __syncthreads();
  // y: thread = ((kz, lz), by, (bx, cx), qz), its three cy
  {
    constexpr int NZ = SYM ? 6 : 9;
    for (int t = tid; t < NZ * 108; t += SF_THREADS) {
      const int qz = t & 3, xx = (t >> 2) % 9, by = (t / 36) % 3, z = t / 108;
      const int kz = SYM ? c_uzpairs[z][0] : c_zpairs[z][0], lz = SYM ? c_uzpairs[z][1] : c_zpairs[z][1];
      const int xt = SYM ? (xx % 3) * 3 + xx / 3 : xx;  // (cx, bx)
      double a0 = 0.0, a1 = 0.0, a2 = 0.0;
      const int nk = c_zn[kz], nl = c_zn[lz];
      for (int ky = 0; ky < nk; ky++)
        for (int ly = 0; ly < nl; ly++) {
          const int g = c_zgroup[kz][ky], h = c_zgroup[lz][ly];
          const double *src = S.M + (SYM && g > h ? (h * 6 + g) * 9 + xt : (g * 6 + h) * 9 + xx) * SF_A1 + qz;
          const double *P = S.P[1] + ((ky * 3 + ly) * 9 + by * 3) * 4;
#pragma unroll
          for (int qy = 0; qy < 4; qy++) {
            const double v = src[4 * qy];
            a0 = fma(P[qy], v, a0);
            a1 = fma(P[4 + qy], v, a1);
            a2 = fma(P[8 + qy], v, a2);
          }
        }
      double *o = S.Dh + (((kz * 3 + lz) * 9 + xx) * 9 + by * 3) * 4 + qz;
      o[0] = a0;
      o[4] = a1;
      o[8] = a2;
    }
  }
  __syncthreads();
  // z: thread = (b, c); SYM: b <= c
  for (int t = tid; t < NB * NB; t += SF_THREADS) {
    const int b = t / NB, c = t - NB * b;
    if (SYM && b > c) continue;
    const int xx = (b / 9) * 3 + c / 9, yy = (b / 3 % 3) * 3 + c / 3 % 3, bz = b % 3, cz = c % 3;
    const int xt = (c / 9) * 3 + b / 9, yt = (c / 3 % 3) * 3 + b / 3 % 3;
    double s = 0.0;
#pragma unroll
    for (int kz = 0; kz < 3; kz++)
#pragma unroll
      for (int lz = 0; lz < 3; lz++) {
        const double *src = S.Dh + (SYM && kz > lz ? ((lz * 3 + kz) * 9 + xt) * 9 + yt : ((kz * 3 + lz) * 9 + xx) * 9 + yy) * 4;
        const double *P = S.P[2] + ((kz * 3 + lz) * 9 + bz * 3 + cz) * 4;
#pragma unroll
        for (int qz = 0; qz < 4; qz++) s = fma(P[qz], src[qz], s);
      }
    s *= S.w[b] * S.w[c];
    if (b <= c) S.Kb[9 * pair_index(b, c) + 3 * d + e] = s;
    if (!SYM && b >= c) S.Kb[9 * pair_index(c, b) + 3 * e + d] = s;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(SF_THREADS, 1)
    sumfac_tangent_kernel(DevMesh m, const double *__restrict__ T, const double *__restrict__ preD, int inertia,
                          double *__restrict__ ebuf)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SfSmem &S = *reinterpret_cast<SfSmem *>(smem_raw);
  const int tid = threadIdx.x, q = tid & 63, r = (tid >> 6) + 1;
  const int64_t el = blockIdx.x;
  const int ei[3] = {(int)(el / ((int64_t)m.nelem[1] * m.nelem[2])), (int)((el / m.nelem[2]) % m.nelem[1]),
                     (int)(el % m.nelem[2])};
  const double *D = preD + el * 900 * SF_Q + q;
  double row[9];
  auto load_row = [&](int d, int e) {
    if (r <= 9)
#pragma unroll
      for (int k = 0; k < 9; k++) row[k] = __ldg(D + (int64_t)(30 * (10 * d + r) + 10 * e + 1 + k) * SF_Q);
  };
  load_row(0, 0);
  for (int i = tid; i < SF_NT * SF_Q; i += SF_THREADS) S.T[i] = __ldg(T + el * (SF_NT * SF_Q) + i);
  for (int i = tid; i < 3 * 324; i += SF_THREADS) {
    const int dir = i / 324, x = i % 324, iq = x & 3, c = (x >> 2) % 3, b = (x / 12) % 3, l = (x / 36) % 3, k = x / 108;
    const double *t = m.tab[dir] + ((size_t)ei[dir] * 4 + iq) * TAB;  // N, N', N'' of three functions
    S.P[dir][x] = __ldg(t + P1 * k + b) * __ldg(t + P1 * l + c);
  }
  if (tid < NB) {
    const int64_t cp = ((int64_t)(ei[0] + tid / 9) * m.nbasis[1] + (ei[1] + (tid / 3) % 3)) * m.nbasis[2] + (ei[2] + tid % 3);
    S.w[tid] = __ldg(m.w + cp);
  }
  __syncthreads();
  for (int d = 0; d < 3; d++)
    for (int e = d; e < 3; e++) {
      double cur[9];
#pragma unroll
      for (int k = 0; k < 9; k++) cur[k] = row[k];
      if (e < 2) load_row(d, e + 1);
      else if (d < 2) load_row(d + 1, d + 1);
      if (d == e)
        sumfac_block<true>(S, cur, inertia ? __ldg(D + (int64_t)(30 * 10 * d + 10 * d) * SF_Q) : 0.0, d, e);
      else
        sumfac_block<false>(S, cur, 0.0, d, e);
    }
  for (int i = tid; i < EBUF; i += SF_THREADS) ebuf[el * EBUF + i] = S.Kb[i];
}

// T of every point, built at the first use outside a capture; false where the
// sum-factorised form does not apply (other than 64 points, no precomputed law
// outputs) or memory is short (37 KB an element beside the element buffers).
bool ensure_sumfac(Context *c, const DevLaw &L)
{
  if (!L.preD || c->nquad != 4 || c->porder != P || c->batch) return false;
  if (c->sf_state >= 0) {
    if (c->sf_state == 1) note_user_capture(c);
    return c->sf_state == 1;
  }
  if (stream_capturing(c)) return false;
  RelaxedCapture relaxed;
  c->sf_state = 0;
  const size_t bytes = sizeof(double) * SF_NT * SF_Q * (size_t)c->nelem_total;
  if (!ensure_ebuf(c) || !cache_fits(bytes)) return false;
  if (cudaMalloc(&c->d_sft, bytes) != cudaSuccess) {
    cudaGetLastError();
    c->d_sft = nullptr;
    return false;
  }
  DevMesh m = c->devmesh();
  m.geo = nullptr;
  sumfac_t_kernel<<<(unsigned)c->nelem_total, 256, 0, c->stream>>>(m, c->d_sft);
  count_launch();
  // complete before a later call on another stream reads it
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(c->stream) != cudaSuccess) return false;
  c->sf_state = 1;
  return true;
}

int launch_sumfac(Context *c, const DevLaw &L, double *vals)
{
  static bool attr = false;
  if (!attr) {
    IGAP_CUDA(cudaFuncSetAttribute(sumfac_tangent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SfSmem)));
    attr = true;
  }
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (c->prof) {
    IGAP_CUDA(cudaEventCreate(&e0));
    IGAP_CUDA(cudaEventCreate(&e1));
    IGAP_CUDA(cudaEventRecord(e0, c->stream));
  }
  sumfac_tangent_kernel<<<(unsigned)c->nelem_total, SF_THREADS, sizeof(SfSmem), c->stream>>>(
      c->devmesh(), c->d_sft, L.preD, c->law == IGAPGPU_LAW_GRADELASTTIME ? 1 : 0, c->d_ebuf);
  count_launch();
  IGAP_CHECK_LAUNCH();
  if (c->prof) {
    IGAP_CUDA(cudaEventRecord(e1, c->stream));
    c->prof_ev[0].emplace_back(e0, e1);
    c->prof_launches[0]++;
    c->prof_elements[0] += c->nelem_total;
  }
  return launch_tangent_gather(c, vals);
}

}  // namespace igap
