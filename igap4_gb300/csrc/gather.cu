// Element buffers to global vectors: every element's 81 residual sums and the
// 378 blocks b <= c of its (symmetric) element matrix are written once, all
// elements in one launch, and a gather adds them per DOF and per CSR slot
// (the additive phase of src/assmcore_iga.c:240-259, :745-764).
//
// The scatter it replaces needs one launch per colour: 27 launches, each as
// long as its slowest element and, below about 4,000 elements, with fewer
// elements than SMs.  The gather writes each slot once (no zeroing, no
// read-modify-write) and adds the contributions in colour order
// (9 (ex mod 3) + 3 (ey mod 3) + ez mod 3), so the sums carry the same bits as
// the colour launches.  Two memory passes of 27 KB per element.
#include <cuda_runtime.h>
#include <stdlib.h>

#include "common.cuh"
#include "element.cuh"
#include "gather.cuh"
#include "gram_common.cuh"

namespace igap {

namespace {
// 567 entries (63 columns from the diagonal on) are three rounds of 192
// threads, seven blocks per SM: 322 -> 240 us at 63x17x15 (256 threads, four
// blocks); the FP32 form's 1125 entries take 505 us with 256, 534 with 192
constexpr int TG_THREADS = 192, TGF_THREADS = 256;
constexpr int TG_NJ = 125;  // control points in a row's stencil

// Elements of one direction that hold both control points i and j, by
// residue: lo..hi consecutive, at most three.
struct Range {
  int lo, n;
};
__device__ __forceinline__ Range shared_elements(int i, int j, int ne)
{
  const int lo = max(max(i, j) - P, 0), hi = min(min(i, j), ne - 1);
  return {lo, hi - lo + 1};
}
// k-th element of the range in the order of the residues mod 3
__device__ __forceinline__ int by_residue(Range r, int e)
{
  // rank of element e among the range's elements, ordered by e mod 3
  int rank = 0;
  for (int k = r.lo; k < r.lo + r.n; k++) rank += (k % 3) < (e % 3) ? 1 : 0;
  return rank;
}

// A control point's place in its lattice and the elements around it.
struct Patch {
  int ix, iy, iz, lox, loy, loz, cy, cz, nj, nb1, nb2;
  int ne0, ne1, ne2;
};

__device__ __forceinline__ Patch patch_of(const DevMesh &m, int64_t cpl)
{
  Patch p;
  const int nb1 = m.nbasis[1], nb2 = m.nbasis[2];
  p.nb1 = nb1;
  p.nb2 = nb2;
  p.ne0 = m.nelem[0];
  p.ne1 = m.nelem[1];
  p.ne2 = m.nelem[2];
  p.iz = (int)(cpl % nb2);
  p.iy = (int)((cpl / nb2) % nb1);
  p.ix = (int)(cpl / ((int64_t)nb1 * nb2));
  p.lox = max(p.ix - P, 0);
  p.loy = max(p.iy - P, 0);
  p.loz = max(p.iz - P, 0);
  p.cy = min(p.iy + P, nb1 - 1) - p.loy + 1;
  p.cz = min(p.iz + P, nb2 - 1) - p.loz + 1;
  p.nj = (min(p.ix + P, m.nbasis[0] - 1) - p.lox + 1) * p.cy * p.cz;
  return p;
}

// Shared tables of one row of control points.  Per column control point j, the
// (element, function) pairs that contribute, in colour order: tab[27 j + rank],
// the row control point's function number b in bits 16.. (it names the element
// of the patch, whose buffer offset is ebase[b]), the entry's offset below.
struct GatherTab {
  int tab[TG_NJ * 27];
  int64_t ebase[27];             // -1: outside the lattice
  unsigned char cnt[TG_NJ];      // contributions of a column
  unsigned char fix[TG_NJ];      // its Dirichlet components (bit e)
  // per direction and (a, c): rank among the shared elements, column offset,
  // number of shared elements
  unsigned char rank[3][9], off[3][9], n[3][9];
};

template <int NT, typename F>
__device__ __forceinline__ void gather_table(GatherTab &G, const Patch &p, int64_t e0, int64_t per_element,
                                             const int *dir, F entry)
{
  if (threadIdx.x < 27) {
    const int t = threadIdx.x;
    const int ex = p.ix - t / 9, ey = p.iy - (t / 3) % 3, ez = p.iz - t % 3;
    const bool in = ex >= 0 && ex < p.ne0 && ey >= 0 && ey < p.ne1 && ez >= 0 && ez < p.ne2;
    G.ebase[t] = in ? (e0 + ((int64_t)ex * p.ne1 + ey) * p.ne2 + ez) * per_element : -1;
    // direction t / 9, element i - a, column function c
    const int dir = t / 9, a = (t / 3) % 3, c = t % 3;
    const int i = dir == 0 ? p.ix : dir == 1 ? p.iy : p.iz, lo = dir == 0 ? p.lox : dir == 1 ? p.loy : p.loz;
    const int ne = dir == 0 ? p.ne0 : dir == 1 ? p.ne1 : p.ne2;
    const Range r = shared_elements(i, i - a + c, ne);
    G.rank[dir][3 * a + c] = (unsigned char)by_residue(r, i - a);
    G.n[dir][3 * a + c] = (unsigned char)max(r.n, 0);
    G.off[dir][3 * a + c] = (unsigned char)(i - a + c - lo);
  }
  for (int j = threadIdx.x; j < p.nj; j += NT) {
    unsigned f = 0;
    if (dir) {
      const int jz = p.loz + j % p.cz, jy = p.loy + (j / p.cz) % p.cy, jx = p.lox + j / (p.cz * p.cy);
      const int *d = dir + 3 * (((int64_t)jx * p.nb1 + jy) * p.nb2 + jz);
      for (int e = 0; e < 3; e++) f |= (__ldg(d + e) ? 1u : 0u) << e;
    }
    G.fix[j] = (unsigned char)f;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 27 * NB; t += NT) {
    const int b = t / NB, c = t % NB;
    if (G.ebase[b] < 0) continue;
    const int x = b / 9 * 3 + c / 9, y = (b / 3) % 3 * 3 + (c / 3) % 3, z = b % 3 * 3 + c % 3;
    const int ny = G.n[1][y], nz = G.n[2][z];
    const int j = (G.off[0][x] * p.cy + G.off[1][y]) * p.cz + G.off[2][z];
    G.tab[j * 27 + (G.rank[0][x] * ny + G.rank[1][y]) * nz + G.rank[2][z]] = b << 16 | entry(b, c);
    G.cnt[j] = (unsigned char)(G.n[0][x] * ny * nz);  // the same value from every pair of the column
  }
  __syncthreads();
}
}  // namespace

// One block per control point: the table of its slots, then a thread per
// entry of the 3 x 3 blocks (nine consecutive threads read one 72-byte block).
// The matrix is symmetric and so are its element blocks: the columns from the
// diagonal on are summed once and stored in both rows (the FP64 additions and
// the reads halve).
__global__ void __launch_bounds__(TG_THREADS, 7) tangent_gather_kernel(GatherMap a, const double *__restrict__ ebuf,
                                                                    double *__restrict__ vals)
{
  __shared__ GatherTab G;
  __shared__ int64_t tbase[TG_NJ];  // slot of this control point's column in row 3 j
  __shared__ int tlen[TG_NJ];       // length of that row
  const int64_t cp = blockIdx.x;
  const int inst = a.cpinst ? __ldg(a.cpinst + cp) : 0;
  const DevMesh &m = a.meshes ? a.meshes[inst] : a.m;
  const int64_t cp0 = m.dof_off / 3;
  const Patch p = patch_of(m, cp - cp0);
  const int self = ((p.ix - p.lox) * p.cy + p.iy - p.loy) * p.cz + p.iz - p.loz;
  for (int j = self + threadIdx.x; j < p.nj; j += TG_THREADS) {
    const int jz = p.loz + j % p.cz, jy = p.loy + (j / p.cz) % p.cy, jx = p.lox + j / (p.cz * p.cy);
    const int64_t r = __ldg(a.rowptr + 3 * (cp0 + ((int64_t)jx * p.nb1 + jy) * p.nb2 + jz));
    const int cx = min(jx + P, m.nbasis[0] - 1) - max(jx - P, 0) + 1, cy = min(jy + P, p.nb1 - 1) - max(jy - P, 0) + 1,
              cz = min(jz + P, p.nb2 - 1) - max(jz - P, 0) + 1;
    tbase[j] = r + 3 * (((p.ix - max(jx - P, 0)) * cy + p.iy - max(jy - P, 0)) * cz + p.iz - max(jz - P, 0));
    tlen[j] = 3 * cx * cy * cz;
  }
  gather_table<TG_THREADS>(G, p, a.eoff ? __ldg(a.eoff + inst) : 0, EBUF, a.dir ? a.dir + m.dof_off : nullptr, [](int b, int c) {  // block offset, bit 15: transposed
    return 9 * pair_index(min(b, c), max(b, c)) | (b > c ? 0x8000 : 0);
  });
  const int64_t r0 = __ldg(a.rowptr + 3 * cp);
  const bool failed = a.err && *a.err;
  const int rfix = G.fix[self];
  for (int t = threadIdx.x; t < 9 * (p.nj - self); t += TG_THREADS) {
    const int j = self + t / 9, q = t % 9, d = q / 3, e = q - 3 * d;
    const int n = G.cnt[j], qt = 3 * e + d;
    const int *tab = G.tab + j * 27;
    double s = 0.0;
#pragma unroll 4
    for (int k = 0; k < n; k++) {
      const int v = tab[k];
      s += __ldg(ebuf + G.ebase[v >> 16] + (v & 0x7fff) + ((v & 0x8000) ? qt : q));
    }
    if ((rfix >> d | G.fix[j] >> e) & 1) s = j == self && d == e ? 1.0 : 0.0;
    if (failed) s = __longlong_as_double(0x7ff8000000000000ll);
    vals[r0 + (int64_t)d * 3 * p.nj + 3 * j + e] = s;
    if (j != self) vals[tbase[j] + (int64_t)e * tlen[j] + d] = s;
  }
}

// The same from FP32 element matrices [27 b][3 d][27 c][3 e] (not symmetric to
// the last bit): a thread per entry of the rows, consecutive threads along
// the columns, in the buffer as in the CSR rows.
__global__ void __launch_bounds__(TGF_THREADS) tangent_gather_f32_kernel(GatherMap a, const float *__restrict__ fbuf,
                                                                        double *__restrict__ vals)
{
  __shared__ GatherTab G;
  const int64_t cp = blockIdx.x;
  const Patch p = patch_of(a.m, cp);
  gather_table<TGF_THREADS>(G, p, 0, NB * 243, a.dir, [](int b, int c) { return 243 * b + 3 * c; });
  const int64_t r0 = __ldg(a.rowptr + 3 * cp);
  const int row = 3 * p.nj;
  const int self = ((p.ix - p.lox) * p.cy + p.iy - p.loy) * p.cz + p.iz - p.loz, rfix = G.fix[self];
  for (int t = threadIdx.x; t < 3 * row; t += TGF_THREADS) {
    const int d = t / row, x = t - d * row, j = x / 3, e = x - 3 * j;
    const int n = G.cnt[j];
    const int *tab = G.tab + j * 27;
    double s = 0.0;
#pragma unroll 4
    for (int k = 0; k < n; k++) {
      const int v = tab[k];
      s += f32_to_f64(__ldg(fbuf + G.ebase[v >> 16] + (v & 0xffff) + 81 * d + e));  // widened on the integer pipe
    }
    if ((rfix >> d | G.fix[j] >> e) & 1) s = j == self && d == e ? 1.0 : 0.0;
    vals[r0 + t] = s;
  }
}

// RR = load + the element sums of every element that holds the control point;
// U - g on the Dirichlet rows.  WARP: a warp per DOF, its lanes an element
// each (small meshes, where 27 loads one after the other are the time); else a
// thread per DOF.  The additions run in colour order either way.
template <bool WARP>
__global__ void __launch_bounds__(256) residual_gather_kernel(GatherMap a, const double *__restrict__ rbuf,
                                                              const double *__restrict__ load, double *__restrict__ RR)
{
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t dof = WARP ? t >> 5 : t;
  if (dof >= a.ndof) return;  // whole warps with WARP
  const int64_t cp = dof / 3;
  const int d = (int)(dof % 3);
  const int inst = a.cpinst ? __ldg(a.cpinst + cp) : 0;
  const DevMesh &m = a.meshes ? a.meshes[inst] : a.m;
  const int64_t e0 = a.eoff ? __ldg(a.eoff + inst) : 0;
  const int64_t cpl = cp - m.dof_off / 3;
  const int nb1 = m.nbasis[1], nb2 = m.nbasis[2];
  const int i[3] = {(int)(cpl / ((int64_t)nb1 * nb2)), (int)((cpl / nb2) % nb1), (int)(cpl % nb2)};
  const int fix = a.dir ? __ldg(a.dir + dof) : 0;
  if (fix) {
    RR[dof] = a.U[dof] - __ldg(a.dir_g + fix - 1);
    return;
  }
  // the sum of residue r's element (0 outside the lattice)
  auto element_sum = [&](int r) {
    const int rr[3] = {r / 9, (r / 3) % 3, r % 3};
    int64_t el = 0;
    int b = 0;
    bool in = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      // the element of this residue among i - 2 .. i
      const int e = i[k] - (i[k] + 3 - rr[k]) % 3;
      in = in && e >= 0 && e < m.nelem[k];
      el = el * m.nelem[k] + e;
      b = b * 3 + i[k] - e;
    }
    double v = 0.0;
    if (in) {
      const double *p = rbuf + (e0 + el) * a.parts * NE + 3 * b + d;
      v = __ldg(p);
      for (int k = 1; k < a.parts; k++) v += __ldg(p + k * NE);
    }
    return v;
  };
  double s = load[dof];
  if constexpr (WARP) {
    const int lane = threadIdx.x & 31;
    const double mine = lane < 27 ? element_sum(lane) : 0.0;
#pragma unroll
    for (int r = 0; r < 27; r++) s += __shfl_sync(0xffffffffu, mine, r);
    if (lane) return;
  } else {
#pragma unroll
    for (int r = 0; r < 27; r++) s += element_sum(r);
  }
  RR[dof] = a.err && *a.err ? __longlong_as_double(0x7ff8000000000000ll) : s;
}

static GatherMap gather_map(Context *c)
{
  GatherMap a;
  a.m = c->devmesh();
  a.rowptr = c->d_rowptr;
  a.ndof = c->ndof;
  a.meshes = nullptr;
  a.eoff = nullptr;
  a.cpinst = nullptr;
  a.err = nullptr;
  a.dir = c->d_dirmap;
  a.dir_g = c->d_dir_g;
  a.U = c->d_Uhist;
  a.parts = 1;
  if (c->batch) batch_gather_map(c, &a);
  return a;
}

int launch_tangent_gather(Context *c, double *vals, const int *err)
{
  GatherMap a = gather_map(c);
  a.err = err;
  tangent_gather_kernel<<<(unsigned)(c->ndof / 3), TG_THREADS, 0, c->stream>>>(a, c->d_ebuf, vals);
  count_launch();
  IGAP_CHECK_LAUNCH();
  return IGAPGPU_OK;
}

int launch_tangent_gather_f32(Context *c, double *vals)
{
  tangent_gather_f32_kernel<<<(unsigned)(c->ndof / 3), TGF_THREADS, 0, c->stream>>>(gather_map(c), c->d_fbuf, vals);
  count_launch();
  IGAP_CHECK_LAUNCH();
  return IGAPGPU_OK;
}

int launch_residual_gather(Context *c, double *RR, int parts, const int *err)
{
  GatherMap a = gather_map(c);
  a.parts = parts;
  a.err = err;
  if (c->ndof < 152 * 64 * 2)  // one wave of warps
    residual_gather_kernel<true><<<(unsigned)((c->ndof + 7) / 8), 256, 0, c->stream>>>(a, c->d_rbuf, c->d_Fneu, RR);
  else
    residual_gather_kernel<false><<<(unsigned)((c->ndof + 255) / 256), 256, 0, c->stream>>>(a, c->d_rbuf, c->d_Fneu, RR);
  count_launch();
  IGAP_CHECK_LAUNCH();
  return IGAPGPU_OK;
}

bool cache_fits(size_t bytes)
{
  size_t freeb = 0, totb = 0;
  return cudaMemGetInfo(&freeb, &totb) == cudaSuccess && bytes <= freeb / 4 && bytes + ((size_t)4 << 30) <= freeb;
}

void note_user_capture(Context *c)
{
  if (!c->user_captured && !c->capturing && stream_capturing(c)) c->user_captured = true;
}

bool release_caches(Context *c)
{
  if (c->user_captured || stream_capturing(c)) return false;
  void **bufs[] = {(void **)&c->d_ebuf, (void **)&c->d_rbuf, (void **)&c->d_fbuf, (void **)&c->d_sft, &c->d_xops};
  bool any = false;
  for (void **p : bufs) any = any || *p;
  if (!any) return false;
  int word = 0;
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return false;
  if (c->exact_state == 1 && c->exact_ran &&
      cudaMemcpy(&word, c->d_xerr + 1, sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess && word)
    c->async_code = word;
  assembly_graphs_release(c);  // they hold the pointers
  for (void **p : bufs) {
    if (*p) cudaFree(*p);
    *p = nullptr;
  }
  c->d_xrow = nullptr;
  c->d_xexp = nullptr;
  c->d_xerr = nullptr;
  c->exact_ran = false;
  c->ebuf_state = c->rbuf_state = c->fbuf_state = c->sf_state = c->exact_state = -1;
  return true;
}

int free_memory(Context *c, size_t need, size_t *freeb)
{
  size_t totb = 0;
  IGAP_CUDA(cudaMemGetInfo(freeb, &totb));
  if (*freeb < need && release_caches(c->owner ? c->owner : c)) IGAP_CUDA(cudaMemGetInfo(freeb, &totb));
  return IGAPGPU_OK;
}

cudaError_t room_malloc_bytes(Context *c, void **p, size_t bytes)
{
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    if (release_caches(c->owner ? c->owner : c)) e = cudaMalloc(p, bytes);
  }
  return e;
}

// Allocated at the first use outside a capture, when it fits beside what else
// the context may need; else the colour launches stay in use (also with
// IGAPGPU_ELEMENT_BUFFERS=0).
template <typename T>
static bool ensure_buffer(Context *c, T **p, int *state, size_t per_element)
{
  if (*state >= 0) {
    if (*state == 1) note_user_capture(c);
    return *state == 1;
  }
  if (stream_capturing(c)) return false;
  RelaxedCapture relaxed;
  *state = 0;
  const char *env = getenv("IGAPGPU_ELEMENT_BUFFERS");
  if (env && env[0] == '0') return false;
  const size_t bytes = sizeof(T) * per_element * (size_t)c->nelem_total;
  if (!cache_fits(bytes)) return false;
  if (cudaMalloc(p, bytes) != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return false;
  }
  *state = 1;
  return true;
}

bool ensure_ebuf(Context *c) { return ensure_buffer(c, &c->d_ebuf, &c->ebuf_state, EBUF); }
bool ensure_fbuf(Context *c) { return ensure_buffer(c, &c->d_fbuf, &c->fbuf_state, NB * 243); }
bool ensure_rbuf(Context *c) { return ensure_buffer(c, &c->d_rbuf, &c->rbuf_state, NE * (size_t)res_parts(c->nelem_total)); }

}  // namespace igap
