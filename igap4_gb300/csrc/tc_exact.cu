// FP64 tangent and residual of the linear isotropic strain-gradient law on
// the tensor cores.  The tangent of the law is a function of the Gram matrix
// G = S S^T of the sqrt(w)-weighted derivatives (tc_gram.cu):
//   K[(b,d),(c,e)] = lam G[(b,d),(c,e)] + mu G[(b,e),(c,d)] + delta_de mu tr G_bc.
// The FP64 pipe (2 FMA per clock and SM) bounds the direct sum: 0.94 M FMA,
// 250 us per element and SM.  Here S is cut error-free into six 9-bit
// slices (Ozaki, Ogita, Oishi, Rump, Numer. Algorithms 59 (2012)) whose BF16
// products the tensor cores sum exactly, and the partial sums are joined in
// 64-bit integers, so that G carries the accuracy of a sum in more than 53
// bits:
//  * row r (81 rows, K = 64 points x 4 slots) is scaled by its own power of
//    two, x = 2^(8 - E_r) S_r, |x| < 256 and |x|_2 <= 2048, rounded to 45
//    fraction bits and split into balanced digits
//      x = D1 + D2 2^-9 + ... + D6 2^-45,  |D_j| <= 256
//    (integers up to 256 are exact in BF16, and so are the stored
//    D_j 2^(-9 (j - 1))); the representation error is 2^-46 of 2^8, 2^-54 of
//    the row's largest entry;
//  * accumulators by weight, s = i + j: acc2 = D1 D1^T; X3 = D1 D2^T;
//    acc4 = the three products with s = 4; X5 = D1 D4^T + D2 D3^T; acc6 = the
//    five with s = 6; acc78 = the eleven with s = 7 and 8 (s >= 9, 2^-63 of
//    the leading term and below, is left out).  G needs X + X^T at the odd
//    weights.  Every partial sum of acc2, X3, acc4 and X5 is an integer
//    multiple of the weight's unit; it stays below 2^24 units (Cauchy-Schwarz
//    on the digits' row norms, checked for every entry of every element when the
//    slices are built; an element that fails keeps the whole context on the FP64
//    kernel: 7 of 6,000 regular box meshes with length scales 0.05 to 0.2),
//    so the FP32 accumulation is exact.  acc6 and acc78 round at 2^-56 and
//    2^-64 of the leading term.
//  * tensor memory holds 512 columns: acc2, acc4, acc6, acc78 with N = 80 and
//    X3, X5 with N = 96.  Column 80 of the symmetric ones is their row 80;
//    the entry (80, 80) is a 256-term FP64 dot product of the row itself.
// Residual: exact for constants as the quadrature loop is not (the state enters
// as differences from the element's middle function: a translation of 5 beside
// displacements of 1e-3 costs the quadrature loop 2e-13, this 1e-15).
// Measured: against 64-bit reference sums the tangent's error is the FP64 kernel's
// (7e-16 at 16x4x4, 3e-15 at 63x17x15 distorted, both from the geometry; the two
// tangents differ by 2e-16).  The residual's error against long double is the
// quadrature loop's within 10 % on random, sinusoidal and most affine states (1e-15 to
// 4e-15 of |F|); on pure bending, whose Hessian terms cancel, the rounding of the
// rows of S adds to the geometry's and it is 1.2 to 1.7 times as large (1.4e-15 to
// 7e-15 there, 2e-15 to 1.2e-14 here; affine states at length scale 0.2 up to 1.3).  Residual and tangent at 16x4x4 7.9 ms (FP64 kernel,
// colour by colour) -> 78 us, 63x17x15 36.7 -> 1.98 ms.  Per element and SM 31 k
// clocks, 27 k of them MMAs (73 clocks each: shared-memory operand reads).
//
// One persistent CTA per SM over all elements; results go to the element
// buffers (gather.cu):
//   warp 0: bulk copies of the chunks (8 points: 6 slices x 2 K-steps x 11 row
//     groups x 256 B) into XS_NS stages,
//   warp 1: 23 MMAs (kind::f16 BF16, M128, N 80 or 96, K16) per K-step,
//   warps 4-6 and 8-10: accumulators -> Y[r][c] in shared memory (int64, units
//     of 2^-36): c > r the symmetric sums and X, c < r X alone, so that
//     G_rc = Y[r][c] + Y[c][r]; the tensor memory is free for the next element
//     after that.  acc78 is drained first and released alone: its products, 11
//     of 23, of the next element's staged chunks run while the others are
//     drained (9 k clocks that the tensor core stood idle: 36 -> 31 k clocks),
//   warps 2-13: a thread per basis pair b <= c forms its 3 x 3 block of K in
//     FP64; the element's blocks leave by one bulk copy, and the residual of
//     the linear law is K_e u_e from the blocks in shared memory (6,561 FMA an
//     element under the next element's MMAs; the quadrature loop takes 93,312
//     on the FP64 pipe).
// Every mbarrier wait is bounded; a CTA that gives up sets the error words
// (the gathers of this launch then write NaN; the context reports the other
// word at its next synchronisation), waits (bounded) for its copies and MMAs in
// flight and frees its tensor memory.  The words are this kernel's own: what
// another kernel left in the context's shared word is not taken for a failure
// of this launch, and another launch does not clear one before it is reported.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include "common.cuh"
#include "element.cuh"
#include "gather.cuh"
#include "gram_common.cuh"
#include "tcgen05.cuh"

namespace igap {

namespace {
constexpr int XS_THREADS = 448;
constexpr int XS_EPI = XS_THREADS - 64;          // epilogue threads: warps 2..13
constexpr int XS_ROWS = NE;                      // 81
constexpr int XS_RG = 11;                        // row groups holding rows 0..87
constexpr int XS_NSL = 6;                        // slices
constexpr int XS_KS_BYTES = XS_RG * 256;         // one K-step of 16 BF16 values
constexpr int XS_SLICE_BYTES = 2 * XS_KS_BYTES;  // a chunk of 8 points (K = 32)
constexpr int XS_CH_BYTES = XS_NSL * XS_SLICE_BYTES;
constexpr int XS_STAGE = XS_CH_BYTES + 5 * 256;  // an M = 128 read of the last K-step stays inside
constexpr int XS_NS = 4;
constexpr int XS_MAXCH = 8;                      // chunks: K <= 256, the exactness bound
constexpr int XS_YP = 83;                        // row stride of Y (odd: conflict-free columns)
constexpr int XS_EXP = 88;
constexpr uint32_t XS_TMEM_COLS = 512;
constexpr uint32_t XS_ACC2 = 0, XS_ACC4 = 80, XS_ACC6 = 160, XS_ACC78 = 240, XS_X3 = 320, XS_X5 = 416;
constexpr uint32_t XS_WAIT_LIMIT = 1u << 26;
constexpr int XO_THREADS = 512;                  // operand kernel
constexpr int XO_LD = (NB * 9 + 31) / 32;        // its loads per lane and point
static_assert(XS_STAGE % 16 == 0 && XS_CH_BYTES % 16 == 0, "bulk copies and descriptors need 16-byte alignment");
static_assert(EBUF * sizeof(double) % 16 == 0, "bulk stores move multiples of 16 bytes");

struct XsSmem {
  unsigned char stage[XS_NS][XS_STAGE];
  double Kb[EBUF];
  long long Y[XS_ROWS * XS_YP];
  unsigned char pb[NPAIRS], pc[NPAIRS];
  double g80;
  double u[NE], rsum[4][NE];
  int ex[XS_EXP];
  uint64_t full[XS_NS], empty[XS_NS], accfull, accempty, empty78;
  uint32_t cp_n[XS_NS], mm_n[XS_NS], accf_n;
  uint32_t taddr;
  int abort;
};
static_assert(sizeof(XsSmem) + 1024 <= 227 * 1024, "one CTA per SM");

struct ExactArgs {
  const unsigned char *ops;   // [element][chunk][XS_CH_BYTES]
  const short *expo;          // [element][XS_EXP]
  const double *row80;        // [element][chunk * 32] row 80 of S
  double *ebuf;               // element matrices out (or null)
  const double *U;            // current state: element residuals K_e u_e to rbuf (or null)
  double *rbuf;
  DevMesh m;
  int64_t nelem;
  int nchunk;
  double lam, mu;
  // batches: law, mesh and first element of every instance, instance of every element
  const DevLaw *laws;
  const DevMesh *meshes;
  const int64_t *eoff;
  const int *einst;
  int *err;  // [0] this launch, [1] until reported
};

__device__ __forceinline__ void mbar_arrive1(uint64_t *mbar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(mbar)) : "memory");
}

__device__ __forceinline__ bool xs_wait(uint64_t *mbar, uint32_t parity, volatile int *abort)
{
  const uint32_t addr = tc::smem_u32(mbar);
  for (uint32_t it = 0; it < XS_WAIT_LIMIT; it++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 255u) == 255u && *abort) return false;
  }
  return false;
}

// v (an integer multiple of 2^-s, or rounded to one) as an integer of that unit
__device__ __forceinline__ long long units(uint32_t v, float scale, int shift)
{
  return (long long)__float2int_rn(__uint_as_float(v) * scale) << shift;
}

// v 2^k on the integer pipe (v an integer below 2^62 in magnitude)
__device__ __forceinline__ double scaled(long long v, int k)
{
  const double d = (double)v;
  if (v == 0) return 0.0;
  return __hiloint2double(__double2hiint(d) + (k << 20), __double2loint(d));
}
}  // namespace

// Slices of every element, once per context (state independent).  One CTA per
// element: S in shared memory (row stride K + 1), row exponents, digits.
// Integer operations and the loads' latency bound it: the digits as bit fields of
// a biased sum with one exact FMA each, and the next point's loads in flight,
// take it from 4.2 to 2.5 ms at 63x17x15 (76 k -> 45 k clocks an element) and the
// first assembly from 7.2 to 5.3 ms.
__global__ void __launch_bounds__(XO_THREADS) exact_operand_kernel(const double *__restrict__ geo, int npts, int nchunk,
                                                                   int64_t nelem, double ell,
                                                                   unsigned char *__restrict__ ops,
                                                                   short *__restrict__ expo,
                                                                   double *__restrict__ row80, int *__restrict__ bad)
{
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  double *S = reinterpret_cast<double *>(smem_raw);
  __shared__ double sw[XS_MAXCH * PW], swl[XS_MAXCH * PW];
  __shared__ int rexp[XS_EXP];
  __shared__ int nrm[XS_EXP][4];
  __shared__ float nf[XS_ROWS][4];
  __shared__ int stop;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = nchunk * 32, ld = K + 1;
  // this lane's values of a point (0: none): place in the cache, second
  // derivative, its two indices (gradient: index), row 3 b
  int off[XO_LD];
#pragma unroll
  for (int i = 0; i < XO_LD; i++) {
    const int u = lane + 32 * i, b = u / 9, s = u % 9, h = s - 3;  // h: xx, xy, xz, yy, yz, zz
    const int i0 = s < 3 ? s : (h < 3 ? 0 : (h < 5 ? 1 : 2)), m0 = s < 3 ? 0 : (h < 3 ? h : (h < 5 ? h - 2 : 2));
    off[i] = u < NB * 9 ? (NDD * b + 1 + s) | (s >= 3) << 10 | i0 << 11 | m0 << 13 | 3 * b << 15 : 0;
  }
  for (int64_t e = blockIdx.x; e < nelem; e += gridDim.x) {
    for (int q = tid; q < nchunk * PW; q += XO_THREADS) {
      double w = q < npts ? geo[(e * npts + q) * GEO_STRIDE + NB * NDD] : 0.0;
      if (q < npts && !(w > 0.0)) {
        atomicExch(bad, 1);
        w = 0.0;
      }
      sw[q] = sqrt(w);
      swl[q] = sqrt(w) * ell;
    }
    for (int i = tid; i < XS_EXP * 4; i += XO_THREADS) nrm[i / 4][i % 4] = 0;
    __syncthreads();
    // column of point q: 32 (q / 8) + q % 8 for the gradient, + 8 + 3 (q % 8) + m for the Hessian row's entry m;
    // a warp per point, the next point's loads in flight
    {
      double v[XO_LD];
      auto fetch = [&](int q) {
        const double *g = geo + (e * npts + q) * GEO_STRIDE;
#pragma unroll
        for (int i = 0; i < XO_LD; i++) v[i] = q < npts && off[i] ? __ldg(g + (off[i] & 0x3ff)) : 0.0;
      };
      fetch(warp);
      for (int q = warp; q < nchunk * PW; q += XO_THREADS / 32) {
        double x[XO_LD];
        const double wq = sw[q], wl = swl[q];
#pragma unroll
        for (int i = 0; i < XO_LD; i++) x[i] = v[i] * ((off[i] >> 10) & 1 ? wl : wq);
        if (q + XO_THREADS / 32 < nchunk * PW) fetch(q + XO_THREADS / 32);
        const int c0 = 32 * (q / PW), p = q % PW;
#pragma unroll
        for (int i = 0; i < XO_LD; i++) {
          if (!off[i]) continue;
          double *row = S + (off[i] >> 15) * ld + c0;  // row 3 b
          const int i0 = (off[i] >> 11) & 3, m0 = (off[i] >> 13) & 3;
          if (!((off[i] >> 10) & 1)) {
            row[i0 * ld + p] = x[i];
          } else {
            row[i0 * ld + PW + 3 * p + m0] = x[i];
            if (i0 != m0) row[m0 * ld + PW + 3 * p + i0] = x[i];
          }
        }
      }
    }
    __syncthreads();
    // E_r: max |S_r| < 2^E_r, and one more where |x|_2 would exceed 2048
    for (int r = warp; r < XS_ROWS; r += XO_THREADS / 32) {
      int hi = 0;
      for (int k = lane; k < K; k += 32) hi = max(hi, __double2hiint(S[r * ld + k]) & 0x7fffffff);
      for (int o = 16; o > 0; o >>= 1) hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      const int ef = hi >> 20;
      int E = ef - 1022;
      if (ef == 0) E = 0;  // a zero row (tinier entries count as zero next to E = -400)
      else if (ef > 1422 || ef < 622) {
        if (lane == 0) atomicExch(bad, 1);
        E = 0;
      }
      // |x|^2 from the leading 24 bits, scaled on the integer pipe (|x| < 2^-100 counts as zero)
      float n2 = 0.f;
      for (int k = lane; k < K; k += 32) {
        const double v = S[r * ld + k];
        const int fe = ((__double2hiint(v) >> 20) & 0x7ff) - 1023 + 8 - E + 127;
        const float x = fe > 27 ? __uint_as_float((uint32_t)fe << 23 | ((uint32_t)__double2hiint(v) & 0xfffffu) << 3 |
                                                  (uint32_t)__double2loint(v) >> 29)
                                : 0.f;
        n2 = fmaf(x, x, n2);
      }
      for (int o = 16; o > 0; o >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, o);
      if (n2 > 4.18e6f) E++;  // 2048^2 less the truncation of x and the rounding of this sum
      if (lane == 0) rexp[r] = E;
    }
    for (int r = XS_ROWS + tid; r < XS_EXP; r += XO_THREADS) rexp[r] = 0;
    __syncthreads();
    unsigned char *oe = ops + (size_t)e * nchunk * XS_CH_BYTES;
    // task: 8 consecutive columns of a row (one 16-byte piece of each slice)
    for (int t = tid; t < nchunk * 4 * XS_RG * 8; t += XO_THREADS) {
      const int r = t % (XS_RG * 8), kq = t / (XS_RG * 8);  // kq: chunk * 4 + K-step * 2 + half
      uint32_t out[XS_NSL][4];
#pragma unroll
      for (int j = 0; j < XS_NSL; j++)
#pragma unroll
        for (int i = 0; i < 4; i++) out[j][i] = 0u;
      if (r < XS_ROWS) {
        const int E = rexp[r];
        float s2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          float f[2][XS_NSL];
#pragma unroll
          for (int u = 0; u < 2; u++) {
            const double v = S[r * ld + kq * 8 + i + u];
            const int hw = __double2hiint(v);
            const int ef = (hw >> 20) & 0x7ff;
            long long X = 0;
            if (ef) {
              // v = m 2^(ef - 1075); x = v 2^(8 - E), 45 fraction bits: m shifted right by E + 1022 - ef >= 0
              const long long mt = ((long long)((hw & 0xfffff) | 0x100000) << 32) | (uint32_t)__double2loint(v);
              const int n = E + 1022 - ef;
              X = n == 0 ? mt : (n < 55 ? (mt + (1ll << (n - 1))) >> n : 0);
              if (hw < 0) X = -X;
            }
            // balanced digits: with 256 added at every digit's place they are the
            // 9-bit fields less 256.  2^23 + field is a float by its bits, and one
            // exact FMA takes off the bias and scales.
            const long long Y = X + 0x1008040201ll * 256;
            const int top = (int)(Y >> 45);  // D1 itself, -256 .. 256
            f[u][0] = __uint_as_float(0x4b000000u | (uint32_t)(top + 256)) - 8388864.f;
            float sc = 1.f / 512.f;
#pragma unroll
            for (int j = 1; j < XS_NSL; j++) {
              const uint32_t d = (uint32_t)(Y >> (9 * (XS_NSL - 1 - j))) & 511u;
              f[u][j] = __fmaf_rn(__uint_as_float(0x4b000000u | d), sc, -8388864.f * sc);
              sc *= 1.f / 512.f;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) s2[j] = fmaf(f[u][j], f[u][j], s2[j]);  // exact: below 2^20 units
          }
#pragma unroll
          for (int j = 0; j < XS_NSL; j++)  // exact in BF16: at most 8 significant bits
            out[j][i / 2] = __byte_perm(__float_as_uint(f[0][j]), __float_as_uint(f[1][j]), 0x7632);
        }
        float un = 1.f;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          atomicAdd(&nrm[r][j], (int)(s2[j] * un));
          un *= 262144.f;
        }
      }
      unsigned char *o = oe + (size_t)(kq / 4) * XS_CH_BYTES + ((kq / 2) % 2) * XS_KS_BYTES + (r / 8) * 256 +
                         (kq % 2) * 128 + (r % 8) * 16;
#pragma unroll
      for (int j = 0; j < XS_NSL; j++)
        *reinterpret_cast<uint4 *>(o + (size_t)j * XS_SLICE_BYTES) = make_uint4(out[j][0], out[j][1], out[j][2], out[j][3]);
    }
    for (int r = tid; r < XS_EXP; r += XO_THREADS) expo[e * XS_EXP + r] = (short)rexp[r];
    for (int k = tid; k < K; k += XO_THREADS) row80[e * K + k] = S[80 * ld + k];
    __syncthreads();
    // partial sums of acc4 and X5 below 2^24 units, entry by entry (the largest
    // norms of an element's rows together refused 28 of 1,500 regular box meshes)
    for (int i = tid; i < XS_ROWS * 4; i += XO_THREADS) nf[i / 4][i % 4] = sqrtf((float)nrm[i / 4][i % 4]);
    if (tid == 0) stop = *(volatile int *)bad;
    __syncthreads();
    bool over = false;
    for (int t = tid; t < XS_ROWS * XS_ROWS; t += XO_THREADS) {
      const float *a = nf[t / XS_ROWS], *b = nf[t % XS_ROWS];
      over |= a[0] * b[2] + a[2] * b[0] + a[1] * b[1] > 1.67e7f || a[0] * b[3] + a[1] * b[2] > 1.67e7f;
    }
    if (over) atomicExch(bad, 1);
    if (stop) break;  // some element failed: no slices for this context
    __syncthreads();
  }
}

__global__ void __launch_bounds__(XS_THREADS, 1) exact_tangent_kernel(ExactArgs a)
{
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  XsSmem &S = *reinterpret_cast<XsSmem *>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int *abort = &S.abort;
  if (warp == 0) {
    tc::tmem_alloc(&S.taddr, XS_TMEM_COLS);
    tc::tmem_relinquish();
  }
  for (int b = tid; b < NB; b += XS_THREADS)
    for (int c = b; c < NB; c++) {
      S.pb[pair_index(b, c)] = (unsigned char)b;
      S.pc[pair_index(b, c)] = (unsigned char)c;
    }
  if (tid == 0) {
    for (int i = 0; i < XS_NS; i++) {
      tc::mbar_init(&S.full[i], 1);
      tc::mbar_init(&S.empty[i], 1);
      S.cp_n[i] = S.mm_n[i] = 0;
    }
    tc::mbar_init(&S.accfull, 1);
    tc::mbar_init(&S.accempty, 192);
    tc::mbar_init(&S.empty78, 192);
    S.accf_n = 0;
    S.abort = 0;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = S.taddr;
  const int nmine = (int64_t)blockIdx.x < a.nelem ? (int)((a.nelem - 1 - blockIdx.x) / gridDim.x) + 1 : 0;
  const uint32_t nchunk = (uint32_t)a.nchunk;
  if (warp == 0) {
    if (lane == 0) {  // producer
      uint32_t s = 0, cpn[XS_NS] = {};
      bool ok = true;
      for (int j = 0; j < nmine && ok; j++) {
        const unsigned char *src = a.ops + (size_t)(blockIdx.x + (int64_t)j * gridDim.x) * nchunk * XS_CH_BYTES;
        for (uint32_t c = 0; c < nchunk; c++, s++) {
          const int st = (int)(s % XS_NS);
          if (s >= (uint32_t)XS_NS && !xs_wait(&S.empty[st], ((s / XS_NS) - 1) & 1, abort)) {
            ok = false;
            break;
          }
          tc::mbar_arrive_expect_tx(&S.full[st], (uint32_t)XS_CH_BYTES);
          tc::bulk_g2s(S.stage[st], src + (size_t)c * XS_CH_BYTES, (uint32_t)XS_CH_BYTES, &S.full[st]);
          cpn[st]++;
        }
      }
      if (!ok) S.abort = 1;
      for (int i = 0; i < XS_NS; i++) S.cp_n[i] = cpn[i];
    }
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issuer
      const uint32_t id80 = tc::instr_desc(1, 128, 80), id96 = tc::instr_desc(1, 128, 96);
      uint32_t s = 0, mmn[XS_NS] = {}, accn = 0;
      bool ok = true;
      auto slices = [&](uint32_t st, int ks, uint64_t *d) {
        const uint32_t base = tc::smem_u32(S.stage[st]);
#pragma unroll
        for (int q = 0; q < XS_NSL; q++)
          d[q] = tc::smem_desc(base + (uint32_t)(q * XS_SLICE_BYTES + ks * XS_KS_BYTES), 128, 256);
      };
      auto low = [&](uint32_t st, uint32_t c) {  // the products of acc78
        for (int ks = 0; ks < 2; ks++) {
          uint64_t d[XS_NSL];
          slices(st, ks, d);
#pragma unroll
          for (int q = 0; q < 6; q++)
            tc::mma_bf16(taddr + XS_ACC78, d[q], d[5 - q], id80, c == 0 && ks == 0 && q == 0 ? 0u : 1u);
#pragma unroll
          for (int q = 1; q < 6; q++) tc::mma_bf16(taddr + XS_ACC78, d[q], d[6 - q], id80, 1u);
        }
      };
      auto high = [&](uint32_t st, uint32_t c) {  // the others
        for (int ks = 0; ks < 2; ks++) {
          uint64_t d[XS_NSL];
          slices(st, ks, d);
          const uint32_t first = (c == 0 && ks == 0) ? 0u : 1u;
          tc::mma_bf16(taddr + XS_ACC2, d[0], d[0], id80, first);
          tc::mma_bf16(taddr + XS_X3, d[0], d[1], id96, first);
          tc::mma_bf16(taddr + XS_ACC4, d[0], d[2], id80, first);
          tc::mma_bf16(taddr + XS_ACC4, d[2], d[0], id80, 1u);
          tc::mma_bf16(taddr + XS_ACC4, d[1], d[1], id80, 1u);
          tc::mma_bf16(taddr + XS_X5, d[0], d[3], id96, first);
          tc::mma_bf16(taddr + XS_X5, d[1], d[2], id96, 1u);
#pragma unroll
          for (int q = 0; q < 5; q++) tc::mma_bf16(taddr + XS_ACC6, d[q], d[4 - q], id80, q == 0 ? first : 1u);
        }
      };
      const uint32_t lead = nchunk < (uint32_t)XS_NS ? nchunk : (uint32_t)XS_NS;  // chunks that the stages hold at once
      for (int j = 0; j < nmine && ok; j++) {
        // acc78 is drained first: its products of the staged chunks run while
        // the other accumulators are drained
        ok = j == 0 || xs_wait(&S.empty78, ((uint32_t)j - 1) & 1, abort);
        uint32_t c = 0;
        for (; c < lead && ok; c++) {
          const uint32_t st = (s + c) % XS_NS;
          if (!(ok = xs_wait(&S.full[st], ((s + c) / XS_NS) & 1, abort))) break;
          tc::fence_after_sync();
          low(st, c);
        }
        ok = ok && (j == 0 || xs_wait(&S.accempty, ((uint32_t)j - 1) & 1, abort));
        if (!ok) {
          if (c > 0) {  // the teardown waits for the products issued
            tc::mma_commit(&S.empty[s % XS_NS]);
            mmn[s % XS_NS]++;
          }
          break;
        }
        tc::fence_after_sync();
        for (c = 0; c < nchunk; c++, s++) {
          const uint32_t st = s % XS_NS;
          if (c >= lead) {
            if (!(ok = xs_wait(&S.full[st], (s / XS_NS) & 1, abort))) break;
            tc::fence_after_sync();
            low(st, c);
          }
          high(st, c);
          tc::mma_commit(&S.empty[st]);
          mmn[st]++;
        }
        if (!ok) break;
        tc::mma_commit(&S.accfull);
        accn++;
      }
      if (!ok) S.abort = 1;
      for (int i = 0; i < XS_NS; i++) S.mm_n[i] = mmn[i];
      S.accf_n = accn;
    }
  } else {
    const int t = tid - 64, quarter = warp & 3;
    const bool drain = warp >= 4 && warp < 11 && quarter < 3;  // 4, 5, 6 and 8, 9, 10
    const int half = warp >= 8 ? 1 : 0;                        // columns 0..47, or 48..80
    bool ok = true;
    for (int j = 0; j < nmine && ok; j++) {
      const int64_t e = blockIdx.x + (int64_t)j * gridDim.x;
      double lam = a.lam, mu = a.mu;
      const int inst = a.laws ? __ldg(a.einst + e) : 0;
      if (a.laws) {
        lam = __ldg(&a.laws[inst].par[0]);
        mu = __ldg(&a.laws[inst].par[1]);
      }
      if (a.U && t >= 32 && t < 32 + NE) {  // the element's state
        const DevMesh &m = a.laws ? a.meshes[inst] : a.m;
        const int64_t el = a.laws ? e - __ldg(a.eoff + inst) : e;
        const int b = (t - 32) / 3, d = (t - 32) % 3;
        const int ez = (int)(el % m.nelem[2]), ey = (int)((el / m.nelem[2]) % m.nelem[1]),
                  ex = (int)(el / ((int64_t)m.nelem[1] * m.nelem[2]));
        const int64_t cp = ((int64_t)(ex + b / 9) * m.nbasis[1] + (ey + (b / 3) % 3)) * m.nbasis[2] + (ez + b % 3);
        // less the middle function's value: constants drop out of the law, and
        // what a rigid translation would lose by cancellation is not formed
        const int64_t mid = ((int64_t)(ex + 1) * m.nbasis[1] + (ey + 1)) * m.nbasis[2] + (ez + 1);
        S.u[t - 32] = __ldg(a.U + m.dof_off + 3 * cp + d) - __ldg(a.U + m.dof_off + 3 * mid + d);
      }
      if (t < 32) {  // entry (80, 80)
        const double *row = a.row80 + (size_t)e * nchunk * 32;
        double s = 0.0;
        for (uint32_t c = 0; c < nchunk; c++) {
          const double v = __ldg(row + c * 32 + lane);
          s = fma(v, v, s);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) S.g80 = s;
      }
      if (t >= XS_EPI - 96 && t < XS_EPI - 96 + XS_EXP)
        S.ex[t - (XS_EPI - 96)] = (int)__ldg(a.expo + e * XS_EXP + t - (XS_EPI - 96));
      // the epilogue warps take the same decision (a named-barrier OR): only
      // the draining warps wait for the accumulators
      const uint32_t got = (!drain || xs_wait(&S.accfull, (uint32_t)j & 1, abort)) ? 1u : 0u;
      uint32_t any_failed;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\t"
          "setp.eq.u32 p, %1, 0;\n\t"
          "bar.red.or.pred q, 1, 384, p;\n\t"
          "selp.u32 %0, 1, 0, q;\n\t}\n"
          : "=r"(any_failed)
          : "r"(got)
          : "memory");
      if (any_failed) {
        ok = false;
        break;
      }
      if (drain) {
        tc::fence_after_sync();
        const int r = quarter * 32 + lane;
        const uint32_t ta = taddr + ((uint32_t)(quarter * 32) << 16);
        const int cb1 = half ? 6 : 3;
        // acc78 first: its integers wait in Y's slots, and the next element's
        // products may overwrite it
        for (int cb = half ? 3 : 0; cb < min(cb1, 5); cb++) {
          uint32_t v8[16];
          tc::tmem_ld_32x32b_x16(ta + XS_ACC78 + cb * 16, v8);
          tc::tmem_wait_ld();
          if (r < XS_ROWS)
#pragma unroll
            for (int i = 0; i < 16; i++)
              S.Y[r * XS_YP + cb * 16 + i] = units(v8[i], 0x1p36f, 0);
        }
        tc::fence_before_sync();
        mbar_arrive1(&S.empty78);
        for (int cb = half ? 3 : 0; cb < cb1; cb++) {
          uint32_t v3[16], v5[16];
          tc::tmem_ld_32x32b_x16(ta + XS_X3 + cb * 16, v3);
          tc::tmem_ld_32x32b_x16(ta + XS_X5 + cb * 16, v5);
          if (cb < 5) {
            uint32_t v2[16], v4[16], v6[16];
            tc::tmem_ld_32x32b_x16(ta + XS_ACC2 + cb * 16, v2);
            tc::tmem_ld_32x32b_x16(ta + XS_ACC4 + cb * 16, v4);
            tc::tmem_ld_32x32b_x16(ta + XS_ACC6 + cb * 16, v6);
            tc::tmem_wait_ld();
            if (r < XS_ROWS)
#pragma unroll
              for (int i = 0; i < 16; i++) {
                const int c = cb * 16 + i;
                const long long x = units(v3[i], 0x1p9f, 27) + units(v5[i], 0x1p27f, 9);
                const long long g = units(v2[i], 1.f, 36) + units(v4[i], 0x1p18f, 18) + units(v6[i], 0x1p36f, 0) +
                                    S.Y[r * XS_YP + c];
                // the symmetric part once per pair: at c > r, and at row 80 for its column's sake
                S.Y[r * XS_YP + c] = c == r ? g + 2 * x : ((c > r || r == 80) ? g + x : x);
              }
          } else {  // column 80
            tc::tmem_wait_ld();
            if (r < XS_ROWS) S.Y[r * XS_YP + 80] = units(v3[0], 0x1p9f, 27) + units(v5[0], 0x1p27f, 9);
          }
        }
        tc::fence_before_sync();
        mbar_arrive1(&S.accempty);  // the next element's MMAs may overwrite the accumulators
      }
      if (t == 0) tc::bulk_wait_read();  // the previous element's blocks have left Kb
      asm volatile("bar.sync 1, 384;" ::: "memory");
      if (t < NPAIRS) {
        const int b = S.pb[t], c = S.pc[t];
        double g[3][3];
#pragma unroll
        for (int d = 0; d < 3; d++)
#pragma unroll
          for (int q = 0; q < 3; q++) {
            const int r = 3 * b + d, col = 3 * c + q;
            const long long y = r == col ? S.Y[r * XS_YP + r] : S.Y[r * XS_YP + col] + S.Y[col * XS_YP + r];
            g[d][q] = scaled(y, S.ex[r] + S.ex[col] - 52);
          }
        if (t == NPAIRS - 1) g[2][2] = S.g80;
        const double mtr = mu * (g[0][0] + g[1][1] + g[2][2]);
#pragma unroll
        for (int d = 0; d < 3; d++)
#pragma unroll
          for (int q = 0; q < 3; q++) {
            double k = fma(mu, g[q][d], lam * g[d][q]);
            if (d == q) k += mtr;
            S.Kb[9 * t + 3 * d + q] = k;
          }
      }
      tc::fence_proxy_async();
      asm volatile("bar.sync 1, 384;" ::: "memory");
      if (t == 0 && a.ebuf) tc::bulk_s2g(a.ebuf + e * EBUF, S.Kb, (uint32_t)(EBUF * sizeof(double)));
      if (a.U) {  // row r of K_e u_e, the 27 functions in four parts
        if (t < 4 * NE) {
          const int r = t % NE, part = t / NE, b = r / 3, d = r - 3 * b;
          double s = 0.0;
          for (int c = 7 * part; c < min(7 * part + 7, NB); c++) {
            const bool up = b <= c;
            const double *k = S.Kb + 9 * (up ? pair_index(b, c) : pair_index(c, b)) + (up ? 3 * d : d);
            const int st = up ? 1 : 3;
#pragma unroll
            for (int q = 0; q < 3; q++) s = fma(k[st * q], S.u[3 * c + q], s);
          }
          S.rsum[part][r] = s;
        }
        asm volatile("bar.sync 1, 384;" ::: "memory");
        if (t < NE) a.rbuf[e * NE + t] = (S.rsum[0][t] + S.rsum[1][t]) + (S.rsum[2][t] + S.rsum[3][t]);
      }
    }
    if (t == 0) tc::bulk_wait_all();
    if (!ok) S.abort = 1;
  }
  tc::fence_before_sync();
  __syncthreads();
  if (S.abort && tid == 0) {
    for (int i = 0; i < XS_NS; i++) {
      if (S.cp_n[i] > 0) tc::mbar_wait(&S.full[i], (S.cp_n[i] - 1) & 1, XS_WAIT_LIMIT);
      if (S.mm_n[i] > 0) tc::mbar_wait(&S.empty[i], (S.mm_n[i] - 1) & 1, XS_WAIT_LIMIT);
    }
    if (S.accf_n > 0) tc::mbar_wait(&S.accfull, (S.accf_n - 1) & 1, XS_WAIT_LIMIT);
    atomicCAS(a.err, 0, 2);
    atomicCAS(a.err + 1, 0, 2);
  }
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, XS_TMEM_COLS);
}

static void exact_free(Context *c)
{
  if (c->d_xops) cudaFree(c->d_xops);  // the others lie behind the slices
  c->d_xops = nullptr;
  c->d_xrow = nullptr;
  c->d_xexp = nullptr;
  c->d_xerr = nullptr;
}

// Builds the slices at the first call that wants them (outside a capture) and
// says whether the tensor-core path is available: the linear law, at most 64
// Gauss points, the FP64 geometry cache of every instance, memory for the slices
// (275 KB an element, cache_fits), and digits within the exactness bound.  The tangent needs the element buffers as well (ensure_ebuf).  One
// allocation, and the residual buffer's beside the operand kernel: an allocation
// takes 70 us and 100 to 150 us a GB.
// IGAPGPU_TC_EXACT=0 keeps the FP64 kernel.
bool ensure_exact(Context *c)
{
  if (c->exact_state >= 0) {
    if (c->exact_state == 1) note_user_capture(c);
    return c->exact_state == 1;
  }
  if (stream_capturing(c)) return false;
  RelaxedCapture relaxed;
  c->exact_state = 0;
  const char *env = getenv("IGAPGPU_TC_EXACT");
  const int npts = c->nquad * c->nquad * c->nquad, nchunk = (npts + PW - 1) / PW;
  if (c->law != IGAPGPU_LAW_LINGRAD || nchunk > XS_MAXCH || (env && env[0] == '0')) return false;
  std::vector<Context *> subs;
  std::vector<int64_t> off;
  if (c->batch) {
    if (!batch_instances(c, &subs, &off)) return false;
  } else {
    subs.push_back(c);
    off.push_back(0);
  }
  for (Context *s : subs)
    if (!s->d_geo) return false;
  const size_t nel = (size_t)c->nelem_total;
  // slices, rows 80, exponents, error words and the exactness flag
  const size_t bytes = nel * nchunk * XS_CH_BYTES, rbytes = nel * nchunk * 32 * sizeof(double),
               ebytes = nel * XS_EXP * sizeof(short), total = bytes + rbytes + ebytes + 3 * sizeof(int);
  if (!cache_fits(total + nel * NE * sizeof(double))) return false;
  bool ok = cudaMalloc(&c->d_xops, total) == cudaSuccess;
  if (ok) {
    unsigned char *p = (unsigned char *)c->d_xops + bytes;
    c->d_xrow = (double *)p;
    c->d_xexp = (short *)(p + rbytes);
    c->d_xerr = (int *)(p + rbytes + ebytes);
    ok = cudaMemsetAsync(c->d_xerr, 0, 3 * sizeof(int), c->stream) == cudaSuccess;
  } else {
    c->d_xops = nullptr;
  }
  int *d_bad = ok ? c->d_xerr + 2 : nullptr;
  const size_t smem = sizeof(double) * XS_ROWS * (nchunk * 32 + 1);
  int bad = 1, dev = 0, nsm = 0;
  ok = ok && cudaFuncSetAttribute(exact_operand_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(double) * XS_ROWS * (XS_MAXCH * 32 + 1))) == cudaSuccess &&
       cudaGetDevice(&dev) == cudaSuccess &&
       cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess;
  for (size_t i = 0; ok && i < subs.size(); i++) {
    const Context *s = subs[i];
    const int64_t grid = s->nelem_total < (int64_t)nsm ? s->nelem_total : (int64_t)nsm;
    exact_operand_kernel<<<(unsigned)grid, XO_THREADS, smem, c->stream>>>(
        s->d_geo, npts, nchunk, s->nelem_total, s->par[2],
        (unsigned char *)c->d_xops + (size_t)off[i] * nchunk * XS_CH_BYTES, c->d_xexp + off[i] * XS_EXP,
        c->d_xrow + off[i] * nchunk * 32, d_bad);
    count_launch();
    ok = cudaGetLastError() == cudaSuccess;
  }
  ok = ok && ensure_rbuf(c) && cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, c->stream) == cudaSuccess &&
       cudaStreamSynchronize(c->stream) == cudaSuccess && !bad;
  if (!ok) {
    cudaGetLastError();
    exact_free(c);
    return false;
  }
  c->exact_state = 1;
  return true;
}

// Element matrices and / or residuals of every element into the element
// buffers, then the gathers (RR, vals null: not wanted).
int launch_exact(Context *c, double *RR, double *vals)
{
  int dev = 0, nsm = 0;
  IGAP_CUDA(cudaGetDevice(&dev));
  IGAP_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int npts = c->nquad * c->nquad * c->nquad;
  ExactArgs a;
  a.ops = (const unsigned char *)c->d_xops;
  a.expo = c->d_xexp;
  a.row80 = c->d_xrow;
  a.ebuf = vals ? c->d_ebuf : nullptr;
  a.U = RR ? c->d_Uhist : nullptr;
  a.rbuf = c->d_rbuf;
  a.m = c->devmesh();
  a.nelem = c->nelem_total;
  a.nchunk = (npts + PW - 1) / PW;
  a.lam = c->par[0];
  a.mu = c->par[1];
  a.laws = nullptr;
  a.meshes = nullptr;
  a.eoff = nullptr;
  a.einst = nullptr;
  a.err = c->d_xerr;
  IGAP_CUDA(cudaMemsetAsync(c->d_xerr, 0, sizeof(int), c->stream));
  if (c->batch) batch_element_map(c, &a.laws, &a.meshes, &a.eoff, &a.einst);
  const size_t smem = sizeof(XsSmem) + 1024;
  static bool attr_set = false;
  if (!attr_set) {
    IGAP_CUDA(cudaFuncSetAttribute(exact_tangent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set = true;
  }
  const unsigned grid = (unsigned)(c->nelem_total < nsm ? c->nelem_total : nsm);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (c->prof) {
    IGAP_CUDA(cudaEventCreate(&e0));
    IGAP_CUDA(cudaEventCreate(&e1));
    IGAP_CUDA(cudaEventRecord(e0, c->stream));
  }
  exact_tangent_kernel<<<grid, XS_THREADS, smem, c->stream>>>(a);
  count_launch();
  IGAP_CHECK_LAUNCH();
  if (c->prof) {
    IGAP_CUDA(cudaEventRecord(e1, c->stream));
    c->prof_ev[0].emplace_back(e0, e1);
    c->prof_launches[0]++;
    c->prof_elements[0] += c->nelem_total;
  }
  c->exact_ran = true;
  const int r = RR ? launch_residual_gather(c, RR, 1, c->d_xerr) : IGAPGPU_OK;
  return r || !vals ? r : launch_tangent_gather(c, vals, c->d_xerr);
}

}  // namespace igap
