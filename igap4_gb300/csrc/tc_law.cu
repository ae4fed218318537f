// Split-precision tangent of the reference's laws (TF32x3 on tcgen05) from
// precomputed FP32 law outputs: the GEMM of tc_tangent.cu,
//   K^T[(d,c,e), b] = sum_{(q,k)} A[(d,c,e),(q,k)] R_q[b,k],
//   A[(d,c,e),(q,k)] = sum_l D_q[(d,k),(e,l)] R_q[c,l],
// with the same products in the same order (bit-identical), its stages on
// separate warps and every element in one launch.
//
// The one-stage kernel spent 125 us per element and SM: loads, the products
// D R (1.56 M FMA; a shared-memory load per FMA), the TF32 split and the
// MMAs waited for each other at CTA barriers, and 27 colour launches left SMs
// idle.  Here a CTA of 12 warps per SM:
//  * warps 8-10 (loader): the next chunk's (8 points) law outputs and FP64
//    basis are in their registers while the current chunk is computed; they
//    write both point-minor ([entry][8 points], FP32) when the buffer is free.
//  * warps 0-3 and 4-7 (two groups, derivative slots 0-4 and 5-9): a thread
//    forms A for one (d, k), 7 functions c, 3 components e and 4 points: 84
//    accumulators, 10 shared 16-byte loads per 84 FMA.  The padded strides
//    spread a warp's 8 distinct loads over all banks.  When its slots' MMAs of
//    the previous chunk are done, the group splits into TF32 hi + lo and
//    stores the operands.  Once per element warps 0-3 also copy the previous
//    element's accumulators (243 rows x 27 columns) to the element buffer.
//  * warp 11 (one thread): 30 MMAs (kind::tf32, M128 N32 K8) per group and
//    chunk, in the order chunk, slot, (hi.hi, hi.lo, lo.hi), into one of two
//    accumulator sets.
// Bound: shared-memory bandwidth (MMA operands 19 k, operand stores 11 k,
// products 6 k clocks per element).
// Every mbarrier wait is bounded; a CTA that gives up sets the error word.
#include <cuda_runtime.h>
#include <stdlib.h>

#include "common.cuh"
#include "element.cuh"
#include "df32.cuh"
#include "gather.cuh"
#include "tcgen05.cuh"

namespace igap {

namespace {
constexpr int TL_THREADS = 384;               // 12 warps: 168 registers a thread
constexpr int TL_LOAD = 96;                   // loader threads
constexpr int TL_SLOTS = 5;                   // derivative slots of a group
constexpr int TL_ATILE = 128 * 8 * 4;         // one (K-step, M-tile) block
constexpr int TL_APIECE = TL_SLOTS * 2 * TL_ATILE;
constexpr int TL_BTILE = 32 * 8 * 4;
constexpr int TL_BPIECE = TL_SLOTS * TL_BTILE;
constexpr int TL_CT = 7;                      // functions per thread: 4 x 7 >= 27
constexpr int TL_DROW = 31;                   // entries per (d, k) row, 30 used
constexpr int TL_RROW = 11;                   // entries per function, 10 used
constexpr uint32_t TL_TMEM_COLS = 128;
constexpr uint32_t TL_WAIT_LIMIT = 1u << 26;
constexpr int TL_ND = 19;                     // 16-byte pieces of the law outputs per loader thread (1800 / 96)
constexpr int TL_NR = 23;                     // basis values per loader thread (2160 / 96)

struct TlSmem {
  unsigned char A[2][2 * TL_APIECE];          // [group][hi, lo][slot][M-tile]
  unsigned char B[2][2 * TL_BPIECE];
  float D[30 * TL_DROW * 8];                  // [group 15 + kq 3 + d][10 e + l][point]
  float R[4 * TL_CT * TL_RROW * 8];           // [c][k][point]
  uint64_t in_full, in_empty, a_full[2], a_empty[2], acc_full[2], acc_empty[2];
  uint32_t mm_n[2], accf_n[2];
  uint32_t taddr;
  int abort;
};
static_assert(sizeof(TlSmem) + 1024 <= 227 * 1024, "one CTA per SM");

__device__ __forceinline__ void tl_arrive(uint64_t *mbar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(mbar)) : "memory");
}

__device__ __forceinline__ bool tl_wait(uint64_t *mbar, uint32_t parity, volatile int *abort)
{
  const uint32_t addr = tc::smem_u32(mbar);
  for (uint32_t it = 0; it < TL_WAIT_LIMIT; it++) {
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
  *abort = 1;
  return false;
}

struct TlArgs {
  const double *geo;   // [element][point][GEO_STRIDE]
  const float *D;      // [element][900][npts]
  float *fbuf;         // [element][27 b][243 (d, c, e)]
  int64_t nelem;
  int npts, nchunk;
  int *err;
};

// The loader's registers of one chunk (this thread's share).
struct TlFetch {
  float4 d[TL_ND];
  double r[TL_NR];
};

// VEC: npts a multiple of 4, so that four points are one aligned 16-byte load.
template <bool VEC>
__device__ __forceinline__ void tl_fetch(TlFetch &f, const TlArgs &a, int64_t e, int ch, int t)
{
  {  // 16-byte piece t + 96 i: entry (t / 2) + 48 i, points 4 (t & 1) ..
    const int q = ch * PW + 4 * (t & 1), left = a.npts - q;
    const float *p = a.D + (e * 900 + (t >> 1)) * a.npts + q;
#pragma unroll
    for (int i = 0; i < TL_ND; i++, p += TL_LOAD / 2 * a.npts) {
      f.d[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i == TL_ND - 1 && t >= 1800 - TL_LOAD * (TL_ND - 1)) continue;
      if (VEC) {
        if (left > 0) f.d[i] = __ldg(reinterpret_cast<const float4 *>(p));
      } else {
        if (left > 0) f.d[i].x = __ldg(p);
        if (left > 1) f.d[i].y = __ldg(p + 1);
        if (left > 2) f.d[i].z = __ldg(p + 2);
        if (left > 3) f.d[i].w = __ldg(p + 3);
      }
    }
  }
  // point (t & 7), entry 12 i + t / 8
  const int q = ch * PW + (t & 7);
  const double *g = a.geo + (e * a.npts + (q < a.npts ? q : 0)) * GEO_STRIDE + (t >> 3);
#pragma unroll
  for (int i = 0; i < TL_NR; i++) {
    f.r[i] = 0.0;
    if (q < a.npts && (i < TL_NR - 1 || (t >> 3) < NB * NDD - TL_LOAD / 8 * (TL_NR - 1))) f.r[i] = __ldg(g + TL_LOAD / 8 * i);
  }
}

__device__ __forceinline__ void tl_store(TlSmem &S, const TlFetch &f, int t)
{
#pragma unroll
  for (int i = 0; i < TL_ND; i++) {
    const int v = t + TL_LOAD * i, entry = v >> 1;
    if (v < 1800) {
      const int dk = entry / 30, d = dk / NDD, k = dk % NDD;
      const int row = (k / TL_SLOTS) * 15 + (k % TL_SLOTS) * 3 + d;
      *reinterpret_cast<float4 *>(S.D + (row * TL_DROW + entry % 30) * 8 + 4 * (v & 1)) = f.d[i];
    }
  }
#pragma unroll
  for (int i = 0; i < TL_NR; i++) {
    const int entry = TL_LOAD / 8 * i + (t >> 3);
    if (entry < NB * NDD)
      S.R[((entry / NDD) * TL_RROW + entry % NDD) * 8 + (t & 7)] = f64_to_pair(f.r[i]).x;
  }
}

__device__ __forceinline__ void tl_split(float4 v, float4 &hi, float4 &lo)
{
  hi.x = tc::to_tf32(v.x);
  hi.y = tc::to_tf32(v.y);
  hi.z = tc::to_tf32(v.z);
  hi.w = tc::to_tf32(v.w);
  lo.x = tc::to_tf32(v.x - hi.x);
  lo.y = tc::to_tf32(v.y - hi.y);
  lo.z = tc::to_tf32(v.z - hi.z);
  lo.w = tc::to_tf32(v.w - hi.w);
}
}  // namespace

template <bool VEC>
__global__ void __launch_bounds__(TL_THREADS, 1) tc_law_kernel(TlArgs a)
{
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  TlSmem &S = *reinterpret_cast<TlSmem *>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int *abort = &S.abort;
  if (warp == 0) {
    tc::tmem_alloc(&S.taddr, TL_TMEM_COLS);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    tc::mbar_init(&S.in_full, TL_LOAD);
    tc::mbar_init(&S.in_empty, 256);
    for (int i = 0; i < 2; i++) {
      tc::mbar_init(&S.a_full[i], 128);
      tc::mbar_init(&S.a_empty[i], 1);
      tc::mbar_init(&S.acc_full[i], 1);
      tc::mbar_init(&S.acc_empty[i], 128);
      S.mm_n[i] = S.accf_n[i] = 0;
    }
    S.abort = 0;
  }
  // rows 243..255 of A, 27..31 of B and function 27 of R stay zero
  for (int i = tid; i < (int)(sizeof(S.A) + sizeof(S.B)) / 16; i += TL_THREADS)
    reinterpret_cast<float4 *>(S.A[0])[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i = tid; i < (int)(sizeof(S.D) + sizeof(S.R)) / 16; i += TL_THREADS)
    reinterpret_cast<float4 *>(S.D)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = S.taddr;
  const int nmine = (int64_t)blockIdx.x < a.nelem ? (int)((a.nelem - 1 - blockIdx.x) / gridDim.x) + 1 : 0;
  const int nchunk = a.nchunk;
  auto element = [&](int j) { return blockIdx.x + (int64_t)j * gridDim.x; };
  if (warp < 8) {
    const int g = warp >> 2;
    const int half = lane & 1, cg = (lane >> 1) & 3, dk = (warp & 3) * 4 + (lane >> 3);
    const bool valid = dk < 15;
    const int d = dk % 3, kq = dk / 3;
    const float *Dp = S.D + (g * 15 + (valid ? dk : 0)) * TL_DROW * 8 + 4 * half;
    const float *Rp = S.R + cg * TL_CT * TL_RROW * 8 + 4 * half;
    const int t = tid & 127;
    unsigned char *Ag = S.A[g], *Bg = S.B[g];
    // accumulators of element j -> element buffer
    auto epilogue = [&](int j) {
      bool got = tl_wait(&S.acc_full[j & 1], (uint32_t)(j >> 1) & 1, abort);
      got = __all_sync(0xffffffffu, got);
      if (!got) return false;
      tc::fence_after_sync();
      float *out = a.fbuf + element(j) * (int64_t)(NB * 243);
      for (int mt = 0; mt < 2; mt++) {
        uint32_t v[32];
        tc::tmem_ld_32x32b_x32(taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)((j & 1) * 64 + mt * 32), v);
        const int r = mt * 128 + (warp * 32) + lane;
        if (r < 243)
#pragma unroll
          for (int b = 0; b < NB; b++) out[b * 243 + r] = __uint_as_float(v[b]);
      }
      tc::fence_before_sync();
      tl_arrive(&S.acc_empty[j & 1]);
      return true;
    };
    uint32_t n = 0;
    bool ok = true;
    for (int j = 0; j < nmine && ok; j++)
      for (int ch = 0; ch < nchunk; ch++, n++) {
        if (!__all_sync(0xffffffffu, tl_wait(&S.in_full, n & 1, abort))) {
          ok = false;
          break;
        }
        float acc[3][TL_CT][4];
#pragma unroll
        for (int e = 0; e < 3; e++)
#pragma unroll
          for (int c = 0; c < TL_CT; c++)
#pragma unroll
            for (int p = 0; p < 4; p++) acc[e][c][p] = 0.f;
#pragma unroll 2
        for (int l = 0; l < NDD; l++) {
          float4 dv[3];
#pragma unroll
          for (int e = 0; e < 3; e++) dv[e] = *reinterpret_cast<const float4 *>(Dp + (NDD * e + l) * 8);
#pragma unroll
          for (int c = 0; c < TL_CT; c++) {
            const float4 rv = *reinterpret_cast<const float4 *>(Rp + (c * TL_RROW + l) * 8);
#pragma unroll
            for (int e = 0; e < 3; e++) {
              acc[e][c][0] = fmaf(dv[e].x, rv.x, acc[e][c][0]);
              acc[e][c][1] = fmaf(dv[e].y, rv.y, acc[e][c][1]);
              acc[e][c][2] = fmaf(dv[e].z, rv.z, acc[e][c][2]);
              acc[e][c][3] = fmaf(dv[e].w, rv.w, acc[e][c][3]);
            }
          }
        }
        // sources of the B operand: 27 functions x 5 slots x 2 halves
        float4 bsrc[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
          const int v = t + 128 * i;
          if (v < 270) bsrc[i] = *reinterpret_cast<const float4 *>(
              S.R + ((v / 10) * TL_RROW + g * TL_SLOTS + (v % 10) / 2) * 8 + 4 * (v & 1));
        }
        tl_arrive(&S.in_empty);
        if (n > 0 && !__all_sync(0xffffffffu, tl_wait(&S.a_empty[g], (n - 1) & 1, abort))) {
          ok = false;
          break;
        }
        if (valid) {
#pragma unroll
          for (int c = 0; c < TL_CT; c++)
#pragma unroll
            for (int e = 0; e < 3; e++) {
              const int cc = cg * TL_CT + c;
              if (cc < NB) {
                const int r = 81 * d + 3 * cc + e;
                const uint32_t off = (uint32_t)((kq * 2 + (r >> 7)) * TL_ATILE) + tc::kmajor_off(r & 127, 4 * half);
                float4 hi, lo;
                tl_split(make_float4(acc[e][c][0], acc[e][c][1], acc[e][c][2], acc[e][c][3]), hi, lo);
                *reinterpret_cast<float4 *>(Ag + off) = hi;
                *reinterpret_cast<float4 *>(Ag + TL_APIECE + off) = lo;
              }
            }
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
          const int v = t + 128 * i;
          if (v < 270) {
            const uint32_t off = (uint32_t)(((v % 10) / 2) * TL_BTILE) + tc::kmajor_off(v / 10, 4 * (v & 1));
            float4 hi, lo;
            tl_split(bsrc[i], hi, lo);
            *reinterpret_cast<float4 *>(Bg + off) = hi;
            *reinterpret_cast<float4 *>(Bg + TL_BPIECE + off) = lo;
          }
        }
        tc::fence_proxy_async();
        tl_arrive(&S.a_full[g]);
        if (g == 0 && ch == 0 && j > 0 && !epilogue(j - 1)) {
          ok = false;
          break;
        }
      }
    if (g == 0 && ok && nmine > 0) epilogue(nmine - 1);
  } else if (warp < 11) {
    const int t = tid - 256;
    bool ok = true;
    TlFetch f;
    uint32_t n = 0;
    if (nmine > 0) tl_fetch<VEC>(f, a, element(0), 0, t);
    for (int j = 0; j < nmine && ok; j++) {
      for (int ch = 0; ch < nchunk && ok; ch++, n++) {
        if (n > 0 && !tl_wait(&S.in_empty, (n - 1) & 1, abort)) {
          ok = false;
          break;
        }
        tl_store(S, f, t);
        tl_arrive(&S.in_full);
        if (ch + 1 < nchunk) tl_fetch<VEC>(f, a, element(j), ch + 1, t);
        else if (j + 1 < nmine) tl_fetch<VEC>(f, a, element(j + 1), 0, t);
      }
    }
  } else if (lane == 0) {
    const uint32_t idesc = tc::instr_desc(2, 128, 32);
    uint32_t n = 0, mmn[2] = {0, 0}, accn[2] = {0, 0};
    bool ok = true;
    for (int j = 0; j < nmine && ok; j++) {
      if (j >= 2 && !tl_wait(&S.acc_empty[j & 1], (uint32_t)((j >> 1) - 1) & 1, abort)) {
        ok = false;
        break;
      }
      const uint32_t acc0 = taddr + (uint32_t)((j & 1) * 64);
      for (int ch = 0; ch < nchunk && ok; ch++, n++)
        for (int g = 0; g < 2; g++) {
          if (!tl_wait(&S.a_full[g], n & 1, abort)) {
            ok = false;
            break;
          }
          tc::fence_after_sync();
          const uint32_t ab = tc::smem_u32(S.A[g]), bb = tc::smem_u32(S.B[g]);
          for (int kt = 0; kt < TL_SLOTS; kt++)
            for (int mt = 0; mt < 2; mt++)
              for (int pp = 0; pp < 3; pp++) {  // hi.hi, hi.lo, lo.hi
                const int pa = (pp == 2) ? 1 : 0, pb = (pp == 1) ? 1 : 0;
                const uint64_t ad = tc::smem_desc(ab + pa * TL_APIECE + (kt * 2 + mt) * TL_ATILE, 128, 256);
                const uint64_t bd = tc::smem_desc(bb + pb * TL_BPIECE + kt * TL_BTILE, 128, 256);
                const uint32_t accum = (ch == 0 && g == 0 && kt == 0 && pp == 0) ? 0u : 1u;
                tc::mma_tf32(acc0 + (uint32_t)(mt * 32), ad, bd, idesc, accum);
              }
          tc::mma_commit(&S.a_empty[g]);
          mmn[g]++;
        }
      if (!ok) break;
      tc::mma_commit(&S.acc_full[j & 1]);
      accn[j & 1]++;
    }
    for (int i = 0; i < 2; i++) {
      S.mm_n[i] = mmn[i];
      S.accf_n[i] = accn[i];
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (S.abort && tid == 0) {
    // MMAs still in flight finish before the tensor memory is freed
    for (int i = 0; i < 2; i++) {
      if (S.mm_n[i] > 0) tc::mbar_wait(&S.a_empty[i], (S.mm_n[i] - 1) & 1, TL_WAIT_LIMIT);
      if (S.accf_n[i] > 0) tc::mbar_wait(&S.acc_full[i], (S.accf_n[i] - 1) & 1, TL_WAIT_LIMIT);
    }
    atomicCAS(a.err, 0, 2);
  }
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, TL_TMEM_COLS);
}

// Whether the reference law's split tangent runs here: precomputed FP32 law
// outputs, the FP64 geometry cache, and room for the FP32 element buffers
// (26 KB an element).  IGAPGPU_TC_PREFETCH=0 keeps the one-stage kernel.
bool tc_law_applies(Context *c, const DevLaw &L)
{
  const char *pf = getenv("IGAPGPU_TC_PREFETCH");
  return c->law != IGAPGPU_LAW_LINGRAD && c->d_geo && L.preR && L.preDf && !(pf && pf[0] == '0') && ensure_fbuf(c);
}

int launch_tc_law(Context *c, double *vals, const DevLaw &L)
{
  int dev = 0, nsm = 0;
  IGAP_CUDA(cudaGetDevice(&dev));
  IGAP_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  TlArgs a;
  a.geo = c->d_geo;
  a.D = L.preDf;
  a.fbuf = c->d_fbuf;
  a.nelem = c->nelem_total;
  a.npts = c->nquad * c->nquad * c->nquad;
  a.nchunk = (a.npts + PW - 1) / PW;
  a.err = c->d_err;
  const bool vec = a.npts % 4 == 0;
  auto kern = vec ? tc_law_kernel<true> : tc_law_kernel<false>;
  const size_t smem = sizeof(TlSmem) + 1024;
  static bool attr[2] = {false, false};
  if (!attr[vec]) {
    IGAP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr[vec] = true;
  }
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (c->prof) {
    IGAP_CUDA(cudaEventCreate(&e0));
    IGAP_CUDA(cudaEventCreate(&e1));
    IGAP_CUDA(cudaEventRecord(e0, c->stream));
  }
  kern<<<(unsigned)(c->nelem_total < nsm ? c->nelem_total : nsm), TL_THREADS, smem, c->stream>>>(a);
  count_launch();
  IGAP_CHECK_LAUNCH();
  if (c->prof) {
    IGAP_CUDA(cudaEventRecord(e1, c->stream));
    c->prof_ev[1].emplace_back(e0, e1);
    c->prof_launches[1]++;
    c->prof_elements[1] += c->nelem_total;
  }
  return launch_tangent_gather_f32(c, vals);
}

}  // namespace igap
