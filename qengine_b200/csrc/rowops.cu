// Row-wise kernels of a decode pass: embedding gather, zero-centred RMSNorm with fused residual,
// BF16 GEMV (off the W4 path), SwiGLU and the vocabulary argmax.
// Boundary: these replace launch_embed .. launch_argmax of the reference (csrc/ops.h:6-14).
// Every kernel treats rows independently and uses a row-count-independent operation order, so
// row r of an n-row call is bit-identical to a 1-row call (the verify == plain-decode property).
#include <algorithm>

#include "common.cuh"
#include "../../include/qengine_b200.h"

namespace qb {
namespace {

// ---------------------------------------------------------------------------------------------
// Embedding gather. Semantics of embed_kernel (reference csrc/basic.cu:16-26): out[r] =
// table[tok[r]], ids outside [0, V) give zeros. 16-byte copies when the rows allow it.
// ---------------------------------------------------------------------------------------------
__global__ void embed_rows_kernel(const bf16* table, const int* tok,
                                  bf16* out, int H, int V, long ldo, int vec) {
  dep_release();
  dep_wait();
  const int r = blockIdx.y;
  const int id = tok[r];
  const bool ok = id >= 0 && id < V;
  bf16* dst = out + (long)r * ldo;
  const bf16* src = table + (size_t)(ok ? id : 0) * H;
  if (vec) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;  // 8 elements per thread
    if (i * 8 < H)
      reinterpret_cast<uint4*>(dst)[i] = ok ? __ldg(reinterpret_cast<const uint4*>(src) + i)
                                            : make_uint4(0, 0, 0, 0);
  } else {
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) * 8, e = min(i + 8, H); i < e; ++i)
      dst[i] = ok ? src[i] : tobf16(0.f);
  }
}

// ---------------------------------------------------------------------------------------------
// RMSNorm1p (+ residual). Semantics of rmsnorm1p_kernel (reference csrc/basic.cu:29-54,
// python/qengine/reference.py:132-136): x = bf16(x + delta) written back when delta is given,
// out = bf16(x * rsqrt(mean x^2 + eps) * (1 + w)), fp32 math, one rounding.
// One CTA per row; a thread owns 8-element packets at stride blockDim, kept in registers
// (PKT packets, enough for H <= 8 * PKT * blockDim) so the row is read once.
// ---------------------------------------------------------------------------------------------
template <int PKT>
__global__ void __launch_bounds__(256)
rmsnorm1p_vec_kernel(bf16* x, const bf16* delta,
                     const bf16* w, bf16* out, int H, long ldx, long ldd,
                     long ldo, float eps) {
  dep_release();
  __shared__ float scratch[32];
  const int row = blockIdx.x, npk = H >> 3;
  // the weight is a constant: fetch it while the producer of x is still running
  uint4 wq[PKT];
#pragma unroll
  for (int p = 0; p < PKT; ++p) {
    const int i = threadIdx.x + p * blockDim.x;
    if (i < npk) wq[p] = __ldg(reinterpret_cast<const uint4*>(w) + i);
  }
  dep_wait();
  uint4* xr = reinterpret_cast<uint4*>(x + (long)row * ldx);
  const uint4* dr = delta ? reinterpret_cast<const uint4*>(delta + (long)row * ldd) : nullptr;
  float v[PKT][8];
  float ss = 0.f;
#pragma unroll
  for (int p = 0; p < PKT; ++p) {
    const int i = threadIdx.x + p * blockDim.x;
    if (i < npk) {
      widen8(xr[i], v[p]);
      if (dr) {
        float d[8];
        widen8(dr[i], d);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[p][e] = rnd(v[p][e] + d[e]);
        xr[i] = narrow8(v[p]);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) ss = fmaf(v[p][e], v[p][e], ss);
    }
  }
  const float inv = rsqrtf(block_allsum(ss, scratch) / (float)H + eps);
  uint4* orow = reinterpret_cast<uint4*>(out + (long)row * ldo);
#pragma unroll
  for (int p = 0; p < PKT; ++p) {
    const int i = threadIdx.x + p * blockDim.x;
    if (i < npk) {
      float g[8], y[8];
      widen8(wq[p], g);
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] = v[p][e] * inv * (1.0f + g[e]);
      orow[i] = narrow8(y);
    }
  }
}

// Any H, any alignment: two passes over the row, same arithmetic per element.
__global__ void __launch_bounds__(256)
rmsnorm1p_any_kernel(bf16* x, const bf16* delta,
                     const bf16* w, bf16* out, int H, long ldx, long ldd,
                     long ldo, float eps) {
  dep_release();
  dep_wait();
  __shared__ float scratch[32];
  const int row = blockIdx.x;
  bf16* xr = x + (long)row * ldx;
  float ss = 0.f;
  for (int c = threadIdx.x; c < H; c += blockDim.x) {
    float v = tofloat(xr[c]);
    if (delta) {
      v = rnd(v + tofloat(delta[(long)row * ldd + c]));
      xr[c] = tobf16(v);  // re-read below by the same thread only
    }
    ss = fmaf(v, v, ss);
  }
  const float inv = rsqrtf(block_allsum(ss, scratch) / (float)H + eps);
  for (int c = threadIdx.x; c < H; c += blockDim.x)
    out[(long)row * ldo + c] = tobf16(tofloat(xr[c]) * inv * (1.0f + tofloat(w[c])));
}

// ---------------------------------------------------------------------------------------------
// BF16 GEMV, NR = 1..8 rows, WR weight rows per warp, weights read once for all rows. Semantics of
// gemv_bf16_kernel (reference csrc/basic.cu:99-155). A lane always walks k in the same order
// whatever NR and WR are, so neither shows in the result.
// Bound by HBM (2 bytes per weight) for one row; with more rows by issue slots, since every 16 bytes of
// weights cost the load and the widening of NR x 16 bytes of activations. Two weight rows per warp share
// them (which sizes take which: gemv_rows_per_warp), and weights leave no L1 lines. 62,080 x 5,120, us before (one
// row per warp) -> now:
// 1 row 90 -> 90, 3 rows 121 -> 99 (6.4 TB/s; 137 -> 102 called on its own), 5 rows 170 -> 134, 8 rows 270 -> 206.
// Four rows per warp: the same at this size, 20 % slower at 1,000 rows x 3. Multiply-adds in pairs (even
// and odd k, fma.rn.f32x2) take another 4 % (3 rows) to 12 % (8 rows) off, but the second accumulator costs
// a single row 2 to 9 % where K is some hundreds, and rows must not depend on how many there are.
// ---------------------------------------------------------------------------------------------
constexpr int kGemvRows = 8;  // weight rows per block: fewer make short rows (K of some hundreds) pay for the blocks

__device__ __forceinline__ uint4 ld_once(const uint4* p) {  // constant and read once: no L1 line, x stays there
  uint4 v;
  asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <int NR, int WR>
__global__ void __launch_bounds__(kGemvRows / WR * 32)
gemv_bf16_rows_kernel(const bf16* W, const bf16* x,
                      bf16* out, int N, int K, long ldx, long ldo) {
  constexpr int U = 4;  // packets of a row in flight
  dep_release();
  const int lane = threadIdx.x & 31;
  const int j = blockIdx.x * kGemvRows + (threadIdx.x >> 5) * WR;
  if (j >= N) { dep_wait(); return; }
  const int npk = K >> 3;
  const uint4* wr[WR];  // rows beyond the last one repeat it and are not stored
#pragma unroll
  for (int i = 0; i < WR; ++i) wr[i] = reinterpret_cast<const uint4*>(W + (size_t)(WR == 1 ? j : min(j + i, N - 1)) * K);
  float acc[WR][NR];
#pragma unroll
  for (int i = 0; i < WR; ++i)
#pragma unroll
    for (int r = 0; r < NR; ++r) acc[i][r] = 0.f;
  bool waited = false;
  for (int p0 = lane; p0 < npk; p0 += 32 * U) {
    uint4 wq[U][WR];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < WR; ++i)
        if (p0 + 32 * u < npk) wq[u][i] = NR == 1 ? __ldg(wr[i] + p0 + 32 * u) : ld_once(wr[i] + p0 + 32 * u);
    if (!waited) { dep_wait(); waited = true; }  // weights are constants; x is produced upstream
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (p0 + 32 * u < npk) {
        float wf[WR][8];
#pragma unroll
        for (int i = 0; i < WR; ++i) widen8(wq[u][i], wf[i]);
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          float xf[8];
          widen8(reinterpret_cast<const uint4*>(x + (long)r * ldx)[p0 + 32 * u], xf);
#pragma unroll
          for (int e = 0; e < 8; ++e)
#pragma unroll
            for (int i = 0; i < WR; ++i) acc[i][r] = fmaf(wf[i][e], xf[e], acc[i][r]);
        }
      }
    }
  }
  if (!waited) dep_wait();
#pragma unroll
  for (int i = 0; i < WR; ++i) {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const float s = warp_allsum(acc[i][r]);
      if (lane == 0 && j + i < N) out[(long)r * ldo + j + i] = tobf16(s);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// SwiGLU on unfused [gate | up] rows: bf16(bf16(silu(g)) * u) (reference csrc/basic.cu:157-170).
// ---------------------------------------------------------------------------------------------
__global__ void swiglu_rows_kernel(const bf16* gu, bf16* out, int I,
                                   long ldg, long ldo) {
  dep_release();
  dep_wait();
  const int r = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= I) return;
  const bf16* g = gu + (long)r * ldg;
  const float s = rnd(silu_acc(tofloat(g[i])));
  out[(long)r * ldo + i] = tobf16(s * tofloat(g[I + i]));
}

// ---------------------------------------------------------------------------------------------
// Argmax, torch semantics (reference csrc/basic.cu:173-239): NaN beats everything, then the
// larger value, then the lower index. A candidate is (value, index); index INT_MAX = "none".
// Stage 1: grid (nb, rows), CTA b scans a contiguous slab of the row with 16-byte loads when
// aligned. Stage 2: one CTA per row merges the nb candidates and maps through idmap.
// ---------------------------------------------------------------------------------------------
constexpr int kNone = 0x7fffffff;

__device__ __forceinline__ bool beats(float a, int ia, float b, int ib) {
  const bool an = a != a, bn = b != b;
  if (an != bn) return an;
  if (!an && a != b) return a > b;
  return ia < ib;
}
__device__ __forceinline__ void merge(float& v, int& i, float ov, int oi) {
  if (beats(ov, oi, v, i)) { v = ov; i = oi; }
}
__device__ __forceinline__ void block_best(float& v, int& i, float* sv, int* si) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    merge(v, i, __shfl_xor_sync(0xffffffffu, v, o), __shfl_xor_sync(0xffffffffu, i, o));
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) { sv[w] = v; si[w] = i; }
  __syncthreads();
  if (w == 0) {
    v = lane < nw ? sv[lane] : -INFINITY;
    i = lane < nw ? si[lane] : kNone;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      merge(v, i, __shfl_xor_sync(0xffffffffu, v, o), __shfl_xor_sync(0xffffffffu, i, o));
  }
}

__global__ void __launch_bounds__(256)
argmax_slab_kernel(const bf16* x, int n, long ldx, float* pv,
                   int* pi) {
  dep_release();
  dep_wait();
  __shared__ float sv[32];
  __shared__ int si[32];
  const int row = blockIdx.y, nb = gridDim.x;
  const bf16* xr = x + (long)row * ldx;
  // slab of this CTA, in 8-element packets
  const int npk = (n + 7) >> 3;
  const int per = (npk + nb - 1) / nb;
  const int p0 = blockIdx.x * per, p1 = min(npk, p0 + per);
  const bool vec = ((reinterpret_cast<uintptr_t>(xr) & 15) == 0);
  float v = -INFINITY;
  int i = kNone;
  for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
    const int k0 = p * 8;
    if (vec && k0 + 8 <= n) {
      float f[8];
      widen8(reinterpret_cast<const uint4*>(xr)[p], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) merge(v, i, f[e], k0 + e);
    } else {
      for (int k = k0; k < min(k0 + 8, n); ++k) merge(v, i, tofloat(xr[k]), k);
    }
  }
  block_best(v, i, sv, si);
  if (threadIdx.x == 0) { pv[row * nb + blockIdx.x] = v; pi[row * nb + blockIdx.x] = i; }
}

__global__ void __launch_bounds__(256)
argmax_final_kernel(const float* pv, const int* pi, int nb,
                    int* out, const int* idmap, float* out_v, int base) {
  dep_release();
  dep_wait();
  __shared__ float sv[32];
  __shared__ int si[32];
  const int row = blockIdx.x;
  float v = -INFINITY;
  int i = kNone;
  for (int k = threadIdx.x; k < nb; k += blockDim.x) merge(v, i, pv[row * nb + k], pi[row * nb + k]);
  block_best(v, i, sv, si);
  if (threadIdx.x == 0) {
    const int a = i == kNone ? 0 : i;  // a row of -inf only: index 0, like torch
    out[row] = (idmap ? idmap[a] : a) + base;
    if (out_v) out_v[row] = v;
  }
}

// Best of nparts (value, index) candidates per row; vals / idx are [nparts, rows]. Used to merge
// the per-rank winners of a vocabulary-split lm_head: same ordering rule as the local argmax, so
// the result equals the argmax over the whole vocabulary (ties go to the lowest global index).
__global__ void argmax_merge_kernel(const float* vals, const int* idx, int nparts, int rows, int* out) {
  dep_release();
  dep_wait();
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= rows) return;
  float v = vals[row];
  int i = idx[row];
  for (int p = 1; p < nparts; ++p) merge(v, i, vals[p * rows + row], idx[p * rows + row]);
  out[row] = i;
}


inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline bool pdl_on() { return pdl_launch_enabled() && pdl_trigger_enabled(); }

}  // namespace
}  // namespace qb

using namespace qb;

extern "C" int qe_embed(const void* table, const int* tok, void* out, int n, int H, int V, long ldo,
                        void* stream) {
  if (n < 1 || H < 1) return QE_ERR_ARG;
  const int vec = (H % 8 == 0) && (ldo % 8 == 0) && aligned16(table) && aligned16(out);
  const int per_block = 256 * 8;
  return (int)launch(embed_rows_kernel, dim3((H + per_block - 1) / per_block, n), dim3(256), 0,
                     (cudaStream_t)stream, pdl_on(), (const bf16*)table, tok, (bf16*)out, H, V, ldo,
                     vec);
}

extern "C" int qe_rmsnorm1p(void* x, const void* delta, const void* w, void* out, int rows, int H,
                            long ldx, long ldd, long ldo, float eps, void* stream) {
  if (rows < 1 || H < 1) return QE_ERR_ARG;
  const bool vec = H % 8 == 0 && ldx % 8 == 0 && ldo % 8 == 0 && (!delta || ldd % 8 == 0) &&
                   aligned16(x) && aligned16(out) && aligned16(w) && (!delta || aligned16(delta));
  cudaStream_t s = (cudaStream_t)stream;
  bf16* X = (bf16*)x;
  const bf16 *D = (const bf16*)delta, *W = (const bf16*)w;
  bf16* O = (bf16*)out;
  if (vec && H <= 8 * 256 * 4) {
    const int npk = H / 8;
    if (npk <= 256) {
      const int threads = std::max(32, (npk + 31) / 32 * 32);
      return (int)launch(rmsnorm1p_vec_kernel<1>, dim3(rows), dim3(threads), 0, s, pdl_on(), X, D, W,
                         O, H, ldx, ldd, ldo, eps);
    }
    if (npk <= 512)
      return (int)launch(rmsnorm1p_vec_kernel<2>, dim3(rows), dim3(256), 0, s, pdl_on(), X, D, W, O,
                         H, ldx, ldd, ldo, eps);
    return (int)launch(rmsnorm1p_vec_kernel<4>, dim3(rows), dim3(256), 0, s, pdl_on(), X, D, W, O, H,
                       ldx, ldd, ldo, eps);
  }
  return (int)launch(rmsnorm1p_any_kernel, dim3(rows), dim3(256), 0, s, pdl_on(), X, D, W, O, H, ldx,
                     ldd, ldo, eps);
}

// Weight rows per warp. Two share the activations, but both forms put 8 rows into a block, so half the
// warps keep loads in flight; and a block costs more, so a last wave of few blocks does, too. Resident blocks per
// SM by their registers: one row per warp 5 (2, 3 activation rows), 4 (4 to 7); two rows per warp 7 (2, 3),
// 6 (4), 5 (5 to 7), 4 (8). Measured, one / two rows per warp, us (148 SMs, graph of 24 calls):
//   * a single row: nothing to share. 8 rows: two (1,000 x 5,120 18.6 / 14.5; 62,080 x 5,120 270 / 206).
//   * 2 to 4 rows: one, except where only two fit into one wave (6,144 x 5,120 16.8 / 13.1, 23.0 / 16.8, 21.3 / 19.6)
//     and behind two full waves of one (three for 4 rows: 12,288 x 5,120, 3 rows 30.8 / 30.6; 62,080 124 / 98;
//     14,336 x 5,120, 4 rows 39.7 / 39.4; 62,080 155 / 120). Between: 8,192 x 5,120, 4 rows 23.1 / 34.0; 10,240 x 5,120,
//     2 rows 20.6 / 23.7. 2 rows, which win least, lose in a thin third wave too (17,300 x 3,584 23.2 / 25.0).
//     Short rows gain from sharing earlier (8,700 x 512, 2 rows 3.6 / 3.2; 13,600 x 1,280, 4 rows 13.1 / 11.4; not yet
//     at 9,500 x 1,440: 7.4 / 8.1, 11.0 / 12.4).
//   * 5 to 7 rows: two (1,000 x 5,120 13.1 / 12.3, 14.6 / 13.5, 17.5 / 15.8; 62,080, 5 rows 174 / 134), except for a
//     thin second wave of long rows (6,144 x 5,120 27.8 / 29.2, 30.1 / 31.5, 34.6 / 35.3; x 800 the other way,
//     7.3 / 7.2, 8.1 / 7.7, 9.1 / 8.7) and 5 rows where one per warp just fits (4,096 x 5,120 15.5 / 16.5; x 2,560
//     9.2 / 8.9).
static int gemv_rows_per_warp(int nr, int N, int K) {
  const int blocks = (N + kGemvRows - 1) / kGemvRows, sms = qe_sm_count();
  auto within = [&](int lo, int hi) { return blocks > lo * sms && blocks <= hi * sms; };  // blocks per SM in (lo, hi]
  auto above = [&](int lo) { return blocks > lo * sms; };
  const bool brief = K < 1536;
  switch (nr) {
    case 1: return 1;
    case 2: return within(5, 7) || (brief ? above(K <= 640 ? 7 : 9) : within(10, 14) || above(15)) ? 2 : 1;
    case 3: return within(5, 7) || above(brief ? K <= 640 ? 7 : 9 : 10) ? 2 : 1;
    case 4: return within(4, 6) || above(brief ? K <= 640 ? 8 : 9 : 12) ? 2 : 1;
    case 5: return (within(3, 4) && K >= 4096) || (within(5, 8) && K >= 2048) ? 1 : 2;
    case 6: return within(5, 7) && K >= 3584 ? 1 : 2;
    case 7: return within(5, 7) && K >= 2048 ? 1 : 2;
    default: return 2;
  }
}

extern "C" int qe_gemv_bf16(const void* W, const void* x, void* out, int nr, int N, int K, long ldx,
                            long ldo, void* stream) {
  if (nr < 1 || nr > QE_MAX_ROWS || K % 8 || N < 1) return QE_ERR_ARG;
  if (!aligned16(W) || !aligned16(x) || ldx % 8) return QE_ERR_ARG;
  const int wr = gemv_rows_per_warp(nr, N, K);
  const dim3 grid((N + kGemvRows - 1) / kGemvRows), block(kGemvRows / wr * 32);
  cudaStream_t s = (cudaStream_t)stream;
  const bf16 *w = (const bf16*)W, *xx = (const bf16*)x;
  bf16* o = (bf16*)out;
  switch (nr) {
#define QB_ROWS(R) \
  case R: return (int)launch(wr == 1 ? gemv_bf16_rows_kernel<R, R == 8 ? 2 : 1> : gemv_bf16_rows_kernel<R, R == 1 ? 1 : 2>, grid, block, 0, s, pdl_on(), w, xx, o, N, K, ldx, ldo);
    QB_ROWS(1) QB_ROWS(2) QB_ROWS(3) QB_ROWS(4) QB_ROWS(5) QB_ROWS(6) QB_ROWS(7) QB_ROWS(8)
#undef QB_ROWS
  }
  return QE_ERR_ARG;
}

extern "C" int qe_swiglu(const void* gu, void* out, int n, int I, long ldg, long ldo, void* stream) {
  if (n < 1 || I < 1) return QE_ERR_ARG;
  return (int)launch(swiglu_rows_kernel, dim3((I + 255) / 256, n), dim3(256), 0,
                     (cudaStream_t)stream, pdl_on(), (const bf16*)gu, (bf16*)out, I, ldg, ldo);
}

extern "C" int qe_argmax_v(const void* x, int rows, int n, long ldx, float* pv, int* pi, int nb,
                           int* out, float* out_v, const int* idmap, int base, void* stream) {
  if (rows < 1 || n < 1 || nb < 1) return QE_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  int e = (int)launch(argmax_slab_kernel, dim3(nb, rows), dim3(256), 0, s, pdl_on(),
                      (const bf16*)x, n, ldx, pv, pi);
  if (e) return e;
  return (int)launch(argmax_final_kernel, dim3(rows), dim3(256), 0, s, pdl_on(), (const float*)pv,
                     (const int*)pi, nb, out, idmap, out_v, base);
}

extern "C" int qe_argmax(const void* x, int rows, int n, long ldx, float* pv, int* pi, int nb,
                         int* out, const int* idmap, void* stream) {
  return qe_argmax_v(x, rows, n, ldx, pv, pi, nb, out, nullptr, idmap, 0, stream);
}

extern "C" int qe_argmax_merge(const float* vals, const int* idx, int nparts, int rows, int* out,
                               void* stream) {
  if (nparts < 1 || rows < 1) return QE_ERR_ARG;
  return (int)launch(argmax_merge_kernel, dim3((rows + 31) / 32), dim3(32), 0, (cudaStream_t)stream,
                     pdl_on(), vals, idx, nparts, rows, out);
}

