// Packing a weight matrix into the W4 wire format on the GPU (qe_w4_pack): int4 symmetric
// round-to-nearest, group 128 along K, one fp16 scale per (row, group), gate / up rows interleaved
// in blocks of 8. The format and the rounding are those of the torch packer in quant.py (the
// reference's python/qengine/quant.py:41-148), bit for bit:
//
//   scale = fp16(max|w| * 2/15),  code = clamp(rint(w / scale) + 8, 0, 15)   (8 where scale is not > 0)
//
// A warp packs one unit, 16 rows x 128 k: lane 4 r + t holds rows r and r + 8, k = 64 c + 16 t + 0..15
// of both 64-k chunks c, which are exactly the 2 x 16 bytes it writes, so nothing is exchanged but
// the two row maxima (over the four lanes of a row). Every weight is read once and every word written
// once, whole sectors on both sides. Bound: HBM. The torch packer goes over the matrix about forty times
// (int64 code words among them): 7.9 ms for a bf16 gate/up pair of 17,408 x 5,120; this kernel 0.080 ms
// (5.6 TB/s; the floor at the copy rate is 0.069 ms). Four operations per weight, two weights to an
// instruction; with a second pass of divisions for every unit that holds a half it was 0.157 ms. Four blocks per SM
// cap the 16-bit types at 64 registers, of which they spill 88 bytes; three blocks without spills take 0.087 ms.
//
// The quotient is only ever rounded to a whole number, so one division per group is enough: w times
// the reciprocal is within 4e-6 of the quotient where the code is not clamped (|w / scale| <= 8, four
// roundings of 2^-24 relative each).
//   * 16-bit types: w = a 2^p and scale = b 2^q with a, b < 2^11, so a quotient that is not exactly half way
//     between two whole numbers is at least 1.2e-4 away from it ((2 a 2^(p-q) - (2 k + 1) b) / (2 b), whose
//     numerator is a multiple of 1/2 or larger). Rounded to a multiple of 2^-14 first, the approximation of a
//     half is the half again, and nothing else is: rounding that, ties to even, gives the code. Halves
//     are common, not rare: a bf16 row maximum that 15 divides gives an exact scale and, where it is
//     negative, the quotient -7.5. (Quantised again with divisions, as below, those were half of all warps.)
//   * fp32: only where the approximation lies within 1e-5 of a half can the rounding differ (2e-5 of
//     random weights): a lane that has one among its 64 weights quantises them all again with divisions.
#include <type_traits>

#include "w4_dev.cuh"

namespace qb {
namespace {

struct PackArgs {
  const void* w[2];  // source of tile rows 0..7 and 8..15 (the same matrix unless gate / up)
  long ld[2];
  int M, K;          // rows of a source, logical K
  int G, tiles;
  int gate_up;
  uint4* qw;
  __half* scales;
};

// 16 consecutive elements of a row, as loaded: 16-bit types stay packed two to a register until each is
// needed (half the registers of fp32 copies, so twice the warps that keep loads in flight).
template <typename T>
struct Row16 {
  static constexpr int W = sizeof(T) * 4;  // 32-bit words
  uint32_t w[W];

  __device__ __forceinline__ void load(const T* p) {
#pragma unroll
    for (int i = 0; i < W / 4; ++i) {
      const uint4 v = reinterpret_cast<const uint4*>(p)[i];
      w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
    }
  }
  __device__ __forceinline__ void load_guarded(const T* p, int n) {  // zeros from element n on
#pragma unroll
    for (int i = 0; i < W; ++i) {
      if constexpr (sizeof(T) == 4) {
        w[i] = i < n ? reinterpret_cast<const uint32_t*>(p)[i] : 0u;
      } else {
        const unsigned short* q = reinterpret_cast<const unsigned short*>(p);
        const uint32_t lo = 2 * i < n ? q[2 * i] : 0u, hi = 2 * i + 1 < n ? q[2 * i + 1] : 0u;
        w[i] = lo | hi << 16;
      }
    }
  }
  // Bits of the largest magnitude. Without the sign bit floating-point numbers are ordered like
  // whole numbers, a NaN above all of them, so the maximum of a row with a NaN is a NaN.
  __device__ __forceinline__ uint32_t max_bits(uint32_t m) const {
#pragma unroll
    for (int i = 0; i < W; ++i) {
      if constexpr (sizeof(T) == 4) m = max(m, w[i] & 0x7fffffffu);
      else m = __vmaxu2(m, w[i] & 0x7fff7fffu);
    }
    return m;
  }
  __device__ __forceinline__ static uint32_t join_max(uint32_t a, uint32_t b) {
    return sizeof(T) == 4 ? max(a, b) : __vmaxu2(a, b);
  }
  __device__ __forceinline__ static float max_value(uint32_t m) {
    if constexpr (sizeof(T) == 4) return __uint_as_float(m);
    m = max(m & 0xffffu, m >> 16);
    if constexpr (std::is_same_v<T, bf16>) return __uint_as_float(m << 16);
    return __half2float(__ushort_as_half((unsigned short)m));
  }
  __device__ __forceinline__ float get(int e) const {
    if constexpr (sizeof(T) == 4) return __uint_as_float(w[e]);
    const uint32_t v = w[e >> 1];
    if constexpr (std::is_same_v<T, bf16>) return __uint_as_float(e & 1 ? v & 0xffff0000u : v << 16);
    return __half2float(__ushort_as_half((unsigned short)(e & 1 ? v >> 16 : v)));
  }
};

// A sum with this number (1.5 * 2^23) is rounded to a whole number, ties to even: rounding costs one
// addition on the FMA pipe instead of a conversion on the quarter-rate one.
constexpr float kRound = 12582912.0f;
// ... with this one (1.5 * 2^9) to a multiple of 2^-14.
constexpr float kSnap = 768.0f;

// max(|a|, |b|, |c|)
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float d;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 2 : 4) pack_kernel(const PackArgs a) {
  const int lane = threadIdx.x & 31, r = lane >> 2, t = lane & 3;
  const long u = (long)blockIdx.x * 8 + (threadIdx.x >> 5);  // unit: tile * G + group
  if (u >= (long)a.tiles * a.G) return;
  const int tile = (int)(u / a.G), g = (int)(u - (long)tile * a.G);
  Row16<T> x[2][2];  // [row half][chunk]
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int row = a.gate_up ? 8 * tile + r : 16 * tile + 8 * j + r;
    const T* src = static_cast<const T*>(a.w[j]) + (long)row * a.ld[j];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int k = 128 * g + 64 * c + 16 * t;
      if (VEC && row < a.M && k + 16 <= a.K) x[j][c].load(src + k);
      else x[j][c].load_guarded(src + k, row < a.M ? a.K - k : 0);
    }
  }
  float s[2], inv[2];
  uint32_t keep = 0xffffffffu;  // nibbles of rows whose scale is a number above zero; the others become 8
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    uint32_t m = x[j][1].max_bits(x[j][0].max_bits(0u));
    m = Row16<T>::join_max(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = Row16<T>::join_max(m, __shfl_xor_sync(0xffffffffu, m, 2));
    const __half h = __float2half_rn(Row16<T>::max_value(m) * (float)(2.0 / 15.0));
    s[j] = __half2float(h);
    inv[j] = (1.0f / s[j]) / 15.f;
    if (!(s[j] > 0.f)) keep &= j ? 0x0f0f0f0fu : 0xf0f0f0f0u;
    if (t == 0) a.scales[(size_t)u * 16 + 8 * j + r] = h;
  }
  // [chunk][word]: k offset 2 j1 + j2 of row half j is nibble j + 2 j1 + 4 j2
  uint32_t word[2][4];
  float far = 0.f;  // largest distance of a quotient from the whole number it is rounded to
  auto quantise = [&](auto exact) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        // the codes are whole numbers below 16: four of them are put together exactly in fp32, those of even
        // k in one half of the word and those of odd k in the other, so two at a time
        float2 half_word = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const float2 v = make_float2(x[j][c].get(4 * w + e), x[j][c].get(4 * w + e + 1));
            float2 minus;  // the codes, negative
            if constexpr (decltype(exact)::value) {
              minus.x = -(fminf(fmaxf((v.x / s[j] + kRound) - kRound, -8.f), 7.f) + 8.f);
              minus.y = -(fminf(fmaxf((v.y / s[j] + kRound) - kRound, -8.f), 7.f) + 8.f);
            } else {
              const float2 y = make_float2(__saturatef(fmaf(v.x, inv[j], 8.f / 15.f)),  // (quotient + 8) / 15, clamped
                                           __saturatef(fmaf(v.y, inv[j], 8.f / 15.f)));
              const float2 k15 = make_float2(15.f, 15.f), round = make_float2(kRound, kRound);
              if constexpr (sizeof(T) == 2) {
                // first to a multiple of 2^-14, which an exact half survives, then to a whole number
                const float2 z = fma2(y, k15, make_float2(kSnap, kSnap));
                const float2 q = fma2(z, make_float2(1.f, 1.f), make_float2(kRound - kSnap, kRound - kSnap));
                minus = fma2(q, make_float2(-1.f, -1.f), round);
              } else {
                minus = fma2(fma2(y, k15, round), make_float2(-1.f, -1.f), round);
                const float2 d = fma2(y, k15, minus);
                far = max3_abs(far, d.x, d.y);
              }
            }
            const float place = -(float)(1 << (4 * (j + e)));
            half_word = fma2(minus, make_float2(place, place), half_word);
          }
        const uint32_t lo = __float_as_uint(half_word.x + kRound), hi = __float_as_uint(half_word.y + kRound);
        word[c][w] = (__byte_perm(lo, hi, 0x5410) & keep) | (0x88888888u & ~keep);
      }
  };
  quantise(std::false_type{});
  if (sizeof(T) == 4 && far > 0.5f - 1e-5f) quantise(std::true_type{});
#pragma unroll
  for (int c = 0; c < 2; ++c)
    a.qw[(size_t)u * 64 + c * 32 + lane] = make_uint4(word[c][0], word[c][1], word[c][2], word[c][3]);
}

template <typename T>
int launch_pack(const PackArgs& a, bool vec, cudaStream_t s) {
  const long blocks = ((long)a.tiles * a.G + 7) / 8;
  if (vec) pack_kernel<T, true><<<(unsigned)blocks, 256, 0, s>>>(a);
  else pack_kernel<T, false><<<(unsigned)blocks, 256, 0, s>>>(a);
  return (int)cudaGetLastError();
}

}  // namespace
}  // namespace qb

using namespace qb;

extern "C" int qe_w4_pack(const void* w0, const void* w1, int dtype, int M, int K, long ld0, long ld1, void* qw,
                          void* scales, void* stream) {
  if (!w0 || !qw || !scales || M < 1 || K < 1 || ld0 < K || (w1 && ld1 < K) || dtype < 0 || dtype > 2) return QE_ERR_ARG;
  PackArgs a{};
  a.gate_up = w1 != nullptr;
  a.w[0] = w0;
  a.w[1] = w1 ? w1 : w0;
  a.ld[0] = ld0;
  a.ld[1] = w1 ? ld1 : ld0;
  a.M = M;
  a.K = K;
  a.G = (K + 127) / 128;
  a.tiles = w1 ? (M + 7) / 8 : (M + 15) / 16;
  if ((long)a.tiles * a.G >= (1L << 30) || (reinterpret_cast<uintptr_t>(qw) & 15)) return QE_ERR_ARG;
  a.qw = static_cast<uint4*>(qw);
  a.scales = static_cast<__half*>(scales);
  const int esz = dtype == 2 ? 4 : 2;
  bool vec = true;  // 16-byte loads: aligned bases, row strides that keep them so
  for (int j = 0; j < 2; ++j)
    vec = vec && (reinterpret_cast<uintptr_t>(a.w[j]) & 15) == 0 && (a.ld[j] * esz) % 16 == 0;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == 0) return launch_pack<bf16>(a, vec, s);
  if (dtype == 1) return launch_pack<__half>(a, vec, s);
  return launch_pack<float>(a, vec, s);
}
