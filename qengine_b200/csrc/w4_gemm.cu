// W4A16 GEMM for up to 64 activation rows on B200 (sm_100a): the weight matrix is streamed from
// HBM once for all rows of a prefill pass, where the GEMV (w4_gemv.cu, 1..8 rows) would stream it
// once per 8 rows.
//
//   out[n, m] = bf16( sum_g fp32(scale[m, g]) * sum_{k in group g} (code[m, k] - 8) * x[n, k] )
//
// No counterpart in the reference, which prefills in passes of at most 8 rows through its GEMV
// (python/qengine/engine.py:558-573). Same packed wire format (w4_dev.cuh) and the GEMV's
// arithmetic per group (exact products of 4-bit integers and bf16 activations, fp32 sums, the
// group scale applied once); the order in which the groups of a tile are added differs from the
// GEMV's, so a row agrees with the GEMV to fp32 rounding, not bit for bit.
//
// Two kernels behind qe_w4_gemm:
//   * w4_gemm_tc_kernel (the default): tcgen05.mma, weights and accumulator in tensor
//     memory; described in front of it, further down.
//   * w4_gemm_kernel (cfg->variant == 1): mma.sync.m16n8k16 on register fragments, described
//     next. With 8 row tiles it issues eight times the mma.sync instructions of the GEMV per
//     unit and saturates near 130 TFLOP/s (mma.sync alone reaches 541 on this part): 64
//     rows cost about as much as the eight GEMV passes they replace. It is kept as the measured
//     baseline of the tensor-memory kernel and as a second implementation the tests compare.
//
// w4_gemm_kernel. With R rows every unit (16 weight rows x 128 k, 1 KB) needs R x 256 B of
// activations: at 64 rows 16 KB per KB of weights, far more than L2 can deliver to 148 SMs at
// the rate the weights arrive. The activations therefore live in shared memory, one slab of GS
// groups (GS x 128 k) of all rows at a time, double-buffered and filled by bulk copies; all warps
// of a CTA walk K slab by slab together. Work is dealt out in whole tiles (16 output rows): a CTA
// owns a contiguous range of tiles, a warp owns one tile per round -- or, when the CTA has fewer
// tiles than warps, 1/2 or 1/4 of the groups of every slab of one tile -- and keeps that tile's
// R x 16 sums in registers across all slabs. Each warp has a private ring of weight stages (its
// units of one slab, contiguous in memory) fed by bulk copies, as in the GEMV. Warps that share
// a tile add their sums through shared memory in ascending warp order after the last slab: no
// atomics, results are bit-identical run to run.
//
// Every mbarrier wait of both kernels is bounded; on expiry the warp records the error word
// (reported by qe_w4_ring_error), requests nothing more and waits, bounded as well, for the copies and
// products it still has in flight. In w4_gemm_kernel the other warps stop at their next wait for it; the
// warps of w4_gemm_tc_kernel each run into their own limit at the latest. Then the CTA frees its tensor
// memory and leaves.
#include <cuda/atomic>

#include <algorithm>
#include <type_traits>

#include "w4_tc.cuh"

namespace qb {
namespace {

using namespace w4;

struct GemmArgs {
  const uint4* qw;
  const __half* scales;
  const bf16* x;
  long ldx;
  OutDesc o;  // o.N = all activation rows (1..8 RT)
  int G, tiles, nctas;
  int kparts;      // tensor-memory kernel: parts of K a super-tile is split into
  float* ws;       // ... their fp32 sums, [super-tile][part][64][128]
  int* counters;   // ... and one arrival counter per super-tile, zero between launches
  int wait_limit;  // tensor-memory kernel: polls after which a wait gives up
};

__device__ int g_gemm_error = 0;

__device__ __forceinline__ void mma_acc(float (&c)[4], const AFrag& f, uint32_t xa, uint32_t xb) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(f.a0), "r"(f.a1), "r"(f.a2), "r"(f.a3), "r"(xa), "r"(xb));
}

// NW warps; RT row tiles of 8 activation rows; slabs of GS groups; STAGES weight stages per warp.
template <int NW, int RT, int GS, int STAGES>
__global__ void __launch_bounds__(NW * 32, 1) w4_gemm_kernel(const __grid_constant__ GemmArgs a) {
  constexpr uint32_t kStageW = GS * 1024, kStageS = GS * 32;
  constexpr uint32_t kRing = STAGES * (kStageW + kStageS);
  constexpr uint32_t kPitch = GS * 256 + 16;  // + 16: the rows of a quarter-warp hit different banks
  constexpr uint32_t kSlab = 8 * RT * kPitch;
  static_assert(2 * kSlab >= (uint32_t)NW * RT * 128 * sizeof(float), "partial sums reuse the slab buffers");
  dep_release();
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t full_w[NW][STAGES];
  __shared__ uint64_t full_x[2], empty_x[2];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = lane >> 2, t = lane & 3;
  unsigned char* ring_w = smem + (size_t)warp * kRing;
  unsigned char* ring_s = ring_w + (size_t)STAGES * kStageW;
  unsigned char* xs = smem + (size_t)NW * kRing;  // two slabs; partial sums after the last slab

  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      bar_init(&full_x[b], 1);
      bar_init(&empty_x[b], NW);
    }
  }
  if (lane == 0) {
    for (int s = 0; s < STAGES; ++s) bar_init(&full_w[warp][s], 1);
    bar_fence_init();
  }
  __syncthreads();

  // ---- this CTA's tiles, this warp's share of them ----
  const int G = a.G, N = a.o.N;
  const int cta = blockIdx.x;
  int T0 = 0, nt = 0;
  if (cta < a.nctas) {
    T0 = share_begin(a.tiles, a.nctas, cta);
    nt = share_begin(a.tiles, a.nctas, cta + 1) - T0;
  }
  int wpt = 1;  // warps per tile: the largest of 1, 2, 4 (<= GS) that the CTA's tiles can keep busy
  while (wpt * 2 <= GS && nt * wpt * 2 <= NW) wpt *= 2;
  const int RS = NW / wpt;              // tiles per round
  const int rounds = (nt + RS - 1) / RS;
  const int SPT = G / GS;               // slabs per tile
  const int n_it = rounds * SPT;        // slabs this CTA walks through
  const int tl = warp / wpt, sub = warp - tl * wpt;
  const int upw = GS / wpt, j0 = sub * upw;  // this warp's groups of a slab
  const int my_rounds = tl < nt ? (nt - tl + RS - 1) / RS : 0;
  const int my_it = my_rounds * SPT;    // weight stages of this warp: the first my_it slabs

  auto unit_of = [&](int q) {  // first unit of weight stage q
    const int round = q / SPT, s = q - round * SPT;
    return (T0 + round * RS + tl) * G + s * GS + j0;
  };
  auto fill_w = [&](int q, int at) {  // lane 0
    const int u = unit_of(q);
    bar_expect(&full_w[warp][at], (uint32_t)upw * (1024 + 32));
    bulk_g2s(ring_w + (size_t)at * kStageW, a.qw + (size_t)u * 64, (uint32_t)upw * 1024, &full_w[warp][at]);
    bulk_g2s(ring_s + (size_t)at * kStageS, a.scales + (size_t)u * 16, (uint32_t)upw * 32, &full_w[warp][at]);
  };
  // warp 0: request slab `it` of the activations (GS groups of every row)
  auto fill_x = [&](int it) {
    const int b = it & 1, s = it % SPT;
    if (lane == 0) bar_expect(&full_x[b], (uint32_t)N * GS * 256);
    __syncwarp();
    for (int row = lane; row < N; row += 32)
      bulk_g2s(xs + (size_t)b * kSlab + (size_t)row * kPitch, a.x + (long)row * a.ldx + (long)s * GS * 128,
               GS * 256, &full_x[b]);
  };

  // weights never depend on the producer of x: the first stages are requested before the
  // programmatic-dependency wait
  if (lane == 0)
    for (int q = 0; q < min(STAGES, my_it); ++q) fill_w(q, q);
  dep_wait();
  if (warp == 0 && n_it > 0) fill_x(0);

  // Lane (r, t) multiplies activation rows 8 rt + r; rows >= N re-read row N - 1 (their mma
  // columns are never stored), row tiles at or beyond N are skipped.
  const int rtu = (N + 7) >> 3;
  uint32_t xoff[RT];
#pragma unroll
  for (int rt = 0; rt < RT; ++rt) xoff[rt] = (uint32_t)min(8 * rt + r, N - 1) * kPitch + 32 * t;

  float acc[RT][4];
#pragma unroll
  for (int rt = 0; rt < RT; ++rt) acc[rt][0] = acc[rt][1] = acc[rt][2] = acc[rt][3] = 0.f;

  auto store_tile = [&](int tile, int rt, const float (&f)[4]) {
    OutDesc d = a.o;
    const size_t esz = d.out_f32 ? 4 : 2;
    d.out = static_cast<unsigned char*>(a.o.out) + (size_t)(8 * rt) * a.o.ldo * esz;
    d.N = min(8, N - 8 * rt);
    tile_out(d, tile, f, lane);
  };

  int slot = 0, phase = 0;
  bool ok = true;
#pragma unroll 1
  for (int it = 0; it < n_it && ok; ++it) {
    const int b = it & 1;
    if (warp == 0 && it + 1 < n_it) {
      // the other buffer is free once every warp has left slab it - 1
      if (it >= 1 && !warp_wait(&empty_x[b ^ 1], ((it - 1) >> 1) & 1)) {
        ok = false;
        atomicExch(&g_gemm_error, 2);
        break;
      }
      if (lane == 0) async_proxy_fence();
      fill_x(it + 1);
    }
    if (!warp_wait(&full_x[b], (it >> 1) & 1)) {
      ok = false;
      atomicExch(&g_gemm_error, 3);
      break;
    }
    if (it < my_it) {
      uint64_t* bar = &full_w[warp][slot];
      if (!warp_wait(bar, phase)) {
        ok = false;
        atomicExch(&g_gemm_error, 1);
        break;
      }
      const uint4* wp = reinterpret_cast<const uint4*>(ring_w + (size_t)slot * kStageW) + lane;
      const unsigned short* sp = reinterpret_cast<const unsigned short*>(ring_s + (size_t)slot * kStageS) + r;
      const unsigned char* xb = xs + (size_t)b * kSlab + (size_t)j0 * 256;
#pragma unroll 1
      for (int i = 0; i < upw; ++i) {
        const uint4 w0 = wp[i * 64], w1 = wp[i * 64 + 32];
        const uint32_t word[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
        float c[RT][4];
#pragma unroll
        for (int rt = 0; rt < RT; ++rt) c[rt][0] = c[rt][1] = c[rt][2] = c[rt][3] = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          // 16 bytes of x per row tile serve two words: k = 64 (q / 2) + 16 t + 8 (q % 2) .. + 7
          const AFrag f0 = unpack_word(word[2 * q]), f1 = unpack_word(word[2 * q + 1]);
          const uint32_t qo = (uint32_t)i * 256 + (q >> 1) * 128 + (q & 1) * 16;
#pragma unroll
          for (int rt = 0; rt < RT; ++rt) {
            if (rt < rtu) {
              const uint4 xv = *reinterpret_cast<const uint4*>(xb + xoff[rt] + qo);
              mma_acc(c[rt], f0, xv.x, xv.y);
              mma_acc(c[rt], f1, xv.z, xv.w);
            }
          }
        }
        const float lo = __half2float(__ushort_as_half(sp[i * 16]));
        const float hi = __half2float(__ushort_as_half(sp[i * 16 + 8]));
#pragma unroll
        for (int rt = 0; rt < RT; ++rt) {
          acc[rt][0] = fmaf(lo, c[rt][0], acc[rt][0]);
          acc[rt][1] = fmaf(lo, c[rt][1], acc[rt][1]);
          acc[rt][2] = fmaf(hi, c[rt][2], acc[rt][2]);
          acc[rt][3] = fmaf(hi, c[rt][3], acc[rt][3]);
        }
      }
      __syncwarp();  // every lane has read this stage: hand its slot back to the copy engine
      if (lane == 0 && it + STAGES < my_it) {
        async_proxy_fence();
        fill_w(it + STAGES, slot);
      }
      if (++slot == STAGES) { slot = 0; phase ^= 1; }
      // last slab of a tile that this warp owns alone: store it and start the next round's tile
      if (wpt == 1 && (it + 1) % SPT == 0) {
        const int tile = T0 + (it / SPT) * RS + tl;
#pragma unroll
        for (int rt = 0; rt < RT; ++rt) {
          if (rt < rtu) store_tile(tile, rt, acc[rt]);
          acc[rt][0] = acc[rt][1] = acc[rt][2] = acc[rt][3] = 0.f;
        }
      }
    }
    __syncwarp();
    if (lane == 0) bar_arrive(&empty_x[b]);  // this warp has left slab `it`
  }

  if (!ok) {
    // Give the copies that are still in flight a bounded chance to land before the CTA exits.
    __syncwarp();
    for (int s = 0; s < STAGES; ++s) bar_wait(&full_w[warp][s], 0, 1 << 10), bar_wait(&full_w[warp][s], 1, 1 << 10);
    for (int b = 0; b < 2; ++b) bar_wait(&full_x[b], 0, 1 << 10), bar_wait(&full_x[b], 1, 1 << 10);
  }
  if (wpt == 1) return;  // (uniform over the CTA) every tile was stored by its warp

  // ---- tiles shared by wpt warps (one round): partial sums through shared memory ----
  __syncthreads();  // every warp has left the last slab: its buffers are free
  float* part = reinterpret_cast<float*>(xs);  // [NW][RT][4][32]
  if (ok && sub != 0 && tl < nt) {
#pragma unroll
    for (int rt = 0; rt < RT; ++rt)
#pragma unroll
      for (int k = 0; k < 4; ++k) part[((warp * RT + rt) * 4 + k) * 32 + lane] = acc[rt][k];
  }
  __syncthreads();
  if (ok && sub == 0 && tl < nt) {
#pragma unroll
    for (int rt = 0; rt < RT; ++rt) {
      if (rt < rtu) {
        for (int w2 = warp + 1; w2 < warp + wpt; ++w2)
#pragma unroll
          for (int k = 0; k < 4; ++k) acc[rt][k] += part[((w2 * RT + rt) * 4 + k) * 32 + lane];
        store_tile(T0 + tl, rt, acc[rt]);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The tensor-core path proper: tcgen05.mma with weights and accumulator in tensor memory.
//
// A job is one super-tile, 128 weight rows (eight 16-row tiles of the wire format), over its part
// of K. A CTA walks its jobs two at a time (same K, so they share the activations) and a last odd
// one alone. One step = one group g (128 k) of a walk; one micro-step = that group of one of its
// super-tiles. Three roles, coupled by mbarriers only:
//   * unpack (warps 9..16, two groups of four that alternate micro-steps): two tiles' 1 KB units per
//     warp come from HBM straight into registers, kTcAhead own micro-steps ahead (a lane's 32 bytes
//     of a unit are contiguous in the wire format, so nothing has to pass through shared memory),
//     are unpacked to the exact bf16 integers code - 8 and stored as the A operand [128 x 128 k] in
//     tensor memory. tcgen05.st.16x256b takes from lane (r, t) the words 2 t, 2 t + 1 of rows r, r + 8
//     of each 8-word block, and a word of the wire format (rows r, r + 8, four consecutive k) unpacks
//     to just these four registers; transpose4 brings the words of a row pair into ascending k;
//   * warp 0 issues a micro-step's eight tcgen05.mma (M 128, K 16, A from tensor memory, B from shared
//     memory) into one of four 64-column accumulators: the group's exact integer dot products D_g[m, n];
//   * drain (warps 1..8): a pair's super-tiles are read by four warps each, a lone one by all eight,
//     half the columns each; scale[m, g] * D_g[m, n] is added to fp32 registers, groups in ascending
//     order -- the arithmetic of the GEMV (exact products, fp32 sums inside a group, the scale applied
//     once per group). They also request the activations (a tensor map over the rows of x, two steps
//     per request, K-major, 128-byte swizzle) and their scales, and store the result through shared
//     memory, four rows at a time.
// A and D have four stages, B has kTcB. A stage of A is free when the products of the micro-step four
// before are complete (the barrier the drain warps wait for, too); a stage of B when a drain warp has
// seen the products of a later step.
//
// What bounds it. Per unit of weights (1 KB, 46 clk of HBM time per SM at the copy rate) an SM issues
// some 270 warp instructions on four schedulers (68 clk) and multiplies for 32 clk; it takes 110 clk:
// the turns of the issuing thread and of a drain warp, barrier waits of 200 clk and more among them,
// come one after the other. 17 warps leave a thread 96 registers; a drain thread (64 sums, 16 values of D,
// its cursors) spills 116 bytes (180 without a tensor map). 64 rows, 27B shapes: gate/up 81.8 -> 44.3 us, in_proj 41.0 -> 26.9,
// down 53.0 -> 35.5, out 25.2 -> 21.2 against the form with A and the weight ring in shared memory,
// where every warp did all three roles in turn and their latencies added up.
//
// A matrix with fewer super-tiles than half the SMs (the 5,120-row out and down projections: 40) is
// also split along K, up to as many jobs as there are SMs; the parts of a super-tile meet in a
// caller-provided fp32 workspace.
// ---------------------------------------------------------------------------------------------
constexpr int kTcThreads = 17 * 32, kTcAhead = 3, kTcB = 8;
constexpr uint32_t kTcBStage = 64 * 256;  // 64 rows x 128 k
constexpr uint32_t kTcPitch = 132;        // floats per row of the output staging: 128 rows of the super-tile + 4
constexpr int kTcChunk = 28;              // groups per request of scales
constexpr uint32_t kTcScaleBytes = kTcChunk * 32;  // of one tile
constexpr uint32_t kTcSmem =
    kTcB * kTcBStage + 2 * 64 * kTcPitch * sizeof(float) + 8 * 2 * 2 * kTcScaleBytes + 1024;
static_assert(kTcSmem + 512 <= 227 * 1024, "shared memory of one block");
constexpr uint32_t kTcACol = 256;         // tensor memory: D in columns 0..255, A in 256..511

// Four sums of the workspace: at once where the caller's array is 16-byte aligned, which nothing asks of it.
__device__ __forceinline__ void ws_put(float* p, const float4& f, bool vec) {
  if (vec) {
    __stcg(reinterpret_cast<float4*>(p), f);
  } else {
    __stcg(p, f.x), __stcg(p + 1, f.y), __stcg(p + 2, f.z), __stcg(p + 3, f.w);
  }
}
__device__ __forceinline__ float4 ws_get(const float* p, bool vec) {
  if (vec) return __ldcg(reinterpret_cast<const float4*>(p));
  return make_float4(__ldcg(p), __ldcg(p + 1), __ldcg(p + 2), __ldcg(p + 3));
}
__device__ __forceinline__ bool ws_vec(const GemmArgs& a) { return (reinterpret_cast<uintptr_t>(a.ws) & 15) == 0; }
// The parts of a super-tile split along K, added in ascending order.
__device__ __forceinline__ void tc_add_parts(const GemmArgs& a, int st, int ti) {
  __threadfence();
  const int KP = a.kparts;
  const bool vec = ws_vec(a);
  const float* wp = a.ws + (size_t)(st * KP) * (64 * 128);
  tc_store(a.o, st * 8, ti, 256, [&](int n, int m0) {
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int p0 = 0; p0 < KP; p0 += 4) {
      float4 x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (p0 + k < KP) x[k] = ws_get(wp + (size_t)(p0 + k) * (64 * 128) + n * 128 + m0, vec);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (p0 + k < KP) f.x += x[k].x, f.y += x[k].y, f.z += x[k].z, f.w += x[k].w;
    }
    return f;
  });
}

template <bool kTma>
__global__ void __launch_bounds__(kTcThreads, 1)
    w4_gemm_tc_kernel(const __grid_constant__ GemmArgs a, const __grid_constant__ CUtensorMap xmap) {
  dep_release();
  extern __shared__ unsigned char smem_raw[];
  // micro-step may be multiplied: its A is stored (one arrival per unpacking warp of its group) and
  // the D of the micro-step four before has been read (eight arrivals: one per drain warp, or two
  // where four of them read it)
  __shared__ uint64_t ready[4];
  __shared__ uint64_t d_full[4];     // its products are complete (tcgen05.commit): D readable, A free
  __shared__ uint64_t b_full[kTcB / 2];  // activations of two steps are stored (bytes, or arrivals of the drain threads)
  __shared__ uint64_t s_full[8][2];      // a drain warp's next scales have landed
  __shared__ uint32_t tmem_slot;
  __shared__ int s_last;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char* Bbase = smem_raw + ((1024u - (sa(smem_raw) & 1023u)) & 1023u);  // swizzle atoms: 1 KB aligned

  if (warp == 1) {  // one barrier per lane
    if (lane < 4) bar_init(&ready[lane], 4 + 8);
    else if (lane < 8) bar_init(&d_full[lane - 4], 1);
    else if (lane < 8 + kTcB / 2) bar_init(&b_full[lane - 8], kTma ? 1 : 2 * 256);
    else if (lane >= 16) bar_init(&s_full[(lane - 16) >> 1][lane & 1], 1);
    bar_fence_init();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sa(&tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  // ---- this CTA's jobs: (super-tile, part of K), dealt out round-robin, walked in pairs ----
  const int G = a.G, N = a.o.N, KP = a.kparts;
  const int J = ((a.tiles + 7) >> 3) * KP;
  const int cta = blockIdx.x, nctas = gridDim.x;
  const int nj = cta < J ? (J - cta + nctas - 1) / nctas : 0;
  // K is split only where every CTA has one job at most
  const int g_begin = KP > 1 ? share_begin(G, KP, cta % KP) : 0;
  const int g_end = KP > 1 ? share_begin(G, KP, cta % KP + 1) : G;
  auto tile0_of = [&](int j) { return (cta + j * nctas) / KP * 8; };

  const int q = warp & 3;  // quarter of the tensor-memory lanes this warp can reach
  constexpr int kLast = 1 << 30;
  // Unpacking warps: cursor over the warp's own micro-steps. Pair walks have one per step and
  // super-tile (group 0 the first super-tile, group 1 the second); a lone super-tile's steps alternate.
  const int grp = ((warp - 1) >> 2) & 1;
  int cj = 0, cg = 0;  // first job of the walk, group
  const uint4* cp = a.qw;
  long second = 0;  // distance of the second tile's unit (0: beyond the matrix, never stored)
  auto enter = [&](int j) {
    cj = j;
    const bool pair = j + 1 < nj;
    if (j >= nj) { cg = kLast; return; }
    cg = g_begin + (pair ? 0 : grp);
    const int tile = min(tile0_of(pair ? j + grp : j) + 2 * q, a.tiles - 1);
    cp = a.qw + ((long)tile * G + cg) * 64 + lane;
    second = tile + 1 < a.tiles ? (long)G * 64 : 0;
  };
  uint4 wreg[kTcAhead][4];
  auto load_next = [&](uint4 (&w)[4]) {  // request the own micro-step under the cursor and move on
    while (cg != kLast && cg >= g_end) enter(cj + 2);
    if (cg == kLast) return;
    w[0] = ld_codes(cp);
    w[1] = ld_codes(cp + 32);
    w[2] = ld_codes(cp + second);
    w[3] = ld_codes(cp + second + 32);
    const int step = cj + 1 < nj ? 1 : 2;
    cg += step;
    cp += step * 64;
  };
  if (warp > 8) {  // weights never depend on the kernel before: requested before anything is waited for
    enter(0);
#pragma unroll
    for (int i = 0; i < kTcAhead; ++i) load_next(wreg[i]);
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
  const int per_job = g_end - g_begin;
  const int V = nj * per_job;              // micro-steps
  const int n16 = (N + 15) >> 4;           // blocks of 16 activation rows
  // Steps are numbered with every walk rounded up to an even count: two share a load of B.
  const int walk = (per_job + 1) & ~1, steps = ((nj + 1) >> 1) * walk;

  if (warp == 0) {
    // ---- the issuing warp ----
    const uint32_t idesc =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n16 * 2) << 17) | ((128u >> 4) << 24);
    const uint64_t db0 = tc_desc(sa(Bbase));
    dep_wait();  // before the first bounded wait: its limit is not for the producer of x to use up
    if (elect_one()) {
      int v = 0, z = 0;  // micro-steps issued, step
      bool ok = true;
#pragma unroll 1
      for (int j = 0; j < nj && ok; j += 2) {
        const bool pair = j + 1 < nj;
#pragma unroll 1
        for (int i = 0; i < per_job && ok; ++i, ++z) {
          const uint64_t db = db0 + (uint64_t)((z & (kTcB - 1)) * (kTcBStage >> 4));
          if (!(i & 1)) {
            ok = bar_wait(&b_full[(z >> 1) & (kTcB / 2 - 1)], (z / kTcB) & 1, a.wait_limit);
            // Copies made by other threads: the fence that shows them to the tensor core is here because
            // it waits for its thread's own outstanding memory operations, of which this one has none.
            if (!kTma) async_proxy_fence();
          }
#pragma unroll 1
          for (int h = 0; h < (pair ? 2 : 1) && ok; ++h) {
            const int s = v & 3;
            ok = bar_wait(&ready[s], (v >> 2) & 1, a.wait_limit);
            tc_fence_after();
            const uint32_t d = tmem + s * 64, ac = tmem + kTcACol + s * 64;
            if (ok) {
#pragma unroll
              for (int k = 0; k < 8; ++k)
                tc_mma(d, ac + 8 * k, db + (uint64_t)((k >> 2) * (8192 >> 4) + (k & 3) * 2), idesc, k ? 1u : 0u);
              tc_commit(&d_full[s]);
              ++v;
            }
          }
        }
        if (per_job & 1) ++z;
      }
      if (!ok) atomicExch(&g_gemm_error, 2);
      // The products in flight, which drain warps that gave up have not waited for.
      if (v > 0) bar_wait(&d_full[(v - 1) & 3], ((v - 1) >> 2) & 1, kGemmWaitLimit);
    }
    __syncwarp();
  } else if (warp > 8) {
    // ---- unpacking warps ----
    const uint32_t t_lane = tmem + kTcACol + ((uint32_t)(32 * q) << 16);
    bool ok = true;
#pragma unroll 1
    for (int v0 = grp; v0 < V && ok; v0 += 2 * kTcAhead) {
#pragma unroll
      for (int i = 0; i < kTcAhead; ++i) {
        const int v = v0 + 2 * i, s = v & 3;
        if (v >= V || !ok) break;
        if (v >= 4) {
          if (v < 6) dep_wait();  // before the group's first bounded wait, as in the issuing warp
          if (!warp_wait(&d_full[s], ((v >> 2) - 1) & 1, a.wait_limit)) {
            ok = false;
            atomicExch(&g_gemm_error, 1);
            break;
          }
        }
        tc_fence_after();
        const uint32_t t0 = t_lane + s * 64;
#pragma unroll
        for (int h = 0; h < 4; ++h) transpose4(wreg[i][h], lane & 3);
        tc_st_chunk(t0, wreg[i][0]);
        tc_st_chunk(t0 + 32, wreg[i][1]);
        tc_st_chunk(t0 + (16u << 16), wreg[i][2]);
        tc_st_chunk(t0 + (16u << 16) + 32, wreg[i][3]);
        load_next(wreg[i]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) bar_arrive(&ready[s]);
      }
    }
  } else {
    // ---- drain warps ----
    const int wd = warp - 1;
    const int m = 32 * q + lane;  // this thread's row of a super-tile
    const uint32_t t_lane = tmem + ((uint32_t)(32 * q) << 16);
    float* const stage = reinterpret_cast<float*>(Bbase + kTcB * kTcBStage);  // [2 groups][64][kTcPitch]
    float* const mine = stage + grp * 64 * kTcPitch;
    // Scales of the warp's two tiles (its 32 rows), kTcChunk groups at a time, two requests ahead. Plain
    // loads into registers, several groups ahead, cost a memory latency per step: they share the few
    // scoreboards of the warp with everything else.
    unsigned char* const scales = Bbase + kTcB * kTcBStage + 2 * 64 * kTcPitch * sizeof(float) + wd * 4 * kTcScaleBytes;
    int sj = 0, sg = 0, snext = 0;  // walk, first group and number of the next request
    auto request_scales = [&] {
      if (sj >= nj) return;
      const int n = min(kTcChunk, per_job - sg);
      if (elect_one()) {
        const int tile = tile0_of(sj + 1 < nj ? sj + grp : sj) + 2 * q;
        unsigned char* dst = scales + (snext & 1) * 2 * kTcScaleBytes;
        uint64_t* bar = &s_full[wd][snext & 1];
        const __half* src = a.scales + ((size_t)min(tile, a.tiles - 1) * G + g_begin + sg) * 16;
        bar_expect(bar, 2 * n * 32);
        bulk_g2s(dst, src, n * 32, bar);
        bulk_g2s(dst + kTcScaleBytes, tile + 1 < a.tiles ? src + (size_t)G * 16 : src, n * 32, bar);
      }
      __syncwarp();
      ++snext;
      sg += kTcChunk;
      if (sg >= per_job) sg = 0, sj += 2;
    };
    request_scales();  // constant like the weights: before the wait
    request_scales();
    auto sync_group = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory"); };
    auto sync_all = [&] { asm volatile("bar.sync 3, 256;" ::: "memory"); };

    int bg = g_begin, bi = 0;  // group of the next step to load, and its number in the walk
    // rows that a tensor map cannot describe: 16-byte pieces, rows 16 i + 2 wd + lane / 16
    const int n0 = 2 * wd + (lane >> 4);
    const bf16* const xsrc = a.x + (long)n0 * a.ldx + (lane & 15) * 8;
    const uint32_t bdst = sa(Bbase) + ((lane >> 3) & 1) * 8192 + n0 * 128 + (((lane & 7) ^ (n0 & 7)) << 4);
    auto load_b = [&](int z) {
      if (z >= steps) return;
      const uint32_t dst = bdst + (z & (kTcB - 1)) * kTcBStage;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i >= n16 || bi >= per_job) break;
        const bool row = n0 + 16 * i < N;
        cp_async16(dst + i * 2048, row ? xsrc + 16 * i * a.ldx + bg * 128 : a.x, row ? 16u : 0u);
      }
      // this thread's copies up to here have landed: one of the 512 arrivals of two steps
      asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];"
                   ::"r"(sa(&b_full[(z >> 1) & (kTcB / 2 - 1)])) : "memory");
      ++bg;
      if (++bi == walk) bi = 0, bg = g_begin;
    };
    dep_wait();
    // Activations by the copy engine: two steps per request, the requests dealt out over the eight
    // warps because each holds up its warp for some hundred clocks.
    auto request_b = [&](int u) {
      if (2 * u < steps && elect_one()) {
        uint64_t* bar = &b_full[u & (kTcB / 2 - 1)];
        bar_expect(bar, 2 * kTcBStage);
        tma_rows(sa(Bbase) + (u & (kTcB / 2 - 1)) * 2 * kTcBStage, &xmap, 2 * g_begin + u % (walk >> 1) * 4, bar);
      }
      __syncwarp();
    };
    int unit = wd;   // next request of this warp (two steps)
    int loaded = 0;  // without a tensor map: steps whose activations have been requested
    if constexpr (kTma) {
      if (wd < kTcB / 2) {
        request_b(wd);
        unit += 8;
      }
    } else {
      for (; loaded < kTcB - 1; ++loaded) load_b(loaded);
    }
    if (lane == 0) {  // nothing to read out of D yet
      for (int s = 0; s < 4; ++s) bar_arrive(&ready[s]);
    }

    bool ok = true;
    int vb = 0, zb = 0, chunk = 0;  // first micro-step and step of the walk, request of scales
    // One walk's sums, left in the staging. A pair: this group's super-tile, all columns. A lone
    // super-tile: all its micro-steps, columns 32 grp .. + 31. Either way one thread adds the groups
    // of a sum in ascending order.
    auto drain = [&](auto is_pair) {
      constexpr bool kPair = decltype(is_pair)::value;
      constexpr int kBlocks = kPair ? 4 : 2;  // of 16 columns
      const int col0 = kPair ? 0 : 32 * grp, blocks = n16 - (kPair ? 0 : 2 * grp);
      float acc[16 * kBlocks];
#pragma unroll
      for (int k = 0; k < 16 * kBlocks; ++k) acc[k] = 0.f;
      int i = 0, v = vb + (kPair ? grp : 0);
#pragma unroll 1
      for (int c0 = 0; c0 < per_job; c0 += kTcChunk, ++chunk) {
        if (!ok) break;
        if (!warp_wait(&s_full[wd][chunk & 1], (chunk >> 1) & 1, a.wait_limit)) {
          ok = false;
          if (lane == 0) atomicExch(&g_gemm_error, 8);
          break;
        }
        const __half* const sc = reinterpret_cast<const __half*>(scales + ((chunk & 1) * 2 + (lane >> 4)) * kTcScaleBytes) +
                                 (lane & 15) - c0 * 16;
        const int end = min(c0 + kTcChunk, per_job);
#pragma unroll 1
        for (; i < end && ok; ++i, v += kPair ? 2 : 1) {
          const int s = v & 3;
          const float scale = __half2float(sc[i * 16]);
          if (!warp_wait(&d_full[s], (v >> 2) & 1, a.wait_limit)) {
            ok = false;
            if (lane == 0) atomicExch(&g_gemm_error, 4);
            break;
          }
          tc_fence_after();
#pragma unroll
          for (int h = 0; h < kBlocks; ++h) {
            if (h >= blocks) break;
            float d[16];
            tc_ld16(t_lane + s * 64 + col0 + h * 16, d);
#pragma unroll
            for (int k = 0; k < 16; k += 2) {
              float* const to = acc + 16 * h + k;
              const float2 sum = fma2(make_float2(scale, scale), make_float2(d[k], d[k + 1]), make_float2(to[0], to[1]));
              to[0] = sum.x, to[1] = sum.y;
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(sa(&ready[s])), "n"(kPair ? 2 : 1) : "memory");
          // all steps before this one are multiplied: their stages of B are free
          if constexpr (kTma) {
            if (2 * unit < zb + i + kTcB - 1) {
              request_b(unit);
              unit += 8;
            }
          } else {
            for (; loaded < min(steps, zb + i + kTcB); ++loaded) load_b(loaded);
          }
        }
        if (!ok) break;
        __syncwarp();  // every lane has read its scales
        request_scales();
      }
      if (!kPair && zb > 0) sync_all();  // both groups have stored the walk before: the staging may be rewritten
      float* const to = (kPair ? mine : stage + col0 * kTcPitch) + m;
#pragma unroll
      for (int k = 0; k < 16 * kBlocks; ++k)
        if (k < 16 * blocks) to[k * kTcPitch] = acc[k];
    };

#pragma unroll 1
    for (int j = 0; j < nj; j += 2) {
      const bool pair = j + 1 < nj;
      if (pair) drain(std::true_type{});
      else drain(std::false_type{});
      // read again after the loops: kept over them, the output's description takes the sums' registers
      const GemmArgs* late = &a;
      asm volatile("" : "+l"(late));
      if (pair) {
        sync_group();
        if (ok)
          tc_store(late->o, tile0_of(j + grp), (tid - 32) & 127, 128,
                   [&](int n, int m0) { return *reinterpret_cast<const float4*>(mine + n * kTcPitch + m0); });
        sync_group();  // the staging may be rewritten
      } else {
        auto sum = [&](int n, int m0) { return *reinterpret_cast<const float4*>(stage + n * kTcPitch + m0); };
        sync_all();
        if (KP == 1 && ok) tc_store(late->o, tile0_of(j), tid - 32, 256, sum);
      }
      vb += (pair ? 2 : 1) * per_job;
      zb += walk;
    }
    if (KP > 1 && nj > 0) {
      // A super-tile split along K (every CTA has one job at most): every part leaves its fp32 sums in
      // the workspace; the CTA that delivers the last part adds them in ascending order of the parts
      // (so the result does not depend on who was last) and stores the tile.
      const GemmArgs* late = &a;
      asm volatile("" : "+l"(late));
      const int ti = tid - 32, st = cta / KP;
      float* wsj = late->ws + (size_t)cta * (64 * 128);
      const bool vec = ws_vec(*late);
#pragma unroll 4
      for (int e = ti; e < late->o.N * 32; e += 256)
        ws_put(wsj + 4 * e, *reinterpret_cast<const float4*>(stage + (e >> 5) * kTcPitch + (e & 31) * 4), vec);
      __threadfence();
      sync_all();
      if (ti == 0) {
        cuda::atomic_ref<int, cuda::thread_scope_device> arrivals(late->counters[st]);
        const int last = arrivals.fetch_add(1, cuda::memory_order_acq_rel) == KP - 1;
        if (last) late->counters[st] = 0;
        s_last = last;
      }
      sync_all();
      if (s_last && ok) tc_add_parts(*late, st, ti);
    }
    if (!ok) {
      // Shared memory may not be left with copies on their way: the last request of scales per slot and
      // this warp's last request of activations (those before it have been waited for; its barrier
      // may be a phase further, never one behind, for a warp requests when the products of the unit's
      // predecessor in the stage are complete).
      for (int r = max(snext - 2, 0); r < snext; ++r) bar_wait(&s_full[wd][r & 1], (r >> 1) & 1, kGemmWaitLimit);
      const int u = unit - 8;
      if (kTma && u >= 0 && 2 * u < steps) bar_wait(&b_full[u & (kTcB / 2 - 1)], (u / (kTcB / 2)) & 1, kGemmWaitLimit);
    }
    if (!kTma) asm volatile("cp.async.wait_all;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

using GemmFn = void (*)(const GemmArgs);

struct GemmGeom {
  GemmFn fn;
  int nw, rt, gs, stages;
  size_t smem() const {
    return (size_t)nw * stages * gs * (1024 + 32) + 2 * (size_t)8 * rt * (gs * 256 + 16);
  }
};
template <int NW, int RT, int GS, int STAGES>
constexpr GemmGeom gemm_geom() {
  return GemmGeom{w4_gemm_kernel<NW, RT, GS, STAGES>, NW, RT, GS, STAGES};
}
// up to 32 rows: slabs of 4 groups; up to 64 rows (or K / 128 not a multiple of 4): slabs of 2
const GemmGeom kGemmGeoms[] = {gemm_geom<16, 4, 4, 2>(), gemm_geom<16, 8, 2, 4>()};

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Parts of K a super-tile is split into (tensor-memory kernel): 1 unless the matrix has fewer
// super-tiles than half the SMs; then as many as keep the job count within the SMs, at least 8
// groups each. Shape (and device) only, never the row count.
int gemm_kparts(int tiles, int G, int epilogue) {
  const int ST = (tiles + 7) / 8, sms = qe_sm_count();
  if (epilogue != QE_EPI_NONE || ST * 2 > sms) return 1;
  return std::max(1, std::min({sms / ST, G / 8, 16}));
}

// The opt-in limit of dynamic shared memory is a per-device, per-function setting: raised once.
cudaError_t allow_smem(const GemmGeom& g, int which) {
  static bool done[2][64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (done[which][dev]) return cudaSuccess;
  e = cudaFuncSetAttribute(g.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem());
  if (e == cudaSuccess) done[which][dev] = true;
  return e;
}

}  // namespace

// Error word of the bounded waits above, for qe_w4_ring_error / qe_w4_clear_error (w4_gemv.cu).
int gemm_error_read() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_gemm_error, sizeof(int)) != cudaSuccess) return -1;
  return v;
}
int gemm_error_clear() {
  const int z = 0;
  return (int)cudaMemcpyToSymbol(g_gemm_error, &z, sizeof(int));
}

}  // namespace qb

using namespace qb;

extern "C" int qe_w4_plan_gemm(const qe_w4_params* p, const qe_w4_cfg* cfg, qe_w4_plan* plan) {
  if (!p || !cfg || !plan || p->Mp <= 0 || p->Kp <= 0 || p->Mp % 16 || p->Kp % 128) return QE_ERR_ARG;
  const int tiles = p->Mp / 16, ST = (tiles + 7) / 8;
  const int kp = cfg->variant == 1 ? 1 : gemm_kparts(tiles, p->Kp / 128, p->epilogue);
  plan->mode = cfg->variant == 1 ? 1 : 0;
  plan->grid_x = std::min(qe_sm_count(), cfg->variant == 1 ? tiles : ST * kp);
  plan->grid_y = 1;
  plan->threads = cfg->variant == 1 ? 512 : kTcThreads;
  plan->ws_floats = kp > 1 ? (long)ST * kp * 64 * 128 : 0;
  plan->counters = kp > 1 ? ST : 0;
  return 0;
}

extern "C" int qe_w4_gemm(const qe_w4_params* p, const qe_w4_cfg* cfg, void* stream) {
  return qe_w4_gemm_bounded(p, cfg, kGemmWaitLimit, stream);
}

extern "C" int qe_w4_gemm_bounded(const qe_w4_params* p, const qe_w4_cfg* cfg, int wait_limit, void* stream) {
  if (!p || !cfg || wait_limit < 0) return QE_ERR_ARG;
  if (p->N < 1 || p->N > QE_MAX_GEMM_ROWS || p->Mp % 16 || p->Kp % 128 || p->Mp <= 0 || p->Kp <= 0) return QE_ERR_ARG;
  if (p->K != p->Kp || p->M <= 0 || p->x_f16 || !p->x || !p->out) return QE_ERR_ARG;
  if (p->epilogue == QE_EPI_SWIGLU ? p->M > p->Mp / 2 : p->M > p->Mp) return QE_ERR_ARG;
  if (p->epilogue != QE_EPI_NONE && p->epilogue != QE_EPI_SWIGLU) return QE_ERR_ARG;
  if ((long)(p->Mp / 16) * (p->Kp / 128) >= (1L << 30)) return QE_ERR_ARG;
  // bulk copies: 16-byte aligned sources, row strides that keep them so
  if (!aligned16(p->qw) || !aligned16(p->scales) || !aligned16(p->x) || (p->ldx & 7)) return QE_ERR_ARG;
  const int G = p->Kp / 128;
  if (cfg->variant != 1) {  // tensor memory path (the default); variant 1: the mma.sync kernels below
    static bool allowed[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
    if (!allowed[dev]) {
      e = cudaFuncSetAttribute(w4_gemm_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(w4_gemm_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem);
      if (e != cudaSuccess) return (int)e;
      allowed[dev] = true;
    }
    GemmArgs a{};
    a.qw = reinterpret_cast<const uint4*>(p->qw);
    a.scales = reinterpret_cast<const __half*>(p->scales);
    a.x = reinterpret_cast<const bf16*>(p->x);
    a.ldx = p->ldx;
    a.o.out = p->out;
    a.o.ldo = p->ldo;
    a.o.M = p->M;
    a.o.N = p->N;
    a.o.epi = p->epilogue;
    a.o.out_f32 = (p->out_f32 && p->epilogue == QE_EPI_NONE) ? 1 : 0;
    a.G = G;
    a.tiles = p->Mp / 16;
    a.wait_limit = wait_limit;
    a.kparts = gemm_kparts(a.tiles, G, p->epilogue);
    if (a.kparts > 1 && (!p->ws || !p->counters)) a.kparts = 1;  // no scratch: whole K per job
    a.ws = p->ws;
    a.counters = p->counters;
    a.nctas = std::min(qe_sm_count(), ((a.tiles + 7) / 8) * a.kparts);
    const bool pdl = cfg->pdl && pdl_launch_enabled() && pdl_trigger_enabled();
    CUtensorMap map{};
    const auto kernel = map_rows(p, 64, 4, &map) ? w4_gemm_tc_kernel<true> : w4_gemm_tc_kernel<false>;
    return (int)launch(kernel, dim3(a.nctas), dim3(kTcThreads), kTcSmem, (cudaStream_t)stream, pdl, a, map);
  }
  int which;
  if (p->N <= 32 && G % 4 == 0) which = 0;
  else if (G % 2 == 0) which = 1;
  else return QE_ERR_ARG;
  const GemmGeom& g = kGemmGeoms[which];
  cudaError_t e = allow_smem(g, which);
  if (e != cudaSuccess) return (int)e;
  GemmArgs a{};
  a.qw = reinterpret_cast<const uint4*>(p->qw);
  a.scales = reinterpret_cast<const __half*>(p->scales);
  a.x = reinterpret_cast<const bf16*>(p->x);
  a.ldx = p->ldx;
  a.o.out = p->out;
  a.o.ldo = p->ldo;
  a.o.M = p->M;
  a.o.N = p->N;
  a.o.epi = p->epilogue;
  a.o.out_f32 = (p->out_f32 && p->epilogue == QE_EPI_NONE) ? 1 : 0;
  a.G = G;
  a.tiles = p->Mp / 16;
  a.nctas = std::min(qe_sm_count(), a.tiles);
  const bool pdl = cfg->pdl && pdl_launch_enabled() && pdl_trigger_enabled();
  return (int)launch(g.fn, dim3(a.nctas), dim3(g.nw * 32), g.smem(), (cudaStream_t)stream, pdl, a);
}
