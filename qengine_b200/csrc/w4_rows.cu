// W4A16 product for up to 128 activation rows with the GEMV's bits (sm_100a): every matrix is read once for
// all rows of a prefill pass, and row r of the result equals qe_w4_gemv of that row, bit for bit.
//
//   out[n, m] = bf16( sum_g fp32(scale[m, g]) * sum_{k in group g} (code[m, k] - 8) * x[n, k] )
//
// No counterpart in the reference, which prefills in passes of at most 8 rows through its GEMV
// (python/qengine/engine.py:558-573).
//
// Why the bits agree. One group's sum is a chain of eight tensor-core products of 16 k each. tcgen05.mma and
// mma.sync leave the same fp32 sum when each step multiplies the same 16 k (measured: 15.7 million sums of
// rows with exponents from -60 to 60, none differs; with the 16 k of a step in another order a third do). The
// GEMV's step s of a 64-k chunk takes word s of the four lanes of a row pair, k = 16 t + 4 s + 0..3; so the
// weights go into tensor memory word by word, as they are stored, and the activations come with each 64-k
// chunk in that order (wire_pos): what produces them writes them so. Between groups the order of the
// additions is the GEMV's deal of the unit stream (w4_dev.cuh, Deal): a warp's range of groups ascending,
// then the ranges of a CTA, then the CTAs. Here one thread adds all of it, and closes a partial sum where a
// range ends (range_end).
//
// Design: the tensor-memory GEMM of w4_gemm.cu (unpacking warps, one issuing thread, drain warps, coupled by
// mbarriers) with another walk. A job is one super-tile of 128 weight rows over the whole of K and all
// activation rows. Where there are fewer super-tiles than half the SMs, a job is a part of the columns, or a part
// of K (a cluster of CTAs then shares a super-tile): parts of K may only meet where a range of the GEMV ends,
// and what each range adds goes through a scratch in L2, to be added up in order. Eighteen warps: one issues the products; one asks
// for the activations (a request holds its warp up for some hundred clocks, which the drain warps cannot
// spare) and passes on that they have landed, so that the issuing thread has one barrier to wait for; the
// other sixteen are shared out by the columns of a job (below). Tensor memory: D in two stages of 128 columns
// or four of 64, A in four of 64.
//   * What bounds it: hand-over latency, as in w4_gemm.cu. A barrier wait costs 270 clk even when there is
//     nothing to wait for, an unpacking warp's turn 700, a drain warp's 500 (32 columns) to 800 (48), and a
//     step (one group of a super-tile) takes 900 clk at 16 columns, 1150 at 64, 1500 at 128. Hence 128 rows.
//   * us, the four matrices of a 27B layer (in the order in_proj, out, gate/up, down): 128 rows 32 + 29 + 64 + 53 = 178,
//     64 rows 26 + 23 + 50 + 43 = 142, 16 rows 23 + 19 + 43 + 37 = 122; eight rows through the GEMV 57, 64 through
//     w4_gemm.cu 130. Parts of the columns instead of K (down: three parts, each of which unpacks the whole
//     matrix): 128 rows 32 + 33 + 65 + 79 = 210, 64 rows 180, 16 rows 157. First form (requests by the drain
//     warps, eight drain and eight unpacking warps whatever the columns): 385, 323, 300.
// Every wait is bounded (see w4_gemm.cu).
#include <algorithm>

#include "w4_tc.cuh"

namespace qb {
w4::Deal gemv_deal(const qe_w4_params& p, const qe_w4_cfg& c);  // w4_gemv.cu
namespace {

using namespace w4;

struct RowsArgs {
  const uint4* qw;
  const __half* scales;
  OutDesc o;  // o.N = all activation rows
  Deal d;
  int G, tiles;
  int wire_out;      // rows of the output in wire order
  int cparts, cols;  // parts the columns (activation rows) are split into, columns of a part (a multiple of 16)
  int wait_limit;
  float* ws;         // split K: pieces of 16 weight rows x `ws_cols` columns, by piece_of
  int ws_cols;
  int kparts, kstride;  // parts of K (the CTAs of a cluster); where they end: see cut_of
};

__device__ int g_rows_error = 0;

constexpr int kThreads = 18 * 32, kAhead = 3, kB = 4;
constexpr uint32_t kBStage = 128 * 256;  // 128 rows x 128 k
constexpr uint32_t kPitch = 132;         // floats per column of the staging: 128 rows of the super-tile + 4
constexpr int kChunk = 16;               // groups per request of scales
constexpr uint32_t kScaleBytes = kChunk * 32;  // of one tile
constexpr uint32_t kSmem = kB * kBStage + 128 * kPitch * sizeof(float) + 12 * 2 * 2 * kScaleBytes + 1024;
static_assert(kB == 4, "the barriers `done` guard the stages of A and of B");
static_assert(kSmem + 2560 <= 227 * 1024, "shared memory of one block");
constexpr uint32_t kACol = 256;  // tensor memory: D in columns 0..255, A in 256..511

// rows x 128 k of the activations from row y: two 64-k chunks from chunk c
__device__ __forceinline__ void tma_step(uint32_t dst, const CUtensorMap* map, int y, int c, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(0), "r"(y), "r"(c), "r"(sa(bar))
      : "memory");
}

// 16 columns of D into registers: asked for, and (with every request before) arrived.
__device__ __forceinline__ void ld16_ask(uint32_t taddr, uint32_t (&u)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
        "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void ld16_wait(uint32_t (&u)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(u[0]), "+r"(u[1]), "+r"(u[2]), "+r"(u[3]), "+r"(u[4]), "+r"(u[5]), "+r"(u[6]), "+r"(u[7]),
                 "+r"(u[8]), "+r"(u[9]), "+r"(u[10]), "+r"(u[11]), "+r"(u[12]), "+r"(u[13]), "+r"(u[14]), "+r"(u[15])
               :
               : "memory");
}

// (Arrived with an earlier wait: what stays is that no use of them moves in front of that.)
__device__ __forceinline__ void ld16_arrived(uint32_t (&u)[16]) {
  asm volatile(""
               : "+r"(u[0]), "+r"(u[1]), "+r"(u[2]), "+r"(u[3]), "+r"(u[4]), "+r"(u[5]), "+r"(u[6]), "+r"(u[7]),
                 "+r"(u[8]), "+r"(u[9]), "+r"(u[10]), "+r"(u[11]), "+r"(u[12]), "+r"(u[13]), "+r"(u[14]), "+r"(u[15])
               :
               : "memory");
}

// ---- split K: where few super-tiles leave SMs without work ----
// Part p of a super-tile's K begins, tile by tile, where a range of the GEMV ends: at the first end from group
// p * kstride on.
__device__ __forceinline__ int cut_of(const RowsArgs& a, int tile, int p) {
  if (p == 0) return 0;
  if (p >= a.kparts) return a.G;
  const int unit0 = tile * a.G;
  return min(range_at(a.d, unit0 + p * a.kstride).end - unit0, a.G);
}
// A piece is what one range of the GEMV adds to one tile. Along the stream either number goes up from piece to
// piece, so their sum names a piece.
__device__ __forceinline__ size_t piece_of(const RowsArgs& a, int tile, const RangeAt& at) {
  return (size_t)(tile + at.cta * a.d.nwarps + at.warp) * a.ws_cols * 16;
}
constexpr int kPieces = 64;  // of a tile, at most (plan_split); a 27B matrix has 8 or 9
constexpr unsigned kCloses = 1u << 31;
// A tile's pieces in order; kCloses: the last one of its CTA.
__device__ __forceinline__ void list_pieces(const RowsArgs& a, int tile, unsigned* list, int& count) {
  RangeAt at = range_at(a.d, tile * a.G);
  int n = 0;
  for (bool more = true; more && n < kPieces; ++n) {
    list[n] = (unsigned)(tile + at.cta * a.d.nwarps + at.warp) | (at.end == at.cta_end ? kCloses : 0);
    more = at.end - tile * a.G < a.G;
    if (more) range_next(a.d, at);
  }
  count = n;
}
// The sums of four rows of a tile for one column, `at` the first of them in piece 0: its pieces, added in the
// order of the drain loop. Asked for kBatch at a time: one by one each would cost a trip to L2.
__device__ __forceinline__ float4 fold_pieces(size_t pitch, const float* at, const unsigned* list, int count) {
  constexpr int kBatch = 10;
  float4 sum = make_float4(0, 0, 0, 0), older = sum;
  auto add = [](float4& to, const float4& v) { to.x += v.x, to.y += v.y, to.z += v.z, to.w += v.w; };
  bool some = false, some_older = false;
#pragma unroll 1
  for (int k0 = 0; k0 < count; k0 += kBatch) {
    float4 v[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k)
      if (k0 + k < count) v[k] = __ldcg(reinterpret_cast<const float4*>(at + (list[k0 + k] & ~kCloses) * pitch));
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      if (k0 + k < count) {
        const bool last = k0 + k == count - 1;  // what the drain loop leaves in registers: not added to a zero
        if (!some) sum = last ? v[k] : make_float4(0, 0, 0, 0);
        if (some || !last) add(sum, v[k]);
        some = true;
        if (last || (list[k0 + k] & kCloses)) {
          const bool whole = last && !some_older;
          if (!some_older) older = last ? sum : make_float4(0, 0, 0, 0);
          if (!whole) add(older, sum);
          some = false;
          some_older = true;
        }
      }
    }
  }
  return older;
}

// kU groups of four unpacking warps, which alternate steps; kP groups of four drain warps, which share the
// columns, at most 48 of them per thread (96 registers). Where the line lies, us of gate/up and of down at
// that many columns: up to 128, <1, 3>, 65 against 106 for two groups of drain warps with 64 sums; up to
// 64, <2, 2>, 50 against 56 for <1, 3>; up to 48, where the unpack is the longer turn, <3, 1>, 43 against 46 for
// <2, 2> at 16 columns, and 79 against 83 for down at 48.
template <int kU, int kP, bool kSplit>
__global__ void __launch_bounds__(kThreads, 1)
    w4_rows_kernel(const __grid_constant__ RowsArgs a, const __grid_constant__ CUtensorMap xmap) {
  constexpr int kDrain = 4 * kP, kBlocks = kP == 2 ? 2 : 3;  // drain warps; 16-column blocks of one of them
  static_assert(2 + kDrain + 4 * kU == kThreads / 32, "warps");
  dep_release();
  extern __shared__ unsigned char smem_raw[];
  // step may be multiplied: its A is stored (one arrival per unpacking warp), its B has landed (one), and the
  // D of the step nd before has been read (one per drain warp)
  __shared__ uint64_t ready[4];
  __shared__ uint64_t done[4];    // its products are complete (tcgen05.commit): D readable, A and B free
  __shared__ uint64_t b_full[kB];    // its activations have landed
  __shared__ uint64_t s_full[kDrain][2];  // a drain warp's next scales have landed
  __shared__ uint32_t tmem_slot;
  __shared__ unsigned pieces[kSplit ? 8 : 1][kSplit ? kPieces : 1];  // split K: see list_pieces
  __shared__ int npieces[8];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char* Bbase = smem_raw + ((1024u - (sa(smem_raw) & 1023u)) & 1023u);  // swizzle atoms: 1 KB aligned

  if (warp == 1) {  // one barrier per lane
    if (lane < 4) bar_init(&ready[lane], 4 + 1 + kDrain);
    else if (lane < 8) bar_init(&done[lane - 4], 1);
    else if (lane < 8 + kB) bar_init(&b_full[lane - 8], 1);
    if (lane < 2 * kDrain) bar_init(&s_full[lane >> 1][lane & 1], 1);
    bar_fence_init();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sa(&tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  // ---- this CTA's jobs: (super-tile, part of the columns), dealt out round-robin ----
  const int G = a.G, N = a.o.N, CP = a.cparts;
  const int J = ((a.tiles + 7) >> 3) * CP;
  int cta = blockIdx.x, nctas = gridDim.x, part = 0;
  if constexpr (kSplit) {  // one job per cluster, a part of its K per CTA
    asm("mov.u32 %0, %%clusterid.x;" : "=r"(cta));
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(part));
    nctas = J;
  }
  int nj = cta < J ? (J - cta + nctas - 1) / nctas : 0;  // jobs
  auto tile0_of = [&](int j) { return (cta + j * nctas) / CP * 8; };
  auto col0_of = [&](int j) { return (cta + j * nctas) % CP * a.cols; };
  auto blocks_of = [&](int j) { return (min(a.cols, N - col0_of(j)) + 15) >> 4; };  // of 16 columns
  int g0 = 0, g1 = G, cut = 0;  // groups of a job; split K: lane i < 8 and i + 8 hold where those of tile i begin and end
  if constexpr (kSplit) {
    cut = cut_of(a, min(tile0_of(0) + (lane & 7), a.tiles - 1), part + (lane >> 3 & 1));
    g0 = __reduce_min_sync(0xffffffffu, lane & 8 ? G : cut);
    g1 = __reduce_max_sync(0xffffffffu, lane & 8 ? cut : 0);
    if (g1 <= g0) nj = 0;
  }
  const int V = nj * (g1 - g0);  // steps

  const int q = warp & 3;  // quarter of the tensor-memory lanes this warp can reach
  // Unpacking warps: a cursor over the group's steps
  const int grp = kU > 1 ? (warp - kDrain - 1) >> 2 : 0;
  int cj = 0, cg = g0 + grp;  // job, group of the step
  const uint4* cp = a.qw;
  long second = 0;  // distance of the second tile's unit (0: beyond the matrix, never stored)
  auto enter = [&] {
    if constexpr (kSplit) cj += cg >= g1;
    else while (cg >= G) cg -= G, ++cj;
    if (cj >= nj) return;
    const int tile = min(tile0_of(cj) + 2 * q, a.tiles - 1);
    cp = a.qw + ((long)tile * G + cg) * 64 + lane;
    second = tile + 1 < a.tiles ? (long)G * 64 : 0;
  };
  uint4 wreg[kAhead][4];
  auto load_next = [&](uint4 (&w)[4]) {  // request the own step under the cursor and move on
    if (cj >= nj) return;
    w[0] = ld_codes(cp);
    w[1] = ld_codes(cp + 32);
    w[2] = ld_codes(cp + second);
    w[3] = ld_codes(cp + second + 32);
    cp += kU * 64;
    cg += kU;
    if (cg >= g1) enter();
  };
  if (warp > kDrain && warp <= kDrain + 4 * kU) {  // weights never depend on the kernel before: requested before anything is waited for
    enter();
#pragma unroll
    for (int i = 0; i < kAhead; ++i) load_next(wreg[i]);
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
  const uint32_t half_bytes = (uint32_t)a.cols * 128;  // one 64-k chunk of a stage of B
  const int nd = a.cols > 64 ? 2 : 4, dcols = 256 / nd;  // stages of D, columns of a stage

  if (warp == 0) {
    // ---- the issuing warp ----
    const uint64_t db0 = tc_desc(sa(Bbase));
    dep_wait();  // before the first bounded wait: its limit is not for the producer of x to use up
    if (elect_one()) {
      int v = 0;
      bool ok = true;
#pragma unroll 1
      for (int j = 0; j < nj && ok; ++j) {
        const uint32_t idesc =
            (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(blocks_of(j) * 2) << 17) | ((128u >> 4) << 24);
#pragma unroll 1
        for (int g = g0; g < g1; ++g, ++v) {
          const int s = v & 3;
          ok = bar_wait(&ready[s], (v >> 2) & 1, a.wait_limit);
          if (!ok) break;
          tc_fence_after();
          const uint32_t d = tmem + (v & (nd - 1)) * dcols, ac = tmem + kACol + s * 64;
          const uint64_t db = db0 + (uint64_t)(s * (kBStage >> 4));
#pragma unroll
          for (int k = 0; k < 8; ++k)
            tc_mma(d, ac + 8 * k, db + (uint64_t)((k >> 2) * (half_bytes >> 4) + (k & 3) * 2), idesc, k ? 1u : 0u);
          tc_commit(&done[s]);
        }
      }
      if (!ok) atomicExch(&g_rows_error, 2);
      // The products in flight, which drain warps that gave up have not waited for.
      if (v > 0) bar_wait(&done[(v - 1) & 3], ((v - 1) >> 2) & 1, kGemmWaitLimit);
    }
    __syncwarp();
  } else if (warp == kDrain + 4 * kU + 1) {
    // ---- the warp that asks for the activations, a step per request, kB ahead (a request holds its warp up
    // for some hundred clocks), and passes on that they have landed ----
    dep_wait();
    if (elect_one()) {
      int z = 0, landed = 0;
      bool ok = true;
      auto pass_on = [&] {
        ok = bar_wait(&b_full[landed & (kB - 1)], (landed / kB) & 1, a.wait_limit);
        if (ok) bar_arrive(&ready[landed & 3]);
        ++landed;
      };
#pragma unroll 1
      for (int j = 0; j < nj && ok; ++j) {
#pragma unroll 1
        for (int g = g0; g < g1 && ok; ++g) {
          uint64_t* const bar = &b_full[z & (kB - 1)];
          // the products that read the stage before are complete
          if (z >= kB) ok = bar_wait(&done[z & (kB - 1)], (z / kB - 1) & 1, a.wait_limit);
          if (!ok) break;
          bar_expect(bar, 2 * half_bytes);
          tma_step(sa(Bbase) + (z & (kB - 1)) * kBStage, &xmap, col0_of(j), 2 * g, bar);
          ++z;
          if (z > 1) pass_on();  // of the request before: the products need not wait for the next one's stage
        }
      }
      while (landed < z && ok) pass_on();
      if (!ok) atomicExch(&g_rows_error, 16);
      // Shared memory may not be left with copies on their way.
      for (int l = max(z - kB, 0); l < z; ++l) bar_wait(&b_full[l & (kB - 1)], (l / kB) & 1, kGemmWaitLimit);
    }
    __syncwarp();
    // (here, while the last products run: in front of the first request it would hold everything up)
    if constexpr (kSplit) {
      if (lane < 8 && tile0_of(0) + lane < a.tiles) list_pieces(a, tile0_of(0) + lane, pieces[lane], npieces[lane]);
    }
  } else if (warp > kDrain) {
    // ---- unpacking warps ----
    const uint32_t t_lane = tmem + kACol + ((uint32_t)(32 * q) << 16);
    bool ok = true;
#pragma unroll 1
    for (int v0 = grp; v0 < V && ok; v0 += kU * kAhead) {
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        const int v = v0 + kU * i, s = v & 3;
        if (v >= V || !ok) break;
        // The stage of A is free when the products of step v - 4 are complete. A lone group asks for two steps at
        // once (a wait costs it 270 clk even when there is nothing to wait for): products complete in order.
        const int z = kU == 1 ? v - 3 : v - 4;
        if (v >= 4 && (kU > 1 || !(v & 1))) {
          if (v < 4 + kU) dep_wait();  // before the first bounded wait, as in the issuing warp
          if (!warp_wait(&done[z & 3], (z >> 2) & 1, a.wait_limit)) {
            ok = false;
            atomicExch(&g_rows_error, 1);
            break;
          }
        }
        tc_fence_after();
        const uint32_t t0 = t_lane + s * 64;
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
    float* const stage = reinterpret_cast<float*>(Bbase + kB * kBStage);  // [128 columns][kPitch]
    // Scales of the warp's two tiles (its 32 rows), kChunk groups at a time, two requests ahead.
    unsigned char* const scales = Bbase + kB * kBStage + 128 * kPitch * sizeof(float) + wd * 4 * kScaleBytes;
    int sj = 0, sg = g0, snext = 0;  // job, first group and number of the next request
    auto request_scales = [&] {
      if (sj >= nj) return;
      const int n = min(kChunk, g1 - sg);
      if (elect_one()) {
        const int tile = tile0_of(sj) + 2 * q;
        unsigned char* dst = scales + (snext & 1) * 2 * kScaleBytes;
        uint64_t* bar = &s_full[wd][snext & 1];
        const __half* src = a.scales + ((size_t)min(tile, a.tiles - 1) * G + sg) * 16;
        bar_expect(bar, 2 * n * 32);
        bulk_g2s(dst, src, n * 32, bar);
        bulk_g2s(dst + kScaleBytes, tile + 1 < a.tiles ? src + (size_t)G * 16 : src, n * 32, bar);
      }
      __syncwarp();
      ++snext;
      sg += kChunk;
      if (sg >= g1) sg = g0, ++sj;
    };
    request_scales();  // constant like the weights: before the wait
    request_scales();
    auto sync_all = [&] { asm volatile("bar.sync 3, %0;" ::"n"(kDrain * 32) : "memory"); };

    dep_wait();
    if (lane == 0) {  // nothing to read out of D yet
      for (int s = 0; s < nd; ++s) bar_arrive(&ready[s]);
    }

    bool ok = true;
    int v = 0, chunk = 0;  // step, request of scales
#pragma unroll 1
    for (int j = 0; j < nj; ++j) {
      const int nb = blocks_of(j), each = (nb + kP - 1) / kP;  // the warps of a quarter share the columns
      const int blocks = min(each, max(0, nb - each * (wd >> 2))), col0 = 16 * each * (wd >> 2);
      float* const mine = stage + col0 * kPitch + m;  // sums of the ranges closed so far
      float* const older = mine + 64 * kPitch;        // ... of the CTAs closed so far (at most 64 columns then)
      float acc[16 * kBlocks];
#pragma unroll
      for (int k = 0; k < 16 * kBlocks; ++k) acc[k] = 0.f;
      // the range of the GEMV that this row's tile begins in, and the group at which it ends
      const int tile = tile0_of(j) + (m >> 4), unit0 = tile * G;
      const int first = kSplit ? __shfl_sync(0xffffffffu, cut, m >> 4) : 0, last = kSplit ? __shfl_sync(0xffffffffu, cut, 8 + (m >> 4)) : G;
      RangeAt at = range_at(a.d, min(unit0 + min(first, G - 1), a.d.total - 1));
      int next = unit0 < a.d.total ? at.end - unit0 : G;  // (a tile beyond the matrix is never stored)
      bool some = false, some_older = false;
      if constexpr (kSplit) {  // `some`: in a piece of this part
        next = tile < a.tiles && first < last ? first : G + 1;
        if (next == g0) some = true, next = min(at.end - unit0, G);
      }
      auto put_piece = [&] {
        float* const to = a.ws + piece_of(a, tile, at) + (size_t)(col0_of(j) + col0) * 16 + (m & 15);
#pragma unroll
        for (int k = 0; k < 16 * kBlocks; ++k) {
          if ((k >> 4) >= blocks) break;
          __stcg(to + k * 16, acc[k]);
        }
      };
      if (j) sync_all();  // the job before is stored: the staging may be written
      int i = g0;
#pragma unroll 1
      for (int c0 = g0; c0 < g1; c0 += kChunk, ++chunk) {
        if (!ok) break;
        if (!warp_wait(&s_full[wd][chunk & 1], (chunk >> 1) & 1, a.wait_limit)) {
          ok = false;
          if (lane == 0) atomicExch(&g_rows_error, 8);
          break;
        }
        const __half* const sc = reinterpret_cast<const __half*>(scales + ((chunk & 1) * 2 + (lane >> 4)) * kScaleBytes) +
                                 (lane & 15) - c0 * 16;
        const int end = min(c0 + kChunk, g1);
#pragma unroll 1
        for (; i < end && ok; ++i, ++v) {
          if constexpr (kSplit) {
            if (i == next) {  // a piece ends here, or this part's first one begins
              if (some) put_piece(), range_next(a.d, at);
              some = true;
              next = i < last ? min(at.end - unit0, G) : G + 1;
#pragma unroll
              for (int k = 0; k < 16 * kBlocks; ++k) acc[k] = 0.f;
            }
          } else if (i == next) {  // a range of the GEMV ends here: its partial sum is closed
            if (at.end == at.cta_end) {
#pragma unroll
              for (int k = 0; k < 16 * kBlocks; ++k) {
                if ((k >> 4) >= blocks) break;
                const float t = (some ? mine[k * kPitch] : 0.f) + acc[k];
                older[k * kPitch] = (some_older ? older[k * kPitch] : 0.f) + t;
                acc[k] = 0.f;
              }
              some = false;
              some_older = true;
            } else {
#pragma unroll
              for (int k = 0; k < 16 * kBlocks; ++k) {
                if ((k >> 4) >= blocks) break;
                mine[k * kPitch] = (some ? mine[k * kPitch] : 0.f) + acc[k];
                acc[k] = 0.f;
              }
              some = true;
            }
            range_next(a.d, at);
            next = at.end - unit0;
          }
          const int s = v & 3;
          const float scale = __half2float(sc[i * 16]);
          if (!warp_wait(&done[s], (v >> 2) & 1, a.wait_limit)) {
            ok = false;
            if (lane == 0) atomicExch(&g_rows_error, 4);
            break;
          }
          tc_fence_after();
          const uint32_t t0 = t_lane + (v & (nd - 1)) * dcols + col0;
          auto add = [&](const uint32_t (&u)[16], int h) {
#pragma unroll
            for (int k = 0; k < 16; k += 2) {
              float* const to = acc + 16 * h + k;
              const float2 sum = fma2(make_float2(scale, scale), make_float2(__uint_as_float(u[k]), __uint_as_float(u[k + 1])),
                                      make_float2(to[0], to[1]));
              to[0] = sum.x, to[1] = sum.y;
            }
          };
          if constexpr (kBlocks == 2) {  // both blocks in one trip to tensor memory (three would spill)
            uint32_t u0[16], u1[16];
            if (blocks > 0) {
              ld16_ask(t0, u0);
              if (blocks > 1) ld16_ask(t0 + 16, u1);
              ld16_wait(u0);
              add(u0, 0);
              if (blocks > 1) {
                ld16_arrived(u1);
                add(u1, 1);
              }
            }
          } else {
#pragma unroll
            for (int h = 0; h < kBlocks; ++h) {
              if (h >= blocks) break;
              uint32_t u[16];
              ld16_ask(t0 + 16 * h, u);
              ld16_wait(u);
              add(u, h);
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) bar_arrive(&ready[(v + nd) & 3]);
        }
        if (!ok) break;
        __syncwarp();  // every lane has read its scales
        request_scales();
      }
      if constexpr (kSplit) {
        if (ok && next == g1) put_piece();
        break;
      }
#pragma unroll
      for (int k = 0; k < 16 * kBlocks; ++k) {
        if ((k >> 4) >= blocks) break;
        float t = acc[k];
        if (some) t = mine[k * kPitch] + t;
        if (some_older) t = older[k * kPitch] + t;
        mine[k * kPitch] = t;
      }
      // read again after the loops: kept over them, the output's description takes the sums' registers
      const RowsArgs* late = &a;
      asm volatile("" : "+l"(late));
      sync_all();
      if (ok) {
        OutDesc o = late->o;
        const int c0 = col0_of(j);
        o.out = static_cast<unsigned char*>(o.out) + (size_t)c0 * o.ldo * (o.out_f32 ? 4 : 2);
        o.N = min(late->cols, o.N - c0);
        tc_store(o, tile0_of(j), tid - 32, kDrain * 32,
                 [&](int n, int m0) { return *reinterpret_cast<const float4*>(stage + n * kPitch + m0); }, late->wire_out != 0);
      }
    }
    if (!ok) {
      // Shared memory may not be left with copies on their way: the last request of scales per slot.
      for (int r = max(snext - 2, 0); r < snext; ++r) bar_wait(&s_full[wd][r & 1], (r >> 1) & 1, kGemmWaitLimit);
    }
  }
  if constexpr (kSplit) {
    __syncwarp();
    // every part of the super-tile is in L2: each CTA of the cluster adds up and stores some of the columns
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    OutDesc o = a.o;
    const int cols = min(a.cols, N - col0_of(0)), each = (cols + a.kparts - 1) / a.kparts, c0 = col0_of(0) + part * each;
    o.out = static_cast<unsigned char*>(o.out) + (size_t)c0 * o.ldo * (o.out_f32 ? 4 : 2);
    o.N = min(each, cols - part * each);
    const int tile0 = tile0_of(0);
    float* const stage = reinterpret_cast<float*>(Bbase + kB * kBStage);
    const int m0 = lane * 4, t = min(m0 >> 4, a.tiles - 1 - tile0);
#pragma unroll 1
    for (int n = warp; n < o.N; n += kThreads / 32)
      *reinterpret_cast<float4*>(stage + n * kPitch + m0) =
          fold_pieces((size_t)a.ws_cols * 16, a.ws + (size_t)(c0 + n) * 16 + (m0 & 15), pieces[t], npieces[t]);
    __syncthreads();
    if (o.N > 0)
      tc_store(o, tile0, tid, kThreads,
               [&](int n, int m) { return *reinterpret_cast<const float4*>(stage + n * kPitch + m); }, a.wire_out != 0);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

using Kernel = void (*)(RowsArgs, CUtensorMap);
template <bool kSplit>
Kernel kernel_for(int cols) {
  return cols > 64 ? w4_rows_kernel<1, 3, kSplit> : cols > 48 ? w4_rows_kernel<2, 2, kSplit> : w4_rows_kernel<3, 1, kSplit>;
}
cudaLaunchConfig_t config(dim3 grid, cudaStream_t stream, cudaLaunchAttribute* at, int kparts, bool pdl) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(kThreads);
  c.dynamicSmemBytes = kSmem;
  c.stream = stream;
  c.attrs = at;
  if (kparts > 1) {
    at[c.numAttrs].id = cudaLaunchAttributeClusterDimension;
    at[c.numAttrs].val.clusterDim.x = kparts;
    at[c.numAttrs].val.clusterDim.y = at[c.numAttrs].val.clusterDim.z = 1;
    ++c.numAttrs;
  }
  if (pdl) {
    at[c.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[c.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++c.numAttrs;
  }
  return c;
}
// Clusters of `kparts` CTAs that the device holds at once (asked once per device and size).
int clusters_at_once(int dev, int kparts) {
  static int known[64][9] = {};
  if (!known[dev][kparts]) {
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t c = config(dim3(kparts), nullptr, at, kparts, false);
    int n = 0;
    for (int cols : {16, 64, 128}) {
      int m = 0;
      if (cudaOccupancyMaxActiveClusters(&m, kernel_for<true>(cols), &c) != cudaSuccess) m = 0, (void)cudaGetLastError();
      n = cols == 16 ? m : std::min(n, m);
    }
    known[dev][kparts] = n + 1;
  }
  return known[dev][kparts] - 1;
}

// How a product is cut into jobs: columns of a job, parts of the columns, parts of K.
struct Split {
  int cols, cparts, kparts, kstride;
};
Split plan_split(const RowsArgs& a, int dev, bool scratch) {
  const int ST = (a.tiles + 7) / 8, sms = qe_sm_count(), n16 = (a.o.N + 15) / 16;
  auto with_parts = [&](int parts) {
    const int cols = 16 * ((n16 + parts - 1) / parts);
    return Split{cols, (a.o.N + cols - 1) / cols, 1, a.G};
  };
  // Few super-tiles: parts of the columns, as many as there are SMs for, so that every SM has a job. Tiles
  // that the GEMV cuts between CTAs need room for a second level of sums: 64 columns at most.
  int parts = ST * 2 > sms ? 1 : std::min(sms / ST, n16);
  if (a.d.cta_quantum != a.G) parts = std::max(parts, (n16 + 3) / 4);
  Split best = with_parts(parts);
  if (!scratch || ST * 2 > sms) return best;
  // ... or parts of K, which unpack every weight once. The GEMV's ranges end at other groups in every tile, so
  // neighbouring parts overlap by a range: each takes an even share of what that makes of G. In clk: a step 870 + 5 per column; the
  // pieces' way through L2 and the meeting of the parts 6000.
  const int range = a.d.quantum * (std::max(a.d.warp_per[0], a.d.cta_rem ? a.d.warp_per[1] : 0) + 1);
  const int shortest = a.d.quantum * std::max(1, std::min(a.d.warp_per[0], a.d.warp_per[1])), pieces = a.G / shortest + 3;
  auto step = [](int cols) { return 870L + 5 * cols; };
  long least = a.G * step(best.cols);
  for (int k = 2; k <= 8 && k * ST <= sms && a.G / k > range && pieces <= kPieces; ++k) {
    Split s = with_parts(std::min(sms / (ST * k), n16));
    s.kparts = k;
    s.kstride = (a.G - range) / k;
    const long cost = (s.kstride + range) * step(s.cols) + 6000;
    if (cost < least && clusters_at_once(dev, k) >= ST * s.cparts) least = cost, best = s;
  }
  return best;
}
size_t ws_floats(const RowsArgs& a) { return (size_t)(a.tiles + a.d.nctas * a.d.nwarps) * ((a.o.N + 15) / 16) * 256; }

int allow_smem(int dev) {
  static bool allowed[64] = {};
  if (allowed[dev]) return 0;
  for (int cols : {16, 64, 128})
    for (const Kernel k : {kernel_for<false>(cols), kernel_for<true>(cols)})
      if (const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem)) return (int)e;
  allowed[dev] = true;
  return 0;
}

// The checks that need no pointers, and the arguments that follow from the sizes.
int prepare(const qe_w4_params* p, const qe_w4_cfg* cfg, RowsArgs& a) {
  if (!p || !cfg) return QE_ERR_ARG;
  if (p->N < 1 || p->N > QE_MAX_PASS_ROWS || p->Mp % 16 || p->Kp % 128 || p->Mp <= 0 || p->Kp <= 0) return QE_ERR_ARG;
  if (p->K != p->Kp || p->M <= 0) return QE_ERR_ARG;
  if (p->epilogue == QE_EPI_SWIGLU ? p->M > p->Mp / 2 : p->M > p->Mp) return QE_ERR_ARG;
  if (p->epilogue != QE_EPI_NONE && p->epilogue != QE_EPI_SWIGLU) return QE_ERR_ARG;
  if ((long)(p->Mp / 16) * (p->Kp / 128) >= (1L << 30)) return QE_ERR_ARG;
  a.o.M = p->M;
  a.o.N = p->N;
  a.o.epi = p->epilogue;
  a.G = p->Kp / 128;
  a.tiles = p->Mp / 16;
  a.d = gemv_deal(*p, *cfg);
  return 0;
}

}  // namespace

// Error word of the bounded waits above, for qe_w4_ring_error / qe_w4_clear_error (w4_gemv.cu).
int rows_error_read() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_rows_error, sizeof(int)) != cudaSuccess) return -1;
  return v;
}
int rows_error_clear() {
  const int z = 0;
  return (int)cudaMemcpyToSymbol(g_rows_error, &z, sizeof(int));
}

}  // namespace qb

using namespace qb;

extern "C" int qe_w4_rows(const qe_w4_params* p, const qe_w4_cfg* cfg, int wire_out, void* stream) {
  return qe_w4_rows_bounded(p, cfg, wire_out, kGemmWaitLimit, stream);
}

extern "C" long qe_w4_rows_ws_floats(const qe_w4_params* p, const qe_w4_cfg* cfg) {
  RowsArgs a{};
  if (const int e = prepare(p, cfg, a)) return e;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || allow_smem(dev)) return 0;
  return plan_split(a, dev, true).kparts > 1 ? (long)ws_floats(a) : 0;
}

extern "C" int qe_w4_rows_bounded(const qe_w4_params* p, const qe_w4_cfg* cfg, int wire_out, int wait_limit, void* stream) {
  RowsArgs a{};
  if (wait_limit < 0) return QE_ERR_ARG;
  if (const int e = prepare(p, cfg, a)) return e;
  if (p->x_f16 || !p->x || !p->out) return QE_ERR_ARG;
  if (!aligned16(p->qw) || !aligned16(p->scales) || !aligned16(p->x) || (p->ldx & 7) || !aligned16(p->ws)) return QE_ERR_ARG;
  if (wire_out && p->M % 64) return QE_ERR_ARG;  // only whole 64-k chunks have a wire order
  int dev = 0;
  if (const cudaError_t e = cudaGetDevice(&dev)) return (int)e;
  if (dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
  if (const int e = allow_smem(dev)) return e;
  a.qw = reinterpret_cast<const uint4*>(p->qw);
  a.scales = reinterpret_cast<const __half*>(p->scales);
  a.o.out = p->out;
  a.o.ldo = p->ldo;
  a.o.out_f32 = (p->out_f32 && p->epilogue == QE_EPI_NONE) ? 1 : 0;
  a.wire_out = wire_out ? 1 : 0;
  a.wait_limit = wait_limit;
  const Split s = plan_split(a, dev, p->ws != nullptr);
  a.cols = s.cols;
  a.cparts = s.cparts;
  a.kparts = s.kparts;
  a.kstride = s.kstride;
  a.ws = p->ws;
  a.ws_cols = (p->N + 15) / 16 * 16;
  CUtensorMap map{};
  if (!map_rows(p, a.cols, 2, &map)) return QE_ERR_ARG;
  const bool pdl = cfg->pdl && pdl_launch_enabled() && pdl_trigger_enabled();
  const int jobs = (a.tiles + 7) / 8 * a.cparts;
  cudaLaunchAttribute at[2];
  const cudaLaunchConfig_t c = config(dim3(a.kparts > 1 ? jobs * a.kparts : std::min(qe_sm_count(), jobs)), (cudaStream_t)stream, at, a.kparts, pdl);
  return (int)cudaLaunchKernelEx(&c, a.kparts > 1 ? kernel_for<true>(a.cols) : kernel_for<false>(a.cols), a, map);
}
