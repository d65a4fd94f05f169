// Gated delta-rule (Gated DeltaNet) decode / verify step for n = 1..8 rows with per-position
// checkpoints for rollback. Boundary: replaces launch_gdn_step_n of the reference
// (csrc/ops.h:20-24, kernel csrc/gdn.cu:65-311); the math follows deltanet_core of the
// reference torch model (python/qengine/reference.py:211-242) including every bf16 rounding.
//
// Rollback scheme (same contract as the reference, csrc/gdn.cu:1-11): the committed state S in
// global memory is the state after position pos - pending. A pass first replays the `pending`
// rows that the previous pass staged and that were accepted -- from their checkpoint
// (k, v, decay, beta), 2 D + 2 floats per position and head -- and writes S back once. Its own
// n rows then run on the register copy of S and are only staged; S is not written for them. A
// rejected draft therefore costs nothing to undo, and a full-state snapshot per position
// (D * D floats) is never needed. Replayed and new rows use the same update routine, so the
// committed state is bit-identical to plain one-row decoding.
//
// Per value head j (q/k head j / (Hv / Hk)), per row at position p:
//   conv  c = w0 x[p-3] + w1 x[p-2] + w2 x[p-1] + w3 x[p] (fp32), y = bf16(silu(bf16(c)))
//   q = y_q * rsqrt(sum y_q^2 + 1e-6) / sqrt(D),  k = y_k * rsqrt(sum y_k^2 + 1e-6),  v = y_v
//   beta = bf16(sigmoid(b)),  decay = exp(-exp(A_log) * softplus(a + dt_bias))
//   S' = decay S + k delta^T with delta = beta (v - decay S^T k);  o = S'^T q
//   out = bf16( bf16(norm_w * bf16(o_b * rsqrt(mean o_b^2 + eps))) * silu(z) ),  o_b = bf16(o)
// Conv history lives in a 16-slot ring keyed by absolute position (slot p & 15); with n <= 8 the
// slots read (p-3..p-1 of the first row) and written (p..p+n-1) never alias.
//
// B200 layout. The columns of S are independent in the recurrence (column d only needs k, q,
// v[d]), so a head is split over a thread-block cluster of D / 32 CTAs, 32 columns each: 192 CTAs
// for the 48 heads of the 27B shape instead of 48. A CTA is 8 warps; warp w owns rows
// [w D/8, (w+1) D/8) of its 32 columns in registers (lane = column, S read and written coalesced).
// One pass over the register state per row gives both S^T k and S^T q of the pre-update state:
//   kv = decay (S^T k),  delta = beta (v - kv),  o = decay (S^T q) + delta (k . q)
// so a row costs one block barrier (partials are double-buffered) instead of several. The gated
// RMSNorm needs the sum of o_b^2 over all D columns of the head: every CTA pushes its partial sum
// into the shared memory of all CTAs of the cluster (distributed shared memory stores), one cluster
// barrier, and each CTA adds the partials in rank order.
//
// Dependency handling: the state, the per-head constants, ctl and the checkpoints of the previous
// pass do not depend on the producer of this pass's projections, so with `early` the state load
// and the whole replay (including the write-back of S) run before the programmatic-dependency
// wait and overlap the in_proj GEMV. `early` requires that the previous pass has completed when
// this pass starts (an engine launches the first kernel of a pass in plain stream order).
#include <cooperative_groups.h>

#include "common.cuh"
#include "../../include/qengine_b200.h"

namespace cg = cooperative_groups;

namespace qb {
namespace {

constexpr int kRing = 16, kMaxRows = QE_MAX_ROWS, kCols = 32, kWarps = 8;

struct GdnArgs {
  const bf16 *qkv, *z, *b, *a;
  long ldp;
  bf16* ring;
  const bf16 *conv_w, *A_log, *dt_bias, *norm_w;
  float *S, *st_k, *st_v, *st_g;
  const int* ctl;
  bf16* out;
  long ldo;
  int n, Hk, Hv;
  float eps;
  int early;
};

template <int D>
__global__ void __launch_bounds__(kWarps * 32) gdn_cluster_kernel(const GdnArgs a) {
  constexpr int RP = D / kWarps;        // state rows per warp
  constexpr int NT = kWarps * 32;
  constexpr int NCTA = D / kCols;       // CTAs per head = cluster size
  dep_release();
  if (!a.early) dep_wait();
  cg::cluster_group cluster = cg::this_cluster();

  __shared__ float q_s[kMaxRows][D], k_s[kMaxRows][D];
  __shared__ float v_s[kMaxRows][kCols], o_s[kMaxRows][kCols];
  __shared__ float gate_s[kMaxRows][2];      // (decay, beta)
  __shared__ float kq_s[kMaxRows];           // k . q per row
  __shared__ float part[2][2][kWarps][kCols];  // [buffer][k or q][warp][column]
  __shared__ float ss_all[NCTA][kMaxRows];   // sum of o_b^2 per row of every CTA of the cluster (pushed)

  const int j = blockIdx.y;                  // value head
  const int cs = blockIdx.x;                 // column slice = rank in the cluster
  const int c0 = cs * kCols;
  const int rep = a.Hv / a.Hk, i_qk = j / rep;
  const int C = 2 * a.Hk * D + a.Hv * D;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = a.n;
  float* Sj = a.S + (size_t)j * D * D + c0 + lane;

  // ---- independent of this pass's producer: state slice, per-head constants, checkpoints ----
  // Every global load of this section is issued into registers before anything is used: a
  // "shared[i] = global[j]" loop stalls on each store until its load is back, one memory round
  // trip per iteration (that was 4 us in front of the replay). Loaded here: ctl, the state (3 MB
  // per layer, from HBM), all eight checkpoint slots (whether or not they are pending: that is
  // only known once ctl arrives), the per-head constants and the conv taps; the conv history
  // needs the position and follows as soon as ctl is there.
  const int ctl_pos = a.ctl[0], ctl_pending = a.ctl[1];
  float s[RP];
#pragma unroll
  for (int i = 0; i < RP; ++i) s[i] = Sj[(size_t)(warp * RP + i) * D];
  constexpr int KPT = kMaxRows * D / NT;  // checkpoint k values per thread
  float kreg[KPT];
#pragma unroll
  for (int u = 0; u < KPT; ++u) {
    const int idx = tid + u * NT, t = idx / D, i = idx - t * D;
    kreg[u] = a.st_k[((size_t)t * a.Hv + j) * D + i];
  }
  const float vreg = a.st_v[((size_t)warp * a.Hv + j) * D + c0 + lane];  // 8 warps = 8 slots, lane = column
  const float greg = lane < 2 ? a.st_g[(warp * a.Hv + j) * 2 + lane] : 0.f;
  const float A_log = tofloat(a.A_log[j]), dt_bias = tofloat(a.dt_bias[j]);
  const float nw = tofloat(a.norm_w[c0 + lane]);
  // conv channels of this thread (q and k: all D channels of the head's q/k head; v: own columns)
  constexpr int CPT = (2 * D + kCols + NT - 1) / NT;  // 2 for D = 128
  float cw[CPT][4], hx[CPT][3];
  int chn[CPT];
#pragma unroll
  for (int u = 0; u < CPT; ++u) {
    const int idx = tid + u * NT;
    chn[u] = -1;
    if (idx < 2 * D + kCols) {
      const int part_id = idx < D ? 0 : idx < 2 * D ? 1 : 2;
      const int c = part_id == 0 ? idx : part_id == 1 ? idx - D : idx - 2 * D;
      chn[u] = part_id == 0 ? i_qk * D + c : part_id == 1 ? a.Hk * D + i_qk * D + c : 2 * a.Hk * D + j * D + c0 + c;
#pragma unroll
      for (int w = 0; w < 4; ++w) cw[u][w] = tofloat(a.conv_w[chn[u] * 4 + w]);
    }
  }
  // ctl and the checkpoints were written by the previous pass, which has completed (the first
  // kernel of a pass is launched in plain stream order): with `early` the whole replay, including
  // the write-back of S, runs before the dependency wait and overlaps the tail of the in_proj GEMV.
  const int P = ctl_pos, pend = min(max(ctl_pending, 0), kMaxRows);
#pragma unroll
  for (int u = 0; u < CPT; ++u) {
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int p = P - 3 + b;
      hx[u][b] = (chn[u] >= 0 && p >= 0) ? tofloat(a.ring[(size_t)(p & (kRing - 1)) * C + chn[u]]) : 0.f;
    }
  }
#pragma unroll
  for (int u = 0; u < KPT; ++u) {
    const int idx = tid + u * NT, t = idx / D, i = idx - t * D;
    k_s[t][i] = kreg[u];
  }
  v_s[warp][lane] = vreg;
  if (lane < 2) gate_s[warp][lane] = greg;

  // S <- decay S + k (beta (v - decay S^T k))^T on this thread's rows of its column; with Q also
  // returns o = S'^T q for the column. Identical arithmetic for replayed and new rows.
  auto row_update = [&](const float* kk, const float* qq, float v, float decay, float beta, float kq,
                        int buf, bool want_o) -> float {
    float pk = 0.f, pq = 0.f;
#pragma unroll
    for (int i = 0; i < RP; ++i) {
      pk = fmaf(s[i], kk[warp * RP + i], pk);
      if (want_o) pq = fmaf(s[i], qq[warp * RP + i], pq);
    }
    part[buf][0][warp][lane] = pk;
    if (want_o) part[buf][1][warp][lane] = pq;
    __syncthreads();
    float kv = part[buf][0][0][lane];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) kv += part[buf][0][w][lane];
    const float delta = (v - decay * kv) * beta;
#pragma unroll
    for (int i = 0; i < RP; ++i) s[i] = fmaf(kk[warp * RP + i], delta, decay * s[i]);
    if (!want_o) return 0.f;
    float qs = part[buf][1][0][lane];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) qs += part[buf][1][w][lane];
    return fmaf(delta, kq, decay * qs);
  };

  // ---- 1. replay the kept rows of the previous pass, write the committed state once ----
  int buf = 0;
  __syncthreads();
  for (int t = 0; t < pend; ++t) {
    row_update(k_s[t], nullptr, v_s[t][lane], gate_s[t][0], gate_s[t][1], 0.f, buf, false);
    buf ^= 1;
  }
  if (pend > 0) {
#pragma unroll
    for (int i = 0; i < RP; ++i) Sj[(size_t)(warp * RP + i) * D] = s[i];
  }
  if (a.early) dep_wait();  // from here on: this pass's projections
  // the gate input of this warp's row is only needed at the very end: fetch it now; likewise the
  // decay / beta inputs of row tid, which the same thread would otherwise only request after its
  // share of the convolution (a second, dependent memory round trip)
  const float z_pre = warp < n ? tofloat(a.z[(long)warp * a.ldp + j * D + c0 + lane]) : 0.f;
  const float b_pre = tid < n ? tofloat(a.b[(long)tid * a.ldp + j]) : 0.f;
  const float a_pre = tid < n ? tofloat(a.a[(long)tid * a.ldp + j]) : 0.f;
  // and every projection value this thread convolves, all rows at once: independent loads in
  // flight together instead of one round trip per row and channel
  bf16 xr[CPT][kMaxRows];
#pragma unroll
  for (int u = 0; u < CPT; ++u)
#pragma unroll
    for (int t = 0; t < kMaxRows; ++t)
      if (chn[u] >= 0 && t < n) xr[u][t] = a.qkv[(long)t * a.ldp + chn[u]];
  __syncthreads();  // k_s / v_s are about to be overwritten by the new rows

  // ---- 2a. causal conv + SiLU of every new row (q, k: all D channels; v: own columns) ----
#pragma unroll
  for (int u = 0; u < CPT; ++u) {
    const int idx = tid + u * NT;
    if (chn[u] < 0) continue;
    const int part_id = idx < D ? 0 : idx < 2 * D ? 1 : 2;
    const int c = part_id == 0 ? idx : part_id == 1 ? idx - D : idx - 2 * D;
    const int ch = chn[u];
    float x0 = hx[u][0], x1 = hx[u][1], x2 = hx[u][2];
    // q/k channels are shared by `rep` heads and by the CTAs of a head: one CTA writes them
    const bool owner = part_id == 2 || ((j % rep) == 0 && cs == 0);
#pragma unroll
    for (int t = 0; t < kMaxRows; ++t) {
      if (t >= n) break;
      const bf16 xb = xr[u][t];
      const float x3 = tofloat(xb);
      float acc = cw[u][0] * x0;
      acc = fmaf(cw[u][1], x1, acc);
      acc = fmaf(cw[u][2], x2, acc);
      acc = fmaf(cw[u][3], x3, acc);
      const float y = rnd(silu_acc(rnd(acc)));
      if (part_id == 0) q_s[t][c] = y;
      else if (part_id == 1) k_s[t][c] = y;
      else v_s[t][c] = y;
      if (owner) a.ring[(size_t)((P + t) & (kRing - 1)) * C + ch] = xb;
      x0 = x1; x1 = x2; x2 = x3;
    }
  }
  if (tid < n) {
    const int t = tid;
    const float bt = rnd(sigmoid_acc(b_pre));
    const float x = a_pre + dt_bias;
    const float sp = x > 20.f ? x : log1pf(expf(x));
    gate_s[t][0] = expf(-expf(A_log) * sp);
    gate_s[t][1] = bt;
  }
  __syncthreads();

  // ---- 2b. l2norm of q and k of every row and k . q: warp t handles row t. Each lane first adds
  // up its own D / 32 elements, so a sum costs ONE butterfly, and the two independent butterflies
  // of q and k overlap (twelve dependent ones were 0.5 us of the step) ----
  for (int t = warp; t < n; t += kWarps) {
    float eq[D / 32], ek[D / 32], sq = 0.f, sk = 0.f;
#pragma unroll
    for (int u = 0; u < D / 32; ++u) {
      eq[u] = q_s[t][lane + 32 * u];
      ek[u] = k_s[t][lane + 32 * u];
      sq = fmaf(eq[u], eq[u], sq);
      sk = fmaf(ek[u], ek[u], sk);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
      sk += __shfl_xor_sync(0xffffffffu, sk, o);
    }
    const float iq = rsqrtf(sq + 1e-6f), ik = rsqrtf(sk + 1e-6f);
    float dot = 0.f;
#pragma unroll
    for (int u = 0; u < D / 32; ++u) {
      const float qn = (eq[u] * iq) / sqrtf((float)D), kn = ek[u] * ik;
      q_s[t][lane + 32 * u] = qn;
      k_s[t][lane + 32 * u] = kn;
      dot = fmaf(qn, kn, dot);
    }
    dot = warp_allsum(dot);
    if (lane == 0) kq_s[t] = dot;
  }
  __syncthreads();

  // ---- 2d. the recurrence, row by row, on the register copy of S ----
  for (int t = 0; t < n; ++t) {
    const float o = row_update(k_s[t], q_s[t], v_s[t][lane], gate_s[t][0], gate_s[t][1], kq_s[t], buf, true);
    buf ^= 1;
    if (warp == 0) o_s[t][lane] = rnd(o);  // the mixer output is a bf16 tensor in the model
  }
  __syncthreads();

  // ---- 2e. gated RMSNorm over the head's D outputs: every CTA pushes its partial sum of squares
  // into the shared memory of all CTAs of the cluster; one cluster barrier makes them visible ----
  for (int t = warp; t < n; t += kWarps) {
    const float ob = o_s[t][lane];
    const float ssum = warp_allsum(ob * ob);
    if (lane < NCTA) *cluster.map_shared_rank(&ss_all[cs][t], lane) = ssum;
  }
  cluster.sync();
  for (int t = warp; t < n; t += kWarps) {
    float total = 0.f;
#pragma unroll
    for (int rk = 0; rk < NCTA; ++rk) total += ss_all[rk][t];
    const float ob = o_s[t][lane];
    const float nn = rnd(ob * rsqrtf(total / (float)D + a.eps));
    const float y = rnd(nw * nn);
    const float zz = t == warp ? z_pre : tofloat(a.z[(long)t * a.ldp + j * D + c0 + lane]);
    a.out[(long)t * a.ldo + j * D + c0 + lane] = tobf16(y * silu_acc(zz));
  }
  // no second barrier: nobody reads remote shared memory after the one above, and every remote
  // store was issued before it
  // ---- 2f. checkpoint every row for the next pass (k, gates: one CTA per head; v: own slice).
  // Last, behind the output: nothing in this pass waits for these stores. The CTA with cs == 0
  // overwrites st_k / st_g, which its siblings read while replaying: the cluster barrier of 2e
  // lies in between, and every CTA passes it only after its replay ----
  for (int t = 0; t < n; ++t) {
    if (cs == 0) {
      for (int i = tid; i < D; i += NT) a.st_k[((size_t)t * a.Hv + j) * D + i] = k_s[t][i];
      if (tid == 0) {
        a.st_g[(t * a.Hv + j) * 2] = gate_s[t][0];
        a.st_g[(t * a.Hv + j) * 2 + 1] = gate_s[t][1];
      }
    }
    if (tid < kCols) a.st_v[((size_t)t * a.Hv + j) * D + c0 + tid] = v_s[t][tid];
  }
}

// ---------------------------------------------------------------------------------------------
// Prefill: n = 8, 16 .. 64 new rows in one launch. What n / 8 calls of the step above do to the
// state, the checkpoints (the last 8 rows stay pending) and the output, bit for bit, with the state
// read and written once instead of once per 8 rows, no replay in between, and convolution,
// normalisation and the gated norm of all rows side by side. Between rows only the recurrence is
// serial, so it decides the layout: warp w owns columns 4 w .. 4 w + 3 of the CTA's 32, lane (g, c) =
// (lane / 4, lane % 4) the rows g D / 8 .. of column c -- the share that warp g of the step kernel
// has. The eight partial sums of a column then meet inside the warp (through 512 bytes of shared
// memory, added in the step kernel's order) and a row needs no block barrier; the step kernel spreads
// a column over its warps because there the loads that fill the state matter more.
// A 1,021-token prompt over 16 layers of the 27B shape (12 of them DeltaNet), with the attention rows of
// a pass in one launch as well: 72.9 -> 56.9 ms.
// ---------------------------------------------------------------------------------------------
constexpr int kWideRows = QE_MAX_GEMM_ROWS, kStaged = QE_MAX_ROWS;

// k and q of a row: four floats of padding per eighth, so that the eight eighths' 16-byte loads hit
// different banks.
template <int D>
struct GdnWideShared {
  static constexpr int RP = D / 8, kPitch = 8 * (RP + 4);
  static __device__ __forceinline__ int at(int i) { return i + i / RP * 4; }
  float q[kWideRows][kPitch], k[kWideRows][kPitch];
  float v[kWideRows][kCols], o[kWideRows][kCols];
  float gate[kWideRows][2], kq[kWideRows];
  float2 part[kWarps][4][8 + 2];  // [warp][column][eighth]: partial sums of S^T k and S^T q
  float ss[D / kCols][kWideRows];
};

template <int D>
__global__ void __launch_bounds__(kWarps * 32, 2) gdn_prefill_kernel(const GdnArgs a) {
  constexpr int NI = D / 32, NT = kWarps * 32, NCTA = D / kCols;
  using Shared = GdnWideShared<D>;
  constexpr int RP = Shared::RP;
  dep_release();
  dep_wait();
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Shared& sh = *reinterpret_cast<Shared*>(smem_raw);

  const int j = blockIdx.y, cs = blockIdx.x, c0 = cs * kCols;
  const int rep = a.Hv / a.Hk, i_qk = j / rep;
  const int C = 2 * a.Hk * D + a.Hv * D;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = a.n, P = a.ctl[0], pend = min(max(a.ctl[1], 0), kStaged);
  const int col = 4 * warp + (lane & 3), g = lane >> 2;
  float* Sj = a.S + ((size_t)j * D + g * RP) * D + c0 + col;

  float2 s[RP / 2];
#pragma unroll
  for (int i = 0; i < RP / 2; ++i) s[i] = make_float2(Sj[(size_t)(2 * i) * D], Sj[(size_t)(2 * i + 1) * D]);
  auto store_state = [&] {
#pragma unroll
    for (int i = 0; i < RP / 2; ++i) {
      Sj[(size_t)(2 * i) * D] = s[i].x;
      Sj[(size_t)(2 * i + 1) * D] = s[i].y;
    }
  };

  // S <- decay S + k (beta (v - decay S^T k))^T; returns o = S'^T q of the lane's column. The
  // arithmetic of the step kernel's row_update, in its order.
  auto row_update = [&](int t, bool want_o) -> float {
    float4 kk[RP / 4];
#pragma unroll
    for (int i = 0; i < RP / 4; ++i) kk[i] = *reinterpret_cast<const float4*>(&sh.k[t][g * (RP + 4) + 4 * i]);
    const float decay = sh.gate[t][0], beta = sh.gate[t][1], v = sh.v[t][col];
    float pk = 0.f, pq = 0.f;
#pragma unroll
    for (int i = 0; i < RP / 4; ++i) {
      pk = fmaf(s[2 * i].x, kk[i].x, pk);
      pk = fmaf(s[2 * i].y, kk[i].y, pk);
      pk = fmaf(s[2 * i + 1].x, kk[i].z, pk);
      pk = fmaf(s[2 * i + 1].y, kk[i].w, pk);
      if (want_o) {
        const float4 qq = *reinterpret_cast<const float4*>(&sh.q[t][g * (RP + 4) + 4 * i]);
        pq = fmaf(s[2 * i].x, qq.x, pq);
        pq = fmaf(s[2 * i].y, qq.y, pq);
        pq = fmaf(s[2 * i + 1].x, qq.z, pq);
        pq = fmaf(s[2 * i + 1].y, qq.w, pq);
      }
    }
    sh.part[warp][lane & 3][g] = make_float2(pk, pq);
    __syncwarp();
    const float4* parts = reinterpret_cast<const float4*>(sh.part[warp][lane & 3]);
    float4 p[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = parts[i];
    const float2 decay2 = make_float2(decay, decay);
#pragma unroll
    for (int i = 0; i < RP / 2; ++i) s[i] = mul2(decay2, s[i]);  // while the partial sums are on their way
    __syncwarp();  // everybody has read: the next row may write
    float kv = p[0].x, qs = p[0].y;
    kv += p[0].z, qs += p[0].w;
#pragma unroll
    for (int i = 1; i < 4; ++i) {
      kv += p[i].x, qs += p[i].y;
      kv += p[i].z, qs += p[i].w;
    }
    const float delta = (v - decay * kv) * beta;
    const float2 delta2 = make_float2(delta, delta);
#pragma unroll
    for (int i = 0; i < RP / 4; ++i) {
      s[2 * i] = fma2(make_float2(kk[i].x, kk[i].y), delta2, s[2 * i]);
      s[2 * i + 1] = fma2(make_float2(kk[i].z, kk[i].w), delta2, s[2 * i + 1]);
    }
    return want_o ? fmaf(delta, sh.kq[t], decay * qs) : 0.f;
  };

  // ---- replay of the kept rows of the previous pass ----
  for (int u = tid; u < kStaged * D; u += NT) {
    const int t = u / D, i = u - t * D;
    sh.k[t][Shared::at(i)] = a.st_k[((size_t)t * a.Hv + j) * D + i];
  }
  sh.v[warp][lane] = a.st_v[((size_t)warp * a.Hv + j) * D + c0 + lane];  // 8 warps = 8 slots
  if (lane < 2) sh.gate[warp][lane] = a.st_g[(warp * a.Hv + j) * 2 + lane];
  __syncthreads();
  for (int t = 0; t < pend; ++t) row_update(t, false);
  cluster.sync();  // k, v, gate are about to be overwritten, k and q by the other CTAs, too

  // ---- causal convolution + SiLU: tasks of 32 channels x 8 rows, dealt out over the warps, a task's
  // loads in flight together. v: own columns, all rows. q and k are the same in all CTAs of the
  // cluster: each takes every NCTA-th block of 8 rows and hands the normalised rows to the others ----
  constexpr int kQk = 2 * D / 32;
  const int nb = n / 8, mine = (nb - cs + NCTA - 1) / NCTA;
  for (int task = warp; task < kQk * mine + nb; task += kWarps) {
    const bool is_v = task >= kQk * mine;
    const int idx = is_v ? 2 * D + lane : task % kQk * 32 + lane;
    const int t0 = 8 * (is_v ? task - kQk * mine : cs + task / kQk * NCTA);
    const int part_id = idx < D ? 0 : idx < 2 * D ? 1 : 2;
    const int c = part_id == 0 ? idx : part_id == 1 ? idx - D : idx - 2 * D;
    const int ch = part_id == 0 ? i_qk * D + c : part_id == 1 ? a.Hk * D + i_qk * D + c : 2 * a.Hk * D + j * D + c0 + c;
    const bf16* src = a.qkv + (long)t0 * a.ldp + ch;
    bf16 raw[11];
#pragma unroll
    for (int u = 0; u < 3; ++u) {  // the three rows before: of this pass, or from the ring
      const int p = P + t0 - 3 + u;
      const bf16* from = t0 ? src + (long)(u - 3) * a.ldp : a.ring + (size_t)(p & (kRing - 1)) * C + ch;
      raw[u] = *from;
      if (p < 0) raw[u] = tobf16(0.f);
    }
#pragma unroll
    for (int u = 3; u < 11; ++u) raw[u] = src[(long)(u - 3) * a.ldp];
    float x[11], w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) w[u] = tofloat(a.conv_w[ch * 4 + u]);
#pragma unroll
    for (int u = 0; u < 11; ++u) x[u] = tofloat(raw[u]);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      float acc = w[0] * x[u];
      acc = fmaf(w[1], x[u + 1], acc);
      acc = fmaf(w[2], x[u + 2], acc);
      acc = fmaf(w[3], x[u + 3], acc);
      const float y = rnd(silu_acc(rnd(acc)));
      if (part_id == 0) sh.q[t0 + u][Shared::at(c)] = y;
      else if (part_id == 1) sh.k[t0 + u][Shared::at(c)] = y;
      else sh.v[t0 + u][c] = y;
    }
  }
  if (tid < n) {
    const float bt = rnd(sigmoid_acc(tofloat(a.b[(long)tid * a.ldp + j])));
    const float x = tofloat(a.a[(long)tid * a.ldp + j]) + tofloat(a.dt_bias[j]);
    const float sp = x > 20.f ? x : log1pf(expf(x));
    sh.gate[tid][0] = expf(-expf(tofloat(a.A_log[j])) * sp);
    sh.gate[tid][1] = bt;
  }
  __syncthreads();

  // ---- l2norm of q and k and k . q of this CTA's rows, one warp per row, into all CTAs ----
  for (int u8 = warp; u8 < 8 * mine; u8 += kWarps) {
    const int t = 8 * (cs + u8 / 8 * NCTA) + (u8 & 7);
    float eq[NI], ek[NI], sq = 0.f, sk = 0.f;
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      eq[u] = sh.q[t][Shared::at(lane + 32 * u)];
      ek[u] = sh.k[t][Shared::at(lane + 32 * u)];
      sq = fmaf(eq[u], eq[u], sq);
      sk = fmaf(ek[u], ek[u], sk);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
      sk += __shfl_xor_sync(0xffffffffu, sk, o);
    }
    const float iq = rsqrtf(sq + 1e-6f), ik = rsqrtf(sk + 1e-6f);
    float dot = 0.f;
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      eq[u] = (eq[u] * iq) / sqrtf((float)D), ek[u] = ek[u] * ik;
      dot = fmaf(eq[u], ek[u], dot);
    }
    dot = warp_allsum(dot);
#pragma unroll
    for (int rk = 0; rk < NCTA; ++rk) {
      Shared& to = *cluster.map_shared_rank(&sh, rk);
#pragma unroll
      for (int u = 0; u < NI; ++u) {
        to.q[t][Shared::at(lane + 32 * u)] = eq[u];
        to.k[t][Shared::at(lane + 32 * u)] = ek[u];
      }
      if (lane == 0) to.kq[t] = dot;
    }
  }
  // gate inputs of this warp's rows, needed at the very end
  constexpr int kRowsPerWarp = kWideRows / kWarps;
  float zz[kRowsPerWarp];
#pragma unroll
  for (int u = 0; u < kRowsPerWarp; ++u)
    zz[u] = warp + kWarps * u < n ? tofloat(a.z[(long)(warp + kWarps * u) * a.ldp + j * D + c0 + lane]) : 0.f;
  cluster.sync();

  // ---- the recurrence; S is written as it stands before the last 8 rows, which stay pending ----
  for (int t = 0; t < n; ++t) {
    if (t == n - kStaged) store_state();
    const float o = row_update(t, true);
    if (g == 0) sh.o[t][col] = rnd(o);  // the mixer output is a bf16 tensor in the model
  }
  __syncthreads();

  // ---- gated RMSNorm over the head's D outputs, as in the step kernel ----
  float ob[kRowsPerWarp];
#pragma unroll
  for (int u = 0; u < kRowsPerWarp; ++u) {
    const int t = warp + kWarps * u;
    ob[u] = t < n ? sh.o[t][lane] : 0.f;
    const float ssum = warp_allsum(ob[u] * ob[u]);
    if (t < n && lane < NCTA) *cluster.map_shared_rank(&sh.ss[cs][t], lane) = ssum;
  }
  const float nw = tofloat(a.norm_w[c0 + lane]);
  cluster.sync();
#pragma unroll
  for (int u = 0; u < kRowsPerWarp; ++u) {
    const int t = warp + kWarps * u;
    if (t >= n) break;
    float total = 0.f;
#pragma unroll
    for (int rk = 0; rk < NCTA; ++rk) total += sh.ss[rk][t];
    const float nn = rnd(ob[u] * rsqrtf(total / (float)D + a.eps));
    const float y = rnd(nw * nn);
    a.out[(long)t * a.ldo + j * D + c0 + lane] = tobf16(y * silu_acc(zz[u]));
  }
  // ---- checkpoints of the last 8 rows; the cluster barrier lies between them and the replay of the
  // CTAs that read the old ones ----
  for (int u = tid; u < kStaged * kCols; u += NT) {
    const int slot = u >> 5, t = n - kStaged + slot;
    a.st_v[((size_t)slot * a.Hv + j) * D + c0 + (u & 31)] = sh.v[t][u & 31];
  }
  if (cs == 0) {
    for (int u = tid; u < kStaged * D; u += NT) {
      const int slot = u / D, t = n - kStaged + slot;
      a.st_k[((size_t)slot * a.Hv + j) * D + (u - slot * D)] = sh.k[t][Shared::at(u - slot * D)];
    }
    if (tid < 2 * kStaged) a.st_g[((tid >> 1) * a.Hv + j) * 2 + (tid & 1)] = sh.gate[n - kStaged + (tid >> 1)][tid & 1];
  }
}

// Conv history: the last 16 rows (or all 8) of a prefill pass into the ring. A launch of its own,
// because the slots alias the history that the CTAs of other heads read at their start.
__global__ void gdn_ring_kernel(const bf16* qkv, long ldp, bf16* ring, const int* ctl, int n, int C) {
  dep_release();
  dep_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x, t = n - gridDim.y + blockIdx.y;
  if (c < C) ring[(size_t)((ctl[0] + t) & (kRing - 1)) * C + c] = qkv[(long)t * ldp + c];
}

}  // namespace

cudaError_t launch_gdn_ring(const bf16* qkv, long ldp, bf16* ring, const int* ctl, int n, int C, cudaStream_t s, bool pdl) {
  return launch(gdn_ring_kernel, dim3((C + 255) / 256, n < kRing ? n : kRing), dim3(256), 0, s, pdl, qkv, ldp, ring, ctl, n,
                C);
}

namespace {

template <int D>
cudaError_t launch_gdn_prefill(const GdnArgs& g, cudaStream_t s, bool pdl) {
  static bool allowed[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!allowed[dev]) {
    e = cudaFuncSetAttribute(gdn_prefill_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GdnWideShared<D>));
    if (e != cudaSuccess) return e;
    allowed[dev] = true;
  }
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(D / kCols, g.Hv, 1);
  c.blockDim = dim3(kWarps * 32, 1, 1);
  c.dynamicSmemBytes = sizeof(GdnWideShared<D>);
  c.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = D / kCols;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = pdl ? 2 : 1;
  e = cudaLaunchKernelEx(&c, gdn_prefill_kernel<D>, g);
  if (e != cudaSuccess) return e;
  return launch_gdn_ring(g.qkv, g.ldp, g.ring, g.ctl, g.n, (2 * g.Hk + g.Hv) * D, s, pdl);
}

// Off by default: the early state load assumes that no launch on the same state is still in
// flight, which a caller that keeps other kernels between two steps of a layer guarantees.
bool g_gdn_early = false;

template <int D>
cudaError_t launch_gdn(const GdnArgs& g, int Hv, cudaStream_t s, bool pdl) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(D / kCols, Hv, 1);
  c.blockDim = dim3(kWarps * 32, 1, 1);
  c.dynamicSmemBytes = 0;
  c.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = D / kCols;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = pdl ? 2 : 1;
  return cudaLaunchKernelEx(&c, gdn_cluster_kernel<D>, g);
}

}  // namespace
}  // namespace qb

using namespace qb;

extern "C" void qe_set_gdn_early(int on) { g_gdn_early = on != 0; }
extern "C" void qe_set_gdn_phases(int) {}

extern "C" int qe_gdn_step_n(const void* qkv, const void* z, const void* b, const void* a, long ldp,
                             void* ring, const void* conv_w, const void* A_log, const void* dt_bias,
                             const void* norm_w, float* S, float* st_k, float* st_v, float* st_g,
                             const int* ctl, void* out, long ldo, int n, int Hk, int Hv, int D,
                             float eps, int q, void* stream) {
  (void)q;
  if (n < 1 || n > QE_MAX_ROWS || Hk < 1 || Hv < 1 || Hv % Hk) return QE_ERR_ARG;
  GdnArgs g{};
  g.qkv = (const bf16*)qkv; g.z = (const bf16*)z; g.b = (const bf16*)b; g.a = (const bf16*)a;
  g.ldp = ldp; g.ring = (bf16*)ring; g.conv_w = (const bf16*)conv_w; g.A_log = (const bf16*)A_log;
  g.dt_bias = (const bf16*)dt_bias; g.norm_w = (const bf16*)norm_w;
  g.S = S; g.st_k = st_k; g.st_v = st_v; g.st_g = st_g; g.ctl = ctl; g.out = (bf16*)out; g.ldo = ldo;
  g.n = n; g.Hk = Hk; g.Hv = Hv; g.eps = eps; g.early = g_gdn_early ? 1 : 0;
  const bool pdl = pdl_launch_enabled() && pdl_trigger_enabled();
  cudaStream_t s = (cudaStream_t)stream;
  if (D == 128) return (int)launch_gdn<128>(g, Hv, s, pdl);
  if (D == 64) return (int)launch_gdn<64>(g, Hv, s, pdl);
  return QE_ERR_ARG;
}

extern "C" int qe_gdn_prefill(const void* qkv, const void* z, const void* b, const void* a, long ldp,
                              void* ring, const void* conv_w, const void* A_log, const void* dt_bias,
                              const void* norm_w, float* S, float* st_k, float* st_v, float* st_g,
                              const int* ctl, void* out, long ldo, int n, int Hk, int Hv, int D,
                              float eps, void* stream) {
  if (n < QE_MAX_ROWS || n > QE_MAX_GEMM_ROWS || n % QE_MAX_ROWS || Hk < 1 || Hv < 1 || Hv % Hk) return QE_ERR_ARG;
  GdnArgs g{};
  g.qkv = (const bf16*)qkv; g.z = (const bf16*)z; g.b = (const bf16*)b; g.a = (const bf16*)a;
  g.ldp = ldp; g.ring = (bf16*)ring; g.conv_w = (const bf16*)conv_w; g.A_log = (const bf16*)A_log;
  g.dt_bias = (const bf16*)dt_bias; g.norm_w = (const bf16*)norm_w;
  g.S = S; g.st_k = st_k; g.st_v = st_v; g.st_g = st_g; g.ctl = ctl; g.out = (bf16*)out; g.ldo = ldo;
  g.n = n; g.Hk = Hk; g.Hv = Hv; g.eps = eps;
  const bool pdl = pdl_launch_enabled() && pdl_trigger_enabled();
  if (D == 128) return (int)launch_gdn_prefill<128>(g, (cudaStream_t)stream, pdl);
  if (D == 64) return (int)launch_gdn_prefill<64>(g, (cudaStream_t)stream, pdl);
  return QE_ERR_ARG;
}
