// Gated delta rule for 8, 16 .. 128 consecutive rows of a prompt, bit for bit what the step kernel
// (deltanet.cu: the math, the rounding points and the checkpoints) leaves when it is called for 8 rows at a
// time. No counterpart in the reference, which prefills at most 8 rows per pass.
//
// gdn_prefill_kernel does all of it in one launch of thread-block clusters, up to 64 rows. Two blocks of a cluster
// land on one SM (96 of 148 SMs work, and a row of the recurrence, which is bound by the instructions of sixteen
// warps there, takes 340 ns instead of 190), and everything that is not serial waits for the cluster's
// barriers: 41 us for 64 rows, 20 of them without a row being advanced. Here the serial part has a kernel to
// itself, and the rest runs row-parallel before and after it:
//   gdn_conv_kernel   convolution + SiLU, l2 norm of q and k, k . q, gates: every 8 rows of a head pair a block;
//   gdn_ring_kernel   conv history (deltanet.cu);
//   gdn_recur_kernel  replay of the pending rows, the recurrence, the state. A head's columns over three blocks
//                     (44, 44, 40 at D 128: 144 blocks of 11 warps, one per SM, no cluster), lanes as in
//                     gdn_prefill_kernel: (g, c) = (lane / 4, lane % 4) owns rows g D / 8 .. of column c of the warp's
//                     four. q, k and v of all rows come into shared memory in groups of asynchronous copies
//                     while the first rows are already being advanced;
//   gdn_gate_kernel   gated RMSNorm, a warp per row and head, the step kernel's order of additions (sums over 32
//                     columns by shuffles, then the groups ascending); checkpoints of the last 8 rows, which must
//                     not be overwritten before every block has replayed the old ones.
// 128 rows of one DeltaNet layer of the 27B shape: 34 us less than two launches of gdn_prefill_kernel (2 x 41 us and
// two rings).
#include "common.cuh"
#include "w4_dev.cuh"  // wire_pos

namespace qb {
// deltanet.cu
cudaError_t launch_gdn_ring(const bf16* qkv, long ldp, bf16* ring, const int* ctl, int n, int C, cudaStream_t s, bool pdl);
namespace {

constexpr int kRing = 16, kStaged = QE_MAX_ROWS, kRows = QE_MAX_PASS_ROWS;

struct RowsArgs {
  const bf16 *qkv, *z, *b, *a;
  long ldp;
  const bf16 *ring, *conv_w, *A_log, *dt_bias, *norm_w;
  float *S, *st_k, *st_v, *st_g;
  const int* ctl;
  bf16* out;
  long ldo;
  int n, Hk, Hv, wire;
  float eps;
  // workspace: normalised q and k [Hk][n][2][D], k . q [Hk][n], (decay, beta) [Hv][n][2], v and o [Hv][n][D]
  float *qk, *kq, *gate;
  bf16 *v, *o;
};

template <int D>
__global__ void __launch_bounds__(2 * D) gdn_conv_kernel(const RowsArgs a) {
  constexpr int NI = D / 32;
  __shared__ float y[2][8][D];
  dep_release();
  dep_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int half = tid / D, c = tid - half * D, t0 = 8 * blockIdx.y, n = a.n;
  const bool is_v = (int)blockIdx.x >= a.Hk;
  const int head = is_v ? 2 * (blockIdx.x - a.Hk) + half : blockIdx.x;  // value head; q/k head
  if (is_v && head >= a.Hv) return;
  const int ch = is_v ? 2 * a.Hk * D + head * D + c : half * a.Hk * D + head * D + c;
  const int C = 2 * a.Hk * D + a.Hv * D, P = a.ctl[0];
  const bf16* src = a.qkv + (long)t0 * a.ldp + ch;
  bf16 raw[11];
#pragma unroll
  for (int u = 0; u < 3; ++u) {  // the three rows before: of this pass, or from the ring
    const int p = P + t0 - 3 + u;
    raw[u] = t0 ? src[(long)(u - 3) * a.ldp] : a.ring[(size_t)(p & (kRing - 1)) * C + ch];
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
    const bf16 r = tobf16(silu_acc(rnd(acc)));
    if (is_v) a.v[((size_t)head * n + t0 + u) * D + c] = r;
    else y[half][u][c] = tofloat(r);
  }
  if (is_v) {
    if (c < 8) {  // gates of this head's eight rows
      const int t = t0 + c;
      const float bt = rnd(sigmoid_acc(tofloat(a.b[(long)t * a.ldp + head])));
      const float xg = tofloat(a.a[(long)t * a.ldp + head]) + tofloat(a.dt_bias[head]);
      const float sp = xg > 20.f ? xg : log1pf(expf(xg));
      float* to = a.gate + ((size_t)head * n + t) * 2;
      to[0] = expf(-expf(tofloat(a.A_log[head])) * sp);
      to[1] = bt;
    }
    return;
  }
  __syncthreads();
  for (int u8 = warp; u8 < 8; u8 += 2 * D / 32) {  // a warp per row
    float eq[NI], ek[NI], sq = 0.f, sk = 0.f;
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      eq[u] = y[0][u8][lane + 32 * u];
      ek[u] = y[1][u8][lane + 32 * u];
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
    float* to = a.qk + ((size_t)head * n + t0 + u8) * 2 * D;
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      eq[u] = (eq[u] * iq) / sqrtf((float)D), ek[u] = ek[u] * ik;
      dot = fmaf(eq[u], ek[u], dot);
      to[lane + 32 * u] = eq[u];
      to[D + lane + 32 * u] = ek[u];
    }
    dot = warp_allsum(dot);
    if (lane == 0) a.kq[(size_t)head * n + t0 + u8] = dot;
  }
}

// k and q of a row: four floats of padding per eighth, so that the eight eighths' 16-byte loads hit
// different banks.
template <int D>
struct RecurShared {
  static constexpr int RP = D / 8, kPitch = 8 * (RP + 4), kCols = D == 128 ? 44 : 24, kWarps = kCols / 4;
  static __device__ __forceinline__ int at(int i) { return i + i / RP * 4; }
  float q[kRows][kPitch], k[kRows][kPitch];
  float k8[kStaged][kPitch];  // the pending rows
  bf16 v[kRows][kCols];
  float v8[kStaged][kCols];
  float gate[kRows][2], gate8[kStaged][2], kq[kRows];
  float2 part[kWarps][4][8 + 2];  // [warp][column][eighth]: partial sums of S^T k and S^T q
};

template <int D>
__global__ void __launch_bounds__(RecurShared<D>::kWarps * 32, 1) gdn_recur_kernel(const RowsArgs a) {
  using Shared = RecurShared<D>;
  constexpr int RP = Shared::RP, PC = Shared::kCols, NT = Shared::kWarps * 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Shared& sh = *reinterpret_cast<Shared*>(smem_raw);
  dep_release();
  dep_wait();
  const int j = blockIdx.y, c0 = blockIdx.x * PC, nc = min(PC, D - c0);
  const int i_qk = j / (a.Hv / a.Hk), n = a.n, pend = min(max(a.ctl[1], 0), kStaged);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int col = min(4 * warp, nc - 4) + (lane & 3), g = lane >> 2;  // (warps beyond the columns repeat the last four)
  const bool mine = 4 * warp < nc;
  float* Sj = a.S + ((size_t)j * D + g * RP) * D + c0 + col;

  float2 s[RP / 2];
#pragma unroll
  for (int i = 0; i < RP / 2; ++i) s[i] = make_float2(Sj[(size_t)(2 * i) * D], Sj[(size_t)(2 * i + 1) * D]);
  auto store_state = [&] {
    if (!mine) return;
#pragma unroll
    for (int i = 0; i < RP / 2; ++i) {
      Sj[(size_t)(2 * i) * D] = s[i].x;
      Sj[(size_t)(2 * i + 1) * D] = s[i].y;
    }
  };

  // q and k of all rows: a group of copies per 16 rows, in the order in which they are needed
  const int chunks = (n + 15) >> 4;
  for (int b = 0; b < chunks; ++b) {
    for (int e = tid; e < min(16, n - 16 * b) * (D / 2); e += NT) {  // 16-byte pieces: D / 4 of q, D / 4 of k per row
      const int t = 16 * b + e / (D / 2), p = e % (D / 2), i = 4 * (p % (D / 4));
      float* to = (p < D / 4 ? sh.q : sh.k)[t] + Shared::at(i);
      const float* from = a.qk + ((size_t)i_qk * n + t) * 2 * D + 4 * p;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(w4::sa(to)), "l"(from) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int e = tid; e < n * nc / 4; e += NT) {  // four columns at a time
    const int t = e / (nc / 4), c = 4 * (e % (nc / 4));
    *reinterpret_cast<uint2*>(&sh.v[t][c]) = *reinterpret_cast<const uint2*>(a.v + ((size_t)j * n + t) * D + c0 + c);
  }
  for (int e = tid; e < 2 * n; e += NT) sh.gate[e >> 1][e & 1] = a.gate[(size_t)j * n * 2 + e];
  for (int e = tid; e < n; e += NT) sh.kq[e] = a.kq[(size_t)i_qk * n + e];
  for (int e = tid; e < kStaged * D; e += NT) sh.k8[e / D][Shared::at(e % D)] = a.st_k[((size_t)(e / D) * a.Hv + j) * D + e % D];
  for (int e = tid; e < kStaged * nc; e += NT) sh.v8[e / nc][e % nc] = a.st_v[((size_t)(e / nc) * a.Hv + j) * D + c0 + e % nc];
  if (tid < 2 * kStaged) sh.gate8[tid >> 1][tid & 1] = a.st_g[((tid >> 1) * a.Hv + j) * 2 + (tid & 1)];
  __syncthreads();

  // S <- decay S + k (beta (v - decay S^T k))^T; returns o = S'^T q of the lane's column. The
  // arithmetic of the step kernel's row_update, in its order.
  auto row_update = [&](const float* kr, const float* qr, float decay, float beta, float v, float kq, bool want_o) -> float {
    float4 kk[RP / 4];
#pragma unroll
    for (int i = 0; i < RP / 4; ++i) kk[i] = *reinterpret_cast<const float4*>(kr + g * (RP + 4) + 4 * i);
    float pk = 0.f, pq = 0.f;
#pragma unroll
    for (int i = 0; i < RP / 4; ++i) {
      pk = fmaf(s[2 * i].x, kk[i].x, pk);
      pk = fmaf(s[2 * i].y, kk[i].y, pk);
      pk = fmaf(s[2 * i + 1].x, kk[i].z, pk);
      pk = fmaf(s[2 * i + 1].y, kk[i].w, pk);
      if (want_o) {
        const float4 qq = *reinterpret_cast<const float4*>(qr + g * (RP + 4) + 4 * i);
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
    return want_o ? fmaf(delta, kq, decay * qs) : 0.f;
  };

  for (int t = 0; t < pend; ++t) row_update(sh.k8[t], nullptr, sh.gate8[t][0], sh.gate8[t][1], sh.v8[t][col], 0.f, false);
  // S is written as it stands before the last 8 rows, which stay pending
  for (int t = 0; t < n; ++t) {
    if (!(t & 15)) {  // the next 16 rows have landed, for every thread
      switch (chunks - 1 - (t >> 4)) {
        case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
        case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
        case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
        case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
        case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
        case 5: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
        case 6: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
        default: asm volatile("cp.async.wait_group 7;" ::: "memory");
      }
      __syncthreads();
    }
    if (t == n - kStaged) store_state();
    const float o = row_update(sh.k[t], sh.q[t], sh.gate[t][0], sh.gate[t][1], tofloat(sh.v[t][col]), sh.kq[t], true);
    if (g == 0 && mine) a.o[((size_t)j * n + t) * D + c0 + col] = tobf16(o);  // the mixer output is a bf16 tensor in the model
  }
}

template <int D>
__global__ void __launch_bounds__(256) gdn_gate_kernel(const RowsArgs a) {
  constexpr int NI = D / 32;
  dep_release();
  dep_wait();
  const int lane = threadIdx.x & 31, n = a.n, warps = n * a.Hv;
  const int id = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (id < warps) {
    const int t = id / a.Hv, j = id - t * a.Hv;
    float ob[NI], zz[NI], total = 0.f;
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      ob[u] = tofloat(a.o[((size_t)j * n + t) * D + lane + 32 * u]);
      zz[u] = tofloat(a.z[(long)t * a.ldp + j * D + lane + 32 * u]);
    }
#pragma unroll
    for (int u = 0; u < NI; ++u) total += warp_allsum(ob[u] * ob[u]);
    const float inv = rsqrtf(total / (float)D + a.eps);
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      const float nn = rnd(ob[u] * inv);
      const float yy = rnd(tofloat(a.norm_w[lane + 32 * u]) * nn);
      const int e = j * D + lane + 32 * u;
      a.out[(long)t * a.ldo + (a.wire ? w4::wire_pos(e) : e)] = tobf16(yy * silu_acc(zz[u]));
    }
    return;
  }
  // checkpoints of the last 8 rows
  const int e = (id - warps) * 32 + lane, per = a.Hv * D;
  if (e >= kStaged * per) return;
  const int slot = e / per, j = e / D % a.Hv, i = e % D, t = n - kStaged + slot;
  a.st_k[e] = a.qk[(((size_t)(j / (a.Hv / a.Hk)) * n + t) * 2 + 1) * D + i];
  a.st_v[e] = tofloat(a.v[((size_t)j * n + t) * D + i]);
  if (i < 2) a.st_g[(slot * a.Hv + j) * 2 + i] = a.gate[((size_t)j * n + t) * 2 + i];
}

template <int D>
int launch_rows(const RowsArgs& a, bf16* ring, cudaStream_t s, bool pdl) {
  static bool allowed[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
  constexpr size_t smem = sizeof(RecurShared<D>);
  static_assert(smem <= 227 * 1024, "shared memory of one block");
  if (!allowed[dev]) {
    e = cudaFuncSetAttribute(gdn_recur_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    allowed[dev] = true;
  }
  e = launch(gdn_conv_kernel<D>, dim3(a.Hk + (a.Hv + 1) / 2, a.n / 8), dim3(2 * D), 0, s, pdl, a);
  if (e == cudaSuccess) e = launch_gdn_ring(a.qkv, a.ldp, ring, a.ctl, a.n, (2 * a.Hk + a.Hv) * D, s, pdl);
  if (e == cudaSuccess)
    e = launch(gdn_recur_kernel<D>, dim3(3, a.Hv), dim3(RecurShared<D>::kWarps * 32), smem, s, pdl, a);
  const int warps = a.n * a.Hv + kStaged * a.Hv * D / 32;
  if (e == cudaSuccess) e = launch(gdn_gate_kernel<D>, dim3((warps + 7) / 8), dim3(256), 0, s, pdl, a);
  return (int)e;
}

}  // namespace
}  // namespace qb

using namespace qb;

extern "C" long qe_gdn_rows_workspace(int n, int Hk, int Hv, int D) {
  // in bytes: q and k, k . q, gates in fp32; v and o in bf16
  return 4L * ((long)Hk * n * 2 * D + (long)Hk * n + 2L * Hv * n + 4) + 4L * Hv * n * D + 64;
}

extern "C" int qe_gdn_rows(const void* qkv, const void* z, const void* b, const void* a, long ldp, void* ring,
                           const void* conv_w, const void* A_log, const void* dt_bias, const void* norm_w, float* S,
                           float* st_k, float* st_v, float* st_g, const int* ctl, void* out, long ldo, int n, int Hk,
                           int Hv, int D, float eps, int wire_out, void* workspace, void* stream) {
  if (n < QE_MAX_ROWS || n > QE_MAX_PASS_ROWS || n % QE_MAX_ROWS || Hk < 1 || Hv < 1 || Hv % Hk || !workspace ||
      (reinterpret_cast<uintptr_t>(workspace) & 15))
    return QE_ERR_ARG;
  RowsArgs r{};
  r.qkv = (const bf16*)qkv; r.z = (const bf16*)z; r.b = (const bf16*)b; r.a = (const bf16*)a;
  r.ldp = ldp; r.ring = (const bf16*)ring; r.conv_w = (const bf16*)conv_w; r.A_log = (const bf16*)A_log;
  r.dt_bias = (const bf16*)dt_bias; r.norm_w = (const bf16*)norm_w;
  r.S = S; r.st_k = st_k; r.st_v = st_v; r.st_g = st_g; r.ctl = ctl; r.out = (bf16*)out; r.ldo = ldo;
  r.n = n; r.Hk = Hk; r.Hv = Hv; r.eps = eps; r.wire = wire_out ? 1 : 0;
  r.qk = (float*)workspace;
  r.v = (bf16*)(r.qk + (size_t)Hk * n * 2 * D);  // 16-byte aligned: rows of D
  r.o = r.v + (size_t)Hv * n * D;
  r.gate = (float*)(r.o + (size_t)Hv * n * D);
  r.kq = r.gate + 2 * (size_t)Hv * n;
  const bool pdl = pdl_launch_enabled() && pdl_trigger_enabled();
  if (D == 128) return launch_rows<128>(r, (bf16*)ring, (cudaStream_t)stream, pdl);
  if (D == 64) return launch_rows<64>(r, (bf16*)ring, (cudaStream_t)stream, pdl);
  return QE_ERR_ARG;
}
