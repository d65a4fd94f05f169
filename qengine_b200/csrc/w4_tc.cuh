// Building blocks of the tensor-memory GEMMs (w4_gemm.cu, w4_rows.cu): tcgen05 wrappers, the unpack of
// the wire format into tensor memory, the epilogue through shared memory.
#pragma once
#include <cuda.h>  // CUtensorMap (types only: the encoder is looked up at run time)

#include "w4_dev.cuh"

namespace qb {
namespace w4 {

constexpr int kGemmWaitLimit = 1 << 20;

// A bounded wait whose verdict is the same in every lane of the (converged) warp.
__device__ __forceinline__ bool warp_wait(uint64_t* b, uint32_t parity, int limit = kGemmWaitLimit) {
  return __all_sync(0xffffffffu, bar_wait(b, parity, limit));
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sa(b)) : "memory");
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t tc_desc(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// D (+)= A * B^T: bf16 x bf16 -> fp32, M = 128, N in the instruction descriptor, K = 16.
__device__ __forceinline__ void tc_mma(uint32_t d, uint32_t a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(sa(bar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t u[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
        "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(u[k]);
}
// One 64-k chunk of a unit (16 bytes of codes per lane) -> 16 rows x 32 words of tensor memory.
__device__ __forceinline__ void tc_st_chunk(uint32_t taddr, const uint4& w) {
  const AFrag f0 = unpack_word(w.x), f1 = unpack_word(w.y), f2 = unpack_word(w.z), f3 = unpack_word(w.w);
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(f0.a0), "r"(f0.a2), "r"(f0.a1), "r"(f0.a3), "r"(f1.a0), "r"(f1.a2), "r"(f1.a1), "r"(f1.a3),
        "r"(f2.a0), "r"(f2.a2), "r"(f2.a1), "r"(f2.a3), "r"(f3.a0), "r"(f3.a2), "r"(f3.a1), "r"(f3.a3)
      : "memory");
}
// Word s of lane t (of the four lanes of a row pair) -> word t of lane s: lane t then holds k = 16 b + 4 t
// .. + 3 in its word b, so that the eight words of a 16-k block are in ascending k and the
// activations need no permutation.
__device__ __forceinline__ void transpose4(uint4& w, int t) {
  const bool hi = t & 2, odd = t & 1;
  const uint32_t r0 = __shfl_xor_sync(0xffffffffu, hi ? w.x : w.z, 2), r1 = __shfl_xor_sync(0xffffffffu, hi ? w.y : w.w, 2);
  const uint32_t y00 = hi ? r0 : w.x, y01 = hi ? r1 : w.y, y10 = hi ? w.z : r0, y11 = hi ? w.w : r1;
  const uint32_t q0 = __shfl_xor_sync(0xffffffffu, odd ? y00 : y01, 1), q1 = __shfl_xor_sync(0xffffffffu, odd ? y10 : y11, 1);
  w = make_uint4(odd ? q0 : y00, odd ? y01 : q0, odd ? q1 : y10, odd ? y11 : q1);
}
// Weights are constant while the kernel runs and read once: no L1 line for them.
__device__ __forceinline__ uint4 ld_codes(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {  // bytes 16, or 0: zero fill
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// 64 rows x 256 k of the activations as four 64-k chunks from chunk c: map dimensions (64 k, rows, chunks).
__device__ __forceinline__ void tma_rows(uint32_t dst, const CUtensorMap* map, int c, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(0), "r"(c), "r"(sa(bar))
      : "memory");
}

// Four consecutive output rows (from `row`) of activation row n.
__device__ __forceinline__ void tc_put4(const OutDesc& o, bool vec, int n, int row, const float4& f, bool wire) {
  if (row >= o.M) return;
  if (wire) row = wire_pos(row);
  const float e[4] = {f.x, f.y, f.z, f.w};
  if (o.out_f32) {
    float* p = static_cast<float*>(o.out) + (long)n * o.ldo + row;
    if (vec && row + 3 < o.M) {
      *reinterpret_cast<float4*>(p) = f;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (row + k < o.M) p[k] = e[k];
    }
  } else {
    bf16* p = static_cast<bf16*>(o.out) + (long)n * o.ldo + row;
    if (vec && row + 3 < o.M) {
      *reinterpret_cast<uint2*>(p) = make_uint2(pack2(f.x, f.y), pack2(f.z, f.w));
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (row + k < o.M) p[k] = tobf16(e[k]);
    }
  }
}
// The finished sums of a super-tile, get(n, m) = those of its rows m .. m + 3, by `threads` threads; wire: the
// columns of an output row in the order of the wire format (wire_pos).
template <typename Get>
__device__ __forceinline__ void tc_store(const OutDesc& o, int tile0, int ti, int threads, Get get, bool wire = false) {
  const bool vec = (o.ldo & 3) == 0 && (reinterpret_cast<uintptr_t>(o.out) & (o.out_f32 ? 15 : 7)) == 0;
  if (o.epi == QE_EPI_SWIGLU) {  // rows 0..7 of a tile are gate rows, 8..15 the matching up rows
#pragma unroll 2
    for (int e = ti; e < o.N * 16; e += threads) {
      const int n = e >> 4, m0 = (e & 14) * 8 + (e & 1) * 4;
      const float4 g = get(n, m0), u = get(n, m0 + 8);
      tc_put4(o, vec, n, tile0 * 8 + (e & 15) * 4,
              make_float4(silu_fast(g.x) * u.x, silu_fast(g.y) * u.y, silu_fast(g.z) * u.z, silu_fast(g.w) * u.w), wire);
    }
  } else {
#pragma unroll 2
    for (int e = ti; e < o.N * 32; e += threads)
      tc_put4(o, vec, e >> 5, tile0 * 16 + (e & 31) * 4, get(e >> 5, (e & 31) * 4), wire);
  }
}
// Tensor map over the rows of x as (64 k, rows, 64-k chunks): boxes of `chunks` chunks of `rows` rows in the
// 128-byte swizzle, rows and chunks beyond the end read as zero. False where a map cannot describe them (rows that overlap, as in an expanded row).
inline bool map_rows(const qe_w4_params* p, int rows, int chunks, CUtensorMap* map) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found);
    return reinterpret_cast<Encode>(e == cudaSuccess && found == cudaDriverEntryPointSuccess ? fn : nullptr);
  }();
  if (!encode || p->ldx < p->K) return false;
  const cuuint64_t dim[3] = {64, (cuuint64_t)p->N, (cuuint64_t)p->K / 64}, stride[2] = {(cuuint64_t)p->ldx * 2, 128};
  const cuuint32_t box[3] = {64, (cuuint32_t)rows, (cuuint32_t)chunks}, step[3] = {1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(p->x), dim, stride, box, step,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}


}  // namespace w4
}  // namespace qb
