// Shared pieces of the flash-attention kernels (forward in attention_sm100.cu, backward in
// attention_bwd_sm100.cu): parameters, swizzled tile stores, operand descriptors, tile loads, tensor maps.
#pragma once
#include "sm100_ptx.cuh"
#include "common.cuh"

namespace gb {

constexpr int AT_BM = 128;   // rows of a score tile (TMEM lanes)
constexpr int AT_BN = 128;   // columns of a score tile
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

struct AttnParams {
  void* o; float* lse;                       // forward outputs
  const float* stats; int Spad;              // backward input: padded row statistics [2][B, Hq, Spad]
  void* dq; void* dk; void* dv;              // backward outputs
  int* status;
  int B, S, Sk, Hq, Hkv;
  int causal, is_bf16;
  float scale;                               // softmax scale
};

// 32 fp32 values of row `row` as 16-bit units u0..u0+3 (16 bytes each) of a 128-byte-swizzled row at `base` (the layout
// TMA SWIZZLE_128B reads and writes).
template <bool BF16>
__device__ __forceinline__ void store_row_chunk_t(uint8_t* base, int u0, int row, const float (&v)[32]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 w;
    w.x = pack2c<BF16>(v[i * 8 + 0], v[i * 8 + 1]);
    w.y = pack2c<BF16>(v[i * 8 + 2], v[i * 8 + 3]);
    w.z = pack2c<BF16>(v[i * 8 + 4], v[i * 8 + 5]);
    w.w = pack2c<BF16>(v[i * 8 + 6], v[i * 8 + 7]);
    *reinterpret_cast<uint4*>(base + (((u0 + i) ^ (row & 7)) << 4)) = w;
  }
}

// K-major operand (contraction inside the 128-byte rows): k-step kk of 16 elements
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t tile_addr, int kk, int rows) {
  return make_smem_desc(tile_addr + (kk >> 2) * rows * 128 + (kk & 3) * 32, 16, 1024);
}
// MN-major operand (contraction over the rows of the tile): k-step kk of 16 rows
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t tile_addr, int kk, int rows) {
  return make_smem_desc(tile_addr + kk * 2048, rows * 128, 1024);
}

template <int D>
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* m, uint64_t* bar, int head, int row0,
                                          int b, int rows) {
#pragma unroll
  for (int dc = 0; dc < D / 64; ++dc) tma_load_4d(dst + dc * rows * 128, m, bar, dc * 64, head, row0, b);
}

#define AT_WAIT(bar, ph, site) mbar_wait((bar), (ph), abort_flag, p.status, (site))

// the same by a whole warp, which stays converged
#define AT_WAIT_ALL(bar, ph, site) __all_sync(0xffffffffu, AT_WAIT(bar, ph, site))

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 2^x for x <= 127 on the FMA pipes, two at a time: x is split into its nearest integer (the low bits of x + 1.5 * 2^23,
// offset by the exponent bias so that a shift turns them into the scale) and a rest in [-1/2, 1/2], whose power is a
// polynomial of degree 5, a least-squares fit on Chebyshev nodes reweighted until its relative error was level: 1.55e-7 in
// exact arithmetic with the constants as rounded here, 2^-22.1 in fp32, as good as ex2.approx.  At -127 the scale's exponent
// bits are all zero, so everything from -126.5 down, -inf included, becomes exactly 0 (ex2.approx.ftz: from -126 down); a
// clamp one higher would leave 2^-126 there, and a row whose scores are all -inf would come out as the mean of V.  NaN
// passes through.
__device__ __forceinline__ float2 poly_exp2(float2 x) {
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x.x) : "f"(-127.f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x.y) : "f"(-127.f));
  constexpr float MAGIC = 12582912.f + 127.f;
  const float2 u = add2(x, make_float2(MAGIC, MAGIC));
  const float2 f = fma2(add2(u, make_float2(-MAGIC, -MAGIC)), make_float2(-1.f, -1.f), x);
  float2 p = fma2(f, make_float2(1.327647129e-3f, 1.327647129e-3f), make_float2(9.675540961e-3f, 9.675540961e-3f));
  p = fma2(p, f, make_float2(5.550713092e-2f, 5.550713092e-2f));
  p = fma2(p, f, make_float2(2.402212024e-1f, 2.402212024e-1f));
  p = fma2(p, f, make_float2(6.931469440e-1f, 6.931469440e-1f));
  p = fma2(p, f, make_float2(1.0000001192f, 1.0000001192f));
  return mul2(p, make_float2(__uint_as_float(__float_as_uint(u.x) << 23), __uint_as_float(__float_as_uint(u.y) << 23)));
}

// ------------------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn4)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static inline EncodeTiledFn4 encode4() {
  static EncodeTiledFn4 fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn4>(ptr);
  }
  return fn;
}

// [B, S, H, D] 16-bit tensor -> map with dims {D, H, S, B}, box {64, 1, 128, 1}, 128-byte swizzle
static inline int make_tmap_bshd(CUtensorMap* out, const void* base, int is_bf16, int B, int S, int H, int D,
                                 int box_rows = 128) {
  EncodeTiledFn4 enc = encode4();
  if (enc == nullptr) return -1;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)D * 2, (cuuint64_t)H * D * 2, (cuuint64_t)S * H * D * 2};
  cuuint32_t box[4] = {64, 1, (cuuint32_t)box_rows, 1};
  cuuint32_t es[4] = {1, 1, 1, 1};
  return (int)enc(out, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                  const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}



// attention of a few query rows (attention_decode_sm100.cu); arguments as checked by gb_attn_fwd.  decode_split: the CTAs that
// share the keys of an item, and how many chunks of keys the longest warp then takes.
void decode_split(const AttnParams& p, int D, int& ranks, int& steps);
int attn_decode(const void* q, const void* k, const void* v, const AttnParams& p, int D, cudaStream_t st);

}  // namespace gb
