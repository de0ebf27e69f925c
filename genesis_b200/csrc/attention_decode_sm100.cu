// Attention of a few query rows against a long key / value cache (decoding steps), forward only, for sm_100a.
//
// A 128-row score tile per query head would be all padding here and would read K and V once per query head.  Instead the
// query rows of all heads of a KV head's group (S * Hq / Hkv of them) are the rows of one 16-row tile, K and V are read
// once per 16 such rows, and the keys are split between the CTAs of a cluster, which combine their partial results
// through distributed shared memory: one launch, no workspace.
//   measured : time on the GPU, inputs cycled past L2: 8 x 1 queries, 32 / 4 heads of 128, 4096 keys: 112 us with 128-row
//              tiles, 18.9 us here (3.6 TB/s of K and V; 64 x 1, 4096 keys: 90 us, 6.0 TB/s); 1 x 1, 14 / 2 heads of 64, 8192
//              keys: 101 -> 12 us.  Launch, ring start and cluster barriers are about 6 us of each: 64 keys take 6.2.  Against the
//              tiled kernel by shape: decode_wins in attention_sm100.cu.
//   bound    : the bytes of K and V.  Every warp streams its own chunks of keys through a private three-stage TMA ring (no
//              barrier between warps in the loop) and multiplies them with mma.sync: with 16 rows the arithmetic is far
//              below what the loads take, and a 128-row tcgen05 tile would be mostly padding.
//   occupancy: 8 KB stages, 4 warps, two CTAs on an SM: 192 KB of loads in flight per SM.
// Statistics, accumulators and partial results are fp32; probabilities are rounded to 16 bits for the second product, as
// in the tiled kernel.
#include "attention_common.cuh"
#include <cooperative_groups.h>

namespace gb {

constexpr int DC_WARPS = 4, DC_ST = 3, DC_ROWS = 16;

template <int D> struct DecCfg {
  static constexpr int KC = D == 128 ? 16 : 32;            // keys per stage
  static constexpr int TILE = KC * D * 2;                  // K or V part of a stage (4 KB)
  static constexpr int RING = DC_ST * 2 * TILE;            // per warp
  static constexpr int PART = DC_ROWS * D * 4;             // a partial result, in the ring's place after the loop
  static constexpr int SMEM = DC_WARPS * RING + 128;
  static_assert(PART <= RING, "partial results replace the ring");
};

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if (BF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// grid: (cluster ranks, row tiles * Hkv, B); row r of a group = query position r / group, head r % group
template <int D, bool BF16>
__global__ void __launch_bounds__(DC_WARPS * 32)
attn_decode_kernel(const __grid_constant__ CUtensorMap tmk, const __grid_constant__ CUtensorMap tmv,
                   const uint16_t* __restrict__ q, const AttnParams p) {
  using C = DecCfg<D>;
  constexpr int KC = C::KC, TILE = C::TILE, NT = KC / 8;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ float sm_m[DC_WARPS][DC_ROWS], sm_l[DC_WARPS][DC_ROWS];
  __shared__ float ct_m[DC_ROWS], ct_l[DC_ROWS];                   // this CTA's result over its warps
  __shared__ int abort_word;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + DC_WARPS * C::RING);     // full[warp][stage]
  volatile int* abort_flag = &abort_word;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = p.Hq / p.Hkv, kvh = (int)blockIdx.y % p.Hkv, tile = (int)blockIdx.y / p.Hkv, b = blockIdx.z;
  const int rows = p.S * group, ranks = gridDim.x, rank = blockIdx.x;
  const int off = p.Sk - p.S;
  const int chunks = (p.Sk + KC - 1) / KC;
  // a poisoned status word or a bad base address leaves no chunks: every CTA still meets the cluster barriers below
  const bool skip = status_poisoned(p.status) || (smem_u32(smem) & 1023) != 0;
  const int c0 = (int)((long long)chunks * rank / ranks) + warp;
  const int c1 = skip ? 0 : (int)((long long)chunks * (rank + 1) / ranks);
  if (threadIdx.x == 0) {
    if ((smem_u32(smem) & 1023) != 0) report_error(p.status, GB_ERR_BAD_ARG, 4, 0);
    abort_word = 0;
    for (int i = 0; i < DC_WARPS * DC_ST; ++i) mbar_init(&bars[i], 1);
    mbar_fence_init();
  }
  __syncthreads();
  uint8_t* ring = smem + warp * C::RING;
  uint64_t* full = bars + warp * DC_ST;
  auto load = [&](int c, int st) {       // one lane
    uint8_t* dst = ring + st * 2 * TILE;
    mbar_expect_tx(&full[st], 2 * TILE);
    load_tile<D>(dst, &tmk, &full[st], kvh, c * KC, b, KC);
    load_tile<D>(dst + TILE, &tmv, &full[st], kvh, c * KC, b, KC);
  };
  if (lane == 0) {
    tma_prefetch_desc(&tmk); tma_prefetch_desc(&tmv);
    for (int i = 0; i < DC_ST; ++i)
      if (c0 + i * DC_WARPS < c1) load(c0 + i * DC_WARPS, i);
  }
  // this thread's rows of the 16: r0 and r0 + 8 of the fragment layout
  int srow[2];
  const uint16_t* qp[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = tile * DC_ROWS + (lane >> 2) + i * 8;
    srow[i] = r < rows ? r / group : -1;
    qp[i] = q + (((size_t)b * p.S + (r < rows ? r / group : 0)) * p.Hq + kvh * group + (r < rows ? r % group : 0)) * D;
  }
  uint32_t qf[D / 16][4];
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
    for (int i = 0; i < 4; ++i)      // a0: row, a1: row + 8, a2 / a3: the same 8 columns on
      qf[kk][i] = srow[i & 1] >= 0 ? *reinterpret_cast<const uint32_t*>(qp[i & 1] + kk * 16 + (i >> 1) * 8 + (lane & 3) * 2) : 0u;
  float o[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[n][i] = 0.f;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  const float sl2 = p.scale * LOG2E;

  int it = 0;
  for (int c = c0; c < c1; c += DC_WARPS, ++it) {
    const int st = it % DC_ST;
    if (!AT_WAIT_ALL(&full[st], (it / DC_ST) & 1, 80)) break;
    const uint32_t aK = smem_u32(ring + st * 2 * TILE), aV = aK + TILE;
    float s[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[n][i] = 0.f;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
        const int row = n * 8 + (lane & 7) + ((lane >> 4) & 1) * 8, unit = (kk & 3) * 2 + ((lane >> 3) & 1);
        uint32_t bk[4];
        ldsm_x4(aK + (kk >> 2) * KC * 128 + row * 128 + ((unit ^ (row & 7)) << 4), bk);
        mma_16816<BF16>(s[n], qf[kk], bk[0], bk[1]);
        mma_16816<BF16>(s[n + 1], qf[kk], bk[2], bk[3]);
      }
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int col = c * KC + n * 8 + (lane & 3) * 2 + (i & 1), sr = srow[i >> 1];
        if (col >= p.Sk || (p.causal && col > sr + off)) s[n][i] = -INFINITY;
        mx[i >> 1] = fmaxf(mx[i >> 1], s[n][i]);
      }
    float alpha[2], nm[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
      const float mn = fmaxf(m[i], mx[i] * sl2);
      nm[i] = mn == -INFINITY ? 0.f : -mn;
      alpha[i] = fast_exp2(m[i] + nm[i]);
      m[i] = mn;
      l[i] *= alpha[i];
    }
    if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
      for (int n = 0; n < D / 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[n][i] *= alpha[i >> 1];
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        s[n][i] = fast_exp2(fmaf(s[n][i], sl2, nm[i >> 1]));
        l[i >> 1] += s[n][i];
      }
#pragma unroll
    for (int kk = 0; kk < KC / 16; ++kk) {
      const uint32_t pa[4] = {pack2c<BF16>(s[2 * kk][0], s[2 * kk][1]), pack2c<BF16>(s[2 * kk][2], s[2 * kk][3]),
                              pack2c<BF16>(s[2 * kk + 1][0], s[2 * kk + 1][1]), pack2c<BF16>(s[2 * kk + 1][2], s[2 * kk + 1][3])};
#pragma unroll
      for (int n = 0; n < D / 8; n += 2) {
        const int row = kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, unit = (n & 7) + ((lane >> 4) & 1);
        uint32_t bv[4];
        ldsm_x4_t(aV + (n >> 3) * KC * 128 + row * 128 + ((unit ^ (row & 7)) << 4), bv);
        mma_16816<BF16>(o[n], pa, bv[0], bv[1]);
        mma_16816<BF16>(o[n + 1], pa, bv[2], bv[3]);
      }
    }
    __syncwarp();                        // all lanes have read the stage
    if (lane == 0 && c + DC_ST * DC_WARPS < c1) load(c + DC_ST * DC_WARPS, st);
  }

  if (__any_sync(0xffffffffu, *abort_flag)) {      // gave up: this warp's last loads have to land first
    const int mine = c1 > c0 ? (c1 - c0 + DC_WARPS - 1) / DC_WARPS : 0;
    drain_copies(full, DC_ST, mine < it + DC_ST ? mine : it + DC_ST);
    __syncwarp();
  }
  // the warps' parts, in shared memory in the place of their rings (every load has arrived and been read)
  float* part = reinterpret_cast<float*>(ring);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    if ((lane & 3) == 0) { sm_m[warp][(lane >> 2) + i * 8] = m[i]; sm_l[warp][(lane >> 2) + i * 8] = l[i]; }
  }
#pragma unroll
  for (int n = 0; n < D / 8; ++n)
#pragma unroll
    for (int i = 0; i < 2; ++i)
      *reinterpret_cast<float2*>(part + ((lane >> 2) + i * 8) * D + n * 8 + (lane & 3) * 2) = make_float2(o[n][2 * i], o[n][2 * i + 1]);
  __syncthreads();
  // weight of a part whose maximum is m against the common maximum
  auto weight = [](float mp, float mc) { return mp == -INFINITY ? 0.f : fast_exp2(mp - mc); };
  float* first = reinterpret_cast<float*>(smem);
  for (int e = threadIdx.x; e < DC_ROWS * D / 4; e += DC_WARPS * 32) {
    const int r = e / (D / 4);
    float mc = -INFINITY, lc = 0.f;
#pragma unroll
    for (int w = 0; w < DC_WARPS; ++w) mc = fmaxf(mc, sm_m[w][r]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < DC_WARPS; ++w) {
      const float wt = weight(sm_m[w][r], mc);
      const float4 v = reinterpret_cast<const float4*>(smem + w * C::RING)[e];
      acc.x += wt * v.x; acc.y += wt * v.y; acc.z += wt * v.z; acc.w += wt * v.w;
      lc += wt * sm_l[w][r];
    }
    reinterpret_cast<float4*>(first)[e] = acc;      // (element e of part 0 is read by this thread only)
    if (e % (D / 4) == 0) { ct_m[r] = mc; ct_l[r] = lc; }
  }
  cluster.sync();
  // ... and the CTAs' parts: every CTA finishes its share of the row tile
  const int total = DC_ROWS * D / 4, e0 = total * rank / ranks, e1 = total * (rank + 1) / ranks;
  for (int e = e0 + (int)threadIdx.x; e < e1 && !skip; e += DC_WARPS * 32) {
    const int rr = e / (D / 4), r = tile * DC_ROWS + rr;
    if (r >= rows) continue;
    float mc = -INFINITY, lc = 0.f;
    for (int k = 0; k < ranks; ++k) mc = fmaxf(mc, cluster.map_shared_rank(ct_m, k)[rr]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < ranks; ++k) {
      const float wt = weight(cluster.map_shared_rank(ct_m, k)[rr], mc);
      const float4 v = reinterpret_cast<const float4*>(cluster.map_shared_rank(first, k))[e];
      acc.x += wt * v.x; acc.y += wt * v.y; acc.z += wt * v.z; acc.w += wt * v.w;
      lc += wt * cluster.map_shared_rank(ct_l, k)[rr];
    }
    const float inv = lc > 0.f ? 1.f / lc : 0.f;
    const int s = r / group, h = kvh * group + r % group, d = e % (D / 4) * 4;
    uint2 w;
    w.x = pack2c<BF16>(acc.x * inv, acc.y * inv);
    w.y = pack2c<BF16>(acc.z * inv, acc.w * inv);
    *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(p.o) + (((size_t)b * p.S + s) * p.Hq + h) * D + d) = w;
    if (d == 0) p.lse[((size_t)b * p.Hq + h) * p.S + s] = lc > 0.f ? (mc + log2f(lc)) * LN2 : -INFINITY;
  }
  cluster.sync();          // nobody leaves while its shared memory is being read
}

// keys are split until two CTAs sit on every SM, as long as a warp keeps two chunks to itself; 8 is the portable limit
void decode_split(const AttnParams& p, int D, int& ranks, int& steps) {
  const int kc = D == 128 ? DecCfg<128>::KC : DecCfg<64>::KC;
  const long long items = ((long long)p.S * (p.Hq / p.Hkv) + DC_ROWS - 1) / DC_ROWS * p.Hkv * p.B;
  const int chunks = (p.Sk + kc - 1) / kc;
  ranks = 1;
  while (ranks < 8 && items * ranks < 2 * sm_count() && chunks >= 4 * ranks * DC_WARPS) ranks *= 2;
  steps = (chunks + ranks * DC_WARPS - 1) / (ranks * DC_WARPS);
}

template <int D, bool BF16>
static int launch_decode(const CUtensorMap& tk, const CUtensorMap& tv, const void* q, const AttnParams& p, cudaStream_t st) {
  using C = DecCfg<D>;
  static unsigned long long cfg = 0;
  int r;
  if ((r = smem_opt_in(attn_decode_kernel<D, BF16>, C::SMEM, cfg)) != 0) return r;
  const int tiles = (p.S * (p.Hq / p.Hkv) + DC_ROWS - 1) / DC_ROWS;
  int ranks, steps;
  decode_split(p, D, ranks, steps);
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(ranks, tiles * p.Hkv, p.B);
  lc.blockDim = dim3(DC_WARPS * 32);
  lc.dynamicSmemBytes = C::SMEM;
  lc.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = ranks; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
  lc.attrs = &at;
  lc.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&lc, attn_decode_kernel<D, BF16>, tk, tv, (const uint16_t*)q, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// (called by gb_attn_fwd, which has checked the arguments)
int attn_decode(const void* q, const void* k, const void* v, const AttnParams& p, int D, cudaStream_t st) {
  CUtensorMap tk, tv;
  int r;
  const int kc = D == 128 ? DecCfg<128>::KC : DecCfg<64>::KC;
  if ((r = make_tmap_bshd(&tk, k, p.is_bf16, p.B, p.Sk, p.Hkv, D, kc)) != 0) return 20000 + r;
  if ((r = make_tmap_bshd(&tv, v, p.is_bf16, p.B, p.Sk, p.Hkv, D, kc)) != 0) return 30000 + r;
  if (D == 64) return p.is_bf16 ? launch_decode<64, true>(tk, tv, q, p, st) : launch_decode<64, false>(tk, tv, q, p, st);
  return p.is_bf16 ? launch_decode<128, true>(tk, tv, q, p, st) : launch_decode<128, false>(tk, tv, q, p, st);
}
}  // namespace gb
