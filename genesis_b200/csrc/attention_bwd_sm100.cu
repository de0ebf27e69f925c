// Flash-attention backward for sm_100a (tcgen05 / TMEM / TMA): row statistics, dQ kernel, dK/dV kernel.
//
// Both kernels work on score tiles of 128 rows and 128 columns (64 where half_tiles says so) with eight arithmetic warps: two
// warpgroups share a tile by columns, every thread owns one row of its half (one TMEM lane).  A TMA warp feeds a ring of
// operand tiles, an MMA warp issues.  P and dS never pass through shared memory: they are written as 16-bit pairs into tensor
// memory, as the A operand of the GEMM that consumes them.
//   dQ    : CTA = (q tile of 128 rows, head); loop over kv tiles:
//           S = Q K^T, dP = dO V^T, dS = P o (dP - delta) * scale, dQ += dS K          (K tile reused MN-major)
//           S and dP of tile j + 1 are issued as soon as those of tile j are in registers, ahead of dQ(j).
//   dK/dV : CTA = (kv tile of 128 rows, some query heads of its group); loop over those heads and their q tiles:
//           S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q                     (dO, Q tiles reused MN-major)
//           P^T replaces S^T and dS^T replaces dP^T in place, so at D = 128 the four tiles fill the 512 columns; the two
//           halves of an iteration alternate: while the warps form dS^T(i) the tensor cores run dV(i) and S^T(i + 1),
//           while they exponentiate S^T(i + 1) the tensor cores run dK(i) and dP^T(i + 1).
// What bounds them: 3 + 4 GEMMs of 128 x 128 x D per score tile (each 512 clocks at D = 128, 256 at D = 64, at the nominal
// rate) against one exponential per score in each kernel (1024 clocks): the tensor pipe at D = 128, the exponentials at D = 64.
// Measured against the kernels they replace (128 x 64 tiles, four arithmetic warps, at D = 64 two CTAs on an SM, one dK/dV CTA
// per query head with fp32 atomics for every group), whole backward pass, bf16 causal, us: 8 x 2048, 14 / 2 heads of 64:
// 543 -> 281; 4 x 4096, 12 / 2 of 128: 1444 -> 676; 8 x 1024, 16 / 4 of 128: 430 -> 174; 1 x 1003, 14 / 2 of 64: 69 -> 48;
// 64 x 197, 12 / 12 of 64: 125 -> 113; 512 x 64, 8 / 8 of 64: 168 -> 163.
// Reference counterpart: genesis/nn/attention.py:162-406 (Triton, 32 x 32 tiles, Hq == Hkv only).
#include "attention_common.cuh"

namespace gb {

constexpr int BW_THREADS = 320;     // 2 x 4 arithmetic warps, TMA warp, MMA warp

// CN: columns of a score tile.  128, or 64 for short rows (see half_tiles): at D = 64 the half tiles leave room for two CTAs on
// an SM, in tensor memory (256 columns each) and in shared memory.
template <int D, int CN> struct BwdCfg {
  static constexpr int TILE = AT_BM * D * 2;                    // one [128 x D] 16-bit tile
  static constexpr int CTILE = CN * D * 2;                      // one [CN x D] tile: what a score tile's columns come from
  static constexpr int ST = D == 64 ? 3 : 2;                    // stages of the operand ring (two CN-row tiles each)
  static constexpr int STATS = 2 * CN * 4;                      // -lse (log2 domain) and -delta of a q tile
  static constexpr int SMEM_DQ = 2 * TILE + ST * 2 * CTILE + 256;
  static constexpr int SMEM_KV = 2 * TILE + ST * (2 * CTILE + STATS) + 256;
  static constexpr int TM_DQ = CN * 5 / 2 + D <= 256 ? 256 : 512;   // tensor-memory columns: S, dP, dS (16-bit), dQ
  static constexpr int TM_KV = 2 * CN + 2 * D <= 256 ? 256 : 512;   // S^T, dP^T, dV, dK
  static constexpr int CTAS = D == 64 && CN == 64 ? 2 : 1;          // on an SM
};

// HC consecutive fp32 columns of a lane (32 or 64), and HC / 2 packed ones back
template <int HC> __device__ __forceinline__ void tmem_ld_cols(uint32_t addr, uint32_t (&r)[HC / 32][32]) {
  tmem_ld_32x32b_x32(addr, r[0]);
  if constexpr (HC == 64) tmem_ld_32x32b_x32(addr + 32, r[1]);
  tmem_ld_wait();
}
__device__ __forceinline__ void tmem_st_cols(uint32_t addr, const uint32_t (&r)[32]) { tmem_st_32x32b_x32(addr, r); }
__device__ __forceinline__ void tmem_st_cols(uint32_t addr, const uint32_t (&r)[16]) { tmem_st_32x32b_x16(addr, r); }

__device__ __forceinline__ void store_out_row(uint16_t* dst, uint32_t tsrc, int ncols, bool valid, int dt,
                                              float mul = 1.f) {
#pragma unroll 1
  for (int c = 0; c < ncols; c += 32) {
    uint32_t r[32];
    tmem_ld_32x32b_x32(tsrc + c, r);
    tmem_ld_wait();
    if (valid) {
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        uint4 w;
        w.x = pack2(__uint_as_float(r[i]) * mul, __uint_as_float(r[i + 1]) * mul, dt);
        w.y = pack2(__uint_as_float(r[i + 2]) * mul, __uint_as_float(r[i + 3]) * mul, dt);
        w.z = pack2(__uint_as_float(r[i + 4]) * mul, __uint_as_float(r[i + 5]) * mul, dt);
        w.w = pack2(__uint_as_float(r[i + 6]) * mul, __uint_as_float(r[i + 7]) * mul, dt);
        *reinterpret_cast<uint4*>(dst + c + i) = w;
      }
    }
  }
}

// =====================================================================================================
// dQ
// =====================================================================================================
template <int D, int CN, bool BF16>
__global__ void __launch_bounds__(BW_THREADS, BwdCfg<D, CN>::CTAS)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmq, const __grid_constant__ CUtensorMap tmk,
                   const __grid_constant__ CUtensorMap tmv, const __grid_constant__ CUtensorMap tmdo,
                   const AttnParams p) {
  using C = BwdCfg<D, CN>;
  constexpr int TILE = C::TILE, CTILE = C::CTILE, ST = C::ST, HC = CN / 2;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if (status_poisoned(p.status)) return;
  if ((reinterpret_cast<uintptr_t>(smem_raw) & 1023) != 0) {
    if (threadIdx.x == 0) report_error(p.status, GB_ERR_BAD_ARG, 2, 0);
    return;
  }
  uint8_t* sQ = smem_raw;
  uint8_t* sdO = sQ + TILE;
  uint8_t* sKV = sdO + TILE;         // ST stages of (K, V)
  uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + ST * 2 * CTILE);
  uint64_t* qdo_full = bars;
  uint64_t* s_full = bars + 1;
  uint64_t* dp_full = bars + 2;
  uint64_t* s_free = bars + 3;
  uint64_t* dp_free = bars + 4;
  uint64_t* ds_ready = bars + 5;
  uint64_t* acc_done = bars + 6;
  uint64_t* kv_full = bars + 7;      // [ST]
  uint64_t* kv_empty = bars + 7 + ST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 7 + 2 * ST);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int bh = p.B * p.Hq, nq = (p.S + AT_BM - 1) / AT_BM;
  const int qt = nq - 1 - (int)blockIdx.x / bh;           // longest (last) rows first
  const int h = (int)blockIdx.x % bh % p.Hq, b = (int)blockIdx.x % bh / p.Hq;
  const int kvh = h / (p.Hq / p.Hkv);
  const int m0 = qt * AT_BM;
  const int off = p.Sk - p.S;
  int n_kv = (p.Sk + CN - 1) / CN;
  if (p.causal) {
    const int lim = (m0 + AT_BM + off + CN - 1) / CN;
    n_kv = lim < n_kv ? lim : n_kv;
  }
  if (n_kv < 1) n_kv = 1;

  if (threadIdx.x == 0) {
    mbar_init(qdo_full, 1); mbar_init(s_full, 1); mbar_init(dp_full, 1); mbar_init(acc_done, 1);
    mbar_init(s_free, 256); mbar_init(dp_free, 256); mbar_init(ds_ready, 256);
    for (int i = 0; i < ST; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) { tmem_alloc(tmem_slot, C::TM_DQ); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem, tdP = tmem + CN, tdS = tmem + 2 * CN, tdQ = tmem + 2 * CN + HC;   // CN + CN + CN / 2 + D columns

  if (warp == 8) {
    if (lane == 0) {   // ---------------- TMA ----------------
      mbar_expect_tx(qdo_full, 2 * TILE);
      load_tile<D>(sQ, &tmq, qdo_full, h, m0, b, AT_BM);
      load_tile<D>(sdO, &tmdo, qdo_full, h, m0, b, AT_BM);
      int j = 0;
      for (; j < n_kv; ++j) {
        const int st = j % ST;
        if (!AT_WAIT(&kv_empty[st], ((j / ST) & 1) ^ 1, 40)) break;
        mbar_expect_tx(&kv_full[st], 2 * CTILE);
        load_tile<D>(sKV + st * 2 * CTILE, &tmk, &kv_full[st], kvh, j * CN, b, CN);
        load_tile<D>(sKV + st * 2 * CTILE + CTILE, &tmv, &kv_full[st], kvh, j * CN, b, CN);
      }
      if (*abort_flag) { drain_copies(qdo_full, 1, 1); drain_copies(kv_full, ST, j); }
    }
  } else if (warp == 9) {
    // ---------------- MMA: the warp stays converged, one elected lane issues ----------------
    constexpr uint32_t fmt = BF16 ? 1u : 0u;
    constexpr uint32_t idesc_s = make_idesc(fmt, 0, 0, AT_BM, CN);
    constexpr uint32_t idesc_dq = make_idesc(fmt, 0, 1, AT_BM, D);
    const uint32_t aQ = smem_u32(sQ), adO = smem_u32(sdO), aKV = smem_u32(sKV);
    auto score = [&](uint32_t d, uint32_t a, uint32_t bb, uint64_t* done) {
      const uint64_t da = desc_kmajor(a, 0, AT_BM), db = desc_kmajor(bb, 0, CN);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)        // (descriptors count 16-byte units)
          umma_f16(d, da + (kk >> 2) * (AT_BM * 128 / 16) + (kk & 3) * 2, db + (kk >> 2) * (CN * 128 / 16) + (kk & 3) * 2,
                   idesc_s, kk > 0);
        umma_commit(done);
      }
      __syncwarp();
    };
    bool ok = AT_WAIT_ALL(qdo_full, 0, 41) && AT_WAIT_ALL(&kv_full[0], 0, 42);
    if (ok) {
      tc_fence_after_sync();
      score(tS, aQ, aKV, s_full);
      score(tdP, adO, aKV + CTILE, dp_full);
    }
    for (int j = 0; ok && j < n_kv; ++j) {
      if (j + 1 < n_kv) {
        const int st = (j + 1) % ST;
        if (!(ok = AT_WAIT_ALL(&kv_full[st], ((j + 1) / ST) & 1, 43) && AT_WAIT_ALL(s_free, j & 1, 44))) break;
        tc_fence_after_sync();
        score(tS, aQ, aKV + st * 2 * CTILE, s_full);
        if (!(ok = AT_WAIT_ALL(dp_free, j & 1, 45))) break;
        tc_fence_after_sync();
        score(tdP, adO, aKV + st * 2 * CTILE + CTILE, dp_full);
      }
      if (!(ok = AT_WAIT_ALL(ds_ready, j & 1, 46))) break;
      tc_fence_after_sync();
      const uint64_t dk = desc_mnmajor(aKV + (j % ST) * 2 * CTILE, 0, CN);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < CN / 16; ++kk)
          umma_f16_ts(tdQ, tdS + kk * 8, dk + kk * (2048 / 16), idesc_dq, j > 0 || kk > 0);
        umma_commit(acc_done);
        umma_commit(&kv_empty[j % ST]);
      }
      __syncwarp();
    }
  } else {
    const int half = warp >> 2;                          // columns half * HC .. + HC - 1 of every score tile
    const int row = m0 + (threadIdx.x & 127);
    const uint32_t lane_base = ((uint32_t)((warp & 3) * 32)) << 16;
    const float sl2 = p.scale * LOG2E;
    const float2 sl2v = make_float2(sl2, sl2);
    const float* stat = p.stats + ((size_t)b * p.Hq + h) * p.Spad + row;
    const float nl = stat[0], nd = stat[(size_t)p.B * p.Hq * p.Spad];
    const float2 nlv = make_float2(nl, nl), ndv = make_float2(nd, nd);
    bool ok = true;
    for (int j = 0; j < n_kv; ++j) {
      if (!(ok = AT_WAIT_ALL(s_full, j & 1, 50))) break;
      tc_fence_after_sync();
      float pr[HC];
      {
        uint32_t s[HC / 32][32];
        tmem_ld_cols<HC>(tS + lane_base + half * HC, s);
        tc_fence_before_sync();
        mbar_arrive(s_free);
        const int col0 = j * CN;
        if ((col0 + CN > p.Sk) || (p.causal && (col0 + CN - 1 > m0 + off)) || (m0 + AT_BM > p.S)) {
          // masked scores become -inf (probability 0) in a pass of their own: the main loop stays branch-free
          int lim = p.causal ? row + off : p.Sk - 1;            // last visible column of this row
          lim = lim < p.Sk - 1 ? lim : p.Sk - 1;
          if (row >= p.S) lim = -1;
          lim -= col0 + half * HC;
#pragma unroll
          for (int c = 0; c < HC / 32; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i) s[c][i] = (c * 32 + i <= lim) ? s[c][i] : 0xff800000u;
        }
#pragma unroll
        for (int i = 0; i < HC; i += 2) {
          const float2 x = fma2(make_float2(__uint_as_float(s[i >> 5][i & 31]), __uint_as_float(s[i >> 5][(i & 31) + 1])),
                                sl2v, nlv);
          pr[i] = fast_exp2(x.x);
          pr[i + 1] = fast_exp2(x.y);
        }
      }
      if (!(ok = AT_WAIT_ALL(dp_full, j & 1, 51))) break;
      tc_fence_after_sync();
      uint32_t dp[HC / 32][32], ds[HC / 2];
      tmem_ld_cols<HC>(tdP + lane_base + half * HC, dp);
      tc_fence_before_sync();
      mbar_arrive(dp_free);
      // dS = P o (dP - delta) as 16-bit pairs (the softmax scale is applied once, to dQ at the end)
#pragma unroll
      for (int i = 0; i < HC; i += 2) {
        const float2 d = mul2(make_float2(pr[i], pr[i + 1]),
                              add2(make_float2(__uint_as_float(dp[i >> 5][i & 31]), __uint_as_float(dp[i >> 5][(i & 31) + 1])), ndv));
        ds[i / 2] = pack2c<BF16>(d.x, d.y);
      }
      // dS is single-buffered: the previous tile's dQ MMA has to be done reading it
      if (j > 0 && !(ok = AT_WAIT_ALL(acc_done, (j - 1) & 1, 52))) break;
      tc_fence_after_sync();
      tmem_st_cols(tdS + lane_base + half * (HC / 2), ds);
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(ds_ready);
    }
    if (ok && AT_WAIT_ALL(acc_done, (n_kv - 1) & 1, 53)) {
      tc_fence_after_sync();
      uint16_t* drow = reinterpret_cast<uint16_t*>(p.dq) + (((size_t)b * p.S + row) * p.Hq + h) * D + half * (D / 2);
      store_out_row(drow, tdQ + lane_base + half * (D / 2), D / 2, row < p.S, BF16 ? DT_BF16 : DT_F16, p.scale);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) { tc_fence_after_sync(); tmem_dealloc(tmem, C::TM_DQ); }
}

// =====================================================================================================
// dK / dV.  One CTA per (kv tile of 128 rows, `1 / splits` of the query heads of a KV head's group, batch).  With
// splits == 1 the CTA owns its output rows and stores them; otherwise (too few kv tiles to fill the GPU with whole
// groups) the parts are added into an fp32 workspace with vector atomics.
// =====================================================================================================
template <int D, int CN, bool BF16>
__global__ void __launch_bounds__(BW_THREADS, BwdCfg<D, CN>::CTAS)
attn_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmq, const __grid_constant__ CUtensorMap tmk,
                     const __grid_constant__ CUtensorMap tmv, const __grid_constant__ CUtensorMap tmdo,
                     const AttnParams p, float* __restrict__ ws, const int splits) {
  using C = BwdCfg<D, CN>;
  constexpr int TILE = C::TILE, CTILE = C::CTILE, ST = C::ST, STAGE = 2 * CTILE, HC = CN / 2;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if (status_poisoned(p.status)) return;
  if ((reinterpret_cast<uintptr_t>(smem_raw) & 1023) != 0) {
    if (threadIdx.x == 0) report_error(p.status, GB_ERR_BAD_ARG, 3, 0);
    return;
  }
  uint8_t* sK = smem_raw;
  uint8_t* sV = sK + TILE;
  uint8_t* sQ = sV + TILE;           // ST stages of (Q, dO)
  uint8_t* sStat = sQ + ST * STAGE;  // ST stages of CN x (-lse), CN x (-delta)
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + ST * C::STATS);
  uint64_t* kv_full = bars;
  uint64_t* s_full = bars + 1;
  uint64_t* dp_full = bars + 2;
  uint64_t* p_ready = bars + 3;
  uint64_t* ds_ready = bars + 4;
  uint64_t* acc_done = bars + 5;
  uint64_t* q_full = bars + 6;       // [ST]
  uint64_t* q_empty = bars + 6 + ST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 6 + 2 * ST);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int group = p.Hq / p.Hkv, parts = p.Hkv * splits;
  const int r = (int)blockIdx.x % (parts * p.B), hs = r % parts, b = r / parts;
  const int n0 = (int)blockIdx.x / (parts * p.B) * AT_BM;     // first kv tiles first: they see the most queries
  const int kvh = hs / splits, part = hs % splits;
  const int h0 = kvh * group + part * group / splits, h1 = kvh * group + (part + 1) * group / splits;
  const int off = p.Sk - p.S;
  const int nq = (p.S + CN - 1) / CN;
  int i_start = 0;
  if (p.causal) { const int first = n0 - off; i_start = first > 0 ? first / CN : 0; }
  const int nqv = nq > i_start ? nq - i_start : 0;
  const int n_it = nqv * (h1 - h0);

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1); mbar_init(s_full, 1); mbar_init(dp_full, 1); mbar_init(acc_done, 1);
    mbar_init(p_ready, 256); mbar_init(ds_ready, 256);
    for (int i = 0; i < ST; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) { tmem_alloc(tmem_slot, C::TM_KV); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem, tdP = tmem + CN, tdV = tmem + 2 * CN, tdK = tmem + 2 * CN + D;

  if (warp == 8) {
    if (lane == 0 && n_it > 0) {   // ---------------- TMA ----------------
      mbar_expect_tx(kv_full, 2 * TILE);
      load_tile<D>(sK, &tmk, kv_full, kvh, n0, b, AT_BM);
      load_tile<D>(sV, &tmv, kv_full, kvh, n0, b, AT_BM);
      const size_t half = (size_t)p.B * p.Hq * p.Spad;
      int h = h0, qt = i_start, it = 0;
      for (; it < n_it; ++it) {
        const int st = it % ST;
        if (!AT_WAIT(&q_empty[st], ((it / ST) & 1) ^ 1, 60)) break;
        mbar_expect_tx(&q_full[st], STAGE + C::STATS);
        load_tile<D>(sQ + st * STAGE, &tmq, &q_full[st], h, qt * CN, b, CN);
        load_tile<D>(sQ + st * STAGE + CTILE, &tmdo, &q_full[st], h, qt * CN, b, CN);
        const float* src = p.stats + ((size_t)b * p.Hq + h) * p.Spad + (size_t)qt * CN;
        bulk_load(sStat + st * C::STATS, src, CN * 4, &q_full[st]);
        bulk_load(sStat + st * C::STATS + CN * 4, src + half, CN * 4, &q_full[st]);
        if (++qt == nq) { qt = i_start; ++h; }
      }
      if (*abort_flag) { drain_copies(kv_full, 1, 1); drain_copies(q_full, ST, it); }
    }
  } else if (warp == 9) {
    // ---------------- MMA: the warp stays converged, one elected lane issues ----------------
    constexpr uint32_t fmt = BF16 ? 1u : 0u;
    constexpr uint32_t idesc_s = make_idesc(fmt, 0, 0, AT_BM, CN);
    constexpr uint32_t idesc_acc = make_idesc(fmt, 0, 1, AT_BM, D);
    const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aQ = smem_u32(sQ);
    auto score = [&](uint32_t d, uint32_t a, uint32_t bb, uint64_t* done) {
      const uint64_t da = desc_kmajor(a, 0, AT_BM), db = desc_kmajor(bb, 0, CN);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)        // (descriptors count 16-byte units)
          umma_f16(d, da + (kk >> 2) * (AT_BM * 128 / 16) + (kk & 3) * 2, db + (kk >> 2) * (CN * 128 / 16) + (kk & 3) * 2,
                   idesc_s, kk > 0);
        umma_commit(done);
      }
      __syncwarp();
    };
    // acc (+)= A B: A = 16-bit pairs in tensor memory, the first half of the columns of each half tile (each warpgroup
    // packs into the columns it read), B = an operand tile as MN-major
    auto accumulate = [&](uint32_t d, uint32_t a, uint32_t tile, bool first) {
      const uint64_t db = desc_mnmajor(tile, 0, CN);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < CN / 16; ++kk)
          umma_f16_ts(d, a + kk / (HC / 16) * HC + kk % (HC / 16) * 8, db + kk * (2048 / 16), idesc_acc, !first || kk > 0);
      }
      __syncwarp();
    };
    bool ok = n_it > 0 && AT_WAIT_ALL(kv_full, 0, 61) && AT_WAIT_ALL(&q_full[0], 0, 62);
    if (ok) {
      tc_fence_after_sync();
      score(tS, aK, aQ, s_full);
      score(tdP, aV, aQ + CTILE, dp_full);
    }
    for (int it = 0; ok && it < n_it; ++it) {
      const uint32_t cur = aQ + (it % ST) * STAGE, nxt = aQ + ((it + 1) % ST) * STAGE;
      const bool more = it + 1 < n_it;
      if (!(ok = AT_WAIT_ALL(p_ready, it & 1, 63))) break;
      tc_fence_after_sync();
      accumulate(tdV, tS, cur + CTILE, it == 0);
      if (more) {
        if (!(ok = AT_WAIT_ALL(&q_full[(it + 1) % ST], ((it + 1) / ST) & 1, 64))) break;
        tc_fence_after_sync();
        score(tS, aK, nxt, s_full);
      }
      if (!(ok = AT_WAIT_ALL(ds_ready, it & 1, 65))) break;
      tc_fence_after_sync();
      accumulate(tdK, tdP, cur, it == 0);
      if (elect_one()) umma_commit(more ? &q_empty[it % ST] : acc_done);
      __syncwarp();
      if (more) score(tdP, aV, nxt + CTILE, dp_full);
    }
  } else {
    const int half = warp >> 2;                          // columns half * HC .. + HC - 1 of every score tile
    const int kvrow = n0 + (threadIdx.x & 127);
    const uint32_t lane_base = ((uint32_t)((warp & 3) * 32)) << 16;
    const uint32_t tSh = tS + lane_base + half * HC, tdPh = tdP + lane_base + half * HC;
    const float sl2 = p.scale * LOG2E;
    const float2 sl2v = make_float2(sl2, sl2);
    bool ok = true;
    int qt = i_start;
    for (int it = 0; it < n_it; ++it) {
      const int q0 = qt * CN + half * HC;
      if (++qt == nq) qt = i_start;
      const int st = it % ST;
      const float4* nl = reinterpret_cast<const float4*>(sStat + st * C::STATS + half * HC * 4);
      const float4* nd = reinterpret_cast<const float4*>(sStat + st * C::STATS + CN * 4 + half * HC * 4);
      // (the statistics are this stage's own: seen through the barrier that their copy completed on)
      if (!(ok = AT_WAIT_ALL(&q_full[st], (it / ST) & 1, 70) && AT_WAIT_ALL(s_full, it & 1, 71))) break;
      tc_fence_after_sync();
      float pr[HC];
      {
        uint32_t s[HC / 32][32], pk[HC / 2];
        tmem_ld_cols<HC>(tSh, s);
        if ((q0 + HC > p.S) || (n0 + AT_BM > p.Sk) || (p.causal && (n0 + AT_BM - 1 > q0 + off))) {
          // this kv row is visible to query columns first..last of the half tile
          const int first = p.causal ? kvrow - off - q0 : 0;
          const int last = kvrow < p.Sk ? p.S - 1 - q0 : -1;
#pragma unroll
          for (int c = 0; c < HC / 32; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              s[c][i] = (c * 32 + i >= first && c * 32 + i <= last) ? s[c][i] : 0xff800000u;   // -inf: probability 0
        }
#pragma unroll
        for (int i = 0; i < HC; i += 4) {
          const float4 n4 = nl[i / 4];
          const uint32_t* v = &s[i >> 5][i & 31];
          const float2 x = fma2(make_float2(__uint_as_float(v[0]), __uint_as_float(v[1])), sl2v, make_float2(n4.x, n4.y));
          const float2 y = fma2(make_float2(__uint_as_float(v[2]), __uint_as_float(v[3])), sl2v, make_float2(n4.z, n4.w));
          pr[i] = fast_exp2(x.x); pr[i + 1] = fast_exp2(x.y); pr[i + 2] = fast_exp2(y.x); pr[i + 3] = fast_exp2(y.y);
          pk[i / 2] = pack2c<BF16>(pr[i], pr[i + 1]);
          pk[i / 2 + 1] = pack2c<BF16>(pr[i + 2], pr[i + 3]);
        }
        tmem_st_cols(tSh, pk);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(p_ready);
      if (!(ok = AT_WAIT_ALL(dp_full, it & 1, 72))) break;
      tc_fence_after_sync();
      uint32_t dp[HC / 32][32], ds[HC / 2];
      tmem_ld_cols<HC>(tdPh, dp);
#pragma unroll
      for (int i = 0; i < HC; i += 4) {       // (the softmax scale is applied once, to dK at the end)
        const float4 n4 = nd[i / 4];
        const uint32_t* v = &dp[i >> 5][i & 31];
        const float2 x = mul2(make_float2(pr[i], pr[i + 1]),
                              add2(make_float2(__uint_as_float(v[0]), __uint_as_float(v[1])), make_float2(n4.x, n4.y)));
        const float2 y = mul2(make_float2(pr[i + 2], pr[i + 3]),
                              add2(make_float2(__uint_as_float(v[2]), __uint_as_float(v[3])), make_float2(n4.z, n4.w)));
        ds[i / 2] = pack2c<BF16>(x.x, x.y);
        ds[i / 2 + 1] = pack2c<BF16>(y.x, y.y);
      }
      tmem_st_cols(tdPh, ds);
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(ds_ready);
    }
    // the first warpgroup writes dV, the second dK
    const size_t orow = (((size_t)b * p.Sk + kvrow) * p.Hkv + kvh) * D;
    const bool valid = kvrow < p.Sk;
    uint16_t* out = reinterpret_cast<uint16_t*>(half ? p.dk : p.dv) + orow;
    const uint32_t src = (half ? tdK : tdV) + lane_base;
    const float mul = half ? p.scale : 1.f;
    if (n_it == 0) {
      // no query row sees this kv tile: its gradient is zero (only the owning-store path has to write it)
      if (ws == nullptr && valid)
        for (int i = 0; i < D / 8; ++i) reinterpret_cast<uint4*>(out)[i] = make_uint4(0, 0, 0, 0);
    } else if (ok && AT_WAIT_ALL(acc_done, 0, 73)) {
      tc_fence_after_sync();
      if (ws == nullptr) {
        store_out_row(out, src, D, valid, BF16 ? DT_BF16 : DT_F16, mul);
      } else {
        // ws = [2][B, Sk, Hkv, D] fp32: dK first, dV second
        float* dst = ws + (half ? 0 : (size_t)p.B * p.Sk * p.Hkv * D) + orow;
#pragma unroll 1
        for (int c = 0; c < D; c += 32) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(src + c, v);
          tmem_ld_wait();
          if (valid) {
#pragma unroll
            for (int i = 0; i < 32; i += 4)
              atomicAdd(reinterpret_cast<float4*>(dst + c + i),
                        make_float4(__uint_as_float(v[i]) * mul, __uint_as_float(v[i + 1]) * mul,
                                    __uint_as_float(v[i + 2]) * mul, __uint_as_float(v[i + 3]) * mul));
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) { tc_fence_after_sync(); tmem_dealloc(tmem, C::TM_KV); }
}

// Row statistics of the backward kernels, rows padded to whole q tiles: stats[0][b, h, s] = -lse in the log2 domain (-inf
// behind the last row: probability 0), stats[1][b, h, s] = -sum_d dO * O.  D / 8 lanes per row, 16 bytes per lane; the lanes
// of row s also write the padding of rows S + s, 2 S + s, ...  (With rows of their own for the padding, and 64-bit indices, the
// backward of 128 x 16 rows, 16 / 16 heads of 64 took 86 us instead of 76.  No GPU holds 2^31 rows of 128 bytes and more.)
template <typename T, int D>
__global__ void attn_stats_kernel(const T* __restrict__ o, const T* __restrict__ dout, const float* __restrict__ lse,
                                  float* __restrict__ stats, unsigned B, unsigned S, unsigned Spad, unsigned H) {
  constexpr unsigned LPR = D / 8;            // lanes per row (8 or 16)
  const unsigned rows = B * S * H;
  const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x / LPR;
  const unsigned sub = tid % LPR;
  // whole warps leave the loop together: rows per pass is a multiple of the rows a warp covers
  for (unsigned r0 = tid / LPR; r0 - (threadIdx.x & 31) / LPR < rows; r0 += step) {
    const unsigned h = r0 % H, bs = r0 / H, s = bs % S, b = bs / S;
    const bool live = r0 < rows;
    float acc = 0.f;
    if (live) {
      const long long at = (long long)r0 * D + sub * 8;
      const Vec16<T> a = ld16(o + at);
      const Vec16<T> g = ld16(dout + at);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc += Cvt<T>::to_f(a.v[i]) * Cvt<T>::to_f(g.v[i]);
    }
#pragma unroll
    for (int m = LPR / 2; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if (live) {
      const size_t head = (size_t)(b * H + h) * Spad, half = (size_t)B * H * Spad;
      if (sub == 0) {
        stats[head + s] = -lse[(size_t)(b * H + h) * S + s] * LOG2E;
        stats[half + head + s] = -acc;
      }
      for (unsigned pad = S + s + sub * S; pad < Spad; pad += LPR * S) {
        stats[head + pad] = -INFINITY;
        stats[half + head + pad] = 0.f;
      }
    }
  }
}

// fp32 workspace [2][n] (dK, dV) -> the 16-bit gradients
template <typename T>
__global__ void attn_dkv_convert_kernel(const float* __restrict__ ws, T* __restrict__ dk, T* __restrict__ dv,
                                        long long n) {
  const long long n4 = n >> 2;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < 2 * n4;
       i += (long long)gridDim.x * blockDim.x) {
    const bool second = i >= n4;
    const long long j = second ? i - n4 : i;
    const float4 v = reinterpret_cast<const float4*>(ws + (second ? n : 0))[j];
    T* dst = (second ? dv : dk) + 4 * j;
    uint2 w;
    w.x = pack2(v.x, v.y, std::is_same<T, __nv_bfloat16>::value ? DT_BF16 : DT_F16);
    w.y = pack2(v.z, v.w, std::is_same<T, __nv_bfloat16>::value ? DT_BF16 : DT_F16);
    *reinterpret_cast<uint2*>(dst) = w;
  }
}

// Into how many parts a KV head's group of query heads is split in the dK/dV kernel: the fewest with which the longest CTA
// takes at most a quarter longer than an even share of all tiles.  Whole groups (1) store their result directly; more
// parts need the zeroed workspace, atomics and a conversion.
static int dkdv_splits(int B, int S, int Sk, int Hq, int Hkv, int causal) {
  const long long nq = (S + AT_BM - 1) / AT_BM, nk = (Sk + AT_BN - 1) / AT_BN;
  const int group = Hq / Hkv;
  const long long pairs = causal ? nq * (nk - nq) + nq * (nq + 1) / 2 : nq * nk;
  const long long total = pairs * Hq * B;
  for (int n = 1; n < group; ++n)
    if (4 * (long long)sm_count() * nq * ((group + n - 1) / n) <= 5 * total) return n;
  return group;
}

template <int D, int CN, bool BF16>
static int launch_dkdv(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const CUtensorMap& dout,
                       const AttnParams& p, float* ws, int splits, int grid, cudaStream_t st) {
  static unsigned long long cfg = 0;
  if (int e = smem_opt_in(attn_bwd_dkdv_kernel<D, CN, BF16>, BwdCfg<D, CN>::SMEM_KV, cfg)) return e;
  attn_bwd_dkdv_kernel<D, CN, BF16><<<grid, BW_THREADS, BwdCfg<D, CN>::SMEM_KV, st>>>(q, k, v, dout, p, ws, splits);
  return (int)cudaGetLastError();
}
template <int D, int CN, bool BF16>
static int launch_dq(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const CUtensorMap& dout,
                     const AttnParams& p, int grid, cudaStream_t st) {
  static unsigned long long cfg = 0;
  if (int e = smem_opt_in(attn_bwd_dq_kernel<D, CN, BF16>, BwdCfg<D, CN>::SMEM_DQ, cfg)) return e;
  attn_bwd_dq_kernel<D, CN, BF16><<<grid, BW_THREADS, BwdCfg<D, CN>::SMEM_DQ, st>>>(q, k, v, dout, p);
  return (int)cudaGetLastError();
}

// Whether a kernel of `grid` CTAs, the longest of which walks through `length` whole score tiles whose columns come from
// sequences of `cols` rows, takes half tiles.  Where the columns fit one, the other half would be padding: 128 x 16, 12 / 12
// heads of 128 135 -> 113 us, 32 x 64, 16 / 16 61 -> 52.  At D = 64 half tiles put two CTAs on an SM, and one's start, epilogue
// and waits are under the other's arithmetic: they win as soon as there are enough CTAs.  Backward pass with whole tiles /
// half tiles, causal, us: 16 / 16 heads, 128 x 64 164 / 92, 128 x 128 193 / 130, 32 x 512 236 / 170, 8 x 1024 150 / 118; 14 / 2
// heads, 8 x 2048 326 / 287.  A CTA that has its SM to itself is faster on whole ones (1 x 1536, 16 / 16 45 / 55), and with less
// than two CTAs for every SM the longest one decides, so there only short ones split.  (1750 shapes: 0.8 % off the better
// of the two on average.)
static bool half_tiles(long long grid, int cols, int length, int D) {
  if (cols <= 64) return true;
  return D == 64 && (grid > 2 * sm_count() || (grid > sm_count() && length <= 8));
}

template <typename T, int D, bool BF16>
static int launch_bwd(const AttnParams& p, const void* q, const void* k, const void* v, const void* o, const void* dout,
                      const float* lse, float* stats, float* ws, int splits, cudaStream_t st) {
  const long long gq = (long long)((p.S + AT_BM - 1) / AT_BM) * p.Hq * p.B;
  const long long gk = (long long)((p.Sk + AT_BM - 1) / AT_BM) * p.Hkv * splits * p.B;
  if (gq > 0x7fffffff || gk > 0x7fffffff) return -5;
  // tiles of 128 rows, and of 64 where they are the columns of half score tiles
  CUtensorMap tq, tk, tv, tdo, hq, hk, hv, hdo;
  const int group = p.Hq / p.Hkv;
  const bool nq = half_tiles(gq, p.Sk, (p.Sk + AT_BN - 1) / AT_BN, D);
  const bool nk = half_tiles(gk, p.S, (p.S + AT_BN - 1) / AT_BN * ((group + splits - 1) / splits), D);
  auto map = [&](CUtensorMap& m, const void* t, int S, int H, int rows) {
    return make_tmap_bshd(&m, t, BF16 ? 1 : 0, p.B, S, H, D, rows);
  };
  int r;
  if ((r = map(tq, q, p.S, p.Hq, 128)) != 0 || (nk && (r = map(hq, q, p.S, p.Hq, 64)) != 0)) return 10000 + r;
  if ((r = map(tk, k, p.Sk, p.Hkv, 128)) != 0 || (nq && (r = map(hk, k, p.Sk, p.Hkv, 64)) != 0)) return 20000 + r;
  if ((r = map(tv, v, p.Sk, p.Hkv, 128)) != 0 || (nq && (r = map(hv, v, p.Sk, p.Hkv, 64)) != 0)) return 30000 + r;
  if ((r = map(tdo, dout, p.S, p.Hq, 128)) != 0 || (nk && (r = map(hdo, dout, p.S, p.Hq, 64)) != 0)) return 40000 + r;
  const long long lanes = (long long)p.B * p.S * p.Hq * (D / 8), nkv = (long long)p.B * p.Sk * p.Hkv * D;
  attn_stats_kernel<T, D><<<gb_grid(lanes, 256), 256, 0, st>>>((const T*)o, (const T*)dout, lse, stats, p.B, p.S,
                                                               p.Spad, p.Hq);
  if (splits > 1 && (r = (int)cudaMemsetAsync(ws, 0, 2 * nkv * sizeof(float), st)) != 0) return r;
  if (splits == 1) ws = nullptr;
  r = nk ? launch_dkdv<D, 64, BF16>(hq, tk, tv, hdo, p, ws, splits, (int)gk, st)
         : launch_dkdv<D, 128, BF16>(tq, tk, tv, tdo, p, ws, splits, (int)gk, st);
  if (r != 0) return r;
  r = nq ? launch_dq<D, 64, BF16>(tq, hk, hv, tdo, p, (int)gq, st) : launch_dq<D, 128, BF16>(tq, tk, tv, tdo, p, (int)gq, st);
  if (r != 0) return r;
  if (splits > 1)
    attn_dkv_convert_kernel<T><<<gb_grid(nkv / 2, 256), 256, 0, st>>>(ws, (T*)p.dk, (T*)p.dv, nkv);
  return (int)cudaGetLastError();
}

}  // namespace gb

using namespace gb;

// Into how many parts the query heads of a group are split (see dkdv_splits).
extern "C" int gb_attn_bwd_splits(int B, int S, int Sk, int Hq, int Hkv, int causal) {
  return dkdv_splits(B, S, Sk, Hq, Hkv, causal);
}

// scratch (fp32, 16-byte aligned): 2 * B * Hq * (S rounded up to 128) row statistics, and behind them
// 2 * B * Sk * Hkv * D elements for dK and dV where gb_attn_bwd_splits() > 1.
extern "C" int gb_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout,
                           const float* lse, float* scratch, void* dq, void* dk, void* dv, int B,
                           int S, int Sk, int Hq, int Hkv, int D, int causal, float scale, int is_bf16,
                           int* status, cudaStream_t st) {
  if (D != 64 && D != 128) return -2;
  if (Hq % Hkv != 0 || Sk < S) return -3;
  if (scratch == nullptr || (reinterpret_cast<uintptr_t>(scratch) & 15) != 0) return -4;
  AttnParams p{};
  p.Spad = (S + AT_BM - 1) / AT_BM * AT_BM;
  p.stats = scratch; p.dq = dq; p.dk = dk; p.dv = dv; p.status = status;
  p.B = B; p.S = S; p.Sk = Sk; p.Hq = Hq; p.Hkv = Hkv; p.causal = causal; p.is_bf16 = is_bf16; p.scale = scale;
  float* ws = scratch + 2 * (long long)B * Hq * p.Spad;
  const int splits = dkdv_splits(B, S, Sk, Hq, Hkv, causal);
  if (D == 64)
    return is_bf16 ? launch_bwd<__nv_bfloat16, 64, true>(p, q, k, v, o, dout, lse, scratch, ws, splits, st)
                   : launch_bwd<__half, 64, false>(p, q, k, v, o, dout, lse, scratch, ws, splits, st);
  return is_bf16 ? launch_bwd<__nv_bfloat16, 128, true>(p, q, k, v, o, dout, lse, scratch, ws, splits, st)
                 : launch_bwd<__half, 128, false>(p, q, k, v, o, dout, lse, scratch, ws, splits, st);
}
