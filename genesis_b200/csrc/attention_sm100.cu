// Flash attention forward for sm_100a on tcgen05 tensor cores (backward: attention_bwd_sm100.cu).
//
// Layout: q [B, S, Hq, D], k/v [B, Sk, Hkv, D], o [B, S, Hq, D], lse [B, Hq, S] (natural log).
// Native GQA (Hkv divides Hq, K/V never replicated), optional causal mask (aligned to the end of
// the keys when Sk > S), any S / Sk, D in {64, 128}, bf16 / fp16.
//
// A persistent CTA works on two q tiles of 128 rows at a time, one per soft-max warpgroup: while one warpgroup
// exponentiates its 128 x 128 score tile, the tensor cores multiply the other's (S = Q K^T, O += P V), so neither waits
// for the other in turn.  One thread row = one TMEM lane, so soft-max statistics never leave the thread, and the
// probabilities go back as 16-bit pairs into the columns of the score tile they came from: P is the tensor-memory A
// operand of the second GEMM and shared memory holds only what TMA wrote (Q tiles, a ring of K / V tiles) and the
// per-warp slabs of the output store.
//   bound       : per tile and SM the exponentials take 1024 clocks (one MUFU result per score, 16 per clock), the products
//                 512 at D = 64 and 1024 at D = 128.  At D = 64 a quarter of the exponentials of a tile without a mask goes to
//                 the FMA pipes, which leaves 768 clocks of MUFU beside the FMA work.
//   registers   : ten warps put three on one scheduler, which caps every warp at 168 registers; the soft-max loop spills 44
//                 bytes at D = 128 and 32 at D = 64.
//   rescaling   : the accumulator is multiplied only when a row maximum grows by more than 2^8 over the reference it was
//                 started with; probabilities up to 2^8 keep their relative precision in 16 and 32 bits, and the final
//                 division by the row sum (taken against the same reference) removes the factor.
//   order       : S(j+1) of a tile is issued after P V(j) of the same tile, which reads the columns S(j+1) overwrites;
//                 the tensor pipe runs them in that order, and the commit of S(j+1) also covers P V(j), so a warpgroup
//                 that sees its scores may touch its accumulator without another wait.
//   work split  : pairs of q tiles, longest first, dealt to the CTAs in alternating direction, which evens out the
//                 causal triangle; when pairs would leave SMs idle each item is one tile.
// Measured against the kernel this replaces (one 128-row tile per CTA, four soft-max warps, P through shared memory),
// bf16 causal, us and TFLOP/s: 8 x 2048, 14 / 2 heads of 64: 174 -> 105 (571); 4 x 4096, 12 / 2 of 128: 383 -> 178 (1162);
// 1 x 16384, 16 / 4 of 128: 1566 -> 848 (1296); 1 x 1003, 14 / 2 of 64: 24.8 -> 20.7.
// Operand tricks: V is consumed as an MN-major operand straight from the tile TMA wrote; nothing is transposed.
// Reference counterpart: Triton kernels of genesis/nn/attention.py:21-519 (32 x 32 tiles, Hq == Hkv only).
#include <type_traits>
#include "attention_common.cuh"

namespace gb {

constexpr int FW_THREADS = 320;          // 2 x 4 soft-max warps, TMA warp, MMA warp
constexpr int FW_SLAB = 32 * 128;        // output slab of a warp: 32 rows x 64 16-bit columns

template <int D> struct FwdCfg {
  static constexpr int TILE = AT_BM * D * 2;             // one [128 x D] 16-bit tile
  static constexpr int ST = D == 64 ? 6 : 4;             // K / V ring
  static constexpr int SMEM = 2 * TILE + ST * TILE + 8 * FW_SLAB + 256;
};

// work item -> q tiles and (head, batch); `tiles` q tiles per item
struct FwdItem { int m0, h, b, n[2], nmax; };
__device__ __forceinline__ FwdItem fwd_item(const AttnParams& p, int item, int tiles) {
  FwdItem w;
  const int nq = (p.S + AT_BM - 1) / AT_BM, npair = (nq + tiles - 1) / tiles;
  const int bh = p.B * p.Hq;
  const int qp = npair - 1 - item / bh, r = item % bh;      // longest (last) rows first
  w.h = r % p.Hq; w.b = r / p.Hq;
  w.m0 = qp * tiles * AT_BM;
  const int off = p.Sk - p.S, full = (p.Sk + AT_BN - 1) / AT_BN;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int m = w.m0 + t * AT_BM;
    int n = full;
    if (p.causal) { const int lim = (m + AT_BM + off + AT_BN - 1) / AT_BN; n = lim < n ? lim : n; }
    w.n[t] = (t < tiles && m < p.S) ? (n < 1 ? 1 : n) : 0;
  }
  w.nmax = w.n[0] > w.n[1] ? w.n[0] : w.n[1];
  return w;
}
// the item of CTA c in round r: rounds run in alternating direction
__device__ __forceinline__ int fwd_deal(int r) {
  return r * (int)gridDim.x + ((r & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
}

template <int D, bool BF16>
__global__ void __launch_bounds__(FW_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmq, const __grid_constant__ CUtensorMap tmk,
                const __grid_constant__ CUtensorMap tmv, const __grid_constant__ CUtensorMap tmo, const AttnParams p,
                const int n_items, const int tiles) {
  using C = FwdCfg<D>;
  constexpr int TILE = C::TILE, ST = C::ST;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if (status_poisoned(p.status)) return;
  if ((reinterpret_cast<uintptr_t>(smem_raw) & 1023) != 0) {     // no room for an alignment pad
    if (threadIdx.x == 0) report_error(p.status, GB_ERR_BAD_ARG, 1, 0);
    return;
  }
  uint8_t* sQ = smem_raw;               // 2 tiles
  uint8_t* sKV = sQ + 2 * TILE;         // ST stages, K and V tiles in turn
  uint8_t* sO = sKV + ST * TILE;        // 8 slabs
  uint64_t* bars = reinterpret_cast<uint64_t*>(sO + 8 * FW_SLAB);
  uint64_t* q_full = bars;              // [2]
  uint64_t* q_empty = bars + 2;         // [2]
  uint64_t* s_full = bars + 4;          // [2]
  uint64_t* p_full = bars + 6;          // [2]
  uint64_t* o_full = bars + 8;          // [2]
  uint64_t* kv_full = bars + 10;        // [ST]
  uint64_t* kv_empty = bars + 10 + ST;  // [ST]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10 + 2 * ST);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; ++t) {
      mbar_init(&q_full[t], 1); mbar_init(&q_empty[t], 1); mbar_init(&s_full[t], 1);
      mbar_init(&p_full[t], 128); mbar_init(&o_full[t], 1);
    }
    for (int s = 0; s < ST; ++s) { mbar_init(&kv_full[s], 1); mbar_init(&kv_empty[s], 1); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tO = tmem + 2 * AT_BN;      // score tiles at tmem and tmem + 128, accumulators behind them
  const int rounds = (n_items + (int)gridDim.x - 1) / (int)gridDim.x;

  if (warp == 8) {
    if (lane == 0) {   // ---------------- TMA ----------------
      tma_prefetch_desc(&tmq); tma_prefetch_desc(&tmk); tma_prefetch_desc(&tmv); tma_prefetch_desc(&tmo);
      int slot = 0;
      uint32_t par = 0;                       // parity of the ring's current lap
      uint32_t qn[2] = {0, 0}, kvn = 0;       // loads issued
      bool ok = true;
      auto load_kv = [&](const CUtensorMap* m, int head, int row, int b) {
        if (!ok || !(ok = AT_WAIT(&kv_empty[slot], par ^ 1, 10))) return;
        mbar_expect_tx(&kv_full[slot], TILE);
        load_tile<D>(sKV + slot * TILE, m, &kv_full[slot], head, row, b, AT_BN);
        ++kvn;
        if (++slot == ST) { slot = 0; par ^= 1; }
      };
      for (int r = 0; ok && r < rounds; ++r) {
        const int item = fwd_deal(r);
        if (item >= n_items) continue;
        const FwdItem w = fwd_item(p, item, tiles);
        const int kvh = w.h / (p.Hq / p.Hkv);
        for (int t = 0; ok && t < 2; ++t) {
          if (w.n[t] == 0) continue;
          if (!(ok = AT_WAIT(&q_empty[t], (qn[t] & 1) ^ 1, 11))) break;
          ++qn[t];
          mbar_expect_tx(&q_full[t], TILE);
          load_tile<D>(sQ + t * TILE, &tmq, &q_full[t], w.h, w.m0 + t * AT_BM, w.b, AT_BM);
          if (t == 0) load_kv(&tmk, kvh, 0, w.b);
        }
        for (int j = 0; ok && j < w.nmax; ++j) {
          load_kv(&tmv, kvh, j * AT_BN, w.b);
          if (j + 1 < w.nmax) load_kv(&tmk, kvh, (j + 1) * AT_BN, w.b);
        }
      }
      if (*abort_flag) {
        drain_copies(kv_full, ST, kvn);
        drain_copies(&q_full[0], 1, qn[0]);
        drain_copies(&q_full[1], 1, qn[1]);
      }
    }
  } else if (warp == 9) {
    // ---------------- MMA: the warp stays converged, one elected lane issues ----------------
    constexpr uint32_t fmt = BF16 ? 1u : 0u;
    constexpr uint32_t idesc_qk = make_idesc(fmt, 0, 0, AT_BM, AT_BN);
    constexpr uint32_t idesc_pv = make_idesc(fmt, 0, 1, AT_BM, D);
    const uint32_t aQ = smem_u32(sQ), aKV = smem_u32(sKV);
    int slot = 0;
    uint32_t par = 0, qpar[2] = {0, 0}, ppar[2] = {0, 0};
    bool ok = true;
    auto qk = [&](int t, int ks) {
      const uint64_t dq = desc_kmajor(aQ + t * TILE, 0, AT_BM), dk = desc_kmajor(aKV + ks * TILE, 0, AT_BN);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t o = (kk >> 2) * (AT_BM * 128 / 16) + (kk & 3) * 2;     // in 16-byte units
          umma_f16(tmem + t * AT_BN, dq + o, dk + o, idesc_qk, kk > 0);
        }
        umma_commit(&s_full[t]);
      }
      __syncwarp();
    };
    auto pv = [&](int t, int vs, bool first) {
      const uint64_t dv = desc_mnmajor(aKV + vs * TILE, 0, AT_BN);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < AT_BN / 16; ++kk)
          umma_f16_ts(tO + t * D, tmem + t * AT_BN + kk * 8, dv + kk * (2048 / 16), idesc_pv, !first || kk > 0);
      }
      __syncwarp();
    };
    auto commit = [&](uint64_t* bar) {
      if (elect_one()) umma_commit(bar);
      __syncwarp();
    };
    auto advance = [&]() { if (++slot == ST) { slot = 0; par ^= 1; } };
    for (int r = 0; ok && r < rounds; ++r) {
      const int item = fwd_deal(r);
      if (item >= n_items) continue;
      const FwdItem w = fwd_item(p, item, tiles);
      if (!(ok = AT_WAIT_ALL(&kv_full[slot], par, 20))) break;
      for (int t = 0; t < 2; ++t) {
        if (w.n[t] == 0) continue;
        if (!(ok = AT_WAIT_ALL(&q_full[t], qpar[t], 21))) break;
        qpar[t] ^= 1;
        tc_fence_after_sync();
        qk(t, slot);
        if (w.n[t] == 1) commit(&q_empty[t]);
      }
      if (!ok) break;
      commit(&kv_empty[slot]);
      advance();
      for (int j = 0; j < w.nmax; ++j) {
        const int vs = slot;
        if (!(ok = AT_WAIT_ALL(&kv_full[vs], par, 22))) break;
        advance();
        const int ks = slot;
        const bool more = j + 1 < w.nmax;
        if (more && !(ok = AT_WAIT_ALL(&kv_full[ks], par, 23))) break;
        for (int t = 0; t < 2; ++t) {
          if (j >= w.n[t]) continue;
          if (!(ok = AT_WAIT_ALL(&p_full[t], ppar[t], 24))) break;
          ppar[t] ^= 1;
          tc_fence_after_sync();
          pv(t, vs, j == 0);
          if (j + 1 < w.n[t]) {
            qk(t, ks);
            if (j + 2 == w.n[t]) commit(&q_empty[t]);
          } else {
            commit(&o_full[t]);
          }
        }
        if (!ok) break;
        commit(&kv_empty[vs]);
        if (more) { commit(&kv_empty[ks]); advance(); }
      }
    }
  } else {
    // ---------------- soft-max warpgroups ----------------
    const int t = warp >> 2;
    const int row_in = threadIdx.x & 127;
    const uint32_t lane_base = ((uint32_t)((warp & 3) * 32)) << 16;
    const uint32_t tS = tmem + t * AT_BN + lane_base, tOt = tO + t * D + lane_base;
    uint8_t* slab = sO + warp * FW_SLAB;
    const float sl2 = p.scale * LOG2E;
    const float2 sl2v = make_float2(sl2, sl2);
    const int off = p.Sk - p.S;
    uint32_t spar = 0, opar = 0;
    bool ok = true;
    for (int r = 0; ok && r < rounds; ++r) {
      const int item = fwd_deal(r);
      if (item >= n_items) continue;
      const FwdItem w = fwd_item(p, item, tiles);
      const int n = t ? w.n[1] : w.n[0];
      if (n == 0) continue;
      const int m0 = w.m0 + t * AT_BM, row = m0 + row_in;
      float m = -INFINITY, l = 0.f;     // reference of the exponentials (scaled, log2 domain) and sum against it
      for (int j = 0; j < n; ++j) {
        if (!(ok = AT_WAIT_ALL(&s_full[t], spar, 30))) break;
        spar ^= 1;
        tc_fence_after_sync();
        uint32_t s[4][32];
        tmem_ld_32x32b_x32(tS, s[0]);
        tmem_ld_32x32b_x32(tS + 32, s[1]);
        tmem_ld_32x32b_x32(tS + 64, s[2]);
        tmem_ld_32x32b_x32(tS + 96, s[3]);
        tmem_ld_wait();
        const int col0 = j * AT_BN;
        const bool masked = (col0 + AT_BN > p.Sk) || (p.causal && (col0 + AT_BN - 1 > m0 + off));
        if (masked) {
          int lim = p.causal ? row + off : p.Sk - 1;               // last visible column of this row
          lim = (lim < p.Sk - 1 ? lim : p.Sk - 1) - col0;
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i) s[c][i] = (c * 32 + i <= lim) ? s[c][i] : 0xff800000u;   // -inf
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; i += 2) mx[c] = max3(mx[c], __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
        const float m_new = fmaxf(m, fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]) * sl2);
        if (j == 0) {
          m = m_new;
        } else {
          const bool grow = m_new > m + 8.f;
          if (__any_sync(0xffffffffu, grow)) {
            const float alpha = grow ? fast_exp2(m - m_new) : 1.f;
            if (grow) m = m_new;
            l *= alpha;
#pragma unroll 1
            for (int c = 0; c < D / 32; ++c) {
              uint32_t o[32];
              tmem_ld_32x32b_x32(tOt + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st_32x32b_x32(tOt + c * 32, o);
            }
          }
        }
        const float nm = m == -INFINITY ? 0.f : -m;
        const float2 nmv = make_float2(nm, nm);
        float2 sum0 = make_float2(0.f, 0.f), sum1 = sum0;
        // D = 64, where the exponentials are the bound: a quarter of them goes to the FMA pipes in tiles without a
        // mask.  1 x 8192, 4 / 4 heads: 93 -> 84 us; 8 x 2048, 14 / 2 heads: 105.4 -> 104.0.
        auto exponentials = [&](auto mixed) {
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            uint32_t pk[32];
#pragma unroll
            for (int i = 0; i < 64; i += 4) {
              const uint32_t* v = &s[hf * 2 + (i >> 5)][i & 31];
              float2 a = fma2(make_float2(__uint_as_float(v[0]), __uint_as_float(v[1])), sl2v, nmv);
              float2 b = fma2(make_float2(__uint_as_float(v[2]), __uint_as_float(v[3])), sl2v, nmv);
              a.x = fast_exp2(a.x); a.y = fast_exp2(a.y);
              if (decltype(mixed)::value && (i & 4)) b = poly_exp2(b);
              else { b.x = fast_exp2(b.x); b.y = fast_exp2(b.y); }
              sum0 = add2(sum0, a);
              sum1 = add2(sum1, b);
              pk[i / 2] = pack2c<BF16>(a.x, a.y);
              pk[i / 2 + 1] = pack2c<BF16>(b.x, b.y);
            }
            tmem_st_32x32b_x32(tS + hf * 32, pk);
          }
        };
        if (D == 64 && !masked) exponentials(std::true_type{});
        else exponentials(std::false_type{});
        tmem_st_wait();
        tc_fence_before_sync();
        mbar_arrive(&p_full[t]);
        sum0 = add2(sum0, sum1);
        l += sum0.x + sum0.y;
      }
      if (!ok || !(ok = AT_WAIT_ALL(&o_full[t], opar, 31))) break;
      opar ^= 1;
      tc_fence_after_sync();
      const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
      for (int c = 0; c < D / 64; ++c) {
        uint32_t o[2][32];
        tmem_ld_32x32b_x32(tOt + c * 64, o[0]);
        tmem_ld_32x32b_x32(tOt + c * 64 + 32, o[1]);
        tmem_ld_wait();
        if (lane == 0) bulk_wait_group_read<0>();        // the slab's last store has read it
        __syncwarp();
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(o[hf][i]) * inv;
          store_row_chunk_t<BF16>(slab + lane * 128, hf * 4, lane, v);
        }
        fence_proxy_async_smem();
        __syncwarp();
        const int r0 = m0 + (warp & 3) * 32;
        if (lane == 0 && r0 < p.S) {
          tma_store_4d(&tmo, slab, c * 64, w.h, r0, w.b);
          bulk_commit_group();
        }
      }
      if (row < p.S) p.lse[((size_t)w.b * p.Hq + w.h) * p.S + row] = (l > 0.f) ? (m + log2f(l)) * LN2 : -INFINITY;
      tc_fence_before_sync();
    }
    if (lane == 0) bulk_wait_group<0>();
    __syncwarp();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) { tc_fence_after_sync(); tmem_dealloc(tmem, 512); }
}

template <int D, bool BF16>
static int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to,
                      const AttnParams& p, cudaStream_t st) {
  static unsigned long long cfg = 0;
  int r;
  if ((r = smem_opt_in(attn_fwd_kernel<D, BF16>, FwdCfg<D>::SMEM, cfg)) != 0) return r;
  const int sms = sm_count();
  const long long nq = (p.S + AT_BM - 1) / AT_BM, bh = (long long)p.B * p.Hq;
  // Two tiles per item wherever that saves a round of the CTAs: two tiles in turn take little longer than one.  One tile / two
  // tiles, us, d = 128, not causal: 24 heads, 1024 rows (2 rounds, 1) 35 / 23; 96 heads, 256 rows (2, 1) 16 / 12; 160 heads,
  // 777 rows (8, 5) 111 / 79; as many rounds of pairs: 96 heads, 384 rows (2, 2) 18.6 / 22.2.  (660 shapes of 4 to 512 heads
  // and 129 to 2048 rows: 0.3 % off the better of the two on average; pairs once they gave every SM an item: 2.7 %.)
  const int tiles = (((nq + 1) / 2) * bh + sms - 1) / sms < (nq * bh + sms - 1) / sms ? 2 : 1;
  const long long items = ((nq + tiles - 1) / tiles) * bh;
  if (items > 0x7fffffff) return -5;
  attn_fwd_kernel<D, BF16><<<(int)(items < sms ? items : sms), FW_THREADS, FwdCfg<D>::SMEM, st>>>(tq, tk, tv, to, p,
                                                                                                (int)items, tiles);
  return (int)cudaGetLastError();
}
}  // namespace gb

using namespace gb;

// A few query rows: the decoding kernel reads K and V once per 16 rows of a group and splits the keys between CTAs; the tiled
// kernel has the faster tensor cores and reads them once per head, 128 rows or not.  Which is faster depends on how both fill
// the GPU, so both times are estimated (us): a start, and per round of CTAs (two on an SM for the decoding kernel) a fixed
// part and the keys a CTA walks through.  Fitted to 2124 shapes (1 to 64 rows of a group, 16 to 16384 keys, 2 to 4096 KV heads
// x batch, inputs cycled past L2), where the choice is 0.3 % off the better of the two on average.  Decoding / tiled kernel:
// 8 x 1 queries, 32 / 4 heads of 128, 4096 keys 19 / 112; 64 x 8, 32 / 4, 1024 keys 82 / 207; one query, 14 / 2 heads of 64, 512
// keys 8.3 / 10.8; the other way: 256 x 16, 16 / 16 heads of 128, 128 keys 140 / 94; 64 x 16, 4 / 4, 256 keys 22.6 / 16.5.
static bool decode_wins(const AttnParams& p, int D) {
  const long long sms = sm_count(), rows = (long long)p.S * (p.Hq / p.Hkv);
  int ranks, steps;
  decode_split(p, D, ranks, steps);
  const long long waves = ((rows + 15) / 16 * p.Hkv * p.B * ranks + 2 * sms - 1) / (2 * sms);
  const long long rounds = ((long long)p.B * p.Hq + sms - 1) / sms, tiles = (p.Sk + AT_BN - 1) / AT_BN;
  const double r = rows < 16 ? (double)rows : 16.0;
  if (D == 64) return 1.5 + waves * (4.8 + 0.87 * steps + 0.05 * r) < 5.8 + rounds * (1.28 + 1.26 * tiles);
  return 0.9 + waves * (6.25 + 0.86 * steps + 0.11 * r) < 5.7 + rounds * (1.5 + 1.63 * tiles);
}

extern "C" int gb_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int S, int Sk,
                           int Hq, int Hkv, int D, int causal, float scale, int is_bf16, int* status,
                           cudaStream_t st) {
  if (D != 64 && D != 128) return -2;
  if (Hq % Hkv != 0 || Sk < S) return -3;
  AttnParams p{};
  p.o = o; p.lse = lse; p.status = status; p.B = B; p.S = S; p.Sk = Sk; p.Hq = Hq; p.Hkv = Hkv;
  p.causal = causal; p.is_bf16 = is_bf16; p.scale = scale;
  if ((long long)S * (Hq / Hkv) <= 64 && B <= 65535 && 4 * Hkv <= 65535 && decode_wins(p, D))
    return attn_decode(q, k, v, p, D, st);
  CUtensorMap tq, tk, tv, to;
  int r;
  if ((r = make_tmap_bshd(&tq, q, is_bf16, B, S, Hq, D)) != 0) return 10000 + r;
  if ((r = make_tmap_bshd(&tk, k, is_bf16, B, Sk, Hkv, D)) != 0) return 20000 + r;
  if ((r = make_tmap_bshd(&tv, v, is_bf16, B, Sk, Hkv, D)) != 0) return 30000 + r;
  if ((r = make_tmap_bshd(&to, o, is_bf16, B, S, Hq, D, 32)) != 0) return 40000 + r;
  if (D == 64) return is_bf16 ? launch_fwd<64, true>(tq, tk, tv, to, p, st) : launch_fwd<64, false>(tq, tk, tv, to, p, st);
  return is_bf16 ? launch_fwd<128, true>(tq, tk, tv, to, p, st) : launch_fwd<128, false>(tq, tk, tv, to, p, st);
}
