// Attention for two query tiles at a time (sm_100a).  The same pipeline as sage_attn_kernel (attn_kernel.cuh, where the
// numerics are described, for int8 and for 16-bit Q and K), with one CTA per SM that holds two 128-row query tiles of
// a head against one ring of K / V tiles:
//   warps 0-3, 4-7 : softmax of tile 0 and of tile 1
//   warp 8         : TMA producer;  warps 9, 10 : MMA issuers of tile 0 and of tile 1
//
// Persistent.  Items are pairs of query tiles; CTA c of G takes items c, c + G, c + 2G, ... whole, in the order of head
// groups (K and V of a few heads at a time stay in the L2).  The loads and the first Q.K^T of the next item run under the end
// of the current one, and the two sides drift against each other by up to the depth of the ring.  An item of few
// KV tiles costs about its steps, where a CTA per tile pays some 5 us of set-up, first loads, epilogue and launch.
// The steps of items left over are cut into equal spans where the items are long, and what such a span holds of an
// item it does not cover goes to the workspace for sage_attn_merge_kernel.
// When it is taken, and what it measured there: sage_takes_pairs (internal.h).
// Where it is not: with head_dim 128 the two-CTA kernel runs at the 1000 W limit, and a good part of that is K and V,
// which every CTA fetches from the L2 for itself (fetched once per stage instead of for every tile: clock 1.60 -> 1.76 GHz,
// 9 % less time for 37 heads of 8192).  Here a tile is fetched once for 256 rows and the clock is 1.73 GHz, but a
// half-step takes more clocks: 1031 us against 1012.
#pragma once

#include "attn_kernel.cuh"

namespace sage {

constexpr int kPairThreads = 352;
constexpr int kPairRows = 2 * kBlockM;

// QKF as in sage_attn_kernel: Q and K in 16 bits.
template <int D, bool QKF>
struct PairSmem {
  static constexpr int kStages = D == 128 ? (QKF ? 2 : 3) : (QKF ? 4 : 5);
  static constexpr int kQBytes = kBlockM * D * (QKF ? 2 : 1);
  static constexpr int kKBytes = kBlockN * D * (QKF ? 2 : 1);
  static constexpr int kVBytes = kBlockN * D * 2;
  static constexpr int kOffQ = 0;
  static constexpr int kOffK = kOffQ + 2 * kQBytes;
  static constexpr int kOffV = kOffK + kStages * kKBytes;
  static constexpr int kOffStage = kOffV + kStages * kVBytes;    // output boxes: 4 KB per softmax warp
  static constexpr int kOffBar = kOffStage + 8 * 4096;
  static constexpr int kSideBars = 10;   // q_full, q_empty, o_final, o_free, s_full[2], p_full[2], pv_done[2]
  static constexpr int kNumBars = 2 * kSideBars + 4 * kStages;
  static constexpr int kOffMisc = kOffBar + 8 * kNumBars;        // tmem base (u32), abort flag, fail code
  static constexpr int kTotal = kOffMisc + 16;
};

// Walks the segments of a CTA: whole items, then its span of the rest.
struct PairIter {
  const AttnParams& p;
  int round;
  long long t, t_end;
  bool first;
  __device__ __forceinline__ explicit PairIter(const AttnParams& pp) : p(pp), round(0), first(true) {
    t = t_end = 0;
    if (blockIdx.x < static_cast<unsigned>(p.pair_spans)) {
      t = (p.sk_total_tiles * blockIdx.x) / p.pair_spans;
      t_end = (p.sk_total_tiles * (blockIdx.x + 1)) / p.pair_spans;
    }
  }
  __device__ __forceinline__ bool next(Segment& s) {
    int item;
    if (round < p.pair_rounds) {
      item = round * gridDim.x + blockIdx.x;
      ++round;
      s.kv_lo = 0;
      s.n_kv = p.sk_nkv_full;
      s.slot = -1;
    } else {
      if (t >= t_end) return false;
      const int rest = static_cast<int>(t / p.sk_nkv_full);
      item = p.pair_rounds * gridDim.x + rest;
      s.kv_lo = static_cast<int>(t - static_cast<long long>(rest) * p.sk_nkv_full);
      s.n_kv = static_cast<int>(min(static_cast<long long>(p.sk_nkv_full - s.kv_lo), t_end - t));
      s.slot = s.n_kv == p.sk_nkv_full ? -1 : (first ? 0 : 1);
      first = false;
      t += s.n_kv;
    }
    int pair;
    pair_item(item, p.B * p.Hq, p.head_group, (p.n_q_tiles + 1) / 2, &s.bh, &pair);
    s.b = s.bh / p.Hq;
    s.hq = s.bh - s.b * p.Hq;
    s.hkv = s.hq / (p.Hq / p.Hkv);
    s.q_base = pair * kPairRows;
    return true;
  }
};

template <int D, bool QKF>
__global__ void __launch_bounds__(kPairThreads, 1)
sage_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o, const AttnParams p) {
  using L = PairSmem<D, QKF>;
  constexpr int kStages = L::kStages;
  constexpr int kHalf = kHalfN;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if ((smem_u32(smem) & 1023u) != 0u) {        // swizzled tiles need 1024-byte alignment
    grid_dependency_wait();
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, kStatusSmemMisaligned);
    return;
  }
  uint8_t* s_q = smem + L::kOffQ;
  uint8_t* s_k = smem + L::kOffK;
  uint8_t* s_v = smem + L::kOffV;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* k_full = bars + 2 * L::kSideBars;
  uint64_t* v_full = k_full + kStages;
  uint64_t* k_empty = v_full + kStages;        // both sides have used the tile
  uint64_t* v_empty = k_empty + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kOffMisc + 4);
  int* fail_code = reinterpret_cast<int*>(smem + L::kOffMisc + 8);
  // Barriers of the side a warp works for (the producer works for both).
  const int side = (warp >= 4 && warp < 8) || warp == 10 ? 1 : 0;
  uint64_t* side_bars = bars + side * L::kSideBars;
  uint64_t* q_full = side_bars + 0;
  uint64_t* q_empty = side_bars + 1;
  uint64_t* o_final = side_bars + 2;
  uint64_t* o_free = side_bars + 3;
  uint64_t* s_full = side_bars + 4;
  uint64_t* p_full = side_bars + 6;
  uint64_t* pv_done = side_bars + 8;

  if (warp == 8 && elect_one()) {
    for (int sd = 0; sd < 2; ++sd) {
      uint64_t* sb = bars + sd * L::kSideBars;
      for (int i = 0; i < L::kSideBars; ++i) mbar_init(sb + i, (i == 3 || i == 6 || i == 7) ? 128 : 1);
    }
    for (int s = 0; s < kStages; ++s) {
      mbar_init(k_full + s, 1);
      mbar_init(v_full + s, 1);
      mbar_init(k_empty + s, 2);
      mbar_init(v_empty + s, 2);
    }
    fence_mbar_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    tma_prefetch_desc(&tm_o);
  }
  grid_dependency_wait();
  if (warp == 9) {                             // after the wait, as in sage_attn_kernel
    tmem_alloc(tmem_slot, 2 * kTmemCols);
    tmem_relinquish();
  }
  if (threadIdx.x == 0) {
    *abort_flag = (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
    *fail_code = 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_launch_dependents();
  const uint32_t tmem_base = *tmem_slot;
  const bool dead_on_arrival = *abort_flag != 0;

#define SAGE_PAIR_WAIT(hinted, bar_ptr, parity, bar_id, action)                   \
  if (!mbar_wait<hinted>((bar_ptr), (parity), abort_flag, p.wait_limit_cycles)) { \
    atomicCAS(fail_code, 0, kStatusWaitTimeout + 16 * (bar_id));                  \
    action;                                                                       \
  }

  if (dead_on_arrival) {
  } else if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      PairIter iter(p);
      Segment g;
      int kt = 0, it = 0;                      // KV tiles / segments so far
      bool ok = true;
#pragma unroll 1
      while (ok && iter.next(g)) {
#pragma unroll 1
        for (int j = 0; j < g.n_kv; ++j) {
          const int t = kt + j, s = t % kStages;
          const uint32_t free_parity = ((t / kStages) & 1) ^ 1u;
          SAGE_PAIR_WAIT(true, k_empty + s, free_parity, 1, { ok = false; break; });
          mbar_arrive_expect_tx(k_full + s, L::kKBytes);
          if constexpr (QKF) {
#pragma unroll
            for (int c = 0; c < D / 64; ++c)
              tma_load_4d(s_k + s * L::kKBytes + c * (kBlockN * 128), &tm_k, k_full + s, c * 64, (g.kv_lo + j) * kBlockN, g.hkv, g.b);
          } else {
            tma_load_3d(s_k + s * L::kKBytes, &tm_k, k_full + s, 0, (g.kv_lo + j) * kBlockN, g.b * p.Hkv + g.hkv);
          }
          if (j == 0) {
            for (int sd = 0; sd < 2; ++sd) {
              uint64_t* sb = bars + sd * L::kSideBars;
              if (it > 0) SAGE_PAIR_WAIT(true, sb + 1, (it - 1) & 1, 13, { ok = false; break; });
              mbar_arrive_expect_tx(sb, L::kQBytes);
              if constexpr (QKF) {
#pragma unroll
                for (int c = 0; c < D / 64; ++c)
                  tma_load_4d(s_q + sd * L::kQBytes + c * (kBlockM * 128), &tm_q, sb, c * 64, g.q_base + sd * kBlockM, g.hq, g.b);
              } else {
                tma_load_3d(s_q + sd * L::kQBytes, &tm_q, sb, 0, g.q_base + sd * kBlockM, g.bh);
              }
            }
            if (!ok) break;
          }
          SAGE_PAIR_WAIT(true, v_empty + s, free_parity, 2, { ok = false; break; });
          if (p.test_drop_v_load && t == 0) continue;       // failure-detection test: v_full never completes
          mbar_arrive_expect_tx(v_full + s, L::kVBytes);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) {
            tma_load_4d(s_v + s * L::kVBytes + c * (kBlockN * 128), &tm_v, v_full + s, c * 64, (g.kv_lo + j) * kBlockN, g.hkv, g.b);
          }
        }
        kt += g.n_kv;
        ++it;
      }
    }
    __syncwarp();
  } else if (warp >= 9) {
    // ------------------------------------------------------------------ MMA issuer of a side
    if (elect_one()) {
      constexpr uint32_t kIdescQK = umma_idesc(2, 1, 1, 0, 0, kBlockM, kHalf);
      constexpr uint32_t kIdescPV = umma_idesc(1, 0, 0, 0, 1, kBlockM, D);
      constexpr uint32_t kSwzQK = (D == 128) ? kSwizzle128B : kSwizzle64B;
      constexpr uint32_t kSboQK = 8 * D;
      const uint64_t desc_q = umma_smem_desc(smem_u32(s_q + side * L::kQBytes), 16, kSboQK, kSwzQK);
      const uint32_t t_base = tmem_base + side * kTmemCols;
      const uint32_t t_o = t_base + kColO;
      const uint32_t idesc_qk16 = umma_idesc(1, p.qk_bf16 ? 1u : 0u, p.qk_bf16 ? 1u : 0u, 0, 0, kBlockM, kHalf);
      auto issue_qk = [&](int stage, int h) {
        if constexpr (QKF) {
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint32_t slab = (k / 4) * (kBlockM * 128);
            const uint64_t dq = umma_smem_desc(smem_u32(s_q + side * L::kQBytes + slab), 16, 1024, kSwizzle128B) + 2 * (k % 4);
            const uint64_t dk =
                umma_smem_desc(smem_u32(s_k + stage * L::kKBytes + slab + h * (kHalf * 128)), 16, 1024, kSwizzle128B) + 2 * (k % 4);
            mma_f16_ss(t_base + kColS + h * kHalf, dq, dk, idesc_qk16, k > 0 ? 1u : 0u);
          }
        } else {
          const uint64_t desc_k = umma_smem_desc(smem_u32(s_k + stage * L::kKBytes + h * kHalf * D), 16, kSboQK, kSwzQK);
#pragma unroll
          for (int k = 0; k < D / 32; ++k)
            mma_i8_ss(t_base + kColS + h * kHalf, desc_q + 2 * k, desc_k + 2 * k, kIdescQK, k > 0 ? 1u : 0u);
        }
        tc_commit(s_full + h);
      };
      PairIter iter(p);
      Segment g;
      int kt = 0, it = 0;
      bool ok = true;
#pragma unroll 1
      while (ok && iter.next(g)) {
        const int n_kv = g.n_kv;
        SAGE_PAIR_WAIT(false, q_full, it & 1, 3, { ok = false; break; });
        {
          const int s0 = kt % kStages;
          SAGE_PAIR_WAIT(false, k_full + s0, (kt / kStages) & 1, 4, { ok = false; break; });
          tc_fence_after();
          issue_qk(s0, 0);
          issue_qk(s0, 1);
          tc_commit(k_empty + s0);
          if (n_kv == 1) tc_commit(q_empty);
        }
#pragma unroll 1
        for (int j = 0; ok && j < n_kv; ++j) {
          const int t = kt + j;
          const int s = t % kStages, s1 = (t + 1) % kStages;
          const uint32_t ph = (t / kStages) & 1, ph1 = ((t + 1) / kStages) & 1;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            SAGE_PAIR_WAIT(false, p_full + h, t & 1, 5, { ok = false; break; });
            if (h == 0) SAGE_PAIR_WAIT(false, v_full + s, ph, 6, { ok = false; break; });
            // the first P.V of a segment overwrites O: the previous segment's O must have been read
            if (h == 0 && j == 0 && it > 0) SAGE_PAIR_WAIT(false, o_free, (it - 1) & 1, 14, { ok = false; break; });
            tc_fence_after();
            const uint64_t desc_v =
                umma_smem_desc(smem_u32(s_v + s * L::kVBytes + h * (kHalf * 128)), kBlockN * 128, 1024, kSwizzle128B);
#pragma unroll
            for (int k = 0; k < kHalf / 16; ++k) {
              mma_f16_ts(t_o, t_base + kColP + h * kHalf + 8 * k, desc_v + 128 * k, kIdescPV, (j > 0 || h > 0 || k > 0) ? 1u : 0u);
            }
            tc_commit(pv_done + h);
            if (h == 1) tc_commit(v_empty + s);
            if (j + 1 < n_kv) {
              if (h == 0) SAGE_PAIR_WAIT(false, k_full + s1, ph1, 7, { ok = false; break; });
              tc_fence_after();
              issue_qk(s1, h);
              if (h == 1) {
                tc_commit(k_empty + s1);
                if (j + 2 == n_kv) tc_commit(q_empty);
              }
            }
          }
        }
        if (!ok) break;
        tc_commit(o_final);
        kt += n_kv;
        ++it;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax / epilogue of a side
    const int wq = warp & 3, tid = threadIdx.x & 127;
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t t_base = tmem_base + side * kTmemCols + lane_base;
    const uint32_t t_o = t_base + kColO;
    bool ok = true;
    int kt = 0, it = 0;
    PairIter iter(p);
    Segment sg;
#pragma unroll 1
    while (ok && iter.next(sg)) {
      const int q_base = sg.q_base + side * kBlockM;
      const int row = q_base + tid;
      float qs = 0.0f;
      if (!QKF && row < p.Sq) {
        const int head = row / p.q_rows;                // 0 unless folded
        qs = __ldg(p.q_scale + (static_cast<long long>(sg.bh) * p.q_fold + head) * p.q_groups + (row - head * p.q_rows) / 32);
      }
      const float* ks_base = p.k_scale + static_cast<long long>(sg.b * p.Hkv + sg.hkv) * p.k_groups;
      float m_used = kMaskValue, l = 0.0f;
      int distrust = 0;
      float ks_next[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int kg = sg.kv_lo * (kBlockN / 16) + g;
        ks_next[g] = (!QKF && kg < p.k_groups) ? __ldg(ks_base + kg) : 0.0f;
      }
      const int n_half = 2 * sg.n_kv;
#pragma unroll 1
      for (int hh = 0; hh < n_half; ++hh) {
        const int t = kt + (hh >> 1), h = hh & 1;
        const int kv_base = (2 * sg.kv_lo + hh) * kHalf;
        const uint32_t t_s = t_base + kColS + h * kHalf;
        float cg[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) cg[g] = QKF ? p.score_scale : __fmul_rn(qs, ks_next[g]);
        SAGE_PAIR_WAIT(false, s_full + h, t & 1, 8, { ok = false; break; });
        tc_fence_after();
        uint32_t sr[2][32];
        tmem_ld32(t_s, sr[0]);
        tmem_ld32(t_s + 32, sr[1]);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int kg = (kv_base + kHalf) / 16 + g;
          ks_next[g] = (!QKF && kg < p.k_groups) ? __ldg(ks_base + kg) : 0.0f;
        }
        tc_wait_ld();
        const bool masked = kv_base + kHalf > p.Skv;
        const int col_end = masked ? p.Skv - kv_base : kHalf;
        uint32_t pk[32];
        f32x2_t cg2[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) cg2[g] = pack2(cg[g], cg[g]);
        auto score_of = [](uint32_t w) -> float {
          if constexpr (QKF) return __uint_as_float(w);
          else return __int2float_rn(static_cast<int>(w));
        };
        auto exp_pass = [&](auto masked_tag, float m_now) -> float {
          constexpr bool kMasked = decltype(masked_tag)::value;
          const f32x2_t neg_m = pack2(-m_now, -m_now);
          f32x2_t acc = pack2(0.0f, 0.0f);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int e = 32 * c + 2 * i;
              const f32x2_t sf = pack2(score_of(sr[c][2 * i]), score_of(sr[c][2 * i + 1]));
              const float2 x = unpack2(ffma2(sf, cg2[e >> 4], neg_m));
              float2 pp = make_float2(fast_exp2(x.x), fast_exp2(x.y));
              if constexpr (kMasked) {
                if (e >= col_end) pp.x = 0.0f;
                if (e + 1 >= col_end) pp.y = 0.0f;
              }
              acc = fadd2(acc, pack2(pp.x, pp.y));
              pk[16 * c + i] = pack_half2(pp.x, pp.y);
            }
          }
          const float2 a = unpack2(acc);
          return a.x + a.y;
        };
        // The steps of sage_attn_kernel: an attempt against the running maximum, else the exact way.
        bool done = false;
        float m_half = kMaskValue;
        const bool attempt = hh != 0 && !masked && distrust < 2;
        if (attempt) {
          const float sum = exp_pass(std::false_type{}, m_used);
          if (!__any_sync(0xffffffffu, !(sum <= kOptimisticSumMax))) {
            l += sum;
            done = true;
          }
        }
        if (attempt) distrust = done ? max(distrust - 1, 0) : min(distrust + 2, 4);
        if (!done) {
          if (!masked && !QKF) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {               // scales are >= 0: max commutes with the scaling
              int mx = static_cast<int>(sr[g >> 1][(g & 1) * 16]);
#pragma unroll
              for (int i = 1; i < 16; ++i) mx = max(mx, static_cast<int>(sr[g >> 1][(g & 1) * 16 + i]));
              m_half = fmaxf(m_half, __int2float_rn(mx) * cg[g]);
            }
          } else {
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const float sv = score_of(sr[c][i]) * cg[(32 * c + i) >> 4];
                if (32 * c + i < col_end) m_half = fmaxf(m_half, sv);
              }
          }
          bool moved = false;
          float alpha = 1.0f;
          if (hh == 0) {
            m_used = m_half;
          } else {
            const bool need = m_half > m_used + (attempt ? kRefusedBarLog2 : kLazyRescaleLog2);
            moved = __any_sync(0xffffffffu, need);
            if (!attempt) distrust = moved ? min(distrust + 1, 4) : distrust - 1;
            alpha = need ? fast_exp2(m_used - m_half) : 1.0f;
            if (need) m_used = m_half;
            l *= alpha;
          }
          if (masked) l += exp_pass(std::true_type{}, m_used);
          else l += exp_pass(std::false_type{}, m_used);
          if (moved) {
            const int hp = h ^ 1;
            const int tp = h ? t : t - 1;
            SAGE_PAIR_WAIT(false, pv_done + hp, tp & 1, 9, { ok = false; break; });
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
              uint32_t orr[32];
              tmem_ld32(t_o + 32 * c, orr);
              tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i) orr[i] = __float_as_uint(__uint_as_float(orr[i]) * alpha);
              tmem_st32(t_o + 32 * c, orr);
            }
          }
        }
        tmem_st32(t_base + kColP + h * kHalf, pk);
        tc_wait_st();
        tc_fence_before();
        mbar_arrive(p_full + h);
      }
      if (!ok) break;

      // ---- epilogue: o = acc * (1/l), as in sage_attn_kernel; the boxes of a warp go out one after the other
      SAGE_PAIR_WAIT(false, o_final, it & 1, 10, { ok = false; break; });
      tc_fence_after();
      const float inv_l = (l > 0.0f) ? (1.0f / l) : 0.0f;
      const bool whole = sg.slot < 0;
      const long long part_row = (static_cast<long long>(blockIdx.x) * 2 + max(sg.slot, 0)) * kPairRows + side * kBlockM + tid;
      if (whole) {
        if (p.lse != nullptr && row < p.Sq) {
          const float lse = (l > 0.0f) ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
          float* dst = p.lse + static_cast<long long>(sg.bh) * p.Sq + row;
          *dst = p.lse_add ? fmaf(p.lse_add_scale, *dst, lse) : lse;
        }
      } else {
        p.part_lse[part_row] = (l > 0.0f) ? (m_used + log2f(l)) : (l == 0.0f) ? -INFINITY : INFINITY;
      }
      uint8_t* stage = smem + L::kOffStage + warp * 4096;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t orr[32];
        tmem_ld32(t_o + 32 * c, orr);
        tc_wait_ld();
        if (c == D / 32 - 1) {                          // O is in registers: the next segment may overwrite it
          tc_fence_before();
          mbar_arrive(o_free);
        }
        if (!whole) {
          float4* dst = reinterpret_cast<float4*>(p.part_o + part_row * D + 32 * c);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            dst[i] = make_float4(__uint_as_float(orr[4 * i]) * inv_l, __uint_as_float(orr[4 * i + 1]) * inv_l,
                                 __uint_as_float(orr[4 * i + 2]) * inv_l, __uint_as_float(orr[4 * i + 3]) * inv_l);
          }
          continue;
        }
        uint32_t out[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float a = __uint_as_float(orr[2 * i]) * inv_l;
          const float bb = __uint_as_float(orr[2 * i + 1]) * inv_l;
          out[i] = p.out_bf16 ? pack_bf162(a, bb) : pack_half2(a, bb);
        }
        if ((c & 1) == 0) {
          if (lane == 0) tma_store_wait_read();         // the box before has left
          __syncwarp();
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int chunk = ((c & 1) * 4 + i) ^ (lane & 7);
          *reinterpret_cast<uint4*>(stage + lane * 128 + chunk * 16) = make_uint4(out[4 * i], out[4 * i + 1], out[4 * i + 2], out[4 * i + 3]);
        }
        if ((c & 1) == 1) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && q_base + wq * 32 < p.Sq) {
            tma_store_4d(&tm_o, stage, (c >> 1) * 64, q_base + wq * 32, sg.hq, sg.b);
            tma_store_commit();
          }
        }
      }
      kt += sg.n_kv;
      ++it;
    }
    if (lane == 0) tma_store_wait_read();               // the staging area is read before the CTA gives it up
    __syncwarp();
  }
#undef SAGE_PAIR_WAIT

  // ---------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // As in sage_attn_kernel: copies and MMAs in flight land before shared memory and TMEM are handed back.
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    if (threadIdx.x == 0) {
      const int code = *fail_code ? *fail_code : kStatusWaitTimeout;
      if (p.status) atomicCAS(p.status, 0, code);
      if (p.status_host) {
        *reinterpret_cast<volatile int*>(p.status_host) = code;
        __threadfence_system();
      }
    }
    __syncthreads();
  }
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * kTmemCols);
  }
}

}  // namespace sage
