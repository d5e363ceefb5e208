// Shared by libsage_b200.so (sage_abi.cu) and _C.so (torch_ops.cpp); not part of the public C ABI.
#pragma once

#include <stdint.h>

#include "../../include/sage_b200.h"

// Rows of a tile that are padding: a 128-row tile holds rows of one head, and with few queries per head
// (some new tokens against a cached prefix) much of it is empty.  The query heads of a GQA group share
// K and V, so without a causal mask their rows can share tiles too: the group becomes one head of
// Hq/Hkv * Sq rows.  The int8 Q and the log-sum-exp are contiguous in that order; the output has to be
// as well (its row stride runs on into the next head).  Returns how many heads become one, 1 for none;
// folded wherever that gives fewer tiles (same work per tile, fewer of them: 32 heads of 64 rows on 8
// kv heads are 16 tiles instead of 32).
static inline int sage_gqa_fold(int64_t Hq, int64_t Hkv, int64_t Sq, int64_t o_stride_h, int64_t o_stride_s, int64_t is_causal) {
  if (is_causal || Hkv <= 0 || Hq <= Hkv || Hq % Hkv != 0 || Sq <= 0) return 1;
  const int64_t rep = Hq / Hkv, rows = rep * Sq;
  if (rows > 0x3fffffff || o_stride_h != Sq * o_stride_s) return 1;
  return (rows + 127) / 128 < rep * ((Sq + 127) / 128) ? (int)rep : 1;
}

// Order of the items (query tile, head) of a plain causal launch.  Heads go `head_group` at a time, the heaviest
// (last) query tiles of a group first.  That balances the SMs as long as a group is followed by another one:
// the next heavy items fill the gaps.  The last group has nothing behind it, so a small one - in particular
// what is left over after whole groups - starts its heaviest items when the other SMs run dry.  The last group
// therefore takes in whole groups before it until it has 1.5 items per CTA slot (two slots per SM), while the
// keys and values of its heads (`kv_bytes` per head) stay in half of the L2.  Attention launch alone, us, groups of 8
// throughout / with the larger last group: D=128 20 heads of 4096 tokens 101 / 83, 10 of 7000 164 / 126, 12 of 8192
// 212 / 190, 64 of 3000 164 / 157, 64 of 2000 (un-quantised) 104 / 94; D=64 32 of 2048 (un-quantised) 44 / 36; where
// the last group is large already (64 heads of 8192) 939 / 941.  One item per slot instead of 1.5: 24 heads of 2304 44
// instead of 42.
// Returns the first head of the last group, a multiple of head_group.
static inline int sage_tail_group_first(int n_heads, int head_group, int n_q_tiles, double kv_bytes, int sms) {
  int tail = n_heads % head_group;
  while (tail < n_heads && (long long)tail * n_q_tiles < 3LL * sms && (tail + head_group) * kv_bytes <= 64e6) tail += head_group;
  return n_heads - tail;
}

// Persistent or plain launch under a causal mask.  The plain launch takes as long as its heaviest item, a CTA by
// itself for most of the time (5 us + 1.15 us per KV tile, 1.4 times that where running maxima move), or as all items
// together on all slots (two CTAs per SM, 6 us + 2 us per tile and slot), whichever is more; its items come heaviest first,
// so the two do not add up.  The persistent launch cuts the steps into equal spans, but a span in the light end of a head
// is many items of one to a few tiles, each with its own start and end, and that span is the last to finish.  So it pays only where
// the heaviest item alone is far above the mean: few heads, long ones.  Time of the persistent launch with its merge over
// that of the plain one, N(0,1) inputs / x20 outliers, ranges over 8 to 48 tiles in the heaviest item:
//   D=64, int8: 1 head 0.40-0.71 / 0.35-0.59, 3 0.69-0.88 / 0.59-0.74, 5 0.90-1.04 / 0.73-0.91, 6 from 14 to 32 tiles
//   0.95-1.05 / 0.81-0.92, 8 0.99-1.29 / 0.82-1.25; un-quantised 5 0.87-0.99 / 0.67-0.85, 8 from 16 to 28 tiles 0.95-1.05 /
//   0.81-0.86, 10 1.14-1.36 / 0.90-1.21;
//   D=128: 1 head 0.50-0.78 / 0.41-0.61, 2 0.68-0.88 / 0.53-0.68, 3 0.83-1.10 / 0.67-0.86, 4 from 20 tiles on 0.93-1.04 / 0.71-0.86,
//   below 0.92-1.19 / 0.71-0.93, 5 1.08-1.30 / 0.86-1.00.
// With 64 tiles 4 heads, D=64, 0.97 / 0.94, 5 heads 1.09 / 1.07: the heaviest item is less than 2.2 times the mean.
// heads: (batch, query head) pairs; heaviest: KV tiles of the heaviest item; mean_steps: KV tiles per CTA of the
// persistent launch.
static inline int sage_causal_streamk(int64_t heads, int64_t heaviest, double mean_steps, int D, int qkf = 0) {
  if (heaviest < 8 || heaviest < 2.2 * mean_steps) return 0;
  if (D == 128) return heads <= 3 || (heads == 4 && heaviest >= 20);
  if (heads <= 5) return 1;
  if (heads == 6) return heaviest >= 14 && heaviest >= 2.8 * mean_steps;
  return qkf && heads <= 8 && heaviest >= 16 && heaviest >= 2.5 * mean_steps;
}

// Whether the un-quantised launch converts a bf16 V itself.  It does so for every item anew, where a launch ahead of it
// converts each tile once; that launch costs about 3.5 us of host time and 3 us on the GPU.  The conversion of an item's
// first tile hides under its first Q.K^T; further ones cost 0.3 us (D=128) or half of that.  us per call, launch
// ahead / inside: 48 items of 1 tile 11.1 / 7.3, 1536 of 1 51.1 / 43.9, D=64 256 of 2 10.7 / 8.6, 160 of 8 20.0 / 19.4, D=128 64 of 4
// 12.5 / 11.8, 384 of 2 (mean, causal) 19.2 / 20.1, 128 of 8 17.9 / 18.4, 512 of 4 26.5 / 31.1.  So: one tile, or at most
// 4 (D=128) or 8 tiles per SM.  One tile, D=128, stays ahead where there are more than 4 items per SM and several of them to
// a tile of V: 1080 items, 45 to a head, 28.1 / 29.1, 1200, 6 to a head, 33.3 / 34.4, but 1100, one to a head, 37.4 / 31.9, and
// 576, 24 to a head, 16.2 / 16.3.  With D=128 and more items than SMs the rings hold one tile, and the conversion stands
// between each load and its use: 160 causal items of 3 (mean) 18.0 / 21.7.
static inline int sage_few_v_tiles(int64_t items, int64_t nq, int64_t nkv, int is_causal, int D, int sms) {
  if (nkv <= 1) return D == 64 || items <= 4 * (int64_t)sms || nq <= 3;
  if (D == 128 && items > sms) return 0;
  const double mean = is_causal && nq <= nkv ? 0.5 * (double)(nq + 1) : (double)nkv;      // tiles of an item
  const double per_sm = mean * (items > sms ? (double)items / sms : 1.0);
  return per_sm <= (D == 128 ? 4.0 : 8.0);
}

// Whether a launch without a causal mask takes two query tiles per CTA (sage_pair_kernel: one persistent CTA per SM, the
// loads and the first Q.K^T of the next item under the end of the current one).  items: pairs of tiles; nq: tiles per
// head.  Figures: time of the attention launch that is taken otherwise (with its merge) over that of this one, from 1600
// combinations of heads, query tiles and KV tiles.  Two kinds of problem gain:
// - many items of few KV tiles, where the start and end of an item is much of it.  From 5 rounds (of 2 tiles per SM) on,
//   at 2 / 4 / 8 / 12 KV tiles: int8 D=128 1.54 / 1.41 / 1.26 / 1.15 (13: 0.95-1.1), D=64 1.39 / 1.31 / 1.16 / 1.08
//   (beyond, 1.03-1.08); un-quantised D=128 1.39 / 1.38 / 1.26 / 1.10, D=64 1.22 / 1.19 / 1.04 / 1.01.  (Otherwise means
//   persistent CTAs of one tile for most of these.  Against one CTA per tile it is 1.0-1.2 up to 4 tiles and 0.9-1.0 at 8.)
//   With 3 or 4 rounds the last, part-filled one weighs more: int8 at 4 / 8 tiles D=64 1.14 / 0.95 (3 rounds), 1.30 / 1.15
//   (4), D=128 0.98 / 0.98 and 1.05 / 0.97; un-quantised D=64 at 1 / 2 / 4 tiles 1.19 / 1.04 / 0.92 and at 3 / 8 1.27 / 1.04 (4),
//   D=128 0.90-1.2 without an order.  Where they are badly filled: sage_pairs_fill.
// - one or two rounds and a few items over, whose steps are cut into spans, where whole tiles on two CTAs per SM fill
//   the last round badly.  int8, D=64, with 0.06 to 0.2 of a round over and up to 96 KV tiles 1.00-1.13 (160 items of 32
//   tiles 77.5 -> 73.5 us); with less over 0.95-1.02 (spans of one tile each, and more to merge), longer items 0.99-1.01.
//   D=128 where the items over are cut into whole spans of 4 tiles 1.03-1.18; where spans reach over the end of an item
//   0.96-1.06, and 0.93-0.96 of what the launch taken otherwise is now; measured up to 0.13 or 0.1 of a round and 40 or 32
//   tiles.  Un-quantised, D=128, up to 0.3 of a round 1.01-1.30.
// Long items are no faster this way: the SM's clock rises (the K and V tiles are fetched once for both query tiles), but
// an item takes more clocks.  An odd number of tiles per head leaves half a pair empty: the rounds are counted in tiles
// (580 tiles fill two rounds of the launch with a CTA per tile, though they are 300 pairs: 20 heads of 3711 tokens, D=64,
// 108 us against 130).  Cut launches, int8, D=64: 0.92-1.00 with more KV tiles than query tiles or less than 0.07 of a round
// over, else 1.00-1.16.  Whole items: with 9 to 15 tiles per head the line lies at half as many KV tiles (from 5 rounds on,
// int8 D=64, 3 / 13 tiles 1.22 / 0.97; un-quantised 4 / 12 1.19 / 0.97), with fewer than 9 they are not taken (0.8-1.4 at 1 to 4 tiles).
#define SAGE_PAIR_WHOLE_ROUNDS 3          // from here on the items left over are not cut into spans
#define SAGE_PAIR_SPAN_TILES 4            // fewest KV tiles of a span, unless the items left over have fewer
static inline int sage_takes_pairs(int64_t items, int64_t nq, int64_t nkv, int D, int qkf, int sms) {
  const int odd = nq % 2 == 1;
  if (odd && nq < 9) return 0;
  const int64_t tiles = odd ? items / ((nq + 1) / 2) * nq : 2 * items;
  const int64_t rounds = tiles / (2 * sms);
  if (rounds >= SAGE_PAIR_WHOLE_ROUNDS) {
    int64_t most;
    if (!qkf) most = rounds >= 5 ? 12 : (rounds == 4 && D == 64) ? 8 : 4;
    else if (D == 128) most = rounds >= 5 ? 12 : 0;
    else most = rounds >= 5 ? 8 : rounds == 4 ? 3 : 1;
    return nkv <= (odd && nq < 17 ? most / 2 : most);
  }
  const double rest = (double)tiles / (2.0 * sms) - (double)rounds;
  if (rounds < 1 || nkv < 16 || items / sms != rounds) return 0;
  if (qkf) return D == 128 && rest <= 0.3;
  if (D == 64) return rest > (odd ? 0.07 : 0.06) && rest <= 0.2 && nkv <= (odd && nq < 96 ? nq : 96);
  if (nkv % SAGE_PAIR_SPAN_TILES != 0 || items % sms * (nkv / SAGE_PAIR_SPAN_TILES) > sms) return 0;
  return rest > 0.0 && rest <= (rounds == 1 ? 0.13 : 0.1) && nkv <= (rounds == 1 ? 40 : 32);
}

// Whether whole pairs fill their rounds well enough, the last of which takes as long as the others, where the other choice
// is one CTA per tile.  Idle slots cost in proportion to the KV tiles of an item.  int8, 3 and 4 rounds, KV tiles times the
// idle share against the speed of one CTA per tile: D=128 up to 0.3 1.02-1.16, 0.35-0.44 1.01-1.02, 0.45-0.7 0.98-1.00 (one
// KV tile, 1.04-1.16 throughout, stays below), 0.8-0.95 0.94-0.99; D=64 0.4-0.5 0.99-1.09, 0.66 0.97, 0.95 0.91.  Where half pairs
// (an odd number of tiles per head) bring one round more than the tiles have, 0.2-0.25 1.04-1.16, 0.26-0.33 0.93-0.99, 0.5
// 0.95.  More rounds and un-quantised calls (sage_takes_pairs) are faster as pairs all the same.
static inline int sage_pairs_fill(int64_t items, int64_t nq, int64_t nkv, int D, int qkf, int sms) {
  const int64_t tiles = items / ((nq + 1) / 2) * nq;
  const int64_t rounds = tiles / (2 * sms), pair_rounds = (items + sms - 1) / sms;
  if (qkf || rounds < SAGE_PAIR_WHOLE_ROUNDS || rounds >= 5) return 1;
  const double idle = 2.0 * (double)sms * (double)pair_rounds / (double)tiles - 1.0;
  const int one_more = pair_rounds > (tiles + 2 * sms - 1) / (2 * sms);
  return (double)nkv * idle <= (one_more ? 0.25 : D == 64 ? 0.5 : 0.44);
}

extern "C" {
// lse[b,h,s] += sm_scale * q[b,h,s,:] . k_mean[b, h / (Hq/Hkv), :], in fp32: refers the log-sum-exp of a
// launch on centred keys (smooth_k) to the original ones.  lse: contiguous [B,Hq,Sq]; k_mean:
// contiguous [B,Hkv,D] in the dtype of q.
int sage_lse_add_q_mean(const sage_strided_t* q, int dtype, const void* k_mean, float* lse, int B, int Hq, int Hkv, int Sq,
                        int D, float sm_scale, void* stream);
// The same without a launch of its own: sage_quant_q_mean_dot quantises Q like sage_quant_qk_int8 and leaves
// q[b,h,s,:] . k_mean[b, h / (Hq/Hkv), :] in lse, and sage_qk_int8_sv_f16_attn_lse_add, which is
// sage_qk_int8_sv_f16_attn_ws otherwise, adds lse_add_scale times that to what it writes there.
int sage_quant_q_mean_dot(const sage_strided_t* q, int dtype, const void* k_mean, int B, int Hq, int Hkv, int Sq, int D,
                          float sm_scale, int8_t* q_i8, float* q_scale, float* lse, void* stream);
int sage_qk_int8_sv_f16_attn_lse_add(const int8_t* q_i8, const int8_t* k_i8, const sage_strided_t* v16, void* o,
                                     int64_t o_stride_b, int64_t o_stride_h, int64_t o_stride_s, const float* q_scale,
                                     const float* k_scale, int out_dtype, int B, int Hq, int Hkv, int Sq, int Skv, int D,
                                     int is_causal, float* lse, float lse_add_scale, int* status, void* workspace,
                                     int64_t workspace_bytes, void* stream);
// Workspace bytes of one launch, as it will plan it: of sage_qk_int8_sv_f16_attn_ws with these sizes and output
// strides (heads folded where the rule above says so), and of sage_direct_attn_ws.  The public
// sage_attn_workspace_bytes knows neither the kv heads nor the strides and gives the most that any of them takes.
int64_t sage_int8_workspace_bytes(int B, int Hq, int Hkv, int Sq, int Skv, int D, int is_causal, int64_t o_stride_h,
                                  int64_t o_stride_s);
int64_t sage_direct_workspace_bytes(int B, int Hq, int Sq, int Skv, int D, int is_causal);
// sage_direct_attn on bf16 tensors with V as it is (bf16, converted inside the launch with the rounding of
// sage_v_to_f16), and whether that is the better way for these sizes.
int sage_direct_attn_bf16_v(const sage_strided_t* q, const sage_strided_t* k, const sage_strided_t* v, void* o,
                            int64_t o_stride_b, int64_t o_stride_h, int64_t o_stride_s, int B, int Hq, int Hkv, int Sq, int Skv,
                            int D, int is_causal, float sm_scale, float* lse, int* status, void* stream);
int sage_direct_takes_bf16_v(int B, int Hq, int Sq, int Skv, int D, int is_causal);
// Test hook: how many CTAs of plain attention launches have started on each SM of the current device (counted
// since the library was loaded; synchronises).
int sage_test_sm_arrivals(unsigned* counts, int n);
}
