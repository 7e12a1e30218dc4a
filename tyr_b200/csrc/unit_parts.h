// How many CTAs of the dK/dV kernel share a key block in launches with few of them.  Plain C++ on sizes alone (SM count
// and cluster capacities are arguments), so that the choice can be checked on the host.
#pragma once
#include <algorithm>

namespace tyr {

struct BwdSizes {
  int n_kblk, n_qblk;      // blocks of 128 keys and of 128 query rows
  int n_kv, n_q;           // KV heads and query heads of the whole batch
  int group, window;       // query heads per KV head; 0: no window
  bool causal;
};
constexpr int kMaxPlanSms = 256;
constexpr int kPartsChoices = 4;  // 1, 2, 4 or 8 CTAs per unit

// A launch of few units takes as long as its longest one (the first keys are seen by every query row of every head
// of the group); with a cluster of CTAs per unit the unit's pairs are shared out, but a cluster costs its merge and
// set-up (kMergePairs streamed pairs), leaves the SMs that hold no whole cluster empty, a cluster that finds no place
// waits for one, and the dQ kernel, which otherwise runs on the SMs that are left, comes after all of them.  So the two
// kernels are laid out on the SMs as they will be: units or clusters longest first, the second round behind the shortest of
// the first, then the dQ kernel's CTAs in their order on the SMs as they fall free.  A dQ pair counts 4/5 of a dK/dV
// pair.  The number with the shortest end wins, more than one only where it is a tenth shorter.
// `capacity[k]`: clusters of 2^k CTAs that are resident at once.  Over 164 launches of 1 to 16 key blocks, up to 32 KV heads
// and groups of 1 to 4, measured with 1, 2, 4 and 8 CTAs each: on average 0.05 % off the best number, 3.7 % at most,
// none slower than with one CTA.  One prompt, one CTA -> the choice, backward alone: 512 rows, 32/8 heads of 128 39.9 ->
// 29.2 us, 8/2 heads 37.2 -> 19.0; 2000 rows, 8/2 heads of 64 98.8 -> 36.2; 1024 rows, 6/6 heads of 64 19.8 -> 17.7.
constexpr int kMergePairs = 3;
inline int choose_unit_parts(const BwdSizes& z, int sms, const int* capacity) {
  if (sms > kMaxPlanSms || z.n_kblk <= 0 || z.n_qblk <= 0) return 1;
  constexpr int kPair = 5, kDqPair = 4;
  auto pairs_of_keys = [&](int blk) {    // streamed pairs of a unit
    const int lo = z.causal ? std::min(blk, z.n_qblk) : 0;
    const int hi = z.window > 0 ? std::min(z.n_qblk, (blk * 128 + 127 + z.window - 1) / 128 + 1) : z.n_qblk;
    return std::max(hi - lo, 0) * z.group;
  };
  auto pairs_of_rows = [&](int blk) {    // KV tiles of a dQ unit
    const int hi = z.causal ? std::min(z.n_kblk, blk + 1) : z.n_kblk;
    const int lo = z.window > 0 ? std::max(0, blk * 128 - z.window + 1) / 128 : 0;
    return std::max(hi - lo, 0);
  };
  const long long units = (long long)z.n_kblk * z.n_kv, row_units = (long long)z.n_qblk * z.n_q;
  if (units >= 2ll * sms) return 1;
  const int n = (int)units, dq_ctas = (int)std::min<long long>(row_units, sms);
  int keys[2 * kMaxPlanSms];   // pairs of each unit, longest first
  for (int b = 0, i = 0; b < z.n_kblk; ++b)
    for (int h = 0, x = pairs_of_keys(b); h < z.n_kv; ++h) keys[i++] = x;
  if (!z.causal || z.window > 0) std::sort(keys, keys + n, [](int a, int b) { return a > b; });
  int rows[kMaxPlanSms] = {};  // KV tiles of each CTA of the dQ kernel: one unit, two in mirrored rounds, or the mean
  if (row_units <= 2ll * dq_ctas) {
    int i = 0;
    for (int b = z.n_qblk - 1; b >= 0; --b)
      for (int h = 0, x = pairs_of_rows(b); h < z.n_q; ++h, ++i) rows[i < dq_ctas ? i : 2 * dq_ctas - 1 - i] += x;
  } else {
    long long total = 0;
    for (int b = 0; b < z.n_qblk; ++b) total += (long long)pairs_of_rows(b) * z.n_q;
    std::fill(rows, rows + dq_ctas, (int)std::min<long long>((total + dq_ctas - 1) / dq_ctas, 1 << 24));
  }
  int best = 0, best_parts = 1;
  for (int k = 0; k < kPartsChoices; ++k) {
    const int parts = 1 << k, slots = k == 0 ? sms : std::min(capacity[k], sms / parts);
    if (slots <= 0) continue;
    auto cost = [&](int i) { return kPair * (((keys[i] + parts - 1) >> k) + (k == 0 ? 1 : kMergePairs)); };
    int end[kMaxPlanSms], all_started = 0;         // when the cluster slots fall free, in order
    if (n <= slots) {
      std::fill(end, end + slots - n, 0);
      for (int s = 0; s < n; ++s) end[slots - 1 - s] = cost(s);
    } else if (n <= 2 * slots) {
      for (int s = 0; s < slots; ++s) end[s] = cost(s) + (2 * slots - 1 - s < n ? cost(2 * slots - 1 - s) : 0);
      std::sort(end, end + slots);
      if (k > 0) all_started = cost(2 * slots - n);
    } else {
      long long total = 0;
      for (int i = 0; i < n; ++i) total += cost(i);
      std::fill(end, end + slots, (int)(total / slots));
      all_started = end[0] - cost(n - 1);
    }
    int span = end[slots - 1];
    const int idle = sms - slots * parts;          // SMs that no cluster takes
    for (int j = 0; j < dq_ctas; ++j)
      span = std::max(span, std::max(j < idle ? 0 : end[(j - idle) >> k], all_started) + kDqPair * rows[j]);
    if (k == 0 || 10ll * span < 9ll * best) {
      best = span;
      best_parts = parts;
    }
  }
  return best_parts;
}

}  // namespace tyr
