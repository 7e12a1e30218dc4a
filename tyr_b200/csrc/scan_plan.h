// How a launch of the decode kernel cuts its keys.  Plain C++ on sizes alone (the SM count is an argument), so that
// the plans can be checked on the host over their whole range.
#pragma once
#include <algorithm>

namespace tyr {

constexpr int kWarpKeys = 16;       // keys of a pipeline stage one warp works on
constexpr int kChunkUnit = 64;      // keys; chunk lengths are multiples of it
constexpr int kMaxWsChunks = 64;    // chunks of a sequence in the workspace form (the merge holds two LSEs per lane)

struct ScanPlan {
  bool cluster = false;  // n_splits CTAs per (sequence, KV head, row group) merge among themselves; else chunk_len keys per CTA
  int n_splits = 1, chunk_len = 0, warps = 4;
  // every key of a sequence of up to max_len is in one of the CTAs' ranges
  bool covers(int max_len) const {
    return cluster ? n_splits >= 2 && n_splits <= 16 : chunk_len > 0 && (long long)chunk_len * n_splits >= max_len;
  }
  bool needs_workspace() const { return !cluster && n_splits > 1; }
};

// The cut of a launch that is done without a workspace: a cluster of CTAs for each (sequence, KV head), or one
// chunk.  `units`: (sequence, KV head, row group) triples.  Always a plan that covers max_len; *pays says whether the
// launch is small enough for it to beat the cut into chunks of the workspace form.
//
// The most CTAs that still run all at once, clusters placed: two per SM less the slots a GPC cannot
// give to whole clusters.  Clusters of 16 leave more of them unused and are only taken where half the
// slots are enough (for head_dim 64 three quarters).  A CTA gets at least one step of its warps' keys (64 or 128); past
// 1024 (head_dim 64: 2048) keys per CTA the workspace form's greater choice of chunk counts wins.
// Device time, workspace form -> this one, 8 KV heads of 128: one sequence of 512 keys 8.2 -> 4.8 us,
// 1537: 8.8 -> 6.7, 4096: 9.5 -> 8.5, 16384: 18.9 -> 18.3 (32768: 29.2 -> 30.7, not taken); 4 x 2051 12.6 -> 10.8,
// 4 x 8192 27.1 -> 24.2; 8 x 1537 14.2 -> 13.2; 12 KV heads of 64: 1537 7.1 -> 5.4, 4 x 8192 23.7 -> 20.0.
// Eight warps per CTA instead of four where one CTA has an SM to itself, and for head_dim 64, whose
// stages are half as large.
inline ScanPlan own_scan_plan(int head_dim, long long units, int max_len, int max_splits, int sm, bool* pays) {
  const int slots = 2 * sm - sm / 4;
  const int warps = head_dim == 64 ? 8 : 4;
  int n = (int)std::min<long long>(8, slots / std::max<long long>(units, 1));
  if (units * 16 <= (head_dim == 64 ? slots * 3 / 4 : slots / 2)) n = 16;
  n = std::min(n, (max_len + kWarpKeys * warps - 1) / (kWarpKeys * warps));
  n = std::max(std::min(n, max_splits), 1);
  *pays = max_len <= (long long)(head_dim == 64 ? 2048 : 1024) * n;
  // few, long pieces that leave a quarter of the slots empty (4 x 24 KV heads, 2000 keys: 29.2 against 25.7 us)
  if (n > 1 && n < 8 && max_len > 512 * n && units * n * 4 < slots * 3) *pays = false;
  ScanPlan s;
  s.cluster = n > 1;
  s.n_splits = n;
  s.chunk_len = n > 1 ? 0 : (max_len + kChunkUnit - 1) / kChunkUnit * kChunkUnit;
  s.warps = n > 1 ? warps : (units <= sm ? 8 : 4);
  return s;
}

// The cut of a typed call with few query rows per KV head (rows = group * q_seq) over kv_seq keys.  Launches that
// the workspace form serves better take it where the caller gives a workspace; without one the cluster is as
// large as fits a wave, whatever the number of keys.  Against the 128-row kernel, which served these calls before:
// 64 x 32/8 heads x 2051 keys (one chunk per pair) 217 -> 84 us; without a workspace 1 x 32/8 x 20000 249 -> 22 us, 4 x 24
// x 2000 36 -> 20, 20 x 8 x 30000 809 -> 381.
inline ScanPlan few_rows_plan(int head_dim, long long units, int kv_seq, bool have_workspace, int sm) {
  bool pays;
  const ScanPlan own = own_scan_plan(head_dim, units, kv_seq, kMaxWsChunks, sm, &pays);
  // One or two (batch, KV head) pairs over long keys: chunks in the workspace reach more of the device than one or two
  // clusters of 16 can, and cost a second launch.  Workspace form against clusters, one pair: heads of 64 6000 keys 7.3
  // against 6.9 us, 8192 7.3 / 7.5, 16384 8.3 / 10.0; of 128 8192 10.6 / 9.6, 12000 11.4 / 11.8, 16384 11.8 / 14.1; two pairs:
  // of 64 8192 7.7 / 7.5, 12000 8.1 / 8.7; of 128 12000 12.4 / 12.0, 16384 13.2 / 14.3.
  const bool long_pair = units <= 2 && kv_seq > (head_dim == 64 ? 8192 : 12288);
  if (!have_workspace || (pays && !long_pair)) return own;
  // chunks that give one wave of CTAs, as in decode_launch_splits
  const int slots = 2 * sm;
  long long c = ((long long)kv_seq * units + slots - 1) / slots;
  c = std::max<long long>(c, (kv_seq + kMaxWsChunks - 1) / kMaxWsChunks);
  c = (c + kChunkUnit - 1) / kChunkUnit * kChunkUnit;
  if (c >= kv_seq) return own;  // one chunk per pair already is a wave: no partials to merge
  ScanPlan s;
  s.chunk_len = (int)c;
  s.n_splits = (kv_seq + s.chunk_len - 1) / s.chunk_len;
  return s;
}

}  // namespace tyr
