// Split-KV flash-decoding for one query token per sequence over a ragged KV
// cache, plus the LSE merge of the partial results.
//
// Replaces the q_seq = 1 call of QwenAttention.forwardStep
// (Tyr/Model/Qwen/Attention.lean:198-200 -> cc/src/tyr.cpp:4100-4133), which
// repeat_interleaves the whole cache per token.  Here every K/V byte is read
// from HBM exactly once: one CTA owns (sequence, KV head, chunk of keys) and
// serves all query heads of that KV head together.  The merge is the formula of
// ringAttnReduce (Tyr/GPU/Kernels/RingAttn.lean:164-180), kept in the log2 domain.
// It runs in one of two places: in the launch itself, when the CTAs that share a sequence and KV head
// form a cluster and exchange their partials through distributed shared memory (small launches), or
// in a second launch over partials in the workspace.
//
// A call with a few query rows per head (the typed call of a generating loop, q_seq = 1, and other
// unmasked calls with group * q_seq <= kMaxFewRows) is served by the same kernel: the rows of a KV head
// are its (query head, query row) pairs.
//
// The kernel is HBM-bound.  Keys stream global -> shared with 16-byte cp.async
// into a 3-stage ring (XOR-swizzled rows, conflict-free for ldmatrix); the tiny
// contractions (<=16 query rows) run on warp-level m16n8k16 MMAs so that issue
// slots stay free for the loads.  Each warp owns 16 of the keys of a stage and
// keeps its own (max, sum, O); the warps merge through shared memory.
// Both products are formed transposed, keys (S^T = K Q^T) and head dims (O^T = V^T P^T) as the 16
// rows of the MMA and query rows as its 8 columns: a warp-level MMA takes about 31 cycles of its SM
// sub-partition here whatever it is used for, and with the up to 8 query rows of a usual group in the
// 16-row operand half of each was wasted.
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "attn_internal.h"
#include "mma_sync.cuh"
#include "ptx_sm100.cuh"
#include "scan_plan.h"

namespace tyr {
namespace {

constexpr int kStages = 3;
constexpr int kMergeThreads = 128;
constexpr int kMaxFewRows = 16;
constexpr int kMinChunk = 256;  // keys; shorter chunks only add merge traffic
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

struct DecodeParams {
  const __nv_bfloat16* q;
  __nv_bfloat16* o;
  float* lse;
  const __nv_bfloat16 *k, *v;
  const void* const* k_ptrs;
  const void* const* v_ptrs;
  const int32_t* kv_lens;
  const int64_t* kv_head_strides;
  int batch, n_head, n_kv_head, max_kv_seq;
  int q_seq;        // query rows per head (1 in the decode entries)
  int rows;         // query rows per KV head: group * q_seq, row r = (head r / q_seq of the group, query r % q_seq)
  int row_groups;   // CTAs (of up to 16 rows each) per KV head and chunk of keys
  int64_t qs[3], os[3], ks[3], vs[3];  // qs, os: batch, head, query row
  float scale_log2;
  int chunk_len, n_splits;
  float* ws_o;    // [batch, n_head * q_seq, n_splits, D] normalised partial outputs
  float* ws_lse;  // [batch, n_head * q_seq, n_splits] log2-domain partial LSE
  int ws_aligned; // ws_o is 16-byte aligned
  int* status;    // per-device status word (out-of-range lengths are reported there)
};

// Row `r` of the KV head's rows (query head and query row) in O and in the LSE array.
__device__ __forceinline__ __nv_bfloat16* o_row(const DecodeParams& p, int b, int hkv, int r) {
  const int h = r / p.q_seq, i = r - h * p.q_seq;
  return p.o + b * p.os[0] + (int64_t)(hkv * (p.rows / p.q_seq) + h) * p.os[1] + i * p.os[2];
}
__device__ __forceinline__ int64_t lse_index(const DecodeParams& p, int b, int hkv, int r) {
  return (int64_t)b * p.n_head * p.q_seq + hkv * p.rows + r;
}

// The value scores are taken relative to, given their maximum so far.  Where all of them are -inf that is 0, so that
// their exponentials and the weight of what was summed before are 0 and not 2^(-inf + inf): a warp sees 16 keys
// at a time, and a key whose products with the query overflow to -inf, or that a caller masks that way, has no weight.
__device__ __forceinline__ float finite_ref(float m) { return m == -INFINITY ? 0.f : m; }

// A length outside [1, max_kv_seq] (the workspace and the grid are sized for max_kv_seq, so a
// longer one would index past both): report it once per sequence, give a sequence without any
// key a defined row (zeros, LSE = -inf), and return the length forced into [0, max_kv_seq].
// Kept out of line so that this rare path costs the scan loop no registers.
template <int D>
__device__ __noinline__ int bad_length(int raw, const DecodeParams& p, int b, int hkv, int row0, int rows_here) {
  const int len = min(max(raw, 0), p.max_kv_seq);
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0 && hkv == 0 && row0 == 0) atomicOr(p.status, kStatusOutOfRange);
    if (len == 0) {
      for (int idx = threadIdx.x; idx < rows_here * D; idx += blockDim.x) {
        const int r = row0 + idx / D, d = idx % D;
        o_row(p, b, hkv, r)[d] = __float2bfloat16_rn(0.f);
        if (d == 0 && p.lse) p.lse[lse_index(p, b, hkv, r)] = -INFINITY;
      }
    }
  }
  return len;
}

template <int D, int kWarps, int kNT>
struct DCfg {
  static constexpr int kRows = 8 * kNT;                 // query rows of a CTA, in column tiles of 8
  static constexpr int kThreads = 32 * kWarps;
  static constexpr int kTileKeys = kWarpKeys * kWarps;  // keys per pipeline stage
  static constexpr int kRowBytes = D * 2;
  static constexpr int kChunksPerRow = D / 8;  // 16-byte chunks
  static constexpr int kTileBytes = kTileKeys * kRowBytes;
  static constexpr int kStageBytes = 2 * kTileBytes;  // K then V
  static constexpr int kSmemBytes = kStages * kStageBytes;
  // cross-warp merge reuses the ring: the warps' rows of D floats, rows padded by 4 floats so that
  // the pieces of four rows a warp stores at once fall on different banks, + 2 floats of (max, sum) per row
  static constexpr int kMergeStride = D + 4;
  // ... and behind it, for a cluster's merge, this CTA's rows of D floats and their (max, sum)
  static constexpr int kPartOff = kWarps * kRows * (kMergeStride + 2);  // in floats
  static_assert((kPartOff + kRows * (D + 2)) * 4 <= kSmemBytes, "merge scratch fits in the ring");
};

// kCluster: the grid's x extent is one cluster, its CTAs cut the sequence's keys evenly and merge among
// themselves; no workspace, no second launch.  Otherwise chunks of p.chunk_len keys, partials to the workspace.
template <int D, int kWarps, int kNT, bool kCluster>
__global__ void __launch_bounds__(32 * kWarps)
decode_kernel(const __grid_constant__ DecodeParams p) {
  using C = DCfg<D, kWarps, kNT>;
  constexpr int kThreads = C::kThreads, kTileKeys = C::kTileKeys, kRows = C::kRows;
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem));

  grid_launch_dependents();
  grid_dependency_wait();
  const int split = blockIdx.x;
  const int hkv = blockIdx.y / p.row_groups;
  const int row0 = (blockIdx.y % p.row_groups) * kRows;   // first of the KV head's rows this CTA serves
  const int rows_here = min(kRows, p.rows - row0);
  const int b = blockIdx.z;
  int len = p.kv_lens ? p.kv_lens[b] : p.max_kv_seq;
  if (len <= 0 || len > p.max_kv_seq) len = bad_length<D>(len, p, b, hkv, row0, rows_here);
  if (kCluster && len == 0) return;  // the whole cluster: its CTAs share the sequence
  int chunk_len = p.chunk_len;
  if (kCluster) chunk_len = ((len + p.n_splits - 1) / p.n_splits + kWarpKeys - 1) / kWarpKeys * kWarpKeys;
  const int n_chunks = (len + chunk_len - 1) / chunk_len;
  if (!kCluster && split >= n_chunks) return;
  const int key_begin = split * chunk_len;
  const int key_end = min(len, key_begin + chunk_len);
  const int n_tiles = max(key_end - key_begin + kTileKeys - 1, 0) / kTileKeys;  // 0: a CTA of the cluster without keys

  const __nv_bfloat16 *kbase, *vbase;
  if (p.k_ptrs) {
    const int64_t hs_k = p.kv_head_strides ? p.kv_head_strides[b] : (int64_t)len * p.ks[2];
    const int64_t hs_v = p.kv_head_strides ? p.kv_head_strides[b] : (int64_t)len * p.vs[2];
    kbase = static_cast<const __nv_bfloat16*>(p.k_ptrs[b]) + hkv * hs_k;
    vbase = static_cast<const __nv_bfloat16*>(p.v_ptrs[b]) + hkv * hs_v;
  } else {
    kbase = p.k + b * p.ks[0] + hkv * p.ks[1];
    vbase = p.v + b * p.vs[0] + hkv * p.vs[1];
  }

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quad = lane >> 2, t4 = lane & 3;

  // ---- stage loader: kTileKeys keys x D bf16 of K and of V, 16 bytes per cp.async
  auto load_tile = [&](int tile, int stage) {
    const uint32_t sk = sbase + stage * C::kStageBytes, sv = sk + C::kTileBytes;
    const int k0 = key_begin + tile * kTileKeys;
#pragma unroll
    for (int it = 0; it < kTileKeys * C::kChunksPerRow / kThreads; ++it) {
      const int idx = it * kThreads + tid;
      const int kr = idx / C::kChunksPerRow, c = idx % C::kChunksPerRow;
      const int key = min(k0 + kr, key_end - 1);  // rows past the end re-read the last valid key
      cp_async16(sk + sw_off<D>(kr, c), kbase + (int64_t)key * p.ks[2] + c * 8);
      cp_async16(sv + sw_off<D>(kr, c), vbase + (int64_t)key * p.vs[2] + c * 8);
    }
  };

#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < n_tiles) load_tile(s, s);
    cp_async_commit();
  }

  // ---- Q fragments (B operand: column = query row of this KV head)
  uint32_t qb[kNT][D / 16][2];
#pragma unroll
  for (int nt = 0; nt < kNT; ++nt) {
    const int r = row0 + nt * 8 + quad, h = r / p.q_seq;
    const bool live = nt * 8 + quad < rows_here;
    const __nv_bfloat16* qr = p.q + b * p.qs[0] + (int64_t)(hkv * (p.rows / p.q_seq) + h) * p.qs[1] + (r - h * p.q_seq) * p.qs[2];
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
      for (int kh = 0; kh < 2; ++kh)          // d, d + 8
        qb[nt][ks][kh] = live ? *reinterpret_cast<const uint32_t*>(qr + ks * 16 + kh * 8 + t4 * 2) : 0u;
  }

  float m_run[kNT][2], l_run[kNT][2];  // query rows nt * 8 + 2 t4, + 1 (log2 domain; l: this lane's keys only)
  float oacc[kNT][D / 16][4];          // O^T: dims 16 m + quad (+ 8 in [2], [3]), the same two query rows
#pragma unroll
  for (int nt = 0; nt < kNT; ++nt) {
    m_run[nt][0] = m_run[nt][1] = -INFINITY;
    l_run[nt][0] = l_run[nt][1] = 0.f;
#pragma unroll
    for (int m = 0; m < D / 16; ++m)
#pragma unroll
      for (int x = 0; x < 4; ++x) oacc[nt][m][x] = 0.f;
  }

  for (int tile = 0; tile < n_tiles; ++tile) {
    cp_async_wait<kStages - 2>();
    __syncthreads();
    if (tile + kStages - 1 < n_tiles) load_tile(tile + kStages - 1, (tile + kStages - 1) % kStages);
    cp_async_commit();

    const int stage = tile % kStages;
    const uint32_t sk = sbase + stage * C::kStageBytes, sv = sk + C::kTileBytes;
    const int wkey0 = warp * kWarpKeys;                              // this warp's keys in the tile
    const int gkey0 = key_begin + tile * kTileKeys + wkey0;   // global index of the first
    if (gkey0 >= key_end) continue;                           // warp-uniform: nothing valid

    // S^T = K Q^T for 16 keys, as two chains over alternate 16-element groups of the head dimension
    // (an MMA's result is some 30 cycles away from the next one's input)
    float sacc[kNT][2][4];
#pragma unroll
    for (int nt = 0; nt < kNT; ++nt)
#pragma unroll
      for (int x = 0; x < 8; ++x) sacc[nt][x >> 2][x & 3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      uint32_t ka[4];
      ldsm_x4(sk + sw_off<D>(wkey0 + (lane & 15), 2 * ks + (lane >> 4)), ka);
#pragma unroll
      for (int nt = 0; nt < kNT; ++nt) mma_bf16_16816(sacc[nt][ks & 1], ka, qb[nt][ks][0], qb[nt][ks][1]);
    }
    // scale, mask the tail, online softmax per query row; this lane has keys quad and quad + 8
    const bool live0 = gkey0 + quad < key_end, live1 = gkey0 + quad + 8 < key_end;
    float sx[kNT][4], mx[kNT][2];
    bool grown = false;
#pragma unroll
    for (int nt = 0; nt < kNT; ++nt)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        sx[nt][x] = live0 ? (sacc[nt][0][x] + sacc[nt][1][x]) * p.scale_log2 : -INFINITY;
        sx[nt][2 + x] = live1 ? (sacc[nt][0][2 + x] + sacc[nt][1][2 + x]) * p.scale_log2 : -INFINITY;
        mx[nt][x] = fmaxf(sx[nt][x], sx[nt][2 + x]);
      }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1)
#pragma unroll
      for (int nt = 0; nt < kNT; ++nt)
#pragma unroll
        for (int x = 0; x < 2; ++x) mx[nt][x] = fmaxf(mx[nt][x], __shfl_xor_sync(0xffffffffu, mx[nt][x], o));
#pragma unroll
    for (int nt = 0; nt < kNT; ++nt)
#pragma unroll
      for (int x = 0; x < 2; ++x) grown = grown || mx[nt][x] > m_run[nt][x];
    if (__any_sync(0xffffffffu, grown)) {  // after the first tiles a row's maximum seldom moves
#pragma unroll
      for (int nt = 0; nt < kNT; ++nt) {
        float alpha[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const float m_new = fmaxf(m_run[nt][x], mx[nt][x]);
          alpha[x] = ex2f(m_run[nt][x] - finite_ref(m_new));   // 0 on the first tile
          m_run[nt][x] = m_new;
          l_run[nt][x] *= alpha[x];
        }
#pragma unroll
        for (int m = 0; m < D / 16; ++m) {
          oacc[nt][m][0] *= alpha[0];
          oacc[nt][m][1] *= alpha[1];
          oacc[nt][m][2] *= alpha[0];
          oacc[nt][m][3] *= alpha[1];
        }
      }
    }
    // P^T as the B operand: the 8 x 8 blocks (keys x query rows) are transposed between the lanes
    uint32_t pb[kNT][2];
#pragma unroll
    for (int nt = 0; nt < kNT; ++nt) {
      const float m0 = finite_ref(m_run[nt][0]), m1 = finite_ref(m_run[nt][1]);
      const float p0 = ex2f(sx[nt][0] - m0), p1 = ex2f(sx[nt][1] - m1);
      const float p2 = ex2f(sx[nt][2] - m0), p3 = ex2f(sx[nt][3] - m1);
      l_run[nt][0] += p0 + p2;
      l_run[nt][1] += p1 + p3;
      pb[nt][0] = transpose_8x8(pack2(p0, p1));
      pb[nt][1] = transpose_8x8(pack2(p2, p3));
    }
    // O^T += V^T P^T : k = this warp's 16 keys, m-tiles of 16 output dims
#pragma unroll
    for (int m = 0; m < D / 16; ++m) {
      uint32_t va[4];
      ldsm_x4_trans(sv + sw_off<D>(wkey0 + (lane & 7) + (lane >> 4) * 8, 2 * m + ((lane >> 3) & 1)), va);
#pragma unroll
      for (int nt = 0; nt < kNT; ++nt) mma_bf16_16816(oacc[nt][m], va, pb[nt][0], pb[nt][1]);
    }
  }

  // ---- merge the warps through shared memory
#pragma unroll
  for (int o = 4; o < 32; o <<= 1)
#pragma unroll
    for (int nt = 0; nt < kNT; ++nt)
#pragma unroll
      for (int x = 0; x < 2; ++x) l_run[nt][x] += __shfl_xor_sync(0xffffffffu, l_run[nt][x], o);
  cp_async_wait<0>();
  __syncthreads();
  constexpr int kMS = C::kMergeStride;
  float* sc_o = reinterpret_cast<float*>(smem);               // [warps][rows][D + 4]
  float* sc_ml = sc_o + kWarps * kRows * kMS;                 // [warps][rows][2]
#pragma unroll
  for (int nt = 0; nt < kNT; ++nt) {
    const int r = warp * kRows + nt * 8 + 2 * t4;
#pragma unroll
    for (int m = 0; m < D / 16; ++m) {
      float* r0 = sc_o + r * kMS + m * 16 + quad;
      r0[0] = oacc[nt][m][0]; r0[kMS] = oacc[nt][m][1];
      r0[8] = oacc[nt][m][2]; r0[kMS + 8] = oacc[nt][m][3];
    }
    if (quad == 0) {
      sc_ml[r * 2] = m_run[nt][0];
      sc_ml[r * 2 + 1] = l_run[nt][0];
      sc_ml[r * 2 + 2] = m_run[nt][1];
      sc_ml[r * 2 + 3] = l_run[nt][1];
    }
  }
  __syncthreads();
  float* part_o = reinterpret_cast<float*>(smem) + C::kPartOff;  // [rows][D] this CTA's unnormalised rows
  float* part_ml = part_o + kRows * D;                           // [rows][2] (max, sum)
  for (int idx = tid; idx < rows_here * D; idx += kThreads) {
    const int r = idx / D, d = idx % D;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) M = fmaxf(M, sc_ml[(w * kRows + r) * 2]);
    float L = 0.f, acc = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float mw = sc_ml[(w * kRows + r) * 2];
      const float f = (mw == -INFINITY) ? 0.f : ex2f(mw - M);
      L += sc_ml[(w * kRows + r) * 2 + 1] * f;
      acc += sc_o[(w * kRows + r) * kMS + d] * f;
    }
    if (kCluster) {
      part_o[r * D + d] = acc;
      if (d == 0) {
        part_ml[2 * r] = M;
        part_ml[2 * r + 1] = L;
      }
      continue;
    }
    // L = 0: every score is -inf.  Of the whole sequence that gives NaN, as from ATen; a chunk of it has no weight.
    const float outv = (n_chunks > 1 && L == 0.f) ? 0.f : acc / L;
    const float lse2 = M + log2f(L);
    if (n_chunks == 1) {
      o_row(p, b, hkv, row0 + r)[d] = __float2bfloat16_rn(outv);
      if (d == 0 && p.lse) p.lse[lse_index(p, b, hkv, row0 + r)] = kLn2 * lse2;
    } else {
      const int64_t slot = lse_index(p, b, hkv, row0 + r) * p.n_splits + split;
      p.ws_o[slot * D + d] = outv;
      if (d == 0) p.ws_lse[slot] = lse2;
    }
  }
  if (kCluster) {
    // every CTA of the cluster merges its share of the (row, dim) outputs over all CTAs' partials,
    // eight CTAs' loads in flight at a time
    cluster_sync();
    const uint32_t ml0 = smem_u32(part_ml), o0 = smem_u32(part_o);
    for (int idx = split * kThreads + tid; idx < rows_here * D; idx += p.n_splits * kThreads) {
      const int r = idx / D, d = idx % D;
      float M = -INFINITY, L = 0.f, acc = 0.f;
      for (int c0 = 0; c0 < n_chunks; c0 += 8) {
        float m8[8], l8[8], a8[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int cc = min(c0 + c, n_chunks - 1);  // a repeated partial is given no weight below
          const uint32_t ml = cluster_map(ml0 + 8 * r, cc);
          m8[c] = cluster_ld_f32(ml);
          l8[c] = cluster_ld_f32(ml + 4);
          a8[c] = cluster_ld_f32(cluster_map(o0 + 4 * (r * D + d), cc));
        }
        float m_new = M;
#pragma unroll
        for (int c = 0; c < 8; ++c) m_new = fmaxf(m_new, m8[c]);
        const float ref = finite_ref(m_new), f0 = ex2f(M - ref);
        L *= f0;
        acc *= f0;
        M = m_new;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float f = c0 + c < n_chunks ? ex2f(m8[c] - ref) : 0.f;
          L = fmaf(l8[c], f, L);
          acc = fmaf(a8[c], f, acc);
        }
      }
      o_row(p, b, hkv, row0 + r)[d] = __float2bfloat16_rn(acc / L);
      if (d == 0 && p.lse) p.lse[lse_index(p, b, hkv, row0 + r)] = kLn2 * (M + log2f(L));
    }
    cluster_sync();  // no CTA's shared memory goes away while another still reads it
  }
}

// One CTA per (query row, sequence): weights w_c = 2^(L_c - max L), O = sum w_c O_c / sum w_c.
// D / 4 lanes hold a row's D values, four floats each, and the CTA's 512 / D lane groups take every
// (512 / D)-th chunk, so that the chunks' loads are in flight together: the kernel is a chain of
// memory latencies, length, then LSEs, then partials.
// Launched with programmatic stream serialisation: its CTAs may become resident while the split
// kernel is still draining, and wait here until that grid has completed and its writes are visible,
// so the launch latency of this second kernel hides behind the tail of the first.
template <int D>
__global__ void __launch_bounds__(kMergeThreads)
decode_merge_kernel(const DecodeParams p) {
  constexpr int kLanes = D / 4, kGroups = kMergeThreads / kLanes;
  __shared__ float4 s_acc[kGroups][kLanes];
  __shared__ float s_w[kGroups];
  grid_launch_dependents();
  grid_dependency_wait();
  const int row = blockIdx.x, b = blockIdx.y;  // row of the sequence: head * q_seq + query
  const int len = p.kv_lens ? min(max(p.kv_lens[b], 0), p.max_kv_seq) : p.max_kv_seq;
  const int n_chunks = (len + p.chunk_len - 1) / p.chunk_len;
  if (n_chunks <= 1) return;  // the split kernel already wrote the final row
  const int g = threadIdx.x / kLanes, l = threadIdx.x % kLanes, lane = threadIdx.x & 31;
  const int64_t slot0 = ((int64_t)b * p.n_head * p.q_seq + row) * p.n_splits;
  // at most 64 chunks: every warp holds all their LSEs, two per lane
  const float l0 = lane < n_chunks ? p.ws_lse[slot0 + lane] : -INFINITY;
  const float l1 = lane + 32 < n_chunks ? p.ws_lse[slot0 + lane + 32] : -INFINITY;
  float M = fmaxf(l0, l1);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
  const float w0 = ex2f(l0 - M), w1 = ex2f(l1 - M);
  float W = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int c0 = 0; c0 < n_chunks; c0 += kGroups) {  // warp-uniform trip count: the shuffle below needs every lane
    const int c = c0 + g;
    const float w = __shfl_sync(0xffffffffu, c < 32 ? w0 : w1, c & 31);
    if (c < n_chunks) {
      const float* vp = p.ws_o + (slot0 + c) * D + 4 * l;
      const float4 v = p.ws_aligned ? *reinterpret_cast<const float4*>(vp) : make_float4(vp[0], vp[1], vp[2], vp[3]);
      W += w;
      acc.x = fmaf(w, v.x, acc.x);
      acc.y = fmaf(w, v.y, acc.y);
      acc.z = fmaf(w, v.z, acc.z);
      acc.w = fmaf(w, v.w, acc.w);
    }
  }
  s_acc[g][l] = acc;
  if (l == 0) s_w[g] = W;
  __syncthreads();
  if (g == 0) {
#pragma unroll
    for (int k = 1; k < kGroups; ++k) {
      const float4 v = s_acc[k][l];
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      W += s_w[k];
    }
    const int head = row / p.q_seq, i = row - head * p.q_seq;
    __nv_bfloat16* o = p.o + b * p.os[0] + (int64_t)head * p.os[1] + i * p.os[2] + 4 * l;
    const float inv = 1.0f / W;
    o[0] = __float2bfloat16_rn(acc.x * inv);  // element stores: the decode entries promise no alignment of O
    o[1] = __float2bfloat16_rn(acc.y * inv);
    o[2] = __float2bfloat16_rn(acc.z * inv);
    o[3] = __float2bfloat16_rn(acc.w * inv);
    if (l == 0 && p.lse) p.lse[(int64_t)b * p.n_head * p.q_seq + row] = kLn2 * (M + log2f(W));
  }
}

// Two-way merge, natural-log LSE (the formula of RingAttn.lean:164-180).
__global__ void merge2_kernel(const float* o_a, const float* lse_a, const float* o_b,
                              const float* lse_b, float* o_out, float* lse_out, int64_t rows, int d) {
  const int64_t r = blockIdx.x;
  if (r >= rows) return;
  const float la = lse_a[r], lb = lse_b[r];
  const float mx = fmaxf(la, lb);
  const float L = (mx == -INFINITY) ? -INFINITY : mx + log1pf(expf(fminf(la, lb) - mx));
  const float wa = (la == -INFINITY) ? 0.f : expf(la - L), wb = (lb == -INFINITY) ? 0.f : expf(lb - L);
  for (int i = threadIdx.x; i < d; i += blockDim.x)
    o_out[r * d + i] = o_a[r * d + i] * wa + o_b[r * d + i] * wb;
  __syncthreads();
  if (threadIdx.x == 0) lse_out[r] = L;
}

template <int D, int kWarps, int kNT, bool kCluster>
cudaError_t launch_scan(const DecodeParams& p, cudaStream_t st) {
  constexpr int kSmem = DCfg<D, kWarps, kNT>::kSmemBytes;
  static std::atomic<bool> attr_set[64] = {};  // per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!attr_set[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(decode_kernel<D, kWarps, kNT, kCluster>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e == cudaSuccess && kCluster)
      e = cudaFuncSetAttribute(decode_kernel<D, kWarps, kNT, kCluster>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    attr_set[dev].store(true, std::memory_order_release);
  }
  return launch_overlapped(decode_kernel<D, kWarps, kNT, kCluster>, dim3(p.n_splits, p.n_kv_head * p.row_groups, p.batch), dim3(32 * kWarps),
                           kSmem, st, kCluster ? p.n_splits : 1, p);
}

template <int D, int kNT>
cudaError_t launch_scan_of(const DecodeParams& p, const ScanPlan& s, cudaStream_t st) {
  if (s.cluster) return s.warps == 8 ? launch_scan<D, 8, kNT, true>(p, st) : launch_scan<D, 4, kNT, true>(p, st);
  return s.warps == 8 ? launch_scan<D, 8, kNT, false>(p, st) : launch_scan<D, 4, kNT, false>(p, st);
}

template <int D>
int launch_d(DecodeParams& p, const ScanPlan& s, cudaStream_t st) {
  if (!s.covers(p.max_kv_seq)) return -TYR_ATTN_ERR_SHAPE;  // (the kernel divides by the chunk length)
  p.n_splits = s.n_splits;
  p.chunk_len = s.chunk_len;
  cudaError_t e = p.rows <= 8 ? launch_scan_of<D, 1>(p, s, st) : launch_scan_of<D, 2>(p, s, st);
  count_launch();
  if (e != cudaSuccess) return (int)e;
  if (s.needs_workspace()) {
    e = launch_overlapped(decode_merge_kernel<D>, dim3(p.n_head * p.q_seq, p.batch), dim3(kMergeThreads), 0, st, 1, p);
    count_launch();
  }
  return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

int max_splits_of(int max_splits) { return max_splits <= 0 || max_splits > kMaxWsChunks ? kMaxWsChunks : max_splits; }

}  // namespace

int decode_num_splits(int max_kv_seq, int max_splits, int* chunk_len) {
  max_splits = max_splits_of(max_splits);
  int chunk = (max_kv_seq + max_splits - 1) / max_splits;
  chunk = (chunk + kChunkUnit - 1) / kChunkUnit * kChunkUnit;
  if (chunk < kMinChunk) chunk = kMinChunk;
  if (chunk_len) *chunk_len = chunk;
  return (max_kv_seq + chunk - 1) / chunk;
}

// Chunk length of a launch that goes through the workspace.  decode_num_splits gives the most chunks the workspace is sized for;
// a launch uses longer chunks than that when it can: every CTA pays for filling its load pipeline,
// the cross-warp merge and a partial output row.
//  * A launch with at least four CTAs for every CTA slot of the device at 2048-key chunks takes
//    those (64 sequences of up to 32 K keys: 5.9 -> 6.95 TB/s against 512-key chunks).
//  * A launch of fewer than three CTAs per slot at 2048-key chunks whose lengths the host knows (one
//    shared length, or the caller's total_kv_len) takes the shortest chunks that still fit in ONE
//    wave of CTAs, all resident at once: each pays its start-up once and none waits for a slot
//    (one sequence of 32 K keys: 37.1 -> 31.3 us; 4 x 32 K: 106 -> 86 us; 8 x 8 K: 66 -> 53 us;
//    eight ragged sequences of up to 32 K, 2.8 CTAs per slot: 149 -> 134 us; 8 x 32 K, 3.5 CTAs per
//    slot, lost 4 % that way and stays with the rule below).
//  * Any other launch halves the chunks from 2048 keys down while it would have fewer than four CTAs
//    per slot (by the longest sequence's count when the lengths are only on the device: ragged
//    lengths leave about half of those with work).
int decode_launch_splits(int max_kv_seq, int max_splits, int batch, int ctas_per_seq_chunk, long long total_kv_len,
                         bool lengths_known, int* chunk_len) {
  int cap_chunk = 0;
  decode_num_splits(max_kv_seq, max_splits, &cap_chunk);
  total_kv_len = std::min<long long>(total_kv_len, (long long)batch * max_kv_seq);  // a hint, not trusted beyond the shapes
  const long long slots = 2ll * sm_count();  // two CTAs are resident per SM
  // CTAs that find work with chunks of `chunk` keys
  auto ctas = [&](int chunk) -> long long {
    if (total_kv_len > 0) return ctas_per_seq_chunk * (total_kv_len / chunk + (batch + 1) / 2);
    return (long long)ctas_per_seq_chunk * batch * ((max_kv_seq + chunk - 1) / chunk);
  };
  const int whole = (max_kv_seq + kChunkUnit - 1) / kChunkUnit * kChunkUnit;  // one chunk per sequence
  int chunk = 2048;
  if (ctas(chunk) < 4 * slots) {
    long long one_wave = 0;  // chunk length of the one-wave cut, 0 when the launch does not take it
    if (lengths_known && ctas(chunk) < 3 * slots) {
      const long long keys = total_kv_len > 0 ? total_kv_len : (long long)batch * max_kv_seq;
      long long c = (keys * ctas_per_seq_chunk + slots - 1) / slots;
      c = (c + kChunkUnit - 1) / kChunkUnit * kChunkUnit;
      c = std::min<long long>(std::max<long long>(c, kMinChunk), whole);
      while (c < whole && ctas((int)c) > slots) c += kChunkUnit;
      // short sequences, many of them: even one CTA per (sequence, KV head) is more than a wave
      if (ctas((int)c) <= slots) one_wave = c;
    }
    if (one_wave > 0) {
      chunk = (int)one_wave;
    } else {
      while (chunk > cap_chunk && ctas(chunk) < 4 * slots) chunk /= 2;
    }
  }
  if (chunk < cap_chunk) chunk = cap_chunk;  // never more chunks than the workspace holds
  *chunk_len = chunk;
  return (max_kv_seq + chunk - 1) / chunk;
}

size_t decode_workspace_bytes(int batch, int n_head, int head_dim, int max_kv_seq, int max_splits) {
  const int n = decode_num_splits(max_kv_seq, max_splits, nullptr);
  if (n <= 1) return 0;
  return (size_t)batch * n_head * n * ((size_t)head_dim + 1) * sizeof(float);
}

int launch_decode(const TyrAttnDecodeArgs& a, float scale, cudaStream_t st) {
  DecodeParams p;
  p.q = static_cast<const __nv_bfloat16*>(a.q);
  p.o = static_cast<__nv_bfloat16*>(a.o);
  p.lse = a.lse;
  p.k = static_cast<const __nv_bfloat16*>(a.k);
  p.v = static_cast<const __nv_bfloat16*>(a.v);
  p.k_ptrs = a.k_ptrs;
  p.v_ptrs = a.v_ptrs;
  p.kv_lens = a.kv_lens;
  p.kv_head_strides = a.kv_head_strides;
  p.batch = a.batch; p.n_head = a.n_head; p.n_kv_head = a.n_kv_head; p.max_kv_seq = a.max_kv_seq;
  p.q_seq = 1;
  p.rows = a.n_head / a.n_kv_head;
  p.row_groups = (p.rows + 15) / 16;
  for (int i = 0; i < 2; ++i) { p.qs[i] = a.q_stride[i]; p.os[i] = a.o_stride[i]; }
  p.qs[2] = p.os[2] = 0;
  for (int i = 0; i < 3; ++i) { p.ks[i] = a.k_stride[i]; p.vs[i] = a.v_stride[i]; }
  p.scale_log2 = scale * kLog2e;
  p.ws_o = nullptr;
  p.ws_lse = nullptr;
  p.ws_aligned = 1;
  {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -TYR_ATTN_ERR_NO_DEVICE;
    DeviceState* ds = device_state(dev);
    if (!ds) return -TYR_ATTN_ERR_NO_DEVICE;
    p.status = ds->status;
  }
  ScanPlan s;
  s.n_splits = decode_launch_splits(a.max_kv_seq, a.max_splits, a.batch, a.n_kv_head * p.row_groups,
                                    a.total_kv_len > 0 ? a.total_kv_len : 0, a.kv_lens == nullptr || a.total_kv_len > 0,
                                    &s.chunk_len);
  if (s.n_splits > 1) {  // the workspace is asked for whether or not this launch then uses it
    const size_t need = decode_workspace_bytes(a.batch, a.n_head, a.head_dim, a.max_kv_seq, a.max_splits);
    if (a.workspace == nullptr || a.workspace_bytes < need) return -TYR_ATTN_ERR_WORKSPACE;
    p.ws_o = static_cast<float*>(a.workspace);
    p.ws_lse = p.ws_o + (size_t)a.batch * a.n_head * s.n_splits * a.head_dim;
    p.ws_aligned = (reinterpret_cast<uintptr_t>(p.ws_o) & 15) == 0;
  }
  bool pays;
  const ScanPlan own = own_scan_plan(a.head_dim, (long long)a.batch * a.n_kv_head * p.row_groups, a.max_kv_seq,
                                     max_splits_of(a.max_splits), sm_count(), &pays);
  if (pays) s = own;
  if (a.head_dim == 128) return launch_d<128>(p, s, st);
  if (a.head_dim == 64) return launch_d<64>(p, s, st);
  return -TYR_ATTN_ERR_HEAD_DIM;
}

// ---- the typed call with few query rows per KV head
static ScanPlan few_rows_plan_of(const TyrAttnPrefillArgs& a, bool have_workspace) {
  const int rows = a.n_head / a.n_kv_head * a.q_seq;
  return few_rows_plan(a.head_dim, (long long)a.batch * a.n_kv_head * ((rows + 15) / 16), a.kv_seq, have_workspace, sm_count());
}

bool few_rows_call(const TyrAttnPrefillArgs& a) {
  return !a.is_causal && a.window_size == 0 && a.key_mask == nullptr && !a.check_mode && a.dtype == TYR_ATTN_BF16 &&
         (a.head_dim == 64 || a.head_dim == 128) && (long long)a.n_head / a.n_kv_head * a.q_seq <= kMaxFewRows;
}

size_t few_rows_workspace_bytes(const TyrAttnPrefillArgs& a) {
  const ScanPlan s = few_rows_plan_of(a, true);
  if (!s.needs_workspace()) return 0;
  return (size_t)a.batch * a.n_head * a.q_seq * s.n_splits * ((size_t)a.head_dim + 1) * sizeof(float);
}

int launch_few_rows(const TyrAttnPrefillArgs& a, float scale, int* status, cudaStream_t st) {
  DecodeParams p;
  p.q = static_cast<const __nv_bfloat16*>(a.q);
  p.o = static_cast<__nv_bfloat16*>(a.o);
  p.lse = a.lse;
  p.k = static_cast<const __nv_bfloat16*>(a.k);
  p.v = static_cast<const __nv_bfloat16*>(a.v);
  p.k_ptrs = p.v_ptrs = nullptr;
  p.kv_lens = nullptr;
  p.kv_head_strides = nullptr;
  p.batch = a.batch; p.n_head = a.n_head; p.n_kv_head = a.n_kv_head; p.max_kv_seq = a.kv_seq;
  p.q_seq = a.q_seq;
  p.rows = a.n_head / a.n_kv_head * a.q_seq;
  p.row_groups = (p.rows + 15) / 16;
  for (int i = 0; i < 3; ++i) { p.qs[i] = a.q_stride[i]; p.os[i] = a.o_stride[i]; p.ks[i] = a.k_stride[i]; p.vs[i] = a.v_stride[i]; }
  p.scale_log2 = scale * kLog2e;
  p.status = status;
  const size_t need = few_rows_workspace_bytes(a);
  const bool ws = a.workspace != nullptr && need > 0 && (size_t)a.workspace_bytes >= need &&
                  (reinterpret_cast<uintptr_t>(a.workspace) & 255) == 0;
  const ScanPlan s = few_rows_plan_of(a, ws);
  p.ws_o = static_cast<float*>(a.workspace);
  p.ws_lse = ws ? p.ws_o + (size_t)a.batch * a.n_head * a.q_seq * s.n_splits * a.head_dim : nullptr;
  p.ws_aligned = 1;
  return a.head_dim == 128 ? launch_d<128>(p, s, st) : launch_d<64>(p, s, st);
}

int launch_merge2(const float* o_a, const float* lse_a, const float* o_b, const float* lse_b,
                  float* o_out, float* lse_out, int64_t rows, int head_dim, cudaStream_t st) {
  if (rows > 0x7fffffffLL) return -TYR_ATTN_ERR_TOO_LARGE;
  merge2_kernel<<<(unsigned)rows, 128, 0, st>>>(o_a, lse_a, o_b, lse_b, o_out, lse_out, rows, head_dim);
  count_launch();
  return (int)cudaGetLastError();
}

}  // namespace tyr

// ---------------------------------------------------------------------------
// Decode without any allocation: the split-KV scratch lives in a fixed array
// inside the library image instead of a caller-provided workspace.
// ---------------------------------------------------------------------------
namespace tyr {
namespace {

constexpr size_t kStaticScratchBytes = TYR_ATTN_DECODE_STATIC_SCRATCH_BYTES;

// Held by every GPU that loads this library until the process exits.
static __device__ __align__(256) unsigned char g_decode_static_scratch[kStaticScratchBytes];

constexpr int kMaxStaticDevices = 64;
std::mutex g_static_mu;
void* g_static_scratch_ptr[kMaxStaticDevices] = {};  // device address of the array, per device

// In host code `g_decode_static_scratch` is only a stand-in for the symbol; the
// address a kernel can use has to be asked for, once per device, with that device current.
int static_scratch_for_current_device(void** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxStaticDevices) return -TYR_ATTN_ERR_NO_DEVICE;
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (g_static_scratch_ptr[dev] == nullptr) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_decode_static_scratch);
    if (e != cudaSuccess) return (int)e;
    if (ptr == nullptr) return -TYR_ATTN_ERR_NO_DEVICE;
    g_static_scratch_ptr[dev] = ptr;
  }
  *out = g_static_scratch_ptr[dev];
  return 0;
}

}  // namespace
}  // namespace tyr

extern "C" int tyr_b200_attn_decode_static(const TyrAttnDecodeArgs* args, void* stream) {
  using namespace tyr;
  if (args == nullptr) return -TYR_ATTN_ERR_NULL;
  if (args->batch <= 0 || args->n_head <= 0 || args->head_dim <= 0 || args->max_kv_seq <= 0)
    return -TYR_ATTN_ERR_SHAPE;
  const size_t need = decode_workspace_bytes(args->batch, args->n_head, args->head_dim,
                                             args->max_kv_seq, args->max_splits);
  if (need > kStaticScratchBytes) return -TYR_ATTN_ERR_TOO_LARGE;
  void* scratch = nullptr;
  int rc = static_scratch_for_current_device(&scratch);
  if (rc != 0) return rc;
  // Nothing in the scratch has to start at zero: the split kernel writes every
  // (row, chunk) slot the merge kernel later reads, so stale contents of an
  // earlier call are never observed.
  TyrAttnDecodeArgs a = *args;
  a.workspace = scratch;
  a.workspace_bytes = kStaticScratchBytes;
  return tyr_b200_attn_decode(&a, stream);
}
