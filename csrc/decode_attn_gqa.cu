// Split-KV paged decode attention, GQA (group <= 8 query heads per KV head, head_dim 128, bf16).
//
// Decode attention is bound by streaming the KV cache from HBM once.  The kernel is organised
// around that stream:
//   * fixed shares: the 16-token KV blocks of all (sequence, kv head) pairs form one linear index
//     space that is cut into gridDim.x equal contiguous shares (two CTAs per SM), so every CTA
//     streams the same number of bytes whatever the batch size or the sequence lengths; a share
//     may end one pair and begin the next;
//   * dynamic tail: SMs do not stream equally fast (the spread is about +-10 % and follows the SM,
//     not the data), so the last dyn_pct percent of every long pair stay out of the fixed shares
//     and form that pair's pool of small chunks.  A CTA that has finished its share draws chunks
//     with one atomic each: first from the pool of the pair it was working on - it then simply
//     keeps accumulating into the same running softmax state, no extra partial result - and, when
//     that pool is empty, from the other pools in turn (one parked partial per visited pool);
//   * every warp of a CTA owns its own 3-stage ring of KV blocks in shared memory and walks blocks
//     warp, warp + W, ... of the CTA's segment, so warps never synchronise while streaming;
//   * K and V blocks arrive by TMA tiled loads (cp.async.bulk.tensor, 128-byte swizzle, one
//     [16 x 64] box per half row) that complete on the warp's mbarrier; the paged layout is
//     handled by the tensor map (coordinates: d, token in page, kv head, page), so both
//     [pages, heads, page, d] and [pages, page, heads, d] caches work;
//   * the 8 query heads of the group form the (padded) 16-row A operand of m16n8k16 tensor-core
//     MMAs: S = Q K^T per block, online softmax in registers in the base-2 domain (the running
//     max is only re-applied when it moves), then O += P V with V fragments read by transposing
//     ldmatrix from the swizzled tile;
//   * the first loads of the next segment are issued before the epilogue of the current one;
//   * when a CTA leaves a pair, its warps' partial (max, sum, O) are merged through shared memory
//     and parked as one normalised piece in scratch memory, unless the CTA saw the whole pair;
//     a second kernel, chained by programmatic launch, folds the pieces with all SMs;
//   * short sequences (gqa_whole_pairs) are not split at all: one CTA per pair, no tables, one launch.
// Measured (B200, launches back to back in a graph): 1 x 131072 tokens 97.3 us with the fold by the pair's last CTA, 91 us
// with the fold kernel (5.9 TB/s); 1 x 300 tokens 18.6 -> 9.6 us, 16 ragged up to 500 tokens 32.7 -> 11.0 us unsplit.
// Every mbarrier wait is bounded; on expiry the kernel raises the error flag and leaves.
#include "attention.h"

#include <algorithm>
#include <climits>

#include "helix_common.cuh"
#include "sm100.cuh"

namespace helix {
namespace {

using namespace sm100;

constexpr int kD = 128;           // head dim
constexpr int kBlockTok = 16;     // tokens per KV block (one MMA k-step of P V)
constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr int kStages = 3;
constexpr int kTileBytes = kBlockTok * kD * 2;        // 4096: one K (or V) block
constexpr int kStageBytes = 2 * kTileBytes;           // K + V
constexpr int kSmemPipe = kWarps * kStages * kStageBytes;   // 98304
constexpr int kMergeBytes = kWarps * 4 * kD * 4;        // 8192: warps' partial O of four heads
constexpr int kSmemBytes = kSmemPipe + kMergeBytes + 1024;   // + alignment slack
constexpr int kMaxList = 2048;                          // pieces one fold can list
constexpr int kMaxPoolChunks = kMaxList - kGqaMaxCtas;   // chunks one pair's pool may hold: a fold lists at most one piece
                                                        // per CTA plus one per chunk of the pair
static_assert(kMaxPoolChunks > 0, "the piece list must hold one piece per CTA");
constexpr int kPlanPairs = 64;                          // up to so many pairs the fold works out by itself what to fold
constexpr int kSerialSeqs = 16;                         // batches up to this size are planned by every thread on its own
constexpr int kMinShare = 8, kWholeBlocks = 96, kWholeExtra = 40;      // 16-token blocks, see gqa_pick_ctas
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

__host__ __device__ __forceinline__ int blocks_of(int seq_len) { return (seq_len + kBlockTok - 1) / kBlockTok; }

// blocks of a pair with `nb` blocks that go to its dynamic pool (a whole number of chunks, always < nb)
__host__ __device__ __forceinline__ int dyn_chunks_of(int nb, int pct, int chunk, int min_blocks) {
  if (pct <= 0 || chunk <= 0 || nb < min_blocks) return 0;
  return (int)(((long long)nb * pct / 100) / chunk);
}

__device__ __forceinline__ int ld_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// sum over this lane and all lanes below
template <class T>
__device__ __forceinline__ T warp_scan(T v) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T below = __shfl_up_sync(0xffffffffu, v, o);
    if ((int)(threadIdx.x & 31) >= o) v += below;
  }
  return v;
}

// Chunks a pair gives to its pool, `want` being what dyn_pct asks for and hb the helper slots handed out so far.
// A pair only gets a pool if what stays in the fixed shares is longer than one share.  A CTA's share then
// never holds such a pair from its first block to its last fixed block, so the share's two piece slots
// (one for a pair it continues, one for a pair it starts) still suffice, and some share ends inside the pair, so
// a CTA is there to take up the pool.  (Two shares were the better line while one CTA folded all pieces of a pair;
// now 24 ragged sequences up to 9000 tokens, 8 kv heads, take 82.6 us with one share and 87.0 with two.)
__device__ __forceinline__ int pool_chunks(const GqaDecodeParams& p, int nb, int want, long long share_max, int hb) {
  if (nb - want * p.dyn_chunk <= share_max) return 0;
  if (hb + want * p.Hkv > p.max_helper || want > kMaxPoolChunks) return 0;    // never more chunks than helper slots
  return want;
}

// Where the pieces of one pair are: CTAs i0 .. i1 stream its fixed part, nc chunks from helper slot hb on form its pool.
struct PairPlan {
  int i0, i1, nc, hb;
};

// The fold's view of the tables the streaming kernel builds (the same rules; see there).
__device__ __forceinline__ PairPlan plan_pair(const GqaDecodeParams& p, int b, int kvh, int* s_nb, unsigned short* s_nc,
                                              long long* s_part) {
  const int tid = threadIdx.x, cd = p.dyn_chunk, G = p.ctas;
  const bool dyn_cfg = p.dyn_pct > 0 && cd > 0 && p.B <= kGqaSeqTable && p.max_helper > 0;
  if (tid < 2) s_part[tid] = 0;
  __syncthreads();
  long long all = 0, before = 0;
  for (int i = tid; i < p.B; i += blockDim.x) {
    const int nb = blocks_of(p.seq_lens[i]);
    all += nb;
    if (i < b) before += nb;
    if (dyn_cfg) {
      s_nb[i] = nb;
      s_nc[i] = (unsigned short)min(dyn_chunks_of(nb, p.dyn_pct, cd, p.dyn_min_blocks), 65535);
    }
  }
  if (before) atomicAdd(reinterpret_cast<unsigned long long*>(&s_part[0]), (unsigned long long)before);
  if (all) atomicAdd(reinterpret_cast<unsigned long long*>(&s_part[1]), (unsigned long long)all);
  __syncthreads();
  PairPlan pl{0, -1, 0, 0};
  long long start = s_part[0], total = s_part[1];
  int ns = blocks_of(p.seq_lens[b]);
  if (dyn_cfg) {
    const long long share_max = (total * p.Hkv + G - 1) / G + 1;
    long long fixed = 0;
    int hb = 0;
    for (int i = 0; i < p.B; ++i) {
      const int nb = s_nb[i], nc = pool_chunks(p, nb, s_nc[i], share_max, hb);
      if (i == b) {
        start = fixed;
        pl.nc = nc;
        pl.hb = hb + kvh * nc;
        ns = nb - nc * cd;
      }
      hb += nc * p.Hkv;
      fixed += nb - nc * cd;
    }
    total = fixed;
  }
  if (ns > 0) {
    const long long share = max((total * p.Hkv + G - 1) / (long long)G, 1LL), sp0 = start * p.Hkv + (long long)kvh * ns;
    pl.i0 = (int)(sp0 / share);
    pl.i1 = (int)((sp0 + ns - 1) / share);
  }
  return pl;
}

// Planning of a launch with many sequences: every lane takes a run of them and shuffles join the runs (all warps alike,
// warp 0 writes the tables).  When every thread walked all sequences, three times, that was a quarter of the streaming kernel
// for 128 sequences of 16 tokens (8 kv heads, a bound that keeps them in shares): 44.9 -> 34.1 us; 512 tokens 74.5 -> 63.0.
// Up to kSerialSeqs sequences the walk is as fast.  Out of line: inside the kernel it costs the launches that do not need it
// 0.2 us of instruction fetch.
struct ManyPlan {
  long long total;       // blocks in the fixed shares
  long long base;        // share-space index of the first block of sequence b, at or a few sequences before this CTA's share
  int b;
  bool pools;            // some pair has a pool
};
__device__ __noinline__ ManyPlan plan_many(const GqaDecodeParams& p, const int* s_nb, const unsigned short* s_nc,
                                           unsigned short* s_ncf, int* s_hb) {
  const int lane = threadIdx.x & 31, G = gridDim.x, Hkv = p.Hkv, n_tab = min(p.B, kGqaSeqTable);
  const int run = (n_tab + 31) / 32, lo = min(lane * run, n_tab), hi = min(lo + run, n_tab);
  long long rest = 0, total = 0;                 // sequences behind the table; all of them
  for (int b = kGqaSeqTable + lane; b < p.B; b += 32) rest += blocks_of(p.seq_lens[b]);
  for (int b = lo; b < hi; ++b) total += s_nb[b];
  rest = warp_sum(rest);
  total = warp_sum(total) + rest;
  const long long share_max = (total * Hkv + G - 1) / G + 1;
  int want = 0;
  for (int b = lo; b < hi; ++b) want += pool_chunks(p, s_nb[b], s_nc[b], share_max, 0);
  int hb = warp_scan(want) * Hkv;
  if (__shfl_sync(0xffffffffu, hb, 31) <= p.max_helper) {
    hb -= want * Hkv;
  } else {                                       // not every pair gets its chunks: who does depends on those before
    hb = 0;
    for (int b = 0; b < lo; ++b) hb += pool_chunks(p, s_nb[b], s_nc[b], share_max, hb) * Hkv;
  }
  long long fixed = 0;
  for (int b = lo; b < hi; ++b) {
    const int nb = s_nb[b], nc = pool_chunks(p, nb, s_nc[b], share_max, hb);
    if (threadIdx.x < 32) {
      s_ncf[b] = (unsigned short)nc;
      s_hb[b] = hb;
    }
    hb += nc * Hkv;
    fixed += nb - nc * p.dyn_chunk;
  }
  const long long end = warp_scan(fixed), table = __shfl_sync(0xffffffffu, end, 31);
  ManyPlan pl;
  pl.total = (table + rest) * Hkv;
  pl.pools = __shfl_sync(0xffffffffu, hb, 31) > 0;
  // the run that holds the first block of this CTA's share, or the sequences behind the table
  const long long g0 = (long long)blockIdx.x * max((pl.total + G - 1) / (long long)G, 1LL);
  const unsigned holds = __ballot_sync(0xffffffffu, g0 < end * Hkv);
  const int src = holds != 0 ? __ffs(holds) - 1 : 31;
  pl.b = holds != 0 ? __shfl_sync(0xffffffffu, lo, src) : n_tab;
  pl.base = (holds != 0 ? __shfl_sync(0xffffffffu, end - fixed, src) : table) * Hkv;
  return pl;
}

// kTrace: the instance that records time stamps (the stamps cost registers the streaming loop needs)
template <bool kTrace>
__global__ void __launch_bounds__(kThreads, 2) gqa_decode_kernel(const __grid_constant__ GqaDecodeParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kWarps][kStages];
  __shared__ float s_m[kWarps][8], s_l[kWarps][8];
  __shared__ int s_flag;                         // first pool with chunks left, while the pools are being probed
  __shared__ int s_draw[2];                      // chunk drawn ahead by thread 0 (two slots, used alternately)
  __shared__ int s_scan;                         // chunk drawn while probing the other pools
  __shared__ int s_nb[kGqaSeqTable];             // KV blocks of each sequence
  __shared__ unsigned short s_nc[kGqaSeqTable];  // chunks a pair of the sequence would give to its pool ...
  __shared__ unsigned short s_ncf[kGqaSeqTable]; // ... and what it does give, after the rules below
  __shared__ int s_hb[kGqaSeqTable];             // first helper slot of the sequence's pools

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int group = p.Hq / p.Hkv;                       // <= 8
  const int g = lane >> 2, t = lane & 3;
  const int Hq = p.Hq, Hkv = p.Hkv;
  const int G = gridDim.x;

  if (tid == 0) {
    for (int w = 0; w < kWarps; ++w)
      for (int s = 0; s < kStages; ++s) mbar_init(&full_bar[w][s], 1);
    mbar_fence_init();
    tma_prefetch_desc(&p.k_map);
    tma_prefetch_desc(&p.v_map);
  }
  const bool early_kv = p.kv_stable != 0;
  if (!early_kv) asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const unsigned long long t_entry = now_ns();
  const unsigned long long deadline = t_entry + p.timeout_ns;
  unsigned long long t_first = 0, t_static = 0, t_dyn = 0;
  unsigned n_drawn = 0, n_visits = 0;

  // ---- per-sequence tables and totals ------------------------------------------------------------
  const int cd = p.dyn_chunk;
  const bool dyn_cfg = p.dyn_pct > 0 && cd > 0 && p.B <= kGqaSeqTable && p.max_helper > 0;
  bool dyn_on = false;                           // some pair of this launch really has a pool
  const int n_tab = min(p.B, kGqaSeqTable);
  for (int i = tid; i < (p.whole ? 0 : n_tab); i += kThreads) {
    // (the divisions are done here, one sequence per thread, not in the serial pass below)
    const int nb = blocks_of(p.seq_lens[i]);
    s_nb[i] = nb;
    s_nc[i] = (unsigned short)min(dyn_cfg ? dyn_chunks_of(nb, p.dyn_pct, cd, p.dyn_min_blocks) : 0, 65535);
  }
  __syncthreads();
  long long total_s = 0;                         // blocks in the fixed shares
  int cur_b = 0;
  long long base = 0;                            // share-space index of block 0 of (cur_b, kvh = 0)
  if (p.whole) {
    // CTA = pair
  } else if (n_tab > kSerialSeqs) {
    const ManyPlan pl = plan_many(p, s_nb, s_nc, s_ncf, s_hb);
    total_s = pl.total;
    cur_b = pl.b;
    base = pl.base;
    dyn_on = pl.pools;
  } else {
    long long total = 0;
    for (int b = 0; b < n_tab; ++b) total += s_nb[b];
    const long long share_max = (total * Hkv + G - 1) / G + 1;
    int hb = 0;
    for (int b = 0; b < n_tab; ++b) {
      const int nb = s_nb[b];
      const int nc = pool_chunks(p, nb, s_nc[b], share_max, hb);
      if (tid == 0) {
        s_ncf[b] = (unsigned short)nc;
        s_hb[b] = hb;
      }
      hb += nc * Hkv;
      total_s += nb - nc * cd;
    }
    total_s *= Hkv;
    dyn_on = hb > 0;
  }
  __syncthreads();
  auto seq_nb = [&](int b) { return b < kGqaSeqTable ? s_nb[b] : blocks_of(p.seq_lens[b]); };
  auto seq_nc = [&](int b) { return (dyn_on && b < kGqaSeqTable) ? (int)s_ncf[b] : 0; };
  auto seq_ns = [&](int b) { return seq_nb(b) - seq_nc(b) * cd; };

  const long long share = max((total_s + G - 1) / (long long)G, 1LL);
  const long long g0 = (long long)blockIdx.x * share;
  const long long g1 = min(total_s, g0 + share);

  int* const pool_ctr = p.counters + (size_t)p.B * Hkv;   // [P]
  int* const helper_flag = p.counters + (size_t)2 * p.B * Hkv + 8;   // [max_helper]
  const int P = p.B * Hkv;

  uint8_t* my_smem = smem + warp * (kStages * kStageBytes);
  const float sl2 = p.scale * kLog2e;
  const int mi = lane >> 3, r8 = lane & 7;
  const uint32_t k_row = (uint32_t)(((mi >> 1) << 3) + r8), k_csel = (uint32_t)(mi & 1);
  const uint32_t v_row = (uint32_t)(((mi & 1) << 3) + r8), v_csel = (uint32_t)(mi >> 1);
  int it_ring = 0;           // TMA iterations issued so far by this warp: fixes stage and parity
  bool ok = true;

  // ---- segments: a run of blocks of one pair that this CTA streams in one go -----------------------
  struct Seg {
    int b, kvh, kb_begin, kb_end, n_blocks, seq_len;
    int slot;                // piece slot, should this segment open a new running state
    bool valid;
  };
  while (!p.whole && cur_b < p.B) {
    const long long span = (long long)seq_ns(cur_b) * Hkv;
    if (g0 < base + span) break;
    base += span;
    ++cur_b;
  }
  long long gcur = p.whole ? g1 : g0;
  auto next_static = [&]() {
    Seg sg;
    sg.valid = false;
    while (gcur < g1 && cur_b < p.B) {
      const int ns = seq_ns(cur_b);
      if (ns == 0) {
        ++cur_b;
        continue;
      }
      sg.b = cur_b;
      sg.seq_len = p.seq_lens[cur_b];
      sg.n_blocks = seq_nb(cur_b);
      sg.kvh = (int)((gcur - base) / ns);
      sg.kb_begin = (int)((gcur - base) - (long long)sg.kvh * ns);
      sg.kb_end = (int)min((long long)ns, (long long)sg.kb_begin + (g1 - gcur));
      sg.slot = blockIdx.x * 2 + (sg.kb_begin == 0 ? 1 : 0);   // slot 1: the piece that starts its pair
      sg.valid = true;
      gcur += (sg.kb_end - sg.kb_begin);
      if (sg.kvh == Hkv - 1 && sg.kb_end == ns) {   // the next segment starts the next sequence
        base += (long long)ns * Hkv;
        ++cur_b;
      }
      break;
    }
    return sg;
  };
  auto chunk_seg = [&](int b, int kvh, int c) {
    Seg sg;
    const int nc = seq_nc(b);
    sg.b = b;
    sg.kvh = kvh;
    sg.n_blocks = seq_nb(b);
    sg.seq_len = p.seq_lens[b];
    sg.kb_begin = sg.n_blocks - (nc - c) * cd;
    sg.kb_end = sg.kb_begin + cd;
    sg.slot = 2 * G + s_hb[b] + kvh * nc + c;
    sg.valid = true;
    return sg;
  };
  // Find a pool that still has chunks, starting at pair `start`, and draw one.  Uniform over the CTA.
  // one thread's look at pool start + off + tid; a stale answer is fine, a pool never refills
  auto probe = [&](int start, int off) {
    bool avail = false;
    if (off + tid < P) {
      const int q = (int)(((long long)start + off + tid) % P);
      const int nc = seq_nc(q / Hkv);
      if (nc > 0) avail = ld_relaxed(pool_ctr + q) < nc;
    }
    return avail;
  };
  // `pre`: the first window's look, taken earlier so that its round trip is over by now
  auto scan_pools = [&](int start, bool have_pre, bool pre) {
    Seg sg;
    sg.valid = false;
    int off = 0;
    while (off < P) {
      const bool avail = (have_pre && off == 0) ? pre : probe(start, off);
      have_pre = false;
      if (tid == 0) s_flag = INT_MAX;
      __syncthreads();
      if (avail) atomicMin(&s_flag, off + tid);
      __syncthreads();
      const int f = s_flag;
      if (f == INT_MAX) {
        off += kThreads;
        __syncthreads();
        continue;
      }
      const int q = (int)(((long long)start + f) % P);
      if (tid == 0) s_scan = atomicAdd(pool_ctr + q, 1);
      __syncthreads();
      const int c = s_scan;
      __syncthreads();
      if (c < seq_nc(q / Hkv)) {
        if (kTrace) ++n_visits;
        if (kTrace) ++n_drawn;
        return chunk_seg(q / Hkv, q % Hkv, c);
      }
      // somebody else took the pool's last chunk in between: it shows as empty on the next probe
    }
    return sg;
  };

  auto issue = [&](const Seg& sg, int ring, int kb, int page) {
    const int tip = (kb * kBlockTok) % p.page_size;
    uint8_t* dst = my_smem + (ring % kStages) * kStageBytes;
    uint64_t* bar = &full_bar[warp][ring % kStages];
    mbar_expect_tx(bar, kStageBytes);
    tma_load_4d(dst, &p.k_map, bar, 0, tip, sg.kvh, page);
    tma_load_4d(dst + 2048, &p.k_map, bar, 64, tip, sg.kvh, page);
    tma_load_4d(dst + kTileBytes, &p.v_map, bar, 0, tip, sg.kvh, page);
    tma_load_4d(dst + kTileBytes + 2048, &p.v_map, bar, 64, tip, sg.kvh, page);
  };
  // first loads of a segment; called while the previous segment is still being merged, so the
  // ramp of one segment hides behind the epilogue of the one before
  auto prologue = [&](const Seg& sg) {
    const int32_t* bt = p.block_table + (int64_t)sg.b * p.bt_stride;
    const int my_first = sg.kb_begin + warp;
    const int my_count = my_first < sg.kb_end ? (sg.kb_end - my_first + kWarps - 1) / kWarps : 0;
    int pg[kStages];
#pragma unroll
    for (int i = 0; i < kStages; ++i)
      pg[i] = i < my_count ? bt[((my_first + i * kWarps) * kBlockTok) / p.page_size] : 0;
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < kStages; ++i)
        if (i < my_count) issue(sg, it_ring + i, my_first + i * kWarps, pg[i]);
    }
  };

  float* s_o = reinterpret_cast<float*>(smem + kSmemPipe);   // [kWarps][4][kD]: merge buffer, not part of the rings

  Seg cur;
  if (p.whole) {                       // CTA = (sequence, kv head) pair, nothing to share out
    cur.b = blockIdx.x / Hkv;
    cur.kvh = blockIdx.x % Hkv;
    cur.seq_len = p.seq_lens[cur.b];
    cur.n_blocks = blocks_of(cur.seq_len);
    cur.kb_begin = 0;
    cur.kb_end = cur.n_blocks;
    cur.slot = 0;
    cur.valid = cur.n_blocks > 0;
  } else {
    cur = next_static();
  }
  if (early_kv) {
    // old KV does not depend on the kernel before us: request the first tiles, then wait for it (q does depend).
    // A segment that reaches the newest token waits first: that token's K/V row may still be on its way.
    const bool touches_newest = cur.valid && cur.kb_end == cur.n_blocks;
    if (touches_newest) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (cur.valid) prologue(cur);
    if (!touches_newest) asm volatile("griddepcontrol.wait;" ::: "memory");
  } else if (cur.valid) {
    prologue(cur);
  }
  int4* const start = reinterpret_cast<int4*>(p.part_lse + gqa_starts_at(G, p.max_helper)) + blockIdx.x;
  const bool note_starts = !p.whole && P > kPlanPairs;
  if (note_starts && tid == 0) start->x = -1;
  bool in_static = cur.valid;
  if (!cur.valid && dyn_on) {          // no fixed share (more CTAs than blocks): go straight to the pools
    cur = scan_pools(blockIdx.x % max(P, 1), false, false);
    if (cur.valid) prologue(cur);
  }

  // ---- running state of the pair this CTA is accumulating ------------------------------------------
  bool st_active = false;
  int st_b = 0, st_kvh = 0, st_slot = 0, st_blocks = 0, st_nb = 0;
  uint32_t qa[8][2];
  float m_run = -INFINITY, l_run = 0.f;      // for head g (quad-uniform max, per-lane partial sum)
  float o_acc[16][4];
#pragma unroll
  for (int i = 0; i < 16; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) o_acc[i][j] = 0.f;
  int dpar = 0;

  while (cur.valid) {
    const int b = cur.b, kvh = cur.kvh, seq_len = cur.seq_len;
    const int kb_begin = cur.kb_begin, kb_end = cur.kb_end;
    if (!st_active) {
      st_active = true;
      st_b = b;
      st_kvh = kvh;
      st_slot = cur.slot;
      st_blocks = 0;
      st_nb = cur.n_blocks;
      // Q fragments (A operand, rows = heads of the group, rows >= group are zero)
      const __nv_bfloat16* qrow = p.q + (int64_t)b * p.q_stride_b + (int64_t)(kvh * group + g) * p.q_stride_h;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        qa[ks][0] = 0u;
        qa[ks][1] = 0u;
        if (g < group) {
          qa[ks][0] = *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 2 * t);
          qa[ks][1] = *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 8 + 2 * t);
        }
      }
    }
    // What follows this segment?  More of the fixed share, or (when that is done) a chunk of this pair's
    // pool, drawn now so that the atomic's round trip hides behind the streaming below.
    const bool static_more = in_static && gcur < g1;
    const int my_nc = seq_nc(b);
    const bool drew = !static_more && dyn_on && my_nc > 0;
    dpar ^= 1;
    if (drew && tid == 0) s_draw[dpar] = atomicAdd(pool_ctr + (b * Hkv + kvh), 1);
    // ... and a look at the other pools, in case this one turns out to be empty
    const bool look = !static_more && dyn_on;
    const bool pre = look ? probe(b * Hkv + kvh + 1, 0) : false;

    const int32_t* bt = p.block_table + (int64_t)b * p.bt_stride;
    // page ids are looked up one iteration ahead of the TMA that needs them, so the (dependent)
    // block-table load never stalls the warp in front of a copy
    auto page_of = [&](int kb) { return bt[(kb * kBlockTok) / p.page_size]; };
    const int my_first = kb_begin + warp;
    const int my_count = my_first < kb_end ? (kb_end - my_first + kWarps - 1) / kWarps : 0;
    int next_page = kStages < my_count ? page_of(my_first + kStages * kWarps) : 0;
    if (note_starts && in_static && tid == 0 && kb_begin == 0 && kb_end < seq_ns(b)) {
      // the last pair of the share, continued by the next CTAs: the fold finds it here (the first tiles are on their way)
      *start = make_int4(b * Hkv + kvh, (int)((gcur - kb_end + seq_ns(b) - 1) / share), my_nc, my_nc > 0 ? s_hb[b] + kvh * my_nc : 0);
    }

    for (int it = 0; it < my_count; ++it) {
      const int ring = it_ring + it;
      const int stage = ring % kStages;
      const int kb = my_first + it * kWarps;
      if (!mbar_wait(&full_bar[warp][stage], (uint32_t)((ring / kStages) & 1), deadline)) {
        ok = false;
        break;
      }
      if (kTrace && t_first == 0) t_first = now_ns();
      const uint32_t kbase = smem_u32(my_smem + stage * kStageBytes);
      const uint32_t vbase = kbase + kTileBytes;

      // S = Q K^T for 16 tokens: two n-tiles of 8 tokens
      float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        const uint32_t c16 = 2u * ks + k_csel;
        uint32_t r0, r1, r2, r3;
        ldmatrix_x4(kbase + (c16 >> 3) * 2048u + swz128(k_row, c16 & 7u), r0, r1, r2, r3);
        mma_bf16_16816(s[0], qa[ks][0], 0u, qa[ks][1], 0u, r0, r1);
        mma_bf16_16816(s[1], qa[ks][0], 0u, qa[ks][1], 0u, r2, r3);
      }
      // scale, mask the tail of the sequence, online softmax (rows g of the quad)
      float mx = -INFINITY;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int tok = kb * kBlockTok + nt * 8 + 2 * t + j;
          float v = s[nt][j] * sl2;
          if (tok >= seq_len) v = -INFINITY;
          s[nt][j] = v;
          mx = fmaxf(mx, v);
        }
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      // the running max only moves when some row saw a larger score: skip the rescale otherwise
      const bool grow = __any_sync(0xffffffffu, mx > m_run);
      float alpha = 1.f;
      if (grow) {
        const float m_new = fmaxf(m_run, mx);     // finite: a block always holds >= 1 valid token
        alpha = fast_exp2(m_run - m_new);         // 0 on the first block (m_run = -inf)
        m_run = m_new;
        l_run *= alpha;
      }
      float psum = 0.f;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          s[nt][j] = fast_exp2(s[nt][j] - m_run);
          psum += s[nt][j];
        }
      l_run += psum;                              // per-lane partial; the quad is reduced at the flush
      const uint32_t pa0 = pack_bf16(s[0][0], s[0][1]);
      const uint32_t pa2 = pack_bf16(s[1][0], s[1][1]);
      // O = O * alpha + P V
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        const uint32_t c16 = 2u * jj + v_csel;
        uint32_t r0, r1, r2, r3;
        ldmatrix_x4_trans(vbase + (c16 >> 3) * 2048u + swz128(v_row, c16 & 7u), r0, r1, r2, r3);
        if (grow) {
          o_acc[2 * jj][0] *= alpha;
          o_acc[2 * jj][1] *= alpha;
          o_acc[2 * jj + 1][0] *= alpha;
          o_acc[2 * jj + 1][1] *= alpha;
        }
        mma_bf16_16816(o_acc[2 * jj], pa0, 0u, pa2, 0u, r0, r1);
        mma_bf16_16816(o_acc[2 * jj + 1], pa0, 0u, pa2, 0u, r2, r3);
      }
      // this stage is free again: fetch the block kStages iterations ahead
      __syncwarp();
      if (lane == 0 && it + kStages < my_count) issue(cur, ring + kStages, kb + kStages * kWarps, next_page);
      if (it + 1 + kStages < my_count) next_page = page_of(kb + (kStages + 1) * kWarps);
    }
    it_ring += my_count;
    st_blocks += kb_end - kb_begin;
    // The vote makes a timeout of one warp a decision of the whole CTA, so no warp is ever left
    // alone at a barrier; it also orders the next merge after the reads of the previous one and
    // publishes thread 0's drawn chunk.
    if (!__syncthreads_and(ok ? 1 : 0)) {
      ok = false;
      break;
    }
    if (kTrace) {
      if (in_static) t_static = now_ns();
      else t_dyn = now_ns();
    }
    // ---- pick the next segment and start streaming it before the epilogue of this one ---------------
    Seg nxt;
    nxt.valid = false;
    if (static_more) nxt = next_static();
    if (!nxt.valid) {
      in_static = false;
      if (dyn_on) {
        const int c = drew ? s_draw[dpar] : INT_MAX;
        if (c < my_nc) {
          nxt = chunk_seg(b, kvh, c);
          if (kTrace) ++n_drawn;
        } else {
          nxt = scan_pools(b * Hkv + kvh + 1, look, pre);
        }
      }
    }
    if (nxt.valid) prologue(nxt);

    if (!nxt.valid || nxt.b != st_b || nxt.kvh != st_kvh) {
      // ---- leave the pair: merge the warps' partials, four heads per round --------------------------
      const bool whole = (st_blocks == st_nb);
      float* part_o = p.part_o + (size_t)st_slot * 8 * kD;
      float* part_l = p.part_lse + (size_t)st_slot * 8;
      float l_quad = l_run;
      l_quad += __shfl_xor_sync(0xffffffffu, l_quad, 1);
      l_quad += __shfl_xor_sync(0xffffffffu, l_quad, 2);
      if (t == 0) {
        s_m[warp][g] = m_run;
        s_l[warp][g] = l_quad;
      }
#pragma unroll
      for (int round = 0; round < 2; ++round) {
        if (round == 1) __syncthreads();          // round 0's reads are done
        if ((g >> 2) == round) {
#pragma unroll
          for (int nt = 0; nt < 16; ++nt) {
            float2 v = make_float2(o_acc[nt][0], o_acc[nt][1]);
            *reinterpret_cast<float2*>(&s_o[(warp * 4 + (g & 3)) * kD + nt * 8 + 2 * t]) = v;
          }
        }
        __syncthreads();
        for (int idx = tid; idx < 4 * kD; idx += kThreads) {
          const int hg = round * 4 + idx / kD, d = idx % kD;
          if (hg >= group) continue;
          float M = -INFINITY;
#pragma unroll
          for (int w = 0; w < kWarps; ++w) M = fmaxf(M, s_m[w][hg]);
          float L = 0.f, O = 0.f;
          if (M != -INFINITY) {
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
              const float sc = fast_exp2(s_m[w][hg] - M);
              L += s_l[w][hg] * sc;
              O += s_o[(w * 4 + (hg & 3)) * kD + d] * sc;
            }
          }
          const float out = L > 0.f ? O / L : 0.f;
          const float lse2 = L > 0.f ? M + log2f(L) : -INFINITY;
          const int h = st_kvh * group + hg;
          if (whole) {
            p.o[((int64_t)st_b * Hq + h) * kD + d] = __float2bfloat16(out);
            if (d == 0) p.lse[(int64_t)st_b * Hq + h] = p.lse_base2 ? lse2 : lse2 * kLn2;
          } else {
            part_o[hg * kD + d] = out;
            if (d == 0) part_l[hg] = lse2;
          }
        }
      }

      // a piece parked in a helper slot is announced to the fold kernel; those of the fixed shares it knows itself
      if (!whole && tid == 0 && st_slot >= 2 * G) helper_flag[st_slot - 2 * G] = 1;
      // the running state is consumed: a fresh one starts with the next segment
      st_active = false;
      m_run = -INFINITY;
      l_run = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o_acc[i][j] = 0.f;
    }
    cur = nxt;
  }

  if (!ok) {
    if (lane == 0) atomicCAS(p.error_flag, 0, (int)kTimeoutMbarrier);
    // bounded grace period for copies that may still be in flight into this warp's ring
    const unsigned long long grace = now_ns() + 2000000ull;
    for (int s = 0; s < kStages; ++s) {
      unsigned spins = 0;
      while (!mbar_try_wait(&full_bar[warp][s], 0) && !mbar_try_wait(&full_bar[warp][s], 1)) {
        if ((++spins & 255u) == 0u && now_ns() > grace) break;
      }
    }
  }

  if (kTrace && p.trace != nullptr && tid == 0) {
    unsigned smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    unsigned long long* tr = p.trace + (size_t)blockIdx.x * 8;
    tr[0] = t_entry;
    tr[1] = t_first;
    tr[2] = t_static;
    tr[3] = now_ns();
    tr[4] = t_dyn;
    tr[5] = (unsigned long long)n_drawn | ((unsigned long long)n_visits << 32);
    tr[6] = smid;
  }

  // sequences without any token: output 0, LSE -inf (CTA 0 sweeps them)
  if (blockIdx.x == 0) {
    for (int bb = 0; bb < p.B; ++bb) {
      if (p.seq_lens[bb] > 0) continue;
      for (int idx = tid; idx < Hq * kD; idx += kThreads) {
        p.o[(int64_t)bb * Hq * kD + idx] = __float2bfloat16(0.f);
        if (idx < Hq) p.lse[(int64_t)bb * Hq + idx] = -INFINITY;
      }
    }
  }
}

// Merges the pieces of every pair that more than one CTA streamed (up to kPlanPairs pairs), one launch behind the streaming kernel: it
// is resident early (its tables are ready before the pieces are) and then has every SM to read them, where a fold by
// the CTA that finished a pair last had one SM read all of its pieces, eight per round trip, behind an acquire-release
// atomic that takes ~4 us while HBM is saturated.  Block (pair, y) merges query heads y, y + gridDim.y, ... of
// the pair's group: warps share out the pieces, lanes the columns.  The last block of a pair clears its pool and flags.
constexpr int kFoldThreads = 128;
__global__ void __launch_bounds__(kFoldThreads) gqa_fold_kernel(const __grid_constant__ GqaDecodeParams p) {
  __shared__ unsigned short s_list[kMaxList];
  __shared__ float4 s_acc[kFoldThreads / 32][32];
  __shared__ float s_max[kFoldThreads / 32], s_sum[kFoldThreads / 32];
  static_assert(kFoldThreads == 128, "four warps");
  __shared__ int s_n;
  __shared__ long long s_part[2];
  __shared__ int s_nb[kGqaSeqTable];
  __shared__ unsigned short s_nc[kGqaSeqTable];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pair = blockIdx.x, b = pair / p.Hkv, kvh = pair % p.Hkv, group = p.Hq / p.Hkv;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // seq_lens is final here: the streaming kernel waits for its predecessors before it lets this one start, or has
  // been promised that they do not touch it (kv_stable)
  const PairPlan pl = plan_pair(p, b, kvh, s_nb, s_nc, s_part);
  const int n_fixed = pl.i1 - pl.i0 + 1;
  for (int i = tid; i < n_fixed; i += kFoldThreads) s_list[i] = (unsigned short)((pl.i0 + i) * 2 + (i == 0 ? 1 : 0));
  if (tid == 0) s_n = n_fixed;
  __syncthreads();
  // Every block waits, also one without work: who waits for this launch counts on the streaming kernel being done.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (n_fixed <= 0 || (n_fixed == 1 && pl.nc == 0)) return;          // empty, or written by the CTA that saw all of it
  int* const helper_flag = p.counters + (size_t)2 * p.B * p.Hkv + 8 + pl.hb;
  for (int c = tid; c < pl.nc; c += kFoldThreads)
    if (__ldcg(helper_flag + c) != 0) s_list[atomicAdd(&s_n, 1)] = (unsigned short)(2 * p.ctas + pl.hb + c);
  __syncthreads();
  const int n = s_n;
  if (pl.nc > 0) {
    if (tid == 0) s_nb[0] = atomicAdd(p.counters + pair, 1) == (int)gridDim.y - 1;
    __syncthreads();
    if (s_nb[0]) {                              // every block of the pair has read the flags
      for (int c = tid; c < pl.nc; c += kFoldThreads) helper_flag[c] = 0;
      if (tid == 0) {
        p.counters[(size_t)p.B * p.Hkv + pair] = 0;
        p.counters[pair] = 0;
      }
    }
  }
  for (int hg = blockIdx.y; hg < group; hg += gridDim.y) {
    // Each warp takes every fourth piece, eight rows and their LSEs per round trip, with a running maximum of its own
    // (one round trip less than weights first: 1 x 32768 tokens 35.4 -> 34.3 us, 1 x 131072 90.8 -> 89.9; batches with few
    // pieces per pair are level, within 1 %).
    float M = -INFINITY, L = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i0 = warp; i0 < n; i0 += 8 * (kFoldThreads / 32)) {
      float4 v[8];
      float l[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = i0 + j * (kFoldThreads / 32);
        l[j] = -INFINITY;
        v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n) {
          const size_t row = (size_t)s_list[i] * 8 + hg;
          l[j] = __ldcg(p.part_lse + row);
          v[j] = __ldcg(reinterpret_cast<const float4*>(p.part_o + row * kD) + lane);
        }
      }
      float top = M;
#pragma unroll
      for (int j = 0; j < 8; ++j) top = fmaxf(top, l[j]);
      const float keep = M == -INFINITY ? 0.f : fast_exp2(M - top);
      M = top;
      L *= keep;
      acc = make_float4(acc.x * keep, acc.y * keep, acc.z * keep, acc.w * keep);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float w = l[j] == -INFINITY ? 0.f : fast_exp2(l[j] - top);
        L += w;
        acc.x += w * v[j].x;
        acc.y += w * v[j].y;
        acc.z += w * v[j].z;
        acc.w += w * v[j].w;
      }
    }
    s_acc[warp][lane] = acc;
    if (lane == 0) {
      s_max[warp] = M;
      s_sum[warp] = L;
    }
    __syncthreads();
    if (warp == 0) {
      M = fmaxf(fmaxf(s_max[0], s_max[1]), fmaxf(s_max[2], s_max[3]));
      L = 0.f;
      acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < kFoldThreads / 32; ++w) {
        const float f = s_max[w] == -INFINITY ? 0.f : fast_exp2(s_max[w] - M);
        const float4 v = s_acc[w][lane];
        L += f * s_sum[w];
        acc.x += f * v.x;
        acc.y += f * v.y;
        acc.z += f * v.z;
        acc.w += f * v.w;
      }
      const float inv = L > 0.f ? 1.f / L : 0.f;
      const int64_t row = (int64_t)b * p.Hq + kvh * group + hg;
      *(reinterpret_cast<uint2*>(p.o + row * kD) + lane) = make_uint2(pack_bf16(acc.x * inv, acc.y * inv), pack_bf16(acc.z * inv, acc.w * inv));
      if (lane == 0) {
        const float lse2 = L > 0.f ? M + log2f(L) : -INFINITY;
        p.lse[row] = p.lse_base2 ? lse2 : lse2 * kLn2;
      }
    }
    __syncthreads();                            // s_acc, s_max and s_sum are free again
  }
}

// The same for more than kPlanPairs pairs.  Most blocks only start when the streaming kernel is done then, and 256 to 2400
// of the blocks above took 8 to 30 us to find out what little there is to fold.  Block (c, y) reads what CTA c noted about
// the one split pair that its share starts: every split pair starts in exactly one CTA.  Up to eight pieces are one round
// trip, so each warp takes a head of its own.  From the end of the streaming kernel to the end of the fold: 128 x 16 tokens
// 22.5 -> 1.6 us, 128 x 2000 17.6 -> 3.9, 24 ragged up to 9000 5.2 -> 4.5.  Up to 64 pairs the kernel above is ahead by 0.5 to
// 1.5 us: its plan is ready before the pieces are, and the note is one more round trip.
constexpr int kFoldWarps = kFoldThreads / 32, kFoldBatch = 8;
__global__ void __launch_bounds__(kFoldThreads) gqa_fold_starts_kernel(const __grid_constant__ GqaDecodeParams p) {
  struct Sum {
    float M, L;
    float4 acc;
  };
  __shared__ unsigned short s_list[kMaxList];
  __shared__ Sum s_sum[kFoldWarps][32];
  __shared__ int s_n, s_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, group = p.Hq / p.Hkv;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int4 start = __ldcg(reinterpret_cast<const int4*>(p.part_lse + gqa_starts_at(p.ctas, p.max_helper)) + blockIdx.x);
  if (start.x < 0) return;
  const int pair = start.x, n_fixed = start.y - (int)blockIdx.x + 1, nc = start.z, hb = start.w;
  for (int i = tid; i < n_fixed; i += kFoldThreads) s_list[i] = (unsigned short)((blockIdx.x + i) * 2 + (i == 0 ? 1 : 0));
  if (tid == 0) s_n = n_fixed;
  __syncthreads();
  if (nc > 0) {
    int* const helper_flag = p.counters + (size_t)2 * p.B * p.Hkv + 8 + hb;
    for (int c = tid; c < nc; c += kFoldThreads)
      if (__ldcg(helper_flag + c) != 0) s_list[atomicAdd(&s_n, 1)] = (unsigned short)(2 * p.ctas + hb + c);
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(p.counters + pair, 1) == (int)gridDim.y - 1;
    __syncthreads();
    if (s_last) {                               // every block of the pair has read the flags
      for (int c = tid; c < nc; c += kFoldThreads) helper_flag[c] = 0;
      if (tid == 0) {
        p.counters[(size_t)p.B * p.Hkv + pair] = 0;
        p.counters[pair] = 0;
      }
    }
  }
  const int n = s_n, b = pair / p.Hkv, kvh = pair % p.Hkv;
  auto store = [&](const Sum& f, int hg) {
    const float inv = f.L > 0.f ? 1.f / f.L : 0.f;
    const int64_t row = (int64_t)b * p.Hq + kvh * group + hg;
    *(reinterpret_cast<uint2*>(p.o + row * kD) + lane) =
        make_uint2(pack_bf16(f.acc.x * inv, f.acc.y * inv), pack_bf16(f.acc.z * inv, f.acc.w * inv));
    if (lane == 0) {
      const float lse2 = f.L > 0.f ? f.M + log2f(f.L) : -INFINITY;
      p.lse[row] = p.lse_base2 ? lse2 : lse2 * kLn2;
    }
  };
  // the pieces i0, i0 + step, ... of one head, kFoldBatch rows and their LSEs per round trip, with a running maximum
  auto rows = [&](int i0, int step, int hg) {
    float M = -INFINITY, L = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (; i0 < n; i0 += kFoldBatch * step) {
      float4 v[kFoldBatch];
      float l[kFoldBatch];
#pragma unroll
      for (int j = 0; j < kFoldBatch; ++j) {
        const int i = i0 + j * step;
        l[j] = -INFINITY;
        v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n) {
          const size_t row = (size_t)s_list[i] * 8 + hg;
          l[j] = __ldcg(p.part_lse + row);
          v[j] = __ldcg(reinterpret_cast<const float4*>(p.part_o + row * kD) + lane);
        }
      }
      float top = M;
#pragma unroll
      for (int j = 0; j < kFoldBatch; ++j) top = fmaxf(top, l[j]);
      const float keep = M == -INFINITY ? 0.f : fast_exp2(M - top);
      M = top;
      L *= keep;
      acc = make_float4(acc.x * keep, acc.y * keep, acc.z * keep, acc.w * keep);
#pragma unroll
      for (int j = 0; j < kFoldBatch; ++j) {
        const float w = l[j] == -INFINITY ? 0.f : fast_exp2(l[j] - top);
        L += w;
        acc.x += w * v[j].x;
        acc.y += w * v[j].y;
        acc.z += w * v[j].z;
        acc.w += w * v[j].w;
      }
    }
    return Sum{M, L, acc};
  };
  if (n <= kFoldBatch) {
    for (int hg = blockIdx.y * kFoldWarps + warp; hg < group; hg += gridDim.y * kFoldWarps) store(rows(0, 1, hg), hg);
    return;
  }
  for (int hg = blockIdx.y; hg < group; hg += gridDim.y) {
    s_sum[warp][lane] = rows(warp, kFoldWarps, hg);
    __syncthreads();
    if (warp == 0) {
      Sum f = s_sum[0][lane];
      for (int w = 1; w < kFoldWarps; ++w) {
        const Sum s = s_sum[w][lane];
        const float top = fmaxf(f.M, s.M);
        const float x = f.M == -INFINITY ? 0.f : fast_exp2(f.M - top), y = s.M == -INFINITY ? 0.f : fast_exp2(s.M - top);
        f.M = top;
        f.L = f.L * x + s.L * y;
        f.acc = make_float4(f.acc.x * x + s.acc.x * y, f.acc.y * x + s.acc.y * y, f.acc.z * x + s.acc.z * y, f.acc.w * x + s.acc.w * y);
      }
      store(f, hg);
    }
    __syncthreads();                            // s_sum is free again
  }
}

}  // namespace

// Number of CTAs for a launch: two per SM, but never so many that a CTA streams fewer than 8 blocks (two per warp).
// With 32 blocks as the limit one sequence of 4000 tokens (8 kv heads) took 19.6 us and four of up to 1000 took
// 21.6 us; with about 128 CTAs each 17.3 and 15.9 us.  Not the best choice everywhere: one sequence of 700 tokens takes 14.5 us
// with the 44 CTAs it gets and 10.6 with 296, and 8 x 1536 tokens take 21.5 where 192 CTAs of 32 blocks took 19.
int gqa_pick_ctas(int B, int Hkv, int max_seq_len, int sm_count) {
  const long long blocks = (long long)std::max(B, 1) * Hkv * std::max((max_seq_len + kBlockTok - 1) / kBlockTok, 1);
  long long ctas = std::min<long long>(2LL * sm_count, std::max<long long>(blocks / kMinShare, 1));
  return (int)std::min<long long>(ctas, kGqaMaxCtas);
}

// One CTA per pair costs the longest sequence's blocks, a quarter per warp at about 0.35 us each; shares cost their
// own length the same way and a fold (about 4 us with its launch).  So pairs stay whole while the longest one is no
// more than kWholeExtra blocks longer than a share would be, and not so long that ragged batches are left with a tail.
bool gqa_whole_pairs(int B, int Hkv, int max_seq_len, int sm_count) {
  const long long blocks = blocks_of(std::max(max_seq_len, 1)), slots = 2LL * sm_count;
  const long long pairs = std::min((long long)std::max(B, 1) * Hkv, slots);
  return blocks <= kWholeBlocks && blocks * (slots - pairs) <= kWholeExtra * slots;
}

void gqa_plan_dynamic(GqaDecodeParams* p, int max_seq_len, int max_helper, int pct_override, int chunk_override) {
  const int nb = std::max(blocks_of(std::max(max_seq_len, 1)), 1);
  const long long blocks = (long long)std::max(p->B, 1) * p->Hkv * nb;
  p->max_helper = std::min(std::max(max_helper, 0), kGqaMaxHelper);
  p->dyn_min_blocks = 64;
  // a dynamic tail only pays when a CTA's fixed share is long compared with a chunk
  int pct = (blocks / std::max(p->ctas, 1) >= 96 && p->B <= kGqaSeqTable) ? 30 : 0;
  if (pct_override >= 0) pct = std::min(pct_override, 50);
  int chunk = chunk_override > 0 ? chunk_override : 20;   // a chunk has a fixed cost (its first loads only start once it is drawn): 16-24 blocks measured best
  if (pct > 0 && p->max_helper > 0) {
    // never more chunks than helper slots, whatever the sequence lengths turn out to be
    const long long worst = (long long)p->B * p->Hkv * ((long long)nb * pct / 100);
    while ((worst + chunk - 1) / chunk > p->max_helper) chunk += 4;
  } else {
    pct = 0;
  }
  p->dyn_pct = pct;
  p->dyn_chunk = chunk;
}

cudaError_t launch_gqa_decode(const GqaDecodeParams& p, bool pdl, cudaStream_t stream) {
  if (p.B <= 0) return cudaSuccess;
  if (p.Hq % p.Hkv != 0 || p.Hq / p.Hkv > 8 || p.page_size % kBlockTok != 0 || p.ctas < 1 || p.ctas > kGqaMaxCtas ||
      p.max_helper < 0 || p.max_helper > kGqaMaxHelper || p.dyn_pct < 0 || p.dyn_pct > 50 ||
      (p.trace != nullptr && gqa_grid(p) > p.trace_rows))
    return cudaErrorInvalidValue;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gqa_decode_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(gqa_decode_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    if (dev < 64) attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(gqa_grid(p), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = pdl ? 1 : 0;
  cudaError_t e = p.trace != nullptr ? cudaLaunchKernelEx(&cfg, gqa_decode_kernel<true>, p)
                                     : cudaLaunchKernelEx(&cfg, gqa_decode_kernel<false>, p);
  if (e != cudaSuccess || p.whole) return e;
  // The fold is always chained to this launch; it waits for the whole grid before it reads a piece.
  const int pairs = p.B * p.Hkv, blocks = pairs <= kPlanPairs ? pairs : p.ctas;
  cfg.gridDim = dim3(blocks, std::max(1, std::min(p.Hq / p.Hkv, 1184 / blocks)), 1);
  cfg.blockDim = dim3(kFoldThreads, 1, 1);
  cfg.dynamicSmemBytes = 0;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, pairs <= kPlanPairs ? gqa_fold_kernel : gqa_fold_starts_kernel, p);
}

}  // namespace helix
