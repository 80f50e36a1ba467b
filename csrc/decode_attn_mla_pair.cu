// Split-KV paged decode attention for MLA over a block-scaled fp8 latent cache, one cluster of two CTAs per
// piece of a sequence.  Same arithmetic as decode_attn_mla.cu (latent dequantised to bf16, fp32 scores and
// sums, bf16 probabilities), both products on the 5th-generation tensor cores.
//
// What bounds it: 278 KFLOP per token (128 heads x (576 + 512) x 2), so the tensor pipe; the fp32 output
// accumulator of all 128 heads, 128 x 512, fills the whole tensor memory of one SM, which is why a single CTA
// has to run Q K^T on the warp-level MMA pipe at a quarter of the rate.  Here the two CTAs of a cluster split
// the LATENT DIMENSIONS, not heads or tokens:
//   * CTA r owns latent dims [256 r, 256 r + 256) and rope dims [32 r, 32 r + 32): it loads and dequantises only
//     those (nothing is loaded, converted or stored twice), and one bf16 tile in shared memory is the K-major
//     operand of its part of Q K^T and, read MN-major, the V operand of its 256 output columns;
//   * tensor memory: O 128 x 256 (256 columns), Q (144 columns, the A operand of every Q K^T straight from tensor
//     memory), P (32 columns, the A operand of P V) and S (64 columns): 496 of 512, and shared memory is left to
//     four tiles of 64 tokens;
//   * a CTA's Q K^T is a partial sum over its dims: it goes to the other CTA as fp32 through distributed shared
//     memory (st.async, completion counted on the receiver's mbarrier), both add the same two numbers and run the
//     same softmax, so nothing else has to be agreed on: fp addition commutes, hence bit-identical decisions.
// Roles per CTA (17 warps): 0..7 softmax (thread = one head x 32 tokens), 8..15 dequantisation fed by register
// prefetch two tiles ahead, 16 issues the MMAs.  The MMA queue runs Q K^T two tiles ahead of P V, so the partial
// sums' way to the peer and the softmax are covered.
// Pieces of a sequence are merged by a second small kernel (mla_pair_fold_kernel) with all SMs.
// Measured against the warp-specialised single-CTA kernel (B200, one call): 32 x 32768 tokens 666 -> 606 us, 16 ragged
// sequences up to 17000 tokens 251 -> 139 us (a last-CTA fold read all pieces through one SM), 2 x 1500 tokens 121 -> 27 us.
// Every wait is bounded; on expiry the error flag is raised, tensor memory is released and the kernel returns.
#include "attention.h"

#include <algorithm>

#include "helix_common.cuh"
#include "sm100.cuh"

namespace helix {
namespace {

using namespace sm100;

constexpr int kH = 128;            // heads
constexpr int kDn = 512;           // latent dims, also the value dims
constexpr int kDr = 64;            // rope dims
constexpr int kDo = kDn / 2;       // latent dims of one CTA
constexpr int kTile = 64;          // tokens per tile
constexpr int kUnit = 16;          // tokens that are sure to share a page
constexpr int kSlots = 4;
constexpr int kSubBytes = kTile * 128;                 // [64 tokens x 64 dims] bf16, 128-byte swizzle
constexpr int kLatBytes = (kDo / 64) * kSubBytes;      // 32768
constexpr int kSlotBytes = kLatBytes + kTile * 64;     // + rope [64 tokens x 32 dims], 64-byte swizzle: 36864
constexpr int kXBytes = kH * kTile * 4;                // partial scores of a tile: 32768
constexpr int kSmem = kSlots * kSlotBytes + 2 * kXBytes + 1024;
constexpr int kSmWarps = 8, kDqWarps = 8;
constexpr int kSmThreads = kSmWarps * 32;
constexpr int kThreads = (kSmWarps + kDqWarps + 4) * 32;      // the last warpgroup only holds the issuing thread
constexpr uint32_t kColO = 0, kColQ = 256, kColP = 400, kColS = 448;
constexpr int kSeqTable = 512;
constexpr int kSmBar = 1;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleThreshold = 8.f;

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&r);
}
__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ void tmem_ld_x32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,"
      "%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]),
        "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]),
        "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st_x16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
      "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[tmem] (+)= A[tmem] * B[smem desc], A with two bf16 of the K index per 32-bit column
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, bool accumulate) {
  const uint32_t acc = accumulate ? 1u : 0u;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(acc)
      : "memory");
}
// K-major operand of 64-byte rows with the 64-byte swizzle, 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t umma_desc_k_sw64(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}
// MN-major operand stored as [K index rows][64 of the MN index], 128-byte swizzle, MN blocks `lbo_bytes` apart
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t addr, uint32_t lbo_bytes) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (uint64_t)(lbo_bytes >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)2 << 61;
}
__device__ __forceinline__ void st_async_f32x4(uint32_t addr, uint32_t bar, float2 a, float2 b) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%2,%3,%4,%5}, [%1];"
               ::"r"(addr), "r"(bar), "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y)
               : "memory");
}
__device__ __forceinline__ float4 lds_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, unsigned long long deadline_ns) {
  unsigned spins = 0;
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((++spins & 255u) == 0u && now_ns() > deadline_ns) return false;
  }
}
__device__ __forceinline__ void bar_sync_named(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ int bar_or_named(int id, int n, int pred) {
  int r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.s32 p, %3, 0;\n"
      "bar.red.or.pred q, %1, %2, p;\n"
      "selp.s32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(r)
      : "r"(id), "r"(n), "r"(pred)
      : "memory");
  return r;
}

// Two e4m3 bytes in the high bytes of the 16-bit halves of x -> the same two numbers times 2^-120 as bf16: the byte
// s.eeee.mmm moved to s.000.0eeee.mmm.0000, subnormals included.
__device__ __forceinline__ __nv_bfloat162 e4m3x2_as_bf16x2(uint32_t x) {
  const uint32_t bits = ((x >> 4) & 0x07FF07FFu) | (x & 0x80008000u);
  return *reinterpret_cast<const __nv_bfloat162*>(&bits);
}

// The tiles of all sequences form one line, sequence after sequence; cluster c takes tiles [c * chunk, (c + 1) * chunk).
// A segment is the part of one sequence inside that range; every role of both CTAs walks the same segments.
struct Segment {
  int b, seq_len, n_tiles, t_begin, count;
};
struct Walk {
  int gcur, g1, base, b;
  __device__ __forceinline__ bool next(const int* s_seq, const MlaDecodeParams& p, Segment& s) {
    while (gcur < g1 && b < p.B) {
      const int len = b < kSeqTable ? s_seq[b] : p.seq_lens[b];
      const int n = (len + kTile - 1) / kTile;
      if (len <= 0 || gcur >= base + n) {
        base += max(n, 0);
        ++b;
        continue;
      }
      s.b = b;
      s.seq_len = len;
      s.n_tiles = n;
      s.t_begin = gcur - base;
      s.count = min(n - s.t_begin, g1 - gcur);
      gcur += s.count;
      return true;
    }
    return false;
  }
};

// one tile's share of a dequantisation thread, in registers between its loads and its conversion
struct Fetch {
  uint4 lat[4], rope;
  float scl[4];
  int live;          // tokens of the tile inside the sequence; 0: no more tiles
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    mla_pair_kernel(const __grid_constant__ MlaDecodeParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t kv_full[kSlots], kv_free[kSlots], s_full, s_free, x_full[2], x_free[2], p_full, q_full, drain;
  __shared__ uint32_t tmem_slot;
  __shared__ float s_red[2][kH];
  __shared__ int s_seq[kSeqTable];
  __shared__ int s_total;

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* x_buf = smem + kSlots * kSlotBytes;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank(), peer = rank ^ 1u;
  const int cluster = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;

  if (tid == 0) {
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&kv_full[i], kDqWarps);
      mbar_init(&kv_free[i], 1);            // tcgen05.commit behind the tile's P V
    }
    mbar_init(&s_full, 1);                  // tcgen05.commit behind a tile's Q K^T
    mbar_init(&s_free, kSmWarps);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&x_full[i], 1);             // + the bytes of the peer's partial scores
      mbar_init(&x_free[i], kSmWarps);      // arrivals from the peer's softmax warps
    }
    mbar_init(&p_full, kSmWarps);
    mbar_init(&q_full, kSmWarps);
    mbar_init(&drain, 1);
    s_total = 0;
    mbar_fence_init();
  }
  if (warp == kSmWarps + kDqWarps) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  tc_fence_before_sync();
  __syncthreads();
  {
    int mine = 0;
    for (int b = tid; b < p.B; b += kThreads) {
      const int len = p.seq_lens[b];
      if (b < kSeqTable) s_seq[b] = len;
      mine += max((len + kTile - 1) / kTile, 0);
    }
    if (mine) atomicAdd(&s_total, mine);
  }
  cluster_arrive();
  cluster_wait();                           // covers the CTA too: barriers, sequence table and tile count are in place
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const unsigned long long deadline = now_ns() + p.timeout_ns;
  const int total = s_total;
  const int chunk = max((total + n_clusters - 1) / n_clusters, 1);
  Walk walk;
  walk.gcur = cluster * chunk;
  walk.g1 = min(total, walk.gcur + chunk);
  walk.base = 0;
  walk.b = 0;
  Segment seg;
  bool ok = true;
  uint32_t gt = 0;                          // tiles this CTA has been through: fixes slots, buffers and phases

  if (warp < kSmWarps) {
    // =========================== softmax ===========================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 136;");
    const int half = warp >> 2, h = 32 * (warp & 3) + lane;
    const uint32_t tq = tmem + ((uint32_t)(32 * (warp & 3)) << 16);     // this warp's lanes of the tensor memory
    const float sl2 = p.scale * kLog2e;
    const float2 sl22 = make_float2(sl2, sl2);
    // an address of this CTA's shared memory plus `to_peer` is the same place in the other CTA
    const uint32_t to_peer = map_to_cta(smem_u32(smem), peer) - smem_u32(smem);
    const uint32_t x_mine = smem_u32(x_buf) + (uint32_t)(half * 8 * kH + h) * 16u;

    while (ok && walk.next(s_seq, p, seg)) {
      const bool whole = seg.count == seg.n_tiles;
      // ---- Q of this segment into tensor memory: [head][256 latent | 32 rope] of this CTA's dims -------------
      {
        const uint8_t* qn = reinterpret_cast<const uint8_t*>(p.q_nope + ((int64_t)seg.b * kH + h) * kDn + rank * kDo);
        const uint8_t* qr = reinterpret_cast<const uint8_t*>(p.q_pe + ((int64_t)seg.b * kH + h) * kDr + rank * (kDr / 2));
        // 9 groups of 16 columns (64 bytes per head): the halves take every other one
        for (int gq = half; gq < 9; gq += 2) {
          const uint4* src = reinterpret_cast<const uint4*>(gq < 8 ? qn + gq * 64 : qr);
          uint32_t v[16];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint4 t = __ldg(src + j);
            v[4 * j] = t.x, v[4 * j + 1] = t.y, v[4 * j + 2] = t.z, v[4 * j + 3] = t.w;
          }
          tmem_st_x16(tq + kColQ + 16 * gq, v);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&q_full);
      }

      float2 cur[16], nxt[16];
      // own partial scores of tile i out of tensor memory (scaled), and on their way to the peer
      auto fetch_and_send = [&](uint32_t n, float2 (&s)[16]) {
        if (!mbar_wait(&s_full, n & 1, deadline)) ok = false;
        tc_fence_after_sync();
        uint32_t v[32];
        tmem_ld_x32(tq + kColS + 32 * half, v);
        tmem_ld_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_free);
#pragma unroll
        for (int j = 0; j < 16; ++j) s[j] = mul2(make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), sl22);
        if (tid == 0) mbar_expect_tx(&x_full[n & 1], kXBytes);
        if (n >= 2 && ok && !mbar_wait_cluster(&x_free[n & 1], ((n >> 1) - 1) & 1, deadline)) ok = false;
        if (ok) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            st_async_f32x4(x_mine + to_peer + (n & 1) * kXBytes + j * (kH * 16), smem_u32(&x_full[n & 1]) + to_peer, s[2 * j],
                           s[2 * j + 1]);
        }
      };

      float m_used = -INFINITY, l_run = 0.f;
      fetch_and_send(gt, cur);
      // A thread whose wait ran out goes on (its data is garbage) until the next vote, where all leave together.
      for (int i = 0; i < seg.count; ++i) {
        const uint32_t n = gt + i;
        if (i + 1 < seg.count) fetch_and_send(n + 1, nxt);
        if (ok && !mbar_wait(&x_full[n & 1], (n >> 1) & 1, deadline)) ok = false;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 x = lds_f32x4(x_mine + (n & 1) * kXBytes + j * (kH * 16));
          cur[2 * j] = add2(cur[2 * j], make_float2(x.x, x.y));
          cur[2 * j + 1] = add2(cur[2 * j + 1], make_float2(x.z, x.w));
        }
        __syncwarp();
        if (lane == 0 && ok) mbar_arrive_remote(smem_u32(&x_free[n & 1]) + to_peer);
        // tokens past the end of the sequence (last tile only)
        const int live = seg.seq_len - (seg.t_begin + i) * kTile - 32 * half;
        if (live < 32) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (2 * j >= live) cur[j].x = -INFINITY;
            if (2 * j + 1 >= live) cur[j].y = -INFINITY;
          }
        }
        float mx = fmaxf(cur[0].x, cur[0].y);
#pragma unroll
        for (int j = 1; j < 16; ++j) mx = fmaxf(mx, fmaxf(cur[j].x, cur[j].y));
        // The running maximum is only re-applied when some head's grew by more than 2^8, so O is rarely rescaled
        // (always at a segment's first tile, where there is nothing to rescale yet).
        if (bar_or_named(kSmBar, kSmThreads, (!ok || i == 0 || mx > m_used + kRescaleThreshold) ? 1 : 0)) {
          s_red[half][h] = mx;
          if (bar_or_named(kSmBar, kSmThreads, ok ? 0 : 1)) {
            ok = false;
            break;
          }
          mx = fmaxf(mx, s_red[half ^ 1][h]);
          float alpha = 1.f;
          if (mx > m_used + kRescaleThreshold || m_used == -INFINITY) {
            const float m_new = fmaxf(m_used, mx);
            alpha = m_used == -INFINITY ? 0.f : fast_exp2(m_used - m_new);
            l_run *= alpha;
            m_used = m_new;
          }
          if (i > 0) {
            // every P V issued so far has to be complete before O is touched
            if (!mbar_wait(&kv_free[(n - 1) % kSlots], ((n - 1) / kSlots) & 1, deadline)) ok = false;
            tc_fence_after_sync();
            for (int c0 = 0; c0 < 128; c0 += 16) {
              uint32_t v[16];
              tmem_ld_32x32b_x16(tq + kColO + 128 * half + c0, v);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * alpha);
              tmem_st_x16(tq + kColO + 128 * half + c0, v);
            }
            tmem_st_wait();
          }
          bar_sync_named(kSmBar, kSmThreads);       // s_red may be written again
        }
        const float m_neg = m_used == -INFINITY ? 0.f : -m_used;
        const float2 mn2 = make_float2(m_neg, m_neg);
        uint32_t pk[16];
        float2 sum = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float2 d = add2(cur[j], mn2);
          const float2 e = make_float2(fast_exp2(d.x), fast_exp2(d.y));
          sum = add2(sum, e);
          pk[j] = pack_bf16(e.x, e.y);
        }
        l_run += sum.x + sum.y;
        // P has one buffer: the P V of the tile before has to be complete
        if (n >= 1 && ok && !mbar_wait(&kv_free[(n - 1) % kSlots], ((n - 1) / kSlots) & 1, deadline)) ok = false;
        tc_fence_after_sync();
        tmem_st_x16(tq + kColP + 16 * half, pk);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full);
#pragma unroll
        for (int j = 0; j < 16; ++j) cur[j] = nxt[j];
      }

      // ---- O of the segment: normalise, write the result or a piece --------------------------------------
      const uint32_t nl = gt + seg.count - 1;
      if (ok && !mbar_wait(&kv_free[nl % kSlots], (nl / kSlots) & 1, deadline)) ok = false;
      if (bar_or_named(kSmBar, kSmThreads, ok ? 0 : 1)) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      s_red[half][h] = l_run;
      bar_sync_named(kSmBar, kSmThreads);
      const float L = s_red[0][h] + s_red[1][h];
      const float inv = L > 0.f ? 1.f / L : 0.f;
      const float lse2 = L > 0.f ? m_used + log2f(L) : -INFINITY;
      // slot 1: the piece that starts its sequence; a cluster holds at most one piece of each kind
      const size_t slot = (size_t)cluster * 2 + (seg.t_begin == 0 ? 1 : 0);
      const int col = (int)rank * kDo + 128 * half;
      for (int c0 = 0; c0 < 128; c0 += 16) {
        uint32_t v[16];
        tmem_ld_32x32b_x16(tq + kColO + 128 * half + c0, v);
        tmem_ld_wait();
        if (whole) {
          uint32_t o16[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) o16[j] = pack_bf16(__uint_as_float(v[2 * j]) * inv, __uint_as_float(v[2 * j + 1]) * inv);
          uint4* dst = reinterpret_cast<uint4*>(p.o + ((int64_t)seg.b * kH + h) * kDn + col + c0);
          dst[0] = make_uint4(o16[0], o16[1], o16[2], o16[3]);
          dst[1] = make_uint4(o16[4], o16[5], o16[6], o16[7]);
        } else {
          float4* dst = reinterpret_cast<float4*>(p.part_o + (slot * kH + h) * kDn + col + c0);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            dst[j] = make_float4(__uint_as_float(v[4 * j]) * inv, __uint_as_float(v[4 * j + 1]) * inv,
                                 __uint_as_float(v[4 * j + 2]) * inv, __uint_as_float(v[4 * j + 3]) * inv);
        }
      }
      if (rank == 0 && half == 0) {
        if (whole) p.lse[(int64_t)seg.b * kH + h] = p.lse_base2 ? lse2 : lse2 * kLn2;
        else p.part_lse[slot * kH + h] = lse2;
      }
      tc_fence_before_sync();
      bar_sync_named(kSmBar, kSmThreads);           // O and s_red are free for the next segment
      gt += seg.count;
    }
    if (!ok && lane == 0) atomicCAS(p.error_flag, 0, (int)kTimeoutMbarrier);
  } else if (warp < kSmWarps + kDqWarps) {
    // =========================== dequantisation ===========================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    const int w8 = warp - kSmWarps;
    // Eight consecutive lanes (one phase of a 16-byte shared-memory access) hold four chunks of an even row and the
    // four of the odd row below: their swizzled stores fall in all eight 16-byte bank groups.
    const int row_lo = 2 * w8 + ((lane & 7) >> 2);                 // row of a 16-token unit
    const int c = 4 * (lane >> 3) + (lane & 3);                    // 16-byte chunk of the fp8 half row
    const int rrow = 8 * w8 + (lane >> 2), rc = lane & 3;          // rope: row of the tile, 16-byte chunk
    const uint8_t* lat_src = p.ckv + (size_t)rank * kDo + c * 16;
    const float* scl_src = p.scales + 2 * rank + (c >> 3);
    const __nv_bfloat16* rope_src = p.kpe + rank * (kDr / 2) + rc * 8;

    // the tile whose page ids have been requested: lane u (mod 4) holds the ones of 16-token unit u
    int tile_left = 0, tile = 0, nx_page = 0, nx_in = 0, nx_live = 0;
    auto advance = [&]() {
      if (tile_left == 0) {
        if (!walk.next(s_seq, p, seg)) {
          nx_live = 0;
          return;
        }
        tile = seg.t_begin;
        tile_left = seg.count;
      }
      // a unit past the end of the sequence reads its last unit again: masked, but inside the block table
      const int tok = min(tile * kTile + (lane & 3) * kUnit, (seg.seq_len - 1) / kUnit * kUnit);
      const int pg = tok / p.page_size;
      nx_page = p.block_table[(int64_t)seg.b * p.bt_stride + pg];
      nx_in = tok - pg * p.page_size;
      nx_live = min(seg.seq_len - tile * kTile, kTile);
      ++tile;
      --tile_left;
    };
    auto load = [&](Fetch& f) {
      f.live = nx_live;
      if (nx_live == 0) return;
      const int64_t row = (int64_t)nx_page * p.page_size + nx_in;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t g = __shfl_sync(0xffffffffu, row, u) + row_lo;
        f.lat[u] = ldg_stream(lat_src + g * kDn);
        f.scl[u] = __ldg(scl_src + g * 4);
      }
      f.rope = ldg_stream(rope_src + (__shfl_sync(0xffffffffu, row, w8 >> 1) + (rrow & 15)) * kDr);
      advance();
    };
    auto convert = [&](Fetch& f) {
      uint8_t* kv = smem + (gt % kSlots) * kSlotBytes;
      if (gt >= kSlots) {
        ok = __all_sync(0xffffffffu, mbar_wait(&kv_free[gt % kSlots], (gt / kSlots - 1) & 1, deadline));
        if (!ok) return;
      }
      uint8_t* sub = kv + (c >> 2) * kSubBytes;
      const uint32_t cc = 2u * (c & 3);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = 16 * u + row_lo;
        const float sc = r < f.live ? f.scl[u] : 0.f;              // rows past the end must not leak into P V
        const uint32_t w[4] = {f.lat[u].x, f.lat[u].y, f.lat[u].z, f.lat[u].w};
        __nv_bfloat162 v[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[2 * j] = e4m3x2_as_bf16x2(__byte_perm(w[j], 0u, 0x1404));
          v[2 * j + 1] = e4m3x2_as_bf16x2(__byte_perm(w[j], 0u, 0x3424));
        }
        // times scale * 2^120, which is a finite bf16 for all but absurd scales: those take two factors
        if (fabsf(sc) < 64.f) {
          const __nv_bfloat162 k = __float2bfloat162_rn(sc * 1.329227995784916e36f);       // 2^120
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = __hmul2(v[j], k);
        } else {
          const __nv_bfloat162 k64 = __float2bfloat162_rn(1.8446744073709552e19f);         // 2^64
          const __nv_bfloat162 k = __float2bfloat162_rn(sc * 7.2057594037927936e16f);      // 2^56
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = __hmul2(__hmul2(v[j], k64), k);
        }
        const uint32_t* o = reinterpret_cast<const uint32_t*>(v);
        *reinterpret_cast<uint4*>(sub + swz128((uint32_t)r, cc)) = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4*>(sub + swz128((uint32_t)r, cc + 1)) = make_uint4(o[4], o[5], o[6], o[7]);
      }
      *reinterpret_cast<uint4*>(kv + kLatBytes + rrow * 64 + ((rc ^ ((rrow >> 1) & 3)) << 4)) = f.rope;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&kv_full[gt % kSlots]);
      ++gt;
    };
    Fetch fa, fb;
    advance();
    load(fa);
    load(fb);
    while (true) {
      if (fa.live == 0) break;
      convert(fa);
      if (!ok) break;
      load(fa);
      if (fb.live == 0) break;
      convert(fb);
      if (!ok) break;
      load(fb);
    }
    if (!ok) atomicCAS(p.error_flag, 0, (int)kTimeoutMbarrier);
  } else {
    // =========================== MMA issue ===========================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    if (warp == kSmWarps + kDqWarps && lane == 0) {
      const uint32_t id_qk = umma_idesc_bf16(kH, kTile);
      const uint32_t id_pv = umma_idesc_bf16(kH, kDo) | (1u << 16);       // B is MN-major
      uint32_t n_seg = 0;
      auto qk = [&](uint32_t n) {
        if (!mbar_wait(&kv_full[n % kSlots], (n / kSlots) & 1, deadline)) return false;
        if (n >= 1 && !mbar_wait(&s_free, (n - 1) & 1, deadline)) return false;
        tc_fence_after_sync();
        const uint32_t kv = smem_u32(smem) + (n % kSlots) * kSlotBytes;
#pragma unroll
        for (int ks = 0; ks < kDo / 16; ++ks)
          umma_bf16_ts(tmem + kColS, tmem + kColQ + ks * 8, umma_desc_k_sw128(kv + (ks >> 2) * kSubBytes + (ks & 3) * 32), id_qk, ks != 0);
#pragma unroll
        for (int ks = 0; ks < kDr / 32; ++ks)
          umma_bf16_ts(tmem + kColS, tmem + kColQ + kDo / 2 + ks * 8, umma_desc_k_sw64(kv + kLatBytes + ks * 32), id_qk, true);
        umma_commit(&s_full);
        return true;
      };
      while (ok && walk.next(s_seq, p, seg)) {
        ok = mbar_wait(&q_full, n_seg & 1, deadline);
        ++n_seg;
        if (ok) {
          tc_fence_after_sync();
          ok = qk(gt);
        }
        if (ok && seg.count > 1) ok = qk(gt + 1);
        for (int i = 0; i < seg.count && ok; ++i) {
          const uint32_t n = gt + i;
          if (i + 2 < seg.count && !qk(n + 2)) {
            ok = false;
            break;
          }
          if (!mbar_wait(&p_full, n & 1, deadline)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t kv = smem_u32(smem) + (n % kSlots) * kSlotBytes;
#pragma unroll
          for (int ks = 0; ks < kTile / 16; ++ks)
            umma_bf16_ts(tmem + kColO, tmem + kColP + ks * 8, umma_desc_mn_sw128(kv + ks * 2048, kSubBytes), id_pv, i != 0 || ks != 0);
          umma_commit(&kv_free[n % kSlots]);
        }
        gt += seg.count;
      }
      if (!ok) {
        atomicCAS(p.error_flag, 0, (int)kTimeoutMbarrier);
        umma_commit(&drain);                           // nothing of this CTA's may be in flight when it leaves
        mbar_wait(&drain, 0, now_ns() + 10000000ull);
      }
    }
  }
  // ---- leave together: neither CTA's shared memory may go while the other still writes to it --------------
  const bool failed = __syncthreads_or(ok ? 0 : 1) != 0;
  cluster_arrive();
  cluster_wait();
  if (failed) {                                      // a wait ran out: give the peer's last stores time to land
    const unsigned long long t = now_ns() + 50000ull;
    while (now_ns() < t) {
    }
  }
  cluster_arrive();
  cluster_wait();
  tc_fence_after_sync();
  if (warp == kSmWarps + kDqWarps) tmem_dealloc(tmem, 512);
}

// Merges the pieces of every sequence that more than one cluster worked on, and writes the empty sequences' zeros.
// Block (b, y) takes `heads` heads of sequence b, thread t output columns [4 t, 4 t + 4).
__global__ void __launch_bounds__(kDn / 4) mla_pair_fold_kernel(const __grid_constant__ MlaDecodeParams p, int n_clusters, int heads) {
  __shared__ int s_sum[2];
  __shared__ float s_w[kDn / 4], s_red[4];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, b = blockIdx.x;
  if (tid < 2) s_sum[tid] = 0;
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  int before = 0, all = 0;
  for (int i = tid; i < p.B; i += blockDim.x) {
    const int n = max((p.seq_lens[i] + kTile - 1) / kTile, 0);
    all += n;
    if (i < b) before += n;
  }
  if (before) atomicAdd(&s_sum[0], before);
  if (all) atomicAdd(&s_sum[1], all);
  const int n_tiles = max((p.seq_lens[b] + kTile - 1) / kTile, 0);
  __syncthreads();
  const int base = s_sum[0], chunk = max((s_sum[1] + n_clusters - 1) / n_clusters, 1);
  const int first = base / chunk, last = (base + max(n_tiles, 1) - 1) / chunk;
  if (n_tiles > 0 && first == last) return;
  for (int h = blockIdx.y * heads; h < min((int)(blockIdx.y + 1) * heads, kH); ++h) {
    uint2* dst = reinterpret_cast<uint2*>(p.o + ((int64_t)b * kH + h) * kDn) + tid;
    if (n_tiles == 0) {
      *dst = make_uint2(0u, 0u);
      if (tid == 0) p.lse[(int64_t)b * kH + h] = -INFINITY;
      continue;
    }
    // the first piece starts its sequence (slot 1); every later one begins where its cluster begins (slot 0)
    auto slot = [&](int c) { return (size_t)c * 2 + (c == first ? 1 : 0); };
    float M = -INFINITY;
    for (int c = first + lane; c <= last; c += 32) M = fmaxf(M, __ldcg(p.part_lse + slot(c) * kH + h));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float L = 0.f;
    for (int c0 = first; c0 <= last; c0 += kDn / 4) {
      const int nb = min(kDn / 4, last - c0 + 1);
      __syncthreads();
      float w = 0.f;
      if (tid < nb && M != -INFINITY) w = fast_exp2(__ldcg(p.part_lse + slot(c0 + tid) * kH + h) - M);
      s_w[tid] = w;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
      if (lane == 0) s_red[warp] = w;
      __syncthreads();
      L += s_red[0] + s_red[1] + s_red[2] + s_red[3];
#pragma unroll 8
      for (int j = 0; j < nb; ++j) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(p.part_o + (slot(c0 + j) * kH + h) * kDn) + tid);
        const float wj = s_w[j];
        acc.x += wj * v.x;
        acc.y += wj * v.y;
        acc.z += wj * v.z;
        acc.w += wj * v.w;
      }
    }
    const float inv = L > 0.f ? 1.f / L : 0.f;
    *dst = make_uint2(pack_bf16(acc.x * inv, acc.y * inv), pack_bf16(acc.z * inv, acc.w * inv));
    if (tid == 0) {
      const float lse2 = L > 0.f ? M + log2f(L) : -INFINITY;
      p.lse[(int64_t)b * kH + h] = p.lse_base2 ? lse2 : lse2 * kLn2;
    }
  }
}

}  // namespace

int mla_pair_pick_ctas(int B, int max_seq_len, int sm_count) {
  const long long tiles = (long long)std::max(B, 1) * std::max((max_seq_len + kTile - 1) / kTile, 1);
  return 2 * (int)std::min<long long>(std::max(sm_count / 2, 1), tiles);
}

cudaError_t launch_mla_decode_pair(const MlaDecodeParams& p, bool pdl, cudaStream_t stream) {
  if (p.B <= 0) return cudaSuccess;
  if (p.page_size % kUnit != 0 || p.ctas < 2 || p.ctas % 2 != 0 || p.ctas > kMlaMaxCtas) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(mla_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(p.ctas, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = pdl ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, mla_pair_kernel, p);
  if (e != cudaSuccess) return e;
  // The fold is always chained to this launch: it waits for the whole grid before it reads anything.
  const int heads = p.B >= 16 ? 8 : p.B >= 4 ? 2 : 1;
  cfg.gridDim = dim3(p.B, kH / heads, 1);
  cfg.blockDim = dim3(kDn / 4, 1, 1);
  cfg.dynamicSmemBytes = 0;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, mla_pair_fold_kernel, p, p.ctas / 2, heads);
}

}  // namespace helix
