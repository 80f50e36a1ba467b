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
//   * a CTA's Q K^T is a partial sum over its dims.  CTA r finishes the 64 heads [64 r, 64 r + 64): it receives the other
//     CTA's fp32 partial scores of these through distributed shared memory (st.async, completion counted on the
//     receiver's mbarrier), runs their softmax and returns the bf16 probabilities (and the factor by which O has to
//     shrink, 1 almost always), which the other CTA puts next to its own as the A operand of its P V.
// Roles per CTA (20 warps): warp 0 issues the MMAs (the oldest warp, so that busier ones do not keep it waiting; the
// whole warp walks the loop and one lane issues, which lets the operands stay in uniform registers); warps 4..7 and 8..11
// are two groups that take tiles in turn (thread = one head; two warps of a group finish this CTA's heads, two forward
// the others), so that one group's way to the peer and back is covered by the other's arithmetic; warps 12..19
// dequantise, fed by register prefetch one tile ahead.  The MMA queue runs Q K^T two tiles ahead of P V.
// Pieces of a sequence are merged by a second small kernel (mla_pair_fold_kernel) with all SMs.
// Measured against the warp-specialised single-CTA kernel (B200, one call): 32 x 32768 tokens 661 -> 416 us, 16 ragged
// sequences up to 17000 tokens 252 -> 84 us (a last-CTA fold read all pieces through one SM), 2 x 1500 tokens 121 -> 26 us.
// Behind it by up to 1.4x: 128 sequences and more of one to four tiles each when the bound given for their lengths is far
// larger (600 x 16 tokens 146 against 180 us), because a cluster takes them one after the other at ~18 us each; with
// their real bound the single-CTA kernel takes 339.
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
constexpr int kHo = kH / 2;                            // heads that one CTA finishes
constexpr int kXBytes = kHo * kTile * 4;               // their partial scores of a tile from the peer: 16384
constexpr int kPxBytes = kHo * kTile * 2;              // the peer's probabilities of the other heads: 8192
constexpr int kSmem = kSlots * kSlotBytes + 2 * kXBytes + 2 * kPxBytes + 1024;
constexpr int kGroupWarps = 4, kSmWarps = 2 * kGroupWarps, kDqWarps = 8;
constexpr int kSmThreads = kSmWarps * 32;
constexpr int kFirstSm = 4, kFirstDq = kFirstSm + kSmWarps;  // warps 1..3 only fill the issuing warp's warpgroup
constexpr int kThreads = (kFirstDq + kDqWarps) * 32;
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
__device__ __forceinline__ void tmem_st_x32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
      "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
      "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
      "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]),
      "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[tmem] (+)= A[tmem] * B[smem desc], A with two bf16 of the K index per 32-bit column; issued by one lane.  The
// descriptor comes as two words: only the lower one, with the address, differs between calls.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t desc_lo, uint32_t desc_hi, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .b64 d;\n\t"
      "mov.b64 d, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d, %4, 1;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "r"(desc_lo), "r"(desc_hi), "r"(idesc)
      : "memory");
}
__device__ __forceinline__ void umma_bf16_ts_first(uint32_t tmem_d, uint32_t tmem_a, uint32_t desc_lo, uint32_t desc_hi, uint32_t idesc,
                                                   uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .b64 d;\n\t.reg .pred p;\n\t"
      "mov.b64 d, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d, %4, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "r"(desc_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// one lane of a warp that has come here together, always the same
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e != 0;
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
__device__ __forceinline__ void st_async_u32x4(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2,%3,%4,%5}, [%1];"
               ::"r"(addr), "r"(bar), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}
__device__ __forceinline__ void st_async_f32(uint32_t addr, uint32_t bar, float v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %2, [%1];" ::"r"(addr), "r"(bar), "f"(v) : "memory");
}
__device__ __forceinline__ uint4 lds_u32x4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 lds_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
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

// Four e4m3 bytes -> the same numbers times 2^-120 as bf16: a byte s.eeee.mmm moved to s.000.0eeee.mmm.0000 IS that
// bf16, subnormals included.  Bytes 0 and 2 land in the first word, 1 and 3 in the second (fewer moves than neighbours
// together); dims 4 i + 1 and 4 i + 2 therefore change places in the tile, in Q on its way to tensor memory (swap_mid)
// and back again where O is read out.
__device__ __forceinline__ void e4m3x4_as_bf16x4(uint32_t w, __nv_bfloat162& even, __nv_bfloat162& odd) {
  const uint32_t e = ((w << 4) & 0x07F007F0u) | ((w << 8) & 0x80008000u);
  const uint32_t o = ((w >> 4) & 0x07F007F0u) | (w & 0x80008000u);
  even = *reinterpret_cast<const __nv_bfloat162*>(&e);
  odd = *reinterpret_cast<const __nv_bfloat162*>(&o);
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
  __shared__ __align__(8) uint64_t kv_full[kSlots], kv_free[kSlots], s_full[2], s_free, x_full[2], px_full[2], inv_full, p_full, q_full, m_bar[kGroupWarps], drain;
  __shared__ uint32_t tmem_slot;
  __shared__ float s_m[kH], s_l[2][kH], s_alpha[2][kHo], s_inv[kHo];
  __shared__ int s_seq[kSeqTable];
  __shared__ int s_total;

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* x_buf = smem + kSlots * kSlotBytes;
  uint8_t* px_buf = x_buf + 2 * kXBytes;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank(), peer = rank ^ 1u;
  const int cluster = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;

  if (tid == 0) {
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&kv_full[i], kDqWarps);
      mbar_init(&kv_free[i], 1);            // tcgen05.commit behind the tile's P V
    }
    mbar_init(&s_free, kGroupWarps);
    for (int i = 0; i < 2; ++i) {           // one set per softmax group: a wait must never be two phases ahead
      mbar_init(&s_full[i], 1);             // tcgen05.commit behind a tile's Q K^T
      mbar_init(&x_full[i], 1);             // + the bytes of the peer's partial scores
      mbar_init(&px_full[i], 1);            // + the bytes of the peer's probabilities and factors
    }
    for (int i = 0; i < kGroupWarps; ++i) mbar_init(&m_bar[i], 1);
    mbar_init(&inv_full, 1);                // + the bytes of the peer's 1 / sum, once per segment
    mbar_init(&p_full, kGroupWarps);
    mbar_init(&q_full, kSmWarps);
    mbar_init(&drain, 1);
    s_total = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
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

  if (warp >= kFirstSm && warp < kFirstDq) {
    // =========================== softmax ===========================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 152;");
    const int quad = warp & 3, h = 32 * quad + lane;
    const uint32_t grp = (uint32_t)(warp - kFirstSm) / kGroupWarps;     // this group takes tiles n with n % 2 == grp
    const uint32_t tq = tmem + ((uint32_t)(32 * quad) << 16);           // this warp's lanes of the tensor memory
    const float sl2 = p.scale * kLog2e;
    const float2 sl22 = make_float2(sl2, sl2);
    // an address of this CTA's shared memory plus `to_peer` is the same place in the other CTA
    const uint32_t to_peer = map_to_cta(smem_u32(smem), peer) - smem_u32(smem);
    const bool mine = (uint32_t)(quad >> 1) == rank;                    // this CTA finishes these heads
    const uint32_t hh = (uint32_t)h & (kHo - 1);
    const uint32_t x_row = smem_u32(x_buf) + grp * kXBytes + hh * 16u, px_row = smem_u32(px_buf) + grp * kPxBytes + hh * 16u;
    uint32_t n_seg = 0;

    while (ok && walk.next(s_seq, p, seg)) {
      const bool whole = seg.count == seg.n_tiles;
      // ---- Q of this segment into tensor memory: [head][256 latent | 32 rope] of this CTA's dims -------------
      {
        const uint8_t* qn = reinterpret_cast<const uint8_t*>(p.q_nope + ((int64_t)seg.b * kH + h) * kDn + rank * kDo);
        const uint8_t* qr = reinterpret_cast<const uint8_t*>(p.q_pe + ((int64_t)seg.b * kH + h) * kDr + rank * (kDr / 2));
        // 9 pieces of 16 columns (64 bytes per head): the groups take every other one
        for (int gq = grp; gq < 9; gq += 2) {
          const uint4* src = reinterpret_cast<const uint4*>(gq < 8 ? qn + gq * 64 : qr);
          uint32_t v[16];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint4 t = __ldg(src + j);
            v[4 * j] = t.x, v[4 * j + 1] = t.y, v[4 * j + 2] = t.z, v[4 * j + 3] = t.w;
          }
          if (gq < 8) {
#pragma unroll
            for (int j = 0; j < 16; j += 2) {            // dims 4 i + 1 and 4 i + 2 change places, as in the tile
              const uint32_t lo = v[j], hi = v[j + 1];
              v[j] = __byte_perm(lo, hi, 0x5410);
              v[j + 1] = __byte_perm(lo, hi, 0x7632);
            }
          }
          tmem_st_x16(tq + kColQ + 16 * gq, v);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&q_full);
      }

      // The maximum in use is per head and shared by the groups through s_m: whoever takes tile n picks it up after
      // tile n - 1 has been through (m_bar) and passes it on.  m_mine is the one that l_run refers to.
      // No credits are needed: the scores of tile n + 2 are sent by a warp that has the probabilities of tile n complete,
      // which were sent after the scores of tile n had been read; and the other way round.
      float m_mine = -INFINITY, l_run = 0.f;
      for (int i = (int)((gt ^ grp) & 1u); i < seg.count; i += 2) {
        const uint32_t n = gt + i, use = n >> 1;         // `use`: how often this group's exchange buffers have been used
        // partial scores out of tensor memory, scaled
        if (!mbar_wait(&s_full[grp], use & 1, deadline)) ok = false;
        tc_fence_after_sync();
        float2 s[32];
        {
          uint32_t v[2][32];
          tmem_ld_x32(tq + kColS, v[0]);
          tmem_ld_x32(tq + kColS + 32, v[1]);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j)
            s[j] = mul2(make_float2(__uint_as_float(v[j >> 4][2 * (j & 15)]), __uint_as_float(v[j >> 4][2 * (j & 15) + 1])), sl22);
        }
        if (!mine && ok) {                               // on their way first: the peer waits for them
#pragma unroll
          for (int j = 0; j < 16; ++j)
            st_async_f32x4(x_row + to_peer + j * (kHo * 16), smem_u32(&x_full[grp]) + to_peer, s[2 * j], s[2 * j + 1]);
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_free);
        uint32_t pk[32];
        float alpha = 1.f;
        if (mine) {
          if ((quad & 1) == 0 && lane == 0) mbar_expect_tx(&x_full[grp], kXBytes);
          if (!mbar_wait(&x_full[grp], use & 1, deadline)) ok = false;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float4 x = lds_f32x4(x_row + j * (kHo * 16));
            s[2 * j] = add2(s[2 * j], make_float2(x.x, x.y));
            s[2 * j + 1] = add2(s[2 * j + 1], make_float2(x.z, x.w));
          }
          // tokens past the end of the sequence (last tile only)
          const int live = seg.seq_len - (seg.t_begin + i) * kTile;
          if (live < kTile) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              if (2 * j >= live) s[j].x = -INFINITY;
              if (2 * j + 1 >= live) s[j].y = -INFINITY;
            }
          }
          float mx[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) mx[j] = fmaxf(s[j].x, s[j].y);
#pragma unroll
          for (int j = 4; j < 32; ++j) mx[j & 3] = fmaxf(mx[j & 3], fmaxf(s[j].x, s[j].y));
          const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
          // The maximum is only moved when a head's grew by more than 2^8, so O is rarely rescaled
          // (always at a segment's first tile, where there is nothing to rescale yet).
          if (n >= 1 && !mbar_wait(&m_bar[quad], (n - 1) & 1, deadline)) ok = false;
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          const float m = i == 0 ? -INFINITY : s_m[h];
          const bool move = top > m + kRescaleThreshold || m == -INFINITY;
          const float m_new = move ? fmaxf(m, top) : m;
          if (move) {
            s_m[h] = m_new;
            alpha = m == -INFINITY ? 0.f : fast_exp2(m - m_new);
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&m_bar[quad]);
          st_async_f32(smem_u32(&s_alpha[grp][hh]) + to_peer, smem_u32(&px_full[grp]) + to_peer, alpha);
          if (m_new != m_mine) {
            l_run = m_mine == -INFINITY ? 0.f : l_run * fast_exp2(m_mine - m_new);
            m_mine = m_new;
          }
          const float m_neg = m_new == -INFINITY ? 0.f : -m_new;
          const float2 mn2 = make_float2(m_neg, m_neg);
          float2 sum = make_float2(0.f, 0.f);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float2 d = add2(s[j], mn2);
            const float2 e = make_float2(fast_exp2(d.x), fast_exp2(d.y));
            sum = add2(sum, e);
            pk[j] = pack_bf16(e.x, e.y);
            if ((j & 3) == 3)
              st_async_u32x4(px_row + to_peer + (j >> 2) * (kHo * 16), smem_u32(&px_full[grp]) + to_peer, pk[j - 3], pk[j - 2],
                             pk[j - 1], pk[j]);
          }
          l_run += sum.x + sum.y;
        } else {
          if ((quad & 1) == 0 && lane == 0) mbar_expect_tx(&px_full[grp], kPxBytes + kHo * 4);
          if (!mbar_wait(&px_full[grp], use & 1, deadline)) ok = false;
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          alpha = s_alpha[grp][hh];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint4 v = lds_u32x4(px_row + j * (kHo * 16));
            pk[4 * j] = v.x, pk[4 * j + 1] = v.y, pk[4 * j + 2] = v.z, pk[4 * j + 3] = v.w;
          }
        }
        // P has one buffer, and O may only be touched between P V products: the one of the tile before is complete
        if (n >= 1) ok = __all_sync(0xffffffffu, mbar_wait(&kv_free[(n - 1) % kSlots], ((n - 1) / kSlots) & 1, deadline));
        if (!ok) break;
        tc_fence_after_sync();
        if (i > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
          for (int c0 = 0; c0 < kDo; c0 += 16) {
            uint32_t v[16];
            tmem_ld_32x32b_x16(tq + kColO + c0, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * alpha);
            tmem_st_x16(tq + kColO + c0, v);
          }
        }
        tmem_st_x32(tq + kColP, pk);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full);
      }

      // ---- O of the segment: normalise, write the result or a piece --------------------------------------
      const uint32_t nl = gt + seg.count - 1;
      if (ok && !mbar_wait(&kv_free[nl % kSlots], (nl / kSlots) & 1, deadline)) ok = false;
      if (bar_or_named(kSmBar, kSmThreads, ok ? 0 : 1)) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      float inv, lse2 = 0.f;
      if (mine) {
        const float m_used = s_m[h];
        s_l[grp][h] = m_mine == -INFINITY ? 0.f : l_run * fast_exp2(m_mine - m_used);
        bar_sync_named(kSmBar, kSmThreads);
        const float L = s_l[0][h] + s_l[1][h];
        inv = L > 0.f ? 1.f / L : 0.f;
        lse2 = L > 0.f ? m_used + log2f(L) : -INFINITY;
        if (grp == 0) st_async_f32(smem_u32(&s_inv[hh]) + to_peer, smem_u32(&inv_full) + to_peer, inv);
      } else {
        if (grp == 0 && (quad & 1) == 0 && lane == 0) mbar_expect_tx(&inv_full, kHo * 4);
        bar_sync_named(kSmBar, kSmThreads);
        if (!mbar_wait(&inv_full, n_seg & 1, deadline)) ok = false;      // the vote at the end of the segment acts on it
        inv = s_inv[hh];
      }
      ++n_seg;
      // slot 1: the piece that starts its sequence; a cluster holds at most one piece of each kind
      const size_t slot = (size_t)cluster * 2 + (seg.t_begin == 0 ? 1 : 0);
      const int col = (int)rank * kDo + 128 * grp;
      for (int c0 = 0; c0 < 128; c0 += 16) {
        uint32_t v[16];
        tmem_ld_32x32b_x16(tq + kColO + 128 * grp + c0, v);
        tmem_ld_wait();
        float o[16];
#pragma unroll
        for (int j = 0; j < 16; ++j)                     // columns 4 i + 1 and 4 i + 2 change places again
          o[j] = __uint_as_float(v[(j & 3) == 1 ? j + 1 : (j & 3) == 2 ? j - 1 : j]) * inv;
        if (whole) {
          uint4* dst = reinterpret_cast<uint4*>(p.o + ((int64_t)seg.b * kH + h) * kDn + col + c0);
#pragma unroll
          for (int j = 0; j < 2; ++j)
            dst[j] = make_uint4(pack_bf16(o[8 * j], o[8 * j + 1]), pack_bf16(o[8 * j + 2], o[8 * j + 3]),
                                pack_bf16(o[8 * j + 4], o[8 * j + 5]), pack_bf16(o[8 * j + 6], o[8 * j + 7]));
        } else {
          float4* dst = reinterpret_cast<float4*>(p.part_o + (slot * kH + h) * kDn + col + c0);
#pragma unroll
          for (int j = 0; j < 4; ++j) dst[j] = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        }
      }
      if (mine && grp == 0) {
        if (whole) p.lse[(int64_t)seg.b * kH + h] = p.lse_base2 ? lse2 : lse2 * kLn2;
        else p.part_lse[slot * kH + h] = lse2;
      }
      tc_fence_before_sync();
      // O, s_m, s_l and s_inv are free for the next segment
      if (bar_or_named(kSmBar, kSmThreads, ok ? 0 : 1)) {
        ok = false;
        break;
      }
      gt += seg.count;
    }
    if (!ok && lane == 0) atomicCAS(p.error_flag, 0, (int)kTimeoutMbarrier);
  } else if (warp >= kFirstDq) {
    // =========================== dequantisation ===========================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    const int w8 = warp - kFirstDq;
    // Eight consecutive lanes (one phase of a 16-byte shared-memory access) hold four chunks of an even row and the
    // four of the odd row below: their swizzled stores fall in all eight 16-byte bank groups.
    const int row_lo = 2 * w8 + ((lane & 7) >> 2);                 // row of a 16-token unit
    const int c = 4 * (lane >> 3) + (lane & 3);                    // 16-byte chunk of the fp8 half row
    const int rrow = 8 * w8 + (lane >> 2), rc = lane & 3;          // rope: row of the tile, 16-byte chunk
    const uint8_t* lat_src = p.ckv + (size_t)rank * kDo + c * 16;
    const float* scl_src = p.scales + 2 * rank + (c >> 3);
    const __nv_bfloat16* rope_src = p.kpe + rank * (kDr / 2) + rc * 8;

    const int page_shift = (p.page_size & (p.page_size - 1)) == 0 ? __ffs(p.page_size) - 1 : -1;
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
      const int pg = page_shift >= 0 ? tok >> page_shift : tok / p.page_size;
      nx_page = p.block_table[(int64_t)seg.b * p.bt_stride + pg];
      nx_in = tok - pg * p.page_size;
      nx_live = min(seg.seq_len - tile * kTile, kTile);
      ++tile;
      --tile_left;
    };
    auto load = [&](Fetch& f) {
      f.live = nx_live;
      if (nx_live == 0) return;
      const uint32_t row = (uint32_t)nx_page * (uint32_t)p.page_size + (uint32_t)nx_in;      // fits: a row is 656 bytes
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t g = __shfl_sync(0xffffffffu, row, u) + row_lo;
        f.lat[u] = ldg_stream(lat_src + (size_t)g * kDn);
        f.scl[u] = __ldg(scl_src + (size_t)g * 4);
      }
      f.rope = ldg_stream(rope_src + (size_t)(__shfl_sync(0xffffffffu, row, w8 >> 1) + (rrow & 15)) * kDr);
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
        for (int j = 0; j < 4; ++j) e4m3x4_as_bf16x4(w[j], v[2 * j], v[2 * j + 1]);
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
    Fetch f;
    advance();
    load(f);
    while (f.live != 0) {
      convert(f);
      if (!ok) break;
      load(f);
    }
    if (!ok) atomicCAS(p.error_flag, 0, (int)kTimeoutMbarrier);
  } else {
    // =========================== MMA issue ===========================
    // 48, taken from the dequantisation warps, which do with 64: with 32 the issuing warp spilled, and a call of one tile per cluster
    // (2 x 1500 tokens) took 26.6 us instead of 25.2
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    if (warp == 0) {
      constexpr uint32_t id_qk = umma_idesc_bf16(kH, kTile);
      constexpr uint32_t id_pv = umma_idesc_bf16(kH, kDo) | (1u << 16);       // B is MN-major
      // All 512 columns are this CTA's, so its tensor memory starts at column 0: no register holds the base.  The tile
      // number goes through a shuffle for the same reason: what is computed from it is then known to be the same in all lanes
      // and stays in uniform registers, which is where the MMA reads its operands (moving them there cost ~60 cycles each).
      constexpr uint32_t td = 0;
      const uint64_t d_lat = umma_desc_k_sw128(smem_u32(smem)), d_rope = umma_desc_k_sw64(smem_u32(smem) + kLatBytes),
                     d_val = umma_desc_mn_sw128(smem_u32(smem), kSubBytes);
      // every lane waits, so that the warp stays together and all agree
      auto wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, deadline)) != 0; };
      // byte offsets enter a descriptor in 16-byte units and never carry out of its 14-bit address field
      auto qk = [&](uint32_t n_lane) {
        const uint32_t n = __shfl_sync(0xffffffffu, n_lane, 0);
        // both at once, a lane each: a wait that has nothing to wait for still takes ~200 cycles
        bool good = true;
        if (lane == 0) good = mbar_wait(&kv_full[n % kSlots], (n / kSlots) & 1, deadline);
        else if (lane == 1 && n >= 1) good = mbar_wait(&s_free, (n - 1) & 1, deadline);
        if (__all_sync(0xffffffffu, good) == 0) return false;
        __syncwarp();                                    // what either lane has seen holds for the one that issues
        tc_fence_after_sync();
        const uint32_t slot = (n % kSlots) * kSlotBytes;
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < kDo / 16; ++ks) {
            const uint32_t lo = (uint32_t)d_lat + ((slot + (ks >> 2) * kSubBytes + (ks & 3) * 32) >> 4);
            if (ks == 0) umma_bf16_ts_first(td + kColS, td + kColQ, lo, (uint32_t)(d_lat >> 32), id_qk, 0u);
            else umma_bf16_ts(td + kColS, td + kColQ + ks * 8, lo, (uint32_t)(d_lat >> 32), id_qk);
          }
#pragma unroll
          for (int ks = 0; ks < kDr / 32; ++ks)
            umma_bf16_ts(td + kColS, td + kColQ + kDo / 2 + ks * 8, (uint32_t)d_rope + ((slot + ks * 32) >> 4), (uint32_t)(d_rope >> 32), id_qk);
          umma_commit(&s_full[n & 1]);
        }
        __syncwarp();
        return true;
      };
      uint32_t n_seg = 0;
      while (ok && walk.next(s_seq, p, seg)) {
        ok = wait(&q_full, n_seg & 1);
        ++n_seg;
        if (ok) {
          tc_fence_after_sync();
          ok = qk(gt);
        }
        if (ok && seg.count > 1) ok = qk(gt + 1);
        for (int i = 0; i < seg.count && ok; ++i) {
          const uint32_t n = __shfl_sync(0xffffffffu, gt + i, 0), later = __shfl_sync(0xffffffffu, i, 0);
          if (i + 2 < seg.count && !qk(n + 2)) {
            ok = false;
            break;
          }
          if (!wait(&p_full, n & 1)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t slot = (n % kSlots) * kSlotBytes;
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < kTile / 16; ++ks) {
              const uint32_t lo = (uint32_t)d_val + ((slot + ks * 2048) >> 4);
              if (ks == 0) umma_bf16_ts_first(td + kColO, td + kColP, lo, (uint32_t)(d_val >> 32), id_pv, later);
              else umma_bf16_ts(td + kColO, td + kColP + ks * 8, lo, (uint32_t)(d_val >> 32), id_pv);
            }
            umma_commit(&kv_free[n % kSlots]);
          }
          __syncwarp();
        }
        gt += seg.count;
      }
      if (!ok) {
        if (lane == 0) atomicCAS(p.error_flag, 0, (int)kTimeoutMbarrier);
        if (elect_one()) umma_commit(&drain);                 // nothing of this CTA's may be in flight when it leaves
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
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// Merges the pieces of every sequence that more than one cluster worked on, and writes the empty sequences' zeros.
// Block (b, y) takes `heads` heads of sequence b.  Threads come in groups of 128 that share out the pieces, thread t of a
// group has output columns [4 t, 4 t + 4); with few sequences there are few blocks and many pieces each, so more groups.
constexpr int kFoldCols = kDn / 4, kFoldMaxGroups = 4;
__global__ void __launch_bounds__(kFoldCols * kFoldMaxGroups)
    mla_pair_fold_kernel(const __grid_constant__ MlaDecodeParams p, int n_clusters, int heads) {
  __shared__ int s_sum[2];
  __shared__ float s_w[kMlaMaxCtas / 2], s_l;
  __shared__ float4 s_acc[kFoldMaxGroups - 1][kFoldCols];
  const int tid = threadIdx.x, lane = tid & 31, b = blockIdx.x;
  const int t = tid % kFoldCols, g = tid / kFoldCols, groups = blockDim.x / kFoldCols;
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
  const int first = base / chunk, last = (base + max(n_tiles, 1) - 1) / chunk, n = last - first + 1;
  if (n_tiles > 0 && n == 1) return;
  for (int h = blockIdx.y * heads; h < min((int)(blockIdx.y + 1) * heads, kH); ++h) {
    uint2* dst = reinterpret_cast<uint2*>(p.o + ((int64_t)b * kH + h) * kDn) + t;
    if (n_tiles == 0) {
      if (g == 0) *dst = make_uint2(0u, 0u);
      if (tid == 0) p.lse[(int64_t)b * kH + h] = -INFINITY;
      continue;
    }
    // the first piece starts its sequence (slot 1); every later one begins where its cluster begins (slot 0)
    auto slot = [&](int i) { return (size_t)(first + i) * 2 + (i == 0 ? 1 : 0); };
    if (tid < 32) {
      float M = -INFINITY, L = 0.f;
      for (int i = lane; i < n; i += 32) {
        const float l = __ldcg(p.part_lse + slot(i) * kH + h);
        s_w[i] = l;
        M = fmaxf(M, l);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
      for (int i = lane; i < n; i += 32) {
        const float w = M == -INFINITY ? 0.f : fast_exp2(s_w[i] - M);
        s_w[i] = w;
        L += w;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
      if (lane == 0) {
        s_l = L;
        const float lse2 = L > 0.f ? M + log2f(L) : -INFINITY;
        p.lse[(int64_t)b * kH + h] = p.lse_base2 ? lse2 : lse2 * kLn2;
      }
    }
    __syncthreads();
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int i = g; i < n; i += groups) {
      const float4 v = __ldcg(reinterpret_cast<const float4*>(p.part_o + (slot(i) * kH + h) * kDn) + t);
      const float w = s_w[i];
      acc.x += w * v.x;
      acc.y += w * v.y;
      acc.z += w * v.z;
      acc.w += w * v.w;
    }
    if (g > 0) s_acc[g - 1][t] = acc;
    __syncthreads();
    if (g == 0) {
      for (int k = 1; k < groups; ++k) {
        const float4 v = s_acc[k - 1][t];
        acc.x += v.x;
        acc.y += v.y;
        acc.z += v.z;
        acc.w += v.w;
      }
      const float inv = s_l > 0.f ? 1.f / s_l : 0.f;
      *dst = make_uint2(pack_bf16(acc.x * inv, acc.y * inv), pack_bf16(acc.z * inv, acc.w * inv));
    }
    __syncthreads();                            // s_w, s_l and s_acc are free again
  }
}

// The same for more sequences than clusters: at most one split sequence per cluster, and most sequences have nothing to
// fold.  With a block per sequence and four heads the device went through 4096 (128 sequences) to 19200 blocks to find that
// out, 5 to 30 us.  Block (c, y) looks for the sequence that cluster c's tiles start and do not end; warp = head, lane = 4 x 4
// columns, four pieces per round trip with a running maximum.
constexpr int kStartsWarps = 4, kStartsBatch = 4;
__global__ void __launch_bounds__(kStartsWarps * 32)
    mla_pair_fold_starts_kernel(const __grid_constant__ MlaDecodeParams p, int n_clusters) {
  __shared__ int s_warp[kStartsWarps], s_b, s_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c = blockIdx.x, h = blockIdx.y * kStartsWarps + warp;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // every thread takes a run of sequences: `end` = tiles up to the end of its run
  const int run = (p.B + (int)blockDim.x - 1) / (int)blockDim.x, lo = min(tid * run, p.B), hi = min(lo + run, p.B);
  int mine = 0;
  for (int b = lo; b < hi; ++b) mine += max((p.seq_lens[b] + kTile - 1) / kTile, 0);
  int end = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int below = __shfl_up_sync(0xffffffffu, end, d);
    if (lane >= d) end += below;
  }
  if (lane == 31) s_warp[warp] = end;
  if (tid == 0) s_b = -1;
  __syncthreads();
  int total = 0;
#pragma unroll
  for (int w = 0; w < kStartsWarps; ++w) {
    if (w < warp) end += s_warp[w];
    total += s_warp[w];
  }
  const int chunk = max((total + n_clusters - 1) / n_clusters, 1), next = (c + 1) * chunk;      // the next cluster's first tile
  if (next < end && next > end - mine) {       // it lies inside this run, behind its first tile
    int first = end - mine, b = lo;
    for (;; ++b) {
      const int n = max((p.seq_lens[b] + kTile - 1) / kTile, 0);
      if (next < first + n) {
        if (first < next && first >= c * chunk) s_b = b, s_last = (first + n - 1) / chunk;
        break;
      }
      first += n;
    }
  }
  __syncthreads();
  for (int b = blockIdx.y * n_clusters + c; b < p.B; b += n_clusters * gridDim.y) {
    if (p.seq_lens[b] > 0) continue;                 // an empty sequence: zeros
    uint4* dst = reinterpret_cast<uint4*>(p.o + (int64_t)b * kH * kDn);
    for (int i = tid; i < kH * kDn / 8; i += blockDim.x) dst[i] = make_uint4(0u, 0u, 0u, 0u);
    p.lse[(int64_t)b * kH + tid] = -INFINITY;
  }
  static_assert(kStartsWarps * 32 == kH, "a thread per LSE of an empty sequence");
  if (s_b < 0) return;
  const int n = s_last - c + 1;
  float M = -INFINITY, L = 0.f;
  float4 acc[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i0 = 0; i0 < n; i0 += kStartsBatch) {
    float4 v[kStartsBatch][4];
    float l[kStartsBatch];
#pragma unroll
    for (int k = 0; k < kStartsBatch; ++k) {
      l[k] = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) v[k][j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i0 + k < n) {
        // the first piece starts its sequence (slot 1); every later one begins where its cluster begins (slot 0)
        const size_t row = ((size_t)(c + i0 + k) * 2 + (i0 + k == 0 ? 1 : 0)) * kH + h;
        l[k] = __ldcg(p.part_lse + row);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[k][j] = __ldcg(reinterpret_cast<const float4*>(p.part_o + row * kDn) + lane + 32 * j);
      }
    }
    float top = M;
#pragma unroll
    for (int k = 0; k < kStartsBatch; ++k) top = fmaxf(top, l[k]);
    const float keep = M == -INFINITY ? 0.f : fast_exp2(M - top);
    M = top;
    L *= keep;
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = make_float4(acc[j].x * keep, acc[j].y * keep, acc[j].z * keep, acc[j].w * keep);
#pragma unroll
    for (int k = 0; k < kStartsBatch; ++k) {
      const float w = l[k] == -INFINITY ? 0.f : fast_exp2(l[k] - top);
      L += w;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[j].x += w * v[k][j].x;
        acc[j].y += w * v[k][j].y;
        acc[j].z += w * v[k][j].z;
        acc[j].w += w * v[k][j].w;
      }
    }
  }
  const float inv = L > 0.f ? 1.f / L : 0.f;
  const int64_t out = (int64_t)s_b * kH + h;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    reinterpret_cast<uint2*>(p.o + out * kDn)[lane + 32 * j] =
        make_uint2(pack_bf16(acc[j].x * inv, acc[j].y * inv), pack_bf16(acc[j].z * inv, acc[j].w * inv));
  if (lane == 0) {
    const float lse2 = L > 0.f ? M + log2f(L) : -INFINITY;
    p.lse[out] = p.lse_base2 ? lse2 : lse2 * kLn2;
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
  cfg.dynamicSmemBytes = 0;
  cfg.numAttrs = 1;
  const int n_clusters = p.ctas / 2;
  if (p.B > n_clusters) {
    cfg.gridDim = dim3(n_clusters, kH / kStartsWarps, 1);
    cfg.blockDim = dim3(kStartsWarps * 32, 1, 1);
    return cudaLaunchKernelEx(&cfg, mla_pair_fold_starts_kernel, p, n_clusters);
  }
  // A block's heads follow one another, 2-3 us each, so it takes several only where one each would be more blocks than
  // the device holds at once (16 of them per SM).
  const int heads = p.B <= 18 ? 1 : p.B <= 37 ? 2 : 4;
  cfg.gridDim = dim3(p.B, kH / heads, 1);
  cfg.blockDim = dim3(kFoldCols * (p.B <= 4 ? 4 : p.B <= 9 ? 2 : 1), 1, 1);
  return cudaLaunchKernelEx(&cfg, mla_pair_fold_kernel, p, n_clusters, heads);
}

}  // namespace helix
