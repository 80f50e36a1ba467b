// Stand-alone LSE-weighted combine for B200: [N, rows, D] partial outputs + [N, rows] LSEs -> [rows, D].
//
//   out[r, :] = sum_n w_n o_n[r, :] / sum_n w_n,   w_n = exp(lse_n[r] - max_n lse_n[r])
//
// The fused exchange applies this as the lines land; this kernel is for callers that already hold every
// rank's rows: users of the plain `alltoall`, and the NCCL path of the vLLM hook.  Counterpart of the
// reference's Triton kernel (patches/dcp_alltoall_helix.py:210-384), with its rules: NaN and +-inf LSEs count
// as -inf (no contribution), a row whose LSEs are all -inf comes out as zeros with a global LSE of -inf,
// base e or base 2.  One warp per row with the online accumulator of the exchange's receive side in registers, or, for short rows,
// half a warp that takes the maximum of the row's LSEs first and then adds up weighted rows (LSEs beyond the sixteenth rank are read
// twice).  16-byte loads; a row is read once and never staged.
#include "lse_combine.h"

#include "exchange_device.cuh"

namespace helix {
namespace {

using namespace dev;

constexpr int kWarpsPerCta = 4;

template <bool BF16, int NIT>
__global__ void __launch_bounds__(kWarpsPerCta * 32) lse_combine_kernel(const __grid_constant__ LseCombineParams p) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (row >= p.rows) return;
  const int nchunks = p.row_bytes >> 4;
  Acc<NIT> acc;
  acc.init();
  for (int n = 0; n < p.n; ++n) {
    const float raw = *reinterpret_cast<const float*>(p.lse + n * p.l_sn + row * p.l_sr);
    float l = p.base2 ? raw : raw * kLog2e;
    if (!(fabsf(l) <= 3.0e38f)) l = -INFINITY;
    if (l == -INFINITY) continue;   // warp-uniform: the row is not even read
    const uint8_t* src = p.o + n * p.o_sn + row * p.o_sr;
    uint64_t lo[NIT], hi[NIT];
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int ch = it * 32 + lane;
      lo[it] = hi[it] = 0ull;
      if (ch < nchunks) {
        const uint4 v = *reinterpret_cast<const uint4*>(src + 16 * ch);
        lo[it] = (uint64_t)v.x | ((uint64_t)v.y << 32);
        hi[it] = (uint64_t)v.z | ((uint64_t)v.w << 32);
      }
    }
    acc.template add<BF16>(l, lo, hi);
  }
  const float inv = acc.s > 0.f ? 1.0f / acc.s : 0.f;
  uint8_t* dst = p.out + row * p.out_sr;
#pragma unroll
  for (int it = 0; it < NIT; ++it) {
    const int ch = it * 32 + lane;
    if (ch < nchunks) {
      float f[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = acc.v[it][j] * inv;
      const uint64_t a = pack4<BF16>(f), b = pack4<BF16>(f + 4);
      uint4 v;
      v.x = (uint32_t)a;
      v.y = (uint32_t)(a >> 32);
      v.z = (uint32_t)b;
      v.w = (uint32_t)(b >> 32);
      *reinterpret_cast<uint4*>(dst + 16 * ch) = v;
    }
  }
  if (p.lse_out != nullptr && lane == 0) {
    float gl = acc.s > 0.f ? (acc.m + log2f(acc.s)) : -INFINITY;
    if (!p.base2) gl *= kLn2;
    p.lse_out[row] = gl;
  }
}

// Rows of up to 16 chunks (head_dim 128 and less): half a warp each, or half of the lanes would be idle, and the lanes share out the
// ranks' LSEs, so that a rank costs a row eight multiply-adds per lane and no exponential.  The kernel above is bound by its
// instructions there: 16384 rows of 128, 8 / 4 / 2 ranks (in a graph) 17.8 / 9.0 / 6.5 -> 13.4 / 5.6 / 4.6 us, 2048 rows 5.0 / 3.4 / 2.7
// -> 4.0 / 3.2 / 2.7.  For rows of 512 it is the other way round: the same arithmetic with a warp per row took 35.7 us against
// 30.6 (8 ranks, 16384 rows), and with two or four ranks' rows in flight at once 35.9 and 42.7.  One or two ranks below 2048 rows
// keep a warp per row too (lse_combine_half_warps).
constexpr int kHalf = 16;
template <bool BF16>
__global__ void __launch_bounds__(kWarpsPerCta * 32) lse_combine_half_kernel(const __grid_constant__ LseCombineParams p) {
  const int lane = threadIdx.x % kHalf;
  const int64_t row = ((int64_t)blockIdx.x * kWarpsPerCta * 32 + threadIdx.x) / kHalf;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const bool inside = row < p.rows;               // a row outside shares its warp with one inside: it walks along
  const int64_t at = inside ? row : p.rows - 1;
  const int nchunks = p.row_bytes >> 4;
  const uint8_t* lse = p.lse + at * p.l_sr;
  auto load_lse = [&](int n) {
    if (n >= p.n) return -INFINITY;
    const float raw = *reinterpret_cast<const float*>(lse + n * p.l_sn);
    const float l = p.base2 ? raw : raw * kLog2e;
    return fabsf(l) <= 3.0e38f ? l : -INFINITY;   // NaN and +-inf: no contribution
  };
  const float first = load_lse(lane);
  float top = first;
  for (int n = kHalf + lane; n < p.n; n += kHalf) top = fmaxf(top, load_lse(n));
#pragma unroll
  for (int o = kHalf / 2; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(kFull, top, o));

  float acc[8], sum = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  const uint8_t* src = p.o + at * p.o_sr + 16 * lane;
  for (int n0 = 0; n0 < p.n; n0 += kHalf) {
    const float l = n0 == 0 ? first : load_lse(n0 + lane);
    const float w = l == -INFINITY ? -1.f : exp2f(l - top);          // below zero: the row is not even read
    sum += fmaxf(w, 0.f);
    const int count = min(kHalf, p.n - n0);
#pragma unroll 2
    for (int k = 0; k < count; ++k) {
      const float wk = __shfl_sync(kFull, w, k, kHalf);
      if (wk >= 0.f && lane < nchunks) {
        const uint4 v = *reinterpret_cast<const uint4*>(src);
        float a[4], b[4];
        unpack4<BF16>((uint64_t)v.x | (uint64_t)v.y << 32, a);
        unpack4<BF16>((uint64_t)v.z | (uint64_t)v.w << 32, b);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[j] += wk * a[j];
          acc[4 + j] += wk * b[j];
        }
      }
      src += p.o_sn;
    }
  }
#pragma unroll
  for (int o = kHalf / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
  if (!inside) return;
  const float inv = sum > 0.f ? 1.0f / sum : 0.f;
  if (lane < nchunks) {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] *= inv;
    const uint64_t a = pack4<BF16>(acc), b = pack4<BF16>(acc + 4);
    *reinterpret_cast<uint4*>(p.out + row * p.out_sr + 16 * lane) =
        make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
  }
  if (p.lse_out != nullptr && lane == 0) {
    float gl = sum > 0.f ? top + log2f(sum) : -INFINITY;
    if (!p.base2) gl *= kLn2;
    p.lse_out[row] = gl;
  }
}

using Fn = void (*)(LseCombineParams);
template <int NIT>
Fn pick(bool bf16) {
  return bf16 ? (Fn)lse_combine_kernel<true, NIT> : (Fn)lse_combine_kernel<false, NIT>;
}

}  // namespace

// Half a warp per row reduces the LSEs over the lanes before the first row is on its way, about 0.2 us.  With one or two ranks and
// few rows nothing makes up for it.  Rows of 128, a warp and half a warp per row, in a graph, us: 1 rank 128 rows 1.84 and 1.99, 2048
// rows 2.05 and 2.15, 4096 rows level; 2 ranks 4 rows 1.92 and 2.09, 1024 rows 2.35 and 2.37 (2.21 and 2.33 where a row's LSEs lie
// together), 2048 rows level, 4096 rows 2.73 and 2.57; 3 ranks 128 rows 2.62 and 2.45 (2.37 and 2.44 there).  The layout is left
// out of the rule, so that both give the same bits.
bool lse_combine_half_warps(int64_t rows, int n, int row_bytes) {
  return row_bytes <= kHalf * 16 && (n > 2 || rows >= 2048);
}

cudaError_t launch_lse_combine(const LseCombineParams& p, bool pdl, cudaStream_t stream) {
  if (p.rows <= 0 || p.n <= 0) return cudaSuccess;
  if (p.row_bytes <= 0 || p.row_bytes % 16 != 0 || p.row_bytes > 4 * 32 * 16) return cudaErrorInvalidValue;
  const int chunks = p.row_bytes / 16;
  const bool half = lse_combine_half_warps(p.rows, p.n, p.row_bytes);
  Fn fn = half            ? (p.is_bf16 ? (Fn)lse_combine_half_kernel<true> : (Fn)lse_combine_half_kernel<false>)
          : chunks <= 32  ? pick<1>(p.is_bf16)
          : chunks <= 64  ? pick<2>(p.is_bf16)
                          : pick<4>(p.is_bf16);
  const int rows_per_cta = half ? 2 * kWarpsPerCta : kWarpsPerCta;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((p.rows + rows_per_cta - 1) / rows_per_cta), 1, 1);
  cfg.blockDim = dim3(kWarpsPerCta * 32, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attrs[1];
  int na = 0;
  if (pdl) {
    attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, fn, p);
}

}  // namespace helix
