// 32-bit products on the tensor cores: out[m, n] = sum_k x[m, k] * w[n, k], all fp32.
//
// A 24-bit significand is exactly three 8-bit ones, so an fp32 value is the sum of three bf16 values without rounding
// (truncation, subtraction, truncation, subtraction).  Of the nine products of two such sums all but the last (a3 b3, below 2^-30 of the
// product) are taken.  Products of bf16 values are exact in fp32; what is not is the tensor core's accumulation, which truncates: a
// long sum would lose a unit in the last place per step, always towards zero.  So an accumulator only ever holds one slab of 64 k,
// small products first, and warps add the slabs up in registers with ordinary rounding.  Error against 64 bits (norm of the
// difference) at 4096 k: 1.2e-7, one running sum in fp32 1.1e-6; a single product is good to 2^-23 (a multiply-add to 2^-24).  (The
// six largest products alone, a sixth faster at 160 rows: 1.5e-7, a single product 2^-21.)
//
// A CTA owns 128 rows of w, BN rows of x and a range of k:
//   warps 0-7   add finished slabs from tensor memory (two accumulators in turn): 128 rows x BN / 2 columns per four warps
//   warps 8-11  a row of w per thread: split a slab of it into three bf16 parts and put them into tensor memory as the MMAs' first
//               operand (two buffers in turn)
//   warp 12     brings w as it is (TMA, a ring of three to six slabs)
//   warp 13     brings the three tiles of x (TMA, two stages), which a kernel before this one has split once
//   warp 14     issues the slab's 32 MMAs
// The ranges of k of one tile go to separate planes that a last kernel adds in order.
//
// Bound by the eight MMAs per product (1.35 us per slab of 160 rows, 1.75 with everything around them) or, with few rows, by the
// splitting (0.95 us per slab, 3.8 TB/s of w over all SMs).  w's parts go through tensor memory because shared memory is full: with
// w and x in stages of their own nothing waits for a load.  (w split into shared memory by the warps that loaded it, stages shared
// with x: 385 us for six products of 301 x 16448 x 4096, 202 in this form.)  4096 k, in us behind a flushed L2, on the CUDA cores (64 x 64 tiles of
// multiply-adds) and here: 301 x 16448 1746 and 232, 301 x 4096 772 and 71, 1 x 16448 398 and 77, 301 x 4096 of 14336 k 2732 and 204.
//
// A result that is not a number is computed again with ordinary multiply-adds (`fs_again`): an infinity times a part that is zero is
// none.  So is one below 2^-100: the third parts of values below 2^-110 lie under bf16's smallest numbers (2^-133), and products of parts
// under those of fp32.  Larger results do not see what is lost there, unless the other operand is beyond 2^10.  Values below 2^-133
// count as zeros.
#include "common.cuh"
#include "gemm_args.h"
#include "api.h"

namespace nkb {

struct F32SplitArgs {
  const float* x;
  const float* w;
  float* out;                 // splits > 1: planes of split_stride
  int m, n, k, kp;            // kp: k in whole slabs
  int splits, slabs_per_split, slabs;
  long long ldx, ldw, ldo, split_stride;
  int* status;
};

constexpr int kFsThreads = 15 * 32;
constexpr int kFsStages = 2;                        // of x, of w's parts and of accumulators
constexpr int kFsRawBytes = kTileRows * kBlockK * 4;
constexpr int kFsMaxRaw = 6;
__host__ __device__ constexpr int fs_x_bytes(int bn) { return 3 * bn * kBlockK * 2; }
__host__ __device__ constexpr int fs_raw_stages(int bn) {
  const int fit = (232448 - 2048 - kFsStages * fs_x_bytes(bn)) / kFsRawBytes;
  return fit < kFsMaxRaw ? fit : kFsMaxRaw;
}
struct FsCtrl {
  uint64_t rfull[kFsMaxRaw], rempty[kFsMaxRaw], xfull[kFsStages], wfull[kFsStages], done[kFsStages], tfull[2], tempty[2];
  uint32_t tmem_base;
  int abort;
};

// The top halves of p[0..2] are the three parts of x.
__device__ __forceinline__ void split_f32(float x, uint32_t (&p)[3]) {
  uint32_t u = __float_as_uint(x);
  float r = x - __uint_as_float(u & 0xffff0000u);
  if ((u & 0x7f800000u) == 0x7f800000u) {       // infinity, or a NaN, which must not become one
    if (u & 0x007fffffu) u |= 0x00400000u;
    r = 0.f;
  }
  p[0] = u;
  p[1] = __float_as_uint(r);
  p[2] = __float_as_uint(r - __uint_as_float(p[1] & 0xffff0000u));
}
// three planes of four values, two bf16 per word
__device__ __forceinline__ void split_f32x4(const float4& v, uint2 (&o)[3]) {
  uint32_t a[3], b[3], c[3], d[3];
  split_f32(v.x, a);
  split_f32(v.y, b);
  split_f32(v.z, c);
  split_f32(v.w, d);
#pragma unroll
  for (int i = 0; i < 3; ++i) o[i] = make_uint2(__byte_perm(a[i], b[i], 0x7632), __byte_perm(c[i], d[i], 0x7632));
}

// planes[3][m][kp] of x, zeros behind k
__global__ void __launch_bounds__(256) f32_planes_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ planes, int m, int k,
                                                         int kp, long long ldx) {
  griddep_wait();
  griddep_launch();
  const int per_row = kp / 4;
  const long long total = (long long)m * per_row;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const long long r = i / per_row;
    const int c = int(i - r * per_row) * 4;
    const float4 v = c < k ? *reinterpret_cast<const float4*>(x + r * ldx + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    uint2 o[3];
    split_f32x4(v, o);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(planes + ((long long)p * m + r) * kp + c) = o[p];
  }
}

__global__ void __launch_bounds__(256) f32_sum_planes_kernel(const float* __restrict__ parts, int splits, long long stride,
                                                             float* __restrict__ out, long long n) {
  griddep_wait();
  griddep_launch();
  for (long long i = (blockIdx.x * 256ll + threadIdx.x) * 4; i < n; i += gridDim.x * 1024ll) {
    float4 a = *reinterpret_cast<const float4*>(parts + i);
#pragma unroll 8
    for (int s = 1; s < splits; ++s) {
      const float4 b = *reinterpret_cast<const float4*>(parts + s * stride + i);
      a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    }
    if (i + 3 < n) {
      *reinterpret_cast<float4*>(out + i) = a;
    } else {
      out[i] = a.x;
      if (i + 1 < n) out[i + 1] = a.y;
      if (i + 2 < n) out[i + 2] = a.z;
    }
  }
}

// Whether a result is computed again.
__device__ __forceinline__ bool fs_doubtful(float y) { return !(fabsf(y) >= 0x1p-100f) && y != 0.f; }

// Doubtful results in rows [r0, r0 + 32) of w and [t0, t1) of x, again by multiply-adds over [k0, k1), a result at a time by the whole warp.  Rows that hold a NaN are left as they are, a sum that has become one ends there.  (301 x 16448 x
// 4096 with every row of x NaN 0.75 ms, with a NaN in every row of w 3.4 ms, with one infinity 0.28 ms; by a thread per row of w, its
// loads 32 rows apart, 104, 104 and 0.55 ms.)
__device__ __noinline__ void fs_again(const float* x, const float* w, float* out, long long ldx, long long ldw, long long ldo, int r0, int n,
                                      int t0, int t1, int k0, int k1) {
  constexpr uint32_t kAll = 0xffffffffu;
  constexpr int kAhead = 8, kStep = kAhead * 128;
  const int lane = threadIdx.x & 31;
  const auto holds_nan = [&](const float* row) {
    bool nan = false;
#pragma unroll 1
    for (int k = k0; k < k1 && !nan; k += kStep) {
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        const int c = k + i * 128 + lane * 4;
        if (c < k1) {
          const float4 a = *reinterpret_cast<const float4*>(row + c);
          nan |= a.x != a.x || a.y != a.y || a.z != a.z || a.w != a.w;
        }
      }
      nan = __any_sync(kAll, nan);
    }
    return nan;
  };
  uint32_t seen = 0, lost = 0;                      // rows of w that have been looked through, and that hold a NaN
#pragma unroll 1
  for (int t = t0; t < t1; ++t) {
    const float y = r0 + lane < n ? out[t * ldo + r0 + lane] : 0.f;
    uint32_t bad = __ballot_sync(kAll, fs_doubtful(y));
    const float* xr = x + t * ldx;
    if (bad && holds_nan(xr)) bad = 0;
#pragma unroll 1
    for (; bad; bad &= bad - 1) {
      const int r = __ffs(bad) - 1;
      const float* wr = w + (long long)(r0 + r) * ldw;
      if (!(seen >> r & 1u)) {
        seen |= 1u << r;
        if (holds_nan(wr)) lost |= 1u << r;
      }
      if (lost >> r & 1u) continue;
      float v = 0.f;
#pragma unroll 1
      for (int k = k0; k < k1; k += kStep) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          const int c = k + i * 128 + lane * 4;
          if (c < k1) {
            const float4 a = *reinterpret_cast<const float4*>(xr + c), b = *reinterpret_cast<const float4*>(wr + c);
            v = fmaf(a.x, b.x, v);
            v = fmaf(a.y, b.y, v);
            v = fmaf(a.z, b.z, v);
            v = fmaf(a.w, b.w, v);
          }
        }
        if (__any_sync(kAll, v != v)) break;
      }
      v = warp_sum(v);
      if (lane == r) out[t * ldo + r0 + r] = v;      // the lane that stored it before
    }
  }
}

template <int BN>
__global__ void __launch_bounds__(kFsThreads, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const F32SplitArgs a) {
  constexpr int kBTile = BN * kBlockK * 2, kXStage = fs_x_bytes(BN), kRaw = fs_raw_stages(BN);
  constexpr int kCols = BN / 2;                     // of an adding warp
  constexpr int kPartCols = 3 * kBlockK / 2;        // tensor memory columns of a slab of w in three parts
  constexpr uint32_t kTmem = 512;
  static_assert(2 * BN + kFsStages * kPartCols <= int(kTmem), "two accumulators and two slabs of w fit tensor memory");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* x_tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* raw_tiles = x_tiles + kFsStages * kXStage;
  __shared__ FsCtrl ctrl;
  const int warp = warp_idx_uniform(), lane = threadIdx.x & 31;
  const int split = blockIdx.x % a.splits, n0 = (blockIdx.x / a.splits) * kTileRows, m0 = blockIdx.y * BN;
  const int s0 = split * a.slabs_per_split, count = min(a.slabs, s0 + a.slabs_per_split) - s0;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW);
    for (int s = 0; s < kRaw; ++s) {
      mbar_init(&ctrl.rfull[s], 1);
      mbar_init(&ctrl.rempty[s], 4);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctrl.xfull[i], 1);
      mbar_init(&ctrl.wfull[i], 4);
      mbar_init(&ctrl.done[i], 1);
      mbar_init(&ctrl.tfull[i], 1);
      mbar_init(&ctrl.tempty[i], 8);
    }
    ctrl.abort = 0;
    mbar_fence_init();
    fence_proxy_async();
  }
  if (warp == 8) {
    tmem_alloc(&ctrl.tmem_base, kTmem);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctrl.tmem_base;
  volatile int* abort_flag = &ctrl.abort;
  griddep_wait();
  griddep_launch();

  if (warp < 8) {
    // ------------------------------------------------------------------ sums of slabs
    const int quad = warp & 3, c0 = (warp >> 2) * kCols;
    float acc[kCols];
#pragma unroll
    for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
    bool ok = true;
    for (int s = 0; s < count; ++s) {
      const int i = s & 1;
      ok = mbar_wait(&ctrl.tfull[i], (s >> 1) & 1, abort_flag, a.status, ERR_WAIT_TMEM_FULL);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      tc_fence_after();
      const uint32_t t0 = tmem + (uint32_t(quad * 32) << 16) + uint32_t(i * BN + c0);
#pragma unroll
      for (int c = 0; c + 32 <= kCols; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32(t0 + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[c + j] += __uint_as_float(v[j]);
      }
      if constexpr (kCols % 32) {
        uint32_t v[16];
        tmem_ld_32x16(t0 + kCols / 32 * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[kCols / 32 * 32 + j] += __uint_as_float(v[j]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctrl.tempty[i]);
    }
    const int row = n0 + quad * 32 + lane;
    bool bad = false;
    if (ok && row < a.n) {
      float* out = a.out + split * a.split_stride + row;
#pragma unroll
      for (int j = 0; j < kCols; ++j) {
        const int t = m0 + c0 + j;
        if (t < a.m) out[t * a.ldo] = acc[j];
        bad |= t < a.m && fs_doubtful(acc[j]);
      }
    }
    if (__any_sync(0xffffffffu, bad))
      fs_again(a.x, a.w, a.out + split * a.split_stride, a.ldx, a.ldw, a.ldo, n0 + quad * 32, a.n, m0 + c0, min(a.m, m0 + c0 + kCols),
               s0 * kBlockK, min(a.k, (s0 + count) * kBlockK));
  } else if (warp < 12) {
    // ------------------------------------------------------------------ parts of w
    const int quad = warp & 3, row = quad * 32 + lane;
    int r = 0;
    uint32_t rphase = 0;
    for (int s = 0; s < count; ++s) {
      const int i = s & 1;
      const bool ok = mbar_wait(&ctrl.rfull[r], rphase, abort_flag, a.status, ERR_WAIT_SMEM_FULL) &&
                      mbar_wait(&ctrl.done[i], ((s >> 1) & 1) ^ 1u, abort_flag, a.status, ERR_WAIT_SMEM_EMPTY);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      const uint32_t t0 = tmem + (uint32_t(quad * 32) << 16) + uint32_t(2 * BN + i * kPartCols);
#pragma unroll
      for (int h = 0; h < 2; ++h) {                 // 32 k: a row of 128 swizzled bytes
        const uint8_t* src = raw_tiles + r * kFsRawBytes + h * (kFsRawBytes / 2) + row * 128;
        uint32_t w[3][16];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint2 o[3];
          split_f32x4(*reinterpret_cast<const float4*>(src + ((c ^ (row & 7)) << 4)), o);
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            w[p][2 * c] = o[p].x;
            w[p][2 * c + 1] = o[p].y;
          }
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) tmem_st_32x16(t0 + p * (kBlockK / 2) + h * 16, w[p]);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&ctrl.rempty[r]);
        mbar_arrive(&ctrl.wfull[i]);
      }
      if (++r == kRaw) { r = 0; rphase ^= 1u; }
    }
  } else if (warp == 12) {
    // ------------------------------------------------------------------ w
    if (elect_one()) {
      int r = 0;
      uint32_t phase = 0;
      for (int s = 0; s < count; ++s) {
        if (!mbar_wait(&ctrl.rempty[r], phase ^ 1u, abort_flag, a.status, ERR_WAIT_SMEM_EMPTY)) break;
        mbar_expect_tx(&ctrl.rfull[r], kFsRawBytes);
        uint8_t* dst = raw_tiles + r * kFsRawBytes;
#pragma unroll
        for (int h = 0; h < 2; ++h)                 // the map counts 16-bit units
          tma_load_2d(dst + h * (kFsRawBytes / 2), &tmW, &ctrl.rfull[r], ((s0 + s) * 2 + h) * 64, n0);
        if (++r == kRaw) { r = 0; phase ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 13) {
    // ------------------------------------------------------------------ x
    if (elect_one()) {
      for (int s = 0; s < count; ++s) {
        const int i = s & 1;
        if (!mbar_wait(&ctrl.done[i], ((s >> 1) & 1) ^ 1u, abort_flag, a.status, ERR_WAIT_SMEM_EMPTY)) break;
        mbar_expect_tx(&ctrl.xfull[i], kXStage);
#pragma unroll
        for (int p = 0; p < 3; ++p)
          tma_load_2d(x_tiles + i * kXStage + p * kBTile, &tmX, &ctrl.xfull[i], (s0 + s) * kBlockK, p * a.m + m0);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ MMAs
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(kTileRows, BN, 0, 0);
      for (int s = 0; s < count; ++s) {
        const int i = s & 1;
        const uint32_t phase = (s >> 1) & 1;
        if (!mbar_wait(&ctrl.tempty[i], phase ^ 1u, abort_flag, a.status, ERR_WAIT_TMEM_EMPTY) ||
            !mbar_wait(&ctrl.xfull[i], phase, abort_flag, a.status, ERR_WAIT_SMEM_FULL) ||
            !mbar_wait(&ctrl.wfull[i], phase, abort_flag, a.status, ERR_WAIT_SMEM_FULL))
          break;
        tc_fence_after();
        const uint32_t d = tmem + uint32_t(i * BN), w0 = tmem + uint32_t(2 * BN + i * kPartCols);
        const uint32_t x0 = smem_u32(x_tiles) + i * kXStage;
        constexpr int kA[8] = {2, 1, 2, 1, 0, 1, 0, 0}, kB[8] = {1, 2, 0, 1, 2, 0, 1, 0};        // small products first
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const uint64_t db = make_smem_desc_sw128(x0 + kB[t] * kBTile, 0, 1024);
#pragma unroll
          for (int k = 0; k < kBlockK / 16; ++k)
            umma_f16_ts(d, w0 + kA[t] * (kBlockK / 2) + k * 8, db + uint64_t(k * 2), idesc, t > 0 || k > 0 ? 1u : 0u);
        }
        umma_commit(&ctrl.done[i]);
        umma_commit(&ctrl.tfull[i]);
      }
    }
    __syncwarp();
  }
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);      // let copies and MMAs in flight drain
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmem);
  }
}

template <int BN>
static int launch_f32_split(const CUtensorMap& tx, const CUtensorMap& tw, const F32SplitArgs& a, cudaStream_t s) {
  constexpr int smem = kFsStages * fs_x_bytes(BN) + fs_raw_stages(BN) * kFsRawBytes + 1024;
  static_assert(smem + int(sizeof(FsCtrl)) <= 232448 && fs_raw_stages(BN) >= 3, "the rings fit a CTA's shared memory");
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return int(e);
    attr_set[dev] = true;
  }
  return launch_pdl(gemm_f32_split_kernel<BN>, dim3((a.n + kTileRows - 1) / kTileRows * a.splits, (a.m + BN - 1) / BN),
                    dim3(kFsThreads), size_t(smem), s, tx, tw, a);
}

}  // namespace nkb

using namespace nkb;

// planes: bf16 scratch [3][m][k in whole slabs of 64]; parts: fp32 scratch [splits][m][n], 16-byte aligned, null with one split; out
// [m][n], contiguous.  Rows of x and w start on 16 bytes and k is a multiple of four (-5 otherwise); block_n one of 32, 64, 96,
// 128, 160; no split is empty.
extern "C" int nkb_gemm_f32_split(const float* x, const float* w, float* out, void* planes, float* parts, int m, int n, int k,
                                  long long ldx, long long ldw, int block_n, int splits, void* stream) {
  if (m <= 0 || n <= 0) return 0;
  if (k <= 0 || splits < 1 || !planes || (splits > 1 && !parts)) return -2;
  if (((k | ldx | ldw) & 3) || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(planes) |
                                 reinterpret_cast<uintptr_t>(parts) | reinterpret_cast<uintptr_t>(out)) & 15))
    return -5;
  if (!status_word() && nkb_init() != 0) return -1;
  F32SplitArgs a{};
  a.x = x;
  a.w = w;
  a.m = m; a.n = n; a.k = k;
  a.slabs = (k + kBlockK - 1) / kBlockK;
  a.kp = a.slabs * kBlockK;
  a.splits = splits;
  a.slabs_per_split = (a.slabs + splits - 1) / splits;
  if ((splits - 1) * a.slabs_per_split >= a.slabs) return -2;
  if ((m + block_n - 1) / block_n > 65535) return -2;
  a.ldx = ldx; a.ldw = ldw; a.ldo = n;
  const long long total = (long long)m * n;
  a.split_stride = splits > 1 ? (total + 3) / 4 * 4 : 0;
  a.out = splits > 1 ? parts : out;
  a.status = status_word();
  CUtensorMap tm, tw;
  if (encode_tmap_bf16_2d(&tm, planes, a.kp, 3ull * m, a.kp, kBlockK, block_n)) return -4;
  // w as pairs of 16-bit units, 32 values (128 bytes) per box row
  if (encode_tmap_bf16_2d(&tw, w, 2ull * k, n, 2ull * ldw, 64, kTileRows)) return -4;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const long long quads = (long long)m * (a.kp / 4);
  const long long pb = (quads + 255) / 256;
  int rc = launch_pdl(f32_planes_kernel, dim3(unsigned(pb < 148 * 16 ? pb : 148 * 16)), dim3(256), 0, s, x,
                      reinterpret_cast<__nv_bfloat16*>(planes), m, k, a.kp, ldx);
  if (rc) return rc;
  switch (block_n) {
    case 32: rc = launch_f32_split<32>(tm, tw, a, s); break;
    case 64: rc = launch_f32_split<64>(tm, tw, a, s); break;
    case 96: rc = launch_f32_split<96>(tm, tw, a, s); break;
    case 128: rc = launch_f32_split<128>(tm, tw, a, s); break;
    case 160: rc = launch_f32_split<160>(tm, tw, a, s); break;
    default: return -2;
  }
  if (rc || splits == 1) return rc;
  const long long sb = (total + 1023) / 1024;
  return launch_pdl(f32_sum_planes_kernel, dim3(unsigned(sb < 148 * 8 ? sb : 148 * 8)), dim3(256), 0, s, (const float*)parts, splits,
                    a.split_stride, out, total);
}
