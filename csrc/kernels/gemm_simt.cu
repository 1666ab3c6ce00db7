// fp32-accumulating GEMM on the CUDA cores: out[m, n] = sum_k x[m, k] * w[n, k], operands fp32 or bf16, output fp32
// or bf16, any sizes and row strides.  Serves models that run in true 32-bit (no tensor-core mode keeps all 24
// mantissa bits) and the projections whose inner size has no 16-byte row pitch, which TMA cannot describe.
//
// Two kernels.  32-bit operands with 16-byte rows run `gemm_f32_kernel` (tiles of up to 64 x 256, up to 16 x 8 results per thread
// in packed pairs, split over k inside a cluster).  Everything else (bf16 without a 16-byte pitch, groups, odd pitches) runs
// `simt_tile`: a CTA of 256 threads owns a 64 x 64 tile of the output, four rows by four columns per thread; k-slabs of 16 are
// prefetched into registers while the previous slab is multiplied from shared memory.
#include "common.cuh"
#include "proj_src.cuh"
#include "api.h"

namespace nkb {

// The body of one tile: rows [m0, m) of x (through row_token when given) against rows of w.
template <typename XT, typename WT, typename OT>
__device__ __forceinline__ void simt_tile(const XT* __restrict__ x, const WT* __restrict__ w, OT* __restrict__ out, int m0,
                                          int m, int n0, int n, int k, long long ldx, long long ldw, long long ldo,
                                          const int* __restrict__ row_token) {
  constexpr int kT = 64, kK = 16;
  __shared__ __align__(16) float xs[kK][kT + 4], ws[kK][kT + 4];
  const int tr = threadIdx.x >> 4, tc = threadIdx.x & 15;
  const int lr = threadIdx.x >> 2, lk = (threadIdx.x & 3) * 4;   // loader: row, first of four k
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  float rx[4], rw[4];
  const long long xr = m0 + lr < m ? (row_token ? row_token[m0 + lr] : m0 + lr) : 0;
  auto fetch = [&](int k0) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int kk = k0 + lk + e;
      rx[e] = (m0 + lr < m && kk < k) ? cast_in<XT>(x[xr * ldx + kk]) : 0.f;
      rw[e] = (n0 + lr < n && kk < k) ? cast_in<WT>(w[(long long)(n0 + lr) * ldw + kk]) : 0.f;
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < k; k0 += kK) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      xs[lk + e][lr] = rx[e];
      ws[lk + e][lr] = rw[e];
    }
    __syncthreads();
    if (k0 + kK < k) fetch(k0 + kK);
#pragma unroll
    for (int kk = 0; kk < kK; ++kk) {
      const float4 a = *reinterpret_cast<const float4*>(&xs[kk][tr * 4]);
      const float4 b = *reinterpret_cast<const float4*>(&ws[kk][tc * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = m0 + tr * 4 + i;
    if (r >= m) break;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = n0 + tc * 4 + j;
      if (c < n) out[(long long)r * ldo + c] = cast_out<OT>(acc[i][j]);
    }
  }
}

template <typename XT, typename WT, typename OT>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const XT* __restrict__ x, const WT* __restrict__ w, OT* __restrict__ out, int m, int n, int k,
                 long long ldx, long long ldw, long long ldo) {
  griddep_wait();
  griddep_launch();
  simt_tile<XT, WT, OT>(x, w, out, blockIdx.y * 64, m, blockIdx.x * 64, n, k, ldx, ldw, ldo, nullptr);
}

// rows of group g: [offsets[g], offsets[g + 1]), weights w + g * n * k
template <typename XT, typename WT, typename OT>
__global__ void __launch_bounds__(256)
gemm_simt_grouped_kernel(const XT* __restrict__ x, const WT* __restrict__ w, OT* __restrict__ out,
                         const int* __restrict__ offsets, const int* __restrict__ row_token, int n, int k, long long ldx,
                         long long ldo) {
  griddep_wait();
  griddep_launch();
  const int g = blockIdx.z, m0 = offsets[g] + blockIdx.y * 64, m = offsets[g + 1];
  if (m0 >= m) return;
  simt_tile<XT, WT, OT>(x, w + (long long)g * n * k, out, m0, m, blockIdx.x * 64, n, k, ldx, k, ldo, row_token);
}

// ------------------------------------------------------------------ 32-bit operands with 16-byte rows
// Bound by the FMA pipe from some ten rows on and by reading w below.  A thread owns TM x 8 results: per k it loads TM + 8 values
// from shared memory for TM * 8 multiply-adds (a 16 x 8 thread keeps the shared-memory pipe busy for three quarters of the time
// of its multiply-adds, a 4 x 4 one for twice that time, which bounded the 64 x 64 tile), and issues them as pairs along n
// (fma.rn.f32x2: the same two roundings in one issue slot; 3 to 10 % faster than single ones).  301 x 16448 x 4096: 1746 us as
// 64 x 64 tiles, 1147 us here (35 of 74 TFLOP/s); 301 x 4096 x 14336: 2732 and 1041 us; 16 x 4096 x 4096: 223 and 58 us.  Slabs of 8 k lie transposed in shared memory, two of them, the next
// one on its way in registers.  The CTAs that share a tile's k range are a cluster: each leaves its sums in shared memory and
// adds up its share of the tile over all of them in the order of k, so results do not depend on timing.
__device__ __forceinline__ uint64_t dup_f32x2(float v) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ uint64_t pack_f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack_f32x2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma_f32x2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

template <int TM>
struct F32Tile {
  static constexpr int kBM = 4 * TM, kBN = 256, kBK = 8;
  // pitches of 4 (mod 8) floats: the two k halves that a warp stores for 16 rows fall into different banks
  static constexpr int kPX = kBM + 4, kPW = kBN + 4;
  static constexpr int kStage = kBK * (kPX + kPW);
  static constexpr int kOut = kBM * kBN;
  static constexpr int smem_bytes(int splits) {
    return 4 * (splits > 1 && kOut > 2 * kStage ? kOut : 2 * kStage);
  }
};

template <int TM, int OCC>
__global__ void __launch_bounds__(128, OCC)
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out, int m, int n, int k,
                long long ldx, long long ldw, long long ldo, int splits) {
  using T = F32Tile<TM>;
  extern __shared__ __align__(16) float sm[];
  const int rank = blockIdx.x % splits;
  const int n0 = (blockIdx.x / splits) * T::kBN, m0 = blockIdx.y * T::kBM;
  const int slabs = (k + T::kBK - 1) / T::kBK;
  const int s0 = int((long long)slabs * rank / splits), s1 = int((long long)slabs * (rank + 1) / splits);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int row4 = (lane >> 3) * 4, col4 = warp * 64 + (lane & 7) * 4;
  const int lq = (t & 1) * 4, lr = t >> 1;               // loader: first of four k, row

  uint64_t acc[TM][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;

  const bool x_on = lr < T::kBM;
  const float* xp = x + (long long)min(m0 + lr, m - 1) * ldx;
  const float* wp[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) wp[i] = w + (long long)min(n0 + lr + 64 * i, n - 1) * ldw;
  float4 rx = make_float4(0.f, 0.f, 0.f, 0.f), rw[4];
  // rows beyond the operand repeat its last row and are not stored; k beyond the end is zero on both sides
  auto fetch = [&](int s) {
    const int kk = s * T::kBK + lq;
    const bool in = kk < k;
    if (x_on) rx = in ? *reinterpret_cast<const float4*>(xp + kk) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) rw[i] = in ? __ldg(reinterpret_cast<const float4*>(wp[i] + kk)) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  auto store = [&](float* st) {
    if (x_on) {
      float* d = st + lq * T::kPX + lr;
      d[0] = rx.x; d[T::kPX] = rx.y; d[2 * T::kPX] = rx.z; d[3 * T::kPX] = rx.w;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float* d = st + T::kBK * T::kPX + lq * T::kPW + lr + 64 * i;
      d[0] = rw[i].x; d[T::kPW] = rw[i].y; d[2 * T::kPW] = rw[i].z; d[3 * T::kPW] = rw[i].w;
    }
  };

  griddep_wait();
  griddep_launch();
  if (s0 < s1) {
    fetch(s0);
    store(sm);
  }
  __syncthreads();
  for (int s = s0; s < s1; ++s) {
    const float* xs = sm + ((s - s0) & 1) * T::kStage;
    const float* ws = xs + T::kBK * T::kPX;
    if (s + 1 < s1) fetch(s + 1);
#pragma unroll
    for (int kk = 0; kk < T::kBK; ++kk) {
      const float4 b0 = *reinterpret_cast<const float4*>(ws + kk * T::kPW + col4);
      const float4 b1 = *reinterpret_cast<const float4*>(ws + kk * T::kPW + col4 + 32);
      const uint64_t b[4] = {pack_f32x2(b0.x, b0.y), pack_f32x2(b0.z, b0.w), pack_f32x2(b1.x, b1.y), pack_f32x2(b1.z, b1.w)};
#pragma unroll
      for (int g = 0; g < TM / 4; ++g) {
        const float4 a4 = *reinterpret_cast<const float4*>(xs + kk * T::kPX + g * 16 + row4);
        const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint64_t a = dup_f32x2(av[i]);
#pragma unroll
          for (int j = 0; j < 4; ++j) fma_f32x2(acc[g * 4 + i][j], a, b[j]);
        }
      }
    }
    if (s + 1 < s1) store(sm + ((s + 1 - s0) & 1) * T::kStage);
    __syncthreads();
  }

  const bool vec = ((ldo | n) & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  auto put = [&](int r, int c, float4 v) {
    if (r >= m || c >= n) return;
    float* o = out + (long long)r * ldo + c;
    if (vec) {
      *reinterpret_cast<float4*>(o) = v;
      return;
    }
    o[0] = v.x;
    if (c + 1 < n) o[1] = v.y;
    if (c + 2 < n) o[2] = v.z;
    if (c + 3 < n) o[3] = v.w;
  };
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float2 u = unpack_f32x2(acc[i][2 * h]), v = unpack_f32x2(acc[i][2 * h + 1]);
      const int r = (i >> 2) * 16 + row4 + (i & 3), c = col4 + 32 * h;
      if (splits == 1)
        put(m0 + r, n0 + c, make_float4(u.x, u.y, v.x, v.y));
      else
        *reinterpret_cast<float4*>(sm + r * T::kBN + c) = make_float4(u.x, u.y, v.x, v.y);
    }
  if (splits == 1) return;
  cluster_sync_all();
  constexpr int kVecs = T::kOut / 4;
  for (int e = rank * 128 + t; e < kVecs; e += splits * 128) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int p = 0; p < splits; ++p) {
      const float4 u = ld_cluster_f4(map_to_cta(sm + 4 * e, p));
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    put(m0 + e / (T::kBN / 4), n0 + (e % (T::kBN / 4)) * 4, v);
  }
  cluster_sync_all();                                   // no CTA leaves while its sums are read
}

template <int TM, int OCC>
static int launch_f32(const float* x, const float* w, float* out, int m, int n, int k, long long ldx, long long ldw,
                      long long ldo, int splits, cudaStream_t s) {
  using T = F32Tile<TM>;
  const int smem = T::smem_bytes(splits);
  static const cudaError_t attr = cudaFuncSetAttribute(gemm_f32_kernel<TM, OCC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       T::smem_bytes(2));
  if (attr != cudaSuccess) return int(attr);
  return launch_pdl_cluster(gemm_f32_kernel<TM, OCC>, dim3((n + T::kBN - 1) / T::kBN * splits, (m + T::kBM - 1) / T::kBM), dim3(128),
                            smem, s, splits, x, w, out, m, n, k, ldx, ldw, ldo, splits);
}

static int gemm_f32(const float* x, const float* w, float* out, int m, int n, int k, long long ldx, long long ldw, long long ldo,
                    cudaStream_t s) {
  // Rows per tile and split of k by the time of the fullest SM: its CTAs (2, 3 or 4 are resident; an incomplete round of them
  // hides less of its loads), times the rows of a tile, over the splits; a split costs an exchange, and a thread with few rows
  // loads more per multiply-add.  Constants fitted to 4096 x 4096, 14336 x 4096, 16448 x 4096 and 4096 x 14336 at 16 to 301
  // rows; the choice is within 8 % of the best of all (rows, splits) there.
  const int tiles_n = (n + 255) / 256;
  int best_tm = 16, best_s = 1;
  float best = 1e30f;
  for (int tm : {4, 8, 16}) {
    const int resident = tm == 16 ? 2 : (tm == 8 ? 3 : 4);
    const long long tiles = (long long)tiles_n * ((m + 4 * tm - 1) / (4 * tm));
    for (int sp = 1; sp <= 8; ++sp) {
      if (sp > 1 && k / sp < 256) break;
      const long long per_sm = (tiles * sp + 147) / 148;
      const float cost = (float(per_sm) + (per_sm % resident ? 0.4f : 0.f)) * float(4 * tm) * (tm == 4 ? 1.6f : 1.f) / sp *
                         (1.f + 0.02f * sp);
      if (cost < best) best = cost, best_tm = tm, best_s = sp;
    }
  }
  if (best_tm == 16) return launch_f32<16, 2>(x, w, out, m, n, k, ldx, ldw, ldo, best_s, s);
  if (best_tm == 8) return launch_f32<8, 3>(x, w, out, m, n, k, ldx, ldw, ldo, best_s, s);
  return launch_f32<4, 4>(x, w, out, m, n, k, ldx, ldw, ldo, best_s, s);
}

template <typename XT, typename WT, typename OT>
static int launch_simt(const void* x, const void* w, void* out, int m, int n, int k, long long ldx, long long ldw,
                       long long ldo, cudaStream_t s) {
  return launch_pdl(gemm_simt_kernel<XT, WT, OT>, dim3((n + 63) / 64, (m + 63) / 64), dim3(256), 0, s,
                    reinterpret_cast<const XT*>(x), reinterpret_cast<const WT*>(w), reinterpret_cast<OT*>(out), m, n, k,
                    ldx, ldw, ldo);
}
template <typename XT, typename WT, typename OT>
static int launch_simt_grouped(const void* x, const void* w, void* out, const int* offsets, const int* row_token,
                               int groups, int max_rows, int n, int k, long long ldx, long long ldo, cudaStream_t s) {
  return launch_pdl(gemm_simt_grouped_kernel<XT, WT, OT>, dim3((n + 63) / 64, (max_rows + 63) / 64, groups), dim3(256), 0, s,
                    reinterpret_cast<const XT*>(x), reinterpret_cast<const WT*>(w), reinterpret_cast<OT*>(out), offsets,
                    row_token, n, k, ldx, ldo);
}

}  // namespace nkb

using namespace nkb;

extern "C" int nkb_gemm_simt(const void* x, int x_bf16, const void* w, int w_bf16, void* out, int out_bf16, int m, int n,
                             int k, long long ldx, long long ldw, long long ldo, void* stream) {
  if (m <= 0 || n <= 0) return 0;
  if (k <= 0 || (m + 63) / 64 > 65535) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  using bf = __nv_bfloat16;
  if (!x_bf16 && !w_bf16 && !out_bf16) {
    const bool rows16 = ((k | ldx | ldw) & 3) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
    if (rows16)
      return gemm_f32(reinterpret_cast<const float*>(x), reinterpret_cast<const float*>(w), reinterpret_cast<float*>(out), m, n, k,
                      ldx, ldw, ldo, s);
    return launch_simt<float, float, float>(x, w, out, m, n, k, ldx, ldw, ldo, s);
  }
  if (x_bf16 && w_bf16 && !out_bf16) return launch_simt<bf, bf, float>(x, w, out, m, n, k, ldx, ldw, ldo, s);
  if (x_bf16 && w_bf16 && out_bf16) return launch_simt<bf, bf, bf>(x, w, out, m, n, k, ldx, ldw, ldo, s);
  return -2;
}

// Rows sorted by group; row_token (may be null) names the row of x behind each sorted row.  w [groups, n, k].
extern "C" int nkb_gemm_simt_grouped(const void* x, int x_bf16, const void* w, int w_bf16, void* out, int out_bf16,
                                     const int* offsets, const int* row_token, int groups, int max_rows, int n, int k,
                                     long long ldx, long long ldo, void* stream) {
  if (groups <= 0 || max_rows <= 0 || n <= 0) return 0;
  if (k <= 0 || (max_rows + 63) / 64 > 65535 || groups > 65535) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  using bf = __nv_bfloat16;
  if (!x_bf16 && !w_bf16 && !out_bf16)
    return launch_simt_grouped<float, float, float>(x, w, out, offsets, row_token, groups, max_rows, n, k, ldx, ldo, s);
  if (x_bf16 && w_bf16 && !out_bf16)
    return launch_simt_grouped<bf, bf, float>(x, w, out, offsets, row_token, groups, max_rows, n, k, ldx, ldo, s);
  if (x_bf16 && w_bf16 && out_bf16)
    return launch_simt_grouped<bf, bf, bf>(x, w, out, offsets, row_token, groups, max_rows, n, k, ldx, ldo, s);
  return -2;
}
