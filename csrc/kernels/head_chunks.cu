// Prompts of the recurrences with one decay per head (head_recurrence.h), sixteen tokens at a time on the matrix units.
//
// With G_t the product of the chunk's decays up to token t, R_tj = G_t / G_j, w_t the write strength and raw keys k (whose unit
// norms are factors i_t of the numbers below), the chunk's tokens obey
//
//     u_t = w_t i_t v_t - w_t i_t^2 (G_t S_0^T k_t + sum_(j<t) R_tj (k_t . k_j) u_j),   so   u = (1 + A)^-1 b
//     o_t = s_t (G_t S_0^T q_t + sum_(j<=t) R_tj (q_t . k_j) u_j)
//     S   = G_15 S_0 + sum_j k_j (R_15,j u_j)^T
//
// A, its inverse and P_tj = s_t R_tj (q_t . k_j) do not depend on the state: four warps prepare them chunks ahead.  A warp of the
// others owns 16 columns of the state for all tokens, transposed ([column][channel]) in the accumulator layout of m16n8k16, which
// is also its A layout: S^T k, u, o and the update pass from product to product in registers, and the warps meet only at the
// chunks' barriers.  The state-space form has u = dt v and neither A nor S^T k.
//
// 32-bit numbers enter products as three bf16 parts (24 bits, taken off by truncation, so exact): with bf16 keys and queries
// three part products are exact; of the nine of two 32-bit numbers all but the last are taken (it is below 2^-28 of a product: a second
// part is up to 2^-7 of a number, a third 2^-14; without the two before it a product was good to 2^-20).  Tensor cores cut off a sum's last bits where fp32 units round: no chain is longer than two steps
// of leading parts, the decayed state never is an accumulator, and 1 + A has its diagonal outside the product.
//
// Bound by issue: of the 4130 clocks a chunk of 128 x 128 takes with the delta rule, 2690 are products (8 clocks each and SM quarter).
// Code is kept small: with the preparation unrolled the two kinds of warps pushed one another out of the instruction cache
// (4 x 2048 tokens of 32 heads 585 us, rolled up 329; token by token 1317).
//
// A number that is not three bf16 parts, because it is infinite, NaN or too small (below 2^-110 a third part may lie under bf16's
// smallest number, 2^-133), leaves bits behind a third part.  A chunk with one in its state, u, A, P or 32-bit keys and queries is
// computed token by token in fp32: infinities and NaN go where they do in the recurrence, and what is tiny keeps its bits.  Only
// where the chunk's own decays multiply to less than 2^-40, what they make tiny loses bits below 2^-133.
#include "common.cuh"
#include "proj_src.cuh"
#include "mma_frag.cuh"
#include "head_recurrence.h"
#include "head_chunks.h"
#include "api.h"

namespace nkb {
namespace {

constexpr int kTok = 16, kPrep = 4;
constexpr int kMatPitch = 48;                          // bytes of a row of a 16 x 16 matrix of bf16, free of bank conflicts

template <int DK, int MW, typename T>
struct Chunk {
  static constexpr bool F32 = sizeof(T) == 4;
  static constexpr int PL = F32 ? 3 : 1;               // bf16 planes of keys and queries
  static constexpr int COLS = 16 * MW, THREADS = 32 * (MW + kPrep);
  static constexpr int NST = F32 || MW == 8 ? 6 : 8;
  static constexpr int KP = DK * 2 + 16, KPLANE = kTok * KP;                    // pitch of a row of keys, a plane
  static constexpr int VP = F32 ? (COLS + 4) * 4 : COLS * 2 + 16;
  static constexpr int oQ = PL * KPLANE, oV = 2 * PL * KPLANE, oT = oV + kTok * VP, oP = oT + 3 * kTok * kMatPitch;
  static constexpr int oF = oP + 3 * kTok * kMatPitch, STAGE = oF + 8 * 16 * 4;
  static constexpr int SP = 20;                        // pitch of the fp32 scratch matrices
  static constexpr int SCRATCH = 2 * kTok * SP * 4;
  static constexpr int oScratch = NST * STAGE, oOut = oScratch + kPrep * SCRATCH, SMEM = oOut + MW * kTok * 48;
};
constexpr float kFaded = 0x1p-40f;
// rows of a stage's factors
enum { F_EV = 0, F_EPG = 1, F_IQG = 2, F_D = 3, F_G = 4, F_EP = 5, F_IQ = 6, F_GC = 7 };  // F_GC: the chunk's decay, then (a whole number) whether it lost bits

struct ChunkParams {
  NkbHeadRec r;
  int* status;
};

__device__ __forceinline__ void hc_cp16(void* dst, const void* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}
// a warp goes on, or gives up, as a whole: matrix instructions and shuffles follow
__device__ __forceinline__ bool hc_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  const bool ok = mbar_wait(bar, parity, abort_flag, status, code);
  return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ float high_part(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
// the upper halves of two words
__device__ __forceinline__ uint32_t pack_high(float lo, float hi) {
  return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
}
// what two parts leave of a number; its lower half is not zero where it is no bf16 number
__device__ __forceinline__ float third_part(float x) {
  const float r = x - high_part(x);
  return r - high_part(r);
}
// two numbers as three pairs of bf16 that add up to them
__device__ __forceinline__ void split3(float x, float y, uint32_t& a, uint32_t& b, uint32_t& c) {
  a = pack_high(x, y);
  b = pack_high(x - high_part(x), y - high_part(y));
  c = pack_high(third_part(x), third_part(y));
}
// unless the lower half of `lost` is set (at once: left to itself, the compiler keeps all third parts to the end and spills)
__device__ __forceinline__ void split3(float x, float y, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& lost) {
  const float xt = third_part(x), yt = third_part(y);
  split3(x, y, a, b, c);
  asm volatile("lop3.b32 %0, %0, %1, %2, 0xfe;" : "+r"(lost) : "r"(__float_as_uint(xt)), "r"(__float_as_uint(yt)));
}
// a 16 x 16 tile in accumulator layout as three A operands
template <typename... Lost>
__device__ __forceinline__ void split_tile(const float (&x)[4], const float (&y)[4], uint32_t (&p)[3][4], Lost&... lost) {
  split3(x[0], x[1], p[0][0], p[1][0], p[2][0], lost...);
  split3(x[2], x[3], p[0][1], p[1][1], p[2][1], lost...);
  split3(y[0], y[1], p[0][2], p[1][2], p[2][2], lost...);
  split3(y[2], y[3], p[0][3], p[1][3], p[2][3], lost...);
}
__device__ __forceinline__ void zero4(float (&x)[4]) { x[0] = x[1] = x[2] = x[3] = 0.f; }
__device__ __forceinline__ void add4(float (&x)[4], const float (&y)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) x[e] += y[e];
}

// the same product as mma_16816, free to move between the others
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Part products of a 16 x 16 tile in three parts and a 16 x 16 matrix in three planes, the smallest first; product i of eight.
constexpr int kPartProducts = 8;
__device__ __forceinline__ void part_product(int i, float (&acc)[2][4], const uint32_t (&a)[3][4], const uint32_t (&m)[3][4]) {
  const int order = i < 2 ? 3 : (i < 5 ? 2 : (i < 7 ? 1 : 0)), j = i < 2 ? i + 1 : (i < 5 ? i - 2 : (i < 7 ? i - 5 : 0));
  mma_bf16(acc[0], a[order - j], m[j][0], m[j][1]);
  mma_bf16(acc[1], a[order - j], m[j][2], m[j][3]);
}
__device__ __forceinline__ void load_planes(uint32_t (&m)[3][4], uint32_t addr) {
#pragma unroll
  for (int j = 0; j < 3; ++j) ldsm_x4(addr + j * kTok * kMatPitch, m[j][0], m[j][1], m[j][2], m[j][3]);
}
// Sums over DK channels of a state's 16 columns times the chunk's keys (KEYS) and queries: the leading parts' sums in `hi`, two steps
// of 16 channels at a time, the others' in `lo`.  Rows and parts of the next step are on their way during a step.
template <int DK, int PL, bool KEYS, int PLANE>
__device__ __forceinline__ void state_products(const float (&S)[DK / 8][4], uint32_t rows, uint32_t q_ofs, float (&hi)[2][2][4],
                                               float (&lo)[2][2][4], uint32_t& lost) {
  constexpr int STEPS = DK / 16, W0 = KEYS ? 0 : 1;     // [0]: keys, [1]: queries
  constexpr int RUN = 2;                                // steps of a chain of leading parts
  float run[2][2][4];
  uint32_t a[2][3][4], m[2][2][PL][4];
#pragma unroll
  for (int w = W0; w < 2; ++w)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      zero4(hi[w][h]);
      zero4(lo[w][h]);
    }
  const auto load = [&](int i) {
#pragma unroll
    for (int w = W0; w < 2; ++w)
#pragma unroll
      for (int j = 0; j < PL; ++j) {
        uint32_t(&z)[4] = m[i & 1][w][j];
        ldsm_x4(rows + w * q_ofs + j * PLANE + i * 32, z[0], z[1], z[2], z[3]);
      }
  };
  load(0);
  split_tile(S[0], S[1], a[0], lost);
#pragma unroll
  for (int i = 0; i < STEPS; ++i) {
    const uint32_t(&x)[3][4] = a[i & 1];
    if (i + 1 < STEPS) load(i + 1);
#pragma unroll
    for (int w = W0; w < 2; ++w)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t(&y)[PL][4] = m[i & 1][w];
        if (i % RUN == 0) zero4(run[w][h]);
        mma_bf16(run[w][h], x[0], y[0][2 * h], y[0][2 * h + 1]);
      }
    if (i + 1 < STEPS) split_tile(S[(2 * i + 2) % (DK / 8)], S[(2 * i + 3) % (DK / 8)], a[(i + 1) & 1], lost);
#pragma unroll
    for (int order = PL > 1 ? 3 : 2; order >= 1; --order)
#pragma unroll
      for (int j = 0; j < PL; ++j)
        if (order - j >= 0 && order - j < 3) {
#pragma unroll
          for (int w = W0; w < 2; ++w)
#pragma unroll
            for (int h = 0; h < 2; ++h) mma_bf16(lo[w][h], x[order - j], m[i & 1][w][j][2 * h], m[i & 1][w][j][2 * h + 1]);
        }
    if (i % RUN == RUN - 1) {
#pragma unroll
      for (int w = W0; w < 2; ++w)
#pragma unroll
        for (int h = 0; h < 2; ++h) add4(hi[w][h], run[w][h]);
    }
  }
}

// MW warps of 16 columns, four warps that prepare.
template <int DK, int MW, bool DELTA, typename T>
__global__ void __launch_bounds__(Chunk<DK, MW, T>::THREADS, 1) head_chunk_kernel(const __grid_constant__ ChunkParams cp) {
  using C = Chunk<DK, MW, T>;
  constexpr int PL = C::PL, NST = C::NST, COLS = C::COLS;
  constexpr bool F32 = C::F32;
  const NkbHeadRec& p = cp.r;
  extern __shared__ __align__(128) uint8_t sm[];
  __shared__ uint64_t full[NST], empty[NST];
  __shared__ int abort_flag;
  const int warp = warp_idx_uniform(), lane = lane_id();
  const int head = blockIdx.y, b = blockIdx.z, col0 = blockIdx.x * COLS;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NST; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], MW);
    }
    abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  griddep_wait();
  griddep_launch();
  const int n = p.q_lens[b], ctx = p.context_lens[b];
  if (n <= 0 || ctx < n) return;
  const long long row0 = p.q_start[b];
  const int chunks = (n + kTok - 1) / kTok;
  const T* x = reinterpret_cast<const T*>(p.x.ptr);

  if (warp >= MW) {
    if constexpr (MW == 8) asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
    // ---------------------------------------------------------------- chunks ahead: operands, factors, inverses
    const int kvh = head / (p.heads / p.groups);
    const int hq = p.q_col + kvh * p.dim, hk = p.k_col + kvh * p.dim, hv = p.v_col + head * p.vdim;
    const float rate = p.rate[head], dtb = p.dt_bias[head];
    float* mk = reinterpret_cast<float*>(sm + C::oScratch + (warp - MW) * C::SCRATCH);     // k.k, then A
    float* mq = mk + kTok * C::SP;                                                         // q.k
    for (int c = warp - MW; c < chunks; c += kPrep) {
      uint8_t* s = sm + c % NST * C::STAGE;
      const int t0 = c * kTok;
      if (!hc_wait(&empty[c % NST], ((c / NST) & 1) ^ 1u, &abort_flag, cp.status, ERR_WAIT_SMEM_EMPTY)) return;
      float a_raw = 0.f, b_raw = 0.f;
      uint32_t lost = 0;
      if (lane < kTok && t0 + lane < n) {
        a_raw = proj_load(p.a, row0 + t0 + lane, head);
        if (DELTA) b_raw = proj_load(p.b, row0 + t0 + lane, head);
      }
      if constexpr (!F32) {
        constexpr int KT = 256 / DK, VT = 256 / COLS;              // tokens that a warp fetches at a time
        {
          int tok = lane / (DK / 8);
          const int ch = lane % (DK / 8) * 8;
          uint8_t* d = s + tok * C::KP + ch * 2;
          const T* row = x + (row0 + t0 + tok) * p.x.ld + ch;
#pragma unroll 2
          for (int i = 0; i < kTok / KT; ++i, tok += KT, d += KT * C::KP, row += KT * p.x.ld) {
            const bool on = t0 + tok < n && ch < p.dim;
            hc_cp16(d, on ? row + hk : x, on);
            hc_cp16(d + C::oQ, on ? row + hq : x, on);
          }
        }
        int tok = lane / (COLS / 8);
        const int ch = lane % (COLS / 8) * 8;
        uint8_t* d = s + C::oV + tok * C::VP + ch * 2;
        const T* row = x + (row0 + t0 + tok) * p.x.ld + hv + col0 + ch;
#pragma unroll 2
        for (int i = 0; i < kTok / VT; ++i, tok += VT, d += VT * C::VP, row += VT * p.x.ld) {
          const bool on = t0 + tok < n && col0 + ch < p.vdim;
          hc_cp16(d, on ? row : x, on);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
      } else {
#pragma unroll 2
        for (int i = 0; i < kTok * COLS / 128; ++i) {
          const int idx = lane + i * 32, tok = idx / (COLS / 4), ch = idx % (COLS / 4) * 4;
          const bool on = t0 + tok < n && col0 + ch < p.vdim;
          hc_cp16(s + C::oV + tok * C::VP + ch * 4, x + (on ? row0 + t0 + tok : row0) * p.x.ld + hv + (on ? col0 + ch : 0), on);
        }
#pragma unroll 2
        for (int i = 0; i < kTok * DK / 128; ++i) {
          const int idx = lane + i * 32, tok = idx / (DK / 4), ch = idx % (DK / 4) * 4;
          const bool on = t0 + tok < n && ch < p.dim;
          float4 k4 = make_float4(0.f, 0.f, 0.f, 0.f), q4 = k4;
          if (on) {
            const T* row = x + (row0 + t0 + tok) * p.x.ld;
            k4 = *reinterpret_cast<const float4*>(row + hk + ch);
            q4 = *reinterpret_cast<const float4*>(row + hq + ch);
          }
          uint32_t u[3], w[3];
          uint8_t* d = s + tok * C::KP + ch * 2;
          split3(k4.x, k4.y, u[0], u[1], u[2], lost);
          split3(k4.z, k4.w, w[0], w[1], w[2], lost);
#pragma unroll
          for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(d + j * C::KPLANE) = make_uint2(u[j], w[j]);
          split3(q4.x, q4.y, u[0], u[1], u[2], lost);
          split3(q4.z, q4.w, w[0], w[1], w[2], lost);
#pragma unroll
          for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(d + C::oQ + j * C::KPLANE) = make_uint2(u[j], w[j]);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
      }
      __syncwarp();

      // products of keys with keys, of queries with keys and (their diagonal only) of queries with queries
      float qq;
      {
        constexpr int W0 = DELTA ? 0 : 1, W1 = DELTA ? 3 : 2, RUN = 2;
        float hi[3][2][4], lo[3][2][4], run[3][2][4];
#pragma unroll
        for (int w = 0; w < 3; ++w)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            zero4(hi[w][h]);
            zero4(lo[w][h]);
          }
        const uint32_t at = smem_u32(s) + ((lane & 7) + ((lane >> 3) & 1) * 8) * C::KP + (lane >> 4) * 16;
#pragma unroll 1
        for (int i0 = 0; i0 < DK / 16; i0 += RUN) {
#pragma unroll
          for (int w = W0; w < W1; ++w)
#pragma unroll
            for (int h = 0; h < 2; ++h) zero4(run[w][h]);
#pragma unroll
          for (int i = 0; i < RUN; ++i) {
            uint32_t ka[PL][4], qa[PL][4];
#pragma unroll
            for (int j = 0; j < PL; ++j) {
              ldsm_x4(at + j * C::KPLANE + (i0 + i) * 32, ka[j][0], ka[j][1], ka[j][2], ka[j][3]);
              ldsm_x4(at + C::oQ + j * C::KPLANE + (i0 + i) * 32, qa[j][0], qa[j][1], qa[j][2], qa[j][3]);
            }
#pragma unroll
            for (int order = PL > 1 ? 3 : 0; order >= 0; --order)
#pragma unroll
              for (int j = 0; j < PL; ++j)
                if (order - j >= 0 && order - j < PL) {
#pragma unroll
                  for (int w = W0; w < W1; ++w)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                      const uint32_t(&l)[4] = w == 0 ? ka[order - j] : qa[order - j];
                      const uint32_t(&r)[4] = w == 2 ? qa[j] : ka[j];
                      mma_bf16(order ? lo[w][h] : run[w][h], l, r[h], r[2 + h]);
                    }
                }
          }
#pragma unroll
          for (int w = W0; w < W1; ++w)
#pragma unroll
            for (int h = 0; h < 2; ++h) add4(hi[w][h], run[w][h]);
        }
        if (PL > 1) {
#pragma unroll
          for (int w = W0; w < W1; ++w)
#pragma unroll
            for (int h = 0; h < 2; ++h) add4(hi[w][h], lo[w][h]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int o = (lane >> 2) * C::SP + h * 8 + (lane & 3) * 2;
          if (DELTA) {
            *reinterpret_cast<float2*>(mk + o) = make_float2(hi[0][h][0], hi[0][h][1]);
            *reinterpret_cast<float2*>(mk + o + 8 * C::SP) = make_float2(hi[0][h][2], hi[0][h][3]);
          }
          *reinterpret_cast<float2*>(mq + o) = make_float2(hi[1][h][0], hi[1][h][1]);
          *reinterpret_cast<float2*>(mq + o + 8 * C::SP) = make_float2(hi[1][h][2], hi[1][h][3]);
        }
        // token t's own product: lane (t % 8) * 4 + (t % 8) / 2, element t % 2 of the tile's diagonal block
        const int from = (lane & 7) * 4 + ((lane & 7) >> 1);
        const float d0 = __shfl_sync(0xffffffffu, hi[2][0][0], from), d1 = __shfl_sync(0xffffffffu, hi[2][0][1], from);
        const float d2 = __shfl_sync(0xffffffffu, hi[2][1][2], from), d3 = __shfl_sync(0xffffffffu, hi[2][1][3], from);
        qq = lane & 8 ? (lane & 1 ? d3 : d2) : (lane & 1 ? d1 : d0);
      }
      __syncwarp();

      // factors; tokens past the end keep the state and write nothing
      float* f = reinterpret_cast<float*>(s + C::oF);
      if (lane < kTok) {
        float g = 1.f, ev = 0.f, ep = 0.f, iq = 0.f;
        if (t0 + lane < n) {
          const float z = a_raw + dtb, dt = fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));
          g = expf(-rate * dt);
          if (DELTA) {
            const float ik = 1.f / sqrtf(mk[lane * C::SP + lane] + p.unit_eps);
            iq = p.q_scale / sqrtf(qq + p.unit_eps);
            ev = ik / (1.f + expf(-b_raw));
            ep = ev * ik;
          } else {
            ev = dt;
            iq = p.q_scale;
          }
        }
        f[F_EV * 16 + lane] = ev;
        f[F_G * 16 + lane] = g;
        f[F_EP * 16 + lane] = ep;
        f[F_IQ * 16 + lane] = iq;
      }
      __syncwarp();
      // lane j < 16: column j of A, decay from token j to the end and up to token j; lane 16 + j: column j of P
      {
        const int j = lane & 15;
        const bool left = lane < 16;
        float* col = (left ? mk : mq) + j;
        const float* scale = f + (left ? F_EP : F_IQ) * 16;
        float r = 1.f, up = 1.f;
#pragma unroll 1
        for (int t4 = 0; t4 < kTok; t4 += 4) {
          const float4 g4 = *reinterpret_cast<const float4*>(f + F_G * 16 + t4), s4 = *reinterpret_cast<const float4*>(scale + t4);
          const float g[4] = {g4.x, g4.y, g4.z, g4.w}, sc[4] = {s4.x, s4.y, s4.z, s4.w};
          float v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = DELTA || !left ? col[(t4 + e) * C::SP] : 0.f;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int t = t4 + e;
            if (t > j) r *= g[e];
            if (t <= j) up *= g[e];
            if (DELTA || !left) col[t * C::SP] = t > j || (!left && t == j) ? sc[e] * r * v[e] : 0.f;
          }
        }
        if (left) {
          f[F_D * 16 + j] = r;
          f[F_EPG * 16 + j] = f[F_EP * 16 + j] * up;
          f[F_IQG * 16 + j] = f[F_IQ * 16 + j] * up;
          if (j == kTok - 1) f[F_GC * 16] = up;
        }
      }
      __syncwarp();
      // column j of (1 + A)^-1 without its diagonal
      if constexpr (DELTA) {
        const int j = lane & 15;
        float inv[kTok];
#pragma unroll
        for (int t = 0; t < kTok; ++t) {
          float r = 0.f;
#pragma unroll
          for (int i4 = 0; i4 < t; i4 += 4) {
            const float4 a4 = *reinterpret_cast<const float4*>(mk + t * C::SP + i4);
            r = fmaf(a4.x, inv[i4], r);
            if (i4 + 1 < t) r = fmaf(a4.y, inv[i4 + 1], r);
            if (i4 + 2 < t) r = fmaf(a4.z, inv[i4 + 2], r);
            if (i4 + 3 < t) r = fmaf(a4.w, inv[i4 + 3], r);
          }
          inv[t] = t == j ? 1.f : (t > j ? -r : 0.f);
        }
        __syncwarp();
        if (lane < kTok) {
#pragma unroll
          for (int t = 0; t < kTok; ++t) mk[t * C::SP + j] = t > j ? inv[t] : 0.f;
        }
        __syncwarp();
      }
      // both in parts, a pair of columns at a time; an infinite key or query shows on the diagonal of P
      uint32_t small = 0;
#pragma unroll 1
      for (int i = lane; i < kTok * 8; i += 32) {
        const int t = i >> 3, j2 = (i & 7) * 2;
        uint8_t* d = s + C::oT + t * kMatPitch + j2 * 2;
        uint32_t w[3];
        if (DELTA) {
          const float2 y = *reinterpret_cast<const float2*>(mk + t * C::SP + j2);
          split3(y.x, y.y, w[0], w[1], w[2], small);
#pragma unroll
          for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(d + k * kTok * kMatPitch) = w[k];
        }
        const float2 y = *reinterpret_cast<const float2*>(mq + t * C::SP + j2);
        split3(y.x, y.y, w[0], w[1], w[2], small);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(d + (C::oP - C::oT) + k * kTok * kMatPitch) = w[k];
      }
      // (all exponent bits: not finite, or such a large one beside a small one)
      if (!(f[F_GC * 16] < kFaded) || (small & 0x7f800000u) == 0x7f800000u) lost |= small;
      lost = __any_sync(0xffffffffu, (lost & 0xffffu) != 0);
      if (lane == 0) f[F_GC * 16 + 1] = __uint_as_float(lost ? 1u : 0u);
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[c % NST]);
    }
    return;
  }

  // ------------------------------------------------------------------ 16 columns of the state
  if constexpr (MW == 8) asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
  constexpr int NT = DK / 8;
  const int slot = p.slot_ids ? p.slot_ids[b] : b, gr = lane >> 2, q2 = (lane & 3) * 2;
  const int cw = warp * 16, ca = col0 + cw + gr;                   // first column of the warp within the CTA, this lane's first of two
  const float skip = !DELTA && p.skip ? p.skip[head] : 0.f;
  float* st = p.state + (((long long)slot * p.heads + head) * p.vdim + ca) * p.dim + q2;
  T* out = reinterpret_cast<T*>(p.out) + (row0 * p.heads + head) * p.vdim + col0 + cw;
  const long long out_ld = (long long)p.heads * p.vdim;
  const bool fresh = ctx == n, ok0 = ca < p.vdim, ok1 = ca + 8 < p.vdim;
  float S[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    float2 u = make_float2(0.f, 0.f), w = u;
    if (!fresh && i * 8 < p.dim) {
      if (ok0) u = *reinterpret_cast<const float2*>(st + i * 8);
      if (ok1) w = *reinterpret_cast<const float2*>(st + 8 * p.dim + i * 8);
    }
    S[i][0] = u.x; S[i][1] = u.y; S[i][2] = w.x; S[i][3] = w.y;
  }
  // places of this lane's rows for ldmatrix: tokens as columns of a product, and tokens summed over
  const int at_n = ((lane & 7) + (lane >> 4) * 8) * C::KP + ((lane >> 3) & 1) * 16;
  const int at_k = ((lane & 7) + ((lane >> 3) & 1) * 8) * C::KP + (lane >> 4) * 16;
  const int at_m = ((lane & 7) + (lane >> 4) * 8) * kMatPitch + ((lane >> 3) & 1) * 16;

#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    const uint8_t* s = sm + c % NST * C::STAGE;
    const float* f = reinterpret_cast<const float*>(s + C::oF);
    const uint32_t base = smem_u32(s);
    const int left = n - c * kTok;                                 // tokens from here on
    if (!hc_wait(&full[c % NST], (c / NST) & 1, &abort_flag, cp.status, ERR_WAIT_SMEM_FULL)) return;
    float U[2][4], O[2][4], v[2][4];
    uint32_t lost = __float_as_uint(f[F_GC * 16 + 1]);
    if constexpr (F32) {
      const float* vr = reinterpret_cast<const float*>(s + C::oV) + cw + gr;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e) v[h][e] = vr[(h * 8 + q2 + (e & 1)) * (C::VP / 4) + (e >> 1) * 8];
    } else {
      uint32_t r[4];
      ldsm_x4_t(base + C::oV + ((lane & 7) + (lane >> 4) * 8) * C::VP + cw * 2 + ((lane >> 3) & 1) * 16, r[0], r[1], r[2], r[3]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 w = unpack_bf16x2(r[e]);
        v[e >> 1][(e & 1) * 2] = w.x;
        v[e >> 1][(e & 1) * 2 + 1] = w.y;
      }
    }
    {
      float hi[2][2][4], lo[2][2][4];
      state_products<DK, PL, DELTA, C::KPLANE>(S, base + at_n, C::oQ, hi, lo, lost);
      // b = w i v - (w i^2 G) S^T k
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float2 ev = *reinterpret_cast<const float2*>(f + F_EV * 16 + h * 8 + q2);
        const float2 eg = *reinterpret_cast<const float2*>(f + F_EPG * 16 + h * 8 + q2);
        const float2 ig = *reinterpret_cast<const float2*>(f + F_IQG * 16 + h * 8 + q2);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          U[h][e] = (e & 1 ? ev.y : ev.x) * v[h][e];
          O[h][e] = (e & 1 ? ig.y : ig.x) * (hi[1][h][e] + lo[1][h][e]);
          if (DELTA) U[h][e] = fmaf(-(e & 1 ? eg.y : eg.x), hi[0][h][e] + lo[0][h][e], U[h][e]);
          else O[h][e] = fmaf(skip, v[h][e], O[h][e]);
        }
      }
    }
    // (1 + A)^-1 b; part products of one order share an accumulator, the two smallest that of the second largest
    if constexpr (DELTA) {
      uint32_t a[3][4], m[3][4];
      float d[3][2][4];
      load_planes(m, base + C::oT + at_m);
      split_tile(U[0], U[1], a, lost);
#pragma unroll
      for (int o = 0; o < 3; ++o)
#pragma unroll
        for (int h = 0; h < 2; ++h) zero4(d[o][h]);
      part_product(0, d[1], a, m);
      part_product(2, d[2], a, m);
      part_product(7, d[0], a, m);
      part_product(1, d[1], a, m);
      part_product(3, d[2], a, m);
      part_product(5, d[1], a, m);
      part_product(4, d[2], a, m);
      part_product(6, d[1], a, m);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        add4(d[1][h], d[2][h]);
        add4(d[0][h], d[1][h]);
        add4(U[h], d[0][h]);
      }
    }
    // u, and decayed to the chunk's end for the state's update
    uint32_t w[3][4], a[3][4];
    split_tile(U[0], U[1], w, lost);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float2 d = *reinterpret_cast<const float2*>(f + F_D * 16 + h * 8 + q2);
#pragma unroll
      for (int e = 0; e < 4; ++e) U[h][e] *= e & 1 ? d.y : d.x;
    }
    const float gc = f[F_GC * 16];
    uint32_t small = 0;
    split_tile(U[0], U[1], a, small);
    if (!(gc < kFaded)) lost |= small;
    if (__any_sync(0xffffffffu, (lost & 0xffffu) != 0)) {
      for (int t = 0; t < min(left, kTok); ++t) {
        float sk0 = 0.f, sk1 = 0.f, sq0 = 0.f, sq1 = 0.f, qk = 0.f;
        const auto two = [&](int at, int col, int i) {
          if constexpr (F32) {                                     // from memory: their parts may have lost bits
            const T* row = x + (row0 + c * kTok + t) * p.x.ld + col + head / (p.heads / p.groups) * p.dim + i * 8 + q2;
            return i * 8 < p.dim ? make_float2(row[0], row[1]) : make_float2(0.f, 0.f);
          } else {
            return unpack_bf16x2(*reinterpret_cast<const uint32_t*>(s + at + t * C::KP + (i * 8 + q2) * 2));
          }
        };
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          const float2 q = two(C::oQ, p.q_col, i), k = two(0, p.k_col, i);
          qk = fmaf(q.x, k.x, fmaf(q.y, k.y, qk));
          sq0 = fmaf(q.x, S[i][0], fmaf(q.y, S[i][1], sq0));
          sq1 = fmaf(q.x, S[i][2], fmaf(q.y, S[i][3], sq1));
          if (DELTA) {
            sk0 = fmaf(k.x, S[i][0], fmaf(k.y, S[i][1], sk0));
            sk1 = fmaf(k.x, S[i][2], fmaf(k.y, S[i][3], sk1));
          }
        }
#pragma unroll
        for (int w = 1; w < 4; w <<= 1) {
          sk0 += __shfl_xor_sync(0xffffffffu, sk0, w);
          sk1 += __shfl_xor_sync(0xffffffffu, sk1, w);
          sq0 += __shfl_xor_sync(0xffffffffu, sq0, w);
          sq1 += __shfl_xor_sync(0xffffffffu, sq1, w);
          qk += __shfl_xor_sync(0xffffffffu, qk, w);
        }
        const T* vr = reinterpret_cast<const T*>(s + C::oV + t * C::VP) + cw + gr;
        const float v0 = cast_in<T>(vr[0]), v1 = cast_in<T>(vr[8]), g = f[F_G * 16 + t], ev = f[F_EV * 16 + t];
        float u0 = ev * v0, u1 = ev * v1;
        if (DELTA) {
          const float es = f[F_EP * 16 + t] * g;
          u0 = fmaf(-es, sk0, u0);
          u1 = fmaf(-es, sk1, u1);
        }
        const float oq = f[F_IQ * 16 + t] * g, ou = f[F_IQ * 16 + t] * qk;
        float o0 = fmaf(oq, sq0, ou * u0), o1 = fmaf(oq, sq1, ou * u1);
        if (!DELTA) {
          o0 = fmaf(skip, v0, o0);
          o1 = fmaf(skip, v1, o1);
        }
        T* o = out + (c * kTok + t) * out_ld + gr;
        if (q2 == 0) {
          if (ok0) o[0] = cast_out<T>(o0);
          if (ok1) o[8] = cast_out<T>(o1);
        }
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          const float2 k = two(0, p.k_col, i);
          S[i][0] = fmaf(k.x, u0, g * S[i][0]);
          S[i][1] = fmaf(k.y, u0, g * S[i][1]);
          S[i][2] = fmaf(k.x, u1, g * S[i][2]);
          S[i][3] = fmaf(k.y, u1, g * S[i][3]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[c % NST]);
      continue;
    }
    // the state's update, and beside it P u
    {
      uint32_t m[3][4];
      float po[2][4];
      load_planes(m, base + C::oP + at_m);
      zero4(po[0]);
      zero4(po[1]);
      // two steps of 16 channels at a time: four tiles whose part products take turns
      uint32_t kb[2][2][PL][4];
      const auto load_keys = [&](int i) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int j = 0; j < PL; ++j) {
            uint32_t(&z)[4] = kb[i & 1][e][j];
            ldsm_x4_t(base + at_k + j * C::KPLANE + (2 * i + e) * 32, z[0], z[1], z[2], z[3]);
          }
      };
      constexpr int STEPS = DK / 32, PER = (kPartProducts + STEPS - 1) / STEPS;
      load_keys(0);
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        if (i + 1 < STEPS) load_keys(i + 1);
        float d[4][4];
#pragma unroll
        for (int h = 0; h < 4; ++h) zero4(d[h]);
#pragma unroll
        for (int order = PL > 1 ? 3 : 2; order >= 0; --order)
#pragma unroll
          for (int j = 0; j < PL; ++j)
            if (order - j >= 0 && order - j < 3) {
#pragma unroll
              for (int h = 0; h < 4; ++h) {
                const uint32_t(&z)[4] = kb[i & 1][h >> 1][j];
                mma_bf16(d[h], a[order - j], z[2 * (h & 1)], z[2 * (h & 1) + 1]);
              }
            }
#pragma unroll
        for (int e = 0; e < PER; ++e)
          if (i * PER + e < kPartProducts) part_product(i * PER + e, po, w, m);
#pragma unroll
        for (int h = 0; h < 4; ++h)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[4 * i + h][e] = fmaf(gc, S[4 * i + h][e], d[h][e]);
      }
      add4(O[0], po[0]);
      add4(O[1], po[1]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[c % NST]);
    if constexpr (F32) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = h * 8 + q2 + (e & 1);
          if (t < left && (e < 2 ? ok0 : ok1)) out[(c * kTok + t) * out_ld + gr + (e >> 1) * 8] = O[h][e];
        }
    } else {
      uint8_t* stage = sm + C::oOut + warp * kTok * 48;
      const uint32_t to = smem_u32(stage) + ((lane & 7) + (lane >> 4) * 8) * 48 + ((lane >> 3) & 1) * 16;
      asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(to),
                   "r"(pack_bf16x2(O[0][0], O[0][1])), "r"(pack_bf16x2(O[0][2], O[0][3])), "r"(pack_bf16x2(O[1][0], O[1][1])),
                   "r"(pack_bf16x2(O[1][2], O[1][3]))
                   : "memory");
      __syncwarp();
      const int t = lane >> 1, half = (lane & 1) * 8;
      const uint4 r = *reinterpret_cast<const uint4*>(stage + t * 48 + half * 2);
      if (t < left && col0 + cw + half < p.vdim) *reinterpret_cast<uint4*>(out + (c * kTok + t) * out_ld + half) = r;
      __syncwarp();
    }
  }
#pragma unroll
  for (int i = 0; i < NT; ++i)
    if (i * 8 < p.dim) {
      if (ok0) *reinterpret_cast<float2*>(st + i * 8) = make_float2(S[i][0], S[i][1]);
      if (ok1) *reinterpret_cast<float2*>(st + 8 * p.dim + i * 8) = make_float2(S[i][2], S[i][3]);
    }
}

template <int DK, int MW, bool DELTA, typename T>
int launch_chunks(const ChunkParams& p, cudaStream_t s) {
  using C = Chunk<DK, MW, T>;
  auto kernel = head_chunk_kernel<DK, MW, DELTA, T>;
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return int(e);
    attr_set[dev] = true;
  }
  return launch_pdl(kernel, dim3((p.r.vdim + C::COLS - 1) / C::COLS, p.r.heads, p.r.batch), dim3(C::THREADS), size_t(C::SMEM), s, p);
}
template <int DK, bool DELTA>
int launch_chunks_form(const ChunkParams& p, cudaStream_t s) {
  if constexpr (DELTA) {
    if (!p.r.bf16) return launch_chunks<DK, 4, DELTA, float>(p, s);
  }
  if (p.r.vdim <= 64 || (long long)p.r.batch * p.r.heads * ((p.r.vdim + 63) / 64) <= 148)
    return launch_chunks<DK, 4, DELTA, __nv_bfloat16>(p, s);
  return launch_chunks<DK, 8, DELTA, __nv_bfloat16>(p, s);
}

}  // namespace

// Sixteen tokens cost a chunk what a few cost it, and a CTA takes a whole SM: token by token (four CTAs an SM) is the faster way for
// short sequences and for single tokens beside short prompts.  us of 32 heads token by token and by chunks, bf16 unless said:
//   128 x 128, delta rule   1 x 16 7.9, 7.4   16 x 16 34, 32   15 x 1 + 64 45, 39   47 x 1 + 64 80, 102   47 x 1 + 128 122, 112
//                           1 x 2048 693, 191   4 x 2048 1317, 329
//   128 x 128, state space  16 x 16 29, 24   47 x 1 + 64 73, 78   47 x 1 + 128 103, 85   1 x 2048 391, 137   4 x 2048 871, 236
//   64 x 64, delta rule     16 x 16 14, 18   16 x 48 34, 25   15 x 1 + 64 27, 21   47 x 1 + 128 57, 55
//   64 x 64, state space    1 x 64 10.3, 6.6   16 x 48 24, 19   47 x 1 + 128 39, 37   24 x 1 + 390 86, 38
//   fp32, 128 x 128, delta  1 x 64 33, 20   16 x 48 118, 130   15 x 1 + 128 105, 97   1 x 301 144, 71   4 x 512 390, 243
bool head_chunks_pay(const NkbHeadRec& a) {
  const bool wide = a.dim > 64, delta = a.b.ptr != nullptr;
  const int longest = a.longest > 0 ? a.longest : a.tokens - a.batch + 1;
  if (!a.bf16) return longest >= 64 && a.tokens >= 24 + 6 * a.batch;
  if (!wide && !delta) return longest >= 64 && a.tokens >= 48 + 8 * a.batch;
  return longest >= (wide ? 16 : 32) && a.tokens >= 16 + 3 * a.batch;
}

// The state-space form of 32-bit models stays token by token: its results were a fifth further from the recurrence in 64 bits (1.27e-7
// against 1.06e-7), those of the delta rule were not (1.60e-7 and 1.64e-7; decays of the served models).
bool head_chunks_ok(const NkbHeadRec& a) {
  if (!a.bf16 && !a.b.ptr) return false;
  const auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (a.dim <= 32 || a.dim > 128 || a.dim % 8 || (a.x.bf16 != 0) != (a.bf16 != 0) || !al16(a.x.ptr) || !al16(a.out)) return false;
  const int run = a.bf16 ? 8 : 4;                      // elements of sixteen bytes
  return (a.vdim | a.q_col | a.k_col | a.v_col) % run == 0 && a.x.ld % run == 0;
}

int head_chunks(const NkbHeadRec& a, cudaStream_t s) {
  if (!status_word() && nkb_init() != 0) return -1;
  const ChunkParams p{a, status_word()};
  const bool delta = a.b.ptr != nullptr;
  if (a.dim <= 64) return delta ? launch_chunks_form<64, true>(p, s) : launch_chunks_form<64, false>(p, s);
  return delta ? launch_chunks_form<128, true>(p, s) : launch_chunks_form<128, false>(p, s);
}

}  // namespace nkb
