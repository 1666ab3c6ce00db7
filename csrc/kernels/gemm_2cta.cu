// bf16 GEMM on CTA pairs: D[m, n] = A[m, k] * B[n, k]^T with output tiles of 256 x 256, or less wide ones.
//
// Two CTAs of a cluster (one SM each) work on one tile with `tcgen05.mma.cta_group::2`: CTA r of
// the pair holds rows [128 r, 128 r + 128) of the A tile and rows [128 r, 128 r + 128) of the B tile in
// its shared memory and the matching 128 accumulator rows in its tensor memory; the MMA is issued by
// one thread of the pair's first CTA and reads both CTAs' shared memory.  Per k-slab each CTA therefore
// loads 32 KB for 128 x 256 outputs (the single-CTA kernel loads 48 KB), which takes the L2 -> shared-
// memory traffic of the prefill GEMMs from about 16 TB/s at tensor-core peak to about 11 TB/s, and the
// ring holds seven stages instead of four.
//
// Synchronisation (all mbarriers; every wait is bounded):
//   full[s]   lives in the first CTA: its TMA warp announces the bytes of both CTAs, both CTAs' loads
//             complete their bytes there;
//   empty[s]  one per CTA: after the MMAs of a stage the issuing thread commits to its own and to the
//             peer's barrier (two plain commits; no cluster-wide broadcast form is used anywhere);
//   tfull[a]  one per CTA, same two commits, wakes both epilogues;
//   tempty[a] lives in the first CTA, count 8: the four epilogue warps of both CTAs arrive.
// Loads are plain (non-broadcast) tiled TMA copies of this GPU's memory.
//
// Tile width: a round of tiles takes as long on 40 SM pairs as on all of them, and products of some hundred rows have two to five rounds.
// Narrower tiles let the last round come out even (the caller picks the width): 414 rows of 2 x 14336 gate / up rows, 4096 of k, 3.03
// rounds of 256 columns 126 us, 4.9 of 160 columns 106 us; at the same number of rounds per column the widest tile is the fastest.
//
// Reference parity: same role as gemm_tcgen05.cuh (the `dot` lowering target, prefill orientation).
#include "gemm_tcgen05.cuh"
#include "api.h"
#include <stdlib.h>

namespace nkb {

struct Gemm2Args {            // <= 128 bytes (see GemmArgs)
  int m, n, k;
  int tiles_m, tiles_n;       // tiles of 256 x tile_n
  int tile_n;                 // multiple of 32 up to 256; gated: half of it gate columns, half up columns
  int kb_total, stages;
  int group_m;                // row tiles that share one sweep over the column tiles (L2 reuse)
  int gated;                  // B holds [gate; up] rows: the pair's first CTA loads gate rows, the second up rows
  int gate_off;               // row offset of the up half in B
  int act;                    // gated: 0 = SiLU, 1 = GELU (tanh form); plain: 2 = squared ReLU, 7 = xIELU of act_a, act_b
  float act_a, act_b;
  int splits;                 // > 1: fp32 partial sums, split s at out + s * split_stride
  int kb_per_split;
  int static_b;               // B (weights) is not written by the kernel before this one: its tiles go ahead of the wait
  long long ldo;
  long long split_stride;
  void* out;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  int* status;
};
static_assert(sizeof(Gemm2Args) <= 128, "Gemm2Args grew past the fast kernel-parameter size");

constexpr int k2TileN = 256;                      // widest tile
constexpr int k2StageBytes = 2 * kATileBytes;     // A rows + B rows of this CTA, 16 KB each

// Rows of A sorted by group, one weight matrix per group (stacked in B): tile t of the list is rows [256 ct, 256 ct + 256) of a
// group.  A struct of its own: the plain kernel's arguments stay small.
struct Group2Args {
  const int* tile_list;       // (group, ct) pairs
  const int* tile_count;
  const int* offsets;         // first row of each group
  int w_rows;                 // rows of B per group
  long long bias_stride;
  float limit, alpha;         // limit > 0: clamped gate (up + 1) * gate * sigmoid(alpha * gate)
};

struct Work2 {
  int tm, tn, sp, kb0, kb1;
  int a_row0, row_end, b_row0, group;    // first row of A and end of its rows, first row of B
};
// group_m row tiles share a sweep over the column tiles so that A and B tiles are re-read from L2; the splits of a tile
// follow one another.  Groups: the column tiles of a row tile follow one another (its weights are read once either way).
template <bool GROUPED>
__device__ __forceinline__ Work2 decode_work2(const Gemm2Args& a, const Group2Args& g, int w) {
  Work2 o;
  if constexpr (GROUPED) {
    const int t = w / a.tiles_n;
    o.tm = 0;
    o.tn = w - t * a.tiles_n;
    o.sp = 0;
    o.kb0 = 0;
    o.kb1 = a.kb_total;
    o.group = g.tile_list[2 * t];
    o.a_row0 = g.offsets[o.group] + g.tile_list[2 * t + 1] * 256;
    o.row_end = g.offsets[o.group + 1];
    o.b_row0 = o.group * g.w_rows;
    return o;
  }
  o.sp = w % a.splits;
  const int t = w / a.splits;
  const int per_group = a.group_m * a.tiles_n;
  const int gr = t / per_group, first = gr * a.group_m;
  const int gsz = min(a.tiles_m - first, a.group_m), in = t - gr * per_group;
  o.tm = first + in % gsz;
  o.tn = in / gsz;
  o.kb0 = o.sp * a.kb_per_split;
  o.kb1 = min(a.kb_total, o.kb0 + a.kb_per_split);
  o.a_row0 = o.tm * 256;
  o.row_end = a.m;
  o.b_row0 = 0;
  o.group = 0;
  return o;
}

template <bool GROUPED>
__device__ __forceinline__ void gemm2_body(const CUtensorMap& tmA, const CUtensorMap& tmB, const Gemm2Args& args,
                                           const Group2Args& grp) {
  extern __shared__ uint8_t smem_raw[];
  // identical layout in both CTAs: [control 1 KB][ring]
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  GemmCtrl* ctrl = reinterpret_cast<GemmCtrl*>(base);
  uint8_t* tiles = base + 1024;
  const int warp = warp_idx_uniform();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();        // 0 = issues the MMAs
  const int stages = args.stages;
  constexpr uint32_t tmem_cols = 2 * k2TileN;     // two accumulators of 256 columns
  const int tile_n = GROUPED ? k2TileN : args.tile_n, half_n = tile_n / 2;     // half_n: rows of B per CTA
  const uint32_t stage_tx = 2u * uint32_t(kATileBytes + half_n * kBlockK * 2);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ctrl->full[s], 1);
      mbar_init(&ctrl->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctrl->tfull[i], 1);
      mbar_init(&ctrl->tempty[i], 8);
    }
    ctrl->abort = 0;
    mbar_fence_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc_pair(&ctrl->tmem_base, tmem_cols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                              // both CTAs' barriers exist before anything remote arrives
  tc_fence_after();
  const uint32_t tmem_base = ctrl->tmem_base;
  volatile int* abort_flag = &ctrl->abort;

  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  // the tile list comes from the kernels before this one: every role waits before it reads the count
  if constexpr (GROUPED) griddep_wait();
  const int total_work = GROUPED ? *grp.tile_count * args.tiles_n : args.tiles_m * args.tiles_n * args.splits;
  griddep_launch();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    auto b_row_of = [&](const Work2& t) {
      return t.b_row0 + (args.gated ? (int(rank) * args.gate_off + t.tn * half_n) : (t.tn * tile_n + int(rank) * half_n));
    };
    // Weight tiles do not depend on the preceding kernel: the first fill of the ring takes them before the wait.  (The second
    // CTA's bytes may arrive before the first one has announced them: a barrier's phase ends only with the announcement.)
    int pre = 0;
    if (!GROUPED && args.static_b && pair < total_work) {
      const Work2 t = decode_work2<GROUPED>(args, grp, pair);
      pre = min(stages, t.kb1 - t.kb0);
      if (lane == 0)
        for (int i = 0; i < pre; ++i) {
          if (rank == 0) mbar_expect_tx(&ctrl->full[i], stage_tx);
          tma_load_2d_pair(tiles + i * k2StageBytes + kATileBytes, &tmB, map_to_cta(&ctrl->full[i], 0), (t.kb0 + i) * kBlockK,
                           b_row_of(t));
        }
      __syncwarp();
    }
    griddep_wait();
    int stage = 0;
    uint32_t phase = 0;
    bool alive = true;
    for (int w = pair; w < total_work && alive; w += npairs) {
      const Work2 t = decode_work2<GROUPED>(args, grp, w);
      const int a_row = t.a_row0 + int(rank) * 128;
      const int b_row = b_row_of(t);
      for (int kb = t.kb0; kb < t.kb1; ++kb) {
        bool ok = mbar_wait(&ctrl->empty[stage], phase ^ 1u, abort_flag, args.status, ERR_WAIT_SMEM_EMPTY);
        if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
        if (lane == 0) {
          const uint32_t full0 = map_to_cta(&ctrl->full[stage], 0);
          uint8_t* a_ptr = tiles + stage * k2StageBytes;
          // the first CTA announces the bytes of both CTAs; the second only lets its loads complete there
          // (its loads of this phase cannot start before the barrier entered the phase: they wait for the
          // stage to be released, which follows the previous phase's completion)
          const bool ahead = w == pair && kb - t.kb0 < pre;
          if (rank == 0 && !ahead) mbar_expect_tx(&ctrl->full[stage], stage_tx);
          tma_load_2d_pair(a_ptr, &tmA, full0, kb * kBlockK, a_row);
          if (!ahead) tma_load_2d_pair(a_ptr + kATileBytes, &tmB, full0, kb * kBlockK, b_row);
        }
        __syncwarp();
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1 && rank == 0) {
    // ------------------------------------------------------------------ MMA issuer (first CTA of the pair)
    // One elected thread runs the whole loop alone: the tensor pipe queues only a few MMAs, so warp votes,
    // reconvergence and descriptor arithmetic between two k-blocks are time in which it drains.
    const uint32_t idesc = make_idesc_bf16(256, tile_n, 0, 0);
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      const uint64_t d_tiles = make_smem_desc_sw128(smem_u32(tiles), 0, 1024);
      const uint64_t d_hi = d_tiles & 0xffffffff00000000ull;
      const uint32_t a_lo0 = uint32_t(d_tiles);
      const uint32_t empty0 = map_to_cta(&ctrl->empty[0], 0), empty1 = map_to_cta(&ctrl->empty[0], 1);
      bool ok = true;
      for (int w = pair; w < total_work && ok; w += npairs) {
        ok = mbar_wait(&ctrl->tempty[acc], acc_phase ^ 1u, abort_flag, args.status, ERR_WAIT_TMEM_EMPTY);
        if (!ok) break;
        const uint32_t d0 = tmem_base + uint32_t(acc * k2TileN);
        const Work2 t = decode_work2<GROUPED>(args, grp, w);
        for (int kb = t.kb0; kb < t.kb1; ++kb) {
          ok = mbar_wait(&ctrl->full[stage], phase, abort_flag, args.status, ERR_WAIT_SMEM_FULL);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_lo = a_lo0 + uint32_t(stage) * uint32_t(k2StageBytes >> 4);
          const uint64_t da = d_hi | a_lo, db = d_hi | (a_lo + uint32_t(kATileBytes >> 4));
#pragma unroll
          for (int k = 0; k < kBlockK / 16; ++k)
            umma_f16_pair(d0, da + uint64_t(k * 2), db + uint64_t(k * 2), idesc, (kb > t.kb0 || k > 0) ? 1u : 0u);
          umma_commit_pair(empty0 + uint32_t(stage) * 8u);
          umma_commit_pair(empty1 + uint32_t(stage) * 8u);
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        umma_commit_pair(map_to_cta(&ctrl->tfull[acc], 0));
        umma_commit_pair(map_to_cta(&ctrl->tfull[acc], 1));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
    __syncwarp();
  } else if (warp >= 2) {
    // ------------------------------------------------------------------ epilogue (warps 2..5, both CTAs)
    const int quad = warp & 3;
    griddep_wait();
    int acc = 0;
    uint32_t acc_phase = 0;
    __nv_bfloat16* out_h = reinterpret_cast<__nv_bfloat16*>(args.out);
    for (int w = pair; w < total_work; w += npairs) {
      const Work2 work = decode_work2<GROUPED>(args, grp, w);
      const int tn = work.tn;
      const __nv_bfloat16* bias = args.bias;
      if constexpr (GROUPED) {
        if (bias) bias += work.group * grp.bias_stride;
      }
      bool ok = mbar_wait(&ctrl->tfull[acc], acc_phase, abort_flag, args.status, ERR_WAIT_TMEM_FULL);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      const uint32_t t0 = tmem_base + (uint32_t(quad * 32) << 16) + uint32_t(acc * k2TileN);
      const int row = work.a_row0 + int(rank) * 128 + quad * 32 + lane;
      if (args.gated) {
        // accumulator columns [0, half_n) = gate, [half_n, tile_n) = up: out[:, tn * half_n + j] = silu(gate_j) * up_j
        const int gcol0 = tn * half_n, cend = min(args.n, gcol0 + half_n);
#pragma unroll 1
        for (int c = 0; c < half_n; c += 32) {
          uint32_t v[32], u[32];
          tmem_ld_32x32(t0 + c, v);
          tmem_ld_32x32(t0 + half_n + c, u);
          tmem_ld_wait();
          if (c + 32 >= half_n) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(map_to_cta(&ctrl->tempty[acc], 0));
          }
          const int cbase = gcol0 + c;
          if (row >= work.row_end || cbase >= cend) continue;
          if constexpr (GROUPED) {
            if (bias) {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                const int c1 = min(cbase + j, args.n - 1);
                v[j] = __float_as_uint(__uint_as_float(v[j]) + __bfloat162float(bias[c1]));
                u[j] = __float_as_uint(__uint_as_float(u[j]) + __bfloat162float(bias[args.gate_off + c1]));
              }
            }
          }
          if (GROUPED && grp.limit > 0.f) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float gg = fminf(__uint_as_float(v[j]), grp.limit);
              const float uu = fminf(fmaxf(__uint_as_float(u[j]), -grp.limit), grp.limit);
              v[j] = __float_as_uint((uu + 1.f) * gg / (1.f + __expf(-grp.alpha * gg)));
            }
          } else if (args.act) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              v[j] = __float_as_uint(gelu_tanh_f(__uint_as_float(v[j])) * __uint_as_float(u[j]));
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              v[j] = __float_as_uint(silu_f(__uint_as_float(v[j])) * __uint_as_float(u[j]));
          }
          const long long off = (long long)row * args.ldo + cbase;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (cbase + 8 * q + 8 <= cend && (off & 7) == 0) {
              reinterpret_cast<uint4*>(out_h + off)[q] =
                  make_uint4(pack_bf16x2(__uint_as_float(v[8 * q]), __uint_as_float(v[8 * q + 1])),
                             pack_bf16x2(__uint_as_float(v[8 * q + 2]), __uint_as_float(v[8 * q + 3])),
                             pack_bf16x2(__uint_as_float(v[8 * q + 4]), __uint_as_float(v[8 * q + 5])),
                             pack_bf16x2(__uint_as_float(v[8 * q + 6]), __uint_as_float(v[8 * q + 7])));
            } else {
#pragma unroll
              for (int j = 8 * q; j < 8 * q + 8; ++j)
                if (cbase + j < cend) out_h[off + j] = __float2bfloat16(__uint_as_float(v[j]));
            }
          }
        }
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
        continue;
      }
      const int col0 = tn * tile_n;
#pragma unroll 1
      for (int c = 0; c < tile_n; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32(t0 + c, v);
        tmem_ld_wait();
        if (c + 32 >= tile_n) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(map_to_cta(&ctrl->tempty[acc], 0));
        }
        const int cbase = col0 + c;
        if (row >= work.row_end || cbase >= args.n) continue;
        if (args.splits > 1) {
          float* o = reinterpret_cast<float*>(args.out) + work.sp * args.split_stride + (long long)row * args.ldo + cbase;
          if (cbase + 32 <= args.n && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              reinterpret_cast<float4*>(o)[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                                            __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
          } else {
            for (int j = 0; j < 32; ++j)
              if (cbase + j < args.n) o[j] = __uint_as_float(v[j]);
          }
          continue;
        }
        if (bias) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (cbase + j < args.n)
              v[j] = __float_as_uint(__uint_as_float(v[j]) + __bfloat162float(bias[cbase + j]));
        }
        if (args.act == 7) {       // xIELU
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(xielu_f(__uint_as_float(v[j]), args.act_a, args.act_b));
        } else if (args.act == 2) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float r = fmaxf(__uint_as_float(v[j]), 0.f);
            v[j] = __float_as_uint(r * r);
          }
        }
        const long long off = (long long)row * args.ldo + cbase;
        if (cbase + 32 <= args.n && ((off & 7) == 0)) {
          uint32_t pk[16];
          if (args.residual) {
            const uint4* rp = reinterpret_cast<const uint4*>(args.residual + off);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint4 rr = rp[q];
              const uint32_t rw[4] = {rr.x, rr.y, rr.z, rr.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 f = unpack_bf16x2(rw[e]);
                pk[q * 4 + e] = pack_bf16x2(__uint_as_float(v[q * 8 + 2 * e]) + f.x,
                                            __uint_as_float(v[q * 8 + 2 * e + 1]) + f.y);
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) pk[j] = pack_bf16x2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
          }
          uint4* p = reinterpret_cast<uint4*>(out_h + off);
#pragma unroll
          for (int q = 0; q < 4; ++q) p[q] = make_uint4(pk[4 * q], pk[4 * q + 1], pk[4 * q + 2], pk[4 * q + 3]);
        } else {
          for (int j = 0; j < 32; ++j) {
            if (cbase + j < args.n) {
              float x = __uint_as_float(v[j]);
              if (args.residual) x += __bfloat162float(args.residual[off + j]);
              out_h[off + j] = __float2bfloat16(x);
            }
          }
        }
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // neither CTA leaves (and frees shared / tensor memory) while its peer still works
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, tmem_cols);
  }
}

__global__ void __launch_bounds__(kGemmThreads, 1)
gemm2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const Gemm2Args args) {
  gemm2_body<false>(tmA, tmB, args, Group2Args{});
}
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm2_grouped_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const Gemm2Args args,
                     const Group2Args grp) {
  gemm2_body<true>(tmA, tmB, args, grp);
}

// Launches `pairs` CTA pairs, at most as many as can be resident at once (the persistent loop strides by their number, and
// pairs need two SMs of one GPC: not every SM can be paired) and as there are tiles.
// resident: of each device, 0 before its first launch.
constexpr int kMaxDevices = 64;
template <typename K, typename... Args>
static int launch_pairs(K kernel, int (&resident)[kMaxDevices], int total, int smem, cudaStream_t stream, int* used, const Args&... args) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (num_sms() / 2));
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = size_t(smem);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (resident[dev] == 0) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e != cudaSuccess) return int(e);
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
    resident[dev] = (e == cudaSuccess && n > 0) ? n : num_sms() / 4;
  }
  const int pairs = resident[dev] < total ? resident[dev] : total;
  if (used) *used = pairs;
  cfg.gridDim = dim3(2 * pairs);
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return int(cudaLaunchKernelEx(&cfg, kernel, args...));
}

static int ring2(Gemm2Args& a) {
  int stages = (232448 - 1024 - 1024) / k2StageBytes;
  if (stages > kMaxStages) stages = kMaxStages;
  a.stages = stages;
  return stages * k2StageBytes + 2048;
}

}  // namespace nkb

using namespace nkb;

// out[m, n] = A[m, k] * B[n, k]^T (+ bias[n]) (+ residual[m, n]); bf16 in and out, row strides in elements.
// tile_n: columns per tile, a multiple of 32 up to 256 (gated: half of them gate, half up).  The launcher returns -5
// for n below 256, which it does not take (callers then use the single-CTA kernel, as they do for 128 rows or fewer).
// Number of CTA pairs that can be resident at once (0 before the first launch).
static int g_pairs_last = 0;
extern "C" int nkb_gemm_2cta_pairs() { return g_pairs_last; }

// gated != 0: B holds [gate; up] (2 x n rows, the up half starting at row gate_off) and out[m, n] =
// silu(A gate^T) * (A up^T); bias / residual are not applied in that mode.  act 1: GELU in place of SiLU; 2 (not gated):
// the square of the positive part of (A B^T + bias); 7 (not gated): xIELU with the parameters act_a, act_b.
extern "C" int nkb_gemm_bf16_2cta(const void* A, const void* B, void* out, int m, int n, int k, long long lda,
                                  long long ldb, long long ldo, const void* bias, const void* residual, int gated,
                                  int gate_off, int act, float act_a, float act_b, int splits, long long split_stride,
                                  int static_b, int tile_n, void* stream) {
  if (splits < 1 || (splits > 1 && (gated || bias || residual || act))) return -2;
  if (act < 0 || (act > 2 && act != 7) || (act >= 2 && gated)) return -2;
  if (!status_word() && nkb_init() != 0) return -1;
  if (m <= 0 || n <= 0 || k <= 0) return -2;
  if ((k & 7) || (lda & 7) || (ldb & 7)) return -2;
  if (tile_n < 32 || tile_n > k2TileN || (tile_n & 31)) return -2;
  if (n < 256) return -5;
  Gemm2Args a{};
  a.m = m; a.n = n; a.k = k;
  a.tiles_m = (m + 255) / 256;
  a.tile_n = tile_n;
  a.tiles_n = gated ? (n + tile_n / 2 - 1) / (tile_n / 2) : (n + tile_n - 1) / tile_n;
  a.gated = gated ? 1 : 0;
  a.gate_off = gate_off;
  a.act = act;
  a.act_a = act_a;
  a.act_b = act_b;
  if (gated && (bias || residual)) return -2;
  a.kb_total = (k + kBlockK - 1) / kBlockK;
  a.splits = splits;
  a.kb_per_split = (a.kb_total + splits - 1) / splits;
  if ((splits - 1) * a.kb_per_split >= a.kb_total) return -2;       // an empty split would leave its partial unwritten
  a.split_stride = split_stride;
  a.static_b = static_b;
  static int group_m = 0;
  if (group_m == 0) {
    const char* e = getenv("NKIPY_B200_2CTA_GROUP");
    group_m = e ? atoi(e) : 16;
    if (group_m < 1) group_m = 16;
  }
  a.group_m = group_m;
  a.ldo = ldo;
  a.out = out;
  a.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  a.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  a.status = status_word();
  const int smem = ring2(a);
  CUtensorMap ta, tb;
  if (encode_tmap_bf16_2d(&ta, A, k, m, lda, kBlockK, kTileRows)) return -4;
  if (encode_tmap_bf16_2d(&tb, B, k, gated ? uint64_t(gate_off) + n : uint64_t(n), ldb, kBlockK, tile_n / 2)) return -4;
  static int resident[kMaxDevices] = {0};
  return launch_pairs(gemm2_kernel, resident, a.tiles_m * a.tiles_n * splits, smem, reinterpret_cast<cudaStream_t>(stream),
                      &g_pairs_last, ta, tb, a);
}

// Per-group products of rows sorted by group: out[r, :] = x[r] * w[g(r)]^T for the row tiles of 256 in tile_list (see
// nkb_moe_dispatch).  w [groups, features (gated: gate_off + features), k], contiguous; bias as in nkb_gemm_bf16_grouped.
extern "C" int nkb_gemm_bf16_2cta_grouped(const void* weights, const void* x_sorted, void* out, const int* group_offsets,
                                          int num_groups, int features, int k, int total_rows, long long ldx, long long ldo,
                                          int gated, int gate_off, const void* bias, long long bias_group_stride,
                                          float act_limit, float act_alpha, const int* tile_list, const int* tile_count,
                                          int max_tiles, void* stream) {
  if (!status_word() && nkb_init() != 0) return -1;
  if (num_groups <= 0 || features <= 0 || k <= 0 || total_rows <= 0) return 0;
  if ((k & 7) || (ldx & 7) || !tile_list || !tile_count || max_tiles <= 0) return -2;
  Gemm2Args a{};
  a.m = total_rows; a.n = features; a.k = k;
  a.tiles_n = gated ? (features + 127) / 128 : (features + 255) / 256;
  a.gated = gated ? 1 : 0;
  a.gate_off = gate_off;
  a.kb_total = (k + kBlockK - 1) / kBlockK;
  a.splits = 1;
  a.kb_per_split = a.kb_total;
  a.group_m = 1;
  a.ldo = ldo;
  a.out = out;
  a.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  a.status = status_word();
  Group2Args g{};
  g.tile_list = tile_list;
  g.tile_count = tile_count;
  g.offsets = group_offsets;
  const long long w_rows = gated ? (long long)gate_off + features : features;
  if (w_rows * num_groups > 0x7fffffffll) return -2;
  g.w_rows = int(w_rows);
  g.bias_stride = bias_group_stride;
  g.limit = act_limit;
  g.alpha = act_alpha;
  const int smem = ring2(a);
  CUtensorMap ta, tb;
  if (encode_tmap_bf16_2d(&ta, x_sorted, k, total_rows, ldx, kBlockK, kTileRows)) return -4;
  if (encode_tmap_bf16_2d(&tb, weights, k, uint64_t(w_rows) * num_groups, k, kBlockK, kTileRows)) return -4;
  static int resident[kMaxDevices] = {0};
  return launch_pairs(gemm2_grouped_kernel, resident, max_tiles * a.tiles_n, smem, reinterpret_cast<cudaStream_t>(stream),
                      nullptr, ta, tb, a, g);
}
