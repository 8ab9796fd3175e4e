// Weight-streaming grouped GEMM for experts with few rows (decoding).
//
//   C[rows of tile t, :] = epilogue( A[tile t, :] . B[expert_ids[t], :, :]^T )
//
// Same operands, epilogues and results as the row-tile kernel of grouped_gemm.cu; what differs is
// the work per weight byte.  A decoding step reads every expert it touches once and uses each
// weight for one to a few rows, so the bound is HBM, and with the chip clocking by power also the
// energy spent per weight.  The row-tile kernel multiplies 128 rows whatever their number.  Here
// the weights are the 128-row operand of tcgen05.mma and the live rows, rounded up to 16, its
// columns: a K block of 256 weight rows is eight 128 x N x 32-byte instructions, and its
// accumulators are 2 N TMEM columns, so for N <= 32 eight K blocks are in flight between the
// tensor core and the promotion of the block-scaled kinds (two in the row-tile kernel).
//
// Work item: (row tile, 256 / KBS weight rows).  A stage is 32 KiB of weights (256 / KBS rows x KBS
// K blocks of 128 bytes, four swizzled 64-row boxes) plus the rows' K blocks, which two warps bring
// with 16-byte asynchronous copies from token order or sorted order; KBS = 2 halves the item
// where there are too few for the chip.
//
// Roles (384 threads): warp 0 weights (TMA), warp 1 MMA issuer + TMEM owner, warps 2-3 rows and
// their scales, warps 4..11 epilogue: warp w owns TMEM lanes 32 (w % 4).., i.e. one weight row per
// thread, and half (w - 4) / 4 of the columns.  Activation scales differ by column here: a thread
// reads them as broadcasts from a ring in shared memory.
//
// Every wait on an mbarrier is bounded; epilogue warps that gave up still meet the others at the
// item's barriers and all leave together.
//
// Measured, up and down projection of one layer in us, row tiles -> this (results equal bit for bit):
// DeepSeek-V3 fp8 (256 experts), 1 token 53 + 35 -> 44 + 27, 96 tokens 1204 + 617 -> 1042 + 542 (6.85
// TB/s of weights), 300 tokens 1228 + 656 -> 1106 + 584; Mixtral bf16, 1 token 84 + 92 -> 81 + 65, 40
// tokens 305 + 148 -> 292 + 147; Qwen3-30B int8, 100 tokens 84 + 54 -> 77 + 39.  Back to back under
// the power limit the gain is larger: the 96-token layer goes from 2179 to 1733 us.
#pragma once

#include <cuda.h>

#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace bolt {
namespace stream {
using namespace tc;

constexpr int kThreads = 384;
constexpr int kRowThreads = 64;
constexpr int kEpilogue = 256;
constexpr int kStages = 4;
constexpr int kWeightBytes = 32768;        // four boxes of 64 rows x 128 bytes
constexpr int kBoxBytes = 8192;
constexpr int kMaxRows = 128;              // rows of an item with one K block per stage
constexpr int kRowBytes = kMaxRows * 128;  // (KBS K blocks of kMaxRows / KBS rows)
constexpr int kAccStages = 8;              // TMEM accumulator stages of the block-scaled kinds, at most
constexpr int kScaleSlots = 16;            // >= kStages + kAccStages + 1
constexpr int kSlotBytes = kMaxRows * 4 + 16;    // activation scales of the rows, the two weight scales
constexpr int kStagePitch = 256 + 4;       // floats
constexpr int kStageOut = 16 * kStagePitch * 4;
constexpr int kSmemBytes =
    kStages * (kWeightBytes + kRowBytes) + kScaleSlots * kSlotBytes + kStageOut + 1024 + 1024;

struct StreamParams {
  const void* a;
  int64_t a_row_bytes;
  const float* a_scale;
  int64_t a_scale_ld;
  const float* b_scale;
  const void* bias;
  int bias_dtype;
  void* c;
  int c_dtype, mid_dtype;
  int64_t c_ld;
  float* c_scale;
  int64_t c_scale_ld;
  int gather, a_scale_tok, scatter, num_tokens, topk, mul_routed_weight, c_vec_ok;
  const int32_t* sorted_ids;
  const float* sorted_weights;
  const int32_t* expert_ids;
  const int32_t* num_valid;
  int32_t* status;
  int n, n_half, num_experts, capacity, tiles_n, num_kb, kb_scale_cols;
  uint32_t idesc;   // instruction descriptor without N
};

// barrier of the epilogue warps
__device__ __forceinline__ void epilogue_sync() {
  asm volatile("barrier.cta.sync 1, 256;" ::: "memory");
}
// the same, and whether any of them is in trouble
__device__ __forceinline__ bool epilogue_any(bool bad) {
  int r;
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.b32 p, %1, 0;\n"
      "barrier.cta.red.or.pred q, 1, 256, p;\nselp.b32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"((int)bad)
      : "memory");
  return r != 0;
}

// TMEM -> registers: this warp's 32 lanes, C consecutive columns
template <int C>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[C]) {
  if constexpr (C == 8) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7])
        : "r"(taddr)
        : "memory");
  } else if constexpr (C == 32) {
    tmem_ld32(taddr, r);
  } else {
    static_assert(C == 16, "8, 16 or 32 columns");
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
        "%12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
  }
}

// 4-byte asynchronous copy global -> shared
__device__ __forceinline__ void cp_async_4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ float round_mid(float v, int mid) {
  if (mid == BOLT_BF16) return __bfloat162float(__float2bfloat16_rn(v));
  if (mid == BOLT_F16) return __half2float(__float2half_rn(v));
  return v;
}
__device__ __forceinline__ uint16_t to_16bit(float v, int dt) {
  if (dt == BOLT_BF16) return __bfloat16_as_ushort(__float2bfloat16_rn(v));
  return __half_as_ushort(__float2half_rn(v));
}

// live rows of the row tile whose 128 ids are held four per lane (they come first in the tile)
__device__ __forceinline__ int live_rows(const int (&id)[4], int num_tokens) {
  int n = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    n += __popc(__ballot_sync(0xffffffffu, (id[i] & 0xFFFFFF) < num_tokens));
  return n;
}
// MMA columns for a number of rows: 16, 32, 64 or 128
__device__ __forceinline__ int columns_for(int rows) {
  return rows <= 16 ? 16 : rows <= 32 ? 32 : rows <= 64 ? 64 : 128;
}
// TMEM stages of the block-scaled kinds (a K block takes 2 N columns, N with KBS = 2)
template <int KBS>
__device__ __forceinline__ int acc_stages(int cols) {
  return min(kAccStages, 512 / ((KBS == 1 ? 2 : 1) * cols));
}

struct Epilogue {
  uint32_t tmem, bar_tfull, bar_tempty, bar_scale, scale_ring;
  uint8_t* out_stage;
  volatile int* abort_flag;
  int warp, lane;       // warp 0..7
  uint32_t parity;      // block-scaled: bit i = parity of the next use of TMEM stage i
  uint32_t count;       // K blocks (block-scaled) or items so far
};

// One work item in the epilogue: rows [row0, row0 + rows) of the sorted layout, 2 t_cols >= rows MMA
// columns, column tile n_blk.  Block-scaled kinds hold their sums in registers and are compiled for
// every t_cols (= T); the others leave them in TMEM (T = 0).  Returns false (in all epilogue warps
// alike) when a wait ran out.
template <int OPK, bool BS, int EPI, int KBS, int T>
__device__ __forceinline__ bool finish_item(const StreamParams& p, Epilogue& ep, int expert,
                                            int n_blk, int row0, int rows, int t_cols) {
  constexpr bool GATED = EPI != BOLT_EPI_STORE;
  constexpr bool QUANT = EPI == BOLT_EPI_SILU_MUL_QUANT;
  constexpr bool CHANNEL = OPK != OP_F16 && !BS;
  constexpr int H = KBS == 1 ? 2 : 1;            // 128-row halves of the item
  constexpr int COLS = GATED ? 128 : 128 * H;    // output columns of the item
  const int q = ep.warp & 3, side = ep.warp >> 2;
  const int lrow = 32 * q + ep.lane;             // weight row within a half
  const uint32_t lane_addr = ep.tmem + ((uint32_t)(32 * q) << 16) + side * t_cols;
  const int n0 = n_blk * COLS;
  const int n_cols = GATED ? p.n_half : p.n;

  float acc[H][BS ? T : 1];
  uint32_t acc_stage = 0;
  bool ok = true;
  if constexpr (BS) {
    constexpr int N = 2 * T;
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
      for (int j = 0; j < T; ++j) acc[h][j] = 0.f;
    const int stages = acc_stages<KBS>(N);
    int t = 0;
    for (int kb = 0; kb < p.num_kb; ++kb) {
      ok = mbar_wait(ep.bar_tfull + 8 * t, (ep.parity >> t) & 1u, ep.abort_flag, p.status, 4);
      if (!ok) break;
      tc_fence_after();
      const uint32_t tbase = lane_addr + t * (H * N);
      const uint32_t slot = ep.count % kScaleSlots;
      ok = mbar_wait(ep.bar_scale + 8 * slot, (ep.count / kScaleSlots) & 1u, ep.abort_flag, p.status, 6);
      if (!ok) break;
      ++ep.count;
      const uint32_t sbase = ep.scale_ring + slot * kSlotBytes;
      // C columns of one half at a time, two loads in flight; the stage goes back to the tensor core
      // as soon as the last column is in registers
      constexpr int C = T <= 32 ? T : 16, CHUNKS = H * (T / C);
      auto column = [&](int i) { return tbase + (i % H) * N + (i / H) * C; };
      uint32_t raw[2][C];
      tmem_ld<C>(column(0), raw[0]);
      float2 b2;
      asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];"
                   : "=f"(b2.x), "=f"(b2.y)
                   : "r"(sbase + kMaxRows * 4));
      float a_s[C];
#pragma unroll
      for (int i = 0; i < CHUNKS; ++i) {
        if (i % H == 0) {
#pragma unroll
          for (int j = 0; j < C; j += 4)
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(a_s[j]), "=f"(a_s[j + 1]), "=f"(a_s[j + 2]), "=f"(a_s[j + 3])
                         : "r"(sbase + (side * T + (i / H) * C + j) * 4));
        }
        tmem_ld_wait();
        if (i + 1 < CHUNKS) {
          tmem_ld<C>(column(i + 1), raw[(i + 1) & 1]);
        } else {
          tc_fence_before();
          __syncwarp();
          if (ep.lane == 0) mbar_arrive(ep.bar_tempty + 8 * t);
        }
        const float b_s = i % H == 0 ? b2.x : b2.y;
        const float2 bb = make_float2(b_s, b_s);
#pragma unroll
        for (int j = 0; j < C; j += 2) {
          float* a = &acc[i % H][(i / H) * C + j];
          const float2 v = __ffma2_rn(
              make_float2(acc_to_f32<OPK>(raw[i & 1][j]), acc_to_f32<OPK>(raw[i & 1][j + 1])),
              __fmul2_rn(make_float2(a_s[j], a_s[j + 1]), bb), make_float2(a[0], a[1]));
          a[0] = v.x;
          a[1] = v.y;
        }
      }
      ep.parity ^= 1u << t;
      if (++t == stages) t = 0;
    }
  } else {
    // the sums over K stay in TMEM; two stages of 256 columns alternate between items
    acc_stage = ep.count & 1u;
    ok = mbar_wait(ep.bar_tfull + 8 * acc_stage, (ep.count >> 1) & 1u, ep.abort_flag, p.status, 4);
    ++ep.count;
    tc_fence_after();
  }
  if (epilogue_any(!ok)) return false;

  // Eight rows of either side at a time pass through shared memory: thread = weight row on the way
  // in, then a warp takes a row and every lane V neighbouring columns of it.  All arithmetic of the
  // epilogue sits behind that, in ONE copy of a rolled loop: written out for every accumulator
  // register it was straight-line code of up to 60 KB that ran once per item at the speed of the
  // instruction fetch, 20 us per item at 128 rows and 4.5 us at 16.  Qwen3-235B fp8, 256 tokens with
  // Zipf-distributed routing: 347 + 195 -> 274 + 162 us for the two GEMMs.
  constexpr int V = COLS / 32;
  const int c0 = n0 + V * ep.lane;               // this lane's first output column
  const bool has_rw = p.mul_routed_weight && p.sorted_weights != nullptr;
  constexpr int G = GATED ? 2 : 1;
  float bias[G][V], b_s[G][V];
  if (CHANNEL || p.bias != nullptr) {
#pragma unroll
    for (int h = 0; h < G; ++h)
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int64_t col = (int64_t)expert * p.n + min(c0 + v, n_cols - 1) + h * p.n_half;
        bias[h][v] = p.bias ? load_bias(p.bias, p.bias_dtype, col) : 0.f;
        b_s[h][v] = CHANNEL ? __ldg(p.b_scale + col) : 1.f;
      }
  }
  float* stage = reinterpret_cast<float*>(ep.out_stage);
#pragma unroll 1
  for (int k = 0; k < t_cols / 8; ++k) {
    if (8 * k >= rows) break;                    // (uniform: the other side's rows come later still)
    if constexpr (BS) {
#pragma unroll
      for (int kk = 0; kk < T / 8; ++kk)
        if (kk == k) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int h = 0; h < H; ++h)
              stage[(side * 8 + j) * kStagePitch + 128 * h + lrow] = acc[h][8 * kk + j];
        }
    } else {
      uint32_t raw[H][8];
#pragma unroll
      for (int h = 0; h < H; ++h)
        tmem_ld<8>(lane_addr + acc_stage * 256 + h * (2 * t_cols) + 8 * k, raw[h]);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int h = 0; h < H; ++h)
          stage[(side * 8 + j) * kStagePitch + 128 * h + lrow] = acc_to_f32<OPK>(raw[h][j]);
    }
    epilogue_sync();
#pragma unroll 1
    for (int u = ep.warp; u < 16; u += kEpilogue / 32) {
      const int r = (u >> 3) * t_cols + 8 * k + (u & 7);
      if (r >= rows) continue;                   // warp-uniform
      const int row = row0 + r;
      const float a_s =
          CHANNEL ? __ldg(p.a_scale + (p.a_scale_tok ? p.sorted_ids[row] & 0xFFFFFF : row)) : 1.f;
      const float rw = has_rw ? __ldg(p.sorted_weights + row) : 1.f;
      float y[G][V];
#pragma unroll
      for (int h = 0; h < G; ++h)
#pragma unroll
        for (int v = 0; v < V; v += 4) {
          const float4 x = *reinterpret_cast<const float4*>(stage + u * kStagePitch + 128 * h +
                                                            V * ep.lane + v);
          y[h][v] = x.x;
          y[h][v + 1] = x.y;
          y[h][v + 2] = x.z;
          y[h][v + 3] = x.w;
        }
#pragma unroll
      for (int h = 0; h < G; ++h)
#pragma unroll
        for (int v = 0; v < V; ++v) {
          if (CHANNEL) {
            const float x = y[h][v] * a_s;
            y[h][v] = p.bias ? fmaf(x, b_s[h][v], bias[h][v]) : x * b_s[h][v];
          } else if (p.bias) {
            y[h][v] += bias[h][v];
          }
          if (has_rw) y[h][v] *= rw;
        }
      if (GATED) {
#pragma unroll
        for (int v = 0; v < V; ++v)
          y[0][v] = round_mid(silu_fast(round_mid(y[0][v], p.mid_dtype)) *
                                  round_mid(y[G - 1][v], p.mid_dtype),
                              p.mid_dtype);
      }
      if constexpr (QUANT) {
        // the row's 128 columns are one 1 x 128 group
        const bool to_i8 = p.c_dtype == BOLT_INT8;
        float m = 0.f;
#pragma unroll
        for (int v = 0; v < V; ++v) m = fmaxf(m, fabsf(y[0][v]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const float scale = __fdiv_rn(fmaxf(m, 1.0e-10f), to_i8 ? 127.0f : 448.0f);
        const float inv = __frcp_rn(scale);
        uint32_t w = 0;
#pragma unroll
        for (int v = 0; v < V; ++v)
          w |= (uint32_t)(to_i8 ? (uint8_t)f32_to_i8(y[0][v] * inv) : f32_to_e4m3(y[0][v] * inv))
               << (8 * v);
        *reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(p.c) + row * p.c_ld + c0) = w;
        if (ep.lane == 0) p.c_scale[(int64_t)n_blk * p.c_scale_ld + row] = scale;
      } else {
        int64_t out_row = row;
        if (p.scatter) {
          const int sid = p.sorted_ids[row];
          out_row = (int64_t)(sid & 0xFFFFFF) * p.topk + ((uint32_t)sid >> 24);
        }
        const int64_t off = out_row * p.c_ld + c0;
        if (p.c_dtype != BOLT_F32 && p.c_vec_ok && c0 + V <= n_cols) {
          uint32_t w[V / 2];
#pragma unroll
          for (int v = 0; v < V; v += 2)
            w[v / 2] = to_16bit(y[0][v], p.c_dtype) | (uint32_t)to_16bit(y[0][v + 1], p.c_dtype) << 16;
          uint16_t* dst = static_cast<uint16_t*>(p.c) + off;
          if constexpr (V == 8) *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
          else *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
        } else {
#pragma unroll
          for (int v = 0; v < V; ++v) {
            if (c0 + v >= n_cols) continue;
            if (p.c_dtype == BOLT_F32) static_cast<float*>(p.c)[off + v] = y[0][v];
            else static_cast<uint16_t*>(p.c)[off + v] = to_16bit(y[0][v], p.c_dtype);
          }
        }
      }
    }
    epilogue_sync();
  }
  if constexpr (!BS) {
    tc_fence_before();
    __syncwarp();
    if (ep.lane == 0) mbar_arrive(ep.bar_tempty + 8 * acc_stage);
  }
  return true;
}

template <int OPK, bool BS, int EPI, int KBS>
__global__ void __launch_bounds__(kThreads, 1)
k_stream_gemm(const __grid_constant__ CUtensorMap tma_b, const StreamParams p) {
  constexpr bool GATED = EPI != BOLT_EPI_STORE;
  static_assert(!GATED || KBS == 1, "a gated item has a gate half and an up half");
  constexpr int H = KBS == 1 ? 2 : 1;
  constexpr int RMAX = kMaxRows / KBS;
  constexpr int kElems = OPK == OP_F16 ? 64 : 128;   // K elements of a 128-byte block
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  uint8_t* rows_smem = smem + kStages * kWeightBytes;
  uint8_t* ring = rows_smem + kStages * kRowBytes;
  uint8_t* out_stage = ring + kScaleSlots * kSlotBytes;
  uint8_t* ctrl = out_stage + kStageOut;
  const uint32_t bar_full = smem_u32(ctrl);                    // [kStages]
  const uint32_t bar_empty = bar_full + 8 * kStages;           // [kStages]
  const uint32_t bar_tfull = bar_empty + 8 * kStages;          // [kAccStages]
  const uint32_t bar_tempty = bar_tfull + 8 * kAccStages;      // [kAccStages]
  const uint32_t bar_scale = bar_tempty + 8 * kAccStages;      // [kScaleSlots]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ctrl + 512);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(ctrl + 516);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar_full + 8 * s, 1 + kRowThreads);   // the weights' byte count, the row copies
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int i = 0; i < kAccStages; ++i) {
      mbar_init(bar_tfull + 8 * i, 1);
      mbar_init(bar_tempty + 8 * i, kEpilogue / 32);
    }
    for (int i = 0; i < kScaleSlots; ++i) mbar_init(bar_scale + 8 * i, kRowThreads);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int num_m = min(*p.num_valid, p.capacity) / 128;
  const int total = num_m * p.tiles_n;
  const int num_st = (p.num_kb + KBS - 1) / KBS;
  // As many CTAs as the fewest rounds need, all with the same number of items (one more or less):
  // a last round of a few items would run at a few CTAs' bandwidth.
  // Measured: Mixtral bf16, 896 items on 148 SMs, 322 -> 307 us; DeepSeek-V3 fp8 with 4 tokens 161 ->
  // 151 us; items of very unequal rows lose a little (Zipf-distributed routing, 213 -> 225 us).
  const int rounds = (total + (int)gridDim.x - 1) / (int)gridDim.x;
  const int stride = rounds > 0 ? (total + rounds - 1) / rounds : 1;
  // expert and the ids of the 128 rows (four per lane) of an item's row tile, one item ahead
  auto fetch = [&](int item, int& expert, int (&id)[4]) {
    const int m_blk = item / p.tiles_n;
    expert = p.expert_ids[m_blk];
#pragma unroll
    for (int i = 0; i < 4; ++i) id[i] = p.sorted_ids[(int64_t)m_blk * 128 + i * 32 + lane];
  };
  // calls body(m_blk, n_blk, expert, first row in the tile, rows, ids) for every item of this CTA in
  // order, whole warps at a time, until it returns false in any lane
  auto for_items = [&](auto body) {
    int expert_n = -1, id_n[4] = {-1, -1, -1, -1};
    int item = (int)blockIdx.x < stride ? (int)blockIdx.x : total;
    if (item < total) fetch(item, expert_n, id_n);
    for (; item < total; item += stride) {
      const int expert = expert_n;
      const int id[4] = {id_n[0], id_n[1], id_n[2], id_n[3]};
      if (item + stride < total) fetch(item + stride, expert_n, id_n);
      if (expert < 0 || expert >= p.num_experts) continue;
      const int m_blk = item / p.tiles_n, n_blk = item - m_blk * p.tiles_n;
      const int live = live_rows(id, p.num_tokens);
      for (int r0 = 0; r0 < live; r0 += RMAX) {
        const bool ok = body(m_blk, n_blk, expert, r0, min(RMAX, live - r0), id);
        if (__any_sync(0xffffffffu, !ok)) return;
      }
    }
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0) {
      // ------------------------------ weights ---------------------------------
      int s = 0;
      uint32_t ph = 0;
      for_items([&](int, int n_blk, int expert, int, int, const int (&)[4]) {
        bool ok = true;
        if (lane == 0) {
          for (int st = 0; st < num_st; ++st) {
            ok = mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, p.status, 1);
            if (!ok) break;
            const uint32_t full = bar_full + 8 * s;
            const int kbn = min(KBS, p.num_kb - st * KBS);
            mbar_expect_tx(full, kbn * (4 / KBS) * kBoxBytes);
            for (int kk = 0; kk < kbn; ++kk) {
#pragma unroll
              for (int b = 0; b < 4 / KBS; ++b) {
                const int brow = GATED ? (b >> 1) * p.n_half + n_blk * 128 + (b & 1) * 64
                                       : n_blk * (256 / KBS) + b * 64;
                tma_load_3d(smem_u32(smem) + s * kWeightBytes + (kk * (4 / KBS) + b) * kBoxBytes,
                            &tma_b, full, (st * KBS + kk) * kElems, brow, expert);
              }
            }
            if (++s == kStages) { s = 0; ph ^= 1; }
          }
        }
        return ok;
      });
    } else if (warp == 1) {
      // ------------------------------ MMA issuer --------------------------------
      int s = 0, last_cols = 0;
      uint32_t ph = 0, parity = 0, count = 0;
      for_items([&](int, int, int, int, int rows, const int (&)[4]) {
        bool ok = true;
        if (lane == 0) {
          const int cols = columns_for(rows);
          const uint32_t idesc = p.idesc | ((uint32_t)(cols >> 3) << 17);
          const int stages = acc_stages<KBS>(cols);
          int t = 0;
          if (BS) {
            if (cols != last_cols) {   // another division of TMEM: wait until all of it is free
              for (int i = 0; ok && i < kAccStages; ++i)
                ok = mbar_wait(bar_tempty + 8 * i, ((parity >> i) & 1u) ^ 1u, abort_flag, p.status, 2);
            }
            last_cols = cols;
          } else {
            t = count & 1u;
            ok = mbar_wait(bar_tempty + 8 * t, ((count >> 1) & 1u) ^ 1u, abort_flag, p.status, 2);
            ++count;
          }
          for (int st = 0; ok && st < num_st; ++st) {
            ok = mbar_wait(bar_full + 8 * s, ph, abort_flag, p.status, 3);
            if (!ok) break;
            const int kbn = min(KBS, p.num_kb - st * KBS);
            for (int kk = 0; kk < kbn; ++kk) {
              if (BS) {
                ok = mbar_wait(bar_tempty + 8 * t, ((parity >> t) & 1u) ^ 1u, abort_flag, p.status, 2);
                if (!ok) break;
              }
              tc_fence_after();
              // rows were written through the generic proxy, the MMA reads through the asynchronous one
              fence_async_smem();
              const uint64_t rdesc = make_smem_desc(smem_u32(rows_smem) + s * kRowBytes + kk * (RMAX * 128));
#pragma unroll
              for (int h = 0; h < H; ++h) {
                const uint64_t wdesc = make_smem_desc(smem_u32(smem) + s * kWeightBytes +
                                                      (kk + h) * (2 * kBoxBytes));
                const uint32_t d = tmem_base + (BS ? t * (H * cols) : t * 256) + h * cols;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  tc_mma<OPK>(d, wdesc + 2 * k, rdesc + 2 * k, idesc,
                              BS ? (k > 0) : (st > 0 || kk > 0 || k > 0));
              }
              if (BS) {
                tc_commit(bar_tfull + 8 * t);
                parity ^= 1u << t;
                if (++t == stages) t = 0;
              }
            }
            if (!ok) break;
            tc_commit(bar_empty + 8 * s);
            if (++s == kStages) { s = 0; ph ^= 1; }
          }
          if (!BS && ok) tc_commit(bar_tfull + 8 * t);
        }
        return ok;
      });
    } else {
      // ------------------------------ rows and scales ----------------------------
      // Thread t brings 16-byte column t % 8 of rows t / 8 + 8 i, placed where the 128-byte-swizzled
      // box copy would put it; rows past the last live one, up to the MMA's columns, are zeros.
      const int tid = (int)threadIdx.x - 64;
      const int c16 = tid & 7, r8 = tid >> 3;
      const uint32_t dst0 = smem_u32(rows_smem) + r8 * 128 + ((c16 ^ r8) << 4);
      const uint8_t* a16 = static_cast<const uint8_t*>(p.a) + c16 * 16;
      int s = 0;
      uint32_t ph = 0, kbi = 0;
      for_items([&](int m_blk, int n_blk, int expert, int r0, int rows, const int (&id)[4]) {
        bool ok = true;
        auto feed = [&](auto count_of) {
          constexpr int Q = decltype(count_of)::value;      // rows of this thread
          int src[Q];
#pragma unroll
          for (int i = 0; i < Q; ++i) {
            const int r = r0 + 8 * i + r8;
            const int w = r >> 5;                           // (the same in the whole warp)
            const int tok = __shfl_sync(0xffffffffu, w < 2 ? (w < 1 ? id[0] : id[1])
                                                           : (w < 3 ? id[2] : id[3]), r & 31) & 0xFFFFFF;
            src[i] = 8 * i + r8 < rows ? (p.gather ? tok : m_blk * 128 + r) : -1;
          }
          const float* sc = BS ? p.a_scale + m_blk * 128 + r0 + 4 * tid : nullptr;
          // weight scales of the two 128-row halves (threads 62 and 63)
          const float* wsc = nullptr;
          if (BS && tid >= 62) {
            const int nblocks = p.n / 128, h = tid - 62;
            const int nb = GATED ? n_blk + h * (p.n_half / 128) : min(n_blk * H + (h & (H - 1)), nblocks - 1);
            wsc = p.b_scale + ((int64_t)expert * nblocks + nb) * p.kb_scale_cols;
          }
          for (int st = 0; st < num_st; ++st) {
            ok = mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, p.status, 5);
            if (!ok) break;
            const int kbn = min(KBS, p.num_kb - st * KBS);
            for (int kk = 0; kk < kbn; ++kk) {
              const int kb = st * KBS + kk;
              const uint32_t dst = dst0 + s * kRowBytes + kk * (RMAX * 128);
#pragma unroll
              for (int i = 0; i < Q; ++i)
                cp_async_16(dst + i * 1024, a16 + (src[i] >= 0 ? src[i] * p.a_row_bytes + kb * 128 : 0),
                            src[i] >= 0 ? 16u : 0u);
              if (BS) {
                const uint32_t slot = kbi % kScaleSlots;
                ++kbi;
                if (tid < 2 * Q)   // 8 Q scales
                  cp_async_16(smem_u32(ring) + slot * kSlotBytes + 16 * tid, sc + kb * p.a_scale_ld, 16u);
                if (tid >= 62)
                  cp_async_4(smem_u32(ring) + slot * kSlotBytes + kMaxRows * 4 + 4 * (tid - 62), wsc + kb);
                cp_async_mbar_arrive_noinc(bar_scale + 8 * slot);
              }
            }
            cp_async_mbar_arrive_noinc(bar_full + 8 * s);
            if (++s == kStages) { s = 0; ph ^= 1; }
          }
        };
        if (rows <= 16) feed(std::integral_constant<int, 2>());
        else if (rows <= 32) feed(std::integral_constant<int, 4>());
        else if (rows <= 64) feed(std::integral_constant<int, 8>());
        else if constexpr (RMAX > 64) feed(std::integral_constant<int, 16>());
        return ok;
      });
      cp_async_wait_all();
    }
  } else {
    // ------------------------------ epilogue -----------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    Epilogue ep;
    ep.tmem = tmem_base;
    ep.bar_tfull = bar_tfull;
    ep.bar_tempty = bar_tempty;
    ep.bar_scale = bar_scale;
    ep.scale_ring = smem_u32(ring);
    ep.out_stage = out_stage;
    ep.abort_flag = abort_flag;
    ep.warp = warp - 4;
    ep.lane = lane;
    ep.parity = 0;
    ep.count = 0;
    for_items([&](int m_blk, int n_blk, int expert, int r0, int rows, const int (&)[4]) {
      const int row0 = m_blk * 128 + r0;
      const int t = columns_for(rows) / 2;
      if constexpr (BS) {
        if (t == 8) return finish_item<OPK, BS, EPI, KBS, 8>(p, ep, expert, n_blk, row0, rows, 8);
        if (t == 16) return finish_item<OPK, BS, EPI, KBS, 16>(p, ep, expert, n_blk, row0, rows, 16);
        if (t == 32) return finish_item<OPK, BS, EPI, KBS, 32>(p, ep, expert, n_blk, row0, rows, 32);
        return finish_item<OPK, BS, EPI, KBS, 64>(p, ep, expert, n_blk, row0, rows, 64);
      } else {
        return finish_item<OPK, BS, EPI, KBS, 0>(p, ep, expert, n_blk, row0, rows, t);
      }
    });
  }

  // ------------------------------ teardown ------------------------------------
  __syncwarp();
  if (*abort_flag) {
    // let copies that are still in flight land before the CTA's memory is released
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u)
                 : "memory");
}

template <int OPK, bool BS, int EPI, int KBS>
int launch(const CUtensorMap& mb, const StreamParams& p, int grid, cudaStream_t st) {
  auto kfn = k_stream_gemm<OPK, BS, EPI, KBS>;
  static std::atomic<bool> configured[kMaxDevices];
  // warps 0-3 drop to 56 registers, the eight epilogue warps rise to 224
  const int rc = configure_kernel(kfn, kSmemBytes, configured, 128, 56, 256, 224);
  if (rc != BOLT_OK) return rc;
  kfn<<<grid, kThreads, kSmemBytes, st>>>(mb, p);
  BOLT_LAUNCH_CHECK();
  return BOLT_OK;
}

template <int OPK, bool BS>
int launch_kind(int epi, int kbs, const CUtensorMap& mb, const StreamParams& p, int grid,
                cudaStream_t st) {
  switch (epi) {
    case BOLT_EPI_STORE:
      if constexpr (!BS) {
        if (kbs == 2) return launch<OPK, BS, BOLT_EPI_STORE, 2>(mb, p, grid, st);
      }
      return launch<OPK, BS, BOLT_EPI_STORE, 1>(mb, p, grid, st);
    case BOLT_EPI_SILU_MUL: return launch<OPK, BS, BOLT_EPI_SILU_MUL, 1>(mb, p, grid, st);
    default:
      if constexpr (BS) return launch<OPK, true, BOLT_EPI_SILU_MUL_QUANT, 1>(mb, p, grid, st);
      set_error("grouped_gemm: fused group quantisation needs a block-scaled kind");
      return BOLT_ERR_UNSUPPORTED;
  }
}

// one per kind, each compiled in a file of its own
#define BOLT_STREAM_KINDS(X) X(OP_F16, false) X(OP_F8, true) X(OP_F8, false) X(OP_I8, false) X(OP_I8, true)
#define BOLT_STREAM_EXTERN(OPK, BS)                                                          \
  extern template int launch_kind<OPK, BS>(int, int, const CUtensorMap&, const StreamParams&, int, \
                                           cudaStream_t);
#define BOLT_STREAM_DEFINE(OPK, BS)                                                          \
  template int launch_kind<OPK, BS>(int, int, const CUtensorMap&, const StreamParams&, int,  \
                                    cudaStream_t);

}  // namespace stream

// mb: tensor map over B [experts, n, k] with boxes of 64 rows x 128 bytes, 128-byte swizzle;
// arguments checked by the caller
int stream_gemm(const bolt_gemm_args* a, const CUtensorMap& mb, cudaStream_t st);

}  // namespace bolt
