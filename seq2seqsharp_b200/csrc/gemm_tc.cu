// Tensor-core GEMM for prefill and large-batch decode: y[M,N] = epilogue(x[M,K] * W[K,N]), fp16 or bf16 in,
// fp32 accumulate.
//
// sm_100a design (5th-generation tensor cores):
//  * operands are staged in shared memory by TMA tensor copies (cp.async.bulk.tensor, 128-byte swizzle, completion
//    on mbarriers): A = activations [M,K] row-major (K-major operand, box 64 k x 128 rows); B = the engine's packed
//    weight tiles, which are stored pre-swizzled (packed_tile_off), so the 128 columns x 32 k a stage needs from a
//    tile are one contiguous 8 KB range that a plain bulk copy lands in operand layout (MN-major, SWIZZLE_128B):
//    decode GEMV and GEMM share ONE copy of the weights;
//  * an elected lane of one warp issues tcgen05.mma (kind::f16) into tensor memory, tcgen05.commit hands shared-memory
//    stages back to the copying warp and signals the epilogue;
//  * epilogue warps read the accumulator with tcgen05.ld (32 lanes x 32 columns per instruction) and apply the
//    same fused epilogue as the GEMV: bias first, activation, gate product on interleaved columns, fp32 residual.
// Three kernels: up to 128 rows 128 x 128 tiles of one CTA (gemm_tc_kernel), more rows pairs of CTAs (gemm_tc_pair_kernel), rows
// sorted by the matrix they meet 128 x 256 tiles of one CTA (gemm_tc_grouped_kernel).
// Rows beyond M and K beyond the tensor are zero-filled by TMA, N is padded by the packed layout.
// Every mbarrier wait is bounded; on timeout an error word is raised, TMEM is freed and the kernel returns.
//
// Replaces cublasGemmEx (TensorSharp.CUDA/MatrixMul/CudaMatrixMulMM.cs:305-362, fp16 accumulate there) plus the bias
// copy, activation and residual kernels around it.
#include <cstdlib>

#include "tc_common.cuh"

namespace tsb {

constexpr int kBM = 128, kBN = 128, kBK = 64;
// Stages of 32 KB.  Three: two CTAs per SM, so one CTA's epilogue overlaps the other's mainloop.  Six: one CTA per SM, taken when there are
// no more CTAs than SMs.  What bounds these launches is the way of the operands (about 1 us from HBM) and a fixed 6 us of prologue and
// epilogue.  Products issued by a warp's elected lane, before (a thread's branch) -> now: 100 x 4096 x 4096 with residual 32 -> 18 us,
// 128 x 8192 x 2048 47 -> 34, 128 x 2048 x 3072 17 -> 12.
constexpr int kTcStages = 3, kTcDeepStages = 6;
constexpr int tc_smem(int stages) { return stages * (kBM + kBN) * kBK * 2 + 1024 + 256; }
constexpr int kTcThreads = 256;
constexpr int kABytes = kBM * kBK * 2;  // 16 KB
constexpr int kBBytes = kBN * kBK * 2;  // 16 KB
// Raised by a kernel whose bounded wait ran out; read and cleared by tc_take_error().
__device__ int g_tc_error;

struct TcArgs {
  int M, N, K;        // logical sizes (N = packed column count actually used, multiple of 8)
  int KB;             // packed 32-row tiles along K
  int ksplit;         // CTAs sharing one output tile along K (grid.z); > 1 only when there are few tiles (small M)
  float* partials;    // [ksplit][M][Npad] raw fp32 accumulators, Npad = gridDim.x * 128
  unsigned int* counters;  // one per output tile, zero on entry, self-resetting
  int* error_flag;
  const unsigned char* Wp;  // packed weight tiles
  unsigned wait_limit;      // polls of a wait before the CTA gives up
  int kind;                 // TcKind: what the 16-byte epilogue has to read and write; kTcAny: element by element
  Epilogue ep;
};

// Fused epilogue for 32 consecutive columns of one row: bias first, activation, gate product on interleaved
// (a_j, g_j) column pairs, gate, fp32 residual, store in the model type or fp32.
template <typename H>
__device__ __forceinline__ void tc_finish(const TcArgs& a, int row, int col0, const float* v) {
  const H* bias = reinterpret_cast<const H*>(a.ep.bias);
  if (!a.ep.glu) {
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int col = col0 + j;
      if (col < a.N) ep_store<H>(a.ep, (size_t)row * a.N + col, ep_act(v[j] + (bias ? to_f<H>(bias[col]) : 0.0f), a.ep.act));
    }
  } else {
    const int No = a.N / 2;
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const int col = col0 + j;
      if (col + 1 < a.N) {
        const float av = v[j] + (bias ? to_f<H>(bias[col]) : 0.0f), gv = v[j + 1] + (bias ? to_f<H>(bias[col + 1]) : 0.0f);
        ep_store<H>(a.ep, (size_t)row * No + (col >> 1), ep_glu(av, gv, a.ep));
      }
    }
  }
}

// The same epilogue for 32 rows x 32 columns of a warp when every pointer is 16-byte aligned and N is a multiple of 32 (TcArgs::kind > 0).
// The sums cross the warp's 4 KB of shared memory (16-byte units XOR-ed with the row: conflict-free both ways), so that a lane finishes
// four neighbouring columns of eight rows and residual, gate and output are whole 32-byte sectors of few rows per instruction.
// What the epilogue reads is on its way one chunk ahead (TcAhead: a register is refilled for the next chunk as soon as it is used): the
// output may be the residual itself, so no load may pass a store by the compiler's hand, and fetched where they were needed the eight
// residual rows of a chunk were eight trips to memory one after the other (4096 x 2048 x 2048 with residual 103 us, now 33).
// Which of these an output has, and its activation, are decided once per chunk and not per element: with the choice inside the loop every
// chunk fetched the code of all activations.
constexpr int kStageFloats = 32 * 32;
enum TcKind { kTcAny = 0, kTcRows16 = 1, kTcResidual = 2, kTcGateResidual = 3, kTcMixed = 4 };   // y | residual -> y32 | gate, residual -> y32 | the rest
struct TcAhead {
  uint2 b;      // as loaded: nothing may wait for it before it is used
  float4 r[8];
  uint2 g[8];
};
// a lane's place in a tile: element of the output at (its first row, its first column), elements between its rows
struct TcLane {
  size_t o;
  int step;
};
__device__ __forceinline__ TcLane tc_lane(const TcArgs& a, int row0, int n0) {
  const int lane = (int)threadIdx.x & 31, No = a.ep.glu ? a.N >> 1 : a.N, col = n0 + (lane & 7) * 4;
  TcLane l;
  l.o = (size_t)(row0 + (lane >> 3)) * No + (a.ep.glu ? col >> 1 : col);
  l.step = 4 * No;
  return l;
}
// bias, and rows `it` of residual and gate, of the chunk that starts c columns into the tile's columns n0 ..
template <typename H>
__device__ __forceinline__ void tc_ahead_bias(const TcArgs& a, int col0, TcAhead& f) {
  if (a.ep.bias && col0 + 32 <= a.N) f.b = *reinterpret_cast<const uint2*>(reinterpret_cast<const H*>(a.ep.bias) + col0 + ((int)threadIdx.x & 7) * 4);
}
template <typename H, int KIND>
__device__ __forceinline__ void tc_ahead_row(const TcArgs& a, const TcLane& l, int c, int it, bool live, TcAhead& f) {
  if (!live) return;
  const size_t o = l.o + c + (size_t)(it * (int64_t)l.step);
  if (KIND == kTcGateResidual) f.g[it] = *reinterpret_cast<const uint2*>(reinterpret_cast<const H*>(a.ep.gate) + o);
  f.r[it] = *reinterpret_cast<const float4*>(a.ep.residual + o);
}
// of a tile's first chunk
template <typename H>
__device__ __forceinline__ void tc_ahead(const TcArgs& a, const TcLane& l, int n_live, int n0, TcAhead& f) {
  if (a.kind == kTcAny) return;
  f.b = make_uint2(0u, 0u);
  tc_ahead_bias<H>(a, n0, f);
  if (a.kind == kTcRows16 || a.kind == kTcMixed || n0 + 32 > a.N) return;
  const int r = ((int)threadIdx.x & 31) >> 3;
  if (a.kind == kTcResidual) {
#pragma unroll
    for (int it = 0; it < 8; ++it) tc_ahead_row<H, kTcResidual>(a, l, 0, it, it * 4 + r < n_live, f);
  } else {
#pragma unroll
    for (int it = 0; it < 8; ++it) tc_ahead_row<H, kTcGateResidual>(a, l, 0, it, it * 4 + r < n_live, f);
  }
}
// chunk c .. c + 31 of the tile's columns n0 ..; f: of this chunk, refilled for the next one if there is one (more)
template <typename H, int ACT, bool GLU, int KIND>
__device__ __forceinline__ void tc_finish_as(const TcArgs& a, const TcLane& l, int n_live, int n0, int c, bool more, const float* stage, TcAhead& f) {
  const int lane = (int)threadIdx.x & 31, r = lane >> 3, q = lane & 7;
  const float2 b01 = Pair16<H>::get(f.b.x), b23 = Pair16<H>::get(f.b.y);
  const float b0 = b01.x, b1 = b01.y, b2 = b23.x, b3 = b23.y;
  if (more) tc_ahead_bias<H>(a, n0 + c + 32, f);
  const size_t o = l.o + (GLU ? c >> 1 : c);
#pragma unroll (ACT == TSB200_ACT_NONE ? 8 : 2)
  for (int it = 0; it < 8; ++it) {
    const bool live = it * 4 + r < n_live;
    float4 t = reinterpret_cast<const float4*>(stage)[(it * 4 + r) * 8 + (q ^ ((it & 1) * 4 + r))];
    t.x += b0; t.y += b1; t.z += b2; t.w += b3;
    const size_t oi = o + (size_t)(it * (int64_t)l.step);
    if constexpr (GLU) {
      Epilogue ep;
      ep.act = ACT; ep.glu_limit = a.ep.glu_limit; ep.glu_slope = a.ep.glu_slope; ep.glu_shift = a.ep.glu_shift;
      const uint32_t y = Pair16<H>::put(ep_glu(t.x, t.y, ep), ep_glu(t.z, t.w, ep));
      if (live) *reinterpret_cast<uint32_t*>(reinterpret_cast<H*>(a.ep.y) + oi) = y;
    } else {
      t.x = ep_act(t.x, ACT); t.y = ep_act(t.y, ACT); t.z = ep_act(t.z, ACT); t.w = ep_act(t.w, ACT);
      if constexpr (KIND == kTcGateResidual) {
        const float2 g0 = Pair16<H>::get(f.g[it].x), g1 = Pair16<H>::get(f.g[it].y);
        t.x = __fmul_rn(t.x, g0.x); t.y = __fmul_rn(t.y, g0.y); t.z = __fmul_rn(t.z, g1.x); t.w = __fmul_rn(t.w, g1.y);   // rounded before the sum
      }
      if constexpr (KIND != kTcRows16) {
        t.x += f.r[it].x; t.y += f.r[it].y; t.z += f.r[it].z; t.w += f.r[it].w;
        if (more) tc_ahead_row<H, KIND>(a, l, c + 32, it, live && n0 + c + 64 <= a.N, f);
        if (live) *reinterpret_cast<float4*>(a.ep.y32 + oi) = t;
      } else {
        if (live) *reinterpret_cast<uint2*>(reinterpret_cast<H*>(a.ep.y) + oi) = make_uint2(Pair16<H>::put(t.x, t.y), Pair16<H>::put(t.z, t.w));
      }
    }
  }
}
// what no model asks for (a 16-bit output with a residual, fp32 without one, a gate alone, a gated product with any of these): small code
template <typename H>
__device__ __forceinline__ void tc_finish_mixed(const TcArgs& a, const TcLane& l, int n_live, int c, const float* stage, uint2 bias) {
  const int lane = (int)threadIdx.x & 31, r = lane >> 3, q = lane & 7;
  const float2 b01 = Pair16<H>::get(bias.x), b23 = Pair16<H>::get(bias.y);
#pragma unroll 1
  for (int it = 0; it < 8; ++it) {
    if (it * 4 + r >= n_live) break;
    const float4 t4 = reinterpret_cast<const float4*>(stage)[(it * 4 + r) * 8 + (q ^ ((it & 1) * 4 + r))];
    float t[4] = {t4.x + b01.x, t4.y + b01.y, t4.z + b23.x, t4.w + b23.y};
    const size_t o = l.o + (a.ep.glu ? c >> 1 : c) + (size_t)(it * (int64_t)l.step);
    if (a.ep.glu) {
      t[0] = ep_glu(t[0], t[1], a.ep);
      t[1] = ep_glu(t[2], t[3], a.ep);
    }
#pragma unroll 1
    for (int e = 0; e < (a.ep.glu ? 2 : 4); ++e) {
      const float v = e == 0 ? t[0] : (e == 1 ? t[1] : (e == 2 ? t[2] : t[3]));
      ep_store<H>(a.ep, o + e, a.ep.glu ? v : ep_act(v, a.ep.act));
    }
  }
}
// all lanes of the warp: v holds row row0 + lane, columns n0 + c .. + 31; rows row0 .. row0 + n_live - 1 exist
template <typename H>
__device__ __forceinline__ void tc_finish_rows(const TcArgs& a, const TcLane& l, int row0, int n_live, int n0, int c, bool more, const float* v, float* stage, TcAhead& f) {
  const int lane = (int)threadIdx.x & 31;
  if (a.kind == kTcAny || n0 + c + 32 > a.N) {
    if (lane < n_live) tc_finish<H>(a, row0 + lane, n0 + c, v);
    return;
  }
  float4* mine = reinterpret_cast<float4*>(stage) + lane * 8;
#pragma unroll
  for (int q = 0; q < 8; ++q) mine[q ^ (lane & 7)] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  __syncwarp();
#define TSB_AS(ACT, GLU, KIND) tc_finish_as<H, ACT, GLU, KIND>(a, l, n_live, n0, c, more, stage, f)
  if (a.kind == kTcResidual) {
    TSB_AS(TSB200_ACT_NONE, false, kTcResidual);
  } else if (a.kind == kTcGateResidual) {
    TSB_AS(TSB200_ACT_NONE, false, kTcGateResidual);
  } else if (a.kind == kTcMixed) {
    tc_finish_mixed<H>(a, l, n_live, c, stage, f.b);
    if (more) tc_ahead_bias<H>(a, n0 + c + 32, f);
  } else if (a.ep.glu) {
    switch (a.ep.act) {
      case TSB200_ACT_SILU:
      case TSB200_ACT_SWIGLU: TSB_AS(TSB200_ACT_SWIGLU, true, kTcRows16); break;
      case TSB200_ACT_CLAMP_GLU: TSB_AS(TSB200_ACT_CLAMP_GLU, true, kTcRows16); break;
      case TSB200_ACT_RELU: TSB_AS(TSB200_ACT_RELU, true, kTcRows16); break;
      case TSB200_ACT_LEAKYRELU: TSB_AS(TSB200_ACT_LEAKYRELU, true, kTcRows16); break;
      case TSB200_ACT_GELU: TSB_AS(TSB200_ACT_GELU, true, kTcRows16); break;
      case TSB200_ACT_SIGMOID: TSB_AS(TSB200_ACT_SIGMOID, true, kTcRows16); break;
      default: TSB_AS(TSB200_ACT_NONE, true, kTcRows16); break;
    }
  } else {
    switch (a.ep.act) {
      case TSB200_ACT_RELU: TSB_AS(TSB200_ACT_RELU, false, kTcRows16); break;
      case TSB200_ACT_SILU:
      case TSB200_ACT_SWIGLU: TSB_AS(TSB200_ACT_SILU, false, kTcRows16); break;
      case TSB200_ACT_LEAKYRELU: TSB_AS(TSB200_ACT_LEAKYRELU, false, kTcRows16); break;
      case TSB200_ACT_GELU: TSB_AS(TSB200_ACT_GELU, false, kTcRows16); break;
      case TSB200_ACT_SIGMOID: TSB_AS(TSB200_ACT_SIGMOID, false, kTcRows16); break;
      default: TSB_AS(TSB200_ACT_NONE, false, kTcRows16); break;
    }
  }
#undef TSB_AS
  __syncwarp();   // the warp's shared memory is free again
}
// One piece of a tile: COLS columns from n0 on of the warp's 32 rows, out of TMEM (acc) and through the epilogue.
// add(c, v): what others have of the sums of columns c .. c + 31.
template <typename H, int COLS, typename Add>
__device__ __forceinline__ void tc_drain(const TcArgs& a, const TcLane& l, uint32_t acc, int row0, int n_live, int n0, float* stage, TcAhead& f, Add add) {
#pragma unroll 1
  for (int c = 0; c < COLS && n_live > 0; c += 32) {
    uint32_t u[32];
    tmem_ld32(acc + c, u);
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(u[j]);
    add(c, v);
    tc_finish_rows<H>(a, l, row0, n_live, n0, c, c + 32 < COLS, v, stage, f);
  }
}

template <typename H, int kTcStages>
__global__ void __launch_bounds__(kTcThreads, kTcStages == 3 ? 2 : 1) gemm_tc_kernel(const __grid_constant__ CUtensorMap mapA, TcArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // carve: [stages][A 16K][B 16K] (1024-byte aligned for the 128B swizzle atoms), then barriers
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sA = s_u32(smem), sB = sA + kTcStages * kABytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kTcStages * (kABytes + kBBytes));
  const uint32_t full = s_u32(bars), empty = full + kTcStages * 8, acc_ready = empty + kTcStages * 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kTcStages + 1);
  __shared__ int s_err;

  const int tid = threadIdx.x, lane = tid & 31, w = warp_index();
  const int n_tile = blockIdx.x;   // one tile of rows
  const int k_total = (a.K + kBK - 1) / kBK;
  const int k_per = (k_total + a.ksplit - 1) / a.ksplit;
  const int k_begin = blockIdx.z * k_per;
  const int k_iters = max(0, min(k_total, k_begin + k_per) - k_begin);  // k blocks of this CTA
  __shared__ int s_last;

  if (tid == 0) {
    for (int i = 0; i < 2 * kTcStages + 1; ++i) tc_mbar_init(bars + i, 1);
    s_err = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (w == 2) {  // TMEM allocation: 128 columns of fp32 accumulator (one warp, whole-warp instruction)
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(kBN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_acc = *tmem_slot;
  pdl_trigger();   // after the allocation: a successor's CTA on this SM cannot take the columns first
  pdl_wait();

  volatile int* err = &s_err;
  if (w == 0) {
    // ---------------- copies.  B: this CTA's 128 columns are boxes (2p, 2p+1) of column tile ct: 8 KB contiguous in every packed k tile
    const unsigned char* wsrc = a.Wp + ((size_t)(n_tile >> 1) * a.KB + k_begin * 2) * 16384 + (size_t)(n_tile & 1) * 8192;
    int s = 0, asked = 0;
    unsigned phase = 1;
    for (; asked < k_iters; ++asked, wsrc += 32768) {
      if (asked >= kTcStages && !tc_wait_or(empty + s * 8, phase, err, a.wait_limit)) break;
      const bool two = (k_begin + asked) * 2 + 1 < a.KB;  // the last 64-k block of an odd tile count has one packed tile only
      const uint32_t bar = full + s * 8, dB = sB + s * kBBytes;
      tc_mbar_expect_el(bar, kABytes + (two ? 16384 : 8192));
      tma_load_2d_el(sA + s * kABytes, &mapA, (k_begin + asked) * kBK, 0, bar);
      tc_bulk_g2s_el(dB, wsrc, 8192, bar);
      if (two) tc_bulk_g2s_el(dB + 8192, wsrc + 16384, 8192, bar);
      if (++s == kTcStages) s = 0, phase ^= 1;
    }
    tc_land(full, kTcStages, asked);
  } else if (w == 1) {
    // ---------------- products.  Instruction descriptor: D fp32, A/B fp16 or bf16, A K-major, B MN-major, N = 128, M = 128
    const uint32_t idesc = (1u << 4) | (Pair16<H>::kUmmaFormat << 7) | (Pair16<H>::kUmmaFormat << 10) | (0u << 15) | (1u << 16) | ((uint32_t)(kBN >> 3) << 17) |
                           ((uint32_t)(kBM >> 4) << 24);
    // A (K-major, SW128): rows of 128 B, 8-row atoms 1024 B apart; 16 k = 32 B along the row.  B (MN-major, SW128), stage = [k tile 2]
    // [64-n box 2][32 k][128 B]: k groups of 8 are 1024 B apart (SBO), the second 64-n box is 4096 B away (LBO); 16 k = two groups = 2048 B;
    // the second k tile starts at 8192 B
    const uint32_t hi = desc_hi(1024), a0 = desc_lo(sA, 16), b0 = desc_lo(sB, 4096);
    int s = 0;
    unsigned phase = 0;
    for (int it = 0; it < k_iters; ++it) {
      if (!tc_wait_or(full + s * 8, phase, err, a.wait_limit)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t ad = a0 + s * (kABytes >> 4), bd = b0 + s * (kBBytes >> 4);
      umma_el(tmem_acc, ad, hi, bd, hi, idesc, it > 0);
      umma_el(tmem_acc, ad + 2, hi, bd + 128, hi, idesc, 1);
      if ((k_begin + it) * 2 + 1 < a.KB) {   // no second packed tile: its stage half was not filled
        umma_el(tmem_acc, ad + 4, hi, bd + 512, hi, idesc, 1);
        umma_el(tmem_acc, ad + 6, hi, bd + 640, hi, idesc, 1);
      }
      umma_commit_el(empty + s * 8);  // frees the stage when these products have read it
      if (++s == kTcStages) s = 0, phase ^= 1;
    }
    umma_commit_el(acc_ready);    // accumulator complete
    tc_wait_short(acc_ready, 0);
  } else if (w >= 4) {
    // ---------------- epilogue: warp (w - 4) owns TMEM lanes 32*(w-4) .. +31 = rows of the tile
    const int q = w - 4;
    const bool ok = tc_wait_or(acc_ready, 0, err, a.wait_limit);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int row = q * 32 + lane;
    const int n0 = n_tile * kBN;
    const bool live = ok && row < a.M;
    const int n_live = ok ? min(32, a.M - q * 32) : 0;
    float* stage = reinterpret_cast<float*>(smem) + q * kStageFloats;   // every product has read its operands
    const size_t Npad = (size_t)gridDim.x * kBN;
    const TcLane at = tc_lane(a, row - lane, n0);
    TcAhead ahead;
    const uint32_t acc = tmem_acc + ((uint32_t)(q * 32) << 16);
    if (a.ksplit == 1) {
      tc_ahead<H>(a, at, n_live, n0, ahead);
      tc_drain<H, kBN>(a, at, acc, row - lane, n_live, n0, stage, ahead, [](int, float*) {});
    } else {
      // raw partial sums of this K slice; the last CTA of the tile adds the slices in a fixed order
#pragma unroll 1
      for (int c = 0; c < kBN; c += 32) {
        uint32_t v[32];
        tmem_ld32(acc + c, v);
        if (!live) continue;
        float4* dst = reinterpret_cast<float4*>(a.partials + ((size_t)blockIdx.z * a.M + row) * Npad + n0 + c);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          dst[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]),
                               __uint_as_float(v[4 * j + 3]));
      }
    }
    if (a.ksplit > 1) {
      __threadfence();
      named_sync<1, 128>();  // the four epilogue warps
      if (w == 4 && lane == 0) {
        const unsigned int prev = atomicAdd(&a.counters[n_tile], 1u);
        s_last = (prev == (unsigned int)(a.ksplit - 1));
        if (s_last) a.counters[n_tile] = 0u;
      }
      named_sync<1, 128>();
      if (s_last) {
        __threadfence();
        tc_ahead<H>(a, at, n_live, n0, ahead);
        tc_drain<H, kBN>(a, at, acc, row - lane, n_live, n0, stage, ahead, [&](int c, float* f) {
#pragma unroll
          for (int j = 0; j < 32; ++j) f[j] = 0.0f;
          // two K slices in flight per round trip, added in slice order (bitwise reproducible)
          int z = live ? 0 : a.ksplit;
          for (; z + 1 < a.ksplit; z += 2) {
            const float4* s0 = reinterpret_cast<const float4*>(a.partials + ((size_t)z * a.M + row) * Npad + n0 + c);
            const float4* s1 = reinterpret_cast<const float4*>(a.partials + ((size_t)(z + 1) * a.M + row) * Npad + n0 + c);
            float4 t0[8], t1[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              t0[j] = __ldcg(s0 + j);
              t1[j] = __ldcg(s1 + j);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              f[4 * j] += t0[j].x; f[4 * j + 1] += t0[j].y; f[4 * j + 2] += t0[j].z; f[4 * j + 3] += t0[j].w;
              f[4 * j] += t1[j].x; f[4 * j + 1] += t1[j].y; f[4 * j + 2] += t1[j].z; f[4 * j + 3] += t1[j].w;
            }
          }
          for (; z < a.ksplit; ++z) {
            const float4* src = reinterpret_cast<const float4*>(a.partials + ((size_t)z * a.M + row) * Npad + n0 + c);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 t = __ldcg(src + j);
              f[4 * j] += t.x; f[4 * j + 1] += t.y; f[4 * j + 2] += t.z; f[4 * j + 3] += t.w;
            }
          }
        });
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (w == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"(kBN) : "memory");
  }
  if (tid == 0 && s_err) {
    g_tc_error = 1;
    if (a.error_flag) *a.error_flag = 1;
  }
}

// ---- persistent kernels of more than one row tile -----------------------------------------------------------------------
// Warp 0: copies; warp 1: TMEM and products; warps 2..9: epilogue (two per quarter of the TMEM lanes, each half of a tile's columns).
// The accumulator is double buffered: the epilogue drains one piece of work while the products of the next are running and the copies
// run ahead across pieces.
constexpr int kPThreads = 320, kPWarps = 8;
constexpr int kPStageBytes = kPWarps * kStageFloats * 4;
constexpr int kP_BN = 256;

struct TcTile {
  int m_tile, n_tile;
};
// bands of `rows` row tiles; inside a band column-major (all rows of a column tile are neighbours in time): the CTAs that run at the same
// time share A and B tiles in L2
__device__ __forceinline__ TcTile tc_tile_of(int t, int m_tiles, int n_tiles, int rows) {
  const int band = t / (rows * n_tiles);
  const int here = min(rows, m_tiles - band * rows);
  const int r = t - band * rows * n_tiles;
  TcTile o;
  o.n_tile = r / here;
  o.m_tile = band * rows + r % here;
  return o;
}
// Rows sorted by the matrix they meet, in blocks of up to 128 (RowGroups): row tile m covers rows [row0, row0 + rows) and multiplies them
// with the packed matrix `matrix`; the number of blocks is read from the device.  One CTA per SM walks tiles of 128 rows x 256 columns
// (blocks of different matrices share no columns, so a CTA pair has nothing to share either).
constexpr int kGStages = 4;
constexpr int kGStage = kABytes + kP_BN * kBK * 2;   // 48 KB
constexpr int kGSmem = kGStages * kGStage + 1024 + 256 + kPStageBytes;
template <typename H>
__global__ void __launch_bounds__(kPThreads, 1) gemm_tc_grouped_kernel(const __grid_constant__ CUtensorMap mapA, TcArgs a, int n_tiles, RowGroups g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sA = s_u32(smem), sB = sA + kGStages * kABytes;
  float* stages = reinterpret_cast<float*>(smem + kGStages * kGStage);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kGStages * kGStage + kPStageBytes);
  const uint32_t full = s_u32(bars), empty = full + kGStages * 8, acc_full = empty + kGStages * 8, acc_empty = acc_full + 16, drain = acc_empty + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kGStages + 5);
  __shared__ int s_err;

  const int tid = threadIdx.x, lane = tid & 31, w = warp_index();
  const int k_total = (a.K + kBK - 1) / kBK;

  if (tid == 0) {
    for (int i = 0; i < 2 * kGStages + 2; ++i) tc_mbar_init(bars + i, 1);
    for (int i = 0; i < 2; ++i) tc_mbar_init(bars + 2 * kGStages + 2 + i, kPWarps);
    tc_mbar_init(bars + 2 * kGStages + 4, 1);
    s_err = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (w == 1) {  // all 512 TMEM columns: two accumulators of 256
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();
  pdl_wait();
  const int m_tiles = min(*g.n_blocks, g.max_blocks), n_total = m_tiles * n_tiles;
  volatile int* err = &s_err;

  if (w == 0) {
    // ---------------- copies
    int s = 0, asked = 0;
    unsigned phase = 1;   // parity of the ring's previous round
    bool ok = true;
    for (int t = blockIdx.x; t < n_total && ok; t += gridDim.x) {
      const TcTile tl = tc_tile_of(t, m_tiles, n_tiles, 16);
      const RowBlock rb = g.table[tl.m_tile];
      const unsigned char* wsrc = a.Wp + (size_t)rb.matrix * g.matrix_bytes + ((size_t)tl.n_tile * a.KB) * 16384;
      for (int it = 0; it < k_total; ++it, wsrc += 32768) {
        if (asked >= kGStages && !(ok = tc_wait_or(empty + s * 8, phase, err, a.wait_limit))) break;
        const bool two = it * 2 + 1 < a.KB;
        const uint32_t bar = full + s * 8, dB = sB + s * 32768;
        tc_mbar_expect_el(bar, kABytes + (two ? 32768 : 16384));
        tma_load_2d_el(sA + s * kABytes, &mapA, it * kBK, rb.row0, bar);
        tc_bulk_g2s_el(dB, wsrc, 16384, bar);
        if (two) tc_bulk_g2s_el(dB + 16384, wsrc + 16384, 16384, bar);
        ++asked;
        if (++s == kGStages) s = 0, phase ^= 1;
      }
    }
    tc_land(full, kGStages, asked);
  } else if (w == 1) {
    // ---------------- products.  Instruction descriptor: fp32 accumulator, A K-major, B MN-major, N = 256, M = 128
    const uint32_t idesc = (1u << 4) | (Pair16<H>::kUmmaFormat << 7) | (Pair16<H>::kUmmaFormat << 10) | (1u << 16) | ((uint32_t)(kP_BN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
    // B stage = [k tile 2][64-n box 4][32 k][128 B]: boxes 4096 B apart (LBO), 8-k groups 1024 B apart (SBO), 16 k = 2048 B, the second k tile
    // at 16384 B
    const uint32_t hi = desc_hi(1024), a0 = desc_lo(sA, 16), b0 = desc_lo(sB, 4096);
    int s = 0, n_done = 0;
    unsigned phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n_total && ok; t += gridDim.x, ++n_done) {
      const int buf = n_done & 1;
      if (n_done >= 2 && !(ok = tc_wait_or(acc_empty + buf * 8, (unsigned)(((n_done >> 1) - 1) & 1), err, a.wait_limit))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem_base + buf * kP_BN;
      for (int it = 0; it < k_total; ++it) {
        if (!(ok = tc_wait_or(full + s * 8, phase, err, a.wait_limit))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t ad = a0 + s * (kABytes >> 4), bd = b0 + s * (32768 >> 4);
        umma_el(acc, ad, hi, bd, hi, idesc, it > 0);
        umma_el(acc, ad + 2, hi, bd + 128, hi, idesc, 1);
        if (it * 2 + 1 < a.KB) {
          umma_el(acc, ad + 4, hi, bd + 1024, hi, idesc, 1);
          umma_el(acc, ad + 6, hi, bd + 1152, hi, idesc, 1);
        }
        umma_commit_el(empty + s * 8);
        if (++s == kGStages) s = 0, phase ^= 1;
      }
      if (ok) umma_commit_el(acc_full + buf * 8);
    }
    umma_commit_el(drain);
    tc_wait_short(drain, 0);
  } else if (w >= 2) {
    // ---------------- epilogue: TMEM lanes 32 (w % 4) .. = rows of the tile, columns 128 ((w - 2) / 4) ..
    const int q = w & 3, half = (w - 2) >> 2;
    float* stage = stages + (w - 2) * kStageFloats;
    TcAhead ahead;
    int n_done = 0;
    for (int t = blockIdx.x; t < n_total; t += gridDim.x, ++n_done) {
      const TcTile tl = tc_tile_of(t, m_tiles, n_tiles, 16);
      const RowBlock rb = g.table[tl.m_tile];
      const int buf = n_done & 1, row0 = rb.row0 + q * 32, n0 = tl.n_tile * kP_BN + half * 128;
      const int n_live = min(32, min(rb.rows - q * 32, a.M - row0));
      const TcLane at = tc_lane(a, row0, n0);
      tc_ahead<H>(a, at, n_live, n0, ahead);
      if (!tc_wait_or(acc_full + buf * 8, (unsigned)((n_done >> 1) & 1), err, a.wait_limit)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      tc_drain<H, 128>(a, at, tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * kP_BN + half * 128), row0, n_live, n0, stage, ahead, [](int, float*) {});
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty + buf * 8) : "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (w == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
  if (tid == 0 && s_err) {
    g_tc_error = 1;
    if (a.error_flag) *a.error_flag = 1;
  }
}

// A cluster of two CTAs works on tiles of 256 rows x BN columns (tcgen05 cta_group::2): each CTA brings 128 rows of A and HALF of the columns
// of B into its shared memory, the leader's one thread issues the products for both, each CTA's TMEM receives its own 128 rows.
// What bounds it: the tensor pipe, from about 4 waves on the power limit (16384 x 2048 x 16384 751 us = 1464 TFLOP/s, cuBLAS 749); an SM takes
// in about 64 bytes per clock from L2, a tile of one CTA needs 94 at full tensor rate (128 x 256) or 128 (128 x 128), a pair 64.  A step of
// 64 k whose operands are there takes 470 clocks for 256 columns and 296 for 128; in whole launches, operands from memory, 0.34 and 0.19 us (launch_pair).  With one 128 x 128 tile per CTA, or 128 x 256 on a CTA of its own,
// products issued by a thread and the epilogue's loads where they are needed, us before -> now: 1024 x 8192 x 2048 with residual 68 -> 30,
// 1024 x 2048 x 16384 gated 62 -> 51, 1273 x 4096 x 4096 with residual 111 -> 42, 1273 x 11008 x 4096 166 -> 100, 16384 x 2048 x 2048 with
// residual 333 -> 112, 256 x 11008 x 4096 80 -> 36.
// The copies of both CTAs report to the leader's barrier (the .cta_group::2 form of the tensor copy), the commits hand stages back to both;
// both operands therefore come by tensor copies, the packed weights as rows of 128 bytes that are laid down as they are stored.
// Tried and not kept: sharing tiles out so that all pairs end together (partial sums through L2): the pairs are then at different k at any time
// and no longer find each other's operands in L2, and the sums cost 5 to 10 us (2048 x 11008 x 4096 190 us against 137, 1273 x 4096 x 4096
// 39 against 42).
template <int BN>
struct PairTile {
  static constexpr int kB = BN / 2 * kBK * 2;               // B bytes of a stage and CTA
  static constexpr int kStages = BN == 256 ? 6 : 8;
  static constexpr int kStage = kABytes + kB;
  static constexpr int kSmem = kStages * kStage + 1024 + 256 + kPStageBytes;
  static constexpr int kCols = BN / 2;                      // columns of an epilogue warp
};

__device__ __forceinline__ uint32_t tc_leader_addr(uint32_t addr) {   // the same place in the shared memory of CTA 0 of the pair
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void tc_pair_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}" ::"r"(dst), "l"(map),
      "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tc_pair_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}" ::"r"(dst), "l"(map),
      "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

template <typename H, int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPThreads, 1)
    gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, TcArgs a, int m_tiles, int n_tiles) {
  typedef PairTile<BN> P;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sA = s_u32(smem), sB = sA + P::kStages * kABytes;
  float* stages = reinterpret_cast<float*>(smem + P::kStages * P::kStage);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + P::kStages * P::kStage + kPStageBytes);
  // full: the leader's counts the copies of both CTAs; acc_empty: the leader's, both CTAs' epilogue warps arrive
  const uint32_t full = s_u32(bars), empty = full + P::kStages * 8, acc_full = empty + P::kStages * 8, acc_empty = acc_full + 16, drain = acc_empty + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * P::kStages + 5);
  __shared__ int s_err;

  const int tid = threadIdx.x, lane = tid & 31, w = warp_index();
  const int rank = (int)(blockIdx.x & 1), pair = (int)(blockIdx.x >> 1), n_pairs = (int)(gridDim.x >> 1);
  const int k_total = (a.K + kBK - 1) / kBK, n_total = m_tiles * n_tiles;
  constexpr uint32_t kTmem = 2 * BN;
  __shared__ int2 s_peer;   // from the other CTA: whether it has given up, and the stages it has asked for
  int asked = 0;            // (warp 0)

  if (tid == 0) {
    for (int i = 0; i < 2 * P::kStages + 2; ++i) tc_mbar_init(bars + i, 1);
    for (int i = 0; i < 2; ++i) tc_mbar_init(bars + 2 * P::kStages + 2 + i, 2 * kPWarps);
    tc_mbar_init(bars + 2 * P::kStages + 4, 1);
    s_err = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (w == 1) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(kTmem) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();   // both CTAs' barriers exist
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();   // after the allocation: a successor's CTA on this SM cannot take the columns first
  pdl_wait();
  volatile int* err = &s_err;

  if (w == 0) {
    // ---------------- copies of this CTA
    const uint32_t full0 = tc_leader_addr(full);
    int s = 0;
    unsigned phase = 1;   // parity of the ring's previous round
    bool ok = true;
    for (int t = pair; t < n_total && ok; t += n_pairs) {
      const TcTile tl = tc_tile_of(t, m_tiles, n_tiles, 8);
      // B: half of the tile's 64-column boxes of a packed tile: [32 k][128 B] each
      const int kb0 = (BN == 256 ? tl.n_tile : tl.n_tile >> 1) * a.KB;
      const int box_row = (BN == 256 ? rank * 2 : (tl.n_tile & 1) * 2 + rank) * 32, row = (tl.m_tile * 2 + rank) * kBM;
      for (int it = 0; it < k_total; ++it) {
        if (asked >= P::kStages && !(ok = tc_wait_or(empty + s * 8, phase, err, a.wait_limit))) break;
        if (rank == 0) tc_mbar_expect_el(full + s * 8, 2 * P::kStage);
        tc_pair_load_2d(sA + s * kABytes, &mapA, it * kBK, row, full0 + s * 8);
        tc_pair_load_3d(sB + s * P::kB, &mapB, 0, box_row, kb0 + it * 2, full0 + s * 8);   // the second k tile of an odd count is not multiplied
        ++asked;
        if (++s == P::kStages) s = 0, phase ^= 1;
      }
    }
  } else if (w == 1 && rank == 0) {
    // ---------------- products.  Instruction descriptor: fp32 accumulator, A K-major, B MN-major, N = BN, M = 256
    const uint32_t idesc = (1u << 4) | (Pair16<H>::kUmmaFormat << 7) | (Pair16<H>::kUmmaFormat << 10) | (1u << 16) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(2 * kBM >> 4) << 24);
    // A: K-major, 8-row atoms 1024 B apart; 16 k = 32 B along the row.  B stage and CTA = [k tile 2][64-n box BN / 128][32 k][128 B]: boxes
    // 4096 B apart (LBO), 8-k groups 1024 B apart (SBO)
    const uint32_t hi = desc_hi(1024), a0 = desc_lo(sA, 16), b0 = desc_lo(sB, 4096);
    int s = 0, n_done = 0;
    unsigned phase = 0;
    bool ok = true;
    for (int t = pair; t < n_total && ok; t += n_pairs, ++n_done) {
      const int buf = n_done & 1;
      if (n_done >= 2 && !(ok = tc_wait_or(acc_empty + buf * 8, (unsigned)(((n_done >> 1) - 1) & 1), err, a.wait_limit))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem_base + buf * BN;
      for (int it = 0; it < k_total; ++it) {
        if (!(ok = tc_wait_or(full + s * 8, phase, err, a.wait_limit))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t ad = a0 + s * (kABytes >> 4), bd = b0 + s * (P::kB >> 4);
        umma_pair_el(acc, ad, hi, bd, hi, idesc, it > 0);
        umma_pair_el(acc, ad + 2, hi, bd + 128, hi, idesc, 1);
        if (it * 2 + 1 < a.KB) {
          umma_pair_el(acc, ad + 4, hi, bd + (P::kB >> 5), hi, idesc, 1);
          umma_pair_el(acc, ad + 6, hi, bd + (P::kB >> 5) + 128, hi, idesc, 1);
        }
        umma_commit_pair_el(empty + s * 8);
        if (++s == P::kStages) s = 0, phase ^= 1;
      }
      if (ok) umma_commit_pair_el(acc_full + buf * 8);
    }
    umma_commit_pair_el(drain);
    tc_wait_short(drain, 0);
  } else if (w >= 2) {
    // ---------------- epilogue: TMEM lanes 32 (w % 4) .. = rows of this CTA's half, columns kCols ((w - 2) / 4) ..
    const int q = w & 3, half = (w - 2) >> 2;
    float* stage = stages + (w - 2) * kStageFloats;
    TcAhead ahead;
    int n_done = 0;
    for (int t = pair; t < n_total; t += n_pairs, ++n_done) {
      const TcTile tl = tc_tile_of(t, m_tiles, n_tiles, 8);
      const int buf = n_done & 1;
      const int row0 = (tl.m_tile * 2 + rank) * kBM + q * 32, n0 = tl.n_tile * BN + half * P::kCols;
      const int n_live = min(32, a.M - row0);
      const TcLane at = tc_lane(a, row0, n0);
      tc_ahead<H>(a, at, n_live, n0, ahead);
      if (!tc_wait_or(acc_full + buf * 8, (unsigned)((n_done >> 1) & 1), err, a.wait_limit)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      tc_drain<H, P::kCols>(a, at, tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN + half * P::kCols), row0, n_live, n0, stage, ahead, [](int, float*) {});
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(tc_leader_addr(acc_empty + buf * 8)) : "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0) {
    uint32_t to;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(s_u32(&s_peer)), "r"(rank ^ 1));
    asm volatile("st.shared::cluster.v2.s32 [%0], {%1, %2};" ::"r"(to), "r"(s_err), "r"(asked) : "memory");
  }
  cluster_sync();   // nobody reports to a CTA that has left
  if (s_err | s_peer.x) {
    // Copies in flight land in both CTAs.  One CTA may have asked for up to kStages stages more than the other, whose part the leader's barrier
    // then waits for in vain, or does not know of: the difference is put right, in the phases that are open, before they are waited for.
    if (w == 0 && rank == 0) {
      for (int j = min(asked, s_peer.y); j < max(asked, s_peer.y); ++j) {
        const uint32_t bar = full + (j % P::kStages) * 8;
        if (asked > s_peer.y) tc_mbar_complete_el(bar, P::kStage);
        else tc_mbar_expect_el(bar, P::kStage);
      }
      tc_land(full, P::kStages, max(asked, s_peer.y));
    }
    cluster_sync();
  }
  if (w == 1) {
    if (rank == 1) tc_wait_short(drain, 0);   // the leader has seen its own arrive
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmem) : "memory");
  }
  if (tid == 0 && s_err) {
    g_tc_error = 1;
    if (a.error_flag) *a.error_flag = 1;
  }
}

// ---- host side ---------------------------------------------------------------------------------------------------------
EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
    else
      cudaGetLastError();
  }
  return fn;
}

int init_tc_attrs(int device) {
  static bool done[kMaxDevices] = {};
  if (done[device]) return 1;
  const auto dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
  TSB_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<__half, kTcStages>, dyn, tc_smem(kTcStages)));
  TSB_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<__nv_bfloat16, kTcStages>, dyn, tc_smem(kTcStages)));
  TSB_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<__half, kTcDeepStages>, dyn, tc_smem(kTcDeepStages)));
  TSB_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<__nv_bfloat16, kTcDeepStages>, dyn, tc_smem(kTcDeepStages)));
  TSB_CUDA(cudaFuncSetAttribute(gemm_tc_grouped_kernel<__nv_bfloat16>, dyn, kGSmem));
  TSB_CUDA(cudaFuncSetAttribute(gemm_tc_pair_kernel<__half, 256>, dyn, PairTile<256>::kSmem));
  TSB_CUDA(cudaFuncSetAttribute(gemm_tc_pair_kernel<__nv_bfloat16, 256>, dyn, PairTile<256>::kSmem));
  TSB_CUDA(cudaFuncSetAttribute(gemm_tc_pair_kernel<__half, 128>, dyn, PairTile<128>::kSmem));
  TSB_CUDA(cudaFuncSetAttribute(gemm_tc_pair_kernel<__nv_bfloat16, 128>, dyn, PairTile<128>::kSmem));
  done[device] = true;
  return 1;
}

// 1 when a tensor-core GEMM on the current device gave up waiting since the last call (and clears the mark).
int tc_take_error() {
  int e = 0;
  if (cudaMemcpyFromSymbol(&e, g_tc_error, sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (e) {
    const int z = 0;
    cudaMemcpyToSymbol(g_tc_error, &z, sizeof(int));
  }
  return e;
}

unsigned tc_wait_limit() {
  static unsigned limit = 0;
  if (!limit) {
    const char* e = getenv("TSB200_WAIT_LIMIT");
    const int n = e ? atoi(e) : 0;
    limit = n > 0 ? (unsigned)n : kTcSpin;
  }
  return limit;
}

int* tc_error_word(int device) {
  static int* word[kMaxDevices] = {};
  if (!word[device]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_tc_error) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    word[device] = reinterpret_cast<int*>(p);
  }
  return word[device];
}

int64_t gemm_tc_workspace_bytes(int M, int N, int sm_count) {
  if (M > kBM) return 0;
  // K slices of the 128 x 128 kernel
  const int64_t tiles = (N + kBN - 1) / kBN;
  if (tiles >= 2 * sm_count) return 0;
  const int64_t ks = (2 * sm_count + tiles - 1) / tiles;
  return 4096 + kWsCounterBytes + ks * M * (int64_t)((N + kBN - 1) / kBN) * kBN * 4;
}

static int tc_map_rows(CUtensorMap* map, int dtype, const void* x, int M, int K) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return 2;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)kBM};
  const cuuint32_t el[2] = {1, 1};
  const CUresult r = enc(map, dtype == TSB200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(x),
                         dims, strides, box, el, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TSB_CHECK(r == CUDA_SUCCESS, "gemm_tc: cuTensorMapEncodeTiled(A) failed with %d", (int)r);
  return 1;
}
// packed weights as [tiles][128 rows of 64 columns]: a box is `rows` rows of two k tiles in a row, laid down as stored
static int tc_map_packed(CUtensorMap* map, int dtype, const void* Wp, int64_t tiles, int rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return 2;
  const cuuint64_t dims[3] = {64, 128, (cuuint64_t)tiles};
  const cuuint64_t strides[2] = {128, 16384};
  const cuuint32_t box[3] = {64, (cuuint32_t)rows, 2};
  const cuuint32_t el[3] = {1, 1, 1};
  const CUresult r = enc(map, dtype == TSB200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(Wp),
                         dims, strides, box, el, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TSB_CHECK(r == CUDA_SUCCESS, "gemm_tc: cuTensorMapEncodeTiled(B) failed with %d", (int)r);
  return 1;
}
static int tc_kind(int N, const Epilogue& ep) {
  const uintptr_t al = (uintptr_t)ep.bias | (uintptr_t)ep.residual | (uintptr_t)ep.y | (uintptr_t)ep.y32 | (uintptr_t)ep.gate;
  if (N % 32 != 0 || al % 16 != 0) return kTcAny;
  if (!ep.residual && !ep.gate && !ep.y32) return kTcRows16;
  if (ep.glu || !ep.residual || !ep.y32 || ep.act != TSB200_ACT_NONE) return kTcMixed;
  return ep.gate ? kTcGateResidual : kTcResidual;
}

int launch_gemm_tc_grouped(int device, DeviceState* st, int dtype, const void* x, const void* Wp, int rows, int K, int N, const Epilogue& ep,
                           const RowGroups& groups, cudaStream_t s) {
  if (dtype != TSB200_BF16 || K % 8 != 0 || ((uintptr_t)x % 16) != 0 || ((uintptr_t)Wp % 16) != 0) return 2;
  TSB_TRY(init_tc_attrs(device));
  CUtensorMap mapA;
  const int r = tc_map_rows(&mapA, dtype, x, rows, K);
  if (r != 1) return r;
  TcArgs a{};
  a.M = rows; a.N = N; a.K = K; a.KB = (K + 31) / 32; a.ep = ep; a.ksplit = 1;
  a.Wp = reinterpret_cast<const unsigned char*>(Wp);
  a.wait_limit = tc_wait_limit();
  a.kind = tc_kind(N, ep);
  TSB_CUDA(launch_k(gemm_tc_grouped_kernel<__nv_bfloat16>, dim3(st->sm_count), dim3(kPThreads), kGSmem, s, mapA, a, (N + kP_BN - 1) / kP_BN, groups));
  count_launch(device);
  return check_launch("gemm_tc_grouped");
}

// Pairs of CTAs.  Tiles of 256 columns or of 128, whichever is done first: whole waves of pairs times 64-k steps (0.33 and 0.19 us; four waves of
// 1024 x 1024 .. 4096 x 18944 0.34, of x 9472 0.19) and the last tile's epilogue (3.3 and 1.6 us).  The estimate names the faster one at 31 of 36 sizes of 160 to
// 16384 rows and costs 3 % at most at the others.
static int launch_pair(int device, DeviceState* st, int dtype, const CUtensorMap& mapA, const TcArgs& a, cudaStream_t s) {
  const int pairs = st->sm_count / 2, m_tiles = (a.M + 2 * kBM - 1) / (2 * kBM), k_total = (a.K + kBK - 1) / kBK;
  const int n256 = (a.N + 255) / 256, n128 = (a.N + 127) / 128;
  const int64_t t256 = (int64_t)m_tiles * n256, t128 = (int64_t)m_tiles * n128;
  TSB_CHECK(t128 < (1 << 30), "gemm_tc: too many tiles");
  const double c256 = (double)((t256 + pairs - 1) / pairs) * k_total * 0.33 + 3.3, c128 = (double)((t128 + pairs - 1) / pairs) * k_total * 0.19 + 1.6;
  const bool wide = c256 <= c128;
  const int64_t t = wide ? t256 : t128;
  CUtensorMap mapB;
  const int r = tc_map_packed(&mapB, dtype, a.Wp, (int64_t)n256 * a.KB, wide ? 64 : 32);
  if (r != 1) return r;
  auto k = dtype == TSB200_BF16 ? (wide ? gemm_tc_pair_kernel<__nv_bfloat16, 256> : gemm_tc_pair_kernel<__nv_bfloat16, 128>)
                                : (wide ? gemm_tc_pair_kernel<__half, 256> : gemm_tc_pair_kernel<__half, 128>);
  TSB_CUDA(launch_k(k, dim3(2 * (int)(t < pairs ? t : pairs)), dim3(kPThreads), wide ? PairTile<256>::kSmem : PairTile<128>::kSmem, s, mapA, mapB, a, m_tiles,
                    wide ? n256 : n128));
  count_launch(device);
  return check_launch("gemm_tc_pair");
}

int launch_gemm_tc(int device, DeviceState* st, int dtype, const void* x, const void* Wp, int M, int K, int N, const Epilogue& ep,
                   int* error_flag, void* ws, int64_t ws_bytes, cudaStream_t s) {
  {
    static int enabled = -1;
    if (enabled < 0) {
      const char* e = getenv("TSB200_TC");  // "0" routes large-M linears to the CUDA-core fallback (A/B measurements)
      enabled = (e && e[0] == '0') ? 0 : 1;
    }
    if (!enabled) return 2;
  }
  if (K % 8 != 0 || ((uintptr_t)x % 16) != 0 || ((uintptr_t)Wp % 16) != 0) return 2;
  TSB_TRY(init_tc_attrs(device));
  const int KB = (K + 31) / 32;
  CUtensorMap mapA;
  {
    const int r = tc_map_rows(&mapA, dtype, x, M, K);
    if (r != 1) return r;
  }
  TcArgs a{};
  a.M = M; a.N = N; a.K = K; a.KB = KB; a.error_flag = error_flag; a.ep = ep;
  a.Wp = reinterpret_cast<const unsigned char*>(Wp);
  a.wait_limit = tc_wait_limit();
  a.kind = tc_kind(N, ep);
  if (M > kBM) return launch_pair(device, st, dtype, mapA, a, s);
  dim3 grid((N + kBN - 1) / kBN, 1, 1);
  // few output tiles (decode-sized M): share each tile's K range among several CTAs so that all SMs stream weights
  a.ksplit = 1;
  {
    const int64_t tiles = grid.x;
    const int k_total = (K + kBK - 1) / kBK;
    // Only for long K: a slice saves its part of 0.37 us per 64 k of a tile alone, and costs the last arriver 2 to 4 us to add.  100 rows
    // with slices / without: 4096 x 4096 67.0 / 27.1 us, 2048 x 3072 32.1 / 17.4, 8192 x 2048 33.4 / 47.  No more slices than SMs, which
    // keeps the deep rings (100 x 11008 x 4096: six slices of three stages 76.9, four of six stages 36.6).
    if (k_total >= 96 && ws) {
      int ks = (int)(st->sm_count / tiles);
      if (ks > 6) ks = 6;
      if (ks > 1) {
        const int k_per = (k_total + ks - 1) / ks;
        ks = (k_total + k_per - 1) / k_per;  // no empty slice
        const int64_t cnt = kWsCounterBytes;
        const int64_t need = cnt + (int64_t)ks * M * grid.x * kBN * 4;
        if (ks > 1 && ws_bytes >= need) {
          a.ksplit = ks;
          a.counters = reinterpret_cast<unsigned int*>(ws);
          a.partials = reinterpret_cast<float*>(reinterpret_cast<char*>(ws) + cnt);
          grid.z = ks;
        }
      }
    }
  }
  const bool deep = (int64_t)grid.x * grid.z <= st->sm_count;
  auto k = dtype == TSB200_BF16 ? (deep ? gemm_tc_kernel<__nv_bfloat16, kTcDeepStages> : gemm_tc_kernel<__nv_bfloat16, kTcStages>)
                                : (deep ? gemm_tc_kernel<__half, kTcDeepStages> : gemm_tc_kernel<__half, kTcStages>);
  TSB_CUDA(launch_k(k, grid, dim3(kTcThreads), tc_smem(deep ? kTcDeepStages : kTcStages), s, mapA, a));
  count_launch(device);
  return check_launch("gemm_tc");
}

}  // namespace tsb
