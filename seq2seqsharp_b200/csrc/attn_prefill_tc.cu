// Causal prompt attention on the 5th-generation tensor cores (tcgen05), for the cached keys / values of the GPT engine (fp16, head
// size 64 or 128) and for the expanded keys / values of the latent layers (bf16, 128 + 64 | 128).
//
// One CTA = (sequence, KV head, 256 rows): two tiles of 128 rows, a row being one (query, head) pair of the KV head's group, so that
// the G heads of a group share every key / value tile.  Roles: warps 0-3 and 4-7 do the softmax of one tile each (a thread owns
// a row: no shuffles), warp 8 brings the tiles in with TMA tensor copies (128-byte swizzle; keys beyond the cached ones are filled
// with zeros, whatever the cache holds there), warp 9 issues the MMAs.  TMEM: S0 | S1 (128 fp32 columns each) | O0 | O1.  Per tile of
// 128 keys: S = Q K^T (operands in shared memory), softmax in registers, P back over S as 16-bit A operand, O += P V (A in TMEM,
// V as the MN-major operand where it was laid down).  The MMAs of one tile run while the other is in its softmax: the order
// PV0(j) QK0(j+1) PV1(j) QK1(j+1) keeps one tile's products behind the other's exponentials.
//
// O lives in TMEM and is rescaled there by its softmax warps, when one of a warp's rows has a new maximum.  That needs no barrier of
// its own: a tile's S arrives after its PV of the step before, because both are issued in that order by one thread.  (Raising the
// maximum in use only once it is 2^8 too small saves 8 % at 16384 tokens, but the largest weight of a row is then no longer exactly 1, and
// the error against 64 bits grows from 2.38e-4 to 2.42e-4 on average, by a tenth for sharp scores.)  The row sum adds the weights as they
// are rounded for the product (add.f32.f16): what rounding a weight does to the numerator it does to the denominator.
//
// What bounds it: the exponentials (16 per clock and SM: at head size 64 a tile's 16384 take twice as long as its products).  Measured, one
// sequence of 16384 tokens, 32 heads, 8 KV heads: head size 64 6.55 ms -> 1.70 ms (645 TFLOP/s), 128 11.6 -> 1.97 ms (1117 TFLOP/s) against the
// kernel on mma.sync with 64 rows per CTA, which short prompts still take (ops_attention.cu); 1024 tokens of head size 64: 48 -> 23 us; 4 x 509 of 128: 71 -> 25 us.
// Three sequences of 1537 tokens, 12 layers of 16 latent heads of 192 | 128: the whole prompt pass 18.9 -> 15.6 ms.
#include "tc_common.cuh"

namespace tsb {

constexpr int kPaThreads = 384, kPaRows = 128, kPaKeys = 128;
constexpr int kPaBox = kPaKeys * 128;        // one 64-column box of 128 rows: 16 KB
// registers per thread: 384 x 168 at launch; two warpgroups hold a row of scores per thread, the third issues copies and products
constexpr int kPaSoftmaxRegs = 224, kPaIssueRegs = 48;
static_assert(256 * kPaSoftmaxRegs + 128 * kPaIssueRegs <= kPaThreads * 168, "the warpgroups' registers come out of the launch's");

struct PaArgs {
  void* out;
  int B, S, T0, H, heads, G, QT;             // heads: KV heads; G query heads each; QT = 128 / G query positions per tile
  int tiles;                                 // CTAs per (sequence, KV head)
  float c;                                   // scale * log2(e)
  int k_boxes;                               // 64-column boxes of a key that mapK holds; the others come from mapR
  int kx, vx, vx0, rx;                       // column of a head's keys / values: head * kx, vx0 + head * vx; of the shared key part: rx
  int z_seq, z_head;                         // outermost coordinate of mapK / mapV: b * z_seq + head * z_head
  const int* starts;                         // packed rows: first row of every sequence (B + 1), or NULL: S rows each
  int vec_out;                               // out is 16-byte aligned
  unsigned wait_limit;                       // polls of a wait before the CTA gives up
  int* error;
};

__device__ __forceinline__ bool pa_wait(uint64_t* bar, unsigned parity, volatile int* err, unsigned limit) {
  const uint32_t a = s_u32(bar);
#pragma unroll 1
  for (unsigned i = 0; i < limit; ++i) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((i & 63) == 63 && *err) return false;
  }
  *err = 1;
  return false;
}
__device__ __forceinline__ void pa_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s_u32(bar)) : "memory");
}
__device__ __forceinline__ void pa_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst), "l"(map),
      "r"(s_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void pa_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst), "l"(map),
      "r"(s_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// D[tmem] += A[tmem] * B[smem]
__device__ __forceinline__ void pa_umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
#define PA_R32(r)                                                                                                                       \
  "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), \
      "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), \
      "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), \
      "+r"(r[31])
// 32 lanes x 32 columns; the registers are valid after pa_ld_wait on them
__device__ __forceinline__ void pa_ld32(uint32_t taddr, uint32_t* r) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void pa_ld_wait(uint32_t* r) {
  __syncwarp();
  asm volatile("tcgen05.wait::ld.sync.aligned;" : PA_R32(r)::"memory");
}
__device__ __forceinline__ void pa_st32(uint32_t taddr, const uint32_t* r) {
  __syncwarp();
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
      "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
      "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void pa_st_wait() {
  __syncwarp();
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ float pa_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// (a0, a1) * (b, b) + (c, c): one instruction for the pair
__device__ __forceinline__ float2 pa_fma2(float a0, float a1, float b, float c) {
  uint64_t a, bb, cc, d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(a0), "f"(a1));
  asm("mov.b64 %0, {%1, %1};" : "=l"(bb) : "f"(b));
  asm("mov.b64 %0, {%1, %1};" : "=l"(cc) : "f"(c));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(bb), "l"(cc));
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
  return r;
}
// sum += the two 16-bit values of a register, in fp32
template <typename H>
__device__ __forceinline__ void pa_add_pair(float& s, uint32_t v) {
  if constexpr (Pair16<H>::kBf16)
    asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %1;\n\tadd.rn.f32.bf16 %0, lo, %0;\n\tadd.rn.f32.bf16 %0, hi, %0;\n\t}" : "+f"(s) : "r"(v));
  else
    asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %1;\n\tadd.rn.f32.f16 %0, lo, %0;\n\tadd.rn.f32.f16 %0, hi, %0;\n\t}" : "+f"(s) : "r"(v));
}
template <int N>
__device__ __forceinline__ void pa_more_registers() {
  __syncwarp();
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void pa_fewer_registers() {
  __syncwarp();
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

template <int QB, int VB>
constexpr int pa_smem(int nks, int nvs) { return (2 * QB + nks * QB + nvs * VB) * kPaBox + 1024 + 256; }

// QB / VB: 64-column boxes of a query-key row / of a value row; NKS / NVS: key / value tiles in flight
template <typename H, int QB, int VB, int NKS, int NVS>
__global__ void __launch_bounds__(kPaThreads, 1) attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                                                                        const __grid_constant__ CUtensorMap mapR, const __grid_constant__ CUtensorMap mapV,
                                                                        PaArgs a) {
  extern __shared__ __align__(1024) unsigned char pa_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)pa_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sQ = s_u32(smem), sK = sQ + 2 * QB * kPaBox, sV = sK + NKS * QB * kPaBox;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (2 * QB + NKS * QB + NVS * VB) * kPaBox);
  uint64_t *q_full = bars, *k_full = q_full + 2, *k_empty = k_full + NKS, *v_full = k_empty + NKS, *v_empty = v_full + NVS;
  uint64_t *s_full = v_empty + NVS, *p_full = s_full + 2, *o_full = p_full + 2, *drain = o_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  __shared__ int s_err;

  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  // the longest key ranges start first, over all sequences and heads
  const int kvh = (int)(blockIdx.x % a.heads), b = (int)((blockIdx.x / a.heads) % a.B);
  const int q0 = (a.tiles - 1 - (int)(blockIdx.x / a.heads / a.B)) * 2 * a.QT;
  const int row0 = a.starts ? a.starts[b] : b * a.S, S = a.starts ? a.starts[b + 1] - row0 : a.S;
  if (q0 >= S) return;   // a shorter sequence
  // key tiles of the two row tiles: up to the last query that exists; the second may have no query at all
  int n_of[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int first = q0 + t * a.QT, last = min(S, first + a.QT) - 1;
    n_of[t] = first < S ? (a.T0 + last + kPaKeys) / kPaKeys : 0;
  }
  const int n_tiles = max(n_of[0], n_of[1]);

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      tc_mbar_init(&q_full[i], 1);
      tc_mbar_init(&s_full[i], 1);
      tc_mbar_init(&p_full[i], kPaRows);
      tc_mbar_init(&o_full[i], 1);
    }
    for (int i = 0; i < NKS; ++i) {
      tc_mbar_init(&k_full[i], 1);
      tc_mbar_init(&k_empty[i], 1);
    }
    for (int i = 0; i < NVS; ++i) {
      tc_mbar_init(&v_full[i], 1);
      tc_mbar_init(&v_empty[i], 1);
    }
    tc_mbar_init(drain, 1);
    s_err = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (w == 9) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();   // after the allocation: a successor's CTA on this SM cannot take the columns first
  pdl_wait();      // (a.starts was there before the pass began)
  volatile int* err = &s_err;

  if (w >= 8) {
    pa_fewer_registers<kPaIssueRegs>();
    if (w == 8 && lane == 0) {
      // ---------------- TMA producer
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (n_of[t] == 0) continue;
        tc_mbar_expect_tx(&q_full[t], QB * kPaBox);
        for (int i = 0; i < QB; ++i) pa_load_4d(sQ + (t * QB + i) * kPaBox, &mapQ, 64 * i, kvh * a.G, (a.starts ? row0 : 0) + q0 + t * a.QT, a.starts ? 0 : b, &q_full[t]);
      }
      const int z = b * a.z_seq + kvh * a.z_head;
      int ks = 0, vs = 0;   // tiles asked for so far
      auto load_k = [&](int j) {
        const int st = j % NKS;
        if (j >= NKS && !pa_wait(&k_empty[st], (unsigned)((j / NKS - 1) & 1), err, a.wait_limit)) return false;
        tc_mbar_expect_tx(&k_full[st], QB * kPaBox);
#pragma unroll
        for (int i = 0; i < QB; ++i) {
          if (i < a.k_boxes) pa_load_3d(sK + (st * QB + i) * kPaBox, &mapK, kvh * a.kx + 64 * i, j * kPaKeys, z, &k_full[st]);
          else pa_load_3d(sK + (st * QB + i) * kPaBox, &mapR, a.rx + 64 * (i - a.k_boxes), j * kPaKeys, b, &k_full[st]);
        }
        ks = j + 1;
        return true;
      };
      bool ok = load_k(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles && !load_k(j + 1)) break;
        const int st = j % NVS;
        if (j >= NVS && !pa_wait(&v_empty[st], (unsigned)((j / NVS - 1) & 1), err, a.wait_limit)) break;
        tc_mbar_expect_tx(&v_full[st], VB * kPaBox);
#pragma unroll
        for (int i = 0; i < VB; ++i) pa_load_3d(sV + (st * VB + i) * kPaBox, &mapV, a.vx0 + kvh * a.vx + 64 * i, j * kPaKeys, z, &v_full[st]);
        vs = j + 1;
      }
      // copies in flight land before the CTA ends (tc_land): they need nobody's help, and a wait may run out after this thread has asked for its last
      for (int t = 0; t < 2; ++t)
        if (n_of[t]) tc_mbar_wait(&q_full[t], 0);
      tc_land(s_u32(k_full), NKS, ks);
      tc_land(s_u32(v_full), NVS, vs);
    } else if (w == 9 && lane == 0) {
      // ---------------- MMA issuer.  Instruction descriptors: fp32 accumulator, A K-major, 128 rows; K: N = 128 K-major; V: N = 64 VB MN-major
      const uint32_t fmt = (1u << 4) | (Pair16<H>::kUmmaFormat << 7) | (Pair16<H>::kUmmaFormat << 10) | ((uint32_t)(kPaRows >> 4) << 24);
      const uint32_t id_qk = fmt | ((uint32_t)(kPaKeys >> 3) << 17), id_pv = fmt | (1u << 16) | ((uint32_t)(VB * 64 >> 3) << 17);
      auto qk = [&](int t, int j) {
        const uint32_t q = sQ + t * QB * kPaBox, k = sK + (j % NKS) * QB * kPaBox;
#pragma unroll
        for (int i = 0; i < QB * 4; ++i) {
          const uint32_t off = (i >> 2) * kPaBox + (i & 3) * 32;
          umma_f16(tmem + t * kPaKeys, make_desc(q + off, 16, 1024), make_desc(k + off, 16, 1024), id_qk, i > 0 ? 1u : 0u);
        }
        umma_commit(&s_full[t]);
      };
      bool ok = pa_wait(&k_full[0], 0, err, a.wait_limit);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (!ok || n_of[t] == 0) continue;
        ok = pa_wait(&q_full[t], 0, err, a.wait_limit);
        if (ok) qk(t, 0);
      }
      umma_commit(&k_empty[0]);
      for (int j = 0; j < n_tiles && ok; ++j) {
        const bool more = j + 1 < n_tiles;
        ok = pa_wait(&v_full[j % NVS], (unsigned)((j / NVS) & 1), err, a.wait_limit);
        if (ok && more) ok = pa_wait(&k_full[(j + 1) % NKS], (unsigned)(((j + 1) / NKS) & 1), err, a.wait_limit);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (!ok || j >= n_of[t]) continue;
          if (!(ok = pa_wait(&p_full[t], (unsigned)(j & 1), err, a.wait_limit))) continue;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // V stage = [box][128 keys][128 B]: 8-key groups 1024 B apart (SBO), boxes kPaBox apart (LBO); 16 keys = 2048 B
          const uint32_t v = sV + (j % NVS) * VB * kPaBox;
#pragma unroll
          for (int i = 0; i < kPaKeys / 16; ++i)
            pa_umma_ts(tmem + 2 * kPaKeys + t * VB * 64, tmem + t * kPaKeys + i * 8, make_desc(v + i * 2048, kPaBox, 1024), id_pv, (j > 0 || i > 0) ? 1u : 0u);
          if (j + 1 < n_of[t]) qk(t, j + 1);
          else umma_commit(&o_full[t]);
        }
        umma_commit(&v_empty[j % NVS]);
        if (more) umma_commit(&k_empty[(j + 1) % NKS]);
      }
    }
  } else {
    // ---------------- softmax: thread = row of tile t
    pa_more_registers<kPaSoftmaxRegs>();
    const int t = w >> 2, row = tid & 127, n = t ? n_of[1] : n_of[0];
    const int pos = q0 + t * a.QT + row / a.G, head = kvh * a.G + row % a.G;
    const bool live = pos < S;
    const int lim = live ? a.T0 + pos + 1 : 0x7fffffff;                            // keys [0, lim) are visible (a row without a query: zeros, never stored)
    const int warp_lim = a.T0 + q0 + t * a.QT + (row & ~31) / a.G + 1;             // the smallest of the warp
    const uint32_t lanes = (uint32_t)((w & 3) * 32) << 16;
    const uint32_t tS = tmem + lanes + t * kPaKeys, tO = tmem + lanes + 2 * kPaKeys + t * VB * 64;
    const float c = a.c;
    float m = -INFINITY, l = 0.0f;
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      ok = __all_sync(0xffffffffu, pa_wait(&s_full[t], (unsigned)(j & 1), err, a.wait_limit));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t s[4][32];
#pragma unroll
      for (int q = 0; q < 4; ++q) pa_ld32(tS + q * 32, s[q]);
#pragma unroll
      for (int q = 0; q < 4; ++q) pa_ld_wait(s[q]);
      if ((j + 1) * kPaKeys > warp_lim) {
        const int left = lim - j * kPaKeys;
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (q * 32 + i >= left) s[q][i] = 0xff800000u;
      }
      float mx[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) mx[q] = __uint_as_float(s[q][0]);
#pragma unroll
      for (int i = 1; i < 32; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) mx[q] = fmaxf(mx[q], __uint_as_float(s[q][i]));
      const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      if (j == 0) {
        m = top;
      } else if (__any_sync(0xffffffffu, top > m)) {
        const float up = fmaxf(m, top);
        const float f = up == -INFINITY ? 1.0f : pa_ex2((m - up) * c);
        m = up;
        l *= f;
#pragma unroll 1
        for (int q = 0; q < VB * 2; ++q) {
          uint32_t o[32];
          pa_ld32(tO + q * 32, o);
          pa_ld_wait(o);
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
          pa_st32(tO + q * 32, o);
        }
      }
      const float mc = m == -INFINITY ? 0.0f : -m * c;   // no key seen yet: every weight is exp2(-inf)
      float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t p[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const uint32_t* e = &s[2 * h + (i >> 4)][2 * (i & 15)];
          float2 x = pa_fma2(__uint_as_float(e[0]), __uint_as_float(e[1]), c, mc);
          x.x = pa_ex2(x.x);
          x.y = pa_ex2(x.y);
          p[i] = Pair16<H>::put(x.x, x.y);
          pa_add_pair<H>(sum[i & 3], p[i]);
        }
        pa_st32(tS + h * 32, p);
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      pa_st_wait();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      pa_arrive(&p_full[t]);
    }
    if (n > 0 && ok && __all_sync(0xffffffffu, pa_wait(&o_full[t], 0, err, a.wait_limit))) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float inv = l > 0.0f ? 1.0f / l : 0.0f;
      H* out = reinterpret_cast<H*>(a.out) + (((int64_t)row0 + pos) * a.H + head) * (VB * 64);
#pragma unroll 1
      for (int q = 0; q < VB * 2; ++q) {
        uint32_t o[32];
        pa_ld32(tO + q * 32, o);
        pa_ld_wait(o);
        if (!live) continue;
        uint32_t y[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = Pair16<H>::put(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv);
        if (a.vec_out) {
#pragma unroll
          for (int i = 0; i < 4; ++i) reinterpret_cast<uint4*>(out + q * 32)[i] = make_uint4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) reinterpret_cast<uint32_t*>(out + q * 32)[i] = y[i];
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (w == 9) {
    if (lane == 0 && s_err) {   // some warp gave up: products in flight end before TMEM is given back
      umma_commit(drain);
      tc_mbar_wait(drain, 0);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
  if (tid == 0 && s_err && a.error) *a.error = 1;
}

// ---- host side ---------------------------------------------------------------------------------------------------------
static int pa_map(CUtensorMap* map, int dtype, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
  EncodeTiledFn enc = get_encode();
  TSB_CHECK(enc, "prompt attention: the driver has no cuTensorMapEncodeTiled");
  const cuuint32_t el[4] = {1, 1, 1, 1};
  const CUresult r = enc(map, dtype == TSB200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, rank, const_cast<void*>(base), dims,
                         strides, box, el, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TSB_CHECK(r == CUDA_SUCCESS, "prompt attention: cuTensorMapEncodeTiled failed with %d", (int)r);
  return 1;
}
// queries [B][S][heads][width], rows of q_rs elements: a box is 64 columns of the G heads of QT positions
static int pa_map_q(CUtensorMap* map, int dtype, const void* q, int width, int H, int S, int B, int64_t q_rs, int G) {
  const cuuint64_t dims[4] = {(cuuint64_t)width, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  const cuuint64_t strides[3] = {(cuuint64_t)width * 2, (cuuint64_t)q_rs * 2, (cuuint64_t)q_rs * 2 * S};
  const cuuint32_t box[4] = {64, (cuuint32_t)G, (cuuint32_t)(kPaRows / G), 1};
  return pa_map(map, dtype, q, 4, dims, strides, box);
}
// rows [n][T][width]: T of every `pitch` elements are used
static int pa_map_rows(CUtensorMap* map, int dtype, const void* x, int width, int T, int n, int64_t row, int64_t pitch) {
  const cuuint64_t dims[3] = {(cuuint64_t)width, (cuuint64_t)T, (cuuint64_t)n};
  const cuuint64_t strides[2] = {(cuuint64_t)row * 2, (cuuint64_t)pitch * 2};
  const cuuint32_t box[3] = {64, kPaKeys, 1};
  return pa_map(map, dtype, x, 3, dims, strides, box);
}

template <typename H, int QB, int VB, int NKS, int NVS>
static int pa_launch(int device, const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& r, const CUtensorMap& v, PaArgs a, cudaStream_t s) {
  constexpr int smem = pa_smem<QB, VB>(NKS, NVS);
  static_assert(smem <= 227 * 1024, "shared memory of a CTA");
  static bool done[kMaxDevices] = {};
  if (!done[device]) {
    TSB_CUDA(cudaFuncSetAttribute(attn_prefill_tc_kernel<H, QB, VB, NKS, NVS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    done[device] = true;
  }
  a.tiles = (a.S + 2 * a.QT - 1) / (2 * a.QT);
  a.vec_out = ((uintptr_t)a.out % 16) == 0 ? 1 : 0;
  a.error = tc_error_word(device);
  a.wait_limit = tc_wait_limit();
  const int64_t grid = (int64_t)a.tiles * a.heads * a.B;
  TSB_CHECK(grid <= 0x7fffffff, "prompt attention: %lld blocks", (long long)grid);
  TSB_CUDA(launch_k(attn_prefill_tc_kernel<H, QB, VB, NKS, NVS>, dim3((unsigned)grid), dim3(kPaThreads), smem, s, q, k, r, v, a));
  count_launch(device);
  return check_launch("attn_prefill_tc");
}

int launch_attn_prefill_tc(int device, void* out, const void* q, int64_t q_rs, const void* cK, const void* cV, int B, int S, int H, int Hkv, int hd, int T0,
                           int Tmax, float scale, const PackedRows* pack, cudaStream_t s) {
  PaArgs a{};
  a.starts = pack ? pack->starts : nullptr;
  a.out = out; a.B = B; a.S = S; a.T0 = T0; a.H = H; a.heads = Hkv; a.G = H / Hkv; a.QT = kPaRows / a.G;
  a.c = scale * 1.44269504088896340736f;
  a.k_boxes = hd / 64; a.z_seq = Hkv; a.z_head = 1;
  CUtensorMap mq, mk, mv;
  TSB_TRY(pa_map_q(&mq, TSB200_F16, q, hd, H, pack ? pack->rows : S, pack ? 1 : B, q_rs, a.G));
  TSB_TRY(pa_map_rows(&mk, TSB200_F16, cK, hd, T0 + S, B * Hkv, hd, (int64_t)Tmax * hd));
  TSB_TRY(pa_map_rows(&mv, TSB200_F16, cV, hd, T0 + S, B * Hkv, hd, (int64_t)Tmax * hd));
  if (hd == 64) return pa_launch<__half, 1, 1, 4, 4>(device, mq, mk, mk, mv, a, s);
  return pa_launch<__half, 2, 2, 2, 2>(device, mq, mk, mk, mv, a, s);
}

bool latent_prefill_tc_shape(int dtype, const LatentShape& a) {
  const int qb = (a.dim + a.rot) / 64;
  return dtype == TSB200_BF16 && a.dim % 64 == 0 && a.rot % 64 == 0 && (qb == 2 || qb == 3) && (a.vdim == 64 || a.vdim == 128) && a.rank % 8 == 0;
}

int launch_latent_prefill_tc(int device, const LatentArgs& l, cudaStream_t s) {
  const LatentShape& sh = l.shape;
  const int T = l.T0 + l.S, kvw = sh.H * (sh.dim + sh.vdim);
  PaArgs a{};
  a.out = l.out; a.B = l.B; a.S = l.S; a.T0 = l.T0; a.H = sh.H; a.heads = sh.H; a.G = 1; a.QT = kPaRows;
  a.c = sh.scale * 1.44269504088896340736f;
  a.k_boxes = sh.dim / 64; a.kx = sh.dim; a.vx0 = sh.H * sh.dim; a.vx = sh.vdim; a.rx = sh.rank; a.z_seq = 1;
  CUtensorMap mq, mk, mr;
  TSB_TRY(pa_map_q(&mq, TSB200_BF16, l.q, sh.dim + sh.rot, sh.H, l.S, l.B, l.q_stride, 1));
  TSB_TRY(pa_map_rows(&mk, TSB200_BF16, l.kv, kvw, T, l.B, kvw, (int64_t)T * kvw));
  TSB_TRY(pa_map_rows(&mr, TSB200_BF16, l.cache, sh.row, T, l.B, sh.row, l.seq_stride));
  typedef __nv_bfloat16 bf16;
  if (sh.dim + sh.rot == 192) {
    if (sh.vdim == 128) return pa_launch<bf16, 3, 2, 2, 1>(device, mq, mk, mr, mk, a, s);
    return pa_launch<bf16, 3, 1, 2, 2>(device, mq, mk, mr, mk, a, s);
  }
  if (sh.vdim == 128) return pa_launch<bf16, 2, 2, 2, 2>(device, mq, mk, mr, mk, a, s);
  return pa_launch<bf16, 2, 1, 3, 3>(device, mq, mk, mr, mk, a, s);
}

}  // namespace tsb
