// Linear layer of 1..64 rows on packed fp16 / bf16 weights: y[M,N] = epilogue(x[M,K] * W[K,N]), the K ranges of an output's columns on
// the CTAs of one cluster, their sums through distributed shared memory.
//
// The WEIGHTS are the 128-row operand of tcgen05.mma (A, read in place from the packed tiles, MN-major, 128-byte swizzle), the activation
// rows its N dimension (B: [16 / 32 / 64 rows][64 k], K-major, one TMA tensor copy per stage, rows beyond M zero-filled).  A CTA owns
// 128 columns over a range of K; the 1, 2, 4 or 8 CTAs of a cluster share the columns.  When its products are done a CTA pushes every
// sum into the shared memory of the CTA that finishes it (each finishes 1 / ks of the columns), one cluster barrier, and the sums
// are added in rank order (bitwise reproducible): no scratch in global memory, no counters, no last arriver that reads the others' slots.
//
// What bounds a decode step's linears is the chain from one launch to the next, not their bytes: a CTA takes at most half of an SM's
// shared memory, so that the next launch's CTAs are resident, have their barriers, TMEM and first weight tiles (at these sizes often
// their whole share) before the current launch ends.  Only the activation tiles wait for it.
// warp 0: copies; warp 1: TMEM and products; warps 2-5: accumulators out of TMEM; all warps: sums and epilogue.
#include "cluster_sums.cuh"
#include "stream_common.cuh"
#include "tc_common.cuh"

namespace tsb {

constexpr int kLcThreads = 192;
constexpr int kLcMaxSections = 4;

struct LcSection {
  int ct_end;   // first column tile (256 columns) after the section
  int N;
  int x_block;  // stacked row block it reads
  int pieces;   // four columns at a time in the epilogue
  Epilogue ep;
};
struct LcArgs {
  const unsigned char* Wp;
  int M, KB, ks, stages;
  int* error;
  int n_sec;
  LcSection sec[kLcMaxSections];
  int rope_on;  // one section only
  RopeFuse rope;
};

template <int NR>
__device__ __forceinline__ void lc_tmem_ld(uint32_t taddr, uint32_t* r) {
  if constexpr (NR == 16) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
  } else {
    tmem_ld32(taddr, r);
  }
}

template <typename H, int NR>
__global__ void __launch_bounds__(kLcThreads) gemm_cluster_tc_kernel(const __grid_constant__ CUtensorMap mapX, LcArgs a) {
  constexpr int kX = NR * 128, kStage = 16384 + kX;
  constexpr uint32_t kCols = NR < 32 ? 32 : NR;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int S = a.stages, ks = a.ks, M = a.M, KB = a.KB;
  float* red = reinterpret_cast<float*>(smem + S * kStage);   // [source rank][items of this CTA][4 columns]
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * kStage + NR * 512);
  uint64_t* empty = full + 8;
  uint64_t* acc = empty + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc + 1);
  __shared__ int s_err;

  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int rank = (int)(blockIdx.x % ks), group = (int)(blockIdx.x / ks);
  int si = 0;
  while (si < a.n_sec - 1 && (group >> 1) >= a.sec[si].ct_end) ++si;
  const Epilogue& ep = a.sec[si].ep;
  const int N = a.sec[si].N, xrow = a.sec[si].x_block * M;
  const int col0 = (group - (si ? a.sec[si - 1].ct_end * 2 : 0)) * 128;   // of the section
  const int KP = (KB + 1) / 2, p0 = KP * rank / ks, n_it = KP * (rank + 1) / ks - p0;   // pairs of k tiles

  if (tid == 0) {
    for (int i = 0; i < S; ++i) {
      tc_mbar_init(&full[i], 1);
      tc_mbar_init(&empty[i], 1);
    }
    tc_mbar_init(acc, 1);
    s_err = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (w == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();
  // weights do not depend on the previous kernel
  const unsigned char* wsrc = a.Wp + ((size_t)(group >> 1) * KB) * kTileBytes + (size_t)(group & 1) * 8192;
  auto weights = [&](int i) {
    const int s = i % S, kb = (p0 + i) * 2;
    const bool two = kb + 1 < KB;
    tc_mbar_expect_tx(&full[s], (two ? 16384 : 8192) + kX);
    tc_bulk_g2s(smem + s * kStage, wsrc + (size_t)kb * kTileBytes, 8192, &full[s]);
    if (two) tc_bulk_g2s(smem + s * kStage + 8192, wsrc + (size_t)(kb + 1) * kTileBytes, 8192, &full[s]);
  };
  const int n_pre = min(S, n_it);
  if (tid == 0)
    for (int i = 0; i < n_pre; ++i) weights(i);
  __syncwarp();
  if (ks > 1) cl_sync();   // the other CTAs exist before anything is pushed to them
  pdl_wait();

  if (tid == 0) {
    // ---------------- copies
    int i = 0;
    for (; i < n_it; ++i) {
      const int s = i % S;
      if (i >= S) {
        if (!tc_mbar_wait(&empty[s], (unsigned)((i / S - 1) & 1))) {
          s_err = 1;
          break;
        }
        weights(i);
      }
      tma_load_2d(smem + s * kStage + 16384, &mapX, (p0 + i) * 64, xrow, &full[s]);   // rows behind the block's are columns nobody reads
    }
    if (s_err)   // copies in flight land first
      for (int j = max(0, i - S); j < i; ++j) tc_mbar_wait(&full[j % S], (unsigned)((j / S) & 1));
  } else if (tid == 32) {
    // ---------------- products.  Instruction descriptor: fp32 accumulator, A MN-major, B K-major, N = NR, M = 128
    const uint32_t idesc = (1u << 4) | (Pair16<H>::kUmmaFormat << 7) | (Pair16<H>::kUmmaFormat << 10) | (1u << 15) | ((uint32_t)(NR >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    for (int i = 0; i < n_it; ++i) {
      const int s = i % S;
      if (!tc_mbar_wait(&full[s], (unsigned)((i / S) & 1))) {
        s_err = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t wb = s_u32(smem + s * kStage), xb = wb + 16384;
      const int kk_end = (p0 + i) * 2 + 1 < KB ? 4 : 2;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        if (kk >= kk_end) break;
        // A: [k tile][64-column box 2][32 k][128 B]: boxes 4096 B apart (LBO), 8-k groups 1024 B apart (SBO); B: rows of 128 B, atoms of 8 rows
        umma_f16(tmem, make_desc(wb + (kk >> 1) * 8192 + (kk & 1) * 2048, 4096, 1024), make_desc(xb + kk * 32, 16, 1024), idesc, (i > 0 || kk > 0) ? 1u : 0u);
      }
      umma_commit(&empty[s]);
    }
    umma_commit(acc);
  }
  __syncwarp();

  // This CTA finishes 128 / ks of the columns, in groups of four, of every row.  The CTA that finishes a column is the same for all rows, and a
  // thread's groups, kLcThreads apart, have the same columns: no index arithmetic per row.  (Rows x columns shared out as one range cost a
  // division per pushed sum; as straight-line code of 40 KB that was the launch's longest part, 0.15 us per row: 64 rows of 64 -> 64 19.5 us,
  // now 10.7; of 4096 -> 22016 53.0, now 42.0.)  Bias and the first group's residual are on their way while the products run.
  const int gsh = 5 - (31 - __clz(ks)), per = M << gsh;   // log2 of a row's groups here; groups of this CTA
  const int c = col0 + ((rank << gsh) + (tid & ((1 << gsh) - 1))) * 4;
  const bool pieces = a.sec[si].pieces != 0;
  float bias[4], res[4];
  cl_bias<H>(ep, N, c, bias);
  if (tid < per) cl_residual(ep, N, tid >> gsh, c, pieces, res);
  if (w >= 2) {
    // ---------------- sums out of TMEM: warp w reads lanes 32 (w % 4) .. = columns of the group
    const bool ok = __all_sync(0xffffffffu, tc_mbar_wait(acc, 0));
    if (!ok) s_err = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int col = (w & 3) * 32 + lane, owner = col >> (gsh + 2);
    float* at = red + ((size_t)rank * per + ((col >> 2) & ((1 << gsh) - 1))) * 4 + (col & 3);   // [source rank][row][group][4]
    const uint32_t local = s_u32(at), step = 16u << gsh;
    uint32_t remote = local;
    if (ks > 1) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(owner));
#pragma unroll
    for (int h = 0; h < (NR + 31) / 32; ++h) {
      uint32_t v[NR < 32 ? NR : 32];
      lc_tmem_ld<NR>(tmem + ((uint32_t)((w & 3) * 32) << 16) + h * 32, v);
#pragma unroll
      for (int r = 0; r < (NR < 32 ? NR : 32); ++r) {
        const int row = h * 32 + r;
        if (row < M) {
          if (ks > 1) asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(remote + row * step), "r"(v[r]) : "memory");
          else asm volatile("st.shared.b32 [%0], %1;" ::"r"(local + row * step), "r"(v[r]) : "memory");
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  if (ks > 1) cl_sync();
  else __syncthreads();

  // ---------------- epilogue
#pragma unroll 1
  for (int i = tid; i < per; i += kLcThreads) {
    float next[4];
    if (i + kLcThreads < per) cl_residual(ep, N, (i + kLcThreads) >> gsh, c, pieces, next);
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int r = 0; r < ks; ++r) {
      const float4 t = *reinterpret_cast<const float4*>(red + (size_t)(r * per + i) * 4);
      v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
    }
    cl_finish4<H>(ep, N, i >> gsh, c, pieces, v, bias, res, a.rope_on, a.rope);
#pragma unroll
    for (int e = 0; e < 4; ++e) res[e] = next[e];
  }
  __syncthreads();
  if (w == 1) {
    if (lane == 0 && s_err) tc_mbar_wait(acc, 0);   // some warp gave up: products in flight end before TMEM is given back
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
  }
  if (tid == 0 && s_err && a.error) *a.error = 1;
}

template <typename H, int NR>
static int lc_launch(int device, const CUtensorMap& map, LcArgs a, int groups, int sms, bool pdl, cudaStream_t s) {
  constexpr int kStage = 16384 + NR * 128;
  // two CTAs per SM; three where that makes one wave of what would be a full and a nearly empty one (two to three groups per SM; 32 rows of
  // 768 -> 50257: 26.4 -> 17.6 us; the rings of more rows than 32 do not fit three times)
  const int per_sm = NR <= 32 && groups > 2 * sms && groups <= 3 * sms ? 75 : 112;
  a.stages = (per_sm * 1024 - 1024 - 256 - NR * 512) / kStage;
  const int smem = a.stages * kStage + NR * 512 + 256 + 1024;
  static bool done[kMaxDevices] = {};
  if (!done[device]) {
    TSB_CUDA(cudaFuncSetAttribute(gemm_cluster_tc_kernel<H, NR>, cudaFuncAttributeMaxDynamicSharedMemorySize, 114 * 1024));
    done[device] = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(groups * a.ks);
  cfg.blockDim = dim3(kLcThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = a.ks;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = (pdl && pdl_enabled()) ? 2 : 1;
  TSB_CUDA(cudaLaunchKernelEx(&cfg, gemm_cluster_tc_kernel<H, NR>, map, a));
  count_launch(device);
  return check_launch("gemm_cluster_tc");
}

// groups: of 128 columns; rows: of x; 1 ok, 0 error, 2 not handled
static int lc_run(int device, DeviceState* st, int dtype, const void* x, int rows, int K, LcArgs a, int groups, bool pdl, cudaStream_t s) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return 2;
  a.KB = (K + 31) / 32;
  // K ranges while all CTAs are resident at once (two per SM), of at least two steps of 64 k each: more copies in flight and a shorter chain
  // per CTA.  Against one CTA per SM (more room for the next launch): 16384-token decode of the 1B-class model 22.3 / 23.2 ms, 7B-class
  // step 2.68 / 2.98 ms, 64 sequences 5.33 / 5.57 ms.
  const int KP = (a.KB + 1) / 2;
  a.ks = 1;
  while (a.ks < 8 && (int64_t)groups * a.ks * 2 <= 2 * st->sm_count && KP / (a.ks * 2) >= 2) a.ks *= 2;
  a.error = tc_error_word(device);
  const int NR = a.M <= 16 ? 16 : (a.M <= 32 ? 32 : 64);
  CUtensorMap map;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)NR};
  const cuuint32_t el[2] = {1, 1};
  const CUresult r = enc(&map, dtype == TSB200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(x), dims, strides, box,
                         el, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TSB_CHECK(r == CUDA_SUCCESS, "gemm_cluster_tc: cuTensorMapEncodeTiled failed with %d", (int)r);
#define TSB_LC(H)                                                     \
  (NR == 16 ? lc_launch<H, 16>(device, map, a, groups, st->sm_count, pdl, s)        \
            : (NR == 32 ? lc_launch<H, 32>(device, map, a, groups, st->sm_count, pdl, s) : lc_launch<H, 64>(device, map, a, groups, st->sm_count, pdl, s)))
  return dtype == TSB200_BF16 ? TSB_LC(__nv_bfloat16) : TSB_LC(__half);
#undef TSB_LC
}

static bool lc_takes(int dtype, const void* x, const void* Wp, int M, int K) {
  return is_16bit(dtype) && M >= 1 && M <= 64 && K % 8 == 0 && (((uintptr_t)x | (uintptr_t)Wp) % 16) == 0;
}

// 1 ok, 0 error, 2 shape not handled (the caller takes another kernel)
int launch_gemm_cluster_tc(int device, DeviceState* st, int dtype, const void* x, const void* Wp, int M, int K, int N, const Epilogue& ep, bool pdl, cudaStream_t s,
                           const RopeFuse* rope) {
  if (!lc_takes(dtype, x, Wp, M, K)) return 2;
  LcArgs a{};
  a.Wp = reinterpret_cast<const unsigned char*>(Wp);
  a.M = M; a.n_sec = 1;
  a.sec[0].ct_end = (N + 255) / 256; a.sec[0].N = N; a.sec[0].ep = ep; a.sec[0].pieces = cl_whole_pieces(ep, N, 2);
  if (rope) {
    if (!cl_rope_fits(*rope, ep, N, 2)) return 2;
    a.rope_on = 1;
    a.rope = *rope;
  }
  return lc_run(device, st, dtype, x, M, K, a, (N + 127) / 128, pdl, s);
}

// several linears of equal K on stacked row blocks, each from a column tile of its own on
int launch_gemm_cluster_sections(int device, DeviceState* st, int dtype, const void* x, const void* Wp, int M, int K, const LinearSection* sec, int n_sec, bool pdl,
                                 cudaStream_t s) {
  if (!lc_takes(dtype, x, Wp, M, K) || n_sec < 1 || n_sec > kLcMaxSections) return 2;
  LcArgs a{};
  a.Wp = reinterpret_cast<const unsigned char*>(Wp);
  a.M = M; a.n_sec = n_sec;
  int ct = 0, blocks = 1;
  for (int i = 0; i < n_sec; ++i) {
    ct += (sec[i].N + 255) / 256;
    a.sec[i].ct_end = ct; a.sec[i].N = sec[i].N; a.sec[i].ep = sec[i].ep; a.sec[i].x_block = sec[i].x_block;
    a.sec[i].pieces = cl_whole_pieces(sec[i].ep, sec[i].N, 2);
    if (sec[i].x_block + 1 > blocks) blocks = sec[i].x_block + 1;
  }
  const int last = sec[n_sec - 1].N;   // an odd half of the last column tile is left out
  return lc_run(device, st, dtype, x, blocks * M, K, a, (ct - (last + 255) / 256) * 2 + (last + 127) / 128, pdl, s);
}

}  // namespace tsb
