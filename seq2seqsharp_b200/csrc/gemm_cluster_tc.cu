// Linear layer of 1..64 rows on packed fp16 / bf16 weights: y[M,N] = epilogue(x[M,K] * W[K,N]), the K ranges of an output's columns on
// the CTAs of one cluster, their sums through distributed shared memory.
//
// The WEIGHTS are the 128-row operand of tcgen05.mma (A, read in place from the packed tiles, MN-major, 128-byte swizzle), the activation
// rows its N dimension (B: [16 / 32 / 64 rows][64 k], K-major, one TMA tensor copy per stage, rows beyond M zero-filled).  A CTA owns
// 128 columns over a range of K; the 1, 2, 4 or 8 CTAs of a cluster share the columns.  When its products are done a CTA pushes every
// sum, four rows at a time, into the shared memory of the CTA that finishes it (each finishes 1 / ks of the columns); the stores report to
// that CTA's mbarrier, and the sums are added in rank order (bitwise reproducible): no scratch in global memory, no counters, no last arriver
// that reads the others' slots, and nobody waits for more than its own sums.
//
// What bounds a decode step's linears is the chain from one launch to the next, not their bytes: a CTA takes at most half of an SM's
// shared memory, so that the next launch's CTAs are resident, have their barriers, TMEM and first weight tiles (at these sizes often
// their whole share) before the current launch ends.  Only the activation tiles wait for it.
// warp 0: copies; warp 1: TMEM and products; warps 2-5: accumulators out of TMEM; all warps: sums and epilogue.
// Parts of a launch in clocks after the one before it has ended (8 rows of 768 -> 768, three steps of 64 k a CTA): first operands 1100, products
// 700, push 270, the cluster's sums 350, epilogue 1000, leaving 400.  Before the products were issued by a whole warp, the sums pushed four
// rows at a time with a barrier of their own and the epilogue's kinds had loops of their own: 1350, 1900, 650, 1400, 1450, 400.  Launches of
// a captured step, before -> now (us): 8 rows of the 768-wide model 4.80 -> 3.58, 32 rows of the 2048-wide one 10.1 -> 8.4, one row of the
// 4096-wide one 16.5 -> 14.7, 64 rows 23.2 -> 20.2.  Four CTAs' registers fit an SM (64 a thread): the kernels behind need room beside two of these.
#include "cluster_sums.cuh"
#include "stream_common.cuh"
#include "tc_common.cuh"

namespace tsb {

constexpr int kLcThreads = 256;
constexpr int kLcMaxSections = 4;

struct LcSection {
  int ct_end;   // first column tile (256 columns) after the section
  int N;
  int x_block;  // stacked row block it reads
  int kind;     // ClKind: which loop finishes it
  Epilogue ep;
};
struct LcArgs {
  const unsigned char* Wp;
  int M, KB, ks, stages;
  unsigned wait_limit;  // polls of a wait before the CTA gives up
  int* error;
  int n_sec;
  LcSection sec[kLcMaxSections];
  // one section only, of kind kClRope
  RopeFuse rope;
};

template <int NR>
__device__ __forceinline__ void lc_tmem_ld(uint32_t taddr, uint32_t* r) {
  if constexpr (NR == 16) {
    __syncwarp();
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
__global__ void __launch_bounds__(kLcThreads, 4) gemm_cluster_tc_kernel(const __grid_constant__ CUtensorMap mapX, LcArgs a) {
  constexpr int kX = NR * 128, kStage = 16384 + kX;
  constexpr uint32_t kCols = NR < 32 ? 32 : NR;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int S = a.stages, ks = a.ks, M = a.M, KB = a.KB;
  float* red = reinterpret_cast<float*>(smem + S * kStage);   // [source rank][row quad][column of a group][group][4 rows]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S * kStage + NR * 512);
  const uint32_t full = s_u32(bars), empty = full + 64, acc = empty + 64, sums = acc + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  __shared__ int s_err, s_asked;   // s_asked: steps whose copies are under way or done (warp 0)

  const int tid = threadIdx.x, lane = tid & 31, w = warp_index();
  const int rank = (int)(blockIdx.x % ks), group = (int)(blockIdx.x / ks);
  int si = 0;
  while (si < a.n_sec - 1 && (group >> 1) >= a.sec[si].ct_end) ++si;
  const Epilogue& ep = a.sec[si].ep;
  const int N = a.sec[si].N, xrow = a.sec[si].x_block * M;
  const int col0 = (group - (si ? a.sec[si - 1].ct_end * 2 : 0)) * 128;   // of the section
  const int KP = (KB + 1) / 2, p0 = KP * rank / ks, n_it = KP * (rank + 1) / ks - p0;   // pairs of k tiles
  const int quads = (M + 3) >> 2;

  if (tid == 0) {
    for (int i = 0; i < S; ++i) {
      tc_mbar_init(bars + i, 1);
      tc_mbar_init(bars + 8 + i, 1);
    }
    tc_mbar_init(bars + 16, 1);
    tc_mbar_init(bars + 17, 1);
    s_err = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (ks > 1) tc_mbar_expect_tx(bars + 17, quads * 2048);   // 128 / ks columns from each of ks CTAs
  }
  if (w == 1) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();
  volatile int* err = &s_err;
  const uint32_t ring = s_u32(smem);
  // weights do not depend on the previous kernel
  const unsigned char* wsrc = a.Wp + ((size_t)(group >> 1) * KB + (size_t)p0 * 2) * kTileBytes + (size_t)(group & 1) * 8192;
  auto weights = [&](int i, int s) {
    const bool two = (p0 + i) * 2 + 1 < KB;
    const unsigned char* src = wsrc + (size_t)i * (2 * kTileBytes);
    const uint32_t dst = ring + s * kStage, bar = full + s * 8;
    tc_mbar_expect_el(bar, (two ? 16384 : 8192) + kX);
    tc_bulk_g2s_el(dst, src, 8192, bar);
    if (two) tc_bulk_g2s_el(dst + 8192, src + kTileBytes, 8192, bar);
  };
  const int n_pre = min(S, n_it);
  if (w == 0) {
    if (elect_one()) asm volatile("prefetch.tensormap [%0];" ::"l"(&mapX) : "memory");
    __syncwarp();
    for (int i = 0; i < n_pre; ++i) weights(i, i);
  }
  // This CTA finishes 128 / ks of the columns, in groups of four, of every row.  A warp takes eight groups of the four rows of a quad at a time
  // (quad-major, so that its reads of a slot are 32 different banks); a thread's columns are the same in all of its quads: no index
  // arithmetic per row.  Bias, position and rotation are asked for before the wait, the first row's residual while the products run.
  const int gsh = 5 - (31 - __clz(ks)), G = 1 << gsh;          // groups here
  const int g = (tid >> 2) & (G - 1);
  const int c = col0 + ((rank << gsh) + g) * 4, row0 = (tid >> (gsh + 2)) * 4 + (tid & 3), step = (kLcThreads >> (gsh + 2)) * 4;
  ClAhead<H> ahead;
  ahead.start(ep, a.sec[si].kind, N, c, row0, M, a.rope);
  if (ks > 1) cluster_sync();   // the other CTAs' barriers exist before anything is pushed to them
  pdl_wait();

  if (w == 0) {
    // ---------------- copies
    int s = 0;
    unsigned phase = 1;   // parity of the ring's previous round
    int i = 0;
    for (; i < n_it; ++i) {
      if (i >= S) {
        if (!tc_wait_or(empty + s * 8, phase, err, a.wait_limit)) break;
        weights(i, s);
      }
      tma_load_2d_el(ring + s * kStage + 16384, &mapX, (p0 + i) * 64, xrow, full + s * 8);   // rows behind the block's are columns nobody reads
      if (++s == S) s = 0, phase ^= 1;
    }
    if (lane == 0) s_asked = i;
    named_arrive<1, 192>();
  } else if (w == 1) {
    // ---------------- products.  Instruction descriptor: fp32 accumulator, A MN-major, B K-major, N = NR, M = 128
    const uint32_t idesc = (1u << 4) | (Pair16<H>::kUmmaFormat << 7) | (Pair16<H>::kUmmaFormat << 10) | (1u << 15) | ((uint32_t)(NR >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    // A: [k tile][64-column box 2][32 k][128 B]: boxes 4096 B apart (LBO), 8-k groups 1024 B apart (SBO); B: rows of 128 B, atoms of 8 rows
    const uint32_t hi = desc_hi(1024), a0 = desc_lo(ring, 4096), b0 = desc_lo(ring + 16384, 16);
    int s = 0;
    unsigned phase = 0;
    for (int i = 0; i < n_it; ++i) {
      if (!tc_wait_or(full + s * 8, phase, err, a.wait_limit)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t ad = a0 + s * (kStage >> 4), bd = b0 + s * (kStage >> 4);
      umma_el(tmem, ad, hi, bd, hi, idesc, i > 0);
      umma_el(tmem, ad + 128, hi, bd + 2, hi, idesc, 1);
      if ((p0 + i) * 2 + 1 < KB) {
        umma_el(tmem, ad + 512, hi, bd + 4, hi, idesc, 1);
        umma_el(tmem, ad + 640, hi, bd + 6, hi, idesc, 1);
      }
      umma_commit_el(empty + s * 8);
      if (++s == S) s = 0, phase ^= 1;
    }
    umma_commit_el(acc);
  }
  __syncwarp();

  ahead.first(ep, a.sec[si].kind, N, c, row0, M, a.rope);
  if (w >= 2 && w < 6) {
    // ---------------- sums out of TMEM: warp w reads lanes 32 (w % 4) .. = columns of the group
    tc_wait_or(acc, 0, err, a.wait_limit);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int col = (w & 3) * 32 + lane, owner = col >> (gsh + 2), e = col & 3, here = ((col >> 2) + 2 * e) & (G - 1);
    const uint32_t local = s_u32(red) + ((uint32_t)rank * quads * (G * 4) + e * G + here) * 16, hop = G * 64;
    uint32_t remote = local, bar = sums;
    if (ks > 1) {
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(owner));
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(sums), "r"(owner));
    }
#pragma unroll
    for (int h = 0; h < (NR + 31) / 32; ++h) {
      uint32_t v[NR < 32 ? NR : 32];
      lc_tmem_ld<NR>(tmem + ((uint32_t)((w & 3) * 32) << 16) + h * 32, v);
#pragma unroll
      for (int r = 0; r < (NR < 32 ? NR : 32); r += 4) {
        const int qd = (h * 32 + r) >> 2;
        if (qd < quads) {
          if (ks > 1)
            asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(remote + qd * hop), "r"(v[r]), "r"(v[r + 1]),
                         "r"(v[r + 2]), "r"(v[r + 3]), "r"(bar)
                         : "memory");
          else
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(local + qd * hop), "r"(v[r]), "r"(v[r + 1]), "r"(v[r + 2]), "r"(v[r + 3]) : "memory");
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    named_arrive<1, 192>();   // TMEM has been read
  }
  if (ks > 1) {
    // arrived when everything is pushed (a CTA that gave up has pushed too); waited for before the CTA leaves, so that nobody pushes to one that has
    cluster_arrive_relaxed();
    tc_wait_or(sums, 0, err, a.wait_limit);
  } else {
    __syncthreads();
  }

  // ---------------- epilogue: rank order; a group's column e lies 2 e groups further on, so that neither the pushes nor these reads meet in a bank
  const float* from = red + ((size_t)(row0 >> 2) * (G * 4)) * 4 + (row0 & 3);
  const int at0 = g * 4, at1 = (G + ((g + 2) & (G - 1))) * 4, at2 = (2 * G + ((g + 4) & (G - 1))) * 4, at3 = (3 * G + ((g + 6) & (G - 1))) * 4;
  const int hop = quads * (G * 16), skip = (step >> 2) * (G * 16);
  auto sum4 = [&](const float* f, float* v) {
    v[0] = f[at0]; v[1] = f[at1]; v[2] = f[at2]; v[3] = f[at3];
    for (int r = 1; r < ks; ++r) {
      f += hop;
      v[0] += f[at0]; v[1] += f[at1]; v[2] += f[at2]; v[3] += f[at3];
    }
  };
  cl_finish_rows<H>(ep, a.sec[si].kind, N, c, row0, M, step, from, skip, ahead, a.rope, sum4);
  if (ks > 1) {
    if (*err) tc_wait_short(sums, 0);   // what is on its way here lands first
    cluster_wait();
  }
  if (w == 1) {
    named_sync<1, 192>();
    if (*err) {   // warp 0, 1 or one of those that read TMEM has given up: copies and products in flight end first (otherwise the products have waited for every
      tc_land(full, S, s_asked);   // copy, and TMEM was read behind the last product)
      tc_wait_short(acc, 0);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
  }
  if (*err && lane == 0 && a.error) *a.error = 1;   // the warp that gave up, at least, sees it
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
  // per CTA.  Against one CTA per SM (fewer ranks, fewer pushes, more room for the next launch), ms of whole calls: 32 steps of one row of the 7B-class
  // model 71.5 / 76.6, 16 of its 64 rows 60.1 / 63.0, 16 of four rows of the 1B-class one after 16384 tokens 17.2 / 17.4; 8 rows of 768 and 32 of
  // 2048 the same (21.6, 28.6): the rule does not look at the rows.
  const int KP = (a.KB + 1) / 2;
  a.ks = 1;
  while (a.ks < 8 && (int64_t)groups * a.ks * 2 <= 2 * st->sm_count && KP / (a.ks * 2) >= 2) a.ks *= 2;
  a.error = tc_error_word(device);
  a.wait_limit = tc_wait_limit();
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
  a.sec[0].ct_end = (N + 255) / 256; a.sec[0].N = N; a.sec[0].ep = ep; a.sec[0].kind = rope ? kClRope : cl_kind(ep, N, 2);
  if (rope) {
    if (!cl_rope_fits(*rope, ep, N, 2)) return 2;
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
    a.sec[i].kind = cl_kind(sec[i].ep, sec[i].N, 2);
    if (sec[i].x_block + 1 > blocks) blocks = sec[i].x_block + 1;
  }
  const int last = sec[n_sec - 1].N;   // an odd half of the last column tile is left out
  return lc_run(device, st, dtype, x, blocks * M, K, a, (ct - (last + 255) / 256) * 2 + (last + 127) / 128, pdl, s);
}

}  // namespace tsb
