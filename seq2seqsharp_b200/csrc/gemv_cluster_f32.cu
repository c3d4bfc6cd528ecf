// fp32 linear of 1..8 rows on packed weights: y[M,N] = epilogue(x[M,K] * W[K,N]), the K ranges of 128 columns on the CTAs of a cluster.
//
// The fp32 counterpart of gemm_cluster_tc.cu (no tensor-core type keeps fp32): a CTA streams its 16 KB tiles ([32 k][128 columns]) through a
// ring of bulk copies, eight warps take four k of a tile each (a lane four columns of every row), the warps' sums meet in shared memory, the
// cluster's through distributed shared memory in rank order.  Two CTAs fit an SM while the rows over a CTA's K range take up to 28 KB; the
// weights are asked for before the launch in front has ended.  What bounds a small model's step is the chain of its launches (512-wide, six layers, one sequence, a
// 128-token request: 42.7 ms with the persistent stream-K kernel, 19.6 with this one).
#include "cluster_sums.cuh"
#include "stream_common.cuh"

namespace tsb {

constexpr int kFcThreads = 288, kFcStages = 5;
// Rows of up to 1024 are normed here instead of by a launch in front, which takes 2.1 us of a step's chain of launches; reading the whole rows
// and their two sums costs this launch about 0.9 us for one row (512 wide: a 128-token request 22.4 -> 20.4 ms).  Longer rows would be read by every
// CTA for more than that, and so are 5 to 8 rows of 512 and more.  us per step of six layers, normed here / by a launch: 512 wide, 1 row 119 / 132,
// 4 143 / 157, 5 221 / 195, 8 227 / 198; 1024 wide, 1 row 170 / 187, 4 241 / 254, 8 390 / 283; 448 wide, 5 rows 179 / 185, 8 209 / 217; 256 wide, 8 146 / 152.
constexpr int kFcNormRegs = 8;   // float4 of a row per lane
static bool fc_norms(int M, int K) { return K > 0 && K % 4 == 0 && K <= kFcNormRegs * 128 && (M <= 4 || K < 512); }

struct FcArgs {
  const float* x;
  const unsigned char* Wp;
  int M, N, K, KB, ks;
  unsigned wait_limit;  // polls of a wait before a warp gives up
  int* error;
  Epilogue ep;
  int kind;    // ClKind
  int norm;    // 0: rows as they are, 1: RMSNorm, 2: LayerNorm of them (gamma, beta, eps) first
  const float* gamma;
  const float* beta;
  float eps;
  RopeFuse rope;
};
// dynamic shared memory: ring | sums of the cluster [M * 32 groups][4] | rows of x over the CTA's range
static size_t fc_smem(int RM, int tiles) { return (size_t)kFcStages * kTileBytes + (size_t)RM * 512 + (size_t)RM * tiles * 128; }

// 5 to 8 rows: nine warps of more than 96 registers are one CTA per SM (a quarter of the register file holds four of 112).  That suits models of less
// than 512, which norm their rows here and whose launches have CTAs for a part of the SMs; of wider models half the launches would take two waves (8 x
// 1024 x 4096 19.7 us, now 10.7; a step of six layers, 8 rows of 1024, 363 and 281).  Those have no norm in their kernel and ask for what the epilogue
// reads behind the products instead of in front of the wait (kLate): 93 registers.
template <int RM, bool NORM>
__global__ void __launch_bounds__(kFcThreads, RM == 8 && !NORM ? 2 : 0) gemv_cluster_f32_kernel(FcArgs a) {
  constexpr bool kLate = RM == 8 && !NORM;
  extern __shared__ __align__(1024) unsigned char fc_raw[];
  __shared__ uint64_t full[kFcStages], empty[kFcStages], sums;
  __shared__ float2 stat[8];   // mean and divisor of a row
  __shared__ int s_err;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int ks = a.ks, M = a.M, rank = (int)(blockIdx.x % ks), group = (int)(blockIdx.x / ks);
  const int t0 = a.KB * rank / ks, n_it = a.KB * (rank + 1) / ks - t0;
  float* red = reinterpret_cast<float*>(fc_raw + kFcStages * kTileBytes);
  float* xs = red + RM * 128;   // [RM][n_it * 32]
  if (tid == 0) {
    for (int i = 0; i < kFcStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 8);
    }
    mbar_init(&sums, 1);
    s_err = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (ks > 1) mbar_expect_tx(&sums, M * 512);   // four columns of M * 32 / ks groups from each of ks CTAs
  }
  __syncthreads();
  pdl_trigger();
  const unsigned char* src = a.Wp + ((size_t)group * a.KB + t0) * kTileBytes;
  const int n_pre = min(kFcStages, n_it);
  if (tid == 256)
    for (int i = 0; i < n_pre; ++i) {
      mbar_expect_tx(&full[i], kTileBytes);
      bulk_g2s(fc_raw + i * kTileBytes, src + (size_t)i * kTileBytes, kTileBytes, &full[i]);
    }
  __syncwarp();
  float g0 = 0.0f, b0 = 0.0f;   // gain and shift of the first element this thread norms
  if (NORM && a.norm) {
    const int k = t0 * 32 + tid % (n_it * 32);
    if (k < a.K) {
      g0 = a.gamma[k];
      if (a.beta) b0 = a.beta[k];
    }
  }
  ClAhead<float> ahead;
  const int per = M * 32 / ks;   // groups of four columns this CTA finishes: at most 256, one per thread
  const int c = group * 128 + ((rank * per + tid) & 31) * 4, row = (rank * per + tid) >> 5;
  if (!kLate && tid < per) ahead.start(a.ep, a.kind, a.N, c, row, M, a.rope);
  if (ks > 1) cluster_sync();   // the other CTAs exist before anything is pushed to them
  pdl_wait();
  if (w == 8) {
    if (lane == 0) {
      int i = n_pre;
      for (; i < n_it; ++i) {
        const int s = i % kFcStages;
        if (!mbar_wait(&empty[s], (unsigned)((i / kFcStages - 1) & 1), a.wait_limit)) {
          s_err = 1;
          break;
        }
        mbar_expect_tx(&full[s], kTileBytes);
        bulk_g2s(fc_raw + s * kTileBytes, src + (size_t)i * kTileBytes, kTileBytes, &full[s]);
      }
      // copies in flight land before the CTA ends, whichever warp has given up
      for (int j = max(0, i - kFcStages); j < i; ++j) mbar_wait(&full[j % kFcStages], (unsigned)((j / kFcStages) & 1));
    }
  } else {
    if (!kLate && tid < per) ahead.first(a.ep, a.kind, a.N, c, row, M, a.rope);
    const int kc = n_it * 32;
    if (NORM && a.norm) {
      // A warp takes the statistics of a row (one row: every warp, so that nobody waits), the arithmetic of the norm kernels
      if (RM == 1 || w < M) {
        const float4* xr = reinterpret_cast<const float4*>(a.x + (size_t)(RM == 1 ? 0 : w) * a.K);
        const int n4 = a.K >> 2;
        float4 v[kFcNormRegs];
        float s = 0.0f, mean = 0.0f;
#pragma unroll
        for (int j = 0; j < kFcNormRegs; ++j) v[j] = lane + j * 32 < n4 ? xr[lane + j * 32] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < kFcNormRegs; ++j)
          s += a.norm == 2 ? (v[j].x + v[j].y) + (v[j].z + v[j].w) : (v[j].x * v[j].x + v[j].y * v[j].y) + (v[j].z * v[j].z + v[j].w * v[j].w);
        s = warp_sum(s);
        if (a.norm == 2) {
          mean = s / a.K;
          s = 0.0f;
#pragma unroll
          for (int j = 0; j < kFcNormRegs; ++j) {
            const float p = v[j].x - mean, q = v[j].y - mean, r = v[j].z - mean, t = v[j].w - mean;
            if (lane + j * 32 < n4) s += (p * p + q * q) + (r * r + t * t);
          }
          s = warp_sum(s);
        }
        stat[RM == 1 ? 0 : w] = make_float2(mean, sqrtf(s / (float)a.K + a.eps));   // every warp of one row writes the same
      }
      if (RM == 1) __syncwarp();
      else named_sync<1, 256>();
    }
    for (int i = tid; i < RM * kc; i += 256) {
      const int m = i / kc, k = t0 * 32 + i % kc;
      float v = m < M && k < a.K ? a.x[(size_t)m * a.K + k] : 0.0f;
      if (NORM && a.norm && m < M && k < a.K) {
        v = (i == tid ? g0 : a.gamma[k]) * ((v - stat[m].x) / stat[m].y);
        if (a.beta) v += i == tid ? b0 : a.beta[k];
      }
      xs[i] = v;
    }
    named_sync<1, 256>();
    float4 acc[RM];
#pragma unroll
    for (int m = 0; m < RM; ++m) acc[m] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int i = 0; i < n_it; ++i) {
      const int s = i % kFcStages;
      if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (unsigned)((i / kFcStages) & 1), a.wait_limit))) {
        s_err = 1;
        break;   // the stage is not handed back: its copy may still be on its way
      }
      const float4* t = reinterpret_cast<const float4*>(fc_raw + s * kTileBytes) + w * 4 * 32 + lane;
      float4 wv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) wv[q] = t[q * 32];
#pragma unroll
      for (int m = 0; m < RM; ++m) {
        const float4 xv = *reinterpret_cast<const float4*>(xs + m * kc + i * 32 + w * 4);
        const float xq[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          acc[m].x = fmaf(xq[q], wv[q].x, acc[m].x);
          acc[m].y = fmaf(xq[q], wv[q].y, acc[m].y);
          acc[m].z = fmaf(xq[q], wv[q].z, acc[m].z);
          acc[m].w = fmaf(xq[q], wv[q].w, acc[m].w);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
    }
    if (kLate && tid < per) {
      ahead.start(a.ep, a.kind, a.N, c, row, M, a.rope);
      ahead.first(a.ep, a.kind, a.N, c, row, M, a.rope);
    }
    named_sync<1, 256>();   // every tile is read: the ring holds the warps' sums now
    float4* part = reinterpret_cast<float4*>(fc_raw);   // [warp][row][32 groups]
#pragma unroll
    for (int m = 0; m < RM; ++m) part[(w * RM + m) * 32 + lane] = acc[m];
    named_sync<1, 256>();
    for (int i = tid; i < M * 32; i += 256) {
      float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 p = part[(q * RM + (i >> 5)) * 32 + (i & 31)];
        v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
      }
      const int owner = i / per;
      float* at = red + (size_t)(rank * per + i - owner * per) * 4;
      if (ks > 1) {
        cl_push4(at, &sums, (uint32_t)owner, v);
      } else {
        *reinterpret_cast<float4*>(at) = v;
      }
    }
    __syncwarp();
  }
  if (ks > 1) {
    // arrived when everything is pushed; waited for before the CTA leaves, so that nobody pushes to one that has
    cluster_arrive_relaxed();
    if (tid < per && !cl_wait(&sums, a.wait_limit)) s_err = 1;
  } else {
    __syncthreads();
  }
  if (tid < per) {
    const int hop = per * 4;
    cl_finish_rows<float>(a.ep, a.kind, a.N, c, row, row + 1, 1, red + tid * 4, 0, ahead, a.rope, [&](const float* f, float* v) {
      v[0] = v[1] = v[2] = v[3] = 0.0f;
      for (int r = 0; r < ks; ++r, f += hop) {
        const float4 t = *reinterpret_cast<const float4*>(f);
        v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
      }
    });
  }
  if (ks > 1) {
    if (*(volatile int*)&s_err) cl_wait(&sums);   // what is on its way here lands first
    cluster_wait();
  }
  if (lane == 0 && *(volatile int*)&s_err && a.error) *a.error = 1;   // the warp that gave up, at least, sees it
}

constexpr size_t kFcAlone = 116 * 1024;   // more than half of an SM's shared memory
template <int RM, bool NORM>
static int fc_launch(int device, const FcArgs& a, int groups, size_t smem, bool pdl, cudaStream_t s) {
  static bool done[kMaxDevices] = {};
  if (!done[device]) {
    TSB_CUDA(cudaFuncSetAttribute(gemv_cluster_f32_kernel<RM, NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024));
    done[device] = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(groups * a.ks);
  cfg.blockDim = dim3(kFcThreads);
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
  if constexpr (RM == 8 && !NORM) {
    // Where two CTAs fit an SM, a small launch's clusters lie two CTAs to an SM and leave others idle: here they get an SM each while all clusters are
    // resident that way (a step of six layers, 8 rows of 512 217 us, so 198; of 768 268 / 234).
    static int fit[kMaxDevices][9] = {};   // clusters of so many CTAs, plus one; 0: not asked yet
    if (!fit[device][a.ks]) {
      int n = 0;
      cfg.dynamicSmemBytes = kFcAlone;
      cfg.numAttrs = 1;
      TSB_CUDA(cudaOccupancyMaxActiveClusters(&n, gemv_cluster_f32_kernel<RM, NORM>, &cfg));
      fit[device][a.ks] = n + 1;
    }
    cfg.dynamicSmemBytes = smem < kFcAlone && groups < fit[device][a.ks] ? kFcAlone : smem;
  }
  cfg.numAttrs = (pdl && pdl_enabled()) ? 2 : 1;
  TSB_CUDA(cudaLaunchKernelEx(&cfg, gemv_cluster_f32_kernel<RM, NORM>, a));
  count_launch(device);
  return check_launch("gemv_cluster_f32");
}

// 1 ok, 0 error, 2 shape not handled (the caller takes another kernel)
int launch_gemv_cluster_f32(int device, DeviceState* st, const float* x, const void* Wp, int M, int K, int N, const Epilogue& ep, bool pdl, cudaStream_t s,
                            const RopeFuse* rope, const RowNorm* norm, int norm_width) {
  if (M < 1 || M > 8 || ((uintptr_t)Wp % 16) != 0) return 2;
  if (norm && (!fc_norms(M, K) || ((uintptr_t)x % 16) != 0)) return 2;
  FcArgs a{};
  if (norm) {
    a.norm = norm->type == 0 ? 2 : 1;
    a.gamma = reinterpret_cast<const float*>(norm->gamma); a.beta = reinterpret_cast<const float*>(norm->beta); a.eps = norm->eps;
  }
  a.x = x; a.Wp = reinterpret_cast<const unsigned char*>(Wp);
  a.M = M; a.N = N; a.K = K; a.KB = (K + 31) / 32; a.ep = ep; a.kind = rope ? kClRope : cl_kind(ep, N, 4);
  if (rope) {
    if (!cl_rope_fits(*rope, ep, N, 4)) return 2;
    a.rope = *rope;
  }
  const int groups = (N + 127) / 128, RM = M <= 1 ? 1 : (M <= 2 ? 2 : (M <= 4 ? 4 : 8));
  auto smem_of = [&](int ks) { return fc_smem(RM, (a.KB + ks - 1) / ks); };
  // K ranges while all CTAs are resident at once, of at least two tiles of 32 k.  An SM holds two CTAs, or one where the rows of a range are
  // long (5 to 8 rows of more than 896 k)
  a.ks = 1;
  while (a.ks < 8 && (int64_t)groups * a.ks * 2 <= (int64_t)(smem_of(a.ks * 2) <= 112 * 1024 ? 2 : 1) * st->sm_count && a.KB / (a.ks * 2) >= 2) a.ks *= 2;
  const size_t smem = smem_of(a.ks);
  if (smem > 220 * 1024) return 2;   // rows too long for the shared memory
  a.error = tc_error_word(device);
  a.wait_limit = tc_wait_limit();
  switch (RM) {
    case 1: return fc_launch<1, true>(device, a, groups, smem, pdl, s);
    case 2: return fc_launch<2, true>(device, a, groups, smem, pdl, s);
    case 4: return fc_launch<4, true>(device, a, groups, smem, pdl, s);
    default:   // one kernel for all launches of a step: two in turn would each fetch their code anew (8 rows of 448: 223 us a step against 209)
      return norm || fc_norms(M, norm_width) ? fc_launch<8, true>(device, a, groups, smem, pdl, s) : fc_launch<8, false>(device, a, groups, smem, pdl, s);
  }
}

}  // namespace tsb
