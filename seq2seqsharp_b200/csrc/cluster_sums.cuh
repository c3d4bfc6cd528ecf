// What the linears whose K ranges lie on the CTAs of a cluster share: pushing sums to the CTA that finishes them, and the epilogue of four
// neighbouring columns.
#pragma once
#include "kernels.cuh"

namespace tsb {

__device__ __forceinline__ void cl_push(float* local, uint32_t cta, float v) {
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(cta));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(ra), "f"(v) : "memory");
}
// four sums; the store reports its 16 bytes to the mbarrier of the CTA that receives them
__device__ __forceinline__ void cl_push4(float* local, uint64_t* bar, uint32_t cta, const float4& v) {
  uint32_t ra, rb;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(cta));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb) : "r"((uint32_t)__cvta_generic_to_shared(bar)), "r"(cta));
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(ra), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(rb) : "memory");
}
// first phase of an mbarrier that other CTAs' pushes complete; bounded
__device__ __forceinline__ bool cl_wait(uint64_t* bar, unsigned limit = 1u << 22) {
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(bar);
#pragma unroll 1
  for (unsigned i = 0; i < limit; ++i) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(at)
        : "memory");
    if (ok) return true;
  }
  return false;
}
template <typename H>
__device__ __forceinline__ void cl_store4(H* dst, const float* t) {
  if constexpr (sizeof(H) == 4) *reinterpret_cast<float4*>(dst) = make_float4(t[0], t[1], t[2], t[3]);
  else *reinterpret_cast<uint2*>(dst) = make_uint2(Pair16<H>::put(t[0], t[1]), Pair16<H>::put(t[2], t[3]));
}

// whether the q | k | v epilogue below can serve a linear: whole heads of a multiple of four elements, rows in the model type, no
// activation / gate / residual, four elements on a boundary of theirs
inline bool cl_rope_fits(const RopeFuse& r, const Epilogue& ep, int N, size_t elem) {
  const uintptr_t al = (uintptr_t)ep.y | (uintptr_t)r.cK | (uintptr_t)r.cV;
  return r.hd % 4 == 0 && r.Hd % r.hd == 0 && r.KVd % r.hd == 0 && r.Hd + 2 * r.KVd == N && N % 4 == 0 && ep.y && !ep.y32 && !ep.residual && !ep.gate && !ep.glu &&
         ep.act == TSB200_ACT_NONE && (!r.use_rope || r.tab) && al % (4 * elem) == 0;
}

// whether four columns of every row lie on a boundary of theirs, in all that an epilogue reads and writes
inline bool cl_whole_pieces(const Epilogue& ep, int N, size_t elem) {
  return N % 4 == 0 && ((uintptr_t)ep.y | (uintptr_t)ep.bias | (uintptr_t)ep.gate) % (4 * elem) == 0 && ((uintptr_t)ep.y32 | (uintptr_t)ep.residual) % 16 == 0;
}

// bias of four columns (zeros where there is none), for cl_finish4
template <typename H>
__device__ __forceinline__ void cl_bias(const Epilogue& ep, int N, int c, float* bias) {
  const H* b = reinterpret_cast<const H*>(ep.bias);
#pragma unroll
  for (int e = 0; e < 4; ++e) bias[e] = b && c + e < N ? to_f<H>(b[c + e]) : 0.0f;
}
// residual of four columns of a row (zeros where there is none)
__device__ __forceinline__ void cl_residual(const Epilogue& ep, int N, int row, int c, bool pieces, float* res) {
  res[0] = res[1] = res[2] = res[3] = 0.0f;
  if (!ep.residual || ep.glu) return;
  const float* r = ep.residual + (size_t)row * N + c;
  if (pieces) {
    if (c < N) {
      const float4 t = *reinterpret_cast<const float4*>(r);
      res[0] = t.x; res[1] = t.y; res[2] = t.z; res[3] = t.w;
    }
    return;
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (c + e < N) res[e] = r[e];
}
// the finished sums v of columns c .. c + 3 of a row: bias first, then gate product, or activation / gate / residual
template <typename H>
__device__ __forceinline__ void cl_finish4(const Epilogue& ep, int N, int row, int c, bool pieces, float* v, const float* bias, const float* res) {
#pragma unroll
  for (int e = 0; e < 4; ++e) v[e] += bias[e];
  if (ep.glu) {
    const int No = N / 2;
    if (pieces && !ep.gate && !ep.residual && !ep.y32) {
      if (c >= N) return;
      const float y0 = ep_glu(v[0], v[1], ep), y1 = ep_glu(v[2], v[3], ep);
      H* dst = reinterpret_cast<H*>(ep.y) + (size_t)row * No + (c >> 1);
      if constexpr (sizeof(H) == 4) *reinterpret_cast<float2*>(dst) = make_float2(y0, y1);
      else *reinterpret_cast<uint32_t*>(dst) = Pair16<H>::put(y0, y1);
      return;
    }
    if (c + 1 < N) ep_store<H>(ep, (size_t)row * No + (c >> 1), ep_glu(v[0], v[1], ep));
    if (c + 3 < N) ep_store<H>(ep, (size_t)row * No + (c >> 1) + 1, ep_glu(v[2], v[3], ep));
    return;
  }
  if (ep.act != TSB200_ACT_NONE) {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = ep_act(v[e], ep.act);
  }
  const size_t o = (size_t)row * N + c;
  if (pieces) {
    if (c >= N) return;
    if (ep.gate) {
      struct __align__(4 * sizeof(H)) Four { H e[4]; };
      const Four g = *reinterpret_cast<const Four*>(reinterpret_cast<const H*>(ep.gate) + o);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] *= to_f<H>(g.e[e]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] += res[e];
    if (ep.y32) cl_store4<float>(ep.y32 + o, v);
    else cl_store4<H>(reinterpret_cast<H*>(ep.y) + o, v);
    return;
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (c + e >= N) continue;
    if (ep.gate) v[e] *= to_f<H>(reinterpret_cast<const H*>(ep.gate)[o + e]);
    v[e] += res[e];
    if (ep.y32) ep.y32[o + e] = v[e];
    else reinterpret_cast<H*>(ep.y)[o + e] = from_f<H>(v[e]);
  }
}

// ---- rows of one thread ----------------------------------------------------------------------------------------------------
// What finishes the four columns of a thread is decided once, and each kind has a loop of its own: with all of cl_finish4's choices inside the
// loop a row took 1300 clocks of mostly instruction fetches (64 rows of 4096 -> 22016, gated: 10200 clocks of a launch's 62000, now 3200).
// What a row reads is on its way one row ahead, the first one's while the products run.
enum ClKind { kClAny = 0, kClScalar = 1, kClResidual = 2, kClGateResidual = 3, kClRows = 4, kClGlu = 5, kClRope = 6 };
inline int cl_kind(const Epilogue& ep, int N, size_t elem) {
  if (!cl_whole_pieces(ep, N, elem)) return kClScalar;
  if (ep.glu) return !ep.gate && !ep.residual && !ep.y32 ? kClGlu : kClAny;
  if (!ep.gate && !ep.residual && !ep.y32) return kClRows;
  if (ep.act == TSB200_ACT_NONE && ep.residual && ep.y32) return ep.gate ? kClGateResidual : kClResidual;
  return kClAny;
}
template <typename H>
struct ClAhead {
  struct __align__(4 * sizeof(H)) Four { H e[4]; };
  float bias[4];
  float4 res;
  Four gate;
  int pos;
  float2 cs0, cs1;
  int sec, head, e0;   // rotation: q, k or v, its head and element
  __device__ __forceinline__ void row(const Epilogue& ep, int kind, int N, int c, int r, const RopeFuse& rf) {
    if (kind == kClResidual || kind == kClGateResidual) {
      if (c >= N) return;
      const size_t o = (size_t)r * N + c;
      res = *reinterpret_cast<const float4*>(ep.residual + o);
      if (kind == kClGateResidual) gate = *reinterpret_cast<const Four*>(reinterpret_cast<const H*>(ep.gate) + o);
    } else if (kind == kClRope) {
      pos = state_len(rf.state, r, rf.T0);
      if (rf.use_rope && sec < 2 && pos < rf.Tmax) {
        cs0 = rf.tab[(int64_t)pos * (rf.hd / 2) + e0 / 2];
        cs1 = rf.tab[(int64_t)pos * (rf.hd / 2) + e0 / 2 + 1];
      }
    }
  }
  // before the wait: weights, and the step state, which was there before the step's first kernel ran (embed_kernel)
  __device__ __forceinline__ void start(const Epilogue& ep, int kind, int N, int c, int row0, int M, const RopeFuse& rf) {
    cl_bias<H>(ep, N, c, bias);
    if (kind == kClRope) {
      sec = c < rf.Hd ? 0 : (c < rf.Hd + rf.KVd ? 1 : 2);
      const int cc = c - (sec == 0 ? 0 : (sec == 1 ? rf.Hd : rf.Hd + rf.KVd));
      head = cc / rf.hd;
      e0 = cc - head * rf.hd;
    }
    if (kind == kClRope && row0 < M) row(ep, kind, N, c, row0, rf);
  }
  // what the launch in front may have written
  __device__ __forceinline__ void first(const Epilogue& ep, int kind, int N, int c, int row0, int M, const RopeFuse& rf) {
    if (kind != kClRope && row0 < M) row(ep, kind, N, c, row0, rf);
  }
};
template <typename H, int ACT, typename Sum>
__device__ __forceinline__ void cl_rows_as(const Epilogue& ep, int N, int c, int row, int M, int step, const float* from, int skip, const float* bias, Sum& sum4) {
  H* y = reinterpret_cast<H*>(ep.y) + (size_t)row * N + c;
#pragma unroll 1
  for (; row < M; row += step, from += skip, y += (size_t)step * N) {
    float v[4];
    sum4(from, v);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = ep_act(v[e] + bias[e], ACT);
    cl_store4<H>(y, v);
  }
}
template <typename H, int ACT, typename Sum>
__device__ __forceinline__ void cl_glu_as(const Epilogue& ep, int N, int c, int row, int M, int step, const float* from, int skip, const float* bias, Sum& sum4) {
  const int No = N >> 1;
  H* y = reinterpret_cast<H*>(ep.y) + (size_t)row * No + (c >> 1);
  Epilogue act = ep;
  act.act = ACT;
#pragma unroll 1
  for (; row < M; row += step, from += skip, y += (size_t)step * No) {
    float v[4];
    sum4(from, v);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] += bias[e];
    const float y0 = ep_glu(v[0], v[1], act), y1 = ep_glu(v[2], v[3], act);
    if constexpr (sizeof(H) == 4) *reinterpret_cast<float2*>(y) = make_float2(y0, y1);
    else *reinterpret_cast<uint32_t*>(y) = Pair16<H>::put(y0, y1);
  }
}
// columns c .. c + 3 of rows row, row + step, ...: sum4(from, v) gives a row's finished sums, `skip` floats lie between a thread's rows
template <typename H, typename Sum>
__device__ __forceinline__ void cl_finish_rows(const Epilogue& ep, int kind, int N, int c, int row, int M, int step, const float* from, int skip, ClAhead<H>& f,
                                               const RopeFuse& rf, Sum sum4) {
  if (c >= N) return;
  if (kind == kClResidual) {
    float* y = ep.y32 + (size_t)row * N + c;
#pragma unroll 1
    for (; row < M; row += step, from += skip, y += (size_t)step * N) {
      const float4 r = f.res;
      if (row + step < M) f.row(ep, kClResidual, N, c, row + step, rf);
      float v[4];
      sum4(from, v);
      v[0] = v[0] + f.bias[0] + r.x; v[1] = v[1] + f.bias[1] + r.y; v[2] = v[2] + f.bias[2] + r.z; v[3] = v[3] + f.bias[3] + r.w;
      cl_store4<float>(y, v);
    }
  } else if (kind == kClRope) {
    // four columns = two rotation pairs of one head; the value is rounded first, as when a second kernel reads it back
#pragma unroll 1
    for (; row < M; row += step, from += skip) {
      const int pos = f.pos;
      const float2 cs0 = f.cs0, cs1 = f.cs1;
      if (row + step < M) f.row(ep, kClRope, N, c, row + step, rf);
      float t[4];
      sum4(from, t);
#pragma unroll
      for (int e = 0; e < 4; ++e) t[e] = to_f<H>(from_f<H>(t[e] + f.bias[e]));
      if (rf.use_rope && f.sec < 2 && pos < rf.Tmax) {
        const float a0 = t[0], b0 = t[1], a1 = t[2], b1 = t[3];
        t[0] = a0 * cs0.x - b0 * cs0.y; t[1] = b0 * cs0.x + a0 * cs0.y;
        t[2] = a1 * cs1.x - b1 * cs1.y; t[3] = b1 * cs1.x + a1 * cs1.y;
      }
      if (f.sec == 0) cl_store4<H>(reinterpret_cast<H*>(ep.y) + (size_t)row * N + c, t);
      else if (pos < rf.Tmax)   // capacity is checked on the host; never write past the cache
        cl_store4<H>(reinterpret_cast<H*>(f.sec == 1 ? rf.cK : rf.cV) + (((int64_t)row * (rf.KVd / rf.hd) + f.head) * rf.Tmax + pos) * rf.hd + f.e0, t);
    }
  } else if (kind == kClGlu) {
    switch (ep.act) {
      case TSB200_ACT_SILU:
      case TSB200_ACT_SWIGLU: return cl_glu_as<H, TSB200_ACT_SWIGLU>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
      case TSB200_ACT_CLAMP_GLU: return cl_glu_as<H, TSB200_ACT_CLAMP_GLU>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
      case TSB200_ACT_RELU: return cl_glu_as<H, TSB200_ACT_RELU>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
      case TSB200_ACT_LEAKYRELU: return cl_glu_as<H, TSB200_ACT_LEAKYRELU>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
      case TSB200_ACT_GELU: return cl_glu_as<H, TSB200_ACT_GELU>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
      case TSB200_ACT_SIGMOID: return cl_glu_as<H, TSB200_ACT_SIGMOID>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
      default: return cl_glu_as<H, TSB200_ACT_NONE>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
    }
  } else if (kind == kClRows) {
    switch (ep.act) {
      case TSB200_ACT_RELU: return cl_rows_as<H, TSB200_ACT_RELU>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
      case TSB200_ACT_SILU:
      case TSB200_ACT_SWIGLU: return cl_rows_as<H, TSB200_ACT_SILU>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
      case TSB200_ACT_LEAKYRELU: return cl_rows_as<H, TSB200_ACT_LEAKYRELU>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
      case TSB200_ACT_GELU: return cl_rows_as<H, TSB200_ACT_GELU>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
      case TSB200_ACT_SIGMOID: return cl_rows_as<H, TSB200_ACT_SIGMOID>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
      default: return cl_rows_as<H, TSB200_ACT_NONE>(ep, N, c, row, M, step, from, skip, f.bias, sum4);
    }
  } else if (kind == kClGateResidual) {
    float* y = ep.y32 + (size_t)row * N + c;
#pragma unroll 1
    for (; row < M; row += step, from += skip, y += (size_t)step * N) {
      const float4 r = f.res;
      const typename ClAhead<H>::Four gt = f.gate;
      if (row + step < M) f.row(ep, kClGateResidual, N, c, row + step, rf);
      float v[4];
      sum4(from, v);
      const float rr[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = __fmul_rn(v[e] + f.bias[e], to_f<H>(gt.e[e])) + rr[e];
      cl_store4<float>(y, v);
    }
  } else {
#pragma unroll 1
    for (; row < M; row += step, from += skip) {
      float v[4], res[4];
      sum4(from, v);
      cl_residual(ep, N, row, c, kind != kClScalar, res);
      cl_finish4<H>(ep, N, row, c, kind != kClScalar, v, f.bias, res);
    }
  }
}

}  // namespace tsb
