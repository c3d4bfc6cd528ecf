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
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
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
// the finished sums v of columns c .. c + 3 of a row: bias first, then rotation and cache append, gate product, or activation / gate / residual
template <typename H>
__device__ __forceinline__ void cl_finish4(const Epilogue& ep, int N, int row, int c, bool pieces, float* v, const float* bias, const float* res, int rope_on, const RopeFuse& rf) {
#pragma unroll
  for (int e = 0; e < 4; ++e) v[e] += bias[e];
  if (rope_on) {
    // four columns = two rotation pairs of one head; the value is rounded first, as when a second kernel reads it back
    if (c + 3 >= N) return;
    const int pos = state_len(rf.state, row, rf.T0);
    const int sec = c < rf.Hd ? 0 : (c < rf.Hd + rf.KVd ? 1 : 2);
    const int cc = c - (sec == 0 ? 0 : (sec == 1 ? rf.Hd : rf.Hd + rf.KVd));
    const int head = cc / rf.hd, e0 = cc % rf.hd;
    float t[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) t[e] = to_f<H>(from_f<H>(v[e]));
    if (rf.use_rope && sec < 2 && pos < rf.Tmax) {
      const float2 cs0 = rf.tab[(int64_t)pos * (rf.hd / 2) + e0 / 2], cs1 = rf.tab[(int64_t)pos * (rf.hd / 2) + e0 / 2 + 1];
      const float a0 = t[0], b0 = t[1], a1 = t[2], b1 = t[3];
      t[0] = a0 * cs0.x - b0 * cs0.y; t[1] = b0 * cs0.x + a0 * cs0.y;
      t[2] = a1 * cs1.x - b1 * cs1.y; t[3] = b1 * cs1.x + a1 * cs1.y;
    }
    if (sec == 0) cl_store4<H>(reinterpret_cast<H*>(ep.y) + (size_t)row * N + c, t);
    else if (pos < rf.Tmax)   // capacity is checked on the host; never write past the cache
      cl_store4<H>(reinterpret_cast<H*>(sec == 1 ? rf.cK : rf.cV) + (((int64_t)row * (rf.KVd / rf.hd) + head) * rf.Tmax + pos) * rf.hd + e0, t);
    return;
  }
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

}  // namespace tsb
