// Helpers shared by the step kernels that give a thread four cells (rfxb_fwdv.cu,
// rfxb_adjv.cu).
#pragma once
#include "rfxb_common.cuh"

namespace rfxb {

#define RFXB_VNST 3   // E plane stages: i, i+1 and one in flight
#define RFXB_VBARS 7  // mbarriers: three E stages, two H stages, two coefficient stages

__host__ __device__ constexpr int vup32(int n) { return (n + 31) / 32 * 32; }

template <int N>
struct IntC { static constexpr int v = N; };

template <int L>
struct Vec {
  float v[L];
  __device__ __forceinline__ float& operator[](int i) { return v[i]; }
  __device__ __forceinline__ const float& operator[](int i) const { return v[i]; }
};

template <int L>
__device__ __forceinline__ Vec<L> vzero() {
  Vec<L> r;
#pragma unroll
  for (int l = 0; l < L; ++l) r.v[l] = 0.f;
  return r;
}
// 16-byte (L = 4, aligned) or single loads and stores
template <int L>
__device__ __forceinline__ Vec<L> vld(const float* p) {
  Vec<L> r;
  if constexpr (L == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
  } else {
    r.v[0] = *p;
  }
  return r;
}
template <int L>
__device__ __forceinline__ void vst(float* p, const Vec<L>& r) {
  if constexpr (L == 4) *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
  else *p = r.v[0];
}

// Block barrier of every thread of the CTA (all roles) with an OR reduction.
template <int NT>
__device__ __forceinline__ bool bar_or(bool v) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.or.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)v), "n"(NT)
      : "memory");
  return r != 0;
}

// z slab of L columns from k on: which of them lie in a slab (bits 0 .. L-1; bit
// 8: the four are one 16-byte access of the psi row, whose padding layers take
// the columns beyond the slab -- their profile is zero, so zeros stay there)
// and the psi element of the first one relative to (low side, q 0) of its row.
// No four columns reach both slabs (plans with fewer than three cells between
// them take the generic kernels).
template <int L>
__device__ __forceinline__ unsigned zslab_of(int k, int ncp, int kb, int nz, int hi, int& off) {
  unsigned m = 0u;
#pragma unroll
  for (int l = 0; l < L; ++l)
    if (k + l < ncp || (k + l >= kb && k + l < nz)) m |= 1u << l;
  off = k < ncp ? k : hi + k - kb;
  if (L == 4 && m != 0u && (k < ncp || k >= kb) && (off & 3) == 0) m |= 256u;
  return m;
}
template <int L>
__device__ __forceinline__ Vec<L> zpsi_load(const float* p, unsigned m) {
  if (L == 4 && (m & 256u)) return vld<L>(p);
  Vec<L> r;
#pragma unroll
  for (int l = 0; l < L; ++l) r.v[l] = (m >> l) & 1u ? p[l] : 0.f;
  return r;
}
template <int L>
__device__ __forceinline__ void zpsi_store(float* p, unsigned m, const Vec<L>& r) {
  if (L == 4 && (m & 256u)) { vst<L>(p, r); return; }
#pragma unroll
  for (int l = 0; l < L; ++l)
    if ((m >> l) & 1u) p[l] = r.v[l];
}

// Whether a work item can be run: its instance exists and its tile and x
// range lie inside that instance's grid on the tiling of the lists.
template <int TY, int ZQ>
__device__ __forceinline__ bool work_item_valid(const RfxbWork& w, const RfxbInst* insts, int n_inst) {
  if (w.inst < 0 || w.inst >= n_inst) return false;
  const RfxbInst& I = insts[w.inst];
  return w.y0 >= 0 && w.y0 < I.ny && w.y0 % TY == 0 && w.z0 >= 0 && w.z0 < I.nz && w.z0 % (4 * ZQ) == 0 &&
         w.xa >= 0 && w.xa < w.xb && w.xb <= I.nx;
}

}  // namespace rfxb
