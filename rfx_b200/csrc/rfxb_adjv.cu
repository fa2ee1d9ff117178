// Fused reverse step of the adjoint, four cells per thread: the tiling, x
// march, staged planes and halo recomputation of the forward step kernel
// (rfxb_fwdv.cu) on the transpose of one forward step (rfxb_adj.cu derives it).
//
// Both halves are written as differences of one flux per cell and direction.
// With q = cb aEm and r_E the transposed psi-E relation of the cell,
//   phase A: aH1_x = aH_x + (Gzy - Gzy|z+1) - (Gyz - Gyz|y+1), and cyclic,
//     Gzy = ze q_y + r_z1, Gyz = ye q_z - r_y1, Gxz = xe q_z + r_x1,
//     Gzx = ze q_x - r_z0, Gyx = ye q_x + r_y0, Gxy = xe q_y - r_x0;
// with p = ch aH1 and r_H the transposed psi-H relation,
//   phase B: aE_x = ca aEm_x + (Kzy - Kzy|z-1) - (Kyz - Kyz|y-1), and cyclic,
//     Kzy = zh p_y - r_z1, Kyz = yh p_z + r_y1, Kxz = xh p_z - r_x1,
//     Kzx = zh p_x + r_z0, Kyx = yh p_x - r_y0, Kxy = xh p_y + r_x0.
// A relation is therefore evaluated once by the cell that owns it (and writes
// its psi) and travels inside the flux: to the next lane in z, to the next
// plane in registers, and in y through shared memory (K) or, for the one row
// above, by evaluating that row's G again, so a plane needs one barrier.
// A flux that travels, s q + r, is rounded once, and the difference to it has its
// own product fused, fma(s, q, -other), with r added by itself: without CPML these
// are the operations of the kernel with one cell per thread (rfxb_adj_fused.cu),
// in the slabs as many roundings.  The differences of phase B that need no other
// row are formed before the barrier, so that nothing but p crosses it.  With every
// product rounded by itself the adjoint fields were 1.04 to 1.17 times as far from
// a float64 march, at 97x83x109 46.5 against 49.4 us a step now, 221x141x69 96.6 /
// 97.5, a 131^3 closed box 41.5 / 42.1, the sweep below 1417 / 1411.
// The probe cotangent of y_{n-1}, the source adjoint and the PEC / edge mask
// follow; adjoint fields and psi are ping-ponged like the forward state.  The
// eps_r gradient over the recorded region is accumulated in phase A from the
// forward history.  Products and sums are rounding intrinsics.
//
// What bounds it: instructions and, in the slabs, instruction fetch (the CPML
// path is 98 KB of code; the rare work -- probes, sources, gradient, failure --
// therefore sits behind single sites over indexed copies: the step of 20 grids
// of 64-160 cells a side 1477 -> 1380 us), and registers: E and cb of the own
// cells are read from their stage where they are used (221x141x69 103 -> 98 us a
// step with them held in registers and 212 instead of 96 bytes spilled).  One cell per
// thread with the relations of the neighbours evaluated again in place -> here,
// reverse steps alone: that sweep 1629 -> 1411 us (three launches against one),
// 221x141x69 with CPML 10 131 -> 97.5, 97x83x109 with CPML 8 58.5 -> 49.4.
#include "rfxb_common.cuh"
#include "rfxb_vec.cuh"

namespace rfxb {

template <int TY, int ZQ>
struct AVDims {
  static constexpr int TZ = 4 * ZQ;
  static constexpr int MAIN = TY * ZQ;
  static constexpr int NT = MAIN + 32;
  static constexpr int EW = TZ + 8;
  static constexpr int CE = (TY + 2) * EW;
  static constexpr int CB = vup32(3 * CE);   // cb follows the three components on a 128-byte boundary
  static constexpr int CH = (TY + 1) * TZ;   // component stride of an adjoint-H stage
  static constexpr int CC = TY * TZ;
  static_assert(MAIN % 32 == 0 && ZQ + TY <= 32, "the halo warp holds the row and the column");
};

// Slots of the prefetched psi of a thread's cells (four floats each), by the
// slabs the cells lie in:
//   z slab: z E q0, q1, z H q0, q1, ce; y E q0, q1 (in a y slab too)
//   y slab: y E q0, q1, y H q0, q1, ce; y E q0, q1 of the next row
//   neither: x E q0, q1 of the next plane, x H q0, q1, ce of the next plane; y E
//            q0, q1 of the next row
// What does not fit is read from global memory where it is used.
#define RFXB_ASLOTS 7

template <int TY, int ZQ, bool CP>
struct __align__(128) AVSmem {
  using D = AVDims<TY, ZQ>;
  float e[RFXB_VNST][D::CB + vup32(D::CE)];   // masked adjoint E, then cb
  float ho[2][3 * D::CH];             // adjoint H, rows y0-1 .. y0+TY-1
  float ca[2][D::CC];                 // ca of the tile
  float k[2][2][TY][D::TZ];           // Kyx, Kyz of plane i in slot i & 1: rows y0-1 .. y0+TY-2
  float kc[2][2][TY];                 // Kzx, Kzy of column z0-1
  float zt[2][D::TZ + 4];             // ze, zh of columns z0 .. z0+TZ
  float zp[3][D::TZ + 4];             // z profile of the same columns
  float ps[CP ? RFXB_ASLOTS : 1][CP ? D::MAIN : 1][4];
  RfxbInst P;
  AdjInst A;
  unsigned long long mbar[RFXB_VBARS];
};

// One transposed relation: nu = psi + SGN s t, psi' = b nu (written when
// WRITE), r = c nu + SGN s km t.
template <int SGN>
__device__ __forceinline__ float rel_nu(float psi, float s, float t) {
  return __fmaf_rn(SGN > 0 ? s : -s, t, psi);
}
template <int SGN>
__device__ __forceinline__ float rel_r(float nu, float s, float t, float c, float km) {
  return __fmaf_rn(SGN > 0 ? s : -s, __fmul_rn(km, t), __fmul_rn(c, nu));
}
// r of a relation of an x or y slab, from its old psi p
template <int L, int SGN, bool WRITE>
__device__ __forceinline__ Vec<L> rel_xy(Vec<L> p, float* out, const float4& c, const Vec<L>& s, const Vec<L>& t,
                                         bool write = true) {
  Vec<L> r;
#pragma unroll
  for (int l = 0; l < L; ++l) {
    const float nu = rel_nu<SGN>(p[l], s[l], t[l]);
    r[l] = rel_r<SGN>(nu, s[l], t[l], c.y, c.z);
    p[l] = __fmul_rn(c.x, nu);
  }
  if (WRITE && write) vst<L>(out, p);
  return r;
}
// the same for a z slab (zero off it): profile per column, psi at the columns' layers
template <int L, int SGN, bool WRITE>
__device__ __forceinline__ Vec<L> rel_z(Vec<L> p, float* out, unsigned m, const Vec<L>& b, const Vec<L>& c,
                                        const Vec<L>& km, const Vec<L>& s, const Vec<L>& t) {
  Vec<L> r;
#pragma unroll
  for (int l = 0; l < L; ++l) {
    const float nu = rel_nu<SGN>(p[l], s[l], t[l]);
    r[l] = (m >> l) & 1u ? rel_r<SGN>(nu, s[l], t[l], c[l], km[l]) : 0.f;
    p[l] = __fmul_rn(b[l], nu);
  }
  if (WRITE) zpsi_store<L>(out, m, p);
  return r;
}

template <int L>
__device__ __forceinline__ Vec<L> vsplat(float a) {
  Vec<L> r;
#pragma unroll
  for (int l = 0; l < L; ++l) r[l] = a;
  return r;
}
template <int L>
__device__ __forceinline__ Vec<L> vmul(const Vec<L>& a, const Vec<L>& b) {
  Vec<L> r;
#pragma unroll
  for (int l = 0; l < L; ++l) r[l] = __fmul_rn(a[l], b[l]);
  return r;
}
// s q + SGN r, rounded once
template <int SGN, int L>
__device__ __forceinline__ Vec<L> vfma(const Vec<L>& s, const Vec<L>& q, const Vec<L>& r) {
  Vec<L> f;
#pragma unroll
  for (int l = 0; l < L; ++l) f[l] = __fmaf_rn(s[l], q[l], SGN > 0 ? r[l] : -r[l]);
  return f;
}
// a flux: with R, r is zero off the slabs; without, no cell has one
template <bool R, int SGN, int L>
__device__ __forceinline__ Vec<L> vflux(const Vec<L>& s, const Vec<L>& q, const Vec<L>& r) {
  return R ? vfma<SGN>(s, q, r) : vmul(s, q);
}
// f += SGN r
template <int SGN, int L>
__device__ __forceinline__ void vacc(Vec<L>& f, const Vec<L>& r) {
#pragma unroll
  for (int l = 0; l < L; ++l) f[l] = SGN > 0 ? __fadd_rn(f[l], r[l]) : __fsub_rn(f[l], r[l]);
}
// a + (b - c), b and c two differences of fluxes
__device__ __forceinline__ float curl_t(float a, float b, float c) { return __fadd_rn(a, __fsub_rn(b, c)); }

// One work item (see fwdv_item): returns false when a bounded wait ran out.
template <int TY, int ZQ, bool CP>
__device__ __forceinline__ bool adjv_item(AVSmem<TY, ZQ, CP>& S, const RfxbInst* __restrict__ insts,
                                          const AdjInst* __restrict__ adjs, const RfxbWork w,
                                          const CUtensorMap* __restrict__ maps, int map0, int n, int par, int apar,
                                          StepPhases& ph, const StepFault& fault, bool first_item) {
  using D = AVDims<TY, ZQ>;
  constexpr int EW = D::EW, CE = D::CE, CB = D::CB, NT = D::NT, TZ = D::TZ, ZPS = TZ + 4, SS = 4 * D::MAIN;
  const int tid = threadIdx.x;
  const int y0 = w.y0, z0 = w.z0, xa = w.xa, xb = w.xb;
  // The boxes of this item.  Plane p: adjoint E and cb in stage (p - xa + 1) % 3,
  // adjoint H in stage (p - xa + 1) % 2, ca in stage (p - xa) % 2; barriers 0-2,
  // 3-4, 5-6.
  const bool producer = tid == NT - 1;
  const CUtensorMap* tm = maps + (size_t)w.inst * RFXB_NMAPS + map0;   // [0|1] aE, [2] cb, [3|4] aH, [5] ca
  const uint32_t ph0 = ph.stage;
  auto sE = [&](int p) { return (p - xa + 1) % RFXB_VNST; };
  auto sH = [&](int p) { return (p - xa + 1) & 1; };
  auto sC = [&](int p) { return (p - xa) & 1; };
  auto issue_e = [&](int p) {
    const uint32_t mb = smem_u32(&S.mbar[sE(p)]);
    mbar_expect_tx(mb, 4u * 4 * CE);
    tma_load_4d(smem_u32(&S.e[sE(p)][0]), tm + apar, z0 - 4, y0, p + 1, 0, mb);
    tma_load_4d(smem_u32(&S.e[sE(p)][CB]), tm + 2, z0 - 4, y0, p + 1, 1, mb);
  };
  auto issue_h = [&](int p) {
    const uint32_t mb = smem_u32(&S.mbar[3 + sH(p)]);
    mbar_expect_tx(mb, 4u * 3 * D::CH);
    tma_load_4d(smem_u32(&S.ho[sH(p)][0]), tm + 3 + apar, z0, y0, p + 1, 3, mb);
  };
  auto issue_c = [&](int p) {
    const uint32_t mb = smem_u32(&S.mbar[5 + sC(p)]);
    mbar_expect_tx(mb, 4u * D::CC);
    tma_load_4d(smem_u32(&S.ca[sC(p)][0]), tm + 5, z0, y0 + 1, p + 1, 0, mb);
  };
  int last_e = min(xa + 1, xb), last_h = xa, last_c = min(xa + 1, xb - 1);   // planes issued so far
  if (producer) {
    const bool skip = first_item && (int)blockIdx.x == fault.cta;
    issue_e(xa - 1);
    if (!skip) issue_e(xa);
    issue_h(xa - 1);
    issue_h(xa);
    issue_c(xa);
    if (xa + 1 <= xb) issue_e(xa + 1);
    if (xa + 1 < xb) issue_c(xa + 1);
  }
  load_inst(S.P, insts + w.inst, tid, NT);
  {
    const int nw = sizeof(AdjInst) / 4;
    const int* s = reinterpret_cast<const int*>(adjs + w.inst);
    int* d = reinterpret_cast<int*>(&S.A);
#pragma unroll 1
    for (int t = tid; t < nw; t += NT) d[t] = __ldg(s + t);
  }
  __syncthreads();
  const RfxbInst& P = S.P;
  const AdjInst& AD = S.A;
  const int wlim = fault.wait_limit;
  const int nx = P.nx, ny = P.ny, nz = P.nz, zs = P.zs, ncp = P.ncp, n4 = P.ncp4;
  const long long ps = P.ps, cs = P.cs;
  const float* Fi = AD.aF[apar][0];
  float* Fo = AD.aF[apar ^ 1][0];
  const unsigned ax_ = CP && ncp > 0 ? P.cpml_axes : 0u;
  const bool cpx = ax_ & 1u, cpy = ax_ & 2u, cpz = ax_ & 4u;
  const int jb = ny - ncp, kb = nz - ncp;
  const int qx = ncp * ny * zs, qy = nx * ncp * zs, qz = nx * ny * n4;

#pragma unroll 1
  for (int t = tid; t < TZ + 1; t += NT) {
    const int k = z0 + t;
    S.zt[0][t] = k <= nz ? __ldg(P.ze + k) : 0.f;
    S.zt[1][t] = k < nz ? __ldg(P.zh + k) : 0.f;
    if (CP) {
      float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
      if (cpz && k < ncp) c = __ldg(P.cpt + 4 * ncp + k);
      else if (cpz && k >= kb && k < nz) c = __ldg(P.cpt + 5 * ncp + (k - kb));
      S.zp[0][t] = c.x;
      S.zp[1][t] = c.y;
      S.zp[2][t] = c.z;
    }
  }

  auto wait = [&](int b) -> bool {
    const bool ok = mbar_wait_bounded(smem_u32(&S.mbar[b]), (ph.stage >> b) & 1u, wlim);
    ph.stage ^= 1u << b;
    return ok;
  };
  // a wait ran out: flag the launch and wait (bounded) for the last box of
  // every stage
  auto bail = [&]() {
    if (producer) {
      atomicOr(P.status, 1);
      auto drain = [&](int b, int fill) { mbar_wait_bounded(smem_u32(&S.mbar[b]), ((ph0 >> b) ^ (uint32_t)fill) & 1u, wlim); };
#pragma unroll 1
      for (int p = max(xa - 1, last_e - 2); p <= last_e; ++p) drain(sE(p), (p - xa + 1) / RFXB_VNST);
#pragma unroll 1
      for (int p = max(xa - 1, last_h - 1); p <= last_h; ++p) drain(3 + sH(p), (p - xa + 1) >> 1);
#pragma unroll 1
      for (int p = max(xa, last_c - 1); p <= last_c; ++p) drain(5 + sC(p), (p - xa) >> 1);
    }
  };
  const bool is_main = tid < D::MAIN;
  const float ch0 = P.ch0;
  const float* ch_arr = P.ch;
  const float* xe_tab = P.xe;
  const float* xh_tab = P.xh;
  const float* psEx = AD.aPsiE[par][0];
  const float* psEy = AD.aPsiE[par][1];
  const float* psEz = AD.aPsiE[par][2];
  // y slab of row j: whether, its profile and psi element of (q 0, plane 0, column k)
  auto yslab = [&](int j, int k, float4& c, int& oy) -> bool {
    if (!CP || !cpy || j >= ny || (j >= ncp && j < jb)) return false;
    const int sd = j < ncp ? 0 : 1, s = sd ? j - jb : j;
    c = __ldg(P.cpt + (2 + sd) * ncp + s);
    oy = 2 * sd * qy + s * zs + k;
    return true;
  };
  auto xslab = [&](int p, float4& c, int& base) -> bool {
    if (!CP || !cpx || p < 0 || (p >= ncp && p < nx - ncp) || p >= nx) return false;
    const int sd = p < ncp ? 0 : 1, s = sd ? p - (nx - ncp) : p;
    c = __ldg(P.cpt + sd * ncp + s);
    base = 2 * sd * qx + s * ny * zs;
    return true;
  };
  auto in_xslab = [&](int p) { return CP && cpx && p >= 0 && p < nx && (p < ncp || p >= nx - ncp); };
  auto xbase_of = [&](int p) {
    const int sd = p < ncp ? 0 : 1, s = sd ? p - (nx - ncp) : p;
    return 2 * sd * qx + s * ny * zs;
  };
  // planes xa-1 and xa have landed; after a wait that ran out all threads leave
  // the loops at the same barrier
  bool bad_end;
  {
    const bool ok0 = wait(0), ok1 = wait(1), ok2 = wait(3);
    bad_end = bar_or<NT>(!(ok0 && ok1 && ok2));
  }

  // Fluxes of L columns with fields ex ey ez and coefficient cb; in a slab, ld(q)
  // gives the old psi and ld(2) the cells' ce.  A flux s q + r is rounded once; in a
  // difference of two the own product is not rounded before it, fma(s, q, -other),
  // and r goes to H by itself.
  // G of the y direction: Gyx = ye q_x + r_y0, Gyz = ye q_z - r_y1.
  auto gy_flux = [&](auto LL, const Vec<decltype(LL)::v>& ex, const Vec<decltype(LL)::v>& ez,
                     const Vec<decltype(LL)::v>& cb, float ye, bool on, const float4& c, auto&& ld,
                     Vec<decltype(LL)::v>& gyx, Vec<decltype(LL)::v>& gyz) {
    constexpr int L = decltype(LL)::v;
    const Vec<L> s = vsplat<L>(ye);
    Vec<L> r0 = vzero<L>(), r1 = vzero<L>();
    if (CP && on) {
      const Vec<L> ce = ld(2);
      r0 = rel_xy<L, +1, false>(ld(0), nullptr, c, ce, ex);
      r1 = rel_xy<L, -1, false>(ld(1), nullptr, c, ce, ez);
    }
    gyx = vflux<CP, +1>(s, vmul(cb, ex), r0);
    gyz = vflux<CP, -1>(s, vmul(cb, ez), r1);
  };
  // Gyx - nyx and Gyz - nyz, nyx and nyz the fluxes of the row above: the products
  // in dyx and dyz, the relations added to hz and hx
  auto gy_diff = [&](auto LL, auto WR, const Vec<decltype(LL)::v>& ex, const Vec<decltype(LL)::v>& ez,
                     const Vec<decltype(LL)::v>& cb, float ye, bool on, const float4& c, int iy, auto&& ld,
                     const Vec<decltype(LL)::v>& nyx, const Vec<decltype(LL)::v>& nyz, Vec<decltype(LL)::v>& dyx,
                     Vec<decltype(LL)::v>& dyz, Vec<decltype(LL)::v>& hx, Vec<decltype(LL)::v>& hz) {
    constexpr int L = decltype(LL)::v;
    constexpr bool W = decltype(WR)::v != 0;
    const Vec<L> s = vsplat<L>(ye);
    dyx = vfma<-1>(s, vmul(cb, ex), nyx);
    dyz = vfma<-1>(s, vmul(cb, ez), nyz);
    if (CP && on) {
      const Vec<L> ce = ld(2);
      float* out = AD.aPsiE[par ^ 1][1];
      vacc<+1>(hz, rel_xy<L, +1, W>(ld(0), out + iy, c, ce, ex));
      vacc<+1>(hx, rel_xy<L, -1, W>(ld(1), out + iy + qy, c, ce, ez));
    }
  };
  // G of the z direction, Gzx = ze q_x - r_z0, Gzy = ze q_y + r_z1; with H the relations are added to hx and hy
  auto gz_flux = [&](auto LL, auto WR, auto HH, const Vec<decltype(LL)::v>& ex, const Vec<decltype(LL)::v>& ey,
                     const Vec<decltype(LL)::v>& cb, const Vec<decltype(LL)::v>& ze, unsigned on, const float* zp, int iz,
                     auto&& ld, Vec<decltype(LL)::v>& gzx, Vec<decltype(LL)::v>& gzy, Vec<decltype(LL)::v>& hx,
                     Vec<decltype(LL)::v>& hy) {
    constexpr int L = decltype(LL)::v;
    constexpr bool W = decltype(WR)::v != 0, H = decltype(HH)::v != 0;
    Vec<L> r0 = vzero<L>(), r1 = vzero<L>();
    if (CP && on) {
      const Vec<L> ce = ld(2);
      const Vec<L> b = vld<L>(zp), c = vld<L>(zp + ZPS), km = vld<L>(zp + 2 * ZPS);
      float* out = AD.aPsiE[par ^ 1][2];
      r0 = rel_z<L, -1, W>(ld(0), out + iz, on, b, c, km, ce, ex);
      r1 = rel_z<L, +1, W>(ld(1), out + iz + qz, on, b, c, km, ce, ey);
      if (H) {
        vacc<+1>(hy, r0);
        vacc<+1>(hx, r1);
      }
    }
    gzx = vflux<CP, -1>(ze, vmul(cb, ex), r0);
    gzy = vflux<CP, +1>(ze, vmul(cb, ey), r1);
  };
  // the products of Gzx - Gzx|z+1 and Gzy - Gzy|z+1 of four columns, nx_ and ny_ the fluxes of the column after them
  auto gz_diff = [&](const Vec<4>& ex, const Vec<4>& ey, const Vec<4>& cb, const Vec<4>& ze, const Vec<4>& gzx,
                     const Vec<4>& gzy, float nx_, float ny_, Vec<4>& dzx, Vec<4>& dzy) {
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      dzx[l] = __fmaf_rn(ze[l], __fmul_rn(cb[l], ex[l]), -(l < 3 ? gzx[l < 3 ? l + 1 : l] : nx_));
      dzy[l] = __fmaf_rn(ze[l], __fmul_rn(cb[l], ey[l]), -(l < 3 ? gzy[l < 3 ? l + 1 : l] : ny_));
    }
  };
  // G of the x direction, Gxy = xe q_y - r_x0, Gxz = xe q_z + r_x1, and its relations (zero off the slabs)
  auto gx_flux = [&](auto LL, const Vec<decltype(LL)::v>& ey, const Vec<decltype(LL)::v>& ez,
                     const Vec<decltype(LL)::v>& cb, float xe, bool on, bool write, const float4& c, int ix, auto&& ld,
                     Vec<decltype(LL)::v>& gxy, Vec<decltype(LL)::v>& gxz, Vec<decltype(LL)::v>& r0,
                     Vec<decltype(LL)::v>& r1) {
    constexpr int L = decltype(LL)::v;
    const Vec<L> s = vsplat<L>(xe);
    r0 = r1 = vzero<L>();
    if (CP && on) {
      const Vec<L> ce = ld(2);
      float* out = AD.aPsiE[par ^ 1][0];
      r0 = rel_xy<L, -1, L == 4>(ld(0), out + ix, c, ce, ey, write);
      r1 = rel_xy<L, +1, L == 4>(ld(1), out + ix + qx, c, ce, ez, write);
    }
    gxy = vflux<CP, -1>(s, vmul(cb, ey), r0);
    gxz = vflux<CP, +1>(s, vmul(cb, ez), r1);
  };
  // loaders from global memory: psi at p (q stride qs), ce at cell e
  auto glob = [&](auto LL, const float* p, int qs, long long e) {
    constexpr int L = decltype(LL)::v;
    const float* ce = P.ce + e;
    return [p, qs, ce](int q) { return q == 2 ? vld<L>(ce) : vld<L>(p + q * qs); };
  };
  auto globz = [&](auto LL, const float* p, int qs, long long e, unsigned m) {
    constexpr int L = decltype(LL)::v;
    const float* ce = P.ce + e;
    return [p, qs, ce, m](int q) { return q == 2 ? vld<L>(ce) : zpsi_load<L>(p + q * qs, m); };
  };
  using L4 = IntC<4>;
  using L1 = IntC<1>;
  using NoW = IntC<0>;
  using Wr = IntC<1>;
  auto ch_at = [&](long long e) {
    Vec<4> c;
    if (ch_arr) c = vld<4>(ch_arr + e);
    else {
#pragma unroll
      for (int l = 0; l < 4; ++l) c[l] = ch0;
    }
    return c;
  };
  // Gzx, Gzy of column z0 + TZ (the one after the tile) at a row's position
  auto gz_after = [&](const float* St, int o, int irow, long long e, float& gx, float& gy) {
    const int k = z0 + TZ;
    if (k >= nz) { gx = 0.f; gy = 0.f; return; }
    Vec<1> ex = vld<1>(St + o), ey = vld<1>(St + o + CE), cb = vld<1>(St + o + CB), ze, a, b;
    ze[0] = S.zt[0][TZ];
    int off = 0;
    const unsigned m = cpz ? zslab_of<1>(k, ncp, kb, nz, 2 * qz, off) : 0u;
    gz_flux(L1{}, NoW{}, NoW{}, ex, ey, cb, ze, m, &S.zp[0][TZ], irow + off, glob(L1{}, psEz + irow + off, qz, e), a, b, a, b);
    gx = a[0];
    gy = b[0];
  };
  // H-probe cotangent of sample n at a cell
  auto h_cot = [&](unsigned m, bool tail, int i, int j, int k, auto&& add) {
    if (!P.g) return;
    int q = 31;
#pragma unroll 1
    while (true) {
      if (m) { q = __ffs(m) - 1; m &= m - 1; }
      else q = max(q + 1, 32);
      if (q >= (tail ? P.nprb : 32)) break;
      const int4 c = __ldg(P.prb + q);
      if (c.x == i && c.y == j && c.z >= k && c.z < k + 4 && (c.w & 7) >= 3)
        add(c.z - k, (c.w & 7) - 3, __ldg(P.g + (long long)n * P.g_ld + q));
    }
  };

  if (bad_end) {
  } else if (is_main) {
    const int r = tid / ZQ, zq = tid % ZQ;
    const int j = y0 + r, k = z0 + 4 * zq;
    const bool own = j < ny && k < nz;
    const int kv = min(4, nz - k);
    const int o = (r + 1) * EW + 4 * zq + 4;
    const long long col = P.off0 + (long long)j * zs + k;
    const int jk = j * zs + k;
    const float ye = own ? __ldg(P.ye + j) : 0.f, ye1 = own ? __ldg(P.ye + j + 1) : 0.f;
    const float yh = own ? __ldg(P.yh + j) : 0.f;
    float4 cy, cyn;
    int oy = 0, oyn = 0;
    const bool yon = own && yslab(j, k, cy, oy);
    const bool ynon = own && j + 1 < ny && yslab(j + 1, k, cyn, oyn);
    int zoff = 0;
    const unsigned zon = own && cpz ? zslab_of<4>(k, ncp, kb, nz, 2 * qz, zoff) : 0u;
    const int orow = j * n4, oz = orow + zoff;
    const float* zp = &S.zp[0][4 * zq];
    const bool last_q = zq == ZQ - 1, first_q = zq == 0;
    unsigned pmask = 0u, smask = 0u;
    if (own) {
#pragma unroll 1
      for (int q = 0; q < min(P.nprb, 32); ++q) {
        const int4 c = __ldg(P.prb + q);
        if (c.y == j && c.z >= k && c.z < k + 4) pmask |= 1u << q;
      }
#pragma unroll 1
      for (int q = 0; q < min(P.nsrc, 32); ++q) {
        const int4 c = __ldg(P.src + q);
        if (c.y == j && c.z >= k && c.z < k + 4) smask |= 1u << q;
      }
    }
    const bool ptail = P.nprb > 32, stail = P.nsrc > 32;
    const unsigned pec = P.pec_axes;
    const bool pec_j = (pec & 2u) && (j == 0 || j == ny - 1);
    const bool pec_k = (pec & 4u) && (k == 0 || k + 3 >= nz - 1);
    const bool in_gyz = P.grad && j >= P.hb[2] && j < P.hb[3] && k < P.hb[5] && k + 4 > P.hb[4] && P.hist &&
                        (n - P.hist_step0) >= 0 && (n - P.hist_step0) < P.hist_nsteps;
    const unsigned char* emask = P.emask;

    const int oh = (r + 1) * TZ + 4 * zq, oc = r * TZ + 4 * zq;   // this thread's place in an H / ca stage
    Vec<4> rx0 = vzero<4>(), rx1 = vzero<4>(), kxyp = vzero<4>(), kxzp = vzero<4>();   // x relations of phase A, x fluxes K
    // prefetch of plane p's psi (and ce) into this thread's slots
    float* const slot = &S.ps[0][CP ? tid : 0][0];
    auto sl = [&](int q) { return vld<4>(slot + q * SS); };
    auto get = [&](int q, const float* p) { cp_async16(slot + q * SS, p); };
    auto getz = [&](int q, const float* p) {
      if (zon & 256u) { get(q, p); return; }
#pragma unroll
      for (int l = 0; l < 4; ++l)
        if ((zon >> l) & 1u) cp_async4(slot + q * SS + l, p + l);
    };
    auto fetch = [&](int p) {
      const long long e = col + (long long)p * ps;
      const int iy = oy + p * ncp * zs;
      if (zon) {
        const int iz = oz + p * ny * n4;
        getz(0, psEz + iz);
        getz(1, psEz + iz + qz);
        getz(2, AD.aPsiH[par][2] + iz);
        getz(3, AD.aPsiH[par][2] + iz + qz);
        get(4, P.ce + e);
        if (yon) {
          get(5, psEy + iy);
          get(6, psEy + iy + qy);
        }
        return;
      }
      if (yon) {
        get(0, psEy + iy);
        get(1, psEy + iy + qy);
        get(2, AD.aPsiH[par][1] + iy);
        get(3, AD.aPsiH[par][1] + iy + qy);
        get(4, P.ce + e);
      } else {
        if (in_xslab(p + 1)) {
          const float* q = psEx + xbase_of(p + 1) + jk;
          get(0, q);
          get(1, q + qx);
          get(4, P.ce + e + ps);
        }
        if (in_xslab(p)) {
          const float* q = AD.aPsiH[par][0] + xbase_of(p) + jk;
          get(2, q);
          get(3, q + qx);
        }
      }
      if (ynon) {
        const int iyn = oyn + p * ncp * zs;
        get(5, psEy + iyn);
        get(6, psEy + iyn + qy);
      }
    };
    // fluxes of column k+4 from the next lane (the last one evaluates them)
    auto z_next = [&](const float* St, const Vec<4>& gzx, const Vec<4>& gzy, int i, float& nx_, float& ny_) {
      nx_ = __shfl_down_sync(0xffffffffu, gzx[0], 1, ZQ);
      ny_ = __shfl_down_sync(0xffffffffu, gzy[0], 1, ZQ);
      if (last_q && own) gz_after(St, o + 4, orow + i * ny * n4, col + 4 + (long long)i * ps, nx_, ny_);
    };

    // ---- prologue: K of the x direction on plane xa-1, G of it on plane xa ----
    {
      const float* St = &S.e[0][0];
      const float* S1 = &S.e[1][0];
      Vec<4> a0[3], cb0, dxy, dxz, dzx, dzy, dyx, dyz;
      const int im = xa - 1;
      float4 cx;
      int xbase = 0;
#pragma unroll
      for (int c = 0; c < 3; ++c) a0[c] = vld<4>(St + o + c * CE);
      cb0 = vld<4>(St + o + CB);
      Vec<4> gzx = vzero<4>(), gzy = vzero<4>();
      const Vec<4> ze = vld<4>(&S.zt[0][4 * zq]);
      const bool pro = own && xa > 0;
      Vec<4> hx, hy = vld<4>(&S.ho[0][oh + D::CH]), hz = vld<4>(&S.ho[0][oh + 2 * D::CH]), nxy, nxz, nyx, nyz, px0, px1;
      float nzx, nzy;
      if (pro) {
        const bool on = xslab(im, cx, xbase);
        gx_flux(L4{}, a0[1], a0[2], cb0, __ldg(xe_tab + im), on, false, cx, xbase + jk,
                glob(L4{}, psEx + xbase + jk, qx, col + (long long)im * ps), nxy, nxz, px0, px1);
        if (CP && on) {
          vacc<+1>(hy, px1);
          vacc<+1>(hz, px0);
        }
        gz_flux(L4{}, NoW{}, Wr{}, a0[0], a0[1], cb0, ze, zon, zp, oz + im * ny * n4,
                globz(L4{}, psEz + oz + im * ny * n4, qz, col + (long long)im * ps, zon), gzx, gzy, hx, hy);
      }
      z_next(St, gzx, gzy, max(im, 0), nzx, nzy);
      if (pro) {
        gz_diff(a0[0], a0[1], cb0, ze, gzx, gzy, nzx, nzy, dzx, dzy);
        gy_flux(L4{}, vld<4>(St + o + EW), vld<4>(St + o + EW + 2 * CE), vld<4>(St + o + EW + CB), ye1, ynon, cyn,
                glob(L4{}, psEy + oyn + im * ncp * zs, qy, col + zs + (long long)im * ps), nyx, nyz);
        gy_diff(L4{}, NoW{}, a0[0], a0[2], cb0, ye, yon, cy, oy + im * ncp * zs,
                glob(L4{}, psEy + oy + im * ncp * zs, qy, col + (long long)im * ps), nyx, nyz, dyx, dyz, hx, hz);
      }
      if (own) {
        xbase = 0;
        const bool on = xslab(xa, cx, xbase);
        gx_flux(L4{}, vld<4>(S1 + o + CE), vld<4>(S1 + o + 2 * CE), vld<4>(S1 + o + CB), __ldg(xe_tab + xa), on, true, cx,
                xbase + jk, glob(L4{}, psEx + xbase + jk, qx, col + (long long)xa * ps), nxy, nxz, rx0, rx1);
      }
      if (pro) {
        const long long e = col + (long long)im * ps;
        const Vec<4> ch = ch_at(e), xe = vsplat<4>(__ldg(xe_tab + im));
        dxy = vfma<-1>(xe, vmul(cb0, a0[1]), nxy);
        dxz = vfma<-1>(xe, vmul(cb0, a0[2]), nxz);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          hy[l] = curl_t(hy[l], dxz[l], dzx[l]);
          hz[l] = curl_t(hz[l], dyx[l], dxy[l]);
        }
        h_cot(pmask, ptail, im, j, k, [&](int l, int c, float g) {
#pragma unroll
          for (int t = 0; t < 4; ++t)
            if (t == l) {
              if (c == 1) hy[t] = hy[t] + g;
              else if (c == 2) hz[t] = hz[t] + g;
            }
        });
        const Vec<4> py = vmul(ch, hy), pz = vmul(ch, hz), xh = vsplat<4>(__ldg(xh_tab + im));
        xbase = 0;
        if (CP && xslab(im, cx, xbase)) {
          const float* q = AD.aPsiH[par][0] + xbase + jk;
          const Vec<4> one = vsplat<4>(1.f);
          kxyp = vfma<+1>(xh, py, rel_xy<4, +1, false>(vld<4>(q), nullptr, cx, one, py));
          kxzp = vfma<-1>(xh, pz, rel_xy<4, -1, false>(vld<4>(q + qx), nullptr, cx, one, pz));
        } else {
          kxyp = vmul(xh, py);
          kxzp = vmul(xh, pz);
        }
      }
    }
    bar_or<NT>(false);   // the stages of plane xa-1 are free
    if (CP && own) fetch(xa);
    if (CP) cp_async_commit();
    bool bad = false;
    float xe1_n = __ldg(xe_tab + xa + 1), xh_n = __ldg(xh_tab + xa), xe = __ldg(xe_tab + xa);
    int sA = 1, sB = 2;
#pragma unroll 1
    for (int i = xa; i < xb; ++i) {
      const long long e = col + (long long)i * ps;
      const float xe1 = xe1_n, xh = xh_n;
      if (i + 1 < xb) { xe1_n = __ldg(xe_tab + i + 2); xh_n = __ldg(xh_tab + i + 1); }
      float4 cx, cx1;
      int xbase = 0, xbase1 = 0;
      const bool xon = own && xslab(i, cx, xbase), x1on = own && xslab(i + 1, cx1, xbase1);
      unsigned em = 0u;
      if (emask && own) em = *reinterpret_cast<const unsigned*>(emask + e);
      bad = !wait(sB) | bad;
      bad = !wait(3 + sH(i)) | bad;
      if (CP) cp_async_wait<0>();   // this plane's psi
      const float* St = &S.e[sA][0];
      const float* S1 = &S.e[sB][0];
      const float* Ho = &S.ho[sH(i)][oh];
      const float* Sa = St + o;
      // ---- phase A ----
      Vec<4> gzx = vzero<4>(), gzy = vzero<4>();
      const int iz = oz + i * ny * n4;
      Vec<4> hx, hy, hz;   // H, then p = ch aH1
      if (own) {
        hx = vld<4>(Ho);
        hy = vld<4>(Ho + D::CH);
        hz = vld<4>(Ho + 2 * D::CH);
        if (CP && xon) {
          vacc<+1>(hy, rx1);
          vacc<+1>(hz, rx0);
        }
        gz_flux(L4{}, Wr{}, Wr{}, vld<4>(Sa), vld<4>(Sa + CE), vld<4>(Sa + CB), vld<4>(&S.zt[0][4 * zq]), zon, zp, iz,
                [&](int q) { return q == 2 ? sl(4) : sl(q); }, gzx, gzy, hx, hy);
      }
      float nzx, nzy;
      z_next(St, gzx, gzy, i, nzx, nzy);
      Vec<4> kzx = vzero<4>(), kzy = vzero<4>(), rz0 = vzero<4>(), rz1 = vzero<4>();
      Vec<4> sx, sy, sz;   // what phase B adds to ca aEm before the terms of the row below
      if (own) {
        Vec<4> nyx, nyz, dyx, dyz, nxy, nxz, dzx, dzy;
        gz_diff(vld<4>(Sa), vld<4>(Sa + CE), vld<4>(Sa + CB), vld<4>(&S.zt[0][4 * zq]), gzx, gzy, nzx, nzy, dzx, dzy);
        gy_flux(L4{}, vld<4>(St + o + EW), vld<4>(St + o + EW + 2 * CE), vld<4>(St + o + EW + CB), ye1, ynon, cyn,
                [&](int q) {
                  if (q == 2) return vld<4>(P.ce + e + zs);
                  return vld<4>(zon ? psEy + oyn + i * ncp * zs + q * qy : slot + (5 + q) * SS);
                }, nyx, nyz);
        gy_diff(L4{}, Wr{}, vld<4>(Sa), vld<4>(Sa + 2 * CE), vld<4>(Sa + CB), ye, yon, cy, oy + i * ncp * zs,
                [&](int q) { return q == 2 ? sl(4) : sl(zon ? 5 + q : q); }, nyx, nyz, dyx, dyz, hx, hz);
#pragma unroll
        for (int l = 0; l < 4; ++l) hx[l] = curl_t(hx[l], dzy[l], dyz[l]);
        gx_flux(L4{}, vld<4>(S1 + o + CE), vld<4>(S1 + o + 2 * CE), vld<4>(S1 + o + CB), xe1, x1on, i + 1 < xb, cx1,
                xbase1 + jk,
                [&](int q) {
                  if (q == 2) return vld<4>((zon || yon) ? P.ce + e + ps : slot + 4 * SS);
                  return vld<4>((zon || yon) ? psEx + xbase1 + jk + q * qx : slot + q * SS);
                }, nxy, nxz, rx0, rx1);
        {
          const Vec<4> s = vsplat<4>(xe), cb = vld<4>(Sa + CB);
          const Vec<4> dxy = vfma<-1>(s, vmul(cb, vld<4>(Sa + CE)), nxy), dxz = vfma<-1>(s, vmul(cb, vld<4>(Sa + 2 * CE)), nxz);
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            hy[l] = curl_t(hy[l], dxz[l], dzx[l]);
            hz[l] = curl_t(hz[l], dyx[l], dxy[l]);
          }
        }
        if (pmask || ptail)
          h_cot(pmask, ptail, i, j, k, [&](int l, int c, float g) {
#pragma unroll
            for (int t = 0; t < 4; ++t)
              if (t == l) {
                if (c == 0) hx[t] = hx[t] + g;
                else if (c == 1) hy[t] = hy[t] + g;
                else hz[t] = hz[t] + g;
              }
          });
        if (kv < 4) {
#pragma unroll
          for (int l = 1; l < 4; ++l)
            if (l >= kv) { hx[l] = 0.f; hy[l] = 0.f; hz[l] = 0.f; }
        }
        vst<4>(Fo + 3 * cs + e, hx);
        vst<4>(Fo + 4 * cs + e, hy);
        vst<4>(Fo + 5 * cs + e, hz);
        if (in_gyz && i >= P.hb[0] && i < P.hb[1]) {
          const int sy = P.hb[3] - P.hb[2], sz = P.hb[5] - P.hb[4];
          const int hc = (P.hb[1] - P.hb[0]) * sy * sz;
          const int c0 = ((i - P.hb[0]) * sy + (j - P.hb[2])) * sz + (k - P.hb[4]);
          const float* hp0 = P.hist + (long long)(n - P.hist_step0) * P.hist_ld + c0;
          float al[3][4];
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            al[0][l] = Sa[l];
            al[1][l] = Sa[CE + l];
            al[2][l] = Sa[2 * CE + l];
          }
#pragma unroll 1
          for (int l = max(0, P.hb[4] - k); l < min(4, P.hb[5] - k); ++l) {
            const float* hp = hp0 + l;
            const float dca = P.dca[c0 + l], dcb = P.dcb[c0 + l];
            const double acc = (double)al[0][l] * ((double)dca * hp[0] + (double)dcb * hp[3 * hc]) +
                               (double)al[1][l] * ((double)dca * hp[hc] + (double)dcb * hp[4 * hc]) +
                               (double)al[2][l] * ((double)dca * hp[2 * hc] + (double)dcb * hp[5 * hc]);
            P.grad[c0 + l] += acc;
          }
        }
        // p = ch aH1 and its fluxes in z
        const Vec<4> ch = ch_at(e), zh = vld<4>(&S.zt[1][4 * zq]);
        hx = vmul(ch, hx);
        hy = vmul(ch, hy);
        hz = vmul(ch, hz);
        if (CP && zon) {   // (hx <- ey, +1, q0), (hy <- ex, -1, q1)
          float* u = AD.aPsiH[par ^ 1][2] + iz;
          const Vec<4> b = vld<4>(zp), c = vld<4>(zp + ZPS), km = vld<4>(zp + 2 * ZPS), one = vsplat<4>(1.f);
          rz0 = rel_z<4, +1, true>(sl(2), u, zon, b, c, km, one, hx);
          rz1 = rel_z<4, -1, true>(sl(3), u + qz, zon, b, c, km, one, hy);
        }
        kzx = vflux<CP, +1>(zh, hx, rz0);
        kzy = vflux<CP, -1>(zh, hy, rz1);
      }
      const int ks = i & 1;
      const float zmx = __shfl_up_sync(0xffffffffu, kzx[3], 1, ZQ), zmy = __shfl_up_sync(0xffffffffu, kzy[3], 1, ZQ);
      if (own) {
        // their differences, but for the first column of the tile (its neighbour's come from the halo warp)
        const Vec<4> zh = vld<4>(&S.zt[1][4 * zq]), one = vsplat<4>(1.f);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          const bool far = l == 0 && first_q;
          sy[l] = far ? 0.f : __fmaf_rn(zh[l], hx[l], -(l ? kzx[l ? l - 1 : 0] : zmx));
          sx[l] = far ? 0.f : __fmaf_rn(zh[l], hy[l], -(l ? kzy[l ? l - 1 : 0] : zmy));
        }
        if (CP && zon) {
          vacc<+1>(sy, rz0);
          vacc<-1>(sx, rz1);
        }
        // the differences in x
        const Vec<4> s = vsplat<4>(xh);
        Vec<4> dz = vfma<-1>(s, hz, kxzp), r0 = vzero<4>(), r1 = vzero<4>();
        sz = vfma<-1>(s, hy, kxyp);
        if (CP && xon) {   // (hy <- ez, +1, q0), (hz <- ey, -1, q1)
          const float* q = AD.aPsiH[par][0] + xbase + jk;
          float* u = AD.aPsiH[par ^ 1][0] + xbase + jk;
          const bool far = zon || yon;
          r0 = rel_xy<4, +1, true>(vld<4>(far ? q : slot + 2 * SS), u, cx, one, hy);
          r1 = rel_xy<4, -1, true>(vld<4>(far ? q + qx : slot + 3 * SS), u + qx, cx, one, hz);
          vacc<+1>(sz, r0);
          vacc<-1>(dz, r1);
        }
        kxyp = vflux<CP, +1>(s, hy, r0);
        kxzp = vflux<CP, -1>(s, hz, r1);
#pragma unroll
        for (int l = 0; l < 4; ++l) sy[l] = __fsub_rn(dz[l], sy[l]);
        // the fluxes in y, to the row above
        Vec<4> ry0 = vzero<4>(), ry1 = vzero<4>();
        if (CP && yon) {   // (hx <- ez, -1, q0), (hz <- ex, +1, q1)
          const int iy = oy + i * ncp * zs;
          const float* q = AD.aPsiH[par][1] + iy;
          float* u = AD.aPsiH[par ^ 1][1] + iy;
          ry0 = rel_xy<4, -1, true>(vld<4>(zon ? q : slot + 2 * SS), u, cy, one, hx);
          ry1 = rel_xy<4, +1, true>(vld<4>(zon ? q + qy : slot + 3 * SS), u + qy, cy, one, hz);
          vacc<+1>(sz, ry0);
          vacc<-1>(sx, ry1);
        }
        if (r + 1 < TY) {
          const Vec<4> s = vsplat<4>(yh);
          vst<4>(&S.k[ks][0][r + 1][4 * zq], vflux<CP, -1>(s, hx, ry0));
          vst<4>(&S.k[ks][1][r + 1][4 * zq], vflux<CP, +1>(s, hz, ry1));
        }
      }
      if (CP && own && i + 1 < xb) fetch(i + 1);
      if (CP) cp_async_commit();
      // the cells' own E: its stage is refilled after the barrier
      Vec<4> a0[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) a0[c] = vld<4>(Sa + c * CE);
      if (bar_or<NT>(bad)) { bad = true; break; }
      bad = !wait(5 + sC(i));
      // ---- phase B ----
      if (own) {
        if (first_q) {
          const float zh0 = S.zt[1][4 * zq];
          sx[0] = __fadd_rn(sx[0], __fmaf_rn(zh0, hy[0], -S.kc[ks][1][r]));
          sy[0] = __fsub_rn(sy[0], __fmaf_rn(zh0, hx[0], -S.kc[ks][0][r]));
        }
        const Vec<4> myx = vld<4>(&S.k[ks][0][r][4 * zq]), myz = vld<4>(&S.k[ks][1][r][4 * zq]);
        const Vec<4> cav = vld<4>(&S.ca[sC(i)][oc]);
        Vec<4> ex, ey, ez;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          ex[l] = __fmaf_rn(cav[l], a0[0][l], __fsub_rn(sx[l], __fmaf_rn(yh, hz[l], -myz[l])));
          ey[l] = __fmaf_rn(cav[l], a0[1][l], sy[l]);
          ez[l] = __fmaf_rn(cav[l], a0[2][l], __fsub_rn(__fmaf_rn(yh, hx[l], -myx[l]), sz[l]));
        }
        if (n >= 1 && (pmask | smask | (unsigned)ptail | (unsigned)stail)) {
          // over an indexed copy: the E-probe cotangents of y_{n-1}, then the source adjoints
          float v[3][4];
#pragma unroll
          for (int l = 0; l < 4; ++l) { v[0][l] = ex[l]; v[1][l] = ey[l]; v[2][l] = ez[l]; }
#pragma unroll 1
          for (int pass = 0; pass < 2; ++pass) {
            const int count = pass ? (P.src_adj ? P.nsrc : 0) : P.g ? P.nprb : 0;
            const int4* list = pass ? P.src : P.prb;
            unsigned m = pass ? smask : pmask;
            int q = 31;
#pragma unroll 1
            while (true) {
              if (m) { q = __ffs(m) - 1; m &= m - 1; }
              else q = max(q + 1, 32);
              if (q >= count) break;
              const int4 c = __ldg(list + q);
              if (c.x != i || c.y != j || c.z < k || c.z >= k + 4) continue;
              if (pass) P.src_adj[(long long)(n - 1) * P.src_ld + q] = v[min(c.w, 2)][c.z - k];
              else if ((c.w & 7) < 3) v[c.w & 7][c.z - k] += __ldg(P.g + (long long)(n - 1) * P.g_ld + q);
            }
          }
#pragma unroll
          for (int l = 0; l < 4; ++l) { ex[l] = v[0][l]; ey[l] = v[1][l]; ez[l] = v[2][l]; }
        }
        if (kv < 4) {
#pragma unroll
          for (int l = 1; l < 4; ++l)
            if (l >= kv) { ex[l] = 0.f; ey[l] = 0.f; ez[l] = 0.f; }
        }
        if ((pec & 1u) && (i == 0 || i == nx - 1)) { ey = vzero<4>(); ez = vzero<4>(); }
        if (pec_j) { ex = vzero<4>(); ez = vzero<4>(); }
        if (pec_k) {
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            if (k + l == 0 || k + l == nz - 1) { ex[l] = 0.f; ey[l] = 0.f; }
            if (k + l == nz - 1) ez[l] = 0.f;
          }
        }
        if (em) {
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            const unsigned m = em >> (8 * l);
            if (m & 1u) ex[l] = 0.f;
            if (m & 2u) ey[l] = 0.f;
            if (m & 4u) ez[l] = 0.f;
          }
        }
        vst<4>(Fo + e, ex);
        vst<4>(Fo + cs + e, ey);
        vst<4>(Fo + 2 * cs + e, ez);
      }
      xe = xe1;
      sA = sB;
      sB = sB == 2 ? 0 : sB + 1;
    }
    bad_end = bad;
  } else {
    // ---- halo warp: row y0-1 (lanes < ZQ, four columns each: Kyx, Kyz),
    // column z0-1 (lanes ZQ .. ZQ+TY-1, one row each: Kzx, Kzy); the last lane
    // issues the boxes ----
    const int lane = tid - D::MAIN;
    const bool is_row = lane < ZQ, is_col = lane >= ZQ && lane - ZQ < TY;
    const bool row = is_row && y0 >= 1 && z0 + 4 * lane < nz;
    const bool colm = is_col && z0 >= 1 && y0 + lane - ZQ < ny;
    const bool on = row || colm;
    const int j = is_row ? y0 - 1 : y0 + lane - ZQ;
    const int k = is_row ? z0 + 4 * lane : z0 - 1;
    const int o = is_row ? 4 * lane + 4 : (lane - ZQ + 1) * EW + 3;
    const long long col = on ? P.off0 + (long long)j * zs + k : 0;
    const int jk = on ? j * zs + k : 0;
    const float ye = on ? __ldg(P.ye + j) : 0.f, ye1 = on ? __ldg(P.ye + j + 1) : 0.f;
    const float yh = on ? __ldg(P.yh + j) : 0.f;
    float4 cy, cyn;
    int oy = 0, oyn = 0;
    const bool yon = on && yslab(j, k, cy, oy);
    const bool ynon = on && j + 1 < ny && yslab(j + 1, k, cyn, oyn);
    const int orow = on ? j * n4 : 0;
    int zoff = 0, zoff0 = 0;
    const unsigned zon_r = row && cpz ? zslab_of<4>(k, ncp, kb, nz, 2 * qz, zoff) : 0u;
    // the column's z slab and that of column z0 (whose profile starts S.zp)
    const unsigned zon_c = colm && cpz ? zslab_of<1>(k, ncp, kb, nz, 2 * qz, zoff) : 0u;
    const unsigned zon_0 = colm && cpz ? zslab_of<1>(z0, ncp, kb, nz, 2 * qz, zoff0) : 0u;
    float ze_c = 0.f, zh_c = 0.f;
    float4 czc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (colm) {
      ze_c = __ldg(P.ze + k);
      zh_c = __ldg(P.zh + k);
      if (zon_c) czc = k < ncp ? __ldg(P.cpt + 4 * ncp + k) : __ldg(P.cpt + 5 * ncp + (k - kb));
    }
    unsigned pmask = 0u;
    if (on)
#pragma unroll 1
      for (int q = 0; q < min(P.nprb, 32); ++q) {
        const int4 c = __ldg(P.prb + q);
        if (c.y == j && (row ? (c.z >= k && c.z < k + 4) : c.z == k)) pmask |= 1u << q;
      }
    const bool ptail = P.nprb > 32;
    // G of the x direction (row Gxy, column Gxz) of plane p and its relation
    auto gx_halo = [&](const float* St, int p, float xe, Vec<4>& gr, Vec<1>& gc, Vec<4>& rr, Vec<1>& rc) {
      float4 cx;
      int xbase = 0;
      const bool xs = xslab(p, cx, xbase);
      const long long e = col + (long long)p * ps;
      if (row) {
        Vec<4> g, d;
        gx_flux(L4{}, vld<4>(St + o + CE), vld<4>(St + o + 2 * CE), vld<4>(St + o + CB), xe, xs, false, cx, xbase + jk,
                glob(L4{}, psEx + xbase + jk, qx, e), gr, g, rr, d);
      } else if (colm) {
        Vec<1> g, d;
        gx_flux(L1{}, vld<1>(St + o + CE), vld<1>(St + o + 2 * CE), vld<1>(St + o + CB), xe, xs, false, cx, xbase + jk,
                glob(L1{}, psEx + xbase + jk, qx, e), g, gc, d, rc);
      }
    };
    Vec<4> rxr, g0r;
    Vec<1> rxc, g0c;
    gx_halo(&S.e[1][0], xa, __ldg(xe_tab + xa), g0r, g0c, rxr, rxc);
    float hc0 = 0.f, hc1 = 0.f;   // the column's adjoint hx, hy, one plane ahead
    auto load_old = [&](int i) {
      if (!colm) return;
      const long long e = col + (long long)i * ps;
      hc0 = Fi[3 * cs + e];
      hc1 = Fi[4 * cs + e];
    };
    load_old(xa);
    bar_or<NT>(false);   // the stages of plane xa-1 are free
    if (producer) {
      if (xa + 2 <= xb) issue_e(xa + 2);
      if (xa + 1 < xb) issue_h(xa + 1);
    }
    last_e = min(xa + 2, xb);
    last_h = min(xa + 1, xb - 1);
    bool bad = false;
    float xe1_n = __ldg(xe_tab + xa + 1), xe = __ldg(xe_tab + xa);
    int sA = 1, sB = 2;
#pragma unroll 1
    for (int i = xa; i < xb; ++i) {
      const float xe1 = xe1_n;
      if (i + 1 < xb) xe1_n = __ldg(xe_tab + i + 2);
      const long long e = col + (long long)i * ps;
      bad = !wait(sB) | bad;
      bad = !wait(3 + sH(i)) | bad;
      const float* St = &S.e[sA][0];
      const float* S1 = &S.e[sB][0];
      const float* Ho = &S.ho[sH(i)][0];
      const int ks = i & 1;
      const int irow = orow + i * ny * n4, iz = irow + zoff;
      Vec<4> nxr, nrr;   // flux and relation of plane i+1
      Vec<1> nxc, nrc;
      gx_halo(S1, i + 1, xe1, nxr, nxc, nrr, nrc);
      const bool xon = in_xslab(i);
      if (is_row) {
        Vec<4> kyx = vzero<4>(), kyz = vzero<4>(), gzx, gzy = vzero<4>(), ex, ez, cb, hx, hz, dz;
        if (row) {
          ex = vld<4>(St + o);
          ez = vld<4>(St + o + 2 * CE);
          cb = vld<4>(St + o + CB);
          hx = vld<4>(Ho + 4 * lane);
          hz = vld<4>(Ho + 2 * D::CH + 4 * lane);
          if (xon) vacc<+1>(hz, rxr);
          gz_flux(L4{}, NoW{}, Wr{}, ex, vld<4>(St + o + CE), cb, vld<4>(&S.zt[0][4 * lane]), zon_r, &S.zp[0][4 * lane], iz,
                  globz(L4{}, psEz + iz, qz, e, zon_r), gzx, gzy, hx, dz);
        }
        float nzy = __shfl_down_sync((1u << ZQ) - 1u, gzy[0], 1, ZQ);
        if (row) {
          if (lane == ZQ - 1) {
            float d;
            gz_after(St, o + 4, irow, e + 4, d, nzy);
          }
          Vec<4> nyx, nyz, dyx, dyz, dzx, dzy;
          gz_diff(ex, vld<4>(St + o + CE), cb, vld<4>(&S.zt[0][4 * lane]), gzx, gzy, 0.f, nzy, dzx, dzy);
          gy_flux(L4{}, vld<4>(St + o + EW), vld<4>(St + o + EW + 2 * CE), vld<4>(St + o + EW + CB), ye1, ynon, cyn,
                  glob(L4{}, psEy + oyn + i * ncp * zs, qy, e + zs), nyx, nyz);
          gy_diff(L4{}, NoW{}, ex, ez, cb, ye, yon, cy, oy + i * ncp * zs, glob(L4{}, psEy + oy + i * ncp * zs, qy, e), nyx,
                  nyz, dyx, dyz, hx, hz);
          const Vec<4> dxr = vfma<-1>(vsplat<4>(xe), vmul(cb, vld<4>(St + o + CE)), nxr);
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            hx[l] = curl_t(hx[l], dzy[l], dyz[l]);
            hz[l] = curl_t(hz[l], dyx[l], dxr[l]);
          }
          if (pmask || ptail)
            h_cot(pmask, ptail, i, j, k, [&](int l, int c, float g) {
#pragma unroll
              for (int t = 0; t < 4; ++t)
                if (t == l) {
                  if (c == 0) hx[t] = hx[t] + g;
                  else if (c == 2) hz[t] = hz[t] + g;
                }
            });
          const Vec<4> ch = ch_at(e), s = vsplat<4>(yh), one = vsplat<4>(1.f);
          hx = vmul(ch, hx);
          hz = vmul(ch, hz);
          if (CP && yon) {
            const float* q = AD.aPsiH[par][1] + oy + i * ncp * zs;
            kyx = vfma<-1>(s, hx, rel_xy<4, -1, false>(vld<4>(q), nullptr, cy, one, hx));
            kyz = vfma<+1>(s, hz, rel_xy<4, +1, false>(vld<4>(q + qy), nullptr, cy, one, hz));
          } else {
            kyx = vmul(s, hx);
            kyz = vmul(s, hz);
          }
        }
        vst<4>(&S.k[ks][0][0][4 * lane], kyx);
        vst<4>(&S.k[ks][1][0][4 * lane], kyz);
      }
      if (is_col) {
        float kzx = 0.f, kzy = 0.f;
        if (colm) {
          const Vec<1> ex = vld<1>(St + o), ey = vld<1>(St + o + CE), ez = vld<1>(St + o + 2 * CE), cb = vld<1>(St + o + CB);
          // z fluxes of this column and of column z0
          Vec<1> ze, nzx, nzy, nyx, nyz, dzx, dzy, dyx, dyz, dxz, hz, hx = vsplat<1>(hc0), hy = vsplat<1>(hc1);
          if (xon) vacc<+1>(hy, rxc);
          ze[0] = S.zt[0][0];
          gz_flux(L1{}, NoW{}, NoW{}, vld<1>(St + o + 1), vld<1>(St + o + 1 + CE), vld<1>(St + o + 1 + CB), ze, zon_0, &S.zp[0][0],
                  irow + zoff0, glob(L1{}, psEz + irow + zoff0, qz, e + 1), nzx, nzy, hx, hy);
          ze[0] = ze_c;
          dzx = vfma<-1>(ze, vmul(cb, ex), nzx);
          dzy = vfma<-1>(ze, vmul(cb, ey), nzy);
          if (CP && zon_c) {
            const Vec<1> ce = vld<1>(P.ce + e);
            vacc<+1>(hy, rel_xy<1, -1, false>(vld<1>(psEz + iz), nullptr, czc, ce, ex));
            vacc<+1>(hx, rel_xy<1, +1, false>(vld<1>(psEz + iz + qz), nullptr, czc, ce, ey));
          }
          gy_flux(L1{}, vld<1>(St + o + EW), vld<1>(St + o + EW + 2 * CE), vld<1>(St + o + EW + CB), ye1, ynon, cyn,
                  glob(L1{}, psEy + oyn + i * ncp * zs, qy, e + zs), nyx, nyz);
          gy_diff(L1{}, NoW{}, ex, ez, cb, ye, yon, cy, oy + i * ncp * zs, glob(L1{}, psEy + oy + i * ncp * zs, qy, e), nyx,
                  nyz, dyx, dyz, hx, hz);
          dxz = vfma<-1>(vsplat<1>(xe), vmul(cb, ez), nxc);
          hx[0] = curl_t(hx[0], dzy[0], dyz[0]);
          hy[0] = curl_t(hy[0], dxz[0], dzx[0]);
          if (pmask || ptail)
            h_cot(pmask, ptail, i, j, k, [&](int l, int c, float g) {
              if (l != 0) return;
              if (c == 0) hx[0] = hx[0] + g;
              else if (c == 1) hy[0] = hy[0] + g;
            });
          const Vec<1> ch = vsplat<1>(ch_arr ? ch_arr[e] : ch0), zh = vsplat<1>(zh_c), one = vsplat<1>(1.f);
          hx = vmul(ch, hx);
          hy = vmul(ch, hy);
          Vec<1> vx, vy;
          if (CP && zon_c) {
            const float* q = AD.aPsiH[par][2] + iz;
            vx = vfma<+1>(zh, hx, rel_xy<1, +1, false>(vld<1>(q), nullptr, czc, one, hx));
            vy = vfma<-1>(zh, hy, rel_xy<1, -1, false>(vld<1>(q + qz), nullptr, czc, one, hy));
          } else {
            vx = vmul(zh, hx);
            vy = vmul(zh, hy);
          }
          kzx = vx[0];
          kzy = vy[0];
        }
        S.kc[ks][0][lane - ZQ] = kzx;
        S.kc[ks][1][lane - ZQ] = kzy;
      }
      rxr = nrr;
      rxc = nrc;
      xe = xe1;
      if (i + 1 < xb) load_old(i + 1);
      if (bar_or<NT>(bad)) { bad = true; break; }
      // phase A of plane i is done: its H stage takes plane i+2 and its E stage
      // plane i+3 (the owners hold plane i's own cells in registers); phase B of
      // plane i-1 is done: its ca stage takes plane i+1
      if (producer) {
        if (i + 3 <= xb) issue_e(i + 3);
        if (i + 2 < xb) issue_h(i + 2);
        if (i > xa && i + 1 < xb) issue_c(i + 1);
      }
      last_e = min(i + 3, xb);
      last_h = min(i + 2, xb - 1);
      last_c = max(last_c, min(i + 1, xb - 1));
      ph.stage ^= 1u << (5 + sC(i));   // the owners wait for ca
      sA = sB;
      sB = sB == 2 ? 0 : sB + 1;
    }
    bad_end = bad;
  }
  if (bar_or<NT>(bad_end)) { bail(); return false; }
  return true;
}

template <int TY, int ZQ, bool CP>
__device__ __forceinline__ void adjv_init_barriers(AVSmem<TY, ZQ, CP>& S) {
  if (threadIdx.x == 0) {
#pragma unroll 1
    for (int q = 0; q < RFXB_VBARS; ++q) mbar_init(smem_u32(&S.mbar[q]), 1);
    mbar_fence_init();
  }
  __syncthreads();
}

// One launch per reverse step: CTA b runs work item b.
template <int TY, int ZQ, bool CP>
__global__ void __launch_bounds__(AVDims<TY, ZQ>::NT, (TY == 24 ? 2 : 5))
adjv_kernel(const RfxbInst* __restrict__ insts, const AdjInst* __restrict__ adjs, const RfxbWork* __restrict__ work,
            const CUtensorMap* __restrict__ maps, int map0, int n, int par, int apar) {
  extern __shared__ __align__(128) unsigned char adjv_smem_raw[];
  RfxbWork w = work[blockIdx.x];
  StepPhases ph;
  if (!CP || (w.inst & RFXB_WORK_PLAIN)) {
    w.inst &= ~RFXB_WORK_PLAIN;
    auto& S = *reinterpret_cast<AVSmem<TY, ZQ, false>*>(adjv_smem_raw);
    adjv_init_barriers<TY, ZQ, false>(S);
    adjv_item<TY, ZQ, false>(S, insts, adjs, w, maps, map0, n, par, apar, ph, StepFault{}, true);
  } else {
    auto& S = *reinterpret_cast<AVSmem<TY, ZQ, CP>*>(adjv_smem_raw);
    adjv_init_barriers<TY, ZQ, CP>(S);
    adjv_item<TY, ZQ, CP>(S, insts, adjs, w, maps, map0, n, par, apar, ph, StepFault{}, true);
  }
}

// Persistent reverse step: one launch per reverse step of as many CTAs as are
// resident, pulling items from three queues (tiles that reach a y slab, the
// other CPML work, the CPML-free tiles) in an order set by the CTA's role.
// Invalid items are skipped and flagged (status bit 2); the last CTA to finish
// clears the fetch counters for the next launch.
template <int TY, int ZQ>
__global__ void __launch_bounds__(AVDims<TY, ZQ>::NT, 5)
adjv_persist_kernel(const RfxbInst* __restrict__ insts, const AdjInst* __restrict__ adjs, int n_inst, RfxbAdjQueues Q,
                    const CUtensorMap* __restrict__ maps, int map0, int n, int par, int apar) {
  extern __shared__ __align__(128) unsigned char adjv_smem_raw[];
  auto& S = *reinterpret_cast<AVSmem<TY, ZQ, true>*>(adjv_smem_raw);
  __shared__ int pick[2];
  const int tid = threadIdx.x;
  adjv_init_barriers<TY, ZQ, true>(S);
  StepPhases ph;
  StepFault fault;
  fault.cta = Q.fault_cta;
  fault.wait_limit = Q.wait_limit;
  static constexpr int kOrder[3][3] = {{2, 1, 0}, {1, 0, 2}, {0, 1, 2}};
  const int role = min(2, (int)blockIdx.x / max(1, Q.role_ctas));
  bool first_item = true;
  bool ok = true;
  while (ok) {
    if (tid == 0) {
      pick[0] = -1;
      for (int t = 0; t < 3; ++t) {
        const int q = kOrder[role][t];
        if (*(volatile int*)&Q.ctr[q] >= Q.count[q]) continue;   // drained (counters only grow): no ticket
        const int k = atomicAdd(&Q.ctr[q], 1);
        if (k < Q.count[q]) { pick[0] = q; pick[1] = k; break; }
      }
    }
    __syncthreads();
    const int q = pick[0], k = pick[1];
    __syncthreads();
    if (q < 0) break;
    const RfxbWork w = Q.list[q][k];
    if (!work_item_valid<TY, ZQ>(w, insts, n_inst)) {
      if (tid == 0) atomicOr(Q.status, 2);
      continue;
    }
    ok = adjv_item<TY, ZQ, true>(S, insts, adjs, w, maps, map0, n, par, apar, ph, fault, first_item);
    first_item = false;
  }
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(&Q.ctr[3], 1) == (int)gridDim.x - 1) {
      Q.ctr[0] = 0;
      Q.ctr[1] = 0;
      Q.ctr[2] = 0;
      Q.ctr[3] = 0;
      __threadfence();
    }
  }
}

#define RFXB_ADJV(TY, ZQ, CP)                                                                                     \
  template __global__ void adjv_kernel<TY, ZQ, CP>(const RfxbInst*, const AdjInst*, const RfxbWork*, const CUtensorMap*, \
                                                   int, int, int, int)
RFXB_ADJV(24, 8, false);
RFXB_ADJV(24, 8, true);
RFXB_ADJV(8, 8, false);
RFXB_ADJV(8, 8, true);
template __global__ void adjv_persist_kernel<8, 8>(const RfxbInst*, const AdjInst*, int, RfxbAdjQueues,
                                                   const CUtensorMap*, int, int, int, int);

size_t adjv_smem_bytes(int tile, bool cp) {
  return tile == 0 ? (cp ? sizeof(AVSmem<24, 8, true>) : sizeof(AVSmem<24, 8, false>))
                   : (cp ? sizeof(AVSmem<8, 8, true>) : sizeof(AVSmem<8, 8, false>));
}
static_assert(2 * (sizeof(AVSmem<24, 8, true>) + 1024) <= 228 * 1024, "two CTAs per SM");

}  // namespace rfxb
