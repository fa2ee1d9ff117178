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
// Every product is rounded by itself before differences are taken: the adjoint
// fields are 1.04 to 1.17 times as far from a float64 march as with one cell per
// thread (rfxb_adj_fused.cu), which fuses one of two products.
// The probe cotangent of y_{n-1}, the source adjoint and the PEC / edge mask
// follow; adjoint fields and psi are ping-ponged like the forward state.  The
// eps_r gradient over the recorded region is accumulated in phase A from the
// forward history.  Products and sums are rounding intrinsics.
//
// What bounds it: instructions and, in the slabs, instruction fetch (the CPML
// path is 98 KB of code; the rare work -- probes, sources, gradient, failure --
// therefore sits behind single sites over indexed copies: the step of 20 grids
// of 64-160 cells a side 1477 -> 1380 us).  One cell per thread with the
// relations of the neighbours evaluated again in place -> here: that step
// 1810 -> 1375 us (three launches against one), 221x141x69 with CPML 10
// 157 -> 100, 97x83x109 with CPML 8 103 -> 43.
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
// f += ADD * r of a relation of an x or y slab, from its old psi p
template <int L, int SGN, int ADD, bool WRITE>
__device__ __forceinline__ void rel_xy(Vec<L>& f, Vec<L> p, float* out, const float4& c, const Vec<L>& s,
                                       const Vec<L>& t, bool write = true) {
#pragma unroll
  for (int l = 0; l < L; ++l) {
    const float nu = rel_nu<SGN>(p[l], s[l], t[l]);
    const float r = rel_r<SGN>(nu, s[l], t[l], c.y, c.z);
    f[l] = ADD > 0 ? __fadd_rn(f[l], r) : __fsub_rn(f[l], r);
    p[l] = __fmul_rn(c.x, nu);
  }
  if (WRITE && write) vst<L>(out, p);
}
// the same for a z slab: profile per column, psi at the columns' layers
template <int L, int SGN, int ADD, bool WRITE>
__device__ __forceinline__ void rel_z(Vec<L>& f, Vec<L> p, float* out, unsigned m, const Vec<L>& b,
                                      const Vec<L>& c, const Vec<L>& km, const Vec<L>& s, const Vec<L>& t) {
#pragma unroll
  for (int l = 0; l < L; ++l) {
    const float nu = rel_nu<SGN>(p[l], s[l], t[l]);
    const float r = rel_r<SGN>(nu, s[l], t[l], c[l], km[l]);
    if ((m >> l) & 1u) f[l] = ADD > 0 ? __fadd_rn(f[l], r) : __fsub_rn(f[l], r);
    p[l] = __fmul_rn(b[l], nu);
  }
  if (WRITE) zpsi_store<L>(out, m, p);
}

template <int L>
__device__ __forceinline__ Vec<L> vscale(float a, const Vec<L>& b, const Vec<L>& c) {   // a (b c)
  Vec<L> r;
#pragma unroll
  for (int l = 0; l < L; ++l) r[l] = __fmul_rn(a, __fmul_rn(b[l], c[l]));
  return r;
}
template <int L>
__device__ __forceinline__ Vec<L> vscale(const Vec<L>& a, const Vec<L>& b, const Vec<L>& c) {
  Vec<L> r;
#pragma unroll
  for (int l = 0; l < L; ++l) r[l] = __fmul_rn(a[l], __fmul_rn(b[l], c[l]));
  return r;
}
// a + ((b - bn) - (c - cn))
__device__ __forceinline__ float curl_t(float a, float b, float bn, float c, float cn) {
  return __fadd_rn(a, __fsub_rn(__fsub_rn(b, bn), __fsub_rn(c, cn)));
}

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

  // fluxes of L columns with fields ex ey ez and coefficient cb; in a slab, ld(q)
  // gives the old psi and ld(2) the cells' ce.
  // G of the y direction: Gyx = ye q_x + r_y0, Gyz = ye q_z - r_y1.
  auto gy_flux = [&](auto LL, auto WR, const Vec<decltype(LL)::v>& ex, const Vec<decltype(LL)::v>& ez,
                     const Vec<decltype(LL)::v>& cb, float ye, bool on, const float4& c, int iy, auto&& ld,
                     Vec<decltype(LL)::v>& gyx, Vec<decltype(LL)::v>& gyz) {
    constexpr int L = decltype(LL)::v;
    constexpr bool W = decltype(WR)::v != 0;
    gyx = vscale<L>(ye, cb, ex);
    gyz = vscale<L>(ye, cb, ez);
    if (CP && on) {
      const Vec<L> ce = ld(2);
      float* out = AD.aPsiE[par ^ 1][1];
      rel_xy<L, +1, +1, W>(gyx, ld(0), out + iy, c, ce, ex);
      rel_xy<L, -1, -1, W>(gyz, ld(1), out + iy + qy, c, ce, ez);
    }
  };
  // G of the z direction: Gzx = ze q_x - r_z0, Gzy = ze q_y + r_z1.
  auto gz_flux = [&](auto LL, auto WR, const Vec<decltype(LL)::v>& ex, const Vec<decltype(LL)::v>& ey,
                     const Vec<decltype(LL)::v>& cb, const Vec<decltype(LL)::v>& ze, unsigned on, const float* zp, int iz,
                     auto&& ld, Vec<decltype(LL)::v>& gzx, Vec<decltype(LL)::v>& gzy) {
    constexpr int L = decltype(LL)::v;
    constexpr bool W = decltype(WR)::v != 0;
    gzx = vscale<L>(ze, cb, ex);
    gzy = vscale<L>(ze, cb, ey);
    if (CP && on) {
      const Vec<L> ce = ld(2);
      const Vec<L> b = vld<L>(zp), c = vld<L>(zp + ZPS), km = vld<L>(zp + 2 * ZPS);
      float* out = AD.aPsiE[par ^ 1][2];
      rel_z<L, -1, -1, W>(gzx, ld(0), out + iz, on, b, c, km, ce, ex);
      rel_z<L, +1, +1, W>(gzy, ld(1), out + iz + qz, on, b, c, km, ce, ey);
    }
  };
  // G of the x direction: Gxy = xe q_y - r_x0, Gxz = xe q_z + r_x1.
  auto gx_flux = [&](auto LL, const Vec<decltype(LL)::v>& ey, const Vec<decltype(LL)::v>& ez,
                     const Vec<decltype(LL)::v>& cb, float xe, bool on, bool write, const float4& c, int ix, auto&& ld,
                     Vec<decltype(LL)::v>& gxy, Vec<decltype(LL)::v>& gxz) {
    constexpr int L = decltype(LL)::v;
    gxy = vscale<L>(xe, cb, ey);
    gxz = vscale<L>(xe, cb, ez);
    if (CP && on) {
      const Vec<L> ce = ld(2);
      float* out = AD.aPsiE[par ^ 1][0];
      rel_xy<L, -1, -1, L == 4>(gxy, ld(0), out + ix, c, ce, ey, write);
      rel_xy<L, +1, +1, L == 4>(gxz, ld(1), out + ix + qx, c, ce, ez, write);
    }
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
  // Gzx, Gzy of column z0 + TZ (the one after the tile) at a row's position
  auto gz_after = [&](const float* St, int o, int irow, long long e, float& gx, float& gy) {
    const int k = z0 + TZ;
    if (k >= nz) { gx = 0.f; gy = 0.f; return; }
    Vec<1> ex = vld<1>(St + o), ey = vld<1>(St + o + CE), cb = vld<1>(St + o + CB), ze, a, b;
    ze[0] = S.zt[0][TZ];
    int off = 0;
    const unsigned m = cpz ? zslab_of<1>(k, ncp, kb, nz, 2 * qz, off) : 0u;
    gz_flux(L1{}, NoW{}, ex, ey, cb, ze, m, &S.zp[0][TZ], irow + off, glob(L1{}, psEz + irow + off, qz, e), a, b);
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

    Vec<4> a0[3], cb0;
    const int oh = (r + 1) * TZ + 4 * zq, oc = r * TZ + 4 * zq;   // this thread's place in an H / ca stage
    Vec<4> gxy = vzero<4>(), gxz = vzero<4>(), kxyp = vzero<4>(), kxzp = vzero<4>();
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
    auto ch_at = [&](long long e) {
      Vec<4> c;
      if (ch_arr) c = vld<4>(ch_arr + e);
      else {
#pragma unroll
        for (int l = 0; l < 4; ++l) c[l] = ch0;
      }
      return c;
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
      Vec<4> pxy = vzero<4>(), pxz = vzero<4>();
      const int im = xa - 1;
      float4 cx;
      int xbase = 0;
#pragma unroll
      for (int c = 0; c < 3; ++c) a0[c] = vld<4>(St + o + c * CE);
      cb0 = vld<4>(St + o + CB);
      Vec<4> gzx = vzero<4>(), gzy = vzero<4>();
      const bool pro = own && xa > 0;
      if (pro) {
        const bool on = xslab(im, cx, xbase);
        gx_flux(L4{}, a0[1], a0[2], cb0, __ldg(xe_tab + im), on, false, cx, xbase + jk,
                glob(L4{}, psEx + xbase + jk, qx, col + (long long)im * ps), pxy, pxz);
        gz_flux(L4{}, NoW{}, a0[0], a0[1], cb0, vld<4>(&S.zt[0][4 * zq]), zon, zp, oz + im * ny * n4,
                globz(L4{}, psEz + oz + im * ny * n4, qz, col + (long long)im * ps, zon), gzx, gzy);
      }
      float nzx, nzy;
      z_next(St, gzx, gzy, max(im, 0), nzx, nzy);
      Vec<4> gyx = vzero<4>(), gyz, nyx = vzero<4>(), nyz;
      if (pro) {
        gy_flux(L4{}, NoW{}, a0[0], a0[2], cb0, ye, yon, cy, oy + im * ncp * zs,
                glob(L4{}, psEy + oy + im * ncp * zs, qy, col + (long long)im * ps), gyx, gyz);
        gy_flux(L4{}, NoW{}, vld<4>(St + o + EW), vld<4>(St + o + EW + 2 * CE), vld<4>(St + o + EW + CB), ye1, ynon, cyn,
                oyn + im * ncp * zs, glob(L4{}, psEy + oyn + im * ncp * zs, qy, col + zs + (long long)im * ps), nyx, nyz);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) a0[c] = vld<4>(S1 + o + c * CE);
      cb0 = vld<4>(S1 + o + CB);
      if (own) {
        xbase = 0;
        const bool on = xslab(xa, cx, xbase);
        gx_flux(L4{}, a0[1], a0[2], cb0, __ldg(xe_tab + xa), on, true, cx, xbase + jk,
                glob(L4{}, psEx + xbase + jk, qx, col + (long long)xa * ps), gxy, gxz);
      }
      if (pro) {
        const long long e = col + (long long)im * ps;
        const Vec<4> h1 = vld<4>(&S.ho[0][oh + D::CH]), h2 = vld<4>(&S.ho[0][oh + 2 * D::CH]), ch = ch_at(e);
        Vec<4> hy, hz;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          hy[l] = curl_t(h1[l], pxz[l], gxz[l], gzx[l], l < 3 ? gzx[l < 3 ? l + 1 : l] : nzx);
          hz[l] = curl_t(h2[l], gyx[l], nyx[l], pxy[l], gxy[l]);
        }
        h_cot(pmask, ptail, im, j, k, [&](int l, int c, float g) {
#pragma unroll
          for (int t = 0; t < 4; ++t)
            if (t == l) {
              if (c == 1) hy[t] = hy[t] + g;
              else if (c == 2) hz[t] = hz[t] + g;
            }
        });
        const float xh = __ldg(xh_tab + im);
        Vec<4> py, pz, one;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          one[l] = 1.f;
          py[l] = __fmul_rn(ch[l], hy[l]);
          pz[l] = __fmul_rn(ch[l], hz[l]);
          kxyp[l] = __fmul_rn(xh, py[l]);
          kxzp[l] = __fmul_rn(xh, pz[l]);
        }
        xbase = 0;
        if (CP && xslab(im, cx, xbase)) {
          const float* q = AD.aPsiH[par][0] + xbase + jk;
          float* u = AD.aPsiH[par ^ 1][0];
          rel_xy<4, +1, +1, false>(kxyp, vld<4>(q), u, cx, one, py);
          rel_xy<4, -1, -1, false>(kxzp, vld<4>(q + qx), u, cx, one, pz);
        }
      }
    }
    bar_or<NT>(false);   // the stages of plane xa-1 are free
    if (CP && own) fetch(xa);
    if (CP) cp_async_commit();
    bool bad = false;
    float xe1_n = __ldg(xe_tab + xa + 1), xh_n = __ldg(xh_tab + xa);
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
      // ---- phase A ----
      Vec<4> gzx = vzero<4>(), gzy = vzero<4>();
      const int iz = oz + i * ny * n4;
      if (own)
        gz_flux(L4{}, Wr{}, a0[0], a0[1], cb0, vld<4>(&S.zt[0][4 * zq]), zon, zp, iz,
                [&](int q) { return q == 2 ? sl(4) : sl(q); }, gzx, gzy);
      float nzx, nzy;
      z_next(St, gzx, gzy, i, nzx, nzy);
      Vec<4> kyx = vzero<4>(), kyz = vzero<4>(), kzx = vzero<4>(), kzy = vzero<4>(), kxy = vzero<4>(), kxz = vzero<4>();
      if (own) {
        Vec<4> gyx, gyz, nyx, nyz, g1xy, g1xz;
        gy_flux(L4{}, Wr{}, a0[0], a0[2], cb0, ye, yon, cy, oy + i * ncp * zs,
                [&](int q) { return q == 2 ? sl(4) : sl(zon ? 5 + q : q); }, gyx, gyz);
        gy_flux(L4{}, NoW{}, vld<4>(St + o + EW), vld<4>(St + o + EW + 2 * CE), vld<4>(St + o + EW + CB), ye1, ynon, cyn,
                oyn + i * ncp * zs,
                [&](int q) {
                  if (q == 2) return vld<4>(P.ce + e + zs);
                  return vld<4>(zon ? psEy + oyn + i * ncp * zs + q * qy : slot + (5 + q) * SS);
                }, nyx, nyz);
        gx_flux(L4{}, vld<4>(S1 + o + CE), vld<4>(S1 + o + 2 * CE), vld<4>(S1 + o + CB), xe1, x1on, i + 1 < xb, cx1,
                xbase1 + jk,
                [&](int q) {
                  if (q == 2) return vld<4>((zon || yon) ? P.ce + e + ps : slot + 4 * SS);
                  return vld<4>((zon || yon) ? psEx + xbase1 + jk + q * qx : slot + q * SS);
                }, g1xy, g1xz);
        Vec<4> hx = vld<4>(Ho), hy = vld<4>(Ho + D::CH), hz = vld<4>(Ho + 2 * D::CH);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          hx[l] = curl_t(hx[l], gzy[l], l < 3 ? gzy[l < 3 ? l + 1 : l] : nzy, gyz[l], nyz[l]);
          hy[l] = curl_t(hy[l], gxz[l], g1xz[l], gzx[l], l < 3 ? gzx[l < 3 ? l + 1 : l] : nzx);
          hz[l] = curl_t(hz[l], gyx[l], nyx[l], gxy[l], g1xy[l]);
        }
        gxy = g1xy;
        gxz = g1xz;
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
            al[0][l] = a0[0][l];
            al[1][l] = a0[1][l];
            al[2][l] = a0[2][l];
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
        // p = ch aH1 and its fluxes
        const Vec<4> ch = ch_at(e), zh = vld<4>(&S.zt[1][4 * zq]);
        Vec<4> one;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          one[l] = 1.f;
          hx[l] = __fmul_rn(ch[l], hx[l]);
          hy[l] = __fmul_rn(ch[l], hy[l]);
          hz[l] = __fmul_rn(ch[l], hz[l]);
          kyx[l] = __fmul_rn(yh, hx[l]);
          kzx[l] = __fmul_rn(zh[l], hx[l]);
          kxy[l] = __fmul_rn(xh, hy[l]);
          kzy[l] = __fmul_rn(zh[l], hy[l]);
          kyz[l] = __fmul_rn(yh, hz[l]);
          kxz[l] = __fmul_rn(xh, hz[l]);
        }
        if (CP && xon) {   // (hy <- ez, +1, q0), (hz <- ey, -1, q1)
          const float* q = AD.aPsiH[par][0] + xbase + jk;
          float* u = AD.aPsiH[par ^ 1][0] + xbase + jk;
          const bool far = zon || yon;
          rel_xy<4, +1, +1, true>(kxy, vld<4>(far ? q : slot + 2 * SS), u, cx, one, hy);
          rel_xy<4, -1, -1, true>(kxz, vld<4>(far ? q + qx : slot + 3 * SS), u + qx, cx, one, hz);
        }
        if (CP && yon) {   // (hx <- ez, -1, q0), (hz <- ex, +1, q1)
          const int iy = oy + i * ncp * zs;
          const float* q = AD.aPsiH[par][1] + iy;
          float* u = AD.aPsiH[par ^ 1][1] + iy;
          rel_xy<4, -1, -1, true>(kyx, vld<4>(zon ? q : slot + 2 * SS), u, cy, one, hx);
          rel_xy<4, +1, +1, true>(kyz, vld<4>(zon ? q + qy : slot + 3 * SS), u + qy, cy, one, hz);
        }
        if (CP && zon) {   // (hx <- ey, +1, q0), (hy <- ex, -1, q1)
          float* u = AD.aPsiH[par ^ 1][2] + iz;
          const Vec<4> b = vld<4>(zp), c = vld<4>(zp + ZPS), km = vld<4>(zp + 2 * ZPS);
          rel_z<4, +1, +1, true>(kzx, sl(2), u, zon, b, c, km, one, hx);
          rel_z<4, -1, -1, true>(kzy, sl(3), u + qz, zon, b, c, km, one, hy);
        }
      }
      if (CP && own && i + 1 < xb) fetch(i + 1);
      if (CP) cp_async_commit();
      const int ks = i & 1;
      if (r + 1 < TY) {
        vst<4>(&S.k[ks][0][r + 1][4 * zq], kyx);
        vst<4>(&S.k[ks][1][r + 1][4 * zq], kyz);
      }
      if (bar_or<NT>(bad)) { bad = true; break; }
      bad = !wait(5 + sC(i));
      // ---- phase B ----
      float zmx = __shfl_up_sync(0xffffffffu, kzx[3], 1, ZQ), zmy = __shfl_up_sync(0xffffffffu, kzy[3], 1, ZQ);
      if (own) {
        if (first_q) { zmx = S.kc[ks][0][r]; zmy = S.kc[ks][1][r]; }
        const Vec<4> myx = vld<4>(&S.k[ks][0][r][4 * zq]), myz = vld<4>(&S.k[ks][1][r][4 * zq]);
        const Vec<4> cav = vld<4>(&S.ca[sC(i)][oc]);
        Vec<4> ex, ey, ez;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          ex[l] = curl_t(__fmul_rn(cav[l], a0[0][l]), kzy[l], l ? kzy[l ? l - 1 : 0] : zmy, kyz[l], myz[l]);
          ey[l] = curl_t(__fmul_rn(cav[l], a0[1][l]), kxz[l], kxzp[l], kzx[l], l ? kzx[l ? l - 1 : 0] : zmx);
          ez[l] = curl_t(__fmul_rn(cav[l], a0[2][l]), kyx[l], myx[l], kxy[l], kxyp[l]);
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
      kxyp = kxy;
      kxzp = kxz;
#pragma unroll
      for (int c = 0; c < 3; ++c) a0[c] = vld<4>(S1 + o + c * CE);
      cb0 = vld<4>(S1 + o + CB);
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
    // G of the x direction on plane i: row Gxy, column Gxz
    Vec<4> gxr = vzero<4>();
    float gxc = 0.f;
    auto gx_halo = [&](const float* St, int p, float xe, Vec<4>& gr, float& gc) {
      float4 cx;
      int xbase = 0;
      const bool xs = xslab(p, cx, xbase);
      const long long e = col + (long long)p * ps;
      if (row) {
        Vec<4> dummy;
        gx_flux(L4{}, vld<4>(St + o + CE), vld<4>(St + o + 2 * CE), vld<4>(St + o + CB), xe, xs, false, cx, xbase + jk,
                glob(L4{}, psEx + xbase + jk, qx, e), gr, dummy);
      } else if (colm) {
        Vec<1> g, d;
        gx_flux(L1{}, vld<1>(St + o + CE), vld<1>(St + o + 2 * CE), vld<1>(St + o + CB), xe, xs, false, cx, xbase + jk,
                glob(L1{}, psEx + xbase + jk, qx, e), d, g);
        gc = g[0];
      }
    };
    gx_halo(&S.e[1][0], xa, __ldg(xe_tab + xa), gxr, gxc);
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
    float xe1_n = __ldg(xe_tab + xa + 1);
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
      Vec<4> g1r = vzero<4>();
      float g1c = 0.f;
      gx_halo(S1, i + 1, xe1, g1r, g1c);
      if (is_row) {
        Vec<4> kyx = vzero<4>(), kyz = vzero<4>(), gzx, gzy = vzero<4>(), ex, ez, cb;
        if (row) {
          ex = vld<4>(St + o);
          ez = vld<4>(St + o + 2 * CE);
          cb = vld<4>(St + o + CB);
          gz_flux(L4{}, NoW{}, ex, vld<4>(St + o + CE), cb, vld<4>(&S.zt[0][4 * lane]), zon_r, &S.zp[0][4 * lane], iz,
                  globz(L4{}, psEz + iz, qz, e, zon_r), gzx, gzy);
        }
        float nzy = __shfl_down_sync((1u << ZQ) - 1u, gzy[0], 1, ZQ);
        if (row) {
          if (lane == ZQ - 1) {
            float d;
            gz_after(St, o + 4, irow, e + 4, d, nzy);
          }
          Vec<4> gyx, gyz, nyx, nyz;
          gy_flux(L4{}, NoW{}, ex, ez, cb, ye, yon, cy, oy + i * ncp * zs, glob(L4{}, psEy + oy + i * ncp * zs, qy, e), gyx, gyz);
          gy_flux(L4{}, NoW{}, vld<4>(St + o + EW), vld<4>(St + o + EW + 2 * CE), vld<4>(St + o + EW + CB), ye1, ynon, cyn,
                  oyn + i * ncp * zs, glob(L4{}, psEy + oyn + i * ncp * zs, qy, e + zs), nyx, nyz);
          Vec<4> hx = vld<4>(Ho + 4 * lane), hz = vld<4>(Ho + 2 * D::CH + 4 * lane);
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            hx[l] = curl_t(hx[l], gzy[l], l < 3 ? gzy[l < 3 ? l + 1 : l] : nzy, gyz[l], nyz[l]);
            hz[l] = curl_t(hz[l], gyx[l], nyx[l], gxr[l], g1r[l]);
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
          Vec<4> one;
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            const float ch = ch_arr ? ch_arr[e + l] : ch0;
            one[l] = 1.f;
            hx[l] = __fmul_rn(ch, hx[l]);
            hz[l] = __fmul_rn(ch, hz[l]);
            kyx[l] = __fmul_rn(yh, hx[l]);
            kyz[l] = __fmul_rn(yh, hz[l]);
          }
          if (CP && yon) {
            const float* q = AD.aPsiH[par][1] + oy + i * ncp * zs;
            rel_xy<4, -1, -1, false>(kyx, vld<4>(q), nullptr, cy, one, hx);
            rel_xy<4, +1, +1, false>(kyz, vld<4>(q + qy), nullptr, cy, one, hz);
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
          Vec<1> ze, gzx, gzy, nzx, nzy, gyx, gyz, nyx, nyz;
          ze[0] = ze_c;
          gzx = vscale<1>(ze, cb, ex);
          gzy = vscale<1>(ze, cb, ey);
          if (CP && zon_c) {
            Vec<1> ce = vld<1>(P.ce + e);
            rel_xy<1, -1, -1, false>(gzx, vld<1>(psEz + iz), nullptr, czc, ce, ex);
            rel_xy<1, +1, +1, false>(gzy, vld<1>(psEz + iz + qz), nullptr, czc, ce, ey);
          }
          ze[0] = S.zt[0][0];
          gz_flux(L1{}, NoW{}, vld<1>(St + o + 1), vld<1>(St + o + 1 + CE), vld<1>(St + o + 1 + CB), ze, zon_0, &S.zp[0][0],
                  irow + zoff0, glob(L1{}, psEz + irow + zoff0, qz, e + 1), nzx, nzy);
          gy_flux(L1{}, NoW{}, ex, ez, cb, ye, yon, cy, oy + i * ncp * zs, glob(L1{}, psEy + oy + i * ncp * zs, qy, e), gyx, gyz);
          gy_flux(L1{}, NoW{}, vld<1>(St + o + EW), vld<1>(St + o + EW + 2 * CE), vld<1>(St + o + EW + CB), ye1, ynon, cyn,
                  oyn + i * ncp * zs, glob(L1{}, psEy + oyn + i * ncp * zs, qy, e + zs), nyx, nyz);
          Vec<1> hx, hy, one;
          hx[0] = curl_t(hc0, gzy[0], nzy[0], gyz[0], nyz[0]);
          hy[0] = curl_t(hc1, gxc, g1c, gzx[0], nzx[0]);
          if (pmask || ptail)
            h_cot(pmask, ptail, i, j, k, [&](int l, int c, float g) {
              if (l != 0) return;
              if (c == 0) hx[0] = hx[0] + g;
              else if (c == 1) hy[0] = hy[0] + g;
            });
          const float ch = ch_arr ? ch_arr[e] : ch0;
          one[0] = 1.f;
          hx[0] = __fmul_rn(ch, hx[0]);
          hy[0] = __fmul_rn(ch, hy[0]);
          Vec<1> vx, vy;
          vx[0] = __fmul_rn(zh_c, hx[0]);
          vy[0] = __fmul_rn(zh_c, hy[0]);
          if (CP && zon_c) {
            const float* q = AD.aPsiH[par][2] + iz;
            rel_xy<1, +1, +1, false>(vx, vld<1>(q), nullptr, czc, one, hx);
            rel_xy<1, -1, -1, false>(vy, vld<1>(q + qz), nullptr, czc, one, hy);
          }
          kzx = vx[0];
          kzy = vy[0];
        }
        S.kc[ks][0][lane - ZQ] = kzx;
        S.kc[ks][1][lane - ZQ] = kzy;
      }
      gxr = g1r;
      gxc = g1c;
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
