// Forward time step, four cells per thread.
//
// One CTA owns a tile of TY rows x 4*ZQ columns of the (y, z) plane and
// marches along x over a range [xa, xb).  A main thread owns one row and four
// consecutive z columns (every field, coefficient and x/y psi access of it is
// one 16-byte access); one further warp computes the H the tile needs from its
// low y row and low z column and issues the E boxes.  Per plane i:
//   1. E of planes i and i+1 (one-cell halo), H^{n-1/2} of plane i (with the low
//      row) and ca, cb of plane i are in shared memory: TMA boxes, three E
//      stages, two of the others, each refilled as soon as its plane is done;
//   2. H^{n+1/2} on the tile and on the halo row and column
//      (rfx/core/yee.py:226-291 / :411-453, rfx/boundaries/cpml.py:804-1065);
//      hx and hz go to shared memory for the next row, z neighbours come from
//      the adjacent lane;
//   3. one block barrier (the exchange array has two slots, so the next
//      plane's H never overwrites values still being read);
//   4. E^{n+1} on the tile (rfx/core/yee.py:347-404 / :456-492,
//      rfx/boundaries/cpml.py:522-801), PEC faces (rfx/boundaries/pec.py:13-47),
//      PEC edge mask (pec.py:179-208), sources, probes
//      (rfx/simulation.py:1518-1567) and the gradient history.
// psi of slab cells (and their ce) is prefetched one plane ahead into slots of
// the thread's own (cp.async), so no slab cell waits on a global load.  Every
// product and sum is written as a rounding intrinsic, so every instantiation
// computes the same bits.
//
// What bounds it: CPML-free items HBM and the latency of one plane (a 257^3 grid
// without CPML 183 us a step, 5.2 TB/s of the 56 bytes per cell); CPML items the
// instructions of the slab terms at 14 warps per SM.  One cell per thread issued
// 360 (CPML-free) and 525 instructions per cell against 130 and 250 here and read
// psi 4 bytes at a time.  24 x 32 tiles take two CTAs per SM (seven warps, 128
// registers, up to 110 KB); taller ones leave one, lower ones reread more halo.
// Measured, one cell per thread -> here: 217x217x121 with CPML 12 182 -> 122 us a
// step, 131x147x103 with CPML 8 96 -> 62, 277^3 with CPML 10 about 325 -> 312 (of
// which CPML-free items 160).  H and the coefficients loaded into registers one
// plane ahead instead of staged: 263 us instead of 183 on 257^3.
#include "rfxb_common.cuh"
#include "rfxb_vec.cuh"

namespace rfxb {

template <int TY, int ZQ>
struct VDims {
  static constexpr int TZ = 4 * ZQ;
  static constexpr int MAIN = TY * ZQ;          // threads that own cells
  static constexpr int NT = MAIN + 32;          // plus the halo warp
  static constexpr int EW = TZ + 8;             // staged E row: z in [z0 - 4, z0 + TZ + 4)
  static constexpr int CE = (TY + 2) * EW;      // component stride of an E stage
  static constexpr int CH = (TY + 1) * TZ;      // of an H stage
  static constexpr int CC = TY * TZ;            // of a coefficient stage
  static_assert(MAIN % 32 == 0 && ZQ + TY <= 32, "the halo warp holds the row and the column");
};

// Slots of the prefetched psi of a thread's cells (four floats each): y psi
// (or, off the y slabs, x psi) H q0, q1, E q0, q1; z psi H q0, q1, E q0, q1; ce.  A
// slot is written (cp.async) and read by its own thread only.
#define RFXB_PSLOTS 9

template <int TY, int ZQ, bool CP>
struct __align__(128) VSmem {
  using D = VDims<TY, ZQ>;
  float e[RFXB_VNST][vup32(3 * D::CE)];   // E^n, rows y0-1 .. y0+TY
  float ho[2][3 * D::CH];                 // H^{n-1/2}, rows y0-1 .. y0+TY-1
  float cab[2][2 * D::CC];                // ca, cb of the tile
  float h[2][2][TY][D::TZ];               // hx, hz of plane i in slot i & 1: rows y0-1 .. y0+TY-2
  float hc[2][2][TY];                     // hx, hy of column z0-1
  float zt[2][D::TZ];                     // zh, ze of the tile's columns
  float zp[3][D::TZ];                     // z profile of the columns (b, c, km)
  float ps[CP ? RFXB_PSLOTS : 1][CP ? D::MAIN : 1][4];
  RfxbInst P;
  unsigned long long mbar[RFXB_VBARS];    // E stages, H stages, coefficient stages
};

// Position of a cell (or four) in the CPML slabs of the axes other than x.
struct VSlab {
  bool y = false;              // in a y slab
  unsigned z = 0u;             // cells in a z slab (zslab_of)
  float4 cy;                   // y profile (b, c, km, w)
  int oy = 0;                  // y psi element of (q 0, plane 0): + i * ncp * zs
  int oz = 0;                  // z psi element of the first cell's (q 0, plane 0): + i * ny * ncp4
};

// One psi term of an x or y slab from the differences d and the old psi p:
// f += SGN s (psi' + km g), psi' written to `out` when WRITE; with K,
// k += SGN (psi' + km g) (the gradient history's correction before its scaling).
template <int L, int SGN, bool WRITE, bool K>
__device__ __forceinline__ void psi_xy(Vec<L>& f, const Vec<L>& s, Vec<L> p, float* out, const float4& c,
                                       const Vec<L>& d, Vec<L>& k, bool rec = false) {
#pragma unroll
  for (int l = 0; l < L; ++l) {
    const float g = __fmul_rn(d[l], c.w);
    p[l] = psi_next(c.x, p[l], c.y, g);
    f[l] = psi_add(f[l], SGN > 0 ? s[l] : -s[l], p[l], c.z, g);
  }
  if (K && rec) {
#pragma unroll
    for (int l = 0; l < L; ++l) {
      const float t = __fmaf_rn(c.z, __fmul_rn(d[l], c.w), p[l]);
      k[l] = SGN > 0 ? __fadd_rn(k[l], t) : __fsub_rn(k[l], t);
    }
  }
  if (WRITE) vst<L>(out, p);
}
// The same for a z slab: profile per column, psi at the columns' layers.
template <int L, int SGN, bool WRITE, bool K>
__device__ __forceinline__ void psi_z(Vec<L>& f, const Vec<L>& s, Vec<L> p, float* out, unsigned m, const float* zp,
                                      int zstride, float w, const Vec<L>& d, Vec<L>& k, bool rec = false) {
  const Vec<L> b = vld<L>(zp), c = vld<L>(zp + zstride), km = vld<L>(zp + 2 * zstride);
#pragma unroll
  for (int l = 0; l < L; ++l) {
    const float g = __fmul_rn(d[l], w);
    p[l] = psi_next(b[l], p[l], c[l], g);
    if ((m >> l) & 1u) f[l] = psi_add(f[l], SGN > 0 ? s[l] : -s[l], p[l], km[l], g);
  }
  if (K && rec) {
#pragma unroll
    for (int l = 0; l < L; ++l) {
      if (!((m >> l) & 1u)) continue;
      const float t = __fmaf_rn(km[l], __fmul_rn(d[l], w), p[l]);
      k[l] = SGN > 0 ? __fadd_rn(k[l], t) : __fsub_rn(k[l], t);
    }
  }
  if (WRITE) zpsi_store<L>(out, m, p);
}

// H^{n+1/2} of L columns from the staged planes A (i) and B (i+1): `o` is the
// position of the first column in component 0 of an E stage.  e0: E of the cells
// on plane i; exz, eyz: ex and ey of the column after the last; hold(c): old H;
// old(axis, q): old psi.  One component after the other, so that only its two
// differences are held.
template <int L, int MASK, bool CP, bool WRITE, int EW, int CE, class Hold, class Old>
__device__ __forceinline__ void h_vec(const float* A, const float* B, int o, const Vec<L>* e0, float exz, float eyz,
                                      Hold&& hold, Old&& old, float xh, float yh, const Vec<L>& zh, const Vec<L>& ch,
                                      const RfxbInst& P, int par, bool xon, const float4& cx, int ox, const VSlab& S,
                                      const float* zp, float wz, int i, int qx, int qy, int qz, int ncp, Vec<L>& hx, Vec<L>& hy,
                                      Vec<L>& hz) {
  constexpr int ZS = EW - 8;
  const int iy = S.oy + i * ncp * P.zs, iz = S.oz + i * P.ny * P.ncp4;
  Vec<L> none;
  if (MASK & 1) {   // Hx -= ch psi(dEz/dy) [y q0], Hx += ch psi(dEy/dz) [z q0]
    Vec<L> gy = vld<L>(A + o + 2 * CE + EW), gz;
    const Vec<L> ho = hold(0);
#pragma unroll
    for (int l = 0; l < L; ++l) {
      gy[l] = gy[l] - e0[2][l];
      gz[l] = (l < L - 1 ? e0[1][l + 1 < L ? l + 1 : l] : eyz) - e0[1][l];
      hx[l] = yee_h(ho[l], ch[l], yee_diff2(gy[l], yh, gz[l], zh[l]));
    }
    if (CP && S.y) psi_xy<L, -1, WRITE, false>(hx, ch, old(1, 0), P.psH[par ^ 1][1] + iy, S.cy, gy, none);
    if (CP && S.z)
      psi_z<L, +1, WRITE, false>(hx, ch, old(2, 0), P.psH[par ^ 1][2] + iz, S.z, zp, ZS, wz, gz, none);
  }
  if (MASK & 2) {   // Hy += ch psi(dEz/dx) [x q0], Hy -= ch psi(dEx/dz) [z q1]
    Vec<L> gx = vld<L>(B + o + 2 * CE), gz;
    const Vec<L> ho = hold(1);
#pragma unroll
    for (int l = 0; l < L; ++l) {
      gx[l] = gx[l] - e0[2][l];
      gz[l] = (l < L - 1 ? e0[0][l + 1 < L ? l + 1 : l] : exz) - e0[0][l];
      hy[l] = yee_h(ho[l], ch[l], yee_diff2(gz[l], zh[l], gx[l], xh));
    }
    if (CP && xon) psi_xy<L, +1, WRITE, false>(hy, ch, old(0, 0), P.psH[par ^ 1][0] + ox, cx, gx, none);
    if (CP && S.z)
      psi_z<L, -1, WRITE, false>(hy, ch, old(2, 1), P.psH[par ^ 1][2] + iz + qz, S.z, zp, ZS, wz, gz, none);
  }
  if (MASK & 4) {   // Hz -= ch psi(dEy/dx) [x q1], Hz += ch psi(dEx/dy) [y q1]
    Vec<L> gx = vld<L>(B + o + CE), gy = vld<L>(A + o + EW);
    const Vec<L> ho = hold(2);
#pragma unroll
    for (int l = 0; l < L; ++l) {
      gx[l] = gx[l] - e0[1][l];
      gy[l] = gy[l] - e0[0][l];
      hz[l] = yee_h(ho[l], ch[l], yee_diff2(gx[l], xh, gy[l], yh));
    }
    if (CP && xon) psi_xy<L, -1, WRITE, false>(hz, ch, old(0, 1), P.psH[par ^ 1][0] + ox + qx, cx, gx, none);
    if (CP && S.y) psi_xy<L, +1, WRITE, false>(hz, ch, old(1, 1), P.psH[par ^ 1][1] + iy + qy, S.cy, gy, none);
  }
}

// One work item.  CP false: neither the tile (its halo row and column
// included) nor planes xa-1 .. xb-1 lie in a CPML slab.  Returns false when a
// bounded wait ran out: the status word is then set and every box the CTA
// issued has been waited for, so the caller must leave.
template <int TY, int ZQ, bool CP>
__device__ __forceinline__ bool fwdv_item(VSmem<TY, ZQ, CP>& S, const RfxbInst* __restrict__ insts, const RfxbWork w,
                                          const CUtensorMap* __restrict__ maps, int map0, int n, int sel,
                                          StepPhases& ph, const StepFault& fault, bool first_item) {
  using D = VDims<TY, ZQ>;
  constexpr int EW = D::EW, CE = D::CE, NT = D::NT, SS = 4 * D::MAIN;
  const int tid = threadIdx.x;
  const int y0 = w.y0, z0 = w.z0, xa = w.xa, xb = w.xb;
  const int fin = sel_in(sel), fout = sel_out(sel), par = sel_psi(sel);
  // The boxes of this item.  Plane p: E in stage (p - xa + 1) % 3, H in stage
  // (p - xa + 1) % 2, coefficients in stage (p - xa) % 2; barriers 0-2, 3-4, 5-6.
  const bool producer = tid == NT - 1;
  const CUtensorMap* tm = maps + (size_t)w.inst * RFXB_NMAPS + map0;   // [0..2] E, [3..5] H of buffer fin, [6] ca/cb
  const uint32_t ph0 = ph.stage;
  auto sE = [&](int p) { return (p - xa + 1) % RFXB_VNST; };
  auto sH = [&](int p) { return (p - xa + 1) & 1; };
  auto sC = [&](int p) { return (p - xa) & 1; };
  auto issue_e = [&](int p) {
    const uint32_t mb = smem_u32(&S.mbar[sE(p)]);
    mbar_expect_tx(mb, 4u * 3 * CE);
    tma_load_4d(smem_u32(&S.e[sE(p)][0]), tm + fin, z0 - 4, y0, p + 1, 0, mb);
  };
  auto issue_h = [&](int p) {
    const uint32_t mb = smem_u32(&S.mbar[3 + sH(p)]);
    mbar_expect_tx(mb, 4u * 3 * D::CH);
    tma_load_4d(smem_u32(&S.ho[sH(p)][0]), tm + 3 + fin, z0, y0, p + 1, 3, mb);
  };
  auto issue_c = [&](int p) {
    const uint32_t mb = smem_u32(&S.mbar[5 + sC(p)]);
    mbar_expect_tx(mb, 4u * 2 * D::CC);
    tma_load_4d(smem_u32(&S.cab[sC(p)][0]), tm + 6, z0, y0 + 1, p + 1, 0, mb);
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
  __syncthreads();
  const RfxbInst& P = S.P;
  const int wlim = fault.wait_limit;
  const int nx = P.nx, ny = P.ny, nz = P.nz, zs = P.zs, ncp = P.ncp, n4 = P.ncp4;
  const long long ps = P.ps, cs = P.cs;
  const float* Fi = P.F[fin][0];
  float* Fo = P.F[fout][0];
  const unsigned ax = CP && ncp > 0 ? P.cpml_axes : 0u;
  const bool cpx = ax & 1u, cpy = ax & 2u, cpz = ax & 4u;
  const int jb = ny - ncp, kb = nz - ncp;
  // q strides of the psi arrays (the sides are two of them apart)
  const int qx = ncp * ny * zs, qy = nx * ncp * zs, qz = nx * ny * n4;

  // the columns' z tables
#pragma unroll 1
  for (int t = tid; t < D::TZ; t += NT) {
    const int k = z0 + t;
    S.zt[0][t] = k < nz ? __ldg(P.zh + k) : 0.f;
    S.zt[1][t] = k < nz ? __ldg(P.ze + k) : 0.f;
    if (CP) {
      float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
      if (cpz && k < ncp) c = __ldg(P.cpu + 4 * ncp + k);
      else if (cpz && k >= kb && k < nz) c = __ldg(P.cpu + 5 * ncp + (k - kb));
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
  const int r = is_main ? tid / ZQ : 0;
  const int zq = is_main ? tid % ZQ : (tid - D::MAIN);   // halo warp: lane
  const float ch0 = P.ch0;
  const float* ch_arr = P.ch;
  const float* xh_tab = P.xh;
  const float* xe_tab = P.xe;

  // position of a row j / columns k.. in the slabs
  auto place = [&](VSlab& B, int j, int k, int cells) {
    if (!CP) return;
    if (cpy && (j < ncp || j >= jb)) {
      const int sd = j < ncp ? 0 : 1, s = sd ? j - jb : j;
      B.y = true;
      B.cy = __ldg(P.cpu + (2 + sd) * ncp + s);
      B.oy = 2 * sd * qy + s * zs + k;
    }
    if (cpz) {
      int off;
      B.z = cells == 4 ? zslab_of<4>(k, ncp, kb, nz, 2 * qz, off) : zslab_of<1>(k, ncp, kb, nz, 2 * qz, off);
      B.oz = j * n4 + off;
    }
  };
  // x slab of plane p
  auto xslab = [&](int p, float4& c, int& base) -> bool {
    if (!CP || !cpx || p < 0 || (p >= ncp && p < nx - ncp) || p >= nx) return false;
    const int sd = p < ncp ? 0 : 1, s = sd ? p - (nx - ncp) : p;
    c = __ldg(P.cpu + sd * ncp + s);
    base = 2 * sd * qx + s * ny * zs;
    return true;
  };
  // Prefetch of the old psi of plane p into this thread's slots (x psi only off
  // the y slabs), H side and E side with ce.
  float* const slot = &S.ps[0][CP && is_main ? tid : 0][0];
  auto in_xslab = [&](int p) { return CP && cpx && p >= 0 && p < nx && (p < ncp || p >= nx - ncp); };
  auto xbase_of = [&](int p) {   // x psi element of (plane p's layer, q 0)
    const int sd = p < ncp ? 0 : 1, s = sd ? p - (nx - ncp) : p;
    return 2 * sd * qx + s * ny * zs;
  };
  auto getz = [&](float* d, const float* p, unsigned m) {
    if (m & 256u) { cp_async16(d, p); return; }
#pragma unroll
    for (int l = 0; l < 4; ++l)
      if ((m >> l) & 1u) cp_async4(d + l, p + l);
  };
  auto fetch = [&](float* const* ps, int p, const VSlab& B, int jk, int first) {   // first: 0 H side, 2 E side
    if (B.y) {
      const float* q = ps[1] + B.oy + p * ncp * zs;
      cp_async16(slot + first * SS, q);
      cp_async16(slot + (first + 1) * SS, q + qy);
    } else if (in_xslab(p)) {
      const float* q = ps[0] + xbase_of(p) + jk;
      cp_async16(slot + first * SS, q);
      cp_async16(slot + (first + 1) * SS, q + qx);
    }
    if (B.z) {
      const float* q = ps[2] + B.oz + p * ny * n4;
      getz(slot + (4 + first) * SS, q, B.z);
      getz(slot + (5 + first) * SS, q + qz, B.z);
    }
  };
  // planes xa-1 and xa have landed, the z tables are written; after a wait that
  // ran out all threads leave the loops at the same barrier
  bool bad_end;
  {
    const bool ok0 = wait(0), ok1 = wait(1), ok2 = wait(3);
    bad_end = bar_or<NT>(!(ok0 && ok1 && ok2));
  }
  if (bad_end) {
  } else if (is_main) {
    const int j = y0 + r, k = z0 + 4 * zq;
    const bool own = j < ny && k < nz;
    const int kv = min(4, nz - k);                      // cells of the four inside the grid
    const int o = (r + 1) * EW + 4 * zq + 4;
    const long long col = P.off0 + (long long)j * zs + k;
    VSlab B;
    if (own) place(B, j, k, 4);
    const int jk = j * zs + k;
    const float yh = own ? __ldg(P.yh + j) : 0.f, ye = own ? __ldg(P.ye + j) : 0.f;
    const float* zp = &S.zp[0][4 * zq];
    const float wz = CP ? P.zw[k >= ncp] : 0.f;
    const bool last_q = zq == ZQ - 1, first_q = zq == 0;
    // sources and probes in this thread's columns
    unsigned smask = 0u, pmask = 0u;
    if (own) {
#pragma unroll 1
      for (int s = 0; s < min(P.nsrc, 32); ++s) {
        const int4 c = __ldg(P.src + s);
        if (c.y == j && c.z >= k && c.z < k + 4) smask |= 1u << s;
      }
#pragma unroll 1
      for (int s = 0; s < min(P.nprb, 32); ++s) {
        const int4 c = __ldg(P.prb + s);
        if (c.y == j && c.z >= k && c.z < k + 4) pmask |= 1u << s;
      }
    }
    const bool tail = P.nsrc > 32 || P.nprb > 32;
    const unsigned pec = P.pec_axes;
    const bool pec_j = (pec & 2u) && (j == 0 || j == ny - 1);
    const bool pec_k = (pec & 4u) && (k == 0 || k + 3 >= nz - 1);
    const bool in_hist = P.hist != nullptr && (n - P.hist_step0) >= 0 && (n - P.hist_step0) < P.hist_nsteps &&
                         j >= P.hb[2] && j < P.hb[3] && k < P.hb[5] && k + 4 > P.hb[4];
    const unsigned char* emask = P.emask;

    Vec<4> e0[3];
    Vec<4> hx = vzero<4>(), hy = vzero<4>(), hz = vzero<4>(), hyp = vzero<4>(), hzp = vzero<4>();
    const float* E0 = &S.e[0][0];
    const int oh = (r + 1) * D::TZ + 4 * zq, oc = r * D::TZ + 4 * zq;   // this thread's place in an H / coefficient stage
    // prologue: hy, hz of plane xa-1 (its owner stores them)
    {
      const float* A = E0;
      const float* Bp = &S.e[1][0];
#pragma unroll
      for (int c = 0; c < 3; ++c) e0[c] = vld<4>(A + o + c * CE);
      const float exz = last_q ? A[o + 4] : 0.f, eyz = last_q ? A[o + 4 + CE] : 0.f;
      const float sx = __shfl_down_sync(0xffffffffu, e0[0][0], 1, ZQ);
      if (xa > 0 && own) {
        const long long e = col + (long long)(xa - 1) * ps;
        Vec<4> ch;
        if (ch_arr) ch = vld<4>(ch_arr + e);
        else {
#pragma unroll
          for (int l = 0; l < 4; ++l) ch[l] = ch0;
        }
        float4 cx;
        int xbase = 0;
        const bool xon = xslab(xa - 1, cx, xbase);
        Vec<4> t;
        const float* H = &S.ho[0][0];
        h_vec<4, 6, CP, false, EW, CE>(
            A, Bp, o, e0, last_q ? exz : sx, eyz, [&](int c) { return vld<4>(H + oh + c * D::CH); },
            [&](int a, int q) {
              const float* p = P.psH[par][a];
              if (a == 0) return vld<4>(p + xbase + jk + q * qx);
              if (a == 1) return vld<4>(p + B.oy + (xa - 1) * ncp * zs + q * qy);
              return zpsi_load<4>(p + B.oz + (xa - 1) * ny * n4 + q * qz, B.z);
            },
            __ldg(xh_tab + xa - 1), yh, vld<4>(&S.zt[0][4 * zq]), ch, P, par, xon, cx, xbase + jk, B, zp, wz, xa - 1, qx, qy, qz,
            ncp, t, hyp, hzp);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) e0[c] = vld<4>(Bp + o + c * CE);
    }
    bar_or<NT>(false);   // the stages of plane xa-1 are free
    if (CP && own) fetch(P.psH[par], xa, B, jk, 0);
    if (CP) cp_async_commit();
    if (CP && own) {
      fetch(P.psE[par], xa, B, jk, 2);
      if (B.y || B.z || in_xslab(xa)) cp_async16(slot + 8 * SS, P.ce + col + (long long)xa * ps);
    }
    if (CP) cp_async_commit();
    bool bad = false;
    float xh_n = __ldg(xh_tab + xa), xe_n = __ldg(xe_tab + xa);
    int sA = 1, sB = 2;   // stages of planes i and i+1
#pragma unroll 1
    for (int i = xa; i < xb; ++i) {
      const long long e = col + (long long)i * ps;
      float4 cx;
      int xbase = 0;
      const bool xon = own && xslab(i, cx, xbase);
      const float xh = xh_n, xe = xe_n;
      if (i + 1 < xb) { xh_n = __ldg(xh_tab + i + 1); xe_n = __ldg(xe_tab + i + 1); }
      Vec<4> ch;
      if (ch_arr) ch = own ? vld<4>(ch_arr + e) : vzero<4>();
      else {
#pragma unroll
        for (int l = 0; l < 4; ++l) ch[l] = ch0;
      }
      unsigned em = 0u;
      if (emask && own) em = *reinterpret_cast<const unsigned*>(emask + e);
      bad = !wait(sB) | bad;
      bad = !wait(3 + sH(i)) | bad;
      if (CP) cp_async_wait<1>();   // this plane's H-side psi (its E side may be in flight)
      // ---- H ----
      const float* H = &S.ho[sH(i)][0];
      const float* A = &S.e[sA][0];
      const float* Bp = &S.e[sB][0];
      {
        float exz = __shfl_down_sync(0xffffffffu, e0[0][0], 1, ZQ), eyz = __shfl_down_sync(0xffffffffu, e0[1][0], 1, ZQ);
        if (last_q) { exz = A[o + 4]; eyz = A[o + 4 + CE]; }
        if (own) {
          h_vec<4, 7, CP, true, EW, CE>(
              A, Bp, o, e0, exz, eyz, [&](int c) { return vld<4>(H + oh + c * D::CH); },
              [&](int a, int q) {
                if (a == 0 && B.y) return vld<4>(P.psH[par][0] + xbase + jk + q * qx);
                return vld<4>(slot + (a == 2 ? 4 + q : q) * SS);
              },
              xh, yh, vld<4>(&S.zt[0][4 * zq]), ch, P, par, xon, cx, xbase + jk, B, zp, wz, i, qx, qy, qz, ncp, hx, hy, hz);
          if (kv < 4) {
#pragma unroll
            for (int l = 1; l < 4; ++l)
              if (l >= kv) { hx[l] = 0.f; hy[l] = 0.f; hz[l] = 0.f; }
          }
          vst<4>(Fo + 3 * cs + e, hx);
          vst<4>(Fo + 4 * cs + e, hy);
          vst<4>(Fo + 5 * cs + e, hz);
          if (CP && i + 1 < xb) fetch(P.psH[par], i + 1, B, jk, 0);
        }
      }
      if (CP) cp_async_commit();
      const int sl = i & 1;
      if (r + 1 < TY) {
        vst<4>(&S.h[sl][0][r + 1][4 * zq], hx);
        vst<4>(&S.h[sl][1][r + 1][4 * zq], hz);
      }
      const bool any = CP && own && (xon || B.y || B.z);
      if (bar_or<NT>(bad)) { bad = true; break; }
      bad = !wait(5 + sC(i));
      if (CP) cp_async_wait<1>();   // this plane's E-side psi
      // ---- E ----
      const float hxu = __shfl_up_sync(0xffffffffu, hx[3], 1, ZQ), hyu = __shfl_up_sync(0xffffffffu, hy[3], 1, ZQ);
      if (own) {
        const float hxm = first_q ? S.hc[sl][0][r] : hxu, hym = first_q ? S.hc[sl][1][r] : hyu;
        const Vec<4> ze = vld<4>(&S.zt[1][4 * zq]);
        const float* C = &S.cab[sC(i)][0];
        const Vec<4> cav = vld<4>(C + oc), cbv = vld<4>(C + oc + D::CC);
        Vec<4> ex, ey, ez, ce, kk = vzero<4>();
        if (CP && any) ce = vld<4>(slot + 8 * SS);
        const int iy = B.oy + i * ncp * zs, iz = B.oz + i * ny * n4, ix = xbase + jk;
        const bool hist_i = in_hist && i >= P.hb[0] && i < P.hb[1];
        float hl[2][3][4];   // curls and CPML corrections for the gradient history
        auto keep = [&](int c, const Vec<4>& curl) {
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            hl[0][c][l] = curl[l];
            hl[1][c][l] = kk[l];
          }
          kk = vzero<4>();
        };
        {   // Ex += ce psi(dHz/dy) [y q0], Ex -= ce psi(dHy/dz) [z q0]
          Vec<4> gy = vld<4>(&S.h[sl][1][r][4 * zq]), gz, cu;
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            gy[l] = hz[l] - gy[l];
            gz[l] = hy[l] - (l ? hy[l ? l - 1 : 0] : hym);
            cu[l] = yee_diff2(gy[l], ye, gz[l], ze[l]);
            ex[l] = yee_e(cav[l], e0[0][l], cbv[l], cu[l]);
          }
          if (CP && B.y) psi_xy<4, +1, true, true>(ex, ce, vld<4>(slot + 2 * SS), P.psE[par ^ 1][1] + iy, B.cy, gy, kk, hist_i);
          if (CP && B.z)
            psi_z<4, -1, true, true>(ex, ce, vld<4>(slot + 6 * SS), P.psE[par ^ 1][2] + iz, B.z, zp, 4 * ZQ, wz, gz, kk, hist_i);
          if (hist_i) keep(0, cu);
        }
        {   // Ey -= ce psi(dHz/dx) [x q0], Ey += ce psi(dHx/dz) [z q1]
          Vec<4> gx, gz, cu;
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            gx[l] = hz[l] - hzp[l];
            gz[l] = hx[l] - (l ? hx[l ? l - 1 : 0] : hxm);
            cu[l] = yee_diff2(gz[l], ze[l], gx[l], xe);
            ey[l] = yee_e(cav[l], e0[1][l], cbv[l], cu[l]);
          }
          if (CP && xon) psi_xy<4, -1, true, true>(ey, ce, vld<4>(B.y ? P.psE[par][0] + ix : slot + 2 * SS), P.psE[par ^ 1][0] + ix, cx, gx, kk, hist_i);
          if (CP && B.z)
            psi_z<4, +1, true, true>(ey, ce, vld<4>(slot + 7 * SS), P.psE[par ^ 1][2] + iz + qz, B.z, zp, 4 * ZQ, wz, gz, kk, hist_i);
          if (hist_i) keep(1, cu);
        }
        {   // Ez += ce psi(dHy/dx) [x q1], Ez -= ce psi(dHx/dy) [y q1]
          Vec<4> gx, gy = vld<4>(&S.h[sl][0][r][4 * zq]), cu;
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            gx[l] = hy[l] - hyp[l];
            gy[l] = hx[l] - gy[l];
            cu[l] = yee_diff2(gx[l], xe, gy[l], ye);
            ez[l] = yee_e(cav[l], e0[2][l], cbv[l], cu[l]);
          }
          if (CP && xon)
            psi_xy<4, +1, true, true>(ez, ce, vld<4>(B.y ? P.psE[par][0] + ix + qx : slot + 3 * SS), P.psE[par ^ 1][0] + ix + qx, cx, gx, kk, hist_i);
          if (CP && B.y)
            psi_xy<4, -1, true, true>(ez, ce, vld<4>(slot + 3 * SS), P.psE[par ^ 1][1] + iy + qy, B.cy, gy, kk, hist_i);
          if (hist_i) keep(2, cu);
        }
        if (hist_i) {
          // d E^{n+1} / d eps_r = dca E^n + dcb curl + dce corr, and
          // dce / dcb = (1 + sigma dt / (2 eps))^2 = (ce / cb)^2: the recorded curl
          // carries the CPML correction (before its ce scaling)
          const int sy = P.hb[3] - P.hb[2], sz = P.hb[5] - P.hb[4];
          const int hc = (P.hb[1] - P.hb[0]) * sy * sz;
          const int c0 = ((i - P.hb[0]) * sy + (j - P.hb[2])) * sz + (k - P.hb[4]);
          float* hp = P.hist + (long long)(n - P.hist_step0) * P.hist_ld + c0;
          float el[3][4], ql[4];
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            el[0][l] = e0[0][l];
            el[1][l] = e0[1][l];
            el[2][l] = e0[2][l];
            const float q = CP && any ? __fdiv_rn(ce[l], cbv[l]) : 0.f;
            ql[l] = __fmul_rn(q, q);
          }
#pragma unroll 1
          for (int c = 0; c < 3; ++c)
#pragma unroll 1
            for (int l = max(0, P.hb[4] - k); l < min(4, P.hb[5] - k); ++l) {
              const float v = hl[0][c][l];
              hp[c * hc + l] = el[c][l];
              hp[(3 + c) * hc + l] = CP && any ? __fmaf_rn(ql[l], hl[1][c][l], v) : v;
            }
        }
        if (kv < 4) {
#pragma unroll
          for (int l = 1; l < 4; ++l)
            if (l >= kv) { ex[l] = 0.f; ey[l] = 0.f; ez[l] = 0.f; }
        }
        // PEC faces
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
            ex[l] = ex[l] * (1.f - (float)(m & 1u));
            ey[l] = ey[l] * (1.f - (float)((m >> 1) & 1u));
            ez[l] = ez[l] * (1.f - (float)((m >> 2) & 1u));
          }
        }
        if (pmask | smask | (unsigned)tail) {   // over an indexed copy: one site per kind
          float v[6][4];
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            v[0][l] = ex[l]; v[1][l] = ey[l]; v[2][l] = ez[l];
            v[3][l] = hx[l]; v[4][l] = hy[l]; v[5][l] = hz[l];
          }
          // probes sampled before the sources, the sources, the other probes
#pragma unroll 1
          for (int pass = 0; pass < 3; ++pass) {
            const bool at_src = pass == 1;
            const int count = at_src ? P.nsrc : P.prb_out ? P.nprb : 0;
            const int4* list = at_src ? P.src : P.prb;
            unsigned m = at_src ? smask : pmask;
            int s = 31;
#pragma unroll 1
            while (true) {
              if (m) { s = __ffs(m) - 1; m &= m - 1; }
              else s = max(s + 1, 32);
              if (s >= count) break;
              const int4 c = __ldg(list + s);
              if (c.x != i || c.y != j || c.z < k || c.z >= k + 4) continue;
              const int l = c.z - k;
              if (at_src) {
                const int comp = min(c.w, 2);
                v[comp][l] = v[comp][l] + __ldg(P.srcw + (long long)n * P.src_ld + s);
              } else if (((c.w >> 4) & 1) == (pass == 0 ? 1 : 0)) {
                P.prb_out[(long long)n * P.prb_ld + s] = v[min(c.w & 7, 5)][l];
              }
            }
          }
#pragma unroll
          for (int l = 0; l < 4; ++l) { ex[l] = v[0][l]; ey[l] = v[1][l]; ez[l] = v[2][l]; }
        }
        vst<4>(Fo + e, ex);
        vst<4>(Fo + cs + e, ey);
        vst<4>(Fo + 2 * cs + e, ez);
        if (CP && i + 1 < xb) {
          fetch(P.psE[par], i + 1, B, jk, 2);
          if (B.y || B.z || in_xslab(i + 1)) cp_async16(slot + 8 * SS, P.ce + e + ps);
        }
      }
      if (CP) cp_async_commit();
#pragma unroll
      for (int c = 0; c < 3; ++c) e0[c] = vld<4>(Bp + o + c * CE);
      hyp = hy;
      hzp = hz;
      sA = sB;
      sB = sB == 2 ? 0 : sB + 1;
    }
    bad_end = bad;
  } else {
    // ---- halo warp: row y0-1 (lanes < ZQ, four columns each: hx, hz), column
    // z0-1 (lanes ZQ .. ZQ+TY-1, one row each: hx, hy); the last lane issues
    // the boxes ----
    const int lane = zq;
    const bool row = lane < ZQ && y0 >= 1 && z0 + 4 * lane < nz;
    const bool colm = lane >= ZQ && lane - ZQ < TY && z0 >= 1 && y0 + lane - ZQ < ny;
    const int j = row ? y0 - 1 : y0 + lane - ZQ;
    const int k = row ? z0 + 4 * lane : z0 - 1;
    const int o = row ? 4 * lane + 4 : (lane - ZQ + 1) * EW + 3;
    const long long col = (row || colm) ? P.off0 + (long long)j * zs + k : 0;
    const int jk = j * zs + k;
    VSlab B;
    if (row) place(B, j, k, 4);
    else if (colm) place(B, j, k, 1);
    const float yh = (row || colm) ? __ldg(P.yh + j) : 0.f;
    float zhc = 0.f;
    float4 czc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (colm) {
      zhc = __ldg(P.zh + k);
      if (CP && cpz && k < ncp) czc = __ldg(P.cpu + 4 * ncp + k);
      else if (CP && cpz && k >= kb) czc = __ldg(P.cpu + 5 * ncp + (k - kb));
    }
    // the column's old hx, hy and old psi (x q0, y q0, z q0, q1), and the row's
    // old psi (x q1, y q0, q1, z q0), one plane ahead
    float hcx = 0.f, hcy = 0.f, pc[4] = {0.f, 0.f, 0.f, 0.f};
    Vec<4> pr[4];
    pr[0] = pr[1] = pr[2] = pr[3] = vzero<4>();
    auto load_old = [&](int i) {
      const float* px = P.psH[par][0] + (in_xslab(i) ? xbase_of(i) + jk : 0);
      const float* py = P.psH[par][1] + B.oy + i * ncp * zs;
      const float* pz = P.psH[par][2] + B.oz + i * ny * n4;
      if (row) {
        if (CP && in_xslab(i)) pr[0] = vld<4>(px + qx);
        if (CP && B.y) { pr[1] = vld<4>(py); pr[2] = vld<4>(py + qy); }
        if (CP && B.z) pr[3] = zpsi_load<4>(pz, B.z);
      } else if (colm) {
        const long long e = col + (long long)i * ps;
        hcx = Fi[3 * cs + e];
        hcy = Fi[4 * cs + e];
        if (CP && in_xslab(i)) pc[0] = px[0];
        if (CP && B.y) pc[1] = py[0];
        if (CP && B.z) {
          pc[2] = pz[0];
          pc[3] = pz[qz];
        }
      }
    };
    load_old(xa);
    bool bad = false;
    float xh_n = __ldg(xh_tab + xa);
    bar_or<NT>(false);   // the stages of plane xa-1 are free
    if (producer) {
      if (xa + 2 <= xb) issue_e(xa + 2);
      if (xa + 1 < xb) issue_h(xa + 1);
    }
    last_e = min(xa + 2, xb);
    last_h = min(xa + 1, xb - 1);
    int sA = 1, sB = 2;
#pragma unroll 1
    for (int i = xa; i < xb; ++i) {
      const float xh = xh_n;
      if (i + 1 < xb) xh_n = __ldg(xh_tab + i + 1);
      const long long e = col + (long long)i * ps;
      float4 cx;
      int xbase = 0;
      const bool xon = xslab(i, cx, xbase);
      bad = !wait(sB) | bad;
      bad = !wait(3 + sH(i)) | bad;
      const float* A = &S.e[sA][0];
      const float* Bp = &S.e[sB][0];
      const float* H = &S.ho[sH(i)][0];
      const int sl = i & 1;
      if (lane < ZQ) {
        Vec<4> hx = vzero<4>(), hy, hz = vzero<4>();
        if (row) {
          Vec<4> ch, e0[3];
          if (ch_arr) ch = vld<4>(ch_arr + e);
          else {
#pragma unroll
            for (int l = 0; l < 4; ++l) ch[l] = ch0;
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) e0[c] = vld<4>(A + o + c * CE);
          h_vec<4, 5, CP, false, EW, CE>(
              A, Bp, o, e0, A[o + 4], A[o + 4 + CE], [&](int c) { return vld<4>(H + c * D::CH + 4 * lane); },
              [&](int a, int q) { return a == 0 ? pr[0] : a == 2 ? pr[3] : q == 0 ? pr[1] : pr[2]; }, xh, yh,
              vld<4>(&S.zt[0][4 * lane]), ch, P, par, xon, cx, xbase + jk, B, &S.zp[0][4 * lane], P.zw[k >= ncp], i, qx, qy, qz, ncp, hx, hy,
              hz);
        }
        vst<4>(&S.h[sl][0][0][4 * lane], hx);
        vst<4>(&S.h[sl][1][0][4 * lane], hz);
      }
      if (lane >= ZQ && lane - ZQ < TY) {
        float hx = 0.f, hy = 0.f;
        if (colm) {
          const float chv = ch_arr ? ch_arr[e] : ch0;
          const float Ex = A[o], Ey = A[o + CE], Ez = A[o + 2 * CE];
          const float dEz_y = A[o + 2 * CE + EW] - Ez, dEy_z = A[o + CE + 1] - Ey, dEx_z = A[o + 1] - Ex;
          const float dEz_x = Bp[o + 2 * CE] - Ez;
          hx = yee_h(hcx, chv, yee_diff2(dEz_y, yh, dEy_z, zhc));
          hy = yee_h(hcy, chv, yee_diff2(dEx_z, zhc, dEz_x, xh));
          if (CP) {
            if (xon) {
              const float g = __fmul_rn(dEz_x, cx.w);
              hy = psi_add(hy, chv, psi_next(cx.x, pc[0], cx.y, g), cx.z, g);
            }
            if (B.y) {
              const float g = __fmul_rn(dEz_y, B.cy.w);
              hx = psi_add(hx, -chv, psi_next(B.cy.x, pc[1], B.cy.y, g), B.cy.z, g);
            }
            if (B.z) {
              const float g0 = __fmul_rn(dEy_z, czc.w), g1 = __fmul_rn(dEx_z, czc.w);
              hx = psi_add(hx, chv, psi_next(czc.x, pc[2], czc.y, g0), czc.z, g0);
              hy = psi_add(hy, -chv, psi_next(czc.x, pc[3], czc.y, g1), czc.z, g1);
            }
          }
        }
        S.hc[sl][0][lane - ZQ] = hx;
        S.hc[sl][1][lane - ZQ] = hy;
      }
      if (i + 1 < xb) load_old(i + 1);
      if (bar_or<NT>(bad)) { bad = true; break; }
      // H of plane i is done: its H stage takes plane i+2 and its E stage plane
      // i+3 (the owners hold E of plane i in registers); E of plane i-1 is done:
      // its coefficient stage takes plane i+1
      if (producer) {
        if (i + 3 <= xb) issue_e(i + 3);
        if (i + 2 < xb) issue_h(i + 2);
        if (i > xa && i + 1 < xb) issue_c(i + 1);
      }
      last_e = min(i + 3, xb);
      last_h = min(i + 2, xb - 1);
      last_c = max(last_c, min(i + 1, xb - 1));
      ph.stage ^= 1u << (5 + sC(i));   // the owners wait for the coefficients
      sA = sB;
      sB = sB == 2 ? 0 : sB + 1;
    }
    bad_end = bad;
  }
  if (bar_or<NT>(bad_end)) { bail(); return false; }
  return true;
}

template <int TY, int ZQ, bool CP>
__device__ __forceinline__ void fwdv_init_barriers(VSmem<TY, ZQ, CP>& S) {
  if (threadIdx.x == 0) {
#pragma unroll 1
    for (int q = 0; q < RFXB_VBARS; ++q) mbar_init(smem_u32(&S.mbar[q]), 1);
    mbar_fence_init();
  }
  __syncthreads();
}

// One launch per step: CTA b runs work item b.  `sel` selects the field
// buffers and the psi parity (step_sel), `map0` the tile shape's E boxes.
template <int TY, int ZQ, bool CP>
__global__ void __launch_bounds__(VDims<TY, ZQ>::NT, (TY == 24 ? 2 : 5))
fwdv_kernel(const RfxbInst* __restrict__ insts, const RfxbWork* __restrict__ work,
            const CUtensorMap* __restrict__ maps, int map0, int n, int sel) {
  extern __shared__ __align__(128) unsigned char fwdv_smem_raw[];
  RfxbWork w = work[blockIdx.x];
  StepPhases ph;
  if (!CP || (w.inst & RFXB_WORK_PLAIN)) {
    w.inst &= ~RFXB_WORK_PLAIN;
    auto& S = *reinterpret_cast<VSmem<TY, ZQ, false>*>(fwdv_smem_raw);
    fwdv_init_barriers<TY, ZQ, false>(S);
    fwdv_item<TY, ZQ, false>(S, insts, w, maps, map0, n, sel, ph, StepFault{}, true);
  } else {
    auto& S = *reinterpret_cast<VSmem<TY, ZQ, CP>*>(fwdv_smem_raw);
    fwdv_init_barriers<TY, ZQ, CP>(S);
    fwdv_item<TY, ZQ, CP>(S, insts, w, maps, map0, n, sel, ph, StepFault{}, true);
  }
}

// Persistent forward step: one launch per step of exactly as many CTAs as
// fit on the GPU at once.  Each CTA takes items from the two lists of the
// step -- queue 0 the tiles that reach a CPML slab, queue 1 the CPML-free
// tiles -- through fetch counters in device memory until both are empty.  The
// first `plain_ctas` CTAs (one per SM when the block scheduler spreads the
// first wave) try queue 1 first, the others queue 0; a CTA whose queue is
// empty helps with the other.  An item outside its instance's grid is skipped
// and flagged (status bit 2).  The last CTA to finish clears the counters for
// the next launch.
template <int TY, int ZQ>
__global__ void __launch_bounds__(VDims<TY, ZQ>::NT, 5)
fwdv_persist_kernel(const RfxbInst* __restrict__ insts, int n_inst, RfxbFwdQueues Q,
                    const CUtensorMap* __restrict__ maps, int map0, int n, int sel) {
  extern __shared__ __align__(128) unsigned char fwdv_smem_raw[];
  auto& S = *reinterpret_cast<VSmem<TY, ZQ, true>*>(fwdv_smem_raw);
  __shared__ int pick[2];
  const int tid = threadIdx.x;
  fwdv_init_barriers<TY, ZQ, true>(S);
  StepPhases ph;
  StepFault fault;
  fault.cta = Q.fault_cta;
  fault.wait_limit = Q.wait_limit;
  const int first = (int)blockIdx.x < Q.plain_ctas ? 1 : 0;
  bool first_item = true;
  bool ok = true;
  while (ok) {
    if (tid == 0) {
      pick[0] = -1;
      for (int t = 0; t < 2; ++t) {
        const int q = t == 0 ? first : 1 - first;
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
    ok = fwdv_item<TY, ZQ, true>(S, insts, w, maps, map0, n, sel, ph, fault, first_item);
    first_item = false;
  }
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(&Q.ctr[2], 1) == (int)gridDim.x - 1) {
      Q.ctr[0] = 0;
      Q.ctr[1] = 0;
      Q.ctr[2] = 0;
      __threadfence();
    }
  }
}

template __global__ void fwdv_kernel<8, 8, false>(const RfxbInst*, const RfxbWork*, const CUtensorMap*, int, int, int);
template __global__ void fwdv_kernel<8, 8, true>(const RfxbInst*, const RfxbWork*, const CUtensorMap*, int, int, int);
template __global__ void fwdv_kernel<24, 8, false>(const RfxbInst*, const RfxbWork*, const CUtensorMap*, int, int, int);
template __global__ void fwdv_kernel<24, 8, true>(const RfxbInst*, const RfxbWork*, const CUtensorMap*, int, int, int);
template __global__ void fwdv_persist_kernel<8, 8>(const RfxbInst*, int, RfxbFwdQueues, const CUtensorMap*, int, int,
                                                   int);

size_t fwdv_smem_bytes(int tile, bool cp) {
  return tile == 0 ? (cp ? sizeof(VSmem<24, 8, true>) : sizeof(VSmem<24, 8, false>))
                   : (cp ? sizeof(VSmem<8, 8, true>) : sizeof(VSmem<8, 8, false>));
}
static_assert(2 * (sizeof(VSmem<24, 8, true>) + 1024) <= 228 * 1024, "two CTAs per SM");

}  // namespace rfxb
