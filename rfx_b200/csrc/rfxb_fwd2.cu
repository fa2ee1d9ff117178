// Two-step forward pass of the CPML-free interior (temporal blocking, depth 2),
// four cells per thread.
//
// One CTA owns a rectangle of at most 13 rows x 56 columns of the (y, z) plane
// over an x range [xa, xb) and advances it from step n to step n+2 in one pass
// over HBM: E^n, H^{n-1/2} and ca/cb are read once with a halo, the intermediate
// state (E^{n+1}, H^{n+1/2}) stays in registers, and only (E^{n+2}, H^{n+3/2})
// of the rectangle are written.  The halo cells of the first step are recomputed
// by every CTA that needs them (overlapped tiling), from step-n values that no
// CTA of the pass overwrites (the pass reads F[par] and writes F[par ^ 1]).
//
// 16 x 16 threads each hold one row and four consecutive columns -- rows y0-2 ..
// y0+13, columns z0-4 .. z0+59 -- and march along x with the second step one
// plane behind the first.  At plane p a thread computes, on its own cells,
//   H^{n+1/2}(p);  E^{n+1}(p), H^{n+3/2}(p-1);  E^{n+2}(p-1)
// with a block barrier at each semicolon: the y neighbour's values of the phase
// before pass through shared memory, the z neighbour's come from the adjacent
// lane, the x neighbour's are the thread's own.  A value at the rim whose
// neighbour no thread holds is wrong and reaches no stored cell: H^{n+1/2} is
// right on rows y0-2 .., E^{n+1} on y0-1 .. y0+13, H^{n+3/2} up to y0+12 and
// E^{n+2} on y0 .. y0+12, alike in z.  The arithmetic is the one-step kernel's
// (rfx/core/yee.py:226-291 and :347-404 through the shared rounding helpers),
// so every value equals the one-step value bit for bit.
//
// The host gives this kernel only cells that, halo included, lie in no CPML slab
// and hold no source, probe or gradient-history cell, in plans with uniform H
// coefficients; items at a grid face take the guarded path (zero outside the
// grid, PEC faces) and a PEC edge mask applies to every E cell as in the
// one-step kernel.  Everything else runs two one-step launches per pass through
// the intermediate buffer F[2].
// Where a one-step neighbour or a per-step observer (DFT plane, flux monitor,
// NTFF face) reads this item's intermediate state, the CTA also stores it to
// F[2] (RfxbWork2::mid).
//
// What bounds it: the latency of a plane (two barriers, two CTAs of eight warps
// per SM) and, on grids far beyond L2, the halo rows read again.  16 x 64 cells
// per plane store 71 % of what they compute; taller CTAs store more but leave
// one per SM, lower ones store less.  One cell per thread on 8 x 32 tiles, with
// the intermediate state in shared memory and four barriers per plane -> here,
// per pass: 257^3 without CPML 399 -> 270 us, 513^3 2679 -> 2381 us (3.2 TB/s of
// the 56 bytes per cell, 82 moved).
#include "rfxb_common.cuh"
#include "rfxb_vec.cuh"

namespace rfxb {

struct Fwd2Smem {
  static constexpr int R = RFXB_D2ROWS, C = RFXB_D2COLS;   // rows and columns of the threads
  static constexpr int CE = (R + 1) * C, CH = R * C;       // component strides of an E and an H / coefficient stage
  float e[3][3 * CE];      // E^n, rows y0-2 .. y0+14, plane p in stage (p - xa + 2) % 3
  float h[2][3 * CH];      // H^{n-1/2}, rows y0-2 .. y0+13
  float cab[2][2 * CH];    // ca, cb
  float x1[2][CH];         // hx, hz of H^{n+1/2}(p)
  float x2[2][2][CH];      // ex, ez of E^{n+1}(p) in slot p & 1
  float x3[2][CH];         // hx, hz of H^{n+3/2}(p-1)
  float zt[2][C];          // zh, ze of the columns
  RfxbInst P;
  unsigned long long mbar[RFXB_VBARS];   // E stages, H stages, coefficient stages
};
static_assert(2 * (sizeof(Fwd2Smem) + 128 + 1024) <= 228 * 1024, "two CTAs per SM");

size_t fwd2_step_smem_bytes() { return sizeof(Fwd2Smem); }

// PEC faces of the E update (rfx/boundaries/pec.py:13-47), as the one-step
// kernel applies them.
__device__ __forceinline__ void pec_faces(unsigned pec, int i, int j, int k, int nx, int ny, int nz, float& ex,
                                          float& ey, float& ez) {
  if ((pec & 1u) && (i == 0 || i == nx - 1)) { ey = 0.f; ez = 0.f; }
  if ((pec & 2u) && (j == 0 || j == ny - 1)) { ex = 0.f; ez = 0.f; }
  if ((pec & 4u) && (k == 0 || k == nz - 1)) { ex = 0.f; ey = 0.f; }
  if ((pec & 4u) && k == nz - 1) ez = 0.f;
}

// One work item.  EDGE: the item's cells reach a grid face (no CPML on that
// axis): cells outside the grid stay zero (the guards the one-step kernel
// reads) and E takes the PEC faces; otherwise every computed cell is an
// interior cell and those checks are compiled out.
template <bool EDGE>
__device__ __forceinline__ void fwd2_item(Fwd2Smem& S, const RfxbWork2& w, const CUtensorMap* __restrict__ maps,
                                          int par, const StepFault& fault) {
  constexpr int C = Fwd2Smem::C, R = Fwd2Smem::R, CE = Fwd2Smem::CE, CH = Fwd2Smem::CH, NT = R * C / 4, ZQ = C / 4;
  const int tid = threadIdx.x, r = tid / ZQ, zq = tid % ZQ;
  const RfxbInst& P = S.P;
  const int y0 = w.y0, z0 = w.z0, xa = w.xa, xb = w.xb;
  const int nx = P.nx, ny = P.ny, nz = P.nz;
  const long long ps = P.ps, cs = P.cs;
  const unsigned pec = P.pec_axes;
  const CUtensorMap* tm = maps + (size_t)w.inst * RFXB_NMAPS;
  const int wlim = fault.wait_limit;
  // The boxes: E of planes xa-2 .. xb+1, H of xa-2 .. xb, coefficients of xa-1 .. xb
  // (map coordinates: z, j + 1, i + 1, component)
  const bool producer = tid == NT - 1;
  auto sE = [&](int p) { return (p - xa + 2) % 3; };
  auto sH = [&](int p) { return (p - xa + 2) & 1; };
  auto sC = [&](int p) { return (p - xa + 1) & 1; };
  auto issue_e = [&](int p) {
    const uint32_t mb = smem_u32(&S.mbar[sE(p)]);
    mbar_expect_tx(mb, 4u * 3 * CE);
    tma_load_4d(smem_u32(&S.e[sE(p)][0]), tm + RFXB_MAP_E2 + par, z0 - 4, y0 - 1, p + 1, 0, mb);
  };
  auto issue_h = [&](int p) {
    const uint32_t mb = smem_u32(&S.mbar[3 + sH(p)]);
    mbar_expect_tx(mb, 4u * 3 * CH);
    tma_load_4d(smem_u32(&S.h[sH(p)][0]), tm + RFXB_MAP_H2 + par, z0 - 4, y0 - 1, p + 1, 3, mb);
  };
  auto issue_c = [&](int p) {
    const uint32_t mb = smem_u32(&S.mbar[5 + sC(p)]);
    mbar_expect_tx(mb, 4u * 2 * CH);
    tma_load_4d(smem_u32(&S.cab[sC(p)][0]), tm + RFXB_MAP_C2, z0 - 4, y0 - 1, p + 1, 0, mb);
  };
  if (producer) {
    issue_e(xa - 2);
    issue_e(xa - 1);
    issue_h(xa - 2);
    issue_h(xa - 1);
    if ((int)blockIdx.x != fault.cta) issue_e(xa);
    issue_c(xa - 1);
    issue_c(xa);
  }
  int last_e = xa, last_h = xa - 1, last_c = xa;   // planes issued so far (xb > xa)
  // spacing tables (entries -1 .. n exist; the cells beyond are zero or unused)
  if (tid < C) {
    const int k = min(max(z0 - 4 + tid, -1), nz);
    S.zt[0][tid] = __ldg(P.zh + k);
    S.zt[1][tid] = __ldg(P.ze + k);
  }
  __syncthreads();   // the first plane reads them before its barrier
  auto xclamp = [&](int i) { return min(max(i, -1), nx); };
  const float ch = P.ch0;
  float* Fo = P.F[par ^ 1][0];
  float* Fm = P.F[2][0];
  const int j = y0 - 2 + r, k = z0 - 4 + 4 * zq;
  const float yh = __ldg(P.yh + min(max(j, -1), ny)), ye = __ldg(P.ye + min(max(j, -1), ny));
  const int oh = r * C + 4 * zq;                       // place in a component of every array here
  const int om = max(r - 1, 0) * C + 4 * zq, op = min(r + 1, R - 1) * C + 4 * zq;   // rows below and above
  const long long col = P.off0 + (long long)j * P.zs + k;
  const bool own = j >= y0 && j < w.yb && k >= z0 && k < w.zb;
  const bool rim = j == 0 || j == ny - 1 || k == 0 || (k < nz && k + 3 >= nz - 1);   // holds a cell of a y or z face
  const bool inyz = j >= 0 && j < ny && k >= 0 && k < nz;
  const unsigned char* emask = P.emask && inyz ? P.emask + col : nullptr;   // PEC edge mask bits (1 ex, 2 ey, 4 ez)
  // zero outside the grid (EDGE)
  auto clip = [&](bool in_x, Vec<4>& a, Vec<4>& b, Vec<4>& c) {
    if (!EDGE) return;
    const int kv = in_x && inyz ? nz - k : 0;
    if (kv >= 4) return;
#pragma unroll
    for (int l = 0; l < 4; ++l)
      if (l >= kv) { a[l] = 0.f; b[l] = 0.f; c[l] = 0.f; }
  };
  // PEC faces and the edge mask of the four cells
  auto finish_e = [&](int i, unsigned em, Vec<4>& ex, Vec<4>& ey, Vec<4>& ez) {
    if (EDGE && (rim || i == 0 || i == nx - 1)) {
#pragma unroll
      for (int l = 0; l < 4; ++l) pec_faces(pec, i, j, k + l, nx, ny, nz, ex[l], ey[l], ez[l]);
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
  };
  // H of the four cells from E (own), the row above, the next plane and the next column
  auto h_update = [&](const Vec<4>* E, const Vec<4>& uex, const Vec<4>& uez, const Vec<4>& ney, const Vec<4>& nez,
                      float xh, Vec<4>& hx, Vec<4>& hy, Vec<4>& hz) {
    const float ex4 = __shfl_down_sync(0xffffffffu, E[0][0], 1, ZQ), ey4 = __shfl_down_sync(0xffffffffu, E[1][0], 1, ZQ);
    const Vec<4> zh = vld<4>(&S.zt[0][4 * zq]);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const float dEz_y = uez[l] - E[2][l], dEx_y = uex[l] - E[0][l];
      const float dEy_z = (l < 3 ? E[1][l < 3 ? l + 1 : l] : ey4) - E[1][l];
      const float dEx_z = (l < 3 ? E[0][l < 3 ? l + 1 : l] : ex4) - E[0][l];
      const float dEz_x = nez[l] - E[2][l], dEy_x = ney[l] - E[1][l];
      hx[l] = yee_h(hx[l], ch, yee_diff2(dEz_y, yh, dEy_z, zh[l]));
      hy[l] = yee_h(hy[l], ch, yee_diff2(dEx_z, zh[l], dEz_x, xh));
      hz[l] = yee_h(hz[l], ch, yee_diff2(dEy_x, xh, dEx_y, yh));
    }
  };
  // E of the four cells from H (own), the row below, the plane before and the column before
  auto e_update = [&](const Vec<4>* H, const Vec<4>& dhx, const Vec<4>& dhz, const Vec<4>& phy, const Vec<4>& phz,
                      float xe, const Vec<4>& ca, const Vec<4>& cb, Vec<4>& ex, Vec<4>& ey, Vec<4>& ez) {
    const float hxm = __shfl_up_sync(0xffffffffu, H[0][3], 1, ZQ), hym = __shfl_up_sync(0xffffffffu, H[1][3], 1, ZQ);
    const Vec<4> ze = vld<4>(&S.zt[1][4 * zq]);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const float dHz_y = H[2][l] - dhz[l], dHx_y = H[0][l] - dhx[l];
      const float dHy_z = H[1][l] - (l ? H[1][l ? l - 1 : 0] : hym);
      const float dHx_z = H[0][l] - (l ? H[0][l ? l - 1 : 0] : hxm);
      const float dHz_x = H[2][l] - phz[l], dHy_x = H[1][l] - phy[l];
      ex[l] = yee_e(ca[l], ex[l], cb[l], yee_diff2(dHz_y, ye, dHy_z, ze[l]));
      ey[l] = yee_e(ca[l], ey[l], cb[l], yee_diff2(dHx_z, ze[l], dHz_x, xe));
      ez[l] = yee_e(ca[l], ez[l], cb[l], yee_diff2(dHy_x, xe, dHx_y, ye));
    }
  };
  auto put = [&](float* F, long long e, const Vec<4>* E, const Vec<4>* H) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      vst<4>(F + c * cs + e, E[c]);
      vst<4>(F + (3 + c) * cs + e, H[c]);
    }
  };
  unsigned phase = 0u;
  auto wait = [&](int b) -> bool {
    const bool ok = mbar_wait_bounded(smem_u32(&S.mbar[b]), (phase >> b) & 1u, wlim);
    phase ^= 1u << b;
    return ok;
  };

  Vec<4> g[3], h1[3], h2y = vzero<4>(), h2z = vzero<4>(), caq = vzero<4>(), cbq = vzero<4>();   // of plane p-1
#pragma unroll
  for (int c = 0; c < 3; ++c) g[c] = h1[c] = vzero<4>();
  unsigned em_q = 0u;
  float xh_n = __ldg(P.xh + xclamp(xa - 2)), xe_n = __ldg(P.xe + xclamp(xa - 2)), xh_q = 0.f, xe_q = 0.f;
  bool bad = !wait(0);
  int sA = 0, sB = 1;   // stages of planes p and p+1
#pragma unroll 1
  for (int p = xa - 2; p <= xb; ++p) {
    const float xh = xh_n, xe = xe_n;
    if (p < xb) { xh_n = __ldg(P.xh + xclamp(p + 1)); xe_n = __ldg(P.xe + xclamp(p + 1)); }
    unsigned em = 0u;
    if (emask && p >= 0 && p < nx) em = *reinterpret_cast<const unsigned*>(emask + p * ps);
    bad = !wait(sB) | bad;
    bad = !wait(3 + sH(p)) | bad;
    // ---- H^{n+1/2}(p) ----
    Vec<4> E[3], H[3];
    {
      const float* A = &S.e[sA][oh];
      const float* B = &S.e[sB][oh];
      const float* Ho = &S.h[sH(p)][oh];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        E[c] = vld<4>(A + c * CE);
        H[c] = vld<4>(Ho + c * CH);
      }
      h_update(E, vld<4>(A + C), vld<4>(A + 2 * CE + C), vld<4>(B + CE), vld<4>(B + 2 * CE), xh, H[0], H[1], H[2]);
      clip(p >= 0 && p < nx, H[0], H[1], H[2]);
      vst<4>(&S.x1[0][oh], H[0]);
      vst<4>(&S.x1[1][oh], H[2]);
    }
    if (bar_or<NT>(bad)) { bad = true; break; }
    // every thread is done with E and H of plane p in shared memory
    if (producer) {
      if (p + 3 <= xb + 1) issue_e(p + 3);
      if (p + 2 <= xb) issue_h(p + 2);
    }
    last_e = min(p + 3, xb + 1);
    last_h = min(p + 2, xb);
    if (p >= xa - 1) {
      bad = !wait(5 + sC(p));
      // ---- E^{n+1}(p) ----
      const Vec<4> ca = vld<4>(&S.cab[sC(p)][oh]), cb = vld<4>(&S.cab[sC(p)][oh + CH]);
      e_update(H, vld<4>(&S.x1[0][om]), vld<4>(&S.x1[1][om]), h1[1], h1[2], xe, ca, cb, E[0], E[1], E[2]);
      finish_e(p, em, E[0], E[1], E[2]);
      clip(p >= 0 && p < nx, E[0], E[1], E[2]);
      // the intermediate state of plane p where a one-step neighbour or an observer reads it
      if (own && p >= xa && p < xb &&
          ((w.mid & RFXB_MID_ALL) || (p == xa && (w.mid & RFXB_MID_LO)) || (p == xb - 1 && (w.mid & RFXB_MID_HI))))
        put(Fm, col + p * ps, E, H);
      vst<4>(&S.x2[p & 1][0][oh], E[0]);
      vst<4>(&S.x2[p & 1][1][oh], E[2]);
      const int q = p - 1;
      if (p >= xa) {
        // ---- H^{n+3/2}(p-1) ----
        h_update(g, vld<4>(&S.x2[q & 1][0][op]), vld<4>(&S.x2[q & 1][1][op]), E[1], E[2], xh_q, h1[0], h1[1], h1[2]);
        clip(q >= 0 && q < nx, h1[0], h1[1], h1[2]);
        vst<4>(&S.x3[0][oh], h1[0]);
        vst<4>(&S.x3[1][oh], h1[2]);
      }
      __syncthreads();
      if (producer && p + 2 <= xb) issue_c(p + 2);   // every thread has its coefficients of plane p
      last_c = max(last_c, min(p + 2, xb));
      if (p >= xa) {
        if (q >= xa) {
          // ---- E^{n+2}(p-1), and the stores ----
          e_update(h1, vld<4>(&S.x3[0][om]), vld<4>(&S.x3[1][om]), h2y, h2z, xe_q, caq, cbq, g[0], g[1], g[2]);
          finish_e(q, em_q, g[0], g[1], g[2]);
          clip(true, g[0], g[1], g[2]);
          if (own) put(Fo, col + q * ps, g, h1);
        }
        h2y = h1[1];
        h2z = h1[2];
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) g[c] = E[c];
      caq = ca;
      cbq = cb;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) h1[c] = H[c];
    em_q = em;
    xh_q = xh;
    xe_q = xe;
    sA = sB;
    sB = sB == 2 ? 0 : sB + 1;
  }
  if (bar_or<NT>(bad) && producer) {
    // a wait ran out: flag the launch and wait (bounded) for the last box of every stage
    atomicOr(P.status, 1);
    auto drain = [&](int b, int fill) { mbar_wait_bounded(smem_u32(&S.mbar[b]), (uint32_t)fill & 1u, wlim); };
#pragma unroll 1
    for (int p = max(xa - 2, last_e - 2); p <= last_e; ++p) drain(sE(p), (p - xa + 2) / 3);
#pragma unroll 1
    for (int p = max(xa - 2, last_h - 1); p <= last_h; ++p) drain(3 + sH(p), (p - xa + 2) >> 1);
#pragma unroll 1
    for (int p = max(xa - 1, last_c - 1); p <= last_c; ++p) drain(5 + sC(p), (p - xa + 1) >> 1);
  }
}

__global__ void __launch_bounds__(RFXB_D2ROWS * RFXB_D2COLS / 4, 2)
fwd2_step_kernel(const RfxbInst* __restrict__ insts, const RfxbWork2* __restrict__ work,
                 const CUtensorMap* __restrict__ maps, int n, int par, StepFault fault) {
  extern __shared__ __align__(128) unsigned char fwd2_smem_raw[];
  Fwd2Smem& S = *reinterpret_cast<Fwd2Smem*>(fwd2_smem_raw);
  const int tid = threadIdx.x;
  const RfxbWork2 w = work[blockIdx.x];
  if (tid == 0) {
#pragma unroll 1
    for (int q = 0; q < RFXB_VBARS; ++q) mbar_init(smem_u32(&S.mbar[q]), 1);
    mbar_fence_init();
  }
  load_inst(S.P, insts + w.inst, tid, blockDim.x);
  __syncthreads();
  if (w.mid & RFXB_MID_EDGE) fwd2_item<true>(S, w, maps, par, fault);
  else fwd2_item<false>(S, w, maps, par, fault);
}

}  // namespace rfxb
