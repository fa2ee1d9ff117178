// Forward steps of a small grid in one launch: the state stays in shared
// memory for all of them.
//
// The grid is cut into at most one block of cells per SM.  A CTA holds its
// block's E (with a one-cell shell), H (with the low layer on each axis), update
// coefficients and CPML psi in shared memory and advances n_steps steps; per step
//   1. H^{n+1/2} on the block and on its low layers (rfx/core/yee.py:226-291 /
//      :411-453, rfx/boundaries/cpml.py:804-1065): the low layers' H and psi are
//      kept twice, by their owner and by this block, with the same bits;
//   2. E^{n+1} on the block (rfx/core/yee.py:347-404 / :456-492,
//      rfx/boundaries/cpml.py:522-801), PEC faces, edge mask, sources and probes;
//      cells within one layer of the block's faces also go to the padded field
//      buffer of the step's parity in global memory;
//   3. a grid barrier (cooperative launch; every wait is bounded), after which
//      the shell is read from there.
// At the end every block writes its cells and psi to the buffers the step count
// makes current.  Every update calls the rounding helpers of the step kernels,
// so the results are theirs bit for bit.
//
// What bounds it: latency -- shared-memory passes over about 1200 cells by 16
// warps, then the barrier and the shell (about 2.5 us of a step).  A launch per
// step leaves the same grid 10 us of plane-by-plane marching and launch gaps:
// 87x47x42 with CPML 8 15.6 -> 6.2 us a step, 61x52x49 with CPML 8 14.5 -> 6.4,
// 43x37x33 with CPML 6 (too thin for the staged kernels) 27.1 -> 5.6.  512
// threads against 768 / 1024: 87x47x42 6.2 / 6.1 / 6.4, 43x37x33 5.6 / 5.8 / 5.9.
#include "rfxb_common.cuh"

namespace rfxb {

// descriptor bits: local coordinates 6 bits each, then
#define RES_VALID (1u << 18)
#define RES_X (1u << 19)        // in a CPML slab of the axis
#define RES_Y (1u << 20)
#define RES_Z (1u << 21)
#define RES_PEC 22              // three bits: component zeroed by a PEC face
#define RES_EM 25               // three bits: component masked by the edge mask
#define RES_EDGE (1u << 28)     // read by a neighbouring block
#define RES_SRC (1u << 29)      // holds a source or a probe

static size_t resident_floats(const ResidentShape& R, int n_axes) {
  const size_t e = (size_t)(R.b[0] + 2) * (R.b[1] + 2) * (R.b[2] + 2);
  const size_t h = (size_t)(R.b[0] + 1) * (R.b[1] + 1) * (R.b[2] + 1);
  const size_t c = (size_t)R.b[0] * R.b[1] * R.b[2];
  const size_t tab = 4 * (size_t)(R.b[0] + R.b[1] + R.b[2] + 6);   // xh, xe, ... of the layers
  const size_t prof = 4 * (size_t)(R.b[0] + R.b[1] + R.b[2] + 3);
  return 3 * e + 4 * h + 4 * c + 2 * n_axes * (h + c) + tab + prof + (e - c) + 64;
}
size_t resident_smem_bytes(const ResidentShape& R, int n_axes) {
  return sizeof(RfxbInst) + 256 + 4 * resident_floats(R, n_axes);
}

// All CTAs of the launch have arrived `gen` times: true, or false when the
// bounded wait ran out.
__device__ __forceinline__ bool grid_barrier(unsigned* ctr, unsigned target, int limit, int* ok_smem) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(ctr, 1u);
    bool ok = false;
    for (int t = 0; t < limit; ++t) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
      if (v >= target) { ok = true; break; }
    }
    __threadfence();
    *ok_smem = ok ? 1 : 0;
  }
  __syncthreads();
  return *ok_smem != 0;
}

__global__ void __launch_bounds__(RFXB_RES_THREADS, 1)
fwd_resident_kernel(const RfxbInst* __restrict__ insts, ResidentShape R, int step0, int n_steps, int par0, int pp0,
                    unsigned* ctr, int wait_limit) {
  constexpr int NT = RFXB_RES_THREADS;
  extern __shared__ __align__(16) unsigned char res_raw[];
  __shared__ int ok_flag, n_shell_s;
  const int tid = threadIdx.x;
  RfxbInst& P = *reinterpret_cast<RfxbInst*>(res_raw);
  load_inst(P, insts, tid, NT);
  if (tid == 0) n_shell_s = 0;
  __syncthreads();
  const int nn[3] = {P.nx, P.ny, P.nz};
  const int ncp = P.ncp;
  const unsigned axes = ncp > 0 ? P.cpml_axes : 0u;
  // this block's cells [lo, lo + d)
  int bi[3], lo[3], d[3];
  {
    int b = blockIdx.x;
    bi[2] = b % R.nb[2];
    b /= R.nb[2];
    bi[1] = b % R.nb[1];
    bi[0] = b / R.nb[1];
    for (int a = 0; a < 3; ++a) {
      lo[a] = bi[a] * R.b[a];
      d[a] = min(R.b[a], nn[a] - lo[a]);
    }
  }
  const int EY = R.b[1] + 2, EZ = R.b[2] + 2, HY = R.b[1] + 1, HZ = R.b[2] + 1;
  const int ES = EY * EZ, NE = (R.b[0] + 2) * ES, HS = HY * HZ, NH = (R.b[0] + 1) * HS;
  const int CS = R.b[1] * R.b[2], NC = R.b[0] * CS;
  // carve the arrays
  float* f = reinterpret_cast<float*>(res_raw + (sizeof(RfxbInst) + 255) / 256 * 256);
  float4* prof = reinterpret_cast<float4*>(f);   // per axis: layers lo-1 .. of the extended block
  int po[3];
  po[0] = 0;
  po[1] = R.b[0] + 1;
  po[2] = po[1] + R.b[1] + 1;
  f += 4 * (po[2] + R.b[2] + 1);
  float* tabs[6];   // xh xe yh ye zh ze at lo-1 .. lo+d-1
  for (int t = 0; t < 6; ++t) {
    tabs[t] = f;
    f += R.b[t / 2] + 2;
  }
  float* E = f;          f += 3 * NE;
  float* H = f;          f += 3 * NH;
  float* ca = f;         f += NC;
  float* cb = f;         f += NC;
  float* psH[3]; float* psE[3];   // [q][cell] per absorbing axis
  for (int a = 0; a < 3; ++a) {
    psH[a] = psE[a] = nullptr;
    if (axes & (1u << a)) {
      psH[a] = f; f += 2 * NH;
      psE[a] = f; f += 2 * NC;
    }
  }
  unsigned* hd = reinterpret_cast<unsigned*>(f); f += NH;
  unsigned* ed = reinterpret_cast<unsigned*>(f); f += NC;
  unsigned* shell = reinterpret_cast<unsigned*>(f);   // packed extended coordinates of the shell cells

  // ---- set-up: tables, descriptors, state ----
  for (int a = 0; a < 3; ++a) {
    const float* th = a == 0 ? P.xh : a == 1 ? P.yh : P.zh;
    const float* te = a == 0 ? P.xe : a == 1 ? P.ye : P.ze;
    for (int t = tid; t < R.b[a] + 1; t += NT) {
      const int x = lo[a] - 1 + t;
      const bool in = x >= 0 && x < nn[a];
      tabs[2 * a][t] = in ? __ldg(th + x) : 0.f;
      tabs[2 * a + 1][t] = in ? __ldg(te + x) : 0.f;
      float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
      if (in && (axes & (1u << a))) {
        int s;
        const int sd = cpml_side(x, nn[a], ncp, s);
        if (sd >= 0) c = __ldg(P.cpu + (2 * a + sd) * ncp + s);
      }
      prof[po[a] + t] = c;
    }
  }
  auto cell = [&](int i, int j, int k) { return P.off0 + (long long)i * P.ps + (long long)j * P.zs + k; };
  auto psi_q = [&](int a, int q, int i, int j, int k) -> long long {
    int s;
    const int x = a == 0 ? i : a == 1 ? j : k;
    const int sd = cpml_side(x, nn[a], ncp, s);
    return a == 0 ? psi_index_x(P, sd, q, s, j, k) : a == 1 ? psi_index_y(P, sd, q, s, i, k) : psi_index_z(P, sd, q, s, i, j);
  };
  __syncthreads();
  for (int t = tid; t < 3 * NE; t += NT) E[t] = 0.f;
  __syncthreads();
  for (int t = tid; t < NE; t += NT) {
    const int li = t / ES, r = t - li * ES, lj = r / EZ, lk = r - lj * EZ;
    const int i = lo[0] - 1 + li, j = lo[1] - 1 + lj, k = lo[2] - 1 + lk;
    if (li > d[0] + 1 || lj > d[1] + 1 || lk > d[2] + 1) continue;
    if (i < 0 || i >= nn[0] || j < 0 || j >= nn[1] || k < 0 || k >= nn[2]) continue;
    const long long e = cell(i, j, k);
    for (int c = 0; c < 3; ++c) E[c * NE + t] = P.F[par0][c][e];
    const int low = (li == 0) + (lj == 0) + (lk == 0), high = (li > d[0]) + (lj > d[1]) + (lk > d[2]);
    if (low + high > 0 && low <= 1 && high <= 1) shell[atomicAdd(&n_shell_s, 1)] = li | (lj << 6) | (lk << 12);
  }
  for (int t = tid; t < NH; t += NT) {
    const int li = t / HS, r = t - li * HS, lj = r / HZ, lk = r - lj * HZ;
    const int i = lo[0] - 1 + li, j = lo[1] - 1 + lj, k = lo[2] - 1 + lk;
    unsigned v = li | (lj << 6) | (lk << 12);
    const bool in = i >= 0 && j >= 0 && k >= 0 && li <= d[0] && lj <= d[1] && lk <= d[2] &&
                    (li == 0) + (lj == 0) + (lk == 0) <= 1;
    for (int c = 0; c < 3; ++c) H[c * NH + t] = in ? P.F[par0][3 + c][cell(i, j, k)] : 0.f;
    if (in) {
      v |= RES_VALID;
      const int x[3] = {li, lj, lk};
      for (int a = 0; a < 3; ++a) {
        if (!psH[a]) continue;
        if (prof[po[a] + x[a]].w == 0.f) continue;
        v |= RES_X << a;
        for (int q = 0; q < 2; ++q) psH[a][q * NH + t] = P.psH[pp0][a][psi_q(a, q, i, j, k)];
      }
    }
    hd[t] = v;
  }
  const unsigned pec = P.pec_axes;
  for (int t = tid; t < NC; t += NT) {
    const int li = t / CS, r = t - li * CS, lj = r / R.b[2], lk = r - lj * R.b[2];
    unsigned v = li | (lj << 6) | (lk << 12);
    float va = 0.f, vb = 0.f;
    if (li < d[0] && lj < d[1] && lk < d[2]) {
      const int i = lo[0] + li, j = lo[1] + lj, k = lo[2] + lk;
      const long long e = cell(i, j, k);
      v |= RES_VALID;
      va = P.ca[e];
      vb = P.cb[e];
      const int x[3] = {li, lj, lk};
      for (int a = 0; a < 3; ++a) {
        if (!psE[a] || prof[po[a] + x[a] + 1].w == 0.f) continue;
        v |= RES_X << a;
        for (int q = 0; q < 2; ++q) psE[a][q * NC + t] = P.psE[pp0][a][psi_q(a, q, i, j, k)];
      }
      unsigned z = 0u;
      if ((pec & 1u) && (i == 0 || i == nn[0] - 1)) z |= 6u;
      if ((pec & 2u) && (j == 0 || j == nn[1] - 1)) z |= 5u;
      if ((pec & 4u) && (k == 0 || k == nn[2] - 1)) z |= 3u;
      if ((pec & 4u) && k == nn[2] - 1) z |= 4u;
      v |= z << RES_PEC;
      if (P.emask) v |= ((unsigned)P.emask[e] & 7u) << RES_EM;
      if (li == 0 || lj == 0 || lk == 0 || li == d[0] - 1 || lj == d[1] - 1 || lk == d[2] - 1) v |= RES_EDGE;
      for (int s = 0; s < P.nsrc; ++s) {
        const int4 c = __ldg(P.src + s);
        if (c.x == i && c.y == j && c.z == k) v |= RES_SRC;
      }
      for (int s = 0; s < P.nprb; ++s) {
        const int4 c = __ldg(P.prb + s);
        if (c.x == i && c.y == j && c.z == k) v |= RES_SRC;
      }
    }
    ca[t] = va;
    cb[t] = vb;
    ed[t] = v;
  }
  __syncthreads();
  const int n_shell = n_shell_s;
  const float ch = P.ch0;
  const float *xh = tabs[0], *xe = tabs[1], *yh = tabs[2], *ye = tabs[3], *zh = tabs[4], *ze = tabs[5];

  // ---- steps ----
  for (int s = 0; s < n_steps; ++s) {
    const int n = step0 + s;
    for (int t = tid; t < NH; t += NT) {
      const unsigned v = hd[t];
      if (!(v & RES_VALID)) continue;
      const int li = v & 63, lj = (v >> 6) & 63, lk = (v >> 12) & 63;
      const int o = li * ES + lj * EZ + lk;
      const float Ex = E[o], Ey = E[NE + o], Ez = E[2 * NE + o];
      const float dEz_y = E[2 * NE + o + EZ] - Ez, dEy_z = E[NE + o + 1] - Ey, dEx_z = E[o + 1] - Ex;
      const float dEz_x = E[2 * NE + o + ES] - Ez, dEy_x = E[NE + o + ES] - Ey, dEx_y = E[o + EZ] - Ex;
      float hx = yee_h(H[t], ch, yee_diff2(dEz_y, yh[lj], dEy_z, zh[lk]));
      float hy = yee_h(H[NH + t], ch, yee_diff2(dEx_z, zh[lk], dEz_x, xh[li]));
      float hz = yee_h(H[2 * NH + t], ch, yee_diff2(dEy_x, xh[li], dEx_y, yh[lj]));
      if (v & RES_X) {
        const float4 c = prof[li];
        const float g0 = __fmul_rn(dEz_x, c.w), g1 = __fmul_rn(dEy_x, c.w);
        const float p0 = psi_next(c.x, psH[0][t], c.y, g0), p1 = psi_next(c.x, psH[0][NH + t], c.y, g1);
        psH[0][t] = p0;
        psH[0][NH + t] = p1;
        hy = psi_add(hy, ch, p0, c.z, g0);
        hz = psi_add(hz, -ch, p1, c.z, g1);
      }
      if (v & RES_Y) {
        const float4 c = prof[po[1] + lj];
        const float g0 = __fmul_rn(dEz_y, c.w), g1 = __fmul_rn(dEx_y, c.w);
        const float p0 = psi_next(c.x, psH[1][t], c.y, g0), p1 = psi_next(c.x, psH[1][NH + t], c.y, g1);
        psH[1][t] = p0;
        psH[1][NH + t] = p1;
        hx = psi_add(hx, -ch, p0, c.z, g0);
        hz = psi_add(hz, ch, p1, c.z, g1);
      }
      if (v & RES_Z) {
        const float4 c = prof[po[2] + lk];
        const float g0 = __fmul_rn(dEy_z, c.w), g1 = __fmul_rn(dEx_z, c.w);
        const float p0 = psi_next(c.x, psH[2][t], c.y, g0), p1 = psi_next(c.x, psH[2][NH + t], c.y, g1);
        psH[2][t] = p0;
        psH[2][NH + t] = p1;
        hx = psi_add(hx, ch, p0, c.z, g0);
        hy = psi_add(hy, -ch, p1, c.z, g1);
      }
      H[t] = hx;
      H[NH + t] = hy;
      H[2 * NH + t] = hz;
    }
    __syncthreads();
    const int fo = (par0 + s + 1) & 1;
    float* Fo = P.F[fo][0];
    const bool last = s + 1 == n_steps;
    for (int t = tid; t < NC; t += NT) {
      const unsigned v = ed[t];
      if (!(v & RES_VALID)) continue;
      const int li = v & 63, lj = (v >> 6) & 63, lk = (v >> 12) & 63;
      const int o = (li + 1) * ES + (lj + 1) * EZ + lk + 1, h = (li + 1) * HS + (lj + 1) * HZ + lk + 1;
      const float hx = H[h], hy = H[NH + h], hz = H[2 * NH + h];
      const float dHz_y = hz - H[2 * NH + h - HZ], dHy_z = hy - H[NH + h - 1], dHx_z = hx - H[h - 1];
      const float dHz_x = hz - H[2 * NH + h - HS], dHy_x = hy - H[NH + h - HS], dHx_y = hx - H[h - HZ];
      const float xev = xe[li + 1], yev = ye[lj + 1], zev = ze[lk + 1];
      const float cav = ca[t], cbv = cb[t];
      float ex = yee_e(cav, E[o], cbv, yee_diff2(dHz_y, yev, dHy_z, zev));
      float ey = yee_e(cav, E[NE + o], cbv, yee_diff2(dHx_z, zev, dHz_x, xev));
      float ez = yee_e(cav, E[2 * NE + o], cbv, yee_diff2(dHy_x, xev, dHx_y, yev));
      const long long e = cell(lo[0] + li, lo[1] + lj, lo[2] + lk);
      if (v & (RES_X | RES_Y | RES_Z)) {
        const float ce = __ldg(P.ce + e);
        if (v & RES_X) {
          const float4 c = prof[li + 1];
          const float g0 = __fmul_rn(dHz_x, c.w), g1 = __fmul_rn(dHy_x, c.w);
          const float p0 = psi_next(c.x, psE[0][t], c.y, g0), p1 = psi_next(c.x, psE[0][NC + t], c.y, g1);
          psE[0][t] = p0;
          psE[0][NC + t] = p1;
          ey = psi_add(ey, -ce, p0, c.z, g0);
          ez = psi_add(ez, ce, p1, c.z, g1);
        }
        if (v & RES_Y) {
          const float4 c = prof[po[1] + lj + 1];
          const float g0 = __fmul_rn(dHz_y, c.w), g1 = __fmul_rn(dHx_y, c.w);
          const float p0 = psi_next(c.x, psE[1][t], c.y, g0), p1 = psi_next(c.x, psE[1][NC + t], c.y, g1);
          psE[1][t] = p0;
          psE[1][NC + t] = p1;
          ex = psi_add(ex, ce, p0, c.z, g0);
          ez = psi_add(ez, -ce, p1, c.z, g1);
        }
        if (v & RES_Z) {
          const float4 c = prof[po[2] + lk + 1];
          const float g0 = __fmul_rn(dHy_z, c.w), g1 = __fmul_rn(dHx_z, c.w);
          const float p0 = psi_next(c.x, psE[2][t], c.y, g0), p1 = psi_next(c.x, psE[2][NC + t], c.y, g1);
          psE[2][t] = p0;
          psE[2][NC + t] = p1;
          ex = psi_add(ex, -ce, p0, c.z, g0);
          ey = psi_add(ey, ce, p1, c.z, g1);
        }
      }
      if (v & (63u << RES_PEC)) {
        if (v & (1u << RES_PEC)) ex = 0.f;
        if (v & (2u << RES_PEC)) ey = 0.f;
        if (v & (4u << RES_PEC)) ez = 0.f;
        ex = ex * (1.f - (float)((v >> RES_EM) & 1u));
        ey = ey * (1.f - (float)((v >> (RES_EM + 1)) & 1u));
        ez = ez * (1.f - (float)((v >> (RES_EM + 2)) & 1u));
      }
      if (v & RES_SRC) {
        const int i = lo[0] + li, j = lo[1] + lj, k = lo[2] + lk;
        auto probes = [&](int pre) {
          if (!P.prb_out) return;
          for (int p = 0; p < P.nprb; ++p) {
            const int4 c = __ldg(P.prb + p);
            if (c.x != i || c.y != j || c.z != k || ((c.w >> 4) & 1) != pre) continue;
            const int m = c.w & 7;
            P.prb_out[(long long)n * P.prb_ld + p] = m == 0 ? ex : m == 1 ? ey : m == 2 ? ez : m == 3 ? hx : m == 4 ? hy : hz;
          }
        };
        probes(1);
        for (int q = 0; q < P.nsrc; ++q) {
          const int4 c = __ldg(P.src + q);
          if (c.x != i || c.y != j || c.z != k) continue;
          const float w = __ldg(P.srcw + (long long)n * P.src_ld + q);
          if (c.w == 0) ex = ex + w;
          else if (c.w == 1) ey = ey + w;
          else ez = ez + w;
        }
        probes(0);
      }
      E[o] = ex;
      E[NE + o] = ey;
      E[2 * NE + o] = ez;
      if (last) {
        Fo[e] = ex;
        Fo[P.cs + e] = ey;
        Fo[2 * P.cs + e] = ez;
        Fo[3 * P.cs + e] = hx;
        Fo[4 * P.cs + e] = hy;
        Fo[5 * P.cs + e] = hz;
      } else if (v & RES_EDGE) {
        Fo[e] = ex;
        Fo[P.cs + e] = ey;
        Fo[2 * P.cs + e] = ez;
      }
    }
    if (last) break;
    if (!grid_barrier(ctr, (unsigned)gridDim.x * (s + 1), wait_limit, &ok_flag)) {
      if (tid == 0) atomicOr(P.status, 1);
      return;
    }
    // the shell, three cells a thread in flight
    for (int t0 = tid; t0 < n_shell; t0 += 3 * NT) {
      float x[3][3];
      int o[3];
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        const int t = t0 + u * NT;
        o[u] = -1;
        if (t >= n_shell) continue;
        const unsigned v = shell[t];
        const int li = v & 63, lj = (v >> 6) & 63, lk = (v >> 12) & 63;
        const float* g = Fo + cell(lo[0] - 1 + li, lo[1] - 1 + lj, lo[2] - 1 + lk);
        o[u] = li * ES + lj * EZ + lk;
        x[u][0] = __ldcg(g);
        x[u][1] = __ldcg(g + P.cs);
        x[u][2] = __ldcg(g + 2 * P.cs);
      }
#pragma unroll
      for (int u = 0; u < 3; ++u)
        if (o[u] >= 0) {
          E[o[u]] = x[u][0];
          E[NE + o[u]] = x[u][1];
          E[2 * NE + o[u]] = x[u][2];
        }
    }
    __syncthreads();
  }
  // psi of the block's cells
  const int pe = pp0 ^ (n_steps & 1);
  for (int t = tid; t < NC; t += NT) {
    const unsigned v = ed[t];
    if (!(v & RES_VALID) || !(v & (RES_X | RES_Y | RES_Z))) continue;
    const int li = v & 63, lj = (v >> 6) & 63, lk = (v >> 12) & 63;
    const int h = (li + 1) * HS + (lj + 1) * HZ + lk + 1;
    for (int a = 0; a < 3; ++a) {
      if (!(v & (RES_X << a))) continue;
      for (int q = 0; q < 2; ++q) {
        const long long p = psi_q(a, q, lo[0] + li, lo[1] + lj, lo[2] + lk);
        P.psH[pe][a][p] = psH[a][q * NH + h];
        P.psE[pe][a][p] = psE[a][q * NC + t];
      }
    }
  }
}

}  // namespace rfxb
