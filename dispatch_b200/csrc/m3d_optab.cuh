// Sampled opacity tables (HOP/optab_mod.f90): a background or line-list opacity
// per unit chi500 tabulated on (wavelength, PC axis 1, PC axis 2) of (ln T, ln ne),
// sampled per (frequency, cell) by a separable tensor-product cubic Hermite with
// precomputed node slopes.
//
// Device layout: one float4 per node (val, dl, dt, de) -- the value and its slopes
// along the wavelength and the two PC axes -- wavelength fastest, so one 16-byte
// load brings everything the collapse needs from a node and the frequencies of a
// window read a contiguous run of nodes.  A second array holds the scattering
// component.  The window's slice of the table (the nodes its frequencies bracket,
// at every (it, je)) stays in L2 while the cells stream through.
#pragma once
#include "m3d_kernels.cuh"

namespace m3d {

struct OptabDev {
  int nnu, ntemp, nne, has_scat;
  const double *lam;
  const float4 *tv, *ts;
  double mu0, mu1, r11, r21, r12, r22, c01, c02, dc1, dc2;
};

// per-frequency bracket on the wavelength nodes: cnt = number of nodes below the
// query, k the 0-based interval, and hermite_coefs of the position in it; node is
// the wavelength node the query sits on (the interval's end with weights 0 and 1
// and vanishing slope weights) or -1
struct OptabFreq {
  int k, cnt;
  float pl, wc0, wc1, wcm0, wcm1;
  int node;
};

// A query on a node: the weights are (c0, c1) = (1, 0) or (0, 1) and cm0 = cm1 = 0,
// so each term the collapse forms from the other node is a product with an exact
// zero and it returns the node's own value and PC slopes.  The node's float4 alone
// then gives the same result for finite tables (a -0 can come out as +0).
__device__ __forceinline__ int optab_on_node(const float c[5], int k) {
  if (c[3] != 0.0f || c[4] != 0.0f) return -1;
  if (c[1] == 1.0f && c[2] == 0.0f) return k;
  if (c[1] == 0.0f && c[2] == 1.0f) return k + 1;
  return -1;
}

// hermite_coefs (interpol_mod.f90:171-188): p, c0, c1, cm0, cm1
__host__ __device__ __forceinline__ void optab_hcoefs(float t, float h, float c[5]) {
  const float t2 = t * t, t3 = t2 * t;
  const float p = 3.0f * t2 - 2.0f * t3;
  c[0] = p;
  c[1] = 1.0f - p;
  c[2] = p;
  c[3] = h * ((t3 - 2.0f * t2) + t);
  c[4] = h * (t3 - t2);
}

// the bracket of optab_mod.f90:214/358 from the count of nodes below x:
// k = min(max(searchsorted, 1), nnu - 1) is that count clamped to [1, nnu - 1]
__device__ __forceinline__ int optab_interval(int nnu, const double *lam, int cnt, double x, float c[5]) {
  int k = cnt < 1 ? 1 : (cnt > nnu - 1 ? nnu - 1 : cnt);
  k -= 1;
  const double l0 = lam[k], l1 = lam[k + 1];
  optab_hcoefs((float)((x - l0) / (l1 - l0)), (float)(l1 - l0), c);
  return k;
}

__global__ void k_optab_freq(int nf, const double *lam_q, int nnu, const double *lam, OptabFreq *fc) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nf) return;
  const double x = lam_q[f];
  int lo = 0, hi = nnu;
  while (lo < hi) {
    const int mid = lo + (hi - lo) / 2;
    if (lam[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  float c[5];
  OptabFreq o;
  o.cnt = lo;
  o.k = optab_interval(nnu, lam, lo, x, c);
  o.pl = c[0];
  o.wc0 = c[1];
  o.wc1 = c[2];
  o.wcm0 = c[3];
  o.wcm1 = c[4];
  o.node = optab_on_node(c, o.k);
  fc[f] = o;
}

// the cell's PC coordinates and Hermite coefficients (optab_mod.f90:225-238)
__device__ __forceinline__ void optab_cell(const OptabDev &T, double temp, double ne, int &it, int &je, float tc[5],
                                           float nc[5]) {
  const double d1 = log(temp) - T.mu0;
  const double d2 = log(ne) - T.mu1;
  const double p1 = __dadd_rn(__dmul_rn(T.r11, d1), __dmul_rn(T.r21, d2));
  const double p2 = __dadd_rn(__dmul_rn(T.r12, d1), __dmul_rn(T.r22, d2));
  const double ft = __dadd_rn(__dmul_rn(p1 - T.c01, __drcp_rn(T.dc1)), 1.0);
  const double fe = __dadd_rn(__dmul_rn(p2 - T.c02, __drcp_rn(T.dc2)), 1.0);
  const double ift = fmin(fmax(floor(ft), 1.0), (double)(T.ntemp - 1));
  const double ife = fmin(fmax(floor(fe), 1.0), (double)(T.nne - 1));
  optab_hcoefs((float)(ft - ift), (float)T.dc1, tc);
  optab_hcoefs((float)(fe - ife), (float)T.dc2, nc);
  it = (int)ift - 1;
  je = (int)ife - 1;
}

// What a cell's queries share, formed by one lane and read by all: the PC coordinates'
// Hermite coefficients (p, 1 - p, cm0, cm1), the table's first node at (it, je), chi500
// and the velocity factor
struct OptabCell {
  float4 tc, nc;
  long long base;
  double vf;
  float ch;
};

__device__ __forceinline__ OptabCell optab_cell_of(const OptabDev &T, double temp, double ne, float ch, double vf) {
  int it, je;
  float tc[5], nc[5];
  optab_cell(T, temp, ne, it, je, tc, nc);
  OptabCell r;
  r.tc = make_float4(tc[0], tc[1], tc[3], tc[4]);
  r.nc = make_float4(nc[0], nc[1], nc[3], nc[4]);
  r.base = (long long)it * T.nnu + (long long)je * T.nnu * T.ntemp;
  r.vf = vf;
  r.ch = ch;
  return r;
}

// collapse (optab_mod.f90:251-286), its PC part: v the wavelength collapses and gt, ge the
// PC slopes at the four (temp, ne) corners; temp, then ne
__device__ __forceinline__ float optab_collapse_pc(const float (&v)[4], const float (&gt)[4], const float (&ge)[4],
                                                   const float4 tc, const float4 nc) {
  const float f0 = fmaf(tc.w, gt[1], fmaf(tc.z, gt[0], fmaf(tc.x, v[1], tc.y * v[0])));
  const float f1 = fmaf(tc.w, gt[3], fmaf(tc.z, gt[2], fmaf(tc.x, v[3], tc.y * v[2])));
  const float ge0 = fmaf(tc.x, ge[1], tc.y * ge[0]);
  const float ge1 = fmaf(tc.x, ge[3], tc.y * ge[2]);
  return fmaf(nc.w, ge1, fmaf(nc.z, ge0, fmaf(nc.x, f1, nc.y * f0)));
}

// the wavelength's part at corner nodes A and B = A + 1, weights w = (p, cm0, cm1)
__device__ __forceinline__ float optab_collapse(const float4 (&A)[4], const float4 (&B)[4], float p, float cm0,
                                                float cm1, const float4 tc, const float4 nc) {
  const float op = 1.0f - p;
  float v[4], gt[4], ge[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    v[c] = fmaf(cm1, B[c].y, fmaf(cm0, A[c].y, fmaf(p, B[c].x, op * A[c].x)));
    gt[c] = fmaf(p, B[c].z, op * A[c].z);
    ge[c] = fmaf(p, B[c].w, op * A[c].w);
  }
  return optab_collapse_pc(v, gt, ge, tc, nc);
}

// the collapse of a query on a node: the node's value and PC slopes at the four corners
__device__ __forceinline__ float optab_collapse_node(const float4 (&A)[4], const float4 tc, const float4 nc) {
  float v[4], gt[4], ge[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    v[c] = A[c].x;
    gt[c] = A[c].z;
    ge[c] = A[c].w;
  }
  return optab_collapse_pc(v, gt, ge, tc, nc);
}

// the nodes of wavelength node k at the four (temp, ne) corners
__device__ __forceinline__ void optab_corners(const float4 *t, long long at, int sit, long long sje, float4 (&A)[4]) {
#pragma unroll
  for (int c = 0; c < 4; c++) A[c] = __ldg(t + at + (c & 1) * sit + (c >> 1) * sje);
}

constexpr int kOptabWarps = 8;
// Both samplers take kOptabCells neighbouring cells a warp and keep the table nodes of the
// last one in registers: neighbours in a row mostly lie in one (T, ne) cell of the table,
// and with the line list's shifts mostly between the same wavelength nodes, so a lane
// rereads its nodes only where they differ.  A cell at a time, the nodes' 16-byte loads
// kept the L1 data pipe 77 and 71 % busy.  64^3 cells of a cube, 256 frequencies:
// 0.44 -> 0.25 and 1.17 -> 1.02 ms.
// Cells a warp and registers were chosen together, by time: 8 cells at 80 registers (4 at
// 64: 0.33 ms, 8 at 122: 0.28, 16 at 122: 0.27), for the line list 4 at 128 (2: 1.32, 3:
// 1.11, 6: 1.43, 4 at 80 with spills: 1.71); its cells' work slots read only where they are
// added to took 1.9.
constexpr int kOptabCells = 8, kOptabCellsLL = 4;

// sample_interpolate (optab_mod.f90:181-287), lanes over the frequencies; back = (kappa +
// kappa_scat) chi500, scat = kappa_scat chi500
__global__ void __launch_bounds__(32 * kOptabWarps, 3) k_optab_sample(OptabDev T, int nf, long long ncell,
                                                                   const double *temp, const double *ne,
                                                                   const float *chi500, const OptabFreq *fc,
                                                                   float *back, float *scat) {
  constexpr int G = kOptabCells;
  __shared__ OptabCell cells[kOptabWarps][G];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const long long w0 = (long long)blockIdx.x * kOptabWarps + wib, nw = (long long)gridDim.x * kOptabWarps;
  const int sit = T.nnu;
  const long long sje = (long long)T.nnu * T.ntemp;
  for (long long c0 = w0 * G; c0 < ncell; c0 += nw * G) {
    const int ncl = (int)min((long long)G, ncell - c0);
    if (lane < ncl) cells[wib][lane] = optab_cell_of(T, temp[c0 + lane], ne[c0 + lane], chi500[c0 + lane], 1.0);
    __syncwarp();
    for (int f = lane; f < nf; f += 32) {
      const int node = fc[f].node;
      const int k = node >= 0 ? node : fc[f].k;
      float4 A[4], As[4];
      long long base = -1;
#pragma unroll
      for (int g = 0; g < G; g++) {
        if (g >= ncl) break;
        const OptabCell &q = cells[wib][g];
        if (q.base != base) {
          base = q.base;
          optab_corners(T.tv, base + k, sit, sje, A);
          optab_corners(T.ts, base + k, sit, sje, As);
        }
        float kap, kas;
        if (node >= 0) {
          kap = optab_collapse_node(A, q.tc, q.nc);
          kas = optab_collapse_node(As, q.tc, q.nc);
        } else {
          const OptabFreq w = fc[f];
          float4 B[4];
          optab_corners(T.tv, base + k + 1, sit, sje, B);
          kap = optab_collapse(A, B, w.pl, w.wcm0, w.wcm1, q.tc, q.nc);
          optab_corners(T.ts, base + k + 1, sit, sje, B);
          kas = optab_collapse(As, B, w.pl, w.wcm0, w.wcm1, q.tc, q.nc);
        }
        const size_t o = (size_t)(c0 + g) * nf + f;
        back[o] = (kap + kas) * q.ch;
        scat[o] = kas * q.ch;
      }
    }
    __syncwarp();
  }
}

// sample_interpolate_ll (optab_mod.f90:300-409): the query wavelength of each
// cell is lam_q (1 + vproj), bracketed by walking from its neighbour's count (the
// unshifted one for the first); xhat, ehat += kappa chi500, and chi_scat += kappa_scat
// chi500 when given.
__global__ void __launch_bounds__(32 * kOptabWarps, 2) k_optab_sample_ll(OptabDev T, int nf, long long ncell,
                                                                      const double *temp, const double *ne,
                                                                      const float *chi500, const float *vproj,
                                                                      const double *lam_q, const OptabFreq *fc,
                                                                      float *xhat, float *ehat, float *chi_scat) {
  constexpr int G = kOptabCellsLL;
  __shared__ OptabCell cells[kOptabWarps][G];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const long long w0 = (long long)blockIdx.x * kOptabWarps + wib, nw = (long long)gridDim.x * kOptabWarps;
  const int sit = T.nnu, nnu = T.nnu;
  const long long sje = (long long)T.nnu * T.ntemp;
  const double *lam = T.lam;
  for (long long c0 = w0 * G; c0 < ncell; c0 += nw * G) {
    const int ncl = (int)min((long long)G, ncell - c0);
    if (lane < ncl)
      cells[wib][lane] = optab_cell_of(T, temp[c0 + lane], ne[c0 + lane], chi500[c0 + lane],
                                       1.0 + (double)vproj[c0 + lane]);
    __syncwarp();
    for (int f = lane; f < nf; f += 32) {
      const double lq = lam_q[f];
      int cnt = fc[f].cnt;
      // the nodes on either side of the count stay at hand: a neighbour's query mostly
      // falls between the same two
      double llo = cnt > 0 ? lam[cnt - 1] : -HUGE_VAL, lhi = cnt < nnu ? lam[cnt] : HUGE_VAL;
      // the work slots of every cell, then their brackets
      float xv[G], ev[G], sv[G], p[G], cm0[G], cm1[G];
      int k[G];
#pragma unroll
      for (int g = 0; g < G; g++) {
        const size_t o = (size_t)(c0 + g) * nf + f;
        xv[g] = g < ncl ? xhat[o] : 0.0f;
        ev[g] = g < ncl ? ehat[o] : 0.0f;
        sv[g] = g < ncl && chi_scat ? chi_scat[o] : 0.0f;
      }
#pragma unroll
      for (int g = 0; g < G; g++) {
        if (g >= ncl) break;
        const double x = __dmul_rn(lq, cells[wib][g].vf);
        // bounded by the count: an infinite x passes no comparison with the ends' marks
        while (cnt < nnu && lhi < x) {
          cnt++;
          llo = lhi;
          lhi = cnt < nnu ? lam[cnt] : HUGE_VAL;
        }
        while (cnt > 0 && llo >= x) {
          cnt--;
          lhi = llo;
          llo = cnt > 0 ? lam[cnt - 1] : -HUGE_VAL;
        }
        float w[5];
        k[g] = (cnt < 1 ? 1 : (cnt > nnu - 1 ? nnu - 1 : cnt)) - 1;
        const bool inside = cnt >= 1 && cnt <= nnu - 1;
        const double l0 = inside ? llo : lam[k[g]], l1 = inside ? lhi : lam[k[g] + 1];
        optab_hcoefs((float)((x - l0) / (l1 - l0)), (float)(l1 - l0), w);
        p[g] = w[0];
        cm0[g] = w[3];
        cm1[g] = w[4];
      }
      auto component = [&](const float4 *t, auto add) {
        float4 A[4], B[4];
        long long at = -1;
#pragma unroll
        for (int g = 0; g < G; g++) {
          if (g >= ncl) break;
          const OptabCell &q = cells[wib][g];
          if (q.base + k[g] != at) {
            at = q.base + k[g];
            optab_corners(t, at, sit, sje, A);
            optab_corners(t, at + 1, sit, sje, B);
          }
          const float w[5] = {p[g], 1.0f - p[g], p[g], cm0[g], cm1[g]};
          const int nd = optab_on_node(w, k[g]);
          const float kap = nd < 0 ? optab_collapse(A, B, p[g], cm0[g], cm1[g], q.tc, q.nc)
                            : nd == k[g] ? optab_collapse_node(A, q.tc, q.nc)
                                         : optab_collapse_node(B, q.tc, q.nc);
          add(g, kap * q.ch);
        }
      };
      component(T.tv, [&](int g, float a) {
        const size_t o = (size_t)(c0 + g) * nf + f;
        xhat[o] = xv[g] + a;
        ehat[o] = ev[g] + a;
      });
      if (chi_scat)
        component(T.ts, [&](int g, float a) { chi_scat[(size_t)(c0 + g) * nf + f] = sv[g] + a; });
    }
    __syncwarp();
  }
}

// ---- a cell a warp ----------------------------------------------------------------
// For cell counts that give the grouped kernels less than the warps they need: the
// neighbours' turns in a warp then only add up.  64 registers at 4 blocks an SM, the
// corners read pair by pair.  Where the line lies: optab_grouped, optab_grouped_ll.

// collapse of a query between the nodes at and at + 1
__device__ __forceinline__ float optab_collapse_at(const float4 *t, long long at, int sit, long long sje,
                                                   const float w[5], const float4 tc, const float4 nc) {
  float v[4], gt[4], ge[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const long long a = at + (c & 1) * sit + (c >> 1) * sje;
    const float4 A = __ldg(t + a), B = __ldg(t + a + 1);
    v[c] = fmaf(w[4], B.y, fmaf(w[3], A.y, fmaf(w[2], B.x, w[1] * A.x)));
    gt[c] = fmaf(w[0], B.z, w[1] * A.z);
    ge[c] = fmaf(w[0], B.w, w[1] * A.w);
  }
  return optab_collapse_pc(v, gt, ge, tc, nc);
}

// and of one on the node at
__device__ __forceinline__ float optab_collapse_node_at(const float4 *t, long long at, int sit, long long sje,
                                                        const float4 tc, const float4 nc) {
  float4 A[4];
  optab_corners(t, at, sit, sje, A);
  return optab_collapse_node(A, tc, nc);
}

__global__ void __launch_bounds__(32 * kOptabWarps, 4) k_optab_sample_one(OptabDev T, int nf, long long ncell,
                                                                       const double *temp, const double *ne,
                                                                       const float *chi500, const OptabFreq *fc,
                                                                       float *back, float *scat) {
  const int lane = threadIdx.x & 31;
  const long long w0 = (long long)blockIdx.x * kOptabWarps + (threadIdx.x >> 5);
  const long long nw = (long long)gridDim.x * kOptabWarps;
  const int sit = T.nnu;
  const long long sje = (long long)T.nnu * T.ntemp;
  for (long long c = w0; c < ncell; c += nw) {
    const OptabCell q = optab_cell_of(T, temp[c], ne[c], chi500[c], 1.0);
    for (int f = lane; f < nf; f += 32) {
      const OptabFreq p = fc[f];
      float kap, kas;
      if (p.node >= 0) {
        kap = optab_collapse_node_at(T.tv, q.base + p.node, sit, sje, q.tc, q.nc);
        kas = optab_collapse_node_at(T.ts, q.base + p.node, sit, sje, q.tc, q.nc);
      } else {
        const float w[5] = {p.pl, p.wc0, p.wc1, p.wcm0, p.wcm1};
        kap = optab_collapse_at(T.tv, q.base + p.k, sit, sje, w, q.tc, q.nc);
        kas = optab_collapse_at(T.ts, q.base + p.k, sit, sje, w, q.tc, q.nc);
      }
      const size_t o = (size_t)c * nf + f;
      back[o] = (kap + kas) * q.ch;
      scat[o] = kas * q.ch;
    }
  }
}

__global__ void __launch_bounds__(32 * kOptabWarps, 4) k_optab_sample_ll_one(OptabDev T, int nf, long long ncell,
                                                                          const double *temp, const double *ne,
                                                                          const float *chi500, const float *vproj,
                                                                          const double *lam_q, const OptabFreq *fc,
                                                                          float *xhat, float *ehat,
                                                                          float *chi_scat) {
  const int lane = threadIdx.x & 31;
  const long long w0 = (long long)blockIdx.x * kOptabWarps + (threadIdx.x >> 5);
  const long long nw = (long long)gridDim.x * kOptabWarps;
  const int sit = T.nnu, nnu = T.nnu;
  const long long sje = (long long)T.nnu * T.ntemp;
  const double *lam = T.lam;
  for (long long c = w0; c < ncell; c += nw) {
    const OptabCell q = optab_cell_of(T, temp[c], ne[c], chi500[c], 1.0 + (double)vproj[c]);
    for (int f = lane; f < nf; f += 32) {
      // the work slots before the bracket and the table
      const size_t o = (size_t)c * nf + f;
      const float xv = xhat[o], ev = ehat[o], sv = chi_scat ? chi_scat[o] : 0.0f;
      const double x = __dmul_rn(lam_q[f], q.vf);
      int cnt = fc[f].cnt;
      while (cnt < nnu && lam[cnt] < x) cnt++;
      while (cnt > 0 && lam[cnt - 1] >= x) cnt--;
      float w[5];
      const int k = optab_interval(nnu, lam, cnt, x, w), nd = optab_on_node(w, k);
      auto kappa = [&](const float4 *t) {
        return nd >= 0 ? optab_collapse_node_at(t, q.base + nd, sit, sje, q.tc, q.nc)
                       : optab_collapse_at(t, q.base + k, sit, sje, w, q.tc, q.nc);
      };
      const float add = kappa(T.tv) * q.ch;
      xhat[o] = xv + add;
      ehat[o] = ev + add;
      if (chi_scat) chi_scat[o] = sv + kappa(T.ts) * q.ch;
    }
  }
}

// sample_build_derivatives (optab_mod.f90:125-166), one thread per node.
// pchip_slopes8 (interpol_mod.f90:240-284) along the fp64 wavelength nodes:
// the interior slope of node i of a line y (stride 1)
__device__ __forceinline__ double pchip8_interior(const double *x, const float *y, int i) {
  const double dxm = x[i] - x[i - 1], dxp = x[i + 1] - x[i];
  const double dym = (double)y[i] - (double)y[i - 1], dyp = (double)y[i + 1] - (double)y[i];
  if (dym == 0 || dyp == 0) return 0.0;
  const double d1 = dym / dxm, d2 = dyp / dxp;
  if (copysign(1.0, d1) != copysign(1.0, d2)) return 0.0;
  const double alpha = (1.0 + dxm / (dxp + dxm)) / 3.0;
  return 1.0 / ((1.0 - alpha) / d1 + alpha / d2);
}

__global__ void k_optab_lam_slopes(int nnu, long long nlines, const double *lam, const float *val, float *dl) {
  const size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (g >= (size_t)nnu * nlines) return;
  const int k = (int)(g % nnu);
  const float *y = val + (g - k);
  double s;
  if (nnu == 2) {
    const double dy = (double)y[1] - (double)y[0], dx = lam[1] - lam[0];
    const double a = 2.0 * dy / dx - dy / dx;
    s = k == 0 ? a : 2.0 * dy / dx - a;
  } else if (k == 0) {
    s = 2.0 * ((double)y[1] - (double)y[0]) / (lam[1] - lam[0]) - pchip8_interior(lam, y, 1);
  } else if (k == nnu - 1) {
    s = 2.0 * ((double)y[k] - (double)y[k - 1]) / (lam[k] - lam[k - 1]) - pchip8_interior(lam, y, k - 1);
  } else {
    s = pchip8_interior(lam, y, k);
  }
  dl[g] = (float)s;
}

// pchip_slopes4 (interpol_mod.f90:193-235) along a regular PC axis, the node
// slopes pchip_mono4 returns at the nodes (:335-362): node i of a line of n
// nodes at stride st; the axis node i is (float)(c0 + i dc)
__device__ __forceinline__ float pchip4_interior(double c0, double dc, const float *y, size_t st, int i) {
  const float xm = (float)(c0 + (double)(i - 1) * dc), x0 = (float)(c0 + (double)i * dc);
  const float xp = (float)(c0 + (double)(i + 1) * dc);
  const float dxm = x0 - xm, dxp = xp - x0;
  const float dym = y[i * st] - y[(i - 1) * st], dyp = y[(i + 1) * st] - y[i * st];
  if (dym == 0 || dyp == 0) return 0.0f;
  const double d1 = (double)(dym / dxm), d2 = (double)(dyp / dxp);
  if (copysign(1.0, d1) != copysign(1.0, d2)) return 0.0f;
  const double alpha = (double)((1.0f + dxm / (dxp + dxm)) / 3.0f);
  return (float)(1.0 / ((1.0 - alpha) / d1 + alpha / d2));
}

__global__ void k_optab_axis_slopes(int nnu, int ntemp, int nne, int dim, double c0, double dc, const float *val,
                                    float *out) {
  const size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (g >= (size_t)nnu * ntemp * nne) return;
  const int it = (int)((g / nnu) % ntemp), je = (int)(g / ((size_t)nnu * ntemp));
  const int n = dim == 1 ? ntemp : nne;
  const int i = dim == 1 ? it : je;
  const size_t st = dim == 1 ? (size_t)nnu : (size_t)nnu * ntemp;
  const float *y = val + (g - (size_t)i * st);
  auto ax = [&](int j) { return (float)(c0 + (double)j * dc); };
  float s;
  if (n == 2) {
    const float dy = y[st] - y[0], dx = ax(1) - ax(0);
    const float a = 2.0f * dy / dx - dy / dx;
    s = i == 0 ? a : 2.0f * dy / dx - a;
  } else if (i == 0) {
    s = 2.0f * (y[st] - y[0]) / (ax(1) - ax(0)) - pchip4_interior(c0, dc, y, st, 1);
  } else if (i == n - 1) {
    s = 2.0f * (y[i * st] - y[(i - 1) * st]) / (ax(i) - ax(i - 1)) - pchip4_interior(c0, dc, y, st, i - 1);
  } else {
    s = pchip4_interior(c0, dc, y, st, i);
  }
  out[g] = s;
}

__global__ void k_optab_pack(size_t n, const float *val, const float *dl, const float *dt, const float *de,
                             float4 *t) {
  const size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (g < n) t[g] = make_float4(val[g], dl[g], dt[g], de[g]);
}

}  // namespace m3d
