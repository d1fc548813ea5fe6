// Discrete adjoint of the 3D Yee step (reverse mode, time reversed).
//
// Forward step n (fdtd3d_kernels.cuh; CPML written generally, the damping
// boundary is the same with psi absent and a per-cell factor `damp`):
//   psiH' = bH psiH + cH D(E)                       D: forward differences
//   H'    = H - a (kH D(E) + S psiH')               S: +psi1 - psi2 per component
//   psiE' = bE psiE + cE G(H')                      G: backward differences
//   E'    = damp (E + cb (kE G(H') + S psiE')) + src
// Its transpose, applied to the adjoint (Ebar', Hbar', psibar') of the
// step's outputs, gives the adjoint of its inputs, in two passes:
//   k3a_pass<true>:  Xbar = cb damp Ebar';  psibarE' += S^T Xbar;
//                    dbarE = kE^T Xbar + cE psibarE';  psibarE = bE psibarE';
//                    Hbar += G^T dbarE (gather from the cell and its upper
//                    neighbours);  dJ/dcb += damp Ebar' X (FP64) with
//                    X = kE G(H') + S psiE' from the stored forward state
//   k3a_pass<false>: Ybar = -a Hbar;  psibarH' += S^T Ybar;
//                    dbarH = kH^T Ybar + cH psibarH';  psibarH = bH psibarH';
//                    Ebar = damp Ebar' + D^T dbarH (cell and lower neighbours)
// Cells outside a component's update range are the identity (no curl term),
// exactly as in the forward step.  Adjoint fields are FP32; dJ/dcb is
// accumulated in FP64.
//
// The difference adjoints dbarE and dbarH are formed where they are gathered,
// from Ebar (Hbar) and psibar of the cell and its three neighbours, instead of
// going through twelve arrays: 3 launches and about 190 bytes per cell and
// step became 2 launches and 130, on a working set (fields, dJ/dcb, psi: 60 MB
// at 96^3) that stays in the L2.  A pass reads one psi set and writes the
// other, because a neighbour's thread reads the value from before the step.
// 96^3, 10-layer CPML, per step: 80 us before, 25 now.
#pragma once

#include "fdtd3d_sweep.cuh"

namespace jxf {

constexpr int ADJ_THREADS = 128;

struct Adj3D {
  int nx, ny, nz;
  float a, cb_const;
  const float* cb;
  const float* damp[3];
  CpmlDev pml;            // tables, slab maps; in / out: adjoint of psi
  const float* fh[3];     // forward H^{n+1/2} after the step
  const float* fpsiE[6];  // forward psi (EXY..EZY) after the step, slab layout
  float* lE[3];           // adjoint of E
  float* lH[3];           // adjoint of H
  double* gcb;            // dJ/dcb accumulator
};

// Adjoint of one difference of a component's curl: the component's adjoint u
// (with the term's sign) through 1/kappa and the psi recurrence.
template <bool KAPPA>
__device__ __forceinline__ float adj_diff(bool slab, float u, float ik, float c, float psi) {
  const float d = KAPPA ? ik * u : u;
  return slab ? d + c * (psi + u) : d;
}

// One thread's cells (x, y, z0 .. z0+V-1).  P1: the pass over the E adjoint
// (updates Hbar and dJ/dcb, neighbours one up); else the pass over the H
// adjoint (updates Ebar, neighbours one down).  XS / YS / ZS (CPML): a cell or
// its neighbour may lie in that axis's psi slab.  Differences by component and
// axis: 0 x/y, 1 x/z, 2 y/z, 3 y/x, 4 z/x, 5 z/y.
template <bool P1, int MODE, int V, bool KAPPA, bool CBARR, bool XS, bool YS, bool ZS>
__device__ __forceinline__ void adj_cells(const Adj3D& p, int x, int y, int z0) {
  constexpr bool CP = MODE == MODE_CPML;
  constexpr bool DAMP = MODE == MODE_ABSORB;
  constexpr int S = P1 ? 1 : -1;  // direction of the neighbours
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  const int plane = ny * nz;
  const long long idx = (long long)x * plane + (y * nz + z0);
  // update conditions of the components, and which neighbours exist
  const bool okx = (CP && !XS) || (P1 ? x >= 1 : x < nx - 1);
  const bool oky = (CP && !YS) || (P1 ? y >= 1 : y < ny - 1);
  const bool ex = (CP && !XS) || (P1 ? x < nx - 1 : x >= 1);
  const bool ey = (CP && !YS) || (P1 ? y < ny - 1 : y >= 1);
  const int zn = P1 ? z0 + V : z0 - 1;  // z neighbour of the vector's end
  const bool ez = (CP && !ZS) || (P1 ? zn < nz : zn >= 0);
  // (a neighbour that does not exist is read at the cell and not used)
  const long long ix = ex ? idx + S * plane : idx;
  const long long iy = ey ? idx + S * nz : idx;
  const long long iz = ez ? (P1 ? idx + V : idx - 1) : idx;
  float* const* const A = P1 ? p.lE : p.lH;
  float* const* const G = P1 ? p.lH : p.lE;
  const VecF<V> a0 = load_v<V>(A[0] + idx), a1 = load_v<V>(A[1] + idx), a2 = load_v<V>(A[2] + idx);
  const VecF<V> a0y = load_v<V>(A[0] + iy), a2y = load_v<V>(A[2] + iy);
  const VecF<V> a1x = load_v<V>(A[1] + ix), a2x = load_v<V>(A[2] + ix);
  const float a0z = A[0][iz], a1z = A[1][iz];
  VecF<V> g0 = load_v<V>(G[0] + idx), g1 = load_v<V>(G[1] + idx), g2 = load_v<V>(G[2] + idx);
  // component adjoint = weight * field adjoint
  VecF<V> w, wx, wy;
  float wz = P1 ? p.cb_const : -p.a;
#pragma unroll
  for (int k = 0; k < V; ++k) w.v[k] = wx.v[k] = wy.v[k] = wz;
  if (P1 && CBARR) {
    w = load_v<V>(p.cb + idx);
    wx = load_v<V>(p.cb + ix);
    wy = load_v<V>(p.cb + iy);
    wz = p.cb[iz];
  }
  VecF<V> damp;
#pragma unroll
  for (int k = 0; k < V; ++k) damp.v[k] = 1.0f;
  if (DAMP) {
    const int xn = ex ? x + S : x, yn = ey ? y + S : y;
    const float dx = __ldg(p.damp[0] + x), dy = __ldg(p.damp[1] + y);
    const float dxn = __ldg(p.damp[0] + xn), dyn = __ldg(p.damp[1] + yn);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const float dz = __ldg(p.damp[2] + z0 + k);
      damp.v[k] = (dx * dy) * dz;
      if (P1) {
        w.v[k] *= damp.v[k];
        wx.v[k] *= (dxn * dy) * dz;
        wy.v[k] *= (dx * dyn) * dz;
      }
    }
    if (P1) wz *= (dx * dy) * __ldg(p.damp[2] + (ez ? zn : z0));
  }
  // forward H of the curl (dJ/dcb)
  VecF<V> f0, f1, f2, f0y, f2y, f1x, f2x;
  float f0z = 0.0f, f1z = 0.0f;
  double gc[V];
  if (P1) {
    const long long jx = okx ? idx - plane : idx, jy = oky ? idx - nz : idx;
    const long long jz = (CP && !ZS) || z0 >= 1 ? idx - 1 : idx;
    f0 = load_v<V>(p.fh[0] + idx);
    f1 = load_v<V>(p.fh[1] + idx);
    f2 = load_v<V>(p.fh[2] + idx);
    f0y = load_v<V>(p.fh[0] + jy);
    f2y = load_v<V>(p.fh[2] + jy);
    f1x = load_v<V>(p.fh[1] + jx);
    f2x = load_v<V>(p.fh[2] + jx);
    f0z = p.fh[0][jz];
    f1z = p.fh[1][jz];
    if constexpr (V == 2) {
      const double2 t = *reinterpret_cast<const double2*>(p.gcb + idx);
      gc[0] = t.x;
      gc[1] = t.y;
    } else {
      gc[0] = p.gcb[idx];
    }
  }
  // psi of the cell and its neighbours, coefficients of their positions
  constexpr int Q = P1 ? PSI_EXY : PSI_HXY;
  constexpr int QXY = Q, QXZ = Q + 1, QYZ = Q + 2, QYX = Q + 3, QZX = Q + 4, QZY = Q + 5;
  constexpr int TB = P1 ? TAB_BE : TAB_BH, TC = P1 ? TAB_CE : TAB_CH, TK = P1 ? TAB_IKE : TAB_IKH;
  VecF<V> zero;
#pragma unroll
  for (int k = 0; k < V; ++k) zero.v[k] = 0.0f;
  VecF<V> qyx = zero, qzx = zero, qxy = zero, qzy = zero;      // of the cell
  VecF<V> nyx = zero, nzx = zero, nxy = zero, nzy = zero;      // of the x / y neighbour
  VecF<V> pxy = zero, pzy = zero, pyx = zero, pzx = zero;      // forward psi
  float qxz[V], qyz[V], nxz = 0.0f, nyz = 0.0f, pxz[V], pyz[V];
  float xc = 0, xk = 1, xcn = 0, xkn = 1, xb = 0, yc = 0, yk = 1, ycn = 0, ykn = 1, yb = 0;
  float zb[V], zc[V], zk[V], zcn = 0.0f, zkn = 1.0f;
  bool sx = false, sxn = false, sy = false, syn = false, sz[V], szn = false;
  long long ox = 0, oy = 0, oz = 0;
  int km[V];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    qxz[k] = qyz[k] = pxz[k] = pyz[k] = zb[k] = zc[k] = 0.0f;
    zk[k] = 1.0f;
    sz[k] = false;
    km[k] = -1;
  }
  if (XS) {
    const int im = slab_map(x, nx, p.pml.P[0]);
    const int imn = ex ? slab_map(x + S, nx, p.pml.P[0]) : -1;
    sx = im >= 0;
    sxn = imn >= 0;
    if (sx) {
      ox = ((long long)im * ny + y) * nz + z0;
      xb = __ldg(p.pml.tab[0][TB] + x);
      xc = __ldg(p.pml.tab[0][TC] + x);
      if (KAPPA) xk = __ldg(p.pml.tab[0][TK] + x);
      qyx = load_v<V>(p.pml.in[QYX] + ox);
      qzx = load_v<V>(p.pml.in[QZX] + ox);
      if (P1) {
        pyx = load_v<V>(p.fpsiE[PSI_EYX - PSI_EXY] + ox);
        pzx = load_v<V>(p.fpsiE[PSI_EZX - PSI_EXY] + ox);
      }
    }
    if (sxn) {
      const long long o = ((long long)imn * ny + y) * nz + z0;
      xcn = __ldg(p.pml.tab[0][TC] + x + S);
      if (KAPPA) xkn = __ldg(p.pml.tab[0][TK] + x + S);
      nyx = load_v<V>(p.pml.in[QYX] + o);
      nzx = load_v<V>(p.pml.in[QZX] + o);
    }
  }
  if (YS) {
    const int jm = slab_map(y, ny, p.pml.P[1]);
    const int jmn = ey ? slab_map(y + S, ny, p.pml.P[1]) : -1;
    sy = jm >= 0;
    syn = jmn >= 0;
    if (sy) {
      oy = ((long long)x * p.pml.L[1] + jm) * nz + z0;
      yb = __ldg(p.pml.tab[1][TB] + y);
      yc = __ldg(p.pml.tab[1][TC] + y);
      if (KAPPA) yk = __ldg(p.pml.tab[1][TK] + y);
      qxy = load_v<V>(p.pml.in[QXY] + oy);
      qzy = load_v<V>(p.pml.in[QZY] + oy);
      if (P1) {
        pxy = load_v<V>(p.fpsiE[PSI_EXY - PSI_EXY] + oy);
        pzy = load_v<V>(p.fpsiE[PSI_EZY - PSI_EXY] + oy);
      }
    }
    if (syn) {
      const long long o = ((long long)x * p.pml.L[1] + jmn) * nz + z0;
      ycn = __ldg(p.pml.tab[1][TC] + y + S);
      if (KAPPA) ykn = __ldg(p.pml.tab[1][TK] + y + S);
      nxy = load_v<V>(p.pml.in[QXY] + o);
      nzy = load_v<V>(p.pml.in[QZY] + o);
    }
  }
  if (ZS) {
    oz = ((long long)x * ny + y) * p.pml.L[2];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      km[k] = slab_map(z0 + k, nz, p.pml.P[2]);
      sz[k] = km[k] >= 0;
      if (sz[k]) {
        zb[k] = __ldg(p.pml.tab[2][TB] + z0 + k);
        zc[k] = __ldg(p.pml.tab[2][TC] + z0 + k);
        if (KAPPA) zk[k] = __ldg(p.pml.tab[2][TK] + z0 + k);
        qxz[k] = p.pml.in[QXZ][oz + km[k]];
        qyz[k] = p.pml.in[QYZ][oz + km[k]];
        if (P1) {
          pxz[k] = p.fpsiE[PSI_EXZ - PSI_EXY][oz + km[k]];
          pyz[k] = p.fpsiE[PSI_EYZ - PSI_EXY][oz + km[k]];
        }
      }
    }
    const int kn = ez ? slab_map(zn, nz, p.pml.P[2]) : -1;
    szn = kn >= 0;
    if (szn) {
      zcn = __ldg(p.pml.tab[2][TC] + zn);
      if (KAPPA) zkn = __ldg(p.pml.tab[2][TK] + zn);
      nxz = p.pml.in[QXZ][oz + kn];
      nyz = p.pml.in[QYZ][oz + kn];
    }
  }

  // z differences of the vector's cells and, at the end the neighbour is on,
  // of the cell beyond
  float d1[V + 1], d2[V + 1];
  constexpr int B = P1 ? 0 : 1;  // cell k is entry k + B, the neighbour the other end
  constexpr int E = P1 ? V : 0;
  d1[E] = ez && oky ? adj_diff<KAPPA>(szn, -(wz * a0z), zkn, zcn, nxz) : 0.0f;
  d2[E] = ez && okx ? adj_diff<KAPPA>(szn, wz * a1z, zkn, zcn, nyz) : 0.0f;
  float d0[V], d3[V], d4[V], d5[V];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int z = z0 + k;
    const bool okz = (CP && !ZS) || (P1 ? z >= 1 : z < nz - 1);
    const bool u0 = oky && okz, u1 = okx && okz, u2 = okx && oky;
    const float x0 = w.v[k] * a0.v[k], x1 = w.v[k] * a1.v[k], x2 = w.v[k] * a2.v[k];
    d0[k] = u0 ? adj_diff<KAPPA>(sy, x0, yk, yc, qxy.v[k]) : 0.0f;
    d1[k + B] = u0 ? adj_diff<KAPPA>(sz[k], -x0, zk[k], zc[k], qxz[k]) : 0.0f;
    d2[k + B] = u1 ? adj_diff<KAPPA>(sz[k], x1, zk[k], zc[k], qyz[k]) : 0.0f;
    d3[k] = u1 ? adj_diff<KAPPA>(sx, -x1, xk, xc, qyx.v[k]) : 0.0f;
    d4[k] = u2 ? adj_diff<KAPPA>(sx, x2, xk, xc, qzx.v[k]) : 0.0f;
    d5[k] = u2 ? adj_diff<KAPPA>(sy, -x2, yk, yc, qzy.v[k]) : 0.0f;
    if (P1) {  // dJ/dcb
      double g = 0.0;
      const float c2z = k > 0 ? f1.v[(k + V - 1) % V] : f1z, c0z = k > 0 ? f0.v[(k + V - 1) % V] : f0z;
      auto term = [&](bool up, float e, float da, float db, float ka, float kb, float pa, float pb) {
        if (!up) return;
        const float X = (KAPPA ? ka * da - kb * db : da - db) + (pa - pb);
        g += (double)e * (double)damp.v[k] * (double)X;
      };
      term(u0, a0.v[k], f2.v[k] - f2y.v[k], f1.v[k] - c2z, yk, zk[k], pxy.v[k], pxz[k]);
      term(u1, a1.v[k], f0.v[k] - c0z, f2.v[k] - f2x.v[k], zk[k], xk, pyz[k], pyx.v[k]);
      term(u2, a2.v[k], f1.v[k] - f1x.v[k], f0.v[k] - f0y.v[k], xk, yk, pzx.v[k], pzy.v[k]);
      gc[k] += g;
    }
    // psi of the cell: b (psi + u); unchanged where the component is not updated
    if (XS && u1) qyx.v[k] = xb * (qyx.v[k] - x1);
    if (XS && u2) qzx.v[k] = xb * (qzx.v[k] + x2);
    if (YS && u0) qxy.v[k] = yb * (qxy.v[k] + x0);
    if (YS && u2) qzy.v[k] = yb * (qzy.v[k] - x2);
    if (ZS && u0) qxz[k] = zb[k] * (qxz[k] - x0);
    if (ZS && u1) qyz[k] = zb[k] * (qyz[k] + x1);
  }
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int z = z0 + k;
    const bool okz = (CP && !ZS) || (P1 ? z >= 1 : z < nz - 1);
    const float n0 = ey && okz ? adj_diff<KAPPA>(syn, wy.v[k] * a0y.v[k], ykn, ycn, nxy.v[k]) : 0.0f;
    const float n5 = ey && okx ? adj_diff<KAPPA>(syn, -(wy.v[k] * a2y.v[k]), ykn, ycn, nzy.v[k]) : 0.0f;
    const float n3 = ex && okz ? adj_diff<KAPPA>(sxn, -(wx.v[k] * a1x.v[k]), xkn, xcn, nyx.v[k]) : 0.0f;
    const float n4 = ex && oky ? adj_diff<KAPPA>(sxn, wx.v[k] * a2x.v[k], xkn, xcn, nzx.v[k]) : 0.0f;
    if (P1) {
      g0.v[k] = g0.v[k] + (d2[k] - d2[k + 1]) + (d5[k] - n5);
      g1.v[k] = g1.v[k] + (d1[k] - d1[k + 1]) + (d4[k] - n4);
      g2.v[k] = g2.v[k] + (d0[k] - n0) + (d3[k] - n3);
    } else {
      g0.v[k] = damp.v[k] * g0.v[k] + ((d2[k] - d2[k + 1]) + (n5 - d5[k]));
      g1.v[k] = damp.v[k] * g1.v[k] + ((d1[k] - d1[k + 1]) + (n4 - d4[k]));
      g2.v[k] = damp.v[k] * g2.v[k] + ((n0 - d0[k]) + (n3 - d3[k]));
    }
  }

  store_v<V>(G[0] + idx, g0);
  store_v<V>(G[1] + idx, g1);
  store_v<V>(G[2] + idx, g2);
  if (P1) {
    if constexpr (V == 2) *reinterpret_cast<double2*>(p.gcb + idx) = make_double2(gc[0], gc[1]);
    else p.gcb[idx] = gc[0];
  }
  if (XS && sx) {
    store_v<V>(p.pml.out[QYX] + ox, qyx);
    store_v<V>(p.pml.out[QZX] + ox, qzx);
  }
  if (YS && sy) {
    store_v<V>(p.pml.out[QXY] + oy, qxy);
    store_v<V>(p.pml.out[QZY] + oy, qzy);
  }
  if (ZS) {
#pragma unroll
    for (int k = 0; k < V; ++k)
      if (sz[k]) {
        p.pml.out[QXZ][oz + km[k]] = qxz[k];
        p.pml.out[QYZ][oz + km[k]] = qyz[k];
      }
  }
}

template <bool P1, int MODE, int V, bool KAPPA, bool CBARR, int REG>
__device__ __forceinline__ void adj_region(const Adj3D& p, const SweepPlan& s, int x, int b) {
  constexpr bool YS = REG == 0 || REG == 2, ZS = REG < 2;
  const int t = b * ADJ_THREADS + (int)threadIdx.x;
  if (t >= s.r[REG].n) return;
  const int j = (int)fdiv((uint32_t)t, s.r[REG].dw);
  const int k = (t - j * s.r[REG].w) * V;
  const int y = YS ? (j < s.y0 ? j : j + (s.y1 - s.y0)) : s.y0 + j;
  const int z = ZS ? (k < s.z0 ? k : k + (s.z1 - s.z0)) : s.z0 + k;
  if (x < s.x0 || x >= s.x1) adj_cells<P1, MODE, V, KAPPA, CBARR, true, YS, ZS>(p, x, y, z);
  else adj_cells<P1, MODE, V, KAPPA, CBARR, false, YS, ZS>(p, x, y, z);
}

// Work split of a plane as in the forward passes (SweepPlan), with one more
// cell of each slab's inner side in its region: a cell's neighbour is read too.
template <bool P1, int MODE, int V, bool KAPPA, bool CBARR>
__global__ void __launch_bounds__(ADJ_THREADS, 5)
    k3a_pass(const __grid_constant__ Adj3D p, const __grid_constant__ SweepPlan s) {
  grid_dep_wait();
  grid_dep_launch_dependents();
  for (int x = blockIdx.y; x < p.nx; x += gridDim.y) {  // (one plane, below 65,536 of them)
    int b = blockIdx.x;
    if (MODE != MODE_CPML) {
      const int t = b * ADJ_THREADS + (int)threadIdx.x;
      if (t >= s.r[3].n) return;
      const int y = (int)fdiv((uint32_t)t, s.r[3].dw);
      adj_cells<P1, MODE, V, KAPPA, CBARR, false, false, false>(p, x, y, (t - y * s.r[3].w) * V);
    } else if (b < s.r[0].nb) {
      adj_region<P1, MODE, V, KAPPA, CBARR, 0>(p, s, x, b);
    } else if ((b -= s.r[0].nb) < s.r[1].nb) {
      adj_region<P1, MODE, V, KAPPA, CBARR, 1>(p, s, x, b);
    } else if ((b -= s.r[1].nb) < s.r[2].nb) {
      adj_region<P1, MODE, V, KAPPA, CBARR, 2>(p, s, x, b);
    } else {
      adj_region<P1, MODE, V, KAPPA, CBARR, 3>(p, s, x, b - s.r[2].nb);
    }
  }
}

// adjoint seeds of the probe readout after step n: lambda[comp][cell] += g[p]
struct Lam6 {
  float* f[6];  // adjoint of Ex, Ey, Ez, Hx, Hy, Hz
};
static __global__ void k3a_seed(Lam6 lam, const long long* cell, const int* comp, int n_probes,
                         const float* grad_row) {
  grid_dep_wait();
  grid_dep_launch_dependents();
  // one thread: probes may repeat a cell, so add in order
  if (blockIdx.x == 0 && threadIdx.x == 0)
    for (int k = 0; k < n_probes; ++k) lam.f[comp[k]][cell[k]] += grad_row[k];
}

// dJ/deps_r = dJ/dcb * dcb/deps_r = -dJ/dcb * cb^2 / coef_e
static __global__ void k3a_finish(const double* gcb, const float* cb, float cb_const, double coef_e,
                           float* grad_eps, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double c = cb ? (double)cb[i] : (double)cb_const;
    grad_eps[i] = (float)(-gcb[i] * c * c / coef_e);
  }
}

}  // namespace jxf
