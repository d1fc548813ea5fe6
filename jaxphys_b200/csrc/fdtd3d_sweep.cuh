// In-place two-pass 3D Yee step for sm_100a ("sweeps").
//
// A step is two launches over one buffer set: the H pass
//   H^{n+1/2} = H^{n-1/2} - a curl E^n
// and the E pass
//   E^{n+1} = (E^n + cb curl H^{n+1/2}) damping + sources
// (jaxphys src/neurosim/em/fdtd3d.py:303-369).  No block waits for another
// inside a launch: a thread owns V consecutive z cells of one plane, loads
// them with their neighbours and writes its own cells back.
//
// Why two passes in place, where the marching kernel needs one: the fields of
// a 128^3 grid and its psi are 70 MB in one buffer set, which stays in the
// 126 MB L2 from step to step, while the marching kernel's two sets do not
// fit, and its march is a serial chain of planes with a barrier in each.  Here
// every load of a thread is in flight at once and there is no barrier.  What
// bounds the passes is the L1 of each SM (0.67 busy in a profiled 128^3 CPML
// pass of 17.7 us that takes 12.2 unprofiled) and the wait for its loads, at
// 66 and 73 bytes per cell, 12 TB/s, in the two passes; below 64^3 the two
// launches of a step (about 2.4 us each).  Measured per step on one B200,
// against the kernels used before: 128^3 10-layer CPML 24.7 us (marching
// kernel 41.1), 64^3 8-layer CPML 8.1 us (10.5), 60^3 absorbing 5.0 us (11),
// 96 x 80 x 64 periodic 6.5 us (per-cell kernels, three launches: 18),
// 75 x 90 x 61 CPML 11.8 us (24).
// Above L2 size it is bound by DRAM (76 bytes per cell and step against 52),
// and the autotuner takes the marching or the blocked kernel there.
#pragma once

#include "fdtd3d_kernels.cuh"

namespace jxf {

// Threads per block.  128: a block of a CPML region holds few rows, and more
// threads leave more of them idle.  With one or two cells per thread and no
// slabs a block of 128 is done so soon that dispatching blocks bounds the pass
// (128^3 of one cell per thread, absorbing: 35.6 us a step against 22.4 with
// 256 threads).
__host__ __device__ constexpr int sweep_threads(int mode, int v0) {
  return mode != MODE_CPML && v0 < 4 ? 256 : 128;
}
// Blocks per SM the compiler must leave registers for: 64 a thread (CPML: 128).
// Without the bound it keeps fewer loads in flight to fit more blocks, 17.1
// against 14.3 us a step for the absorbing 128^3 grid; a tighter bound spills
// the CPML kernel.
__host__ __device__ constexpr int sweep_min_blocks(int mode, int v0) {
  return (mode == MODE_CPML ? 512 : 1024) / sweep_threads(mode, v0);
}

// Work split of one plane x.  CPML grids: the cells of a plane fall in four
// regions by whether their y / z lies in a psi slab, each cut into blocks of
// sweep_threads() threads (V0 cells per thread outside the z slabs, V1 inside),
// so that a block runs code for its slabs alone: with one code for all, every
// warp of a 128-cell row holds z-slab lanes and pays for the CPML update (37
// against 25 us a step at 128^3).  Other grids: one region.
struct SweepRegion {
  int n;       // work items (threads) of the region in a plane
  int w;       // items per row
  int nb;      // blocks
  FastDiv dw;  // divide by w
};
struct SweepPlan {
  SweepRegion r[4];  // [0 y slab + z slab, 1 z slab, 2 y slab, 3 neither]
  int y0, y1;        // rows outside the y slabs: [y0, y1)
  int z0, z1;        // columns of the regions outside the z slabs: [z0, z1)
  int x0, x1;        // planes outside the x slabs: [x0, x1)
  int nblk;          // blocks per plane
  // soft sources of the E pass: cells grouped by block (CSR over plane * nblk
  // + block), terms of a cell in list order
  const int* src_ptr;
  const SrcCell* src_cell;
  const SrcTerm* src_term;
};

// Where an E pass leaves H and the E psi of the step as well (the adjoint's
// recompute keeps them after every step; a copy would read them again).
struct SweepSnap {
  static constexpr bool on = true;
  float* h[3];
  float* psi[6];  // EXY .. EZY
};
struct NoSnap {
  static constexpr bool on = false;
};

template <int V>
struct VecF {
  float v[V];
};
template <int V>
__device__ __forceinline__ VecF<V> load_v(const float* p) {
  VecF<V> r;
  if constexpr (V == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    r.v[0] = t.x;
    r.v[1] = t.y;
    r.v[2] = t.z;
    r.v[3] = t.w;
  } else if constexpr (V == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    r.v[0] = t.x;
    r.v[1] = t.y;
  } else {
    r.v[0] = *p;
  }
  return r;
}
template <int V>
__device__ __forceinline__ void store_v(float* p, const VecF<V>& r) {
  if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
  else if constexpr (V == 2) *reinterpret_cast<float2*>(p) = make_float2(r.v[0], r.v[1]);
  else *p = r.v[0];
}

// One thread's cells (x, y, z0 .. z0+V-1) of the H pass (H = true: forward
// differences of E) or the E pass (backward differences of H).  XS / YS / ZS
// (CPML): the cells may lie in that axis's psi slab; outside it neither psi
// nor that axis's outer index range can occur, so their code compiles away.
// Every load is issued before the first store: the psi arrays are updated in
// place, and a store in between would hold back the loads behind it.
template <bool H, int MODE, int V, bool KAPPA, bool CBARR, bool XS, bool YS, bool ZS, class SNAP>
__device__ __forceinline__ void sweep_cells(const Step3D& p, const SNAP& sn, int x, int y, int z0) {
  constexpr bool CP = MODE == MODE_CPML;
  constexpr bool PER = MODE == MODE_PERIODIC;
  constexpr int F = H ? 0 : 3, G = H ? 3 : 0;  // fields read with neighbours / updated
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  const int plane = ny * nz;
  const long long idx = (long long)x * plane + (y * nz + z0);
  // the component updates need a neighbour along x / y (interior of the slabs'
  // complement: always there)
  const bool xn = (CP && !XS) || PER || (H ? x < nx - 1 : x >= 1);
  const bool yn = (CP && !YS) || PER || (H ? y < ny - 1 : y >= 1);
  const bool ze = (CP && !ZS) || (H ? z0 + V < nz : z0 >= 1);  // outer z neighbour in range
  // neighbour cells; one that does not exist is read at the cell itself and
  // not used (loads without a condition can all be in flight together)
  long long ix = !xn ? idx : (H ? idx + plane : idx - plane);
  long long iy = !yn ? idx : (H ? idx + nz : idx - nz);
  long long iz = !ze ? idx : (H ? idx + V : idx - 1);
  if (PER) {
    const long long dx = (long long)(nx - 1) * plane, dy = (long long)(ny - 1) * nz;
    if (H ? x == nx - 1 : x == 0) ix = H ? idx - dx : idx + dx;
    if (H ? y == ny - 1 : y == 0) iy = H ? idx - dy : idx + dy;
    if (!ze) iz = H ? idx - (nz - V) : idx + (nz - 1);
  }
  const VecF<V> f0 = load_v<V>(p.in[F] + idx);
  const VecF<V> f1 = load_v<V>(p.in[F + 1] + idx);
  const VecF<V> f2 = load_v<V>(p.in[F + 2] + idx);
  const VecF<V> f0y = load_v<V>(p.in[F] + iy), f2y = load_v<V>(p.in[F + 2] + iy);
  const VecF<V> f1x = load_v<V>(p.in[F + 1] + ix), f2x = load_v<V>(p.in[F + 2] + ix);
  // (from the next lane by a shuffle instead: 128^3 CPML 26.6 us a step, not 24.3)
  const float f0z = p.in[F][iz], f1z = p.in[F + 1][iz];
  VecF<V> g0 = load_v<V>(p.in[G] + idx);
  VecF<V> g1 = load_v<V>(p.in[G + 1] + idx);
  VecF<V> g2 = load_v<V>(p.in[G + 2] + idx);
  VecF<V> cb;
  if (!H && CBARR) cb = load_v<V>(p.cb + idx);

  // psi of the cells and the coefficients of their positions
  constexpr int Q = H ? 0 : PSI_EXY;
  constexpr int TB = H ? TAB_BH : TAB_BE, TC = H ? TAB_CH : TAB_CE, TK = H ? TAB_IKH : TAB_IKE;
  VecF<V> qxy, qzy, qyx, qzx, zb, zc, zk;
  constexpr int ZP = V > 1 ? 2 : 1;
  float qxz[V], qyz[V];
  int km[V], kp[V / ZP];
  float xb = 0.0f, xc = 0.0f, xk = 1.0f, yb = 0.0f, yc = 0.0f, yk = 1.0f;
  int ox = 0, oy = 0, oz = 0;
  if (XS) {
    const int im = slab_map(x, nx, p.pml.P[0]);
    ox = (im * ny + y) * nz + z0;
    xb = __ldg(p.pml.tab[0][TB] + x);
    xc = __ldg(p.pml.tab[0][TC] + x);
    if (KAPPA) xk = __ldg(p.pml.tab[0][TK] + x);
    qyx = load_v<V>(p.pml.in[Q + PSI_HYX] + ox);
    qzx = load_v<V>(p.pml.in[Q + PSI_HZX] + ox);
  }
  if (YS) {
    const int jm = slab_map(y, ny, p.pml.P[1]);
    oy = (x * p.pml.L[1] + jm) * nz + z0;
    yb = __ldg(p.pml.tab[1][TB] + y);
    yc = __ldg(p.pml.tab[1][TC] + y);
    if (KAPPA) yk = __ldg(p.pml.tab[1][TK] + y);
    qxy = load_v<V>(p.pml.in[Q + PSI_HXY] + oy);
    qzy = load_v<V>(p.pml.in[Q + PSI_HZY] + oy);
  }
  // psi of the z slabs, in pairs (V > 1: nz and so the slab rows are even).
  // A z region starts and ends on a multiple of V, so a few of its cells lie
  // outside the slab: they read a psi entry that they do not use.
  if (ZS) {
    oz = (x * ny + y) * p.pml.L[2];
    zb = load_v<V>(p.pml.tab[2][TB] + z0);
    zc = load_v<V>(p.pml.tab[2][TC] + z0);
    if (KAPPA) zk = load_v<V>(p.pml.tab[2][TK] + z0);
#pragma unroll
    for (int k = 0; k < V; ++k) km[k] = slab_map(z0 + k, nz, p.pml.P[2]);
#pragma unroll
    for (int k = 0; k < V; k += ZP) {
      int o = km[k];
      if (ZP == 2 && o < 0) o = km[(k + 1) % V] - 1;
      kp[k / ZP] = oz + max(o, 0);
      const VecF<ZP> u = load_v<ZP>(p.pml.in[Q + PSI_HXZ] + kp[k / ZP]);
      const VecF<ZP> v = load_v<ZP>(p.pml.in[Q + PSI_HYZ] + kp[k / ZP]);
#pragma unroll
      for (int i = 0; i < ZP; ++i) {
        qxz[k + i] = u.v[i];
        qyz[k + i] = v.v[i];
      }
    }
  }

#pragma unroll
  for (int k = 0; k < V; ++k) {
    // d1 / d2: the two differences of each component's curl
    float d1x, d2x, d1y, d2y, d1z, d2z;
    if (H) {
      d1x = fsub(f2y.v[k], f2.v[k]);
      d2x = fsub(k + 1 < V ? f1.v[(k + 1) % V] : f1z, f1.v[k]);
      d1y = fsub(k + 1 < V ? f0.v[(k + 1) % V] : f0z, f0.v[k]);
      d2y = fsub(f2x.v[k], f2.v[k]);
      d1z = fsub(f1x.v[k], f1.v[k]);
      d2z = fsub(f0y.v[k], f0.v[k]);
    } else {
      d1x = fsub(f2.v[k], f2y.v[k]);
      d2x = fsub(f1.v[k], k > 0 ? f1.v[(k + V - 1) % V] : f1z);
      d1y = fsub(f0.v[k], k > 0 ? f0.v[(k + V - 1) % V] : f0z);
      d2y = fsub(f2.v[k], f2x.v[k]);
      d1z = fsub(f1.v[k], f1x.v[k]);
      d2z = fsub(f0.v[k], f0y.v[k]);
    }
    const bool zn = (CP && !ZS) || PER || (H ? z0 + k < nz - 1 : z0 + k >= 1);
    const bool ux = yn && zn, uy = xn && zn, uz = xn && yn;
    const float c = H ? p.a : (CBARR ? cb.v[k] : p.cb_const);
    if (XS || YS || ZS) {
      float p1x = 0.0f, p2x = 0.0f, p1y = 0.0f, p2y = 0.0f, p1z = 0.0f, p2z = 0.0f;
      if (YS) {
        if (zn) qxy.v[k] = psi_next(yb, qxy.v[k], yc, d1x);
        p1x = qxy.v[k];
        p2z = qzy.v[k] = psi_next(yb, qzy.v[k], yc, d2z);
      }
      if (XS) {
        if (zn) qyx.v[k] = psi_next(xb, qyx.v[k], xc, d2y);
        p2y = qyx.v[k];
        p1z = qzx.v[k] = psi_next(xb, qzx.v[k], xc, d1z);
      }
      const bool zon = ZS && km[k] >= 0;
      const float zkk = (KAPPA && ZS) ? zk.v[k] : 1.0f;
      if (ZS) {
        if (zn) qxz[k] = psi_next(zb.v[k], qxz[k], zc.v[k], d2x);
        if (zn) qyz[k] = psi_next(zb.v[k], qyz[k], zc.v[k], d1y);
        p2x = zon ? qxz[k] : 0.0f;
        p1y = zon ? qyz[k] : 0.0f;
      }
      if (H) {
        if (ux) g0.v[k] = h_sel<KAPPA>(g0.v[k], c, d1x, d2x, YS, zon, p1x, p2x, yk, zkk);
        if (uy) g1.v[k] = h_sel<KAPPA>(g1.v[k], c, d1y, d2y, zon, XS, p1y, p2y, zkk, xk);
        if (uz) g2.v[k] = h_sel<KAPPA>(g2.v[k], c, d1z, d2z, XS, YS, p1z, p2z, xk, yk);
      } else {
        if (ux) g0.v[k] = e_sel<KAPPA>(g0.v[k], c, d1x, d2x, YS, zon, p1x, p2x, yk, zkk);
        if (uy) g1.v[k] = e_sel<KAPPA>(g1.v[k], c, d1y, d2y, zon, XS, p1y, p2y, zkk, xk);
        if (uz) g2.v[k] = e_sel<KAPPA>(g2.v[k], c, d1z, d2z, XS, YS, p1z, p2z, xk, yk);
      }
    } else if (H) {
      if (ux) g0.v[k] = h_plain(g0.v[k], c, d1x, d2x);
      if (uy) g1.v[k] = h_plain(g1.v[k], c, d1y, d2y);
      if (uz) g2.v[k] = h_plain(g2.v[k], c, d1z, d2z);
    } else {
      if (ux) g0.v[k] = e_plain(g0.v[k], c, d1x, d2x);
      if (uy) g1.v[k] = e_plain(g1.v[k], c, d1y, d2y);
      if (uz) g2.v[k] = e_plain(g2.v[k], c, d1z, d2z);
    }
    if (!H && MODE == MODE_ABSORB) {
      const float f =
          fmul(fmul(__ldg(p.damp[0] + x), __ldg(p.damp[1] + y)), __ldg(p.damp[2] + z0 + k));
      g0.v[k] = fmul(g0.v[k], f);
      g1.v[k] = fmul(g1.v[k], f);
      g2.v[k] = fmul(g2.v[k], f);
    }
  }

  store_v<V>(p.out[G] + idx, g0);
  store_v<V>(p.out[G + 1] + idx, g1);
  store_v<V>(p.out[G + 2] + idx, g2);
  auto put_psi = [&](float* const* psi) {  // the six arrays of the pass
    if (XS && xn) {
      store_v<V>(psi[PSI_HYX] + ox, qyx);
      if (yn) store_v<V>(psi[PSI_HZX] + ox, qzx);
    }
    if (YS && yn) {
      store_v<V>(psi[PSI_HXY] + oy, qxy);
      if (xn) store_v<V>(psi[PSI_HZY] + oy, qzy);
    }
    if constexpr (ZS) {
#pragma unroll
      for (int k = 0; k < V; k += ZP) {
        float* const u = psi[PSI_HXZ] + kp[k / ZP];
        float* const v = psi[PSI_HYZ] + kp[k / ZP];
        const int k1 = (k + ZP - 1) % V;
        if (km[k] >= 0 && km[k1] >= 0) {
          if (ZP == 2) {
            if (yn) *reinterpret_cast<float2*>(u) = make_float2(qxz[k], qxz[k1]);
            if (xn) *reinterpret_cast<float2*>(v) = make_float2(qyz[k], qyz[k1]);
          } else {
            if (yn) *u = qxz[k];
            if (xn) *v = qyz[k];
          }
        } else if (ZP == 2 && (km[k] >= 0 || km[k1] >= 0)) {
          const int i = km[k] >= 0 ? 0 : 1;
          if (yn) u[i] = i ? qxz[k1] : qxz[k];
          if (xn) v[i] = i ? qyz[k1] : qyz[k];
        }
      }
    }
  };
  if (CP) put_psi(p.pml.out + Q);
  if constexpr (SNAP::on && !H) {
    store_v<V>(sn.h[0] + idx, f0);
    store_v<V>(sn.h[1] + idx, f1);
    store_v<V>(sn.h[2] + idx, f2);
    if (CP) put_psi(sn.psi);
  }
}

// One block of region REG (SweepPlan::r) of plane x.
template <bool H, int MODE, int V0, int V1, bool KAPPA, bool CBARR, int REG, class SNAP>
__device__ __forceinline__ void sweep_region(const Step3D& p, const SweepPlan& s, const SNAP& sn,
                                             int x, int b) {
  constexpr bool YS = REG == 0 || REG == 2, ZS = REG < 2;
  constexpr int V = ZS ? V1 : V0, NT = sweep_threads(MODE, V0);
  const int t = b * NT + (int)threadIdx.x;
  if (t >= s.r[REG].n) return;
  const int j = (int)fdiv((uint32_t)t, s.r[REG].dw);
  const int k = (t - j * s.r[REG].w) * V;
  const int y = YS ? (j < s.y0 ? j : j + (s.y1 - s.y0)) : s.y0 + j;
  const int z = ZS ? (k < s.z0 ? k : k + (s.z1 - s.z0)) : s.z0 + k;
  if (x < s.x0 || x >= s.x1) sweep_cells<H, MODE, V, KAPPA, CBARR, true, YS, ZS>(p, sn, x, y, z);
  else sweep_cells<H, MODE, V, KAPPA, CBARR, false, YS, ZS>(p, sn, x, y, z);
}

// Block b of plane x of one grid.
template <bool H, int MODE, int V0, int V1, bool KAPPA, bool CBARR, class SNAP = NoSnap>
__device__ __forceinline__ void sweep_block(const Step3D& p, const SweepPlan& s, int x, int b,
                                            const SNAP& sn = SNAP()) {
  constexpr int NT = sweep_threads(MODE, V0);
  // probes of the state after the previous step: its E components are final
  // until this step's E pass, its H components were recorded by its E pass.
  // Spread over the planes: one block for all of them took 150 us a step for
  // 16,384 probes (33^3 CPML: 6.2 us a step with one probe); over all blocks,
  // the test in every block costs 1.5 % of a 128^3 CPML step.  (With the whole
  // test up front and the loop not unrolled, the kernels keep the registers
  // they have without it: two more cost the one-cell CPML kernels a block per
  // SM, 155 against 140 us a step for 60,000 x 8 x 9 cells.)
  if (p.probe_out != nullptr && b == 0 && x * NT < p.n_probes) {
#pragma unroll 1
    for (int i = x * NT + (int)threadIdx.x; i < p.n_probes; i += p.nx * NT) {
      const int c = p.probe_comp[i];
      if ((c < 3) == H) p.probe_out[i] = p.in[c][p.probe_cell[i]];
    }
  }
  int s0 = 0, s1 = 0;
  if (!H && s.src_ptr != nullptr) {
    const int* q = s.src_ptr + (x * s.nblk + b);
    s0 = __ldg(q);
    s1 = __ldg(q + 1);
  }
  if (MODE != MODE_CPML) {
    const int t = b * NT + (int)threadIdx.x;
    if (t < s.r[3].n) {
      const int y = (int)fdiv((uint32_t)t, s.r[3].dw);
      sweep_cells<H, MODE, V0, KAPPA, CBARR, false, false, false>(p, sn, x, y,
                                                                  (t - y * s.r[3].w) * V0);
    }
  } else if (b < s.r[0].nb) {
    sweep_region<H, MODE, V0, V1, KAPPA, CBARR, 0>(p, s, sn, x, b);
  } else if ((b -= s.r[0].nb) < s.r[1].nb) {
    sweep_region<H, MODE, V0, V1, KAPPA, CBARR, 1>(p, s, sn, x, b);
  } else if ((b -= s.r[1].nb) < s.r[2].nb) {
    sweep_region<H, MODE, V0, V1, KAPPA, CBARR, 2>(p, s, sn, x, b);
  } else {
    sweep_region<H, MODE, V0, V1, KAPPA, CBARR, 3>(p, s, sn, x, b - s.r[2].nb);
  }
  // soft sources of the block's cells, after its E update
  if (!H && s0 < s1) {
    __syncthreads();
    for (int i = s0 + (int)threadIdx.x; i < s1; i += NT) {
      const SrcCell c = s.src_cell[i];
      float* f = p.out[c.comp] + c.cell;
      float v = *f;
      for (int k = 0; k < c.count; ++k) {
        const SrcTerm t = s.src_term[c.first + k];
        v = fadd(v, fmul(t.amp, p.wave[(long long)t.wave * p.wave_len + p.step]));
      }
      *f = v;
    }
  }
}

template <bool H, int MODE, int V0, int V1, bool KAPPA, bool CBARR>
__global__ void __launch_bounds__(sweep_threads(MODE, V0), sweep_min_blocks(MODE, V0))
    k3d_sweep(const __grid_constant__ Step3D p, const __grid_constant__ SweepPlan s) {
  grid_dep_wait();
  grid_dep_launch_dependents();
  sweep_block<H, MODE, V0, V1, KAPPA, CBARR>(p, s, blockIdx.y, blockIdx.x);
}

// E pass that leaves a snapshot too.
template <int MODE, int V0, int V1, bool KAPPA, bool CBARR>
__global__ void __launch_bounds__(sweep_threads(MODE, V0), sweep_min_blocks(MODE, V0))
    k3d_sweep_snap(const __grid_constant__ Step3D p, const __grid_constant__ SweepPlan s,
                   const __grid_constant__ SweepSnap sn) {
  grid_dep_wait();
  grid_dep_launch_dependents();
  sweep_block<false, MODE, V0, V1, KAPPA, CBARR, SweepSnap>(p, s, blockIdx.y, blockIdx.x, sn);
}

// The same pass over several grids of a batch in one launch.  Their parameters
// ride in the launch (constant memory): read from global memory they would put
// a dependent load in front of every block's first field load.
constexpr int SWEEP_GROUP = 8;
struct SweepGroup {
  int n;
  int end[SWEEP_GROUP];       // blocks of grids 0 .. k
  FastDiv dblk[SWEEP_GROUP];  // divide by a grid's blocks per plane
  Step3D p[SWEEP_GROUP];
  SweepPlan s[SWEEP_GROUP];
};
template <bool H, int MODE, int V0, int V1, bool KAPPA, bool CBARR>
__global__ void __launch_bounds__(sweep_threads(MODE, V0), sweep_min_blocks(MODE, V0))
    k3d_sweep_group(const __grid_constant__ SweepGroup g) {
  grid_dep_wait();
  grid_dep_launch_dependents();
  int k = 0;
  while ((int)blockIdx.x >= g.end[k]) ++k;
  const int b = (int)blockIdx.x - (k > 0 ? g.end[k - 1] : 0);
  const int x = (int)fdiv((uint32_t)b, g.dblk[k]);
  sweep_block<H, MODE, V0, V1, KAPPA, CBARR>(g.p[k], g.s[k], x, b - x * g.s[k].nblk);
}

}  // namespace jxf
